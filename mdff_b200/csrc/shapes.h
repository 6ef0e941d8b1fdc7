// shapes.h -- launch shapes that also size buffers: plain host arithmetic, no
// CUDA, so that a host test can run it over whole ranges of ions and meshes.
#pragma once
#include <algorithm>
#include <cstddef>

#ifdef __CUDACC__
#define MDFF_HD __host__ __device__
#else
#define MDFF_HD
#endif

namespace mdff {

inline int ceil_div(long a, long b) { return (int)((a + b - 1) / b); }

// ---------------------------------------------------------------------------
// FP64 structure factor of the single engine (k_rho_dm)

constexpr int kDmRows = 64;  // mesh rows per block

// n tiles (of four n) per pass over the ions, and passes: as many as their
// accumulators allow (registers: 8 a tile, 16 with dipoles).  Charges alone have
// one product per tile for the same loads of the ions' phases: 13700 ions, kz 20, two
// passes of three tiles 141 us, one of six 108 us.
inline int rho_dm_nt(int kz, bool hm) {
  const int most = hm ? 5 : 8, tiles = kz / 4 + 1, groups = (tiles + most - 1) / most;
  return (tiles + groups - 1) / groups;
}
// shared memory of k_rho_dm staging ci ions a buffer, and the largest ci (32, 16
// or 8) whose two buffers fit half an SM (0: the mesh does not fit)
inline size_t rho_dm_smem(int kx, int ky, int nt, int ci) {
  const size_t ent = (size_t)(kx + 1 + ky + 1 + 4 * nt);
  const size_t b = 2 * (ent * (ci + 4) * 16 + (size_t)ci * 32), red = 8 * 32 * 8 * 8;
  return b > red ? b : red;
}
inline int rho_dm_ci(int kx, int ky, int nt) {
  for (int ci = 32; ci >= 8; ci /= 2)
    if (rho_dm_smem(kx, ky, nt, ci) <= (ci > 8 ? 110 * 1024 : 227 * 1024)) return ci;
  return 0;
}

// ion chunks wanted: one block per SM over (row blocks x chunks x n passes)
inline int rho_dm_want(int nsm, int nrows, int groups) {
  return std::max(1, (nsm > 0 ? nsm : 148) / std::max(ceil_div(nrows, kDmRows) * std::max(groups, 1), 1));
}
// ions per chunk (at least 16, a multiple of 8) and the chunks of nion ions.  The
// count is not monotone in nion: 148 SMs, 181 rows, 5103 ions are 46 chunks of 112, 3402
// of them 48 chunks of 72.
inline void rho_dm_split(int nion, int want, int* chunk, int* nchunk) {
  *chunk = std::max(16, ceil_div(ceil_div(nion, want), 8) * 8);
  *nchunk = ceil_div(nion, *chunk);
}
// most chunks of any subset of natm ions: a chunk holds at least nion / want ions
// and at least 16
inline int rho_dm_most(int natm, int want) { return std::min(want, ceil_div(natm, 16)); }

// ---------------------------------------------------------------------------
// Optional caches of pair terms: an eighth of the device's memory at most and half
// of what is free, so that later allocations, other handles and the caller's own
// tensors find room.
inline size_t pair_cache_room(size_t mfree, size_t mtotal) { return std::min(mtotal / 8, mfree / 2); }
inline bool pair_cache_fits(size_t bytes, size_t mfree, size_t mtotal) { return bytes <= pair_cache_room(mfree, mtotal); }

// ---------------------------------------------------------------------------
// reciprocal sums of the batched engine (brho_t, bfld_t)

constexpr int kBStage = 16384;  // least bytes of the shared staging buffer

// bytes of an ion's phase record: X, Y, then (c, s) of n = 0..kz padded with
// zeros to whole tiles of brho (4 n) and steps of bfld (2 n, at least 3 steps);
// 32 mod 128, so that the lanes of a fragment load hit distinct banks
MDFF_HD inline int brec_bytes(int kx, int ky, int kz) {
  const int z1 = (kz / 4 + 1) * 64, z2 = (kz / 2 < 2 ? 3 : kz / 2 + 1) * 32;
  const int b = (kx + 1 + ky + 1) * 16 + (z1 > z2 ? z1 : z2);
  return (b + 95) / 128 * 128 + 32;
}

// The staging buffer of brho_t: the weights (nw of 32 bytes for each of cnt ions) lie in
// its first `weights` bytes when they take at most a third of it and leave two buffers
// of four records of rs bytes (a step takes four ions), else in the field's scratch (weights
// = 0); ch: records per buffer, at most 32, fewer than four only where the whole
// buffer has no room for eight records (kx + ky above 110 in the least buffer).
struct BStaging {
  int weights, ch;
};
MDFF_HD inline BStaging brec_staging(int stage_bytes, int cnt, int nw, int rs) {
  const int bytes = (cnt * 32 * nw + 127) / 128 * 128;
  const bool in_stage = cnt * 32 * nw <= stage_bytes / 3 && (stage_bytes - bytes) / (2 * rs) >= 4;
  BStaging s;
  s.weights = in_stage ? bytes : 0;
  const int ch = (stage_bytes - s.weights) / (2 * rs);
  s.ch = ch >= 32 ? 32 : ch >= 4 ? ch / 4 * 4 : ch;
  return s;
}

}  // namespace mdff
