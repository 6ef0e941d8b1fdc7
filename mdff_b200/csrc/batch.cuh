// batch.cuh -- batched engforce: many independent configurations of uneven
// ion counts in one persistent kernel.
//
// The reference evaluates one configuration per engforce call
// (engforce_driver.f90:102-190); a batch of small boxes would leave a B200
// mostly idle, one launch sequence per box.  Here one thread-block cluster of
// C CTAs owns one configuration at a time and takes the next one from a
// device work queue (configurations are queued in descending cost order, so
// the tail is short).  Inside a cluster each CTA owns a slice of the ions (pair
// sums, forces, partial structure factors) and a slice of the polarisable ions
// (solver vectors and fields); the CTAs exchange vectors and partial sums
// through L2 and meet at hardware cluster barriers.  Boxes are small (the
// real-space cutoff is clamped to half the box, coulomb.f90:377-383): one FP32
// sweep over all pairs of a box writes each ion's partners within the cutoffs
// plus a margin, every pair loop walks those with the exact minimum image and
// inclusion test (the pair set and each pair's arithmetic are those of the
// list-based engine), and the dipole operator's pair tensor is formed once per
// box and cached.
//
// What bounds it: the FP64 pipe in the reciprocal products (batch_rec.cuh), L2
// latency in the pair loops, then the tail (the largest box on its cluster).
// Measured on one B200 against all-pairs loops with a phase recurrence per k
// tile and the pair tensor recomputed per operator, each with its default shape:
// 256 boxes of 64-1000 ions, mixed, 28.1 -> 4.9 ms; 24 boxes of 64-300 ions,
// FP64, 3.7 -> 0.7 ms; 64 MgO boxes of 216-512 ions, FP64 at 1e-11, 9.6 -> 2.6
// ms.  Time of the CTAs of the first batch (sum 735 CTA-ms): structure factors
// 113, fields 145, cached dipole fields 112, force pass 92, partner lists 60,
// the other pair loops 82.
//
// Per configuration, in order:
//   load      direct coordinates (kardir, lattice.f90:183-225), phase tables
//   short     engforce_bmhftd_pbc / engforce_nmlj_pbc (FP64)
//   static    damped charge (+ static dipole) field (moment_from_pola.f90:327-330)
//   solve     PCG on (alpha^-1 - T) mu = E_stat with FP64 residual refinement
//             (calc = 'other': the first guess is alpha E_stat)
//   force     multipole_ES with forces, energy, stress (ewald.f90:49-314)
// Scalars land in the single-configuration engine's slot layout.
#pragma once
#include <cooperative_groups.h>

#include "common.cuh"
#include "realspace.cuh"
#include "recip.cuh"
#include "batch_rec.cuh"

namespace mdff {

namespace cgx = cooperative_groups;

constexpr int kBMaxT = 4;          // types of a batched configuration
constexpr int kBPart = 16;         // values per CTA partial slot
constexpr int kBMaxC = 8;          // largest cluster
constexpr int kBSlots = 48;        // per-configuration scalar slots

// scalar slots of a configuration (same offsets as the single engine)
enum {
  BS_SR = 0,     // 16
  BS_DIR = 16,   // 7
  BS_REC = 23,   // 7
  BS_MOM = 30,   // 8
  BS_UPOL = 38,
  BS_ITER = 39,
  BS_CONV = 40,
  BS_RMSD = 41,
  BS_CATA = 42,
  BS_STAT = 43   // 0 = ok, else an MDFF_ERR_* code
};

enum {
  BF_COUL = 1, BF_SR = 2, BF_BMH = 4, BF_BMHFTD = 8, BF_LJ = 16, BF_POLAR = 32,
  BF_QQ = 64, BF_QD = 128, BF_DD = 256, BF_SURF = 512, BF_DIPST = 1024, BF_THOLE = 2048,
  BF_WFC = 4096, BF_TT4 = 8192  // BF_TT4: every damped ion pair uses order 4
};

struct BConf {
  int off, n, ntype, flags;
  int nk, nrows, row_off, k_off;
  int kx, ky, kz;
  int trunc, maxit, npol;
  int nb_off, es_off, pad0, pad1;
  double A[9], B[9], omega;
  double alpha, rc2, coul_unit, tol;
  int lwfc[kBMaxT];      // Wannier centres per type (BF_WFC): < 0 centre type
  int ldip_wfc, pad2;
  double rcut_wfc;
  // phase records of the reciprocal sums (batch_rec.cuh): byte offset of the
  // box, bytes per ion, byte offset of Z in a record; offset of apm
  long long rec;
  int rs, zo, apm_off, pad3;
  double rs2;            // largest squared short-range cutoff of the box
};

struct BatchArgs {
  int nconf, ntot;
  const BConf* conf;
  const int* order;      // queue position -> configuration (descending cost)
  int* queue;            // zeroed before every launch
  const double* pos;     // [3][ntot] Cartesian
  const int* typ;        // [ntot] packed type, polarisable flag and ranks (btyp, bpol, brank, bpl)
  const double* q;       // [ntot]
  const int* ipol;       // [ntot] polarisable flag (ldip_polar of the type)
  const double* pol;     // [ntot][9]
  const double* inv;     // [ntot][9]
  const double4* dip;    // [ntot] static dipoles
  const NBPair* nbtab;   // per configuration, [ntype][ntype] at nb_off
  const ESPair* estab;
  const int4* rows;      // per configuration at row_off: (nx, ny, nz_lo, k)
  const double* Ak;      // per configuration at k_off
  const double4* kvec;
  const double2* apm;    // (A(+n), A(-n)) by (row, n), per configuration at apm_off
  double4* s;            // [ntot] direct coordinates, w = q
  unsigned char* rec;    // phase records of every configuration
  // workspace of the resident CTAs (blockIdx.x) and clusters (blockIdx.x / C)
  double4* rpart;        // [CTA][2][rpart_ld] structure-factor partials
  size_t rpart_ld;
  double* gpart;         // [CTA][kBSplit][6][wn] field sums per row subset
  int wn;                // ions per row of the workspaces (nmax)
  int stage_extra;       // bytes of staging buffer after the shared layout (0: the 16 KB within it)
  unsigned short* nbl;   // [cluster][2][wn][wn] partners within the long / short cutoff
  int* nbn;              // [cluster][2][wn]
  // pair cache of the dipole operator, rows of the box's polarisable ions
  // (npol entries each) when npol^2 <= ccap, else the pairs are recomputed
  size_t ccap;           // entries per cluster
  unsigned short* cj;
  int* cn;               // [cluster][wn]
  double4* c64;          // (rx, ry, rz, B2)
  double* b64;           // B1
  float4* c32;
  float* b32;
  double4 *Estat, *x, *r, *z, *p, *mu;  // [ntot]
  double4* E;            // [ntot] final field
  double* force;         // [3][ntot]
  double* part;          // [nconf][kBMaxC][2][kBPart]
  double* out;           // [nconf][kBSlots]
};

// shared-memory layout of one CTA for configurations of up to nmax ions
struct BShared {
  double4* s;      // [nmax]
  double4* v;      // [nmax] vector operand (FP64)
  float4* v32;     // [nmax] vector operand (FP32)
  int* t;          // [nmax]
  NBPair* nb;      // [kBMaxT^2]
  ESPair* es;      // [kBMaxT^2]
  double* red;     // [kBPart * 32]
  double* res;     // [kBPart]
  int* cfg;        // [1]
  unsigned char* stage;  // staging buffer of the reciprocal sums
  int stage_bytes;
};

__host__ __device__ inline size_t batch_smem_bytes(int nmax) {
  size_t b = 0;
  b += sizeof(double4) * nmax * 2;
  b += kBStage;
  b += sizeof(float4) * nmax;
  b += sizeof(NBPair) * kBMaxT * kBMaxT;
  b += sizeof(ESPair) * kBMaxT * kBMaxT;
  b += sizeof(double) * kBPart * 33;
  b += sizeof(int) * nmax + 16;
  return b;
}

// offset of the adjoint's extra [nmax] double4 array after the layout
// (rounded up to 16 bytes: vector loads need the alignment)
__host__ __device__ inline size_t batch_smem_extra_offset(int nmax) {
  return (batch_smem_bytes(nmax) + 15) & ~(size_t)15;
}

__device__ inline BShared batch_smem(unsigned char* base, int nmax) {
  BShared S;
  size_t o = 0;
  S.s = reinterpret_cast<double4*>(base + o); o += sizeof(double4) * nmax;
  S.v = reinterpret_cast<double4*>(base + o); o += sizeof(double4) * nmax;
  S.stage = base + o; o += kBStage;
  S.v32 = reinterpret_cast<float4*>(base + o); o += sizeof(float4) * nmax;
  S.nb = reinterpret_cast<NBPair*>(base + o); o += sizeof(NBPair) * kBMaxT * kBMaxT;
  S.es = reinterpret_cast<ESPair*>(base + o); o += sizeof(ESPair) * kBMaxT * kBMaxT;
  S.red = reinterpret_cast<double*>(base + o); o += sizeof(double) * kBPart * 32;
  S.res = reinterpret_cast<double*>(base + o); o += sizeof(double) * kBPart;
  S.t = reinterpret_cast<int*>(base + o); o += sizeof(int) * nmax;
  S.cfg = reinterpret_cast<int*>(base + o);
  S.stage_bytes = kBStage;
  return S;
}

// what one CTA knows about the configuration it works on
struct BCtx {
  const BConf* c;
  int cfg, rank, C, i0, i1, n, off;
  int p0, p1, npol;  // this CTA's polarisable ions (ranks), of npol in the box
  int slot;          // cluster index in the launch
  double* part;   // this configuration's partial slots
  int parity, rpar;
};

// Sum NV values over the cluster; every thread of every CTA receives the
// same result (partials are summed in rank order).  Slots are double-buffered
// by parity: a slot is rewritten two reductions later, after a barrier that
// every reader has passed.
template <int NV>
__device__ void cluster_sum(cgx::cluster_group& cl, BCtx& X, const BShared& S, double (&v)[NV]) {
  block_sum<NV>(v, S.red);
  double* mine = X.part + ((size_t)X.rank * 2 + X.parity) * kBPart;
  if (threadIdx.x == 0)
#pragma unroll
    for (int k = 0; k < NV; ++k) mine[k] = v[k];
  cl.sync();
  if ((int)threadIdx.x < NV) {
    double acc = 0.0;
    for (int c = 0; c < X.C; ++c)
      acc += __ldcg(X.part + ((size_t)c * 2 + X.parity) * kBPart + threadIdx.x);
    S.res[threadIdx.x] = acc;
  }
  __syncthreads();
#pragma unroll
  for (int k = 0; k < NV; ++k) v[k] = S.res[k];
  __syncthreads();
  X.parity ^= 1;
}

// L2 load of a 4-vector written by another CTA of the cluster
__device__ __forceinline__ double4 ldcg4(const double4* p) {
  const double2* q = reinterpret_cast<const double2*>(p);
  double2 a = __ldcg(q), b = __ldcg(q + 1);
  return make_double4(a.x, a.y, b.x, b.y);
}

// all ions' 4-vectors of the configuration from global memory into shared
__device__ inline void gather_vec(const BCtx& X, const double4* __restrict__ g, double4* sh) {
  for (int i = threadIdx.x; i < X.n; i += blockDim.x) sh[i] = ldcg4(g + X.off + i);
}
// the polarisable ions' 4-vectors by rank (R = float: FP32 copies)
__device__ inline void gather_pol(const BCtx& X, const int* t, const double4* __restrict__ g, double4* sh) {
  for (int k = threadIdx.x; k < X.npol; k += blockDim.x) sh[k] = ldcg4(g + X.off + bpl(t[k]));
}
__device__ inline void gather_pol32(const BCtx& X, const int* t, const double4* __restrict__ g, float4* sh) {
  for (int k = threadIdx.x; k < X.npol; k += blockDim.x) {
    const double4 v = ldcg4(g + X.off + bpl(t[k]));
    sh[k] = make_float4((float)v.x, (float)v.y, (float)v.z, 0.f);
  }
}

// m = 2 pi B^T mu (so that k.mu = n.m)
__device__ __forceinline__ double3 bmvec(const BConf& c, double mx, double my, double mz) {
  return make_double3(kTwoPi * (c.B[0] * mx + c.B[3] * my + c.B[6] * mz),
                      kTwoPi * (c.B[1] * mx + c.B[4] * my + c.B[7] * mz),
                      kTwoPi * (c.B[2] * mx + c.B[5] * my + c.B[8] * mz));
}

// ---------------------------------------------------------------------------
// weights (q, 2 pi B^T mu) of list entry k: mode 0 all ions (q and mu from S.s,
// S.v by ion), 1 / 2 the polarisable ions (no charge, mu from S.v / S.v32 by rank)
struct BWeights {
  const BConf* c;
  const double4* s;
  const double4* v;
  const float4* v32;
  int n0, mode;
  bool has_q, has_mu;
  __device__ __forceinline__ void operator()(int k, double (&w)[4]) const {
    double mx = 0.0, my = 0.0, mz = 0.0;
    if (has_mu) {
      if (mode == 2) {
        const float4 m = v32[n0 + k];
        mx = m.x;
        my = m.y;
        mz = m.z;
      } else {
        const double4 m = v[n0 + k];
        mx = m.x;
        my = m.y;
        mz = m.z;
      }
    }
    const double3 m = bmvec(*c, mx, my, mz);
    w[0] = (mode == 0 && has_q) ? s[n0 + k].w : 0.0;
    w[1] = m.x;
    w[2] = m.y;
    w[3] = m.z;
  }
};

struct BRecArgs {
  const BConf* c;
  const int4* rows;
  BList src, dst;        // ions of the structure factor / of the field
  const int* t;
  const unsigned char* rec;
  const double2* apm;
  const double4* w;      // weights of src
  unsigned char* buf;    // two buffers of CH records
  int CH;
  bool rot;              // (brho of kind 2) the sums times i
  double4* out;          // this CTA's partials
  const double4* part;   // rank 0's partials
  size_t pld;
  int C;
  unsigned char* stage;
  int stage_bytes;
  double* gp;
  int gld;
  BWeights wd;           // dipole weights of dst
};

template <int NT, int HM>
__device__ __noinline__ void brho_n(const BRecArgs& r) {
  const BConf& c = *r.c;
  brho_t<NT, HM>(r.rec, c.rs, c.zo, c.kx, c.kz, r.rows, c.nrows, r.src, r.t, r.w, r.buf, r.CH, r.out, r.rot);
}
template <int HM>
__device__ __forceinline__ void brho(const BRecArgs& r) {
  switch (r.c->kz / 4) {
    case 0: brho_n<1, HM>(r); break;
    case 1: brho_n<2, HM>(r); break;
    case 2: brho_n<3, HM>(r); break;
    default: brho_n<4, HM>(r); break;
  }
}
template <int KS, bool MUF>
__device__ __noinline__ int bfld_n(const BRecArgs& r) {
  const BConf& c = *r.c;
  return bfld_t<KS, MUF>(r.rec, c.rs, c.zo, c.kx, c.kz, r.rows, c.nrows, r.apm, r.part, r.pld, r.C, r.dst, r.t,
                         r.stage, r.stage_bytes, r.gp, r.gld, r.wd);
}
template <bool MUF>
__device__ __forceinline__ int bfld(const BRecArgs& r) {
  switch (r.c->kz / 2) {
    case 0: case 1: case 2: return bfld_n<3, MUF>(r);
    case 3: return bfld_n<4, MUF>(r);
    case 4: return bfld_n<5, MUF>(r);
    case 5: return bfld_n<6, MUF>(r);
    default: return bfld_n<7, MUF>(r);
  }
}

// set-up of a pass: ions, workspaces (mode, dst_pol as brec)
__device__ __forceinline__ BRecArgs brec_args(const BatchArgs& a, BCtx& X, const BShared& S, int mode, bool dst_pol) {
  const BConf& c = *X.c;
  BRecArgs r;
  r.c = X.c;
  r.rows = a.rows + c.row_off;
  r.src = mode == 0 ? BList{X.i0, X.i1 - X.i0, false} : BList{X.p0, X.p1 - X.p0, true};
  r.dst = dst_pol ? BList{X.p0, X.p1 - X.p0, true} : BList{X.i0, X.i1 - X.i0, false};
  r.t = S.t;
  r.rec = a.rec + c.rec;
  r.apm = a.apm + c.apm_off;
  r.pld = 2 * a.rpart_ld;  // CTA to CTA
  // (the partials are double-buffered: a reader of the previous pass's half
  // has passed this pass's barrier before that half is written again)
  r.part = a.rpart + ((size_t)(blockIdx.x - X.rank) * 2 + X.rpar) * a.rpart_ld;
  r.out = a.rpart + ((size_t)blockIdx.x * 2 + X.rpar) * a.rpart_ld;
  X.rpar ^= 1;
  r.rot = false;
  r.C = X.C;
  r.stage = S.stage;
  r.stage_bytes = S.stage_bytes;
  r.gp = a.gpart + (size_t)blockIdx.x * kBSplit * 6 * a.wn;
  r.gld = a.wn;
  r.wd = BWeights{X.c, S.s, S.v, S.v32, r.dst.n0, 0, false, true};
  return r;
}
// room for nw weights per ion, the rest of the staging buffer for the records in
// passing (brec_staging)
__device__ __forceinline__ double4* brec_weights(BRecArgs& r, const BShared& S, int nw) {
  const BStaging st = brec_staging(S.stage_bytes, r.src.cnt, nw, r.c->rs);
  double4* w = st.weights ? reinterpret_cast<double4*>(S.stage) : reinterpret_cast<double4*>(r.gp);
  r.buf = S.stage + st.weights;
  r.CH = st.ch;
  r.w = w;
  return w;
}

// Reciprocal pass of one configuration.  mode 0: the weights of all of this
// CTA's ions with charges and / or the dipoles in S.v; 1 / 2: of its
// polarisable ions with the vector in S.v / S.v32 by rank.  The field sums are
// left in this CTA's gpart for all its ions or (dst_pol) its polarisable ones;
// bfld_get reads them.  With do_str, es[0..6] receives this CTA's share of
// (u_rec, tau_rec) scaled as in k_rec_field_sum.  Returns the number of row subsets.
__device__ __noinline__ int brec(cgx::cluster_group& cl, const BatchArgs& a, BCtx& X, const BShared& S, int mode,
                                 bool has_q, bool has_mu, bool dst_pol, bool muf, bool do_str, double (&es)[7]) {
  const BConf& c = *X.c;
  for (int k = 0; k < 7; ++k) es[k] = 0.0;
  if (c.nk == 0) return 0;
  BRecArgs r = brec_args(a, X, S, mode, dst_pol);
  {
    // weights once per ion: in the staging buffer, else in the field's scratch
    const BWeights ws{X.c, S.s, S.v, S.v32, r.src.n0, mode, has_q, has_mu};
    double4* w = brec_weights(r, S, 1);
    __syncthreads();
    for (int k = threadIdx.x; k < r.src.cnt; k += blockDim.x) {
      double v[4];
      ws(k, v);
      w[k] = make_double4(v[0], v[1], v[2], v[3]);
    }
    __syncthreads();
  }
  if (has_mu) brho<1>(r);
  else brho<0>(r);
  cl.sync();
  if (do_str) {
    // energy and stress of this CTA's share of the rows
    const int nz = c.kz + 1;
    const double4* kv0 = a.kvec + c.k_off;
    const double* Ak = a.Ak + c.k_off;
    const int r0 = (int)((long long)c.nrows * X.rank / X.C), r1 = (int)((long long)c.nrows * (X.rank + 1) / X.C);
    for (int e = threadIdx.x; e < (r1 - r0) * nz; e += blockDim.x) {
      const int row = r0 + e / nz, n = e % nz;
      const int4 ri = r.rows[row];
      double2 rp, rm;
      brho_pm(r.part, r.pld, X.C, (size_t)row * nz + n, nullptr, rp, rm);
      for (int sg = 0; sg < 2; ++sg) {
        if (sg ? !(n > 0 && ri.z < 0) : n < ri.z) continue;
        const int k = ri.w + (sg ? -n : n) - ri.z;
        const double2 v = sg ? rm : rp;
        const double st = (v.x * v.x + v.y * v.y) * Ak[k];
        const double4 kv = kv0[k];
        es[0] += st;
        es[1] += (1.0 - kv.w * kv.x * kv.x) * st;
        es[2] += (1.0 - kv.w * kv.y * kv.y) * st;
        es[3] += (1.0 - kv.w * kv.z * kv.z) * st;
        es[4] -= kv.w * kv.x * kv.y * st;
        es[5] -= kv.w * kv.x * kv.z * st;
        es[6] -= kv.w * kv.y * kv.z * st;
      }
    }
    const double tpi_V = kTwoPi / c.omega;
    es[0] *= 2.0 * tpi_V;
    for (int k = 1; k < 7; ++k) es[k] *= 2.0 * tpi_V / c.omega;
  }
  if (muf) return bfld<true>(r);
  return bfld<false>(r);
}

// field e (and dipole force fm) of list entry k from the row subsets' sums
__device__ __forceinline__ void bfld_get(const BatchArgs& a, const BConf& c, int RS, int k, bool muf,
                                         double (&e)[3], double (&fm)[3]) {
  const double* gp = a.gpart + (size_t)blockIdx.x * kBSplit * 6 * a.wn;
  double G[3] = {0, 0, 0}, H[3] = {0, 0, 0};
  for (int s = 0; s < RS; ++s)
#pragma unroll
    for (int d = 0; d < 3; ++d) {
      G[d] += gp[(size_t)(s * 6 + d) * a.wn + k];
      if (muf) H[d] += gp[(size_t)(s * 6 + 3 + d) * a.wn + k];
    }
  const double scale = 2.0 * (2.0 * (kTwoPi / c.omega));
#pragma unroll
  for (int d = 0; d < 3; ++d) {
    e[d] = -kTwoPi * (c.B[3 * d] * G[0] + c.B[3 * d + 1] * G[1] + c.B[3 * d + 2] * G[2]) * scale;
    fm[d] = kTwoPi * (c.B[3 * d] * H[0] + c.B[3 * d + 1] * H[1] + c.B[3 * d + 2] * H[2]) * scale;
  }
}

// ---------------------------------------------------------------------------
// Partner lists of this CTA's ions, ascending, within the long-range (which =
// 0) and the short-range (1) cutoff plus a margin: every later pair loop walks
// these (and takes the exact inclusion decision itself) instead of all ions of
// the box, half of which lie outside the half-box cutoff and nearly all
// outside a 4-6 A short-range cutoff.  The test is FP32 on coordinates wrapped
// to [-0.5, 0.5); the margin covers its rounding, and a pair whose image is
// ambiguous at that precision is always kept, as is one whose distance is not a
// number (the pair loops carry it into the results).
__device__ __forceinline__ unsigned short* bnbl(const BatchArgs& a, const BCtx& X, int which, int i) {
  return a.nbl + (((size_t)X.slot * 2 + which) * a.wn + i) * a.wn;
}
__device__ __forceinline__ int* bnbn(const BatchArgs& a, const BCtx& X, int which) {
  return a.nbn + ((size_t)X.slot * 2 + which) * a.wn;
}
__device__ __noinline__ void blists(const BatchArgs& a, const BCtx& X, const BShared& S, bool coul, bool sr) {
  const BConf& c = *X.c;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarp = blockDim.x >> 5;
  for (int i = threadIdx.x; i < X.n; i += blockDim.x) {
    const double4 s = S.s[i];
    S.v32[i] = make_float4((float)(s.x - rint(s.x)), (float)(s.y - rint(s.y)), (float)(s.z - rint(s.z)), 0.f);
  }
  __syncthreads();
  float A[9];
  float amax = 0.f;
#pragma unroll
  for (int k = 0; k < 9; ++k) {
    A[k] = (float)c.A[k];
    amax += fabsf(A[k]);
  }
  // rounding of r: 3 coordinates of 2^-24 each times the cell, 4x margin
  const float rl = sqrtf((float)c.rc2), rs = sqrtf((float)c.rs2);
  const float l2 = coul ? (float)c.rc2 * 1.00001f + 2e-6f * amax * rl : -1.f;
  const float s2 = sr ? (float)c.rs2 * 1.00001f + 2e-6f * amax * rs : -1.f;
  for (int i = X.i0 + warp; i < X.i1; i += nwarp) {
    const float4 si = S.v32[i];
    unsigned short *ll = bnbl(a, X, 0, i), *ls = bnbl(a, X, 1, i);
    int ml = 0, ms = 0;
    for (int j0 = 0; j0 < X.n; j0 += 32) {
      const int j = j0 + lane;
      bool kl = false, ksr = false;
      if (j < X.n && j != i) {
        const float4 sj = S.v32[j];
        float dx = si.x - sj.x, dy = si.y - sj.y, dz = si.z - sj.z;
        // nearest integer by the 2^23 shift (|d| <= 1)
        dx -= __fadd_rn(__fadd_rn(dx, 12582912.f), -12582912.f);
        dy -= __fadd_rn(__fadd_rn(dy, 12582912.f), -12582912.f);
        dz -= __fadd_rn(__fadd_rn(dz, 12582912.f), -12582912.f);
        const float x = A[0] * dx + A[1] * dy + A[2] * dz;
        const float y = A[3] * dx + A[4] * dy + A[5] * dz;
        const float z = A[6] * dx + A[7] * dy + A[8] * dz;
        const float r2 = x * x + y * y + z * z;
        const bool edge = fmaxf(fabsf(dx), fmaxf(fabsf(dy), fabsf(dz))) > 0.49999f;
        kl = coul && (!(r2 > l2) || edge);
        ksr = sr && (!(r2 > s2) || edge);
      }
      const unsigned bl = __ballot_sync(FULL_MASK, kl), bs = __ballot_sync(FULL_MASK, ksr);
      const unsigned lt = (1u << lane) - 1u;
      if (kl) ll[ml + __popc(bl & lt)] = (unsigned short)j;
      if (ksr) ls[ms + __popc(bs & lt)] = (unsigned short)j;
      ml += __popc(bl);
      ms += __popc(bs);
    }
    if (lane == 0) {
      bnbn(a, X, 0)[i] = ml;
      bnbn(a, X, 1)[i] = ms;
    }
  }
  __syncthreads();
}
// the lists are rewritten for every box a cluster takes and may have been
// written by another CTA: read through L2, one visit ahead of their use
__device__ __forceinline__ int bnbr(const unsigned short* l, int k) { return (int)__ldcg(l + k); }

// ---------------------------------------------------------------------------
// real-space field of the vector in S.v / S.v32 on this CTA's polarisable ions
// (warp per ion, lanes over its partner list), added into E.  QQ: damped charge field; DD:
// dipole field.  pol = false: vectors by ion, the reference's condition (both
// dipoles nonzero); true: vectors by rank, both ions polarisable.
template <typename R, bool QQ, bool DD, int K = 0>
__device__ __noinline__ void bfield(const BatchArgs& a, const BCtx& X, const BShared& S, int damp, bool pol,
                       double4* __restrict__ E) {
  const BConf& c = *X.c;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarp = blockDim.x >> 5;
  const R rc2 = (R)c.rc2;
  for (int p = X.p0 + warp; p < X.p1; p += nwarp) {
    const int i = bpl(S.t[p]);
    const double4 si = S.s[i];
    const int ti = btyp(S.t[i]);
    bool dip_i = pol;
    if (DD && !pol) {
      const double4 m = S.v[i];
      dip_i = m.x != 0 || m.y != 0 || m.z != 0;
    }
    R ex = R(0), ey = R(0), ez = R(0);
    const unsigned short* row = bnbl(a, X, 0, i);
    const int nn = (QQ || dip_i) ? __ldcg(bnbn(a, X, 0) + i) : 0;
    int jn = lane < nn ? bnbr(row, lane) : 0;
    for (int k = lane; k < nn; k += 32) {
      const int j = jn;
      if (k + 32 < nn) jn = bnbr(row, k + 32);
      const double4 sj = S.s[j];
      const int tj = S.t[j];
      R rx, ry, rz;
      const R r2 = pair_vec<R>(c.A, si, sj, rx, ry, rz);
      if (r2 > rc2) continue;  // ewald_dir.f90:202
      R mx = R(0), my = R(0), mz = R(0);
      bool dd = false;
      if (DD && dip_i) {
        if (pol) {
          dd = bpol(tj);
          if (dd) {
            if (sizeof(R) == 4) {
              const float4 m = S.v32[brank(tj)];
              mx = (R)m.x; my = (R)m.y; mz = (R)m.z;
            } else {
              const double4 m = S.v[brank(tj)];
              mx = (R)m.x; my = (R)m.y; mz = (R)m.z;
            }
          }
        } else {
          const double4 m = S.v[j];
          mx = (R)m.x; my = (R)m.y; mz = (R)m.z;
          dd = m.x != 0 || m.y != 0 || m.z != 0;
        }
      }
      const double qj = QQ ? sj.w : 0.0;
      if (!dd && (!QQ || qj == 0.0)) continue;
      es_field_pair<R, QQ, DD, K>(S.es, c.ntype, i, j, ti, btyp(tj), rx, ry, rz, r2, (R)c.alpha, damp,
                               qj, dd, mx, my, mz, ex, ey, ez, (c.flags & BF_THOLE) ? 1 : 0);
    }
    const double dx = warp_sum((double)ex), dy = warp_sum((double)ey), dz = warp_sum((double)ez);
    if (lane == 0) {
      const int gi = X.off + i;
      const double4 o = E[gi];
      E[gi] = make_double4(o.x + dx, o.y + dy, o.z + dz, 0.0);
    }
  }
}

// Pair cache of the dipole operator: for every polarisable ion of this CTA the
// terms of T2(r) mu = B2 r (r.mu) - B1 mu of its polarisable partners within
// the cutoff, formed once per box in FP64 (the operator is applied a dozen
// times); MIXED keeps an FP32 copy for the inner iterations.  Row p (rank)
// starts at p * npol.
__device__ __forceinline__ bool bcached(const BatchArgs& a, const BCtx& X) {
  return (size_t)X.npol * X.npol <= a.ccap;
}
template <bool MIXED>
__device__ __noinline__ void bcache(const BatchArgs& a, const BCtx& X, const BShared& S) {
  const BConf& c = *X.c;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarp = blockDim.x >> 5;
  const int thole = (c.flags & BF_THOLE) ? 1 : 0;
  for (int p = X.p0 + warp; p < X.p1; p += nwarp) {
    const int i = bpl(S.t[p]);
    const double4 si = S.s[i];
    const int ti = btyp(S.t[i]);
    const unsigned short* row = bnbl(a, X, 0, i);
    const int nn = __ldcg(bnbn(a, X, 0) + i);
    const size_t base = (size_t)X.slot * a.ccap + (size_t)p * X.npol;
    int m = 0;
    int jn = lane < nn ? bnbr(row, lane) : 0;
    for (int k0 = 0; k0 < nn; k0 += 32) {
      const int k = k0 + lane;
      bool keep = false;
      double rx = 0, ry = 0, rz = 0, B1 = 0, B2 = 0;
      int rk = 0;
      const int j = jn;
      if (k + 32 < nn) jn = bnbr(row, k + 32);
      if (k < nn) {
        const int tj = S.t[j];
        if (bpol(tj)) {
          const double r2 = pair_vec<double>(c.A, si, S.s[j], rx, ry, rz);
          if (r2 <= c.rc2) {
            keep = true;
            rk = brank(tj);
            Radial<double> g;
            radial<double, false>(r2, c.alpha, g);
            double F1 = g.F1, F2 = g.F2;
            if (thole) {
              const bool ia = half_mask(i, j);
              const int tjt = btyp(tj);
              const ESPair& P = S.es[(ia ? ti : tjt) * c.ntype + (ia ? tjt : ti)];
              if (P.thole) thole_radial<double>(P, g.d, F1, F2);
            }
            B1 = F1 * g.dm3;
            B2 = 3.0 * F2 * g.dm5;
          }
        }
      }
      const unsigned bal = __ballot_sync(FULL_MASK, keep);
      if (keep) {
        const size_t o = base + m + __popc(bal & ((1u << lane) - 1u));
        a.cj[o] = (unsigned short)rk;
        a.c64[o] = make_double4(rx, ry, rz, B2);
        a.b64[o] = B1;
        if (MIXED) {
          a.c32[o] = make_float4((float)rx, (float)ry, (float)rz, (float)B2);
          a.b32[o] = (float)B1;
        }
      }
      m += __popc(bal);
    }
    if (lane == 0) a.cn[(size_t)X.slot * a.wn + p] = m;
  }
  __syncthreads();
}

// T2 v of the cached pairs on this CTA's polarisable ions (vector in S.v / S.v32
// by rank), added into E.  Eight lanes per row, four rows per warp, and the
// next four entries of a lane in flight while the current ones are used: the
// cache streams from L2, so what counts is the bytes in flight (a warp per row
// with four entries a lane left most lanes idle in every row's last round and
// paid its reduction per row).
template <typename R>
struct BPairs {
  R x[4], y[4], z[4], b2[4], b1[4];
  int j[4];
};
template <typename R>
__device__ __forceinline__ void bpairs_load(const BatchArgs& a, size_t base, int k0, int n, BPairs<R>& q) {
#pragma unroll
  for (int u = 0; u < 4; ++u) {
    const int k = k0 + 8 * u;
    const bool ok = k < n;
    const size_t o = base + (ok ? k : 0);
    q.j[u] = a.cj[o];
    if (sizeof(R) == 4) {
      const float4 r = a.c32[o];
      q.x[u] = (R)r.x; q.y[u] = (R)r.y; q.z[u] = (R)r.z; q.b2[u] = (R)r.w;
      q.b1[u] = (R)a.b32[o];
    } else {
      const double4 r = a.c64[o];
      q.x[u] = (R)r.x; q.y[u] = (R)r.y; q.z[u] = (R)r.z; q.b2[u] = (R)r.w;
      q.b1[u] = (R)a.b64[o];
    }
    if (!ok) q.b2[u] = q.b1[u] = R(0);
  }
}
template <typename R>
__device__ __noinline__ void bfield_cached(const BatchArgs& a, const BCtx& X, const BShared& S, double4* __restrict__ E) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarp = blockDim.x >> 5;
  const int sub = lane >> 3, l8 = lane & 7;
  for (int pb = X.p0 + 4 * warp; pb < X.p1; pb += 4 * nwarp) {
    const int p = pb + sub;
    const bool ok = p < X.p1;
    const size_t base = (size_t)X.slot * a.ccap + (size_t)(ok ? p : pb) * X.npol;
    const int n = ok ? a.cn[(size_t)X.slot * a.wn + p] : 0;
    // rounds of the longest of the four rows (entry 0 of an empty row is read
    // but not used; a row of the workspace always exists)
    const int nm = __reduce_max_sync(FULL_MASK, n);
    R ex = R(0), ey = R(0), ez = R(0);
    BPairs<R> q;
    if (nm > 0) bpairs_load<R>(a, base, l8, n, q);
    for (int k0 = 0; k0 < nm; k0 += 32) {
      const BPairs<R> c = q;
      if (k0 + 32 < nm) bpairs_load<R>(a, base, k0 + 32 + l8, n, q);
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        R mx, my, mz;
        const int j = k0 + l8 + 8 * u < n ? c.j[u] : 0;
        if (sizeof(R) == 4) {
          const float4 m = S.v32[j];
          mx = (R)m.x; my = (R)m.y; mz = (R)m.z;
        } else {
          const double4 m = S.v[j];
          mx = (R)m.x; my = (R)m.y; mz = (R)m.z;
        }
        const R rm = c.b2[u] * (c.x[u] * mx + c.y[u] * my + c.z[u] * mz);
        if (k0 + l8 + 8 * u < n) {
          ex += rm * c.x[u] - c.b1[u] * mx;
          ey += rm * c.y[u] - c.b1[u] * my;
          ez += rm * c.z[u] - c.b1[u] * mz;
        }
      }
    }
    double d[3] = {(double)ex, (double)ey, (double)ez};
#pragma unroll
    for (int o = 1; o < 8; o <<= 1)
#pragma unroll
      for (int c = 0; c < 3; ++c) d[c] += __shfl_xor_sync(FULL_MASK, d[c], o);
    if (ok && l8 == 0) {
      const int gi = X.off + bpl(S.t[p]);
      const double4 o = E[gi];
      E[gi] = make_double4(o.x + d[0], o.y + d[1], o.z + d[2], 0.0);
    }
  }
}

// ---------------------------------------------------------------------------
// short range (FP64) on this CTA's ions: forces overwrite force[own];
// acc[16] as k_shortrange.
__device__ __noinline__ void bshort(const BatchArgs& a, const BCtx& X, const BShared& S, double (&acc)[kSRPart]) {
  const BConf& c = *X.c;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarp = blockDim.x >> 5;
  const int do_bmh = (c.flags & BF_BMH) ? 1 : 0, do_lj = (c.flags & BF_LJ) ? 1 : 0;
  const int lbmhftd = (c.flags & BF_BMHFTD) ? 1 : 0;
  for (int k = 0; k < kSRPart; ++k) acc[k] = 0.0;
  for (int i = X.i0 + warp; i < X.i1; i += nwarp) {
    double4 si = S.s[i];
    int ti = btyp(S.t[i]);
    double fb[3] = {0, 0, 0}, fl[3] = {0, 0, 0};
    const unsigned short* row = bnbl(a, X, 1, i);
    const int nn = bnbn(a, X, 1)[i];
    int jn = lane < nn ? bnbr(row, lane) : 0;
    for (int k = lane; k < nn; k += 32) {
      const int j = jn;
      if (k + 32 < nn) jn = bnbr(row, k + 32);
      double4 sj = S.s[j];
      double rx, ry, rz;
      double r2 = min_image_exact(c.A, xsub(si.x, sj.x), xsub(si.y, sj.y), xsub(si.z, sj.z), rx,
                                  ry, rz);
      const NBPair& P = S.nb[ti * c.ntype + btyp(S.t[j])];
      if (r2 >= P.rcutsq) continue;  // non_bonded.f90:1154 strict <
      if (do_bmh && (P.A != 0.0 || P.wall != 0.0)) {
        double u, wij;
        sr_pair_bmh<double>(P, lbmhftd, r2, u, wij);
        double fx = wij * rx, fy = wij * ry, fz = wij * rz;
        fb[0] += fx;
        fb[1] += fy;
        fb[2] += fz;
        acc[0] += 0.5 * u;
        acc[1] += 0.5 * (rx * fx + ry * fy + rz * fz);
        acc[4] += rx * fx;
        acc[5] += ry * fy;
        acc[6] += rz * fz;
        acc[7] += 0.5 * (rx * fy + ry * fx);
        acc[8] += 0.5 * (rx * fz + rz * fx);
        acc[9] += 0.5 * (ry * fz + rz * fy);
      }
      if (do_lj) {
        double e, wij;
        sr_pair_lj<double>(P, c.trunc, r2, e, wij);
        double fx = wij * rx, fy = wij * ry, fz = wij * rz;
        fl[0] += fx;
        fl[1] += fy;
        fl[2] += fz;
        acc[2] += 0.5 * e;
        acc[3] += 0.5 * (wij * r2);
        acc[10] += rx * fx;
        acc[11] += ry * fy;
        acc[12] += rz * fz;
        acc[13] += 0.5 * (rx * fy + ry * fx);
        acc[14] += 0.5 * (rx * fz + rz * fx);
        acc[15] += 0.5 * (ry * fz + rz * fy);
      }
    }
#pragma unroll
    for (int d = 0; d < 3; ++d) {
      fb[d] = warp_sum(fb[d]);
      fl[d] = warp_sum(fl[d]);
    }
    if (lane == 0) {
      const double* f = do_bmh ? fb : fl;  // non_bonded.f90:699-701, 1104-1106
      int gi = X.off + i;
      a.force[gi] = f[0];
      a.force[a.ntot + gi] = f[1];
      a.force[2 * (size_t)a.ntot + gi] = f[2];
    }
  }
}

// final real-space pass (k_es_force) on this CTA's ions; mu in S.v (FP64).  K,
// THOLE as k_es_force.  The pair's vector and the cutoff decision are the exact FP64
// ones and the lane sums FP64 in both engines: the mixed one evaluates the pair's terms in
// FP32 and nothing else.
template <typename R, int K, bool THOLE>
__device__ __noinline__ void bforce_n(const BatchArgs& a, const BCtx& X, const BShared& S, double (&acc)[kESPart]) {
  const BConf& c = *X.c;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarp = blockDim.x >> 5;
  const int task_qq = (c.flags & BF_QQ) ? 1 : 0, task_qd = (c.flags & BF_QD) ? 1 : 0;
  const int task_dd = (c.flags & BF_DD) ? 1 : 0;
  double la[kESPart];
#pragma unroll
  for (int k = 0; k < kESPart; ++k) la[k] = 0.0;
  for (int i = X.i0 + warp; i < X.i1; i += nwarp) {
    const double4 si = S.s[i];
    const int ti = btyp(S.t[i]);
    const double4 mui = S.v[i];
    const R qi = (R)si.w, mi[3] = {(R)mui.x, (R)mui.y, (R)mui.z};
    const bool dip_i = mui.x != 0.0 || mui.y != 0.0 || mui.z != 0.0;
    double e[3] = {0, 0, 0}, f[3] = {0, 0, 0};
    const unsigned short* row = bnbl(a, X, 0, i);
    const int nn = bnbn(a, X, 0)[i];
    int jn = lane < nn ? bnbr(row, lane) : 0;
    for (int k = lane; k < nn; k += 32) {
      const int j = jn;
      if (k + 32 < nn) jn = bnbr(row, k + 32);
      const double4 sj = S.s[j];
      double rd[3];
      const double r2 = pair_vec<double>(c.A, si, sj, rd[0], rd[1], rd[2]);
      if (r2 > c.rc2) continue;
      const R r[3] = {(R)rd[0], (R)rd[1], (R)rd[2]};
      const int tj = btyp(S.t[j]);
      const double4 muj = S.v[j];
      const bool i_is_a = half_mask(i, j);
      const ESPair& P = S.es[(i_is_a ? ti : tj) * c.ntype + (i_is_a ? tj : ti)];
      const R mj[3] = {(R)muj.x, (R)muj.y, (R)muj.z};
      const bool dip_j = muj.x != 0.0 || muj.y != 0.0 || muj.z != 0.0;
      R u, fi[3], Ei[3];
      // the single engine's pair (i's frame)
      es_force_ipair<R, K, THOLE>(P, i_is_a, P.ldamp != 0, (R)r2, (R)c.alpha, r, qi, (R)sj.w, mi, mj, dip_i, dip_j,
                                  task_qq, task_qd, task_dd, u, fi, Ei);
#pragma unroll
      for (int d = 0; d < 3; ++d) {
        f[d] += (double)fi[d];
        e[d] += (double)Ei[d];
      }
      la[0] += 0.5 * (double)u;
      la[1] += (double)(r[0] * fi[0]);
      la[2] += (double)(r[1] * fi[1]);
      la[3] += (double)(r[2] * fi[2]);
      la[4] += 0.5 * (double)(r[0] * fi[1] + r[1] * fi[0]);
      la[5] += 0.5 * (double)(r[0] * fi[2] + r[2] * fi[0]);
      la[6] += 0.5 * (double)(r[1] * fi[2] + r[2] * fi[1]);
    }
#pragma unroll
    for (int d = 0; d < 3; ++d) {
      e[d] = warp_sum(e[d]);
      f[d] = warp_sum(f[d]);
    }
    if (lane == 0) {
      int gi = X.off + i;
      a.E[gi] = make_double4(e[0], e[1], e[2], 0.0);
      a.force[gi] += f[0] * c.coul_unit;
      a.force[a.ntot + gi] += f[1] * c.coul_unit;
      a.force[2 * (size_t)a.ntot + gi] += f[2] * c.coul_unit;
    }
  }
#pragma unroll
  for (int k = 0; k < kESPart; ++k) acc[k] = la[k];
}
template <typename R>
__device__ __forceinline__ void bforce(const BatchArgs& a, const BCtx& X, const BShared& S, double (&acc)[kESPart]) {
  const int fl = X.c->flags;
  if (fl & BF_THOLE) bforce_n<R, 0, true>(a, X, S, acc);
  else if (fl & BF_TT4) bforce_n<R, 4, false>(a, X, S, acc);
  else bforce_n<R, 0, false>(a, X, S, acc);
}

__device__ __forceinline__ double4 bmat3(const double* m, double4 v) {
  return make_double4(m[0] * v.x + m[1] * v.y + m[2] * v.z, m[3] * v.x + m[4] * v.y + m[5] * v.z,
                      m[6] * v.x + m[7] * v.y + m[8] * v.z, 0.0);
}

// self (+ surface) field of the vector v on own ions: E += 2 selfa2 v_i
// (- fpi_3V (qtot + vtot) with lsurf), ewald.f90:182-213
__device__ void bself(const BatchArgs& a, const BCtx& X, const double4* __restrict__ v, double selfa2,
                      bool lsurf, double fpi_3V, const double* tot, double4* __restrict__ E) {
  for (int i = X.i0 + threadIdx.x; i < X.i1; i += blockDim.x) {
    int gi = X.off + i;
    double4 m = v[gi];
    double s0 = 0.0, s1 = 0.0, s2 = 0.0;
    if (lsurf) {
      s0 = -(tot[0] + tot[3]) * fpi_3V;
      s1 = -(tot[1] + tot[4]) * fpi_3V;
      s2 = -(tot[2] + tot[5]) * fpi_3V;
    }
    double4 o = E[gi];
    E[gi] = make_double4(o.x + s0 + 2.0 * selfa2 * m.x, o.y + s1 + 2.0 * selfa2 * m.y,
                         o.z + s2 + 2.0 * selfa2 * m.z, 0.0);
  }
}

// moments [sum q r (3), sum v (3), sum q^2, sum v^2] over the cluster
__device__ void bmoments(cgx::cluster_group& cl, const BatchArgs& a, BCtx& X, const BShared& S,
                         const double4* __restrict__ v, bool has_q, double (&m)[8]) {
  for (int k = 0; k < 8; ++k) m[k] = 0.0;
  for (int i = X.i0 + threadIdx.x; i < X.i1; i += blockDim.x) {
    int gi = X.off + i;
    double qi = has_q ? S.s[i].w : 0.0;
    double4 u = v ? ldcg4(v + gi) : make_double4(0, 0, 0, 0);
    m[0] += qi * a.pos[gi];
    m[1] += qi * a.pos[a.ntot + gi];
    m[2] += qi * a.pos[2 * (size_t)a.ntot + gi];
    m[3] += u.x;
    m[4] += u.y;
    m[5] += u.z;
    m[6] += qi * qi;
    m[7] += u.x * u.x + u.y * u.y + u.z * u.z;
  }
  cluster_sum<8>(cl, X, S, m);
}

// the same sums added to the field of the polarisable ions: reciprocal field of
// entry k - p0 plus self (+ surface) field of v
__device__ void bfinish_pol(const BatchArgs& a, const BCtx& X, const BShared& S, int RS,
                            const double4* __restrict__ v, double selfa2, bool lsurf, double fpi_3V,
                            const double* tot, double4* __restrict__ E) {
  const BConf& c = *X.c;
  for (int p = X.p0 + threadIdx.x; p < X.p1; p += blockDim.x) {
    const int gi = X.off + bpl(S.t[p]);
    double e[3], fm[3];
    bfld_get(a, c, RS, p - X.p0, false, e, fm);
    const double4 m = ldcg4(v + gi);
    double s[3] = {0.0, 0.0, 0.0};
    if (lsurf)
      for (int d = 0; d < 3; ++d) s[d] = -(tot[d] + tot[3 + d]) * fpi_3V;
    const double4 o = E[gi];
    E[gi] = make_double4(o.x + e[0] + s[0] + 2.0 * selfa2 * m.x, o.y + e[1] + s[1] + 2.0 * selfa2 * m.y,
                         o.z + e[2] + s[2] + 2.0 * selfa2 * m.z, 0.0);
  }
}

// T v (field of a dipole set alone: dd undamped between polarisable ions,
// reciprocal dipole part, self / surface) on this CTA's polarisable ions into
// Tv.  The vector must be in global memory (vg) for all polarisable ions of the
// box; it is gathered here by rank.
template <typename R>
__device__ void bmatvec(cgx::cluster_group& cl, const BatchArgs& a, BCtx& X, const BShared& S,
                        const double4* __restrict__ vg, double4* __restrict__ Tv) {
  const BConf& c = *X.c;
  cl.sync();  // every CTA's slice of vg is written
  if (sizeof(R) == 4) gather_pol32(X, S.t, vg, S.v32);
  else gather_pol(X, S.t, vg, S.v);
  for (int p = X.p0 + threadIdx.x; p < X.p1; p += blockDim.x)
    Tv[X.off + bpl(S.t[p])] = make_double4(0, 0, 0, 0);
  __syncthreads();
  double es[7];
  const int RS = brec(cl, a, X, S, sizeof(R) == 4 ? 2 : 1, false, true, true, false, false, es);
  if (bcached(a, X)) bfield_cached<R>(a, X, S, Tv);
  else bfield<R, false, true>(a, X, S, 0, true, Tv);
  double tot[6] = {0, 0, 0, 0, 0, 0};
  if (c.flags & BF_SURF) {
    double m[8];
    bmoments(cl, a, X, S, vg, false, m);
    for (int k = 0; k < 6; ++k) tot[k] = m[k];
  }
  __syncthreads();
  double al = c.alpha;
  double selfa2 = 2.0 * (al / sqrt(kPi)) * al * al / 3.0;
  bfinish_pol(a, X, S, RS, vg, selfa2, (c.flags & BF_SURF) != 0, 2.0 * (kTwoPi / c.omega / 3.0), tot, Tv);
  __syncthreads();
}

// PCG on (alpha^-1 - T) x = b over the polarisable ions of the configuration,
// x holding the first guess (zero on the other ions).  Each CTA owns the
// polarisable ions of its rank range, so that a box whose polarisable ions
// are one type block still splits evenly over the cluster.  The true residual is formed with the FP64
// operator; with MIXED the inner iterations use the FP32 operator and stop
// at 1e-4 of that residual (iterative refinement), else they run to tol.
// Stops on the reference's rmsd measure (get_rmsd_mu, moment_from_pola.f90:
// 998-1027) <= tol, or after maxit inner iterations / 8 refinements.
template <bool MIXED>
__device__ void bsolve(cgx::cluster_group& cl, const BatchArgs& a, BCtx& X, const BShared& S,
                       const double4* __restrict__ b, double4* __restrict__ x, double tol,
                       int maxit, int& iters, double& rmsd) {
  typedef typename std::conditional<MIXED, float, double>::type RM;
  const BConf& c = *X.c;
  const double npol = (double)max(c.npol, 1);
  int outer = 0;
  iters = 0;
  while (true) {
    // true residual with the FP64 operator
    bmatvec<double>(cl, a, X, S, x, a.p);
    // (the gather of x read every CTA's slice before this one changes)
    double v2[2] = {0.0, 0.0};
    for (int p = X.p0 + threadIdx.x; p < X.p1; p += blockDim.x) {
      const int gi = X.off + bpl(S.t[p]);
      double4 ax = bmat3(a.inv + 9 * (size_t)gi, ldcg4(x + gi));
      double4 bi = ldcg4(b + gi), tx = a.p[gi];
      double4 ri = make_double4(bi.x + tx.x - ax.x, bi.y + tx.y - ax.y, bi.z + tx.z - ax.z, 0.0);
      double4 zi = bmat3(a.pol + 9 * (size_t)gi, ri);
      const double* pl = a.pol + 9 * (size_t)gi;
      double rr[3] = {ri.x, ri.y, ri.z};
      for (int d = 0; d < 3; ++d)
        if (pl[4 * d] != 0.0) v2[1] += rr[d] * rr[d];
      a.r[gi] = ri;
      a.z[gi] = zi;
      a.p[gi] = zi;
      v2[0] += ri.x * zi.x + ri.y * zi.y + ri.z * zi.z;
    }
    cluster_sum<2>(cl, X, S, v2);
    double rz = v2[0];
    rmsd = sqrt(v2[1] / npol);
    if (rmsd <= tol || iters >= maxit || outer >= 8) break;
    ++outer;
    // FP64 operator: the recurrence residual is final.  FP32 operator: trusted
    // to half the tolerance when the starting residual is small (the drift from
    // the true residual is ~ the FP32 matvec error times that start), else a
    // 1e-4 reduction and a new FP64 residual (iterative refinement).
    const double kGap = 3e-6;
    const bool trust = !MIXED || kGap * rmsd <= 0.5 * tol;
    const double tol_in = !MIXED ? tol : (trust ? 0.5 * tol : fmax(tol, 1e-4 * rmsd));
    double rms_last = rmsd;
    while (true) {
      // T p into a.E (the field buffer is free until the final pass)
      bmatvec<RM>(cl, a, X, S, a.p, a.E);
      double pq[1] = {0.0};
      for (int p = X.p0 + threadIdx.x; p < X.p1; p += blockDim.x) {
        const int gi = X.off + bpl(S.t[p]);
        const double4 pi = a.p[gi];
        const double4 ap = bmat3(a.inv + 9 * (size_t)gi, pi);
        const double4 tp = a.E[gi];
        const double4 qi = make_double4(ap.x - tp.x, ap.y - tp.y, ap.z - tp.z, 0.0);
        a.E[gi] = qi;  // q = A p
        pq[0] += pi.x * qi.x + pi.y * qi.y + pi.z * qi.z;
      }
      cluster_sum<1>(cl, X, S, pq);
      double alp = (pq[0] != 0.0) ? rz / pq[0] : 0.0;
      double u2[2] = {0.0, 0.0};
      for (int p = X.p0 + threadIdx.x; p < X.p1; p += blockDim.x) {
        const int gi = X.off + bpl(S.t[p]);
        double4 xi = ldcg4(x + gi), ri = a.r[gi], pi = a.p[gi], qi = a.E[gi];
        xi.x += alp * pi.x;
        xi.y += alp * pi.y;
        xi.z += alp * pi.z;
        ri.x -= alp * qi.x;
        ri.y -= alp * qi.y;
        ri.z -= alp * qi.z;
        double4 zi = bmat3(a.pol + 9 * (size_t)gi, ri);
        x[gi] = xi;
        a.r[gi] = ri;
        a.z[gi] = zi;
        u2[0] += ri.x * zi.x + ri.y * zi.y + ri.z * zi.z;
        const double* pl = a.pol + 9 * (size_t)gi;
        double rr[3] = {ri.x, ri.y, ri.z};
        for (int d = 0; d < 3; ++d)
          if (pl[4 * d] != 0.0) u2[1] += rr[d] * rr[d];
      }
      cluster_sum<2>(cl, X, S, u2);
      ++iters;
      double rms_in = sqrt(u2[1] / npol);
      rms_last = rms_in;
      if (!(rms_in > tol_in && iters < maxit)) break;
      double be = (rz != 0.0) ? u2[0] / rz : 0.0;
      rz = u2[0];
      for (int p = X.p0 + threadIdx.x; p < X.p1; p += blockDim.x) {
        const int gi = X.off + bpl(S.t[p]);
        double4 pi = a.p[gi], zi = a.z[gi];
        a.p[gi] = make_double4(zi.x + be * pi.x, zi.y + be * pi.y, zi.z + be * pi.z, 0.0);
      }
    }
    if (trust && (rms_last <= tol_in || iters >= maxit)) {
      rmsd = rms_last;
      break;
    }
  }
}

// ---------------------------------------------------------------------------
// one configuration, whole cluster
template <bool MIXED>
__device__ void bconfig(cgx::cluster_group& cl, const BatchArgs& a, BCtx& X, const BShared& S) {
  typedef typename std::conditional<MIXED, float, double>::type RM;
  const BConf& c = *X.c;
  double* out = a.out + (size_t)X.cfg * kBSlots;
  const bool coul = (c.flags & BF_COUL) != 0;
  // ---- load --------------------------------------------------------------
  for (int i = X.i0 + threadIdx.x; i < X.i1; i += blockDim.x) {
    int gi = X.off + i;
    double sx, sy, sz;
    kardir_exact(c.B, a.pos[gi], a.pos[a.ntot + gi], a.pos[2 * (size_t)a.ntot + gi], sx, sy, sz);
    a.s[gi] = make_double4(sx, sy, sz, a.q[gi]);
    if (coul && c.nk > 0) {
      // e^{2 pi i n s}, s wrapped to [-0.5, 0.5) (k_rec_tables)
      double sv[3] = {sx, sy, sz};
      const int km[3] = {c.kx, c.ky, c.kz};
      int e0 = 0;
      for (int d = 0; d < 3; ++d) {
        double w = sv[d] - rint(sv[d]);
        for (int m = 0; m <= km[d]; ++m) {
          double sn, cs;
          sincospi(2.0 * (double)m * w, &sn, &cs);
          // (entries of n > kz stay zero)
          unsigned char* rp = a.rec + c.rec + (size_t)i * c.rs;
          if (d < 2) reinterpret_cast<double2*>(rp)[e0 + m] = make_double2(cs, sn);
          else reinterpret_cast<double2*>(rp + c.zo)[m] = make_double2(cs, sn);
        }
        e0 += km[d] + 1;
      }
    }
  }
  for (int k = threadIdx.x; k < c.ntype * c.ntype; k += blockDim.x) {
    S.nb[k] = a.nbtab[c.nb_off + k];
    S.es[k] = a.estab[c.es_off + k];
  }
  cl.sync();
  for (int i = threadIdx.x; i < X.n; i += blockDim.x) {
    S.s[i] = ldcg4(a.s + X.off + i);
    S.t[i] = a.typ[X.off + i];
  }
  __syncthreads();
  blists(a, X, S, coul, (c.flags & BF_SR) != 0);
  // ---- short range -------------------------------------------------------
  {
    double acc[kSRPart];
    if (c.flags & BF_SR) {
      bshort(a, X, S, acc);
    } else {
      for (int k = 0; k < kSRPart; ++k) acc[k] = 0.0;
      for (int i = X.i0 + threadIdx.x; i < X.i1; i += blockDim.x) {
        int gi = X.off + i;
        a.force[gi] = a.force[a.ntot + gi] = a.force[2 * (size_t)a.ntot + gi] = 0.0;
      }
    }
    cluster_sum<kSRPart>(cl, X, S, acc);
    if (X.rank == 0 && threadIdx.x == 0)
      for (int k = 0; k < kSRPart; ++k) out[BS_SR + k] = acc[k];
  }
  if (!coul) {
    for (int i = X.i0 + threadIdx.x; i < X.i1; i += blockDim.x) {
      a.mu[X.off + i] = make_double4(0, 0, 0, 0);
      a.E[X.off + i] = make_double4(0, 0, 0, 0);
    }
    return;
  }
  const double al = c.alpha;
  const double selfa2 = 2.0 * (al / sqrt(kPi)) * al * al / 3.0;
  const double fpi_3V = 2.0 * (kTwoPi / c.omega / 3.0);
  const bool lsurf = (c.flags & BF_SURF) != 0;
  const bool dipst = (c.flags & BF_DIPST) != 0;
  const bool task_qq = (c.flags & BF_QQ) != 0;
  int iters = 0, conv = 1;
  double rmsd = 0.0;
  for (int i = X.i0 + threadIdx.x; i < X.i1; i += blockDim.x) a.x[X.off + i] = make_double4(0, 0, 0, 0);
  if (c.flags & BF_POLAR) {
    // the partner lists and the zeroed dipoles of every ion are in place
    cl.sync();
    // ---- static field: damped charges + static dipoles, at the polarisable
    // ions (the solver reads it there) ----------------------------------------
    for (int p = X.p0 + threadIdx.x; p < X.p1; p += blockDim.x)
      a.Estat[X.off + bpl(S.t[p])] = make_double4(0, 0, 0, 0);
    gather_vec(X, a.dip, S.v);
    __syncthreads();
    if (task_qq && dipst) bfield<RM, true, true>(a, X, S, 1, false, a.Estat);
    else if (task_qq && (c.flags & BF_TT4)) bfield<RM, true, false, 4>(a, X, S, 1, false, a.Estat);
    else if (task_qq) bfield<RM, true, false>(a, X, S, 1, false, a.Estat);
    else if (dipst) bfield<RM, false, true>(a, X, S, 1, false, a.Estat);
    if (bcached(a, X)) bcache<MIXED>(a, X, S);
    __syncthreads();
    double es[7];
    const int RS = brec(cl, a, X, S, 0, task_qq, dipst, true, false, false, es);
    double tot[6] = {0, 0, 0, 0, 0, 0};
    if (lsurf) {
      double m[8];
      bmoments(cl, a, X, S, a.dip, true, m);
      for (int k = 0; k < 6; ++k) tot[k] = m[k];
    }
    __syncthreads();
    bfinish_pol(a, X, S, RS, a.dip, selfa2, lsurf, fpi_3V, tot, a.Estat);
    __syncthreads();
    // ---- PCG: (alpha^-1 - T) x = E_stat, x0 = alpha E_stat ----------------
    for (int p = X.p0 + threadIdx.x; p < X.p1; p += blockDim.x) {
      const int gi = X.off + bpl(S.t[p]);
      a.x[gi] = bmat3(a.pol + 9 * (size_t)gi, a.Estat[gi]);
    }
    const double tol = c.tol;
    bsolve<MIXED>(cl, a, X, S, a.Estat, a.x, tol, c.maxit, iters, rmsd);
    conv = rmsd <= tol ? 1 : 0;
    cl.sync();  // the converged dipoles of every CTA are in place
  }
  // ---- u_pol, total dipoles (+ Wannier centres), catastrophe -------------
  {
    const bool wfc = (c.flags & BF_WFC) != 0;
    double v[3] = {0.0, 0.0, 0.0};
    for (int i = X.i0 + threadIdx.x; i < X.i1; i += blockDim.x) {
      int gi = X.off + i;
      double4 m = ldcg4(a.x + gi);
      if (a.ipol[gi]) {
        const double* iv = a.inv + 9 * (size_t)gi;
        double mm[3] = {m.x, m.y, m.z};
        for (int p = 0; p < 3; ++p)
          for (int q2 = 0; q2 < 3; ++q2) v[0] += mm[p] * iv[3 * p + q2] * mm[q2];
      }
      double4 d = a.dip[gi];
      double4 t = make_double4(d.x + m.x, d.y + m.y, d.z + m.z, 0.0);
      if (wfc && c.lwfc[btyp(S.t[i])] >= 0) {
        // moment_from_WFc (moment_from_pola.f90:686-738): -2 sum (r_c - r_i)
        // over the centres c with |r|^2 < rcut_wfc, in ascending centre order
        const double4 si = S.s[i];
        double w[3] = {0.0, 0.0, 0.0};
        int cnt = 0;
        for (int j = 0; j < X.n; ++j) {
          if (c.lwfc[btyp(S.t[j])] >= 0) continue;
          const double4 sj = S.s[j];
          double rx, ry, rz;
          const double r2 = min_image_exact(c.A, xsub(sj.x, si.x), xsub(sj.y, si.y), xsub(sj.z, si.z),
                                            rx, ry, rz);
          if (r2 < c.rcut_wfc) {
            ++cnt;
            w[0] += rx;
            w[1] += ry;
            w[2] += rz;
          }
        }
        if (c.lwfc[btyp(S.t[i])] > 0 && cnt != c.lwfc[btyp(S.t[i])]) v[2] = 1.0;  // :731-737
        if (c.ldip_wfc) {
          t.x = t.x + -2.0 * w[0];
          t.y = t.y + -2.0 * w[1];
          t.z = t.z + -2.0 * w[2];
        }
      }
      a.mu[gi] = t;
      if (t.x > 10.0 || t.y > 10.0 || t.z > 10.0) v[1] = 1.0;  // moment_from_pola.f90:176-178
    }
    cluster_sum<3>(cl, X, S, v);
    if (X.rank == 0 && threadIdx.x == 0) {
      out[BS_UPOL] = v[0];
      out[BS_ITER] = iters;
      out[BS_CONV] = conv;
      out[BS_RMSD] = rmsd;
      out[BS_CATA] = v[1] > 0.0 ? 1.0 : 0.0;
      out[BS_STAT] = v[2] > 0.0 ? (double)MDFF_ERR_BAD_ARGS : 0.0;
    }
  }
  // ---- final pass: forces, energy, field, stress --------------------------
  cl.sync();
  gather_vec(X, a.mu, S.v);
  __syncthreads();
  {
    double acc[kESPart];
    bforce<RM>(a, X, S, acc);
    cluster_sum<kESPart>(cl, X, S, acc);
    if (X.rank == 0 && threadIdx.x == 0)
      for (int k = 0; k < kESPart; ++k) out[BS_DIR + k] = acc[k];
  }
  __syncthreads();
  {
    bool has_mu = (c.flags & (BF_QD | BF_DD)) != 0;
    double es[7];
    const int RS = brec(cl, a, X, S, 0, task_qq, has_mu, false, has_mu, true, es);
    cluster_sum<7>(cl, X, S, es);
    if (X.rank == 0 && threadIdx.x == 0)
      for (int k = 0; k < 7; ++k) out[BS_REC + k] = es[k];
    for (int i = X.i0 + threadIdx.x; i < X.i1; i += blockDim.x) {
      const int gi = X.off + i;
      double e[3], fm[3];
      bfld_get(a, c, RS, i - X.i0, has_mu, e, fm);
      const double4 o = a.E[gi];
      a.E[gi] = make_double4(o.x + e[0], o.y + e[1], o.z + e[2], 0.0);
      const double qi = S.s[i].w;
      a.force[gi] += (qi * e[0] + fm[0]) * c.coul_unit;
      a.force[a.ntot + gi] += (qi * e[1] + fm[1]) * c.coul_unit;
      a.force[2 * (size_t)a.ntot + gi] += (qi * e[2] + fm[2]) * c.coul_unit;
    }
  }
  double m[8];
  bmoments(cl, a, X, S, a.mu, true, m);
  if (X.rank == 0 && threadIdx.x == 0)
    for (int k = 0; k < 8; ++k) out[BS_MOM + k] = m[k];
  __syncthreads();
  bself(a, X, a.mu, selfa2, lsurf, fpi_3V, m, a.E);
}

// configuration cfg becomes the cluster's: ion and polarisable-ion ranges of this CTA
__device__ __forceinline__ void bctx_set(const BatchArgs& a, BCtx& X, int cfg) {
  const BConf* c = a.conf + cfg;
  X.c = c;
  X.cfg = cfg;
  X.n = c->n;
  X.off = c->off;
  X.i0 = (int)((long long)X.n * X.rank / X.C);
  X.i1 = (int)((long long)X.n * (X.rank + 1) / X.C);
  X.npol = c->npol;
  X.p0 = (int)((long long)X.npol * X.rank / X.C);
  X.p1 = (int)((long long)X.npol * (X.rank + 1) / X.C);
  X.slot = (int)(blockIdx.x / X.C);
  X.part = a.part + (size_t)cfg * kBMaxC * 2 * kBPart;
  X.parity = 0;
  X.rpar = 0;
}

// Persistent kernel: one cluster per configuration at a time, configurations
// taken from the queue in descending cost order.
template <bool MIXED>
__global__ void __launch_bounds__(512) k_batch(BatchArgs a, int nmax) {
  extern __shared__ __align__(16) unsigned char bsm[];
  BShared S = batch_smem(bsm, nmax);
  if (a.stage_extra) {
    S.stage = bsm + batch_smem_extra_offset(nmax);
    S.stage_bytes = a.stage_extra;
  }
  cgx::cluster_group cl = cgx::this_cluster();
  BCtx X;
  X.rank = (int)cl.block_rank();
  X.C = (int)cl.num_blocks();
  X.parity = 0;
  while (true) {
    if (X.rank == 0 && threadIdx.x == 0) *S.cfg = atomicAdd(a.queue, 1);
    cl.sync();
    int qpos = *cl.map_shared_rank(S.cfg, 0);
    cl.sync();  // rank 0 may overwrite its slot only after every CTA read it
    if (qpos >= a.nconf) break;
    int cfg = a.order[qpos];
    bctx_set(a, X, cfg);
    bconfig<MIXED>(cl, a, X, S);
    __syncthreads();
  }
}

}  // namespace mdff
