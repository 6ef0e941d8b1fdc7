// recip_dm.cuh -- FP64 reciprocal sums of the single-configuration engine as
// tensor-core products (dmma.cuh; multipole_ES_rec, ewald_rec.f90:38-365).
//
// With the factorised phases and Z_{-n} = conj Z_n both signs of nz come from one
// product over n = 0..kz (batch_rec.cuh has the same forms): with P = X_nx Y_ny,
// U = (q + i (nx m1 + ny m2)) P and V = i m3 P of the row (nx, ny),
//   S(+-n) = a1 +- a2,  a1 = sum_i [ U c_n + i n V s_n ],  a2 = sum_i [ i U s_n + n V c_n ]
// and, sigma = rho'(n) + rho'(-n), delta = rho'(n) - rho'(-n),
//   T_p = sum_nz nz^p rho' conj(Z): T_0 = sum_n (sigma c_n - i delta s_n),
//   T_1 = sum_n n (delta c_n - i sigma s_n), T_2 = sum_n n^2 (sigma c_n - i delta s_n);
// the field, the dipole force and the field gradient follow from conj(P) T_p.
// 4 multiply-adds per (k, ion) with dipoles against about 10 operations of a phase
// recurrence with its weights.
//
//   k_rho_dm  : M = (re, im) of U and V of the rows, N = (c_n, s_n), K = ions
//   k_field_dm: M = ions, N = (re, im) of the rows, K = (c_n, s_n), times n and n^2
//
// Both are bound by the FP64 pipe (18.5e12 multiply-adds a second).  Measured on
// one B200 (cold caches, in isolation): 8000-ion MgO, kmax 16 (17,968 k), the
// 4000 dipoles of an operator application: structure factor 132 -> 39 us (the
// recurrence ran over all ions; 15.5 us at the pipe's rate), field 81 -> 39 us.
// 13,700-ion NaCl, kmax 20 (34,460 k), charges, where the FP32 recurrence ran
// in the mixed engine: 272 -> 108 us.  Whole calls: 8000-ion MgO, FP64 SCF from
// scratch (43 iterations) 12.1 -> 7.1 ms with these kernels alone; 5100-ion silica, FP64 CG
// and field gradients 1.99 -> 1.34 ms (the gradient's reciprocal part 405 -> 18 us).
#pragma once
#include "dmma.cuh"
#include "recip.cuh"
#include "shapes.h"

namespace mdff {

constexpr int kDmThreads = 512;    // k_rho_dm: 8 groups of 8 rows x 2 ion halves
constexpr int kDmFldThreads = 256; // k_field_dm: 8 warps of 16 ions
constexpr int kDmFldIons = 128;

__device__ __forceinline__ void dm_cp16(void* smem, const void* g) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((unsigned)__cvta_generic_to_shared(smem)), "l"(g)
               : "memory");
}

// Structure-factor partials: grid (row blocks, ion chunks, n passes).  imap: the
// ions with weights (nion of them; nullptr: all); w by ion; part[chunk][k].
template <int NT, bool HM>
static __global__ void __launch_bounds__(kDmThreads, 1) k_rho_dm(
    const double2* __restrict__ tab, const double4* __restrict__ w, int natm, const int* __restrict__ imap,
    int nion, int chunk, int ci, RecMesh M, double2* __restrict__ part, const int* __restrict__ stop) {
  extern __shared__ __align__(16) unsigned char dms[];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int g = lane >> 2, tt = lane & 3, rg = warp & 7, half = warp >> 3;
  const int kx = M.kmax[0], ky = M.kmax[1], kz = M.kmax[2];
  const int n0 = blockIdx.z * 4 * NT;
  const int nxy = kx + 1 + ky + 1, ent = nxy + 4 * NT, ld = ci + 4;  // ions of an entry, padded: bank spread
  double2* sp = reinterpret_cast<double2*>(dms);
  double4* sw = reinterpret_cast<double4*>(sp + (size_t)2 * ent * ld);
  const int a0 = blockIdx.y * chunk, a1 = a0 + chunk < nion ? a0 + chunk : nion;
  const int nch = (a1 - a0 + ci - 1) / ci;
  // a thread copies one ion slot of every (512 / ci)-th entry (the weights are the
  // last two); its ion index is fetched one chunk ahead
  const int fk = threadIdx.x & (ci - 1), fe = threadIdx.x / ci, fs = kDmThreads / ci;
  auto slot_ion = [&](int c) {
    const int sl = a0 + c * ci + fk < a1 ? a0 + c * ci + fk : a1 - 1;
    return imap ? imap[sl] : sl;
  };
  int inext = slot_ion(0), icur = inext;
  auto fetch_tab = [&](int c) {
    const int i = icur = inext;
    if (c + 1 < nch) inext = slot_ion(c + 1);
    double2* o = sp + (size_t)(c & 1) * ent * ld + fk;
    const double2* tb = tab + i;
    for (int en = fe; en < ent; en += fs) {
      // (entries of n > kz repeat the last one: their columns are not stored)
      const int te = en < nxy ? en : nxy + (n0 + en - nxy < kz ? n0 + en - nxy : kz);
      dm_cp16(o + en * ld, tb + (size_t)te * natm);
    }
  };
  auto fetch_w = [&](int c) {
    if (fe < 2)
      dm_cp16(reinterpret_cast<double2*>(sw + (c & 1) * ci + fk) + fe,
              reinterpret_cast<const double2*>(w + icur) + fe);
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  const int row = blockIdx.x * kDmRows + rg * 8 + g;
  const int4 ri = M.rows[row < M.nrows ? row : M.nrows - 1];
  const double fx = (double)ri.x, fy = (double)ri.y;
  const int xo = ri.x * ld, yo = (kx + 1 + (ri.y < 0 ? -ri.y : ri.y)) * ld;
  const bool yn = ri.y < 0;
  double u[NT][4], v[HM ? NT : 1][4];
#pragma unroll
  for (int s = 0; s < NT; ++s)
#pragma unroll
    for (int d = 0; d < 4; ++d) {
      u[s][d] = 0.0;
      if (HM) v[HM ? s : 0][d] = 0.0;
    }
  // the first phases travel while the weights' kernel finishes (the tables and
  // the ion map are older than it: every kernel between waits before it lets its
  // successor start)
  fetch_tab(0);
  pdl_wait();
  pdl_trigger();
  fetch_w(0);
  if (loop_stopped(stop)) {
    asm volatile("cp.async.wait_all;" ::: "memory");
    return;
  }
  for (int c = 0; c < nch; ++c) {
    if (c + 1 < nch) {
      fetch_tab(c + 1);
      fetch_w(c + 1);
      asm volatile("cp.async.wait_group 1;" ::: "memory");
    } else {
      asm volatile("cp.async.wait_group 0;" ::: "memory");
    }
    __syncthreads();
    const double2* rb = sp + (size_t)(c & 1) * ent * ld;
    const double4* wbuf = sw + (c & 1) * ci;
    const int m = a1 - a0 - c * ci < ci ? a1 - a0 - c * ci : ci;
#pragma unroll 2
    for (int k0 = 4 * half; k0 < m; k0 += 8) {
      const int k = k0 + tt;  // (past the end: the last ion's phases, weight zero)
      const double2 X = rb[xo + k];
      double2 Y = rb[yo + k];
      Y.y = flip_if(Y.y, yn);
      double4 wi = wbuf[k];
      if (k >= m) wi = make_double4(0.0, 0.0, 0.0, 0.0);
      const double2 P = cmul(X, Y);
      double Ur = wi.x * P.x, Ui = wi.x * P.y;
      if (HM) {
        const double km = fx * wi.y + fy * wi.z;
        Ur -= km * P.y;
        Ui += km * P.x;
      }
      const double Vr = -wi.w * P.y, Vi = wi.w * P.x;
      const double* zb = reinterpret_cast<const double*>(rb + (size_t)(nxy + (g >> 1)) * ld + k) + (g & 1);
#pragma unroll
      for (int s = 0; s < NT; ++s) {
        const double b = zb[(size_t)8 * s * ld];  // column g of the tile: (c, s) of n = 4 s + g / 2
        dmma(u[s], Ur, Ui, b);
        if (HM) dmma(v[HM ? s : 0], Vr, Vi, b);
      }
    }
    __syncthreads();
  }
  // the two ion halves, then S(+-n) = a1 +- a2
  double* red = reinterpret_cast<double*>(dms) + (size_t)rg * 8 * 32 + lane;
  double2* out = part + (size_t)blockIdx.y * M.nk;
#pragma unroll
  for (int s = 0; s < NT; ++s) {
    double* U = u[s];
    double* V = v[HM ? s : 0];
    if (half) {
#pragma unroll
      for (int d = 0; d < 4; ++d) {
        red[d * 32] = U[d];
        if (HM) red[(4 + d) * 32] = V[d];
      }
    }
    __syncthreads();
    if (!half) {
#pragma unroll
      for (int d = 0; d < 4; ++d) {
        U[d] += red[d * 32];
        if (HM) V[d] += red[(4 + d) * 32];
      }
      const int n = n0 + 4 * s + tt;
      if (row < M.nrows && n <= kz) {
        const double fn = (double)n;
        double p = U[0], q = U[2], r = -U[3], t = U[1];
        if (HM) {
          p -= fn * V[3];
          q += fn * V[1];
          r += fn * V[0];
          t += fn * V[2];
        }
        if (n >= ri.z) out[ri.w + n - ri.z] = make_double2(p + r, q + t);
        if (n > 0 && ri.z < 0) out[ri.w - n - ri.z] = make_double2(p - r, q - t);
      }
    }
    __syncthreads();
  }
}

// rho over the chunks (as k_rec_sum): 32 k x 8 chunk subsets per block, the
// subsets added in order; up to a few tens of chunks
static __global__ void __launch_bounds__(256) k_rec_sum8(const double2* __restrict__ part, int nchunk, RecMesh M,
                                                         double2* __restrict__ rhoA, double* __restrict__ epart,
                                                         double2* __restrict__ acc, const int* __restrict__ stop) {
  const bool stopped = loop_stopped(stop);
  pdl_wait();
  pdl_trigger();
  if (stopped) return;
  __shared__ double2 sh[8][32];
  const int lx = threadIdx.x & 31, ly = threadIdx.x >> 5;
  const int k = blockIdx.x * 32 + lx;
  double r = 0.0, im = 0.0;
  if (k < M.nk)
    for (int c = ly; c < nchunk; c += 8) {
      const double2 v = part[(size_t)c * M.nk + k];
      r += v.x;
      im += v.y;
    }
  sh[ly][lx] = make_double2(r, im);
  __syncthreads();
  if (ly != 0) return;
#pragma unroll
  for (int y = 1; y < 8; ++y) {
    r += sh[y][lx].x;
    im += sh[y][lx].y;
  }
  double ev[7] = {0, 0, 0, 0, 0, 0, 0};
  if (k < M.nk) {
    const double A = M.Ak[k];
    const double2 ra = make_double2(A * r, A * im);
    rhoA[k] = ra;
    if (acc) acc[k] = ra;
    if (epart) rec_energy_terms((r * r + im * im) * A, M.kvec[k], ev);
  }
  if (!epart) return;
#pragma unroll
  for (int a = 0; a < 7; ++a) ev[a] = warp_sum(ev[a]);
  if (lx == 0)
    for (int a = 0; a < 7; ++a) epart[(size_t)blockIdx.x * 7 + a] = ev[a];
}

// ---------------------------------------------------------------------------
// what k_field_dm sums per ion: the field (G = sum n recarg), the field and the
// dipole force (H = sum n (k.m) recarg2), the field gradient (G = sum (nx^2, ny^2,
// nz^2) recarg2, H = sum (nx ny, nx nz, ny nz) recarg2)
enum { DM_FIELD = 0, DM_FORCE = 1, DM_EFG = 2 };

// steps of two n (instantiated counts), doubles per staged row
inline int field_dm_ks(int kz) {
  const int ks = kz / 2 + 1;
  if (ks > 16) return 0;
  return ks <= 3 ? 3 : ks <= 9 ? ks : ks <= 11 ? 11 : ks <= 13 ? 13 : 16;
}
__host__ __device__ constexpr int field_dm_rl(int ks) { return 8 * ks + (ks % 2 == 0 ? 8 : 0); }

// Field partials: grid (ion tiles of 128, row groups of rpg rows, a multiple of
// 4); dynamic shared memory for rc staged rows.  imap (nion entries): the ions
// whose sums are wanted (nullptr: all).  A warp holds (c, s) of its 16 ions and
// walks the rows four at a time: lane (g, tt) ends with row tt's T of ions g, g + 8.
template <int KS, int MODE>
static __global__ void __launch_bounds__(kDmFldThreads, KS <= 9 ? 2 : 1) k_field_dm(
    const double2* __restrict__ tab, const double4* __restrict__ w, int natm, const int* __restrict__ imap,
    int nion, RecMesh M, const double2* __restrict__ rhoA, int rpg, int rc, double4* __restrict__ Gpart,
    double4* __restrict__ Hpart, const int* __restrict__ stop) {
  constexpr int KN = 2 * KS, RL = field_dm_rl(KS);
  const bool stopped = loop_stopped(stop);
  constexpr bool AN = KS <= 9 && MODE == DM_FIELD;  // n (c, s) in registers too
  extern __shared__ __align__(16) unsigned char dms[];
  int4* srow = reinterpret_cast<int4*>(dms);  // the chunk's rows
  double* sc = reinterpret_cast<double*>(srow + rc);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int g = lane >> 2, tt = lane & 3;
  const int kx = M.kmax[0], ky = M.kmax[1], kz = M.kmax[2];
  // B fragment: k = (n, c or s) of lane tt, column = (row, re or im) of lane g,
  // picked from the staged (sigma_r, sigma_i, delta_r, delta_i) by index and sign
  const int isS = tt & 1, comp = g & 1;
  const int i0 = isS ? 3 - comp : comp, i1 = isS ? 1 - comp : 2 + comp;
  const bool neg = isS && comp;
  const int boff = (g >> 1) * RL + (tt >> 1) * 4;
  const int s0 = blockIdx.x * kDmFldIons + warp * 16;
  const bool wact = s0 < nion;
  int ion[2];
  double a[2][KS], an[2][AN ? KS : 1];
  double4 wi[2];
#pragma unroll
  for (int q = 0; q < 2; ++q) {
    int sl = s0 + 8 * q + g;
    sl = sl < nion ? sl : nion - 1;
    ion[q] = imap ? imap[sl] : sl;
#pragma unroll
    for (int s = 0; s < KS; ++s) {
      const int n = 2 * s + (tt >> 1);
      double z = 0.0;
      if (n <= kz) z = reinterpret_cast<const double*>(tab + (size_t)(kx + 1 + ky + 1 + n) * natm + ion[q])[isS];
      a[q][s] = z;
      if (AN) an[q][AN ? s : 0] = (double)n * z;
    }
  }
  // (the phases above are older than the kernel that sums rho', as in k_rho_dm)
  pdl_wait();
  pdl_trigger();
  if (stopped) return;
  if (MODE == DM_FORCE)
#pragma unroll
    for (int q = 0; q < 2; ++q) wi[q] = w[ion[q]];
  double G[2][3], H[2][3];
#pragma unroll
  for (int q = 0; q < 2; ++q)
#pragma unroll
    for (int d = 0; d < 3; ++d) G[q][d] = H[q][d] = 0.0;
  const int r0 = blockIdx.y * rpg, r1 = r0 + rpg < M.nrows ? r0 + rpg : M.nrows;
  for (int ra = r0; ra < r1; ra += rc) {
    const int nr = r1 - ra < rc ? r1 - ra : rc, nr4 = (nr + 3) / 4;
    __syncthreads();
    for (int r = threadIdx.x; r < nr4 * 4; r += kDmFldThreads) srow[r] = M.rows[ra + (r < nr ? r : nr - 1)];
    __syncthreads();
#pragma unroll 4
    for (int e = threadIdx.x; e < nr4 * 4 * KN; e += kDmFldThreads) {
      const int rr = e / KN, n = e - rr * KN;
      const int4 ri = srow[rr];
      // (a row past the end and an n past kz have zero coefficients)
      const bool hp = rr < nr && n <= kz && n >= ri.z, hm = rr < nr && n <= kz && n > 0 && ri.z < 0;
      double2 rp = rhoA[hp ? ri.w + n - ri.z : 0], rm = rhoA[hm ? ri.w - n - ri.z : 0];
      if (!hp) rp = make_double2(0.0, 0.0);
      if (!hm) rm = make_double2(0.0, 0.0);
      double2* o = reinterpret_cast<double2*>(sc + (size_t)rr * RL + 4 * n);
      o[0] = make_double2(rp.x + rm.x, rp.y + rm.y);
      o[1] = n ? make_double2(rp.x - rm.x, rp.y - rm.y) : make_double2(0.0, 0.0);
    }
    __syncthreads();
    if (wact) {
      // this lane's row of the four, X and Y of its ions one step ahead
      double2 Xn[2], Yn[2];
      auto next = [&](int r4) {
        const int4 rn = srow[r4 * 4 + tt];
        const int ye = kx + 1 + (rn.y < 0 ? -rn.y : rn.y);
#pragma unroll
        for (int q = 0; q < 2; ++q) {
          Xn[q] = tab[(size_t)rn.x * natm + ion[q]];
          Yn[q] = tab[(size_t)ye * natm + ion[q]];
        }
      };
      next(0);
      for (int r4 = 0; r4 < nr4; ++r4) {
        const double2 X[2] = {Xn[0], Xn[1]}, Y[2] = {Yn[0], Yn[1]};
        if (r4 + 1 < nr4) next(r4 + 1);
        double d0[4] = {0, 0, 0, 0}, d1[4] = {0, 0, 0, 0}, d2[4] = {0, 0, 0, 0};
        const double* b = sc + (size_t)r4 * 4 * RL + boff;
#pragma unroll
        for (int s = 0; s < KS; ++s) {
          const double b0 = flip_if(b[8 * s + i0], neg), b1 = flip_if(b[8 * s + i1], neg);
          const double fn = (double)(2 * s + (tt >> 1));
          double n0, n1;
          if (AN) {
            n0 = an[0][AN ? s : 0];
            n1 = an[1][AN ? s : 0];
          } else {
            n0 = fn * a[0][s];
            n1 = fn * a[1][s];
          }
          dmma(d0, a[0][s], a[1][s], b0);
          dmma(d1, n0, n1, b1);
          if (MODE != DM_FIELD) dmma(d2, fn * n0, fn * n1, b0);
        }
        const int4 ri = srow[r4 * 4 + tt];
        const double fx = (double)ri.x, fy = (double)ri.y;
#pragma unroll
        for (int q = 0; q < 2; ++q) {
          const double2 P = cmul(X[q], make_double2(Y[q].x, flip_if(Y[q].y, ri.y < 0)));
          const double tr = d0[2 * q], ti = d0[2 * q + 1], ur = d1[2 * q], ui = d1[2 * q + 1];
          if (MODE != DM_EFG) {
            const double S0 = P.x * ti - P.y * tr, S1 = P.x * ui - P.y * ur;
            G[q][0] += fx * S0;
            G[q][1] += fy * S0;
            G[q][2] += S1;
          }
          if (MODE != DM_FIELD) {
            const double vr = d2[2 * q], vi = d2[2 * q + 1];
            const double R0 = P.x * tr + P.y * ti, R1 = P.x * ur + P.y * ui, R2 = P.x * vr + P.y * vi;
            if (MODE == DM_FORCE) {
              const double am = fx * wi[q].y + fy * wi[q].z;
              const double y0 = am * R0 + wi[q].w * R1;
              H[q][0] += fx * y0;
              H[q][1] += fy * y0;
              H[q][2] += am * R1 + wi[q].w * R2;
            } else {
              const double xr = fx * R0;
              G[q][0] += fx * xr;
              G[q][1] += fy * (fy * R0);
              G[q][2] += R2;
              H[q][0] += fy * xr;
              H[q][1] += fx * R1;
              H[q][2] += fy * R1;
            }
          }
        }
      }
    }
  }
  if (!wact) return;
#pragma unroll
  for (int q = 0; q < 2; ++q) {
#pragma unroll
    for (int d = 0; d < 3; ++d) {
      G[q][d] += __shfl_xor_sync(FULL_MASK, G[q][d], 1);
      G[q][d] += __shfl_xor_sync(FULL_MASK, G[q][d], 2);
      if (MODE != DM_FIELD) {
        H[q][d] += __shfl_xor_sync(FULL_MASK, H[q][d], 1);
        H[q][d] += __shfl_xor_sync(FULL_MASK, H[q][d], 2);
      }
    }
    if (s0 + 8 * q + g >= nion) continue;
    const size_t o = (size_t)blockIdx.y * natm + ion[q];
    if (tt == 0) Gpart[o] = make_double4(G[q][0], G[q][1], G[q][2], 0.0);
    if (MODE != DM_FIELD && tt == 1) Hpart[o] = make_double4(H[q][0], H[q][1], H[q][2], 0.0);
  }
}

// reciprocal electric field gradient from the row groups' sums (ewald_rec.f90:
// 209-217): k_a k_b = 4 pi^2 sum_pq B_ap B_bq n_p n_q, upper triangle only, as the
// reference; scaled by 2 fpi_V and added into efg[i][9]
static __global__ void k_efg_rec_sum(const double4* __restrict__ Gpart, const double4* __restrict__ Hpart, int ng,
                                     int natm, const CellC* __restrict__ cell, double scale,
                                     double* __restrict__ efg) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= natm) return;
  double N[6] = {0, 0, 0, 0, 0, 0};  // xx yy zz xy xz yz
  for (int c = 0; c < ng; ++c) {
    const double4 a = Gpart[(size_t)c * natm + i], b = Hpart[(size_t)c * natm + i];
    N[0] += a.x;
    N[1] += a.y;
    N[2] += a.z;
    N[3] += b.x;
    N[4] += b.y;
    N[5] += b.z;
  }
  const double* B = cell->B;
  const double Nm[3][3] = {{N[0], N[3], N[4]}, {N[3], N[1], N[5]}, {N[4], N[5], N[2]}};
  for (int a = 0; a < 3; ++a)
    for (int b = a; b < 3; ++b) {
      double v = 0.0;
      for (int p = 0; p < 3; ++p)
        for (int q = 0; q < 3; ++q) v += B[3 * a + p] * B[3 * b + q] * Nm[p][q];
      efg[9 * (size_t)i + 3 * a + b] += kTwoPi * kTwoPi * v * scale;
    }
}

}  // namespace mdff
