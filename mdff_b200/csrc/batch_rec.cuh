// batch_rec.cuh -- reciprocal space (multipole_ES_rec, ewald_rec.f90:38-365)
// of one configuration of the batched engine, as FP64 tensor-core products.
//
// The mesh is rows (nx, ny) of nz = -kz..kz, and Z_{-n} = conj Z_n, so both
// signs of nz come from one product over n = 0..kz: with P = X_nx Y_ny, the
// ion's row weight U = (q + i (nx m1 + ny m2)) P and V = i m3 P,
//   S(+-n) = a1 +- a2,  a1 = sum_i [ U c_n + i n V s_n ],  a2 = sum_i [ i U s_n + n V c_n ],
// (c_n, s_n) = Z_n: a product with M = (re, im) of U and V of the rows, N =
// (c_n, s_n), K = ions, 8 multiply-adds per (row, n) for two k vectors and no phase
// recurrence.  The field is the transpose: with sigma = rho'(n) + rho'(-n) and
// delta = rho'(n) - rho'(-n),
//   T  = sum_nz rho' conj(Z) = sum_n (sigma c_n - i delta s_n),
//   T1 = sum_nz nz rho' conj(Z) = sum_n n (delta c_n - i sigma s_n),
// a product with M = ions, K = (c_n, s_n) (times n, n^2), N = (re, im) of the rows; the recarg
// sums are Im(conj(P) T), Im(conj(P) T1).
//
// Bound: the FP64 pipe.  brho: a warp owns 8 mesh rows and all ions of its CTA
// (no sum over warps), four ions a step; the ions' phase records (X, Y, then
// (c, s) per n, contiguous) pass through shared memory in two buffers.  Every
// CTA of the cluster takes its own ions and all rows; the CTAs' partial sums
// meet in the field's staging.  bfld: a warp owns 16 ions, their (c, s) in
// registers, and a subset of the rows, four rows a step, whose coefficients are
// staged in shared memory.  Measured inside the batch kernel (256 boxes of
// 64-1000 ions, mixed, 2 CTAs x 512 threads), one structure factor of the dipole
// operator on one CTA, 133 ions x 113 rows on average: 22 us (43 us with the
// records read through L1; 31 us as FP32 register tiles of one lane per row
// pair, whose 16-byte broadcast loads and sums over warps cost more than their
// FMAs; the FMAs alone at the FP64 rate 8.6 us); one field 25 us (27 us in FP32).
#pragma once
#include "common.cuh"
#include "dmma.cuh"
#include "realspace.cuh"
#include "recip.cuh"
#include "shapes.h"

namespace mdff {

constexpr int kBSplit = 8;      // most row subsets of the field's ion blocks

// words of an ion: type (4 bits), polarisable flag (1), its rank among the
// polarisable ions (11); bits 16-26 of word k: the k-th polarisable ion
__host__ __device__ __forceinline__ int btyp(int t) { return t & 15; }
__host__ __device__ __forceinline__ bool bpol(int t) { return ((t >> 4) & 1) != 0; }
__host__ __device__ __forceinline__ int brank(int t) { return (t >> 5) & 2047; }
__host__ __device__ __forceinline__ int bpl(int t) { return (t >> 16) & 2047; }

// the ions of a reciprocal pass on one CTA: ions n0.. (all ions) or the
// polarisable ions of rank n0.. (pol), cnt of them
struct BList {
  int n0, cnt;
  bool pol;
};
__device__ __forceinline__ int blist_ion(const BList& L, const int* t, int k) {
  return L.pol ? bpl(t[L.n0 + k]) : L.n0 + k;
}

__device__ __forceinline__ void cp_async16(void* smem, const void* g) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((unsigned)__cvta_generic_to_shared(smem)), "l"(g)
               : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() {
  asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}

// Partial structure factor of this CTA's ions over all rows: out[row * (kz + 1)
// + n] = (a1, a2).  w: weights (q, m1, m2, m3) of the list entries.  NT: tiles of
// four n, covering kz + 1.  The records pass through shared memory (buf, two
// buffers of CH records), every warp reading all of them.
// HM: 0 charges only, 1 charges and dipoles, 2 the product with a second vector u
// (weights (., u1, u2, u3) at w + cnt): sum_i (k.u_i)(q_i + i k.m_i) P_i.  Its row weight
// is a polynomial in n, alpha + n beta + n^2 gamma; gamma's share goes to U's
// accumulator with n^2 (c_n, s_n) as operand.  rot: the sums times i.
template <int NT, int HM>
__device__ __forceinline__ void brho_t(const unsigned char* __restrict__ rec, int stride, int zoff, int kx,
                                       int kz, const int4* __restrict__ rows, int nrows, const BList& L,
                                       const int* t, const double4* w, unsigned char* buf, int CH,
                                       double4* __restrict__ out, bool rot = false) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
  const int g = lane >> 2, tt = lane & 3;
  const int ng = (nrows + 7) / 8, nz = kz + 1;
  const int pieces = stride / 16, nch = (L.cnt + CH - 1) / CH;
  // a warp copies whole records, a lane a 16-byte piece of each
  auto fetch = [&](int c) {
    const int k0 = c * CH, m = L.cnt - k0 < CH ? L.cnt - k0 : CH;
    unsigned char* o = buf + (size_t)(c & 1) * CH * stride;
    for (int k = warp; k < m; k += nw) {
      const unsigned char* rp = rec + (size_t)blist_ion(L, t, k0 + k) * stride;
      for (int pc = lane; pc < pieces; pc += 32) cp_async16(o + k * stride + pc * 16, rp + pc * 16);
    }
    cp_async_commit();
  };
  for (int it0 = 0; it0 < ng; it0 += nw) {
    const int it = it0 + warp;
    const bool act = it < ng;
    const int row = it * 8 + g;
    const int4 ri = rows[row < nrows ? row : nrows - 1];
    const double fx = (double)ri.x, fy = (double)ri.y;
    const int xo = ri.x * 16, yo = (kx + 1 + (ri.y < 0 ? -ri.y : ri.y)) * 16;
    const bool yn = ri.y < 0;
    double u[NT][4], v[HM ? NT : 1][4];
#pragma unroll
    for (int q = 0; q < NT; ++q)
#pragma unroll
      for (int d = 0; d < 4; ++d) {
        u[q][d] = 0.0;
        if (HM) v[HM ? q : 0][d] = 0.0;
      }
    if (nch > 0) fetch(0);
    for (int c = 0; c < nch; ++c) {
      if (c + 1 < nch) {
        fetch(c + 1);
        cp_async_wait<1>();
      } else {
        cp_async_wait<0>();
      }
      __syncthreads();
      if (act) {
        const int kb = c * CH, m = L.cnt - kb < CH ? L.cnt - kb : CH;
        const unsigned char* rb = buf + (size_t)(c & 1) * CH * stride;
#pragma unroll 2
        for (int k0 = 0; k0 < m; k0 += 4) {
          const bool ok = k0 + tt < m;  // weights zero past the end
          const int k = ok ? k0 + tt : k0;
          const unsigned char* rp = rb + k * stride;
          const double2 X = *reinterpret_cast<const double2*>(rp + xo);
          double2 Y = *reinterpret_cast<const double2*>(rp + yo);
          Y.y = flip_if(Y.y, yn);
          const double2* wp = reinterpret_cast<const double2*>(w + kb + k);
          double2 wa = wp[0], wb = wp[1];
          if (!ok) wa.x = wa.y = wb.x = wb.y = 0.0;
          const double2 P = cmul(X, Y);
          if (HM == 2) {
            const double2* up = wp + 2 * (size_t)L.cnt;
            double2 ua = up[0], ub = up[1];
            if (!ok) ua.y = ub.x = ub.y = 0.0;
            const double km = fx * wa.y + fy * wb.x, ku = fx * ua.y + fy * ub.x;
            const double a0 = ku * wa.x, a1 = ku * km, b0 = wa.x * ub.y, b1 = km * ub.y + ku * wb.y, g1 = wb.y * ub.y;
            const double Ur = a0 * P.x - a1 * P.y, Ui = a0 * P.y + a1 * P.x;
            const double Vr = b0 * P.x - b1 * P.y, Vi = b0 * P.y + b1 * P.x;
            const double Gr = -g1 * P.y, Gi = g1 * P.x;
#pragma unroll
            for (int s = 0; s < NT; ++s) {
              const double b = reinterpret_cast<const double*>(rp + zoff)[8 * s + g];
              const double fn = (double)(4 * s + (g >> 1));
              dmma(u[s], Ur, Ui, b);
              dmma(v[HM ? s : 0], Vr, Vi, b);
              dmma(u[s], Gr, Gi, fn * fn * b);
            }
            continue;
          }
          double Ur = wa.x * P.x, Ui = wa.x * P.y;
          if (HM) {
            const double km = fx * wa.y + fy * wb.x;
            Ur -= km * P.y;
            Ui += km * P.x;
          }
          const double Vr = -wb.y * P.y, Vi = wb.y * P.x;
#pragma unroll
          for (int s = 0; s < NT; ++s) {
            const double b = reinterpret_cast<const double*>(rp + zoff)[8 * s + g];
            dmma(u[s], Ur, Ui, b);
            if (HM) dmma(v[HM ? s : 0], Vr, Vi, b);
          }
        }
      }
      __syncthreads();
    }
    if (act && row < nrows) {
#pragma unroll
      for (int s = 0; s < NT; ++s) {
        // columns 2 tt, 2 tt + 1 = c_n, s_n of n
        const int n = 4 * s + tt;
        if (n >= nz) continue;
        const double fn = (double)n;
        const double* U = u[s];
        const double* V = v[HM ? s : 0];
        double4 o = make_double4(U[0], U[2], -U[3], U[1]);
        if (HM) {
          o.x -= fn * V[3];
          o.y += fn * V[1];
          o.z += fn * V[0];
          o.w += fn * V[2];
        }
        if (HM == 2 && rot) o = make_double4(-o.y, o.x, -o.w, o.z);
        out[(size_t)row * nz + n] = o;
      }
    }
  }
}

// A_k rho(+n), A_k rho(-n) of (row, n) from the C CTAs' partials (summed in rank
// order); apm: (A(+n), A(-n)) by (row, n), zero where the mesh has no such k
__device__ __forceinline__ void brho_pm(const double4* __restrict__ part, size_t ld, int C, size_t e,
                                        const double2* __restrict__ apm, double2& rp, double2& rm) {
  const double2 A = apm ? apm[e] : make_double2(1.0, 1.0);
  double s[4] = {0.0, 0.0, 0.0, 0.0};
  for (int c = 0; c < C; c += 2) {
    const double2* p = reinterpret_cast<const double2*>(part + (size_t)c * ld + e);
    const double2* p2 = reinterpret_cast<const double2*>(part + (size_t)(c + 1 < C ? c + 1 : c) * ld + e);
    const double2 u = __ldcg(p), v = __ldcg(p + 1);
    double2 u2 = __ldcg(p2), v2 = __ldcg(p2 + 1);
    if (c + 1 >= C) u2.x = u2.y = v2.x = v2.y = 0.0;
    s[0] = s[0] + u.x + u2.x;
    s[1] = s[1] + u.y + u2.y;
    s[2] = s[2] + v.x + v2.x;
    s[3] = s[3] + v.y + v2.y;
  }
  rp = make_double2(A.x * (s[0] + s[2]), A.x * (s[1] + s[3]));
  rm = make_double2(A.y * (s[0] - s[2]), A.y * (s[1] - s[3]));
}

// row subsets per ion block: the count (up to kBSplit) that leaves the fewest
// warps idle in the last round, less 4 % per subset for an item's start-up
// (loading the ions' phases, summing over lanes)
__device__ __forceinline__ int bfld_split(int nib, int nw) {
  int best = 1;
  double eff = 0.0;
  for (int s = 1; s <= kBSplit; ++s) {
    const int items = nib * s, rounds = (items + nw - 1) / nw;
    const double e = (double)items / (double)(rounds * nw) - 0.04 * s;
    if (e > eff) {
      eff = e;
      best = s;
    }
  }
  return best;
}

// Field (and dipole-force) sums of this CTA's ions over all k:
// gp[(s * 6 + d) * gld + k], d = 0..2: sum_k n recarg, 3..5 (MUF): sum_k n
// (k.m) recarg2, for row subset s = 0..split-1 of list entry k; returns split.
// part: the CTAs' structure-factor partials.  KS: steps of two n, covering kz + 1.
// W(k, w): dipole weights of list entry k (MUF).
template <int KS, bool MUF, typename W>
__device__ __forceinline__ int bfld_t(const unsigned char* __restrict__ rec, int stride, int zoff, int kx, int kz,
                                      const int4* __restrict__ rows, int nrows, const double2* __restrict__ apm,
                                      const double4* __restrict__ part, size_t pld, int C, const BList& L,
                                      const int* t, unsigned char* stage, int stage_bytes, double* __restrict__ gp,
                                      int gld, const W& wfun) {
  constexpr int KN = 2 * KS;                             // padded n count
  constexpr int RL = 4 * KN + (KS % 2 == 0 ? 8 : 0);     // doubles per staged row (bank spread)
  const int RC = stage_bytes / (RL * 8) / 4 * 4;         // rows per staged chunk
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
  const int g = lane >> 2, tt = lane & 3;
  const int nib = (L.cnt + 15) / 16, nz = kz + 1;
  const int RS = nib > 0 ? bfld_split(nib, nw) : 1;
  double* sc = reinterpret_cast<double*>(stage);
  // B[k][col]: k = (n, c or s) of lane tt, col = (row, re or im) of lane g; the
  // values sigma, delta (re, im) of (row, n) are staged once and picked by index and sign:
  //   T:  re = sigma_r c + delta_i s,  im = sigma_i c - delta_r s
  //   T1: re = delta_r (n c) + sigma_i (n s),  im = delta_i (n c) - sigma_r (n s)
  const int isS = tt & 1, comp = g & 1;
  const int i0 = isS ? 3 - comp : comp, i1 = isS ? 1 - comp : 2 + comp;
  const bool neg = isS && comp;
  const int boff = (g >> 1) * RL + (tt >> 1) * 4;
  for (int ra = 0; ra < nrows; ra += RC) {
    const int nr = nrows - ra < RC ? nrows - ra : RC, nr4 = (nr + 3) / 4;
    __syncthreads();
    for (int e = threadIdx.x; e < nr4 * 4 * KN; e += blockDim.x) {
      const int rr = e / KN, n = e % KN;
      double2 rp = make_double2(0.0, 0.0), rm = rp;
      if (n < nz && rr < nr) brho_pm(part, pld, C, (size_t)(ra + rr) * nz + n, apm, rp, rm);
      double2* o = reinterpret_cast<double2*>(sc + (size_t)rr * RL + 4 * n);
      o[0] = make_double2(rp.x + rm.x, rp.y + rm.y);
      o[1] = n ? make_double2(rp.x - rm.x, rp.y - rm.y) : make_double2(0.0, 0.0);
    }
    __syncthreads();
    for (int it = warp; it < nib * RS; it += nw) {
      const int ib = it % nib, rs = it / nib;
      const unsigned char* rp[2];
      double a[2][KS], an[2][KS], w[2][4];
#pragma unroll
      for (int q = 0; q < 2; ++q) {
        const int k = ib * 16 + 8 * q + g;
        const int kc = k < L.cnt ? k : L.cnt - 1;
        rp[q] = rec + (size_t)blist_ion(L, t, kc) * stride;
        const double* z = reinterpret_cast<const double*>(rp[q] + zoff);
#pragma unroll
        for (int s = 0; s < KS; ++s) {
          a[q][s] = z[4 * s + tt];
          an[q][s] = (double)(2 * s + (tt >> 1)) * a[q][s];
        }
        if (MUF) wfun(kc, w[q]);
      }
      double G[2][3], H[2][3];
#pragma unroll
      for (int q = 0; q < 2; ++q)
#pragma unroll
        for (int d = 0; d < 3; ++d) G[q][d] = H[q][d] = 0.0;
      const int q0 = nr4 * rs / RS, q1 = nr4 * (rs + 1) / RS;
      // this lane's row of the four: indices two steps ahead, X and Y one
      auto row_of = [&](int r4) {
        const int r = ra + r4 * 4 + tt;
        return rows[r < nrows ? r : nrows - 1];
      };
      int4 r1 = row_of(q0), r2 = row_of(q0 + 1);
      double2 Xn[2], Yn[2];
      auto next = [&](const int4& rn) {
        const int ye = kx + 1 + (rn.y < 0 ? -rn.y : rn.y);
#pragma unroll
        for (int q = 0; q < 2; ++q) {
          Xn[q] = reinterpret_cast<const double2*>(rp[q])[rn.x];
          Yn[q] = reinterpret_cast<const double2*>(rp[q])[ye];
        }
      };
      next(r1);
      for (int r4 = q0; r4 < q1; ++r4) {
        const int4 ri = r1;
        const double2 X[2] = {Xn[0], Xn[1]}, Y[2] = {Yn[0], Yn[1]};
        r1 = r2;
        next(r1);
        r2 = row_of(r4 + 2);
        double d0[4] = {0, 0, 0, 0}, d1[4] = {0, 0, 0, 0}, d2[4] = {0, 0, 0, 0};
        const double* b = sc + (size_t)r4 * 4 * RL + boff;
#pragma unroll
        for (int s = 0; s < KS; ++s) {
          const double b0 = flip_if(b[8 * s + i0], neg), b1 = flip_if(b[8 * s + i1], neg);
          dmma(d0, a[0][s], a[1][s], b0);
          dmma(d1, an[0][s], an[1][s], b1);
          if (MUF) {
            const double fn = (double)(2 * s + (tt >> 1));
            dmma(d2, fn * an[0][s], fn * an[1][s], b0);
          }
        }
        const double fx = (double)ri.x, fy = (double)ri.y;
#pragma unroll
        for (int q = 0; q < 2; ++q) {
          const double2 P = cmul(X[q], make_double2(Y[q].x, flip_if(Y[q].y, ri.y < 0)));
          const double tr = d0[2 * q], ti = d0[2 * q + 1], ur = d1[2 * q], ui = d1[2 * q + 1];
          const double S0 = P.x * ti - P.y * tr, S1 = P.x * ui - P.y * ur;
          G[q][0] += fx * S0;
          G[q][1] += fy * S0;
          G[q][2] += S1;
          if (MUF) {
            const double vr = d2[2 * q], vi = d2[2 * q + 1];
            const double R0 = P.x * tr + P.y * ti, R1 = P.x * ur + P.y * ui, R2 = P.x * vr + P.y * vi;
            const double am = fx * w[q][1] + fy * w[q][2];
            const double y0 = am * R0 + w[q][3] * R1;
            H[q][0] += fx * y0;
            H[q][1] += fy * y0;
            H[q][2] += am * R1 + w[q][3] * R2;
          }
        }
      }
      // (a row past the end has zero coefficients)
#pragma unroll
      for (int q = 0; q < 2; ++q)
#pragma unroll
        for (int d = 0; d < 3; ++d) {
          G[q][d] += __shfl_xor_sync(FULL_MASK, G[q][d], 1);
          G[q][d] += __shfl_xor_sync(FULL_MASK, G[q][d], 2);
          if (MUF) {
            H[q][d] += __shfl_xor_sync(FULL_MASK, H[q][d], 1);
            H[q][d] += __shfl_xor_sync(FULL_MASK, H[q][d], 2);
          }
        }
      // lane tt writes component tt of its two ions
      if (tt < 3) {
#pragma unroll
        for (int q = 0; q < 2; ++q) {
          const int k = ib * 16 + 8 * q + g;
          if (k >= L.cnt) continue;
          double* o = gp + (size_t)(rs * 6 + tt) * gld + k;
          o[0] = (ra ? o[0] : 0.0) + (tt == 0 ? G[q][0] : tt == 1 ? G[q][1] : G[q][2]);
          if (MUF) {
            double* oh = o + 3 * (size_t)gld;
            oh[0] = (ra ? oh[0] : 0.0) + (tt == 0 ? H[q][0] : tt == 1 ? H[q][1] : H[q][2]);
          }
        }
      }
    }
  }
  __syncthreads();
  return RS;
}

}  // namespace mdff
