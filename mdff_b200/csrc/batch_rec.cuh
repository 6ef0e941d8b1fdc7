// batch_rec.cuh -- reciprocal space (multipole_ES_rec, ewald_rec.f90:38-365)
// of one configuration of the batched engine, as register-tiled products.
//
// The mesh is rows (nx, ny) of nz = -kz..kz, and Z_{-n} = conj Z_n, so both
// signs of nz come from one pass over n = 0..kz: with P = X_nx Y_ny, the
// ion's row weight U = (q + i (nx m1 + ny m2)) P and V = i m3 P,
//   S(+-n) = a1 +- a2,  a1 = sum_i [ U c_n + i V n s_n ],  a2 = sum_i [ i U s_n + V n c_n ],
// (c_n, s_n) = Z_n: 8 multiply-adds per (row, n) for two k vectors, no phase
// recurrence, and the weights are formed once per (row, ion) instead of once
// per k.  The field is the transpose: with sigma = rho'(n) + rho'(-n) and
// delta = rho'(n) - rho'(-n),
//   T  = sum_n rho' conj(Z) = sum_n (sigma c_n - i delta s_n),
//   T1 = sum_nz nz rho' conj(Z) = sum_n n (delta c_n - i sigma s_n),
// then recarg sums are Im(conj(P) T), Im(conj(P) T1).
//
// Bound: FMA issue of the structure factor (FP32 or FP64 pipe) and the
// broadcast loads that feed it.  brho: one lane per mesh row, the ion's phase
// record (X, Y, and (c, s, n c, n s) per n, contiguous) read as broadcasts
// through L1; the warps of a CTA split (row block, ion subset), every CTA
// of the cluster takes its own ions and all rows, so a record is read by one
// CTA only; the ion subsets are summed through shared memory in FP64 in a fixed order.
// bfld: one lane per ion, (c, s) in registers, the coefficients of a row
// broadcast from shared memory; the warps split (ion block, row subset).
// Against one thread per (k tile, ion) with a phase recurrence and FP64
// weights formed per tile: see the batch kernel's figures in batch.cuh.
#pragma once
#include "common.cuh"
#include "realspace.cuh"
#include "recip.cuh"

namespace mdff {

constexpr int kBStage = 16384;  // bytes of the shared staging buffer (BShared::rho)
constexpr int kBSplit = 8;      // most row subsets of the field's ion blocks

// words of an ion: type (4 bits), polarisable flag (1), its rank among the
// polarisable ions (11); bits 16-26 of word k: the k-th polarisable ion
__host__ __device__ __forceinline__ int btyp(int t) { return t & 15; }
__host__ __device__ __forceinline__ bool bpol(int t) { return ((t >> 4) & 1) != 0; }
__host__ __device__ __forceinline__ int brank(int t) { return (t >> 5) & 2047; }
__host__ __device__ __forceinline__ int bpl(int t) { return (t >> 16) & 2047; }

// n tile of the structure factor for kz + 1 values of n (FP64: at most 8 in
// registers, more in two tiles) and the field's padded n count
inline int brho_tile(int nz, bool fp64) {
  if (fp64) {
    const int nt = (nz + 7) / 8, t = (nz + nt - 1) / nt;
    return t < 5 ? 5 : t;
  }
  return nz <= 6 ? 6 : nz <= 10 ? nz : 13;
}
inline int bfld_tile(int nz) { return nz <= 6 ? 6 : nz <= 8 ? 8 : nz <= 10 ? 10 : 13; }

// (x, y, z, w) of a record entry
__device__ __forceinline__ void bld4(const float* p, float (&v)[4]) {
  const float4 a = *reinterpret_cast<const float4*>(p);
  v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w;
}
__device__ __forceinline__ void bld4(const double* p, double (&v)[4]) {
  const double2 a = *reinterpret_cast<const double2*>(p), b = *reinterpret_cast<const double2*>(p + 2);
  v[0] = a.x; v[1] = a.y; v[2] = b.x; v[3] = b.y;
}

// the ions of a reciprocal pass on one CTA: ions n0.. (all ions) or the
// polarisable ions of rank n0.. (pol), cnt of them; the weights of entry k are
// w(k) = (q, m1, m2, m3)
struct BList {
  int n0, cnt;
  bool pol;
};
__device__ __forceinline__ int blist_ion(const BList& L, const int* t, int k) {
  return L.pol ? bpl(t[L.n0 + k]) : L.n0 + k;
}

// Partial structure factor of this CTA's ions over all rows:
// out[row * (kz + 1) + n] = (a1, a2).  stage: kBStage bytes.  W(k, w): weights
// of list entry k.
template <typename R, int T, bool HM, typename W>
__device__ __forceinline__ void brho_t(const unsigned char* __restrict__ rec, int stride, int zoff, int kx,
                                       int kz, const int4* __restrict__ rows, int nrows, const BList& L,
                                       const int* t, unsigned char* stage, double4* __restrict__ out,
                                       const W& wfun) {
  typedef typename cplx<R>::T C2;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
  const int nrb = (nrows + 31) / 32, NR = nrb < nw ? nrb : nw, ks = nw / NR;
  const int rbw = warp / ks, kk = warp % ks;
  const bool act = rbw < NR;
  const int nz = kz + 1;
  constexpr int CAP = kBStage / (4 * (int)sizeof(R));
  R* sw = reinterpret_cast<R*>(stage);
  for (int rb0 = 0; rb0 < nrb; rb0 += NR)
    for (int t0 = 0; t0 < nz; t0 += T) {
      const int row = (rb0 + rbw) * 32 + lane;
      const int4 ri = rows[row < nrows ? row : nrows - 1];
      const R fx = (R)ri.x, fy = (R)ri.y;
      const int ye = kx + 1 + (ri.y < 0 ? -ri.y : ri.y);
      const R ys = ri.y < 0 ? R(-1) : R(1);
      R acc[T][4];
#pragma unroll
      for (int u = 0; u < T; ++u) acc[u][0] = acc[u][1] = acc[u][2] = acc[u][3] = R(0);
      for (int c0 = 0; c0 < L.cnt; c0 += CAP) {
        const int cc = L.cnt - c0 < CAP ? L.cnt - c0 : CAP;
        __syncthreads();
        for (int k = threadIdx.x; k < cc; k += blockDim.x) {
          R w[4];
          wfun(c0 + k, w);
#pragma unroll
          for (int d = 0; d < 4; ++d) sw[4 * k + d] = w[d];
        }
        __syncthreads();
        if (act)
          for (int k = kk; k < cc; k += ks) {
            const unsigned char* rp = rec + (size_t)blist_ion(L, t, c0 + k) * stride;
            const C2* xy = reinterpret_cast<const C2*>(rp);
            const R* z = reinterpret_cast<const R*>(rp + zoff) + 4 * t0;
            const C2 X = xy[ri.x];
            C2 Y = xy[ye];
            Y.y *= ys;
            R w[4];
            bld4(sw + 4 * k, w);
            const C2 P = cmul(X, Y);
            const R km = fx * w[1] + fy * w[2];
            R Ur, Ui;
            if (HM) {
              Ur = w[0] * P.x - km * P.y;
              Ui = w[0] * P.y + km * P.x;
            } else {
              Ur = w[0] * P.x;
              Ui = w[0] * P.y;
            }
            const R Vr = -w[3] * P.y, Vi = w[3] * P.x;
#pragma unroll
            for (int u = 0; u < T; ++u) {
              R v[4];
              bld4(z + 4 * u, v);
              acc[u][0] += Ur * v[0];
              acc[u][1] += Ui * v[0];
              acc[u][2] -= Ui * v[1];
              acc[u][3] += Ur * v[1];
              if (HM) {
                acc[u][0] -= Vi * v[3];
                acc[u][1] += Vr * v[3];
                acc[u][2] += Vr * v[2];
                acc[u][3] += Vi * v[2];
              }
            }
          }
      }
      // sum the ion subsets (warps of one row block) in order, FP64
      constexpr int NB = sizeof(R) == 4 ? 2 : 1;  // n per round of the buffer (16 warps x 32 lanes)
#pragma unroll
      for (int u0 = 0; u0 < T; u0 += NB) {
        __syncthreads();
#pragma unroll
        for (int b = 0; b < NB; ++b)
          if (u0 + b < T) {
            R* o = sw + 4 * ((b * nw + warp) * 32 + lane);
#pragma unroll
            for (int d = 0; d < 4; ++d) o[d] = acc[u0 + b < T ? u0 + b : 0][d];
          }
        __syncthreads();
        for (int e = threadIdx.x; e < NB * NR * 32; e += blockDim.x) {
          const int b = e / (NR * 32), rr = e % (NR * 32), n = t0 + u0 + b;
          const int orow = rb0 * 32 + rr;
          if (u0 + b >= T || n >= nz || orow >= nrows) continue;
          double s[4] = {0.0, 0.0, 0.0, 0.0};
          for (int c = 0; c < ks; ++c) {
            const R* o = sw + 4 * ((b * nw + (rr >> 5) * ks + c) * 32 + (rr & 31));
#pragma unroll
            for (int d = 0; d < 4; ++d) s[d] += (double)o[d];
          }
          out[(size_t)orow * nz + n] = make_double4(s[0], s[1], s[2], s[3]);
        }
      }
    }
  __syncthreads();
}

// rho'(+n), rho'(-n) of (row, n) from the CTAs' partials (summed in rank
// order), A_k scaled; for n = 0 and the half row (0, 0) the missing partner is zero
__device__ __forceinline__ void brho_pm(const double4* __restrict__ part, size_t ld, int C, int nz,
                                        const int4& ri, int row, int n, const double* __restrict__ Ak,
                                        double2& rp, double2& rm) {
  double s[4] = {0.0, 0.0, 0.0, 0.0};
  for (int c = 0; c < C; ++c) {
    const double2* p = reinterpret_cast<const double2*>(part + (size_t)c * ld + (size_t)row * nz + n);
    const double2 u = __ldcg(p), v = __ldcg(p + 1);
    s[0] += u.x;
    s[1] += u.y;
    s[2] += v.x;
    s[3] += v.y;
  }
  // the row (0, 0) holds nz = 1..kz only (ri.z = 1), every other row -kz..kz
  const bool hp = n >= ri.z, hm = n > 0 && ri.z < 0;
  rp = hp ? make_double2(s[0] + s[2], s[1] + s[3]) : make_double2(0.0, 0.0);
  rm = hm ? make_double2(s[0] - s[2], s[1] - s[3]) : make_double2(0.0, 0.0);
  if (Ak) {
    const double Ap = hp ? Ak[ri.w + n - ri.z] : 0.0, Am = hm ? Ak[ri.w - n - ri.z] : 0.0;
    rp.x *= Ap;
    rp.y *= Ap;
    rm.x *= Am;
    rm.y *= Am;
  }
}

// row subsets per ion block: the count (up to kBSplit) that leaves the fewest
// warps idle in the last round
__device__ __forceinline__ int bfld_split(int nib, int nw) {
  int best = 1;
  double eff = 0.0;
  for (int s = 1; s <= kBSplit; ++s) {
    const int items = nib * s, rounds = (items + nw - 1) / nw;
    const double e = (double)items / (double)(rounds * nw) - 0.01 * s;
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
// tab: phase tables [entry][ion] of leading dimension ld; part: the CTAs'
// structure-factor partials.
template <typename R, int KT, bool MUF, typename W>
__device__ __forceinline__ int bfld_t(const typename cplx<R>::T* __restrict__ tab, int ld, int kx, int ky,
                                      int kz, const int4* __restrict__ rows, int nrows,
                                      const double* __restrict__ Ak, const double4* __restrict__ part,
                                      size_t pld, int C, const BList& L, const int* t,
                                      unsigned char* stage, double* __restrict__ gp, int gld, const W& wfun) {
  typedef typename cplx<R>::T C2;
  constexpr bool F32 = sizeof(R) == 4;
  constexpr int RC = kBStage / (4 * (int)sizeof(R) * KT);  // rows per staged chunk
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
  const int nib = (L.cnt + 31) / 32, nz = kz + 1;
  const int RS = nib > 0 ? bfld_split(nib, nw) : 1;
  R* sc = reinterpret_cast<R*>(stage);
  for (int ra = 0; ra < nrows; ra += RC) {
    const int nr = nrows - ra < RC ? nrows - ra : RC;
    __syncthreads();
    for (int e = threadIdx.x; e < nr * KT; e += blockDim.x) {
      const int rr = e / KT, n = e % KT;
      double2 rp = make_double2(0.0, 0.0), rm = rp;
      if (n < nz) {
        brho_pm(part, pld, C, nz, rows[ra + rr], ra + rr, n, Ak, rp, rm);
      }
      R* o = sc + 4 * e;
      o[0] = (R)(rp.x + rm.x);
      o[1] = (R)(rp.y + rm.y);
      o[2] = n ? (R)(rp.x - rm.x) : R(0);
      o[3] = n ? (R)(rp.y - rm.y) : R(0);
    }
    __syncthreads();
    for (int it = warp; it < nib * RS; it += nw) {
      const int ib = it % nib, rs = it / nib;
      const int k = ib * 32 + lane;
      const int kc = k < L.cnt ? k : L.cnt - 1;
      const C2* tb = tab + blist_ion(L, t, kc);
      // (FP64 keeps only (c, s) in registers and scales the products by n)
      R c[KT], s[KT], nc[F32 ? KT : 1], ns[F32 ? KT : 1];
#pragma unroll
      for (int n = 0; n < KT; ++n) {
        C2 z;
        z.x = z.y = R(0);
        if (n < nz) z = tb[(size_t)(kx + 1 + ky + 1 + n) * ld];
        c[n] = z.x;
        s[n] = z.y;
        if constexpr (F32) {
          nc[n] = R(n) * z.x;
          ns[n] = R(n) * z.y;
        }
      }
      R w[4] = {R(0), R(0), R(0), R(0)};
      if (MUF) wfun(kc, w);
      double G[3] = {0.0, 0.0, 0.0}, H[3] = {0.0, 0.0, 0.0};
      R g0 = R(0), g1 = R(0), g2 = R(0), h0 = R(0), h1 = R(0), h2 = R(0);
      const int q0 = (int)((long long)nr * rs / RS), q1 = (int)((long long)nr * (rs + 1) / RS);
      int nxc = q0 < q1 ? rows[ra + q0].x : 0;
      C2 X = tb[(size_t)nxc * ld];
      for (int r = q0; r < q1; ++r) {
        const int4 ri = rows[ra + r];
        if (ri.x != nxc) {
          // the sums of one nx in R, the nx sums in FP64
          G[0] += (double)nxc * (double)g0;
          G[1] += (double)g1;
          G[2] += (double)g2;
          if (MUF) {
            H[0] += (double)nxc * (double)h0;
            H[1] += (double)h1;
            H[2] += (double)h2;
          }
          g0 = g1 = g2 = h0 = h1 = h2 = R(0);
          nxc = ri.x;
          X = tb[(size_t)nxc * ld];
        }
        C2 Y = tb[(size_t)(kx + 1 + (ri.y < 0 ? -ri.y : ri.y)) * ld];
        if (ri.y < 0) Y.y = -Y.y;
        const C2 P = cmul(X, Y);
        R tr = R(0), ti = R(0), t1r = R(0), t1i = R(0), t2r = R(0), t2i = R(0);
        const R* q = sc + 4 * r * KT;
#pragma unroll
        for (int n = 0; n < KT; ++n) {
          R v[4];  // sigma, delta
          bld4(q + 4 * n, v);
          tr += v[0] * c[n];
          tr += v[3] * s[n];
          ti += v[1] * c[n];
          ti -= v[2] * s[n];
          if constexpr (F32) {
            t1r += v[2] * nc[n];
            t1r += v[1] * ns[n];
            t1i += v[3] * nc[n];
            t1i -= v[0] * ns[n];
          } else {
            t1r += R(n) * (v[2] * c[n] + v[1] * s[n]);
            t1i += R(n) * (v[3] * c[n] - v[0] * s[n]);
          }
          if (MUF) {
            t2r += R(n * n) * (v[0] * c[n] + v[3] * s[n]);
            t2i += R(n * n) * (v[1] * c[n] - v[2] * s[n]);
          }
        }
        const R S0 = P.x * ti - P.y * tr, S1 = P.x * t1i - P.y * t1r;
        const R fy = (R)ri.y;
        g0 += S0;
        g1 += fy * S0;
        g2 += S1;
        if (MUF) {
          const R R0 = P.x * tr + P.y * ti, R1 = P.x * t1r + P.y * t1i, R2 = P.x * t2r + P.y * t2i;
          const R am = (R)ri.x * w[1] + fy * w[2];
          const R y0 = am * R0 + w[3] * R1;
          h0 += y0;
          h1 += fy * y0;
          h2 += am * R1 + w[3] * R2;
        }
      }
      G[0] += (double)nxc * (double)g0;
      G[1] += (double)g1;
      G[2] += (double)g2;
      if (MUF) {
        H[0] += (double)nxc * (double)h0;
        H[1] += (double)h1;
        H[2] += (double)h2;
      }
      if (k < L.cnt)
#pragma unroll
        for (int d = 0; d < 3; ++d) {
          double* o = gp + (size_t)(rs * 6 + d) * gld + k;
          o[0] = (ra ? o[0] : 0.0) + G[d];
          if (MUF) {
            double* oh = o + 3 * (size_t)gld;
            oh[0] = (ra ? oh[0] : 0.0) + H[d];
          }
        }
    }
  }
  __syncthreads();
  return RS;
}

}  // namespace mdff
