// pim.cuh -- induced-dipole (PIM) solve and the self / surface terms.
//
//  * SCF: moment_from_pola_scf (moment_from_pola.f90:240-485) step by step:
//    induced_moment (:955-993), ASPC predictor/corrector (:493-598),
//    u_pol (:387-395), get_rmsd_mu (:998-1027).
//  * CG:  preconditioned conjugate gradients on (alpha^-1 - T) mu = E_stat,
//    the linear system whose fixed point the SCF iterates to; preconditioner
//    alpha; stop on the reference's rmsd measure (for diagonal alpha the CG
//    residual E - alpha^-1 mu is exactly (mu/alpha_aa - E) up to sign).
//  * self and surface field terms of multipole_ES (ewald.f90:182-213).
// Vectors are double4 [natm] (xyz + pad).  Reductions are per-block partials
// summed in a fixed order (deterministic).
#pragma once
#include "common.cuh"

namespace mdff {

struct PolDev {
  const double* pol;     // [natm][9] poldipia (row-major a,b)
  const double* invpol;  // [natm][9]
  const int* ipolar;     // [natm]
};

__device__ __forceinline__ double4 matvec3(const double* m, double4 v) {
  return make_double4(m[0] * v.x + m[1] * v.y + m[2] * v.z, m[3] * v.x + m[4] * v.y + m[5] * v.z,
                      m[6] * v.x + m[7] * v.y + m[8] * v.z, 0.0);
}

// mu_i = alpha_i E_i on polarisable ions, 0 elsewhere (induced_moment)
__global__ void k_induce(const double4* __restrict__ E, PolDev P, int natm, double4* __restrict__ mu) {
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= natm) return;
  const double* a = P.pol + 9 * (size_t)i;
  mu[i] = P.ipolar[i] ? make_double4(((a[0] * E[i].x) + a[1] * E[i].y) + a[2] * E[i].z,
                                     ((a[3] * E[i].x) + a[4] * E[i].y) + a[5] * E[i].z,
                                     ((a[6] * E[i].x) + a[7] * E[i].y) + a[8] * E[i].z, 0.0)
                      : make_double4(0, 0, 0, 0);
}

// ASPC predictor: mu = sum_k B_k hist[k]; hist[k] = hist[k-1] for k = ord..1
__global__ void k_aspc_predict(double4* __restrict__ hist, int natm, int ord, double b0, double b1,
                               double b2, double b3, double b4, double4* __restrict__ mu) {
  pdl_wait();
  pdl_trigger();
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= natm) return;
  double B[5] = {b0, b1, b2, b3, b4};
  double4 s = make_double4(0, 0, 0, 0);
  for (int k = 0; k <= ord; ++k) {
    double4 h = hist[(size_t)k * natm + i];
    s.x = s.x + B[k] * h.x;
    s.y = s.y + B[k] * h.y;
    s.z = s.z + B[k] * h.z;
  }
  mu[i] = s;
  for (int k = ord; k >= 1; --k) hist[(size_t)k * natm + i] = hist[(size_t)(k - 1) * natm + i];
}

// ASPC corrector: mu = w alpha E + (1 - w) mu
__global__ void k_aspc_correct(const double4* __restrict__ E, PolDev P, int natm, double wgt,
                               double4* __restrict__ mu) {
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= natm) return;
  double4 m = make_double4(0, 0, 0, 0);
  if (P.ipolar[i]) m = matvec3(P.pol + 9 * (size_t)i, E[i]);
  double4 o = mu[i];
  mu[i] = make_double4(wgt * m.x + (1.0 - wgt) * o.x, wgt * m.y + (1.0 - wgt) * o.y,
                       wgt * m.z + (1.0 - wgt) * o.z, 0.0);
}

// partials of u_pol = 1/2 sum mu alpha^-1 mu  (slot 0)
__global__ void k_upol_part(const double4* __restrict__ mu, PolDev P, int natm,
                            double* __restrict__ part) {
  pdl_wait();
  pdl_trigger();
  __shared__ double red[32];
  double v[1] = {0.0};
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < natm && P.ipolar[i]) {
    const double* a = P.invpol + 9 * (size_t)i;
    double m[3] = {mu[i].x, mu[i].y, mu[i].z};
    for (int x = 0; x < 3; ++x)
      for (int y = 0; y < 3; ++y) v[0] += m[x] * a[3 * x + y] * m[y];
  }
  block_sum<1>(v, red);
  if (threadIdx.x == 0) part[blockIdx.x] = v[0];
}

// partials of get_rmsd_mu: sum over polarisable ions, components with
// alpha_aa /= 0, of (mu_a/alpha_aa - E_a)^2.  Slot 0 of each block.
__global__ void k_rmsd_part(const double4* __restrict__ mu, const double4* __restrict__ E, PolDev P,
                            int natm, double* __restrict__ part) {
  __shared__ double red[32];
  double v[1] = {0.0};
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < natm && P.ipolar[i]) {
    const double* a = P.pol + 9 * (size_t)i;
    double m[3] = {mu[i].x, mu[i].y, mu[i].z}, e[3] = {E[i].x, E[i].y, E[i].z};
    for (int x = 0; x < 3; ++x) {
      double al = a[4 * x];
      if (al == 0.0) continue;
      double d = m[x] / al - e[x];
      v[0] += d * d;
    }
  }
  block_sum<1>(v, red);
  if (threadIdx.x == 0) part[blockIdx.x] = v[0];
}

// out = a + b
__global__ void k_add4(const double4* __restrict__ a, const double4* __restrict__ b, int n,
                       double4* __restrict__ out) {
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  out[i] = make_double4(a[i].x + b[i].x, a[i].y + b[i].y, a[i].z + b[i].z, 0.0);
}

// moments for self / surface terms: partial sums of
// [qtot(3) = sum q r, mutot(3), qsq, musq]
__global__ void k_moments_part(const double* __restrict__ pos, const double* __restrict__ q,
                               const double4* __restrict__ mu, int natm, int has_q,
                               double* __restrict__ part) {
  pdl_wait();
  pdl_trigger();
  __shared__ double red[8 * 32];
  double v[8] = {0, 0, 0, 0, 0, 0, 0, 0};
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < natm) {
    double qi = has_q ? q[i] : 0.0;
    double4 m = mu ? mu[i] : make_double4(0, 0, 0, 0);
    v[0] = qi * pos[i];
    v[1] = qi * pos[natm + i];
    v[2] = qi * pos[2 * natm + i];
    v[3] = m.x;
    v[4] = m.y;
    v[5] = m.z;
    v[6] = qi * qi;
    v[7] = m.x * m.x + m.y * m.y + m.z * m.z;
  }
  block_sum<8>(v, red);
  if (threadIdx.x == 0)
    for (int k = 0; k < 8; ++k) part[(size_t)blockIdx.x * 8 + k] = v[k];
}

// E += 2 selfa2 mu  (+ surface  -fpi_3V (qtot + mutot)  when lsurf);
// mom = reduced [qtot(3), mutot(3), qsq, musq]
__global__ void k_self_surf_field(const double4* __restrict__ mu, int natm, double selfa2,
                                  int lsurf, double fpi_3V, const double* __restrict__ mom,
                                  double4* __restrict__ E) {
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= natm) return;
  double4 m = mu ? mu[i] : make_double4(0, 0, 0, 0);
  double4 o = E[i];
  double s0 = 0.0, s1 = 0.0, s2 = 0.0;
  if (lsurf) {
    s0 = -(mom[0] + mom[3]) * fpi_3V;
    s1 = -(mom[1] + mom[4]) * fpi_3V;
    s2 = -(mom[2] + mom[5]) * fpi_3V;
  }
  E[i] = make_double4(o.x + s0 + 2.0 * selfa2 * m.x, o.y + s1 + 2.0 * selfa2 * m.y,
                      o.z + s2 + 2.0 * selfa2 * m.z, 0.0);
}

// ---- SCF iterations on the device -------------------------------------------
// From the second on, an SCF iteration (moment_from_pola.f90:340-460) is the dipole
// field of the iterate mun (cached real-space part on the side stream, rho, field
// sums) and
//   k_scf_tail: mu = mun, E_ind = real + reciprocal + self, the residual and u_pol;
//   the next iterate mun = alpha (E_stat + E_ind) and its reciprocal weights; the last
//   block to finish adds the partials in fixed order and sets rmsd, count, u_pol and
//   the WHILE condition of the graph that runs the iterations,
// so that a solve needs no host round trip per iteration.  An iterate formed after
// the last iteration is not used.  At 216 ions an iteration is a chain of launch
// latencies: with step, field sum and check as three kernels 24 us, as one 20.5, with
// four iterations per pass of the loop (a pass has about 5 us of its own) 18.

// mun = alpha (E_stat + E_ind) and its weights, for the first iteration of the loop
__device__ __forceinline__ void scf_iterate(const double* al, const double (&E)[3], const CellC* __restrict__ cell,
                                            int i, double4* __restrict__ mun, double4* __restrict__ w) {
  double m[3];
#pragma unroll
  for (int x = 0; x < 3; ++x) m[x] = ((al[3 * x] * E[0]) + al[3 * x + 1] * E[1]) + al[3 * x + 2] * E[2];
  mun[i] = make_double4(m[0], m[1], m[2], 0.0);
  const double* B = cell->B;
  w[i] = make_double4(0.0, kTwoPi * (B[0] * m[0] + B[3] * m[1] + B[6] * m[2]),
                      kTwoPi * (B[1] * m[0] + B[4] * m[1] + B[7] * m[2]),
                      kTwoPi * (B[2] * m[0] + B[5] * m[1] + B[8] * m[2]));
}
__global__ void k_scf_step(const double4* __restrict__ Estat, const double4* __restrict__ Eind, PolDev P,
                           int natm, const CellC* __restrict__ cell, double4* __restrict__ mun,
                           double4* __restrict__ w) {
  pdl_wait();
  pdl_trigger();
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= natm || !P.ipolar[i]) return;
  const double4 a = Estat[i], b = Eind[i];
  const double E[3] = {a.x + b.x, a.y + b.y, a.z + b.z};
  scf_iterate(P.pol + 9 * (size_t)i, E, cell, i, mun, w);
}

// four threads per polarisable ion split the field partials, as k_rec_field_sum
__global__ void __launch_bounds__(256) k_scf_tail(const double4* __restrict__ Gpart, int nchunk, int natm,
                                                  const int* __restrict__ polidx, int npol,
                                                  const CellC* __restrict__ cell, double scale, double selfa2,
                                                  const double4* __restrict__ Estat, PolDev P,
                                                  double4* __restrict__ mun, double4* __restrict__ mu,
                                                  double4* __restrict__ Eind, double4* __restrict__ w,
                                                  double* __restrict__ part, int* __restrict__ ticket, int npol_r, double tol,
                                                  int miniter, int maxiter, double* __restrict__ sc,
                                                  double* __restrict__ upol, int* __restrict__ stop,
                                                  cudaGraphConditionalHandle hc) {
  if (loop_stopped(stop)) return;
  __shared__ double red[2 * 32];
  __shared__ int last;
  double v[2] = {0.0, 0.0};
  const int t = blockIdx.x * blockDim.x + threadIdx.x, sl = t >> 2, sub = t & 3;
  double g[3] = {0.0, 0.0, 0.0};
  int i = 0;
  double4 m, o, st;
  double al[9], iv[9];
  if (sl < npol) {
    i = polidx[sl];
    m = mun[i];
    o = Eind[i];
    st = Estat[i];
#pragma unroll
    for (int a = 0; a < 9; ++a) {
      al[a] = P.pol[9 * (size_t)i + a];
      iv[a] = P.invpol[9 * (size_t)i + a];
    }
    chunk_sum4(Gpart, nchunk, natm, i, sub, g);
  }
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    g[a] += __shfl_xor_sync(FULL_MASK, g[a], 1);
    g[a] += __shfl_xor_sync(FULL_MASK, g[a], 2);
  }
  if (sl < npol && sub == 0) {
    const double* B = cell->B;
    const double mm[3] = {m.x, m.y, m.z}, oo[3] = {o.x, o.y, o.z}, ss[3] = {st.x, st.y, st.z};
    double e[3], E[3];
#pragma unroll
    for (int a = 0; a < 3; ++a) {
      const double er = -kTwoPi * (B[3 * a] * g[0] + B[3 * a + 1] * g[1] + B[3 * a + 2] * g[2]) * scale;
      e[a] = oo[a] + er + 2.0 * selfa2 * mm[a];
      E[a] = ss[a] + e[a];
      if (al[4 * a] != 0.0) {  // get_rmsd_mu (:998-1027)
        const double d = mm[a] / al[4 * a] - E[a];
        v[0] += d * d;
      }
#pragma unroll
      for (int b = 0; b < 3; ++b) v[1] += mm[a] * iv[3 * a + b] * mm[b];
    }
    mu[i] = m;
    Eind[i] = make_double4(e[0], e[1], e[2], 0.0);
    scf_iterate(al, E, cell, i, mun, w);
  }
  block_sum<2>(v, red);
  if (threadIdx.x == 0) {
    part[(size_t)blockIdx.x * 2] = v[0];
    part[(size_t)blockIdx.x * 2 + 1] = v[1];
    __threadfence();
    last = atomicAdd(ticket, 1) == (int)gridDim.x - 1;
  }
  __syncthreads();
  if (!last) return;
  __threadfence();
  v[0] = v[1] = 0.0;
  for (int b = threadIdx.x; b < (int)gridDim.x; b += blockDim.x) {
    v[0] += __ldcg(part + (size_t)b * 2);
    v[1] += __ldcg(part + (size_t)b * 2 + 1);
  }
  block_sum<2>(v, red);
  if (threadIdx.x != 0) return;
  *ticket = 0;
  const double rmsd = sqrt(v[0] / (double)npol_r);
  const int it = (int)sc[0] + 1;
  sc[0] = (double)it;
  sc[1] = rmsd;
  *upol = v[1];
  const bool more = (it < maxiter && rmsd > tol) || it < miniter;
  if (!more) *stop = 1;
  cudaGraphSetConditional(hc, more ? 1u : 0u);
}

// head of the loop: sc[0] = iterations, sc[1] = rmsd from the residual sum r2 of
// the first iteration.  The condition is the host loop's.
__global__ void k_scf_check(const double* __restrict__ r2, int npol, double tol, int miniter, int maxiter,
                            double* __restrict__ sc, int* __restrict__ stop, cudaGraphConditionalHandle hc) {
  if (threadIdx.x != 0) return;
  *stop = 0;
  const double rmsd = sqrt(*r2 / (double)npol);
  sc[0] = 1.0;
  sc[1] = rmsd;
  cudaGraphSetConditional(hc, ((1 < maxiter && rmsd > tol) || 1 < miniter) ? 1u : 0u);
}

// ---- conjugate gradients ----------------------------------------------------
// A x = alpha^-1 x - T x on polarisable ions (T x = field of x).  The step
// scalars (r.z, p.q) stay on the device; only the rmsd goes to the host.

// r = b + Tx - alpha^-1 x ; z = alpha r ; p = z ; partial r.z and rmsd
// FP32 operands of the next operator application of the direction p (when w32
// is given): w32 = (0, m), m = 2 pi B^T p, mu32 = p, as k_rec_weights writes them
// (and w32 again at the ion's slot in w32s, when the ion has one)
__device__ __forceinline__ void cg_dir_weights(const CellC* __restrict__ cell, double4 u, int i,
                                               float4* __restrict__ w32, float4* __restrict__ mu32,
                                               const SlotW& sw) {
  const double* B = cell->B;
  double m1 = kTwoPi * (B[0] * u.x + B[3] * u.y + B[6] * u.z);
  double m2 = kTwoPi * (B[1] * u.x + B[4] * u.y + B[7] * u.z);
  double m3 = kTwoPi * (B[2] * u.x + B[5] * u.y + B[8] * u.z);
  const float4 wv = make_float4(0.f, (float)m1, (float)m2, (float)m3);
  w32[i] = wv;
  mu32[i] = make_float4((float)u.x, (float)u.y, (float)u.z, 0.f);
  sw.put(i, wv);
}

// FP64 operator: w = (0, m)
__device__ __forceinline__ void cg_dir_weights64(const CellC* __restrict__ cell, double4 u, int i,
                                                 double4* __restrict__ w) {
  const double* B = cell->B;
  w[i] = make_double4(0.0, kTwoPi * (B[0] * u.x + B[3] * u.y + B[6] * u.z),
                      kTwoPi * (B[1] * u.x + B[4] * u.y + B[7] * u.z),
                      kTwoPi * (B[2] * u.x + B[5] * u.y + B[8] * u.z));
}

__global__ void k_cg_init(const double4* __restrict__ b, const double4* __restrict__ Tx,
                          const double4* __restrict__ x, PolDev P, int natm, double4* __restrict__ r,
                          double4* __restrict__ z, double4* __restrict__ p, double* __restrict__ part,
                          const CellC* __restrict__ cell, float4* __restrict__ w32,
                          float4* __restrict__ mu32, SlotW sw, double4* __restrict__ w64) {
  pdl_wait();
  pdl_trigger();
  __shared__ double red[2 * 32];
  double v[2] = {0.0, 0.0};
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < natm) {
    double4 ri = make_double4(0, 0, 0, 0), zi = make_double4(0, 0, 0, 0);
    if (P.ipolar[i]) {
      double4 ax = matvec3(P.invpol + 9 * (size_t)i, x[i]);
      // b = nullptr: Tx already holds b + T x (the merged static pass)
      const double4 bi = b ? b[i] : make_double4(0.0, 0.0, 0.0, 0.0);
      ri = make_double4(bi.x + Tx[i].x - ax.x, bi.y + Tx[i].y - ax.y, bi.z + Tx[i].z - ax.z, 0);
      zi = matvec3(P.pol + 9 * (size_t)i, ri);
      const double* a = P.pol + 9 * (size_t)i;
      double rr[3] = {ri.x, ri.y, ri.z};
      for (int c = 0; c < 3; ++c)
        if (a[4 * c] != 0.0) v[1] += rr[c] * rr[c];
    }
    r[i] = ri;
    z[i] = zi;
    p[i] = zi;
    if (w32) cg_dir_weights(cell, zi, i, w32, mu32, sw);
    if (w64) cg_dir_weights64(cell, zi, i, w64);
    v[0] = ri.x * zi.x + ri.y * zi.y + ri.z * zi.z;
  }
  block_sum<2>(v, red);
  if (threadIdx.x == 0) {
    part[(size_t)blockIdx.x * 2] = v[0];
    part[(size_t)blockIdx.x * 2 + 1] = v[1];
  }
}

// q = alpha^-1 p - Tp (polarisable ions); partial p.q
__global__ void k_cg_Ap(const double4* __restrict__ p, const double4* __restrict__ Tp, PolDev P,
                        int natm, double4* __restrict__ qv, double* __restrict__ part) {
  pdl_wait();
  pdl_trigger();
  __shared__ double red[32];
  double v[1] = {0.0};
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < natm) {
    double4 qi = make_double4(0, 0, 0, 0);
    if (P.ipolar[i]) {
      double4 ap = matvec3(P.invpol + 9 * (size_t)i, p[i]);
      qi = make_double4(ap.x - Tp[i].x, ap.y - Tp[i].y, ap.z - Tp[i].z, 0);
    }
    qv[i] = qi;
    v[0] = p[i].x * qi.x + p[i].y * qi.y + p[i].z * qi.z;
  }
  block_sum<1>(v, red);
  if (threadIdx.x == 0) part[blockIdx.x] = v[0];
}

// al = rz / pq ; x += al p ; r -= al q ; z = alpha_pol r ;
// partial r.z (new) and rmsd^2
// (acc: the structure factor is linear in the dipoles, so acc += al rho'(p)
// with rho'(p) = rhoA of this step's operator keeps acc = rho' of the charges
// and the current x; nk k vectors, grid-stride)
__global__ void k_cg_update(const double* __restrict__ rz_p, const double* __restrict__ pq_p,
                            PolDev P, int natm, const double4* __restrict__ p,
                            const double4* __restrict__ qv, double4* __restrict__ x,
                            double4* __restrict__ r, double4* __restrict__ z,
                            double* __restrict__ part, double2* __restrict__ acc = nullptr,
                            const double2* __restrict__ rhoA = nullptr, int nk = 0) {
  pdl_wait();
  pdl_trigger();
  __shared__ double red[2 * 32];
  double v[2] = {0.0, 0.0};
  double rz = *rz_p, pq = *pq_p;
  double al = (pq != 0.0) ? rz / pq : 0.0;
  if (acc)
    for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < nk; k += gridDim.x * blockDim.x) {
      const double2 a = acc[k], d = rhoA[k];
      acc[k] = make_double2(a.x + al * d.x, a.y + al * d.y);
    }
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < natm && P.ipolar[i]) {
    double4 xi = x[i], ri = r[i], pi = p[i], qi = qv[i];
    xi.x += al * pi.x;
    xi.y += al * pi.y;
    xi.z += al * pi.z;
    ri.x -= al * qi.x;
    ri.y -= al * qi.y;
    ri.z -= al * qi.z;
    double4 zi = matvec3(P.pol + 9 * (size_t)i, ri);
    x[i] = xi;
    r[i] = ri;
    z[i] = zi;
    v[0] = ri.x * zi.x + ri.y * zi.y + ri.z * zi.z;
    const double* a = P.pol + 9 * (size_t)i;
    double rr[3] = {ri.x, ri.y, ri.z};
    for (int c = 0; c < 3; ++c)
      if (a[4 * c] != 0.0) v[1] += rr[c] * rr[c];
  }
  block_sum<2>(v, red);
  if (threadIdx.x == 0) {
    part[(size_t)blockIdx.x * 2] = v[0];
    part[(size_t)blockIdx.x * 2 + 1] = v[1];
  }
}

// p = z + beta p with beta = rz_new / rz
__global__ void k_cg_dir(const double* __restrict__ rz_p, const double* __restrict__ rzn_p,
                         int natm, const double4* __restrict__ z, double4* __restrict__ p,
                         const CellC* __restrict__ cell, float4* __restrict__ w32,
                         float4* __restrict__ mu32, SlotW sw) {
  pdl_wait();
  pdl_trigger();
  double rz = *rz_p, rzn = *rzn_p;
  double be = (rz != 0.0) ? rzn / rz : 0.0;
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < natm) {
    double4 pi = p[i], zi = z[i];
    double4 pn = make_double4(zi.x + be * pi.x, zi.y + be * pi.y, zi.z + be * pi.z, 0.0);
    p[i] = pn;
    if (w32) cg_dir_weights(cell, pn, i, w32, mu32, sw);
  }
}

// ---------------------------------------------------------------------------
// The three vector kernels of a CG iteration whose operator's parts are deferred
// to it (field partials per row group, real-space field in Edd), over the
// polarisable ions (polidx):
//   k_cg_q     T p = real + reciprocal + self (+ surface), q = alpha^-1 p - T p, p.q
//   k_cg_step  al; x, r, z updated (and the accumulated rho'); r.z, |r|^2
//   k_cg_next  beta; p <- z + beta p with the next operator's weights; the step
//              scalars and the loop's condition
// Each kernel sums its predecessor's block partials itself (every block the same
// order): a sum of a few hundred numbers costs a block about 1 us, a launch of its
// own 4 us.  Scalars are read and written by different kernels: sc[3] is r.z for
// k_cg_step (whose block 0 moves it to sc[0]), sc[0] is r.z for k_cg_next (whose block
// 0 leaves the new one in sc[3]).  So is the stop flag: k_cg_next sets it and cannot leave
// by it (a block that starts late would see this launch's own), it leaves by
// the copy that this iteration's k_cg_step took.  An iteration of 8000 MgO ions had ten kernels, 66 us,
// of which 23 us were these and their reductions; now six.
template <int NV>
__device__ __forceinline__ void block_partials(const double* __restrict__ part, int nblk, double (&v)[NV],
                                               double* red, double* out) {
#pragma unroll
  for (int k = 0; k < NV; ++k) v[k] = 0.0;
  for (int b = threadIdx.x; b < nblk; b += blockDim.x)
#pragma unroll
    for (int k = 0; k < NV; ++k) v[k] += part[(size_t)b * NV + k];
  block_sum<NV>(v, red);
  if (threadIdx.x == 0)
#pragma unroll
    for (int k = 0; k < NV; ++k) out[k] = v[k];
  __syncthreads();
#pragma unroll
  for (int k = 0; k < NV; ++k) v[k] = out[k];
}

// four threads per ion split the field partials, as k_rec_field_sum
__global__ void __launch_bounds__(256) k_cg_q(const double4* __restrict__ Gpart, int nchunk, int natm,
                                              const int* __restrict__ polidx, int npol,
                                              const CellC* __restrict__ cell, double scale, SelfField sf,
                                              const double4* __restrict__ Edd, const double4* __restrict__ p, PolDev P,
                                              double4* __restrict__ qv, double* __restrict__ part) {
  pdl_trigger();  // (a plain launch: everything before it is complete)
  __shared__ double red[32];
  double v[1] = {0.0};
  const int sub = threadIdx.x & 3;
  for (int s0 = blockIdx.x * (blockDim.x / 4); s0 < npol; s0 += gridDim.x * (blockDim.x / 4)) {
    const int sl = s0 + (threadIdx.x >> 2);
    const bool ok = sl < npol;
    const int i = polidx[ok ? sl : npol - 1];
    double g[3] = {0.0, 0.0, 0.0};
    const double4 pi = p[i], o = Edd[i];
    chunk_sum4(Gpart, nchunk, natm, i, sub, g);
#pragma unroll
    for (int a = 0; a < 3; ++a) {
      g[a] += __shfl_xor_sync(FULL_MASK, g[a], 1);
      g[a] += __shfl_xor_sync(FULL_MASK, g[a], 2);
    }
    if (!ok || sub != 0) continue;
    const double* B = cell->B;
    const double4 ap = matvec3(P.invpol + 9 * (size_t)i, pi);
    const double pp[3] = {pi.x, pi.y, pi.z}, oo[3] = {o.x, o.y, o.z}, aa[3] = {ap.x, ap.y, ap.z};
    double q[3];
#pragma unroll
    for (int a = 0; a < 3; ++a) {
      const double er = -kTwoPi * (B[3 * a] * g[0] + B[3 * a + 1] * g[1] + B[3 * a + 2] * g[2]) * scale;
      double self = 2.0 * sf.selfa2 * pp[a];
      if (sf.lsurf) self -= (sf.mom[a] + sf.mom[3 + a]) * sf.fpi_3V;
      q[a] = aa[a] - (oo[a] + er + self);
      v[0] += pp[a] * q[a];
    }
    qv[i] = make_double4(q[0], q[1], q[2], 0.0);
  }
  block_sum<1>(v, red);
  if (threadIdx.x == 0) part[blockIdx.x] = v[0];
}

__global__ void __launch_bounds__(256) k_cg_step(double* __restrict__ sc, const double* __restrict__ pq_part, int npq,
                                                 PolDev P, const int* __restrict__ polidx, int npol,
                                                 const double4* __restrict__ p, const double4* __restrict__ qv,
                                                 double4* __restrict__ x, double4* __restrict__ r,
                                                 double4* __restrict__ z, double* __restrict__ part,
                                                 double2* __restrict__ acc, const double2* __restrict__ rhoA, int nk,
                                                 const int* __restrict__ stop, int* __restrict__ stop_copy) {
  const bool stopped = loop_stopped(stop);
  __shared__ double red[2 * 32], bc[2];
  const int t0 = blockIdx.x * blockDim.x + threadIdx.x, nt = gridDim.x * blockDim.x;
  // what k_cg_q does not write is read before the wait for it
  const int i0 = polidx[t0 < npol ? t0 : npol - 1];
  const double4 x0 = x[i0], r0 = r[i0], p0 = p[i0];
  double a0[9];
#pragma unroll
  for (int c = 0; c < 9; ++c) a0[c] = P.pol[9 * (size_t)i0 + c];
  const double rz = sc[3];
  pdl_wait();
  pdl_trigger();
  if (blockIdx.x == 0 && threadIdx.x == 0) *stop_copy = stopped ? 1 : 0;
  if (stopped) return;
  const double4 q0 = qv[i0];
  double pq[1], v[2] = {0.0, 0.0};
  block_partials<1>(pq_part, npq, pq, red, bc);
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    sc[0] = rz;
    sc[2] = pq[0];
  }
  const double al = (pq[0] != 0.0) ? rz / pq[0] : 0.0;
  auto step = [&](int i, double4 xi, double4 ri, const double4& pi, const double4& qi, const double* a) {
    xi.x += al * pi.x;
    xi.y += al * pi.y;
    xi.z += al * pi.z;
    ri.x -= al * qi.x;
    ri.y -= al * qi.y;
    ri.z -= al * qi.z;
    const double4 zi = matvec3(a, ri);
    x[i] = xi;
    r[i] = ri;
    z[i] = zi;
    v[0] += ri.x * zi.x + ri.y * zi.y + ri.z * zi.z;
    const double rr[3] = {ri.x, ri.y, ri.z};
#pragma unroll
    for (int c = 0; c < 3; ++c)
      if (a[4 * c] != 0.0) v[1] += rr[c] * rr[c];
  };
  if (t0 < npol) step(i0, x0, r0, p0, q0, a0);
  for (int sl = t0 + nt; sl < npol; sl += nt) {
    const int i = polidx[sl];
    step(i, x[i], r[i], p[i], qv[i], P.pol + 9 * (size_t)i);
  }
  if (acc)  // (k_cg_update)
    for (int k = t0; k < nk; k += nt) {
      const double2 a = acc[k], d = rhoA[k];
      acc[k] = make_double2(a.x + al * d.x, a.y + al * d.y);
    }
  block_sum<2>(v, red);
  if (threadIdx.x == 0) {
    part[(size_t)blockIdx.x * 2] = v[0];
    part[(size_t)blockIdx.x * 2 + 1] = v[1];
  }
}

__global__ void __launch_bounds__(256) k_cg_next(double* __restrict__ sc, const double* __restrict__ rz_part, int nrz,
                                                 int npol_r, const int* __restrict__ polidx, int npol,
                                                 const double4* __restrict__ z, double4* __restrict__ p,
                                                 const CellC* __restrict__ cell, float4* __restrict__ w32,
                                                 float4* __restrict__ mu32, SlotW sw, double4* __restrict__ w64,
                                                 const int* __restrict__ stop_copy, int* __restrict__ stop,
                                                 cudaGraphConditionalHandle hc) {
  __shared__ double red[2 * 32], bc[2];
  const int t0 = blockIdx.x * blockDim.x + threadIdx.x, nt = gridDim.x * blockDim.x;
  // (as k_cg_step: only z, the partials and the flag's copy are its)
  const int i0 = polidx[t0 < npol ? t0 : npol - 1];
  const double4 p0 = p[i0];
  pdl_wait();
  pdl_trigger();
  if (loop_stopped(stop_copy)) return;
  const double4 z0 = z[i0];
  double v[2];
  block_partials<2>(rz_part, nrz, v, red, bc);
  const double rz = sc[0];
  const double be = (rz != 0.0) ? v[0] / rz : 0.0;
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    sc[3] = v[0];
    sc[4] = v[1];
    const double it = sc[6] + 1.0, rm = sqrt(v[1] / (double)npol_r);
    sc[6] = it;
    sc[8] = rm;
    const bool more = rm > sc[5] && it < sc[7];
    if (!more) *stop = 1;
    cudaGraphSetConditional(hc, more ? 1u : 0u);
  }
  auto next = [&](int i, const double4& pi, const double4& zi) {
    const double4 pn = make_double4(zi.x + be * pi.x, zi.y + be * pi.y, zi.z + be * pi.z, 0.0);
    p[i] = pn;
    if (w32) cg_dir_weights(cell, pn, i, w32, mu32, sw);
    if (w64) cg_dir_weights64(cell, pn, i, w64);
  };
  if (t0 < npol) next(i0, p0, z0);
  for (int sl = t0 + nt; sl < npol; sl += nt) next(polidx[sl], p[polidx[sl]], z[polidx[sl]]);
}

// moment_from_WFc (moment_from_pola.f90:632-807), warp per ion over its
// (full, ascending) neighbour row: every ion of a type with lwfc >= 0 sums
// r_j - r_i (minimum image, the reference's two-rounding arithmetic) over
// the Wannier centres j (lwfc < 0) with |r_ij|^2 < rcut_wfc, in ascending j as
// the reference does; mu_wfc = -2 sum.  An ion of a type with lwfc > 0 that
// finds a different number of centres sets *bad (the reference STOPs).
__global__ void k_wfc_dipoles(const double4* __restrict__ s, const int* __restrict__ itype,
                              const int* __restrict__ lwfc, const int* __restrict__ nbr,
                              const int* __restrict__ nnb, int cap, int natm,
                              const CellC* __restrict__ cell, double rcut_wfc,
                              double4* __restrict__ mu_wfc, int* __restrict__ bad) {
  int lane = threadIdx.x & 31;
  int i = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  if (i >= natm) return;
  const int lw = lwfc[itype[i]];
  if (lw < 0) {
    if (lane == 0) mu_wfc[i] = make_double4(0, 0, 0, 0);
    return;
  }
  const double4 si = s[i];
  const int n = nnb[i];
  double ax = 0.0, ay = 0.0, az = 0.0;
  int cnt = 0;
  for (int k0 = 0; k0 < n; k0 += 32) {
    int k = k0 + lane;
    bool hit = false;
    double rx = 0.0, ry = 0.0, rz = 0.0;
    if (k < n) {
      int j = nbr[(size_t)i * cap + k];
      if (lwfc[itype[j]] < 0) {
        double4 sj = s[j];
        double r2 = min_image_exact(cell->A, xsub(sj.x, si.x), xsub(sj.y, si.y), xsub(sj.z, si.z), rx, ry, rz);
        hit = r2 < rcut_wfc;
      }
    }
    unsigned m = __ballot_sync(FULL_MASK, hit);
    while (m) {  // in ascending neighbour order
      int l = __ffs(m) - 1;
      m &= m - 1;
      double x = __shfl_sync(FULL_MASK, rx, l), y = __shfl_sync(FULL_MASK, ry, l),
             z = __shfl_sync(FULL_MASK, rz, l);
      ax = ax + x;
      ay = ay + y;
      az = az + z;
      cnt++;
    }
  }
  if (lane == 0) {
    mu_wfc[i] = make_double4(-2.0 * ax, -2.0 * ay, -2.0 * az, 0.0);
    if (lw > 0 && cnt != lw) atomicExch(bad, 1);
  }
}

// mu_tot = (dipia + mu_ind) [+ mu_wfc] ; catastrophe flag if any component > 10
// (moment_from_pola.f90:136-147, 176-178: positive components only)
// qm32 (optional): (mu_x, mu_y, mu_z, q) in FP32 for the mixed final pass
__global__ void k_mu_total(const double4* __restrict__ dip, const double4* __restrict__ mu_ind,
                           const double4* __restrict__ mu_wfc, int natm, double4* __restrict__ mu_tot,
                           int* __restrict__ flag, const double* __restrict__ q = nullptr,
                           float4* __restrict__ qm32 = nullptr) {
  pdl_wait();
  pdl_trigger();
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= natm) return;
  double4 a = dip[i], b = mu_ind[i];
  double4 m = make_double4(a.x + b.x, a.y + b.y, a.z + b.z, 0.0);
  if (mu_wfc) {
    double4 w = mu_wfc[i];
    m = make_double4(m.x + w.x, m.y + w.y, m.z + w.z, 0.0);
  }
  mu_tot[i] = m;
  if (qm32) qm32[i] = make_float4((float)m.x, (float)m.y, (float)m.z, (float)q[i]);
  if (m.x > 10.0 || m.y > 10.0 || m.z > 10.0) atomicExch(flag, 1);
}

}  // namespace mdff
