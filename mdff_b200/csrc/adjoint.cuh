// adjoint.cuh -- gradients of a batched evaluation with respect to
// force-field parameters (the differentiable fitting path).  No counterpart
// in the reference, which has no derivatives with respect to its potential
// parameters.
//
// For one configuration let J = g_U U + u_F . F + u_mu . mu (the upstream
// gradients of the total energy, the forces and the induced dipoles).  The
// dipoles solve R(mu, theta) = alpha^-1 mu - E(mu, theta) = 0 with H = dR/dmu
// = alpha^-1 - T symmetric, so
//     dJ/dtheta = dJ/dtheta|_mu - lambda . dR/dtheta,   H lambda = dJ/dmu,
// one adjoint solve with the forward's own PCG operator.  Every term
// differentiates the expressions the forward evaluates (es_force_ipair, the
// short-range pair, the reciprocal sums), not an idealised energy, so the
// gradient is that of the computed forces to the solver tolerance.
//
//   dJ/dmu_j = g_U cu R_j + d(u_F . F)/dmu_j + u_mu_j, with
//     real space  -cu d(Du . f_ab)/dm   per pair (Du = u_a - u_b)
//     reciprocal  cu (8 pi/V) sum_k A_k k [ (k.u_j) Re(rho P_j*) - Re(sigma P_j*) ],
//                 sigma(k) = sum_i (k.u_i)(q_i + i k.mu_i) P_i, P_i = e^{i k.r_i}
//   parameters: Buckingham A, rho, C per type pair (short-range forces and
//   energy); isotropic polarisability per type (u_pol and alpha^-1 in R);
//   Tang-Toennies b, c of the charge field on a dipole type (damped qd
//   forces / energy and the damped static field); one charge scale s on all
//   charges (qq terms scale with s^2, qd terms and the charge field with s).
//
// Bound: the dipole solve (to 1e-12, twice the forward's iterations), FP64
// throughout.  The structure-factor channels are the forward's tensor-core
// products (brho_t; sigma's weight is a polynomial in nz), the right-hand side's k
// sums two passes of its field product; the pair loops walk the partner lists
// with partners fetched ahead, the right-hand side over the CTA's share of the
// polarisable ions, and form each pair's parameter derivatives once, selected
// into the gradient by per-type-pair masks.  Measured, 64 boxes of 216-512 ions, all ten
// parameters of the MgO model: 7.6 -> 3.1 ms (SM time at 2 CTAs: right-hand side's and
// charge-scale channels 99 -> 46 ms, pair loops 72 -> 47, solve 229 -> 196; the
// rest from the launch shape: clusters of 2 instead of 8).
#pragma once
#include "batch.cuh"

namespace mdff {

enum { FIT_A = 0, FIT_RHO = 1, FIT_C = 2, FIT_POL = 3, FIT_TTB = 4, FIT_TTC = 5, FIT_QSCALE = 6 };
constexpr int kFitMax = 16;

struct FitParam {
  int kind, t1, t2, pad;
};

struct AdjArgs {
  const double* gE;    // [nconf] dJ/dU (U = u_lj + u_bmhft + u_coul, eV)
  const double* gF;    // [3][ntot] dJ/dF
  const double* gmu;   // [ntot][3] dJ/dmu or null
  double4* w;          // [ntot] u_F as 4-vectors
  double4* rhs;        // [ntot]
  double4* lam;        // [ntot]
  double2 *rq, *rm, *sq, *sm, *rl;  // [sum nk] structure-factor channels
  double* grad;        // [nconf][kFitMax]
  double* info;        // [nconf][4]: adjoint iterations, rmsd, tolerance
  double qscale;       // current charge scale (s in the s-derivatives)
  double tol_rel;      // adjoint solve tolerance relative to rms(rhs)
  int nparam;
  FitParam prm[kFitMax];
};

// One Tang-Toennies role (b, c, order) at distance r: F1d = 1 - f and fd of
// tt_damp, from f1, fd1 of c = 1 (f = 1 - c (1 - f1), fd = c fd1).  c = 0 damps
// nothing; its derivatives are formed only where a parameter asks (need).
template <int K>
__device__ __forceinline__ void tt_role(double b, double c, double r, int order, bool need, double& F1d,
                                        double& fd, double& f1, double& fd1) {
  F1d = fd = fd1 = 0.0;
  f1 = 1.0;
  if (c != 0.0) tt_damp_k<double, K>(b, 1.0, r, order, f1, fd1);
  else if (need) tt_damp<double>(b, 1.0, r, order, f1, fd1);
  F1d = c * (1.0 - f1);
  fd = c * fd1;
}

// d f / d b and d f / d c of tt_damp (f = 1 - c e^{-x} sum_k x^k/k!, fd = c b
// e^{-x} x^n/n!, x = b r) from f1, fd1 of c = 1:
//   df/dc = (f - 1)/c ... evaluated without dividing by c:  -e^{-x} S(x)
//   dfd/dc = b e^{-x} x^n/n!
//   df/db = r c e^{-x} x^n/n! = (r/b) fd
//   dfd/db = c e^{-x} x^n/n! (1 + n - x)
__device__ __forceinline__ void tt_damp_grad(double b, double c, double r, int n, double f1, double fd1,
                                             double& dfdb, double& dfddb, double& dfdc, double& dfddc) {
  double x = b * r;
  double en = (b != 0.0) ? fd1 / b : 0.0;  // e^{-x} x^n / n!
  if (b == 0.0) {
    // x = 0: e^{-x} x^n/n! = 1 for n = 0, else 0
    en = (n == 0) ? 1.0 : 0.0;
  }
  dfdc = f1 - 1.0;
  dfddc = fd1;
  // order 0 keeps the reference's f = 1 - c (1 + x) e^{-x} (tt_damp.f90:85-93)
  dfdb = (n == 0) ? c * r * x * en : c * r * en;
  dfddb = c * en * (1.0 + (double)n - x);
}

struct PairAdj {
  double gU, cu, rs;  // rs = 1 / (charge scale)
  int qs;             // mask of the charge-scale parameters
  int nparam;
};

__device__ __forceinline__ double dot3(const double (&a)[3], const double4& b) {
  return a[0] * b.x + a[1] * b.y + a[2] * b.z;
}
__device__ __forceinline__ double dot3(const double4& a, const double4& b) {
  return a.x * b.x + a.y * b.y + a.z * b.z;
}

// One real-space pair from the visit of ion i (r = r_i - r_j; the expressions
// of es_force_ipair, in i's frame; roles by i_is_a).
//   GRAD = false: dm += d(u_F . F)/dm_i.
//   GRAD = true:  this visit's share of the parameter gradient (half of the
//   energy, the force on i, the charge field on i against lambda_i) into g;
//   hit_i / hit_j: masks of the damping parameters of the field on i / on j.
template <int K, bool GRAD>
__device__ __forceinline__ void es_pair_adjoint(const PairAdj& J, const AdjArgs& A, const ESPair& P, bool i_is_a,
                                                double d2, double alpha, const double (&r)[3], double qi, double qj,
                                                const double4& mi, const double4& mj, int task_qq, int task_qd,
                                                int task_dd, const double4& wi, const double4& wj,
                                                const double4& li, int hit_i, int hit_j, double (&dm)[3],
                                                double (&g)[kFitMax]) {
  Radial<double> rd;
  radial<double, !GRAD>(d2, alpha, rd);
  const bool dip_i = mi.x != 0.0 || mi.y != 0.0 || mi.z != 0.0;
  const bool dip_j = mj.x != 0.0 || mj.y != 0.0 || mj.z != 0.0;
  const double B0 = rd.dm1 * rd.F0, B1 = rd.F1 * rd.dm3, B2 = 3.0 * rd.F2 * rd.dm5;
  double C1i = B1, C2i = B2, C1j = B1, C2j = B2;  // B - B_damped for the field on i / on j
  double bi = 0, ci = 0, bj = 0, cj = 0, f1i = 1, fd1i = 0, f1j = 1, fd1j = 0;
  int ki = 0, kj = 0;
  if (P.ldamp) {
    double F1d, fd;
    bi = i_is_a ? P.ba : P.bb;
    ci = i_is_a ? P.ca : P.cb;
    ki = i_is_a ? P.ka : P.kb;
    tt_role<K>(bi, ci, rd.d, ki, GRAD && hit_i, F1d, fd, f1i, fd1i);
    C1i = B1 - F1d * rd.dm3;
    C2i = B2 - 3.0 * (F1d + (rd.d / 3.0) * fd) * rd.dm5;
    if (GRAD) {  // (the field on j does not enter dm_i)
      bj = i_is_a ? P.bb : P.ba;
      cj = i_is_a ? P.cb : P.ca;
      kj = i_is_a ? P.kb : P.ka;
      tt_role<K>(bj, cj, rd.d, kj, hit_j != 0, F1d, fd, f1j, fd1j);
      C1j = B1 - F1d * rd.dm3;
      C2j = B2 - 3.0 * (F1d + (rd.d / 3.0) * fd) * rd.dm5;
    }
  }
  const bool qd = task_qd && (dip_i || dip_j);
  const double rmj = dot3(r, mj);
  if (!GRAD) {
    const double4 D = make_double4(wi.x - wj.x, wi.y - wj.y, wi.z - wj.z, 0.0);
    const double Dr = dot3(r, D), Dmj = dot3(D, mj);
    double fr = 0.0, fD = 0.0, fm = 0.0;  // coefficients of r, D, m_j
    if (task_dd && dip_i && dip_j) {
      const double B3 = 15.0 * rd.F3 * rd.dm7;
      fr += B3 * rmj * Dr - B2 * Dmj;
      fm -= B2 * Dr;
      fD -= B2 * rmj;
    }
    if (qd) {
      fr += qj * C2i * Dr;
      fD -= qj * C1i;
    }
    // u_F . F = -cu D . f
    dm[0] -= J.cu * (fr * r[0] + fD * D.x + fm * mj.x);
    dm[1] -= J.cu * (fr * r[1] + fD * D.y + fm * mj.y);
    dm[2] -= J.cu * (fr * r[2] + fD * D.z + fm * mj.z);
    return;
  }
  const double rmi = dot3(r, mi), wr = dot3(r, wi), lr = dot3(r, li);
  const double wmi = dot3(wi, mi), wmj = dot3(wi, mj);
  double vq = 0.0, vb[2] = {0.0, 0.0}, vc[2] = {0.0, 0.0};
  if (J.qs) {
    if (task_qq)  // w.f_qq and u_qq scale with s^2; the charge field on i with s
      vq += 2.0 * J.cu * qi * qj * B1 * wr + J.gU * J.cu * qi * qj * B0 + qj * C1i * lr;
    if (qd)
      vq += J.cu * (qi * (C2j * wr * rmj - C1j * wmj) - qj * (C2i * wr * rmi - C1i * wmi)) +
            0.5 * J.gU * J.cu * (qi * C1j * rmj - qj * C1i * rmi);
    vq *= J.rs;
  }
  if (P.ldamp && hit_i) {
    double dfdb, dfddb, dfdc, dfddc;
    tt_damp_grad(bi, ci, rd.d, ki, f1i, fd1i, dfdb, dfddb, dfdc, dfddc);
    auto val = [&](double df, double dfd) {
      const double dB1 = -df * rd.dm3, dB2 = 3.0 * (-df + (rd.d / 3.0) * dfd) * rd.dm5;  // of the damped parts
      double v = 0.0;
      if (qd) v += J.cu * qj * (dB2 * wr * rmi - dB1 * wmi) + 0.5 * J.gU * J.cu * qj * dB1 * rmi;
      if (task_qq) v -= qj * dB1 * lr;
      return v;
    };
    vb[0] = val(dfdb, dfddb);
    vc[0] = val(dfdc, dfddc);
  }
  if (P.ldamp && hit_j && qd) {
    double dfdb, dfddb, dfdc, dfddc;
    tt_damp_grad(bj, cj, rd.d, kj, f1j, fd1j, dfdb, dfddb, dfdc, dfddc);
    auto val = [&](double df, double dfd) {
      const double dB1 = -df * rd.dm3, dB2 = 3.0 * (-df + (rd.d / 3.0) * dfd) * rd.dm5;
      return -J.cu * qi * (dB2 * wr * rmj - dB1 * wmj) - 0.5 * J.gU * J.cu * qi * dB1 * rmj;
    };
    vb[1] = val(dfdb, dfddb);
    vc[1] = val(dfdc, dfddc);
  }
#pragma unroll
  for (int p = 0; p < kFitMax; ++p) {
    if (p >= J.nparam) break;
    const int kind = A.prm[p].kind;
    if (kind == FIT_QSCALE) {
      g[p] += vq;
    } else if (kind == FIT_TTB || kind == FIT_TTC) {
      if ((hit_i >> p) & 1) g[p] += kind == FIT_TTB ? vb[0] : vc[0];
      if ((hit_j >> p) & 1) g[p] += kind == FIT_TTB ? vb[1] : vc[1];
    }
  }
}

// Buckingham / BMH pair parameters from the visit of ion i (r = r_i - r_j):
// w_i . r dwij/dtheta + 1/2 g_U du/dtheta (hit: mask of the pair's parameters)
__device__ __forceinline__ void sr_pair_adjoint(const PairAdj& J, const AdjArgs& A, const NBPair& P, int lbmhftd,
                                                int hit, double rijsq, const double (&r)[3], const double4& wi,
                                                double (&g)[kFitMax]) {
  if (P.A == 0.0) return;  // the reference skips the pair (non_bonded.f90:1153)
  const double d = sqrt(rijsq), dinv = 1.0 / d;
  const double wr = dot3(r, wi);
  const double e = exp(-P.B * d);
  const double ir2 = dinv * dinv, ir6 = ir2 * ir2 * ir2;
  double f6 = 1.0, fd6 = 0.0;
  if (lbmhftd) tt_damp_k<double, 6>(P.BD, 1.0, d, 6, f6, fd6);
  const double hg = 0.5 * J.gU;
  const double vA = wr * (P.B * e * dinv) + hg * e;
  // B = 1/rho: d/drho = -B^2 d/dB
  const double vR = -P.B * P.B * (wr * (P.A * e * (1.0 - P.B * d) * dinv) - hg * P.A * d * e);
  const double vC = wr * ((-6.0 * f6 * ir6 * dinv + fd6 * ir6) * dinv) - hg * f6 * ir6;
#pragma unroll
  for (int p = 0; p < kFitMax; ++p) {
    if (p >= J.nparam) break;
    const int kind = A.prm[p].kind;
    if ((hit >> p) & 1) g[p] += kind == FIT_A ? vA : kind == FIT_RHO ? vR : vC;
  }
}

// ---------------------------------------------------------------------------
// Structure-factor partials of this CTA's ions over all rows (brho_t), visible
// to the cluster on return:
//   sum_i [ (has_q ? q_i : 0) + i (has_m ? k.v_i : 0) ] (has_w ? k.w_i : 1) P_i,
// v from S.v, w from Sw by ion; rot: times i (has_w only).  r: the pass, for the
// field (bfld) or badj_store of the same partials.
__device__ __noinline__ void badj_rho(cgx::cluster_group& cl, const BatchArgs& a, BCtx& X, const BShared& S,
                                      const double4* Sw, bool has_q, bool has_m, bool has_w, bool rot, BRecArgs& r) {
  const BConf& c = *X.c;
  r = brec_args(a, X, S, 0, false);
  r.rot = rot;
  double4* w = brec_weights(r, S, has_w ? 2 : 1);
  const BWeights ws{X.c, S.s, S.v, S.v32, r.src.n0, 0, has_q, has_m};
  __syncthreads();
  for (int k = threadIdx.x; k < r.src.cnt; k += blockDim.x) {
    double v[4];
    ws(k, v);
    w[k] = make_double4(v[0], v[1], v[2], v[3]);
    if (has_w) {
      const double4 u = Sw[r.src.n0 + k];
      const double3 m = bmvec(c, u.x, u.y, u.z);
      w[r.src.cnt + k] = make_double4(0.0, m.x, m.y, m.z);
    }
  }
  __syncthreads();
  if (has_w) brho<2>(r);
  else if (has_m) brho<1>(r);
  else brho<0>(r);
  cl.sync();
}
// the sums of this CTA's share of the rows, by k
__device__ __noinline__ void badj_store(const BatchArgs& a, const BCtx& X, const BRecArgs& r, double2* __restrict__ out) {
  const BConf& c = *X.c;
  const int nz = c.kz + 1;
  const int r0 = (int)((long long)c.nrows * X.rank / X.C), r1 = (int)((long long)c.nrows * (X.rank + 1) / X.C);
  for (int e = threadIdx.x; e < (r1 - r0) * nz; e += blockDim.x) {
    const int row = r0 + e / nz, n = e % nz;
    const int4 ri = r.rows[row];
    double2 rp, rm;
    brho_pm(r.part, r.pld, X.C, (size_t)row * nz + n, nullptr, rp, rm);
    double2* o = out + c.k_off + ri.w - ri.z;
    if (n >= ri.z) o[n] = rp;
    if (n > 0 && ri.z < 0) o[-n] = rm;
  }
}

// real-space right-hand side of this CTA's polarisable ions (warp per ion)
template <int K>
__device__ __noinline__ void badj_rhs(const BatchArgs& a, const AdjArgs& J, const PairAdj& PJ, const BCtx& X,
                                      const BShared& S, const double4* Sw) {
  const BConf& c = *X.c;
  const int task_qq = (c.flags & BF_QQ) ? 1 : 0, task_qd = (c.flags & BF_QD) ? 1 : 0;
  const int task_dd = (c.flags & BF_DD) ? 1 : 0;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarp = blockDim.x >> 5;
  for (int p = X.p0 + warp; p < X.p1; p += nwarp) {
    const int i = bpl(S.t[p]);
    const double4 si = S.s[i], mi = S.v[i], wi = Sw[i];
    const int ti = btyp(S.t[i]);
    double dm[3] = {0, 0, 0}, g[kFitMax];
    const unsigned short* row = bnbl(a, X, 0, i);
    const int nn = __ldcg(bnbn(a, X, 0) + i);
    int jn = lane < nn ? bnbr(row, lane) : 0;
    for (int k = lane; k < nn; k += 32) {
      const int j = jn;
      if (k + 32 < nn) jn = bnbr(row, k + 32);
      const double4 sj = S.s[j];
      double r[3];
      const double r2 = pair_vec<double>(c.A, si, sj, r[0], r[1], r[2]);
      if (r2 > c.rc2) continue;
      const int tj = btyp(S.t[j]);
      const bool ia = half_mask(i, j);
      es_pair_adjoint<K, false>(PJ, J, S.es[(ia ? ti : tj) * c.ntype + (ia ? tj : ti)], ia, r2, c.alpha, r, si.w, sj.w,
                                mi, S.v[j], task_qq, task_qd, task_dd, wi, Sw[j], wi, 0, 0, dm, g);
    }
#pragma unroll
    for (int d = 0; d < 3; ++d) dm[d] = warp_sum(dm[d]);
    if (lane == 0) J.rhs[X.off + i] = make_double4(dm[0], dm[1], dm[2], 0.0);
  }
}

// pair terms of the parameter gradient (warp per ion of this CTA), added to g.
// S.es[ti * ntype + tj].thole: bit p, damping parameter p is the field on type ti by
// charges of type tj; bit 16 + p, short-range parameter p is of the pair.
template <int K>
__device__ __noinline__ void badj_pairs(const BatchArgs& a, const AdjArgs& J, const PairAdj& PJ, const BCtx& X,
                                        const BShared& S, const double4* Sw, bool any_sr, bool any_es,
                                        double (&gout)[kFitMax]) {
  const BConf& c = *X.c;
  const int task_qq = (c.flags & BF_QQ) ? 1 : 0, task_qd = (c.flags & BF_QD) ? 1 : 0;
  const int task_dd = (c.flags & BF_DD) ? 1 : 0, lbmhftd = (c.flags & BF_BMHFTD) ? 1 : 0;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarp = blockDim.x >> 5;
  double g[kFitMax];
#pragma unroll
  for (int p = 0; p < kFitMax; ++p) g[p] = 0.0;
  for (int i = X.i0 + warp; i < X.i1; i += nwarp) {
    const double4 si = S.s[i], mi = S.v[i], wi = Sw[i];
    const int ti = btyp(S.t[i]);
    if (any_sr) {
      const unsigned short* row = bnbl(a, X, 1, i);
      const int nn = __ldcg(bnbn(a, X, 1) + i);
      int jn = lane < nn ? bnbr(row, lane) : 0;
      for (int k = lane; k < nn; k += 32) {
        const int j = jn;
        if (k + 32 < nn) jn = bnbr(row, k + 32);
        const int tp = ti * c.ntype + btyp(S.t[j]), h = (S.es[tp].thole >> 16) & 0xffff;
        if (!h) continue;
        double r[3];
        const double r2 = pair_vec<double>(c.A, si, S.s[j], r[0], r[1], r[2]);
        const NBPair& P = S.nb[tp];
        if (r2 < P.rcutsq) sr_pair_adjoint(PJ, J, P, lbmhftd, h, r2, r, wi, g);
      }
    }
    const double4 li = ldcg4(J.lam + X.off + i);
    const unsigned short* row = bnbl(a, X, 0, i);
    const int nn = any_es ? __ldcg(bnbn(a, X, 0) + i) : 0;
    int jn = lane < nn ? bnbr(row, lane) : 0;
    for (int k = lane; k < nn; k += 32) {
      const int j = jn;
      if (k + 32 < nn) jn = bnbr(row, k + 32);
      const int tj = btyp(S.t[j]);
      const int hi = S.es[ti * c.ntype + tj].thole & 0xffff, hj = S.es[tj * c.ntype + ti].thole & 0xffff;
      if (!PJ.qs && !hi && !hj) continue;
      const double4 sj = S.s[j];
      double r[3], dm[3];
      const double r2 = pair_vec<double>(c.A, si, sj, r[0], r[1], r[2]);
      if (r2 > c.rc2) continue;
      const bool ia = half_mask(i, j);
      es_pair_adjoint<K, true>(PJ, J, S.es[(ia ? ti : tj) * c.ntype + (ia ? tj : ti)], ia, r2, c.alpha, r, si.w, sj.w,
                               mi, S.v[j], task_qq, task_qd, task_dd, wi, wi, li, hi, hj, dm, g);
    }
  }
#pragma unroll
  for (int p = 0; p < kFitMax; ++p) gout[p] += g[p];
}

// ---------------------------------------------------------------------------
// adjoint of one configuration (the forward of the same positions has run:
// a.s, a.rec, a.x (induced dipoles), a.mu (total), a.E (field) are valid)
__device__ void bconfig_adjoint(cgx::cluster_group& cl, const BatchArgs& a, const AdjArgs& J, BCtx& X,
                                const BShared& S, double4* Sw) {
  const BConf& c = *X.c;
  const bool coul = (c.flags & BF_COUL) != 0, polar = (c.flags & BF_POLAR) != 0;
  const int task_qq = (c.flags & BF_QQ) ? 1 : 0;
  const bool tt4 = (c.flags & BF_TT4) != 0;
  const double cu = c.coul_unit;
  const double gU = J.gE[X.cfg];
  PairAdj PJ;
  PJ.nparam = J.nparam;
  PJ.gU = gU;
  PJ.cu = cu;
  PJ.rs = 1.0 / J.qscale;
  PJ.qs = 0;
  bool any_sr = false, any_es = false;
  for (int p = 0; p < J.nparam; ++p) {
    if (J.prm[p].kind <= FIT_C) any_sr = true;
    if (J.prm[p].kind >= FIT_TTB) any_es = true;
    if (J.prm[p].kind == FIT_QSCALE) PJ.qs |= 1 << p;
  }
  any_sr = any_sr && (c.flags & BF_SR) && (c.flags & BF_BMH);
  any_es = any_es && coul;
  // ---- load -------------------------------------------------------------
  for (int i = X.i0 + threadIdx.x; i < X.i1; i += blockDim.x) {
    int gi = X.off + i;
    J.w[gi] = make_double4(J.gF[gi], J.gF[a.ntot + gi], J.gF[2 * (size_t)a.ntot + gi], 0.0);
  }
  for (int k = threadIdx.x; k < c.ntype * c.ntype; k += blockDim.x) {
    S.nb[k] = a.nbtab[c.nb_off + k];
    S.es[k] = a.estab[c.es_off + k];
    const int ti = k / c.ntype, tj = k % c.ntype;
    int h = 0;
    for (int p = 0; p < J.nparam; ++p) {
      const FitParam& fp = J.prm[p];
      const bool ord = ti == fp.t1 && tj == fp.t2, rev = ti == fp.t2 && tj == fp.t1;
      if ((fp.kind == FIT_TTB || fp.kind == FIT_TTC) && ord) h |= 1 << p;
      if (fp.kind <= FIT_C && (ord || rev)) h |= 1 << (16 + p);
    }
    S.es[k].thole = h;  // (fits have no Thole functions)
  }
  cl.sync();
  for (int i = threadIdx.x; i < X.n; i += blockDim.x) {
    S.s[i] = ldcg4(a.s + X.off + i);
    S.t[i] = a.typ[X.off + i];
    S.v[i] = ldcg4(a.mu + X.off + i);
    Sw[i] = ldcg4(J.w + X.off + i);
  }
  __syncthreads();
  blists(a, X, S, coul, (c.flags & BF_SR) != 0);
  if (coul && polar) {
    cl.sync();  // every CTA's partner lists
    if (bcached(a, X)) bcache<false>(a, X, S);
  }
  double g[kFitMax];
  for (int p = 0; p < kFitMax; ++p) g[p] = 0.0;
  int iters = 0;
  double rmsd = 0.0, tol = 0.0;
  if (coul && polar) {
    // ---- right-hand side: g_U cu R + d(u_F.F)/dmu + u_mu ---------------------
    if (tt4) badj_rhs<4>(a, J, PJ, X, S, Sw);
    else badj_rhs<0>(a, J, PJ, X, S, Sw);
    // reciprocal: rho = sum (q + i k.mu) P and i sigma = i sum (k.u)(q + i k.mu) P;
    // sum_k A n [ (k.w) Re(rho P*) - Re(sigma P*) ] is the dipole force of rho on
    // the vectors w plus the field sum of i sigma (bfld_get's fm and e)
    for (int ch = 0; ch < 2 && c.nk > 0; ++ch) {
      BRecArgs r;
      badj_rho(cl, a, X, S, Sw, task_qq != 0, true, ch == 1, ch == 1, r);
      r.wd = BWeights{X.c, S.s, Sw, S.v32, X.i0, 0, false, true};
      const int RS = ch == 0 ? bfld<true>(r) : bfld<false>(r);
      for (int i = X.i0 + threadIdx.x; i < X.i1; i += blockDim.x) {
        double e[3], fm[3];
        bfld_get(a, c, RS, i - X.i0, ch == 0, e, fm);
        const double4 o = J.lam[X.off + i];  // lam as scratch
        J.lam[X.off + i] = ch == 0 ? make_double4(fm[0], fm[1], fm[2], 0.0)
                                   : make_double4(o.x + e[0], o.y + e[1], o.z + e[2], 0.0);
      }
      __syncthreads();
    }
    cl.sync();  // every CTA's rows of rhs
    double v1[1] = {0.0};
    for (int i = X.i0 + threadIdx.x; i < X.i1; i += blockDim.x) {
      int gi = X.off + i;
      double4 o = make_double4(0, 0, 0, 0);
      if (a.ipol[gi]) {
        double4 rr = ldcg4(J.rhs + gi), rc = c.nk > 0 ? J.lam[gi] : make_double4(0, 0, 0, 0);
        double4 ax = bmat3(a.inv + 9 * (size_t)gi, ldcg4(a.x + gi));
        double4 E = ldcg4(a.E + gi);
        double R[3] = {ax.x - E.x, ax.y - E.y, ax.z - E.z};
        double gm[3] = {0, 0, 0};
        if (J.gmu) {
          gm[0] = J.gmu[3 * (size_t)gi];
          gm[1] = J.gmu[3 * (size_t)gi + 1];
          gm[2] = J.gmu[3 * (size_t)gi + 2];
        }
        o.x = rr.x + cu * rc.x + gU * cu * R[0] + gm[0];
        o.y = rr.y + cu * rc.y + gU * cu * R[1] + gm[1];
        o.z = rr.z + cu * rc.z + gU * cu * R[2] + gm[2];
        v1[0] += o.x * o.x + o.y * o.y + o.z * o.z;
      }
      J.rhs[gi] = o;
    }
    cluster_sum<1>(cl, X, S, v1);
    double rms = sqrt(v1[0] / (3.0 * max(c.npol, 1)));
    tol = fmax(J.tol_rel * rms, 1e-300);
    // ---- adjoint solve H lambda = rhs, lambda0 = alpha rhs -------------------
    for (int i = X.i0 + threadIdx.x; i < X.i1; i += blockDim.x) {
      int gi = X.off + i;
      J.lam[gi] = a.ipol[gi] ? bmat3(a.pol + 9 * (size_t)gi, J.rhs[gi]) : make_double4(0, 0, 0, 0);
    }
    if (rms > 0.0) bsolve<false>(cl, a, X, S, J.rhs, J.lam, tol, 4 * c.maxit, iters, rmsd);
    cl.sync();
    for (int i = threadIdx.x; i < X.n; i += blockDim.x) S.v[i] = ldcg4(a.mu + X.off + i);
    __syncthreads();
  } else {
    for (int i = X.i0 + threadIdx.x; i < X.i1; i += blockDim.x) J.lam[X.off + i] = make_double4(0, 0, 0, 0);
  }
  // ---- parameter gradient ----------------------------------------------------
  if (tt4) badj_pairs<4>(a, J, PJ, X, S, Sw, any_sr, any_es, g);
  else badj_pairs<0>(a, J, PJ, X, S, Sw, any_sr, any_es, g);
  // per-ion terms: polarisability, self energy of the charges
  const double selfa = c.alpha / sqrt(kPi);
  for (int i = X.i0 + threadIdx.x; i < X.i1; i += blockDim.x) {
    int gi = X.off + i;
    int ti = btyp(S.t[i]);
    for (int p = 0; p < J.nparam; ++p) {
      const FitParam& fp = J.prm[p];
      if (fp.kind == FIT_POL && ti == fp.t1 && a.ipol[gi]) {
        double al = a.pol[9 * (size_t)gi];
        double4 m = ldcg4(a.x + gi), l = ldcg4(J.lam + gi);
        double mm = m.x * m.x + m.y * m.y + m.z * m.z, lm = l.x * m.x + l.y * m.y + l.z * m.z;
        g[p] += lm / (al * al) - 0.5 * gU * cu * mm / (al * al);
      }
      if (fp.kind == FIT_QSCALE && coul && task_qq) {
        double q = S.s[i].w;
        g[p] += gU * cu * (-2.0 * selfa * q * q) / J.qscale;
      }
    }
  }
  // reciprocal charge-scale terms: rho_lambda, then per k over this CTA's rows
  if (PJ.qs && coul && task_qq && c.nk > 0) {
    // channels: rq = rho_q, rm = rho_mu, sq = sigma_q, sm = sigma_mu, rl = rho_lambda
    for (int ch = 0; ch < 5; ++ch) {
      if (ch == 4) {  // (S.v = mu until here; every CTA's lambda is visible)
        __syncthreads();
        for (int i = threadIdx.x; i < X.n; i += blockDim.x) S.v[i] = ldcg4(J.lam + X.off + i);
        __syncthreads();
      }
      BRecArgs r;
      badj_rho(cl, a, X, S, Sw, ch == 0 || ch == 2, ch != 0 && ch != 2, ch == 2 || ch == 3, false, r);
      badj_store(a, X, r, ch == 0 ? J.rq : ch == 1 ? J.rm : ch == 2 ? J.sq : ch == 3 ? J.sm : J.rl);
    }
    __syncthreads();
    const double fpi_V = 2.0 * (kTwoPi / c.omega), epi_V = 2.0 * fpi_V;
    double acc = 0.0;
    int r0 = (int)((long long)c.nrows * X.rank / X.C), r1 = (int)((long long)c.nrows * (X.rank + 1) / X.C);
    int k0 = a.rows[c.row_off + r0].w;
    int k1 = (r1 < c.nrows) ? a.rows[c.row_off + r1].w : c.nk;
    if (r0 >= r1) k1 = k0;
    for (int k = k0 + threadIdx.x; k < k1; k += blockDim.x) {
      size_t gk = (size_t)c.k_off + k;
      double A = a.Ak[gk];
      double2 q = __ldcg(J.rq + gk), m = __ldcg(J.rm + gk), sq = __ldcg(J.sq + gk);
      double2 sm = __ldcg(J.sm + gk), l = __ldcg(J.rl + gk);
      double qq = q.x * q.x + q.y * q.y, qm = q.x * m.x + q.y * m.y;  // Re(conj(q) m)
      // Im(conj(x) y) = x.re y.im - x.im y.re
      double iqsq = q.x * sq.y - q.y * sq.x, iqsm = q.x * sm.y - q.y * sm.x;
      double imsq = m.x * sq.y - m.y * sq.x;
      double rql = q.x * l.x + q.y * l.y;
      acc += A * (gU * cu * fpi_V * (2.0 * qq + 2.0 * qm) +
                  cu * epi_V * (2.0 * iqsq + iqsm + imsq) - epi_V * rql);
    }
    for (int p = 0; p < J.nparam; ++p)
      if (J.prm[p].kind == FIT_QSCALE) g[p] += acc / J.qscale;
  }
  cluster_sum<kFitMax>(cl, X, S, g);
  if (X.rank == 0 && threadIdx.x == 0) {
    for (int p = 0; p < kFitMax; ++p) J.grad[(size_t)X.cfg * kFitMax + p] = g[p];
    J.info[4 * (size_t)X.cfg] = iters;
    J.info[4 * (size_t)X.cfg + 1] = rmsd;
    J.info[4 * (size_t)X.cfg + 2] = tol;
  }
}

__global__ void __launch_bounds__(512) k_batch_adjoint(const __grid_constant__ BatchArgs a,
                                                       const __grid_constant__ AdjArgs J, int nmax) {
  extern __shared__ __align__(16) unsigned char bsm[];
  BShared S = batch_smem(bsm, nmax);
  double4* Sw = reinterpret_cast<double4*>(bsm + batch_smem_extra_offset(nmax));
  if (a.stage_extra) {
    S.stage = reinterpret_cast<unsigned char*>(Sw + nmax);
    S.stage_bytes = a.stage_extra;
  }
  cgx::cluster_group cl = cgx::this_cluster();
  BCtx X;
  X.rank = (int)cl.block_rank();
  X.C = (int)cl.num_blocks();
  while (true) {
    if (X.rank == 0 && threadIdx.x == 0) *S.cfg = atomicAdd(a.queue, 1);
    cl.sync();
    int qpos = *cl.map_shared_rank(S.cfg, 0);
    cl.sync();
    if (qpos >= a.nconf) break;
    int cfg = a.order[qpos];
    bctx_set(a, X, cfg);
    bconfig_adjoint(cl, a, J, X, S, Sw);
    __syncthreads();
  }
}

}  // namespace mdff
