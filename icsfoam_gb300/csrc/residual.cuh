// Pieces of the residual pipeline shared by its kernels (k_residual.cu) and
// the reverse-mode derivative of the residual (k_adjoint.cu): scheme
// parameters, the reconstruction of a face value, and the host helpers that
// fill them from a handle.
#pragma once

#include <type_traits>

#include "flux.cuh"
#include "hb.cuh"
#include "ics_internal.cuh"

namespace ics {

template <typename Real>
constexpr bool is_fp64 = std::is_same<Real, double>::value;

struct ResParams {
  double R, Cv, gamma, cstarFac;
  int scheme, reconRho, reconU, reconT, lowMach;
  double entropyFix;
};

__device__ __forceinline__ int recon_of(const ResParams& P, int q) {
  if (q == Q_RHO || q == Q_P) return P.reconRho;
  if (q == Q_UX || q == Q_UY || q == Q_UZ) return P.reconU;
  return P.reconT;
}

// Sums of products with every rounding written out.  The residual, its forward
// product (Real = Dual, whose value takes the same roundings) and its reverse
// product decide their limiter branches on these values; left to the compiler's
// contraction the kernels could round them differently and, at a tie, take
// different branches.
__device__ __forceinline__ double madd(double a, double b, double c) { return ::fma(a, b, c); }
__device__ __forceinline__ Dual madd(double a, const Dual& b, const Dual& c) {
  return Dual(::fma(a, b.v, c.v), ::fma(a, b.d, c.d));
}
// d . g
template <typename Real>
__device__ __forceinline__ Real project(double d0, double d1, double d2, const Real& g0, const Real& g1,
                                        const Real& g2) {
  return madd(d2, g2, madd(d1, g1, madd(d0, g0, Real(0.0))));
}
// specific total energy Cv T + |U|^2 / 2
__device__ __forceinline__ double total_energy(double Cv, double T, double U0, double U1, double U2) {
  return ::fma(Cv, T, 0.5 * ::fma(U2, U2, ::fma(U1, U1, __dmul_rn(U0, U0))));
}
__device__ __forceinline__ Dual total_energy(double Cv, const Dual& T, const Dual& U0, const Dual& U1,
                                             const Dual& U2) {
  return Dual(total_energy(Cv, T.v, U0.v, U1.v, U2.v), Cv * T.d + U0.v * U0.d + U1.v * U1.d + U2.v * U2.d);
}
// numerator and denominator of Venkatakrishnan's (r^2 + 2 r) / (r^2 + r + 2),
// r = ra / rb; equal where r = 2 exactly, a linear profile on uniform cells
__device__ __forceinline__ void venkatakrishnan(double ra, double rb, double& num, double& den) {
  const double aa = __dmul_rn(ra, ra), ab = __dmul_rn(ra, rb), bb = __dmul_rn(rb, rb);
  num = ::fma(2.0, ab, aa);
  den = __dadd_rn(::fma(2.0, bb, ab), aa);
}
__device__ __forceinline__ void venkatakrishnan(const Dual& ra, const Dual& rb, Dual& num, Dual& den) {
  venkatakrishnan(ra.v, rb.v, num.v, den.v);
  num.d = 2.0 * (ra.d * (ra.v + rb.v) + ra.v * rb.d);
  den.d = ra.d * (2.0 * ra.v + rb.v) + rb.d * (ra.v + 4.0 * rb.v);
}

// TVD limitedScheme face value from the two cell values and the upwind
// cell's gradient projected on C_nei - C_own (NVD/TVD r with vanLeer or Minmod)
template <typename Real, typename GT>
__device__ __forceinline__ Real tvd_face(int scheme, double wf, double wUp, const Real& qo, const Real& qn,
                                         const GT& gradcf) {
  const Real gradf = qn - qo;
  Real r;
  if (fabs(gradcf) >= 1000 * fabs(gradf))
    r = 2 * 1000 * (gradcf >= 0 ? 1.0 : -1.0) * (gradf >= 0 ? 1.0 : -1.0) - 1.0;
  else
    r = 2 * (gradcf / gradf) - 1;
  Real lim;
  if (scheme == ICS_RECON_VANLEER)
    lim = (r + fabs(r)) / (1 + fabs(r));
  else
    lim = fmax(fmin(fmin(r, 1.0), 2.0), 0.0);
  const Real wgt = lim * wf + (1.0 - lim) * wUp;
  return wgt * (qo - qn) + qn;
}

// reconstruct field k on face f for direction dir (+1 owner side, -1 neighbour side)
template <typename Real>
__device__ __forceinline__ Real reconstruct(const DevMesh& m, int scheme, int k, int f, int o, int nb, const Real& qo,
                                            const Real& qn, const Real* __restrict__ grad, double dir) {
  const int N = m.N, F = m.F;
  const double wUp = dir > 0 ? 1.0 : 0.0;
  if (scheme == ICS_RECON_UPWIND) return dir > 0 ? qo : qn;
  if (scheme == ICS_RECON_VANLEER || scheme == ICS_RECON_MINMOD) {
    const int c = dir > 0 ? o : nb;
    const double d0 = m.dCC[f], d1 = m.dCC[F + f], d2 = m.dCC[2 * F + f];
    const Real gradcf = project(d0, d1, d2, grad[(3 * k) * N + c], grad[(3 * k + 1) * N + c], grad[(3 * k + 2) * N + c]);
    return tvd_face(scheme, m.w[f], wUp, qo, qn, gradcf);
  }
  // MUSCL: upwind value + limited-gradient extrapolation (the small products
  // are summed before they meet the value: one rounding at its size)
  const int c = dir > 0 ? o : nb;
  const double* d = dir > 0 ? m.dOwn : m.dNei;
  const Real base = dir > 0 ? qo : qn;
  return base + project(d[f], d[F + f], d[2 * F + f], grad[(3 * k) * N + c], grad[(3 * k + 1) * N + c],
                        grad[(3 * k + 2) * N + c]);
}

ResParams res_params(const Handle& h);
// fields with a reconstruction gradient (bit k = q field k) and the limiter
// kind of the MUSCL groups (0 none, 1 minmod, 2 Venkatakrishnan)
unsigned grad_mask(const Handle& h, int* limited);

}  // namespace ics
