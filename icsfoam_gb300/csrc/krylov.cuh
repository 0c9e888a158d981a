// Pieces of the GMRES cycle shared by its kernels (k_column.cu, k_linalg.cu):
// 16-byte vectors of the Krylov element types and the Givens update of a
// Hessenberg column.
#pragma once

#include "ics_internal.cuh"

namespace ics {

// 16-byte vector of the Krylov element type
template <typename TV>
struct V16;
template <>
struct V16<float> {
  using T = float4;
  static constexpr int n = 4;
};
template <>
struct V16<double> {
  using T = double2;
  static constexpr int n = 2;
};

__device__ __forceinline__ void axpy16(float4& x, float h, const float4& p) {
  x.x -= h * p.x;
  x.y -= h * p.y;
  x.z -= h * p.z;
  x.w -= h * p.w;
}
__device__ __forceinline__ void axpy16(double2& x, double h, const double2& p) {
  x.x -= h * p.x;
  x.y -= h * p.y;
}
// acc + a . b, one multiply-add per product
__device__ __forceinline__ float dot16(const float4& a, const float4& b, float acc) {
  return fmaf(a.w, b.w, fmaf(a.z, b.z, fmaf(a.y, b.y, fmaf(a.x, b.x, acc))));
}
__device__ __forceinline__ double dot16(const double2& a, const double2& b, double acc) {
  return fma(a.y, b.y, fma(a.x, b.x, acc));
}

__device__ __forceinline__ void givens(double h, double beta, double& c, double& s) {
  if (beta == 0) {
    c = 1;
    s = 0;
  } else if (fabs(beta) > fabs(h)) {
    const double tau = -h / beta;
    s = 1.0 / sqrt(1.0 + tau * tau);
    c = s * tau;
  } else {
    const double tau = -beta / h;
    c = 1.0 / sqrt(1.0 + tau * tau);
    s = c * tau;
  }
}

// after the Gram-Schmidt of direction i: H[j][i] for j <= i are in H, nrm2[i]
// holds |w|^2; rotate column i with the previous Givens rotations and make a
// new one (gmres.C:1013-1027, rotation gmres.C:44-69)
__device__ __forceinline__ void dev_hess(KrylovScalars* ks, int i, int m) {
  if (ks->status) return;
  double* H = ks->H;
  const double beta = sqrt(ks->nrm2[i]);
  for (int j = 0; j < i; ++j) {
    const double Hji = H[j * m + i];
    H[j * m + i] = ks->c[j] * Hji - ks->s[j] * H[(j + 1) * m + i];
    H[(j + 1) * m + i] = ks->s[j] * Hji + ks->c[j] * H[(j + 1) * m + i];
  }
  givens(H[i * m + i], beta, ks->c[i], ks->s[i]);
  const double bhi = ks->bh[i];
  ks->bh[i] = ks->c[i] * bhi - ks->s[i] * ks->bh[i + 1];
  ks->bh[i + 1] = ks->s[i] * bhi + ks->c[i] * ks->bh[i + 1];
  H[i * m + i] = ks->c[i] * H[i * m + i] - ks->s[i] * beta;
}

// start of a cycle: bh = (beta, 0...)
__device__ __forceinline__ void dev_beta0(KrylovScalars* ks, double beta, int m) {
  for (int i = 0; i <= m; ++i) ks->bh[i] = 0.0;
  ks->bh[0] = beta;
  if (!(beta > 0.0)) ks->status = isfinite(beta) ? 2 : 4;
}

}  // namespace ics
