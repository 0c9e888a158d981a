// Pieces of the GMRES cycle shared by its kernels (k_column.cu, k_linalg.cu):
// 16-byte vectors of the Krylov element types and the Givens update of a
// Hessenberg column.
#pragma once

#include "dual.cuh"
#include "ics_internal.cuh"

namespace ics {

__device__ __forceinline__ int ld_relaxed_int(const int* p) {
  int v;
  asm volatile("ld.relaxed.gpu.global.b32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}

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

// Conversions without the FP64 pipe (which a conversion occupies as long as an
// addition): the exponent is rebiased in integers, and FP64 to FP32 rounds to
// nearest even.  Subnormal numbers, infinities and NaN take the conversion.
__device__ __forceinline__ double widen(float f) {
  const unsigned b = __float_as_uint(f), a = b & 0x7fffffffu, sign = b & 0x80000000u;
  if (a - 0x00800000u < 0x7f000000u) return __hiloint2double(sign | ((a >> 3) + (896u << 20)), b << 29);
  return a == 0 ? __hiloint2double(sign, 0) : double(f);
}
__device__ __forceinline__ double widen(double f) { return f; }

__device__ __forceinline__ float narrow(double d) {
  const unsigned hi = __double2hiint(d), lo = __double2loint(d), a = hi & 0x7fffffffu, sign = hi & 0x80000000u;
  if (a - (897u << 20) < (253u << 20)) {  // a result of exponent 2^-126 .. 2^126, whose rounding may carry
    const unsigned f = ((a - (896u << 20)) << 3) | (lo >> 29), rest = lo & 0x1fffffffu;
    return __uint_as_float(sign | (f + (rest > 0x10000000u - (f & 1))));
  }
  return (a | lo) == 0 ? __uint_as_float(sign) : float(d);
}
template <typename TD>
__device__ __forceinline__ TD convert(double x) {
  if constexpr (sizeof(TD) == 4)
    return narrow(x);
  else
    return x;
}

// x / b from the reciprocal r = fl(1/b) and its error term rl = r (1 - b r), after
// Markstein:
// two operations, within a half unit and 2^-50 of the quotient
template <typename TV>
__device__ __forceinline__ TV quotient(TV x, TV r, TV rl) {
  return fma(x, r, x * rl);
}

// Sums of NV values per thread over a block of W warps.  An FP64 instruction
// takes 64 cycles of its scheduler whichever lanes are active, so a warp folds
// its values together -- every exchange halves the values a lane carries, 9
// additions for 8 values instead of 40 -- and one warp folds the warps' sums on
// all its lanes.  In warp 0, lane FOLD_GROUP<NV> k returns the sum of value k
// (as do the lanes after it up to the next value's); sm is free after a barrier.
template <int NV>
constexpr int FOLD_VALUES = NV <= 1 ? 1 : NV <= 2 ? 2 : NV <= 4 ? 4 : 8;
template <int NV>
constexpr int FOLD_GROUP = 32 / FOLD_VALUES<NV>;

template <int NV, int W>
__device__ __forceinline__ double block_sums(const double (&v)[NV], double (*sm)[FOLD_VALUES<NV>]) {
  static_assert(NV <= 8 && (W & (W - 1)) == 0 && W <= 32, "");
  constexpr int P = FOLD_VALUES<NV>, G = FOLD_GROUP<NV>;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  double a[P];
#pragma unroll
  for (int k = 0; k < P; ++k) a[k] = k < NV ? v[k] : 0.0;
  int n = P;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    if (n > 1) {
      n >>= 1;
      const bool high = lane & o;
#pragma unroll
      for (int k = 0; k < P / 2; ++k)
        if (k < n) {
          const double keep = high ? a[k + n] : a[k], send = high ? a[k] : a[k + n];
          a[k] = keep + __shfl_xor_sync(0xffffffffu, send, o);
        }
    } else {
      a[0] += __shfl_xor_sync(0xffffffffu, a[0], o);
    }
  }
  if (lane % G == 0) sm[warp][lane / G] = a[0];
  __syncthreads();
  double t = 0.0;
  if (warp == 0) {
    constexpr int SPAN = G < W ? G : W;  // lanes that share a value's warps
    if (lane % G < SPAN) {
      t = sm[lane % G][lane / G];
#pragma unroll
      for (int w = SPAN; w < W; w += SPAN) t += sm[w + lane % G][lane / G];
    }
#pragma unroll
    for (int o = SPAN / 2; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
  }
  return t;
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

// Hessenberg column i with |w|^2 = nrm2: rotate it with the previous Givens
// rotations and make a new one (gmres.C:1013-1027, rotation gmres.C:44-69).
// One thread; the loads of eight rows are in flight together (as dependent
// loads and stores a column of 8 takes 5 us).
__device__ __forceinline__ void hess_column(double* H, double* cs, double* sn, double* bh, int i, int m, double nrm2) {
  const double beta = sqrt(nrm2);
  double a = H[i];
  for (int j0 = 0; j0 < i; j0 += 8) {
    double b[8], c[8], s[8];
#pragma unroll
    for (int k = 0; k < 8; ++k)
      if (j0 + k < i) {
        b[k] = H[(j0 + k + 1) * m + i];
        c[k] = cs[j0 + k];
        s[k] = sn[j0 + k];
      }
#pragma unroll
    for (int k = 0; k < 8; ++k)
      if (j0 + k < i) {
        H[(j0 + k) * m + i] = c[k] * a - s[k] * b[k];
        a = s[k] * a + c[k] * b[k];
      }
  }
  const double b0 = bh[i], b1 = bh[i + 1];
  double c, s;
  givens(a, beta, c, s);
  cs[i] = c;
  sn[i] = s;
  bh[i] = c * b0 - s * b1;
  bh[i + 1] = s * b0 + c * b1;
  H[i * m + i] = c * a - s * beta;
}

// H y = bh, H upper triangular of m <= 64 rows: one warp, a lane holds the sums
// of rows lane and lane + 32; the diagonal's reciprocals are made together and
// eight columns are loaded at a time
__device__ __forceinline__ void back_substitute(const double* __restrict__ H, const double* __restrict__ bh,
                                                double* __restrict__ y, int m) {
  static_assert(MAX_DIRS <= 64, "two rows per lane");
  const int lane = threadIdx.x & 31;
  double sum[2], st[2], r[2];
#pragma unroll
  for (int q = 0; q < 2; ++q) {
    const int row = lane + 32 * q;
    const double h = row < m ? H[row * m + row] : 1.0;
    sum[q] = row < m ? bh[row] : 0.0;
    st[q] = h >= 0 ? h + VSMALL : h - VSMALL;
    r[q] = 1.0 / st[q];
  }
  for (int i0 = m - 1; i0 >= 0; i0 -= 8) {
    double h[8][2];
#pragma unroll
    for (int k = 0; k < 8; ++k)
#pragma unroll
      for (int q = 0; q < 2; ++q) {
        const int row = lane + 32 * q, i = i0 - k;
        h[k][q] = row < i ? H[row * m + i] : 0.0;
      }
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      const int i = i0 - k;
      if (i < 0) break;
      const double yi = __shfl_sync(0xffffffffu, i < 32 ? quot(sum[0], st[0], r[0]) : quot(sum[1], st[1], r[1]), i & 31);
      sum[0] -= h[k][0] * yi;
      if (m > 32) sum[1] -= h[k][1] * yi;
      if (lane == 0) y[i] = yi;
    }
  }
}

// after the Gram-Schmidt of direction i: H[j][i] for j <= i are in H, nrm2[i]
// holds |w|^2
__device__ __forceinline__ void dev_hess(KrylovScalars* ks, int i, int m) {
  if (!ks->status) hess_column(ks->H, ks->c, ks->s, ks->bh, i, m, ks->nrm2[i]);
}

// start of a cycle: bh = (beta, 0...)
__device__ __forceinline__ void dev_beta0(KrylovScalars* ks, double beta, int m) {
  for (int i = 0; i <= m; ++i) ks->bh[i] = 0.0;
  ks->bh[0] = beta;
  if (!(beta > 0.0)) atomicOr(&ks->status, isfinite(beta) ? 2 : 4);  // beside bit 8 of a wait that gave up
}

}  // namespace ics
