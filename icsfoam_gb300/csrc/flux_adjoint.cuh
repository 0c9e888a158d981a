// Reverse-mode derivatives of the per-face flux functions (flux.cuh): given
// the adjoint Fb of the five fluxes, the adjoints of the two face states.
//
// Each function recomputes the flux's intermediate values in the flux's own
// order, takes the branches it takes (decided on the values, with the
// conventions of the dual numbers at ties), and walks the expressions
// backwards.  One value pass and one backward pass, about 500 FP64 operations
// for HLLC, stand where 16 forward-mode passes (one per input, value and
// derivative: about 14,000) stood: the reverse product is bound by GB300's
// FP64 pipe.  465k-cell swept bump, HLLC: k_adj_face 13.8 -> 1.09 ms.
//
// The Roe flux is differentiated in its wave form: with c^2 = (gamma - 1)(H -
// |U|^2/2) the product P |Lambda| P^-1 dW of flux_roe is the sum of the
// entropy, shear and acoustic waves, in which the Roe density cancels.  That
// holds for a fixed frame (um = 0) only.
#pragma once

#include "flux.cuh"

namespace ics {

// adjoints of the Roe averages U = (k Ur + Ul)/(k + 1), H likewise, k =
// sqrt(rr/rl), into the two sides' adjoints
__device__ __forceinline__ void roe_average_adjoint(const FState& L, const FState& R, double k, double icr,
                                                    const double U[3], double H, const double Ub[3], double Hb,
                                                    FState& Lb, FState& Rb) {
  double kb = Hb * (R.H - H);
  const double wr = k * icr;
#pragma unroll
  for (int i = 0; i < 3; ++i) {
    kb += Ub[i] * (R.U[i] - U[i]);
    Rb.U[i] += Ub[i] * wr;
    Lb.U[i] += Ub[i] * icr;
  }
  Rb.H += Hb * wr;
  Lb.H += Hb * icr;
  const double h = 0.5 * kb * wr;  // kb icr dk, dk = k/2 (drr/rr - drl/rl)
  if (R.rho >= VSMALL) Rb.rho += h / R.rho;
  if (L.rho >= VSMALL) Lb.rho -= h / L.rho;
}

// c = sqrt(|z|), z = (g - 1)(H - |U|^2/2)
__device__ __forceinline__ void roe_sound_adjoint(double g, double z, double c, const double U[3], double cb,
                                                  double Ub[3], double& Hb) {
  const double zb = c > 0.0 ? (z >= 0.0 ? 0.5 : -0.5) * (g - 1.0) * cb / c : 0.0;
  Hb += zb;
#pragma unroll
  for (int i = 0; i < 3; ++i) Ub[i] -= zb * U[i];
}

// false where several wave regions have a non-zero switch (flux_hllc's
// general sum): the caller differentiates those faces by dual numbers
__device__ __forceinline__ bool flux_hllc_adjoint(const FState& L, const FState& R, const double n[3], double magS,
                                                  double g, double um, const double Fb[5], FState& Lb, FState& Rb) {
  const double k = sqrt(fmax(VSMALL, R.rho) / fmax(VSMALL, L.rho));
  const double icr = 1.0 / (k + 1.0);
  double uA[3];
#pragma unroll
  for (int i = 0; i < 3; ++i) uA[i] = (k * R.U[i] + L.U[i]) * icr;
  const double HA = (k * R.H + L.H) * icr;
  const double z = (g - 1.0) * (HA - 0.5 * dot3(uA, uA));
  const double cA = sqrt(fabs(z));
  const double ul = dot3(L.U, n) - um, ur = dot3(R.U, n) - um, ua = dot3(uA, n) - um;
  const bool slOwn = ul - L.c <= ua - cA, srOwn = ur + R.c >= ua + cA;
  const double Sl = slOwn ? ul - L.c : ua - cA;
  const double Sr = srOwn ? ur + R.c : ua + cA;
  const double A = Sr - ur, C = Sl - ul;
  const double iden = 1.0 / (R.rho * A - L.rho * C);
  const double Sm = (R.rho * ur * A - L.rho * ul * C + L.p - R.p) * iden;
  const double coefSl = pos0d(Sl), coefSr = negd(Sr), coefSm = pos0d(Sm);
  const double coefSlm = (1.0 - coefSl) * coefSm, coefSmr = (1.0 - coefSm) * (1.0 - coefSr);
  if ((coefSl != 0.0) + (coefSlm != 0.0) + (coefSmr != 0.0) + (coefSr != 0.0) != 1) return false;
  const bool left = coefSl != 0.0 || coefSlm != 0.0;
  const FState& X = left ? L : R;
  FState Xb{0, 0, {0, 0, 0}, 0, 0, 0};
  const double uX = left ? ul : ur;
  double a[5];
#pragma unroll
  for (int i = 0; i < 5; ++i) a[i] = Fb[i] * magS;
  const double an = a[1] * n[0] + a[2] * n[1] + a[3] * n[2];
  double uXb = 0.0;
  Lb = FState{0, 0, {0, 0, 0}, 0, 0, 0};
  Rb = Lb;
  if (coefSl != 0.0 || coefSr != 0.0) {  // the plain flux of one side
    const double m = X.rho * uX;
    const double mb = a[0] + a[1] * X.U[0] + a[2] * X.U[1] + a[3] * X.U[2] + a[4] * X.H;
#pragma unroll
    for (int i = 0; i < 3; ++i) Xb.U[i] = a[1 + i] * m + mb * X.rho * n[i];
    Xb.p = an;
    Xb.H = a[4] * m;
    Xb.rho = mb * uX;
    (left ? Lb : Rb) = Xb;
    return true;
  }
  const double SX = left ? Sl : Sr;
  const double iX = 1.0 / (SX - Sm);
  const double d = SX - uX;
  const double rs = iX * d * X.rho;  // star density
  const double v = uX - Sm;
  const double pS = X.p - X.rho * d * v;
  const double es = iX * (pS * Sm - X.p * uX);  // rhoE* = rs E + es
  const double q = iX * (pS - X.p);             // (rho U)*_k = rs U_k + q n_k
  const double aU = a[1] * X.U[0] + a[2] * X.U[1] + a[3] * X.U[2];
  const double rsb = Sm * (a[0] + aU + a[4] * X.E);
  double Smb = rs * (a[0] + aU + a[4] * X.E) + q * an + a[4] * (es + pS) + a[4] * Sm * iX * pS;
  const double iXb = Sm * (an * (pS - X.p) + a[4] * (pS * Sm - X.p * uX)) + rsb * d * X.rho;
  const double pSb = an + a[4] * (Sm + um) + iX * Sm * (an + a[4] * Sm);
  const double t = -iXb * iX * iX;  // adjoint of SX - Sm
  const double db = rsb * iX * X.rho;
  uXb = -a[4] * Sm * iX * X.p - db + pSb * X.rho * (v - d);
  double SXb = t + db - pSb * X.rho * v;
  Smb += pSb * X.rho * d - t;
  Xb.rho = rsb * iX * d - pSb * d * v;
  Xb.p = pSb - iX * Sm * (an + a[4] * uX);
  Xb.E = a[4] * Sm * rs;
#pragma unroll
  for (int i = 0; i < 3; ++i) Xb.U[i] = a[1 + i] * Sm * rs;
  (left ? Lb : Rb) = Xb;
  double ulb = left ? uXb : 0.0, urb = left ? 0.0 : uXb;
  double Slb = left ? SXb : 0.0, Srb = left ? 0.0 : SXb;
  // Sm = (rr ur A - rl ul C + pl - pr) / (rr A - rl C)
  const double nb = Smb * iden, dnb = -nb * Sm;
  Rb.rho += (nb * ur + dnb) * A;
  Lb.rho -= (nb * ul + dnb) * C;
  Lb.p += nb;
  Rb.p -= nb;
  const double Ab = (nb * ur + dnb) * R.rho, Cb = -(nb * ul + dnb) * L.rho;
  urb += nb * R.rho * A - Ab;
  ulb -= nb * L.rho * C + Cb;
  Srb += Ab;
  Slb += Cb;
  double uab = 0.0, cAb = 0.0;
  if (slOwn) {
    ulb += Slb;
    Lb.c -= Slb;
  } else {
    uab += Slb;
    cAb -= Slb;
  }
  if (srOwn) {
    urb += Srb;
    Rb.c += Srb;
  } else {
    uab += Srb;
    cAb += Srb;
  }
#pragma unroll
  for (int i = 0; i < 3; ++i) {
    Lb.U[i] += ulb * n[i];
    Rb.U[i] += urb * n[i];
  }
  if (slOwn && srOwn) return true;  // the averages decided neither wave speed
  double uAb[3] = {uab * n[0], uab * n[1], uab * n[2]}, HAb = 0.0;
  roe_sound_adjoint(g, z, cA, uA, cAb, uAb, HAb);
  roe_average_adjoint(L, R, k, icr, uA, HA, uAb, HAb, Lb, Rb);
  return true;
}

__device__ __forceinline__ void flux_ausm_adjoint(const FState& L, const FState& R, const double S[3], double magS,
                                                  int lowMach, double um, const double Fb[5], FState& Lb, FState& Rb) {
  const double im = 1.0 / magS;
  const double uL = dot3(L.U, S) * im - um, uR = dot3(R.U, S) * im - um;
  const bool cOwnL = L.c >= uL, cOwnR = R.c >= -uR;
  const double mL = cOwnL ? L.c : uL, mR = cOwnR ? R.c : -uR;
  const double cl = L.c * L.c / mL, cr = R.c * R.c / mR;  // ordered by flux_ausm's own quotients
  const double imL = 1.0 / mL, imR = 1.0 / mR;
  const bool cfL = cl <= cr;
  const double cf = cfL ? cl : cr;
  const double icf = 1.0 / cf;
  const double ML = uL * icf, MR = uR * icf;
  double Mp, pp, dMp, dpp;
  if (fabs(ML) < 1.0) {
    const double p2 = 0.25 * sq(ML + 1), m2 = -0.25 * sq(ML - 1);
    const double dp2 = 0.5 * (ML + 1), dm2 = -0.5 * (ML - 1);
    const double w = 2 - ML - 3 * ML * m2;
    Mp = p2 * (1 - 2 * m2);
    pp = p2 * w;
    dMp = dp2 * (1 - 2 * m2) - 2 * p2 * dm2;
    dpp = dp2 * w + p2 * (-1 - 3 * m2 - 3 * ML * dm2);
  } else {
    Mp = fmax(ML, 0.0);
    pp = ML > 0 ? 1.0 : 0.0;
    dMp = ML >= 0 ? 1.0 : 0.0;
    dpp = 0.0;
  }
  double Mm, pm, dMm, dpm;
  if (fabs(MR) < 1.0) {
    const double m2 = -0.25 * sq(MR - 1), p2 = 0.25 * sq(MR + 1);
    const double dm2 = -0.5 * (MR - 1), dp2 = 0.5 * (MR + 1);
    const double w = -2 - MR + 3 * MR * p2;
    Mm = m2 * (1 + 2 * p2);
    pm = m2 * w;
    dMm = dm2 * (1 + 2 * p2) + 2 * m2 * dp2;
    dpm = dm2 * w + m2 * (-1 + 3 * p2 + 3 * MR * dp2);
  } else {
    Mm = fmin(MR, 0.0);
    pm = MR < 0 ? 1.0 : 0.0;
    dMm = MR <= 0 ? 1.0 : 0.0;
    dpm = 0.0;
  }
  double M12 = Mp + Mm;
  const double Mmean = 0.5 * (sq(uL) + sq(uR)) * sq(icf);
  const double rs = L.rho + R.rho, dp = R.p - L.p;
  const double iD = 1.0 / (0.5 * rs * sq(cf));
  const double f = fmax(1.0 - Mmean, 0.0);
  const double MD = -0.25 * f * dp * iD;
  const double w12 = (M12 > 0.0 && M12 + MD <= 0.0) || (M12 < 0.0 && M12 + MD >= 0.0) ? 0.2 : 1.0;
  M12 += w12 * MD;
  const double du = uR - uL;
  const bool left = M12 >= 0;
  const FState& up = left ? L : R;
  const double ra = M12 * cf * up.rho;
  // backwards
  const double rab = magS * (Fb[0] + Fb[1] * up.U[0] + Fb[2] * up.U[1] + Fb[3] * up.U[2] + Fb[4] * up.H);
  const double pb = Fb[1] * S[0] + Fb[2] * S[1] + Fb[3] * S[2] + Fb[4] * um * magS;
  Lb = FState{0, 0, {0, 0, 0}, 0, 0, 0};
  Rb = Lb;
  FState& ub = left ? Lb : Rb;
  const double rm = ra * magS;
#pragma unroll
  for (int i = 0; i < 3; ++i) ub.U[i] = Fb[1 + i] * rm;
  ub.H = Fb[4] * rm;
  ub.rho = rab * M12 * cf;
  const double M12b = rab * cf * up.rho;
  double cfb = rab * M12 * up.rho;
  double ppb = pb * L.p, pmb = pb * R.p, rsb = 0.0, uLb = 0.0, uRb = 0.0;
  Lb.p = pb * pp;
  Rb.p = pb * pm;
  if (lowMach) {
    const double q = -0.25 * pb, ppm = pp * pm;
    ppb += q * pm * rs * cf * du;
    pmb += q * pp * rs * cf * du;
    rsb += q * ppm * cf * du;
    cfb += q * ppm * rs * du;
    uRb += q * ppm * rs * cf;
    uLb -= q * ppm * rs * cf;
  }
  const double MDb = w12 * M12b;
  const double fb = -0.25 * MDb * dp * iD;
  const double dpb = -0.25 * MDb * f * iD;
  const double Db = -MDb * MD * iD;
  Rb.p += dpb;
  Lb.p -= dpb;
  rsb += 0.5 * Db * sq(cf);
  cfb += Db * rs * cf;
  if (1.0 - Mmean >= 0.0) {
    const double mb = -fb * sq(icf);
    uLb += mb * uL;
    uRb += mb * uR;
    cfb += 2.0 * fb * Mmean * icf;
  }
  Lb.rho += rsb;
  Rb.rho += rsb;
  const double MLb = M12b * dMp + ppb * dpp, MRb = M12b * dMm + pmb * dpm;
  uLb += MLb * icf;
  uRb += MRb * icf;
  cfb -= (MLb * ML + MRb * MR) * icf;
  if (cfL) {
    if (cOwnL) {
      Lb.c = cfb;
    } else {
      Lb.c = 2.0 * cfb * L.c * imL;
      uLb -= cfb * cl * imL;
    }
  } else {
    if (cOwnR) {
      Rb.c = cfb;
    } else {
      Rb.c = 2.0 * cfb * R.c * imR;
      uRb += cfb * cr * imR;
    }
  }
#pragma unroll
  for (int i = 0; i < 3; ++i) {
    Lb.U[i] += uLb * im * S[i];
    Rb.U[i] += uRb * im * S[i];
  }
}

// entropy-fixed wave speed l(x, eps): l = x, or (x^2 + eps^2)/(2 eps) below
// eps; adds the adjoint of eps, returns the one of x
__device__ __forceinline__ double harten(double x, double eps) { return x < eps ? (x * x + eps * eps) / (2.0 * eps) : x; }
__device__ __forceinline__ double harten_adjoint(double x, double eps, double lb, double& epsb) {
  if (!(x < eps)) return lb;
  const double r = x / eps;
  epsb += lb * (0.5 - 0.5 * r * r);
  return lb * r;
}

// fixed frame only (um = 0)
__device__ __forceinline__ void flux_roe_adjoint(const FState& L, const FState& R, const double n[3], double magS,
                                                 double g, double fix, const double Fb[5], FState& Lb, FState& Rb) {
  const double k = sqrt(fmax(VSMALL, R.rho) / fmax(VSMALL, L.rho));
  const double icr = 1.0 / (k + 1.0);
  double U[3];
#pragma unroll
  for (int i = 0; i < 3; ++i) U[i] = (k * R.U[i] + L.U[i]) * icr;
  const double H = (k * R.H + L.H) * icr;
  const double ke = 0.5 * dot3(U, U);
  const double z = (g - 1.0) * (H - ke);
  const double c = sqrt(fabs(z));
  const double un = dot3(U, n);
  const double L1 = fabs(un), L2 = fabs(un + c), L3 = fabs(un - c);
  const double eps = fix * fmax(L2, L3);
  const double l1 = harten(L1, eps), l2 = harten(L2, eps), l3 = harten(L3, eps);
  // jumps and wave strengths (w = d(rho U) - U d(rho))
  const double d0 = R.rho - L.rho, dE = R.rho * R.E - L.rho * L.E;
  double dm[3], w[3];
#pragma unroll
  for (int i = 0; i < 3; ++i) {
    dm[i] = R.rho * R.U[i] - L.rho * L.U[i];
    w[i] = dm[i] - U[i] * d0;
  }
  const double wn = dot3(w, n);
  const double dp = (g - 1.0) * (ke * d0 - dot3(U, dm) + dE);
  const double ic = 1.0 / c, hc2 = 0.5 * ic * ic;
  const double a2 = (dp + c * wn) * hc2, a3 = (dp - c * wn) * hc2, a1 = d0 - 2.0 * dp * hc2;
  double sh[3];
#pragma unroll
  for (int i = 0; i < 3; ++i) sh[i] = w[i] - n[i] * wn;
  // backwards through the dissipation -0.5 |S| (waves)
  const double h = 0.5 * magS;
  const double A0 = -h * Fb[0], AE = -h * Fb[4];
  const double Am[3] = {-h * Fb[1], -h * Fb[2], -h * Fb[3]};
  const double AmU = dot3(Am, U), Amn = dot3(Am, n);
  const double e1 = A0 + AmU + AE * ke;
  const double e2 = A0 + AmU + c * Amn + AE * (H + c * un);
  const double e3 = A0 + AmU - c * Amn + AE * (H - c * un);
  const double l1b = a1 * e1 + dot3(Am, sh) + AE * dot3(U, sh);
  const double l2b = a2 * e2, l3b = a3 * e3;
  const double a1b = l1 * e1, a2b = l2 * e2, a3b = l3 * e3;
  const double s2 = l2 * a2, s3 = l3 * a3, sm = l1 * a1 + s2 + s3;
  double Ub[3], shb[3];
#pragma unroll
  for (int i = 0; i < 3; ++i) {
    shb[i] = l1 * (Am[i] + AE * U[i]);
    Ub[i] = sm * Am[i] + l1 * AE * (sh[i] + a1 * U[i]);
  }
  double cb = (s2 - s3) * (Amn + AE * un);
  double unb = AE * c * (s2 - s3);
  double Hb = AE * (s2 + s3);
  const double dpb = (a2b + a3b - 2.0 * a1b) * hc2;
  const double wnb = (a2b - a3b) * c * hc2 - dot3(shb, n);
  cb += (a2b - a3b) * wn * hc2 - 2.0 * ic * (a2b * a2 + a3b * a3) + 4.0 * a1b * dp * hc2 * ic;
  double d0b = a1b;
  const double G = (g - 1.0) * dpb;
  double dmb[3];
#pragma unroll
  for (int i = 0; i < 3; ++i) {
    const double wb = shb[i] + wnb * n[i];
    dmb[i] = wb - G * U[i];
    Ub[i] += G * (U[i] * d0 - dm[i]) - wb * d0;
    d0b -= wb * U[i];
  }
  d0b += G * ke;
  double epsb = 0.0;
  const double L1b = harten_adjoint(L1, eps, l1b, epsb);
  double L2b = harten_adjoint(L2, eps, l2b, epsb), L3b = harten_adjoint(L3, eps, l3b, epsb);
  if (L2 >= L3)
    L2b += fix * epsb;
  else
    L3b += fix * epsb;
  const double s2b = un + c >= 0.0 ? L2b : -L2b, s3b = un - c >= 0.0 ? L3b : -L3b;
  unb += (un >= 0.0 ? L1b : -L1b) + s2b + s3b;
  cb += s2b - s3b;
#pragma unroll
  for (int i = 0; i < 3; ++i) Ub[i] += unb * n[i];
  roe_sound_adjoint(g, z, c, U, cb, Ub, Hb);
  // the central flux and the jumps of each side
  const double an = h * (Fb[1] * n[0] + Fb[2] * n[1] + Fb[3] * n[2]);
  auto side = [&](const FState& X, FState& Xb, double sgn) {
    const double u = dot3(X.U, n), m = X.rho * u;
    const double mb = h * (Fb[0] + Fb[1] * X.U[0] + Fb[2] * X.U[1] + Fb[3] * X.U[2] + Fb[4] * X.H);
    Xb.rho = mb * u + sgn * (d0b + dot3(dmb, X.U) + G * X.E);
#pragma unroll
    for (int i = 0; i < 3; ++i) Xb.U[i] = h * Fb[1 + i] * m + mb * X.rho * n[i] + sgn * dmb[i] * X.rho;
    Xb.p = an;
    Xb.E = sgn * G * X.rho;
    Xb.H = h * Fb[4] * m;
    Xb.c = 0.0;
  };
  side(L, Lb, -1.0);
  side(R, Rb, 1.0);
  roe_average_adjoint(L, R, k, icr, U, H, Ub, Hb, Lb, Rb);
}

}  // namespace ics
