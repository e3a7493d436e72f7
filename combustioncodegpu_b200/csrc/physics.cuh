// Device physics of the residual path, templated on the bulk precision T
// (double for the plain path, float for the mixed path) and on the species
// count NS (n > 0: n species; -n: a runtime count of at most n; 0: perfect air).
//
// Reference counterparts (file:line in CombustionCodeGPU):
//   NASA-7 h/cp with linear h below T_low ......... Thermo.cu:7-63
//   total energy .................................. Thermo.cu:66-86
//   temperature Newton (FP64 in every precision) .. Thermo.cu:89-125
//   Sutherland ..................................... Transport.cu:7-10
//   Wilke / constant-Schmidt transport ............. Transport.cu:43-96 (X[l])
//   MUSCL + minmod + face thermo ................... Reconstruction.cu:26-89, Limiter.cuh:13-16
//   AUSM+ ........................................... InviscidScheme.cu:24-108
// The polynomials are evaluated in Horner form and sqrt(mu_m/mu_n) as
// sqrt(mu_m)/sqrt(mu_n); both differ from the reference only by rounding.
#pragma once
#include <cuda_runtime.h>

#include "cc_common.h"

namespace ccb {

template <typename T>
__device__ __forceinline__ const SpecTables<T> &tab(const ChemParams &C);
template <>
__device__ __forceinline__ const SpecTables<double> &tab<double>(const ChemParams &C) {
  return C.d;
}
template <>
__device__ __forceinline__ const SpecTables<float> &tab<float>(const ChemParams &C) {
  return C.f;
}

template <int NS>
struct SpecCount {
  static constexpr int kArr = NS > 0 ? NS : (NS == 0 ? 1 : -NS);
  __device__ __forceinline__ static int n(const ChemParams &C) { return NS >= 0 ? NS : C.ns; }
};

// Division, reciprocal, square root and x^-0.145 of the bulk precision: IEEE
// in FP64 (the plain path), hardware approximations in FP32 (the mixed path;
// relative error of a few ulp, far below the path's 1e-5 error budget).
// These take denormal operands: a density of 1e-40 is far from any flow, but
// flushed to zero it divides to infinity.
__device__ __forceinline__ double fdiv(double a, double b) { return a / b; }
__device__ __forceinline__ float fdiv(float a, float b) { return __fdividef(a, b); }
__device__ __forceinline__ double frcp(double a) { return 1.0 / a; }
__device__ __forceinline__ float frcp(float a) { return __fdividef(1.0f, a); }
__device__ __forceinline__ double fsqrt(double a) { return sqrt(a); }
__device__ __forceinline__ float fsqrt(float a) { return a * rsqrtf(a); }

// The same where the operand taken by the hardware is a normal number whatever
// the state's density and pressure: sums over mole fractions that add up to
// one, specific heats, a temperature and what is formed of it and the species'
// constants (normal down to 1e-30 K).  Numerators may be denormal.  These
// flush denormal operands (.ftz), which saves the scaling of every operand:
// the update of 128^3 mixed takes 0.314 ms a stage with them and 0.318 with the
// others, the halo program of 12 blocks 0.307 and 0.320, the 128^3 step 2.637 and
// 2.655.
__device__ __forceinline__ double rcp_normal(double a) { return 1.0 / a; }
__device__ __forceinline__ float rcp_normal(float a) {
  float r;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(a));
  return r;
}
__device__ __forceinline__ double div_normal(double a, double b) { return a / b; }
__device__ __forceinline__ float div_normal(float a, float b) { return a * rcp_normal(b); }
__device__ __forceinline__ double sqrt_normal(double a) { return sqrt(a); }
__device__ __forceinline__ float sqrt_normal(float a) {
  float r;
  asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(a));
  return a * r;
}

// Length of the face vector, from its square, and the reciprocal of that
// length.  The mass flux takes the product of both, so what counts is that
// they are reciprocal.  FP32: the reciprocal of the length as computed; the
// reciprocal root itself leaves twice its error in the product, the same at
// every face of a uniform grid (velocity error after 20 steps of the 32^3 box
// 1.73e-7 against 1.30e-7).  FP64: its error is far below the rounding of the
// fluxes, and root and division cost 1 % of the faces.
__device__ __forceinline__ void length_and_reciprocal(double kk, double &len, double &inv) {
  inv = rsqrt(kk);
  len = kk * inv;
}
__device__ __forceinline__ void length_and_reciprocal(float kk, float &len, float &inv) {
  len = fsqrt(kk);
  inv = frcp(len);
}

// NASA-7 records (SpecTables::rec) are read through a pointer `rec` to the
// [kMaxSpec][kRecRanges][kRecLen] array: the stage kernels point it at a copy
// in shared memory, other kernels at the constant bank (param_rec).  The
// range is chosen per thread by the record address, so a warp whose points
// straddle t_mid reads two records in one vector load instead of serialising
// on divergent constant addresses, and the coefficients cannot be hoisted
// out of the surrounding loops into registers.
//
// A record holds a0..a5 of one range, times R_u / W: cp = a0 + a1 T + .. +
// a4 T^4 and h = a5 + T (a0 + a1 T/2 + .. + a4 T^4/5), per unit mass.  Below
// t_low, where h continues linearly with cp(t_low) (Thermo.cu:7-63), both are
// polynomials of the same form, so range 0 is a record too.
template <typename T>
__device__ __forceinline__ const T *param_rec(const ChemParams &C) {
  return &tab<T>(C).rec[0][0][0];
}

template <typename T>
__device__ __forceinline__ void load_rec(const T *r, T (&x)[6]);
template <>
__device__ __forceinline__ void load_rec<float>(const float *r, float (&x)[6]) {
  const float4 w = *reinterpret_cast<const float4 *>(r);
  const float2 y = *reinterpret_cast<const float2 *>(r + 4);
  x[0] = w.x, x[1] = w.y, x[2] = w.z, x[3] = w.w, x[4] = y.x, x[5] = y.y;
}
template <>
__device__ __forceinline__ void load_rec<double>(const double *r, double (&x)[6]) {
  const double2 *v = reinterpret_cast<const double2 *>(r);
#pragma unroll
  for (int q = 0; q < 3; ++q) {
    const double2 w = v[q];
    x[2 * q] = w.x, x[2 * q + 1] = w.y;
  }
}

// Record of species k at temperature t.
template <typename T>
__device__ __forceinline__ const T *species_rec(const SpecTables<T> &S, const T *rec, int k, T t) {
  const int r = t < S.t_low[k] ? 0 : (t < S.t_mid[k] ? 1 : 2);
  return rec + (kRecRanges * k + r) * kRecLen;
}

// The range of every species at temperature t at once, or -1 where they
// differ: with the usual tables (one t_low and t_mid for all species) two
// comparisons serve the whole mixture.
template <typename T>
__device__ __forceinline__ int common_range(const SpecTables<T> &S, T t) {
  if (t < S.t_low_min) return 0;
  if (t < S.t_mid_min) return t >= S.t_low_max ? 1 : -1;
  return t >= S.t_high_max ? 2 : -1;
}

template <typename T>
__device__ __forceinline__ T poly_cp(const T (&x)[6], T t) {
  return x[0] + t * (x[1] + t * (x[2] + t * (x[3] + t * x[4])));
}
template <typename T>
__device__ __forceinline__ T poly_h(const T (&x)[6], T t) {
  return x[5] + t * (x[0] + t * (T(0.5) * x[1] + t * (T(1.0 / 3.0) * x[2] + t * (T(0.25) * x[3] + t * (T(0.2) * x[4])))));
}

template <typename T>
__device__ __forceinline__ T nasa_h(const SpecTables<T> &S, const T *rec, int k, T t) {
  T x[6];
  load_rec<T>(species_rec(S, rec, k, t), x);
  return poly_h(x, t);
}

template <typename T>
__device__ __forceinline__ T nasa_cp(const SpecTables<T> &S, const T *rec, int k, T t) {
  T x[6];
  load_rec<T>(species_rec(S, rec, k, t), x);
  return poly_cp(x, t);
}

// Coefficients of the mixture sum_k w_k (h_k, cp_k) at temperature t: the
// species share the form of the polynomial, so their weighted coefficients
// are summed (6 multiply-adds per species) and one polynomial is evaluated,
// instead of two per species (about 20 operations each).  Where the species
// lie in different ranges (r < 0) each record is chosen by itself.
template <typename T, int NS>
__device__ __forceinline__ void nasa_mix(const ChemParams &C, const T *rec, T t, int r, const T *w, T (&c)[6]) {
  const SpecTables<T> &S = tab<T>(C);
  constexpr int A = SpecCount<NS>::kArr;
  const int ns = SpecCount<NS>::n(C);
#pragma unroll
  for (int q = 0; q < 6; ++q) c[q] = T(0);
  if (r >= 0) {
    const T *base = rec + r * kRecLen;
#pragma unroll
    for (int l = 0; l < A; ++l) {
      if (l < ns) {
        T x[6];
        load_rec<T>(base + kRecRanges * kRecLen * l, x);
#pragma unroll
        for (int q = 0; q < 6; ++q) c[q] += w[l] * x[q];
      }
    }
  } else {
#pragma unroll
    for (int l = 0; l < A; ++l) {
      if (l < ns) {
        T x[6];
        load_rec<T>(species_rec(S, rec, l, t), x);
#pragma unroll
        for (int q = 0; q < 6; ++q) c[q] += w[l] * x[q];
      }
    }
  }
}

template <typename T>
__device__ __forceinline__ T sutherland(T t) {
  // 1.716e-5 (T/273)^1.5 (273+111)/(T+111)
  const T r = t / T(273);
  return T(1.716e-5) * (r * sqrt(r)) * T(384) / (t + T(111));
}

template <typename T>
__device__ __forceinline__ T pow_m0145(T x);
template <>
__device__ __forceinline__ double pow_m0145<double>(double x) {
  return pow(x, -0.145);
}
template <>
__device__ __forceinline__ float pow_m0145<float>(float x) {
  float l, r;  // x: reduced temperature
  asm("lg2.approx.ftz.f32 %0, %1;" : "=f"(l) : "f"(x));
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(-0.145f * l));
  return r;
}

// Wilke mixture viscosity, modified-Wilke conductivity and constant-Schmidt
// rho*D_k.  cp[k] is the species cp per unit mass at temp.
template <typename T, int NS>
__device__ __forceinline__ void transport(const ChemParams &C, T temp, const T *Y, T mw_total, const T *cp,
                                          T &mu_out, T &lam_out, T *rhod) {
  const SpecTables<T> &S = tab<T>(C);
  constexpr int A = SpecCount<NS>::kArr;
  const int ns = SpecCount<NS>::n(C);
  T X[A], vis[A], svis[A], isvis[A];
  const T sqt = sqrt_normal(temp);
#pragma unroll
  for (int l = 0; l < A; ++l) {
    if (l < ns) {
      X[l] = Y[l] * mw_total * S.inv_mw[l];
      const T t_dl = temp * S.lj_inv[l];
      const T tp = t_dl + T(0.5);
      const T omega = T(1.147) * pow_m0145<T>(t_dl) + rcp_normal(tp * tp);
      vis[l] = div_normal(S.vis_coeff[l] * sqt, omega);
      svis[l] = sqrt_normal(vis[l]);
      isvis[l] = rcp_normal(svis[l]);
    }
  }
  T viscosity = 0, conductivity = 0;
#pragma unroll
  for (int m = 0; m < A; ++m) {
    if (m < ns) {
      T vt = 0;
#pragma unroll
      for (int n = 0; n < A; ++n) {
        if (n < ns) {
          T phi;
          if (m == n) {
            phi = T(1);
          } else {
            const T num = T(1) + svis[m] * isvis[n] * S.wj[m * kMaxSpec + n];
            phi = num * num * S.sw[m * kMaxSpec + n];
          }
          vt += phi * X[n];
        }
      }
      const T lam_m = vis[m] * (cp[m] + S.lam_shift[m]);
      viscosity += div_normal(vis[m] * X[m], vt);
      conductivity += div_normal(lam_m * X[m], T(1.065) * vt - T(0.065) * X[m]);
    }
  }
  mu_out = viscosity;
  lam_out = conductivity;
  const T inv_sc = T(1) / T(C.Sc);
#pragma unroll
  for (int l = 0; l < A; ++l) {
    if (l < ns) {
      const T d = X[l] - T(1);
      rhod[l] = (fabs(d) < T(1e-3)) ? viscosity * inv_sc : div_normal((T(1) - Y[l]) * viscosity, (T(1) - X[l]) * T(C.Sc));
    }
  }
}

// Point properties used by the stage update and the time step:
// mu, lambda, rho*D_k (stored) and gamma, acoustic speed (for dt).
template <typename T, int NS>
__device__ __forceinline__ void point_props(const ChemParams &C, const T *rec, T temp, const T *Y, T &mu, T &lam,
                                            T *rhod, T &gamma, T &c) {
  constexpr int A = SpecCount<NS>::kArr;
  const int ns = SpecCount<NS>::n(C);
  if (NS == 0 || (NS < 0 && ns == 0)) {
    const T c_temp = T(kGammaAir * kRu / kMwAir);
    c = sqrt(c_temp * temp);
    mu = sutherland<T>(temp);
    lam = mu * c_temp / T(kGammaAir - 1) / T(C.Pr);
    gamma = T(kGammaAir);
    return;
  }
  const SpecTables<T> &S = tab<T>(C);
  T cp[A], mwi = 0, cp_mix = 0;
#pragma unroll
  for (int l = 0; l < A; ++l)
    if (l < ns) cp[l] = nasa_cp<T>(S, rec, l, temp);
#pragma unroll
  for (int l = 0; l < A; ++l)
    if (l < ns) mwi += Y[l] * S.inv_mw[l], cp_mix += Y[l] * cp[l];
  const T gas = T(kRu) * mwi;
  gamma = div_normal(cp_mix, cp_mix - gas);
  c = sqrt_normal(gamma * gas * temp);
  transport<T, NS>(C, temp, Y, rcp_normal(mwi), cp, mu, lam, rhod);
}

// Temperature from internal energy by Newton iteration (tolerance 1e-3 on
// |1 - T1/T|, at most C.newton_max_iter iterations (1000 by default, as the
// reference), warm start t) in FP32, for the full-FP32 study; the FP64 Newton
// of the other precisions is in point_finish.
template <int NS>
__device__ __forceinline__ float newton_temperature_f32(const ChemParams &C, const float *rec, float e, const float *Y,
                                                        float gas_const, float t, bool &capped) {
  float err = 1;
  int iter = 0, range = -2;
  float x[6];  // the mixture's coefficients, summed again only where t has left their range
  while (err > 1e-3f && iter++ < C.newton_max_iter) {
    const int r = common_range(C.f, t);
    if (r != range || r < 0) nasa_mix<float, NS>(C, rec, t, r, Y, x), range = r;
    const float t1 = t - (poly_h(x, t) - gas_const * t - e) / (poly_cp(x, t) - gas_const);
    err = fabsf(1.0f - t1 / t);
    t = t1;
  }
  capped = err > 1e-3f;
  return t;
}

// 0.5 (sgn a + sgn b) min(|a|, |b|): the median of a, b and 0 in FP32 (four
// min/max instructions); in FP64, whose comparisons run on the slow FP64
// pipe, the smaller magnitude where the sign bits agree.
__device__ __forceinline__ float minmod(float a, float b) {
  return fmaxf(fminf(a, b), fminf(fmaxf(a, b), 0.0f));
}
__device__ __forceinline__ double minmod(double a, double b) {
  const double m = fmin(fabs(a), fabs(b));
  return (__double2hiint(a) ^ __double2hiint(b)) < 0 ? 0.0 : copysign(m, a);
}

// AUSM+ pressure splitting P+(M) = (M+1)^2 (2-M)/4 + a M (M^2-1)^2 and
// P-(M) = (M-1)^2 (2+M)/4 - a M (M^2-1)^2 for |M| <= 1, 1 / 0 beyond, with
// P+(M) + P-(M) = 1.  Returns P+(ml) + P-(mr) - 1 without the cancellation of
// forming the sum: in the subsonic case it is P+(ml) - P+(mr) = (ml - mr) x
// the divided difference of P+(M) = 1/2 + 3M/4 - M^3/4 + a (M^5 - 2M^3 + M).
template <typename T>
__device__ __forceinline__ T ausm_pressure_defect(T ml, T mr, T a) {
  auto p_plus = [&](T m) {
    const T q = m * m - T(1);
    return (m + T(1)) * (m + T(1)) * (T(2) - m) * T(0.25) + a * m * q * q;
  };
  auto p_minus = [&](T m) {
    const T q = m * m - T(1);
    return (m - T(1)) * (m - T(1)) * (T(2) + m) * T(0.25) - a * m * q * q;
  };
  const bool sl = !(fabs(ml) > T(1)), sr = !(fabs(mr) > T(1));
  if (sl && sr) {
    const T x2 = ml * ml, y2 = mr * mr, xy = ml * mr;
    const T s2 = x2 + xy + y2;
    const T s4 = x2 * x2 + x2 * xy + xy * xy + xy * y2 + y2 * y2;
    return (ml - mr) * (T(0.75) - T(0.25) * s2 + a * (s4 - T(2) * s2 + T(1)));
  }
  if (!sl) {                                        // P+(ml) is 1 or 0
    if (ml > T(0)) return sr ? p_minus(mr) : (mr < T(0) ? T(1) : T(0));
    return sr ? -p_plus(mr) : (mr < T(0) ? T(0) : T(-1));
  }
  return mr < T(0) ? p_plus(ml) : -p_minus(ml);     // P-(mr) is 1 or 0
}

// MUSCL (kappa = 1/3, minmod) or first-order states at the face between
// points 1 and 2 of v[0..3], face thermodynamics, then AUSM+.
// v[t][0..4] = rho,u,v,w,p ; v[t][5+l] = Y_l.  F receives n_var values.
template <typename T, int NS>
__device__ __forceinline__ void face_inviscid(const ChemParams &C, const T *rec, const T (&v)[4][5 + SpecCount<NS>::kArr],
                                              const T k[3], T *F) {
  constexpr int A = SpecCount<NS>::kArr;
  constexpr int NV = 5 + A;
  const int ns = SpecCount<NS>::n(C);
  const int nv = 5 + ns;
  T L[NV], R[NV];
  if (C.reconstruction == 2) {
#pragma unroll
    for (int l = 0; l < NV; ++l) {
      if (l < nv) {
        const T d_i = v[1][l] - v[0][l];
        const T d_i1 = v[2][l] - v[1][l];
        const T d_i2 = v[3][l] - v[2][l];
        const T m1 = minmod(d_i, d_i1);
        const T m2 = minmod(d_i1, d_i2);
        // minmod is symmetric: ((1-k) mm(a,b) + (1+k) mm(b,a)) / 4 = mm(a,b) / 2
        L[l] = v[1][l] + T(0.5) * m1;
        R[l] = v[2][l] - T(0.5) * m2;
      }
    }
  } else {
#pragma unroll
    for (int l = 0; l < NV; ++l)
      if (l < nv) L[l] = v[1][l], R[l] = v[2][l];
  }
  // L[4], R[4] hold the gauge pressure p - p_ref (p_ref = 0 in FP64)
  const T pref = T(C.p_ref);
  const T pl = L[4] + pref, pr = R[4] + pref;
  // el, er: total enthalpy per unit mass, (rho E + p) / rho; c2l, c2r: gamma p / rho
  T el = T(0.5) * (L[1] * L[1] + L[2] * L[2] + L[3] * L[3]);
  T er = T(0.5) * (R[1] * R[1] + R[2] * R[2] + R[3] * R[3]);
  T c2l, c2r;
  if (NS == 0 || (NS < 0 && ns == 0)) {
    c2l = fdiv(T(kGammaAir) * pl, L[0]);
    c2r = fdiv(T(kGammaAir) * pr, R[0]);
    el += c2l * T(1.0 / (kGammaAir - 1));
    er += c2r * T(1.0 / (kGammaAir - 1));
  } else {
    const SpecTables<T> &S = tab<T>(C);
    T gas_l = 0, gas_r = 0;  // R_u / W
#pragma unroll
    for (int l = 0; l < A; ++l)
      if (l < ns) gas_l += L[5 + l] * S.cv_shift[l], gas_r += R[5 + l] * S.cv_shift[l];
    const T t_l = fdiv(pl, L[0] * gas_l);
    const T t_r = fdiv(pr, R[0] * gas_r);
    T xl[6], xr[6];
    const int rl = common_range(S, t_l), rr = common_range(S, t_r);
    if (rl == rr && rl >= 0) {  // one load of each record serves both states
      const T *base = rec + rl * kRecLen;
#pragma unroll
      for (int q = 0; q < 6; ++q) xl[q] = xr[q] = T(0);
#pragma unroll
      for (int l = 0; l < A; ++l) {
        if (l < ns) {
          T x[6];
          load_rec<T>(base + kRecRanges * kRecLen * l, x);
#pragma unroll
          for (int q = 0; q < 6; ++q) xl[q] += L[5 + l] * x[q], xr[q] += R[5 + l] * x[q];
        }
      }
    } else {
      nasa_mix<T, NS>(C, rec, t_l, -1, L + 5, xl);
      nasa_mix<T, NS>(C, rec, t_r, -1, R + 5, xr);
    }
    const T cpl = poly_cp(xl, t_l), cpr = poly_cp(xr, t_r);
    el += poly_h(xl, t_l);
    er += poly_h(xr, t_r);
    c2l = fdiv(cpl, cpl - gas_l) * gas_l * t_l;
    c2r = fdiv(cpr, cpr - gas_r) * gas_r * t_r;
  }
  const T alpha = T(3.0 / 16.0);
  const T k1 = k[0], k2 = k[1], k3 = k[2];
  T gk, igk;
  length_and_reciprocal(k1 * k1 + k2 * k2 + k3 * k3, gk, igk);
  const T ul = (k1 * L[1] + k2 * L[2] + k3 * L[3]) * igk;
  const T ur = (k1 * R[1] + k2 * R[2] + k3 * R[3]) * igk;
  const T rho_l = L[0], rho_r = R[0];
  const T c = T(0.5) * (fsqrt(c2l) + fsqrt(c2r));
  const T ic = frcp(c);
  const T mach_l = ul * ic, mach_r = ur * ic;
  T mlp, mrn, plp, prn;
  if (fabs(mach_l) > T(1)) {
    mlp = T(0.5) * (mach_l + fabs(mach_l));
    plp = fdiv(mlp, mach_l);
  } else {
    const T a = (mach_l + T(1)) * (mach_l + T(1)) * T(0.25);
    const T b = (mach_l * mach_l - T(1)) * (mach_l * mach_l - T(1));
    mlp = a + T(0.125) * b;
    plp = a * (T(2) - mach_l) + alpha * mach_l * b;
  }
  if (fabs(mach_r) > T(1)) {
    mrn = T(0.5) * (mach_r - fabs(mach_r));
    prn = fdiv(mrn, mach_r);
  } else {
    const T a = (mach_r - T(1)) * (mach_r - T(1)) * T(0.25);
    const T b = (mach_r * mach_r - T(1)) * (mach_r * mach_r - T(1));
    mrn = -a - T(0.125) * b;
    prn = a * (T(2) + mach_r) - alpha * mach_r * b;
  }
  // pressure term of the momentum flux, less p_ref k: plp p'_l + prn p'_r
  // + p_ref (plp + prn - 1), the last factor evaluated without cancellation
  T p_coeff;
  if (C.p_ref == 0.0) {
    p_coeff = plp * pl + prn * pr;
  } else {
    p_coeff = plp * L[4] + prn * R[4] + pref * ausm_pressure_defect(mach_l, mach_r, alpha);
  }
  // interface Mach number M+(ml) + M-(mr); at low Mach both terms are near
  // +-3/8 and their FP32 sum loses ~5 bits, so the FP32 path uses the
  // cancellation-free form (the FP64 path keeps the reference's sum)
  T m_half = mlp + mrn;
  if (sizeof(T) == 4 && !(fabs(mach_l) > T(1)) && !(fabs(mach_r) > T(1))) {
    // M+(M) + M-(M) = M: M+(ml) + M-(mr) = mr + (ml - mr) [1/2 + (ml + mr)(1/4 + (ml^2 + mr^2 - 2)/8)]
    m_half = mach_r + (mach_l - mach_r) *
                          (T(0.5) + (mach_l + mach_r) * (T(0.25) + T(0.125) * (mach_l * mach_l + mach_r * mach_r - T(2))));
  }
  const T mach_pos = T(0.5) * (m_half + fabs(m_half));
  const T mach_neg = T(0.5) * (m_half - fabs(m_half));
  const T mass_flux_half = c * (rho_l * mach_pos + rho_r * mach_neg);
  const T coeff = mass_flux_half * gk;
  const bool up = mass_flux_half >= T(0);
  F[0] = coeff;
  F[1] = coeff * (up ? L[1] : R[1]) + p_coeff * k1;
  F[2] = coeff * (up ? L[2] : R[2]) + p_coeff * k2;
  F[3] = coeff * (up ? L[3] : R[3]) + p_coeff * k3;
  F[4] = coeff * (up ? el : er);
#pragma unroll
  for (int l = 0; l < A; ++l)
    if (l < ns) F[5 + l] = coeff * (up ? L[5 + l] : R[5 + l]);
}

}  // namespace ccb
