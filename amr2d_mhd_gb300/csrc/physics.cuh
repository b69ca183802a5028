// Device physics of the per-face update: slope limiters, WENO weights, MHD
// wave speeds and the Riemann solvers.  Templated on the arithmetic type T.
// The double instantiation is compiled without FMA contraction and evaluates
// every expression in the reference's order, so it reproduces the reference
// bit for bit; the float instantiation is the FP32 bulk path.  Divisions and
// square roots go through the arithmetic M (softfp.cuh): the type's operators,
// or for double the same results off the FP64 pipe.
#pragma once

#include "amr_common.h"
#include "softfp.cuh"

namespace amr {

// defs.hpp:110-111 macros and std::min / std::max (they differ for equal and
// NaN arguments; each call site uses the form of the reference)
template <typename T> __device__ __forceinline__ T mmin(T a, T b) { return a < b ? a : b; }
template <typename T> __device__ __forceinline__ T mmax(T a, T b) { return a > b ? a : b; }
template <typename T> __device__ __forceinline__ T smin(T a, T b) { return b < a ? b : a; }
template <typename T> __device__ __forceinline__ T smax(T a, T b) { return a < b ? b : a; }
template <typename T> __device__ __forceinline__ T sgn(T v) { return v > T(0) ? T(1) : (v < T(0) ? T(-1) : T(0)); }
template <typename T> __device__ __forceinline__ T eps_of();
template <> __device__ __forceinline__ double eps_of<double>() { return 1.0E-15; }
// The FP32 bulk path keeps the FP64 scheme's epsilon (representable in
// float): defs.hpp:20 would switch to 1e-6 in a float build, which changes
// the WENO weights and limiter ratios, i.e. the scheme, not just the rounding.
template <> __device__ __forceinline__ float eps_of<float>() { return 1.0E-15f; }

// Classification of a value from its bit pattern in the integer pipe: the
// same predicates as isfinite / == 0 / isnan, which would take slots of the
// FP64 pipe (on GB300 2 per SM per clock) in the FP64-bound face kernel.
__device__ __forceinline__ bool bits_finite(double x) {
  return (__double_as_longlong(x) & 0x7ff0000000000000LL) != 0x7ff0000000000000LL;
}
__device__ __forceinline__ bool bits_finite(float x) { return (__float_as_uint(x) & 0x7f800000u) != 0x7f800000u; }
__device__ __forceinline__ bool bits_zero(double x) {
  return (static_cast<unsigned long long>(__double_as_longlong(x)) << 1) == 0ull;
}
__device__ __forceinline__ bool bits_zero(float x) { return (__float_as_uint(x) << 1) == 0u; }
__device__ __forceinline__ bool bits_nan(double x) {
  return (__double_as_longlong(x) & 0x7fffffffffffffffLL) > 0x7ff0000000000000LL;
}
__device__ __forceinline__ bool bits_nan(float x) { return (__float_as_uint(x) & 0x7fffffffu) > 0x7f800000u; }

// sgn() of a double from its bits
template <> __device__ __forceinline__ double sgn<double>(double v) {
  return bits_zero(v) || bits_nan(v) ? 0.0 : (__double2hiint(v) < 0 ? -1.0 : 1.0);
}

// slopelimiter.cpp:14-18 and :23-27, max(0, min(1, r)) and max(0, min(2r,
// (1+r)/2, 2)) with the macros of defs.hpp.  The Soft forms give the same
// bits: a negative r gives +0 and -0 gives -0; the rest are comparisons of
// values that are not negative.
template <typename T>
__device__ __forceinline__ T minmod_of(Native<T> &, T r) { return mmax(T(0), mmin(T(1), r)); }
__device__ __forceinline__ double minmod_of(Soft &m, double r) {
  const double c = m.least(r, 1.0);
  return __double2hiint(r) < 0 ? (m.nonzero(r) ? 0.0 : r) : c;
}
// FP32 faces: single instructions for the comparisons
__device__ __forceinline__ float minmod_of(Quick &, float r) { return bits_nan(r) ? r : fmaxf(0.f, fminf(1.f, r)); }
__device__ __forceinline__ float mc_of(Quick &, float r) {
  return fmaxf(0.f, fminf(fminf(2.f * r, 0.5f + 0.5f * r), 2.f));
}
template <typename T>
__device__ __forceinline__ T mc_of(Native<T> &, T r) {
  const T a = T(2) * r, b = T(0.5) * (T(1) + r);
  return mmax(T(0), mmin(mmin(a, b), T(2)));
}
__device__ __forceinline__ double mc_of(Soft &m, double r) {
  const double c = m.least(m.least(m.twice(r), m.half(1.0 + fabs(r))), 2.0);
  return __double2hiint(r) < 0 ? (m.nonzero(r) ? 0.0 : r) : c;
}

// slopelimiter.cpp:6-54
template <typename T, class M>
__device__ __forceinline__ T slope_limiter(M &m, int lim, T r, T eta) {
  const T E = eps_of<T>();
  switch (lim) {
    case LIM_1ST: return T(0);
    case LIM_NOSL: return r;
    case LIM_MINMOD: return minmod_of(m, r);
    case LIM_VANLEER: return m.div(fabs(r) + r, T(1) + fabs(r));
    case LIM_SUPERBEE: {
      T a = T(2) * r;
      T b = mmin(a, T(1));
      a = mmin(r, T(2));
      T c = mmax(a, b);
      return mmax(T(0), c);
    }
    case LIM_MC: return mc_of(m, r);
    case LIM_KOREN: {
      T a = m.template by<3>(T(1) + T(2) * r);
      T b = mmin(a, T(2));
      a = T(2) * r;
      T c = mmin(a, b);
      return mmax(T(0), c);
    }
    case LIM_CADA3RD: {
      const T third = m.template by<3>(T(2) + r);
      T a = mmin(T(2) * r, third);
      T b = mmin(a, T(1.6));
      T ph = mmax(T(-0.5) * r, b);
      a = mmin(third, ph);
      ph = mmax(T(0), a);
      if (eta <= T(1) - E) return third;
      if (eta >= T(1) + E) return ph;
      const T w = m.div(eta - T(1), E);
      return T(0.5) * (m.template by<3>((T(1) - w) * (T(2) + r)) + (T(1) + w) * ph);
    }
    default: return T(0);
  }
}

// The limiter ratio num/den (celledges.cpp:38,41), skipping the division when
// the limiter's value does not need it: num = +-0 gives r = +-0 exactly (sign
// rule of IEEE division), and for minmod, MC, Superbee and Koren every
// negative r gives phi = +0, so any negative stand-in does; "1st" ignores r.
// FP32 faces: a difference plus 1e-15 is zero or a normal number
__device__ __forceinline__ float limiter_ratio(Quick &m, int, float num, float den) { return m.ratio(num, den); }
// FP64 faces: always the division, so that those of a face's variables overlap
// (a branch around each puts them one after the other: KH 256 blocks 90 against
// 79 us, 196-block rotor, with uniform regions a branch could skip, 109 against
// 95, one warp alone 26.7 against 21.7)
__device__ __forceinline__ double limiter_ratio(Soft &m, int lim, double num, double den) {
  return lim == LIM_1ST ? 0.0 : m.div(num, den);
}
template <typename T, class M>
__device__ __forceinline__ T limiter_ratio(M &m, int lim, T num, T den) {
  if (lim == LIM_1ST) return T(0);
  if (!bits_zero(den) && bits_finite(den) && bits_finite(num)) {
    const bool neg = signbit(num) != signbit(den);
    if (bits_zero(num)) return neg ? T(-0.0) : T(0.0);
    if (neg && (lim == LIM_MINMOD || lim == LIM_MC || lim == LIM_SUPERBEE || lim == LIM_KOREN)) return T(-1);
  }
  return m.div(num, den);
}

// celledges.cpp:38-43 for one variable of one face.  dA = W[i]-W[i-1],
// dB = W[i+1]-W[i], dC = W[i+2]-W[i+1] around the face i+1/2; returns the
// left state wxL[i] and right state wxR[i+1].  inv2 = 1/(dx*dx) for Cada3rd.
template <typename T, class M>
__device__ __forceinline__ void muscl_face(M &m, int lim, T wi, T wip, T dA, T dB, T dC, T h,
                                           T &left, T &right) {
  const T E = eps_of<T>();
  T etaL = T(0), etaR = T(0);
  if (lim == LIM_CADA3RD) {
    etaL = m.div(dB * dB + dA * dA, (T(1) * h) * (T(1) * h));
    etaR = m.div(dC * dC + dB * dB, (T(1) * h) * (T(1) * h));
  }
  T r = limiter_ratio(m, lim, dB, dA + E);
  T phi = slope_limiter<T>(m, lim, r, etaL);
  left = wi + m.half(phi) * dA;
  r = limiter_ratio(m, lim, dB, dC + E);
  phi = slope_limiter<T>(m, lim, r, etaR);
  right = wip - m.half(phi) * dC;
}

// WENO2D_primvar.cpp:43-87: the two WENO3 face values of a cell with
// neighbours wm, wp.  vR is the value at its left face (wxR), vL at its right
// face (wxL).
template <typename T, class M>
__device__ __forceinline__ void weno3_cell(M &m, T wm, T w, T wp, T &vL, T &vR) {
  const T e = eps_of<T>();
  {
    T p0n = m.half(wm) + m.half(w), p1n = T(1.5) * w - m.half(wp);
    T B0n = (w - wm) * (w - wm), B1n = (wp - w) * (wp - w);
    T d0n = T(2.) / T(3.), d1n = T(1.) / T(3.);
    T a0n = m.ratio(d0n, (e + B0n) * (e + B0n)), a1n = m.ratio(d1n, (e + B1n) * (e + B1n));
    T asn = a0n + a1n;
    T w0n = m.div(a0n, asn), w1n = m.div(a1n, asn);
    vR = w0n * p0n + w1n * p1n;
  }
  {
    T p0p = T(1.5) * w - m.half(wm), p1p = m.half(wp) + m.half(w);
    T B0p = (w - wm) * (w - wm), B1p = (wp - w) * (wp - w);
    T d0p = T(1.) / T(3.), d1p = T(2.) / T(3.);
    T a0p = m.ratio(d0p, (e + B0p) * (e + B0p)), a1p = m.ratio(d1p, (e + B1p) * (e + B1p));
    T asp = a0p + a1p;
    T w0p = m.div(a0p, asp), w1p = m.div(a1p, asp);
    vL = w0p * p0p + w1p * p1p;
  }
}

// WENO2D_primvar.cpp:140-193 (beta_1 takes the -2 neighbour, :145,174).
// RIGHT selects wxR (value at the cell's left face) or wxL.
template <typename T, bool RIGHT, class M>
__device__ __forceinline__ T weno5_cell(M &m, T wmm, T wm, T w, T wp, T wpp) {
  const T e = eps_of<T>();
  const T c13 = T(13.) / T(12.);
  T t, t2;
  if (RIGHT) {
    T p0n = m.template by<6>(-wmm + T(5) * wm + m.twice(w));
    T p1n = m.template by<6>(m.twice(wm) + T(5) * w - wp);
    T p2n = m.template by<6>(T(11) * w - T(7) * wp + m.twice(wpp));
    t = wmm - m.twice(wm) + w; t2 = wmm - m.quad(wm) + T(3) * w;
    T B0 = c13 * (t * t) + m.quarter(t2 * t2);
    t = wmm - m.twice(w) + wp; t2 = wm - wp;
    T B1 = c13 * (t * t) + m.quarter(t2 * t2);
    t = w - m.twice(wp) + wpp; t2 = T(3) * w - m.quad(wp) + wpp;
    T B2 = c13 * (t * t) + m.quarter(t2 * t2);
    T d0 = T(1.) / T(10.), d1 = T(6.) / T(10.), d2 = T(3.) / T(10.);
    T a0 = m.ratio(d0, (e + B0) * (e + B0)), a1 = m.ratio(d1, (e + B1) * (e + B1)), a2 = m.ratio(d2, (e + B2) * (e + B2));
    T as = a0 + a1 + a2;
    T w0 = m.div(a0, as), w1 = m.div(a1, as), w2 = m.div(a2, as);
    return w0 * p0n + w1 * p1n + w2 * p2n;
  } else {
    T p0p = m.template by<6>(m.twice(wmm) - T(7) * wm + T(11) * w);
    T p1p = m.template by<6>(-wm + T(5) * w + m.twice(wp));
    T p2p = m.template by<6>(m.twice(w) + T(5) * wp - wpp);
    t = wmm - m.twice(wm) + w; t2 = wmm - m.quad(wm) + T(3) * w;
    T B0 = c13 * (t * t) + m.quarter(t2 * t2);
    t = wmm - m.twice(w) + wp; t2 = wm - wp;
    T B1 = c13 * (t * t) + m.quarter(t2 * t2);
    t = w - m.twice(wp) + wpp; t2 = T(3) * w - m.quad(wp) + wpp;
    T B2 = c13 * (t * t) + m.quarter(t2 * t2);
    T d0 = T(3.) / T(10.), d1 = T(6.) / T(10.), d2 = T(1.) / T(10.);
    T a0 = m.ratio(d0, (e + B0) * (e + B0)), a1 = m.ratio(d1, (e + B1) * (e + B1)), a2 = m.ratio(d2, (e + B2) * (e + B2));
    T as = a0 + a1 + a2;
    T w0 = m.div(a0, as), w1 = m.div(a1, as), w2 = m.div(a2, as);
    return w0 * p0p + w1 * p1p + w2 * p2p;
  }
}

// misc.cpp:71-79, fast magnetosonic speed along component `norm`
template <typename T, class M>
__device__ __forceinline__ T fast_speed(M &m, const T *w, T gamma, int norm) {
  T ca = m.root(m.div(w[5] * w[5] + w[6] * w[6] + w[7] * w[7], w[0]));
  T a = m.root(m.div(gamma * w[4], w[0]));
  T can = m.root(m.div(w[norm] * w[norm], w[0]));
  T i0 = (ca * ca) + (a * a);
  T i1 = (ca * ca) - (a * a);
  return m.root(m.half(i0 + m.root(i1 * i1 + m.quad(a * a) * ((ca * ca) - (can * can)))));
}

// FP32 faces: the squares of the sound and Alfven speeds as they are, without
// the roots that the FP64 path takes and squares again, and the transverse
// field's share as a sum instead of a difference (fewer roundings, and never
// negative).  A negative square is NaN, as its root is there: the trap for face
// states of negative pressure or density.
__device__ __forceinline__ float real_speed(float a2, float c2, float cf) {
  return fminf(a2, c2) < 0.f ? __int_as_float(0x7fffffff) : cf;
}
__device__ __forceinline__ float fast_speed_of(Quick &m, const float *w, float gamma) {
  const float ir = m.div(1.f, w[0]);
  const float t2 = (w[6] * w[6] + w[7] * w[7]) * ir, c2 = w[5] * w[5] * ir + t2, a2 = gamma * w[4] * ir;
  const float d = c2 - a2;
  return real_speed(a2, c2, m.root(0.5f * (c2 + a2 + m.root(d * d + 4.f * a2 * t2))));
}

// the same for norm 5 (x) and 6 (y), whose first two terms are the same values
template <typename T, class M>
__device__ __forceinline__ void fast_speeds(M &m, const T *w, T gamma, T *cf) {
  const T ca = m.root(m.div(w[5] * w[5] + w[6] * w[6] + w[7] * w[7], w[0]));
  const T a = m.root(m.div(gamma * w[4], w[0]));
  const T i0 = (ca * ca) + (a * a), i1 = (ca * ca) - (a * a);
#pragma unroll
  for (int q = 0; q < 2; q++) {
    const T can = m.root(m.div(w[5 + q] * w[5 + q], w[0]));
    cf[q] = m.root(m.half(i0 + m.root(i1 * i1 + m.quad(a * a) * ((ca * ca) - (can * can)))));
  }
}

// FP32: as fast_speed_of, with one reciprocal for both.  Error against 64 bits
// over rotor, blast, low-beta and KH states: rms 3.8e-8, at most 1.9e-7 (the
// form with the roots, each quotient correctly rounded: 4.8e-8 and 2.1e-6, as its
// difference c_a^2 - c_n^2 cancels).
__device__ __forceinline__ void fast_speeds_of(Native<float> &m, const float *w, float gamma, float *cf) {
  const float ir = 1.f / w[0];
  const float bx = w[5] * w[5] * ir, by = w[6] * w[6] * ir, bz = w[7] * w[7] * ir, a2 = gamma * w[4] * ir;
  const float c2 = bx + by + bz, d = c2 - a2;
  cf[0] = real_speed(a2, c2, m.root(0.5f * (c2 + a2 + m.root(d * d + 4.f * a2 * (by + bz)))));
  cf[1] = real_speed(a2, c2, m.root(0.5f * (c2 + a2 + m.root(d * d + 4.f * a2 * (bx + bz)))));
}
template <class M>
__device__ __forceinline__ void fast_speeds_of(M &m, const double *w, double gamma, double *cf) {
  fast_speeds<double>(m, w, gamma, cf);
}

// riemannS.cpp:59-108 for one side: the energy, the total pressure and the
// fast speed; then, from those, the enthalpy, conserved state and physical flux
template <typename T>
struct Side {
  T q[8], F[8], H, pt, cf, e;
};

template <typename T, class M>
__device__ __forceinline__ void side_scalars(M &m, const T *w, T gamma, T &cf, T &pt, T &e) {
  cf = fast_speed<T>(m, w, gamma, 5);
  const T b2 = w[5] * w[5] + w[6] * w[6] + w[7] * w[7];
  // the reference's 0.5*b2/rho: halving is exact, so it is half of the b2/rho
  // the fast speed has
  e = m.div(w[4], w[0] * (gamma - T(1))) + m.half(w[1] * w[1] + w[2] * w[2] + w[3] * w[3]) + m.half(m.div(b2, w[0]));
  e = e * w[0];
  pt = w[4] + m.half(b2);
}

// FP32 faces: the energy as p/(gamma - 1) + rho v^2/2 + B^2/2, without the
// reference's detour over the energy per mass (fewer roundings)
template <typename T>
__device__ __forceinline__ void side_scalars(Quick &m, const float *w, float gamma, float &cf, float &pt, float &e) {
  const float b2 = w[5] * w[5] + w[6] * w[6] + w[7] * w[7];
  cf = fast_speed_of(m, w, gamma);
  e = m.div(w[4], gamma - 1.f) + 0.5f * (w[0] * (w[1] * w[1] + w[2] * w[2] + w[3] * w[3]) + b2);
  pt = w[4] + 0.5f * b2;
}

template <typename T, class M>
__device__ __forceinline__ T enthalpy(M &m, const T *w, T e) {
  return m.div(e + w[4] + m.half(w[5] * w[5] + w[6] * w[6] + w[7] * w[7]), w[0]);
}

template <typename T>
__device__ __forceinline__ void side_flux(const T *w, T pt, T e, T H, T *q, T *F) {
  const T vn = w[1], Bn = w[5];
  q[0] = w[0]; q[1] = w[0] * w[1]; q[2] = w[0] * w[2]; q[3] = w[0] * w[3];
  q[4] = e; q[5] = w[5]; q[6] = w[6]; q[7] = w[7];
  F[0] = w[0] * vn;
  F[1] = w[0] * vn * w[1] + pt - Bn * w[5];
  F[2] = w[0] * vn * w[2] - Bn * w[6];
  F[3] = w[0] * vn * w[3] - Bn * w[7];
  F[4] = w[0] * vn * H - Bn * (w[1] * w[5] + w[2] * w[6] + w[3] * w[7]);
  F[5] = vn * w[5] - Bn * w[1];
  F[6] = vn * w[6] - Bn * w[2];
  F[7] = vn * w[7] - Bn * w[3];
}

template <typename T, class M>
__device__ __forceinline__ void side_state(M &m, const T *w, T gamma, Side<T> &s) {
  side_scalars<T>(m, w, gamma, s.cf, s.pt, s.e);
  s.H = enthalpy<T>(m, w, s.e);
  side_flux<T>(w, s.pt, s.e, s.H, s.q, s.F);
}

// misc.cpp:95-140 Roe averages (sqrt(rhoL + sqrt(rhoR)) denominator as in
// the reference, :98,100) and the outer eigenvalues lambda_0 / lambda_6
template <typename T, class M>
__device__ __forceinline__ void roe_outer(M &m, const T *wL, const T *wR, T HL, T HR, T gamma, T &vx,
                                          T &l0, T &l6) {
  T v[3], B[3];
  const T sl = m.root(wL[0]), sr = m.root(wR[0]);
  const T sd = m.root(wL[0] + sr);
#pragma unroll
  for (int i = 0; i < 3; i++) {
    v[i] = m.div(sl * wL[i + 1] + sr * wR[i + 1], sd);
    B[i] = m.div(sl * wL[i + 5] + sr * wR[i + 5], sd);
  }
  const T RT = m.root(m.div(wR[0], wL[0]));
  const T d = m.root(wR[0] * wL[0]);
  const T d6 = wL[6] - wR[6], d7 = wL[7] - wR[7];
  const T Xfac = m.div(T(0.5) * (d6 * d6 + d7 * d7), sl + sr);
  const T Yfac = m.div(T(0.5) * (wL[0] + wR[0]), d);
  const T h = m.div(HL + RT * HR, T(1) + RT);
  const T vsq = v[0] * v[0] + v[1] * v[1] + v[2] * v[2];
  const T btsq = B[1] * B[1] + B[2] * B[2];
  const T bt_starsq = (gamma - T(1.) - (gamma - T(2)) * Yfac) * btsq;
  const T vaxsq = m.div(B[0] * B[0], d);
  const T hp = h - (vaxsq + m.div(btsq, d));
  T twid_asq = ((gamma - T(1.)) * (hp - T(0.5) * vsq) - (gamma - T(2.)) * Xfac);
  twid_asq = mmax(twid_asq, eps_of<T>());
  const T ct2 = m.div(bt_starsq, d);
  const T tsum = vaxsq + ct2 + twid_asq;
  const T tdif = vaxsq + ct2 - twid_asq;
  const T cf2_cs2 = m.root(tdif * tdif + T(4.) * twid_asq * ct2);
  const T cfsq = T(0.5) * (tsum + cf2_cs2);
  const T cfast = m.root(cfsq);
  vx = v[0];
  l0 = v[0] - cfast;
  l6 = v[0] + cfast;
}

// riemannS.cpp:58-116
template <typename T, class M>
__device__ __forceinline__ int flux_rusa(M &m, const T *wL, const T *wR, T gamma, T *f) {
  Side<T> L, R;
  side_state<T>(m, wL, gamma, L);
  side_state<T>(m, wR, gamma, R);
  const T a = L.cf + fabs(wL[1]), b = R.cf + fabs(wR[1]);
  const T im = m.std_most(a, b);
#pragma unroll
  for (int k = 0; k < 8; k++) f[k] = m.half(L.F[k] + R.F[k]) - m.half(im) * (R.q[k] - L.q[k]);
  return 0;
}

// riemannS.cpp:118-189
template <typename T, class M>
__device__ __forceinline__ int flux_hlle(M &m, const T *wL, const T *wR, T gamma, T *f) {
  Side<T> L, R;
  side_state<T>(m, wL, gamma, L);
  side_state<T>(m, wR, gamma, R);
  T vx, l0, l6;
  roe_outer<T>(m, wL, wR, L.H, R.H, gamma, vx, l0, l6);
  T SL = smin(wL[1] - L.cf, l0);
  SL = mmin(SL, T(0.));
  T SR = smax(wR[1] + R.cf, l6);
  SR = mmax(SR, T(0.));
#pragma unroll
  for (int k = 0; k < 8; k++) f[k] = m.div(SR * L.F[k] - SL * R.F[k] + SL * SR * (R.q[k] - L.q[k]), SR - SL);
  return 0;
}

// riemannS.cpp:192-295 (Linde 1998 with the heuristic alpha)
template <typename T, class M>
__device__ __forceinline__ int flux_hllc(M &m, const T *wL, const T *wR, T gamma, T *f) {
  Side<T> L, R;
  side_state<T>(m, wL, gamma, L);
  side_state<T>(m, wR, gamma, R);
  T vx, l0, l6;
  roe_outer<T>(m, wL, wR, L.H, R.H, gamma, vx, l0, l6);
  const T SL = smin(wL[1] - L.cf, l0);
  const T SR = smax(wR[1] + R.cf, l6);
  const T SM = vx;
  T s1 = T(0.), s2 = T(0.);
#pragma unroll
  for (int k = 0; k < 8; k++) s1 += fabs(R.q[k] - L.q[k]);
#pragma unroll
  for (int k = 0; k < 8; k++) s2 += fabs((R.F[k] - L.F[k]) - vx * (R.q[k] - L.q[k]));
  const T interm = T(1.) - m.div(s2, s1 + eps_of<T>());
  const T alpha = mmax(T(0.), interm);
  if (alpha > T(1) || alpha < T(0) || isnan(alpha)) return DERR_HLLC;
  if (SR - SL == T(0)) return DERR_HLLC;
  int br = -1;
  if (SL > T(0.)) br = 0;
  else if (SL <= T(0.) && SM >= T(0.)) br = 1;
  else if (SM <= T(0.) && SR >= T(0.)) br = 2;
  else if (SR < T(0.)) br = 3;
#pragma unroll
  for (int k = 0; k < 8; k++) {
    T v = T(0);
    if (br == 0) v = L.F[k];
    else if (br == 1)
      v = m.div(SL * ((T(1) - alpha) * SR + alpha * vx), SR - SL) * (R.q[k] - L.q[k]) -
          m.div(SL, SR - SL) * R.F[k] + m.div(SR, SR - SL) * L.F[k];
    else if (br == 2)
      v = m.div(SR * ((T(1) - alpha) * SL + alpha * vx), SR - SL) * (R.q[k] - L.q[k]) -
          m.div(SL, SR - SL) * R.F[k] + m.div(SR, SR - SL) * L.F[k];
    else if (br == 3) v = R.F[k];
    f[k] = v;
  }
  return 0;
}

template <typename T>
__device__ __forceinline__ T dot13_57(T a1, T a2, T a3, T a5, T a6, T a7) {  // misc.cpp:51-61
  T s = T(0.);
  s += a1 * a5;
  s += a2 * a6;
  s += a3 * a7;
  return s;
}

// riemannS.cpp:397-549 (Miyoshi & Kusano).  The wave fan selects one of six
// regions; both star states and the waves are evaluated, then one side's
// state, flux and star state are picked and the region's flux assembled once,
// with the reference's operations in the reference's order.  (Evaluating
// every region a warp's faces fall into, as a switch over them does, and both
// sides' fluxes takes 40 % more FP64 instructions on the rotor.)
template <typename T, class M>
__device__ __forceinline__ int flux_hlld(M &m, const T *wL, const T *wR, T gamma, T *f) {
  T cfL, ptL, eL, cfR, ptR, eR;
  side_scalars<T>(m, wL, gamma, cfL, ptL, eL);
  side_scalars<T>(m, wR, gamma, cfR, ptR, eR);
  const T vnL = wL[1], vnR = wR[1];
  const T cf = m.std_most(cfL, cfR);
  const T SL = smin(vnL, vnR) - cf;
  const T SR = smax(vnL, vnR) + cf;
  const T mL = (SL - vnL) * wL[0], mR = (SR - vnR) * wR[0];
  const T SM = m.div(mR * vnR - mL * vnL - ptR + ptL, mR - mL);
  const T pts = m.div(mR * ptL - mL * ptR + wL[0] * wR[0] * (SR - vnR) * (SL - vnL) * (vnR - vnL), mR - mL);
  // left and right * states (:467-497)
  auto star = [&](const T *w, T S, T e, T pt, T ms, T &r, T &v, T &wz, T &by, T &bz, T &d, T &es) {
    r = m.div(ms, S - SM);   // w0 * (S - vn) is (S - vn) * w0
    const T den = ms * (S - SM) - w[5] * w[5];
    if (m.nonzero(den)) {
      const T k = m.div(SM - w[1], den);
      const T h = m.div(w[0] * ((S - w[1]) * (S - w[1])) - w[5] * w[5], den);
      v = w[2] - w[5] * w[6] * k;
      wz = w[3] - w[5] * w[7] * k;
      by = w[6] * h;
      bz = w[7] * h;
    } else {
      v = w[2]; wz = w[3]; by = T(0.); bz = T(0.);
    }
    d = dot13_57(SM, v, wz, w[5], by, bz);
    es = m.div((S - w[1]) * e - pt * w[1] + pts * SM +
                   w[5] * (dot13_57(w[1], w[2], w[3], w[5], w[6], w[7]) - d),
               S - SM);
  };
  T rLs, vLs, wzLs, byLs, bzLs, dLs, eLs, rRs, vRs, wzRs, byRs, bzRs, dRs, eRs;
  star(wL, SL, eL, ptL, mL, rLs, vLs, wzLs, byLs, bzLs, dLs, eLs);
  star(wR, SR, eR, ptR, mR, rRs, vRs, wzRs, byRs, bzRs, dRs, eRs);
  const T sLs = m.root(rLs), sRs = m.root(rRs);
  const T SLs = SM - m.div(fabs(wL[5]), sLs);
  const T SRs = SM + m.div(fabs(wR[5]), sRs);
  int br = -1;
  if (m.positive(SL)) br = 0;
  else if (m.nonpositive(SL) && m.nonnegative(SLs)) br = 1;
  else if (m.nonpositive(SLs) && m.nonnegative(SM)) br = 2;
  else if (m.nonpositive(SM) && m.nonnegative(SRs)) br = 3;
  else if (m.nonpositive(SRs) && m.nonnegative(SR)) br = 4;
  else if (m.negative(SR)) br = 5;
  const bool left = br <= 2, mid = br == 2 || br == 3, fan = mid || br == 1 || br == 4;
  // the picked side: its state, flux, star state and waves
  T w[8], q[8], F[8];
#pragma unroll
  for (int k = 0; k < 8; k++) w[k] = left ? wL[k] : wR[k];
  const T e = left ? eL : eR;
  side_flux<T>(w, left ? ptL : ptR, e, enthalpy<T>(m, w, e), q, F);
  const T S = left ? SL : SR, Ss = left ? SLs : SRs, ss = left ? sLs : sRs;
  const T rs = left ? rLs : rRs, es = left ? eLs : eRs;
  const T vs = left ? vLs : vRs, wzs = left ? wzLs : wzRs, bys = left ? byLs : byRs, bzs = left ? bzLs : bzRs;
  // conserved * state (w2u, misc.cpp:82-92; energy replaced, :524,527)
  const T qs[8] = {rs, rs * SM, rs * vs, rs * wzs, es, w[5], bys, bzs};
  T x[8];   // the state the wave Sx multiplies: the ** state (:501-519) or the * state
  T Sx = S;
#pragma unroll
  for (int k = 0; k < 8; k++) x[k] = qs[k];
  if (mid) {  // the right ** state is a copy of the left one (:517)
    const T sg = sgn(wL[5]), sum = sLs + sRs, rr = m.root(rLs * rRs);
    const T vss = m.div(sLs * vLs + sRs * vRs + (byRs - byLs) * sg, sum);
    const T wss = m.div(sLs * wzLs + sRs * wzRs + (bzRs - bzLs) * sg, sum);
    const T byss = m.div(sLs * byRs + sRs * byLs + rr * (vRs - vLs) * sg, sum);
    const T bzss = m.div(sLs * bzRs + sRs * bzLs + rr * (wzRs - wzLs) * sg, sum);
    const T dss = dot13_57(SM, vss, wss, wL[5], byss, bzss);
    const T de = ss * ((left ? dLs : dRs) - dss) * (left ? sg : sgn(wR[5]));
    x[0] = rLs; x[1] = rLs * SM; x[2] = rLs * vss; x[3] = rLs * wss;
    x[4] = es + (left ? -de : de); x[5] = wL[5]; x[6] = byss; x[7] = bzss;
    Sx = Ss;
  }
#pragma unroll
  for (int k = 0; k < 8; k++) {
    T v = F[k] + Sx * x[k];
    const T v2 = v - (Ss - S) * qs[k];
    v = (mid ? v2 : v) - S * q[k];
    f[k] = fan ? v : (br < 0 ? T(0) : F[k]);
  }
  return 0;
}

// riemannS.cpp:297-395: the hydrodynamic Roe solver (Toro's, "not suited
// for MHD"), which riemannS only reaches in the reference's configuration
// without a magnetic field (riemannS.cpp:39-40).  The normal is x (xnorm = 1,
// ynorm = 0, written out as the reference does; a field enters only the
// physical fluxes).  The reference's (gamma-1)/pow(a,2) is (gamma-1)/(a*a)
// here, the correctly rounded square; the C library's pow rounds a few in a
// thousand squares differently, so this solver matches the reference to a
// few ulp rather than bit for bit.
template <typename T, class M>
__device__ __forceinline__ int flux_roe(M &m, const T *wL, const T *wR, T gamma, T *flux) {
  const T xnorm = T(1.0), ynorm = T(0.0);
  const T vnL = wL[1] * xnorm + wL[2] * ynorm, BnL = wL[5] * xnorm + wL[6] * ynorm;
  T eL = (wL[4] / (wL[0] * (gamma - T(1)))) + T(0.5) * (wL[1] * wL[1] + wL[2] * wL[2] + wL[3] * wL[3]) +
         T(0.5) * (wL[5] * wL[5] + wL[6] * wL[6] + wL[7] * wL[7]) / wL[0];
  eL = eL * wL[0];
  const T HL = (eL + wL[4] + T(0.5) * (wL[5] * wL[5] + wL[6] * wL[6] + wL[7] * wL[7])) / wL[0];
  const T vnR = wR[1] * xnorm + wR[2] * ynorm, BnR = wR[5] * xnorm + wR[6] * ynorm;
  T eR = (wR[4] / (wR[0] * (gamma - T(1)))) + T(0.5) * (wR[1] * wR[1] + wR[2] * wR[2] + wR[3] * wR[3]) +
         T(0.5) * (wR[5] * wR[5] + wR[6] * wR[6] + wR[7] * wR[7]) / wR[0];
  eR = eR * wR[0];
  const T HR = (eR + wR[4] + T(0.5) * (wR[5] * wR[5] + wR[6] * wR[6] + wR[7] * wR[7])) / wR[0];
  const T qL[5] = {wL[0], wL[0] * wL[1], wL[0] * wL[2], wL[0] * wL[3], eL};
  const T qR[5] = {wR[0], wR[0] * wR[1], wR[0] * wR[2], wR[0] * wR[3], eR};
  // Roe averages, eigenvalues, right eigenvectors (rows K[j], columns 0..4;
  // the field columns are zero)
  const T RT = sqrt(wR[0] / wL[0]);
  const T u = (wL[1] + RT * wR[1]) / (T(1) + RT);
  const T v = (wL[2] + RT * wR[2]) / (T(1) + RT);
  const T w = (wL[3] + RT * wR[3]) / (T(1) + RT);
  const T H = (HL + RT * HR) / (T(1) + RT);
  const T a = sqrt((gamma - T(1)) * (H - T(0.5) * (u * u + v * v + w * w)));
  const T lambda[5] = {u - a, u, u, u, u + a};
  const T K[5][5] = {{T(1.), u - a, v, w, H - u * a},
                     {T(1.), u, v, w, T(0.5) * (u * u + v * v + w * w)},
                     {T(0.), T(0.), T(1.), T(0.), v},
                     {T(0.), T(0.), T(0.), T(1.), w},
                     {T(1.), u + a, v, w, H + u * a}};
  // wave strengths
  T alpha[5];
  alpha[2] = (qR[2] - qL[2]) - v * (qR[0] - qL[0]);
  alpha[3] = (qR[3] - qL[3]) - w * (qR[0] - qL[0]);
  const T du5bar = (qR[4] - qL[4]) - (alpha[2]) * v - (alpha[3]) * w;
  alpha[1] = ((gamma - T(1)) / (a * a)) * ((qR[0] - qL[0]) * (H - u * u) + u * (qR[1] - qL[1]) - du5bar);
  alpha[0] = T(0.5) * (T(1) / a) * ((qR[0] - qL[0]) * (u + a) - (qR[1] - qL[1]) - a * alpha[1]);
  alpha[4] = (qR[0] - qL[0]) - (alpha[0] + alpha[1]);
  // physical fluxes
  const T ptL = wL[4] + T(0.5) * (wL[5] * wL[5] + wL[6] * wL[6] + wL[7] * wL[7]);
  const T ptR = wR[4] + T(0.5) * (wR[5] * wR[5] + wR[6] * wR[6] + wR[7] * wR[7]);
  const T FL[8] = {wL[0] * vnL,
                   wL[0] * vnL * wL[1] + xnorm * ptL - BnL * wL[5],
                   wL[0] * vnL * wL[2] + ynorm * ptL - BnL * wL[6],
                   wL[0] * vnL * wL[3] - BnL * wL[7],
                   wL[0] * vnL * HL - BnL * (wL[1] * wL[5] + wL[2] * wL[6] + wL[3] * wL[7]),
                   vnL * wL[5] - BnL * wL[1],
                   vnL * wL[6] - BnL * wL[2],
                   vnL * wL[7] - BnL * wL[3]};
  const T FR[8] = {wR[0] * vnR,
                   wR[0] * vnR * wR[1] + xnorm * ptR - BnR * wR[5],
                   wR[0] * vnR * wR[2] + ynorm * ptR - BnR * wR[6],
                   wR[0] * vnR * wR[3] - BnR * wR[7],
                   wR[0] * vnR * HR - BnR * (wR[1] * wR[5] + wR[2] * wR[6] + wR[3] * wR[7]),
                   vnR * wR[5] - BnR * wR[1],
                   vnR * wR[6] - BnR * wR[2],
                   vnR * wR[7] - BnR * wR[3]};
#pragma unroll
  for (int k = 0; k < 8; k++) {
    T summ = T(0.);
#pragma unroll
    for (int j = 0; j < 5; j++) summ += alpha[j] * fabs(lambda[j]) * (k < 5 ? K[j][k] : T(0.));
    flux[k] = T(0.5) * (FL[k] + FR[k]) - T(0.5) * summ;
  }
  return 0;
}

template <int FLUX, typename T, class M>
__device__ __forceinline__ int riemann(M &m, const T *wL, const T *wR, T gamma, T *f) {
  if (FLUX == FLX_RUSA) return flux_rusa<T>(m, wL, wR, gamma, f);
  if (FLUX == FLX_HLLE) return flux_hlle<T>(m, wL, wR, gamma, f);
  if (FLUX == FLX_HLLC) return flux_hllc<T>(m, wL, wR, gamma, f);
  if (FLUX == FLX_ROE) return flux_roe<T>(m, wL, wR, gamma, f);
  return flux_hlld<T>(m, wL, wR, gamma, f);
}

}  // namespace amr
