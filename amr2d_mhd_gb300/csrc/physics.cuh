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

// slopelimiter.cpp:6-54
template <typename T, class M>
__device__ __forceinline__ T slope_limiter(M &m, int lim, T r, T eta) {
  const T E = eps_of<T>();
  switch (lim) {
    case LIM_1ST: return T(0);
    case LIM_NOSL: return r;
    case LIM_MINMOD: { T a = mmin(T(1), r); return mmax(T(0), a); }
    case LIM_VANLEER: return m.div(fabs(r) + r, T(1) + fabs(r));
    case LIM_SUPERBEE: {
      T a = T(2) * r;
      T b = mmin(a, T(1));
      a = mmin(r, T(2));
      T c = mmax(a, b);
      return mmax(T(0), c);
    }
    case LIM_MC: {
      T a = T(2) * r, b = T(0.5) * (T(1) + r);
      T c = mmin(a, b);
      a = mmin(c, T(2));
      return mmax(T(0), a);
    }
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
  T r = limiter_ratio<T>(m, lim, dB, dA + E);
  T phi = slope_limiter<T>(m, lim, r, etaL);
  left = wi + T(0.5) * phi * dA;
  r = limiter_ratio<T>(m, lim, dB, dC + E);
  phi = slope_limiter<T>(m, lim, r, etaR);
  right = wip - T(0.5) * phi * dC;
}

// WENO2D_primvar.cpp:43-87: the two WENO3 face values of a cell with
// neighbours wm, wp.  vR is the value at its left face (wxR), vL at its right
// face (wxL).
template <typename T, class M>
__device__ __forceinline__ void weno3_cell(M &m, T wm, T w, T wp, T &vL, T &vR) {
  const T e = eps_of<T>();
  {
    T p0n = T(0.5) * wm + T(0.5) * w, p1n = T(1.5) * w - T(0.5) * wp;
    T B0n = (w - wm) * (w - wm), B1n = (wp - w) * (wp - w);
    T d0n = T(2.) / T(3.), d1n = T(1.) / T(3.);
    T a0n = m.div(d0n, (e + B0n) * (e + B0n)), a1n = m.div(d1n, (e + B1n) * (e + B1n));
    T asn = a0n + a1n;
    T w0n = m.div(a0n, asn), w1n = m.div(a1n, asn);
    vR = w0n * p0n + w1n * p1n;
  }
  {
    T p0p = T(1.5) * w - T(0.5) * wm, p1p = T(0.5) * wp + T(0.5) * w;
    T B0p = (w - wm) * (w - wm), B1p = (wp - w) * (wp - w);
    T d0p = T(1.) / T(3.), d1p = T(2.) / T(3.);
    T a0p = m.div(d0p, (e + B0p) * (e + B0p)), a1p = m.div(d1p, (e + B1p) * (e + B1p));
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
  const T c13 = T(13.) / T(12.), c14 = T(1.) / T(4.);
  T t, t2;
  if (RIGHT) {
    T p0n = m.template by<6>(T(-1) * wmm + T(5) * wm + T(2) * w);
    T p1n = m.template by<6>(T(2) * wm + T(5) * w - wp);
    T p2n = m.template by<6>(T(11) * w - T(7) * wp + T(2) * wpp);
    t = wmm - T(2) * wm + w; t2 = wmm - T(4) * wm + T(3) * w;
    T B0 = c13 * (t * t) + c14 * (t2 * t2);
    t = wmm - T(2) * w + wp; t2 = wm - wp;
    T B1 = c13 * (t * t) + c14 * (t2 * t2);
    t = w - T(2) * wp + wpp; t2 = T(3) * w - T(4) * wp + wpp;
    T B2 = c13 * (t * t) + c14 * (t2 * t2);
    T d0 = T(1.) / T(10.), d1 = T(6.) / T(10.), d2 = T(3.) / T(10.);
    T a0 = m.div(d0, (e + B0) * (e + B0)), a1 = m.div(d1, (e + B1) * (e + B1)), a2 = m.div(d2, (e + B2) * (e + B2));
    T as = a0 + a1 + a2;
    T w0 = m.div(a0, as), w1 = m.div(a1, as), w2 = m.div(a2, as);
    return w0 * p0n + w1 * p1n + w2 * p2n;
  } else {
    T p0p = m.template by<6>(T(2) * wmm - T(7) * wm + T(11) * w);
    T p1p = m.template by<6>(T(-1) * wm + T(5) * w + T(2) * wp);
    T p2p = m.template by<6>(T(2) * w + T(5) * wp - wpp);
    t = wmm - T(2) * wm + w; t2 = wmm - T(4) * wm + T(3) * w;
    T B0 = c13 * (t * t) + c14 * (t2 * t2);
    t = wmm - T(2) * w + wp; t2 = wm - wp;
    T B1 = c13 * (t * t) + c14 * (t2 * t2);
    t = w - T(2) * wp + wpp; t2 = T(3) * w - T(4) * wp + wpp;
    T B2 = c13 * (t * t) + c14 * (t2 * t2);
    T d0 = T(3.) / T(10.), d1 = T(6.) / T(10.), d2 = T(1.) / T(10.);
    T a0 = m.div(d0, (e + B0) * (e + B0)), a1 = m.div(d1, (e + B1) * (e + B1)), a2 = m.div(d2, (e + B2) * (e + B2));
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
  return m.root(T(0.5) * (i0 + m.root(i1 * i1 + T(4.) * (a * a) * ((ca * ca) - (can * can)))));
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
    cf[q] = m.root(T(0.5) * (i0 + m.root(i1 * i1 + T(4.) * (a * a) * ((ca * ca) - (can * can)))));
  }
}

// conserved state, physical flux, enthalpy, total pressure and energy of one
// side (riemannS.cpp:59-108)
template <typename T>
struct Side {
  T q[8], F[8], H, pt, cf, e;
};

template <typename T, class M>
__device__ __forceinline__ void side_state(M &m, const T *w, T gamma, Side<T> &s) {
  s.cf = fast_speed<T>(m, w, gamma, 5);
  const T vn = w[1], Bn = w[5];
  T e = m.div(w[4], w[0] * (gamma - T(1))) + T(0.5) * (w[1] * w[1] + w[2] * w[2] + w[3] * w[3]) +
        m.div(T(0.5) * (w[5] * w[5] + w[6] * w[6] + w[7] * w[7]), w[0]);
  e = e * w[0];
  s.e = e;
  s.H = m.div(e + w[4] + T(0.5) * (w[5] * w[5] + w[6] * w[6] + w[7] * w[7]), w[0]);
#pragma unroll
  for (int k = 0; k < 8; k++) s.q[k] = w[k];
  s.q[1] = w[0] * w[1]; s.q[2] = w[0] * w[2]; s.q[3] = w[0] * w[3];
  s.q[4] = e;
  const T pt = w[4] + T(0.5) * (w[5] * w[5] + w[6] * w[6] + w[7] * w[7]);
  s.pt = pt;
  s.F[0] = w[0] * vn;
  s.F[1] = w[0] * vn * w[1] + pt - Bn * w[5];
  s.F[2] = w[0] * vn * w[2] - Bn * w[6];
  s.F[3] = w[0] * vn * w[3] - Bn * w[7];
  s.F[4] = w[0] * vn * s.H - Bn * (w[1] * w[5] + w[2] * w[6] + w[3] * w[7]);
  s.F[5] = vn * w[5] - Bn * w[1];
  s.F[6] = vn * w[6] - Bn * w[2];
  s.F[7] = vn * w[7] - Bn * w[3];
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
  const T im = smax(a, b);
#pragma unroll
  for (int k = 0; k < 8; k++) f[k] = T(0.5) * (L.F[k] + R.F[k]) - T(0.5) * im * (R.q[k] - L.q[k]);
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

// riemannS.cpp:397-549 (Miyoshi & Kusano).  Only the branch the wave fan
// selects is assembled; its arithmetic is that of the reference.
template <typename T, class M>
__device__ __forceinline__ int flux_hlld(M &m, const T *wL, const T *wR, T gamma, T *f) {
  Side<T> L, R;
  side_state<T>(m, wL, gamma, L);
  side_state<T>(m, wR, gamma, R);
  const T vnL = wL[1], vnR = wR[1], ptL = L.pt, ptR = R.pt;
  const T SL = smin(vnL, vnR) - smax(L.cf, R.cf);
  const T SR = smax(vnL, vnR) + smax(L.cf, R.cf);
  const T SM = m.div((SR - vnR) * wR[0] * vnR - (SL - vnL) * wL[0] * vnL - ptR + ptL,
                     (SR - vnR) * wR[0] - (SL - vnL) * wL[0]);
  const T pts = m.div((SR - vnR) * wR[0] * ptL - (SL - vnL) * wL[0] * ptR +
                          wL[0] * wR[0] * (SR - vnR) * (SL - vnL) * (vnR - vnL),
                      (SR - vnR) * wR[0] - (SL - vnL) * wL[0]);
  // left * state (:467-481)
  const T rLs = m.div(wL[0] * (SL - vnL), SL - SM);
  T vLs, wzLs, byLs, bzLs;
  if ((wL[0] * (SL - wL[1]) * (SL - SM) - wL[5] * wL[5]) != T(0)) {
    const T den = wL[0] * (SL - wL[1]) * (SL - SM) - wL[5] * wL[5];
    vLs = wL[2] - wL[5] * wL[6] * m.div(SM - wL[1], den);
    wzLs = wL[3] - wL[5] * wL[7] * m.div(SM - wL[1], den);
    byLs = wL[6] * m.div(wL[0] * ((SL - wL[1]) * (SL - wL[1])) - wL[5] * wL[5], den);
    bzLs = wL[7] * m.div(wL[0] * ((SL - wL[1]) * (SL - wL[1])) - wL[5] * wL[5], den);
  } else {
    vLs = wL[2]; wzLs = wL[3]; byLs = T(0.); bzLs = T(0.);
  }
  const T eLs = m.div((SL - wL[1]) * L.e - ptL * wL[1] + pts * SM +
                          wL[5] * (dot13_57(wL[1], wL[2], wL[3], wL[5], wL[6], wL[7]) -
                                   dot13_57(SM, vLs, wzLs, wL[5], byLs, bzLs)),
                      SL - SM);
  // right * state (:483-497)
  const T rRs = m.div(wR[0] * (SR - vnR), SR - SM);
  T vRs, wzRs, byRs, bzRs;
  if ((wR[0] * (SR - wR[1]) * (SR - SM) - wR[5] * wR[5]) != T(0)) {
    const T den = wR[0] * (SR - wR[1]) * (SR - SM) - wR[5] * wR[5];
    vRs = wR[2] - wR[5] * wR[6] * m.div(SM - wR[1], den);
    wzRs = wR[3] - wR[5] * wR[7] * m.div(SM - wR[1], den);
    byRs = wR[6] * m.div(wR[0] * ((SR - wR[1]) * (SR - wR[1])) - wR[5] * wR[5], den);
    bzRs = wR[7] * m.div(wR[0] * ((SR - wR[1]) * (SR - wR[1])) - wR[5] * wR[5], den);
  } else {
    vRs = wR[2]; wzRs = wR[3]; byRs = T(0); bzRs = T(0);
  }
  const T eRs = m.div((SR - wR[1]) * R.e - ptR * wR[1] + pts * SM +
                          wR[5] * (dot13_57(wR[1], wR[2], wR[3], wR[5], wR[6], wR[7]) -
                                   dot13_57(SM, vRs, wzRs, wR[5], byRs, bzRs)),
                      SR - SM);
  const T sLs = m.root(rLs), sRs = m.root(rRs);
  const T SLs = SM - m.div(fabs(wL[5]), sLs);
  const T SRs = SM + m.div(fabs(wR[5]), sRs);
  int br = -1;
  if (SL > T(0)) br = 0;
  else if (SL <= T(0.) && SLs >= T(0.)) br = 1;
  else if (SLs <= T(0.) && SM >= T(0.)) br = 2;
  else if (SM <= T(0.) && SRs >= T(0.)) br = 3;
  else if (SRs <= T(0.) && SR >= T(0.)) br = 4;
  else if (SR < T(0.)) br = 5;
  // conserved * states (w2u, misc.cpp:82-92; energy replaced, :524,527)
  const T qLs[8] = {rLs, rLs * SM, rLs * vLs, rLs * wzLs, eLs, wL[5], byLs, bzLs};
  const T qRs[8] = {rRs, rRs * SM, rRs * vRs, rRs * wzRs, eRs, wR[5], byRs, bzRs};
  T qss[8];
  if (br == 2 || br == 3) {
    // ** states (:501-519); the right ** state is a copy of the left one (:517)
    const T sg = sgn(wL[5]);
    const T vss = m.div(sLs * vLs + sRs * vRs + (byRs - byLs) * sg, sLs + sRs);
    const T wss = m.div(sLs * wzLs + sRs * wzRs + (bzRs - bzLs) * sg, sLs + sRs);
    const T byss = m.div(sLs * byRs + sRs * byLs + m.root(rLs * rRs) * (vRs - vLs) * sg, sLs + sRs);
    const T bzss = m.div(sLs * bzRs + sRs * bzLs + m.root(rLs * rRs) * (wzRs - wzLs) * sg, sLs + sRs);
    const T dss = dot13_57(SM, vss, wss, wL[5], byss, bzss);
    T ess;
    if (br == 2)
      ess = eLs - sLs * (dot13_57(SM, vLs, wzLs, wL[5], byLs, bzLs) - dss) * sg;
    else
      ess = eRs + sRs * (dot13_57(SM, vRs, wzRs, wR[5], byRs, bzRs) - dss) * sgn(wR[5]);
    qss[0] = rLs; qss[1] = rLs * SM; qss[2] = rLs * vss; qss[3] = rLs * wss;
    qss[4] = ess; qss[5] = wL[5]; qss[6] = byss; qss[7] = bzss;
  }
#pragma unroll
  for (int k = 0; k < 8; k++) {
    T v = T(0);
    switch (br) {
      case 0: v = L.F[k]; break;
      case 1: v = L.F[k] + SL * qLs[k] - SL * L.q[k]; break;
      case 2: v = L.F[k] + SLs * qss[k] - (SLs - SL) * qLs[k] - SL * L.q[k]; break;
      case 3: v = R.F[k] + SRs * qss[k] - (SRs - SR) * qRs[k] - SR * R.q[k]; break;
      case 4: v = R.F[k] + SR * qRs[k] - SR * R.q[k]; break;
      case 5: v = R.F[k]; break;
      default: break;
    }
    f[k] = v;
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
