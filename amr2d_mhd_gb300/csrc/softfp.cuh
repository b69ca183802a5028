// Correctly rounded FP64 division and square root on the integer and FP32
// pipes.
//
// GB300 issues FP64 at 2 lanes per SM and clock, 1/64 of the FP32 rate, so a
// warp's FP64 instruction holds the SM's FP64 pipe for 16 clocks; the
// compiler's division and square root take 8 to 10 of them.  The FP64
// kernels of this library were bound by that pipe (83 % busy) while the issue
// slots stood at 8 %.  The routines below take about 45 integer instructions
// and one MUFU each, none of them on the FP64 pipe, and return the same bits
// as IEEE division and square root in round to nearest even.  Measured on one
// GB300, 12 warps per SM: 26 clocks per SM and warp for an addition and a
// division (115 with the compiler's), 25 for an addition and a square root
// (115).  The face kernel with the Soft arithmetic, 196-block rotor (MC +
// HLLD): 257 -> 90 us; 256-block KH layer (MC + RUSA): 207 -> 79 us and 2.87 ->
// 1.12 M FP64-pipe instructions; 256-block Orszag-Tang (WENO5 + HLLD): 790 ->
// 280 us.
//
// Method (long division with a large radix, two digits; e.g. Ercegovac &
// Lang, Digital Arithmetic, ch. 5 and 7): a 23-bit reciprocal from MUFU,
// rounded so that it never exceeds the true one, is refined by one Newton step
// in 32-bit fixed point to R (relative error below 2^-29); the first
// quotient digit is the high word of a * R, the exact remainder follows
// modulo 2^64 (it is small, so its low 64 bits are all of it), the second
// digit is the high word of remainder * R.  Both digits are too small by a
// few units at most, which leaves the quotient within 2^-57 below the true
// one.  From it comes n, the rounded 53-bit quotient or one less, and the
// sign of the exact (2n + 1) b - 2 a 2^k (modulo 2^64 again) decides.  A
// quotient of two 53-bit numbers and a square root never lie halfway between
// two 53-bit numbers.
//
// Zero numerators and arguments are handled.  Everything else outside the
// normal range (subnormal, infinite or NaN operands, negative square roots,
// results near the ends of the exponent range) is left to the caller: `bad`
// is set, the value returned is meaningless, and the caller repeats its
// computation with the native operators (Soft / Native below).
#pragma once

#include <stdint.h>
#include <string.h>

#include <cmath>

#ifdef __CUDACC__
#define AMR_HD __host__ __device__ __forceinline__
#else
#define AMR_HD inline
#endif

namespace amr {

AMR_HD uint64_t f64_bits(double x) {
#ifdef __CUDA_ARCH__
  return static_cast<uint64_t>(__double_as_longlong(x));
#else
  uint64_t u;
  memcpy(&u, &x, 8);
  return u;
#endif
}
AMR_HD double bits_f64(uint32_t hi, uint32_t lo) {
#ifdef __CUDA_ARCH__
  return __hiloint2double(static_cast<int>(hi), static_cast<int>(lo));
#else
  const uint64_t u = (static_cast<uint64_t>(hi) << 32) | lo;
  double x;
  memcpy(&x, &u, 8);
  return x;
#endif
}
AMR_HD uint32_t mulhi32(uint32_t a, uint32_t b) {
#ifdef __CUDA_ARCH__
  return __umulhi(a, b);
#else
  return static_cast<uint32_t>((static_cast<uint64_t>(a) * b) >> 32);
#endif
}
// (hi:lo << s) >> 32 and the low word of (hi:lo >> s), 0 < s < 32
AMR_HD uint32_t shl_hi(uint32_t lo, uint32_t hi, int s) {
#ifdef __CUDA_ARCH__
  return __funnelshift_l(lo, hi, s);
#else
  return (hi << s) | (lo >> (32 - s));
#endif
}
AMR_HD uint32_t shr_lo(uint32_t lo, uint32_t hi, int s) {
#ifdef __CUDA_ARCH__
  return __funnelshift_r(lo, hi, s);
#else
  return (lo >> s) | (hi << (32 - s));
#endif
}

// The 23-bit seeds as 32-bit fractions of 2^32: r + 1 truncated to a float in
// [1.4, 2) has r in its mantissa, which the shift moves to the top.  The host
// build (for tests) stands in for MUFU with a float operation, moved by
// `seed_ulp` units to cover MUFU's error bounds (2^-23 and 2^-22.9).
#ifdef __CUDA_ARCH__
__device__ __forceinline__ uint32_t seed_rcp(uint32_t fbits) {
  float r;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(__uint_as_float(fbits)));
  return __float_as_uint(__fadd_rz(r, 1.0f)) << 9;
}
__device__ __forceinline__ uint32_t seed_rsqrt(uint32_t fbits) {
  float r;
  asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(__uint_as_float(fbits)));
  return __float_as_uint(__fadd_rz(r, 1.0f)) << 9;
}
#else
inline double &seed_rel() {
  static double v = 0.0;
  return v;
}
inline uint32_t seed_fix(double r) {
  return static_cast<uint32_t>(r * (1.0 + seed_rel()) * 8388608.0) << 9;  // truncated, as __fadd_rz
}
inline uint32_t seed_rcp(uint32_t fbits) {
  float f;
  memcpy(&f, &fbits, 4);
  return seed_fix(1.0 / f);
}
inline uint32_t seed_rsqrt(uint32_t fbits) {
  float f;
  memcpy(&f, &fbits, 4);
  return seed_fix(1.0 / std::sqrt(static_cast<double>(f)));
}
#endif

// floor-like reciprocal of the significand b32 = floor(mb 2^-21): R <= 2^63 / (mb 2^-21)
AMR_HD uint32_t rcp_digit(uint32_t b32) {
  // R0 below the reciprocal, relative error in (0, 7.1 2^-23]: the float of
  // b's top 24 bits raised by 4 units, which covers the bits cut off and
  // MUFU's error
  const uint32_t R0 = seed_rcp((b32 >> 8) + 0x3f000004u);
  // one Newton step; 2^31 - p is too large by less than 2, taken back by the
  // 4 in 2 (2^31 - p) - 4, so that R stays below: error in [0, 2^-29.9)
  const uint32_t p = mulhi32(b32, R0);
  return R0 + mulhi32(R0, 0u - 2u * p - 4u);
}

// a / b with R = rcp_digit(top 32 bits of b's significand)
AMR_HD double div_with(double a, double b, uint32_t R, bool &bad) {
  const uint64_t ua = f64_bits(a), ub = f64_bits(b);
  const uint32_t ah = static_cast<uint32_t>(ua >> 32), al = static_cast<uint32_t>(ua);
  const uint32_t bh = static_cast<uint32_t>(ub >> 32), bl = static_cast<uint32_t>(ub);
  const uint32_t sign = (ah ^ bh) & 0x80000000u;
  const uint32_t ea = ah & 0x7ff00000u, eb = bh & 0x7ff00000u;
  const bool zero = ((ah << 1) | al) == 0u;
  // both operands normal and the exponent of the result two steps inside the normal range
  const uint32_t er = ea - eb + (1021u << 20);   // (exponent of a / b) - 2, if in range
  bad |= !(eb - (1u << 20) < (2046u << 20) &&
           (zero || (ea - (1u << 20) < (2046u << 20) && er < (2043u << 20))));
  // 53-bit significands ma, mb; the top 32 bits of ma
  const uint32_t mah = (ah & 0xfffffu) | 0x100000u, mbh = (bh & 0xfffffu) | 0x100000u;
  const uint32_t a32 = shl_hi(al, mah, 11);
  // first digit, floor(2^31 a / b) less 0..6, and its remainder in [0, 6.1 mb)
  const uint32_t q1 = mulhi32(a32, R);
  const uint64_t mb = (static_cast<uint64_t>(mbh) << 32) | bl, nb = 0u - mb;
  const uint64_t ma31 = (static_cast<uint64_t>(shr_lo(al, mah, 1)) << 32) | (al << 31);
  const uint64_t rem = ma31 + static_cast<uint64_t>(q1) * static_cast<uint32_t>(nb) +
                       (static_cast<uint64_t>(q1 * static_cast<uint32_t>(nb >> 32)) << 32);
  // second digit: 2^28 rem / mb (below 2^31)
  const uint32_t q2 = mulhi32(shr_lo(static_cast<uint32_t>(rem), static_cast<uint32_t>(rem >> 32), 24), R);
  // Q = 2^59 a / b less 0..8; normalised to [2^59, 2^60) (less 0..16)
  uint64_t Q = (static_cast<uint64_t>(q1) << 28) + q2;
  const bool below = static_cast<uint32_t>(Q >> 32) < (1u << 27);
  if (below) Q += Q;
  // n = v >> 7, the rounded quotient or one less; u = 2 n + 1
  const uint64_t v = Q + 64u;
  const uint32_t vl = static_cast<uint32_t>(v), vh = static_cast<uint32_t>(v >> 32);
  const uint32_t ul = shr_lo(vl, vh, 6) | 1u, uh = vh >> 6;
  const uint32_t nl = shr_lo(vl, vh, 7), nh = vh >> 7;
  // the sign of u mb - 2^(k+1) ma, k = 52 (quotient >= 1) or 53
  const uint64_t t = static_cast<uint64_t>(ul) * bl - (static_cast<uint64_t>(al << (below ? 22 : 21)) << 32) +
                     (static_cast<uint64_t>(ul * mbh + uh * bl) << 32);
  const uint32_t up = static_cast<uint32_t>(t >> 63);
  const uint64_t n = ((static_cast<uint64_t>(nh) << 32) | nl) + up;
  const uint32_t e = ea - eb + (below ? 1021u << 20 : 1022u << 20);
  const uint32_t hi = static_cast<uint32_t>(n >> 32) + e;
  return bits_f64((zero ? 0u : hi) | sign, zero ? 0u : static_cast<uint32_t>(n));
}

// a / b; several quotients of one b share its R (the compiler merges them)
AMR_HD double div_rn(double a, double b, bool &bad) {
  const uint64_t ub = f64_bits(b);
  const uint32_t mbh = (static_cast<uint32_t>(ub >> 32) & 0xfffffu) | 0x100000u;
  return div_with(a, b, rcp_digit(shl_hi(static_cast<uint32_t>(ub), mbh, 11)), bad);
}

// a / B for a small whole number B: its R is a constant
template <int B>
AMR_HD double div_by(double a, bool &bad) {
  constexpr int lead = B < 2 ? 0 : (B < 4 ? 1 : (B < 8 ? 2 : 3));
  static_assert(B > 0 && B < 16, "B in [1, 16)");
  constexpr uint32_t b32 = static_cast<uint32_t>(B) << (31 - lead);
  constexpr uint64_t r = (1ull << 63) / b32;
  return div_with(a, static_cast<double>(B), r > 0xffffffffull ? 0xffffffffu : static_cast<uint32_t>(r), bad);
}

// sqrt(x)
AMR_HD double sqrt_rn(double x, bool &bad) {
  const uint64_t ux = f64_bits(x);
  const uint32_t xh = static_cast<uint32_t>(ux >> 32), xl = static_cast<uint32_t>(ux);
  const bool zero = ((xh << 1) | xl) == 0u;
  bad |= !(zero || xh - (1u << 20) < (2046u << 20));   // positive and normal
  // x = M 2^-52 4^h, M in [2^52, 2^54): the significand, doubled for odd exponents
  const uint32_t odd = (~xh >> 20) & 1u;
  const uint32_t mh = (xh & 0xfffffu) | 0x100000u;
  const uint32_t Mh = (mh << odd) | (odd ? xl >> 31 : 0u), Ml = xl << odd;
  const uint32_t M32 = shl_hi(Ml, Mh, 10);
  // R0 <= 2^32 / sqrt(M 2^-52), relative error in (0, 6.1 2^-23]: the float of
  // M's top bits raised by 6 units
  const uint32_t R0 = seed_rsqrt(shl_hi(xl, (xh & 0x1fffffu) ^ 0x100000u, 3) + 0x3f800006u);
  // one Newton step: 2^30 - (M R0^2) is too large by less than 3, taken back
  const uint32_t v0 = mulhi32(mulhi32(M32, R0), R0);
  const uint32_t R = R0 + mulhi32(R0, 0x80000000u - 6u - 2u * v0);
  // first digit, 2^30 sqrt less 0..6, its remainder (below 2^35), second digit
  const uint32_t s1 = mulhi32(M32, R);
  const uint64_t M8 = (static_cast<uint64_t>(shl_hi(Ml, Mh, 8)) << 32) | (Ml << 8);
  const uint64_t rem = M8 - static_cast<uint64_t>(s1) * s1;
  const uint32_t s2 = mulhi32(shr_lo(static_cast<uint32_t>(rem), static_cast<uint32_t>(rem >> 32), 3), R);
  // 2^58 sqrt less 0..8; n = v >> 6, the rounded root or one less; u = 2 n + 1
  const uint64_t v = (static_cast<uint64_t>(s1) << 28) + s2 + 32u;
  const uint32_t vl = static_cast<uint32_t>(v), vh = static_cast<uint32_t>(v >> 32);
  const uint32_t ul = shr_lo(vl, vh, 5) | 1u, uh = vh >> 5;
  const uint32_t nl = shr_lo(vl, vh, 6), nh = vh >> 6;
  // the sign of u^2 - 2^54 M
  const uint64_t t = static_cast<uint64_t>(ul) * ul - (static_cast<uint64_t>(Ml << 22) << 32) +
                     (static_cast<uint64_t>(2u * ul * uh) << 32);
  const uint32_t up = static_cast<uint32_t>(t >> 63);
  const uint64_t n = ((static_cast<uint64_t>(nh) << 32) | nl) + up;
  const uint32_t e = (((xh + (1023u << 20)) >> 1) & 0x7ff00000u) - (1u << 20);
  const uint32_t hi = static_cast<uint32_t>(n >> 32) + e;
  return zero ? x : bits_f64(hi, static_cast<uint32_t>(n));
}

// a * b, for kernels whose FP64 instructions are few among memory accesses (the
// CT face update): about 50 integer instructions, 17 clocks per SM and warp
// beside additions on the FP64 pipe, which takes 20 for a product.  (In the face
// kernels, which have a quarter of the warps in flight to hide those 50
// instructions, products stayed faster on the FP64 pipe.)
AMR_HD double mul_rn(double a, double b, bool &bad) {
  const uint64_t ua = f64_bits(a), ub = f64_bits(b);
  const uint32_t ah = static_cast<uint32_t>(ua >> 32), al = static_cast<uint32_t>(ua);
  const uint32_t bh = static_cast<uint32_t>(ub >> 32), bl = static_cast<uint32_t>(ub);
  const uint32_t ea = ah & 0x7ff00000u, eb = bh & 0x7ff00000u;
  // a zero operand, or exponents so small together that the product, below 2^-1075, rounds to zero
  const bool za = ((ah << 1) | al) == 0u, zb = ((bh << 1) | bl) == 0u;
  const bool zero = za || zb || ea + eb <= (969u << 20);
  // normal operands and a result exponent inside the normal range, or zeros and normal operands
  const uint32_t er = ea + eb - (1024u << 20);   // (exponent of the product) - 1, if it is not doubled
  bad |= !((za || ea - (1u << 20) < (2046u << 20)) && (zb || eb - (1u << 20) < (2046u << 20)) &&
           (zero || er < (2044u << 20)));
  // the 106-bit product of the significands: h 2^64 + (low word of c) 2^32 + (low word of p)
  const uint32_t mah = (ah & 0xfffffu) | 0x100000u, mbh = (bh & 0xfffffu) | 0x100000u;
  const uint64_t p = static_cast<uint64_t>(al) * bl;
  const uint64_t c = static_cast<uint64_t>(al) * mbh + (static_cast<uint64_t>(mah) * bl + (p >> 32));
  const uint64_t h = static_cast<uint64_t>(mah) * mbh + (c >> 32);
  const uint32_t hh = static_cast<uint32_t>(h >> 32), hl = static_cast<uint32_t>(h), w = static_cast<uint32_t>(c);
  const uint32_t top = hh >> 9;                  // 1 if the product is in [2, 4)
  const int s = 12 - static_cast<int>(top);
  const uint32_t nl = shl_hi(w, hl, s), nh = shl_hi(hl, hh, s);
  // what is cut off, its last bit standing for everything below; round to nearest even
  const uint32_t rest = (w << s) | (static_cast<uint32_t>(p) != 0u ? 1u : 0u);
  const uint32_t up = static_cast<uint32_t>((static_cast<uint64_t>(rest) + 0x7fffffffu + (nl & 1u)) >> 32);
  const uint64_t n = ((static_cast<uint64_t>(nh) << 32) | nl) + up;
  const uint32_t hi = static_cast<uint32_t>(n >> 32) + er + (top << 20);
  const uint32_t sign = (ah ^ bh) & 0x80000000u;
  return bits_f64((zero ? 0u : hi) | sign, zero ? 0u : static_cast<uint32_t>(n));
}

// double to float (to nearest even) and back on the integer pipe, where the
// conversion instructions take the FP64 pipe; outside the float's normal range
// the conversion itself
AMR_HD float to_f32(double x) {
  const uint64_t u = f64_bits(x);
  const uint32_t h = static_cast<uint32_t>(u >> 32), l = static_cast<uint32_t>(u);
  const uint32_t e = (h >> 20) & 0x7ffu;
  if ((h << 1 | l) != 0u && e - 897u >= 253u) return static_cast<float>(x);
  const uint32_t m = shl_hi(l, h & 0xfffffu, 3);
  const uint32_t up = static_cast<uint32_t>((static_cast<uint64_t>(l << 3) + 0x7fffffffu + (m & 1u)) >> 32);
  const uint32_t b = (h & 0x80000000u) | ((h << 1 | l) == 0u ? 0u : ((e - 896u) << 23) + m + up);
#ifdef __CUDA_ARCH__
  return __uint_as_float(b);
#else
  float f;
  memcpy(&f, &b, 4);
  return f;
#endif
}
AMR_HD double to_f64(float x) {
#ifdef __CUDA_ARCH__
  const uint32_t b = __float_as_uint(x);
#else
  uint32_t b;
  memcpy(&b, &x, 4);
#endif
  const uint32_t e = (b >> 23) & 0xffu, m = b & 0x7fffffu;
  if ((b << 1) != 0u && e - 1u >= 254u) return static_cast<double>(x);
  return (b << 1) == 0u ? bits_f64(b, 0u) : bits_f64((b & 0x80000000u) | ((e + 896u) << 20) | (m >> 3), m << 29);
}

// 2^K x, exact: the exponent field moved, zeros kept.  A result or operand
// outside the normal range sets `bad`.
template <int K>
AMR_HD double scale_pow2(double x, bool &bad) {
  const uint64_t u = f64_bits(x);
  const uint32_t h = static_cast<uint32_t>(u >> 32), l = static_cast<uint32_t>(u);
  const uint32_t t = h << 1;
  const bool zero = (t | l) == 0u;
  constexpr uint32_t down = K < 0 ? -K : 0, up = K > 0 ? K : 0;
  bad |= !(zero || t - ((1u + down) << 21) < ((2046u - up - down) << 21));
  return bits_f64(zero ? h : h + (static_cast<uint32_t>(K) << 20), l);
}

// x * p for p a power of two, exact, as scale_pow2
AMR_HD double times_pow2(double x, double p, bool &bad) {
  const uint64_t u = f64_bits(x);
  const uint32_t h = static_cast<uint32_t>(u >> 32), l = static_cast<uint32_t>(u);
  const uint32_t t = h << 1;
  const bool zero = (t | l) == 0u;
  const int e = static_cast<int>(t >> 21), k = static_cast<int>((f64_bits(p) >> 52) & 0x7ff) - 1023;
  bad |= !(zero || (e - 1u < 2046u && e + k - 1u < 2046u));
  return bits_f64(zero ? h : h + (static_cast<uint32_t>(k) << 20), l);
}

#ifdef __CUDACC__
// The arithmetic a formula is evaluated with: the operators of the type, or,
// for double, the routines above and comparisons and multiplications by
// powers of two on the bit patterns (3 to 7 integer instructions each, where
// the FP64 pipe takes 16 clocks per warp).  After a Soft evaluation that reports
// failed(), some operand was outside the routines' range and the results are
// meaningless: evaluate again with Native.
template <typename T>
struct Native {
  __device__ __forceinline__ T div(T a, T b) { return a / b; }
  __device__ __forceinline__ T ratio(T a, T b) { return a / b; }   // b not subnormal (Quick)
  __device__ __forceinline__ T root(T x) { return sqrt(x); }
  template <int B> __device__ __forceinline__ T by(T a) { return a / T(B); }
  __device__ __forceinline__ T mul(T a, T b) { return a * b; }
  // the larger of two values that are not negative; Soft compares the bits,
  // where a NaN counts as the largest (and the division it reaches fails)
  __device__ __forceinline__ T most(T a, T b) { return a > b ? a : b; }
  __device__ __forceinline__ T std_most(T a, T b) { return a < b ? b : a; }   // std::max, for a NaN in b
  __device__ __forceinline__ T least(T a, T b) { return a < b ? a : b; }
  // multiplications by powers of two
  __device__ __forceinline__ T half(T a) { return T(0.5) * a; }
  __device__ __forceinline__ T quarter(T a) { return T(0.25) * a; }
  __device__ __forceinline__ T twice(T a) { return T(2) * a; }
  __device__ __forceinline__ T quad(T a) { return T(4) * a; }
  __device__ __forceinline__ T scaled(T a, T p) { return a * p; }   // p a positive power of two
  // comparisons with zero
  __device__ __forceinline__ bool positive(T a) { return a > T(0); }
  __device__ __forceinline__ bool negative(T a) { return a < T(0); }
  __device__ __forceinline__ bool nonpositive(T a) { return a <= T(0); }
  __device__ __forceinline__ bool nonnegative(T a) { return a >= T(0); }
  __device__ __forceinline__ bool nonzero(T a) { return a != T(0); }
  __device__ __forceinline__ bool failed() const { return false; }
};
struct Soft {
  bool bad = false;
  __device__ __forceinline__ double div(double a, double b) { return div_rn(a, b, bad); }
  __device__ __forceinline__ double ratio(double a, double b) { return div(a, b); }
  __device__ __forceinline__ double root(double x) { return sqrt_rn(x, bad); }
  template <int B> __device__ __forceinline__ double by(double a) { return div_by<B>(a, bad); }
  __device__ __forceinline__ double mul(double a, double b) { return mul_rn(a, b, bad); }
  __device__ __forceinline__ double most(double a, double b) { return f64_bits(a) > f64_bits(b) ? a : b; }
  __device__ __forceinline__ double std_most(double a, double b) { return most(a, b); }
  __device__ __forceinline__ double least(double a, double b) { return f64_bits(a) < f64_bits(b) ? a : b; }
  __device__ __forceinline__ double half(double a) { return scale_pow2<-1>(a, bad); }
  __device__ __forceinline__ double quarter(double a) { return scale_pow2<-2>(a, bad); }
  __device__ __forceinline__ double twice(double a) { return scale_pow2<1>(a, bad); }
  __device__ __forceinline__ double quad(double a) { return scale_pow2<2>(a, bad); }
  __device__ __forceinline__ double scaled(double a, double p) { return times_pow2(a, p, bad); }
  // of numbers (a NaN fails in the divisions around them)
  __device__ __forceinline__ bool positive(double a) { return __double_as_longlong(a) > 0; }
  __device__ __forceinline__ bool negative(double a) { return __double_as_longlong(a) < 0 && nonzero(a); }
  __device__ __forceinline__ bool nonpositive(double a) { return !positive(a); }
  __device__ __forceinline__ bool nonnegative(double a) { return !negative(a); }
  __device__ __forceinline__ bool nonzero(double a) { return (f64_bits(a) << 1) != 0; }
  __device__ __forceinline__ bool failed() const { return bad; }
};
// The FP32 face kernels': quotients and roots from MUFU without the
// compiler's handling of subnormal operands (2 and 1 instructions; a quotient
// is a * rcp(b), within 2 ulp, and quotients of one b share the reciprocal).
// MUFU takes a divisor above 2^126 for infinite (reciprocal zero) and a
// subnormal divisor or radicand for zero: `low`, the smallest of all three,
// notes those, and the face is then evaluated again with Native, as after Soft.
// (The check costs 1 % of a step of 32 MC + HLLD rotors or 24 HLLE blasts, 3.5 %
// of a 512^2 WENO3 layer.)
struct Quick : Native<float> {
  float low = 1.0f;
  __device__ __forceinline__ float div(float a, float b) {
    low = fminf(low, fabsf(b));
    return ratio(a, b);
  }
  // a / b where a zero b is as good as any (infinite or NaN, as IEEE) and a subnormal one does not occur
  __device__ __forceinline__ float ratio(float a, float b) {
    float r;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(b));
    low = fminf(low, fabsf(r));
    return a * r;
  }
  __device__ __forceinline__ float root(float x) {
    float r;
    asm("sqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    low = fminf(low, fabsf(x));
    return r;
  }
  template <int B> __device__ __forceinline__ float by(float a) { return a * (1.0f / B); }
  __device__ __forceinline__ bool failed() const { return low < 0x1p-126f; }
};
template <typename T> struct FaceArith { using type = Soft; };
template <> struct FaceArith<float> { using type = Quick; };
template <typename T> struct ArithOf { using type = Native<T>; };
template <> struct ArithOf<double> { using type = Soft; };

// f(m) with the arithmetic of T, repeated with Native where that failed; f
// only writes values that the repetition overwrites
template <typename T, class F>
__device__ __forceinline__ void evaluate(F &&f) {
  typename ArithOf<T>::type m;
  f(m);
  if (m.failed()) {
    // as a loop (of one round), which stays a branch: a short body would be
    // predicated, and its FP64 instructions issued to the pipe all the same
    // (k_ct_face, 6272 leaves: 55 us predicated, 42 with the branch)
    Native<T> n;
    int rounds = 1;
    asm volatile("" : "+r"(rounds));
    for (; rounds > 0; rounds--) f(n);
  }
}
#endif

}  // namespace amr
