// softfp.cuh -- binary64 arithmetic computed on the integer and FP32 pipes:
// correctly rounded division, square root and multiplication, comparisons,
// fmin / fmax and scalings by powers of two.
//
// GB300 executes binary64 at 1/64 of its FP32 rate: one warp-wide binary64
// instruction holds that pipe for as long as ~32-64 integer instructions
// issue, and a hardware division or square root takes 7-8 of them.  These
// routines return exactly the IEEE round-to-nearest-even result (the same
// bits as x / y, sqrt(x), x * y) for finite normal operands with a normal
// result and for zero operands, and defer every other case (subnormals,
// infinities, NaNs, division by zero, overflow, underflow) to the hardware
// instruction.
//
// They are bound by the integer instructions they issue (the ALU pipe takes
// one warp instruction in two cycles), so each is laid out to need few of
// them: a 30-bit reciprocal (or reciprocal square root) from the FP32 seed and
// one Newton step in 32-bit words, the result's 53 bits in two digits of ~30
// and 23 bits (each digit one 32x32 high product), one exact remainder in
// 64-bit words that decides the rounding, exponents added in place, and one
// range test for all operands.  Instructions per call: division 97 (an exact
// 64-bit reciprocal word, refined and corrected in 128-bit products, took
// over 200), two quotients by one divisor 151, square root 89, product 59,
// two products in one call 98.  With them and the shorter HLLC flux of
// physics.cuh a Kelvin-Helmholtz 2048^2 step (PLM, HLLC) went from 1.66 to
// 1.10 ms, a Sedov one from 1.33 to 1.01 ms.
//
// The core routines also compile for the host (plain C++), where
// tests/softfp_harness.cpp runs them against the host's binary64 arithmetic.
#pragma once

#include <stdint.h>
#ifndef __CUDACC__
#include <math.h>
#include <string.h>
#endif

#ifdef __CUDACC__
#define FV2D_SF __host__ __device__ __forceinline__
#define FV2D_SF_CALL static __host__ __device__ __noinline__
#else
#define FV2D_SF inline
#define FV2D_SF_CALL static
#endif

namespace fv2d {
namespace softfp {

#ifndef __CUDACC__
struct double2 {
  double x, y;
};
inline double2 make_double2(double x, double y) { return double2{x, y}; }
// units in the last place the host's seeds are moved by (the tests sweep it:
// the device's approximations are only accurate to an ulp or two)
static int seed_ulps = 0;
#endif

// On the device the moves are opaque to the optimiser: a plain bit cast lets
// it recognise the integer tests below as floating-point classifications and
// lower them back to binary64 instructions (abs.f64 + setp).
FV2D_SF uint64_t bits(double x) {
  uint64_t b;
#ifdef __CUDA_ARCH__
  asm("mov.b64 %0, %1;" : "=l"(b) : "d"(x));
#else
  memcpy(&b, &x, 8);
#endif
  return b;
}
FV2D_SF double from_bits(uint64_t b) {
  double x;
#ifdef __CUDA_ARCH__
  asm("mov.b64 %0, %1;" : "=d"(x) : "l"(b));
#else
  memcpy(&x, &b, 8);
#endif
  return x;
}
FV2D_SF uint32_t mulhi32(uint32_t a, uint32_t b) { return (uint32_t)(((uint64_t)a * b) >> 32); }

// FP32 seeds as bit patterns: 1/f and 1/sqrt(f).
FV2D_SF uint32_t seed_bits(uint32_t fb, bool root) {
  uint32_t rb;
#ifdef __CUDA_ARCH__
  if (root)
    asm("{\n\t.reg .f32 f, r;\n\tmov.b32 f, %1;\n\trsqrt.approx.ftz.f32 r, f;\n\tmov.b32 %0, r;\n\t}" : "=r"(rb) : "r"(fb));
  else
    asm("{\n\t.reg .f32 f, r;\n\tmov.b32 f, %1;\n\trcp.approx.ftz.f32 r, f;\n\tmov.b32 %0, r;\n\t}" : "=r"(rb) : "r"(fb));
#else
  float f;
  memcpy(&f, &fb, 4);
  const float r = root ? (float)(1.0 / sqrt((double)f)) : (float)(1.0 / (double)f);
  memcpy(&rb, &r, 4);
#ifndef __CUDACC__
  rb += (uint32_t)seed_ulps;
#endif
#endif
  // in [1/2, 1): the 24-bit significand becomes the top of the fixed-point word
  rb = rb < 0x3F000000u ? 0x3F000000u : rb;
  return rb > 0x3F7FFFFFu ? 0x3F7FFFFFu : rb;
}

constexpr uint64_t MAG = 0x7FFFFFFFFFFFFFFFull, INF_BITS = 0x7FF0000000000000ull, SIGN = 0x8000000000000000ull;
constexpr uint64_t FRAC = 0xFFFFFFFFFFFFFull, ONE52 = 1ull << 52;

// Hardware instructions for the special cases, behind calls so that the
// compiler cannot if-convert their expansion into the common path (issued
// predicated-off instructions still occupy the binary64 pipe).
FV2D_SF_CALL double div_hw(double a, double b) { return a / b; }
FV2D_SF_CALL double sqrt_hw(double x) { return sqrt(x); }
FV2D_SF_CALL double mul_hw(double x, double y) { return x * y; }
FV2D_SF_CALL bool prod_neg_hw(double x, double y) { return x * y < 0.0; }

FV2D_SF uint32_t hi32(uint64_t x) { return (uint32_t)(x >> 32); }
FV2D_SF uint32_t lo32(uint64_t x) { return (uint32_t)x; }
FV2D_SF uint64_t join(uint32_t hi, uint32_t lo) { return ((uint64_t)hi << 32) | lo; }
constexpr uint32_t EXP_HI = 0x7FF00000u, FRAC_HI = 0xFFFFFu, ONE_HI = 0x100000u, SIGN_HI = 0x80000000u;

FV2D_SF uint64_t significand(uint64_t ib) { return (ib & FRAC) | ONE52; }
FV2D_SF int exponent(uint64_t ib) { return (int)(hi32(ib) >> 20) & 0x7ff; }
FV2D_SF bool normal_exp(int e) { return (unsigned)(e - 1) < 0x7FEu; }

// The operand range of the common paths, tested on the high words of all of a
// routine's operands together (two instructions an operand): biased exponents
// 768..1279 (adding 256 makes bits 10 and 9 read 10), whose products,
// quotients, and products divided by a third operand are normal.
struct Range {
  uint32_t acc = 0xFFFFFFFFu;
  FV2D_SF void add(uint64_t x) { acc &= (hi32(x) + 0x10000000u) ^ 0x20000000u; }
  FV2D_SF bool ok() const { return (acc & 0x60000000u) == 0x60000000u; }
};

// Reciprocal word of a significand mb in [2^52, 2^53): x = 2^83 / mb with a
// relative error below 2^-30, x in [2^30, 2^31].  With B = mb / 2^21
// truncated to 32 bits, X0 = 2^32 (1 + e) 2^31 / B from the seed (|e| < 2^-21:
// 24-bit truncation of B and two ulps of the approximation), one Newton step
// X0 (2 - B X0 / 2^63) / 2 leaves e^2 < 2^-42 and three truncations of
// 2^-31 each.
FV2D_SF uint32_t recip_word(uint64_t mb) {
  const uint32_t B = (uint32_t)(mb >> 21);
  const uint32_t X0 = (seed_bits(0x3F800000u | ((B >> 8) & 0x7FFFFFu), false) << 8) | 0x80000000u;
  return mulhi32(X0, 0u - mulhi32(B, X0));
}

// n / mb rounded to nearest, as a 53-bit integer Q = n 2^52 / mb, for n in
// [mb, 2 mb) (n below 2^54) and x = recip_word(mb).  The high digit qa (30
// bits, scale 2^-29) is taken one below its estimate: the estimate is off by
// (-3, 1) units, so the remainder r1 = (n 2^29 - qa mb) lies in (0, 4 mb),
// below 2^55.  The low digit qb (scale 2^-52) is rounded to nearest with an
// error of 0.58, so |r2| < 0.58 mb and one step either way rounds Q.  A
// quotient of two 53-bit significands is never midway between two results
// ((2 Q + 1) mb = 2^53 n would need 2^53 | mb), so there are no ties.
FV2D_SF uint64_t quotient(uint64_t n, uint64_t mb, uint32_t x) {
  const uint32_t qa = mulhi32((uint32_t)(n >> 22), x) - 1u;
  const uint64_t r1 = (n << 29) - (uint64_t)qa * mb;
  const uint32_t qb = (mulhi32((uint32_t)(r1 >> 23), x) + 16u) >> 5;
  const int64_t r2 = (int64_t)((r1 << 23) - (uint64_t)qb * mb) * 2;
  uint64_t Q = ((uint64_t)qa << 23) + qb;
  Q += r2 > (int64_t)mb ? 1u : 0u;
  Q -= r2 < -(int64_t)mb ? 1u : 0u;
  return Q;
}

// The sign of s's bit 31 on a positive high word.
FV2D_SF uint32_t with_sign(uint32_t h, uint32_t s) { return h | (s & SIGN_HI); }

// a / b for normal a, b with a normal quotient, x = recip_word of b's
// significand.  Exponents stay in place in the high words; a significand of
// 2^53 carries into the exponent.
FV2D_SF double div_core(uint64_t a, uint64_t b, uint32_t x) {
  const uint64_t ma = significand(a), mb = significand(b);
  const bool big = ma >= mb;
  const uint64_t Q = quotient(big ? ma : ma << 1, mb, x);
  const uint32_t h = hi32(Q) + (hi32(a) & EXP_HI) - (hi32(b) & EXP_HI) + (big ? 1022u << 20 : 1021u << 20);
  return from_bits(join(with_sign(h, hi32(a) ^ hi32(b)), lo32(Q)));
}
// Operands outside the common range: zeros (quiescent regions: a zero with
// the xor of the signs), else the hardware instruction.
FV2D_SF double div_rare(double a, double b) {
  const uint64_t ia = bits(a), ib = bits(b);
  if ((ia & MAG) == 0 && normal_exp(exponent(ib))) return from_bits((ia ^ ib) & SIGN);
  return div_hw(a, b);
}
FV2D_SF double div_with(double a, double b, uint32_t x) {
  Range r;
  r.add(bits(a));
  r.add(bits(b));
  if (!r.ok()) return div_rare(a, b);
  return div_core(bits(a), bits(b), x);
}
// the reciprocal word of b, for any b (meaningless unless b is normal)
FV2D_SF uint32_t recip_of(double b) { return recip_word(significand(bits(b))); }

// Division, square root and multiplication are called rather than inlined:
// the step kernel uses them dozens of times per cell, and one shared copy
// keeps its code within the instruction caches.
FV2D_SF_CALL double div_rn(double a, double b) { return div_with(a, b, recip_of(b)); }

// {a1 / b, a2 / b} (returned by value: outputs through references would live
// on the stack across the call)
FV2D_SF_CALL double2 div2_rn(double a1, double a2, double b) {
  const uint32_t x = recip_of(b);
  Range r;
  r.add(bits(a1));
  r.add(bits(a2));
  r.add(bits(b));
  if (!r.ok()) return make_double2(div_with(a1, b, x), div_with(a2, b, x));
  return make_double2(div_core(bits(a1), bits(b), x), div_core(bits(a2), bits(b), x));
}

// {a1 / b1, a2 / b2} in one call
FV2D_SF_CALL double2 quot2_rn(double a1, double b1, double a2, double b2) {
  Range r;
  r.add(bits(a1));
  r.add(bits(b1));
  r.add(bits(a2));
  r.add(bits(b2));
  if (!r.ok()) return make_double2(div_with(a1, b1, recip_of(b1)), div_with(a2, b2, recip_of(b2)));
  return make_double2(div_core(bits(a1), bits(b1), recip_of(b1)), div_core(bits(a2), bits(b2), recip_of(b2)));
}

// Quotients by one divisor b: recip_of(b) forms its reciprocal word once,
// div_by(a, b, x) each quotient.
FV2D_SF_CALL double div_by(double a, double b, uint32_t x) { return div_with(a, b, x); }
FV2D_SF_CALL double2 div2_by(double a1, double a2, double b, uint32_t x) {
  Range r;
  r.add(bits(a1));
  r.add(bits(a2));
  r.add(bits(b));
  if (!r.ok()) return make_double2(div_with(a1, b, x), div_with(a2, b, x));
  return make_double2(div_core(bits(a1), bits(b), x), div_core(bits(a2), bits(b), x));
}

// recip_of(b) for a divisor known on the host (the mesh spacings): 2^83 / mb
// rounded down.
inline uint32_t recip_of_host(double b) {
  union {
    double f;
    uint64_t u;
  } c{b};
  return (uint32_t)(((unsigned __int128)1 << 83) / ((c.u & FRAC) | ONE52));
}

// sqrt of the significand: M = m 2^(52 + odd) in [2^104, 2^106), g = M 2^-104;
// S = sqrt(M) rounded to nearest, in [2^52, 2^53].  Y = 2^31 / sqrt(g) to
// 2^-29.4 (one Newton step from the seed), the high digit S1 (scale 2^-29)
// two below its estimate, which is off by (-3, 1.5), so r1 = M 2^-46 - S1^2 is
// positive and below 2^34; the low digit's error is below 0.85 (rounding 0.5,
// second-order term 0.2, truncations), and the exact remainder R = M - S^2
// (its low 64 bits carry it) settles the rounding: a step up when R > S, down
// when R <= -S.
FV2D_SF uint64_t root(uint64_t m, int odd) {
  const uint32_t Z = (uint32_t)(m >> (22 - odd));  // g 2^30
  const uint32_t g = ((uint32_t)(127 + odd) << 23) | ((uint32_t)(m >> 29) & 0x7FFFFFu);
  const uint32_t X0 = (seed_bits(g, true) << 8) | 0x80000000u;
  const uint32_t U = mulhi32(mulhi32(X0, X0), Z);
  const uint32_t Y = mulhi32(X0, 0xC0000000u - U);
  const uint32_t S1 = mulhi32(Z, Y) - 2u;
  const uint64_t r1 = (m << (6 + odd)) - (uint64_t)S1 * S1;
  const uint32_t S2 = (mulhi32((uint32_t)(r1 >> 2), Y) + 8u) >> 4;
  const uint64_t S = ((uint64_t)S1 << 23) + S2;
  const int64_t R = (int64_t)(join((uint32_t)m << (20 + odd), 0u) - S * S);
  return S + (R > (int64_t)S ? 1u : 0u) - (R <= -(int64_t)S ? 1u : 0u);
}

// sqrt(x) of a positive normal x, round to nearest even.
FV2D_SF double sqrt_core(uint64_t ix) {
  const int E = (int)(hi32(ix) >> 20);
  const int odd = (E & 1) ^ 1;  // x = m 2^(E - 1075), E - 1075 - odd even
  const uint64_t S = root(significand(ix), odd);
  return from_bits(S + join((uint32_t)((E - odd + 1021) >> 1) << 20, 0u));
}
FV2D_SF_CALL double sqrt_rn(double x) {
  const uint64_t ix = bits(x);
  if ((ix << 1) == 0) return x;  // sqrt(+-0) = +-0
  if (!normal_exp((int)(ix >> 52))) return sqrt_hw(x);  // sign bit included: negative values fail the test
  return sqrt_core(ix);
}

// x * y, round to nearest even, for normal operands with a normal result:
// the 106-bit product of the significands, one of them aligned to bit 63 so
// that the product's high 64 bits hold the result's 52 or 53 bits and the low
// ones decide the rounding.
FV2D_SF double mul_core(uint64_t a, uint64_t b) {
  const uint64_t A = (a << 11) | SIGN;
  const uint32_t al = lo32(A), ah = hi32(A), bl = lo32(b), bh = (hi32(b) & FRAC_HI) | ONE_HI;
  const uint64_t p0 = (uint64_t)al * bl;
  const uint64_t p1 = (uint64_t)ah * bl + hi32(p0);
  const uint64_t p2 = (uint64_t)al * bh + lo32(p1);
  const uint64_t H = (uint64_t)ah * bh + hi32(p1) + hi32(p2);  // in [2^51, 2^53)
  const uint32_t top = hi32(H) & ONE_HI;                       // product of the significands >= 2
  const int k = top ? 0 : 1;
  const uint32_t F = (uint32_t)(((join(lo32(p2), lo32(p0))) << k) >> 32), G = lo32(p0) << k;
  uint64_t M = join((uint32_t)((H << k) >> 32), (uint32_t)((join(lo32(H), lo32(p2)) << k) >> 32)) + (F >> 31);
  if (((F ^ 0x80000000u) | G) == 0) M &= ~1ull;  // tie: to even
  const uint32_t h = hi32(M) + (hi32(a) & EXP_HI) + (hi32(b) & EXP_HI) + top - (1024u << 20);
  return from_bits(join(with_sign(h, hi32(a) ^ hi32(b)), lo32(M)));
}
// Operands outside the common range: zero times finite (zero velocities)
// keeps the xor of the signs, the rest takes the hardware instruction.
FV2D_SF double mul_rare(double x, double y) {
  const uint64_t a = bits(x), b = bits(y);
  if (((a & MAG) == 0 || (b & MAG) == 0) && exponent(a) != 0x7FF && exponent(b) != 0x7FF)
    return from_bits((a ^ b) & SIGN);
  return mul_hw(x, y);
}
FV2D_SF double mul_with(double x, double y) {
  Range r;
  r.add(bits(x));
  r.add(bits(y));
  if (!r.ok()) return mul_rare(x, y);
  return mul_core(bits(x), bits(y));
}
FV2D_SF_CALL double mul_rn(double x, double y) { return mul_with(x, y); }
// two independent products in one call
FV2D_SF_CALL double2 mul2_rn(double x0, double y0, double x1, double y1) {
  Range r;
  r.add(bits(x0));
  r.add(bits(y0));
  r.add(bits(x1));
  r.add(bits(y1));
  if (!r.ok()) return make_double2(mul_with(x0, y0), mul_with(x1, y1));
  return make_double2(mul_core(bits(x0), bits(y0)), mul_core(bits(x1), bits(y1)));
}

// ---------------------------------------------------------------------------
// Comparisons and power-of-two scalings on the bit patterns.  Each returns
// exactly what the IEEE operation returns (NaN compares false; +0 == -0),
// so a binary64 DSETP / DMUL on the 1/64-rate pipe becomes a few integer
// instructions.  Operands outside the cheap range (results that would be
// subnormal, overflow, NaN/inf inputs of a product) go to the hardware
// instruction through a call that is not if-converted.

FV2D_SF bool isnan_b(uint64_t b) { return (b & MAG) > INF_BITS; }

// x > 0, x < 0, x >= 0, x <= 0
FV2D_SF bool gt0(double x) { return bits(x) - 1ull < INF_BITS; }
FV2D_SF bool lt0(double x) { return bits(x) - (SIGN + 1ull) < INF_BITS; }
FV2D_SF bool ge0(double x) {
  const uint64_t b = bits(x);
  return b <= INF_BITS || b == SIGN;
}
FV2D_SF bool le0(double x) {
  const uint64_t b = bits(x);
  return (b & MAG) == 0 || b - SIGN <= INF_BITS;
}

// Order key with -0 == +0 (IEEE comparison order for non-NaN values).
FV2D_SF int64_t key_ieee(uint64_t b) {
  const int64_t m = (int64_t)(b & MAG);
  return (int64_t)b < 0 ? -m : m;
}
// x < y (IEEE: false when either is NaN)
FV2D_SF bool lt(double x, double y) {
  const uint64_t a = bits(x), b = bits(y);
  return !isnan_b(a) && !isnan_b(b) && key_ieee(a) < key_ieee(b);
}

// maximumNumber / minimumNumber: a NaN operand yields the other one; -0 < +0.
// (The C fmax / fmin of the aarch64 C library, FMAXNM / FMINNM.)
FV2D_SF int64_t key_total(uint64_t b) { return (int64_t)(b ^ ((uint64_t)((int64_t)b >> 63) >> 1)); }
FV2D_SF double fmax_nm(double x, double y) {
  const uint64_t a = bits(x), b = bits(y);
  if (isnan_b(b)) return x;
  if (isnan_b(a)) return y;
  return key_total(a) > key_total(b) ? x : y;
}
FV2D_SF double fmin_nm(double x, double y) {
  const uint64_t a = bits(x), b = bits(y);
  if (isnan_b(b)) return x;
  if (isnan_b(a)) return y;
  return key_total(a) < key_total(b) ? x : y;
}
// {fmin_nm(x, y), fmax_nm(x, y)} from one comparison
FV2D_SF double2 minmax_nm(double x, double y) {
  const uint64_t a = bits(x), b = bits(y);
  if (isnan_b(b)) return make_double2(x, x);
  if (isnan_b(a)) return make_double2(y, y);
  const bool less = key_total(a) < key_total(b);
  return make_double2(less ? x : y, less ? y : x);
}

// |x| < |y|
FV2D_SF bool lt_abs(double x, double y) {
  const uint64_t a = bits(x) & MAG, b = bits(y) & MAG;
  return a < b && b <= INF_BITS;
}

// x * y < 0.  Nonzero non-NaN factors of opposite signs give a negative
// product unless it underflows to -0, impossible when the biased exponents
// sum to at least 972 (|x y| >= 2^-1074); smaller products, zeros, subnormals,
// infinities and NaNs go through the call.
FV2D_SF bool prod_neg(double x, double y) {
  const uint32_t a = (uint32_t)(bits(x) >> 32), b = (uint32_t)(bits(y) >> 32);
  if (!((a ^ b) >> 31)) return false;
  const uint32_t xa = a & 0x7FF00000u, xb = b & 0x7FF00000u;
  if (xa - 1u < 0x7FEFFFFFu && xb - 1u < 0x7FEFFFFFu && xa + xb >= (972u << 20)) return true;
  if ((bits(x) & MAG) == 0 || (bits(y) & MAG) == 0) return false;
  return prod_neg_hw(x, y);
}

// x * 2^k for y == 2^k (k = unbiased exponent of y): exact exponent shift
// when x and the result are normal; zeros keep their sign.
FV2D_SF double mul_pow2(double x, double y, int k) {
  const uint64_t a = bits(x);
  const int e = exponent(a);
  if (normal_exp(e) && normal_exp(e + k)) return from_bits(a + ((uint64_t)((uint32_t)k << 20) << 32));
  if ((a & MAG) == 0) return x;
  return mul_hw(x, y);
}

// x * 0.5
FV2D_SF double half(double x) { return mul_pow2(x, 0.5, -1); }

// The sound speeds of two states, sqrt(gamma p / r) with each operation
// rounded, in one call with two independent chains: both of them
// (sound2), or the larger one (sound_max: the square root of the larger
// quotient, a correctly rounded square root being monotone).  Positive
// operands of the common range keep every intermediate normal.
FV2D_SF bool sound_range(double pL, double rL, double pR, double rR, double gamma) {
  Range r;
  r.add(bits(pL));
  r.add(bits(rL));
  r.add(bits(pR));
  r.add(bits(rR));
  r.add(bits(gamma));
  const uint32_t signs = hi32(bits(pL)) | hi32(bits(rL)) | hi32(bits(pR)) | hi32(bits(rR)) | hi32(bits(gamma));
  return r.ok() && (int32_t)signs >= 0;
}
FV2D_SF uint64_t sound_quotient(double p, double r, double gamma) {
  return bits(div_core(bits(mul_core(bits(gamma), bits(p))), bits(r), recip_of(r)));
}
FV2D_SF_CALL double sound_max_rare(double pL, double rL, double pR, double rR, double gamma) {
  return sqrt_rn(fmax_nm(div_rn(mul_rn(pL, gamma), rL), div_rn(mul_rn(pR, gamma), rR)));
}
FV2D_SF_CALL double sound_max(double pL, double rL, double pR, double rR, double gamma) {
  if (!sound_range(pL, rL, pR, rR, gamma)) return sound_max_rare(pL, rL, pR, rR, gamma);
  const uint64_t a = sound_quotient(pL, rL, gamma), b = sound_quotient(pR, rR, gamma);
  return sqrt_core(a > b ? a : b);
}
FV2D_SF_CALL double sound_rare(double p, double r, double gamma) { return sqrt_rn(div_rn(mul_rn(p, gamma), r)); }
FV2D_SF_CALL double2 sound2(double pL, double rL, double pR, double rR, double gamma) {
  if (!sound_range(pL, rL, pR, rR, gamma))
    return make_double2(sound_rare(pL, rL, gamma), sound_rare(pR, rR, gamma));
  return make_double2(sqrt_core(sound_quotient(pL, rL, gamma)), sqrt_core(sound_quotient(pR, rR, gamma)));
}

}  // namespace softfp
}  // namespace fv2d
