// FP64 division on the integer units.
//
// The GB300 has two FP64 lanes per SM and 64 integer ones: a warp's DFMA
// occupies the SM's FP64 pipe for 16 cycles, in which the integer units take
// 32 warp instructions.  An IEEE quotient costs about ten FP64 instructions,
// and the eliminations here need one to three of them per row, so the FP64
// solvers were bound by their divisions (FP64 pipe 86-89 % busy, 90-98 FP64
// instructions a row).  Here the reciprocal of the divisor's significand is
// formed in 64-bit fixed point (a single-precision seed, one third-order
// Newton-Raphson step) and multiplied by the numerator's significand, so a
// division issues no FP64 instruction at all; several quotients by one
// divisor share its reciprocal.  In place of the IEEE division in the same
// kernels: 16384 x 1024 CR 2939 -> 1456 us, 4096 x 1000 any-size 683 -> 257 us.
//
// Accuracy: the reciprocal is within 2^-60 of 1/b relative, the product is
// rounded to nearest once: the quotient is within (1/2 + 2^-7) ulp of a / b,
// exact where a / b is representable.  Zero, subnormal, infinite or NaN
// operands and quotients that leave the normal range take the IEEE division.
#pragma once
#include <cstdint>
#include <cstring>
#include <cuda_runtime.h>

namespace tridi {

#ifdef __CUDA_ARCH__
__device__ __forceinline__ float div64_seed(float f) {
  float r;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(f));
  return r;
}
// (a PTX move, so that the compiler does not see the value behind the bits:
// it would turn tests of the exponent field into FP64 compares)
__device__ __forceinline__ uint64_t div64_bits(double v) {
  uint64_t u;
  asm("mov.b64 %0, %1;" : "=l"(u) : "d"(v));
  return u;
}
__device__ __forceinline__ double div64_value(uint64_t v) { return __longlong_as_double((long long)v); }
__device__ __forceinline__ uint32_t div64_fbits(float v) { return __float_as_uint(v); }
__device__ __forceinline__ float div64_fvalue(uint32_t v) { return __uint_as_float(v); }
__device__ __forceinline__ uint64_t div64_mulhi(uint64_t a, uint64_t b) { return __umul64hi(a, b); }
#else
// host form, for checking the arithmetic without a GPU
inline float div64_seed(float f) { return 1.0f / f; }
inline uint64_t div64_bits(double v) { uint64_t u; memcpy(&u, &v, 8); return u; }
inline double div64_value(uint64_t u) { double v; memcpy(&v, &u, 8); return v; }
inline uint32_t div64_fbits(float v) { uint32_t u; memcpy(&u, &v, 4); return u; }
inline float div64_fvalue(uint32_t u) { float v; memcpy(&v, &u, 4); return v; }
inline uint64_t div64_mulhi(uint64_t a, uint64_t b) { return (uint64_t)(((unsigned __int128)a * b) >> 64); }
#endif

// The reciprocal of b: r / 2^64 = 1 / (2 m) for b's significand m in [1/2, 1),
// truncated to just below 2^64 for a power of two.
struct Inv64 {
  uint64_t r;
  double b;
};

__host__ __device__ __forceinline__ uint64_t reciprocal_q64(uint64_t bits) {
  const uint64_t M = (bits << 11) | 0x8000000000000000ull;  // significand in [2^63, 2^64)
  const uint32_t mh = (uint32_t)(M >> 32), ml = (uint32_t)M;
  // seed: y = Y0 / 2^32 near 1 / (2 m), relative error below 2^-21
  float y = div64_seed(div64_fvalue(0x3f800000u | ((mh >> 8) & 0x7fffffu)));
  y = y < 1.0f ? y : div64_fvalue(0x3f7fffffu);  // keep Y0 in 32 bits
  const uint32_t y0 = (div64_fbits(y) << 8) | 0x80000000u;
  // e = 1 - 2 m y in units of 2^-63
  const uint64_t s = (uint64_t)mh * y0 + (((uint64_t)ml * y0) >> 32);
  const int64_t e = (int64_t)(0x8000000000000000ull - s);
  // y (1 + e + e^2): what is left is e^3 < 2^-63
  const int32_t eh = (int32_t)(e >> 20);
  const int64_t e2 = e + (((int64_t)eh * eh) >> 23);
  const int32_t e2h = (int32_t)(e2 >> 32);
  const uint32_t e2l = (uint32_t)e2;
  const uint64_t corr = (uint64_t)(((int64_t)e2h * (int64_t)(uint64_t)y0) * 2) + (((uint64_t)e2l * y0) >> 31);
  return ((uint64_t)y0 << 32) + corr;
}

__host__ __device__ __forceinline__ Inv64 invert64(double b) { return Inv64{reciprocal_q64(div64_bits(b)), b}; }

// The IEEE quotient, for the operands that quotient_fast() refuses.  Out of
// line, with the bits passed as integers: rare, and any part of it that the
// compiler moved ahead of the test would cost FP64 issue at every division.
#ifdef __CUDACC__
static __device__ __noinline__ uint64_t quotient_ieee_bits(uint64_t a, uint64_t b) {
  return (uint64_t)__double_as_longlong(__ddiv_rn(__longlong_as_double((long long)a), __longlong_as_double((long long)b)));
}
#endif
__host__ __device__ __forceinline__ double quotient_ieee(double a, double b) {
#ifdef __CUDA_ARCH__
  return div64_value(quotient_ieee_bits(div64_bits(a), div64_bits(b)));
#else
  return a / b;
#endif
}

// a / v.b into q; false where an operand or the quotient is zero-divisor,
// subnormal, infinite or NaN (q is then meaningless).  A zero a is fine.
__host__ __device__ __forceinline__ bool quotient_fast(double a, const Inv64& v, double& q) {
  const uint64_t ba = div64_bits(a), bb = div64_bits(v.b);
  const uint32_t ha = (uint32_t)(ba >> 32), hb = (uint32_t)(bb >> 32);
  const int ea = (int)((ha >> 20) & 0x7ff), eb = (int)((hb >> 20) & 0x7ff);
  const uint64_t A = (ba << 11) | 0x8000000000000000ull;
  const uint64_t p = div64_mulhi(A, v.r);  // a's significand times 1 / (2 m): [2^62, 2^64)
  const uint32_t top = (uint32_t)(p >> 63);
  // to 53 bits, to nearest; a carry out of the significand moves the exponent
  const uint64_t t = ((p >> (9 + top)) + 1) >> 1;
  const int ex = ea - eb + 1022 + (int)top;  // biased exponent of the quotient
  const bool zero = (ba << 1) == 0;
  const uint64_t mag = zero ? 0 : ((uint64_t)(uint32_t)(ex - 1) << 52) + t;
  q = div64_value(((uint64_t)((ha ^ hb) & 0x80000000u) << 32) | mag);
  return (unsigned)(eb - 1) < 2046u && (zero || ((unsigned)(ea - 1) < 2046u && (unsigned)(ex - 1) < 2045u));
}

__host__ __device__ __forceinline__ double div64(double a, const Inv64& v) {
  double q;
  if (quotient_fast(a, v, q)) return q;
  return quotient_ieee(a, v.b);
}

// Three quotients by one divisor (a row divided by its diagonal): one
// reciprocal and one test for the rare case.
__host__ __device__ __forceinline__ void div64x3(double a, double c, double d, double b, double& qa, double& qc,
                                                 double& qd) {
  const Inv64 v = invert64(b);
  const bool fa = quotient_fast(a, v, qa), fc = quotient_fast(c, v, qc), fd = quotient_fast(d, v, qd);
  if (!(fa && fc && fd)) {
    qa = quotient_ieee(a, b);
    qc = quotient_ieee(c, b);
    qd = quotient_ieee(d, b);
  }
}

// Two quotients by one divisor.
__host__ __device__ __forceinline__ void div64x2(double c, double d, double b, double& qc, double& qd) {
  const Inv64 v = invert64(b);
  const bool fc = quotient_fast(c, v, qc), fd = quotient_fast(d, v, qd);
  if (!(fc && fd)) {
    qc = quotient_ieee(c, b);
    qd = quotient_ieee(d, b);
  }
}

}  // namespace tridi
