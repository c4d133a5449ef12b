// sr_math.cuh — the evaluator's own single-precision sin, cos and log, and paired
// division, reciprocal and square root.
//
// CUDA's accurate sinf / cosf / logf are general-purpose routines (each with
// a slow path for arguments its fast path cannot reduce) that cost 30+
// instructions a datapoint and, DPT times inlined into the interpreter's
// dispatch switch, overflow the instruction cache, so the interpreter had to
// call them out of line.  These versions are short enough to be expanded at
// their switch case:
//
//   * sin / cos: Cody and Waite's argument reduction (W. J. Cody, W. Waite,
//     Software Manual for the Elementary Functions, 1980) by pi/2, with a
//     three-part float constant applied by fused multiply-adds, and minimax
//     polynomials on [-pi/4, pi/4] (Remez exchange algorithm, coefficients
//     derived by csrc/gen_minimax.py): sin r = r + r^3 S(r^2), cos r = 1 +
//     r^2 (-1/2 + r^2 C(r^2)), S and C of degree 2; the quadrant picks the
//     polynomial and the sign.  Arguments with |x| > 32768 and non-finite
//     ones go to CUDA's sinf / cosf, out of line.
//   * log: x = 2^e m with m in [sqrt(1/2), sqrt(2)), f = m - 1 (exact),
//     log x = e ln2 + f - f^2/2 + f^3 R(f) (R of degree 7, minimax, same
//     script), ln2 split in two so that e * ln2_hi is exact; subnormal
//     arguments are scaled by 2^23 first.
//
// The interpreter evaluates two datapoints at once with the paired FP32
// instructions of sm_100 (fma.rn.f32x2 and friends: sincos_parts2,
// sr_log_normal2); each half is the same correctly rounded operation as the
// scalar form, so both forms give identical results.
//
// Their accuracy is measured on every float argument against the correctly
// rounded value (sr_check_math, tests/test_gpu_math.py) and is the device
// column of the parity rule's error table.  Every kernel of this library that
// evaluates these operators calls these functions, so results do not depend
// on which kernel or dispatch path evaluates an operator.
#pragma once
#include <cuda_runtime.h>
#include <math.h>

namespace sr {
namespace {  // one copy per kernel translation unit

// pi/2 = kPio2Hi + kPio2Mid + kPio2Lo to about 1e-23.
constexpr float kTwoOverPi = 0.636619772f;
constexpr float kPio2Hi = 1.57079637f;
constexpr float kPio2Mid = -4.37113883e-08f;
constexpr float kPio2Lo = -1.71512451e-15f;
constexpr float kSinCosFastMax = 32768.0f;  // larger |x|: CUDA's sinf / cosf
// 1.5 * 2^23: adding it rounds a float of magnitude below 2^22 to an integer
// held in the low mantissa bits.
constexpr float kRoundMagic = 12582912.0f;

// sin r = r + r^3 (kS0 + z (kS1 + z kS2)), z = r^2
constexpr float kS0 = -0.166666546743f;
constexpr float kS1 = 0.00833210095313f;
constexpr float kS2 = -0.000195039631257f;
// cos r = 1 + z (-1/2 + z (kC0 + z (kC1 + z kC2)))
constexpr float kC0 = 0.0416666546518f;
constexpr float kC1 = -0.00138876543845f;
constexpr float kC2 = 2.4463837439e-05f;

// Reduced argument, quadrant and both polynomials of x (|x| <= 32768).
struct SinCosParts {
  float s, c;  // sin r, cos r
  int q;       // quadrant (x = q pi/2 + r)
};

__device__ __forceinline__ SinCosParts sincos_parts(float x) {
  const float t = fmaf(x, kTwoOverPi, kRoundMagic);
  const float j = __fsub_rn(t, kRoundMagic);
  SinCosParts p;
  p.q = __float_as_int(t);  // low bits: j mod 2^22
  float r = fmaf(-j, kPio2Hi, x);
  r = fmaf(-j, kPio2Mid, r);
  r = fmaf(-j, kPio2Lo, r);
  const float z = __fmul_rn(r, r);
  float ps = fmaf(kS2, z, kS1);
  ps = fmaf(ps, z, kS0);
  p.s = fmaf(__fmul_rn(r, z), ps, r);
  float pc = fmaf(kC2, z, kC1);
  pc = fmaf(pc, z, kC0);
  pc = fmaf(pc, z, -0.5f);
  p.c = fmaf(z, pc, 1.0f);
  return p;
}

// sin (q_offset 0) or cos (q_offset 1) from the parts.
__device__ __forceinline__ float sincos_pick(const SinCosParts &p, int q_offset) {
  const int q = p.q + q_offset;
  const float y = (q & 1) ? p.c : p.s;
  return __int_as_float(__float_as_int(y) ^ ((q & 2) << 30));
}

__device__ __forceinline__ bool sincos_fast_ok(float x) { return fabsf(x) <= kSinCosFastMax; }

__device__ __noinline__ float sincos_slow(float x, int q_offset) {
  return q_offset ? cosf(x) : sinf(x);
}

__device__ __forceinline__ float sr_sinf(float x) {
  if (!sincos_fast_ok(x)) return sincos_slow(x, 0);
  const float y = sincos_pick(sincos_parts(x), 0);
  return x == 0.0f ? x : y;  // sin(-0) = -0
}

__device__ __forceinline__ float sr_cosf(float x) {
  if (!sincos_fast_ok(x)) return sincos_slow(x, 1);
  return sincos_pick(sincos_parts(x), 1);
}

// sin and cos of the same argument (one reduction): the values sr_sinf and
// sr_cosf return.
__device__ __forceinline__ void sr_sincosf(float x, float *s, float *c) {
  if (!sincos_fast_ok(x)) {
    *s = sincos_slow(x, 0);
    *c = sincos_slow(x, 1);
    return;
  }
  const SinCosParts p = sincos_parts(x);
  const float sv = sincos_pick(p, 0);
  *s = x == 0.0f ? x : sv;
  *c = sincos_pick(p, 1);
}

// Two arguments at once in paired FP32 operations (fma.rn.f32x2 and friends:
// each half is the same correctly rounded operation as the scalar form, so
// the results are those of sincos_parts).
__device__ __forceinline__ float2 f2(float a) { return make_float2(a, a); }
__device__ __forceinline__ void sincos_parts2(float2 x, SinCosParts &p0, SinCosParts &p1) {
  const float2 t = __ffma2_rn(x, f2(kTwoOverPi), f2(kRoundMagic));
  const float2 j = __fadd2_rn(t, f2(-kRoundMagic));
  p0.q = __float_as_int(t.x);
  p1.q = __float_as_int(t.y);
  float2 r = __ffma2_rn(j, f2(-kPio2Hi), x);
  r = __ffma2_rn(j, f2(-kPio2Mid), r);
  r = __ffma2_rn(j, f2(-kPio2Lo), r);
  const float2 z = __fmul2_rn(r, r);
  float2 ps = __ffma2_rn(f2(kS2), z, f2(kS1));
  ps = __ffma2_rn(ps, z, f2(kS0));
  const float2 s = __ffma2_rn(__fmul2_rn(r, z), ps, r);
  float2 pc = __ffma2_rn(f2(kC2), z, f2(kC1));
  pc = __ffma2_rn(pc, z, f2(kC0));
  pc = __ffma2_rn(pc, z, f2(-0.5f));
  const float2 c = __ffma2_rn(z, pc, f2(1.0f));
  p0.s = s.x; p1.s = s.y; p0.c = c.x; p1.c = c.y;
}

// Largest and smallest magnitude of N values (at least 2), two values an
// instruction; _nan: NaN when one is, otherwise NaNs are passed over.
__device__ __forceinline__ float max3_abs(float a, float b, float c) {
  float r;
  asm("max.abs.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
  return r;
}
__device__ __forceinline__ float min3_abs(float a, float b, float c) {
  float r;
  asm("min.abs.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
  return r;
}
__device__ __forceinline__ float max3_abs_nan(float a, float b, float c) {
  float r;
  asm("max.NaN.abs.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
  return r;
}
template <int N>
__device__ __forceinline__ float max_abs(const float (&v)[N]) {
  float m = max3_abs(v[0], v[1], v[N > 2 ? 2 : 1]);
#pragma unroll
  for (int k = 3; k < N; k += 2) m = max3_abs(m, v[k], v[k + 1 < N ? k + 1 : k]);
  return m;
}
template <int N>
__device__ __forceinline__ float max_abs_nan(const float (&v)[N]) {
  float m = max3_abs_nan(v[0], v[1], v[N > 2 ? 2 : 1]);
#pragma unroll
  for (int k = 3; k < N; k += 2) m = max3_abs_nan(m, v[k], v[k + 1 < N ? k + 1 : k]);
  return m;
}
template <int N>
__device__ __forceinline__ float min_abs(const float (&v)[N]) {
  float m = min3_abs(v[0], v[1], v[N > 2 ? 2 : 1]);
#pragma unroll
  for (int k = 3; k < N; k += 2) m = min3_abs(m, v[k], v[k + 1 < N ? k + 1 : k]);
  return m;
}

// Correctly rounded division and square root of two values at once for
// arguments of middling magnitude, in paired operations: an approximate
// reciprocal (reciprocal square root), one Newton step, and exact residuals by
// fused multiply-add (P. Markstein, IA-64 and Elementary Functions, 2000;
// J.-M. Muller et al., Handbook of Floating-Point Arithmetic, ch. 4).  Within
// the ranges below no intermediate over- or underflows, so the last step
// rounds correctly, as __fdiv_rn and __fsqrt_rn do; every other argument goes to
// those.  tests/test_gpu_interpreter.py compares them with IEEE results on the
// quotients closest to a rounding boundary and on every mantissa.
constexpr float kDivMin = 8.67361738e-19f, kDivMax = 1.15292150e18f;     // 2^-60, 2^60
constexpr float kSqrtMin = 7.88860905e-31f, kSqrtMax = 1.26765060e30f;   // 2^-100, 2^100

__device__ __forceinline__ float rcp_approx(float x) {
  float r;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
}
__device__ __forceinline__ float rsqrt_approx(float x) {
  float r;
  asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
}

// a / b, |a| and |b| in [kDivMin, kDivMax] (NaN gives NaN).
__device__ __forceinline__ float2 div2_mid(float2 a, float2 b) {
  const float2 nb = __fmul2_rn(b, f2(-1.0f));
  float2 r = make_float2(rcp_approx(b.x), rcp_approx(b.y));
  r = __ffma2_rn(r, __ffma2_rn(nb, r, f2(1.0f)), r);
  float2 q = __fmul2_rn(a, r);
  q = __ffma2_rn(__ffma2_rn(nb, q, a), r, q);
  return __ffma2_rn(__ffma2_rn(nb, q, a), r, q);
}

// 1 / b, |b| in [kDivMin, kDivMax] (NaN gives NaN).
__device__ __forceinline__ float2 rcp2_mid(float2 b) {
  const float2 nb = __fmul2_rn(b, f2(-1.0f));
  float2 r = make_float2(rcp_approx(b.x), rcp_approx(b.y));
  r = __ffma2_rn(r, __ffma2_rn(nb, r, f2(1.0f)), r);
  const float2 q = __ffma2_rn(__ffma2_rn(nb, r, f2(1.0f)), r, r);
  return __ffma2_rn(__ffma2_rn(nb, q, f2(1.0f)), r, q);
}

// a / b into a and 1 / b into r: both from one reciprocal, the same values as
// div2_mid and rcp2_mid.
__device__ __forceinline__ void div_rcp2_mid(float2 &a, float2 b, float2 &r) {
  const float2 nb = __fmul2_rn(b, f2(-1.0f));
  r = make_float2(rcp_approx(b.x), rcp_approx(b.y));
  r = __ffma2_rn(r, __ffma2_rn(nb, r, f2(1.0f)), r);
  float2 q = __fmul2_rn(a, r);
  q = __ffma2_rn(__ffma2_rn(nb, q, a), r, q);
  a = __ffma2_rn(__ffma2_rn(nb, q, a), r, q);
  q = __ffma2_rn(__ffma2_rn(nb, r, f2(1.0f)), r, r);
  r = __ffma2_rn(__ffma2_rn(nb, q, f2(1.0f)), r, q);
}

// sqrt(x), x in [kSqrtMin, kSqrtMax] (NaN gives NaN).
__device__ __forceinline__ float2 sqrt2_mid(float2 x) {
  const float2 nx = __fmul2_rn(x, f2(-1.0f));
  const float2 y = make_float2(rsqrt_approx(x.x), rsqrt_approx(x.y));
  float2 g = __fmul2_rn(x, y);          // sqrt x
  float2 nh = __fmul2_rn(y, f2(-0.5f)); // -1 / (2 sqrt x)
  const float2 e = __ffma2_rn(nh, g, f2(0.5f));
  g = __ffma2_rn(g, e, g);
  nh = __ffma2_rn(nh, e, nh);
  return __ffma2_rn(__ffma2_rn(g, g, nx), nh, g);
}

// log(1 + f) = f + f^2 (-1/2 + f R(f)), R(f) = kR0 + f (kR1 + ... f kR7)
constexpr float kR0 = 0.333333317078f;
constexpr float kR1 = -0.250008210321f;
constexpr float kR2 = 0.20001226863f;
constexpr float kR3 = -0.166233574103f;
constexpr float kR4 = 0.142017583522f;
constexpr float kR5 = -0.13160182163f;
constexpr float kR6 = 0.127615745496f;
constexpr float kR7 = -0.0763449398631f;
// ln 2 = kLn2Hi + kLn2Lo; kLn2Hi has 10 trailing zero bits, so e * kLn2Hi
// is exact for every exponent e.
constexpr float kLn2Hi = 0.693115234f;
constexpr float kLn2Lo = 3.19461833e-05f;

// log(a) for a >= 0 (+inf and NaN pass through, log(0) = -inf).
__device__ __forceinline__ float sr_log_nonneg(float a) {
  const bool sub = a < 1.17549435e-38f;
  const float as = sub ? __fmul_rn(a, 8388608.0f) : a;
  const int ia = __float_as_int(as);
  // e such that as / 2^e lies in [sqrt(1/2), sqrt(2)); 0x3f3504f3 is
  // sqrt(1/2) rounded to float.
  const int e = (ia - 0x3f3504f3) >> 23;
  const float m = __int_as_float(ia - (e << 23));
  const float f = __fsub_rn(m, 1.0f);
  const float ef = static_cast<float>(sub ? e - 23 : e);
  float p = fmaf(kR7, f, kR6);
  p = fmaf(p, f, kR5);
  p = fmaf(p, f, kR4);
  p = fmaf(p, f, kR3);
  p = fmaf(p, f, kR2);
  p = fmaf(p, f, kR1);
  p = fmaf(p, f, kR0);
  p = fmaf(p, f, -0.5f);
  const float y = fmaf(__fmul_rn(f, f), p, f);
  const float r = fmaf(ef, kLn2Hi, fmaf(ef, kLn2Lo, y));
  return (a == 0.0f) ? __int_as_float(0xff800000) : (a < INFINITY ? r : a);
}

// sr_log_nonneg of two positive normal arguments: no scaling, no special cases
// (the exponent becomes a float by adding it to the low bits of 1.5 * 2^23).
__device__ __forceinline__ float2 sr_log_normal2(float a0, float a1) {
  const int ia0 = __float_as_int(a0), ia1 = __float_as_int(a1);
  const int k0 = ia0 - 0x3f3504f3, k1 = ia1 - 0x3f3504f3;
  const float2 m = make_float2(__int_as_float(ia0 - (k0 & 0xff800000)),
                               __int_as_float(ia1 - (k1 & 0xff800000)));
  const float2 f = __fadd2_rn(m, f2(-1.0f));
  const int magic = __float_as_int(kRoundMagic);
  const float2 ef = __fadd2_rn(make_float2(__int_as_float((k0 >> 23) + magic),
                                           __int_as_float((k1 >> 23) + magic)),
                               f2(-kRoundMagic));
  float2 p = __ffma2_rn(f2(kR7), f, f2(kR6));
  p = __ffma2_rn(p, f, f2(kR5));
  p = __ffma2_rn(p, f, f2(kR4));
  p = __ffma2_rn(p, f, f2(kR3));
  p = __ffma2_rn(p, f, f2(kR2));
  p = __ffma2_rn(p, f, f2(kR1));
  p = __ffma2_rn(p, f, f2(kR0));
  p = __ffma2_rn(p, f, f2(-0.5f));
  const float2 y = __ffma2_rn(__fmul2_rn(f, f), p, f);
  return __ffma2_rn(ef, f2(kLn2Hi), __ffma2_rn(ef, f2(kLn2Lo), y));
}
constexpr float kMinNormal = 1.17549435e-38f;

// logf semantics: NaN for negative arguments.
__device__ __forceinline__ float sr_logf(float x) {
  return x < 0.0f ? __int_as_float(0x7fc00000) : sr_log_nonneg(x);
}

// Protected log (reference LOOSE_LOG): -1e9 at 0, else log|x|.
__device__ __forceinline__ float sr_loose_logf(float x) {
  return x == 0.0f ? -1e9f : sr_log_nonneg(fabsf(x));
}

}  // namespace
}  // namespace sr
