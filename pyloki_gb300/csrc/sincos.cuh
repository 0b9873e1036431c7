// Sine and cosine of the Fourier folds' float32 angles and of 64 bins.
#pragma once

#include "loki_common.cuh"

namespace loki {

// cos and sin of 2 pi k / 64, the nearest floats.
__device__ constexpr float kCos64[17] = {
    1.0f, 0.99518472667219693f, 0.98078528040323043f, 0.95694033573220882f, 0.92387953251128674f,
    0.88192126434835505f, 0.83146961230254524f, 0.77301045336273699f, 0.70710678118654752f,
    0.63439328416364549f, 0.55557023301960218f, 0.47139673682599764f, 0.38268343236508977f,
    0.29028467725446233f, 0.19509032201612825f, 0.09801714032956060f, 0.0f};
__device__ __forceinline__ constexpr float cos64(int k) {
  k &= 63;
  if (k > 32) k = 64 - k;
  return k <= 16 ? kCos64[k] : -kCos64[32 - k];
}
__device__ __forceinline__ constexpr float sin64(int k) { return cos64(k + 48); }

// sin and cos of a float32 angle by Cody and Waite's additive reduction
// ("Software Manual for the Elementary Functions", 1980): 2 pi split into
// three float32 parts, the first two with 8 significant bits so that k times
// them is exact for |k| < 2^15 (angles up to about 2e5 rad), subtracted with
// fused multiply-adds; sincosf of the reduced angle then stays on its short
// path. The parts come from 2 pi to 60 digits: 0x1.92p+2 + 0x1.fbp-10 +
// 0x1.5110b4p-20 (their sum is 2 pi to 2e-14).
__device__ __forceinline__ void sincos_reduced(float a, float* s, float* c) {
  constexpr float kC1 = 0x1.92p+2f, kC2 = 0x1.fbp-10f, kC3 = 0x1.5110b4p-20f;
  const float k = rintf(__fmul_rn(a, 0.15915494f));
  if (fabsf(k) < 32768.0f) {
    float r = __fmaf_rn(-k, kC1, a);
    r = __fmaf_rn(-k, kC2, r);
    r = __fmaf_rn(-k, kC3, r);
    sincosf(r, s, c);
  } else {
    sincosf(a, s, c);
  }
}

// Sine and cosine of r, |r| < 0.86, by minimax polynomials on [-pi/4, pi/4] in
// r^2 (Remez exchange in float64, rounded: sin to 4e-9, cos to 1e-10 before
// rounding), turned by the quadrant q.
__device__ __forceinline__ void sincos_poly(float r, unsigned q, float* s, float* c) {
  const float r2 = __fmul_rn(r, r);
  float p = __fmaf_rn(r2, -0x1.994cfap-13f, 0x1.11075cp-7f);
  p = __fmaf_rn(r2, p, -0x1.555546p-3f);
  const float sr = __fmaf_rn(__fmul_rn(r, r2), p, r);
  float t = __fmaf_rn(r2, 0x1.9a00cep-16f, -0x1.6c0c86p-10f);
  t = __fmaf_rn(r2, t, 0x1.55554ap-5f);
  const float cr = __fmaf_rn(__fmul_rn(r2, r2), t, __fmaf_rn(r2, -0.5f, 1.0f));
  const float sv = q & 1u ? cr : sr, cv = q & 1u ? sr : cr;
  *s = __uint_as_float(__float_as_uint(sv) ^ ((q << 30) & 0x80000000u));
  *c = __uint_as_float(__float_as_uint(cv) ^ (((q + 1u) << 30) & 0x80000000u));
}

// The same for a caller that knows |a| < 2e5: reduction by pi / 2 in four
// parts (the first three with 7 significant bits, so k times them is exact for
// |k| < 2^17 and the subtractions are exact; the parts, truncations of pi / 2
// to 60 digits, sum to it within 6e-15). Both results are within 1.6 x 2^-24 of
// the exact values (1.56 over 1.2e7 angles): as accurate as sincosf there, in
// about half its instructions.
__device__ __forceinline__ void sincos_small(float a, float* s, float* c) {
  const float kf = __fmaf_rn(a, 0x1.45f306p-1f, 12582912.0f);  // 2^23 + 2^22: k in the low bits
  const float k = __fsub_rn(kf, 12582912.0f);
  float r = __fmaf_rn(-k, 0x1.9p+0f, a);
  r = __fmaf_rn(-k, 0x1.0cp-7f, r);
  r = __fmaf_rn(-k, 0x1.ecp-14f, r);
  r = __fmaf_rn(-k, 0x1.5110b4p-22f, r);
  sincos_poly(r, __float_as_uint(kf), s, c);
}

// For |a| < 1.6e6 (|k| < 2^20), as accurate: pi / 2 = C1 + C2 to 2^-49, C1 its
// nearest float. a and k C1 are multiples of 2^-23 (or, |a| < 1, of 2^-24) and
// differ by less than 1, so the first subtraction is exact and the second rounds
// once. k may be off by 0.043 before it is rounded: |r| < 0.86.
__device__ __forceinline__ void sincos_mid(float a, float* s, float* c) {
  const float kf = __fmaf_rn(a, 0x1.45f306p-1f, 12582912.0f);
  const float k = __fsub_rn(kf, 12582912.0f);
  const float r = __fmaf_rn(-k, -0x1.777a5cp-25f, __fmaf_rn(-k, 0x1.921fb6p+0f, a));
  sincos_poly(r, __float_as_uint(kf), s, c);
}

}  // namespace loki
