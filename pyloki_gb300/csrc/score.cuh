// Boxcar matched-filter scoring of one warp-tile of profiles held in shared
// memory (detection/scoring.py:42-165, 249-282).
//
// Layout: row r of the tile starts at tile + r * stride and holds the
// normalised profile in [0, nbins); the circular prefix sum is built in place
// and extended to nbins + wmax entries. stride is odd so that the 32 lanes,
// each walking its own row, hit 32 different banks.
//
// Each lane owns one row and runs the prefix sum sequentially in float32,
// exactly as circular_prefix_sum does, so the sums (and the S/N derived from
// them in float64) are bit-identical to the reference.
#pragma once

#include <float.h>

#include "loki_common.cuh"

namespace loki {

__host__ __device__ __forceinline__ int score_stride(int nbins, int wmax) {
  int s = nbins + (wmax > 0 ? wmax : 1);
  return (s & 1) ? s : s + 1;
}

// Circular prefix sum of length nbins + wmax, in place (scoring.py:42-71).
__device__ __forceinline__ float prefix_row(float* row, int nbins, int wmax) {
  float s = row[0];
  int i = 1;
  for (; i + 8 <= nbins; i += 8) {  // eight loads ahead of the eight stores
    float x[8];
#pragma unroll
    for (int k = 0; k < 8; ++k) x[k] = row[i + k];
#pragma unroll
    for (int k = 0; k < 8; ++k) row[i + k] = s = __fadd_rn(s, x[k]);
  }
  for (; i < nbins; ++i) {
    s = __fadd_rn(s, row[i]);
    row[i] = s;
  }
  const float last = s;
  const int nsum = nbins + wmax;
  if (nsum > nbins) {
    const int n_wraps = nsum / nbins;
    const int extra = nsum % nbins;
    for (int w = 1; w < n_wraps; ++w) {
      const float add = __fmul_rn((float)w, last);
      for (int j = 0; j < nbins; ++j) row[w * nbins + j] = __fadd_rn(row[j], add);
    }
    if (extra > 0) {
      const float add = __fmul_rn((float)n_wraps, last);
      for (int j = 0; j < extra; ++j) row[n_wraps * nbins + j] = __fadd_rn(row[j], add);
    }
  }
  return last;  // prefix_sum[nbins - 1] == total
}

// Largest differences P[i + w] - P[i] of N widths at once: the row is walked
// once for all of them. A NaN difference is passed over, as the reference's
// d > max does.
template <int N>
__device__ __forceinline__ void dmax_widths(const float* row, int nbins, const int (&w)[4],
                                            float (&m)[4]) {
#pragma unroll
  for (int q = 0; q < N; ++q) m[q] = -FLT_MAX;
#pragma unroll 4
  for (int i = 0; i < nbins; ++i) {
    const float p = row[i];
#pragma unroll
    for (int q = 0; q < N; ++q) m[q] = fmaxf(m[q], __fsub_rn(row[i + w[q]], p));
  }
}

// ---- fast path: nbins == 64, widths of a compiled series ----------------------
//
// The widths of a configuration are max(w + 1, floor(r w)) of the one before.
// For r = 2 (1, 2, 4, ...) and r = 1.5 (1, 2, 3, 4, 6, 9, ..., the default) up
// to 32 bins the prefix stays in registers and the differences have constant
// indices: 64 to 96 instructions a width, where the walk over a row in shared
// memory takes 200 (widths 1 to 9, score kernel of 64 pruning runs: 15.0 -> 13.7 ms).
//
// The reference's S/N of one width is RN32(RN64(RN64(hb*d) - RN64(b*T))) with
// d = max prefix difference and T = total (both float32). It is estimated in
// two-float FP32 (hb, b split into hi/lo floats, exact products by FMA, exact
// two-sum); when the estimate is farther than 2^-40 * max(|hb d|, |b T|) from
// an f32 rounding midpoint the rounding of the FP64 chain is certain,
// otherwise the FP64 chain is evaluated.
struct ScoreK {
  float hb_hi[LOKI_MAX_WIDTHS], hb_lo[LOKI_MAX_WIDTHS];
  float b_hi[LOKI_MAX_WIDTHS], b_lo[LOKI_MAX_WIDTHS];
  int pow2_64;  // nbins == 64 and widths == 1, 2, 4, ... (<= 32)
  int list64;   // nbins == 64: 1 as pow2_64, 2 widths == 1, 2, 3, 4, 6, 9, ... (<= 28)
  int inv_one;  // inv_stdnoise == 1
};

inline ScoreK make_score_k(const LokiScoreSpec& sp, int nbins) {
  ScoreK k;
  bool pow2 = nbins == 64 && sp.nwidths <= 6, seq15 = nbins == 64 && sp.nwidths <= 9;
  const int w15[9] = {1, 2, 3, 4, 6, 9, 13, 19, 28};
  for (int i = 0; i < sp.nwidths; ++i) {
    k.hb_hi[i] = (float)sp.hb[i];
    k.hb_lo[i] = (float)(sp.hb[i] - (double)k.hb_hi[i]);
    k.b_hi[i] = (float)sp.b[i];
    k.b_lo[i] = (float)(sp.b[i] - (double)k.b_hi[i]);
    if (sp.widths[i] != (1 << i)) pow2 = false;
    if (i < 9 && sp.widths[i] != w15[i]) seq15 = false;
  }
  k.pow2_64 = pow2 ? 1 : 0;
  k.list64 = pow2 ? 1 : seq15 ? 2 : 0;
  k.inv_one = sp.inv_stdnoise == 1.0 ? 1 : 0;
  return k;
}

// Exact FP64 chain; out of line so the compiler cannot evaluate it
// speculatively on the (common) fast path.
static __device__ __noinline__ float snr_exact(float d, float T, double hb, double b) {
  return __double2float_rn(__dsub_rn(__dmul_rn(hb, (double)d), __dmul_rn(b, (double)T)));
}

__device__ __forceinline__ float snr_fast(float d, float T, float hbh, float hbl, float bh,
                                          float bl, double hb, double b) {
  const float p1 = hbh * d;
  float e1 = fmaf(hbh, d, -p1);
  e1 = fmaf(hbl, d, e1);
  const float p2 = bh * T;
  float e2 = fmaf(bh, T, -p2);
  e2 = fmaf(bl, T, e2);
  const float s = p1 - p2;
  const float bb = s - p1;
  const float es = (p1 - (s - bb)) + (-p2 - bb);
  const float lo = (e1 - e2) + es;
  const float r = s + lo;
  const float res = (s - r) + lo;
  const unsigned bits = __float_as_uint(fabsf(r));
  const unsigned expo = bits >> 23;
  if (expo > 30 && expo < 255 && (bits & 0x7FFFFFu) != 0u) {
    const float half_ulp = __uint_as_float((expo - 24u) << 23);
    const float margin = fmaxf(fabsf(p1), fabsf(p2)) * 9.094947e-13f;  // 2^-40
    if (fabsf(res) < half_ulp - margin) return r;
  }
  return snr_exact(d, T, hb, b);
}

// Two IEEE round-to-nearest subtractions in one instruction (sm_100+ f32x2).
__device__ __forceinline__ void sub2(float a0, float a1, float b0, float b1, float& d0,
                                     float& d1) {
  unsigned long long a, b, d;
  asm("mov.b64 %0, {%1, %2};" : "=l"(a) : "f"(a0), "f"(a1));
  asm("mov.b64 %0, {%1, %2};" : "=l"(b) : "f"(b0), "f"(b1));
  asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
  asm("mov.b64 {%0, %1}, %2;" : "=f"(d0), "=f"(d1) : "l"(d));
}

// max of three; a NaN input is ignored like Python's max(acc, nan) == acc.
__device__ __forceinline__ float max3(float a, float b, float c) {
  float m;
  asm("max.f32 %0, %1, %2, %3;" : "=f"(m) : "f"(a), "f"(b), "f"(c));
  return m;
}

__device__ __forceinline__ unsigned long long pack2(float a, float b) {
  unsigned long long x;
  asm("mov.b64 %0, {%1, %2};" : "=l"(x) : "f"(a), "f"(b));
  return x;
}

__device__ __forceinline__ void unpack2(unsigned long long x, float& a, float& b) {
  asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(x));
}

// The prefix is held as 48 register pairs P2[k] = (P[2k], P[2k+1]); for even
// widths both operands of the packed subtraction are register pairs already.
template <int H>  // width W = 2H
__device__ __forceinline__ float dmax64_even(const unsigned long long (&P2)[48]) {
  float m = -FLT_MAX;
#pragma unroll
  for (int k = 0; k < 32; ++k) {
    unsigned long long d;
    asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(P2[k + H]), "l"(P2[k]));
    float d0, d1;
    unpack2(d, d0, d1);
    m = max3(m, d0, d1);
  }
  return m;
}

template <int W>  // odd
__device__ __forceinline__ float dmax64_odd(const unsigned long long (&P2)[48]) {
  float m = -FLT_MAX;
#pragma unroll
  for (int k = 0; k < 32; ++k) {
    float a0, a1, b0, b1, c0, c1;
    unpack2(P2[k], a0, a1);
    unpack2(P2[k + (W - 1) / 2], b0, b1);
    unpack2(P2[k + (W + 1) / 2], c0, c1);
    m = max3(m, __fsub_rn(b1, a0), __fsub_rn(c0, a1));
  }
  return m;
}

// Sequential prefix in registers, then the width scans with compile-time
// indices (no shared-memory traffic after the row is read once).
__device__ __forceinline__ void score_row64(const float* row, const LokiScoreSpec& sp,
                                                 const ScoreK& K, float* out) {
  unsigned long long P2[48];
  float s = row[0];
#pragma unroll
  for (int k = 0; k < 32; ++k) {
    const float s0 = k == 0 ? s : __fadd_rn(s, row[2 * k]);
    s = __fadd_rn(s0, row[2 * k + 1]);
    P2[k] = pack2(s0, s);
  }
  const float total = s;
  const unsigned long long tt = pack2(total, total);
#pragma unroll
  for (int k = 0; k < 16; ++k)  // circular extension: P[64 + j] = P[j] + total
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(P2[32 + k]) : "l"(P2[k]), "l"(tt));
  float best = -FLT_MAX;
  for (int iw = 0; iw < sp.nwidths; ++iw) {
    float dm;
    if (K.list64 == 1) {
      switch (iw) {
        case 0: dm = dmax64_odd<1>(P2); break;
        case 1: dm = dmax64_even<1>(P2); break;
        case 2: dm = dmax64_even<2>(P2); break;
        case 3: dm = dmax64_even<4>(P2); break;
        case 4: dm = dmax64_even<8>(P2); break;
        default: dm = dmax64_even<16>(P2); break;
      }
    } else {
      switch (iw) {
        case 0: dm = dmax64_odd<1>(P2); break;
        case 1: dm = dmax64_even<1>(P2); break;
        case 2: dm = dmax64_odd<3>(P2); break;
        case 3: dm = dmax64_even<2>(P2); break;
        case 4: dm = dmax64_even<3>(P2); break;
        case 5: dm = dmax64_odd<9>(P2); break;
        case 6: dm = dmax64_odd<13>(P2); break;
        case 7: dm = dmax64_odd<19>(P2); break;
        default: dm = dmax64_even<14>(P2); break;
      }
    }
    float s;
    if (K.inv_one) {
      s = snr_fast(dm, total, K.hb_hi[iw], K.hb_lo[iw], K.b_hi[iw], K.b_lo[iw], sp.hb[iw],
                   sp.b[iw]);
    } else {
      const double x = __dsub_rn(__dmul_rn(sp.hb[iw], (double)dm),
                                 __dmul_rn(sp.b[iw], (double)total));
      s = __double2float_rn(__dmul_rn(x, sp.inv_stdnoise));
    }
    if (sp.mode == 0) out[iw] = s;
    else if (s > best) best = s;
  }
  if (sp.mode != 0) out[0] = best;
}

// Score the row owned by this lane. mode 0 writes nwidths values at out,
// mode 1 writes the max over widths at out[0].
__device__ __forceinline__ void score_row(float* row, int nbins, const LokiScoreSpec& sp,
                                          const ScoreK& K, float* out) {
  const float total = prefix_row(row, nbins, sp.wmax);
  // (generic path: any nbins and width list, prefix in shared memory). With
  // stdnoise 1 the S/N is snr_fast's float, the rounding of the same float64
  // chain; the largest float is then the rounding of the largest float64.
  double best = -(double)FLT_MAX;
  float best_f = -FLT_MAX;
  for (int w0 = 0; w0 < sp.nwidths; w0 += 4) {
    int w[4];
    float m[4];
#pragma unroll
    for (int q = 0; q < 4; ++q) w[q] = sp.widths[min(w0 + q, sp.nwidths - 1)];
    // a single profile of 500 bins, kernel time: one width 14.6 us by four, 9 by itself
    const int left = sp.nwidths - w0;
    if (left == 1) dmax_widths<1>(row, nbins, w, m);
    else if (left == 2) dmax_widths<2>(row, nbins, w, m);
    else dmax_widths<4>(row, nbins, w, m);
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const int iw = w0 + q;
      if (iw >= sp.nwidths) break;
      if (K.inv_one) {
        const float f = snr_fast(m[q], total, K.hb_hi[iw], K.hb_lo[iw], K.b_hi[iw], K.b_lo[iw],
                                 sp.hb[iw], sp.b[iw]);
        if (sp.mode == 0) out[iw] = f;
        else if (f > best_f) best_f = f;
        continue;
      }
      // S/N of one width (scoring.py:131-138)
      const double s = __dmul_rn(__dsub_rn(__dmul_rn(sp.hb[iw], (double)m[q]),
                                           __dmul_rn(sp.b[iw], (double)total)),
                                 sp.inv_stdnoise);
      if (sp.mode == 0) out[iw] = __double2float_rn(s);
      else if (s > best) best = s;
    }
  }
  if (sp.mode != 0) out[0] = K.inv_one ? best_f : __double2float_rn(best);
}

// Normalised bin j of a complex fold: the inverse transform of both components
// (tw: cos, then sin, of 2 pi r / nbins), then e / sqrt(v).
__device__ __forceinline__ float norm_bin_complex(const float2* __restrict__ fold, int j,
                                                  int nbins, int nbf,
                                                  const float* __restrict__ tw) {
  float val[2];
  for (int c = 0; c < 2; ++c) {
    const float2* x = fold + c * nbf;
    float acc = x[0].x;
    int r = 0;
    for (int m = 1; m < nbf; ++m) {
      // the imaginary parts of the DC and (for even nbins) Nyquist terms are
      // ignored; other terms count twice
      r += j;
      if (r >= nbins) r -= nbins;
      const float cth = tw[r], s = tw[nbins + r];
      const float2 xm = x[m];
      if (2 * m == nbins) {
        acc = __fmaf_rn(xm.x, cth, acc);
      } else {
        acc = __fmaf_rn(2.0f * xm.x, cth, acc);
        acc = __fmaf_rn(-2.0f * xm.y, s, acc);
      }
    }
    val[c] = __fdiv_rn(acc, (float)nbins);
  }
  return __fdiv_rn(val[0], __fsqrt_rn(val[1]));
}

}  // namespace loki
