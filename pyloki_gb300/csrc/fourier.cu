// Fourier-domain FFA (use_fourier=True): complex brute fold, complex DP level
// with fractional phase shifts, and the inverse-FFT fold norm.
//
// Profiles are (2, nbins_f) complex64 rows, nbins_f = nbins / 2 + 1, stored
// as float2 (re, im). The arithmetic follows the reference's float32 /
// complex64 expressions; its BLAS sgemm, numpy cos/sin and pocketfft inverse
// transform are not reproduced bit for bit, so this path is compared with the
// reference to a stated float32 tolerance.
#include <algorithm>

#include "loki_common.cuh"
#include "resolve.cuh"
#include "score.cuh"
#include "sincos.cuh"

namespace loki {

// brutefold_start_complex_opt (core/fold.py:395-481): for every (segment,
// frequency, harmonic h) the DFT sum_t x[t] exp(-2 pi i f_h t tsamp) of both
// components, f_h = float32(f * h), the angle formed in float32 as
// f_h * float32(t * float32(-2 pi tsamp)); then the t_ref phase correction
// exp(i float32(2 pi t_ref) f_h). One thread owns one (frequency, harmonic)
// and kSegs segments, so each basis value serves kSegs segments.
constexpr int kSegs = 16;

__global__ void __launch_bounds__(128)
brutefold_complex_kernel(const float* __restrict__ ts_e, const float* __restrict__ ts_v,
                         const double* __restrict__ freqs, int64_t nfreq, int64_t seg_len,
                         int64_t nseg, int nbf, float tfac, float corr_factor,
                         float2* __restrict__ fold) {
  const int64_t ncomb = nfreq * nbf;
  const int64_t comb = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  const int64_t s0 = (int64_t)blockIdx.y * kSegs;
  if (comb >= ncomb) return;
  const int64_t fi = comb / nbf;
  const int h = (int)(comb - fi * nbf);
  const float fh = (float)(freqs[fi] * (double)h);
  const int ns = (int)std::min<int64_t>(kSegs, nseg - s0);
  float er[kSegs], ei[kSegs], vr[kSegs], vi[kSegs];
#pragma unroll
  for (int k = 0; k < kSegs; ++k) er[k] = ei[k] = vr[k] = vi[k] = 0.0f;
  // ts_v NULL: all ones, so every segment's variance sums are the running sums
  // of the basis values (fmaf(1, c, acc) = acc + c), taken once in vr[0]/vi[0]
  const bool unit = ts_v == nullptr;
  int64_t t = 0;
  // four samples per step with 16-byte (broadcast) loads of each segment;
  // every accumulator still takes its terms in sample order
  const bool vec = (seg_len & 3) == 0 &&
                   ((reinterpret_cast<uintptr_t>(ts_e) | reinterpret_cast<uintptr_t>(ts_v)) &
                    15) == 0;
  if (unit && vec) {
    for (; t < seg_len; t += 4) {
      float sn[4], cs[4];
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const float tv = __fmul_rn((float)(t + q), tfac);
        sincos_reduced(__fmul_rn(fh, tv), &sn[q], &cs[q]);
        vr[0] = fmaf(1.0f, cs[q], vr[0]);
        vi[0] = fmaf(1.0f, sn[q], vi[0]);
      }
#pragma unroll
      for (int k = 0; k < kSegs; ++k) {
        if (k < ns) {
          const float4 xe =
              __ldg(reinterpret_cast<const float4*>(ts_e + (s0 + k) * seg_len + t));
          const float e4[4] = {xe.x, xe.y, xe.z, xe.w};
#pragma unroll
          for (int q = 0; q < 4; ++q) {
            er[k] = fmaf(e4[q], cs[q], er[k]);
            ei[k] = fmaf(e4[q], sn[q], ei[k]);
          }
        }
      }
    }
  }
  if (vec && !unit) {
    for (; t < seg_len; t += 4) {
      float sn[4], cs[4];
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const float tv = __fmul_rn((float)(t + q), tfac);
        sincos_reduced(__fmul_rn(fh, tv), &sn[q], &cs[q]);
      }
#pragma unroll
      for (int k = 0; k < kSegs; ++k) {
        if (k < ns) {
          const int64_t at = (s0 + k) * seg_len + t;
          const float4 xe = __ldg(reinterpret_cast<const float4*>(ts_e + at));
          const float4 xv = __ldg(reinterpret_cast<const float4*>(ts_v + at));
          const float e4[4] = {xe.x, xe.y, xe.z, xe.w}, v4[4] = {xv.x, xv.y, xv.z, xv.w};
#pragma unroll
          for (int q = 0; q < 4; ++q) {
            er[k] = fmaf(e4[q], cs[q], er[k]);
            ei[k] = fmaf(e4[q], sn[q], ei[k]);
            vr[k] = fmaf(v4[q], cs[q], vr[k]);
            vi[k] = fmaf(v4[q], sn[q], vi[k]);
          }
        }
      }
    }
  }
  for (; t < seg_len; ++t) {
    const float tv = __fmul_rn((float)t, tfac);
    const float ang = __fmul_rn(fh, tv);
    float sn, cs;
    sincos_reduced(ang, &sn, &cs);
    if (unit) {
      vr[0] = fmaf(1.0f, cs, vr[0]);
      vi[0] = fmaf(1.0f, sn, vi[0]);
    }
#pragma unroll
    for (int k = 0; k < kSegs; ++k) {
      if (k < ns) {
        const int64_t at = (s0 + k) * seg_len + t;
        const float xe = __ldg(ts_e + at);
        er[k] = fmaf(xe, cs, er[k]);
        ei[k] = fmaf(xe, sn, ei[k]);
        if (!unit) {
          const float xv = __ldg(ts_v + at);
          vr[k] = fmaf(xv, cs, vr[k]);
          vi[k] = fmaf(xv, sn, vi[k]);
        }
      }
    }
  }
  if (unit) {
#pragma unroll
    for (int k = 1; k < kSegs; ++k) {
      vr[k] = vr[0];
      vi[k] = vi[0];
    }
  }
  // correction phasor exp(i * float32(corr_factor * f_h)), complex64 multiply
  const float th = __fmul_rn(corr_factor, fh);
  float cs_c, sn_c;
  sincos_reduced(th, &sn_c, &cs_c);
#pragma unroll
  for (int k = 0; k < kSegs; ++k) {  // constant indices keep the sums in registers
    if (k >= ns) break;
    float2* row = fold + ((s0 + k) * nfreq + fi) * 2 * nbf;
    row[h] = make_float2(__fsub_rn(__fmul_rn(er[k], cs_c), __fmul_rn(ei[k], sn_c)),
                         __fadd_rn(__fmul_rn(er[k], sn_c), __fmul_rn(ei[k], cs_c)));
    row[nbf + h] = make_float2(__fsub_rn(__fmul_rn(vr[k], cs_c), __fmul_rn(vi[k], sn_c)),
                               __fadd_rn(__fmul_rn(vr[k], sn_c), __fmul_rn(vi[k], cs_c)));
  }
}

__device__ __forceinline__ float2 cmul(float2 a, float2 b) {
  return make_float2(__fsub_rn(__fmul_rn(a.x, b.x), __fmul_rn(a.y, b.y)),
                     __fadd_rn(__fmul_rn(a.x, b.y), __fmul_rn(a.y, b.x)));
}

// Rotation step of shift_add_complex (core/common.py:344-372): the angle
// float32(float32(-2 pi) * shift) / nbins and its unit phasor.
__device__ __forceinline__ float2 shift_phasor(float shift, int nbins) {
  const float step = __fdiv_rn(__fmul_rn((float)(-2.0 * 3.14159265358979323846), shift),
                               (float)nbins);
  float sn, cs;
  sincosf(step, &sn, &cs);
  return make_float2(cs, sn);
}

// One complex DP level (dynamic/dyn_pffa.py:435-489 with shift_add_complex):
// thread per (output segment, parameter set, component); the plan gives the
// tail / head rows and their float32 phase shifts.
__global__ void ffa_level_complex_kernel(const LokiFFACoord* __restrict__ plan, int64_t Q,
                                         int64_t P_in, int64_t nseg_out, int nbins, int nbf,
                                         const float2* __restrict__ in,
                                         float2* __restrict__ out) {
  const int64_t k = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  const int64_t total = nseg_out * Q * 2;
  if (k >= total) return;
  const int c = (int)(k & 1);
  const int64_t q = (k >> 1) % Q;
  const int64_t ip = (k >> 1) / Q;
  const LokiFFACoord co = plan[q];
  const float2* t = in + (((2 * ip) * P_in + co.i_tail) * 2 + c) * nbf;
  const float2* h = in + (((2 * ip + 1) * P_in + co.i_head) * 2 + c) * nbf;
  float2* o = out + ((ip * Q + q) * 2 + c) * nbf;
  const float2 dt = shift_phasor(co.shift_tail, nbins);
  const float2 dh = shift_phasor(co.shift_head, nbins);
  float2 pt = make_float2(1.0f, 0.0f), ph = make_float2(1.0f, 0.0f);
  for (int j = 0; j < nbf; ++j) {
    const float2 a = cmul(t[j], pt), b = cmul(h[j], ph);
    o[j] = make_float2(__fadd_rn(a.x, b.x), __fadd_rn(a.y, b.y));
    pt = cmul(pt, dt);
    ph = cmul(ph, dh);
  }
}

// ---------------------------------------------------------------------------
// The same level without a plan table: each warp owns up to 32 output
// parameters and a range of segment pairs, a lane resolves one parameter (the
// two-float resolve of the time-domain levels; the float32 shift from the same
// two-float product), then the warp streams whole rows, lane by harmonic, with
// the phasor of every harmonic taken directly. A thread walking a row by phasor
// recurrence read 264-byte rows lane by lane, and the float64 plan cost a pass
// of its own: 8.7 ms for the six levels of a 2^20 search (15 100 frequencies at
// level 0), now 2.8 ms. Bound: HBM, the rows in and out once a level.
// ---------------------------------------------------------------------------

// Unit phasor exp(-2 pi i k shift / nbins): the turns k shift / nbins are formed
// with the product's rounding error kept (1 / nbins = inv_nb + inv_lo), so the
// angle is good to 2^-24.
__device__ __forceinline__ float2 harmonic_phasor(int k, float shift, float inv_nb,
                                                  float inv_lo) {
  const float p = __fmul_rn((float)k, shift);
  const float e = __fmaf_rn((float)k, shift, -p);
  const float t = __fmul_rn(p, inv_nb);
  const float et = __fmaf_rn(p, inv_lo, __fmaf_rn(p, inv_nb, -t));  // 0 for a power of two
  float fr = __fsub_rn(t, rintf(t));
  fr = __fadd_rn(fr, __fadd_rn(et, __fmul_rn(e, inv_nb)));
  float sn, cs;
  sincos_small(__fmul_rn(-6.2831853f, fr), &sn, &cs);
  return make_float2(cs, sn);
}

// Relative shift of one trial in bins: the plan's float32 value (the turns are
// kept as a float pair until the product with nbins is rounded).
__device__ __forceinline__ float trial_shift_bins(const OtherRes& o, float f_hi, float f_lo,
                                                  int nbins) {
  const float p = o.g_hi * f_hi;
  float e = fmaf(o.g_hi, f_hi, -p);
  e = fmaf(o.g_hi, f_lo, e);
  e = fmaf(o.g_lo, f_hi, e);
  const float a = p - floorf(p);  // exact
  float s = __fadd_rn(a, e);
  const float bb = __fsub_rn(s, a);
  const float lo = __fadd_rn(__fsub_rn(a, __fsub_rn(s, bb)), __fsub_rn(e, bb));
  s = __fsub_rn(s, floorf(s));
  const float x = __fmul_rn(s, (float)nbins);
  return __fadd_rn(x, __fmaf_rn(lo, (float)nbins, __fmaf_rn(s, (float)nbins, -x)));
}

constexpr int kClWarps = 8;

// kSlots x 32 float2 of a row (2 nbf); nbins 64: 66, three slots
template <int kSlots>
__global__ void __launch_bounds__(kClWarps * 32)
ffa_level_complex_rows_kernel(LokiFFALevel L, LevelK K, int pw, int64_t pairs,
                              const float2* __restrict__ in, float2* __restrict__ out,
                              int32_t* __restrict__ err) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int nbf = L.nbins / 2 + 1, row = 2 * nbf, n = L.nparams;
  int64_t Q = 1, P_in = 1;
  for (int d = 0; d < n; ++d) {
    Q *= L.counts_cur[d];
    P_in *= L.counts_prev[d];
  }
  const int64_t q0 = ((int64_t)blockIdx.x * kClWarps + warp) * pw;
  if (q0 >= Q) return;
  const int kmax = (int)min((int64_t)pw, Q - q0);
  int64_t my_t = 0, my_h = 0;
  float my_st = 0.0f, my_sh = 0.0f;
  bool my_ok = false;
  if (lane < kmax) {
    int64_t other, last;
    q_split(L, K, q0 + lane, other, last);
    const OtherRes ot = make_other(L, K, other, 0), oh = make_other(L, K, other, 1);
    const double f = L.param_arr[n - 1][last];
    float f_hi, f_lo;
    split2(f, &f_hi, &f_lo);
    const int64_t it = trial_index(ot, f, f_hi, f_lo, L, K);
    const int64_t ih = trial_index(oh, f, f_hi, f_lo, L, K);
    my_t = ot.prefix * L.in_width + it;
    my_h = oh.prefix * L.in_width + ih;
    my_ok = my_t < P_in && my_h < P_in;
    if (!my_ok) atomicOr(err, LOKI_DEVERR_WINDOW);
    my_st = trial_shift_bins(ot, f_hi, f_lo, L.nbins);
    my_sh = trial_shift_bins(oh, f_hi, f_lo, L.nbins);
  }
  const float inv_nb = 1.0f / (float)L.nbins;
  const float inv_lo = (float)(1.0 / (double)L.nbins - (double)inv_nb);
  const int64_t ip0 = blockIdx.y * pairs, ip1 = min(ip0 + pairs, L.nseg_in / 2);
  for (int k = 0; k < kmax; ++k) {
    const int64_t t = __shfl_sync(0xFFFFFFFFu, my_t, k), h = __shfl_sync(0xFFFFFFFFu, my_h, k);
    const float st = __shfl_sync(0xFFFFFFFFu, my_st, k), sh = __shfl_sync(0xFFFFFFFFu, my_sh, k);
    if (!__shfl_sync(0xFFFFFFFFu, my_ok, k)) continue;
    float2 pt[kSlots], ph[kSlots];
#pragma unroll
    for (int u = 0; u < kSlots; ++u) {
      const int e = lane + 32 * u, m = e < nbf ? e : e - nbf;
      if (e < row) {
        pt[u] = harmonic_phasor(m, st, inv_nb, inv_lo);
        ph[u] = harmonic_phasor(m, sh, inv_nb, inv_lo);
      }
    }
    const float2* tp = in + ((2 * ip0) * P_in + t) * row + lane;
    const float2* hp = in + ((2 * ip0 + 1) * P_in + h) * row + lane;
    float2* op = out + (ip0 * Q + q0 + k) * row + lane;
    for (int64_t ip = ip0; ip < ip1; ++ip) {
      float2 a[kSlots], b[kSlots];
#pragma unroll
      for (int u = 0; u < kSlots; ++u)
        if (lane + 32 * u < row) {
          a[u] = __ldg(tp + 32 * u);
          b[u] = __ldg(hp + 32 * u);
        }
#pragma unroll
      for (int u = 0; u < kSlots; ++u)
        if (lane + 32 * u < row) {
          const float2 x = cmul(a[u], pt[u]), y = cmul(b[u], ph[u]);
          op[32 * u] = make_float2(__fadd_rn(x.x, y.x), __fadd_rn(x.y, y.y));
        }
      tp += 2 * P_in * row;
      hp += 2 * P_in * row;
      op += Q * row;
    }
  }
}

// ---------------------------------------------------------------------------
// Final folds of 64 bins to S/N in one pass: rows staged in shared memory, a
// thread per fold makes both inverse transforms in registers (a 32-point
// complex transform of the packed coefficients), normalises and scores. The
// table-driven transform (fold_norm_complex_kernel) takes 4 224 multiply-adds
// a fold and a pass over the normalised profiles: 10.1 + 0.4 ms for 3.87e6
// folds and 5 widths against 1.1 ms here. Bound: instruction issue (about 4 000 a fold).
// ---------------------------------------------------------------------------

constexpr int kSnrThreads = 64;
constexpr int kSnrRow = 67;  // float2 of a staged fold (66) and one of padding

// In-place inverse transform (positive exponent, unscaled) of 2^LOG complex
// values in registers, decimation in frequency; the output is bit-reversed.
template <int LOG>
__device__ __forceinline__ void ifft_dif(float2 (&z)[1 << LOG]) {
#pragma unroll
  for (int s = LOG; s >= 1; --s) {
    const int half = 1 << (s - 1);
#pragma unroll
    for (int i = 0; i < (1 << LOG) / 2; ++i) {
      const int j = i & (half - 1), a = ((i >> (s - 1)) << s) + j, b = a + half;
      const float2 u = z[a], v = z[b];
      z[a] = make_float2(u.x + v.x, u.y + v.y);
      const float dx = u.x - v.x, dy = u.y - v.y;
      const int k = j * (64 >> s);  // twiddle exp(2 pi i k / 64)
      if (k == 0) {
        z[b] = make_float2(dx, dy);
      } else if (k == 16) {
        z[b] = make_float2(-dy, dx);
      } else {
        const float c = cos64(k), w = sin64(k);
        z[b] = make_float2(fmaf(dx, c, -(dy * w)), fmaf(dx, w, dy * c));
      }
    }
  }
}

__device__ __forceinline__ constexpr int rev5(int k) {
  return ((k & 1) << 4) | ((k & 2) << 2) | (k & 4) | ((k & 8) >> 2) | ((k & 16) >> 4);
}

// x[2 n] + i x[2 n + 1] = z[rev5(n)] / 64 of the 33 coefficients X of a row:
// Z[k] = (X[k] + conj X[32 - k]) + i exp(2 pi i k / 64) (X[k] - conj X[32 - k]).
// The imaginary parts of the first and last coefficient are not used.
__device__ __forceinline__ void irfft64(const float2* __restrict__ X, float2 (&z)[32]) {
#pragma unroll
  for (int k = 0; k <= 16; ++k) {
    float2 a = X[k], b = X[32 - k];
    if (k == 0) a.y = b.y = 0.0f;
    const float2 s = make_float2(a.x + b.x, a.y - b.y);
    const float2 d = make_float2(a.x - b.x, a.y + b.y);
    const float c = cos64(k), w = sin64(k);
    // i (c + i w) d
    const float2 r = make_float2(fmaf(d.x, -w, -(d.y * c)), fmaf(d.x, c, -(d.y * w)));
    z[k] = make_float2(s.x + r.x, s.y + r.y);
    if (k > 0 && k < 16) z[32 - k] = make_float2(s.x - r.x, r.y - s.y);
  }
  ifft_dif<5>(z);
}

__global__ void __launch_bounds__(kSnrThreads)
fold_snr_complex64_kernel(const float2* __restrict__ folds, int64_t n, LokiScoreSpec sp,
                          ScoreK SK, float* __restrict__ out) {
  extern __shared__ float2 st[];  // [threads][kSnrRow]; later a prefix row of floats a thread
  const int tid = threadIdx.x;
  const int64_t p0 = (int64_t)blockIdx.x * kSnrThreads;
  const int rows = (int)min((int64_t)kSnrThreads, n - p0);
  for (int k = tid; k < rows * 66; k += kSnrThreads) {
    const int r = k / 66;
    st[r * kSnrRow + (k - r * 66)] = __ldg(folds + p0 * 66 + k);
  }
  __syncthreads();
  if (tid >= rows) return;  // no block-level synchronisation follows
  float2* row = st + tid * kSnrRow;
  float2 e[32], v[32];
  irfft64(row, e);
  irfft64(row + 33, v);
  // both transforms carry the factor 64, as numpy's irfft is divided by nbins
  float* x = reinterpret_cast<float*>(row);
#pragma unroll
  for (int k = 0; k < 32; ++k) {
    const float2 a = e[rev5(k)], b = v[rev5(k)];
    x[2 * k] = __fdiv_rn(a.x * (1.0f / 64.0f), __fsqrt_rn(b.x * (1.0f / 64.0f)));
    x[2 * k + 1] = __fdiv_rn(a.y * (1.0f / 64.0f), __fsqrt_rn(b.y * (1.0f / 64.0f)));
  }
  const int nout = sp.mode == 0 ? sp.nwidths : 1;
  if (SK.list64) score_row64(x, sp, SK, out + (size_t)(p0 + tid) * nout);
  else score_row(x, 64, sp, SK, out + (size_t)(p0 + tid) * nout);
}

// get_fold_norm for Fourier folds (ffa.py:401-411): irfft of each component
// (nbins real samples from nbins_f coefficients, computed in float64 with
// exact twiddles and rounded to float32), then e / sqrt(v).
// irfft (numpy, n = nbins) of each component, then e / sqrt(v). Twiddle
// factors cos/sin(2 pi r / nbins) depend only on r = (m j) mod nbins: a block
// fills a float32 table of nbins entries (float64 sincospi, rounded once) and
// every term reads it; the sums run in float32 with fused multiply-adds, as
// numpy's float32 transform of a complex64 fold does (float64 sums would
// leave the FP64 pipe, a small fraction of GB300's float32 rate, the limit).
__global__ void fold_norm_complex_kernel(const float2* __restrict__ folds, int64_t n, int nbins,
                                         int nbf, float* __restrict__ out) {
  extern __shared__ float tw[];  // [nbins] cos, [nbins] sin
  for (int r = threadIdx.x; r < nbins; r += blockDim.x) {
    double s, c;
    sincospi(2.0 * (double)r / (double)nbins, &s, &c);
    tw[r] = (float)c;
    tw[nbins + r] = (float)s;
  }
  __syncthreads();
  const int64_t k = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (k >= n * nbins) return;
  const int64_t p = k / nbins;
  const int j = (int)(k - p * nbins);
  out[k] = norm_bin_complex(folds + p * 2 * nbf, j, nbins, nbf, tw);
}

}  // namespace loki

using namespace loki;

extern "C" int loki_brutefold_complex(const float* ts_e, const float* ts_v, int64_t nsamps,
                                      const double* freqs, int64_t nfreqs, int64_t segment_len,
                                      int32_t nbins, double tsamp, double t_ref, void* fold_out,
                                      void* stream) {
  if (!ts_e || !freqs || !fold_out)  // ts_v NULL: all ones
    return set_error(LOKI_ERR_INVALID, "null pointer argument");
  if (nsamps <= 0 || nfreqs <= 0 || segment_len <= 0 || nbins < 2)
    return set_error(LOKI_ERR_INVALID, "bad sizes");
  if (nsamps % segment_len != 0)
    return set_error(LOKI_ERR_INVALID,
                     "the Fourier brute fold needs nsamps a multiple of segment_len");
  const int nbf = nbins / 2 + 1;
  const int64_t nseg = nsamps / segment_len;
  const int64_t ncomb = nfreqs * nbf;
  const float tfac = (float)(-2.0 * 3.14159265358979323846 * tsamp);
  const float corr = (float)(2.0 * 3.14159265358979323846 * t_ref);
  const int64_t gx = (ncomb + 127) / 128, gy = (nseg + kSegs - 1) / kSegs;
  if (gx > 0x7FFFFFFF || gy > 65535) return set_error(LOKI_ERR_UNSUPPORTED, "grid too large");
  note_launch();
  brutefold_complex_kernel<<<dim3((unsigned)gx, (unsigned)gy), 128, 0, (cudaStream_t)stream>>>(
      ts_e, ts_v, freqs, nfreqs, segment_len, nseg, nbf, tfac, corr,
      reinterpret_cast<float2*>(fold_out));
  return check_launch("brutefold_complex");
}

extern "C" int loki_ffa_level_complex(const LokiFFALevel* lvl, const LokiFFACoord* plan,
                                      const void* fold_in, void* fold_out, void* stream) {
  if (!lvl || !plan || !fold_in || !fold_out)
    return set_error(LOKI_ERR_INVALID, "null pointer argument");
  int64_t Q = 1, P_in = 1;
  for (int d = 0; d < lvl->nparams; ++d) {
    Q *= lvl->counts_cur[d];
    P_in *= lvl->counts_prev[d];
  }
  if (lvl->out_start != 0 || lvl->out_width != lvl->counts_cur[lvl->nparams - 1] ||
      lvl->in_start != 0 || lvl->in_width != lvl->counts_prev[lvl->nparams - 1])
    return set_error(LOKI_ERR_UNSUPPORTED, "Fourier levels are materialised whole");
  if (lvl->nseg_in < 2 || lvl->nseg_in % 2)
    return set_error(LOKI_ERR_INVALID, "nseg_in must be even");
  const int nbf = lvl->nbins / 2 + 1;
  const int64_t nseg_out = lvl->nseg_in / 2;
  const int64_t total = nseg_out * Q * 2;
  note_launch();
  ffa_level_complex_kernel<<<(unsigned)((total + 255) / 256), 256, 0, (cudaStream_t)stream>>>(
      plan, Q, P_in, nseg_out, lvl->nbins, nbf, reinterpret_cast<const float2*>(fold_in),
      reinterpret_cast<float2*>(fold_out));
  return check_launch("ffa_level_complex");
}

extern "C" int loki_fold_norm_complex(const void* folds, int64_t n, int32_t nbins, float* out,
                                      void* stream) {
  if (n < 0 || nbins < 2) return set_error(LOKI_ERR_INVALID, "bad sizes");
  if (n == 0) return LOKI_OK;
  if (!folds || !out) return set_error(LOKI_ERR_INVALID, "null pointer argument");
  const int64_t total = n * nbins;
  if (nbins > 8192) return set_error(LOKI_ERR_UNSUPPORTED, "nbins above 8192");
  note_launch();
  fold_norm_complex_kernel<<<(unsigned)((total + 255) / 256), 256, 8 * nbins,
                             (cudaStream_t)stream>>>(
      reinterpret_cast<const float2*>(folds), n, nbins, nbins / 2 + 1, out);
  return check_launch("fold_norm_complex");
}

extern "C" int loki_ffa_level_complex_rows(const LokiFFALevel* lvl, const void* fold_in,
                                           void* fold_out, int32_t* dev_err, void* stream) {
  if (!lvl || !fold_in || !fold_out || !dev_err)
    return set_error(LOKI_ERR_INVALID, "null pointer argument");
  if (lvl->nparams < 1 || lvl->nparams > LOKI_MAX_PARAMS || lvl->nbins < 2 || lvl->nbins % 2 ||
      lvl->level < 1 || lvl->level > 62)
    return set_error(LOKI_ERR_INVALID, "bad level descriptor");
  const int n = lvl->nparams;
  int64_t Q = 1;
  for (int d = 0; d < n; ++d) {
    if (!lvl->param_arr[d] || lvl->counts_cur[d] < 1 || lvl->counts_prev[d] < 1)
      return set_error(LOKI_ERR_INVALID, "bad grid in dim %d", d);
    Q *= lvl->counts_cur[d];
  }
  if (lvl->out_start != 0 || lvl->out_width != lvl->counts_cur[n - 1] || lvl->in_start != 0 ||
      lvl->in_width != lvl->counts_prev[n - 1])
    return set_error(LOKI_ERR_UNSUPPORTED, "Fourier levels are materialised whole");
  if (lvl->nseg_in < 2 || lvl->nseg_in % 2)
    return set_error(LOKI_ERR_INVALID, "nseg_in must be even");
  const int slots = (2 * (lvl->nbins / 2 + 1) + 31) / 32;
  if (slots > 9) return set_error(LOKI_ERR_UNSUPPORTED, "nbins above 286");
  const LevelK K = make_level_k(*lvl);
  // warps to fill the GPU twice: split over segment pairs, then 8 parameters a warp
  const int64_t pairs = lvl->nseg_in / 2, want = 152 * 4 * kClWarps * 2;
  const int64_t w32 = (Q + 31) / 32;
  int64_t parts = std::min<int64_t>({pairs, 65535, (want + w32 - 1) / w32});
  const int64_t per = (pairs + parts - 1) / parts;
  parts = (pairs + per - 1) / per;
  const int pw = parts * w32 < want / 2 ? 8 : 32;
  const int64_t gx = (Q + pw * kClWarps - 1) / (pw * kClWarps);
  if (gx > 0x7FFFFFFF) return set_error(LOKI_ERR_UNSUPPORTED, "grid too large");
  auto kern = slots <= 1   ? ffa_level_complex_rows_kernel<1>
              : slots <= 2 ? ffa_level_complex_rows_kernel<2>
              : slots <= 3 ? ffa_level_complex_rows_kernel<3>
              : slots <= 5 ? ffa_level_complex_rows_kernel<5>
                           : ffa_level_complex_rows_kernel<9>;
  note_launch();
  kern<<<dim3((unsigned)gx, (unsigned)parts), kClWarps * 32, 0, (cudaStream_t)stream>>>(
      *lvl, K, pw, per, static_cast<const float2*>(fold_in), static_cast<float2*>(fold_out),
      dev_err);
  return check_launch("ffa_level_complex_rows");
}

extern "C" int loki_fold_snr_complex64(const void* folds, int64_t n, const LokiScoreSpec* spec,
                                       float* snr, void* stream) {
  if (!spec) return set_error(LOKI_ERR_INVALID, "null score spec");
  if (n < 0) return set_error(LOKI_ERR_INVALID, "n < 0");
  if (spec->nwidths < 1 || spec->nwidths > LOKI_MAX_WIDTHS)
    return set_error(LOKI_ERR_INVALID, "nwidths %d out of range", spec->nwidths);
  int wmax = 0;
  for (int i = 0; i < spec->nwidths; ++i) {
    if (spec->widths[i] < 1) return set_error(LOKI_ERR_INVALID, "width < 1");
    wmax = std::max(wmax, (int)spec->widths[i]);
  }
  if (wmax != spec->wmax) return set_error(LOKI_ERR_INVALID, "wmax != max(widths)");
  // the prefix row of 64 + wmax floats takes the place of the fold
  if (64 + wmax > 2 * kSnrRow)
    return set_error(LOKI_ERR_UNSUPPORTED, "widths above %d", 2 * kSnrRow - 64);
  if (n == 0) return LOKI_OK;
  if (!folds || !snr) return set_error(LOKI_ERR_INVALID, "null pointer argument");
  const int64_t blocks = (n + kSnrThreads - 1) / kSnrThreads;
  if (blocks > 0x7FFFFFFF) return set_error(LOKI_ERR_UNSUPPORTED, "grid too large");
  const ScoreK SK = make_score_k(*spec, 64);
  note_launch();
  fold_snr_complex64_kernel<<<(unsigned)blocks, kSnrThreads,
                              kSnrThreads * kSnrRow * (int)sizeof(float2),
                              (cudaStream_t)stream>>>(static_cast<const float2*>(folds), n, *spec,
                                                      SK, snr);
  return check_launch("fold_snr_complex64");
}
