// Complex brute fold of the Fourier-domain FFA on the tensor cores
// (core/fold.py:395-481 brutefold_start_complex_opt).
//
// The fold is a product: for every (frequency f, harmonic h) and segment row
// the sums over t of x[row, t] cos(angle) and x[row, t] sin(angle), with the
// reference's float32 angle f_h * float32(t * float32(-2 pi tsamp)). The basis
// (f, h, t) is 2 nfreq nbf x seg_len, used once per segment, and has to be made
// from each rounded angle (no recurrence reproduces them), so each CTA makes
// its 128 rows of it on the fly and multiplies them with every segment.
//
// Both operands are split into three bfloat16 parts, x = x1 + x2 + x3 (24
// significant bits), and the products down to 2^-16 of the largest (11, 12, 21,
// 13, 31, 22) are summed: what is dropped is below 2^-24 of |x| |c|, the size
// of one float32 rounding. Tensor memory holds the sums of 144 samples, which
// the threads add up in float32.
//
// CTA (one per SM, 544 threads): warps 0-15 make the basis, a row (f, h) per
// lane of tensor memory and four threads a row, a quarter of a chunk's samples
// each, and put its cosine and sine parts into tensor memory as the A operands;
// warp 16 fetches the segments' parts (B, laid out in global memory as the MMA
// reads them, one bulk copy a chunk) and issues the MMAs. Chunks of 48 samples
// pass through two stages with mbarriers both ways, every wait bounded: where
// one runs out the CTA waits (bounded again) for its MMAs and copies in flight,
// writes NaN for the sums that it did not finish and sets the error word.
//
// Bound: making the basis (about 48 instructions per (f, h, sample) with the
// splitting: 10.5 ms at full issue for 15 100 frequencies x 33 harmonics x
// 16 384 samples) beside the MMAs (24 a 32 samples, about 8 ms). Measured there
// with 64 segments of unit variance: 15.3 ms; the direct sums, which make every
// basis value four times and add in float32, take 126.5 ms.
#include <algorithm>
#include <cuda_bf16.h>

#include "loki_common.cuh"
#include "sincos.cuh"
#include "tcgen05.cuh"

namespace loki {

constexpr int kFmGen = 512;             // basis threads
constexpr int kFmSplit = kFmGen / 128;  // threads per row, each a share of a chunk's samples
constexpr int kFmThreads = kFmGen + 32;
constexpr int kFmRows = 128;            // (f, h) rows per CTA

// Samples per chunk. 48 where two stages of A fit beside the sums of N columns
// (64 segments and a row of ones, 9208 frequencies: 9.2 ms against 10.2 with
// three stages of 32), 32 for more columns.
__host__ __device__ constexpr int fm_k(int N) { return N <= 96 ? 48 : 32; }
// Chunks summed in tensor memory: 144 (128) samples. Its float32 sums round
// toward zero, so their error grows with the length: against float64 over the
// same angles the folds of 16 384 samples are 7.0e-7 sqrt(n) off (rms; the
// direct sums 1.6e-6), with 512 samples 2.2e-6 and 3 % faster.
__host__ __device__ constexpr int fm_group(int N) { return 144 / fm_k(N); }
// Tensor-memory columns of one A stage: two comps, three parts, two samples a column.
__host__ __device__ constexpr int fm_acols(int N) { return 3 * fm_k(N); }

// Six products of the parts, the largest first.
__device__ constexpr int kFmPart[6][2] = {{0, 0}, {0, 1}, {1, 0}, {0, 2}, {2, 0}, {1, 1}};

__host__ __device__ constexpr int fm_stages(int N) {
  return 2 * N + 3 * fm_acols(N) <= 512 ? 3 : 2;
}
__host__ __device__ constexpr int fm_b_bytes(int N) { return 3 * N * fm_k(N) * 2; }

// Rows of the product: segments of ts_e, then those of ts_v, or one row of ones
// when ts_v is NULL. Tiles of N rows each (N a multiple of 16, at most 128).
struct FmRows {
  int64_t rows;
  int N, tiles;
};

static FmRows fm_rows(int64_t nseg, bool unit) {
  FmRows r;
  r.rows = unit ? nseg + 1 : 2 * nseg;
  r.tiles = (int)((r.rows + 127) / 128);
  const int need = (int)((r.rows + r.tiles - 1) / r.tiles);
  r.N = need <= 32 ? 32 : need <= 64 ? 64 : need <= 80 ? 80 : need <= 96 ? 96 : 128;
  r.tiles = (int)((r.rows + r.N - 1) / r.N);
  return r;
}

// The segments' bfloat16 parts: [tile][chunk][part][N x K, K-major core
// matrices of 8 rows x 16 bytes]; one thread makes 8 samples of one row. times:
// float32(t * tfac) of every sample.
template <int K>
__global__ void __launch_bounds__(256)
fm_split_kernel(const float* __restrict__ ts_e, const float* __restrict__ ts_v, int64_t seg_len,
                int64_t nseg, int64_t rows, int N, int64_t nch, int64_t total,
                float tfac, uint4* __restrict__ out, float* __restrict__ times) {
  const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (i < nch * K) times[i] = __fmul_rn((float)i, tfac);
  if (i >= total) return;
  constexpr int kGroups = K / 8;
  const int kg = (int)(i % kGroups);
  const int64_t u = i / kGroups;
  const int n = (int)(u % N);
  const int64_t ch = u / N % nch, tile = u / N / nch;
  const int64_t row = tile * N + n, t0 = ch * K + kg * 8;
  uint32_t p[3][4];
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    float x[2];
#pragma unroll
    for (int z = 0; z < 2; ++z) {
      const int64_t t = t0 + 2 * q + z;
      x[z] = 0.0f;
      if (row < rows && t < seg_len)
        x[z] = row < nseg ? ts_e[row * seg_len + t]
               : ts_v     ? ts_v[(row - nseg) * seg_len + t]
                          : 1.0f;
    }
#pragma unroll
    for (int s = 0; s < 3; ++s) {
      const __nv_bfloat162 b = __floats2bfloat162_rn(x[0], x[1]);
      const uint32_t w = *reinterpret_cast<const uint32_t*>(&b);
      p[s][q] = w;
      x[0] = __fsub_rn(x[0], __uint_as_float(w << 16));
      x[1] = __fsub_rn(x[1], __uint_as_float(w & 0xFFFF0000u));
    }
  }
  const int64_t base = (tile * nch + ch) * (3 * N * K * 2 / 16);
#pragma unroll
  for (int s = 0; s < 3; ++s)
    out[base + s * (N * K * 2 / 16) + (n >> 3) * (8 * kGroups) + kg * 8 + (n & 7)] =
        make_uint4(p[s][0], p[s][1], p[s][2], p[s][3]);
}

__device__ __forceinline__ void mbar_arrive(uint64_t* bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}
__device__ __forceinline__ void mbar_expect(uint64_t* bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)),
               "r"(bytes)
               : "memory");
}
__device__ __forceinline__ void bulk_load(void* dst, const void* src, uint32_t bytes,
                                          uint64_t* bar) {
  asm volatile(
      "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::
          "r"(smem_u32(dst)),
      "l"(src), "r"(bytes), "r"(smem_u32(bar))
      : "memory");
}

// D (+)= A (tensor memory) * B (shared memory)^T, bf16 inputs, f32 accumulate.
// Run by a whole warp, issued by its elected lane: the operands then stay in
// uniform registers (issued from a branch of one lane, the 24 MMAs of a chunk
// took 2400 clocks instead of 1600).
__device__ __forceinline__ void mma_bf16_ta(uint32_t d_tmem, uint32_t a_tmem, uint64_t bdesc,
                                            uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n.reg .pred p, q;\n"
      "elect.sync _|q, 0xFFFFFFFF;\n"
      "setp.ne.b32 p, %4, 0;\n"
      "@q tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n}" ::"r"(d_tmem),
      "r"(a_tmem), "l"(bdesc), "r"(idesc), "r"(accumulate)
      : "memory");
}

__device__ __forceinline__ void tmem_store(uint32_t taddr, const uint32_t (&r)[4]) {
  asm volatile("tcgen05.st.sync.aligned.32x32b.x4.b32 [%0], {%1, %2, %3, %4};" ::"r"(taddr),
               "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3])
               : "memory");
}
__device__ __forceinline__ void tmem_store(uint32_t taddr, const uint32_t (&r)[6]) {
  asm volatile("tcgen05.st.sync.aligned.32x32b.x4.b32 [%0], {%1, %2, %3, %4};" ::"r"(taddr),
               "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3])
               : "memory");
  asm volatile("tcgen05.st.sync.aligned.32x32b.x2.b32 [%0], {%1, %2};" ::"r"(taddr + 4),
               "r"(r[4]), "r"(r[5])
               : "memory");
}
__device__ __forceinline__ void tmem_ld4(uint32_t taddr, uint32_t (&r)[4]) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x4.b32 {%0, %1, %2, %3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
               : "r"(taddr));
}

// Two values' three bfloat16 parts, packed.
__device__ __forceinline__ void split3(float a, float b, uint32_t& p0, uint32_t& p1,
                                       uint32_t& p2) {
  __nv_bfloat162 h = __floats2bfloat162_rn(a, b);
  p0 = *reinterpret_cast<const uint32_t*>(&h);
  a = __fsub_rn(a, __uint_as_float(p0 << 16));
  b = __fsub_rn(b, __uint_as_float(p0 & 0xFFFF0000u));
  h = __floats2bfloat162_rn(a, b);
  p1 = *reinterpret_cast<const uint32_t*>(&h);
  a = __fsub_rn(a, __uint_as_float(p1 << 16));
  b = __fsub_rn(b, __uint_as_float(p1 & 0xFFFF0000u));
  h = __floats2bfloat162_rn(a, b);
  p2 = *reinterpret_cast<const uint32_t*>(&h);
}

__device__ __forceinline__ void fm_commit(uint64_t* bar) {
  asm volatile(
      "{\n.reg .pred q;\nelect.sync _|q, 0xFFFFFFFF;\n"
      "@q tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n}" ::"r"(
          smem_u32(bar))
      : "memory");
}

// Test hook (loki_fourier_force_timeout): one wait that completed counts as run
// out, 1: the issuing warp's for the basis of the second chunk, 2: the basis
// warps' for the first sums. Nothing of the tensor cores' is left in flight by
// it that a wait that really ran out would not leave.
__device__ int g_fm_force_timeout = 0;

struct FmBars {
  uint64_t full[3], empty[3], done, drained, last;
  uint32_t tmem;
  int dead;    // a wait ran out: nothing more is issued, arrived at or waited for
  int loaded;  // chunks that were copied for, of a CTA whose wait ran out
  int force;   // g_fm_force_timeout
};

// Bounded wait. False, at once and for good in every thread that has to wait,
// after any wait ran out; `expired`: one that completed counts as run out.
__device__ __forceinline__ bool fm_wait(FmBars& S, uint64_t* bar, uint32_t parity,
                                        bool expired = false) {
  for (long long i = 0; i < kSpinLimit; ++i) {
    if (mbar_try_wait(bar, parity)) {
      if (!expired) return true;
      break;
    }
    if (*reinterpret_cast<volatile int*>(&S.dead)) return false;
  }
  *reinterpret_cast<volatile int*>(&S.dead) = 1;
  return false;
}

template <int N>
__global__ void __launch_bounds__(kFmThreads, 1)
brutefold_complex_mma_kernel(const uint8_t* __restrict__ parts, const float* __restrict__ times,
                             const double* __restrict__ freqs,
                             int64_t nfreq, int64_t seg_len, int64_t nseg, int64_t rows, int unit,
                             int nbf, float tfac, float corr_factor, int nch,
                             float2* __restrict__ fold, int32_t* __restrict__ err) {
  constexpr int K = fm_k(N), S = fm_stages(N), kGroup = fm_group(N);
  constexpr int kPer = K / kFmSplit;  // samples of a chunk per thread
  constexpr int kB = fm_b_bytes(N);
  constexpr int kCols = N / kFmSplit;  // columns summed by one thread, of cos and of sin
  constexpr uint32_t kColA = 2 * N;
  extern __shared__ __align__(128) uint8_t bs[];  // [S][kB]
  __shared__ FmBars B;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int64_t ncomb = nfreq * nbf;
  const int64_t m0 = (int64_t)blockIdx.x * kFmRows;
  const int64_t row0 = (int64_t)blockIdx.y * N;
  if (tid == 0) {
    for (int s = 0; s < S; ++s) {
      mbar_init(&B.full[s], kFmGen + 1);
      mbar_init(&B.empty[s], 1);
    }
    mbar_init(&B.done, 1);
    mbar_init(&B.drained, kFmGen);
    mbar_init(&B.last, 1);
    B.dead = 0;
    B.force = g_fm_force_timeout;
  }
  if (warp == kFmGen / 32) tmem_alloc(&B.tmem, 512);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tm = B.tmem;
  // chunks whose copy was waited for, or (basis warps) arrived for: nch unless a
  // wait ran out
  int mine = nch;

  if (warp == kFmGen / 32) {
    const uint8_t* src = parts + (int64_t)blockIdx.y * nch * kB;
    int loaded = std::min(S, nch), taken = 0;  // chunks copied for, and waited for
    for (int i = 0; i < loaded; ++i) {
      if (lane == 0) {
        mbar_expect(&B.full[i], kB);
        bulk_load(bs + i * kB, src + i * kB, kB, &B.full[i]);
      }
    }
    // the warp's wait: all of its lanes go on, or none
    auto wait = [&](uint64_t* bar, uint32_t parity, bool expired = false) {
      return __all_sync(0xFFFFFFFFu, fm_wait(B, bar, parity, expired));
    };
    constexpr uint32_t idesc = idesc_bf16(128, N);
    for (int i = 0; i < nch; ++i) {
      const int s = i % S;
      const bool expired = i == 1 && B.force == 1;
      if (!wait(&B.full[s], (uint32_t)(i / S) & 1u, expired)) break;
      ++taken;
      const bool first = i % kGroup == 0;
      if (first && i > 0 && !wait(&B.drained, (uint32_t)(i / kGroup - 1) & 1u)) break;
      tc_fence_after();
      const uint32_t a = tm + kColA + s * fm_acols(N);
      const uint32_t b = smem_u32(bs + s * kB);
#pragma unroll
      for (int ks = 0; ks < K / 16; ++ks)
#pragma unroll
        for (int comp = 0; comp < 2; ++comp)
#pragma unroll
          for (int p = 0; p < 6; ++p)
            mma_bf16_ta(tm + comp * N, a + (comp * 3 + kFmPart[p][0]) * (K / 2) + ks * 8,
                        smem_desc(b + kFmPart[p][1] * (N * K * 2) + ks * 256, 128, K / 8 * 128),
                        idesc, first && ks == 0 && p == 0 ? 0u : 1u);
      fm_commit(&B.empty[s]);
      if (i % kGroup == kGroup - 1 || i == nch - 1) fm_commit(&B.done);
      // refill the stage of the chunk before this one, whose MMAs are done first
      if (i > 0 && loaded < nch) {
        const int r = (i - 1) % S;
        if (!wait(&B.empty[r], (uint32_t)((i - 1) / S) & 1u)) break;
        if (lane == 0) {
          mbar_expect(&B.full[r], kB);
          bulk_load(bs + r * kB, src + (int64_t)loaded * kB, kB, &B.full[r]);
        }
        __syncwarp();
        ++loaded;
      }
    }
    // no MMA of this CTA's is in flight when its tensor memory is freed
    fm_commit(&B.last);
    for (long long k = 0; k < kSpinLimit && !mbar_try_wait(&B.last, 0); ++k) {
    }
    if (lane == 0) B.loaded = loaded;
    mine = taken;
    __syncwarp();
  } else {
    const int quad = warp & 3, g = warp >> 2;  // tensor-memory lanes, sample group
    const int64_t comb = m0 + quad * 32 + lane;
    const int64_t fi = std::min<int64_t>(comb, ncomb - 1) / nbf;
    const int h = (int)(std::min<int64_t>(comb, ncomb - 1) - fi * nbf);
    const float fh = (float)(freqs[fi] * (double)h);
    // The largest angle of this row decides how its sines are taken, for all rows of
    // the warp alike: rows of a warp taking two ways each cost both, and sincosf above
    // 2e5 its slow one (2500 frequencies up to 500 Hz, one segment of 2^16 samples:
    // 45 ms, and 42 by the direct sums). False for NaN.
    const float top = fabsf(fh * tfac) * (float)(nch * K);
    const int way = __all_sync(0xFFFFFFFFu, top < 1.9e5f)   ? 0
                    : __all_sync(0xFFFFFFFFu, top < 1.6e6f) ? 1
                                                            : 2;
    const uint32_t lane_base = tm + ((uint32_t)(quad * 32) << 16);
    float accc[kCols], accs[kCols];
#pragma unroll
    for (int j = 0; j < kCols; ++j) accc[j] = accs[j] = 0.0f;
    // sums of a finished group of chunks out of tensor memory
    // (`arrived`: chunks arrived for so far)
    auto drain = [&](int group, int arrived) {
      if (mine == nch && !fm_wait(B, &B.done, (uint32_t)group & 1u, group == 0 && B.force == 2))
        mine = arrived + (arrived == nch);  // another number than that of a sum that is whole
      __syncwarp();
      tc_fence_after();
#pragma unroll
      for (int j = 0; j < kCols; j += 4) {
        uint32_t c[4], s[4];
        tmem_ld4(lane_base + g * kCols + j, c);
        tmem_ld4(lane_base + N + g * kCols + j, s);
        asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          accc[j + k] = __fadd_rn(accc[j + k], __uint_as_float(c[k]));
          accs[j + k] = __fadd_rn(accs[j + k], __uint_as_float(s[k]));
        }
      }
      tc_fence_before();
      if (mine == nch) mbar_arrive(&B.drained);
    };
    // after a wait that ran out a thread arrives at no barrier any more; its warp
    // goes on together, as tcgen05.st and ld want it, to the next group's end
    for (int i = 0; i < nch; ++i) {
      const int s = i % S;
      float tv[kPer];
#pragma unroll
      for (int q = 0; q < kPer; q += 4) {
        const float4 v = __ldg(reinterpret_cast<const float4*>(times + i * K + g * kPer + q));
        tv[q] = v.x, tv[q + 1] = v.y, tv[q + 2] = v.z, tv[q + 3] = v.w;
      }
      if (i >= S) {
        if (mine == nch && !fm_wait(B, &B.empty[s], (uint32_t)(i / S - 1) & 1u)) mine = i;
        tc_fence_after();
      }
      uint32_t pc[3][kPer / 2], ps[3][kPer / 2];
      auto basis = [&](auto sine) {
#pragma unroll
        for (int q = 0; q < kPer / 2; ++q) {
          float sn[2], cs[2];
          sine(__fmul_rn(fh, tv[2 * q]), &sn[0], &cs[0]);
          sine(__fmul_rn(fh, tv[2 * q + 1]), &sn[1], &cs[1]);
          split3(cs[0], cs[1], pc[0][q], pc[1][q], pc[2][q]);
          split3(sn[0], sn[1], ps[0][q], ps[1][q], ps[2][q]);
        }
      };
      if (way == 0) basis([](float x, float* s, float* c) { sincos_small(x, s, c); });
      else if (way == 1) basis([](float x, float* s, float* c) { sincos_mid(x, s, c); });
      else basis([](float x, float* s, float* c) { sincos_reduced(x, s, c); });
      __syncwarp();
      const uint32_t a = lane_base + kColA + s * fm_acols(N) + g * (kPer / 2);
#pragma unroll
      for (int p = 0; p < 3; ++p) {
        tmem_store(a + p * (K / 2), pc[p]);
        tmem_store(a + (3 + p) * (K / 2), ps[p]);
      }
      asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
      tc_fence_before();
      if (mine == nch) mbar_arrive(&B.full[s]);
      if (i % kGroup == 0 && i > 0) {
        drain(i / kGroup - 1, i + 1);
        if (!__all_sync(0xFFFFFFFFu, mine == nch)) break;
      }
    }
    drain((nch - 1) / kGroup, nch);
    if (mine != nch) {  // sums that were not finished are not handed out as numbers
#pragma unroll
      for (int j = 0; j < kCols; ++j) accc[j] = accs[j] = nanf("");
    }
    // correction phasor exp(i * float32(corr_factor * f_h)), complex64 multiply
    if (comb < ncomb) {
      float cs_c, sn_c;
      sincos_reduced(__fmul_rn(corr_factor, fh), &sn_c, &cs_c);
#pragma unroll
      for (int j = 0; j < kCols; ++j) {
        const int64_t row = row0 + g * kCols + j;
        if (row >= rows) continue;
        const float2 z = make_float2(
            __fsub_rn(__fmul_rn(accc[j], cs_c), __fmul_rn(accs[j], sn_c)),
            __fadd_rn(__fmul_rn(accc[j], sn_c), __fmul_rn(accs[j], cs_c)));
        if (row < nseg) {
          fold[(row * nfreq + fi) * 2 * nbf + h] = z;
        } else if (!unit) {
          fold[((row - nseg) * nfreq + fi) * 2 * nbf + nbf + h] = z;
        } else {  // the row of ones: every segment's variance
          for (int64_t seg = 0; seg < nseg; ++seg)
            fold[(seg * nfreq + fi) * 2 * nbf + nbf + h] = z;
        }
      }
    }
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  if (B.dead) {
    // Copies ahead of the products may still be on their way into this CTA's
    // shared memory. Each lands on a barrier that the basis warps had not all
    // arrived at: they arrive now, and the issuing warp waits (bounded).
    if (warp < kFmGen / 32) {
      for (int j = mine; j < B.loaded; ++j) mbar_arrive(&B.full[j % S]);
    } else {
      for (int j = mine; j < B.loaded; ++j)
        for (long long k = 0;
             k < kSpinLimit && !mbar_try_wait(&B.full[j % S], (uint32_t)(j / S) & 1u); ++k) {
        }
    }
  }
  if (warp == kFmGen / 32) {
    if (lane == 0 && B.dead) atomicOr(err, LOKI_DEVERR_TIMEOUT);
    __syncwarp();
    tmem_dealloc(tm, 512);
  }
}

}  // namespace loki

using namespace loki;

extern "C" int loki_fourier_force_timeout(int32_t wait) {
  const int v = wait;
  if (wait < 0 || wait > 2) return set_error(LOKI_ERR_INVALID, "wait %d outside 0..2", wait);
  if (cudaMemcpyToSymbol(g_fm_force_timeout, &v, sizeof(v)) != cudaSuccess)
    return set_error(LOKI_ERR_CUDA, "cudaMemcpyToSymbol failed");
  return LOKI_OK;
}

extern "C" int64_t loki_brutefold_complex_scratch_bytes(int64_t nsamps, int64_t segment_len,
                                                        int32_t unit_variance) {
  // sample numbers are exact in float32 below 2^24
  if (nsamps <= 0 || segment_len <= 0 || segment_len > (1 << 24) || nsamps % segment_len) return 0;
  const FmRows r = fm_rows(nsamps / segment_len, unit_variance != 0);
  const int64_t nch = (segment_len + fm_k(r.N) - 1) / fm_k(r.N);
  return nch * (r.tiles * (int64_t)fm_b_bytes(r.N) + fm_k(r.N) * 4);
}

template <int N>
static int launch_fm(dim3 grid, const uint8_t* parts, const float* times, const double* freqs,
                     int64_t nfreqs, int64_t seg_len, int64_t nseg, int64_t rows, int unit, int nbf, float tfac,
                     float corr, int64_t nch, float2* fold, int32_t* err, cudaStream_t s) {
  // more than half of an SM's shared memory: tensor memory has room for one CTA
  const int smem = std::max(116 * 1024, fm_stages(N) * fm_b_bytes(N));
  if (set_smem_limit(brutefold_complex_mma_kernel<N>, smem) != cudaSuccess)
    return set_error(LOKI_ERR_CUDA, "cudaFuncSetAttribute failed");
  note_launch();
  brutefold_complex_mma_kernel<N><<<grid, kFmThreads, smem, s>>>(
      parts, times, freqs, nfreqs, seg_len, nseg, rows, unit, nbf, tfac, corr, (int)nch, fold, err);
  return LOKI_OK;
}

extern "C" int loki_brutefold_complex_scratch(const float* ts_e, const float* ts_v,
                                              int64_t nsamps, const double* freqs,
                                              int64_t nfreqs, int64_t segment_len, int32_t nbins,
                                              double tsamp, double t_ref, void* scratch,
                                              int64_t scratch_bytes, void* fold_out,
                                              int32_t* dev_err, void* stream) {
  if (!ts_e || !freqs || !scratch || !fold_out || !dev_err)  // ts_v NULL: all ones
    return set_error(LOKI_ERR_INVALID, "null pointer argument");
  if (nsamps <= 0 || nfreqs <= 0 || segment_len <= 0 || nbins < 2)
    return set_error(LOKI_ERR_INVALID, "bad sizes");
  if (nsamps % segment_len != 0)
    return set_error(LOKI_ERR_INVALID,
                     "the Fourier brute fold needs nsamps a multiple of segment_len");
  if (segment_len > (1 << 24))
    return set_error(LOKI_ERR_UNSUPPORTED, "segments above 2^24 samples");
  if (scratch_bytes < loki_brutefold_complex_scratch_bytes(nsamps, segment_len, !ts_v))
    return set_error(LOKI_ERR_CAPACITY, "complex fold scratch too small");
  if ((reinterpret_cast<uintptr_t>(scratch) & 15) != 0)
    return set_error(LOKI_ERR_INVALID, "scratch must be 16-byte aligned");
  const int nbf = nbins / 2 + 1;
  const int64_t nseg = nsamps / segment_len;
  const FmRows r = fm_rows(nseg, !ts_v);
  const int64_t nch = (segment_len + fm_k(r.N) - 1) / fm_k(r.N);
  const float tfac = (float)(-2.0 * 3.14159265358979323846 * tsamp);
  const float corr = (float)(2.0 * 3.14159265358979323846 * t_ref);
  const int64_t gx = (nfreqs * nbf + kFmRows - 1) / kFmRows;
  const int64_t total = (int64_t)r.tiles * nch * r.N * (fm_k(r.N) / 8);
  if (gx > 0x7FFFFFFF || r.tiles > 65535 || (total + 255) / 256 > 0x7FFFFFFF)
    return set_error(LOKI_ERR_UNSUPPORTED, "grid too large");
  cudaStream_t s = (cudaStream_t)stream;
  uint8_t* parts = static_cast<uint8_t*>(scratch);
  float* times = reinterpret_cast<float*>(parts + r.tiles * nch * fm_b_bytes(r.N));
  note_launch();
  auto split = fm_k(r.N) == 48 ? fm_split_kernel<48> : fm_split_kernel<32>;
  split<<<(unsigned)((total + 255) / 256), 256, 0, s>>>(
      ts_e, ts_v, segment_len, nseg, r.rows, r.N, nch, total, tfac,
      reinterpret_cast<uint4*>(parts), times);
  const dim3 grid((unsigned)gx, (unsigned)r.tiles);
  auto go = [&](auto launch) {
    return launch(grid, parts, times, freqs, nfreqs, segment_len, nseg,
                  r.rows, ts_v ? 0 : 1, nbf, tfac, corr, nch, static_cast<float2*>(fold_out),
                  dev_err, s);
  };
  const int rc = r.N == 32   ? go(launch_fm<32>)
                 : r.N == 64 ? go(launch_fm<64>)
                 : r.N == 80 ? go(launch_fm<80>)
                 : r.N == 96 ? go(launch_fm<96>)
                             : go(launch_fm<128>);
  if (rc) return rc;
  return check_launch("brutefold_complex_mma");
}
