// Brute fold at the start of the FFA (core/fold.py:108-171 brutefold_start).
//
// Two paths give the same bit-identical sums: with nbins <= 256 and room for
// it in the scratch, the chain path below; otherwise the per-thread walk
// described next.
//
// The reference computes a phase-bin map per (frequency, sample in segment)
// and then, per segment and frequency, adds every sample into its bin in time
// order. In the walk the map is built once per frequency chunk
// (phase_map_kernel, FP64 with the reference's rounding) and shared by all
// segments; the fold kernel gives each thread one (segment, frequency) and
// walks the samples in time order exactly like the reference loop, so every
// bin sum is bit-identical.
//
// Per thread the running sums of the current bin stay in registers; all 2 x
// nbins sums live in shared memory laid out [bin][thread] (conflict-free).
// The map row is read 16 bytes at a time and the series 4 samples at a time
// (the 8 threads' series loads of one block are broadcasts of the same
// addresses). Blocks are ordered segment-fastest so that the map rows of the
// frequencies in flight stay in L2 while every segment consumes them.
#include <algorithm>

#include "loki_common.cuh"

namespace loki {

template <typename T>
__global__ void phase_map_kernel(const double* __restrict__ freqs, int64_t nfreq,
                                 int64_t seg_len, int nbins, double tsamp, double t_ref,
                                 T* __restrict__ map) {
  const int64_t total = nfreq * seg_len;
  for (int64_t k = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; k < total;
       k += (int64_t)gridDim.x * blockDim.x) {
    const int64_t f = k / seg_len;
    const int64_t i = k - f * seg_len;
    const double pt = __dsub_rn(__dmul_rn((double)i, tsamp), t_ref);
    int b = round_shift(phase_idx(pt, freqs[f], nbins, 0.0), nbins);
    // Only a non-finite frequency can leave [0, nbins); keep every
    // accumulator index in bounds (the host rejects such grids up front).
    if (b < 0 || b >= nbins) b = 0;
    map[k] = (T)b;
  }
}

template <typename T>
struct MapVec;
template <>
struct MapVec<uint8_t> {
  static constexpr int N = 16;
  __device__ static int get(const uint4& v, int k) {
    const unsigned w = k < 4 ? v.x : k < 8 ? v.y : k < 12 ? v.z : v.w;
    return (w >> (8 * (k & 3))) & 0xFF;
  }
};
template <>
struct MapVec<uint16_t> {
  static constexpr int N = 8;
  __device__ static int get(const uint4& v, int k) {
    const unsigned w = k < 2 ? v.x : k < 4 ? v.y : k < 6 ? v.z : v.w;
    return (w >> (16 * (k & 1))) & 0xFFFF;
  }
};

__device__ __forceinline__ float f4get(const float4& v, int k) {
  return k == 0 ? v.x : k == 1 ? v.y : k == 2 ? v.z : v.w;
}

// kUnit: ts_v is all ones, so only the ts_e sums are taken here (half the
// shared memory per thread); brutefold_count_kernel writes the variance rows.
template <typename T, bool kUnit>
__global__ void __launch_bounds__(128)
brutefold_seq_kernel(const float* __restrict__ ts_e, const float* __restrict__ ts_v,
                     int64_t nsamps, const T* __restrict__ map, int64_t nfreq_chunk,
                     int64_t f_offset, int64_t nfreq_total, int64_t seg_len, int64_t nseg,
                     int nbins, float* __restrict__ fold) {
  extern __shared__ float acc[];  // [NC * nbins][blockDim.x]
  constexpr int NC = kUnit ? 1 : 2;
  const int BS = blockDim.x;
  const int t = threadIdx.x;
  const int64_t seg = blockIdx.x % nseg;
  const int64_t fi = (blockIdx.x / nseg) * BS + t;
  if (fi >= nfreq_chunk) return;  // no block-level synchronisation follows
  for (int b = 0; b < NC * nbins; ++b) acc[b * BS + t] = 0.0f;
  const int64_t start = seg * seg_len;
  const int64_t len = std::min<int64_t>(seg_len, nsamps - start);
  const T* m = map + fi * seg_len;
  const float* e = ts_e + start;
  const float* v = kUnit ? e : ts_v + start;
  int cur = 0;
  float ae = 0.0f, av = 0.0f;
  constexpr int VN = MapVec<T>::N;
  int64_t i = 0;
  const bool aligned = ((reinterpret_cast<uintptr_t>(m) | reinterpret_cast<uintptr_t>(e) |
                         reinterpret_cast<uintptr_t>(v)) & 15) == 0;
  if (aligned && len >= VN) {
    // software pipeline: the map word and series of the next VN samples are
    // loaded while the current VN samples are added
    uint4 mv = *reinterpret_cast<const uint4*>(m);
    float4 ev[VN / 4], vv[VN / 4];
#pragma unroll
    for (int q = 0; q < VN / 4; ++q) {
      ev[q] = __ldg(reinterpret_cast<const float4*>(e) + q);
      if constexpr (!kUnit) vv[q] = __ldg(reinterpret_cast<const float4*>(v) + q);
    }
    for (; i + VN <= len; i += VN) {
      const bool more = i + 2 * VN <= len;
      uint4 mv_n = mv;
      float4 ev_n[VN / 4], vv_n[VN / 4];
#pragma unroll
      for (int q = 0; q < VN / 4; ++q) {
        ev_n[q] = ev[q];
        if constexpr (!kUnit) vv_n[q] = vv[q];
      }
      if (more) {
        mv_n = *reinterpret_cast<const uint4*>(m + i + VN);
#pragma unroll
        for (int q = 0; q < VN / 4; ++q) {
          ev_n[q] = __ldg(reinterpret_cast<const float4*>(e + i + VN) + q);
          if constexpr (!kUnit) vv_n[q] = __ldg(reinterpret_cast<const float4*>(v + i + VN) + q);
        }
      }
#pragma unroll
      for (int k = 0; k < VN; ++k) {
        const int b = MapVec<T>::get(mv, k);
        if (b != cur) {
          acc[cur * BS + t] = ae;
          ae = acc[b * BS + t];
          if constexpr (!kUnit) {
            acc[(nbins + cur) * BS + t] = av;
            av = acc[(nbins + b) * BS + t];
          }
          cur = b;
        }
        ae = __fadd_rn(ae, f4get(ev[k >> 2], k & 3));
        if constexpr (!kUnit) av = __fadd_rn(av, f4get(vv[k >> 2], k & 3));
      }
      mv = mv_n;
#pragma unroll
      for (int q = 0; q < VN / 4; ++q) {
        ev[q] = ev_n[q];
        if constexpr (!kUnit) vv[q] = vv_n[q];
      }
    }
  }
  for (; i < len; ++i) {
    const int b = (int)m[i];
    if (b != cur) {
      acc[cur * BS + t] = ae;
      ae = acc[b * BS + t];
      if constexpr (!kUnit) {
        acc[(nbins + cur) * BS + t] = av;
        av = acc[(nbins + b) * BS + t];
      }
      cur = b;
    }
    ae = __fadd_rn(ae, e[i]);
    if constexpr (!kUnit) av = __fadd_rn(av, v[i]);
  }
  acc[cur * BS + t] = ae;
  if constexpr (!kUnit) acc[(nbins + cur) * BS + t] = av;
  float* out = fold + ((size_t)seg * nfreq_total + f_offset + fi) * 2 * nbins;
  if ((reinterpret_cast<uintptr_t>(out) & 15) == 0 && ((NC * nbins) & 3) == 0) {
    for (int b = 0; b < NC * nbins; b += 4)
      *reinterpret_cast<float4*>(out + b) =
          make_float4(acc[b * BS + t], acc[(b + 1) * BS + t], acc[(b + 2) * BS + t],
                      acc[(b + 3) * BS + t]);
  } else {
    for (int b = 0; b < NC * nbins; ++b) out[b] = acc[b * BS + t];
  }
}

// Variance rows of a unit-variance fold: with ts_v all ones every (segment,
// frequency, bin) sum of the reference is the bin's sample count (exact in
// float32 below 2^24 samples per segment). The map depends only on the sample
// position within a segment, so every full segment has the same counts: one
// histogram per frequency (and one more for a shorter last segment).
template <typename T>
__global__ void __launch_bounds__(256)
brutefold_count_kernel(const T* __restrict__ map, int64_t nfreq_chunk, int64_t f_offset,
                       int64_t nfreq_total, int64_t seg_len, int64_t nsamps, int64_t nseg,
                       int nbins, float* __restrict__ fold) {
  extern __shared__ int hist[];  // [2][nbins]: full segments, last segment
  const int64_t fi = blockIdx.x;
  if (fi >= nfreq_chunk) return;
  const T* m = map + fi * seg_len;
  const int64_t last_len = nsamps - (nseg - 1) * seg_len;
  for (int b = threadIdx.x; b < 2 * nbins; b += blockDim.x) hist[b] = 0;
  __syncthreads();
  for (int64_t i = threadIdx.x; i < seg_len; i += blockDim.x) {
    const int b = (int)m[i];
    atomicAdd(&hist[b], 1);
    if (i < last_len) atomicAdd(&hist[nbins + b], 1);
  }
  __syncthreads();
  for (int64_t k = threadIdx.x; k < nseg * nbins; k += blockDim.x) {
    const int64_t seg = k / nbins;
    const int b = (int)(k - seg * nbins);
    const int c = seg == nseg - 1 ? hist[nbins + b] : hist[b];
    fold[((size_t)seg * nfreq_total + f_offset + fi) * 2 * nbins + nbins + b] = (float)c;
  }
}


// ---------------------------------------------------------------------------
// Chain path (nbins <= 256). Each (row, frequency, bin) sum is a chain of adds
// in sample order, a row being one segment of ts_e or (general variance) of
// ts_v. Which samples reach a bin depends only on the position within a
// segment, so the order is built once per frequency, not once per row:
//
// 1. series_rows_kernel lays the series out by time chunk: for a group of NS
//    rows and a chunk of T samples, [t][row], so that a chunk is one contiguous
//    copy and the rows of one sample are one conflict-free shared-memory load.
// 2. chain_list_kernel sorts each chunk's T positions by bin (stable) for one
//    frequency and writes them as steps of two neighbouring bins: two
//    positions of the even bin, two of the odd one, in time order, padded with
//    position T, a row of zeros. Adding +0 leaves a sum unchanged (a sum that
//    starts at +0 is never -0).
// 3. brutefold_chain_kernel: each lane owns V rows (NS = 32 V; groups of 4 rows
//    where there are no more, which 28 lanes then read with the others), each warp
//    up to 32 chains (bins of one frequency) whose sums stay in registers over the
//    whole segment (or, with little scratch, over a run of chunks: the sums then
//    pass from launch to launch through the fold). A step loads its four positions
//    (one broadcast) and four samples of V rows and adds them in order, two chains
//    side by side.
//
// Bound: shared-memory bandwidth, 4 bytes per add at 128 bytes a clock and SM:
// 4.6 ms with padding for 2^21 samples x 15 100 frequencies, 64 bins, 128
// segments, where the walk takes 6.2 ms and the lists 1.1 ms. A walk of
// 512-sample chunks with one row a lane and the sums in shared memory took
// 13.6 ms (four loads of loop state per 10 samples of a chain), its float64
// phase map 4.5 ms and the sort of it by warp matches 2.7 ms.
// ---------------------------------------------------------------------------

constexpr int kChains = 32;      // chains (bins) per warp, sums in registers
constexpr int kChainWarps = 16;  // most warps per fold block
constexpr int kMaxPer = 16;      // samples of a chunk per lane of the list kernel

// Shape of one chain launch, fixed by nbins, the rows and the frequencies.
struct ChainShape {
  int NS;   // rows per group: 4, 32 or 64 (0: the chain path does not apply)
  int T;    // samples per time chunk, a multiple of 32, at most 32 kMaxPer
  int wpf;  // warps per frequency
  int bpw;  // bins per warp (even)
  int F;    // frequencies per block
  int LB;   // bytes of one (frequency, chunk) list
};

// List of one (frequency, chunk): wpf 32-bit first entries, wpf x 16 step
// counts (bytes), then the 16-bit entries (twice the position). A bin of n
// positions takes ceil(n / 2) steps, a pair of bins the larger of the two, so
// there are at most (T + nbins) / 2 steps of four entries.
__host__ __device__ inline int list_counts_off(int wpf) { return (4 * wpf + 15) & ~15; }
__host__ __device__ inline int list_entries_off(int wpf) {
  return list_counts_off(wpf) + kChains / 2 * wpf;
}
__host__ __device__ inline int list_bytes(int T, int nbins, int wpf) {
  return (list_entries_off(wpf) + 4 * (T + nbins) + 15) & ~15;
}

// Bin of a warp's chain: the warps of a frequency take pairs of neighbouring bins
// in turn. A chunk of a slow pulsar's series covers a run of neighbouring bins (10
// of 64 at 0.2 s), which fell to one warp while the others of the block waited for
// it when each took its bins in one piece (2^20 samples at 1-10 Hz: walk 0.55 ->
// 0.40 ms; 100 bins at 20-150 Hz 2.58 -> 2.47; 50-500 Hz 6.76 -> 6.69).
__host__ __device__ inline int chain_bin(int warp, int chain, int wpf) {
  return 2 * ((chain >> 1) * wpf + warp) + (chain & 1);
}

// Rows [0, nseg) are the segments of ts_e, rows [nseg, 2 nseg) those of ts_v.
// out: [row group][chunk - c0][t][NS] for nc chunks from c0, zeros beyond the
// series and the last row.
template <int NS>
__global__ void __launch_bounds__(256)
series_rows_kernel(const float* __restrict__ ts_e, const float* __restrict__ ts_v,
                   int64_t nsamps, int64_t seg_len, int64_t nseg, int64_t nrows, int T,
                   int64_t c0, int64_t nc, float* __restrict__ out) {
  __shared__ float tile[NS][33];
  const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
  const int64_t nt = T / 32;  // a block per 32 positions of a chunk
  const int64_t tc = blockIdx.x / nt, t = tc % nc, rg = tc / nc;
  const int t0 = (int)(blockIdx.x - tc * nt) * 32;
  const int64_t i = (c0 + t) * T + t0 + tx;  // position within the segment
#pragma unroll
  for (int q0 = 0; q0 < NS; q0 += 8) {
    const int q = q0 + ty;
    const int64_t row = rg * NS + q, seg = row < nseg ? row : row - nseg;
    const int64_t p = seg * seg_len + i;
    float x = 0.0f;
    if (q < NS && row < nrows && i < seg_len && p < nsamps)
      x = __ldg((row < nseg ? ts_e : ts_v) + p);
    if (q < NS) tile[q][tx] = x;
  }
  __syncthreads();
  float* o = out + ((rg * nc + t) * (int64_t)T + t0) * NS;
#pragma unroll
  for (int k = threadIdx.x; k < 32 * NS; k += 256) o[k] = tile[k % NS][k / NS];
}

// Turns per sample (and at position 0) of one frequency as 64-bit fixed-point
// fractions: the bin of position i is round(frac(i step + first) nbins). They
// carry the exact product to 2^-64, the reference's float64 chain deviates
// from it by at most 2^-50 of the turns counted from t_ref, and its float32
// half-up rounding moves a bin edge by less than nbins 2^-23 bins. A position
// farther than `margin` (2^-32 bins) from every edge therefore has a certain
// bin; the others take the float64 chain (margin 2^31: every position does).
struct BinStep {
  unsigned long long step, first;
  unsigned margin;
};

__device__ __forceinline__ unsigned long long turn_fraction(double a, double b) {
  const double p = __dmul_rn(a, b), e = __fma_rn(a, b, -p);  // a b = p + e
  const double fr = __dsub_rn(p, floor(p));                  // exact
  unsigned long long u = fr >= 1.0 ? 0ull : (unsigned long long)__dmul_rn(fr, 0x1p64);
  return u + (unsigned long long)(long long)__dmul_rn(e, 0x1p64);
}

__device__ __forceinline__ BinStep make_bin_step(double f, int64_t seg_len, int nbins,
                                                 double tsamp, double t_ref) {
  BinStep s{0, 0, 0x80000000u};
  const double span = fmax((double)seg_len * tsamp, fabs(t_ref)) * f;  // turns
  if (span >= 0.0 && span < 0x1p24) {  // false for NaN and for negative frequencies
    s.step = turn_fraction(tsamp, f);
    s.first = 0ull - turn_fraction(t_ref, f);
    s.margin = (unsigned)((double)nbins * (0x1p10 + span * 0x1p-17)) + 64u;
  }
  return s;
}

// Bin of one position from the float64 chain (out of line: rarely taken).
static __device__ __noinline__ int bin_exact(int64_t i, double f, int nbins, double tsamp,
                                             double t_ref) {
  const double pt = __dsub_rn(__dmul_rn((double)i, tsamp), t_ref);
  const int b = round_shift(phase_idx(pt, f, nbins, 0.0), nbins);
  return b < 0 || b >= nbins ? 0 : b;  // as phase_map_kernel
}

// Lists of nc chunks from c0. The blocks of a frequency (grid y) share its chunks,
// a warp per chunk. counts (unit variance): [frequency][2][nbins] sample counts of
// these chunks of a full and of the last segment, added up over the blocks where
// there are several (whole numbers below 2^24: exact in any order; the caller
// clears them). The
// bins are integer arithmetic kept in registers and sorted by per-lane counts
// whose rows are padded to an odd number of words (without the padding 16-way
// bank conflicts made it 2.2 ms instead of 1.0). Bound: instruction issue (79 %).
constexpr int kCntRow = 36;    // bytes of a bin's 32 per-lane counts (9 words: no bank conflicts)
constexpr int kPlaceRow = 34;  // 16-bit ranks of a bin's 32 lanes, its first entry (17 words)
__host__ __device__ inline int list_warp_bytes(int nbins, int LB) {
  return ((nbins * (kCntRow + 2 * kPlaceRow) + 15) & ~15) + LB;
}

__global__ void __launch_bounds__(256, 3)
chain_list_kernel(const double* __restrict__ freqs, int64_t seg_len, int nbins, double tsamp,
                  double t_ref, ChainShape cs, int64_t c0, int64_t nc, int64_t last_len,
                  uint8_t* __restrict__ lists, float* __restrict__ counts) {
  extern __shared__ __align__(16) uint8_t lsm[];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, nwarps = blockDim.x >> 5;
  const int per_warp = list_warp_bytes(nbins, cs.LB);  // list, counts u8, places u16
  uint8_t* list = lsm + warp * per_warp;
  uint8_t* cnt = list + cs.LB;
  uint16_t* place = reinterpret_cast<uint16_t*>(cnt + nbins * kCntRow);
  int* hist = reinterpret_cast<int*>(lsm + nwarps * per_warp);  // [2][nbins]
  uint32_t* first = reinterpret_cast<uint32_t*>(list);
  uint8_t* steps = list + list_counts_off(cs.wpf);
  uint16_t* entry = reinterpret_cast<uint16_t*>(list + list_entries_off(cs.wpf));
  const int64_t f = blockIdx.x;
  const double fr = freqs[f];
  const BinStep bs = make_bin_step(fr, seg_len, nbins, tsamp, t_ref);
  const int per = cs.T / 32;
  for (int k = tid; k < 2 * nbins; k += blockDim.x) hist[k] = 0;
  for (int k = lane; k < list_entries_off(cs.wpf); k += 32) list[k] = 0;
  __syncthreads();
  for (int64_t tl = (int64_t)blockIdx.y * nwarps + warp; tl < nc;
       tl += (int64_t)gridDim.y * nwarps) {
    const int64_t t = c0 + tl;
    const int clen = (int)min((int64_t)cs.T, seg_len - t * cs.T);
    for (int k = lane; k < nbins * (kCntRow / 4); k += 32) reinterpret_cast<uint32_t*>(cnt)[k] = 0;
    __syncwarp();
    // this lane's positions: bin, and rank among the lane's earlier ones
    const int i0 = lane * per;
    unsigned long long ph = bs.step * (unsigned long long)(t * cs.T + i0) + bs.first;
    uint16_t br[kMaxPer];
#pragma unroll
    for (int k = 0; k < kMaxPer; ++k) {
      br[k] = 0;
      if (k < per && i0 + k < clen) {
        const unsigned long long x =
            (unsigned long long)(unsigned)(ph >> 32) * (unsigned)nbins + 0x80000000ull;
        int b = (int)(x >> 32);
        if (b >= nbins) b = 0;
        if ((unsigned)x + bs.margin <= 2u * bs.margin - 1u)
          b = bin_exact(t * cs.T + i0 + k, fr, nbins, tsamp, t_ref);
        const int r = cnt[b * kCntRow + lane];
        cnt[b * kCntRow + lane] = (uint8_t)(r + 1);
        br[k] = (uint16_t)(b | (r << 8));
        if (counts && last_len < seg_len && t * cs.T + i0 + k < last_len)
          atomicAdd(&hist[nbins + b], 1);
      }
      ph += bs.step;
    }
    __syncwarp();
    // per bin (a lane each): the rank of every lane's first position, the
    // steps of its pair of bins and where they begin
    int base = 0;  // steps of the bins before (in the order of the warps' chains)
    for (int s0 = 0; s0 < cs.wpf * cs.bpw; s0 += 32) {
      const int kb = (s0 + lane) / cs.bpw, kc = s0 + lane - kb * cs.bpw;
      const int b = kb < cs.wpf ? chain_bin(kb, kc, cs.wpf) : nbins;
      uint32_t w[8] = {0, 0, 0, 0, 0, 0, 0, 0};
      int c = 0;
      if (b < nbins) {
#pragma unroll
        for (int k = 0; k < 8; ++k) {
          w[k] = reinterpret_cast<const uint32_t*>(cnt + b * kCntRow)[k];
          c += (int)((w[k] * 0x01010101u) >> 24);
        }
      }
      const int g = (c + 1) >> 1;
      const int st = max(g, __shfl_xor_sync(0xFFFFFFFFu, g, 1));
      int incl = lane & 1 ? 0 : st;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int y = __shfl_up_sync(0xFFFFFFFFu, incl, o);
        if (lane >= o) incl += y;
      }
      if (b < nbins) {
        const int at = 4 * (base + incl - st);  // the pair's first entry
        if (!(kc & 1)) steps[kb * (kChains / 2) + kc / 2] = (uint8_t)st;
        if (kc == 0) first[kb] = (uint32_t)at;
        if (counts) atomicAdd(&hist[b], c);
        uint32_t run = 0;
        uint32_t* o = reinterpret_cast<uint32_t*>(place + b * kPlaceRow);
#pragma unroll
        for (int k = 0; k < 8; ++k) {
          const uint32_t in = w[k] * 0x01010101u, ex = in - w[k];  // per-byte prefix sums
          o[2 * k] = (run + (ex & 0xFFu)) | ((run + ((ex >> 8) & 0xFFu)) << 16);
          o[2 * k + 1] = (run + ((ex >> 16) & 0xFFu)) | ((run + (ex >> 24)) << 16);
          run += in >> 24;
        }
        o[16] = (uint32_t)(at + 2 * (b & 1));
      }
      base += __shfl_sync(0xFFFFFFFFu, incl, 31);
    }
    const uint32_t pad = 2u * (uint32_t)cs.T * 0x10001u;  // the zero row
    for (int k = lane; k < base; k += 32)
      reinterpret_cast<uint2*>(entry)[k] = make_uint2(pad, pad);
    __syncwarp();
#pragma unroll
    for (int k = 0; k < kMaxPer; ++k)
      if (k < per && i0 + k < clen) {
        const uint16_t* o = place + (br[k] & 0xFF) * kPlaceRow;
        const int r = o[lane] + (br[k] >> 8);
        entry[o[32] + 4 * (r >> 1) + (r & 1)] = (uint16_t)(2 * (i0 + k));
      }
    __syncwarp();
    uint4* dst = reinterpret_cast<uint4*>(lists + (f * nc + tl) * cs.LB);
    const int used = (list_entries_off(cs.wpf) + 8 * base + 15) / 16;
    for (int k = lane; k < used; k += 32) dst[k] = reinterpret_cast<const uint4*>(list)[k];
    __syncwarp();
  }
  if (!counts) return;
  __syncthreads();
  for (int b = tid; b < nbins; b += blockDim.x) {
    const float full = (float)hist[b], end = (float)hist[last_len < seg_len ? nbins + b : b];
    if (gridDim.y == 1) {
      counts[(f * 2) * nbins + b] = full;
      counts[(f * 2 + 1) * nbins + b] = end;
    } else {
      atomicAdd(counts + (f * 2) * nbins + b, full);
      atomicAdd(counts + (f * 2 + 1) * nbins + b, end);
    }
  }
}

__device__ __forceinline__ void cp_async16(void* dst, const void* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(
                   (uint32_t)__cvta_generic_to_shared(dst)),
               "l"(src)
               : "memory");
}

__device__ __forceinline__ uint2 lds_u32x2(uint32_t addr) {
  uint2 v;
  asm volatile("ld.shared.v2.u32 {%0, %1}, [%2];" : "=r"(v.x), "=r"(v.y) : "r"(addr));
  return v;
}
// One sample of this lane's V rows.
__device__ __forceinline__ void lds_rows(uint32_t addr, float (&x)[1]) {
  asm volatile("ld.shared.f32 %0, [%1];" : "=f"(x[0]) : "r"(addr));
}
__device__ __forceinline__ void lds_rows(uint32_t addr, float (&x)[2]) {
  asm volatile("ld.shared.v2.f32 {%0, %1}, [%2];" : "=f"(x[0]), "=f"(x[1]) : "r"(addr));
}

// Block: NS rows x F frequencies, F * wpf warps, over nc chunks. Shared
// memory, double buffered by chunk: rows [T + 1][NS] f32 (row T zeros), lists
// [F][LB]; the next chunk is copied while this one is walked. The sums leave
// through the same memory, whole profiles at a time; `go_on`: they start from
// what an earlier launch left in the fold.
template <int NS>
__global__ void __launch_bounds__(kChainWarps * 32, 1)
brutefold_chain_kernel(const float* __restrict__ rows, const uint8_t* __restrict__ lists,
                       const float* __restrict__ counts, ChainShape cs, int64_t nfreq_chunk,
                       int64_t f_offset, int64_t nfreq_total, int64_t nc, int64_t nseg,
                       int64_t nrows, int64_t nrg, int nbins, int go_on,
                       float* __restrict__ fold) {
  constexpr int V = NS == 64 ? 2 : 1;    // rows per lane
  constexpr int kU = NS < 16 ? NS : 16;  // rows of the fold in flight
  extern __shared__ __align__(16) uint8_t csm[];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, nthr = blockDim.x;
  const int64_t rg = blockIdx.x % nrg, f0 = blockIdx.x / nrg * cs.F;
  const int nfb = (int)min((int64_t)cs.F, nfreq_chunk - f0);
  const int rbytes = (cs.T + 1) * NS * 4, lbytes = cs.F * cs.LB + 16;
  uint8_t* buf[2] = {csm, csm + rbytes + lbytes};
  const float* src_r = rows + rg * nc * (int64_t)cs.T * NS;
  auto fetch = [&](int64_t t) {
    uint8_t* b = buf[t & 1];
    const uint8_t* r = reinterpret_cast<const uint8_t*>(src_r + t * (int64_t)cs.T * NS);
    for (int k = tid; k < cs.T * NS / 4; k += nthr) cp_async16(b + 16 * k, r + 16 * k);
    const int lq = cs.LB / 16;
    for (int k = tid; k < nfb * lq; k += nthr) {
      const int fi = k / lq, q = k - fi * lq;
      cp_async16(b + rbytes + 16 * k, lists + ((f0 + fi) * nc + t) * cs.LB + 16 * q);
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  // the frequencies side by side: those of a slow pulsar are all in the same bins,
  // whose warps would otherwise share one of the SM's four schedulers
  const int kb = warp / cs.F, fi = warp - kb * cs.F;
  const bool active = fi < nfb;
  const int nv = (int)min((int64_t)NS, nrows - rg * NS);  // rows of this block
  // a row's profiles of the block's frequencies in the fold
  auto profiles = [&](int r) {
    const int64_t row = rg * NS + r, seg = row < nseg ? row : row - nseg;
    return fold + ((size_t)seg * nfreq_total + f_offset + f0) * 2 * nbins +
           (row < nseg ? 0 : nbins);
  };
  float* out_s = reinterpret_cast<float*>(csm);  // [row][F nbins]
  const int fn = cs.F * nbins, stride = fn + 1;
  float acc[kChains][V];
#pragma unroll
  for (int c = 0; c < kChains; ++c)
#pragma unroll
    for (int v = 0; v < V; ++v) acc[c][v] = 0.0f;
  if (go_on) {
    for (int k = tid; k < nfb * nbins; k += nthr) {
      const int q = k / nbins, at = q * 2 * nbins + (k - q * nbins);
      for (int r0 = 0; r0 < nv; r0 += kU) {
        float x[kU];
#pragma unroll
        for (int u = 0; u < kU; ++u) x[u] = profiles(min(r0 + u, nv - 1))[at];
#pragma unroll
        for (int u = 0; u < kU; ++u) out_s[min(r0 + u, nv - 1) * stride + k] = x[u];
      }
    }
    __syncthreads();
#pragma unroll
    for (int c = 0; c < kChains; ++c) {
      const int b = chain_bin(kb, c, cs.wpf);
      if (active && c < cs.bpw && b < nbins)
#pragma unroll
        for (int v = 0; v < V; ++v)
          if (lane * V + v < nv) acc[c][v] = out_s[(lane * V + v) * stride + fi * nbins + b];
    }
    __syncthreads();
  }
  for (int k = tid; k < NS; k += nthr)
    for (int q = 0; q < 2; ++q) reinterpret_cast<float*>(buf[q])[cs.T * NS + k] = 0.0f;
  fetch(0);
  for (int64_t t = 0; t < nc; ++t) {
    if (t + 1 < nc) {
      fetch(t + 1);
      asm volatile("cp.async.wait_group 1;" ::: "memory");
    } else {
      asm volatile("cp.async.wait_group 0;" ::: "memory");
    }
    __syncthreads();
    if (active) {
      const uint8_t* l = buf[t & 1] + rbytes + fi * cs.LB;
      const uint4 c4 = *reinterpret_cast<const uint4*>(l + list_counts_off(cs.wpf) +
                                                       kb * (kChains / 2));
      const uint32_t cw[4] = {c4.x, c4.y, c4.z, c4.w};
      // 32-bit shared addresses: this lane's rows, the warp's entries
      const uint32_t xb =
          (uint32_t)__cvta_generic_to_shared(buf[t & 1]) + lane % (NS / V) * (4 * V);
      uint32_t e = (uint32_t)__cvta_generic_to_shared(l) + list_entries_off(cs.wpf) +
                   2 * reinterpret_cast<const uint32_t*>(l)[kb];
      // a sample's bytes are 2 NS per unit of an entry: one 16 x 8-bit dot product per address
      constexpr uint32_t kLo = 2 * NS, kHi = kLo << 8;
      uint2 next = lds_u32x2(e);  // one step ahead: the warp's steps are one run
#pragma unroll
      for (int c = 0; c < kChains; c += 2) {
        const uint32_t end = e + ((cw[c >> 3] >> (8 * ((c >> 1) & 3))) & 0xFFu) * 8;
        // One row a lane is where a walk has few warps and, at the low
        // frequencies of few segments, long runs of one bin: four steps' loads
        // in flight there (32 segments at 1-10 Hz: 0.66 -> 0.55 ms; eight: 7 %
        // slower than four).
        if constexpr (V == 1) {
          constexpr int N = 4;
#pragma unroll 1
          while (end - e >= 8 * N) {
            uint2 w[N];
            w[0] = next;
#pragma unroll
            for (int k = 1; k < N; ++k) w[k] = lds_u32x2(e + 8 * k);
            e += 8 * N;
            next = lds_u32x2(e);
            float x[N][4][V];
#pragma unroll
            for (int k = 0; k < N; ++k) {
              lds_rows(__dp2a_lo(w[k].x, kLo, xb), x[k][0]);
              lds_rows(__dp2a_lo(w[k].x, kHi, xb), x[k][1]);
              lds_rows(__dp2a_lo(w[k].y, kLo, xb), x[k][2]);
              lds_rows(__dp2a_lo(w[k].y, kHi, xb), x[k][3]);
            }
#pragma unroll
            for (int k = 0; k < N; ++k) {
              acc[c][0] = __fadd_rn(__fadd_rn(acc[c][0], x[k][0][0]), x[k][1][0]);
              acc[c + 1][0] = __fadd_rn(__fadd_rn(acc[c + 1][0], x[k][2][0]), x[k][3][0]);
            }
          }
        }
#pragma unroll 1
        while (e != end) {
          const uint2 w = next;
          e += 8;
          next = lds_u32x2(e);
          float a0[V], a1[V], b0[V], b1[V];
          lds_rows(__dp2a_lo(w.x, kLo, xb), a0);
          lds_rows(__dp2a_lo(w.x, kHi, xb), a1);
          lds_rows(__dp2a_lo(w.y, kLo, xb), b0);
          lds_rows(__dp2a_lo(w.y, kHi, xb), b1);
#pragma unroll
          for (int v = 0; v < V; ++v) {
            acc[c][v] = __fadd_rn(__fadd_rn(acc[c][v], a0[v]), a1[v]);
            acc[c + 1][v] = __fadd_rn(__fadd_rn(acc[c + 1][v], b0[v]), b1[v]);
          }
        }
      }
    }
    __syncthreads();
  }
  // sums to shared memory, then whole profiles to the fold
  if (active) {
#pragma unroll
    for (int c = 0; c < kChains; ++c) {
      const int b = chain_bin(kb, c, cs.wpf);
      if (c < cs.bpw && b < nbins && lane < NS / V)
#pragma unroll
        for (int v = 0; v < V; ++v) out_s[(lane * V + v) * stride + fi * nbins + b] = acc[c][v];
    }
  }
  __syncthreads();
  const int per = counts ? 2 * nbins : nbins;  // unit variance: every row is a segment's
  for (int k = tid; k < nfb * per; k += nthr) {
    const int q = k / per, j = k - q * per, at = q * 2 * nbins + j;
    if (j < nbins) {
      for (int r = 0; r < nv; ++r) profiles(r)[at] = out_s[r * stride + q * nbins + j];
      continue;
    }
    const float* cn = counts + (f0 + q) * 2 * nbins + j - nbins;
    const float full = __ldg(cn), end = __ldg(cn + nbins);
    for (int r0 = 0; r0 < nv; r0 += kU) {
      float x[kU];
#pragma unroll
      for (int u = 0; u < kU; ++u) x[u] = go_on ? profiles(min(r0 + u, nv - 1))[at] : 0.0f;
#pragma unroll
      for (int u = 0; u < kU; ++u)
        if (r0 + u < nv) profiles(r0 + u)[at] = x[u] + (rg * NS + r0 + u == nseg - 1 ? end : full);
    }
  }
}

}  // namespace loki

using namespace loki;

namespace loki {

static int64_t round256(int64_t x) { return (x + 255) & ~int64_t(255); }

constexpr int kChainSmem = 226 * 1024;

static int chain_smem(const ChainShape& c, int nbins) {
  const int walk = 2 * ((c.T + 1) * c.NS * 4 + c.F * c.LB + 16);
  const int out = c.NS * (c.F * nbins + 1) * 4;
  return std::max(walk, out);
}

constexpr int64_t kChainSms = 152;

// NS: two rows a lane (64 rows share a list walk, 8-byte loads) once there are
// more than 32, unless blocks of 32 rows and one frequency all fit on the GPU
// at once; four rows where there are no more (one fold of 2^23 samples: 28 ms,
// and 56 with copies of 32 rows, most of them zeros). F: as many frequencies as
// 16 warps hold, fewer where that leaves SMs without a block; the warps that
// this leaves free share a frequency's bins. T: the longest chunk two buffers of
// which fit, since each (chain, chunk) pays a loop and half a padding entry, but
// no longer than an even share of a segment.
static ChainShape chain_shape(int nbins, int64_t nrows, int64_t nfreqs, int64_t seg_len) {
  ChainShape c{0, 0, 0, 0, 0, 0};
  if (nbins < 1 || nbins > 256) return c;
  const int ns = nrows <= 4                                            ? 4
                 : nrows > 32 && (nrows + 31) / 32 * nfreqs > kChainSms ? 64
                                                                        : 32;
  const int least = (nbins + kChains - 1) / kChains;  // warps that hold a frequency's bins
  c.F = kChainWarps / least;
  const int64_t nrg = (nrows + ns - 1) / ns;
  // waves of blocks times the work of one (its copies cost about 0.8 of a frequency's walk)
  const int fmax = c.F;
  double best = 0.0;
  for (int f = fmax; f >= 1; --f) {
    const int64_t blocks = nrg * ((nfreqs + f - 1) / f);
    const double cost = (double)((blocks + kChainSms - 1) / kChainSms) * (f + 0.8);
    if (f == fmax || cost < best) {
      best = cost;
      c.F = f;
    }
  }
  c.wpf = std::max(least, std::min(kChainWarps / c.F, (nbins + 1) / 2));
  c.bpw = ((nbins + c.wpf - 1) / c.wpf + 1) & ~1;
  for (c.T = ns < 64 ? 480 : 384; c.T >= 32; c.T -= 32) {
    c.LB = list_bytes(c.T, nbins, c.wpf);
    c.NS = ns;
    if (chain_smem(c, nbins) > kChainSmem) continue;
    const int64_t nch = (seg_len + c.T - 1) / c.T;
    c.T = (int)(((seg_len + nch - 1) / nch + 31) / 32 * 32);
    c.LB = list_bytes(c.T, nbins, c.wpf);
    return c;
  }
  c.NS = 0;
  return c;
}

static int64_t chain_chunks(const ChainShape& c, int64_t seg_len) {
  return (seg_len + c.T - 1) / c.T;
}
static int64_t chain_groups(const ChainShape& c, int64_t nrows) {
  return (nrows + c.NS - 1) / c.NS;
}

// Scratch of the chain path: the series layout of `run` chunks of every
// segment, then their lists (and sample counts) for `freqs` frequencies (0: the
// path does not apply).
struct ChainPlan {
  ChainShape c;
  int64_t run, freqs;
};

static int64_t chain_rows_bytes(const ChainShape& c, int64_t nrows, int64_t run) {
  return chain_groups(c, nrows) * run * c.T * c.NS * 4;
}
static int64_t chain_freq_bytes(const ChainShape& c, int64_t run, int nbins) {
  return run * c.LB + 2 * nbins * 4;
}
static int64_t chain_bytes(const ChainPlan& p, int64_t nrows, int nbins) {
  return 4 * 256 + chain_rows_bytes(p.c, nrows, p.run) +
         p.freqs * chain_freq_bytes(p.c, p.run, nbins);
}

// Everything in one run over all frequencies where that fits. Otherwise a run of
// fewer chunks, of every row: the layout is made once and each list once whatever
// the split, but every run after the first reads the sums back from the fold, so
// runs are as long as leaves room for frequencies that fill the GPU twice; where
// one chunk at a time does not, the phase map is made instead.
// (16 MiB for 2^23 samples of general
// variance, 15 100 frequencies: a launch of 20 blocks for every 64 rows and 157
// frequencies took 432 ms.) Of five to eight rows, padded to 32, the runs keep the
// layout within kPadded.
constexpr int64_t kPadded = int64_t(64) << 20;

static ChainPlan chain_plan(int nbins, int64_t nrows, int64_t nfreqs, int64_t seg_len,
                            int64_t scratch_bytes) {
  const ChainPlan none = {{0, 0, 0, 0, 0, 0}, 0, 0};
  ChainPlan p = {chain_shape(nbins, nrows, nfreqs, seg_len), 0, nfreqs};
  if (!p.c.NS) return none;
  const int64_t nch = chain_chunks(p.c, seg_len);
  p.run = nch;
  if (p.c.NS == 32 && nrows <= 8)
    p.run = std::max<int64_t>(1, std::min(nch, kPadded / chain_rows_bytes(p.c, nrows, 1)));
  if (chain_bytes(p, nrows, nbins) <= scratch_bytes) return p;
  for (int64_t run = p.run; run >= 1; run = run == 1 ? 0 : (run + 1) / 2) {
    // where a launch does not fill the GPU, the shape is one for its frequencies
    int64_t nf = nfreqs;
    for (int pass = 0; pass < 3 && nf > 0; ++pass) {
      const ChainShape c = chain_shape(nbins, nrows, nf, seg_len);
      const int64_t avail = scratch_bytes - 4 * 256 - chain_rows_bytes(c, nrows, run);
      const int64_t fit = avail < 0 ? 0 : avail / chain_freq_bytes(c, run, nbins);
      const int64_t take = std::min(fit, nf);
      if (take < 1) break;
      const int64_t nrg = chain_groups(c, nrows), blocks = nrg * ((take + c.F - 1) / c.F);
      if (take == nfreqs) return {c, run, take};
      if (blocks >= 2 * kChainSms)  // whole waves of blocks
        return {c, run, std::min(take, blocks / kChainSms * kChainSms / nrg * c.F)};
      if (take == nf) break;
      nf = take;
    }
  }
  return none;
}

static int brutefold_chain(const float* ts_e, const float* ts_v, bool unit, int64_t nsamps,
                           const double* freqs, int64_t nfreqs, int64_t seg_len, int nbins,
                           double tsamp, double t_ref, char* scratch, const ChainPlan& p,
                           float* fold_out, cudaStream_t s) {
  const ChainShape& c = p.c;
  const int64_t nseg = (nsamps + seg_len - 1) / seg_len, nrows = nseg * (unit ? 1 : 2);
  const int64_t nch = chain_chunks(c, seg_len), nrg = chain_groups(c, nrows);
  const int64_t last_len = nsamps - (nseg - 1) * seg_len;
  auto kf = c.NS == 4    ? brutefold_chain_kernel<4>
            : c.NS == 32 ? brutefold_chain_kernel<32>
                         : brutefold_chain_kernel<64>;
  auto kr = c.NS == 4    ? series_rows_kernel<4>
            : c.NS == 32 ? series_rows_kernel<32>
                         : series_rows_kernel<64>;
  const int smem = chain_smem(c, nbins);
  const int lwarps = nbins <= 128 ? 8 : 4;  // about 230 KB at 256 bins and 8 warps
  const int lsmem = lwarps * list_warp_bytes(nbins, c.LB) + 2 * nbins * (int)sizeof(int);
  if (set_smem_limit(kf, smem) != cudaSuccess ||
      set_smem_limit(chain_list_kernel, lsmem) != cudaSuccess)
    return set_error(LOKI_ERR_CUDA, "cudaFuncSetAttribute failed");
  float* rows = reinterpret_cast<float*>(scratch);
  char* at = scratch + round256(chain_rows_bytes(c, nrows, p.run));
  float* counts = unit ? reinterpret_cast<float*>(at) : nullptr;
  uint8_t* lists = reinterpret_cast<uint8_t*>(at + round256(p.freqs * 2 * nbins * 4));
  if (nrg * p.run * (c.T / 32) > 0x7FFFFFFF || p.freqs > 0x7FFFFFFF ||
      nrg * ((p.freqs + c.F - 1) / c.F) > 0x7FFFFFFF)
    return set_error(LOKI_ERR_UNSUPPORTED, "grid too large");
  for (int64_t c0 = 0; c0 < nch; c0 += p.run) {
    const int64_t nc = std::min(p.run, nch - c0);
    note_launch();
    kr<<<(unsigned)(nrg * nc * (c.T / 32)), 256, 0, s>>>(ts_e, ts_v, nsamps, seg_len, nseg,
                                                          nrows, c.T, c0, nc, rows);
    for (int64_t f0 = 0; f0 < nfreqs; f0 += p.freqs) {
      const int64_t nf = std::min(p.freqs, nfreqs - f0);
      // blocks a frequency: three on every SM, two chunks a warp at least (the counts
      // of several have to be cleared first)
      const int64_t ny = std::max<int64_t>(
          1, std::min<int64_t>((3 * kChainSms + nf - 1) / nf, nc / (2 * lwarps)));
      if (counts && ny > 1 &&
          cudaMemsetAsync(counts, 0, nf * 2 * nbins * sizeof(float), s) != cudaSuccess)
        return set_error(LOKI_ERR_CUDA, "cudaMemsetAsync failed");
      note_launch();
      chain_list_kernel<<<dim3((unsigned)nf, (unsigned)ny), 32 * lwarps, lsmem, s>>>(
          freqs + f0, seg_len, nbins, tsamp, t_ref, c, c0, nc, last_len, lists, counts);
      note_launch();
      kf<<<(unsigned)(nrg * ((nf + c.F - 1) / c.F)), c.F * c.wpf * 32, smem, s>>>(
          rows, lists, counts, c, nf, f0, nfreqs, nc, nseg, nrows, nrg, nbins, c0 > 0, fold_out);
    }
    int rc = check_launch("brutefold_chain");
    if (rc) return rc;
  }
  return LOKI_OK;
}

// unit: ts_v is all ones (ts_v may be NULL): only the ts_e sums are made from
// samples, the variance rows are the per-frequency sample counts.
static int brutefold_impl(const float* ts_e, const float* ts_v, bool unit, int64_t nsamps,
                          const double* freqs, int64_t nfreqs, int64_t segment_len,
                          int32_t nbins, double tsamp, double t_ref, void* phase_scratch,
                          int64_t scratch_bytes, float* fold_out, void* stream) {
  if (!ts_e || (!ts_v && !unit) || !freqs || !phase_scratch || !fold_out)
    return set_error(LOKI_ERR_INVALID, "null pointer argument");
  if (nsamps <= 0 || nfreqs <= 0 || segment_len <= 0)
    return set_error(LOKI_ERR_INVALID, "nsamps, nfreqs and segment_len must be > 0");
  if (nbins < 1 || nbins > 768)
    return set_error(LOKI_ERR_UNSUPPORTED, "nbins %d outside [1, 768]", nbins);
  if (unit && segment_len >= (int64_t(1) << 24))
    return set_error(LOKI_ERR_UNSUPPORTED, "unit-variance counts need segments below 2^24");
  cudaStream_t s = (cudaStream_t)stream;
  const int nc = unit ? 1 : 2;
  const int64_t nseg = (nsamps + segment_len - 1) / segment_len;
  const int elem = nbins <= 256 ? 1 : 2;
  if (scratch_bytes / (segment_len * elem) < 1)
    return set_error(LOKI_ERR_CAPACITY, "phase scratch of %lld bytes holds no frequency",
                     (long long)scratch_bytes);
  {  // the chain path when it applies and a chunk of every row and one frequency's list fit
    const ChainPlan p = chain_plan(nbins, nseg * nc, nfreqs, segment_len, scratch_bytes);
    if (p.freqs > 0 && (reinterpret_cast<uintptr_t>(phase_scratch) & 15) == 0)
      return brutefold_chain(ts_e, ts_v, unit, nsamps, freqs, nfreqs, segment_len, nbins, tsamp,
                             t_ref, reinterpret_cast<char*>(phase_scratch), p, fold_out, s);
  }
  const int64_t chunk = std::min(scratch_bytes / (segment_len * elem), nfreqs);
  int bs = 128;  // nc * nbins floats of shared memory per thread, <= 200 KB a block
  while (bs > 32 && (size_t)bs * nc * nbins * sizeof(float) > 200 * 1024) bs >>= 1;
  const size_t smem = (size_t)bs * nc * nbins * sizeof(float);
  if (smem > 200 * 1024) return set_error(LOKI_ERR_UNSUPPORTED, "nbins too large");
  auto k8 = unit ? brutefold_seq_kernel<uint8_t, true> : brutefold_seq_kernel<uint8_t, false>;
  auto k16 =
      unit ? brutefold_seq_kernel<uint16_t, true> : brutefold_seq_kernel<uint16_t, false>;
  if (set_smem_limit(k8, (int)smem) != cudaSuccess ||
      set_smem_limit(k16, (int)smem) != cudaSuccess)
    return set_error(LOKI_ERR_CUDA, "cudaFuncSetAttribute failed");
  const int hsmem = 2 * nbins * (int)sizeof(int);
  for (int64_t f0 = 0; f0 < nfreqs; f0 += chunk) {
    const int64_t nf = std::min(chunk, nfreqs - f0);
    const int64_t total = nf * segment_len;
    const int mblocks = (int)std::min<int64_t>((total + 255) / 256, 152 * 64);
    const int64_t blocks = nseg * ((nf + bs - 1) / bs);
    if (blocks > 0x7FFFFFFF || nf > 0x7FFFFFFF)
      return set_error(LOKI_ERR_UNSUPPORTED, "grid too large");
    note_launch();
    note_launch();
    if (unit) note_launch();
    if (elem == 1) {
      uint8_t* map = (uint8_t*)phase_scratch;
      phase_map_kernel<uint8_t><<<mblocks, 256, 0, s>>>(freqs + f0, nf, segment_len, nbins,
                                                       tsamp, t_ref, map);
      k8<<<(unsigned)blocks, bs, smem, s>>>(ts_e, ts_v, nsamps, map, nf, f0, nfreqs,
                                            segment_len, nseg, nbins, fold_out);
      if (unit)
        brutefold_count_kernel<uint8_t><<<(unsigned)nf, 256, hsmem, s>>>(
            map, nf, f0, nfreqs, segment_len, nsamps, nseg, nbins, fold_out);
    } else {
      uint16_t* map = (uint16_t*)phase_scratch;
      phase_map_kernel<uint16_t><<<mblocks, 256, 0, s>>>(freqs + f0, nf, segment_len, nbins,
                                                        tsamp, t_ref, map);
      k16<<<(unsigned)blocks, bs, smem, s>>>(ts_e, ts_v, nsamps, map, nf, f0, nfreqs,
                                             segment_len, nseg, nbins, fold_out);
      if (unit)
        brutefold_count_kernel<uint16_t><<<(unsigned)nf, 256, hsmem, s>>>(
            map, nf, f0, nfreqs, segment_len, nsamps, nseg, nbins, fold_out);
    }
    int rc = check_launch("brutefold");
    if (rc) return rc;
  }
  return LOKI_OK;
}

}  // namespace loki

extern "C" int64_t loki_brutefold_series_scratch_bytes(int64_t nsamps, int64_t nfreqs,
                                                      int64_t segment_len, int32_t nbins,
                                                      int32_t unit_variance) {
  if (nsamps <= 0 || nfreqs <= 0 || segment_len <= 0 || nbins < 1) return 0;
  const int64_t nrows = (nsamps + segment_len - 1) / segment_len * (unit_variance ? 1 : 2);
  const ChainPlan p = chain_plan(nbins, nrows, nfreqs, segment_len, INT64_MAX / 2);
  if (!p.freqs) return nfreqs * segment_len * (nbins <= 256 ? 1 : 2);
  return std::max(segment_len, chain_bytes(p, nrows, nbins));  // what any fold asks for at least
}

extern "C" int64_t loki_brutefold_scratch_bytes(int64_t nfreqs, int64_t segment_len,
                                                int32_t nbins) {
  return loki_brutefold_series_scratch_bytes(segment_len * 64, nfreqs, segment_len, nbins, 1);
}

extern "C" int loki_brutefold(const float* ts_e, const float* ts_v, int64_t nsamps,
                              const double* freqs, int64_t nfreqs, int64_t segment_len,
                              int32_t nbins, double tsamp, double t_ref, void* phase_scratch,
                              int64_t scratch_bytes, float* fold_out, void* stream) {
  return brutefold_impl(ts_e, ts_v, false, nsamps, freqs, nfreqs, segment_len, nbins, tsamp,
                        t_ref, phase_scratch, scratch_bytes, fold_out, stream);
}

extern "C" int loki_brutefold_unit_variance(const float* ts_e, int64_t nsamps,
                                            const double* freqs, int64_t nfreqs,
                                            int64_t segment_len, int32_t nbins, double tsamp,
                                            double t_ref, void* phase_scratch,
                                            int64_t scratch_bytes, float* fold_out,
                                            void* stream) {
  return brutefold_impl(ts_e, nullptr, true, nsamps, freqs, nfreqs, segment_len, nbins, tsamp,
                        t_ref, phase_scratch, scratch_bytes, fold_out, stream);
}

// Fixed scratch of loki_brutefold_noalloc: the series layout and the sample lists
// of a run of chunks (chain_plan), or the phase map of as many frequencies as it
// holds. The limits on segment_len are the map's: 16 MiB hold one frequency of
// up to 16 Mi samples (nbins <= 256, one byte a sample) or 8 Mi (two bytes).
static constexpr int64_t kNoAllocScratchBytes = int64_t(16) << 20;
static __device__ __align__(256) unsigned char g_noalloc_phase_scratch[kNoAllocScratchBytes];

namespace {
// Device address of the array in the current context. Looked up on every call
// (the lookup allocates nothing): an address cached per device ordinal would
// go stale after cudaDeviceReset or under a non-primary context.
int noalloc_scratch(void** out) {
  void* p = nullptr;
  const cudaError_t e = cudaGetSymbolAddress(&p, g_noalloc_phase_scratch);
  if (e != cudaSuccess || !p)
    return set_error(LOKI_ERR_CUDA, "cudaGetSymbolAddress of the phase scratch failed: %s",
                     cudaGetErrorString(e));
  *out = p;
  return LOKI_OK;
}
}  // namespace

extern "C" int64_t loki_brutefold_noalloc_scratch_bytes(void) { return kNoAllocScratchBytes; }

extern "C" int loki_brutefold_noalloc(const float* ts_e, const float* ts_v, int64_t nsamps,
                                      const double* freqs, int64_t nfreqs, int64_t segment_len,
                                      int32_t nbins, double tsamp, double t_ref, float* fold_out,
                                      void* stream) {
  if (!ts_e || !ts_v || !freqs || !fold_out)
    return set_error(LOKI_ERR_INVALID, "null pointer argument");
  if (nsamps <= 0 || nfreqs <= 0 || segment_len <= 0)
    return set_error(LOKI_ERR_INVALID, "nsamps, nfreqs and segment_len must be > 0");
  if (nbins < 1 || nbins > 768)
    return set_error(LOKI_ERR_UNSUPPORTED, "nbins %d outside [1, 768]", nbins);
  const int64_t elem = nbins <= 256 ? 1 : 2;
  if (segment_len > kNoAllocScratchBytes / elem)
    return set_error(LOKI_ERR_CAPACITY,
                     "segment_len %lld above the no-alloc limit of %lld samples for nbins %d "
                     "(fixed %lld-byte phase scratch)",
                     (long long)segment_len, (long long)(kNoAllocScratchBytes / elem), nbins,
                     (long long)kNoAllocScratchBytes);
  void* scratch = nullptr;
  const int rc = noalloc_scratch(&scratch);
  if (rc) return rc;
  // What a launch reads of the scratch (rows and lists, or the map) is written by
  // launches of the same call before it, and every fold_out element by one thread
  // (which reads it again where its sums go on): nothing is left to be cleared.
  return loki_brutefold(ts_e, ts_v, nsamps, freqs, nfreqs, segment_len, nbins, tsamp, t_ref,
                        scratch, kNoAllocScratchBytes, fold_out, stream);
}
