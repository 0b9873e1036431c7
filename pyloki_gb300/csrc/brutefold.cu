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
//    rows (32 V lanes' worth) and a chunk of T samples, [t][row], so that a
//    chunk is one contiguous copy and the rows of one sample are one
//    conflict-free shared-memory load.
// 2. chain_list_kernel sorts each chunk's T positions by bin (stable) for one
//    frequency and writes them as steps of two neighbouring bins: two
//    positions of the even bin, two of the odd one, in time order, padded with
//    position T, a row of zeros. Adding +0 leaves a sum unchanged (a sum that
//    starts at +0 is never -0).
// 3. brutefold_chain_kernel: each lane owns V rows, each warp up to 32 chains
//    (consecutive bins of one frequency) whose sums stay in registers over the
//    whole segment. A step loads its four positions (one broadcast) and four
//    samples of V rows and adds them in order, two chains side by side.
//
// Bound: shared-memory bandwidth, 4 bytes per add at 128 bytes a clock and SM:
// 4.6 ms with padding for 2^21 samples x 15 100 frequencies, 64 bins, 128
// segments, where the walk takes 6.8 ms and the lists 1.1 ms. A walk of
// 512-sample chunks with one row a lane and the sums in shared memory took
// 13.6 ms (four loads of loop state per 10 samples of a chain), its float64
// phase map 4.5 ms and the sort of it by warp matches 2.7 ms.
// ---------------------------------------------------------------------------

constexpr int kChains = 32;      // chains (bins) per warp, sums in registers
constexpr int kChainWarps = 16;  // most warps per fold block
constexpr int kMaxPer = 16;      // samples of a chunk per lane of the list kernel

// Shape of one chain launch, fixed by nbins, the rows and the frequencies.
struct ChainShape {
  int V;    // rows per lane (0: the chain path does not apply)
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
// out: [row group][chunk][t][NS], zeros beyond the series and the last row.
__global__ void __launch_bounds__(256)
series_rows_kernel(const float* __restrict__ ts_e, const float* __restrict__ ts_v,
                   int64_t nsamps, int64_t seg_len, int64_t nseg, int64_t nrows, int64_t rg0,
                   int T, int NS, int64_t nch, float* __restrict__ out) {
  __shared__ float tile[32][33];
  const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
  const int64_t nt = T / 32;  // a block per 32 positions of a chunk; rg: within this launch
  const int64_t tc = blockIdx.x / nt, t = tc % nch, rg = tc / nch;
  const int t0 = (int)(blockIdx.x - tc * nt) * 32;
  float* o = out + (rg * nch + t) * (int64_t)T * NS;
  for (int r0 = 0; r0 < NS; r0 += 32) {
    __syncthreads();
    for (int q = ty; q < 32; q += 8) {
      const int64_t row = (rg0 + rg) * NS + r0 + q;
      const int64_t seg = row < nseg ? row : row - nseg;
      const int64_t i = t * T + t0 + tx;  // position within the segment
      const int64_t p = seg * seg_len + i;
      float x = 0.0f;
      if (row < nrows && i < seg_len && p < nsamps) x = __ldg((row < nseg ? ts_e : ts_v) + p);
      tile[q][tx] = x;
    }
    __syncthreads();
    for (int q = ty; q < 32; q += 8) o[(int64_t)(t0 + q) * NS + r0 + tx] = tile[tx][q];
  }
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

// One block per frequency, a warp per time chunk. counts (unit variance):
// [frequency][2][nbins] sample counts of a full and of the last segment. The
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
                  double t_ref, ChainShape cs, int64_t nch, int64_t last_len,
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
  for (int64_t t = warp; t < nch; t += nwarps) {
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
    uint4* dst = reinterpret_cast<uint4*>(lists + (f * nch + t) * cs.LB);
    const int used = (list_entries_off(cs.wpf) + 8 * base + 15) / 16;
    for (int k = lane; k < used; k += 32) dst[k] = reinterpret_cast<const uint4*>(list)[k];
    __syncwarp();
  }
  if (!counts) return;
  __syncthreads();
  for (int b = tid; b < nbins; b += blockDim.x) {
    counts[(f * 2) * nbins + b] = (float)hist[b];
    counts[(f * 2 + 1) * nbins + b] = (float)hist[last_len < seg_len ? nbins + b : b];
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

// Block: NS = 32 V rows x F frequencies, F * wpf warps. Shared memory, double
// buffered by chunk: rows [T + 1][NS] f32 (row T zeros), lists [F][LB]; the
// next chunk is copied while this one is walked. The sums leave through the
// same memory, whole profiles at a time.
template <int V>
__global__ void __launch_bounds__(kChainWarps * 32, 1)
brutefold_chain_kernel(const float* __restrict__ rows, const uint8_t* __restrict__ lists,
                       const float* __restrict__ counts, ChainShape cs, int64_t nfreq_chunk,
                       int64_t f_offset, int64_t nfreq_total, int64_t nch, int64_t nseg,
                       int64_t nrows, int64_t rg0, int64_t nrg, int nbins,
                       float* __restrict__ fold) {
  constexpr int NS = 32 * V;
  extern __shared__ __align__(16) uint8_t csm[];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, nthr = blockDim.x;
  const int64_t rg = blockIdx.x % nrg, f0 = blockIdx.x / nrg * cs.F;
  const int nfb = (int)min((int64_t)cs.F, nfreq_chunk - f0);
  const int rbytes = (cs.T + 1) * NS * 4, lbytes = cs.F * cs.LB + 16;
  uint8_t* buf[2] = {csm, csm + rbytes + lbytes};
  const float* src_r = rows + rg * nch * (int64_t)cs.T * NS;
  auto fetch = [&](int64_t t) {
    uint8_t* b = buf[t & 1];
    const uint8_t* r = reinterpret_cast<const uint8_t*>(src_r + t * (int64_t)cs.T * NS);
    for (int k = tid; k < cs.T * NS / 4; k += nthr) cp_async16(b + 16 * k, r + 16 * k);
    const int lq = cs.LB / 16;
    for (int k = tid; k < nfb * lq; k += nthr) {
      const int fi = k / lq, q = k - fi * lq;
      cp_async16(b + rbytes + 16 * k, lists + ((f0 + fi) * nch + t) * cs.LB + 16 * q);
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  for (int k = tid; k < NS; k += nthr)
    for (int q = 0; q < 2; ++q) reinterpret_cast<float*>(buf[q])[cs.T * NS + k] = 0.0f;
  float acc[kChains][V];
#pragma unroll
  for (int c = 0; c < kChains; ++c)
#pragma unroll
    for (int v = 0; v < V; ++v) acc[c][v] = 0.0f;
  const int fi = warp / cs.wpf, kb = warp - fi * cs.wpf;
  const bool active = fi < nfb;
  fetch(0);
  for (int64_t t = 0; t < nch; ++t) {
    if (t + 1 < nch) {
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
      const uint32_t xb = (uint32_t)__cvta_generic_to_shared(buf[t & 1]) + lane * (4 * V);
      uint32_t e = (uint32_t)__cvta_generic_to_shared(l) + list_entries_off(cs.wpf) +
                   2 * reinterpret_cast<const uint32_t*>(l)[kb];
      // a row's bytes are 64 V per unit of an entry: one 16 x 8-bit dot product per address
      constexpr uint32_t kLo = 64 * V, kHi = kLo << 8;
      uint2 next = lds_u32x2(e);  // one step ahead: the warp's steps are one run
#pragma unroll
      for (int c = 0; c < kChains; c += 2) {
        const uint32_t end = e + ((cw[c >> 3] >> (8 * ((c >> 1) & 3))) & 0xFFu) * 8;
        // One row a lane is where a walk has few warps and, at the low
        // frequencies of few segments, long runs of one bin: four steps' loads
        // in flight there (32 segments at 1-10 Hz: 0.66 -> 0.55 ms).
        if constexpr (V == 1) {
#pragma unroll 1
          while (end - e >= 32) {
            uint2 w[4];
            w[0] = next;
#pragma unroll
            for (int k = 1; k < 4; ++k) w[k] = lds_u32x2(e + 8 * k);
            e += 32;
            next = lds_u32x2(e);
            float x[4][4][V];
#pragma unroll
            for (int k = 0; k < 4; ++k) {
              lds_rows(__dp2a_lo(w[k].x, kLo, xb), x[k][0]);
              lds_rows(__dp2a_lo(w[k].x, kHi, xb), x[k][1]);
              lds_rows(__dp2a_lo(w[k].y, kLo, xb), x[k][2]);
              lds_rows(__dp2a_lo(w[k].y, kHi, xb), x[k][3]);
            }
#pragma unroll
            for (int k = 0; k < 4; ++k) {
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
  // sums to shared memory [row][F nbins], then whole profiles to the fold
  float* out_s = reinterpret_cast<float*>(csm);
  const int fn = cs.F * nbins, stride = fn + 1;
  if (active) {
#pragma unroll
    for (int c = 0; c < kChains; ++c) {
      const int b = chain_bin(kb, c, cs.wpf);
      if (c < cs.bpw && b < nbins)
#pragma unroll
        for (int v = 0; v < V; ++v) out_s[(lane * V + v) * stride + fi * nbins + b] = acc[c][v];
    }
  }
  __syncthreads();
  const int ncomp = counts ? 1 : 2;
  for (int r = 0; r < NS; ++r) {
    const int64_t row = (rg0 + rg) * NS + r;
    if (row >= nrows) break;
    const int64_t seg = row < nseg ? row : row - nseg;
    float* o = fold + ((size_t)seg * nfreq_total + f_offset + f0) * 2 * nbins +
               (row < nseg ? 0 : nbins);
    if (ncomp == 1) {
      const float* cn = counts + (f0 * 2 + (seg == nseg - 1 ? 1 : 0)) * nbins;
      for (int k = tid; k < nfb * 2 * nbins; k += nthr) {
        const int q = k / (2 * nbins), j = k - q * 2 * nbins;
        o[k] = j < nbins ? out_s[r * stride + q * nbins + j]
                         : __ldg(cn + q * 2 * nbins + j - nbins);
      }
    } else {
      for (int k = tid; k < nfb * nbins; k += nthr) {
        const int q = k / nbins;
        o[q * 2 * nbins + (k - q * nbins)] = out_s[r * stride + k];
      }
    }
  }
}

}  // namespace loki

using namespace loki;

namespace loki {

static int64_t round256(int64_t x) { return (x + 255) & ~int64_t(255); }

constexpr int kChainSmem = 226 * 1024;

static int chain_smem(const ChainShape& c, int nbins) {
  const int ns = 32 * c.V;
  const int walk = 2 * ((c.T + 1) * ns * 4 + c.F * c.LB + 16);
  const int out = ns * (c.F * nbins + 1) * 4;
  return std::max(walk, out);
}

// V: two rows a lane (64 rows share a list walk, 8-byte loads) once there are
// more than 32. F: as many frequencies as 16 warps hold, fewer where that
// leaves SMs without a block. T: the longest chunk two buffers of which
// fit, since each (chain, chunk) pays a loop and half a padding entry.
static ChainShape chain_shape(int nbins, int64_t nrows, int64_t nfreqs, int V) {
  ChainShape c{0, 0, 0, 0, 0, 0};
  if (nbins < 1 || nbins > 256) return c;
  c.wpf = (nbins + kChains - 1) / kChains;
  c.bpw = ((nbins + c.wpf - 1) / c.wpf + 1) & ~1;
  c.F = kChainWarps / c.wpf;
  const int64_t nrg = (nrows + 32 * V - 1) / (32 * V);
  // waves of blocks times the work of one (its copies cost about 0.8 of a frequency's walk)
  const int fmax = c.F;
  double best = 0.0;
  for (int f = fmax; f >= 1; --f) {
    const int64_t blocks = nrg * ((nfreqs + f - 1) / f);
    const double cost = (double)((blocks + 151) / 152) * (f + 0.8);
    if (f == fmax || cost < best) {
      best = cost;
      c.F = f;
    }
  }
  for (c.T = V == 1 ? 480 : 384; c.T >= 32; c.T -= 32) {
    c.LB = list_bytes(c.T, nbins, c.wpf);
    c.V = V;
    if (chain_smem(c, nbins) <= kChainSmem) return c;
  }
  c.V = 0;
  return c;
}

static int64_t chain_chunks(const ChainShape& c, int64_t seg_len) {
  return (seg_len + c.T - 1) / c.T;
}
// Scratch bytes of one row group of the series layout, and of one frequency
// (lists and counts).
static int64_t chain_group_bytes(const ChainShape& c, int64_t seg_len) {
  return chain_chunks(c, seg_len) * c.T * 32 * c.V * 4;
}
static int64_t chain_freq_bytes(const ChainShape& c, int64_t seg_len, int nbins) {
  return chain_chunks(c, seg_len) * c.LB + 2 * nbins * 4;
}

// Scratch of the chain path: `groups` row groups of the series at a time (all
// of them when they fit in half of it) and `chunk` frequencies.
struct ChainPlan {
  ChainShape c;
  int64_t groups, chunk;
};

static ChainPlan chain_plan(int nbins, int64_t nrows, int64_t nfreqs, int64_t seg_len,
                            int64_t scratch_bytes) {
  for (int V = nrows > 32 ? 2 : 1; V >= 1; --V) {
    const ChainShape c = chain_shape(nbins, nrows, nfreqs, V);
    if (!c.V) continue;
    const int64_t avail = scratch_bytes - 4 * 256;
    const int64_t g = chain_group_bytes(c, seg_len), q = chain_freq_bytes(c, seg_len, nbins);
    const int64_t nrg = (nrows + 32 * V - 1) / (32 * V);
    if (avail < g + q) continue;
    int64_t groups = nrg;
    if (nrg * g + nfreqs * q > avail) groups = std::min(nrg, std::max<int64_t>(1, avail / 2 / g));
    return {c, groups, std::min(nfreqs, std::max<int64_t>(1, (avail - groups * g) / q))};
  }
  return {{0, 0, 0, 0, 0, 0}, 0, 0};
}

static int brutefold_chain(const float* ts_e, const float* ts_v, bool unit, int64_t nsamps,
                           const double* freqs, int64_t nfreqs, int64_t seg_len, int nbins,
                           double tsamp, double t_ref, char* scratch, const ChainPlan& p,
                           float* fold_out, cudaStream_t s) {
  const ChainShape& c = p.c;
  const int64_t nseg = (nsamps + seg_len - 1) / seg_len, nrows = nseg * (unit ? 1 : 2);
  const int64_t nch = chain_chunks(c, seg_len), nrg = (nrows + 32 * c.V - 1) / (32 * c.V);
  const int64_t last_len = nsamps - (nseg - 1) * seg_len;
  auto kf = c.V == 1 ? brutefold_chain_kernel<1> : brutefold_chain_kernel<2>;
  const int smem = chain_smem(c, nbins);
  const int lwarps = nbins <= 128 ? 8 : 4;  // about 230 KB at 256 bins and 8 warps
  const int lsmem = lwarps * list_warp_bytes(nbins, c.LB) + 2 * nbins * (int)sizeof(int);
  if (set_smem_limit(kf, smem) != cudaSuccess ||
      set_smem_limit(chain_list_kernel, lsmem) != cudaSuccess)
    return set_error(LOKI_ERR_CUDA, "cudaFuncSetAttribute failed");
  float* rows = reinterpret_cast<float*>(scratch);
  char* at = scratch + round256(p.groups * chain_group_bytes(c, seg_len));
  float* counts = unit ? reinterpret_cast<float*>(at) : nullptr;
  uint8_t* lists = reinterpret_cast<uint8_t*>(at + round256(p.chunk * 2 * nbins * 4));
  const int threads = c.F * c.wpf * 32;
  auto lay_out = [&](int64_t rg0, int64_t n) {
    note_launch();
    series_rows_kernel<<<(unsigned)(n * nch * (c.T / 32)), 256, 0, s>>>(ts_e, ts_v, nsamps, seg_len, nseg,
                                                           nrows, rg0, c.T, 32 * c.V, nch, rows);
  };
  if (p.groups * nch * (c.T / 32) > 0x7FFFFFFF || p.chunk > 0x7FFFFFFF ||
      p.groups * ((p.chunk + c.F - 1) / c.F) > 0x7FFFFFFF)
    return set_error(LOKI_ERR_UNSUPPORTED, "grid too large");
  if (p.groups == nrg) lay_out(0, nrg);
  for (int64_t f0 = 0; f0 < nfreqs; f0 += p.chunk) {
    const int64_t nf = std::min(p.chunk, nfreqs - f0);
    note_launch();
    chain_list_kernel<<<(unsigned)nf, 32 * lwarps, lsmem, s>>>(freqs + f0, seg_len, nbins, tsamp,
                                                              t_ref, c, nch, last_len, lists,
                                                              counts);
    for (int64_t r0 = 0; r0 < nrg; r0 += p.groups) {
      const int64_t n = std::min(p.groups, nrg - r0);
      if (p.groups < nrg) lay_out(r0, n);
      note_launch();
      kf<<<(unsigned)(n * ((nf + c.F - 1) / c.F)), threads, smem, s>>>(
          rows, lists, counts, c, nf, f0, nfreqs, nch, nseg, nrows, r0, n, nbins, fold_out);
    }
    int rc = check_launch("brutefold_chain");
    if (rc) return rc;
  }
  return LOKI_OK;
}

// unit: ts_v is all ones (ts_v may be NULL); the ts_e sums come from the
// sequential kernel and the variance rows from the per-frequency counts.
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
  {  // the chain path when it applies and one row group and frequency of it fit
    const ChainPlan p = chain_plan(nbins, nseg * nc, nfreqs, segment_len, scratch_bytes);
    if (p.chunk > 0 && (reinterpret_cast<uintptr_t>(phase_scratch) & 15) == 0)
      return brutefold_chain(ts_e, ts_v, unit, nsamps, freqs, nfreqs, segment_len, nbins, tsamp,
                             t_ref, reinterpret_cast<char*>(phase_scratch), p, fold_out, s);
  }
  const int elem = nbins <= 256 ? 1 : 2;
  int64_t chunk = scratch_bytes / (segment_len * elem);
  if (chunk < 1)
    return set_error(LOKI_ERR_CAPACITY, "phase scratch of %lld bytes holds no frequency",
                     (long long)scratch_bytes);
  chunk = std::min(chunk, nfreqs);
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
  const int V = nrows > 32 ? 2 : 1;
  const ChainShape c = chain_shape(nbins, nrows, nfreqs, V);
  if (!c.V) return nfreqs * segment_len * (nbins <= 256 ? 1 : 2);
  return 4 * 256 + (nrows + 32 * V - 1) / (32 * V) * chain_group_bytes(c, segment_len) +
         nfreqs * chain_freq_bytes(c, segment_len, nbins);
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

// Fixed phase-map scratch of loki_brutefold_noalloc. 16 MiB holds the map of
// one frequency for segments of up to 16 Mi samples (nbins <= 256, one byte a
// sample) or 8 Mi samples (nbins > 256, two bytes); larger frequency grids are
// processed in chunks of as many frequencies as the array holds.
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
  // Every map entry a fold reads is written by the phase-map launch of the same
  // chunk, and every fold_out element by one fold thread: nothing is cleared.
  return loki_brutefold(ts_e, ts_v, nsamps, freqs, nfreqs, segment_len, nbins, tsamp, t_ref,
                        scratch, kNoAllocScratchBytes, fold_out, stream);
}
