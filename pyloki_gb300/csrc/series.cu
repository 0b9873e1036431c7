// Input conditioning of a time series: the running-median deredden, order
// statistics, the mean and the normalisation that io/timeseries.py:198-236
// (TimeSeries.from_tim) applies through sigpyproc's TimeSeries.deredden and
// TimeSeries.normalise before a search.
//
// Definitions (sigpyproc is not part of the reference tree, so its filters are
// restated here with these semantics):
// - running median over `window` samples: output i is the order statistic of
//   rank window / 2 (the upper median for an even window) of the samples at
//   i - window/2 .. i - window/2 + window - 1, with half-sample symmetric
//   reflection at the ends (scipy.ndimage.median_filter, mode "reflect");
// - k-th order statistic of a float32 array (0-based, ascending);
// - the mean accumulated in float64.
#include <algorithm>

#include "loki_common.cuh"

namespace loki {

constexpr int kMedThreads = 512;
constexpr int kMedMaxWindow = 32768;

// Index of position j in [0, n) after half-sample symmetric reflection
// (period 2n).
__device__ __forceinline__ int64_t reflect_idx(int64_t j, int64_t n) {
  const int64_t p = 2 * n;
  int64_t m = j % p;
  if (m < 0) m += p;
  return m < n ? m : p - 1 - m;
}

// Order-preserving key of the float at p (NaN after +inf). Its bits are loaded
// as an integer: made from a loaded float, u | 0x80000000 (which is -|x|) of a
// positive NaN came out as 0x7FFFFFFF, the key of -0.
__device__ __forceinline__ unsigned load_key(const float* __restrict__ p) {
  const unsigned u = __ldg(reinterpret_cast<const unsigned*>(p));
  return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}
__device__ __forceinline__ float key2f(unsigned k) {
  return __uint_as_float((k & 0x80000000u) ? (k & 0x7FFFFFFFu) : ~k);
}

// Number of entries of the ascending window s[0..w) below v (lower bound),
// found by warp `lane`s with a 32-way search.
__device__ __forceinline__ int warp_lower_bound(const float* s, int w, float v, int lane) {
  int lo = 0, hi = w;  // answer in [lo, hi]
  while (hi - lo > 32) {
    const int step = (hi - lo + 31) / 32;
    const int idx = lo + (lane + 1) * step - 1;  // last element of lane's slice
    const bool below = idx < hi && s[idx] < v;
    const unsigned m = __ballot_sync(0xFFFFFFFFu, below);
    const int nb = __popc(m);  // slices entirely below v
    lo = lo + nb * step;
    hi = min(hi, lo + step);
  }
  const int idx = lo + lane;
  const bool below = idx < hi && s[idx] < v;
  return lo + __popc(__ballot_sync(0xFFFFFFFFu, below));
}

// Block b computes outputs [b * chunk, min((b + 1) * chunk, n)). The window is
// kept sorted in shared memory: a bitonic sort of the first window, then per
// output one removal and one insertion (two warp searches and a shift).
__global__ void __launch_bounds__(kMedThreads)
running_median_kernel(const float* __restrict__ x, int64_t n, int w, int pw, int64_t chunk,
                      int subtract, float* __restrict__ out) {
  extern __shared__ float s[];  // [pw]
  __shared__ int pos[2];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int64_t i0 = (int64_t)blockIdx.x * chunk;
  if (i0 >= n) return;  // uniform over the block
  const int64_t i1 = min(i0 + chunk, n);
  const int half = w / 2;
  for (int k = tid; k < pw; k += kMedThreads)
    s[k] = k < w ? x[reflect_idx(i0 - half + k, n)] : __int_as_float(0x7F800000);
  __syncthreads();
  for (int size = 2; size <= pw; size <<= 1) {  // bitonic sort, ascending
    for (int stride = size >> 1; stride > 0; stride >>= 1) {
      for (int k = tid; k < pw / 2; k += kMedThreads) {
        const int a = 2 * k - (k & (stride - 1));
        const int b = a + stride;
        const bool up = (a & size) == 0;
        const float va = s[a], vb = s[b];
        if ((va > vb) == up) {
          s[a] = vb;
          s[b] = va;
        }
      }
      __syncthreads();
    }
  }
  // the samples leaving and entering the window for output i + 1, loaded one
  // output ahead
  float vo = x[reflect_idx(i0 - half, n)];
  float vn = x[reflect_idx(i0 - half + w, n)];
  for (int64_t i = i0;; ++i) {
    if (tid == 0) {
      const float m = s[half];
      out[i] = subtract ? __fsub_rn(x[i], m) : m;
    }
    if (i + 1 >= i1) break;
    const float co = vo, cn = vn;
    if (i + 2 < i1) {
      vo = x[reflect_idx(i + 1 - half, n)];
      vn = x[reflect_idx(i + 1 - half + w, n)];
    }
    if (co == cn) continue;  // the window's sorted content is unchanged
    if (warp < 2) {
      const int r = warp_lower_bound(s, w, warp == 0 ? co : cn, lane);
      if (lane == 0) pos[warp] = r;
    }
    __syncthreads();
    const int p = pos[0], q = pos[1];
    // cn > co: s[p+1 .. q-1] move down one and cn lands at q - 1;
    // cn < co: s[q .. p-1] move up one and cn lands at q
    const int src = cn > co ? p + 1 : q;
    const int dst = cn > co ? p : q + 1;
    const int len = cn > co ? q - 1 - p : p - q;
    constexpr int kPer = kMedMaxWindow / kMedThreads;
    float v[kPer];
#pragma unroll
    for (int j = 0; j < kPer; ++j) {
      if (j * kMedThreads >= len) break;  // uniform over the block
      const int k = tid + j * kMedThreads;
      if (k < len) v[j] = s[src + k];
    }
    __syncthreads();
#pragma unroll
    for (int j = 0; j < kPer; ++j) {
      if (j * kMedThreads >= len) break;
      const int k = tid + j * kMedThreads;
      if (k < len) s[dst + k] = v[j];
    }
    if (tid == 0) s[cn > co ? q - 1 : q] = cn;
    __syncthreads();
  }
}

// ---------------------------------------------------------------------------
// Running median over a wavelet matrix (Claude, Navarro & Ordonez 2015): the
// reflected series' keys are stably partitioned bit by bit, most significant
// first, zeros before ones, keeping per level the bits and the running count
// of ones. The order statistic of a window is then read off level by level:
// the window's zeros are a contiguous range of the next level, and its ones
// another, so 32 pairs of rank lookups give the k-th smallest key, whatever
// the window length. Every output is independent. The sorted window that one
// block slides over its outputs (running_median_kernel) pays a search and a
// shift of the window for each sample, one after the other: 2^22 samples with
// a 15 625-sample window took 79 ms there and take 0.60 ms here, where the 32
// partition passes (one launch each, L2-resident) are most of it.
// ---------------------------------------------------------------------------

constexpr int kWmThreads = 512;
constexpr int kWmTile = 8192;                           // keys per block
constexpr int kWmPer = kWmTile / kWmThreads;            // keys per lane
constexpr int kWmWords = kWmTile / 32;                  // rank words per tile

struct WmScratch {
  uint2* level;    // [32][ntiles * kWmWords]: ones before the word, the word's bits
  uint32_t* keys;  // [2][ntiles * kWmTile]
  int32_t* count;  // [32][ntiles]: ones of the tile at that level (level 0: top bit)
  uint32_t* zeros; // [32]: zeros of the level
  int64_t ntiles;
};

static int64_t wm_tiles(int64_t m) { return m / kWmTile + 1; }  // position m has a word too
static int64_t wm_bytes(int64_t nt) {
  return nt * (32 * kWmWords * 8 + 2 * kWmTile * 4 + 32 * 4) + 32 * 4 + 256;
}
static WmScratch wm_layout(void* p, int64_t nt) {
  WmScratch w;
  w.ntiles = nt;
  w.level = reinterpret_cast<uint2*>(p);
  w.keys = reinterpret_cast<uint32_t*>(w.level + 32 * nt * kWmWords);
  w.count = reinterpret_cast<int32_t*>(w.keys + 2 * nt * kWmTile);
  w.zeros = reinterpret_cast<uint32_t*>(w.count + 32 * nt);
  return w;
}

// Keys of the m = n + w - 1 reflected samples; the tiles' counts of the top bit.
__global__ void __launch_bounds__(kWmThreads)
wm_keys_kernel(const float* __restrict__ x, int64_t n, int half, int64_t m, WmScratch W) {
  __shared__ int total;
  if (threadIdx.x == 0) total = 0;
  __syncthreads();
  const int64_t base = (int64_t)blockIdx.x * kWmTile;
  int ones = 0;
  for (int k = threadIdx.x; k < kWmTile; k += kWmThreads) {
    const int64_t p = base + k;
    const uint32_t key = p < m ? load_key(x + reflect_idx(p - half, n)) : 0u;
    W.keys[p] = key;
    ones += (int)(key >> 31);
  }
  atomicAdd(&total, ones);
  __syncthreads();
  if (threadIdx.x == 0) W.count[blockIdx.x] = total;
}

// One level: the tile's rank words, and its keys to the next level's order
// (level < 31), whose tiles' counts of the next bit are added up on the way
// (a tile's zeros, and its ones, land in at most two tiles).
__global__ void __launch_bounds__(kWmThreads)
wm_level_kernel(int level, int64_t m, WmScratch W) {
  __shared__ uint32_t red[2], wsum[kWmThreads / 32];
  __shared__ int nxt[4];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int64_t nt = W.ntiles, blk = blockIdx.x;
  const int bit = 31 - level;
  if (tid < 2) red[tid] = 0;
  if (tid < 4) nxt[tid] = 0;
  __syncthreads();
  uint32_t pre = 0, tot = 0;  // ones before this tile, ones of the level
  for (int64_t j = tid; j < nt; j += kWmThreads) {
    const uint32_t c = (uint32_t)W.count[level * nt + j];
    tot += c;
    if (j < blk) pre += c;
  }
  for (int o = 16; o > 0; o >>= 1) {
    pre += __shfl_down_sync(0xFFFFFFFFu, pre, o);
    tot += __shfl_down_sync(0xFFFFFFFFu, tot, o);
  }
  if (lane == 0) {
    atomicAdd(&red[0], pre);
    atomicAdd(&red[1], tot);
  }
  const uint32_t* src = W.keys + (level & 1) * nt * kWmTile;
  uint32_t* dst = W.keys + ((level & 1) ^ 1) * nt * kWmTile;
  const int64_t base = blk * kWmTile + warp * (32 * kWmPer);
  uint32_t key[kWmPer];
  int ones = 0;
#pragma unroll
  for (int k = 0; k < kWmPer; ++k) {
    const int64_t p = base + 32 * k + lane;
    key[k] = p < m ? src[p] : 0u;
    ones += __popc(__ballot_sync(0xFFFFFFFFu, (key[k] >> bit) & 1u));
  }
  if (lane == 0) wsum[warp] = (uint32_t)ones;
  __syncthreads();
  const uint32_t tile_pre = red[0], zeros = (uint32_t)(m - red[1]);
  if (blk == 0 && tid == 0) W.zeros[level] = zeros;
  uint32_t run = tile_pre;
  for (int k = 0; k < warp; ++k) run += wsum[k];
  // first destination tile of this tile's zeros and ones
  const uint32_t z0 = ((uint32_t)(blk * kWmTile) - tile_pre) / kWmTile;
  const uint32_t o0 = (zeros + tile_pre) / kWmTile;
  int n4[4] = {0, 0, 0, 0};
#pragma unroll
  for (int k = 0; k < kWmPer; ++k) {
    const int64_t p = base + 32 * k + lane;
    const bool one = (key[k] >> bit) & 1u;
    const uint32_t bal = __ballot_sync(0xFFFFFFFFu, one);
    if (lane == 0) W.level[(int64_t)level * nt * kWmWords + (p >> 5)] = make_uint2(run, bal);
    const uint32_t before = run + __popc(bal & lanemask_lt());
    run += __popc(bal);
    if (level == 31) continue;
    const uint32_t d = one ? zeros + before : (uint32_t)p - before;
    if (p < m) dst[d] = key[k];
    const bool nb = p < m && ((key[k] >> (bit - 1)) & 1u);
    const bool second = d / kWmTile != (one ? o0 : z0);
    const uint32_t b_nb = __ballot_sync(0xFFFFFFFFu, nb);
    const uint32_t b_s = __ballot_sync(0xFFFFFFFFu, second);
    n4[0] += __popc(b_nb & ~bal & ~b_s);
    n4[1] += __popc(b_nb & ~bal & b_s);
    n4[2] += __popc(b_nb & bal & ~b_s);
    n4[3] += __popc(b_nb & bal & b_s);
  }
  if (level == 31) return;
  if (lane == 0)
    for (int q = 0; q < 4; ++q)
      if (n4[q]) atomicAdd(&nxt[q], n4[q]);
  __syncthreads();
  if (tid < 4 && nxt[tid])
    atomicAdd(&W.count[(level + 1) * nt + (tid < 2 ? z0 : o0) + (tid & 1)], nxt[tid]);
}

// out[i]: the key of rank w / 2 among positions [i, i + w), or x[i] minus it.
__global__ void __launch_bounds__(256)
wm_median_kernel(const float* __restrict__ x, int64_t n, int w, int subtract, WmScratch W,
                 float* __restrict__ out) {
  __shared__ uint32_t zeros[32];
  if (threadIdx.x < 32) zeros[threadIdx.x] = W.zeros[threadIdx.x];
  __syncthreads();
  const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (i >= n) return;
  uint32_t l = (uint32_t)i, r = (uint32_t)i + (uint32_t)w, k = (uint32_t)w / 2, key = 0;
  const int64_t stride = W.ntiles * kWmWords;
#pragma unroll 4
  for (int level = 0; level < 32; ++level) {
    const uint2* L = W.level + level * stride;
    const uint2 a = __ldg(L + (l >> 5)), b = __ldg(L + (r >> 5));
    const uint32_t ol = a.x + __popc(a.y & ((1u << (l & 31)) - 1u));
    const uint32_t orr = b.x + __popc(b.y & ((1u << (r & 31)) - 1u));
    const uint32_t nz = (r - l) - (orr - ol);
    if (k < nz) {
      l -= ol;
      r -= orr;
    } else {
      k -= nz;
      l = zeros[level] + ol;
      r = zeros[level] + orr;
      key |= 0x80000000u >> level;
    }
  }
  const float med = key2f(key);
  out[i] = subtract ? __fsub_rn(x[i], med) : med;
}

// ---------------------------------------------------------------------------
// Order statistics: up to four ranks by radix select over 11 + 11 + 10 bits of
// the key. One launch a digit: every block adds its histograms to the global
// ones, and the last block to finish picks each rank's digit.
// ---------------------------------------------------------------------------

constexpr int kSelRanks = 4;
constexpr int kSelBins = 2048;
constexpr int kSelThreads = 512;

struct SelMulti {
  unsigned prefix[kSelRanks];
  long long k[kSelRanks];
  unsigned done;  // blocks finished with the current digit
};

struct SelRanks {
  long long k[kSelRanks];
  int n;
};

__global__ void __launch_bounds__(kSelThreads)
select_multi_kernel(const float* __restrict__ x, int64_t n, int digit, SelRanks ranks,
                    SelMulti* __restrict__ st, unsigned* __restrict__ hist,
                    float* __restrict__ out) {
  __shared__ unsigned h[kSelRanks * kSelBins];
  __shared__ unsigned wtot[kSelThreads / 32];
  __shared__ bool last;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int shift = digit == 0 ? 21 : digit == 1 ? 10 : 0;
  const int bins = digit == 2 ? 1024 : 2048;
  const unsigned mask = digit == 0 ? 0u : digit == 1 ? 0xFFE00000u : 0xFFFFFC00u;
  const int nh = digit == 0 ? 1 : ranks.n;  // the first digit's histogram serves every rank
  unsigned prefix[kSelRanks];
#pragma unroll
  for (int q = 0; q < kSelRanks; ++q) prefix[q] = digit && q < nh ? st->prefix[q] : 0u;
  for (int j = tid; j < nh * kSelBins; j += kSelThreads) h[j] = 0;
  __syncthreads();
  for (int64_t i = blockIdx.x * (int64_t)kSelThreads + tid; i < n;
       i += (int64_t)gridDim.x * kSelThreads) {
    const unsigned key = load_key(x + i);
#pragma unroll
    for (int q = 0; q < kSelRanks; ++q)
      if (q < nh && (key & mask) == prefix[q])
        atomicAdd(&h[q * kSelBins + ((key >> shift) & (unsigned)(bins - 1))], 1u);
  }
  __syncthreads();
  for (int j = tid; j < nh * kSelBins; j += kSelThreads)
    if (h[j]) atomicAdd(&hist[j], h[j]);
  __threadfence();
  __syncthreads();
  if (tid == 0) last = atomicAdd(&st->done, 1u) == gridDim.x - 1;
  __syncthreads();
  if (!last) return;
  __threadfence();
  for (int q = 0; q < ranks.n; ++q) {
    const unsigned* hq = hist + (digit == 0 ? 0 : q) * kSelBins;
    const long long k = digit == 0 ? ranks.k[q] : st->k[q];
    constexpr int kPer = kSelBins / kSelThreads;
    unsigned c[kPer], sum = 0;
#pragma unroll
    for (int j = 0; j < kPer; ++j) sum += c[j] = __ldcg(hq + tid * kPer + j);
    unsigned incl = sum;
    for (int o = 1; o < 32; o <<= 1) {
      const unsigned y = __shfl_up_sync(0xFFFFFFFFu, incl, o);
      if (lane >= o) incl += y;
    }
    if (lane == 31) wtot[warp] = incl;
    __syncthreads();
    long long before = incl - sum;
    for (int j = 0; j < warp; ++j) before += wtot[j];
    __syncthreads();
    if (k >= before && k < before + sum) {  // exactly one thread: its bins hold the rank
      long long kk = k - before;
      int j = 0;
#pragma unroll
      for (int u = 0; u < kPer - 1; ++u)
        if (j == u && kk >= c[u]) {
          kk -= c[u];
          j = u + 1;
        }
      const unsigned p = (digit ? st->prefix[q] : 0u) | ((unsigned)(tid * kPer + j) << shift);
      st->prefix[q] = p;
      st->k[q] = kk;
      if (digit == 2) out[q] = key2f(p);
    }
    __syncthreads();
  }
  for (int j = tid; j < nh * kSelBins; j += kSelThreads) hist[j] = 0;
  if (tid == 0) st->done = 0;
}

// sum of x (or of x^2) in float64: per-block partial sums, then one block
// adds them
__global__ void __launch_bounds__(256)
sum_f64_kernel(const float* __restrict__ x, int64_t n, int square, double* __restrict__ part) {
  __shared__ double w[8];
  double a = 0.0;
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n;
       i += (int64_t)gridDim.x * blockDim.x) {
    const double v = (double)x[i];
    a += square ? v * v : v;
  }
  for (int o = 16; o > 0; o >>= 1) a += __shfl_down_sync(0xFFFFFFFFu, a, o);
  if ((threadIdx.x & 31) == 0) w[threadIdx.x >> 5] = a;
  __syncthreads();
  if (threadIdx.x == 0) {
    double t = 0.0;
    for (int k = 0; k < 8; ++k) t += w[k];
    part[blockIdx.x] = t;
  }
}

__global__ void sum_parts_kernel(const double* __restrict__ part, int nparts,
                                 double* __restrict__ out) {
  __shared__ double w[32];
  double a = 0.0;
  for (int k = threadIdx.x; k < nparts; k += blockDim.x) a += part[k];
  for (int o = 16; o > 0; o >>= 1) a += __shfl_down_sync(0xFFFFFFFFu, a, o);
  if ((threadIdx.x & 31) == 0) w[threadIdx.x >> 5] = a;
  __syncthreads();
  if (threadIdx.x == 0) {
    double t = 0.0;
    for (int k = 0; k < (int)(blockDim.x + 31) / 32; ++k) t += w[k];
    *out = t;
  }
}

// y = (x - loc) / scale, float32 arithmetic, or |x - loc| when scale == 0
__global__ void affine_kernel(const float* __restrict__ x, int64_t n, float loc, float scale,
                              float* __restrict__ y) {
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n;
       i += (int64_t)gridDim.x * blockDim.x) {
    const float d = __fsub_rn(x[i], loc);
    y[i] = scale == 0.0f ? fabsf(d) : __fdiv_rn(d, scale);
  }
}

}  // namespace loki

using namespace loki;

extern "C" int loki_running_median(const float* x, int64_t n, int32_t window,
                                   int32_t subtract, float* out, void* stream) {
  if (!x || !out) return set_error(LOKI_ERR_INVALID, "null pointer argument");
  if (n <= 0) return set_error(LOKI_ERR_INVALID, "n must be > 0");
  if (window < 1) return set_error(LOKI_ERR_INVALID, "window %d must be >= 1", window);
  if (window > kMedMaxWindow)
    return set_error(LOKI_ERR_UNSUPPORTED, "window %d above %d", window, kMedMaxWindow);
  int pw = 1;
  while (pw < window) pw <<= 1;
  pw = std::max(pw, 2);
  const int smem = pw * (int)sizeof(float);
  if (set_smem_limit(running_median_kernel, smem) != cudaSuccess)
    return set_error(LOKI_ERR_CUDA, "cudaFuncSetAttribute failed");
  int dev = 0, nsm = 0;
  if (cudaGetDevice(&dev) != cudaSuccess ||
      cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess)
    return set_error(LOKI_ERR_CUDA, "device query failed");
  // one block per SM (registers and the window's shared memory), each output
  // chunk long enough to pay for its sort
  const int64_t blocks = std::max<int64_t>(
      1, std::min<int64_t>((int64_t)nsm, (n + 4 * (int64_t)window - 1) / (4 * window)));
  const int64_t chunk = (n + blocks - 1) / blocks;
  note_launch();
  running_median_kernel<<<(unsigned)blocks, kMedThreads, smem, (cudaStream_t)stream>>>(
      x, n, window, pw, chunk, subtract, out);
  return check_launch("running_median");
}

extern "C" int64_t loki_running_median_scratch_bytes(int64_t n, int32_t window) {
  if (n <= 0 || window < 1 || window > kMedMaxWindow || n + window > (int64_t(1) << 31)) return 0;
  return wm_bytes(wm_tiles(n + window - 1));
}

extern "C" int loki_running_median_scratch(const float* x, int64_t n, int32_t window,
                                           int32_t subtract, float* out, void* scratch,
                                           int64_t scratch_bytes, void* stream) {
  if (!x || !out || !scratch) return set_error(LOKI_ERR_INVALID, "null pointer argument");
  if (n <= 0) return set_error(LOKI_ERR_INVALID, "n must be > 0");
  if (window < 1) return set_error(LOKI_ERR_INVALID, "window %d must be >= 1", window);
  if (window > kMedMaxWindow)
    return set_error(LOKI_ERR_UNSUPPORTED, "window %d above %d", window, kMedMaxWindow);
  const int64_t need = loki_running_median_scratch_bytes(n, window);
  if (need == 0)
    return set_error(LOKI_ERR_UNSUPPORTED, "%lld samples above 2^31", (long long)n);
  if (scratch_bytes < need)
    return set_error(LOKI_ERR_CAPACITY, "median scratch below %lld bytes", (long long)need);
  if ((reinterpret_cast<uintptr_t>(scratch) & 15) != 0)
    return set_error(LOKI_ERR_INVALID, "scratch must be 16-byte aligned");
  cudaStream_t s = (cudaStream_t)stream;
  const int64_t m = n + window - 1, nt = wm_tiles(m);
  const WmScratch W = wm_layout(scratch, nt);
  if (cudaMemsetAsync(W.count, 0, 32 * nt * sizeof(int32_t), s) != cudaSuccess)
    return set_error(LOKI_ERR_CUDA, "cudaMemsetAsync failed");
  for (int i = 0; i < 34; ++i) note_launch();
  wm_keys_kernel<<<(unsigned)nt, kWmThreads, 0, s>>>(x, n, window / 2, m, W);
  for (int level = 0; level < 32; ++level)
    wm_level_kernel<<<(unsigned)nt, kWmThreads, 0, s>>>(level, m, W);
  wm_median_kernel<<<(unsigned)((n + 255) / 256), 256, 0, s>>>(x, n, window, subtract, W, out);
  return check_launch("running_median");
}

extern "C" int64_t loki_select_scratch_bytes(void) {
  return kSelRanks * kSelBins * (int64_t)sizeof(unsigned) + (int64_t)sizeof(SelMulti) + 64;
}

extern "C" int loki_select_ranks(const float* x, int64_t n, const int64_t* ranks, int32_t nranks,
                                 float* out, void* scratch, int64_t scratch_bytes,
                                 void* stream) {
  if (!x || !ranks || !out || !scratch)
    return set_error(LOKI_ERR_INVALID, "null pointer argument");
  if (nranks < 1 || nranks > kSelRanks)
    return set_error(LOKI_ERR_INVALID, "need 1..%d ranks", kSelRanks);
  SelRanks r{};
  r.n = nranks;
  for (int q = 0; q < nranks; ++q) {
    if (n <= 0 || ranks[q] < 0 || ranks[q] >= n)
      return set_error(LOKI_ERR_INVALID, "need 0 <= k < n");
    r.k[q] = ranks[q];
  }
  if (scratch_bytes < loki_select_scratch_bytes())
    return set_error(LOKI_ERR_CAPACITY, "select scratch below %lld bytes",
                     (long long)loki_select_scratch_bytes());
  cudaStream_t s = (cudaStream_t)stream;
  SelMulti* st = reinterpret_cast<SelMulti*>(scratch);
  unsigned* hist = reinterpret_cast<unsigned*>(st + 1);
  if (cudaMemsetAsync(scratch, 0, sizeof(SelMulti) + kSelRanks * kSelBins * sizeof(unsigned), s) !=
      cudaSuccess)
    return set_error(LOKI_ERR_CUDA, "cudaMemsetAsync failed");
  const int blocks = (int)std::min<int64_t>((n + 4095) / 4096, 152 * 4);
  for (int digit = 0; digit < 3; ++digit) {
    note_launch();
    select_multi_kernel<<<blocks, kSelThreads, 0, s>>>(x, n, digit, r, st, hist, out);
  }
  return check_launch("select_ranks");
}

extern "C" int loki_select_kth(const float* x, int64_t n, int64_t k, float* out,
                               void* scratch, int64_t scratch_bytes, void* stream) {
  return loki_select_ranks(x, n, &k, 1, out, scratch, scratch_bytes, stream);
}

extern "C" int loki_sum_f64(const float* x, int64_t n, int32_t square, double* out,
                            void* scratch, int64_t scratch_bytes, void* stream) {
  if (!x || !out || !scratch) return set_error(LOKI_ERR_INVALID, "null pointer argument");
  if (n < 0) return set_error(LOKI_ERR_INVALID, "n must be >= 0");
  const int blocks = (int)std::max<int64_t>(1, std::min<int64_t>((n + 255) / 256, 1024));
  if (scratch_bytes < blocks * (int64_t)sizeof(double))
    return set_error(LOKI_ERR_CAPACITY, "sum scratch below %d doubles", blocks);
  cudaStream_t s = (cudaStream_t)stream;
  double* part = reinterpret_cast<double*>(scratch);
  note_launch();
  note_launch();
  sum_f64_kernel<<<blocks, 256, 0, s>>>(x, n, square, part);
  sum_parts_kernel<<<1, 256, 0, s>>>(part, blocks, out);
  return check_launch("sum_f64");
}

extern "C" int loki_affine(const float* x, int64_t n, float loc, float scale, float* y,
                           void* stream) {
  if (!x || !y) return set_error(LOKI_ERR_INVALID, "null pointer argument");
  if (n <= 0) return LOKI_OK;
  const int blocks = (int)std::min<int64_t>((n + 255) / 256, 152 * 16);
  note_launch();
  affine_kernel<<<blocks, 256, 0, (cudaStream_t)stream>>>(x, n, loc, scale, y);
  return check_launch("affine");
}
