// Enumerate-prune kernels for the Taylor basis with float32 folds
// (prune.py:165-332 pruning_iteration_batched with the PrunePolyTaylorDPFuncts
// plugin, dynamic/dyn_poly_taylor.py:396-690).
//
// One level = branch (per parent) -> exclusive scan of child counts -> score
// (per child: branch value, FP64 resolve, gather + roll + add, boxcar S/N) ->
// selection (in child order, with the exact overflow rule when needed) ->
// emit (transform the survivors, write the new tree). Child order is parent
// order then the C-order odometer over the branched parameters, which is the
// order the reference appends survivors in.
//
// FP64 arithmetic follows the reference's numpy operations with round-to-
// nearest intrinsics (no contraction); the batched Taylor shifts reproduce
// the BLAS matrix product, which accumulates each output with forward fused
// multiply-adds (acc = fma(x_j, T_ij, acc), j = 0..P).
#include <algorithm>
#include <vector>

#include "loki_common.cuh"
#include "score.cuh"
#include "sincos.cuh"

namespace loki {

int score_smem_bytes(int nbins, int wmax, int warps);

// ---------------------------------------------------------------------------
// exclusive scan of int64 (counts) or of score >= threshold flags
// ---------------------------------------------------------------------------

constexpr int kScanBlock = 1024;

template <bool FLAGS>
__device__ __forceinline__ int64_t scan_in(const void* in, int64_t i, int64_t n, double thr) {
  if (i >= n) return 0;
  if (FLAGS) return ((double)reinterpret_cast<const float*>(in)[i] >= thr) ? 1 : 0;
  return reinterpret_cast<const int64_t*>(in)[i];
}

// One kScanBlock-element tile of the scan: exclusive within the tile, the
// tile's total in sums[tile].
template <bool FLAGS>
__device__ __forceinline__ void scan_tile(const void* in, int64_t n, double thr, int64_t* out,
                                          int64_t* sums, int64_t tile, int64_t* warp_tot) {
  const int64_t i = tile * kScanBlock + threadIdx.x;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int64_t x = scan_in<FLAGS>(in, i, n, thr);
  int64_t v = x;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int64_t y = __shfl_up_sync(0xFFFFFFFFu, v, o);
    if (lane >= o) v += y;
  }
  if (lane == 31) warp_tot[warp] = v;
  __syncthreads();
  if (warp == 0) {
    int64_t w = warp_tot[lane];
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int64_t y = __shfl_up_sync(0xFFFFFFFFu, w, o);
      if (lane >= o) w += y;
    }
    warp_tot[lane] = w;  // inclusive over warps
  }
  __syncthreads();
  const int64_t incl = v + (warp ? warp_tot[warp - 1] : 0);
  if (i < n) out[i] = incl - x;  // exclusive within the block
  if (threadIdx.x == kScanBlock - 1) sums[tile] = incl;
  __syncthreads();  // warp_tot is reused by the next tile
}

// n_dev, when not null, holds the element count on the device: the blocks
// then stride over its tiles.
template <bool FLAGS>
__global__ void __launch_bounds__(kScanBlock)
scan_block_kernel(const void* in, int64_t n, const int64_t* n_dev, double thr, int64_t* out,
                  int64_t* sums) {
  __shared__ int64_t warp_tot[32];
  if (!n_dev) {
    scan_tile<FLAGS>(in, n, thr, out, sums, blockIdx.x, warp_tot);
    return;
  }
  n = *n_dev;
  const int64_t ntiles = (n + kScanBlock - 1) / kScanBlock;
  for (int64_t t = blockIdx.x; t < ntiles; t += gridDim.x)  // uniform over the block
    scan_tile<FLAGS>(in, n, thr, out, sums, t, warp_tot);
}

// Single block: exclusive scan of the block sums (any count), carry-chained.
// With n_dev the block count and the total's slot (out + n) come from the
// device count.
__global__ void __launch_bounds__(kScanBlock)
scan_sums_kernel(int64_t* sums, int64_t nblocks, int64_t* total, const int64_t* n_dev,
                 int64_t* out) {
  __shared__ int64_t warp_tot[32];
  __shared__ int64_t carry;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if (n_dev) {
    const int64_t n = *n_dev;
    nblocks = (n + kScanBlock - 1) / kScanBlock;
    total = out + n;
  }
  if (threadIdx.x == 0) carry = 0;
  __syncthreads();
  for (int64_t base = 0; base < nblocks; base += kScanBlock) {
    const int64_t i = base + threadIdx.x;
    const int64_t x = i < nblocks ? sums[i] : 0;
    int64_t v = x;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int64_t y = __shfl_up_sync(0xFFFFFFFFu, v, o);
      if (lane >= o) v += y;
    }
    if (lane == 31) warp_tot[warp] = v;
    __syncthreads();
    if (warp == 0) {
      int64_t w = warp_tot[lane];
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int64_t y = __shfl_up_sync(0xFFFFFFFFu, w, o);
        if (lane >= o) w += y;
      }
      warp_tot[lane] = w;
    }
    __syncthreads();
    const int64_t incl = v + (warp ? warp_tot[warp - 1] : 0);
    const int64_t c = carry;
    if (i < nblocks) sums[i] = c + incl - x;
    __syncthreads();
    if (threadIdx.x == kScanBlock - 1) carry = c + incl;
    __syncthreads();
  }
  if (threadIdx.x == 0) *total = carry;
}

__global__ void scan_add_kernel(int64_t* out, int64_t n, const int64_t* n_dev,
                                const int64_t* sums) {
  if (!n_dev) {
    const int64_t i = (int64_t)blockIdx.x * kScanBlock + threadIdx.x;
    if (i < n) out[i] += sums[blockIdx.x];
    return;
  }
  n = *n_dev;
  for (int64_t i = (int64_t)blockIdx.x * kScanBlock + threadIdx.x; i < n;
       i += (int64_t)gridDim.x * kScanBlock)
    out[i] += sums[i / kScanBlock];
}

// out[0..n) exclusive scan, out[n] = total.
template <bool FLAGS>
static int exclusive_scan(const void* in, int64_t n, double thr, int64_t* out, void* scratch,
                          int64_t scratch_bytes, cudaStream_t s) {
  const int64_t nblocks = std::max<int64_t>(1, (n + kScanBlock - 1) / kScanBlock);
  if (scratch_bytes < nblocks * (int64_t)sizeof(int64_t))
    return set_error(LOKI_ERR_CAPACITY, "scan scratch too small");
  int64_t* sums = reinterpret_cast<int64_t*>(scratch);
  if (n == 0) {
    if (cudaMemsetAsync(out, 0, sizeof(int64_t), s) != cudaSuccess)
      return set_error(LOKI_ERR_CUDA, "cudaMemsetAsync failed");
    return LOKI_OK;
  }
  for (int i = 0; i < 3; ++i) note_launch();
  scan_block_kernel<FLAGS><<<(unsigned)nblocks, kScanBlock, 0, s>>>(in, n, nullptr, thr, out,
                                                                    sums);
  scan_sums_kernel<<<1, kScanBlock, 0, s>>>(sums, nblocks, out + n, nullptr, nullptr);
  scan_add_kernel<<<(unsigned)nblocks, kScanBlock, 0, s>>>(out, n, nullptr, sums);
  return check_launch("exclusive_scan");
}

// The same scan over a device-held count *n_dev <= n_cap (no host wait):
// out[0..n) exclusive scan, out[n] = total. At most `grid` blocks stride over
// the tiles.
template <bool FLAGS>
static int exclusive_scan_dev(const void* in, int64_t n_cap, const int64_t* n_dev, double thr,
                              int64_t* out, void* scratch, int64_t scratch_bytes, int grid,
                              cudaStream_t s) {
  const int64_t ntiles = std::max<int64_t>(1, (n_cap + kScanBlock - 1) / kScanBlock);
  if (scratch_bytes < ntiles * (int64_t)sizeof(int64_t))
    return set_error(LOKI_ERR_CAPACITY, "scan scratch too small");
  const unsigned blocks = (unsigned)std::max<int64_t>(1, std::min<int64_t>(ntiles, grid));
  int64_t* sums = reinterpret_cast<int64_t*>(scratch);
  for (int i = 0; i < 3; ++i) note_launch();
  scan_block_kernel<FLAGS><<<blocks, kScanBlock, 0, s>>>(in, n_cap, n_dev, thr, out, sums);
  scan_sums_kernel<<<1, kScanBlock, 0, s>>>(sums, ntiles, nullptr, n_dev, out);
  scan_add_kernel<<<blocks, kScanBlock, 0, s>>>(out, n_cap, n_dev, sums);
  return check_launch("exclusive_scan_dev");
}

// ---------------------------------------------------------------------------
// shared FP64 pieces
// ---------------------------------------------------------------------------

// y_i = sum_j x_j T_ij accumulated with forward fused multiply-adds.
__device__ __forceinline__ double tdot(const double* x, const double (*T)[LOKI_MAX_PARAMS + 1],
                                       int i, int m) {
  double acc = 0.0;
  for (int j = 0; j < m; ++j) acc = __fma_rn(x[j], T[i][j], acc);
  return acc;
}

// get_nearest_indices_2d_batch for one axis (utils/psr_utils.py:517-554).
__device__ __forceinline__ int64_t axis_index(double v, double vmin, double inv, int64_t n) {
  if (!(inv > 0.0)) return 0;
  const double raw = __dmul_rn(__dsub_rn(v, vmin), inv);
  int64_t idx = (int64_t)__dadd_rn(raw, LOKI_FLOAT_EPSILON);
  if (idx < 0) idx = 0;
  else if (idx >= n) idx = n - 1;
  return idx;
}

// The tree's order as a constant where the kernel has one (KP > 0): the loops
// over it unroll and a child's parameters stay in registers instead of local
// memory.
template <int KP>
__device__ __forceinline__ int tree_order(const LokiPruneLevel& D) {
  return KP > 0 ? KP : D.poly_order;
}

// Child leaf parameters [d_P .. d_1] from the parent's branching info.
__device__ __forceinline__ void child_params(const LokiBranchInfo& B, int P, int64_t local,
                                             double* pv) {
  // a parent has at most branch_max^P children: 32-bit arithmetic, and none for
  // the parameters that did not split
  uint32_t rest = (uint32_t)local;
  for (int j = P - 1; j >= 0; --j) {
    const uint32_t c = (uint32_t)B.count[j];
    if (c == 1) {
      pv[j] = B.first[j];
      continue;
    }
    const uint32_t q = rest / c, k = rest - q * c;
    rest = q;
    pv[j] = __dadd_rn(B.first[j], __dmul_rn((double)k, B.dact[j]));
  }
}

struct ChildRes {
  int32_t ia, iff;  // (accel, freq) FFA grid indices
  double phase;
};

// cheby_to_taylor (utils/transforms.py:556-583) of coefficients a[0..P]
// (alpha_P..alpha_0), lowest three Taylor orders only: d_k =
// ((rev(a) @ R)[k] * k!) / scale**k for k = 2 (accel), 1 (velocity), 0 (delay).
__device__ __forceinline__ void cheby_low3(const LokiPruneLevel& D, const double* a, int m,
                                           double* d2, double* d1, double* d0) {
  double ar[LOKI_MAX_PARAMS + 1];
  for (int i = 0; i < m; ++i) ar[i] = a[m - 1 - i];
  double d[3];
  for (int k = 0; k < 3; ++k)
    d[k] = __ddiv_rn(__dmul_rn(tdot(ar, D.tm_r, k, m), D.cfact[k]), D.ctsk[k]);
  *d0 = d[0];
  *d1 = d[1];
  *d2 = d[2];
}

// Chebyshev resolve (core/chebyshev.py:180-277): shift the coefficients to
// t_add (and t_init on the moving grid) at the current scale, then read the
// Taylor accel / velocity / delay there.
__device__ __forceinline__ void cheby_kinematics(const LokiPruneLevel& D, int P,
                                                 const double* pv, double* accel, double* vel,
                                                 double* dd) {
  const int m = P + 1;
  double a[LOKI_MAX_PARAMS + 1];
  for (int i = 0; i < m; ++i) a[i] = tdot(pv, D.tm_a, i, m);
  double a2, a1, a0;
  cheby_low3(D, a, m, &a2, &a1, &a0);
  *accel = a2;
  if (D.moving) {
    for (int i = 0; i < m; ++i) a[i] = tdot(pv, D.tm_i, i, m);
    double i2, i1, i0;
    cheby_low3(D, a, m, &i2, &i1, &i0);
    *vel = __dsub_rn(a1, i1);
    *dd = __dsub_rn(a0, i0);
  } else {
    *vel = a1;
    *dd = a0;
  }
}

// poly_taylor_resolve_batch (moving) / poly_taylor_fixed_resolve_batch
// (core/taylor.py:172-277) for one child with params pv[0..P] (d_P..d_1, d_0).
__device__ __forceinline__ ChildRes resolve_child(const LokiPruneLevel& D, int P,
                                                  const double* pv, double f0) {
  const int m = P + 1;
  double accel, vel, dd;
  if (D.basis == 1) {
    cheby_kinematics(D, P, pv, &accel, &vel, &dd);
  } else if (D.moving) {
    accel = tdot(pv, D.tm_a, P - 2, m);
    vel = __dsub_rn(tdot(pv, D.tm_a, P - 1, m), tdot(pv, D.tm_i, P - 1, m));
    dd = __dsub_rn(tdot(pv, D.tm_a, P, m), tdot(pv, D.tm_i, P, m));
  } else {
    accel = tdot(pv, D.tm_a, P - 2, m);
    vel = tdot(pv, D.tm_a, P - 1, m);
    dd = tdot(pv, D.tm_a, P, m);
  }
  const double freq = __dmul_rn(f0, __dsub_rn(1.0, div_c(vel)));
  const double delay = div_c(dd);
  ChildRes r;
  r.phase = phase_idx(D.dt_phase, f0, D.nbins, delay);
  r.ia = (int32_t)axis_index(accel, D.accel_min, D.accel_inv, D.n_accel);
  r.iff = (int32_t)axis_index(freq, D.freq_min, D.freq_inv, D.n_freq);
  return r;
}

// ---------------------------------------------------------------------------
// branch
// ---------------------------------------------------------------------------

// The level's steps, factors and shift limit in float32, for branch_quick.
struct BranchF {
  float dfc[LOKI_MAX_PARAMS], fac[LOKI_MAX_PARAMS], eta;
};

__device__ __forceinline__ BranchF branch_floats(const LokiPruneLevel& D) {
  BranchF F;
  for (int j = 0; j < LOKI_MAX_PARAMS; ++j) {
    F.dfc[j] = (float)D.dfc[j];
    F.fac[j] = (float)D.fac[j];
  }
  F.eta = (float)D.eta_m;
  return F;
}

// Whether parameter j (step dcur) splits, and into how many (*num), where
// float32 settles what float64 decides: 1 or 0; -1 where it does not (a value
// within the rounding of a limit or of a whole ratio, out of float32's range,
// not positive, or beyond branch_max) and the float64 chain has to be run. Each
// approximation is off by at most 10 roundings of 2^-24 (6e-7); the margins are
// 2e-6 and more. The FP64 unit (16 clocks of the SM for an instruction of a warp)
// was 73 % busy in the branch kernel, most of it with the divisions of the split
// and the ratio, 9 to 13 a parent of order 4; what is left is one for each
// parameter that splits into a count that is no power of two. 64 runs of 128
// levels: 5.5 -> 2.8 ms; 16 of the circular tree: 4.0 -> 1.7.
__device__ __forceinline__ int branch_quick(const BranchF& F, int j, float f0, float rf0,
                                            double dcur, int64_t branch_max, int* num) {
  const float dc = (float)dcur, dn = F.dfc[j] * rf0;
  const float fb = F.fac[j] * f0 * (float)(1.0 / LOKI_C_VAL);
  const float lo = 1e-30f, hi = 1e30f;
  if (!(dc > lo && dc < hi && dn > lo && dn < hi && fb > lo && fb < hi && F.eta > 1e-20f &&
        F.eta < 1e20f))
    return -1;
  const float shift = fabsf(dc - dn) * fb, err = (dc + dn) * fb * 2e-6f;
  const float ratio = __fdividef(dc, dn), bm = (float)branch_max;
  if (shift + err < F.eta * (1.0f - 2e-6f)) return ratio * (1.0f + 4e-6f) < bm ? 0 : -1;
  if (!(shift - err > F.eta * (1.0f + 2e-6f)) || !(ratio < 1e5f)) return -1;
  const float x = ratio - (float)LOKI_FLOAT_EPSILON, m = ratio * 4e-6f + 1e-9f;
  const float c = ceilf(x - m);
  if (c != ceilf(x + m) || c > bm) return -1;
  *num = max((int)c, 1);
  return 1;
}

// dcur / num: by a power of two exact scaling.
__device__ __forceinline__ double branch_step(double dcur, int64_t num) {
  return num == 1                 ? dcur
         : (num & (num - 1)) == 0 ? __dmul_rn(dcur, 1.0 / (double)num)
                                  : __ddiv_rn(dcur, (double)num);
}

// Parent i: per-parameter child counts, steps and first values (info[i]) and
// its child count (counts[i]).
template <int KP = 0>
__device__ __forceinline__ void branch_one(const LokiPruneLevel& D,
                                           const double* __restrict__ leaves, int64_t i,
                                           LokiBranchInfo* __restrict__ info,
                                           int64_t* __restrict__ counts,
                                           int32_t* __restrict__ err,
                                           const uint8_t* __restrict__ mask,
                                           const BranchF& F) {
  const int P = tree_order<KP>(D), m = P + 1;
  const double* lf = leaves + i * (P + 2) * 2;
  const double f0 = lf[(P + 1) * 2];
  const float f0f = (float)f0, rf0 = __frcp_rn(f0f);
  // Parent values and errors in the current domain: as stored (Taylor), or
  // shifted from the previous to the current Chebyshev domain with
  // shift_cheby_full (utils/transforms.py:650-701).
  double pval[LOKI_MAX_PARAMS + 1], perr[LOKI_MAX_PARAMS + 1];
  if (D.basis == 1) {
    double raw[LOKI_MAX_PARAMS + 1], rawe[LOKI_MAX_PARAMS + 1];
    for (int k = 0; k < m; ++k) {
      raw[k] = lf[2 * k];
      rawe[k] = lf[2 * k + 1];
    }
    for (int k = 0; k < m; ++k) pval[k] = tdot(raw, D.tm_b, k, m);
    if (D.tiling == 0) {
      for (int k = 0; k < m; ++k) perr[k] = __dmul_rn(rawe[k], fabs(D.tm_b[k][k]));
    } else if (D.tiling == 2) {
      for (int k = 0; k < m; ++k) perr[k] = tdot(rawe, D.tm_be, k, m);
    } else {
      double e2[LOKI_MAX_PARAMS + 1];
      for (int k = 0; k < m; ++k) e2[k] = __dmul_rn(rawe[k], rawe[k]);
      for (int k = 0; k < m; ++k) perr[k] = __dsqrt_rn(tdot(e2, D.tm_be, k, m));
    }
  } else {
    for (int k = 0; k < m; ++k) {
      pval[k] = lf[2 * k];
      perr[k] = lf[2 * k + 1];
    }
  }
  // Halving is exact, so x / 2 is computed as x * 0.5 (the same rounded
  // value as the reference's division).
  LokiBranchInfo B;
  B.d0 = pval[P];
  int64_t total = 1;
  for (int j = 0; j < P; ++j) {
    const double pcur = pval[j], dcur = perr[j];
    int quick_num = 1;
    const int quick = branch_quick(F, j, f0f, rf0, dcur, D.branch_max, &quick_num);
    bool split = quick > 0;
    int64_t num = quick_num;
    if (quick < 0) {
      const double dnew = __ddiv_rn(D.dfc[j], f0);
      const double fb = __dmul_rn(D.fac[j], __ddiv_rn(f0, LOKI_C_VAL));
      const double shift = __dmul_rn(fabs(__dsub_rn(dcur, dnew)), fb);
      split = !(shift < D.eta_m);
      num = 1;
      if (!(dcur > 0.0) || !(dnew > 0.0)) {
        atomicOr(err, LOKI_DEVERR_BRANCH);
        split = false;
      } else if (split || dcur > __dmul_rn(dnew, 0.5 * (double)D.branch_max)) {
        // The child count is needed for a split, and for the reference's
        // branch_max check of every parameter; a parameter that does not
        // split and whose step is at most half of branch_max new steps cannot
        // exceed branch_max (ratio <= branch_max / 2 up to rounding), so its
        // division is skipped.
        const double ratio = __ddiv_rn(dcur, dnew);
        num = (int64_t)ceil(__dsub_rn(ratio, LOKI_FLOAT_EPSILON));
        if (num < 1) num = 1;
        if (num > D.branch_max) {
          atomicOr(err, LOKI_DEVERR_BRANCH);
          num = D.branch_max;
        }
      }
    }
    double dact = dcur, first = pcur;
    if (split) {
      dact = branch_step(dcur, num);
      first = __dadd_rn(__dsub_rn(pcur, __dmul_rn(dcur, 0.5)), __dmul_rn(dact, 0.5));
    } else {
      num = 1;
    }
    B.first[j] = first;
    B.dact[j] = dact;
    B.count[j] = (int32_t)num;
    total *= num;
  }
  info[i] = B;
  counts[i] = (mask && !mask[i]) ? 0 : total;  // a masked-out parent has no children
}

__global__ void prune_branch_kernel(LokiPruneLevel D, const double* __restrict__ leaves,
                                    int64_t n, LokiBranchInfo* __restrict__ info,
                                    int64_t* __restrict__ counts, int32_t* __restrict__ err,
                                    const uint8_t* __restrict__ mask,
                                    const int64_t* __restrict__ n_dev) {
  if (n_dev) n = *n_dev;  // parent count held on the device
  const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (i >= n) return;
  branch_one(D, leaves, i, info, counts, err, mask, branch_floats(D));
}

// ---------------------------------------------------------------------------
// score: warp per 32 children
// ---------------------------------------------------------------------------

constexpr int kPruneWarps = 4;

__device__ __forceinline__ int64_t find_parent(const int64_t* offsets, int64_t n, int64_t c) {
  int64_t lo = 0, hi = n;  // offsets[lo] <= c < offsets[hi]
  while (hi - lo > 1) {
    const int64_t mid = (lo + hi) >> 1;
    if (offsets[mid] <= c) lo = mid;
    else hi = mid;
  }
  return lo;
}

// find_parent for a warp: lanes k < kmax hold ascending children c. The first
// lane's parent by a 32-way search, the others' among the 32 parents after it
// (a few windows; a lane beyond them searches alone). Four to five dependent
// loads where a binary search of every lane takes 12 to 16.
__device__ __forceinline__ int64_t warp_find_parents(const int64_t* __restrict__ offsets,
                                                     int64_t n, int64_t c, int kmax) {
  const int lane = threadIdx.x & 31;
  const int64_t c0 = __shfl_sync(0xFFFFFFFFu, c, 0);
  if (lane >= kmax) c = c0;
  int64_t lo = 0, hi = n;  // offsets[lo] <= c0 < offsets[hi]
  while (hi - lo > 32) {
    const int64_t step = (hi - lo + 31) / 32, i = lo + lane * step;
    const unsigned m = __ballot_sync(0xFFFFFFFFu, i < hi && offsets[i] <= c0);
    lo += (31 - __clz(m)) * step;
    hi = min(hi, lo + step);
  }
  lo += __popc(__ballot_sync(0xFFFFFFFFu, lo + lane < hi && offsets[lo + lane] <= c0)) - 1;
  int64_t par = -1;
  for (int w = 0; w < 4; ++w, lo += 32) {
    const int64_t off = offsets[min(lo + 1 + lane, n)];
    int k = 0;  // entries of the window at or below c
#pragma unroll
    for (int s = 16; s >= 1; s >>= 1)
      if (__shfl_sync(0xFFFFFFFFu, off, k + s - 1) <= c) k += s;
    if (__shfl_sync(0xFFFFFFFFu, off, k) <= c) ++k;
    if (par < 0 && k < 32) par = lo + k;
    if (__ballot_sync(0xFFFFFFFFu, par < 0) == 0) break;
  }
  return par >= 0 ? par : find_parent(offsets, n, c);
}

__device__ __forceinline__ unsigned float_key(float x) {
  const unsigned u = __float_as_uint(x);
  return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}

__device__ __forceinline__ float key_float(unsigned k) {
  return __uint_as_float((k & 0x80000000u) ? (k & 0x7FFFFFFFu) : ~k);
}

// Rows of 32 children (parent row, segment row and roll held lane by lane):
// shift-add, e / sqrt(v), one normalised profile per tile row.
__device__ __forceinline__ void gather_norm_rows(const float* __restrict__ folds,
                                                 const float* __restrict__ seg, int64_t my_par,
                                                 int64_t my_row, int my_shift, int kmax, int nb,
                                                 float* tile, int stride) {
  const int lane = threadIdx.x & 31;
  if (nb == 64) {
    // four children's rows in flight per lane (bins lane and lane + 32); eight cost
    // the batch kernel registers: 13.7 instead of 13.1 ms of score, 7.2 instead of
    // 6.2 in the circular tree
    constexpr int kU = 4;
    for (int k0 = 0; k0 < kmax; k0 += kU) {
      float pe[kU][2], pw[kU][2], se[kU][2], sw[kU][2];
#pragma unroll
      for (int u = 0; u < kU; ++u) {
        const int k = k0 + u;
        const int src = k < kmax ? k : 0;
        // (rows of 512 bytes: their numbers fit 32 bits)
        const uint32_t par = __shfl_sync(0xFFFFFFFFu, (uint32_t)my_par, src);
        const uint32_t row = __shfl_sync(0xFFFFFFFFu, (uint32_t)my_row, src);
        const int sh = __shfl_sync(0xFFFFFFFFu, my_shift, src);
        if (k < kmax) {
          const float* pf = folds + (size_t)par * 128;
          const float* sf = seg + (size_t)row * 128;
#pragma unroll
          for (int c = 0; c < 2; ++c) {
            const int j = lane + 32 * c;
            const int js = (j - sh) & 63;
            pe[u][c] = __ldg(pf + j);
            pw[u][c] = __ldg(pf + 64 + j);
            se[u][c] = __ldg(sf + js);
            sw[u][c] = __ldg(sf + 64 + js);
          }
        }
      }
#pragma unroll
      for (int u = 0; u < kU; ++u) {
        const int k = k0 + u;
        if (k >= kmax) break;
        float* trow = tile + k * stride;
#pragma unroll
        for (int c = 0; c < 2; ++c) {
          const float e = __fadd_rn(pe[u][c], se[u][c]);
          const float v = __fadd_rn(pw[u][c], sw[u][c]);
          trow[lane + 32 * c] = __fdiv_rn(e, __fsqrt_rn(v));
        }
      }
    }
  } else {
    for (int k = 0; k < kmax; ++k) {
      const int64_t par = __shfl_sync(0xFFFFFFFFu, my_par, k);
      const int64_t row = __shfl_sync(0xFFFFFFFFu, my_row, k);
      const int sh = __shfl_sync(0xFFFFFFFFu, my_shift, k);
      const float* pf = folds + par * 2 * nb;
      const float* sf = seg + row * 2 * nb;
      float* trow = tile + k * stride;
      for (int j = lane; j < nb; j += 32) {
        int js = j - sh;
        js += (js < 0) ? nb : 0;
        const float e = __fadd_rn(pf[j], sf[js]);
        const float v = __fadd_rn(pf[nb + j], sf[nb + js]);
        trow[j] = __fdiv_rn(e, __fsqrt_rn(v));
      }
    }
  }
  __syncwarp();
}

// Lane k scores row k of the tile; the level's score range is reduced over the
// warp before it reaches the run's two words.
__device__ __forceinline__ void score_tile_rows(float* tile, int stride, int nb,
                                                const LokiScoreSpec& sp, const ScoreK& SK,
                                                float* __restrict__ scores, int kmax,
                                                unsigned* __restrict__ minmax_keys) {
  const int lane = threadIdx.x & 31;
  unsigned lo = 0xFFFFFFFFu, hi = 0u;
  if (lane < kmax) {
    float* row = tile + lane * stride;
    float s;
    if (SK.list64) score_row64(row, sp, SK, &s);
    else score_row(row, nb, sp, SK, &s);
    scores[lane] = s;
    if (s == s) lo = hi = float_key(s);  // NaN scores do not enter min/max (like np.min)
  }
  lo = __reduce_min_sync(0xFFFFFFFFu, lo);
  hi = __reduce_max_sync(0xFFFFFFFFu, hi);
  if (lane == 0 && lo != 0xFFFFFFFFu) {
    atomicMin(minmax_keys, lo);
    atomicMax(minmax_keys + 1, hi);
  }
}

// Children c0 .. c0 + 31 (those below n_children) of one warp.
template <int KP = 0>
__device__ __forceinline__ void score_tile(
    const LokiPruneLevel& D, const double* __restrict__ leaves, const float* __restrict__ folds,
    int64_t n_parents, const LokiBranchInfo* __restrict__ info,
    const int64_t* __restrict__ offsets, int64_t n_children, const float* __restrict__ seg,
    const LokiScoreSpec& sp, const ScoreK& SK, float* __restrict__ scores,
    int32_t* __restrict__ cidx, double* __restrict__ cphase, unsigned* __restrict__ minmax_keys,
    float* tile, int64_t c0, int width = 32) {
  const int lane = threadIdx.x & 31;
  const int nb = D.nbins, P = tree_order<KP>(D);
  const int stride = score_stride(nb, sp.wmax);
  const int kmax = (int)std::min<int64_t>(width, n_children - c0);
  // lane k resolves child c0 + k
  int64_t my_par = warp_find_parents(offsets, n_parents, c0 + lane, kmax), my_row = 0;
  int my_shift = 0;
  if (lane < kmax) {
    const int64_t c = c0 + lane, par = my_par;
    const LokiBranchInfo B = info[par];
    const double* lf = leaves + par * (P + 2) * 2;
    double pv[LOKI_MAX_PARAMS + 1];
    child_params(B, P, c - offsets[par], pv);
    pv[P] = B.d0;  // d_0 (alpha_0 in the current domain for Chebyshev)
    const ChildRes r = resolve_child(D, P, pv, lf[(P + 1) * 2]);
    cidx[2 * c] = r.ia;
    cidx[2 * c + 1] = r.iff;
    cphase[c] = r.phase;
    my_row = (int64_t)r.ia * D.n_freq + r.iff;
    my_shift = round_shift(r.phase, nb);
  }
  gather_norm_rows(folds, seg, my_par, my_row, my_shift, kmax, nb, tile, stride);
  score_tile_rows(tile, stride, nb, sp, SK, scores + c0, kmax, minmax_keys);
}

__global__ void __launch_bounds__(kPruneWarps * 32)
prune_score_kernel(LokiPruneLevel D, const double* __restrict__ leaves,
                   const float* __restrict__ folds, int64_t n_parents,
                   const LokiBranchInfo* __restrict__ info, const int64_t* __restrict__ offsets,
                   int64_t n_children, const float* __restrict__ seg, LokiScoreSpec sp,
                   ScoreK SK, float* __restrict__ scores, int32_t* __restrict__ cidx,
                   double* __restrict__ cphase, unsigned* __restrict__ minmax_keys,
                   int64_t* cnt_dev, int64_t child_cap, LokiPruneLevelStats* st,
                   int32_t* err) {
  extern __shared__ float tiles[];
  const int warp = threadIdx.x >> 5;
  float* tile = tiles + (size_t)warp * 32 * score_stride(D.nbins, sp.wmax);
  if (!cnt_dev) {
    const int64_t c0 = ((int64_t)blockIdx.x * kPruneWarps + warp) * 32;
    if (c0 < n_children)
      score_tile(D, leaves, folds, n_parents, info, offsets, n_children, seg, sp, SK, scores,
                 cidx, cphase, minmax_keys, tile, c0);
    return;
  }
  // device counts: cnt_dev[0] parents; the children are offsets[parents],
  // none when they exceed the workspace (the run is then flagged). Block 0
  // records them for the later kernels of the level. Warps stride over the
  // 32-child tiles.
  n_parents = cnt_dev[0];
  const int64_t total = offsets[n_parents];
  n_children = total > child_cap ? 0 : total;
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    cnt_dev[1] = n_children;
    st->n_parents = n_parents;
    st->n_children = total;
    st->n_valid = total;
    if (total > child_cap) atomicOr(err, LOKI_DEVERR_CAPACITY);
  }
  for (int64_t t = (int64_t)blockIdx.x * kPruneWarps + warp; t * 32 < n_children;
       t += (int64_t)gridDim.x * kPruneWarps) {
    score_tile(D, leaves, folds, n_parents, info, offsets, n_children, seg, sp, SK, scores,
               cidx, cphase, minmax_keys, tile, t * 32);
    __syncwarp();  // the tile rows are rewritten by the next tile
  }
}

__global__ void minmax_init_kernel(unsigned* keys) {
  keys[0] = 0xFFFFFFFFu;
  keys[1] = 0u;
}

__global__ void minmax_finish_kernel(const unsigned* keys, float* out) {
  if (keys[0] == 0xFFFFFFFFu) {  // no finite score
    out[0] = 0.0f;
    out[1] = 0.0f;
  } else {
    out[0] = key_float(keys[0]);
    out[1] = key_float(keys[1]);
  }
}

// ---------------------------------------------------------------------------
// selection without overflow
// ---------------------------------------------------------------------------

__global__ void select_scatter_kernel(const float* __restrict__ scores, int64_t n, double thr,
                                      const int64_t* __restrict__ pos, int64_t* __restrict__ ids,
                                      const int64_t* __restrict__ n_dev) {
  if (n_dev) {  // device count: grid-stride walk
    n = *n_dev;
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n;
         i += (int64_t)gridDim.x * blockDim.x)
      if ((double)scores[i] >= thr) ids[pos[i]] = i;
    return;
  }
  const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (i < n && (double)scores[i] >= thr) ids[pos[i]] = i;
}

// ---------------------------------------------------------------------------
// selection with the overflow rule (single block, sequential over batches)
// ---------------------------------------------------------------------------

constexpr int kSelThreads = 1024;

// Block-wide exclusive scan of one flag per thread; returns the offset of this
// thread and writes the block total.
__device__ __forceinline__ int block_scan_flag(int f, int* total, int* wsum) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const unsigned b = __ballot_sync(0xFFFFFFFFu, f);
  const int before = __popc(b & lanemask_lt());
  if (lane == 0) wsum[warp] = __popc(b);
  __syncthreads();
  if (warp == 0) {
    int w = lane < (int)(blockDim.x >> 5) ? wsum[lane] : 0;
    int v = w;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int y = __shfl_up_sync(0xFFFFFFFFu, v, o);
      if (lane >= o) v += y;
    }
    wsum[lane] = v - w;  // exclusive
    if (lane == 31) wsum[32] = v;
  }
  __syncthreads();
  const int off = wsum[warp] + before;
  *total = wsum[32];
  __syncthreads();
  return off;
}

// Value of ascending rank r among keys[0..n) (radix select, 4 x 8 bits).
__device__ unsigned block_select(const unsigned* keys, int64_t n, int64_t r, unsigned* hist) {
  unsigned prefix = 0, mask = 0;
  for (int shift = 24; shift >= 0; shift -= 8) {
    for (int b = threadIdx.x; b < 256; b += blockDim.x) hist[b] = 0;
    __syncthreads();
    for (int64_t i = threadIdx.x; i < n; i += blockDim.x) {
      const unsigned k = keys[i];
      if ((k & mask) == prefix) atomicAdd(&hist[(k >> shift) & 0xFF], 1u);
    }
    __syncthreads();
    __shared__ unsigned sel_digit;
    __shared__ long long sel_r;
    if (threadIdx.x == 0) {
      long long acc = 0;
      int d = 0;
      for (; d < 256; ++d) {
        if (acc + hist[d] > r) break;
        acc += hist[d];
      }
      sel_digit = (unsigned)(d < 256 ? d : 255);
      sel_r = r - acc;
    }
    __syncthreads();
    prefix |= sel_digit << shift;
    mask |= 0xFFu << shift;
    r = sel_r;
    __syncthreads();
  }
  return prefix;
}

// The overflow rule over the whole selection, by one block (any multiple of
// 32 threads up to 1024): batch by batch of parents, the passing children are
// appended while they fit, otherwise prune_on_overload raises the threshold.
// Writes ids[0 .. *n_out) and the final threshold.
__device__ void select_overflow_block(const float* __restrict__ scores,
                                      const int64_t* __restrict__ offsets, int64_t n_parents,
                                      int64_t batch, double thr, int64_t cap,
                                      int64_t* __restrict__ ids, int64_t* n_out,
                                      double* __restrict__ thr_out,
                                      int64_t* __restrict__ tmp_ids,
                                      unsigned* __restrict__ keys) {
  __shared__ int wsum[33];
  __shared__ unsigned hist[256];
  __shared__ long long vs_sh;
  __shared__ double cur_sh;
  const int nthr = blockDim.x;  // the loops stride by the block
  if (threadIdx.x == 0) {
    vs_sh = 0;
    cur_sh = thr;
  }
  __syncthreads();
  for (int64_t p0 = 0; p0 < n_parents; p0 += batch) {
    const int64_t p1 = std::min(p0 + batch, n_parents);
    const int64_t c_lo = offsets[p0], c_hi = offsets[p1];
    if (c_hi == c_lo) continue;
    const double eff_in = fmax(thr, cur_sh);
    // pass 1: count passing children of the batch
    int64_t m = 0;
    for (int64_t base = c_lo; base < c_hi; base += nthr) {
      const int64_t c = base + threadIdx.x;
      const int f = (c < c_hi && (double)scores[c] >= eff_in) ? 1 : 0;
      int tot;
      block_scan_flag(f, &tot, wsum);
      m += tot;
    }
    int64_t vs = vs_sh;
    if (m <= cap - vs) {  // fast path: append in order
      int64_t w = vs;
      for (int64_t base = c_lo; base < c_hi; base += nthr) {
        const int64_t c = base + threadIdx.x;
        const int f = (c < c_hi && (double)scores[c] >= eff_in) ? 1 : 0;
        int tot;
        const int off = block_scan_flag(f, &tot, wsum);
        if (f) ids[w + off] = c;
        w += tot;
      }
      if (threadIdx.x == 0) vs_sh = vs + m;
      __syncthreads();
      continue;
    }
    // prune_on_overload: keys of the current tree and of the passing batch
    int64_t w = vs;
    for (int64_t i = threadIdx.x; i < vs; i += nthr) keys[i] = float_key(scores[ids[i]]);
    for (int64_t base = c_lo; base < c_hi; base += nthr) {
      const int64_t c = base + threadIdx.x;
      const int f = (c < c_hi && (double)scores[c] >= eff_in) ? 1 : 0;
      int tot;
      const int off = block_scan_flag(f, &tot, wsum);
      if (f) {
        keys[w + off] = float_key(scores[c]);
        tmp_ids[w - vs + off] = c;
      }
      w += tot;
    }
    __syncthreads();
    const int64_t total = vs + m;
    const unsigned kth = block_select(keys, total, total - cap, hist);
    const unsigned mid = block_select(keys, total, total - total / 2 - 1, hist);
    double eff = cur_sh;
    const double tk = nextafter((double)key_float(kth), INFINITY);
    const double tm = nextafter((double)key_float(mid), INFINITY);
    eff = fmax(eff, fmax(tk, tm));
    // keep tree entries >= eff (stable)
    int64_t kept = 0;
    for (int64_t base = 0; base < vs; base += nthr) {
      const int64_t i = base + threadIdx.x;
      int64_t id = 0;
      int f = 0;
      if (i < vs) {
        id = ids[i];
        f = (double)scores[id] >= eff ? 1 : 0;
      }
      int tot;
      const int off = block_scan_flag(f, &tot, wsum);
      if (f) keys[kept + off] = (unsigned)(id & 0xFFFFFFFFu), tmp_ids[m + kept + off] = id;
      kept += tot;
    }
    __syncthreads();
    for (int64_t i = threadIdx.x; i < kept; i += nthr) ids[i] = tmp_ids[m + i];
    __syncthreads();
    // pending batch entries >= eff, in order, up to the free space
    const int64_t space = cap - kept;
    int64_t added = 0;
    for (int64_t base = 0; base < m; base += nthr) {
      const int64_t i = base + threadIdx.x;
      int64_t id = 0;
      int f = 0;
      if (i < m) {
        id = tmp_ids[i];
        f = (double)scores[id] >= eff ? 1 : 0;
      }
      int tot;
      const int off = block_scan_flag(f, &tot, wsum);
      if (f && added + off < space) ids[kept + added + off] = id;
      added += tot;
    }
    if (threadIdx.x == 0) {
      vs_sh = kept + std::min(added, space);
      cur_sh = eff;
    }
    __syncthreads();
  }
  if (threadIdx.x == 0) {
    *n_out = vs_sh;
    *thr_out = cur_sh;
  }
  __syncthreads();
}

// With cnt_dev (device counts: [0] parents) the plain selection's survivor
// count is pos[*n_in] (n_in: its inputs, the children): it is stored at
// *n_out, and the kernel does nothing more unless it exceeds cap (then
// *ovf_flag is set and the overflow rule rewrites the selection and *n_out).
// n_out points into the same counters, so neither pointer is restrict.
__global__ void __launch_bounds__(kSelThreads)
select_overflow_kernel(const float* __restrict__ scores, const int64_t* __restrict__ offsets,
                       int64_t n_parents, int64_t batch, double thr, int64_t cap,
                       int64_t* __restrict__ ids, int64_t* n_out,
                       double* __restrict__ thr_out, int64_t* __restrict__ tmp_ids,
                       unsigned* __restrict__ keys, const int64_t* cnt_dev,
                       int32_t* __restrict__ ovf_flag, const int64_t* __restrict__ pos,
                       const int64_t* n_in) {
  if (cnt_dev) {
    const int64_t n_sel = pos[*n_in];  // the selection's total over its n_in inputs
    n_parents = cnt_dev[0];
    __syncthreads();  // every thread has read the counters
    if (threadIdx.x == 0) *n_out = n_sel;
    if (n_sel <= cap) return;  // uniform over the block
    if (threadIdx.x == 0) *ovf_flag = 1;
  }
  select_overflow_block(scores, offsets, n_parents, batch, thr, cap, ids, n_out, thr_out, tmp_ids,
                        keys);
}

// ---------------------------------------------------------------------------
// emit: thread per survivor for the leaf, warp per 32 survivors for folds
// ---------------------------------------------------------------------------

// What the level-synchronous batch adds to an emission: the run's backtrack
// history row of every survivor, and the level's best leaf.
struct EmitExtra {
  int32_t* bt_hist = nullptr;  // row of the level's first survivor
  int64_t best = -1;           // survivor with the best score
  double* best_leaf = nullptr;
  float* best_score = nullptr;
};

__device__ __forceinline__ void emit_extra(const EmitExtra& X, int64_t s, const double* lo,
                                           float sc, const int32_t* bt, int P) {
  if (X.bt_hist) {
    int32_t* h = X.bt_hist + s * (P + 2);
    for (int j = 0; j < P + 2; ++j) h[j] = bt[j];
  }
  if (s == X.best) {
    for (int j = 0; j < (P + 2) * 2; ++j) X.best_leaf[j] = lo[j];
    *X.best_score = sc;
  }
}

// Rows of 32 survivors (as gather_norm_rows): shift-added, written to fout.
__device__ __forceinline__ void gather_add_rows(const float* __restrict__ folds,
                                                const float* __restrict__ seg, int64_t my_par,
                                                int64_t my_row, int my_shift, int kmax, int nb,
                                                float* __restrict__ fout) {
  const int lane = threadIdx.x & 31;
  if (nb == 64) {
    // four survivors' rows in flight per lane (bins lane and lane + 32)
    constexpr int kU = 4;
    for (int k0 = 0; k0 < kmax; k0 += kU) {
      float pe[kU][2], pw[kU][2], se[kU][2], sw[kU][2];
#pragma unroll
      for (int u = 0; u < kU; ++u) {
        const int k = k0 + u;
        const int src = k < kmax ? k : 0;
        // (rows of 512 bytes: their numbers fit 32 bits)
        const uint32_t par = __shfl_sync(0xFFFFFFFFu, (uint32_t)my_par, src);
        const uint32_t row = __shfl_sync(0xFFFFFFFFu, (uint32_t)my_row, src);
        const int sh = __shfl_sync(0xFFFFFFFFu, my_shift, src);
        if (k < kmax) {
          const float* pf = folds + (size_t)par * 128;
          const float* sf = seg + (size_t)row * 128;
#pragma unroll
          for (int c = 0; c < 2; ++c) {
            const int j = lane + 32 * c;
            const int js = (j - sh) & 63;
            pe[u][c] = __ldg(pf + j);
            pw[u][c] = __ldg(pf + 64 + j);
            se[u][c] = __ldg(sf + js);
            sw[u][c] = __ldg(sf + 64 + js);
          }
        }
      }
#pragma unroll
      for (int u = 0; u < kU; ++u) {
        const int k = k0 + u;
        if (k >= kmax) break;
        float* o = fout + k * 128;
#pragma unroll
        for (int c = 0; c < 2; ++c) {
          o[lane + 32 * c] = __fadd_rn(pe[u][c], se[u][c]);
          o[64 + lane + 32 * c] = __fadd_rn(pw[u][c], sw[u][c]);
        }
      }
    }
    return;
  }
  for (int k = 0; k < kmax; ++k) {
    const int64_t par = __shfl_sync(0xFFFFFFFFu, my_par, k);
    const int64_t row = __shfl_sync(0xFFFFFFFFu, my_row, k);
    const int sh = __shfl_sync(0xFFFFFFFFu, my_shift, k);
    const float* pf = folds + par * 2 * nb;
    const float* sf = seg + row * 2 * nb;
    float* o = fout + k * 2 * nb;
    for (int j = lane; j < nb; j += 32) {
      int js = j - sh;
      js += (js < 0) ? nb : 0;
      o[j] = __fadd_rn(pf[j], sf[js]);
      o[nb + j] = __fadd_rn(pf[nb + j], sf[nb + js]);
    }
  }
}

// Survivors s0 .. s0 + 31 (those below n_surv) of one warp.
template <int KP = 0>
__device__ __forceinline__ void emit_tile(
    const LokiPruneLevel& D, const double* __restrict__ leaves, const float* __restrict__ folds,
    const LokiBranchInfo* __restrict__ info, const int64_t* __restrict__ offsets,
    int64_t n_parents, const float* __restrict__ seg, const int64_t* __restrict__ surv,
    int64_t n_surv, const float* __restrict__ cscores, const int32_t* __restrict__ cidx,
    const double* __restrict__ cphase, double* __restrict__ lout, float* __restrict__ fout,
    float* __restrict__ sout, float* __restrict__ seout, int32_t* __restrict__ bout, int64_t s0,
    const EmitExtra& X = EmitExtra(), int width = 32) {
  const int lane = threadIdx.x & 31;
  const int nb = D.nbins, P = tree_order<KP>(D), m = P + 1;
  const int kmax = (int)std::min<int64_t>(width, n_surv - s0);
  const int64_t my_c = surv[s0 + min(lane, kmax - 1)];
  int64_t my_par = warp_find_parents(offsets, n_parents, my_c, kmax), my_row = 0;
  int my_shift = 0;
  if (lane < kmax) {
    const int64_t s = s0 + lane, c = my_c, par = my_par;
    const LokiBranchInfo B = info[par];
    const double* lf = leaves + par * (P + 2) * 2;
    double pv[LOKI_MAX_PARAMS + 1], ev[LOKI_MAX_PARAMS + 1];
    child_params(B, P, c - offsets[par], pv);
    pv[P] = B.d0;
    for (int j = 0; j < P; ++j) ev[j] = B.dact[j];
    ev[P] = 0.0;
    double* lo = lout + s * (P + 2) * 2;
    if (D.moving) {
      for (int i = 0; i < m; ++i) lo[2 * i] = tdot(pv, D.tm_n, i, m);
      if (D.tiling == 0) {
        for (int i = 0; i < m; ++i) lo[2 * i + 1] = __dmul_rn(ev[i], fabs(D.tm_n[i][i]));
      } else if (D.tiling == 2) {
        for (int i = 0; i < m; ++i) lo[2 * i + 1] = tdot(ev, D.tm_e, i, m);
      } else {
        double e2[LOKI_MAX_PARAMS + 1];
        for (int j = 0; j < m; ++j) e2[j] = __dmul_rn(ev[j], ev[j]);
        for (int i = 0; i < m; ++i) lo[2 * i + 1] = __dsqrt_rn(tdot(e2, D.tm_e, i, m));
      }
    } else {
      for (int i = 0; i < m; ++i) {
        lo[2 * i] = pv[i];
        lo[2 * i + 1] = ev[i];
      }
    }
    lo[2 * m] = lf[2 * m];          // f0
    lo[2 * m + 1] = lf[2 * m + 1];  // basis flag
    const float sc = cscores[c];
    sout[s] = sc;
    seout[s] = sc;
    int32_t* bt = bout + s * (P + 2);
    const int ia = cidx[2 * c], iff = cidx[2 * c + 1];
    bt[0] = (int32_t)par;
    for (int j = 1; j < P + 1; ++j) bt[j] = 0;
    bt[D.nparams_ffa - 1] = ia;  // column 1 + (nparams_ffa - 2)
    bt[D.nparams_ffa] = iff;     // column 1 + (nparams_ffa - 1)
    bt[P + 1] = (int32_t)cphase[c];
    emit_extra(X, s, lo, sc, bt, P);
    my_row = (int64_t)ia * D.n_freq + iff;
    my_shift = round_shift(cphase[c], nb);
  }
  gather_add_rows(folds, seg, my_par, my_row, my_shift, kmax, nb, fout + s0 * 2 * nb);
}

__global__ void __launch_bounds__(kPruneWarps * 32)
prune_emit_kernel(LokiPruneLevel D, const double* __restrict__ leaves,
                  const float* __restrict__ folds, const LokiBranchInfo* __restrict__ info,
                  const int64_t* __restrict__ offsets, int64_t n_parents,
                  const float* __restrict__ seg, const int64_t* __restrict__ surv,
                  int64_t n_surv, const float* __restrict__ cscores,
                  const int32_t* __restrict__ cidx, const double* __restrict__ cphase,
                  double* __restrict__ lout, float* __restrict__ fout,
                  float* __restrict__ sout, float* __restrict__ seout,
                  int32_t* __restrict__ bout, const int64_t* __restrict__ cnt_dev) {
  const int warp = threadIdx.x >> 5;
  if (!cnt_dev) {
    const int64_t s0 = ((int64_t)blockIdx.x * kPruneWarps + warp) * 32;
    if (s0 < n_surv)
      emit_tile(D, leaves, folds, info, offsets, n_parents, seg, surv, n_surv, cscores, cidx,
                cphase, lout, fout, sout, seout, bout, s0);
    return;
  }
  // device counts: cnt_dev[0] parents, cnt_dev[2] survivors
  n_parents = cnt_dev[0];
  n_surv = cnt_dev[2];
  for (int64_t t = (int64_t)blockIdx.x * kPruneWarps + warp; t * 32 < n_surv;
       t += (int64_t)gridDim.x * kPruneWarps)
    emit_tile(D, leaves, folds, info, offsets, n_parents, seg, surv, n_surv, cscores, cidx,
              cphase, lout, fout, sout, seout, bout, t * 32);
}

// ---------------------------------------------------------------------------
// circular-orbit propagation, shared by the circular tree and its ascend
// ---------------------------------------------------------------------------

// get_circ_mask (core/circular.py:13-79): 1 snap-circular, 2 crackle-circular
// (the snap/accel hole), 0 Taylor.
__device__ __forceinline__ int circ_class(const double* v, const double* e, double sig) {
  const double crackle = v[0], snap = v[1], jerk = v[2], accel = v[3];
  const bool sig_snap = fabs(snap) > __dmul_rn(sig, e[1]);
  const bool sig_accel = fabs(accel) > __dmul_rn(sig, e[3]);
  const bool sig_jerk = fabs(jerk) > __dmul_rn(sig, e[2]);
  const bool snap_circ = sig_snap && sig_accel && __dmul_rn(-snap, accel) > 0.0;
  if (snap_circ) return 1;
  if (sig_jerk && __dmul_rn(-crackle, jerk) > 0.0) return 2;
  return 0;
}

// shift_taylor_circular_params (utils/transforms.py:246-299): closed-form
// circular-orbit propagation of [d5 .. d0] by dt (values only). cos and sin
// are CUDA's double-precision functions.
__device__ __forceinline__ void circ_shift(const double* p, double dt, bool hole, double* out) {
  const double d5 = p[0], d4 = p[1], d3 = p[2], d2 = p[3], d1 = p[4], d0 = p[5];
  const double wsq = hole ? __ddiv_rn(-d5, d3) : __ddiv_rn(-d4, d2);
  const double w = __dsqrt_rn(wsq);
  const double wdt = __dmul_rn(w, dt);
  const double c = cos(wdt), s = sin(wdt);
  const double d2j = __dadd_rn(__dmul_rn(d2, c), __dmul_rn(__ddiv_rn(d3, w), s));
  const double d3j = __dsub_rn(__dmul_rn(d3, c), __dmul_rn(__dmul_rn(d2, w), s));
  const double d1ci = __ddiv_rn(-d3, wsq);
  const double d1cj = __ddiv_rn(-d3j, wsq);
  const double e1 = __dsub_rn(d1, d1ci);
  const double d0cj = __ddiv_rn(-d2j, wsq);
  const double d0ci = __ddiv_rn(-d2, wsq);
  out[0] = __dmul_rn(-wsq, d3j);
  out[1] = __dmul_rn(-wsq, d2j);
  out[2] = d3j;
  out[3] = d2j;
  out[4] = __dadd_rn(d1cj, e1);
  out[5] = __dadd_rn(__dadd_rn(d0cj, __dsub_rn(d0, d0ci)), __dmul_rn(e1, dt));
}

// ---------------------------------------------------------------------------
// ascend: warp per 32 survivors, segments accumulated in order
// ---------------------------------------------------------------------------

// Survivors s0 .. s0 + 31 (those below n) of one warp; acc and tile are the
// warp's accumulators (32 x 2 nb) and score tile.
__device__ __forceinline__ void ascend_tile(
    const LokiPruneLevel& D, const double* __restrict__ leaves, float* __restrict__ folds,
    float* __restrict__ scores, float* __restrict__ scores_ep, int64_t n, int nseg,
    const double* __restrict__ tm_seg, const double* __restrict__ dt_seg,
    const int32_t* __restrict__ seg_idx, const float* __restrict__ ffa, int64_t seg_stride,
    const LokiScoreSpec& sp, const ScoreK& SK, float* acc, float* tile, int64_t s0) {
  const int lane = threadIdx.x & 31;
  const int nb = D.nbins, P = D.poly_order, m = P + 1;
  const int stride = score_stride(nb, sp.wmax);
  const int kmax = (int)std::min<int64_t>(32, n - s0);
  for (int k = 0; k < kmax; ++k)
    for (int j = lane; j < 2 * nb; j += 32) acc[k * 2 * nb + j] = 0.0f;
  double pv[LOKI_MAX_PARAMS + 1];
  double f0 = 1.0;
  int cls = 0;  // circular tree: class of the survivor (core/circular.py:597-666)
  if (lane < kmax) {
    const double* lf = leaves + (s0 + lane) * (P + 2) * 2;
    double ev[LOKI_MAX_PARAMS + 1];
    for (int i = 0; i < m; ++i) {
      pv[i] = lf[2 * i];
      ev[i] = lf[2 * i + 1];
    }
    f0 = lf[2 * m];
    if (D.basis == 2) cls = circ_class(pv, ev, D.circ_sig_prop);
  }
  __syncwarp();
  for (int sg = 0; sg < nseg; ++sg) {
    const double(*T)[LOKI_MAX_PARAMS + 1] =
        reinterpret_cast<const double(*)[LOKI_MAX_PARAMS + 1]>(tm_seg + sg * 36);
    int64_t my_row = 0;
    int my_shift = 0;
    if (lane < kmax) {
      double accel, vel, dd;
      if (D.basis == 1) {  // core/chebyshev.py:280-320: shift to t0_seg, then Taylor
        double a[LOKI_MAX_PARAMS + 1];
        for (int i = 0; i < m; ++i) a[i] = tdot(pv, T, i, m);
        cheby_low3(D, a, m, &accel, &vel, &dd);
      } else if (cls != 0) {  // circular survivors: closed-form propagation
        double a[6];
        circ_shift(pv, dt_seg[sg], cls == 2, a);
        accel = a[3];
        vel = a[4];
        dd = a[5];
      } else {
        accel = tdot(pv, T, P - 2, m);
        vel = tdot(pv, T, P - 1, m);
        dd = tdot(pv, T, P, m);
      }
      const double freq = __dmul_rn(f0, __dsub_rn(1.0, div_c(vel)));
      const double delay = div_c(dd);
      const double ph = phase_idx(dt_seg[sg], f0, nb, delay);
      const int64_t ia = axis_index(accel, D.accel_min, D.accel_inv, D.n_accel);
      const int64_t iff = axis_index(freq, D.freq_min, D.freq_inv, D.n_freq);
      my_row = ia * D.n_freq + iff;
      my_shift = round_shift(ph, nb);
    }
    const float* fseg = ffa + (int64_t)seg_idx[sg] * seg_stride;
    if (nb == 64) {
      // eight survivors' segment rows in flight per lane (bins lane, lane + 32)
      constexpr int kU = 8;
      for (int k0 = 0; k0 < kmax; k0 += kU) {
        float se[kU][2], sw[kU][2];
#pragma unroll
        for (int u = 0; u < kU; ++u) {
          const int k = k0 + u;
          const int src = k < kmax ? k : 0;
          const int64_t row = __shfl_sync(0xFFFFFFFFu, my_row, src);
          const int sh = __shfl_sync(0xFFFFFFFFu, my_shift, src);
          if (k < kmax) {
            const float* sf = fseg + row * 128;
#pragma unroll
            for (int c = 0; c < 2; ++c) {
              const int js = (lane + 32 * c - sh) & 63;
              se[u][c] = __ldg(sf + js);
              sw[u][c] = __ldg(sf + 64 + js);
            }
          }
        }
#pragma unroll
        for (int u = 0; u < kU; ++u) {
          const int k = k0 + u;
          if (k >= kmax) break;
          float* a = acc + k * 128;
#pragma unroll
          for (int c = 0; c < 2; ++c) {
            const int j = lane + 32 * c;
            a[j] = __fadd_rn(a[j], se[u][c]);
            a[64 + j] = __fadd_rn(a[64 + j], sw[u][c]);
          }
        }
      }
      continue;
    }
    for (int k = 0; k < kmax; ++k) {
      const int64_t row = __shfl_sync(0xFFFFFFFFu, my_row, k);
      const int sh = __shfl_sync(0xFFFFFFFFu, my_shift, k);
      const float* sf = fseg + row * 2 * nb;
      float* a = acc + k * 2 * nb;
      for (int j = lane; j < nb; j += 32) {
        int js = j - sh;
        js += (js < 0) ? nb : 0;
        a[j] = __fadd_rn(a[j], sf[js]);
        a[nb + j] = __fadd_rn(a[nb + j], sf[nb + js]);
      }
    }
  }
  __syncwarp();
  for (int k = 0; k < kmax; ++k) {
    const float* a = acc + k * 2 * nb;
    float* o = folds + (s0 + k) * 2 * nb;
    float* trow = tile + k * stride;
    for (int j = lane; j < nb; j += 32) {
      o[j] = a[j];
      o[nb + j] = a[nb + j];
      trow[j] = __fdiv_rn(a[j], __fsqrt_rn(a[nb + j]));
    }
  }
  __syncwarp();
  if (lane < kmax) {
    scores_ep[s0 + lane] = scores[s0 + lane];
    float s;
    float* row = tile + lane * stride;
    if (SK.list64) score_row64(row, sp, SK, &s);
    else score_row(row, nb, sp, SK, &s);
    scores[s0 + lane] = s;
  }
}

__global__ void __launch_bounds__(kPruneWarps * 32)
prune_ascend_kernel(LokiPruneLevel D, const double* __restrict__ leaves,
                    float* __restrict__ folds, float* __restrict__ scores,
                    float* __restrict__ scores_ep, int64_t n, int nseg,
                    const double* __restrict__ tm_seg, const double* __restrict__ dt_seg,
                    const int32_t* __restrict__ seg_idx, const float* __restrict__ ffa,
                    int64_t seg_stride, LokiScoreSpec sp, ScoreK SK,
                    const int64_t* __restrict__ n_dev) {
  extern __shared__ float tiles[];
  const int warp = threadIdx.x >> 5;
  // per warp: the 32 accumulators (2 * nb each) followed by the score tile
  const int stride = score_stride(D.nbins, sp.wmax);
  float* acc = tiles + (size_t)warp * 32 * (2 * D.nbins + stride);
  float* tile = acc + 32 * 2 * D.nbins;
  if (!n_dev) {
    const int64_t s0 = ((int64_t)blockIdx.x * kPruneWarps + warp) * 32;
    if (s0 < n)
      ascend_tile(D, leaves, folds, scores, scores_ep, n, nseg, tm_seg, dt_seg, seg_idx, ffa,
                  seg_stride, sp, SK, acc, tile, s0);
    return;
  }
  n = *n_dev;  // survivors held on the device: warps stride over their tiles
  for (int64_t t = (int64_t)blockIdx.x * kPruneWarps + warp; t * 32 < n;
       t += (int64_t)gridDim.x * kPruneWarps) {
    ascend_tile(D, leaves, folds, scores, scores_ep, n, nseg, tm_seg, dt_seg, seg_idx, ffa,
                seg_stride, sp, SK, acc, tile, t * 32);
    __syncwarp();  // the accumulators are reused by the next tile
  }
}

// ---------------------------------------------------------------------------
// circular-orbit Taylor tree (core/circular.py, dynamic/dyn_circular_taylor.py)
//
// Leaves are [d5 (crackle), d4 (snap), d3, d2, d1, d0, (f0, flag)]. Children
// of one parent batch are ordered as the reference builds them: first every
// child that keeps the parent's crackle (cartesian order over the batch),
// then the children whose crackle is expanded, each expansion in crackle
// order. Physical validation drops children before scoring, so the scored
// list is the compacted list of valid children.
// ---------------------------------------------------------------------------

// One child of the circular tree: parent, index in the parent's cartesian
// product over d4..d1, and the crackle sub-index (-1: parent crackle kept).
struct CircChild {
  int32_t parent, cart, crackle, pad;
};

// circ_validate_batch (core/circular.py:82-124) for one child.
__device__ __forceinline__ bool circ_valid(const LokiPruneLevel& D, const double* v,
                                           const double* e) {
  const double snap = v[1], accel = v[3], sig = D.circ_sig_valid;
  const bool sig_snap = fabs(snap) > __dmul_rn(sig, e[1]);
  const bool sig_accel = fabs(accel) > __dmul_rn(sig, e[3]);
  if (!(sig_snap && sig_accel)) return true;
  if (!(__dmul_rn(-snap, accel) > 0.0)) return false;
  const double wsq = __ddiv_rn(-snap, accel);
  const double limit = __dmul_rn(D.circ_x_mass, pow(wsq, 2.0 / 3.0));
  return wsq <= D.circ_omega_max_sq && fabs(accel) <= limit;
}

// Parameters and errors of one circular child (core/circular.py:204-394).
__device__ __forceinline__ void circ_child(const LokiBranchInfo& B, const double* lf,
                                           const CircChild& ch, double* pv, double* ev) {
  const int P = 5;
  child_params(B, P, ch.cart, pv);
  pv[P] = B.d0;
  for (int j = 0; j < P; ++j) ev[j] = B.dact[j];
  ev[P] = 0.0;
  if (ch.crackle >= 0) {  // branch_param_padded on the parent crackle cell
    const double dact = B.dact[0];
    const double first = __dadd_rn(__dsub_rn(lf[0], __dmul_rn(lf[1], 0.5)),
                                   __dmul_rn(dact, 0.5));
    pv[0] = __dadd_rn(first, __dmul_rn((double)ch.crackle, dact));
  }
}

// Branch every parent (circ_taylor_branch_batch): per-parameter branching of
// d4..d1 as in the Taylor tree, crackle deferred; counts the children that
// keep the parent crackle and those produced by crackle expansion.
__device__ __forceinline__ void circ_branch_one(const LokiPruneLevel& D,
                                                const double* __restrict__ leaves, int64_t i,
                                                LokiBranchInfo* __restrict__ info,
                                                int64_t* __restrict__ n_keep,
                                                int64_t* __restrict__ n_exp,
                                                int32_t* __restrict__ err, const BranchF& F);

// n_dev, when not null, holds the parent count on the device (grid-stride).
__global__ void circ_branch_kernel(LokiPruneLevel D, const double* __restrict__ leaves,
                                   int64_t n, LokiBranchInfo* __restrict__ info,
                                   int64_t* __restrict__ n_keep, int64_t* __restrict__ n_exp,
                                   int32_t* __restrict__ err, const int64_t* __restrict__ n_dev) {
  if (n_dev) {
    n = *n_dev;
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n;
         i += (int64_t)gridDim.x * blockDim.x)
      circ_branch_one(D, leaves, i, info, n_keep, n_exp, err, branch_floats(D));
    return;
  }
  const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (i < n) circ_branch_one(D, leaves, i, info, n_keep, n_exp, err, branch_floats(D));
}

__device__ __forceinline__ void circ_branch_one(const LokiPruneLevel& D,
                                                const double* __restrict__ leaves, int64_t i,
                                                LokiBranchInfo* __restrict__ info,
                                                int64_t* __restrict__ n_keep,
                                                int64_t* __restrict__ n_exp,
                                                int32_t* __restrict__ err, const BranchF& F) {
  const int P = 5;
  const double* lf = leaves + i * (P + 2) * 2;
  const double f0 = lf[(P + 1) * 2];
  const float f0f = (float)f0, rf0 = __frcp_rn(f0f);
  LokiBranchInfo B;
  B.d0 = lf[2 * P];
  bool needs0 = false;
  int64_t num_c = 1;
  int64_t total = 1;
  for (int j = 0; j < P; ++j) {
    const double pcur = lf[2 * j], dcur = lf[2 * j + 1];
    int quick_num = 1;
    const int quick = branch_quick(F, j, f0f, rf0, dcur, D.branch_max, &quick_num);
    bool needs = quick > 0;
    int64_t num = quick_num;
    if (quick < 0) {
      const double dnew = __ddiv_rn(D.dfc[j], f0);
      const double fb = __dmul_rn(D.fac[j], __ddiv_rn(f0, LOKI_C_VAL));
      const double shift = __dmul_rn(fabs(__dsub_rn(dcur, dnew)), fb);
      needs = shift >= D.eta_m;
      num = 0;  // no step to split: an error, values kept
      if (!(dcur > 0.0) || !(dnew > 0.0)) {
        atomicOr(err, LOKI_DEVERR_BRANCH);
      } else {
        const double ratio = __ddiv_rn(dcur, dnew);
        num = (int64_t)ceil(__dsub_rn(ratio, LOKI_FLOAT_EPSILON));
        if (num < 1) num = 1;
        if (num > D.branch_max) {
          atomicOr(err, LOKI_DEVERR_BRANCH);
          num = D.branch_max;
        }
      }
    }
    double dact = dcur, first = pcur;
    if (needs && num > 0) {
      dact = branch_step(dcur, num);
      first = __dadd_rn(__dsub_rn(pcur, __dmul_rn(dcur, 0.5)), __dmul_rn(dact, 0.5));
    }
    if (num < 1) num = 1;
    if (j == 0) {  // crackle keeps the parent value; its step is the would-be child step
      needs0 = needs;
      num_c = num;
      first = pcur;
      num = 1;
    }
    if (!needs) num = 1;
    B.first[j] = first;
    B.dact[j] = dact;
    B.count[j] = (int32_t)num;
    total *= num;
  }
  B.reserved = needs0 ? (int32_t)num_c : 0;
  // first cartesian product: which children fall in the hole and expand crackle
  const double sig = D.circ_sig_prop;
  int64_t keep = 0, exp = 0;
  double pv[LOKI_MAX_PARAMS + 1];
  if (!needs0) keep = total;  // none expands
  for (int64_t k = 0; needs0 && k < total; ++k) {
    child_params(B, P, k, pv);
    const double snap = pv[1], jerk = pv[2], accel = pv[3];
    const bool snap_circ = fabs(snap) > __dmul_rn(sig, B.dact[1]) &&
                           fabs(accel) > __dmul_rn(sig, B.dact[3]) &&
                           __dmul_rn(-snap, accel) > 0.0;
    const bool expand = !snap_circ && fabs(jerk) > __dmul_rn(sig, B.dact[2]);
    if (expand) exp += num_c;
    else ++keep;
  }
  info[i] = B;
  n_keep[i] = keep;
  n_exp[i] = exp;
}

// Children of every parent at their batch-ordered positions, plus a validity
// flag (1.0 / 0.0) per child for the compaction.
__device__ __forceinline__ void circ_map_one(const LokiPruneLevel& D,
                                             const double* __restrict__ leaves, int64_t n,
                                             int64_t batch, const LokiBranchInfo* __restrict__ info,
                                             const int64_t* __restrict__ keep_off,
                                             const int64_t* __restrict__ exp_off,
                                             CircChild* __restrict__ map,
                                             float* __restrict__ validf, int64_t i);

// With cnt (device counts) the parents are cnt[0] and the children
// keep_off[n] + exp_off[n]; block 0 records the children in cnt[1] and the
// level's statistics, and above child_cap the level gets none (flagged).
__global__ void circ_map_kernel(LokiPruneLevel D, const double* __restrict__ leaves, int64_t n,
                                int64_t batch, const LokiBranchInfo* __restrict__ info,
                                const int64_t* __restrict__ keep_off,
                                const int64_t* __restrict__ exp_off,
                                CircChild* __restrict__ map, float* __restrict__ validf,
                                int64_t* cnt, int64_t child_cap, LokiPruneLevelStats* st,
                                int32_t* err) {
  if (cnt) {
    n = cnt[0];
    const int64_t total = keep_off[n] + exp_off[n];
    const bool fits = total <= child_cap;
    if (blockIdx.x == 0 && threadIdx.x == 0) {
      cnt[1] = fits ? total : 0;
      st->n_parents = n;
      st->n_children = total;
      if (!fits) atomicOr(err, LOKI_DEVERR_CAPACITY);
    }
    if (!fits) return;
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n;
         i += (int64_t)gridDim.x * blockDim.x)
      circ_map_one(D, leaves, n, batch, info, keep_off, exp_off, map, validf, i);
    return;
  }
  const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (i < n) circ_map_one(D, leaves, n, batch, info, keep_off, exp_off, map, validf, i);
}

__device__ __forceinline__ void circ_map_one(const LokiPruneLevel& D,
                                             const double* __restrict__ leaves, int64_t n,
                                             int64_t batch, const LokiBranchInfo* __restrict__ info,
                                             const int64_t* __restrict__ keep_off,
                                             const int64_t* __restrict__ exp_off,
                                             CircChild* __restrict__ map,
                                             float* __restrict__ validf, int64_t i) {
  const int P = 5;
  const int64_t b0 = (i / batch) * batch, b1 = std::min(b0 + batch, n);
  int64_t pk = keep_off[i] + exp_off[b0];
  int64_t pe = keep_off[b1] + exp_off[i];
  const LokiBranchInfo B = info[i];
  const double* lf = leaves + i * (P + 2) * 2;
  const int64_t num_c = B.reserved;
  int64_t total = 1;
  for (int j = 0; j < P; ++j) total *= B.count[j];
  const double sig = D.circ_sig_prop;
  double pv[LOKI_MAX_PARAMS + 1], ev[LOKI_MAX_PARAMS + 1];
  for (int64_t k = 0; k < total; ++k) {
    CircChild ch = {(int32_t)i, (int32_t)k, -1, 0};
    circ_child(B, lf, ch, pv, ev);
    const double snap = pv[1], jerk = pv[2], accel = pv[3];
    const bool snap_circ = fabs(snap) > __dmul_rn(sig, ev[1]) &&
                           fabs(accel) > __dmul_rn(sig, ev[3]) &&
                           __dmul_rn(-snap, accel) > 0.0;
    const bool expand = !snap_circ && fabs(jerk) > __dmul_rn(sig, ev[2]) && num_c > 0;
    const float ok = circ_valid(D, pv, ev) ? 1.0f : 0.0f;  // crackle does not enter
    if (!expand) {
      map[pk] = ch;
      validf[pk] = ok;
      ++pk;
    } else {
      for (int64_t c = 0; c < num_c; ++c) {
        ch.crackle = (int32_t)c;
        map[pe] = ch;
        validf[pe] = ok;
        ++pe;
      }
    }
  }
}

// Position of the first valid child at or after child index c.
__device__ __forceinline__ int64_t lower_bound64(const int64_t* a, int64_t n, int64_t c) {
  int64_t lo = 0, hi = n;
  while (lo < hi) {
    const int64_t mid = (lo + hi) >> 1;
    if (a[mid] < c) lo = mid + 1;
    else hi = mid;
  }
  return lo;
}

// Valid-child offsets at parent-batch boundaries (for the overflow rule).
__global__ void circ_boff_kernel(const int64_t* __restrict__ keep_off,
                                 const int64_t* __restrict__ exp_off, int64_t n,
                                 const int64_t* __restrict__ valid_ids, int64_t n_valid,
                                 int64_t* __restrict__ boff, const int64_t* __restrict__ cnt) {
  if (cnt) {  // device counts: cnt[0] parents, cnt[4] valid children
    n = cnt[0];
    n_valid = cnt[4];
    for (int64_t p = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; p <= n;
         p += (int64_t)gridDim.x * blockDim.x)
      boff[p] = lower_bound64(valid_ids, n_valid, keep_off[p] + exp_off[p]);
    return;
  }
  const int64_t p = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (p > n) return;
  boff[p] = lower_bound64(valid_ids, n_valid, keep_off[p] + exp_off[p]);
}

// Resolve (circ_taylor_resolve_batch / circ_taylor_fixed_resolve_batch) of
// one valid child; returns its class.
__device__ __forceinline__ int circ_resolve(const LokiPruneLevel& D, const double* pv,
                                            const double* ev, double f0, ChildRes* r) {
  const int m = 6;
  const int cls = circ_class(pv, ev, D.circ_sig_prop);
  double accel, vel, dd;
  if (cls != 0) {
    double a[6], b[6];
    circ_shift(pv, D.circ_dt_add, cls == 2, a);
    accel = a[3];
    if (D.moving) {
      circ_shift(pv, D.circ_dt_init, cls == 2, b);
      vel = __dsub_rn(a[4], b[4]);
      dd = __dsub_rn(a[5], b[5]);
    } else {
      vel = a[4];
      dd = a[5];
    }
  } else if (D.moving) {
    accel = tdot(pv, D.tm_a, 3, m);
    vel = __dsub_rn(tdot(pv, D.tm_a, 4, m), tdot(pv, D.tm_i, 4, m));
    dd = __dsub_rn(tdot(pv, D.tm_a, 5, m), tdot(pv, D.tm_i, 5, m));
  } else {
    accel = tdot(pv, D.tm_a, 3, m);
    vel = tdot(pv, D.tm_a, 4, m);
    dd = tdot(pv, D.tm_a, 5, m);
  }
  const double freq = __dmul_rn(f0, __dsub_rn(1.0, div_c(vel)));
  const double delay = div_c(dd);
  r->phase = phase_idx(D.dt_phase, f0, D.nbins, delay);
  r->ia = (int32_t)axis_index(accel, D.accel_min, D.accel_inv, D.n_accel);
  r->iff = (int32_t)axis_index(freq, D.freq_min, D.freq_inv, D.n_freq);
  return cls;
}

// Valid children v0 .. v0 + 31 (those below n_valid) of one warp.
__device__ __forceinline__ void circ_score_tile(
    const LokiPruneLevel& D, const double* __restrict__ leaves, const float* __restrict__ folds,
    int64_t batch, const LokiBranchInfo* __restrict__ info, const CircChild* __restrict__ map,
    const int64_t* __restrict__ valid_ids, int64_t n_valid, const float* __restrict__ seg,
    const LokiScoreSpec& sp, const ScoreK& SK, float* __restrict__ scores,
    int32_t* __restrict__ cidx, double* __restrict__ cphase, int8_t* __restrict__ ccls,
    int32_t* __restrict__ batch_taylor, unsigned* __restrict__ minmax_keys, float* tile,
    int64_t v0, int width = 32) {
  const int lane = threadIdx.x & 31;
  const int nb = D.nbins, P = 5;
  const int stride = score_stride(nb, sp.wmax);
  const int kmax = (int)std::min<int64_t>(width, n_valid - v0);
  int64_t my_par = 0, my_row = 0;
  int my_shift = 0;
  if (lane < kmax) {
    const int64_t v = v0 + lane;
    const CircChild ch = map[valid_ids[v]];
    const LokiBranchInfo B = info[ch.parent];
    const double* lf = leaves + (int64_t)ch.parent * (P + 2) * 2;
    double pv[6], ev[6];
    circ_child(B, lf, ch, pv, ev);
    ChildRes r;
    const int cls = circ_resolve(D, pv, ev, lf[(P + 1) * 2], &r);
    if (cls == 0) atomicOr(batch_taylor + ch.parent / batch, 1);
    cidx[2 * v] = r.ia;
    cidx[2 * v + 1] = r.iff;
    cphase[v] = r.phase;
    ccls[v] = (int8_t)cls;
    my_par = ch.parent;
    my_row = (int64_t)r.ia * D.n_freq + r.iff;
    my_shift = round_shift(r.phase, nb);
  }
  gather_norm_rows(folds, seg, my_par, my_row, my_shift, kmax, nb, tile, stride);
  score_tile_rows(tile, stride, nb, sp, SK, scores + v0, kmax, minmax_keys);
}

// With cnt (device counts) the valid children are pos_v[cnt[1]] (the
// validity compaction's total); block 0 records them in cnt[4] and st.
__global__ void __launch_bounds__(kPruneWarps * 32)
circ_score_kernel(LokiPruneLevel D, const double* __restrict__ leaves,
                  const float* __restrict__ folds, int64_t batch,
                  const LokiBranchInfo* __restrict__ info, const CircChild* __restrict__ map,
                  const int64_t* __restrict__ valid_ids, int64_t n_valid,
                  const float* __restrict__ seg, LokiScoreSpec sp, ScoreK SK,
                  float* __restrict__ scores, int32_t* __restrict__ cidx,
                  double* __restrict__ cphase, int8_t* __restrict__ ccls,
                  int32_t* __restrict__ batch_taylor, unsigned* __restrict__ minmax_keys,
                  int64_t* cnt, const int64_t* __restrict__ pos_v, LokiPruneLevelStats* st) {
  extern __shared__ float tiles[];
  const int warp = threadIdx.x >> 5;
  float* tile = tiles + (size_t)warp * 32 * score_stride(D.nbins, sp.wmax);
  if (!cnt) {
    const int64_t v0 = ((int64_t)blockIdx.x * kPruneWarps + warp) * 32;
    if (v0 < n_valid)
      circ_score_tile(D, leaves, folds, batch, info, map, valid_ids, n_valid, seg, sp, SK,
                      scores, cidx, cphase, ccls, batch_taylor, minmax_keys, tile, v0);
    return;
  }
  n_valid = pos_v[cnt[1]];
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    cnt[4] = n_valid;
    st->n_valid = n_valid;
  }
  for (int64_t t = (int64_t)blockIdx.x * kPruneWarps + warp; t * 32 < n_valid;
       t += (int64_t)gridDim.x * kPruneWarps) {
    circ_score_tile(D, leaves, folds, batch, info, map, valid_ids, n_valid, seg, sp, SK, scores,
                    cidx, cphase, ccls, batch_taylor, minmax_keys, tile, t * 32);
    __syncwarp();
  }
}

// New tree from the survivors: circ_taylor_transform_batch
// (core/circular.py:669-705, moving grid), the basis flag written by the
// moving-grid resolve (core/circular.py:478-509: 1 snap, 2 crackle, and 0 for
// the crackle children of a batch that also holds Taylor children), backtracks
// and folds.
// Survivors s0 .. s0 + 31 (those below n_surv) of one warp.
__device__ __forceinline__ void circ_emit_tile(
    const LokiPruneLevel& D, const double* __restrict__ leaves, const float* __restrict__ folds,
    int64_t batch, const LokiBranchInfo* __restrict__ info, const CircChild* __restrict__ map,
    const int64_t* __restrict__ valid_ids, const float* __restrict__ seg,
    const int64_t* __restrict__ surv, int64_t n_surv, const float* __restrict__ cscores,
    const int32_t* __restrict__ cidx, const double* __restrict__ cphase,
    const int8_t* __restrict__ ccls, const int32_t* __restrict__ batch_taylor,
    double* __restrict__ lout, float* __restrict__ fout, float* __restrict__ sout,
    float* __restrict__ seout, int32_t* __restrict__ bout, int64_t s0,
    const EmitExtra& X = EmitExtra(), int width = 32) {
  const int lane = threadIdx.x & 31;
  const int nb = D.nbins, P = 5, m = 6;
  const int kmax = (int)std::min<int64_t>(width, n_surv - s0);
  int64_t my_par = 0, my_row = 0;
  int my_shift = 0;
  if (lane < kmax) {
    const int64_t s = s0 + lane;
    const int64_t v = surv[s];
    const CircChild ch = map[valid_ids[v]];
    const LokiBranchInfo B = info[ch.parent];
    const double* lf = leaves + (int64_t)ch.parent * (P + 2) * 2;
    double pv[6], ev[6];
    circ_child(B, lf, ch, pv, ev);
    const int cls = ccls[v];
    double* lo = lout + s * (P + 2) * 2;
    double flag = lf[2 * m + 1];
    if (D.moving) {
      if (cls == 1) flag = 1.0;
      else if (cls == 2) flag = batch_taylor[ch.parent / batch] ? 0.0 : 2.0;
      if (cls != 0) {
        double o[6];
        circ_shift(pv, D.circ_dt_next, cls == 2, o);
        for (int i = 0; i < m; ++i) {
          lo[2 * i] = o[i];
          lo[2 * i + 1] = ev[i];
        }
      } else {
        for (int i = 0; i < m; ++i) lo[2 * i] = tdot(pv, D.tm_n, i, m);
        if (D.tiling == 0) {
          for (int i = 0; i < m; ++i) lo[2 * i + 1] = __dmul_rn(ev[i], fabs(D.tm_n[i][i]));
        } else if (D.tiling == 2) {
          for (int i = 0; i < m; ++i) lo[2 * i + 1] = tdot(ev, D.tm_e, i, m);
        } else {
          double e2[6];
          for (int j = 0; j < m; ++j) e2[j] = __dmul_rn(ev[j], ev[j]);
          for (int i = 0; i < m; ++i) lo[2 * i + 1] = __dsqrt_rn(tdot(e2, D.tm_e, i, m));
        }
      }
    } else {
      for (int i = 0; i < m; ++i) {
        lo[2 * i] = pv[i];
        lo[2 * i + 1] = ev[i];
      }
    }
    lo[2 * m] = lf[2 * m];
    lo[2 * m + 1] = flag;
    const float sc = cscores[v];
    sout[s] = sc;
    seout[s] = sc;
    int32_t* bt = bout + s * (P + 2);
    const int ia = cidx[2 * v], iff = cidx[2 * v + 1];
    bt[0] = ch.parent;
    for (int j = 1; j < P + 1; ++j) bt[j] = 0;
    bt[D.nparams_ffa - 1] = ia;
    bt[D.nparams_ffa] = iff;
    bt[P + 1] = (int32_t)cphase[v];
    emit_extra(X, s, lo, sc, bt, P);
    my_par = ch.parent;
    my_row = (int64_t)ia * D.n_freq + iff;
    my_shift = round_shift(cphase[v], nb);
  }
  gather_add_rows(folds, seg, my_par, my_row, my_shift, kmax, nb, fout + s0 * 2 * nb);
}

__global__ void __launch_bounds__(kPruneWarps * 32)
circ_emit_kernel(LokiPruneLevel D, const double* __restrict__ leaves,
                 const float* __restrict__ folds, int64_t batch,
                 const LokiBranchInfo* __restrict__ info, const CircChild* __restrict__ map,
                 const int64_t* __restrict__ valid_ids, const float* __restrict__ seg,
                 const int64_t* __restrict__ surv, int64_t n_surv,
                 const float* __restrict__ cscores, const int32_t* __restrict__ cidx,
                 const double* __restrict__ cphase, const int8_t* __restrict__ ccls,
                 const int32_t* __restrict__ batch_taylor, double* __restrict__ lout,
                 float* __restrict__ fout, float* __restrict__ sout,
                 float* __restrict__ seout, int32_t* __restrict__ bout,
                 const int64_t* __restrict__ cnt) {
  const int warp = threadIdx.x >> 5;
  if (!cnt) {
    const int64_t s0 = ((int64_t)blockIdx.x * kPruneWarps + warp) * 32;
    if (s0 < n_surv)
      circ_emit_tile(D, leaves, folds, batch, info, map, valid_ids, seg, surv, n_surv, cscores,
                     cidx, cphase, ccls, batch_taylor, lout, fout, sout, seout, bout, s0);
    return;
  }
  n_surv = cnt[2];  // device counts: warps stride over the survivors' tiles
  for (int64_t t = (int64_t)blockIdx.x * kPruneWarps + warp; t * 32 < n_surv;
       t += (int64_t)gridDim.x * kPruneWarps)
    circ_emit_tile(D, leaves, folds, batch, info, map, valid_ids, seg, surv, n_surv, cscores,
                   cidx, cphase, ccls, batch_taylor, lout, fout, sout, seout, bout, t * 32);
}

// ---------------------------------------------------------------------------
// complex (Fourier) folds: PrunePolyTaylorComplexDPFuncts and the Chebyshev
// counterpart. Tree folds and FFA segment rows are (2, nbf) complex64, nbf =
// nbins / 2 + 1 (float2 re, im). One lane owns one child: it rotates the
// segment row with the phasor recurrence of shift_add_complex_batch
// (core/common.py:403-429), adds the parent fold, and scores the irfft of the
// sum (detection/scoring.py:285-292).
// ---------------------------------------------------------------------------

// Phasor step exp(-2 pi i shift / nbins) with the reference's float32 angle
// float32(-2 * float32(pi)) * float32(shift) / nbins.
__device__ __forceinline__ float2 prune_phasor(double phase, int nbins) {
  const float m2pi = -2.0f * (float)3.14159265358979323846;
  const float ang = __fdiv_rn(__fmul_rn(m2pi, (float)phase), (float)nbins);
  float sn, cs;
  sincosf(ang, &sn, &cs);
  return make_float2(cs, sn);
}

__device__ __forceinline__ float2 cmul_rn(float2 a, float2 b) {
  return make_float2(__fsub_rn(__fmul_rn(a.x, b.x), __fmul_rn(a.y, b.y)),
                     __fadd_rn(__fmul_rn(a.x, b.y), __fmul_rn(a.y, b.x)));
}

// comb = seg * phasor^k + par, both components (par may be null: seg only).
__device__ __forceinline__ void rotate_add(const float2* __restrict__ seg,
                                           const float2* __restrict__ par, float2 delta, int nbf,
                                           float2* __restrict__ comb) {
  for (int c = 0; c < 2; ++c) {
    float2 ph = make_float2(1.0f, 0.0f);
    for (int k = 0; k < nbf; ++k) {
      const float2 r = cmul_rn(seg[c * nbf + k], ph);
      const float2 p = par ? par[c * nbf + k] : make_float2(0.0f, 0.0f);
      comb[c * nbf + k] = make_float2(__fadd_rn(r.x, p.x), __fadd_rn(r.y, p.y));
      ph = cmul_rn(ph, delta);
    }
  }
}

// irfft (n = nbins, even) of both components, then e / sqrt(v) into row.
// tw holds cos, then sin, of 2 pi t / nbins (float32 of the exact value).
__device__ __forceinline__ void irfft_norm(const float2* __restrict__ comb, int nbins, int nbf,
                                           const float* __restrict__ tw, float* row) {
  const float inv = 1.0f / (float)nbins;
  for (int j = 0; j < nbins; ++j) {
    float x[2];
    for (int c = 0; c < 2; ++c) {
      const float2* X = comb + c * nbf;
      float acc = X[0].x;
      const float nyq = X[nbf - 1].x;
      acc = (j & 1) ? __fsub_rn(acc, nyq) : __fadd_rn(acc, nyq);
      int idx = 0;
      for (int m = 1; m < nbf - 1; ++m) {
        idx += j;
        if (idx >= nbins) idx -= nbins;
        const float t = __fsub_rn(__fmul_rn(X[m].x, tw[idx]), __fmul_rn(X[m].y, tw[nbins + idx]));
        acc = __fadd_rn(acc, __fmul_rn(2.0f, t));
      }
      x[c] = __fmul_rn(acc, inv);
    }
    row[j] = __fdiv_rn(x[0], __fsqrt_rn(x[1]));
  }
}

__device__ __forceinline__ void load_twiddles(float* tw, int nbins) {
  for (int t = threadIdx.x; t < nbins; t += blockDim.x) {
    double s, c;
    sincospi(2.0 * (double)t / (double)nbins, &s, &c);
    tw[t] = (float)c;
    tw[nbins + t] = (float)s;
  }
}

// Per-warp shared memory of the complex kernels: 32 lanes x (2, nbf) float2
// sums, then the 32-row score tile.
__host__ __device__ inline size_t cplx_warp_floats(int nbins, int stride) {
  return (size_t)32 * 2 * (nbins / 2 + 1) * 2 + (size_t)32 * stride;
}

// One child of the complex tree: resolve, rotate-add the segment row onto the
// parent fold, score the sum through its irfft (comb and trow: this lane's
// scratch, tw: the block's twiddles).
__device__ __forceinline__ void score_child_complex(
    const LokiPruneLevel& D, const double* __restrict__ leaves, const float2* __restrict__ folds,
    int64_t n_parents, const LokiBranchInfo* __restrict__ info,
    const int64_t* __restrict__ offsets, const float2* __restrict__ seg, const LokiScoreSpec& sp,
    const ScoreK& SK,
    float* __restrict__ scores, int32_t* __restrict__ cidx, double* __restrict__ cphase,
    unsigned* __restrict__ minmax_keys, const float* tw, float2* comb, float* trow, int64_t c) {
  const int nb = D.nbins, nbf = nb / 2 + 1, P = D.poly_order;
  const int64_t par = find_parent(offsets, n_parents, c);
  const LokiBranchInfo B = info[par];
  const double* lf = leaves + par * (P + 2) * 2;
  double pv[LOKI_MAX_PARAMS + 1];
  child_params(B, P, c - offsets[par], pv);
  pv[P] = B.d0;
  const ChildRes r = resolve_child(D, P, pv, lf[(P + 1) * 2]);
  cidx[2 * c] = r.ia;
  cidx[2 * c + 1] = r.iff;
  cphase[c] = r.phase;
  const int64_t row = (int64_t)r.ia * D.n_freq + r.iff;
  rotate_add(seg + row * 2 * nbf, folds + par * 2 * nbf, prune_phasor(r.phase, nb), nbf, comb);
  irfft_norm(comb, nb, nbf, tw, trow);
  float s;
  score_row(trow, nb, sp, SK, &s);
  scores[c] = s;
  if (s == s) {
    atomicMin(minmax_keys, float_key(s));
    atomicMax(minmax_keys + 1, float_key(s));
  }
}

__global__ void __launch_bounds__(kPruneWarps * 32)
prune_score_complex_kernel(LokiPruneLevel D, const double* __restrict__ leaves,
                           const float2* __restrict__ folds, int64_t n_parents,
                           const LokiBranchInfo* __restrict__ info,
                           const int64_t* __restrict__ offsets, int64_t n_children,
                           const float2* __restrict__ seg, LokiScoreSpec sp, ScoreK SK,
                           float* __restrict__ scores, int32_t* __restrict__ cidx,
                           double* __restrict__ cphase, unsigned* __restrict__ minmax_keys) {
  extern __shared__ float smem[];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int nb = D.nbins, nbf = nb / 2 + 1;
  const int stride = score_stride(nb, sp.wmax);
  float* tw = smem;
  load_twiddles(tw, nb);
  __syncthreads();
  float* wbase = smem + 2 * nb + (size_t)warp * cplx_warp_floats(nb, stride);
  float2* comb = reinterpret_cast<float2*>(wbase) + (size_t)lane * 2 * nbf;
  float* tile = wbase + (size_t)32 * 2 * nbf * 2;
  const int64_t c = ((int64_t)blockIdx.x * kPruneWarps + warp) * 32 + lane;
  if (c >= n_children) return;
  score_child_complex(D, leaves, folds, n_parents, info, offsets, seg, sp, SK, scores, cidx, cphase,
                      minmax_keys, tw, comb, tile + lane * stride, c);
}

// The rows one survivor's fold is made of.
struct EmitRow {
  int64_t par, row;
  double phase;
};

// One survivor of the complex tree: transform and backtrack, its fold's rows
// returned.
template <int KP = 0>
__device__ __forceinline__ EmitRow emit_one_complex_leaf(
    const LokiPruneLevel& D, const double* __restrict__ leaves,
    const LokiBranchInfo* __restrict__ info, const int64_t* __restrict__ offsets,
    const int64_t* __restrict__ surv, const float* __restrict__ cscores,
    const int32_t* __restrict__ cidx, const double* __restrict__ cphase,
    double* __restrict__ lout, float* __restrict__ sout, float* __restrict__ seout,
    int32_t* __restrict__ bout, int64_t s, int64_t par, const EmitExtra& X = EmitExtra()) {
  const int P = tree_order<KP>(D), m = P + 1;
  const int64_t c = surv[s];
  const LokiBranchInfo B = info[par];
  const double* lf = leaves + par * (P + 2) * 2;
  double pv[LOKI_MAX_PARAMS + 1], ev[LOKI_MAX_PARAMS + 1];
  child_params(B, P, c - offsets[par], pv);
  pv[P] = B.d0;
  for (int j = 0; j < P; ++j) ev[j] = B.dact[j];
  ev[P] = 0.0;
  double* lo = lout + s * (P + 2) * 2;
  if (D.moving) {
    for (int i = 0; i < m; ++i) lo[2 * i] = tdot(pv, D.tm_n, i, m);
    if (D.tiling == 0) {
      for (int i = 0; i < m; ++i) lo[2 * i + 1] = __dmul_rn(ev[i], fabs(D.tm_n[i][i]));
    } else if (D.tiling == 2) {
      for (int i = 0; i < m; ++i) lo[2 * i + 1] = tdot(ev, D.tm_e, i, m);
    } else {
      double e2[LOKI_MAX_PARAMS + 1];
      for (int j = 0; j < m; ++j) e2[j] = __dmul_rn(ev[j], ev[j]);
      for (int i = 0; i < m; ++i) lo[2 * i + 1] = __dsqrt_rn(tdot(e2, D.tm_e, i, m));
    }
  } else {
    for (int i = 0; i < m; ++i) {
      lo[2 * i] = pv[i];
      lo[2 * i + 1] = ev[i];
    }
  }
  lo[2 * m] = lf[2 * m];
  lo[2 * m + 1] = lf[2 * m + 1];
  sout[s] = cscores[c];
  seout[s] = cscores[c];
  int32_t* bt = bout + s * (P + 2);
  const int ia = cidx[2 * c], iff = cidx[2 * c + 1];
  bt[0] = (int32_t)par;
  for (int j = 1; j < P + 1; ++j) bt[j] = 0;
  bt[D.nparams_ffa - 1] = ia;
  bt[D.nparams_ffa] = iff;
  bt[P + 1] = (int32_t)cphase[c];
  emit_extra(X, s, lo, cscores[c], bt, P);
  return {par, (int64_t)ia * D.n_freq + iff, cphase[c]};
}

__device__ __forceinline__ void emit_one_complex(
    const LokiPruneLevel& D, const double* __restrict__ leaves, const float2* __restrict__ folds,
    const LokiBranchInfo* __restrict__ info, const int64_t* __restrict__ offsets,
    int64_t n_parents, const float2* __restrict__ seg, const int64_t* __restrict__ surv,
    const float* __restrict__ cscores, const int32_t* __restrict__ cidx,
    const double* __restrict__ cphase, double* __restrict__ lout, float2* __restrict__ fout,
    float* __restrict__ sout, float* __restrict__ seout, int32_t* __restrict__ bout,
    int64_t s) {
  const int nb = D.nbins, nbf = nb / 2 + 1;
  const EmitRow r = emit_one_complex_leaf(D, leaves, info, offsets, surv, cscores, cidx, cphase,
                                          lout, sout, seout, bout, s,
                                          find_parent(offsets, n_parents, surv[s]));
  rotate_add(seg + r.row * 2 * nbf, folds + r.par * 2 * nbf, prune_phasor(r.phase, nb), nbf,
             fout + s * 2 * nbf);
}

// Survivors of the complex tree: transform / backtrack exactly as
// prune_emit_kernel, the fold written as the complex sum.
__global__ void __launch_bounds__(kPruneWarps * 32)
prune_emit_complex_kernel(LokiPruneLevel D, const double* __restrict__ leaves,
                          const float2* __restrict__ folds,
                          const LokiBranchInfo* __restrict__ info,
                          const int64_t* __restrict__ offsets, int64_t n_parents,
                          const float2* __restrict__ seg, const int64_t* __restrict__ surv,
                          int64_t n_surv, const float* __restrict__ cscores,
                          const int32_t* __restrict__ cidx, const double* __restrict__ cphase,
                          double* __restrict__ lout, float2* __restrict__ fout,
                          float* __restrict__ sout, float* __restrict__ seout,
                          int32_t* __restrict__ bout) {
  const int64_t s = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (s >= n_surv) return;
  emit_one_complex(D, leaves, folds, info, offsets, n_parents, seg, surv, cscores, cidx, cphase,
                   lout, fout, sout, seout, bout, s);
}

// Ascend of the complex tree (dyn_poly_taylor.py:632-679 with
// core/common.py:460-490): per survivor the rotated segment rows are summed
// over the segments in order, then the sum is scored through its irfft.
// Ascend of one survivor of the complex tree.
__device__ __forceinline__ void ascend_one_complex(
    const LokiPruneLevel& D, const double* __restrict__ leaves, float2* __restrict__ folds,
    float* __restrict__ scores, float* __restrict__ scores_ep, int nseg,
    const double* __restrict__ tm_seg, const double* __restrict__ dt_seg,
    const int32_t* __restrict__ seg_idx, const float2* __restrict__ ffa, int64_t seg_stride,
    const LokiScoreSpec& sp, const ScoreK& SK, const float* tw, float2* comb, float* trow,
    int64_t r) {
  const int nb = D.nbins, nbf = nb / 2 + 1, P = D.poly_order, m = P + 1;
  const double* lf = leaves + r * (P + 2) * 2;
  double pv[LOKI_MAX_PARAMS + 1], ev[LOKI_MAX_PARAMS + 1];
  for (int i = 0; i < m; ++i) {
    pv[i] = lf[2 * i];
    ev[i] = lf[2 * i + 1];
  }
  const double f0 = lf[2 * m];
  // circular tree: class of the survivor (core/circular.py:597-666)
  const int cls = D.basis == 2 ? circ_class(pv, ev, D.circ_sig_prop) : 0;
  for (int k = 0; k < 2 * nbf; ++k) comb[k] = make_float2(0.0f, 0.0f);
  for (int sg = 0; sg < nseg; ++sg) {
    const double(*T)[LOKI_MAX_PARAMS + 1] =
        reinterpret_cast<const double(*)[LOKI_MAX_PARAMS + 1]>(tm_seg + sg * 36);
    double accel, vel, dd;
    if (D.basis == 1) {
      double a[LOKI_MAX_PARAMS + 1];
      for (int i = 0; i < m; ++i) a[i] = tdot(pv, T, i, m);
      cheby_low3(D, a, m, &accel, &vel, &dd);
    } else if (cls != 0) {  // circular survivors: closed-form propagation
      double a[6];
      circ_shift(pv, dt_seg[sg], cls == 2, a);
      accel = a[3];
      vel = a[4];
      dd = a[5];
    } else {
      accel = tdot(pv, T, P - 2, m);
      vel = tdot(pv, T, P - 1, m);
      dd = tdot(pv, T, P, m);
    }
    const double freq = __dmul_rn(f0, __dsub_rn(1.0, div_c(vel)));
    const double delay = div_c(dd);
    const double ph = phase_idx(dt_seg[sg], f0, nb, delay);
    const int64_t ia = axis_index(accel, D.accel_min, D.accel_inv, D.n_accel);
    const int64_t iff = axis_index(freq, D.freq_min, D.freq_inv, D.n_freq);
    const float2* row = ffa + (int64_t)seg_idx[sg] * seg_stride + (ia * D.n_freq + iff) * 2 * nbf;
    const float2 delta = prune_phasor(ph, nb);
    for (int c = 0; c < 2; ++c) {  // res += row * phasor^k
      float2 p = make_float2(1.0f, 0.0f);
      for (int k = 0; k < nbf; ++k) {
        const float2 t = cmul_rn(row[c * nbf + k], p);
        float2& a = comb[c * nbf + k];
        a = make_float2(__fadd_rn(a.x, t.x), __fadd_rn(a.y, t.y));
        p = cmul_rn(p, delta);
      }
    }
  }
  float2* o = folds + r * 2 * nbf;
  for (int k = 0; k < 2 * nbf; ++k) o[k] = comb[k];
  irfft_norm(comb, nb, nbf, tw, trow);
  scores_ep[r] = scores[r];
  float s;
  score_row(trow, nb, sp, SK, &s);
  scores[r] = s;
}

__global__ void __launch_bounds__(kPruneWarps * 32)
prune_ascend_complex_kernel(LokiPruneLevel D, const double* __restrict__ leaves,
                            float2* __restrict__ folds, float* __restrict__ scores,
                            float* __restrict__ scores_ep, int64_t n, int nseg,
                            const double* __restrict__ tm_seg,
                            const double* __restrict__ dt_seg,
                            const int32_t* __restrict__ seg_idx,
                            const float2* __restrict__ ffa, int64_t seg_stride,
                            LokiScoreSpec sp, ScoreK SK) {
  extern __shared__ float smem[];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int nb = D.nbins, nbf = nb / 2 + 1;
  const int stride = score_stride(nb, sp.wmax);
  float* tw = smem;
  load_twiddles(tw, nb);
  __syncthreads();
  float* wbase = smem + 2 * nb + (size_t)warp * cplx_warp_floats(nb, stride);
  float2* comb = reinterpret_cast<float2*>(wbase) + (size_t)lane * 2 * nbf;
  float* tile = wbase + (size_t)32 * 2 * nbf * 2;
  const int64_t r = ((int64_t)blockIdx.x * kPruneWarps + warp) * 32 + lane;
  if (r >= n) return;
  ascend_one_complex(D, leaves, folds, scores, scores_ep, nseg, tm_seg, dt_seg, seg_idx, ffa,
                     seg_stride, sp, SK, tw, comb, tile + lane * stride, r);
}

// ---------------------------------------------------------------------------
// circular-orbit tree over complex folds (PruneCircTaylorComplexDPFuncts,
// dynamic/dyn_circular_taylor.py:168-330): the circular branch, validation,
// resolve and transform of the real-fold circular kernels, with the complex
// shift-add (core/common.py:403-429) and irfft scoring
// (detection/scoring.py:285-292) of the complex Taylor kernels.
// ---------------------------------------------------------------------------

// Valid child v of the complex circular tree: resolve, rotate + add into
// the lane's comb buffer, irfft into trow, score (tw: the block's twiddles).
__device__ __forceinline__ void circ_score_one_complex(
    const LokiPruneLevel& D, const double* __restrict__ leaves, const float2* __restrict__ folds,
    int64_t batch, const LokiBranchInfo* __restrict__ info, const CircChild* __restrict__ map,
    const int64_t* __restrict__ valid_ids, const float2* __restrict__ seg,
    const LokiScoreSpec& sp, const ScoreK& SK, const float* tw, float2* comb, float* trow,
    float* __restrict__ scores, int32_t* __restrict__ cidx, double* __restrict__ cphase,
    int8_t* __restrict__ ccls, int32_t* __restrict__ batch_taylor,
    unsigned* __restrict__ minmax_keys, int64_t v) {
  const int nb = D.nbins, nbf = nb / 2 + 1, P = 5;
  const CircChild ch = map[valid_ids[v]];
  const LokiBranchInfo B = info[ch.parent];
  const double* lf = leaves + (int64_t)ch.parent * (P + 2) * 2;
  double pv[6], ev[6];
  circ_child(B, lf, ch, pv, ev);
  ChildRes r;
  const int cls = circ_resolve(D, pv, ev, lf[(P + 1) * 2], &r);
  if (cls == 0) atomicOr(batch_taylor + ch.parent / batch, 1);
  cidx[2 * v] = r.ia;
  cidx[2 * v + 1] = r.iff;
  cphase[v] = r.phase;
  ccls[v] = (int8_t)cls;
  const int64_t row = (int64_t)r.ia * D.n_freq + r.iff;
  rotate_add(seg + row * 2 * nbf, folds + (int64_t)ch.parent * 2 * nbf,
             prune_phasor(r.phase, nb), nbf, comb);
  irfft_norm(comb, nb, nbf, tw, trow);
  float s;
  score_row(trow, nb, sp, SK, &s);
  scores[v] = s;
  if (s == s) {
    atomicMin(minmax_keys, float_key(s));
    atomicMax(minmax_keys + 1, float_key(s));
  }
}

__global__ void __launch_bounds__(kPruneWarps * 32)
circ_score_complex_kernel(LokiPruneLevel D, const double* __restrict__ leaves,
                          const float2* __restrict__ folds, int64_t batch,
                          const LokiBranchInfo* __restrict__ info,
                          const CircChild* __restrict__ map,
                          const int64_t* __restrict__ valid_ids, int64_t n_valid,
                          const float2* __restrict__ seg, LokiScoreSpec sp, ScoreK SK,
                          float* __restrict__ scores, int32_t* __restrict__ cidx,
                          double* __restrict__ cphase, int8_t* __restrict__ ccls,
                          int32_t* __restrict__ batch_taylor,
                          unsigned* __restrict__ minmax_keys) {
  extern __shared__ float smem[];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int nb = D.nbins, nbf = nb / 2 + 1;
  const int stride = score_stride(nb, sp.wmax);
  float* tw = smem;
  load_twiddles(tw, nb);
  __syncthreads();
  float* wbase = smem + 2 * nb + (size_t)warp * cplx_warp_floats(nb, stride);
  float2* comb = reinterpret_cast<float2*>(wbase) + (size_t)lane * 2 * nbf;
  float* tile = wbase + (size_t)32 * 2 * nbf * 2;
  const int64_t v = ((int64_t)blockIdx.x * kPruneWarps + warp) * 32 + lane;
  if (v >= n_valid) return;
  circ_score_one_complex(D, leaves, folds, batch, info, map, valid_ids, seg, sp, SK, tw, comb,
                         tile + lane * stride, scores, cidx, cphase, ccls, batch_taylor,
                         minmax_keys, v);
}

// Survivor s of the complex circular tree (circ_emit_one's leaves, basis
// flag and backtracks; the fold written as the complex sum).
__device__ __forceinline__ EmitRow circ_emit_one_complex_leaf(
    const LokiPruneLevel& D, const double* __restrict__ leaves, int64_t batch,
    const LokiBranchInfo* __restrict__ info, const CircChild* __restrict__ map,
    const int64_t* __restrict__ valid_ids, const int64_t* __restrict__ surv,
    const float* __restrict__ cscores,
    const int32_t* __restrict__ cidx, const double* __restrict__ cphase,
    const int8_t* __restrict__ ccls, const int32_t* __restrict__ batch_taylor,
    double* __restrict__ lout, float* __restrict__ sout,
    float* __restrict__ seout, int32_t* __restrict__ bout, int64_t s,
    const EmitExtra& X = EmitExtra()) {
  const int P = 5, m = 6;
  const int64_t v = surv[s];
  const CircChild ch = map[valid_ids[v]];
  const LokiBranchInfo B = info[ch.parent];
  const double* lf = leaves + (int64_t)ch.parent * (P + 2) * 2;
  double pv[6], ev[6];
  circ_child(B, lf, ch, pv, ev);
  const int cls = ccls[v];
  double* lo = lout + s * (P + 2) * 2;
  double flag = lf[2 * m + 1];
  if (D.moving) {
    if (cls == 1) flag = 1.0;
    else if (cls == 2) flag = batch_taylor[ch.parent / batch] ? 0.0 : 2.0;
    if (cls != 0) {
      double o[6];
      circ_shift(pv, D.circ_dt_next, cls == 2, o);
      for (int i = 0; i < m; ++i) {
        lo[2 * i] = o[i];
        lo[2 * i + 1] = ev[i];
      }
    } else {
      for (int i = 0; i < m; ++i) lo[2 * i] = tdot(pv, D.tm_n, i, m);
      if (D.tiling == 0) {
        for (int i = 0; i < m; ++i) lo[2 * i + 1] = __dmul_rn(ev[i], fabs(D.tm_n[i][i]));
      } else if (D.tiling == 2) {
        for (int i = 0; i < m; ++i) lo[2 * i + 1] = tdot(ev, D.tm_e, i, m);
      } else {
        double e2[6];
        for (int j = 0; j < m; ++j) e2[j] = __dmul_rn(ev[j], ev[j]);
        for (int i = 0; i < m; ++i) lo[2 * i + 1] = __dsqrt_rn(tdot(e2, D.tm_e, i, m));
      }
    }
  } else {
    for (int i = 0; i < m; ++i) {
      lo[2 * i] = pv[i];
      lo[2 * i + 1] = ev[i];
    }
  }
  lo[2 * m] = lf[2 * m];
  lo[2 * m + 1] = flag;
  sout[s] = cscores[v];
  seout[s] = cscores[v];
  int32_t* bt = bout + s * (P + 2);
  const int ia = cidx[2 * v], iff = cidx[2 * v + 1];
  bt[0] = ch.parent;
  for (int j = 1; j < P + 1; ++j) bt[j] = 0;
  bt[D.nparams_ffa - 1] = ia;
  bt[D.nparams_ffa] = iff;
  bt[P + 1] = (int32_t)cphase[v];
  emit_extra(X, s, lo, cscores[v], bt, P);
  return {(int64_t)ch.parent, (int64_t)ia * D.n_freq + iff, cphase[v]};
}

__device__ __forceinline__ void circ_emit_one_complex(
    const LokiPruneLevel& D, const double* __restrict__ leaves, const float2* __restrict__ folds,
    int64_t batch, const LokiBranchInfo* __restrict__ info, const CircChild* __restrict__ map,
    const int64_t* __restrict__ valid_ids, const float2* __restrict__ seg,
    const int64_t* __restrict__ surv, const float* __restrict__ cscores,
    const int32_t* __restrict__ cidx, const double* __restrict__ cphase,
    const int8_t* __restrict__ ccls, const int32_t* __restrict__ batch_taylor,
    double* __restrict__ lout, float2* __restrict__ fout, float* __restrict__ sout,
    float* __restrict__ seout, int32_t* __restrict__ bout, int64_t s) {
  const int nb = D.nbins, nbf = nb / 2 + 1;
  const EmitRow r = circ_emit_one_complex_leaf(D, leaves, batch, info, map, valid_ids, surv,
                                               cscores, cidx, cphase, ccls, batch_taylor, lout,
                                               sout, seout, bout, s);
  rotate_add(seg + r.row * 2 * nbf, folds + r.par * 2 * nbf, prune_phasor(r.phase, nb), nbf,
             fout + s * 2 * nbf);
}

// Survivors of the complex circular tree: leaves, basis flag and backtracks as
// circ_emit_kernel, the fold written as the complex sum.
__global__ void __launch_bounds__(kPruneWarps * 32)
circ_emit_complex_kernel(LokiPruneLevel D, const double* __restrict__ leaves,
                         const float2* __restrict__ folds, int64_t batch,
                         const LokiBranchInfo* __restrict__ info,
                         const CircChild* __restrict__ map,
                         const int64_t* __restrict__ valid_ids, const float2* __restrict__ seg,
                         const int64_t* __restrict__ surv, int64_t n_surv,
                         const float* __restrict__ cscores, const int32_t* __restrict__ cidx,
                         const double* __restrict__ cphase, const int8_t* __restrict__ ccls,
                         const int32_t* __restrict__ batch_taylor, double* __restrict__ lout,
                         float2* __restrict__ fout, float* __restrict__ sout,
                         float* __restrict__ seout, int32_t* __restrict__ bout) {
  const int64_t s = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (s >= n_surv) return;
  circ_emit_one_complex(D, leaves, folds, batch, info, map, valid_ids, seg, surv, cscores, cidx,
                        cphase, ccls, batch_taylor, lout, fout, sout, seout, bout, s);
}

// ---------------------------------------------------------------------------
// Complex rows of 32 children at a time, 64 bins, with the arithmetic of
// rotate_add and irfft_norm. Every lane runs its child's phasor recurrence once,
// into a table of shared memory; then the warp combines the children's parent and
// segment rows whole, lane by harmonic (loads and stores of full lines), and, to
// score, each lane transforms its own child: every bin summed over the harmonics
// in order with each product and sum rounded. The angles of bins j, 64 - j, 32 - j
// and 32 + j have the same cosine and sine up to sign, so their four sums share
// two products, and the 64 sums are independent registers. A lane walking its
// rows in global memory and the bins one after the other took 56 ms for the 8.0e6
// children of a 16-run search; now 9.4, of which 2 are the latency of the 100
// levels with fewer than 500 children a run.
// ---------------------------------------------------------------------------

constexpr int kCplxRow = 33;  // float2 of one component; odd, so lanes miss each other's banks
__host__ __device__ constexpr int cplx64_warp_bytes() { return 2 * 32 * kCplxRow * 8; }

// Powers 0 .. 32 of each lane's phasor.
__device__ __forceinline__ void phasor_table(float2 delta, float2* T) {
  float2* t = T + (threadIdx.x & 31) * kCplxRow;
  float2 ph = make_float2(1.0f, 0.0f);
#pragma unroll 3
  for (int k = 0; k < 33; ++k) {
    t[k] = ph;
    ph = cmul_rn(ph, delta);
  }
  __syncwarp();
}

__device__ __forceinline__ float2 rotate_add1(float2 b, float2 ph, float2 a) {
  const float2 r = cmul_rn(b, ph);
  return make_float2(__fadd_rn(r.x, a.x), __fadd_rn(r.y, a.y));
}

// One component of the combined rows of children k < kmax: harmonic h of child k
// to out[k * stride + h].
__device__ __forceinline__ void combine_rows64(const float2* __restrict__ folds,
                                               const float2* __restrict__ seg, int64_t my_par,
                                               int64_t my_row, int kmax, int comp,
                                               const float2* T, float2* out, int stride) {
  const int lane = threadIdx.x & 31;
  const float2* fa = folds + comp * 33 + lane;
  const float2* fb = seg + comp * 33 + lane;
  constexpr int kU = 8;
  for (int k0 = 0; k0 < kmax; k0 += kU) {
    float2 a[kU], b[kU];
#pragma unroll
    for (int u = 0; u < kU; ++u) {
      const int k = min(k0 + u, kmax - 1);
      a[u] = __ldg(fa + (size_t)__shfl_sync(0xFFFFFFFFu, (uint32_t)my_par, k) * 66);
      b[u] = __ldg(fb + (size_t)__shfl_sync(0xFFFFFFFFu, (uint32_t)my_row, k) * 66);
    }
#pragma unroll
    for (int u = 0; u < kU; ++u)
      if (k0 + u < kmax)
        out[(k0 + u) * stride + lane] = rotate_add1(b[u], T[(k0 + u) * kCplxRow + lane], a[u]);
  }
  if (lane < kmax)  // the last harmonic, child by lane
    out[lane * stride + 32] =
        rotate_add1(__ldg(seg + my_row * 66 + comp * 33 + 32), T[lane * kCplxRow + 32],
                    __ldg(folds + my_par * 66 + comp * 33 + 32));
  __syncwarp();
}

// Twiddles by harmonic: W[m * 16 + j] = (cos, sin) of 2 pi m j / 64 for harmonics
// m = 1 .. 31 (row m - 1), after the 64 angles they are taken from.
constexpr int kTwiddle64Bytes = 512 + 31 * 16 * 8;

__device__ __forceinline__ void load_twiddles64(float* smem) {
  float2 *tw = reinterpret_cast<float2*>(smem), *W = tw + 64;
  for (int t = threadIdx.x; t < 64; t += blockDim.x) tw[t] = make_float2(cos64(t), sin64(t));
  __syncthreads();
  for (int t = threadIdx.x; t < 31 * 16; t += blockDim.x)
    W[t] = tw[((t >> 4) + 1) * (t & 15) & 63];
}

// The 64 sums of one component: p[j] = (bin j, bin 64 - j), q[j] = (bin 32 + j,
// bin 32 - j) for j = 1 .. 15, and bins 0, 32, 16 and 48.
struct Sums64 {
  unsigned long long p[16], q[16];
  float b0, b32, b16, b48;
};

__device__ __forceinline__ unsigned long long fma2_rn(unsigned long long a, unsigned long long b,
                                                      unsigned long long c) {
  unsigned long long d;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
  return d;
}

// Harmonic m (M = m mod 4) into the sums: doubling is exact, so 2 t + acc rounds
// once, as the sum of the doubled term.
template <int M>
__device__ __forceinline__ void irfft64_step(const float2 x, const float2* __restrict__ W,
                                             Sums64& S) {
  constexpr bool odd = M & 1;
  constexpr float sg = odd ? -2.0f : 2.0f, v = (M & 2) ? -2.0f : 2.0f;
  const unsigned long long two = pack2(2.0f, 2.0f), sgn = pack2(sg, sg), xx = pack2(x.x, x.y);
  S.b0 = __fmaf_rn(2.0f, x.x, S.b0);
  S.b32 = __fmaf_rn(sg, x.x, S.b32);
  S.b16 = __fmaf_rn(odd ? -v : v, odd ? x.y : x.x, S.b16);
  S.b48 = __fmaf_rn(v, odd ? x.y : x.x, S.b48);
#pragma unroll
  for (int j2 = 0; j2 < 16; j2 += 2) {
    const ulonglong2 w = *reinterpret_cast<const ulonglong2*>(W + j2);
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int j = j2 + h;
      if (j == 0) continue;
      unsigned long long ab;
      asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(ab) : "l"(xx), "l"(h ? w.y : w.x));
      float a, b;
      unpack2(ab, a, b);
      const unsigned long long uz = pack2(__fsub_rn(a, b), __fadd_rn(a, b));
      S.p[j] = fma2_rn(two, uz, S.p[j]);
      S.q[j] = fma2_rn(sgn, uz, S.q[j]);
    }
  }
}

// irfft_norm's sums of one component (unscaled).
__device__ __forceinline__ void irfft64_sums(const float2* __restrict__ X,
                                             const float2* __restrict__ W, Sums64& S) {
  const float x0 = X[0].x, nyq = X[32].x;
  const float even = __fadd_rn(x0, nyq), odd = __fsub_rn(x0, nyq);
  S.b0 = S.b32 = S.b16 = S.b48 = even;
#pragma unroll
  for (int j = 1; j < 16; ++j) S.p[j] = S.q[j] = (j & 1) ? pack2(odd, odd) : pack2(even, even);
#pragma unroll 1
  for (int m = 1; m < 29; m += 4) {
    irfft64_step<1>(X[m], W + (m - 1) * 16, S);
    irfft64_step<2>(X[m + 1], W + m * 16, S);
    irfft64_step<3>(X[m + 2], W + (m + 1) * 16, S);
    irfft64_step<0>(X[m + 3], W + (m + 2) * 16, S);
  }
  irfft64_step<1>(X[29], W + 28 * 16, S);
  irfft64_step<2>(X[30], W + 29 * 16, S);
  irfft64_step<3>(X[31], W + 30 * 16, S);
}

// The same by four lanes a child: this one's bins of j = 4 part + h, h < 4 (p[h],
// q[h]; j = 0 stands for none), and bins 0, 32, 16 and 48.
struct Sums16 {
  unsigned long long p[4], q[4];
  float b0, b32, b16, b48;
};

template <int M>
__device__ __forceinline__ void irfft16_step(const float2 x, const float2* __restrict__ W,
                                             Sums16& S) {
  constexpr bool odd = M & 1;
  constexpr float sg = odd ? -2.0f : 2.0f, v = (M & 2) ? -2.0f : 2.0f;
  const unsigned long long two = pack2(2.0f, 2.0f), sgn = pack2(sg, sg), xx = pack2(x.x, x.y);
  S.b0 = __fmaf_rn(2.0f, x.x, S.b0);
  S.b32 = __fmaf_rn(sg, x.x, S.b32);
  S.b16 = __fmaf_rn(odd ? -v : v, odd ? x.y : x.x, S.b16);
  S.b48 = __fmaf_rn(v, odd ? x.y : x.x, S.b48);
#pragma unroll
  for (int h = 0; h < 4; h += 2) {
    const ulonglong2 w = *reinterpret_cast<const ulonglong2*>(W + h);
#pragma unroll
    for (int g = 0; g < 2; ++g) {
      unsigned long long ab;
      asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(ab) : "l"(xx), "l"(g ? w.y : w.x));
      float a, b;
      unpack2(ab, a, b);
      const unsigned long long uz = pack2(__fsub_rn(a, b), __fadd_rn(a, b));
      S.p[h + g] = fma2_rn(two, uz, S.p[h + g]);
      S.q[h + g] = fma2_rn(sgn, uz, S.q[h + g]);
    }
  }
}

__device__ __forceinline__ void irfft16_sums(const float2* __restrict__ X,
                                             const float2* __restrict__ W, int part, Sums16& S) {
  const float x0 = X[0].x, nyq = X[32].x;
  const float even = __fadd_rn(x0, nyq), odd = __fsub_rn(x0, nyq);
  W += 4 * part;  // j has the parity of h
  S.b0 = S.b32 = S.b16 = S.b48 = even;
#pragma unroll
  for (int h = 0; h < 4; ++h) S.p[h] = S.q[h] = (h & 1) ? pack2(odd, odd) : pack2(even, even);
#pragma unroll 1
  for (int m = 1; m < 29; m += 4) {
    irfft16_step<1>(X[m], W + (m - 1) * 16, S);
    irfft16_step<2>(X[m + 1], W + m * 16, S);
    irfft16_step<3>(X[m + 2], W + (m + 1) * 16, S);
    irfft16_step<0>(X[m + 3], W + (m + 2) * 16, S);
  }
  irfft16_step<1>(X[29], W + 28 * 16, S);
  irfft16_step<2>(X[30], W + 29 * 16, S);
  irfft16_step<3>(X[31], W + 30 * 16, S);
}

// e / sqrt(v) of two bins' sums.
__device__ __forceinline__ unsigned long long norm64(unsigned long long e, unsigned long long v) {
  const float inv = 1.0f / 64.0f;
  float e0, e1, v0, v1;
  unpack2(e, e0, e1);
  unpack2(v, v0, v1);
  return pack2(__fdiv_rn(__fmul_rn(e0, inv), __fsqrt_rn(__fmul_rn(v0, inv))),
               __fdiv_rn(__fmul_rn(e1, inv), __fsqrt_rn(__fmul_rn(v1, inv))));
}

// Bins j, 64 - j, 32 + j and 32 - j (j = 0: bins 0, 32, 16 and 48) of a row.
__device__ __forceinline__ void put_bins(float* row, int j, unsigned long long p,
                                         unsigned long long q) {
  float x0, x1, y0, y1;
  unpack2(p, x0, x1);
  unpack2(q, y0, y1);
  row[j] = x0;
  row[j == 0 ? 32 : 64 - j] = x1;
  row[j == 0 ? 16 : 32 + j] = y0;
  row[j == 0 ? 48 : 32 - j] = y1;
}

// Scores of the warp's children (rows and phasor held lane by lane).
__device__ __forceinline__ void cplx64_score(const float2* __restrict__ folds,
                                             const float2* __restrict__ seg, int64_t my_par,
                                             int64_t my_row, float2 delta, int kmax,
                                             const float2* tw, float2* buf,
                                             const LokiScoreSpec& sp, const ScoreK& SK,
                                             float* __restrict__ scores,
                                             unsigned* __restrict__ minmax_keys) {
  const int lane = threadIdx.x & 31;
  float2 *A = buf, *T = buf + 32 * kCplxRow;
  const float2* row = A + lane * kCplxRow;
  unsigned long long* keep = reinterpret_cast<unsigned long long*>(T + lane * kCplxRow);
  const int stride = score_stride(64, sp.wmax);
  float* tile = reinterpret_cast<float*>(buf);
  phasor_table(delta, T);
  if (kmax <= 8) {  // four lanes a child (a level of 100 children a run: 44 -> 20 us)
    const int part = lane & 3;
    const float2* sub = A + (lane >> 2) * kCplxRow;
    Sums16 E, V;
    combine_rows64(folds, seg, my_par, my_row, kmax, 0, T, A, kCplxRow);
    irfft16_sums(sub, tw, part, E);
    __syncwarp();
    combine_rows64(folds, seg, my_par, my_row, kmax, 1, T, A, kCplxRow);
    irfft16_sums(sub, tw, part, V);
    if (part == 0) {
      E.p[0] = pack2(E.b0, E.b32), E.q[0] = pack2(E.b16, E.b48);
      V.p[0] = pack2(V.b0, V.b32), V.q[0] = pack2(V.b16, V.b48);
    }
    __syncwarp();  // the buffer becomes the score tile
#pragma unroll
    for (int h = 0; h < 4; ++h)
      put_bins(tile + (lane >> 2) * stride, 4 * part + h, norm64(E.p[h], V.p[h]),
               norm64(E.q[h], V.q[h]));
    __syncwarp();
    score_tile_rows(tile, stride, 64, sp, SK, scores, kmax, minmax_keys);
    return;
  }
  Sums64 S;
  combine_rows64(folds, seg, my_par, my_row, kmax, 0, T, A, kCplxRow);
  irfft64_sums(row, tw, S);
  __syncwarp();  // every lane has read its row
  combine_rows64(folds, seg, my_par, my_row, kmax, 1, T, A, kCplxRow);
  // the phasors have been used: their rows keep the first component's sums, which
  // would be 64 more registers. (Three blocks an SM spill 108 bytes a thread and
  // were 5 % slower.)
#pragma unroll
  for (int j = 1; j < 16; ++j) {
    keep[j] = S.p[j];
    keep[16 + j] = S.q[j];
  }
  keep[0] = pack2(S.b0, S.b32);
  keep[16] = pack2(S.b16, S.b48);
  irfft64_sums(row, tw, S);
  S.p[0] = pack2(S.b0, S.b32);
  S.q[0] = pack2(S.b16, S.b48);
#pragma unroll
  for (int j = 0; j < 16; ++j) {
    S.p[j] = norm64(keep[j], S.p[j]);
    S.q[j] = norm64(keep[16 + j], S.q[j]);
  }
  __syncwarp();  // every lane has read its rows: the buffer becomes the score tile
#pragma unroll
  for (int j = 0; j < 16; ++j) put_bins(tile + lane * stride, j, S.p[j], S.q[j]);
  __syncwarp();
  score_tile_rows(tile, stride, 64, sp, SK, scores, kmax, minmax_keys);
}

// Complex sums of the warp's survivors, whole rows to fout.
__device__ __forceinline__ void cplx64_emit(const float2* __restrict__ folds,
                                            const float2* __restrict__ seg, int64_t my_par,
                                            int64_t my_row, float2 delta, int kmax, float2* buf,
                                            float2* __restrict__ fout) {
  phasor_table(delta, buf);
  for (int comp = 0; comp < 2; ++comp)
    combine_rows64(folds, seg, my_par, my_row, kmax, comp, buf, fout + comp * 33, 66);
}

// ---------------------------------------------------------------------------
// launchers
// ---------------------------------------------------------------------------

static int check_prune(const LokiPruneLevel* D) {
  if (!D) return set_error(LOKI_ERR_INVALID, "null prune level descriptor");
  if (D->poly_order < 2 || D->poly_order > LOKI_MAX_PARAMS)
    return set_error(LOKI_ERR_INVALID, "poly_order %d outside [2, %d]", D->poly_order,
                     LOKI_MAX_PARAMS);
  if (D->nbins < 2) return set_error(LOKI_ERR_INVALID, "nbins < 2");
  if (D->nparams_ffa < 2 || D->nparams_ffa > D->poly_order)
    return set_error(LOKI_ERR_INVALID, "nparams_ffa %d outside [2, poly_order]",
                     D->nparams_ffa);
  if (D->n_accel < 1 || D->n_freq < 1) return set_error(LOKI_ERR_INVALID, "empty FFA grid");
  if (D->tiling < 0 || D->tiling > 2) return set_error(LOKI_ERR_INVALID, "bad tiling");
  return LOKI_OK;
}

static int prune_spec_check(const LokiScoreSpec* sp, int nbins) {
  if (!sp || sp->nwidths < 1 || sp->nwidths > LOKI_MAX_WIDTHS)
    return set_error(LOKI_ERR_INVALID, "bad score spec");
  if (nbins + sp->wmax > 1024)
    return set_error(LOKI_ERR_UNSUPPORTED, "nbins + wmax above 1024 for pruning");
  return LOKI_OK;
}

}  // namespace loki

using namespace loki;

extern "C" int64_t loki_scan_scratch_bytes(int64_t n) {
  return std::max<int64_t>(1, (n + kScanBlock - 1) / kScanBlock) * (int64_t)sizeof(int64_t);
}

static int prune_branch_impl(const LokiPruneLevel* lvl, const double* leaves,
                             int64_t n_parents, const uint8_t* mask, LokiBranchInfo* info,
                             int64_t* offsets, void* scan_scratch, int64_t scan_scratch_bytes,
                             int32_t* dev_err, void* stream);

// End of a device-resident level (single thread): the level's record (score
// range from the ordered keys, as minmax_finish_kernel), then the survivors
// become the next level's parents and the keys restart.
__device__ __forceinline__ void level_end(int64_t* cnt, unsigned* keys, int32_t* ovf_flag,
                                          LokiPruneLevelStats* st) {
  st->n_surv = cnt[2];
  const bool none = keys[0] == 0xFFFFFFFFu;  // no finite score
  st->score_min = none ? 0.0f : key_float(keys[0]);
  st->score_max = none ? 0.0f : key_float(keys[1]);
  st->overflow = *ovf_flag;
  st->reserved = 0;
  *ovf_flag = 0;
  keys[0] = 0xFFFFFFFFu;
  keys[1] = 0u;
  cnt[3] += cnt[2];  // backtrack history rows
  cnt[0] = cnt[2];
}

// Best leaf of a tree (max score, first index on ties, as torch.argmax):
// one block reduces (score, index), then copies the leaf row and its score.
__device__ void block_best(const float* __restrict__ scores, int64_t n,
                           const double* __restrict__ leaves, int row,
                           double* __restrict__ leaf_out, float* __restrict__ score_out) {
  __shared__ float sv[32];
  __shared__ int64_t si[32];
  float bv = -INFINITY;
  int64_t bi = -1;
  // each thread visits its elements in increasing index order, so it keeps
  // its first maximum; float4 loads, four in flight, when the scores are
  // 16-byte aligned
  int64_t head = 0;
  if ((reinterpret_cast<uintptr_t>(scores) & 15) == 0) {
    const float4* s4 = reinterpret_cast<const float4*>(scores);
    const int64_t n4 = n >> 2;
    const int64_t step = blockDim.x;
    int64_t q = threadIdx.x;
    for (; q + 3 * step < n4; q += 4 * step) {
      float4 a[4];
#pragma unroll
      for (int u = 0; u < 4; ++u) a[u] = s4[q + u * step];
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const float c[4] = {a[u].x, a[u].y, a[u].z, a[u].w};
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          if (bi < 0 || c[k] > bv) {
            bv = c[k];
            bi = 4 * (q + u * step) + k;
          }
        }
      }
    }
    for (; q < n4; q += step) {
      const float4 a = s4[q];
      const float c[4] = {a.x, a.y, a.z, a.w};
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        if (bi < 0 || c[k] > bv) {
          bv = c[k];
          bi = 4 * q + k;
        }
      }
    }
    head = n4 << 2;
  }
  for (int64_t i = head + threadIdx.x; i < n; i += blockDim.x) {
    const float v = scores[i];
    if (bi < 0 || v > bv) {
      bv = v;
      bi = i;
    }
  }
  for (int o = 16; o > 0; o >>= 1) {
    const float ov = __shfl_down_sync(0xFFFFFFFFu, bv, o);
    const int64_t oi = __shfl_down_sync(0xFFFFFFFFu, bi, o);
    if (oi >= 0 && (bi < 0 || ov > bv || (ov == bv && oi < bi))) {
      bv = ov;
      bi = oi;
    }
  }
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if (lane == 0) {
    sv[warp] = bv;
    si[warp] = bi;
  }
  __syncthreads();
  if (warp == 0) {
    const int nw = (blockDim.x + 31) >> 5;
    bv = lane < nw ? sv[lane] : -INFINITY;
    bi = lane < nw ? si[lane] : -1;
    for (int o = 16; o > 0; o >>= 1) {
      const float ov = __shfl_down_sync(0xFFFFFFFFu, bv, o);
      const int64_t oi = __shfl_down_sync(0xFFFFFFFFu, bi, o);
      if (oi >= 0 && (bi < 0 || ov > bv || (ov == bv && oi < bi))) {
        bv = ov;
        bi = oi;
      }
    }
    bi = __shfl_sync(0xFFFFFFFFu, bi, 0);
    if (bi >= 0)
      for (int j = lane; j < row; j += 32) leaf_out[j] = leaves[bi * row + j];
    if (lane == 0 && bi >= 0) *score_out = scores[bi];
  }
}

__global__ void __launch_bounds__(1024)
prune_best_kernel(const float* __restrict__ scores, int64_t n, const double* __restrict__ leaves,
                  int row, double* __restrict__ leaf_out, float* __restrict__ score_out,
                  int64_t* lvl_cnt, unsigned* lvl_keys, int32_t* lvl_ovf,
                  LokiPruneLevelStats* lvl_st) {
  if (lvl_cnt) n = lvl_cnt[2];  // the level's survivors; 0 writes nothing
  block_best(scores, n, leaves, row, leaf_out, score_out);
  // every thread read the count before block_best's barrier
  if (threadIdx.x == 0 && lvl_cnt) level_end(lvl_cnt, lvl_keys, lvl_ovf, lvl_st);
}

extern "C" int loki_prune_best(const float* scores, int64_t n, const double* leaves,
                               int32_t row_len, double* leaf_out, float* score_out,
                               void* stream) {
  if (n < 0 || row_len < 1) return set_error(LOKI_ERR_INVALID, "bad sizes");
  if (n == 0) return LOKI_OK;
  if (!scores || !leaves || !leaf_out || !score_out)
    return set_error(LOKI_ERR_INVALID, "null pointer argument");
  note_launch();
  prune_best_kernel<<<1, 1024, 0, (cudaStream_t)stream>>>(scores, n, leaves, row_len, leaf_out,
                                                         score_out, nullptr, nullptr, nullptr,
                                                         nullptr);
  return check_launch("prune_best");
}

extern "C" int loki_prune_branch(const LokiPruneLevel* lvl, const double* leaves,
                                 int64_t n_parents, LokiBranchInfo* info, int64_t* offsets,
                                 void* scan_scratch, int64_t scan_scratch_bytes,
                                 int32_t* dev_err, void* stream) {
  return prune_branch_impl(lvl, leaves, n_parents, nullptr, info, offsets, scan_scratch,
                           scan_scratch_bytes, dev_err, stream);
}

extern "C" int loki_prune_branch_masked(const LokiPruneLevel* lvl, const double* leaves,
                                        int64_t n_parents, const uint8_t* parent_mask,
                                        LokiBranchInfo* info, int64_t* offsets,
                                        void* scan_scratch, int64_t scan_scratch_bytes,
                                        int32_t* dev_err, void* stream) {
  if (n_parents > 0 && !parent_mask) return set_error(LOKI_ERR_INVALID, "null parent mask");
  return prune_branch_impl(lvl, leaves, n_parents, parent_mask, info, offsets, scan_scratch,
                           scan_scratch_bytes, dev_err, stream);
}

static int prune_branch_impl(const LokiPruneLevel* lvl, const double* leaves,
                             int64_t n_parents, const uint8_t* mask, LokiBranchInfo* info,
                             int64_t* offsets, void* scan_scratch, int64_t scan_scratch_bytes,
                             int32_t* dev_err, void* stream) {
  int rc = check_prune(lvl);
  if (rc) return rc;
  if (n_parents < 0) return set_error(LOKI_ERR_INVALID, "n_parents < 0");
  if (!offsets || !dev_err || (n_parents && (!leaves || !info)))
    return set_error(LOKI_ERR_INVALID, "null pointer argument");
  cudaStream_t s = (cudaStream_t)stream;
  if (n_parents > 0) {
    // child counts go to offsets[0..n), scanned in place
    note_launch();
    prune_branch_kernel<<<(unsigned)((n_parents + 255) / 256), 256, 0, s>>>(
        *lvl, leaves, n_parents, info, offsets, dev_err, mask, nullptr);
    rc = check_launch("prune_branch");
    if (rc) return rc;
  }
  return exclusive_scan<false>(offsets, n_parents, 0.0, offsets, scan_scratch,
                               scan_scratch_bytes, s);
}

extern "C" int loki_prune_score(const LokiPruneLevel* lvl, const double* leaves,
                                const float* folds, int64_t n_parents,
                                const LokiBranchInfo* info, const int64_t* offsets,
                                int64_t n_children, const float* fold_segment,
                                const LokiScoreSpec* spec, float* child_scores,
                                int32_t* child_idx, double* child_phase, float* score_minmax,
                                int32_t* dev_err, void* stream) {
  int rc = check_prune(lvl);
  if (rc) return rc;
  rc = prune_spec_check(spec, lvl->nbins);
  if (rc) return rc;
  if (!score_minmax || !dev_err) return set_error(LOKI_ERR_INVALID, "null pointer argument");
  cudaStream_t s = (cudaStream_t)stream;
  unsigned* keys = reinterpret_cast<unsigned*>(score_minmax);  // reused as ordered keys
  note_launch();
  minmax_init_kernel<<<1, 1, 0, s>>>(keys);
  if (n_children > 0) {
    if (!leaves || !folds || !info || !offsets || !fold_segment || !child_scores ||
        !child_idx || !child_phase)
      return set_error(LOKI_ERR_INVALID, "null pointer argument");
    LokiScoreSpec sp = *spec;
    sp.mode = 1;
    const ScoreK SK = make_score_k(sp, lvl->nbins);
    const int smem = score_smem_bytes(lvl->nbins, sp.wmax, kPruneWarps);
    if (smem > 200 * 1024)
      return set_error(LOKI_ERR_UNSUPPORTED, "nbins + wmax too large for pruning");
    if (smem > 48 * 1024 &&
        set_smem_limit(prune_score_kernel, smem) != cudaSuccess)
      return set_error(LOKI_ERR_CUDA, "cudaFuncSetAttribute failed");
    const int64_t blocks = (n_children + kPruneWarps * 32 - 1) / (kPruneWarps * 32);
    if (blocks > 0x7FFFFFFF) return set_error(LOKI_ERR_UNSUPPORTED, "grid too large");
    note_launch();
    prune_score_kernel<<<(unsigned)blocks, kPruneWarps * 32, smem, s>>>(
        *lvl, leaves, folds, n_parents, info, offsets, n_children, fold_segment, sp, SK,
        child_scores, child_idx, child_phase, keys, nullptr, 0, nullptr, nullptr);
  }
  note_launch();
  minmax_finish_kernel<<<1, 1, 0, s>>>(keys, score_minmax);
  return check_launch("prune_score");
}

extern "C" int loki_prune_select(const float* child_scores, int64_t n_children,
                                 double threshold, int64_t* surv_ids, int64_t* n_surv,
                                 void* scan_scratch, int64_t scan_scratch_bytes, void* stream) {
  if (n_children < 0 || !n_surv) return set_error(LOKI_ERR_INVALID, "bad select arguments");
  if (n_children > 0 && (!child_scores || !surv_ids))
    return set_error(LOKI_ERR_INVALID, "null pointer argument");
  cudaStream_t s = (cudaStream_t)stream;
  // positions are scanned into surv_ids' tail-free temp: reuse surv_ids is not
  // possible (scatter reads positions), so positions live in the scratch
  // after the block sums.
  const int64_t sums_bytes = loki_scan_scratch_bytes(n_children);
  const int64_t need = sums_bytes + (n_children + 1) * (int64_t)sizeof(int64_t);
  if (scan_scratch_bytes < need)
    return set_error(LOKI_ERR_CAPACITY, "select scratch needs %lld bytes", (long long)need);
  int64_t* pos = reinterpret_cast<int64_t*>(reinterpret_cast<char*>(scan_scratch) + sums_bytes);
  int rc = exclusive_scan<true>(child_scores, n_children, threshold, pos, scan_scratch,
                                sums_bytes, s);
  if (rc) return rc;
  if (n_children > 0) note_launch();
  if (n_children > 0)
    select_scatter_kernel<<<(unsigned)((n_children + 255) / 256), 256, 0, s>>>(
        child_scores, n_children, threshold, pos, surv_ids, nullptr);
  if (cudaMemcpyAsync(n_surv, pos + n_children, sizeof(int64_t), cudaMemcpyDeviceToDevice, s) !=
      cudaSuccess)
    return set_error(LOKI_ERR_CUDA, "cudaMemcpyAsync failed");
  return check_launch("prune_select");
}

extern "C" int loki_prune_select_overflow(const float* child_scores, const int64_t* offsets,
                                          int64_t n_parents, int64_t batch_size,
                                          double threshold, int64_t capacity,
                                          int64_t* surv_ids, int64_t* n_surv, double* thr_out,
                                          int64_t* scratch_ids, float* scratch_keys,
                                          int64_t scratch_len, void* stream) {
  if (batch_size < 1 || capacity < 1 || n_parents < 0)
    return set_error(LOKI_ERR_INVALID, "bad overflow selection arguments");
  if (!child_scores || !offsets || !surv_ids || !n_surv || !thr_out || !scratch_ids ||
      !scratch_keys)
    return set_error(LOKI_ERR_INVALID, "null pointer argument");
  note_launch();
  select_overflow_kernel<<<1, kSelThreads, 0, (cudaStream_t)stream>>>(
      child_scores, offsets, n_parents, batch_size, threshold, capacity, surv_ids, n_surv,
      thr_out, scratch_ids, reinterpret_cast<unsigned*>(scratch_keys), nullptr, nullptr,
      nullptr, nullptr);
  (void)scratch_len;
  return check_launch("prune_select_overflow");
}

extern "C" int loki_prune_emit(const LokiPruneLevel* lvl, const double* leaves,
                               const float* folds, const LokiBranchInfo* info,
                               const int64_t* offsets, int64_t n_parents,
                               const float* fold_segment, const int64_t* surv_ids,
                               int64_t n_surv, const float* child_scores,
                               const int32_t* child_idx, const double* child_phase,
                               double* leaves_out, float* folds_out, float* scores_out,
                               float* scores_ep_out, int32_t* bt_out, void* stream) {
  int rc = check_prune(lvl);
  if (rc) return rc;
  if (n_surv <= 0) return LOKI_OK;
  if (!leaves || !folds || !info || !offsets || !fold_segment || !surv_ids || !child_scores ||
      !child_idx || !child_phase || !leaves_out || !folds_out || !scores_out ||
      !scores_ep_out || !bt_out)
    return set_error(LOKI_ERR_INVALID, "null pointer argument");
  const int64_t blocks = (n_surv + kPruneWarps * 32 - 1) / (kPruneWarps * 32);
  note_launch();
  prune_emit_kernel<<<(unsigned)blocks, kPruneWarps * 32, 0, (cudaStream_t)stream>>>(
      *lvl, leaves, folds, info, offsets, n_parents, fold_segment, surv_ids, n_surv,
      child_scores, child_idx, child_phase, leaves_out, folds_out, scores_out, scores_ep_out,
      bt_out, nullptr);
  return check_launch("prune_emit");
}

extern "C" int loki_prune_ascend(const LokiPruneLevel* lvl, const double* leaves, float* folds,
                                 float* scores, float* scores_ep, int64_t n, int32_t nseg,
                                 const double* tm_seg, const double* dt_seg,
                                 const int32_t* seg_idx, const float* ffa_fold,
                                 int64_t seg_stride, const LokiScoreSpec* spec,
                                 int32_t* dev_err, void* stream) {
  int rc = check_prune(lvl);
  if (rc) return rc;
  rc = prune_spec_check(spec, lvl->nbins);
  if (rc) return rc;
  if (n <= 0) return LOKI_OK;
  if (nseg < 1 || !leaves || !folds || !scores || !scores_ep || !tm_seg || !dt_seg ||
      !seg_idx || !ffa_fold || !dev_err)
    return set_error(LOKI_ERR_INVALID, "bad ascend arguments");
  LokiScoreSpec sp = *spec;
  sp.mode = 1;
  const ScoreK SK = make_score_k(sp, lvl->nbins);
  const int nb = lvl->nbins;
  const int smem = kPruneWarps * 32 * (2 * nb + score_stride(nb, sp.wmax)) * (int)sizeof(float);
  if (smem > 200 * 1024) return set_error(LOKI_ERR_UNSUPPORTED, "nbins too large for ascend");
  if (smem > 48 * 1024 &&
      set_smem_limit(prune_ascend_kernel, smem) != cudaSuccess)
    return set_error(LOKI_ERR_CUDA, "cudaFuncSetAttribute failed");
  const int64_t blocks = (n + kPruneWarps * 32 - 1) / (kPruneWarps * 32);
  note_launch();
  prune_ascend_kernel<<<(unsigned)blocks, kPruneWarps * 32, smem, (cudaStream_t)stream>>>(
      *lvl, leaves, folds, scores, scores_ep, n, nseg, tm_seg, dt_seg, seg_idx, ffa_fold,
      seg_stride, sp, SK, nullptr);
  return check_launch("prune_ascend");
}

extern "C" int loki_prune_ascend_dev(const LokiPruneLevel* lvl, const double* leaves,
                                     float* folds, float* scores, float* scores_ep,
                                     const int64_t* n_dev, int64_t n_cap, int32_t nseg,
                                     const double* tm_seg, const double* dt_seg,
                                     const int32_t* seg_idx, const float* ffa_fold,
                                     int64_t seg_stride, const LokiScoreSpec* spec,
                                     int32_t* dev_err, void* stream) {
  int rc = check_prune(lvl);
  if (rc) return rc;
  rc = prune_spec_check(spec, lvl->nbins);
  if (rc) return rc;
  if (n_cap < 1 || nseg < 1 || !n_dev || !leaves || !folds || !scores || !scores_ep ||
      !tm_seg || !dt_seg || !seg_idx || !ffa_fold || !dev_err)
    return set_error(LOKI_ERR_INVALID, "bad ascend arguments");
  LokiScoreSpec sp = *spec;
  sp.mode = 1;
  const ScoreK SK = make_score_k(sp, lvl->nbins);
  const int nb = lvl->nbins;
  const int smem = kPruneWarps * 32 * (2 * nb + score_stride(nb, sp.wmax)) * (int)sizeof(float);
  if (smem > 200 * 1024) return set_error(LOKI_ERR_UNSUPPORTED, "nbins too large for ascend");
  if (smem > 48 * 1024 && set_smem_limit(prune_ascend_kernel, smem) != cudaSuccess)
    return set_error(LOKI_ERR_CUDA, "cudaFuncSetAttribute failed");
  int dev = 0, nsm = 0, occ = 0;
  if (cudaGetDevice(&dev) != cudaSuccess ||
      cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess ||
      cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, prune_ascend_kernel,
                                                    kPruneWarps * 32, smem) != cudaSuccess)
    return set_error(LOKI_ERR_CUDA, "occupancy query failed");
  const int64_t need = (n_cap + kPruneWarps * 32 - 1) / (kPruneWarps * 32);
  const unsigned blocks = (unsigned)std::max<int64_t>(
      1, std::min<int64_t>(need, (int64_t)nsm * std::max(1, occ)));
  note_launch();
  prune_ascend_kernel<<<blocks, kPruneWarps * 32, smem, (cudaStream_t)stream>>>(
      *lvl, leaves, folds, scores, scores_ep, 0, nseg, tm_seg, dt_seg, seg_idx, ffa_fold,
      seg_stride, sp, SK, n_dev);
  return check_launch("prune_ascend_dev");
}

// ---- circular-orbit tree --------------------------------------------------

static int check_circ(const LokiPruneLevel* lvl) {
  int rc = check_prune(lvl);
  if (rc) return rc;
  if (lvl->basis != 2 || lvl->poly_order != 5)
    return set_error(LOKI_ERR_INVALID, "the circular tree needs basis 2 and poly_order 5");
  return LOKI_OK;
}

extern "C" int loki_prune_circ_branch(const LokiPruneLevel* lvl, const double* leaves,
                                      int64_t n_parents, LokiBranchInfo* info,
                                      int64_t* keep_off, int64_t* exp_off, void* scan_scratch,
                                      int64_t scan_scratch_bytes, int32_t* dev_err,
                                      void* stream) {
  int rc = check_circ(lvl);
  if (rc) return rc;
  if (n_parents < 0) return set_error(LOKI_ERR_INVALID, "n_parents < 0");
  if (!keep_off || !exp_off || !dev_err || (n_parents && (!leaves || !info)))
    return set_error(LOKI_ERR_INVALID, "null pointer argument");
  cudaStream_t s = (cudaStream_t)stream;
  if (n_parents > 0) {
    note_launch();
    circ_branch_kernel<<<(unsigned)((n_parents + 255) / 256), 256, 0, s>>>(
        *lvl, leaves, n_parents, info, keep_off, exp_off, dev_err, nullptr);
    rc = check_launch("prune_circ_branch");
    if (rc) return rc;
  }
  rc = exclusive_scan<false>(keep_off, n_parents, 0.0, keep_off, scan_scratch,
                             scan_scratch_bytes, s);
  if (rc) return rc;
  return exclusive_scan<false>(exp_off, n_parents, 0.0, exp_off, scan_scratch,
                               scan_scratch_bytes, s);
}

extern "C" int loki_prune_circ_map(const LokiPruneLevel* lvl, const double* leaves,
                                   int64_t n_parents, int64_t batch_size,
                                   const LokiBranchInfo* info, const int64_t* keep_off,
                                   const int64_t* exp_off, void* child_map, float* valid_flags,
                                   void* stream) {
  int rc = check_circ(lvl);
  if (rc) return rc;
  if (batch_size < 1 || n_parents < 0) return set_error(LOKI_ERR_INVALID, "bad batch size");
  if (n_parents == 0) return LOKI_OK;
  if (!leaves || !info || !keep_off || !exp_off || !child_map || !valid_flags)
    return set_error(LOKI_ERR_INVALID, "null pointer argument");
  note_launch();
  circ_map_kernel<<<(unsigned)((n_parents + 255) / 256), 256, 0, (cudaStream_t)stream>>>(
      *lvl, leaves, n_parents, batch_size, info, keep_off, exp_off,
      reinterpret_cast<CircChild*>(child_map), valid_flags, nullptr, 0, nullptr, nullptr);
  return check_launch("prune_circ_map");
}

extern "C" int loki_prune_circ_score(const LokiPruneLevel* lvl, const double* leaves,
                                     const float* folds, int64_t n_parents, int64_t batch_size,
                                     const LokiBranchInfo* info, const void* child_map,
                                     const int64_t* keep_off, const int64_t* exp_off,
                                     const int64_t* valid_ids, int64_t n_valid,
                                     const float* fold_segment, const LokiScoreSpec* spec,
                                     float* child_scores, int32_t* child_idx,
                                     double* child_phase, int8_t* child_class,
                                     int32_t* batch_taylor, int64_t* batch_offsets,
                                     float* score_minmax, int32_t* dev_err, void* stream) {
  int rc = check_circ(lvl);
  if (rc) return rc;
  rc = prune_spec_check(spec, lvl->nbins);
  if (rc) return rc;
  if (batch_size < 1 || n_parents < 0 || n_valid < 0)
    return set_error(LOKI_ERR_INVALID, "bad circular score arguments");
  if (!score_minmax || !dev_err || !batch_taylor || !batch_offsets || !keep_off || !exp_off)
    return set_error(LOKI_ERR_INVALID, "null pointer argument");
  cudaStream_t s = (cudaStream_t)stream;
  const int64_t nbatch = (n_parents + batch_size - 1) / batch_size;
  if (nbatch > 0 && cudaMemsetAsync(batch_taylor, 0, nbatch * sizeof(int32_t), s) != cudaSuccess)
    return set_error(LOKI_ERR_CUDA, "cudaMemsetAsync failed");
  unsigned* keys = reinterpret_cast<unsigned*>(score_minmax);
  note_launch();
  minmax_init_kernel<<<1, 1, 0, s>>>(keys);
  if (n_valid > 0) {
    if (!leaves || !folds || !info || !child_map || !valid_ids || !fold_segment ||
        !child_scores || !child_idx || !child_phase || !child_class)
      return set_error(LOKI_ERR_INVALID, "null pointer argument");
    LokiScoreSpec sp = *spec;
    sp.mode = 1;
    const ScoreK SK = make_score_k(sp, lvl->nbins);
    const int smem = score_smem_bytes(lvl->nbins, sp.wmax, kPruneWarps);
    if (smem > 200 * 1024)
      return set_error(LOKI_ERR_UNSUPPORTED, "nbins + wmax too large for pruning");
    if (smem > 48 * 1024 &&
        set_smem_limit(circ_score_kernel, smem) != cudaSuccess)
      return set_error(LOKI_ERR_CUDA, "cudaFuncSetAttribute failed");
    const int64_t blocks = (n_valid + kPruneWarps * 32 - 1) / (kPruneWarps * 32);
    if (blocks > 0x7FFFFFFF) return set_error(LOKI_ERR_UNSUPPORTED, "grid too large");
    note_launch();
    circ_score_kernel<<<(unsigned)blocks, kPruneWarps * 32, smem, s>>>(
        *lvl, leaves, folds, batch_size, info, reinterpret_cast<const CircChild*>(child_map),
        valid_ids, n_valid, fold_segment, sp, SK, child_scores, child_idx, child_phase,
        child_class, batch_taylor, keys, nullptr, nullptr, nullptr);
  }
  note_launch();
  minmax_finish_kernel<<<1, 1, 0, s>>>(keys, score_minmax);
  note_launch();
  circ_boff_kernel<<<(unsigned)((n_parents + 1 + 255) / 256), 256, 0, s>>>(
      keep_off, exp_off, n_parents, valid_ids, n_valid, batch_offsets, nullptr);
  return check_launch("prune_circ_score");
}

extern "C" int loki_prune_circ_emit(const LokiPruneLevel* lvl, const double* leaves,
                                    const float* folds, int64_t batch_size,
                                    const LokiBranchInfo* info, const void* child_map,
                                    const int64_t* valid_ids, const float* fold_segment,
                                    const int64_t* surv_ids, int64_t n_surv,
                                    const float* child_scores, const int32_t* child_idx,
                                    const double* child_phase, const int8_t* child_class,
                                    const int32_t* batch_taylor, double* leaves_out,
                                    float* folds_out, float* scores_out, float* scores_ep_out,
                                    int32_t* bt_out, void* stream) {
  int rc = check_circ(lvl);
  if (rc) return rc;
  if (n_surv <= 0) return LOKI_OK;
  if (batch_size < 1) return set_error(LOKI_ERR_INVALID, "bad batch size");
  if (!leaves || !folds || !info || !child_map || !valid_ids || !fold_segment || !surv_ids ||
      !child_scores || !child_idx || !child_phase || !child_class || !batch_taylor ||
      !leaves_out || !folds_out || !scores_out || !scores_ep_out || !bt_out)
    return set_error(LOKI_ERR_INVALID, "null pointer argument");
  const int64_t blocks = (n_surv + kPruneWarps * 32 - 1) / (kPruneWarps * 32);
  note_launch();
  circ_emit_kernel<<<(unsigned)blocks, kPruneWarps * 32, 0, (cudaStream_t)stream>>>(
      *lvl, leaves, folds, batch_size, info, reinterpret_cast<const CircChild*>(child_map),
      valid_ids, fold_segment, surv_ids, n_surv, child_scores, child_idx, child_phase,
      child_class, batch_taylor, leaves_out, folds_out, scores_out, scores_ep_out, bt_out,
      nullptr);
  return check_launch("prune_circ_emit");
}

static int cplx_smem(const LokiPruneLevel* lvl, const LokiScoreSpec& sp, int* smem);

extern "C" int loki_prune_circ_score_complex(
    const LokiPruneLevel* lvl, const double* leaves, const void* folds, int64_t n_parents,
    int64_t batch_size, const LokiBranchInfo* info, const void* child_map,
    const int64_t* keep_off, const int64_t* exp_off, const int64_t* valid_ids, int64_t n_valid,
    const void* fold_segment, const LokiScoreSpec* spec, float* child_scores,
    int32_t* child_idx, double* child_phase, int8_t* child_class, int32_t* batch_taylor,
    int64_t* batch_offsets, float* score_minmax, int32_t* dev_err, void* stream) {
  int rc = check_circ(lvl);
  if (rc) return rc;
  rc = prune_spec_check(spec, lvl->nbins);
  if (rc) return rc;
  if (batch_size < 1 || n_parents < 0 || n_valid < 0)
    return set_error(LOKI_ERR_INVALID, "bad circular score arguments");
  if (!score_minmax || !dev_err || !batch_taylor || !batch_offsets || !keep_off || !exp_off)
    return set_error(LOKI_ERR_INVALID, "null pointer argument");
  cudaStream_t s = (cudaStream_t)stream;
  const int64_t nbatch = (n_parents + batch_size - 1) / batch_size;
  if (nbatch > 0 && cudaMemsetAsync(batch_taylor, 0, nbatch * sizeof(int32_t), s) != cudaSuccess)
    return set_error(LOKI_ERR_CUDA, "cudaMemsetAsync failed");
  unsigned* keys = reinterpret_cast<unsigned*>(score_minmax);
  note_launch();
  minmax_init_kernel<<<1, 1, 0, s>>>(keys);
  if (n_valid > 0) {
    if (!leaves || !folds || !info || !child_map || !valid_ids || !fold_segment ||
        !child_scores || !child_idx || !child_phase || !child_class)
      return set_error(LOKI_ERR_INVALID, "null pointer argument");
    LokiScoreSpec sp = *spec;
    sp.mode = 1;
    const ScoreK SK = make_score_k(sp, lvl->nbins);
    int smem = 0;
    rc = cplx_smem(lvl, sp, &smem);
    if (rc) return rc;
    if (smem > 48 * 1024 &&
        set_smem_limit(circ_score_complex_kernel, smem) != cudaSuccess)
      return set_error(LOKI_ERR_CUDA, "cudaFuncSetAttribute failed");
    const int64_t blocks = (n_valid + kPruneWarps * 32 - 1) / (kPruneWarps * 32);
    if (blocks > 0x7FFFFFFF) return set_error(LOKI_ERR_UNSUPPORTED, "grid too large");
    note_launch();
    circ_score_complex_kernel<<<(unsigned)blocks, kPruneWarps * 32, smem, s>>>(
        *lvl, leaves, static_cast<const float2*>(folds), batch_size, info,
        reinterpret_cast<const CircChild*>(child_map), valid_ids, n_valid,
        static_cast<const float2*>(fold_segment), sp, SK, child_scores, child_idx,
        child_phase, child_class, batch_taylor, keys);
  }
  note_launch();
  minmax_finish_kernel<<<1, 1, 0, s>>>(keys, score_minmax);
  note_launch();
  circ_boff_kernel<<<(unsigned)((n_parents + 1 + 255) / 256), 256, 0, s>>>(
      keep_off, exp_off, n_parents, valid_ids, n_valid, batch_offsets, nullptr);
  return check_launch("prune_circ_score_complex");
}

extern "C" int loki_prune_circ_emit_complex(
    const LokiPruneLevel* lvl, const double* leaves, const void* folds, int64_t batch_size,
    const LokiBranchInfo* info, const void* child_map, const int64_t* valid_ids,
    const void* fold_segment, const int64_t* surv_ids, int64_t n_surv,
    const float* child_scores, const int32_t* child_idx, const double* child_phase,
    const int8_t* child_class, const int32_t* batch_taylor, double* leaves_out,
    void* folds_out, float* scores_out, float* scores_ep_out, int32_t* bt_out, void* stream) {
  int rc = check_circ(lvl);
  if (rc) return rc;
  if (lvl->nbins % 2) return set_error(LOKI_ERR_INVALID, "complex folds need an even nbins");
  if (n_surv <= 0) return LOKI_OK;
  if (batch_size < 1) return set_error(LOKI_ERR_INVALID, "bad batch size");
  if (!leaves || !folds || !info || !child_map || !valid_ids || !fold_segment || !surv_ids ||
      !child_scores || !child_idx || !child_phase || !child_class || !batch_taylor ||
      !leaves_out || !folds_out || !scores_out || !scores_ep_out || !bt_out)
    return set_error(LOKI_ERR_INVALID, "null pointer argument");
  note_launch();
  circ_emit_complex_kernel<<<(unsigned)((n_surv + 127) / 128), 128, 0, (cudaStream_t)stream>>>(
      *lvl, leaves, static_cast<const float2*>(folds), batch_size, info,
      reinterpret_cast<const CircChild*>(child_map), valid_ids,
      static_cast<const float2*>(fold_segment), surv_ids, n_surv, child_scores, child_idx,
      child_phase, child_class, batch_taylor, leaves_out, static_cast<float2*>(folds_out),
      scores_out, scores_ep_out, bt_out);
  return check_launch("prune_circ_emit_complex");
}

// ---- complex (Fourier) folds -----------------------------------------------

static int cplx_smem(const LokiPruneLevel* lvl, const LokiScoreSpec& sp, int* smem) {
  if (lvl->nbins % 2) return set_error(LOKI_ERR_INVALID, "complex folds need an even nbins");
  const size_t bytes = ((size_t)2 * lvl->nbins +
                        kPruneWarps * cplx_warp_floats(lvl->nbins,
                                                       score_stride(lvl->nbins, sp.wmax))) *
                       sizeof(float);
  if (bytes > 200 * 1024)
    return set_error(LOKI_ERR_UNSUPPORTED, "nbins too large for complex pruning");
  *smem = (int)bytes;
  return LOKI_OK;
}

extern "C" int loki_prune_score_complex(const LokiPruneLevel* lvl, const double* leaves,
                                        const void* folds, int64_t n_parents,
                                        const LokiBranchInfo* info, const int64_t* offsets,
                                        int64_t n_children, const void* fold_segment,
                                        const LokiScoreSpec* spec, float* child_scores,
                                        int32_t* child_idx, double* child_phase,
                                        float* score_minmax, int32_t* dev_err, void* stream) {
  int rc = check_prune(lvl);
  if (rc) return rc;
  rc = prune_spec_check(spec, lvl->nbins);
  if (rc) return rc;
  if (!score_minmax || !dev_err) return set_error(LOKI_ERR_INVALID, "null pointer argument");
  cudaStream_t s = (cudaStream_t)stream;
  unsigned* keys = reinterpret_cast<unsigned*>(score_minmax);
  note_launch();
  minmax_init_kernel<<<1, 1, 0, s>>>(keys);
  if (n_children > 0) {
    if (!leaves || !folds || !info || !offsets || !fold_segment || !child_scores ||
        !child_idx || !child_phase)
      return set_error(LOKI_ERR_INVALID, "null pointer argument");
    LokiScoreSpec sp = *spec;
    sp.mode = 1;
    const ScoreK SK = make_score_k(sp, lvl->nbins);
    int smem = 0;
    rc = cplx_smem(lvl, sp, &smem);
    if (rc) return rc;
    if (set_smem_limit(prune_score_complex_kernel, smem) != cudaSuccess)
      return set_error(LOKI_ERR_CUDA, "cudaFuncSetAttribute failed");
    const int64_t blocks = (n_children + kPruneWarps * 32 - 1) / (kPruneWarps * 32);
    if (blocks > 0x7FFFFFFF) return set_error(LOKI_ERR_UNSUPPORTED, "grid too large");
    note_launch();
    prune_score_complex_kernel<<<(unsigned)blocks, kPruneWarps * 32, smem, s>>>(
        *lvl, leaves, reinterpret_cast<const float2*>(folds), n_parents, info, offsets,
        n_children, reinterpret_cast<const float2*>(fold_segment), sp, SK, child_scores,
        child_idx, child_phase, keys);
  }
  note_launch();
  minmax_finish_kernel<<<1, 1, 0, s>>>(keys, score_minmax);
  return check_launch("prune_score_complex");
}

extern "C" int loki_prune_emit_complex(const LokiPruneLevel* lvl, const double* leaves,
                                       const void* folds, const LokiBranchInfo* info,
                                       const int64_t* offsets, int64_t n_parents,
                                       const void* fold_segment, const int64_t* surv_ids,
                                       int64_t n_surv, const float* child_scores,
                                       const int32_t* child_idx, const double* child_phase,
                                       double* leaves_out, void* folds_out, float* scores_out,
                                       float* scores_ep_out, int32_t* bt_out, void* stream) {
  int rc = check_prune(lvl);
  if (rc) return rc;
  if (n_surv <= 0) return LOKI_OK;
  if (!leaves || !folds || !info || !offsets || !fold_segment || !surv_ids || !child_scores ||
      !child_idx || !child_phase || !leaves_out || !folds_out || !scores_out ||
      !scores_ep_out || !bt_out)
    return set_error(LOKI_ERR_INVALID, "null pointer argument");
  note_launch();
  prune_emit_complex_kernel<<<(unsigned)((n_surv + 127) / 128), 128, 0, (cudaStream_t)stream>>>(
      *lvl, leaves, reinterpret_cast<const float2*>(folds), info, offsets, n_parents,
      reinterpret_cast<const float2*>(fold_segment), surv_ids, n_surv, child_scores, child_idx,
      child_phase, leaves_out, reinterpret_cast<float2*>(folds_out), scores_out, scores_ep_out,
      bt_out);
  return check_launch("prune_emit_complex");
}

extern "C" int loki_prune_ascend_complex(const LokiPruneLevel* lvl, const double* leaves,
                                         void* folds, float* scores, float* scores_ep,
                                         int64_t n, int32_t nseg, const double* tm_seg,
                                         const double* dt_seg, const int32_t* seg_idx,
                                         const void* ffa_fold, int64_t seg_stride,
                                         const LokiScoreSpec* spec, int32_t* dev_err,
                                         void* stream) {
  int rc = check_prune(lvl);
  if (rc) return rc;
  rc = prune_spec_check(spec, lvl->nbins);
  if (rc) return rc;
  if (n <= 0) return LOKI_OK;
  if (nseg < 1 || !leaves || !folds || !scores || !scores_ep || !tm_seg || !dt_seg ||
      !seg_idx || !ffa_fold || !dev_err)
    return set_error(LOKI_ERR_INVALID, "bad ascend arguments");
  LokiScoreSpec sp = *spec;
  sp.mode = 1;
  const ScoreK SK = make_score_k(sp, lvl->nbins);
  int smem = 0;
  rc = cplx_smem(lvl, sp, &smem);
  if (rc) return rc;
  if (set_smem_limit(prune_ascend_complex_kernel, smem) != cudaSuccess)
    return set_error(LOKI_ERR_CUDA, "cudaFuncSetAttribute failed");
  const int64_t blocks = (n + kPruneWarps * 32 - 1) / (kPruneWarps * 32);
  note_launch();
  prune_ascend_complex_kernel<<<(unsigned)blocks, kPruneWarps * 32, smem,
                                (cudaStream_t)stream>>>(
      *lvl, leaves, reinterpret_cast<float2*>(folds), scores, scores_ep, n, nseg, tm_seg, dt_seg,
      seg_idx, reinterpret_cast<const float2*>(ffa_fold), seg_stride, sp, SK);
  return check_launch("prune_ascend_complex");
}

// ---------------------------------------------------------------------------
// device-resident run: every level of one reference segment with the counts
// kept on the device (counts[0] parents, [1] children, [2] survivors)
// ---------------------------------------------------------------------------

namespace loki {

__global__ void run_seed_kernel(int64_t* cnt, int64_t n, unsigned* keys) {
  cnt[0] = n;
  for (int k = 1; k < 8; ++k) cnt[k] = 0;
  keys[0] = 0xFFFFFFFFu;  // score min / max keys of the first level
  keys[1] = 0u;
}

__global__ void run_level_end_kernel(int64_t* cnt, unsigned* keys, int32_t* ovf_flag,
                                     LokiPruneLevelStats* st) {
  level_end(cnt, keys, ovf_flag, st);
}

// survivors' backtracks appended to the history at row counts[3]
__global__ void run_bt_copy_kernel(const int32_t* __restrict__ bt, const int64_t* cnt, int row,
                                   int32_t* __restrict__ hist, int64_t hist_rows,
                                   int32_t* err) {
  const int64_t start = cnt[3], rows = cnt[2];
  if (start + rows > hist_rows) {
    if (blockIdx.x == 0 && threadIdx.x == 0) atomicOr(err, LOKI_DEVERR_CAPACITY);
    return;
  }
  int32_t* out = hist + start * row;
  const int64_t n = rows * row;
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n;
       i += (int64_t)gridDim.x * blockDim.x)
    out[i] = bt[i];
}

}  // namespace loki

// One circular-orbit level with device counts (counts[4] = valid children):
// branch (kept and crackle-expanded children per parent), the two scans, the
// batch-ordered child map, validation compaction, resolve + score, batch
// offsets of the valid children, selection with the overflow rule, emit.
static int circ_level_dev(const LokiPruneLevel& D, const LokiPruneTree& in,
                          const LokiPruneTree& out, const LokiPruneWork& w,
                          const LokiPruneRun* run, const float* seg, double thr,
                          const LokiScoreSpec& sp, const ScoreK& SK, int smem, int64_t max_sugg,
                          int64_t batch, unsigned g_par, unsigned g_flat, unsigned g_score,
                          unsigned g_emit, int scan_grid, int64_t* cnt, int64_t* pos,
                          int64_t sums_bytes, unsigned* keys, LokiPruneLevelStats* st,
                          int32_t* dev_err, cudaStream_t s) {
  LokiBranchInfo* info = reinterpret_cast<LokiBranchInfo*>(w.info);
  CircChild* map = reinterpret_cast<CircChild*>(run->child_map);
  note_launch();
  circ_branch_kernel<<<g_par, 256, 0, s>>>(D, in.leaves, 0, info, w.offsets, run->exp_off,
                                           dev_err, cnt);
  int rc = exclusive_scan_dev<false>(w.offsets, w.par_cap, cnt, 0.0, w.offsets, w.scan,
                                     w.scan_bytes, scan_grid, s);
  if (rc) return rc;
  rc = exclusive_scan_dev<false>(run->exp_off, w.par_cap, cnt, 0.0, run->exp_off, w.scan,
                                 w.scan_bytes, scan_grid, s);
  if (rc) return rc;
  note_launch();
  circ_map_kernel<<<g_par, 256, 0, s>>>(D, in.leaves, 0, batch, info, w.offsets, run->exp_off,
                                        map, run->valid_flags, cnt, w.child_cap, st, dev_err);
  // validation compaction: valid flags are 1.0 / 0.0
  rc = exclusive_scan_dev<true>(run->valid_flags, w.child_cap, cnt + 1, 0.5, pos, w.sscan,
                                sums_bytes, scan_grid, s);
  if (rc) return rc;
  for (int i = 0; i < 3; ++i) note_launch();
  select_scatter_kernel<<<g_flat, 256, 0, s>>>(run->valid_flags, 0, 0.5, pos, run->valid_ids,
                                               cnt + 1);
  if (cudaMemsetAsync(run->batch_taylor, 0,
                      (size_t)(w.par_cap / batch + 1) * sizeof(int32_t), s) != cudaSuccess)
    return set_error(LOKI_ERR_CUDA, "cudaMemsetAsync failed");
  circ_score_kernel<<<g_score, kPruneWarps * 32, smem, s>>>(
      D, in.leaves, in.folds, batch, info, map, run->valid_ids, 0, seg, sp, SK, w.child_scores,
      w.child_idx, w.child_phase, run->child_class, run->batch_taylor, keys, cnt, pos, st);
  circ_boff_kernel<<<g_par, 256, 0, s>>>(w.offsets, run->exp_off, 0, run->valid_ids, 0,
                                         run->batch_offsets, cnt);
  rc = exclusive_scan_dev<true>(w.child_scores, w.child_cap, cnt + 4, thr, pos, w.sscan,
                                sums_bytes, scan_grid, s);
  if (rc) return rc;
  for (int i = 0; i < 3; ++i) note_launch();
  select_scatter_kernel<<<g_flat, 256, 0, s>>>(w.child_scores, 0, thr, pos, w.surv, cnt + 4);
  select_overflow_kernel<<<1, kSelThreads, 0, s>>>(
      w.child_scores, run->batch_offsets, 0, batch, thr, max_sugg, w.surv, cnt + 2, w.ovf_thr,
      w.ovf_ids, reinterpret_cast<unsigned*>(w.ovf_keys), cnt, run->ovf_flag, pos, cnt + 4);
  circ_emit_kernel<<<g_emit, kPruneWarps * 32, 0, s>>>(
      D, in.leaves, in.folds, batch, info, map, run->valid_ids, seg, w.surv, 0, w.child_scores,
      w.child_idx, w.child_phase, run->child_class, run->batch_taylor, out.leaves, out.folds,
      out.scores, out.scores_ep, out.backtracks, cnt);
  return LOKI_OK;
}

extern "C" int loki_prune_run(const LokiPruneLevel* lvls, int32_t nlevels, const float* ffa_folds,
                              int64_t seg_stride, const int32_t* seg_idx,
                              const double* thresholds, const LokiScoreSpec* spec,
                              int64_t seed_n, int64_t max_sugg, int64_t batch_size,
                              const LokiPruneRun* run, int32_t* dev_err, void* stream) {
  if (!lvls || nlevels < 1 || !ffa_folds || !seg_idx || !thresholds || !spec || !run ||
      !dev_err)
    return set_error(LOKI_ERR_INVALID, "null pointer or no level");
  if (max_sugg < 1 || batch_size < 1 || seed_n < 0 || seed_n > max_sugg || seg_stride < 1)
    return set_error(LOKI_ERR_INVALID, "bad sizes");
  const LokiPruneWork& w = run->work;
  const LokiPruneTree* tr = run->trees;
  if (tr[0].cap < max_sugg || tr[1].cap < max_sugg || w.par_cap < max_sugg || w.child_cap < 1 ||
      w.ovf_cap < max_sugg + w.child_cap + 1)
    return set_error(LOKI_ERR_CAPACITY, "run workspace below max_sugg / child_cap");
  if (!run->counts || !run->ovf_flag || !run->stats || !w.info || !w.offsets || !w.scan ||
      !w.child_scores || !w.child_idx || !w.child_phase || !w.surv || !w.sscan || !w.minmax ||
      !w.ovf_ids || !w.ovf_keys || !w.ovf_thr)
    return set_error(LOKI_ERR_INVALID, "null workspace pointer");
  for (int l = 0; l < nlevels; ++l) {
    int rc = check_prune(&lvls[l]);
    if (rc) return rc;
    if (lvls[l].basis != lvls[0].basis || lvls[l].poly_order != lvls[0].poly_order ||
        lvls[l].nbins != lvls[0].nbins)
      return set_error(LOKI_ERR_INVALID, "levels of different trees");
  }
  const bool circ = lvls[0].basis == 2;
  if (circ && (lvls[0].poly_order != 5 || !run->exp_off || !run->child_map ||
               !run->valid_flags || !run->valid_ids || !run->child_class ||
               !run->batch_taylor || !run->batch_offsets))
    return set_error(LOKI_ERR_INVALID, "the circular-orbit tree needs poly_order 5 and its "
                                       "workspace");
  int rc = prune_spec_check(spec, lvls[0].nbins);
  if (rc) return rc;
  const int64_t sums_bytes = loki_scan_scratch_bytes(w.child_cap);
  if (w.scan_bytes < loki_scan_scratch_bytes(w.par_cap + 1) ||
      w.sscan_bytes < sums_bytes + (w.child_cap + 1) * (int64_t)sizeof(int64_t))
    return set_error(LOKI_ERR_CAPACITY, "scan scratch below par_cap / child_cap");
  cudaStream_t s = (cudaStream_t)stream;
  const int nb = lvls[0].nbins, P = lvls[0].poly_order;
  LokiScoreSpec sp = *spec;
  sp.mode = 1;
  const ScoreK SK = make_score_k(sp, nb);
  const int smem = score_smem_bytes(nb, sp.wmax, kPruneWarps);
  if (smem > 200 * 1024)
    return set_error(LOKI_ERR_UNSUPPORTED, "nbins + wmax too large for pruning");
  if (smem > 48 * 1024 && (set_smem_limit(prune_score_kernel, smem) != cudaSuccess ||
                           set_smem_limit(circ_score_kernel, smem) != cudaSuccess))
    return set_error(LOKI_ERR_CUDA, "cudaFuncSetAttribute failed");
  int dev = 0, nsm = 0, occ_s = 0, occ_e = 0;
  if (cudaGetDevice(&dev) != cudaSuccess ||
      cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess ||
      (circ ? cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ_s, circ_score_kernel,
                                                            kPruneWarps * 32, smem)
            : cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ_s, prune_score_kernel,
                                                            kPruneWarps * 32, smem)) !=
          cudaSuccess ||
      (circ ? cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ_e, circ_emit_kernel,
                                                            kPruneWarps * 32, 0)
            : cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ_e, prune_emit_kernel,
                                                            kPruneWarps * 32, 0)) !=
          cudaSuccess)
    return set_error(LOKI_ERR_CUDA, "occupancy query failed");
  // grids: one full wave of the score / emit kernels, and enough blocks for
  // the parent-sized and child-sized passes to stride through
  const unsigned g_score = (unsigned)std::max(1, nsm * std::max(1, occ_s));
  const unsigned g_emit = (unsigned)std::max(1, nsm * std::max(1, occ_e));
  const unsigned g_par = (unsigned)std::min<int64_t>((w.par_cap + 255) / 256, 8 * nsm);
  const unsigned g_flat = (unsigned)(4 * nsm);
  const int scan_grid = 2 * nsm;
  int64_t* cnt = run->counts;
  int64_t* pos = reinterpret_cast<int64_t*>(reinterpret_cast<char*>(w.sscan) + sums_bytes);
  unsigned* keys = reinterpret_cast<unsigned*>(w.minmax);
  const int row_bt = P + 2, row_leaf = (P + 2) * 2;
  note_launch();
  run_seed_kernel<<<1, 1, 0, s>>>(cnt, seed_n, keys);
  for (int l = 1; l <= nlevels; ++l) {
    const LokiPruneLevel& D = lvls[l - 1];
    const LokiPruneTree& in = tr[(l - 1) & 1];
    const LokiPruneTree& out = tr[l & 1];
    const float* seg = ffa_folds + (int64_t)seg_idx[l - 1] * seg_stride;
    const double thr = thresholds[l - 1];
    LokiPruneLevelStats* st = run->stats + (l - 1);
    LokiBranchInfo* info = reinterpret_cast<LokiBranchInfo*>(w.info);
    if (circ) {
      rc = circ_level_dev(D, in, out, w, run, seg, thr, sp, SK, smem, max_sugg, batch_size,
                          g_par, g_flat, g_score, g_emit, scan_grid, cnt, pos, sums_bytes, keys,
                          st, dev_err, s);
      if (rc) return rc;
    } else {
    note_launch();
    prune_branch_kernel<<<g_par, 256, 0, s>>>(D, in.leaves, w.par_cap, info, w.offsets, dev_err,
                                              nullptr, cnt);
    rc = exclusive_scan_dev<false>(w.offsets, w.par_cap, cnt, 0.0, w.offsets, w.scan,
                                   w.scan_bytes, scan_grid, s);
    if (rc) return rc;
    note_launch();
    prune_score_kernel<<<g_score, kPruneWarps * 32, smem, s>>>(
        D, in.leaves, in.folds, 0, info, w.offsets, 0, seg, sp, SK, w.child_scores, w.child_idx,
        w.child_phase, keys, cnt, w.child_cap, st, dev_err);
    rc = exclusive_scan_dev<true>(w.child_scores, w.child_cap, cnt + 1, thr, pos, w.sscan,
                                  sums_bytes, scan_grid, s);
    if (rc) return rc;
    for (int i = 0; i < 3; ++i) note_launch();
    select_scatter_kernel<<<g_flat, 256, 0, s>>>(w.child_scores, 0, thr, pos, w.surv, cnt + 1);
    select_overflow_kernel<<<1, kSelThreads, 0, s>>>(
        w.child_scores, w.offsets, 0, batch_size, thr, max_sugg, w.surv, cnt + 2, w.ovf_thr,
        w.ovf_ids, reinterpret_cast<unsigned*>(w.ovf_keys), cnt, run->ovf_flag, pos, cnt + 1);
    prune_emit_kernel<<<g_emit, kPruneWarps * 32, 0, s>>>(
        D, in.leaves, in.folds, info, w.offsets, 0, seg, w.surv, 0, w.child_scores, w.child_idx,
        w.child_phase, out.leaves, out.folds, out.scores, out.scores_ep, out.backtracks, cnt);
    }
    if (run->bt_hist) {  // before the level end moves the counters on
      note_launch();
      run_bt_copy_kernel<<<g_flat, 256, 0, s>>>(out.backtracks, cnt, row_bt, run->bt_hist,
                                                run->bt_rows, dev_err);
    }
    note_launch();
    if (run->best_leaves && run->best_scores) {  // best leaf, then the level end
      prune_best_kernel<<<1, 1024, 0, s>>>(out.scores, 0, out.leaves, row_leaf,
                                           run->best_leaves + (int64_t)(l - 1) * row_leaf,
                                           run->best_scores + (l - 1), cnt, keys,
                                           run->ovf_flag, st);
    } else {
      run_level_end_kernel<<<1, 1, 0, s>>>(cnt, keys, run->ovf_flag, st);
    }
    rc = check_launch("prune_run");
    if (rc) return rc;
  }
  return LOKI_OK;
}

// ---------------------------------------------------------------------------
// block-per-run driver: one thread block runs every level of one job (a
// reference segment of a fold) with block barriers between the steps, so a
// batch of jobs is one launch instead of ~13 dependent launches per level
// and job. The steps are those of loki_prune_run (Taylor and Chebyshev
// trees): branch, scan, score, select (with the overflow rule), emit,
// backtrack history, best leaf and level record.
// ---------------------------------------------------------------------------

namespace loki {

constexpr int kRunThreads = 512;  // 16 warps a job

// Exclusive scan of in[0..n) (int64 counts, or score >= thr flags) into
// out[0..n), out[n] = total, by one block; in may be out. Returns the total.
template <bool FLAGS>
__device__ int64_t block_scan64(const void* in, int64_t n, double thr, int64_t* out,
                                int64_t* warp_tot) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
  int64_t carry = 0;
  for (int64_t base = 0; base < n; base += blockDim.x) {
    const int64_t i = base + threadIdx.x;
    const int64_t x = scan_in<FLAGS>(in, i, n, thr);
    int64_t v = x;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int64_t y = __shfl_up_sync(0xFFFFFFFFu, v, o);
      if (lane >= o) v += y;
    }
    if (lane == 31) warp_tot[warp] = v;
    __syncthreads();
    if (warp == 0) {
      int64_t w = lane < nw ? warp_tot[lane] : 0;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int64_t y = __shfl_up_sync(0xFFFFFFFFu, w, o);
        if (lane >= o) w += y;
      }
      warp_tot[lane] = w;  // inclusive over warps
    }
    __syncthreads();
    const int64_t incl = v + (warp ? warp_tot[warp - 1] : 0);
    if (i < n) out[i] = carry + incl - x;
    carry += warp_tot[nw - 1];
    __syncthreads();  // warp_tot is rewritten by the next tile
  }
  if (threadIdx.x == 0) out[n] = carry;
  __syncthreads();
  return carry;
}

__global__ void __launch_bounds__(kRunThreads, 1)
prune_block_run_kernel(const LokiPruneJob* __restrict__ jobs,
                       const LokiPruneLevel* __restrict__ levels,
                       const int32_t* __restrict__ seg_idx, const double* __restrict__ thr_all,
                       int32_t nlevels, LokiScoreSpec sp, ScoreK SK, int64_t max_sugg,
                       int64_t batch) {
  extern __shared__ float tiles[];
  __shared__ int64_t warp_tot[32];
  __shared__ int64_t n_sh;
  const LokiPruneJob& J = jobs[blockIdx.x];
  const LokiPruneRun& R = J.run;
  const LokiPruneWork& w = R.work;
  const int tid = threadIdx.x, warp = tid >> 5, nwarps = blockDim.x >> 5;
  float* tile = tiles + (size_t)warp * 32 * score_stride(levels[0].nbins, sp.wmax);
  int64_t* cnt = R.counts;
  unsigned* keys = reinterpret_cast<unsigned*>(w.minmax);
  LokiBranchInfo* info = reinterpret_cast<LokiBranchInfo*>(w.info);
  // selection positions after the scan sums, as loki_prune_run places them
  const int64_t sums_bytes = (int64_t)max((int64_t)1, (w.child_cap + kScanBlock - 1) / kScanBlock) * 8;
  int64_t* pos = reinterpret_cast<int64_t*>(reinterpret_cast<char*>(w.sscan) + sums_bytes);
  const int P = levels[0].poly_order;
  const int row_bt = P + 2, row_leaf = (P + 2) * 2;
  if (tid == 0) {
    cnt[0] = J.seed_n;
    for (int k = 1; k < 8; ++k) cnt[k] = 0;
    keys[0] = 0xFFFFFFFFu;
    keys[1] = 0u;
    *R.ovf_flag = 0;
  }
  __syncthreads();
  int64_t n_par = J.seed_n;
  for (int l = 1; l <= nlevels; ++l) {
    const LokiPruneLevel& D = levels[(size_t)blockIdx.x * nlevels + (l - 1)];
    const LokiPruneTree& in = R.trees[(l - 1) & 1];
    const LokiPruneTree& out = R.trees[l & 1];
    const float* seg = J.ffa_fold + (int64_t)seg_idx[(size_t)blockIdx.x * nlevels + (l - 1)] *
                                        J.seg_stride;
    const double thr = thr_all[(size_t)blockIdx.x * nlevels + (l - 1)];
    LokiPruneLevelStats* st = R.stats + (l - 1);
    // branch and the child offsets
    for (int64_t i = tid; i < n_par; i += blockDim.x)
      branch_one(D, in.leaves, i, info, w.offsets, J.dev_err, nullptr, branch_floats(D));
    __syncthreads();
    const int64_t total = block_scan64<false>(w.offsets, n_par, 0.0, w.offsets, warp_tot);
    const int64_t n_child = total > w.child_cap ? 0 : total;
    if (tid == 0) {
      cnt[1] = n_child;
      st->n_parents = n_par;
      st->n_children = total;
      st->n_valid = total;
      if (total > w.child_cap) atomicOr(J.dev_err, LOKI_DEVERR_CAPACITY);
    }
    // score every child
    for (int64_t t = warp; t * 32 < n_child; t += nwarps) {
      score_tile(D, in.leaves, in.folds, n_par, info, w.offsets, n_child, seg, sp, SK,
                 w.child_scores, w.child_idx, w.child_phase, keys, tile, t * 32);
      __syncwarp();  // the tile rows are rewritten by the next tile
    }
    __syncthreads();
    // select: survivors in order, then the overflow rule when they exceed max_sugg
    const int64_t n_sel = block_scan64<true>(w.child_scores, n_child, thr, pos, warp_tot);
    for (int64_t i = tid; i < n_child; i += blockDim.x)
      if ((double)w.child_scores[i] >= thr) w.surv[pos[i]] = i;
    if (tid == 0) n_sh = n_sel;
    __syncthreads();
    if (n_sel > max_sugg) {  // uniform over the block
      if (tid == 0) *R.ovf_flag = 1;
      select_overflow_block(w.child_scores, w.offsets, n_par, batch, thr, max_sugg, w.surv,
                            &n_sh, w.ovf_thr, w.ovf_ids, reinterpret_cast<unsigned*>(w.ovf_keys));
    }
    const int64_t n_surv = n_sh;
    // the next tree
    for (int64_t t = warp; t * 32 < n_surv; t += nwarps)
      emit_tile(D, in.leaves, in.folds, info, w.offsets, n_par, seg, w.surv, n_surv,
                w.child_scores, w.child_idx, w.child_phase, out.leaves, out.folds, out.scores,
                out.scores_ep, out.backtracks, t * 32);
    __syncthreads();
    // backtrack history, best leaf, level record
    if (R.bt_hist) {
      const int64_t start = cnt[3];
      if (start + n_surv > R.bt_rows) {
        if (tid == 0) atomicOr(J.dev_err, LOKI_DEVERR_CAPACITY);
      } else {
        int32_t* h = R.bt_hist + start * row_bt;
        for (int64_t i = tid; i < n_surv * row_bt; i += blockDim.x) h[i] = out.backtracks[i];
      }
    }
    if (R.best_leaves && R.best_scores)
      block_best(out.scores, n_surv, out.leaves, row_leaf,
                 R.best_leaves + (int64_t)(l - 1) * row_leaf, R.best_scores + (l - 1));
    __syncthreads();
    if (tid == 0) {
      cnt[2] = n_surv;
      level_end(cnt, keys, R.ovf_flag, st);
    }
    __syncthreads();
    n_par = n_surv;
  }
}

}  // namespace loki

extern "C" int64_t loki_prune_run_blocks_scratch_bytes(int32_t njobs, int32_t nlevels) {
  if (njobs < 1 || nlevels < 1) return 0;
  const int64_t nl = (int64_t)njobs * nlevels;
  return ((int64_t)njobs * sizeof(LokiPruneJob) + 255) / 256 * 256 +
         (nl * (int64_t)sizeof(LokiPruneLevel) + 255) / 256 * 256 +
         (nl * 4 + 255) / 256 * 256 + nl * 8;
}

extern "C" int loki_prune_run_blocks(const LokiPruneJob* jobs, int32_t njobs,
                                     const LokiPruneLevel* levels, const int32_t* seg_idx,
                                     const double* thresholds, int32_t nlevels,
                                     const LokiScoreSpec* spec, int64_t max_sugg,
                                     int64_t batch_size, void* dev_scratch,
                                     int64_t dev_scratch_bytes, void* stream) {
  if (!jobs || njobs < 1 || !levels || !seg_idx || !thresholds || nlevels < 1 || !spec ||
      !dev_scratch)
    return set_error(LOKI_ERR_INVALID, "null pointer, no job or no level");
  if (max_sugg < 1 || batch_size < 1)
    return set_error(LOKI_ERR_INVALID, "bad sizes");
  if (dev_scratch_bytes < loki_prune_run_blocks_scratch_bytes(njobs, nlevels))
    return set_error(LOKI_ERR_CAPACITY, "job scratch below %lld bytes",
                     (long long)loki_prune_run_blocks_scratch_bytes(njobs, nlevels));
  const int nb = levels[0].nbins;
  for (int64_t k = 0; k < (int64_t)njobs * nlevels; ++k) {
    int rc = check_prune(&levels[k]);
    if (rc) return rc;
    if (levels[k].basis != levels[0].basis || levels[k].poly_order != levels[0].poly_order ||
        levels[k].nbins != nb)
      return set_error(LOKI_ERR_INVALID, "levels of different trees");
  }
  if (levels[0].basis == 2)
    return set_error(LOKI_ERR_UNSUPPORTED, "the circular-orbit tree runs in loki_prune_run");
  for (int j = 0; j < njobs; ++j) {
    const LokiPruneJob& J = jobs[j];
    const LokiPruneRun& R = J.run;
    const LokiPruneWork& w = R.work;
    if (!J.ffa_fold || J.seg_stride < 1 || !J.dev_err || J.seed_n < 0 || J.seed_n > max_sugg)
      return set_error(LOKI_ERR_INVALID, "job %d: bad fold, error word or seed", j);
    if (R.trees[0].cap < max_sugg || R.trees[1].cap < max_sugg || w.par_cap < max_sugg ||
        w.child_cap < 1 || w.ovf_cap < max_sugg + w.child_cap + 1)
      return set_error(LOKI_ERR_CAPACITY, "job %d: workspace below max_sugg / child_cap", j);
    if (!R.counts || !R.ovf_flag || !R.stats || !w.info || !w.offsets || !w.child_scores ||
        !w.child_idx || !w.child_phase || !w.surv || !w.sscan || !w.minmax || !w.ovf_ids ||
        !w.ovf_keys || !w.ovf_thr)
      return set_error(LOKI_ERR_INVALID, "job %d: null workspace pointer", j);
    if (w.sscan_bytes <
        loki_scan_scratch_bytes(w.child_cap) + (w.child_cap + 1) * (int64_t)sizeof(int64_t))
      return set_error(LOKI_ERR_CAPACITY, "job %d: selection scratch below child_cap", j);
    for (int t = 0; t < 2; ++t)
      if (!R.trees[t].leaves || !R.trees[t].folds || !R.trees[t].scores ||
          !R.trees[t].scores_ep || !R.trees[t].backtracks)
        return set_error(LOKI_ERR_INVALID, "job %d: null tree pointer", j);
  }
  int rc = prune_spec_check(spec, nb);
  if (rc) return rc;
  LokiScoreSpec sp = *spec;
  sp.mode = 1;
  const ScoreK SK = make_score_k(sp, nb);
  const int smem = (kRunThreads / 32) * 32 * score_stride(nb, sp.wmax) * (int)sizeof(float);
  if (smem > 200 * 1024)
    return set_error(LOKI_ERR_UNSUPPORTED, "nbins + wmax too large for the block driver");
  if (set_smem_limit(prune_block_run_kernel, smem) != cudaSuccess)
    return set_error(LOKI_ERR_CUDA, "cudaFuncSetAttribute failed");
  const int64_t nl = (int64_t)njobs * nlevels;
  char* base = reinterpret_cast<char*>(dev_scratch);
  const int64_t o_lv = ((int64_t)njobs * sizeof(LokiPruneJob) + 255) / 256 * 256;
  const int64_t o_si = o_lv + (nl * (int64_t)sizeof(LokiPruneLevel) + 255) / 256 * 256;
  const int64_t o_th = o_si + (nl * 4 + 255) / 256 * 256;
  cudaStream_t s = (cudaStream_t)stream;
  if (cudaMemcpyAsync(base, jobs, njobs * sizeof(LokiPruneJob), cudaMemcpyHostToDevice, s) !=
          cudaSuccess ||
      cudaMemcpyAsync(base + o_lv, levels, nl * sizeof(LokiPruneLevel), cudaMemcpyHostToDevice,
                      s) != cudaSuccess ||
      cudaMemcpyAsync(base + o_si, seg_idx, nl * 4, cudaMemcpyHostToDevice, s) != cudaSuccess ||
      cudaMemcpyAsync(base + o_th, thresholds, nl * 8, cudaMemcpyHostToDevice, s) != cudaSuccess)
    return set_error(LOKI_ERR_CUDA, "copy of the job tables failed");
  note_launch();
  prune_block_run_kernel<<<(unsigned)njobs, kRunThreads, smem, s>>>(
      reinterpret_cast<const LokiPruneJob*>(base),
      reinterpret_cast<const LokiPruneLevel*>(base + o_lv),
      reinterpret_cast<const int32_t*>(base + o_si), reinterpret_cast<const double*>(base + o_th),
      nlevels, sp, SK, max_sugg, batch_size);
  return check_launch("prune_block_run");
}

// ---------------------------------------------------------------------------
// level-synchronous batch: every step of a level is one launch over all jobs
// (blockIdx.y = job), so a batch of jobs costs the launches of one run and
// each step spreads over the whole GPU. The device code is that of
// loki_prune_run; the counters, records and results of job j are those a
// loki_prune_run of job j writes.
// ---------------------------------------------------------------------------

namespace loki {

struct BatchTabs {
  const LokiPruneJob* jobs;
  const LokiPruneLevel* levels;  // [job][level]
  const int32_t* seg_idx;        // [job][level]
  const double* thr;             // [job][level]
  int32_t nlevels;
};

// counts[] of a job between the kernels of a level: parents, children (0 when
// they exceed the workspace), survivors, backtrack rows of the levels before,
// valid children (circular tree), and for the emission the parents, the first
// backtrack row and the best survivor of the level.
enum { kCntPar, kCntChild, kCntSurv, kCntBt, kCntValid, kCntOldPar, kCntBtRow, kCntBest };

__global__ void bj_seed_kernel(BatchTabs T) {
  const LokiPruneJob& J = T.jobs[blockIdx.x];
  int64_t* cnt = J.run.counts;
  cnt[0] = J.seed_n;
  for (int k = 1; k < 8; ++k) cnt[k] = 0;
  unsigned* keys = reinterpret_cast<unsigned*>(J.run.work.minmax);
  keys[0] = 0xFFFFFFFFu;
  keys[1] = 0u;
  *J.run.ovf_flag = 0;
}

// ---- work of a level's wide kernels -------------------------------------------
//
// A wide kernel (branch, map, score, emit) runs one block per resident slot of
// the GPU over the tiles of up to kQueueJobs jobs: every block sums the jobs'
// tile counts (from one of their counters) and takes an equal run of
// consecutive tiles, so most blocks see one job. A job's level descriptor
// (2.3 KB of matrices and limits, read by every step of the resolve) is copied
// to shared memory when the block turns to it. With a grid of blocks per job
// instead, sized for the largest job, most blocks only read their job's
// counters and left (60 us a level for 64 jobs in branch alone), and the
// descriptor's lines were fetched one dependent load after another.
// What every wide kernel of a batch takes beside its tables.
struct LevelArgs {
  LokiScoreSpec sp;
  ScoreK SK;
  int64_t batch;  // parents a batch (circular tree)
  int nb;         // phase bins
};

constexpr int kQueueJobs = 256;
constexpr int kTile = kPruneWarps * 32;  // parents, children or survivors a tile

struct JobQueue {
  alignas(16) LokiPruneLevel lvl;
  BranchF bf;
  int width;                // items a warp takes of a tile
  int pre[kQueueJobs + 1];  // tiles before each job
};

// Widths a warp may take: the narrowest and the widest below 32, packed.
enum { kWide = 32 << 5, kNarrow8 = 8 << 5 | 8, kNarrow16 = 8 << 5 | 16 };

// Tiles [t0, t1) of this block over jobs j0 .. j0 + nj, counts[idx] items each. A
// warp takes 32 items of a tile; where the level is so small that the grid holds
// all tiles at once even then, `narrow` (8) or twice that: a warp's time is latency
// there (rows are gathered a few at a time, complex ones transformed by four lanes
// a child), and 100 of the 127 levels of a search have a few hundred children a run
// (score of such a level 20 -> 16 us, circular 20 -> 14, complex 44 -> 20, emission
// 13 -> 11). The complex scores take 8 or 32: between, a lane transforms a child by
// itself and half of the lanes would idle.
__device__ __forceinline__ void queue_open(JobQueue& Q, const BatchTabs& T, int j0, int nj,
                                           int idx, int narrow, int* t0, int* t1) {
  const int lane = threadIdx.x & 31;
  int64_t cnt[kQueueJobs / kTile];
#pragma unroll
  for (int k = 0; k < kQueueJobs / kTile; ++k) {
    const int t = threadIdx.x + k * kTile;
    cnt[k] = t < nj ? T.jobs[j0 + t].run.counts[idx] : 0;
  }
  const int narrow_top = narrow & 31;
  int width = narrow >> 5, total;
  for (;; width = width < narrow_top ? 2 * width : 32) {
    const int items = width * kPruneWarps;
#pragma unroll
    for (int k = 0; k < kQueueJobs / kTile; ++k) {
      const int t = threadIdx.x + k * kTile;
      if (t < nj) Q.pre[t + 1] = (int)((cnt[k] + items - 1) / items);
    }
    if (threadIdx.x == 0) Q.pre[0] = 0;
    __syncthreads();
    if (threadIdx.x < 32) {
      int carry = 0;
      for (int base = 0; base < nj; base += 32) {
        int v = base + lane < nj ? Q.pre[base + lane + 1] : 0;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
          const int y = __shfl_up_sync(0xFFFFFFFFu, v, o);
          if (lane >= o) v += y;
        }
        if (base + lane < nj) Q.pre[base + lane + 1] = v + carry;
        carry += __shfl_sync(0xFFFFFFFFu, v, 31);
      }
    }
    __syncthreads();
    total = Q.pre[nj];
    if (width == 32 || total <= (int)gridDim.x) break;
    __syncthreads();  // every thread has read the total
  }
  if (threadIdx.x == 0) Q.width = width;
  const int per = (total + (int)gridDim.x - 1) / (int)gridDim.x;
  *t0 = min((int)blockIdx.x * per, total);
  *t1 = min(*t0 + per, total);
}

// Job of tile t; its level descriptor in Q.lvl (loaded when the job changes:
// every thread of the block comes here for every tile). Returns the job.
__device__ __forceinline__ int queue_job(JobQueue& Q, const BatchTabs& T, int j0, int nj, int l,
                                         int t, int cur) {
  int lo = 0, hi = nj;  // pre[lo] <= t < pre[hi]
  while (hi - lo > 1) {
    const int mid = (lo + hi) >> 1;
    if (Q.pre[mid] <= t) lo = mid;
    else hi = mid;
  }
  if (lo != cur) {
    __syncthreads();  // the previous job's descriptor is no longer read
    static_assert(sizeof(LokiPruneLevel) % 8 == 0, "copied by 8-byte words");
    const uint64_t* src = reinterpret_cast<const uint64_t*>(
        T.levels + (size_t)(j0 + lo) * T.nlevels + (l - 1));
    uint64_t* dst = reinterpret_cast<uint64_t*>(&Q.lvl);
    for (int k = threadIdx.x; k < (int)(sizeof(LokiPruneLevel) / 8); k += blockDim.x)
      dst[k] = src[k];
    if (threadIdx.x == 0)
      Q.bf = branch_floats(T.levels[(size_t)(j0 + lo) * T.nlevels + (l - 1)]);
    __syncthreads();
  }
  return lo;
}

// Runs body(job index, tile within the job, level descriptor) over this block's
// tiles.
template <typename F>
__device__ __forceinline__ void queue_run(JobQueue& Q, const BatchTabs& T, int l, int j0, int nj,
                                          int idx, int narrow, F body) {
  int t0, t1, cur = -1;
  queue_open(Q, T, j0, nj, idx, narrow, &t0, &t1);
  for (int t = t0; t < t1; ++t) {
    cur = queue_job(Q, T, j0, nj, l, t, cur);
    body(j0 + cur, (int64_t)(t - Q.pre[cur]));
  }
}

__device__ __forceinline__ const void* job_segment(const BatchTabs& T, const LokiPruneJob& J,
                                                   int job, int l, int bytes) {
  const size_t li = (size_t)job * T.nlevels + (l - 1);
  return reinterpret_cast<const char*>(J.ffa_fold) +
         (int64_t)T.seg_idx[li] * J.seg_stride * bytes;
}

template <int KP>
__global__ void __launch_bounds__(kTile)
bj_branch_kernel(BatchTabs T, int l, int j0, int nj, LevelArgs A) {
  __shared__ JobQueue Q;
  queue_run(Q, T, l, j0, nj, kCntPar, kWide, [&](int job, int64_t tile) {
    const LokiPruneJob& J = T.jobs[job];
    const int64_t i = tile * kTile + threadIdx.x;
    if (i < J.run.counts[kCntPar])
      branch_one<KP>(Q.lvl, J.run.trees[(l - 1) & 1].leaves, i,
                     reinterpret_cast<LokiBranchInfo*>(J.run.work.info), J.run.work.offsets,
                     J.dev_err, nullptr, Q.bf);
  });
}

// ---- per-job kernels: one block of 1024 threads a job ---------------------------

constexpr int kJobThreads = 1024;
constexpr int kJobPer = 8;  // consecutive items a thread takes per pass

// Exclusive block scan of one value a thread; the total to *tot.
__device__ __forceinline__ int64_t job_scan(int64_t x, int64_t* wsum, int64_t* tot) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  int64_t v = x;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int64_t y = __shfl_up_sync(0xFFFFFFFFu, v, o);
    if (lane >= o) v += y;
  }
  __syncthreads();  // wsum of the previous pass has been read
  if (lane == 31) wsum[warp] = v;
  __syncthreads();
  int64_t before = 0, total = 0;
  const int64_t w = wsum[lane];
  int64_t z = w;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int64_t y = __shfl_up_sync(0xFFFFFFFFu, z, o);
    if (lane >= o) z += y;
  }
  total = __shfl_sync(0xFFFFFFFFu, z, 31);
  before = __shfl_sync(0xFFFFFFFFu, z - w, warp);
  *tot = total;
  return before + v - x;
}

// A warp's share of n items, in order (its sum over the warp scanned once).
__device__ __forceinline__ void job_range(int64_t n, int64_t* b, int64_t* e) {
  const int64_t per = ((n + kJobThreads / 32 - 1) / (kJobThreads / 32) + 255) & ~int64_t(255);
  *b = min(n, (int64_t)(threadIdx.x >> 5) * per);
  *e = min(n, *b + per);
}

// Exclusive scan in place of the n counts at a; a[n] = the total. One pass over a
// small level; on a larger one every warp sums its share, the block scans the sums
// once, and the warps scan their shares (pass after pass, with the block's barriers
// in each, a single run of 870 000 children a level took 4 % longer than with the
// scans spread over the GPU).
__device__ __forceinline__ int64_t job_scan_counts(int64_t* a, int64_t n, int64_t* wsum) {
  int64_t tot;
  if (n <= kJobThreads * kJobPer) {
    const int64_t i0 = (int64_t)threadIdx.x * kJobPer;
    int64_t c[kJobPer], sum = 0;
#pragma unroll
    for (int k = 0; k < kJobPer; ++k) {
      c[k] = i0 + k < n ? a[i0 + k] : 0;
      sum += c[k];
    }
    int64_t run = job_scan(sum, wsum, &tot);
#pragma unroll
    for (int k = 0; k < kJobPer; ++k) {
      if (i0 + k < n) a[i0 + k] = run;
      run += c[k];
    }
  } else {
    const int lane = threadIdx.x & 31;
    int64_t b, e, sum = 0;
    job_range(n, &b, &e);
    for (int64_t i0 = b; i0 < e; i0 += 32 * kJobPer)
#pragma unroll
      for (int k = 0; k < kJobPer; ++k) {
        const int64_t i = i0 + 32 * k + lane;
        sum += i < e ? a[i] : 0;
      }
    for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(0xFFFFFFFFu, sum, o);
    int64_t run = __shfl_sync(0xFFFFFFFFu, job_scan(lane == 0 ? sum : 0, wsum, &tot), 0);
    constexpr int kPer = 4;
    for (int64_t i0 = b + kPer * lane; i0 - kPer * lane < e; i0 += 32 * kPer) {
      int64_t c[kPer], v = 0;
#pragma unroll
      for (int k = 0; k < kPer; ++k) {
        c[k] = i0 + k < e ? a[i0 + k] : 0;
        v += c[k];
      }
      int64_t incl = v;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int64_t y = __shfl_up_sync(0xFFFFFFFFu, incl, o);
        if (lane >= o) incl += y;
      }
      int64_t at = run + incl - v;
#pragma unroll
      for (int k = 0; k < kPer; ++k) {
        if (i0 + k < e) a[i0 + k] = at;
        at += c[k];
      }
      run += __shfl_sync(0xFFFFFFFFu, incl, 31);
    }
  }
  if (threadIdx.x == 0) a[n] = tot;
  return tot;
}

// After branch: the children's offsets (and, circular tree, the expansions'),
// their number and the level's record; the circular tree's A.batch flags cleared.
__global__ void __launch_bounds__(kJobThreads) bj_scan_kernel(BatchTabs T, int l, int j0,
                                                              int circ, int64_t batch) {
  __shared__ int64_t wsum[32];
  const LokiPruneJob& J = T.jobs[j0 + blockIdx.x];
  const LokiPruneRun& R = J.run;
  int64_t* cnt = R.counts;
  const int64_t n = cnt[kCntPar];
  int64_t total = job_scan_counts(R.work.offsets, n, wsum);
  if (circ) {
    total += job_scan_counts(R.exp_off, n, wsum);
    for (int64_t i = threadIdx.x; i <= n / batch; i += blockDim.x) R.batch_taylor[i] = 0;
  }
  if (threadIdx.x == 0) {
    cnt[kCntChild] = total > R.work.child_cap ? 0 : total;
    LokiPruneLevelStats* st = R.stats + (l - 1);
    st->n_parents = n;
    st->n_children = total;
    if (!circ) st->n_valid = total;
    if (total > R.work.child_cap) atomicOr(J.dev_err, LOKI_DEVERR_CAPACITY);
  }
}

// Indices of the n values v with v >= thr, in order, to ids; returns how many.
// *best: position among them of the largest, the first of equals (-1: none).
__device__ __forceinline__ int64_t job_compact(const float* __restrict__ v, int64_t n, float thr,
                                               int64_t* __restrict__ ids, int64_t* wsum,
                                               int64_t* best) {
  int64_t tot, bi = -1;
  float bv = 0.0f;
  auto take = [&](float x, int64_t i, int64_t at) {
    if (bi < 0 || x > bv) {
      bv = x;
      bi = at;
    }
    ids[at] = i;
  };
  if (n <= kJobThreads * kJobPer) {  // one pass, as job_scan_counts
    const int64_t i0 = (int64_t)threadIdx.x * kJobPer;
    float x[kJobPer];
    unsigned f = 0;
    if (i0 + kJobPer <= n && (reinterpret_cast<uintptr_t>(v) & 15) == 0) {
#pragma unroll
      for (int k = 0; k < kJobPer; k += 4) {
        const float4 q = *reinterpret_cast<const float4*>(v + i0 + k);
        x[k] = q.x, x[k + 1] = q.y, x[k + 2] = q.z, x[k + 3] = q.w;
      }
    } else {
#pragma unroll
      for (int k = 0; k < kJobPer; ++k) x[k] = i0 + k < n ? v[i0 + k] : nanf("");
    }
#pragma unroll
    for (int k = 0; k < kJobPer; ++k) f |= x[k] >= thr ? 1u << k : 0u;
    int64_t at = job_scan(__popc(f), wsum, &tot);
#pragma unroll
    for (int k = 0; k < kJobPer; ++k)
      if (f >> k & 1u) take(x[k], i0 + k, at++);
  } else {
    int64_t b, e;
    job_range(n, &b, &e);
    const int lane = threadIdx.x & 31;
    int cnt = 0;
    for (int64_t i0 = b; i0 < e; i0 += 32 * kJobPer)
#pragma unroll
      for (int k = 0; k < kJobPer; ++k) {
        const int64_t i = i0 + 32 * k + lane;
        cnt += i < e && v[i] >= thr ? 1 : 0;
      }
    cnt = (int)__reduce_add_sync(0xFFFFFFFFu, (unsigned)cnt);
    int64_t run = __shfl_sync(0xFFFFFFFFu, job_scan(lane == 0 ? cnt : 0, wsum, &tot), 0);
    for (int64_t i0 = b; i0 < e; i0 += 32 * kJobPer) {
      float x[kJobPer];
#pragma unroll
      for (int k = 0; k < kJobPer; ++k) {
        const int64_t i = i0 + 32 * k + lane;
        x[k] = i < e ? v[i] : nanf("");
      }
#pragma unroll
      for (int k = 0; k < kJobPer; ++k) {
        const unsigned m = __ballot_sync(0xFFFFFFFFu, x[k] >= thr);
        if (x[k] >= thr) take(x[k], i0 + 32 * k + lane, run + __popc(m & lanemask_lt()));
        run += __popc(m);
      }
    }
  }
  // the block's best: a thread's own is its first maximum already
  __shared__ float sv[32];
  __shared__ int64_t si[32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  auto fold = [&]() {
    for (int o = 16; o > 0; o >>= 1) {
      const float ov = __shfl_down_sync(0xFFFFFFFFu, bv, o);
      const int64_t oi = __shfl_down_sync(0xFFFFFFFFu, bi, o);
      if (oi >= 0 && (bi < 0 || ov > bv || (ov == bv && oi < bi))) {
        bv = ov;
        bi = oi;
      }
    }
  };
  fold();
  if (lane == 0) {
    sv[warp] = bv;
    si[warp] = bi;
  }
  __syncthreads();
  bv = sv[lane];
  bi = si[lane];
  fold();
  *best = __shfl_sync(0xFFFFFFFFu, bi, 0);
  __syncthreads();
  return tot;
}

// Circular tree: the valid children in order and their number.
__global__ void __launch_bounds__(kJobThreads) bj_circ_valid_kernel(BatchTabs T, int l, int j0) {
  __shared__ int64_t wsum[32];
  const LokiPruneRun& R = T.jobs[j0 + blockIdx.x].run;
  int64_t best;
  const int64_t n = job_compact(R.valid_flags, R.counts[kCntChild], 0.5f, R.valid_ids, wsum, &best);
  if (threadIdx.x == 0) {
    R.counts[kCntValid] = n;
    R.stats[l - 1].n_valid = n;
  }
}

// After score: the survivors in child order (by the overflow rule when they
// exceed max_sugg), the best of them, the level's record, and the counters
// turned to the next level.
__global__ void __launch_bounds__(kJobThreads)
bj_select_kernel(BatchTabs T, int l, int j0, int64_t max_sugg, int64_t batch, int circ) {
  __shared__ int64_t wsum[32];
  const int job = j0 + blockIdx.x;
  const LokiPruneJob& J = T.jobs[job];
  const LokiPruneRun& R = J.run;
  const LokiPruneWork& w = R.work;
  int64_t* cnt = R.counts;
  const int64_t n_par = cnt[kCntPar], n_valid = cnt[kCntValid];
  const double thr = T.thr[(size_t)job * T.nlevels + (l - 1)];
  int64_t best;
  // a float is at or above thr exactly if it is at or above the first float there
  int64_t n = job_compact(w.child_scores, circ ? n_valid : cnt[kCntChild],
                          __double2float_ru(thr), w.surv, wsum, &best);
  const bool ovf = n > max_sugg;
  if (ovf) {
    const int64_t* off = w.offsets;
    if (circ) {  // the rule's batches are over the valid children
      for (int64_t q = threadIdx.x; q <= (n_par + batch - 1) / batch; q += blockDim.x) {
        const int64_t p = min(q * batch, n_par);
        R.batch_offsets[p] = lower_bound64(R.valid_ids, n_valid, w.offsets[p] + R.exp_off[p]);
      }
      off = R.batch_offsets;
    }
    __syncthreads();
    select_overflow_block(w.child_scores, off, n_par, batch, thr, max_sugg, w.surv, &wsum[0],
                          w.ovf_thr, w.ovf_ids, reinterpret_cast<unsigned*>(w.ovf_keys));
    n = wsum[0];
    __syncthreads();
    // the best of what the rule kept
    unsigned long long* key = reinterpret_cast<unsigned long long*>(&wsum[1]);
    if (threadIdx.x == 0) *key = 0ull;
    __syncthreads();
    for (int64_t i = threadIdx.x; i < n; i += blockDim.x)
      // + 0.0f: zeros of either sign are equal
      atomicMax(key, ((unsigned long long)float_key(w.child_scores[w.surv[i]] + 0.0f) << 32) |
                         (0xFFFFFFFFu - (unsigned)i));
    __syncthreads();
    best = n > 0 ? (int64_t)(0xFFFFFFFFu - (unsigned)*key) : -1;
  }
  if (threadIdx.x != 0) return;
  LokiPruneLevelStats* st = R.stats + (l - 1);
  unsigned* keys = reinterpret_cast<unsigned*>(w.minmax);
  cnt[kCntOldPar] = n_par;
  cnt[kCntBtRow] = cnt[kCntBt];
  cnt[kCntBest] = best;
  cnt[kCntSurv] = n;
  if (R.bt_hist && cnt[kCntBt] + n > R.bt_rows) atomicOr(J.dev_err, LOKI_DEVERR_CAPACITY);
  *R.ovf_flag = ovf ? 1 : 0;
  level_end(cnt, keys, R.ovf_flag, st);
}

// ---- score and emission ------------------------------------------------------

template <int KP>
__global__ void __launch_bounds__(kTile, 3)
bj_score_kernel(BatchTabs T, int l, int j0, int nj, LevelArgs A) {
  extern __shared__ float tiles[];
  __shared__ JobQueue Q;
  const int warp = threadIdx.x >> 5;
  queue_run(Q, T, l, j0, nj, kCntChild, kNarrow16, [&](int job, int64_t t) {
    const LokiPruneJob& J = T.jobs[job];
    const LokiPruneWork& w = J.run.work;
    const LokiPruneTree& in = J.run.trees[(l - 1) & 1];
    const int64_t n_child = J.run.counts[kCntChild], c0 = (t * kPruneWarps + warp) * Q.width;
    if (c0 >= n_child) return;
    float* tile = tiles + (size_t)warp * 32 * score_stride(Q.lvl.nbins, A.sp.wmax);
    score_tile<KP>(Q.lvl, in.leaves, in.folds, J.run.counts[kCntPar],
               reinterpret_cast<LokiBranchInfo*>(w.info), w.offsets, n_child,
               static_cast<const float*>(job_segment(T, J, job, l, 4)), A.sp, A.SK, w.child_scores,
               w.child_idx, w.child_phase, reinterpret_cast<unsigned*>(w.minmax), tile, c0,
               Q.width);
    __syncwarp();
  });
}

// The emission's extras of a job: its backtrack history row and best survivor.
__device__ __forceinline__ EmitExtra job_extra(const LokiPruneRun& R, int l, int P) {
  EmitExtra X;
  const int64_t row = R.counts[kCntBtRow];
  if (R.bt_hist && row + R.counts[kCntSurv] <= R.bt_rows) X.bt_hist = R.bt_hist + row * (P + 2);
  if (R.best_leaves && R.best_scores) {
    X.best = R.counts[kCntBest];
    X.best_leaf = R.best_leaves + (int64_t)(l - 1) * (P + 2) * 2;
    X.best_score = R.best_scores + (l - 1);
  }
  return X;
}

template <int KP>
__global__ void __launch_bounds__(kTile, 4)
bj_emit_kernel(BatchTabs T, int l, int j0, int nj, LevelArgs A) {
  __shared__ JobQueue Q;
  const int warp = threadIdx.x >> 5;
  queue_run(Q, T, l, j0, nj, kCntSurv, kNarrow16, [&](int job, int64_t t) {
    const LokiPruneJob& J = T.jobs[job];
    const LokiPruneRun& R = J.run;
    const LokiPruneWork& w = R.work;
    const LokiPruneTree &in = R.trees[(l - 1) & 1], &out = R.trees[l & 1];
    const int64_t n_surv = R.counts[kCntSurv], s0 = (t * kPruneWarps + warp) * Q.width;
    if (s0 >= n_surv) return;
    emit_tile<KP>(Q.lvl, in.leaves, in.folds, reinterpret_cast<LokiBranchInfo*>(w.info), w.offsets,
              R.counts[kCntOldPar], static_cast<const float*>(job_segment(T, J, job, l, 4)),
              w.surv, n_surv, w.child_scores, w.child_idx, w.child_phase, out.leaves, out.folds,
              out.scores, out.scores_ep, out.backtracks, s0, job_extra(R, l, Q.lvl.poly_order),
                  Q.width);
  });
}

// Shared memory of the complex kernels: twiddles, then per warp either the 64-bin
// rows or (other bin counts) every lane's sums and score row.
__host__ __device__ inline int cplx_smem_bytes(int nbins, int wmax, bool score) {
  const int stride = score_stride(nbins, wmax);
  if (nbins == 64)
    return score ? kTwiddle64Bytes + kPruneWarps * max(cplx64_warp_bytes(), 32 * stride * 4)
                 : kPruneWarps * cplx64_warp_bytes() / 2;
  return score ? (int)((2 * nbins + kPruneWarps * cplx_warp_floats(nbins, stride)) * 4) : 0;
}

template <int KP>
__global__ void __launch_bounds__(kTile, 2)
bj_score_complex_kernel(BatchTabs T, int l, int j0, int nj, LevelArgs A) {
  extern __shared__ __align__(16) float smem[];
  __shared__ JobQueue Q;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int stride = score_stride(A.nb, A.sp.wmax), nbf = A.nb / 2 + 1;
  const float2* W = reinterpret_cast<const float2*>(smem) + 64;
  if (A.nb == 64) load_twiddles64(smem);
  else load_twiddles(smem, A.nb);
  queue_run(Q, T, l, j0, nj, kCntChild, kNarrow8, [&](int job, int64_t t) {
    const LokiPruneJob& J = T.jobs[job];
    const LokiPruneWork& w = J.run.work;
    const LokiPruneTree& in = J.run.trees[(l - 1) & 1];
    const LokiBranchInfo* info = reinterpret_cast<LokiBranchInfo*>(w.info);
    const float2* folds = reinterpret_cast<const float2*>(in.folds);
    const float2* seg = static_cast<const float2*>(job_segment(T, J, job, l, 8));
    unsigned* keys = reinterpret_cast<unsigned*>(w.minmax);
    const int64_t n_par = J.run.counts[kCntPar], n_child = J.run.counts[kCntChild];
    const int64_t c0 = (t * kPruneWarps + warp) * Q.width, c = c0 + lane;
    if (c0 >= n_child) return;
    const int kmax = (int)min((int64_t)Q.width, n_child - c0);
    const LokiPruneLevel& D = Q.lvl;
    if (A.nb != 64) {
      float* wbase = smem + 2 * A.nb + (size_t)warp * cplx_warp_floats(A.nb, stride);
      if (lane < kmax)
        score_child_complex(D, in.leaves, folds, n_par, info, w.offsets, seg, A.sp, A.SK,
                            w.child_scores, w.child_idx, w.child_phase, keys, smem,
                            reinterpret_cast<float2*>(wbase) + (size_t)lane * 2 * nbf,
                            wbase + (size_t)32 * 2 * nbf * 2 + lane * stride, c);
      return;
    }
    const int64_t par = warp_find_parents(w.offsets, n_par, c, kmax);
    int64_t row = 0;
    float2 delta = make_float2(1.0f, 0.0f);
    if (lane < kmax) {
      const int P = tree_order<KP>(D);
      const LokiBranchInfo B = info[par];
      double pv[LOKI_MAX_PARAMS + 1];
      child_params(B, P, c - w.offsets[par], pv);
      pv[P] = B.d0;
      const ChildRes r = resolve_child(D, P, pv, in.leaves[(par * (P + 2) + P + 1) * 2]);
      w.child_idx[2 * c] = r.ia;
      w.child_idx[2 * c + 1] = r.iff;
      w.child_phase[c] = r.phase;
      row = (int64_t)r.ia * D.n_freq + r.iff;
      delta = prune_phasor(r.phase, 64);
    }
    const int wb = max(cplx64_warp_bytes(), 32 * stride * 4);
    cplx64_score(folds, seg, par, row, delta, kmax, W,
                 reinterpret_cast<float2*>(reinterpret_cast<char*>(smem) + kTwiddle64Bytes +
                                           warp * wb),
                 A.sp, A.SK, w.child_scores + c0, keys);
    __syncwarp();
  });
}

template <int KP>
__global__ void __launch_bounds__(kTile, 4)
bj_emit_complex_kernel(BatchTabs T, int l, int j0, int nj, LevelArgs A) {
  extern __shared__ __align__(16) float smem[];
  __shared__ JobQueue Q;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  queue_run(Q, T, l, j0, nj, kCntSurv, kNarrow16, [&](int job, int64_t t) {
    const LokiPruneJob& J = T.jobs[job];
    const LokiPruneRun& R = J.run;
    const LokiPruneWork& w = R.work;
    const LokiPruneTree &in = R.trees[(l - 1) & 1], &out = R.trees[l & 1];
    const LokiBranchInfo* info = reinterpret_cast<LokiBranchInfo*>(w.info);
    const float2* folds = reinterpret_cast<const float2*>(in.folds);
    const float2* seg = static_cast<const float2*>(job_segment(T, J, job, l, 8));
    const int64_t n_surv = R.counts[kCntSurv], s0 = (t * kPruneWarps + warp) * Q.width;
    const int64_t s = s0 + lane;
    if (s0 >= n_surv) return;
    const int kmax = (int)min((int64_t)Q.width, n_surv - s0), nbf = A.nb / 2 + 1;
    const int64_t par = warp_find_parents(w.offsets, R.counts[kCntOldPar],
                                          w.surv[s0 + min(lane, kmax - 1)], kmax);
    EmitRow r = {0, 0, 0.0};
    if (lane < kmax)
      r = emit_one_complex_leaf<KP>(Q.lvl, in.leaves, info, w.offsets, w.surv, w.child_scores,
                                w.child_idx, w.child_phase, out.leaves, out.scores,
                                out.scores_ep, out.backtracks, s, par,
                                job_extra(R, l, Q.lvl.poly_order));
    float2* fout = reinterpret_cast<float2*>(out.folds);
    if (A.nb == 64)
      cplx64_emit(folds, seg, r.par, r.row, prune_phasor(r.phase, A.nb), kmax,
                  reinterpret_cast<float2*>(smem) + warp * 32 * kCplxRow,
                  fout + s0 * 66);
    else if (lane < kmax)
      rotate_add(seg + r.row * 2 * nbf, folds + r.par * 2 * nbf, prune_phasor(r.phase, A.nb), nbf,
                 fout + s * 2 * nbf);
  });
}

// ---- circular-orbit tree -------------------------------------------------------

__global__ void __launch_bounds__(kTile)
bj_circ_branch_kernel(BatchTabs T, int l, int j0, int nj, LevelArgs A) {
  __shared__ JobQueue Q;
  queue_run(Q, T, l, j0, nj, kCntPar, kWide, [&](int job, int64_t tile) {
    const LokiPruneJob& J = T.jobs[job];
    const int64_t i = tile * kTile + threadIdx.x;
    if (i < J.run.counts[kCntPar])
      circ_branch_one(Q.lvl, J.run.trees[(l - 1) & 1].leaves, i,
                      reinterpret_cast<LokiBranchInfo*>(J.run.work.info), J.run.work.offsets,
                      J.run.exp_off, J.dev_err, Q.bf);
  });
}

// the batch-ordered child map and validity flags (none of a level whose
// children exceed the workspace)
__global__ void __launch_bounds__(kTile)
bj_circ_map_kernel(BatchTabs T, int l, int j0, int nj, LevelArgs A) {
  __shared__ JobQueue Q;
  queue_run(Q, T, l, j0, nj, kCntPar, kWide, [&](int job, int64_t tile) {
    const LokiPruneRun& R = T.jobs[job].run;
    const int64_t i = tile * kTile + threadIdx.x, n = R.counts[kCntPar];
    if (i < n && R.counts[kCntChild] > 0)
      circ_map_one(Q.lvl, R.trees[(l - 1) & 1].leaves, n, A.batch,
                   reinterpret_cast<const LokiBranchInfo*>(R.work.info), R.work.offsets,
                   R.exp_off, reinterpret_cast<CircChild*>(R.child_map), R.valid_flags, i);
  });
}

__global__ void __launch_bounds__(kTile)
bj_circ_score_kernel(BatchTabs T, int l, int j0, int nj, LevelArgs A) {
  extern __shared__ float tiles[];
  __shared__ JobQueue Q;
  const int warp = threadIdx.x >> 5;
  queue_run(Q, T, l, j0, nj, kCntValid, kNarrow16, [&](int job, int64_t t) {
    const LokiPruneJob& J = T.jobs[job];
    const LokiPruneRun& R = J.run;
    const LokiPruneWork& w = R.work;
    const LokiPruneTree& in = R.trees[(l - 1) & 1];
    const int64_t n_valid = R.counts[kCntValid], v0 = (t * kPruneWarps + warp) * Q.width;
    if (v0 >= n_valid) return;
    circ_score_tile(Q.lvl, in.leaves, in.folds, A.batch,
                    reinterpret_cast<const LokiBranchInfo*>(w.info),
                    reinterpret_cast<const CircChild*>(R.child_map), R.valid_ids, n_valid,
                    static_cast<const float*>(job_segment(T, J, job, l, 4)), A.sp, A.SK,
                    w.child_scores, w.child_idx, w.child_phase, R.child_class, R.batch_taylor,
                    reinterpret_cast<unsigned*>(w.minmax),
                    tiles + (size_t)warp * 32 * score_stride(Q.lvl.nbins, A.sp.wmax), v0, Q.width);
    __syncwarp();
  });
}

__global__ void __launch_bounds__(kTile)
bj_circ_emit_kernel(BatchTabs T, int l, int j0, int nj, LevelArgs A) {
  __shared__ JobQueue Q;
  const int warp = threadIdx.x >> 5;
  queue_run(Q, T, l, j0, nj, kCntSurv, kNarrow16, [&](int job, int64_t t) {
    const LokiPruneJob& J = T.jobs[job];
    const LokiPruneRun& R = J.run;
    const LokiPruneWork& w = R.work;
    const LokiPruneTree &in = R.trees[(l - 1) & 1], &out = R.trees[l & 1];
    const int64_t n_surv = R.counts[kCntSurv], s0 = (t * kPruneWarps + warp) * Q.width;
    if (s0 >= n_surv) return;
    circ_emit_tile(Q.lvl, in.leaves, in.folds, A.batch,
                   reinterpret_cast<const LokiBranchInfo*>(w.info),
                   reinterpret_cast<const CircChild*>(R.child_map), R.valid_ids,
                   static_cast<const float*>(job_segment(T, J, job, l, 4)), w.surv, n_surv,
                   w.child_scores, w.child_idx, w.child_phase, R.child_class, R.batch_taylor,
                   out.leaves, out.folds, out.scores, out.scores_ep, out.backtracks, s0,
                   job_extra(R, l, 5), Q.width);
  });
}

__global__ void __launch_bounds__(kTile, 2)
bj_circ_score_complex_kernel(BatchTabs T, int l, int j0, int nj, LevelArgs A) {
  extern __shared__ __align__(16) float smem[];
  __shared__ JobQueue Q;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int stride = score_stride(A.nb, A.sp.wmax), nbf = A.nb / 2 + 1;
  const float2* W = reinterpret_cast<const float2*>(smem) + 64;
  if (A.nb == 64) load_twiddles64(smem);
  else load_twiddles(smem, A.nb);
  queue_run(Q, T, l, j0, nj, kCntValid, kNarrow8, [&](int job, int64_t t) {
    const LokiPruneJob& J = T.jobs[job];
    const LokiPruneRun& R = J.run;
    const LokiPruneWork& w = R.work;
    const LokiPruneTree& in = R.trees[(l - 1) & 1];
    const LokiBranchInfo* info = reinterpret_cast<const LokiBranchInfo*>(w.info);
    const CircChild* map = reinterpret_cast<const CircChild*>(R.child_map);
    const float2* folds = reinterpret_cast<const float2*>(in.folds);
    const float2* seg = static_cast<const float2*>(job_segment(T, J, job, l, 8));
    unsigned* keys = reinterpret_cast<unsigned*>(w.minmax);
    const int64_t n_valid = R.counts[kCntValid], v0 = (t * kPruneWarps + warp) * Q.width;
    const int64_t v = v0 + lane;
    if (v0 >= n_valid) return;
    const int kmax = (int)min((int64_t)Q.width, n_valid - v0);
    const LokiPruneLevel& D = Q.lvl;
    if (A.nb != 64) {
      float* wbase = smem + 2 * A.nb + (size_t)warp * cplx_warp_floats(A.nb, stride);
      if (lane < kmax)
        circ_score_one_complex(D, in.leaves, folds, A.batch, info, map, R.valid_ids, seg, A.sp,
                               A.SK, smem, reinterpret_cast<float2*>(wbase) + (size_t)lane * 2 * nbf,
                               wbase + (size_t)32 * 2 * nbf * 2 + lane * stride, w.child_scores,
                               w.child_idx, w.child_phase, R.child_class, R.batch_taylor, keys,
                               v);
      return;
    }
    int64_t par = 0, row = 0;
    float2 delta = make_float2(1.0f, 0.0f);
    if (lane < kmax) {
      const CircChild ch = map[R.valid_ids[v]];
      const LokiBranchInfo I = info[ch.parent];
      const double* lf = in.leaves + (int64_t)ch.parent * 14;
      double pv[6], ev[6];
      circ_child(I, lf, ch, pv, ev);
      ChildRes r;
      const int cls = circ_resolve(D, pv, ev, lf[12], &r);
      if (cls == 0) atomicOr(R.batch_taylor + ch.parent / A.batch, 1);
      w.child_idx[2 * v] = r.ia;
      w.child_idx[2 * v + 1] = r.iff;
      w.child_phase[v] = r.phase;
      R.child_class[v] = (int8_t)cls;
      par = ch.parent;
      row = (int64_t)r.ia * D.n_freq + r.iff;
      delta = prune_phasor(r.phase, 64);
    }
    const int wb = max(cplx64_warp_bytes(), 32 * stride * 4);
    cplx64_score(folds, seg, par, row, delta, kmax, W,
                 reinterpret_cast<float2*>(reinterpret_cast<char*>(smem) + kTwiddle64Bytes +
                                           warp * wb),
                 A.sp, A.SK, w.child_scores + v0, keys);
    __syncwarp();
  });
}

__global__ void __launch_bounds__(kTile)
bj_circ_emit_complex_kernel(BatchTabs T, int l, int j0, int nj, LevelArgs A) {
  extern __shared__ __align__(16) float smem[];
  __shared__ JobQueue Q;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  queue_run(Q, T, l, j0, nj, kCntSurv, kNarrow16, [&](int job, int64_t t) {
    const LokiPruneJob& J = T.jobs[job];
    const LokiPruneRun& R = J.run;
    const LokiPruneWork& w = R.work;
    const LokiPruneTree &in = R.trees[(l - 1) & 1], &out = R.trees[l & 1];
    const float2* folds = reinterpret_cast<const float2*>(in.folds);
    const float2* seg = static_cast<const float2*>(job_segment(T, J, job, l, 8));
    const int64_t n_surv = R.counts[kCntSurv], s0 = (t * kPruneWarps + warp) * Q.width;
    const int64_t s = s0 + lane;
    if (s0 >= n_surv) return;
    const int kmax = (int)min((int64_t)Q.width, n_surv - s0), nbf = A.nb / 2 + 1;
    EmitRow r = {0, 0, 0.0};
    if (lane < kmax)
      r = circ_emit_one_complex_leaf(Q.lvl, in.leaves, A.batch,
                                     reinterpret_cast<const LokiBranchInfo*>(w.info),
                                     reinterpret_cast<const CircChild*>(R.child_map),
                                     R.valid_ids, w.surv, w.child_scores, w.child_idx,
                                     w.child_phase, R.child_class, R.batch_taylor, out.leaves,
                                     out.scores, out.scores_ep, out.backtracks, s,
                                     job_extra(R, l, 5));
    float2* fout = reinterpret_cast<float2*>(out.folds);
    if (A.nb == 64)
      cplx64_emit(folds, seg, r.par, r.row, prune_phasor(r.phase, A.nb), kmax,
                  reinterpret_cast<float2*>(smem) + warp * 32 * kCplxRow,
                  fout + s0 * 66);
    else if (lane < kmax)
      rotate_add(seg + r.row * 2 * nbf, folds + r.par * 2 * nbf, prune_phasor(r.phase, A.nb), nbf,
                 fout + s * 2 * nbf);
  });
}

// The wide kernels of a batch: of the circular tree, or of a polynomial tree whose
// order is a constant in them (3 and 4, every configured search; KP 0: any).
struct BatchKernels {
  using Wide = void (*)(BatchTabs, int, int, int, LevelArgs);
  Wide branch, map, score, emit;
};

template <int KP>
BatchKernels tree_kernels(bool cplx) {
  return {bj_branch_kernel<KP>, nullptr,
          cplx ? bj_score_complex_kernel<KP> : bj_score_kernel<KP>,
          cplx ? bj_emit_complex_kernel<KP> : bj_emit_kernel<KP>};
}

inline BatchKernels batch_kernels(bool circ, bool cplx, int order) {
  if (circ)
    return {bj_circ_branch_kernel, bj_circ_map_kernel,
            cplx ? bj_circ_score_complex_kernel : bj_circ_score_kernel,
            cplx ? bj_circ_emit_complex_kernel : bj_circ_emit_kernel};
  return order == 3   ? tree_kernels<3>(cplx)
         : order == 4 ? tree_kernels<4>(cplx)
                      : tree_kernels<0>(cplx);
}

}  // namespace loki

// Host checks of a batch and the copy of its tables into dev_scratch; fills
// the grid sizes of the enqueue.
struct BatchShape {
  int nbins, poly_order;
  int64_t max_par, max_child;
  int fourier;  // complex (Fourier-domain) folds
  int circ;     // circular-orbit tree (real folds, poly_order 5)
};

static int batch_tables(const LokiPruneJob* jobs, int32_t njobs, const LokiPruneLevel* levels,
                        const int32_t* seg_idx, const double* thresholds, int32_t nlevels,
                        const LokiScoreSpec* spec, int64_t max_sugg, int64_t batch_size,
                        void* dev_scratch, int64_t dev_scratch_bytes, cudaStream_t s,
                        BatchShape* shape, int fourier = 0) {
  if (!jobs || njobs < 1 || njobs > 65535 || !levels || !seg_idx || !thresholds ||
      nlevels < 1 || !spec || !dev_scratch)
    return set_error(LOKI_ERR_INVALID, "null pointer, no job (or above 65535) or no level");
  if (max_sugg < 1 || batch_size < 1) return set_error(LOKI_ERR_INVALID, "bad sizes");
  if (dev_scratch_bytes < loki_prune_run_blocks_scratch_bytes(njobs, nlevels))
    return set_error(LOKI_ERR_CAPACITY, "job scratch below %lld bytes",
                     (long long)loki_prune_run_blocks_scratch_bytes(njobs, nlevels));
  const int nb = levels[0].nbins, P = levels[0].poly_order;
  int64_t max_par = 0, max_child = 0;
  for (int64_t k = 0; k < (int64_t)njobs * nlevels; ++k) {
    int rc = check_prune(&levels[k]);
    if (rc) return rc;
    if (levels[k].basis != levels[0].basis || levels[k].poly_order != P ||
        levels[k].nbins != nb)
      return set_error(LOKI_ERR_INVALID, "levels of different trees");
  }
  const bool circ = levels[0].basis == 2;
  if (circ && P != 5)
    return set_error(LOKI_ERR_UNSUPPORTED, "the circular-orbit tree has poly_order 5");
  for (int j = 0; j < njobs; ++j) {
    const LokiPruneJob& J = jobs[j];
    const LokiPruneRun& R = J.run;
    const LokiPruneWork& w = R.work;
    if (!J.ffa_fold || J.seg_stride < 1 || !J.dev_err || J.seed_n < 0 || J.seed_n > max_sugg)
      return set_error(LOKI_ERR_INVALID, "job %d: bad fold, error word or seed", j);
    if (circ && (!R.exp_off || !R.child_map || !R.valid_flags || !R.valid_ids ||
                 !R.child_class || !R.batch_taylor || !R.batch_offsets))
      return set_error(LOKI_ERR_INVALID, "job %d: no circular-orbit workspace", j);
    if (R.trees[0].cap < max_sugg || R.trees[1].cap < max_sugg || w.par_cap < max_sugg ||
        w.child_cap < 1 || w.ovf_cap < max_sugg + w.child_cap + 1)
      return set_error(LOKI_ERR_CAPACITY, "job %d: workspace below max_sugg / child_cap", j);
    if (!R.counts || !R.ovf_flag || !R.stats || !w.info || !w.offsets || !w.scan ||
        !w.child_scores || !w.child_idx || !w.child_phase || !w.surv || !w.sscan || !w.minmax ||
        !w.ovf_ids || !w.ovf_keys || !w.ovf_thr)
      return set_error(LOKI_ERR_INVALID, "job %d: null workspace pointer", j);
    if (w.scan_bytes < loki_scan_scratch_bytes(w.par_cap + 1) ||
        w.sscan_bytes <
            loki_scan_scratch_bytes(w.child_cap) + (w.child_cap + 1) * (int64_t)sizeof(int64_t))
      return set_error(LOKI_ERR_CAPACITY, "job %d: scan scratch below par_cap / child_cap", j);
    for (int t = 0; t < 2; ++t)
      if (!R.trees[t].leaves || !R.trees[t].folds || !R.trees[t].scores ||
          !R.trees[t].scores_ep || !R.trees[t].backtracks)
        return set_error(LOKI_ERR_INVALID, "job %d: null tree pointer", j);
    max_par = std::max(max_par, w.par_cap);
    max_child = std::max(max_child, w.child_cap);
  }
  int rc = prune_spec_check(spec, nb);
  if (rc) return rc;
  const int64_t nl = (int64_t)njobs * nlevels;
  char* base = reinterpret_cast<char*>(dev_scratch);
  const int64_t o_lv = ((int64_t)njobs * sizeof(LokiPruneJob) + 255) / 256 * 256;
  const int64_t o_si = o_lv + (nl * (int64_t)sizeof(LokiPruneLevel) + 255) / 256 * 256;
  const int64_t o_th = o_si + (nl * 4 + 255) / 256 * 256;
  if (cudaMemcpyAsync(base, jobs, njobs * sizeof(LokiPruneJob), cudaMemcpyHostToDevice, s) !=
          cudaSuccess ||
      cudaMemcpyAsync(base + o_lv, levels, nl * sizeof(LokiPruneLevel), cudaMemcpyHostToDevice,
                      s) != cudaSuccess ||
      cudaMemcpyAsync(base + o_si, seg_idx, nl * 4, cudaMemcpyHostToDevice, s) != cudaSuccess ||
      cudaMemcpyAsync(base + o_th, thresholds, nl * 8, cudaMemcpyHostToDevice, s) != cudaSuccess)
    return set_error(LOKI_ERR_CUDA, "copy of the job tables failed");
  shape->nbins = nb;
  shape->poly_order = P;
  shape->max_par = max_par;
  shape->max_child = max_child;
  shape->fourier = fourier ? 1 : 0;
  shape->circ = circ ? 1 : 0;
  return LOKI_OK;
}

// The kernels of a batch over tables already in dev_scratch (no host
// access to them: the enqueue can be captured in a CUDA graph and replayed
// after new tables of the same shape are copied in).
static int batch_enqueue(void* dev_scratch, int32_t njobs, int32_t nlevels,
                         const LokiScoreSpec* spec, int64_t max_sugg, int64_t batch_size,
                         const BatchShape& shape, cudaStream_t s,
                         cudaEvent_t* ev_score = nullptr) {
  const int nb = shape.nbins;
  const bool cplx = shape.fourier != 0;
  LokiScoreSpec sp = *spec;
  sp.mode = 1;
  const ScoreK SK = make_score_k(sp, nb);
  const int smem = cplx ? cplx_smem_bytes(nb, sp.wmax, true)
                        : score_smem_bytes(nb, sp.wmax, kPruneWarps);
  const int smem_emit = cplx ? cplx_smem_bytes(nb, sp.wmax, false) : 0;
  if (smem > 200 * 1024)
    return set_error(LOKI_ERR_UNSUPPORTED, "nbins + wmax too large for pruning");
  const BatchKernels K = batch_kernels(shape.circ, cplx, shape.poly_order);
  const LevelArgs A = {sp, SK, batch_size, nb};
  if (set_smem_limit(K.score, smem) != cudaSuccess ||
      set_smem_limit(K.emit, smem_emit) != cudaSuccess)
    return set_error(LOKI_ERR_CUDA, "cudaFuncSetAttribute failed");
  int dev = 0, nsm = 0;
  if (cudaGetDevice(&dev) != cudaSuccess ||
      cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess)
    return set_error(LOKI_ERR_CUDA, "device query failed");
  const int64_t nl = (int64_t)njobs * nlevels;
  char* base = reinterpret_cast<char*>(dev_scratch);
  const int64_t o_lv = ((int64_t)njobs * sizeof(LokiPruneJob) + 255) / 256 * 256;
  const int64_t o_si = o_lv + (nl * (int64_t)sizeof(LokiPruneLevel) + 255) / 256 * 256;
  const int64_t o_th = o_si + (nl * 4 + 255) / 256 * 256;
  BatchTabs T;
  T.jobs = reinterpret_cast<const LokiPruneJob*>(base);
  T.levels = reinterpret_cast<const LokiPruneLevel*>(base + o_lv);
  T.seg_idx = reinterpret_cast<const int32_t*>(base + o_si);
  T.thr = reinterpret_cast<const double*>(base + o_th);
  T.nlevels = nlevels;
  // Wide kernels: one block per resident slot (see JobQueue), no more than the
  // largest workspace has tiles. Per-job kernels: one block a job.
  const int64_t max_par = shape.max_par, max_child = shape.max_child;
  const int nj_max = std::min<int>(njobs, kQueueJobs);
  auto wide = [&](BatchKernels::Wide kern, int bytes, int64_t items, unsigned* g) {
    int per = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, kern, kTile, bytes) != cudaSuccess)
      return set_error(LOKI_ERR_CUDA, "occupancy query failed");
    const int64_t tiles = (items + kPruneWarps * 8 - 1) / (kPruneWarps * 8) * nj_max;
    *g = (unsigned)std::max<int64_t>(1,
                                     std::min<int64_t>((int64_t)nsm * std::max(1, per), tiles));
    return (int)LOKI_OK;
  };
  unsigned g_branch = 1, g_map = 1, g_score = 1, g_emit = 1;
  if (int rc = wide(K.branch, 0, max_par, &g_branch)) return rc;
  if (shape.circ)
    if (int rc = wide(K.map, 0, max_par, &g_map)) return rc;
  if (int rc = wide(K.score, smem, max_child, &g_score)) return rc;
  if (int rc = wide(K.emit, smem_emit, max_par, &g_emit)) return rc;
  note_launch();
  bj_seed_kernel<<<(unsigned)njobs, 1, 0, s>>>(T);
  for (int l = 1; l <= nlevels; ++l) {
    // steps of the level for every job at once, kQueueJobs jobs a launch; the
    // score launches come together so that their time can be taken
    for (int step = 0; step < 7; ++step) {
      if (step == 4 && ev_score) cudaEventRecord(ev_score[2 * (l - 1)], s);
      if (step == 5 && ev_score) cudaEventRecord(ev_score[2 * (l - 1) + 1], s);
      if (!shape.circ && (step == 2 || step == 3)) continue;
      for (int j0 = 0; j0 < njobs; j0 += kQueueJobs) {
        const int nj = std::min(kQueueJobs, njobs - j0);
        note_launch();
        switch (step) {
          case 0: K.branch<<<g_branch, kTile, 0, s>>>(T, l, j0, nj, A); break;
          case 1:
            bj_scan_kernel<<<(unsigned)nj, kJobThreads, 0, s>>>(T, l, j0, shape.circ, batch_size);
            break;
          case 2: K.map<<<g_map, kTile, 0, s>>>(T, l, j0, nj, A); break;
          case 3: bj_circ_valid_kernel<<<(unsigned)nj, kJobThreads, 0, s>>>(T, l, j0); break;
          case 4: K.score<<<g_score, kTile, smem, s>>>(T, l, j0, nj, A); break;
          case 5:
            bj_select_kernel<<<(unsigned)nj, kJobThreads, 0, s>>>(T, l, j0, max_sugg, batch_size,
                                                                  shape.circ);
            break;
          default: K.emit<<<g_emit, kTile, smem_emit, s>>>(T, l, j0, nj, A);
        }
      }
    }
    int rc = check_launch("prune_run_batch");
    if (rc) return rc;
  }
  return LOKI_OK;
}

extern "C" int loki_prune_run_batch(const LokiPruneJob* jobs, int32_t njobs,
                                    const LokiPruneLevel* levels, const int32_t* seg_idx,
                                    const double* thresholds, int32_t nlevels,
                                    const LokiScoreSpec* spec, int64_t max_sugg,
                                    int64_t batch_size, void* dev_scratch,
                                    int64_t dev_scratch_bytes, void* stream) {
  cudaStream_t s = (cudaStream_t)stream;
  BatchShape shape;
  int rc = batch_tables(jobs, njobs, levels, seg_idx, thresholds, nlevels, spec, max_sugg,
                        batch_size, dev_scratch, dev_scratch_bytes, s, &shape);
  if (rc) return rc;
  return batch_enqueue(dev_scratch, njobs, nlevels, spec, max_sugg, batch_size, shape, s);
}

extern "C" int loki_prune_batch_tables(const LokiPruneJob* jobs, int32_t njobs,
                                       const LokiPruneLevel* levels, const int32_t* seg_idx,
                                       const double* thresholds, int32_t nlevels,
                                       const LokiScoreSpec* spec, int64_t max_sugg,
                                       int64_t batch_size, int32_t fourier, void* dev_scratch,
                                       int64_t dev_scratch_bytes, int64_t* shape_out,
                                       void* stream) {
  if (!shape_out) return set_error(LOKI_ERR_INVALID, "null shape pointer");
  BatchShape shape;
  int rc = batch_tables(jobs, njobs, levels, seg_idx, thresholds, nlevels, spec, max_sugg,
                        batch_size, dev_scratch, dev_scratch_bytes, (cudaStream_t)stream,
                        &shape, fourier);
  if (rc) return rc;
  shape_out[0] = shape.nbins;
  shape_out[1] = shape.poly_order;
  shape_out[2] = shape.max_par;
  shape_out[3] = shape.max_child;
  shape_out[4] = shape.fourier;
  shape_out[5] = shape.circ;
  return LOKI_OK;
}

extern "C" int loki_prune_batch_score_times(void* dev_scratch, int32_t njobs, int32_t nlevels,
                                            const LokiScoreSpec* spec, int64_t max_sugg,
                                            int64_t batch_size, const int64_t* shape_in,
                                            float* score_ms, void* stream) {
  if (!dev_scratch || !spec || !shape_in || !score_ms || njobs < 1 || njobs > 65535 ||
      nlevels < 1 || max_sugg < 1 || batch_size < 1)
    return set_error(LOKI_ERR_INVALID, "bad batch timing arguments");
  BatchShape shape;
  shape.nbins = (int)shape_in[0];
  shape.poly_order = (int)shape_in[1];
  shape.max_par = shape_in[2];
  shape.max_child = shape_in[3];
  shape.fourier = shape_in[4] != 0;
  shape.circ = shape_in[5] != 0;
  if (shape.nbins < 1 || shape.poly_order < 1 || shape.poly_order > LOKI_MAX_PARAMS ||
      shape.max_par < 1 || shape.max_child < 1 ||
      (shape.circ && shape.poly_order != 5))
    return set_error(LOKI_ERR_INVALID, "bad batch shape");
  int rc = prune_spec_check(spec, shape.nbins);
  if (rc) return rc;
  std::vector<cudaEvent_t> ev(2 * (size_t)nlevels, nullptr);
  for (auto& e : ev)
    if (cudaEventCreate(&e) != cudaSuccess) {
      for (auto& f : ev)
        if (f) cudaEventDestroy(f);
      return set_error(LOKI_ERR_CUDA, "cudaEventCreate failed");
    }
  cudaStream_t s = (cudaStream_t)stream;
  rc = batch_enqueue(dev_scratch, njobs, nlevels, spec, max_sugg, batch_size, shape, s,
                     ev.data());
  if (!rc && cudaStreamSynchronize(s) != cudaSuccess)
    rc = set_error(LOKI_ERR_CUDA, "cudaStreamSynchronize failed");
  for (int l = 0; l < nlevels && !rc; ++l)
    if (cudaEventElapsedTime(&score_ms[l], ev[2 * l], ev[2 * l + 1]) != cudaSuccess)
      rc = set_error(LOKI_ERR_CUDA, "cudaEventElapsedTime failed");
  for (auto& e : ev) cudaEventDestroy(e);
  return rc;
}

extern "C" int loki_prune_batch_enqueue(void* dev_scratch, int32_t njobs, int32_t nlevels,
                                        const LokiScoreSpec* spec, int64_t max_sugg,
                                        int64_t batch_size, const int64_t* shape_in,
                                        void* stream) {
  if (!dev_scratch || !spec || !shape_in || njobs < 1 || njobs > 65535 || nlevels < 1 ||
      max_sugg < 1 || batch_size < 1)
    return set_error(LOKI_ERR_INVALID, "bad batch enqueue arguments");
  BatchShape shape;
  shape.nbins = (int)shape_in[0];
  shape.poly_order = (int)shape_in[1];
  shape.max_par = shape_in[2];
  shape.max_child = shape_in[3];
  shape.fourier = shape_in[4] != 0;
  shape.circ = shape_in[5] != 0;
  if (shape.nbins < 1 || shape.poly_order < 1 || shape.poly_order > LOKI_MAX_PARAMS ||
      shape.max_par < 1 || shape.max_child < 1 ||
      (shape.circ && shape.poly_order != 5))
    return set_error(LOKI_ERR_INVALID, "bad batch shape");
  int rc = prune_spec_check(spec, shape.nbins);
  if (rc) return rc;
  return batch_enqueue(dev_scratch, njobs, nlevels, spec, max_sugg, batch_size, shape,
                       (cudaStream_t)stream);
}

// ---------------------------------------------------------------------------
// batched ascend and read-back of many jobs' final trees
// ---------------------------------------------------------------------------

namespace loki {

__global__ void __launch_bounds__(kPruneWarps * 32)
prune_ascend_batch_kernel(const LokiAscendJob* __restrict__ jobs, int nseg, LokiScoreSpec sp,
                          ScoreK SK) {
  extern __shared__ float tiles[];
  const LokiAscendJob& J = jobs[blockIdx.y];
  const LokiPruneLevel& D = J.lvl;
  const int warp = threadIdx.x >> 5;
  const int stride = score_stride(D.nbins, sp.wmax);
  float* acc = tiles + (size_t)warp * 32 * (2 * D.nbins + stride);
  float* tile = acc + 32 * 2 * D.nbins;
  const int64_t n = *J.n_dev;
  for (int64_t t = (int64_t)blockIdx.x * kPruneWarps + warp; t * 32 < n;
       t += (int64_t)gridDim.x * kPruneWarps) {
    ascend_tile(D, J.leaves, J.folds, J.scores, J.scores_ep, n, nseg, J.tm_seg, J.dt_seg,
                J.seg_idx, J.ffa_fold, J.seg_stride, sp, SK, acc, tile, t * 32);
    __syncwarp();  // the accumulators are reused by the next tile
  }
}

// The same over complex trees (folds and segment strides in float2 units).
__global__ void __launch_bounds__(kPruneWarps * 32)
prune_ascend_batch_complex_kernel(const LokiAscendJob* __restrict__ jobs, int nseg,
                                  LokiScoreSpec sp, ScoreK SK) {
  extern __shared__ float smem[];
  const LokiAscendJob& J = jobs[blockIdx.y];
  const LokiPruneLevel& D = J.lvl;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int nb = D.nbins, nbf = nb / 2 + 1;
  const int stride = score_stride(nb, sp.wmax);
  float* tw = smem;
  load_twiddles(tw, nb);
  __syncthreads();
  float* wbase = smem + 2 * nb + (size_t)warp * cplx_warp_floats(nb, stride);
  float2* comb = reinterpret_cast<float2*>(wbase) + (size_t)lane * 2 * nbf;
  float* trow = wbase + (size_t)32 * 2 * nbf * 2 + lane * stride;
  const int64_t n = *J.n_dev;
  for (int64_t r = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; r < n;
       r += (int64_t)gridDim.x * blockDim.x)
    ascend_one_complex(D, J.leaves, reinterpret_cast<float2*>(J.folds), J.scores, J.scores_ep,
                       nseg, J.tm_seg, J.dt_seg, J.seg_idx,
                       reinterpret_cast<const float2*>(J.ffa_fold), J.seg_stride, sp, SK, tw, comb,
                       trow, r);
}

// Block y copies part y: src[y][0 .. bytes[y]) to dst + off[y] (16-byte
// words where both ends allow, else bytes).
__global__ void gather_parts_kernel(const LokiGatherPart* __restrict__ parts,
                                    char* __restrict__ dst) {
  const LokiGatherPart& P = parts[blockIdx.y];
  const char* src = reinterpret_cast<const char*>(P.src);
  char* d = dst + P.dst_off;
  const int64_t nb = P.bytes;
  const int64_t step = (int64_t)gridDim.x * blockDim.x;
  const int64_t i0 = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (((reinterpret_cast<uintptr_t>(src) | reinterpret_cast<uintptr_t>(d)) & 15) == 0) {
    const int64_t n16 = nb >> 4;
    for (int64_t i = i0; i < n16; i += step)
      reinterpret_cast<uint4*>(d)[i] = reinterpret_cast<const uint4*>(src)[i];
    for (int64_t i = (n16 << 4) + i0; i < nb; i += step) d[i] = src[i];
  } else {
    for (int64_t i = i0; i < nb; i += step) d[i] = src[i];
  }
}

}  // namespace loki

extern "C" int loki_prune_ascend_batch(const LokiAscendJob* jobs, int32_t njobs, int32_t nseg,
                                       const LokiScoreSpec* spec, int64_t n_cap,
                                       int32_t fourier, void* dev_scratch,
                                       int64_t dev_scratch_bytes, void* stream) {
  if (!jobs || njobs < 1 || njobs > 65535 || nseg < 1 || !spec || n_cap < 1 || !dev_scratch)
    return set_error(LOKI_ERR_INVALID, "bad batched ascend arguments");
  if (dev_scratch_bytes < (int64_t)njobs * (int64_t)sizeof(LokiAscendJob))
    return set_error(LOKI_ERR_CAPACITY, "ascend job scratch below %lld bytes",
                     (long long)njobs * (long long)sizeof(LokiAscendJob));
  const int nb = jobs[0].lvl.nbins;
  for (int j = 0; j < njobs; ++j) {
    const LokiAscendJob& J = jobs[j];
    int rc = check_prune(&J.lvl);
    if (rc) return rc;
    if (J.lvl.nbins != nb || J.lvl.basis != jobs[0].lvl.basis)
      return set_error(LOKI_ERR_INVALID, "ascend jobs of different trees");
    if (!J.n_dev || !J.leaves || !J.folds || !J.scores || !J.scores_ep || !J.tm_seg ||
        !J.dt_seg || !J.seg_idx || !J.ffa_fold || J.seg_stride < 1 || !J.dev_err)
      return set_error(LOKI_ERR_INVALID, "ascend job %d: null pointer or bad stride", j);
  }
  int rc = prune_spec_check(spec, nb);
  if (rc) return rc;
  LokiScoreSpec sp = *spec;
  sp.mode = 1;
  const ScoreK SK = make_score_k(sp, nb);
  const int stride = score_stride(nb, sp.wmax);
  const int smem =
      fourier ? (int)((2 * nb + kPruneWarps * cplx_warp_floats(nb, stride)) * sizeof(float))
              : kPruneWarps * 32 * (2 * nb + stride) * (int)sizeof(float);
  if (smem > 200 * 1024) return set_error(LOKI_ERR_UNSUPPORTED, "nbins too large for ascend");
  if (smem > 48 * 1024 && (fourier ? set_smem_limit(prune_ascend_batch_complex_kernel, smem)
                                   : set_smem_limit(prune_ascend_batch_kernel, smem)) !=
                              cudaSuccess)
    return set_error(LOKI_ERR_CUDA, "cudaFuncSetAttribute failed");
  int dev = 0, nsm = 0, occ = 0;
  if (cudaGetDevice(&dev) != cudaSuccess ||
      cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess ||
      (fourier ? cudaOccupancyMaxActiveBlocksPerMultiprocessor(
                     &occ, prune_ascend_batch_complex_kernel, kPruneWarps * 32, smem)
               : cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, prune_ascend_batch_kernel,
                                                               kPruneWarps * 32, smem)) !=
          cudaSuccess)
    return set_error(LOKI_ERR_CUDA, "occupancy query failed");
  cudaStream_t s = (cudaStream_t)stream;
  if (cudaMemcpyAsync(dev_scratch, jobs, njobs * sizeof(LokiAscendJob), cudaMemcpyHostToDevice,
                      s) != cudaSuccess)
    return set_error(LOKI_ERR_CUDA, "copy of the ascend jobs failed");
  const int64_t need = (n_cap + kPruneWarps * 32 - 1) / (kPruneWarps * 32);
  const int64_t wave = ((int64_t)nsm * std::max(1, occ) + njobs - 1) / njobs;
  const unsigned bx = (unsigned)std::max<int64_t>(1, std::min<int64_t>(need, wave));
  note_launch();
  if (fourier)
    prune_ascend_batch_complex_kernel<<<dim3(bx, njobs), kPruneWarps * 32, smem, s>>>(
        reinterpret_cast<const LokiAscendJob*>(dev_scratch), nseg, sp, SK);
  else
    prune_ascend_batch_kernel<<<dim3(bx, njobs), kPruneWarps * 32, smem, s>>>(
        reinterpret_cast<const LokiAscendJob*>(dev_scratch), nseg, sp, SK);
  return check_launch("prune_ascend_batch");
}

extern "C" int loki_gather_parts(const LokiGatherPart* parts, int32_t nparts, void* dst,
                                 int64_t dst_bytes, void* dev_scratch,
                                 int64_t dev_scratch_bytes, void* stream) {
  if (!parts || nparts < 1 || nparts > 65535 || !dst || !dev_scratch)
    return set_error(LOKI_ERR_INVALID, "bad gather arguments");
  if (dev_scratch_bytes < (int64_t)nparts * (int64_t)sizeof(LokiGatherPart))
    return set_error(LOKI_ERR_CAPACITY, "gather scratch below %lld bytes",
                     (long long)nparts * (long long)sizeof(LokiGatherPart));
  int64_t maxb = 0;
  for (int i = 0; i < nparts; ++i) {
    if (parts[i].bytes < 0 || parts[i].dst_off < 0 ||
        parts[i].dst_off + parts[i].bytes > dst_bytes || (parts[i].bytes > 0 && !parts[i].src))
      return set_error(LOKI_ERR_INVALID, "gather part %d outside the destination", i);
    maxb = std::max(maxb, parts[i].bytes);
  }
  if (maxb == 0) return LOKI_OK;
  cudaStream_t s = (cudaStream_t)stream;
  if (cudaMemcpyAsync(dev_scratch, parts, nparts * sizeof(LokiGatherPart),
                      cudaMemcpyHostToDevice, s) != cudaSuccess)
    return set_error(LOKI_ERR_CUDA, "copy of the gather parts failed");
  const unsigned bx = (unsigned)std::max<int64_t>(1, std::min<int64_t>(64, (maxb / 16 + 255) / 256));
  note_launch();
  gather_parts_kernel<<<dim3(bx, nparts), 256, 0, s>>>(
      reinterpret_cast<const LokiGatherPart*>(dev_scratch), reinterpret_cast<char*>(dst));
  return check_launch("gather_parts");
}

namespace loki {

// Block y seeds job y: leaves copied, the segment rows copied into the tree
// and scored (normalised e / sqrt(v), boxcar S/N as loki_snr_score_batch),
// scores_ep and the seed record set, backtracks and the error word cleared.
__global__ void __launch_bounds__(kPruneWarps * 32)
prune_seed_batch_kernel(const LokiSeedJob* __restrict__ jobs, int nb, int P, LokiScoreSpec sp,
                        ScoreK SK) {
  extern __shared__ float tiles[];
  const LokiSeedJob& J = jobs[blockIdx.y];
  const int64_t n = J.n;
  const int row_leaf = (P + 2) * 2, row_bt = P + 2;
  const int64_t gtid = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  const int64_t gstep = (int64_t)gridDim.x * blockDim.x;
  for (int64_t i = gtid; i < n * row_leaf; i += gstep) J.leaves_out[i] = J.seed_leaves[i];
  for (int64_t i = gtid; i < n * 2 * nb; i += gstep) J.folds_out[i] = J.fold_rows[i];
  for (int64_t i = gtid; i < n * row_bt; i += gstep) J.bt_out[i] = 0;
  if (gtid == 0) *J.dev_err = 0;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int stride = score_stride(nb, sp.wmax);
  float* tile = tiles + (size_t)warp * 32 * stride;
  for (int64_t p0 = ((int64_t)blockIdx.x * kPruneWarps + warp) * 32; p0 < n;
       p0 += (int64_t)gridDim.x * kPruneWarps * 32) {
    const int kmax = (int)min((int64_t)32, n - p0);
    for (int k = 0; k < kmax; ++k) {
      const float* src = J.fold_rows + (p0 + k) * 2 * nb;
      float* trow = tile + k * stride;
      for (int j = lane; j < nb; j += 32) trow[j] = __fdiv_rn(src[j], __fsqrt_rn(src[nb + j]));
    }
    __syncwarp();
    if (lane < kmax) {
      float s;
      float* row = tile + lane * stride;
      if (SK.list64) score_row64(row, sp, SK, &s);
      else score_row(row, nb, sp, SK, &s);
      J.scores_out[p0 + lane] = s;
      J.scores_ep_out[p0 + lane] = s;
      J.seed_scores_out[p0 + lane] = s;
    }
    __syncwarp();
  }
}

// The same of complex folds: rows of 2 (nb / 2 + 1) float2, eight a warp (a run's
// few hundred seeds are one wave), normalised as fold_norm_complex_kernel does.
// Per-run launches and copies (eight for each job) left the GPU idle for most of
// 6 ms before the levels of 16 runs.
constexpr int kSeedRows = 8;

__global__ void __launch_bounds__(kPruneWarps * 32)
prune_seed_batch_complex_kernel(const LokiSeedJob* __restrict__ jobs, int nb, int P,
                                LokiScoreSpec sp, ScoreK SK) {
  extern __shared__ float smem[];
  const LokiSeedJob& J = jobs[blockIdx.y];
  const int64_t n = J.n;
  const int row_leaf = (P + 2) * 2, row_bt = P + 2, nbf = nb / 2 + 1;
  const float2* rows = reinterpret_cast<const float2*>(J.fold_rows);
  float2* fout = reinterpret_cast<float2*>(J.folds_out);
  const int64_t gtid = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  const int64_t gstep = (int64_t)gridDim.x * blockDim.x;
  for (int64_t i = gtid; i < n * row_leaf; i += gstep) J.leaves_out[i] = J.seed_leaves[i];
  for (int64_t i = gtid; i < n * 2 * nbf; i += gstep) fout[i] = rows[i];
  for (int64_t i = gtid; i < n * row_bt; i += gstep) J.bt_out[i] = 0;
  if (gtid == 0) *J.dev_err = 0;
  load_twiddles(smem, nb);
  __syncthreads();
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int stride = score_stride(nb, sp.wmax);
  float* tile = smem + 2 * nb + (size_t)warp * kSeedRows * stride;
  for (int64_t p0 = ((int64_t)blockIdx.x * kPruneWarps + warp) * kSeedRows; p0 < n;
       p0 += (int64_t)gridDim.x * kPruneWarps * kSeedRows) {
    const int kmax = (int)min((int64_t)kSeedRows, n - p0);
    for (int k = 0; k < kmax; ++k)
      for (int j = lane; j < nb; j += 32)
        tile[k * stride + j] = norm_bin_complex(rows + (p0 + k) * 2 * nbf, j, nb, nbf, smem);
    __syncwarp();
    if (lane < kmax) {
      float s;
      float* row = tile + lane * stride;
      if (SK.list64) score_row64(row, sp, SK, &s);
      else score_row(row, nb, sp, SK, &s);
      J.scores_out[p0 + lane] = s;
      J.scores_ep_out[p0 + lane] = s;
      J.seed_scores_out[p0 + lane] = s;
    }
    __syncwarp();
  }
}

}  // namespace loki

static int seed_batch(const LokiSeedJob* jobs, int32_t njobs, int32_t nbins, int32_t poly_order,
                      const LokiScoreSpec* spec, void* dev_scratch, int64_t dev_scratch_bytes,
                      bool cplx, void* stream);

extern "C" int loki_prune_seed_batch(const LokiSeedJob* jobs, int32_t njobs, int32_t nbins,
                                     int32_t poly_order, const LokiScoreSpec* spec,
                                     void* dev_scratch, int64_t dev_scratch_bytes,
                                     void* stream) {
  return seed_batch(jobs, njobs, nbins, poly_order, spec, dev_scratch, dev_scratch_bytes, false,
                    stream);
}

extern "C" int loki_prune_seed_batch_complex(const LokiSeedJob* jobs, int32_t njobs,
                                             int32_t nbins, int32_t poly_order,
                                             const LokiScoreSpec* spec, void* dev_scratch,
                                             int64_t dev_scratch_bytes, void* stream) {
  if (nbins % 2) return set_error(LOKI_ERR_INVALID, "complex folds need an even nbins");
  return seed_batch(jobs, njobs, nbins, poly_order, spec, dev_scratch, dev_scratch_bytes, true,
                    stream);
}

static int seed_batch(const LokiSeedJob* jobs, int32_t njobs, int32_t nbins, int32_t poly_order,
                      const LokiScoreSpec* spec, void* dev_scratch, int64_t dev_scratch_bytes,
                      bool cplx, void* stream) {
  if (!jobs || njobs < 1 || njobs > 65535 || !spec || !dev_scratch || nbins < 2 ||
      poly_order < 1 || poly_order > LOKI_MAX_PARAMS)
    return set_error(LOKI_ERR_INVALID, "bad seed batch arguments");
  if (dev_scratch_bytes < (int64_t)njobs * (int64_t)sizeof(LokiSeedJob))
    return set_error(LOKI_ERR_CAPACITY, "seed job scratch below %lld bytes",
                     (long long)njobs * (long long)sizeof(LokiSeedJob));
  int64_t maxn = 0;
  for (int j = 0; j < njobs; ++j) {
    const LokiSeedJob& J = jobs[j];
    if (J.n < 0 || (J.n > 0 && (!J.seed_leaves || !J.fold_rows || !J.leaves_out ||
                                !J.folds_out || !J.scores_out || !J.scores_ep_out ||
                                !J.seed_scores_out || !J.bt_out)) ||
        !J.dev_err)
      return set_error(LOKI_ERR_INVALID, "seed job %d: null pointer or negative size", j);
    maxn = std::max(maxn, J.n);
  }
  int rc = prune_spec_check(spec, nbins);
  if (rc) return rc;
  LokiScoreSpec sp = *spec;
  sp.mode = 1;
  const ScoreK SK = make_score_k(sp, nbins);
  const int rows = cplx ? kSeedRows : 32;  // a warp's
  const int smem = cplx ? (int)((2 * nbins + kPruneWarps * kSeedRows *
                                                 score_stride(nbins, sp.wmax)) * sizeof(float))
                        : score_smem_bytes(nbins, sp.wmax, kPruneWarps);
  if (smem > 200 * 1024) return set_error(LOKI_ERR_UNSUPPORTED, "nbins + wmax too large");
  const auto kern = cplx ? prune_seed_batch_complex_kernel : prune_seed_batch_kernel;
  if (smem > 48 * 1024 && set_smem_limit(kern, smem) != cudaSuccess)
    return set_error(LOKI_ERR_CUDA, "cudaFuncSetAttribute failed");
  cudaStream_t s = (cudaStream_t)stream;
  if (cudaMemcpyAsync(dev_scratch, jobs, njobs * sizeof(LokiSeedJob), cudaMemcpyHostToDevice,
                      s) != cudaSuccess)
    return set_error(LOKI_ERR_CUDA, "copy of the seed jobs failed");
  const unsigned bx =
      (unsigned)std::max<int64_t>(1, std::min<int64_t>(32, (maxn + kPruneWarps * rows - 1) /
                                                               (kPruneWarps * rows)));
  note_launch();
  kern<<<dim3(bx, njobs), kPruneWarps * 32, smem, s>>>(
      reinterpret_cast<const LokiSeedJob*>(dev_scratch), nbins, poly_order, sp, SK);
  return check_launch("prune_seed_batch");
}
