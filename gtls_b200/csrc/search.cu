// TLS period search kernels for sm_100a.
//
// Per trial period the reference (src/gputls/core.py:770-875 with the kernels
// of src/gputls/GPUFun.py) folds the light curve, sorts it by phase, pads the
// sorted flux with its first maxD samples, and evaluates for every duration d
// and phase start k the template chi2
//
//   chi2(d,k) = sum_{i<w} (y_{k+i} - 1 + s_i c)^2 w_{k+i}          (in transit)
//             + sum over the other samples of (1 - y)^2 w            (out of transit)
//             - edge correction (the wrapped tail)                  (GPUFun.py:425-434)
//
// with c = 2 * overshoot_d * mean depth of the window.  Written in terms of
// v = y - 1, u = v w and the baseline E = sum_{i<n} v_i^2 w_i (a constant of
// the light curve: the reference's E[M-1] - edge), this is exactly
//
//   chi2(d,k) = E + c (2 B_k + c C_k),  B_k = sum_i s_i u_{k+i},  C_k = sum_i s_i^2 w_{k+i}
//
// with B and C sliding correlations of the template with the folded (u, w)
// records.  Only the minimum over (d, k) is wanted, so every start is first
// bounded from block sums and only those that can hold the minimum get their
// sums (screen.cuh, chi2.cuh).  A start whose window mean fails the depth test
// carries the value n (GPUFun.py:407,437), and so do the starts that are not
// multiples of skip(d) = w / skip_point (for w > skip_point) in the main pass
// (GPUFun.py:402,409).
//
// Kernels:
//   curve_setup_kernel   (v, w) records per original sample and their sums.
//   prepare_kernel       one CTA per period: FP64 fold (GPUFun.py:30-41) and
//                        stable bucket ranking of the phases (cupy argsort):
//                        the original index of every sorted position.
//   chi2_kernel          one CTA per (period, range of starts): (min, argmin).
//   finish_kernel        per-period minimum over ranges (first occurrence).
#include <cuda_runtime.h>

#include <algorithm>
#include <cfloat>
#include <cmath>
#include <cstdint>
#include <cstring>
#include <vector>

#include "chi2_core.cuh"
#include "common.cuh"
#include "screen.cuh"

namespace gtls {

constexpr int kPrepThreads = 1024;
constexpr int kPrepThreadsSmall = 512;   // curves of at most kPrepSmallMaxN samples: two CTAs per SM
constexpr int kPrepSmallMaxN = 1 << 15;
constexpr int kSmallBucket = 8;     // entries of buckets up to this size are ranked by their own thread
constexpr int kSmallBucketSm = 32;  // the same, for buckets in shared memory
constexpr int kBigBuckets = 512;    // capacity of the list of larger buckets (warp-ranked)
constexpr int kMaxRounds = 96;      // rounds of the shared-memory prepare path
constexpr int kRoundShift = 20;     // hist entries of that path: position | round << kRoundShift
constexpr int kPosMask = (1 << kRoundShift) - 1;
constexpr int kPrepStaticSmem = 4096;  // static shared memory of prepare_kernel, rounded up
// ------------------------------------------------------------ descriptors
// Sums over a curve.  vscale and wscale are powers of two that bring v and w
// to the order of one for the FP32 bounds (screen.cuh): u scales with both,
// delta with dscale = vscale^2 wscale.
struct CurveConst {
  double ebase;            // sum v^2 w
  double vscale, wscale, dscale;
  double spike_u, spike_w; // samples of larger |u| or w (scaled) are spikes; infinite: none
  float wbar, qbar;        // mean of the scaled w and u^2, of samples that are no spikes
  int kind;                // kUniform: all weights equal; kNoValue or more: E is not finite
  int pad;
};
constexpr int kUniform = 1, kNoValue = 2;

// Per-light-curve parameters and buffers on the device.  A search covers one
// or many light curves; every kernel finds its curve through these.
template <typename Real>
struct CurveDev {
  const double* t;              // [n] times
  const double* y;              // [n] flux
  const double* dy;             // [n] uncertainties
  const double* periods;        // [np] this curve's trial periods
  double* chi2_out;             // [np]
  int64_t* loc_out;             // [np] or NULL
  int* late;                    // [np] 1: a list ran over, the period is searched again (scratch)
  double2* vw;                  // [n] (v, w) per original sample (scratch)
  CurveConst* cst;              // sums over the curve (scratch)
  double* sums;                 // [setup blocks * kSetupSums] their parts (scratch)
  int* arrived;                 // setup blocks done (0 at first)
  const int* widths;            // [D]
  const double* overshoot;      // [D]
  const double* templates;      // [D * max_width]
  const int* skips;             // [D]
  const int* trow_off;          // [D] offsets into trows
  typename Tr<Real>::R2* trows; // template rows (s, s^2), w_d entries each
  ScreenRow* srows;             // [2 D] bounds of the chi2 of a start: constants per duration and table,
  ScreenCell* scells;           // its cells,
  const int* sends;             // and their ends
  int* union_cnt;               // [nbatch]
  int* union_list;              // [nbatch * D] ascending duration indices
  long long np;
  int n, maxd, D, max_width, batch, nbatch;
  int tile, ntiles, nb_log2;    // starts of a chi2 CTA, CTAs of a period, bucket bits (global-scatter ordering)
  int rnb_log2, rcap;           // shared-memory prepare path: bucket bits and round capacity (0: off)
  int coarse, vstride;          // chi2: step of the coarse prefix (0: none), row of the prefix of v of a CTA
  float span;
};

// A run: consecutive periods of one curve inside a chunk of the period list,
// with the offsets of their scratch rows.  Chunk items and chi2 CTAs are
// numbered run after run.
struct Run {
  int curve;
  int item0;          // first item (period) of the run in its chunk
  int count;          // periods in the run
  int tile0;          // first chi2 CTA of the run in its chunk
  long long pidx0;    // index of the run's first period within its curve
  long long slot_off; // element offset of the run's first row of sorted indices (and of slots)
  long long v_off;    // element offset of the run's first row of prefixes of v
};

// Largest i in [lo, hi) with key(i) <= x (keys ascending, key(lo) <= x).
template <typename F>
__device__ __forceinline__ int upper_find(int lo, int hi, long long x, F key) {
  while (hi - lo > 1) {
    const int mid = (lo + hi) >> 1;
    if (key(mid) <= x) lo = mid;
    else hi = mid;
  }
  return lo;
}

// ------------------------------------------------------------ curve set-up
// (v, w) per original sample: v = y - 1 (exact), w = 1/(dy*dy)
// (calcInverseSquaredPatchedDy GPUFun.py:134-142), and the curve's sums, E =
// sum v^2 w (calculate_base_error GPUFun.py:293-312 summed over the n samples)
// first.  One CTA per kSetupItems samples (one CTA per curve took 25 us on
// 70,000 samples); the last of a curve's CTAs adds their parts, in order.
constexpr int kSetupThreads = 256;
constexpr int kSetupItems = 1024;
constexpr int kSetupSums = 8;   // E, sum v^2, sum w, sum u^2, min w, max w, sum |u|^(1/2), sum w^(1/2)
static_assert(kSetupSums <= kSetupThreads / 32, "a warp adds up each");

// Square root of x >= 0 to 6%: the exponent halved and half of the fraction with it
// (0 becomes 2^-511).
__device__ __forceinline__ double rough_root(double x) {
  return __longlong_as_double((__double_as_longlong(x) >> 1) + (1023LL << 51));
}

__device__ __forceinline__ double sums_join(int k, double x, double y) {
  return k == 4 ? fmin(x, y) : (k == 5 ? fmax(x, y) : x + y);
}
__device__ __forceinline__ double sums_none(int k) { return k == 4 ? INFINITY : (k == 5 ? -INFINITY : 0.0); }

// Power of two that brings x to [1, 2), or 1 where there is none.
__device__ __forceinline__ double unit_scale(double x) {
  if (!(x > 1e-290 && x < 1e290)) return 1.0;
  return exp2(-(double)ilogb(x));
}

// Spikes.  The bounds of a start (screen.cuh) come from differences of FP32
// prefix sums, which one sample of a million times the others' |u| (its u^2 a
// 10^12-fold) or w would leave without a digit for every cell after it: the list of
// waiting starts ran over, and 300 periods of 70,000 samples with one dy
// a thousandth of the others took 92 ms (now 2.0; clean 1.8).  Such samples, at most 2
// kSpikeMax of a curve, are left out of the prefix sums and added to the bounds of the
// windows that hold them.  The sums round to 2^-23 of the whole (kPrefixErr), so a
// curve has spikes where its sum of u^2 is so far above that of its samples but the largest
// kSpikeMax that a cell's u^2 would round by 128 of their mean (flares of 50%,
// 20 of it, cost 10% more with spikes than without), or where weights are above 2^20 typical ones.
// A sample is a spike from the largest power of two (times the typical |u|)
// on below which that rounding is at most 32.  Typical is the square of the mean
// square root, which spikes hardly move; curves whose sum is below 2^30 typical
// ones are not looked at.  1,024, not 256 with their v in the prefix sums: 300 periods of
// 70,000 samples, 700 of them up to 400 times the flux, 4.3 ms (39; dense sums 2.1);
// 350 up to 5 times 2.3 (11.4; 2.1); 700 lowered by up to 80% 2.8 (2.1; 3.7).
constexpr int kSpikeMax = 1024;
constexpr int kSpikes = 4 * kSpikeMax;   // of a CTA: a window may run once more around the curve
constexpr double kSpikeSum = 0x1p30, kSpikeRest = 0x1p28, kSpikeW = 0x1p20;

// The curve's thresholds of |u| and w (infinite: none), and where there are
// any its sums 1 to 3 (kSetupSums) without its spikes, by one CTA.
template <typename Real>
__device__ __noinline__ void find_spikes(const CurveDev<Real>& C, double typical_u, double typical_w, double (&sums)[4],
                            double (&thr)[2]) {
  constexpr int kBins = 96, kFirst = 4;   // |u| of 2^kFirst typical ones on, by powers of two
  __shared__ int hist[kBins], heavy;
  __shared__ double bin_q[kBins], limit[2], red[3][kSetupThreads / 32];
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const double inv_u = 1.0 / typical_u;
  auto sum_over = [&](double x) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
    return x;
  };
  for (int b = threadIdx.x; b < kBins; b += kSetupThreads) {
    hist[b] = 0;
    bin_q[b] = 0.0;
  }
  if (threadIdx.x == 0) heavy = 0;
  __syncthreads();
  double low_q = 0.0;
#pragma unroll 4
  for (int i = threadIdx.x; i < C.n; i += kSetupThreads) {
    const double2 g = __ldcg(&C.vw[i]);
    const double u = fabs(g.x * g.y), x = u * inv_u;
    if (x >= (double)(1 << kFirst)) {
      const int b = min(kBins - 1, ilogb(x) - kFirst);
      atomicAdd(&hist[b], 1);
      atomicAdd(&bin_q[b], u * u);
    } else {
      low_q += u * u;
    }
    if (g.y > kSpikeW * typical_w) atomicAdd(&heavy, 1);
  }
  low_q = sum_over(low_q);
  if (lane == 0) red[0][wid] = low_q;
  __syncthreads();
  if (threadIdx.x == 0) {
    double rest = 0.0, unit = (double)(1 << kFirst);   // unit: the least |u| of bin j, in typical ones
    for (int q = 0; q < kSetupThreads / 32; ++q) rest += red[0][q];
    int above = 0, j = 0;
    for (int b = 0; b < kBins; ++b) above += hist[b];
    for (; above > kSpikeMax; ++j, unit *= 2.0) {
      above -= hist[j];
      rest += bin_q[j];
    }
    limit[0] = INFINITY;
    if (sums[3] * C.n > kSpikeSum * rest) {
      double below = rest;
      for (; j < kBins && (below + bin_q[j]) * C.n <= kSpikeRest * rest; ++j, unit *= 2.0) below += bin_q[j];
      limit[0] = typical_u * unit;
    }
    limit[1] = heavy > 0 && heavy <= kSpikeMax ? kSpikeW * typical_w : INFINITY;
  }
  __syncthreads();
  thr[0] = limit[0];
  thr[1] = limit[1];
  if (thr[0] == INFINITY && thr[1] == INFINITY) return;
  double s[3] = {0.0, 0.0, 0.0};
#pragma unroll 4
  for (int i = threadIdx.x; i < C.n; i += kSetupThreads) {
    const double2 g = __ldcg(&C.vw[i]);
    const double u = g.x * g.y;
    if (fabs(u) >= thr[0] || g.y > thr[1]) continue;
    s[0] += g.x * g.x;
    s[1] += g.y;
    s[2] += u * u;
  }
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    s[k] = sum_over(s[k]);
    if (lane == 0) red[k][wid] = s[k];
  }
  __syncthreads();
  for (int k = 0; k < 3; ++k) {
    sums[1 + k] = 0.0;
    for (int q = 0; q < kSetupThreads / 32; ++q) sums[1 + k] += red[k][q];
  }
}

template <typename Real>
__device__ void curve_setup(const CurveDev<Real>& C, int blk, int nblk) {
  __shared__ double red[kSetupSums][kSetupThreads / 32];
  __shared__ int last;
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  double s[kSetupSums];
#pragma unroll
  for (int k = 0; k < kSetupSums; ++k) s[k] = sums_none(k);
  for (int i = blk * kSetupItems + threadIdx.x; i < min(C.n, (blk + 1) * kSetupItems); i += kSetupThreads) {
    const double v = C.y[i] - 1.0;
    const double d = C.dy[i];
    const double w = 1.0 / (d * d);
    C.vw[i] = make_double2(v, w);
    s[0] += v * v * w;
    s[1] += v * v;
    s[2] += w;
    s[3] += (v * w) * (v * w);
    s[4] = fmin(s[4], w);
    s[5] = fmax(s[5], w);
    s[6] += rough_root(fabs(v * w));
    s[7] += rough_root(w);
  }
#pragma unroll
  for (int k = 0; k < kSetupSums; ++k) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) s[k] = sums_join(k, s[k], __shfl_xor_sync(0xffffffffu, s[k], o));
    if (lane == 0) red[k][wid] = s[k];
  }
  __syncthreads();
  if (threadIdx.x < kSetupSums) {
    double x = red[threadIdx.x][0];
    for (int i = 1; i < kSetupThreads / 32; ++i) x = sums_join(threadIdx.x, x, red[threadIdx.x][i]);
    C.sums[(size_t)blk * kSetupSums + threadIdx.x] = x;
    __threadfence();
  }
  __syncthreads();
  // (thread 0's fence above comes after a barrier: it covers the CTA's (v, w) as well)
  if (threadIdx.x == 0) last = atomicAdd(C.arrived, 1) == nblk - 1;
  __syncthreads();
  if (!last) return;
  __threadfence();
  if (wid < kSetupSums) {
    const int k = wid;
    double x = sums_none(k);
    for (int b = lane; b < nblk; b += 32) x = sums_join(k, x, __ldcg(&C.sums[(size_t)b * kSetupSums + k]));
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) x = sums_join(k, x, __shfl_xor_sync(0xffffffffu, x, o));
    if (lane == 0) red[k][0] = x;
  }
  __syncthreads();
  double sums[4] = {red[0][0], red[1][0], red[2][0], red[3][0]}, thr[2] = {INFINITY, INFINITY};
  const double root_u = red[6][0] / C.n, root_w = red[7][0] / C.n;
  const double typical_u = root_u * root_u, typical_w = root_w * root_w;
  const double spread = sums[3] / typical_u / typical_u;
  if ((spread > kSpikeSum && spread < INFINITY) || (red[5][0] > kSpikeW * typical_w && red[5][0] < INFINITY))
    find_spikes(C, typical_u, typical_w, sums, thr);
  if (threadIdx.x == 0) {
    CurveConst cc;
    cc.ebase = sums[0];
    cc.vscale = unit_scale(sqrt(sums[1] / C.n));
    cc.wscale = unit_scale(sums[2] / C.n);
    cc.dscale = cc.vscale * cc.vscale * cc.wscale;
    cc.spike_u = thr[0] * (cc.vscale * cc.wscale);
    cc.spike_w = thr[1] * cc.wscale;
    cc.wbar = (float)(sums[2] * cc.wscale / C.n);
    cc.qbar = (float)(sums[3] * (cc.vscale * cc.wscale) * (cc.vscale * cc.wscale) / C.n);
    cc.kind = (red[4][0] == red[5][0] ? kUniform : 0) | (fabs(sums[0]) < INFINITY ? 0 : kNoValue);
    *C.cst = cc;
  }
}

// ------------------------------------------------------------ block scans
// Exclusive scan of an int array in shared memory, in place; returns the
// total.  Warp w owns the contiguous range [w*per, (w+1)*per) and walks it 32
// consecutive entries at a time, so that lanes never share a bank.
__device__ int block_exclusive_scan_smem(int* a, int len, int* warp_tmp) {
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, nw = blockDim.x >> 5;
  const int per = ((len + nw - 1) / nw + 31) & ~31;
  const int beg = min(len, wid * per), end = min(len, beg + per);
  int sum = 0;
  for (int i = beg + lane; i < end; i += 32) sum += a[i];
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
  if (lane == 0) warp_tmp[wid] = sum;
  __syncthreads();
  int carry = lane < wid ? warp_tmp[lane] : 0;
  int total = lane < nw ? warp_tmp[lane] : 0;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    carry += __shfl_xor_sync(0xffffffffu, carry, o);
    total += __shfl_xor_sync(0xffffffffu, total, o);
  }
  for (int i0 = beg; i0 < end; i0 += 32) {
    const int i = i0 + lane;
    const int x = i < end ? a[i] : 0;
    int inc = x;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int yv = __shfl_up_sync(0xffffffffu, inc, o);
      if (lane >= o) inc += yv;
    }
    if (i < end) a[i] = carry + inc - x;
    carry += __shfl_sync(0xffffffffu, inc, 31);
  }
  __syncthreads();
  return total;
}

// ---------------------------------------------------------------- prepare
// Phase of sample t for period P: t/P minus its truncation, as foldFast
// (GPUFun.py:38-39) computes it (IEEE division, int truncation).
__device__ __forceinline__ double fold_phase(double t, double P) {
  double x = __ddiv_rn(t, P);
  return x - (double)(int)x;
}

// Bucket (y) of a phase and its key within the bucket (x): the bucket is
// floor(phase * NB), NB a power of two, clamped so that out-of-range phases
// land in the first or last one; the key is 32 bits of the fraction, rounded
// down, which never reverses an order.  The key resolves 2^-46 of a turn at
// 2^14 buckets: phases of samples more than 64 turns from t = 0 are no finer,
// so that their keys differ wherever they do (a float's 24 bits left ties
// by the hundred on periods commensurate with the cadence).
__device__ __forceinline__ uint2 phase_key(double phase, int nb_log2) {
  const int nb = 1 << nb_log2;
  const double x = phase * (double)nb;
  const double b = floor(x);
  if (!(b >= 0.0)) return make_uint2(0u, 0u);
  if (b >= (double)nb) return make_uint2(~0u, (unsigned)(nb - 1));
  return make_uint2(__double2uint_rd((x - b) * 0x1p32), (unsigned)b);
}

// The same of sample times.  The quotient is the correctly rounded t / P
// without a division: from the rounded reciprocal r of P, two corrections
// q += r (t - q P), each remainder a fused multiply-add.  The first leaves q
// within one unit of the last place, and from such a q the second rounds
// correctly when r is itself rounded correctly (P. Markstein, IBM J. Res. Dev.
// 34, 1990, theorem on the final step of division).  Adding 2^52 rounded down
// then leaves the whole turns, and adding 2^20 / NB to the phase its bucket
// and key in the sum's two words: no branch and no conversion, so
// that a thread's samples overlap (the divide's own branch kept them one after
// the other; 70,000 samples: 0.95 -> 0.88 us a period).  Turn counts outside [2^-200, 2^31) and extreme periods
// are divided.
struct FoldKey {
  double P, r, place;
  int nb_log2;
  __device__ __forceinline__ FoldKey(double P_, int nbl) : P(P_), nb_log2(nbl) {
    r = P_ >= 0x1p-200 && P_ <= 0x1p200 ? __drcp_rn(P_) : __longlong_as_double(0x7ff8000000000000LL);
    place = __hiloint2double((1023 + 20 - nbl) << 20, 0);
  }
  template <int kB>
  __device__ __forceinline__ void operator()(const double (&t)[kB], uint2 (&w)[kB]) const {
    double x[kB];
#pragma unroll
    for (int u = 0; u < kB; ++u) x[u] = __dmul_rn(t[u], r);
#pragma unroll
    for (int c = 0; c < 2; ++c)
#pragma unroll
      for (int u = 0; u < kB; ++u) x[u] = __fma_rn(__fma_rn(-x[u], P, t[u]), r, x[u]);
#pragma unroll
    for (int u = 0; u < kB; ++u) {
      const double z = __dadd_rd(__dsub_rn(x[u], __dsub_rn(__dadd_rd(x[u], 0x1p52), 0x1p52)), place);
      w[u] = make_uint2((unsigned)__double2loint(z), (unsigned)__double2hiint(z) & 0xfffffu);
    }
#pragma unroll
    for (int u = 0; u < kB; ++u)
      if ((unsigned)__double2hiint(x[u]) - 0x33700000u >= 0x41e00000u - 0x33700000u)
        w[u] = phase_key(fold_phase(t[u], P), nb_log2);
  }
};

// Strict order of two slots of the same bucket: by phase, then by original
// index (the order of a stable argsort).  Equal keys are decided on the exact
// FP64 phases, recomputed.
// Slot index words hold the sample index, and in the bits above it a bucket
// where there is room (the same for two slots of one bucket, so comparing
// whole words compares the indices): index_bits is 17 for curves of at most
// 2^17 samples.
constexpr int kPackedShift = 17;
constexpr int kPackedMaxN = 1 << kPackedShift;
constexpr int kRoundMaxN = (1 << 20) - 1;   // positions of the rounds' hist entries; 12 bits for a bucket of a round
__host__ __device__ __forceinline__ int index_bits(int n) {
  int b = kPackedShift;
  while ((1 << b) < n) ++b;
  return b;
}
__device__ __forceinline__ bool slot_less(uint2 a, uint2 b, const double* __restrict__ t, double P, unsigned imask) {
  if (a.x != b.x) return a.x < b.x;
  const double pa = fold_phase(t[a.y & imask], P), pb = fold_phase(t[b.y & imask], P);
  if (pa != pb) return pa < pb;
  return a.y < b.y;
}

// Rank of every entry of bucket slots [s, e) among the bucket (emit(s + rank,
// original index)), by a whole warp: each lane ranks one entry of a group of
// 32 against the bucket, streamed 32 entries at a time and broadcast by
// shuffles.  Used for large buckets, whose O(k^2) comparisons would
// otherwise fall on single threads, where sort_bucket_warp cannot be.
template <typename Emit>
__device__ __forceinline__ void rank_bucket_warp(const uint2* __restrict__ slot, int s, int e,
                                                 const double* __restrict__ t, double P, unsigned imask, Emit emit) {
  const int lane = threadIdx.x & 31;
  for (int j0 = s; j0 < e; j0 += 32) {
    const int j = j0 + lane;
    const uint2 mine = slot[min(j, e - 1)];
    int r = 0;
    for (int m0 = s; m0 < e; m0 += 32) {
      const uint2 oth = slot[min(m0 + lane, e - 1)];
      const int cnt = min(32, e - m0);
      for (int q = 0; q < cnt; ++q) {
        uint2 o;
        o.x = __shfl_sync(0xffffffffu, oth.x, q);
        o.y = __shfl_sync(0xffffffffu, oth.y, q);
        if (o.y != mine.y && slot_less(o, mine, t, P, imask)) ++r;
      }
    }
    if (j < e) emit(s + r, (int)(mine.y & imask));
  }
}

// The same by sorting the bucket in place in shared memory, for buckets of a
// period commensurate with the cadence (hundreds to thousands of samples at a
// few phases; by comparing all pairs, a division in most, such a period
// took milliseconds: 800 periods of a 70,000-sample curve, of which a few are
// so, 2.2 -> 0.84 us each on average).  Each entry becomes one 64-bit word, the fraction of the
// bucket in fixed point above the ib bits of its index: with 64 - ib bits
// every phase is exact but those below 2^-10 of the samples before the first
// turn ends, so that the words sort as a stable argsort does.  A bucket with a
// fraction that is not exact takes rank_bucket_warp.  A network of
// ascending comparators (each merge starts with the mirrored pairs) works on any
// length: pairs that reach past the end are left out.  The slots keep
// their index words.
template <typename Emit>
__device__ __noinline__ void sort_bucket_warp(uint2* __restrict__ slot, int s, int e, int b, int nb_log2, int ib,
                                              unsigned high, const double* __restrict__ t, double P, Emit emit) {
  const int lane = threadIdx.x & 31, k = e - s;
  const unsigned imask = (1u << ib) - 1u;
  unsigned long long* const w = reinterpret_cast<unsigned long long*>(slot) + s;
  const double unit = (double)(1ULL << (63 - ib)) * 2.0;
  bool exact = true;
  for (int j = lane; j < k; j += 32) {
    const unsigned i = slot[s + j].y & imask;
    const double y = (fold_phase(t[i], P) * (double)(1 << nb_log2) - (double)b) * unit;
    const bool ok = y >= 0.0 && y < unit && y == floor(y);
    exact = exact && ok;
    w[j] = (ok ? (unsigned long long)y << ib : 0ULL) | i;
  }
  __syncwarp();
  if (!__all_sync(0xffffffffu, exact)) {
    for (int j = lane; j < k; j += 32) {
      const unsigned i = (unsigned)w[j] & imask;
      slot[s + j] = make_uint2(phase_key(fold_phase(t[i], P), nb_log2).x, i | high);
    }
    __syncwarp();
    rank_bucket_warp(slot, s, e, t, P, imask, emit);
    return;
  }
  auto order = [&](int i, int j) {
    if (j >= k) return;
    const unsigned long long x = w[i], y = w[j];
    if (y < x) {
      w[i] = y;
      w[j] = x;
    }
  };
  int half = 1;   // pairs of the padded length
  while (2 * half < k) half *= 2;
  for (int p = 1; p <= half; p *= 2) {   // sorted runs of p become runs of 2 p
    for (int c = lane; c < half; c += 32) {
      const int i = 2 * c - (c & (p - 1));
      order(i, i ^ (2 * p - 1));
    }
    __syncwarp();
    for (int q = p / 2; q > 0; q /= 2) {
      for (int c = lane; c < half; c += 32) {
        const int i = 2 * c - (c & (q - 1));
        order(i, i + q);
      }
      __syncwarp();
    }
  }
  for (int j = lane; j < k; j += 32) {
    const unsigned i = (unsigned)w[j] & imask;
    emit(s + j, (int)i);
    slot[s + j].y = i | high;
  }
}

// Round tables of the shared-memory prepare path.
struct RoundTables {
  int nrounds;               // rounds; -1: the period takes the global-scatter path
  int rb[kMaxRounds + 1];    // first bucket of each round (rb[nrounds] = NB)
  int rpos[kMaxRounds + 1];  // first sorted position of each round (rpos[nrounds] = n)
  int cursor[kMaxRounds];    // append cursors of the round-partitioned sample words
};

// Shared-memory prepare of one period (curves of at most kRoundMaxN
// samples).  The samples are folded (GPUFun.py:30-41) and counted into NB
// phase buckets; the buckets are cut greedily into rounds of whole buckets
// holding at most `cap` samples each (and no more buckets than the index word
// has room for); a second fold appends each sample's word (in-bucket key,
// index | bucket << ib, ib = index_bits(n), of which the low bits stay) to its round's range
// of the scratch row `stage` (warp-aggregated, so the stores stay nearly
// coalesced).  Each round then
//   (a) reads its words (coalesced) into shared-memory slots by bucket,
//   (b) ranks every slot within its bucket (the stable argsort order of
//       the fold, as slot_less defines it) and writes its original index at
//       the resulting sorted position (close to the slot's, so nearly
//       coalesced),
// so that nothing is scattered through global memory.  Returns false, having
// written nothing, when a single bucket holds more than `cap` samples or more
// than kMaxRounds rounds would be needed; the caller then takes the global
// path.  Dynamic shared memory: hist [NB] ints, slots [cap] words.
// kIndexBits: index_bits(n) where it is kPackedShift (every bucket number fits
// above it), else 0.
template <int kIndexBits>
__device__ __noinline__ bool prepare_rounds(int* dyn, int* wtmp_i, int* big, int* nbig, RoundTables& rt,
                               const double* __restrict__ t, int n, double P, int nb_log2, int cap,
                               uint2* __restrict__ stage, int* __restrict__ ord) {
  const int nb = 1 << nb_log2;
  const int ib = kIndexBits ? kIndexBits : index_bits(n);
  const unsigned imask = (1u << ib) - 1u;
  int* hist = dyn;
  uint2* slots = reinterpret_cast<uint2*>(dyn + nb);
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, nwarp = blockDim.x >> 5;
  constexpr int kB = 3;   // elements per thread in flight in each pass (2 and 4: 5% slower, short curves 8%)
  const int stride = blockDim.x * kB;

  const FoldKey fold(P, nb_log2);
  for (int b = threadIdx.x; b < nb; b += blockDim.x) hist[b] = 0;
  __syncthreads();
  // (1) fold and histogram of buckets
  for (int i0 = threadIdx.x; i0 < n; i0 += stride) {
    double tv[kB];
#pragma unroll
    for (int u = 0; u < kB; ++u) {
      const int i = i0 + u * blockDim.x;
      tv[u] = i < n ? t[i] : P;   // (a padding of 0 would take the divide)
    }
    uint2 wd[kB];
    fold(tv, wd);
#pragma unroll
    for (int u = 0; u < kB; ++u) {
      const int i = i0 + u * blockDim.x;
      if (i < n) atomicAdd(&hist[wd[u].y], 1);
    }
  }
  __syncthreads();
  block_exclusive_scan_smem(hist, nb, wtmp_i);   // hist[b]: first position of bucket b
  // (2) rounds, by warp 0: from bucket b0, the largest b1 with
  //     start(b1) <= start(b0) + cap (a 32-way search of the bucket starts)
  if (wid == 0) {
    auto S = [&](int x) { return x < nb ? hist[x] : n; };
    int r = 0, b0 = 0;
    bool ok = true;
    if (lane == 0) {
      rt.rb[0] = 0;
      rt.rpos[0] = 0;
    }
    while (b0 < nb) {
      const int lim = S(b0) + cap;
      int lo = b0, hi = min(nb, b0 + (int)(~0u >> ib) + 1);   // S(lo) <= lim; the answer lies in [lo, hi]
      while (lo < hi) {
        const int step = (hi - lo + 31) >> 5;
        const int x = min(hi, lo + (lane + 1) * step);
        const int c = __popc(__ballot_sync(0xffffffffu, S(x) <= lim));   // a prefix of the lanes
        const int nlo = min(hi, lo + c * step);
        const int nhi = c == 32 ? hi : min(hi, lo + (c + 1) * step) - 1;
        lo = nlo;
        hi = nhi;
      }
      if (lo == b0 || r == kMaxRounds) {   // bucket b0 alone exceeds cap, or too many rounds
        ok = false;
        break;
      }
      if (lane == 0) {
        rt.cursor[r] = S(b0);
        rt.rb[r + 1] = lo;
        rt.rpos[r + 1] = S(lo);
      }
      ++r;
      b0 = lo;
    }
    if (lane == 0) rt.nrounds = ok ? r : -1;
  }
  __syncthreads();
  const int nr = rt.nrounds;
  if (nr < 0) return false;
  // each bucket's round in the bits of hist above the positions
  for (int b = threadIdx.x; b < nb; b += blockDim.x)
    hist[b] |= upper_find(0, nr, b, [&](int q) { return (long long)rt.rb[q]; }) << kRoundShift;
  auto H = [&](int b) { return hist[b] & kPosMask; };
  // the bucket of a word of the round from b0 on, from its low bits
  auto bucket_of = [&](unsigned y, int b0) { 
    return kIndexBits ? (int)(y >> ib) : b0 + (int)(((y >> ib) - (unsigned)b0) & (~0u >> ib));
  };
  __syncthreads();
  // (3) fold again; each sample's word to its round's range of the scratch
  //     row (the loop runs over whole warps for the warp-wide match)
  for (int i0 = threadIdx.x - lane; i0 < n; i0 += stride) {
    double tv[kB];
#pragma unroll
    for (int u = 0; u < kB; ++u) {
      const int i = i0 + lane + u * blockDim.x;
      tv[u] = i < n ? t[i] : P;   // (a padding of 0 would take the divide)
    }
    uint2 wds[kB];
    fold(tv, wds);
#pragma unroll
    for (int u = 0; u < kB; ++u) {
      const int i = i0 + lane + u * blockDim.x;
      const int r = i < n ? hist[wds[u].y] >> kRoundShift : -1;
      const uint2 wd = make_uint2(wds[u].x, (unsigned)i | wds[u].y << ib);
      const unsigned peers = __match_any_sync(0xffffffffu, r);
      const int leader = __ffs(peers) - 1;
      int pos = 0;
      if (lane == leader && r >= 0) pos = atomicAdd(&rt.cursor[r], __popc(peers));
      pos = __shfl_sync(0xffffffffu, pos, leader) + __popc(peers & ((1u << lane) - 1u));
      if (r >= 0 && pos < rt.rpos[r + 1]) stage[pos] = wd;   // always true: the counts of pass (1)
    }
  }
  __syncthreads();
  for (int r = 0; r < nr; ++r) {
    const int rs = rt.rpos[r], cnt = rt.rpos[r + 1] - rs;
    const int b0 = rt.rb[r], b1 = rt.rb[r + 1];
    // (a) the round's words into slots by bucket; afterwards the position
    //     H(b) is the end of bucket b and H(b - 1) its start (for the round's
    //     first bucket that is the end of the previous round's last one, rs)
    for (int q0 = threadIdx.x; q0 < cnt; q0 += stride) {
      uint2 wd[kB];
#pragma unroll
      for (int u = 0; u < kB; ++u) {
        const int q = q0 + u * blockDim.x;
        wd[u] = q < cnt ? stage[rs + q] : make_uint2(0u, 0u);
      }
#pragma unroll
      for (int u = 0; u < kB; ++u) {
        const int q = q0 + u * blockDim.x;
        if (q < cnt) {
          const int b = bucket_of(wd[u].y, b0);
          const int sl = (atomicAdd(&hist[b], 1) & kPosMask) - rs;
          if ((unsigned)sl < (unsigned)cnt) slots[sl] = wd[u];   // always true: the counts of pass (1)
        }
      }
    }
    if (threadIdx.x == 0) *nbig = 0;
    __syncthreads();
    // the scratch lines read so far, whole 128-byte lines inside this
    // period's row, are dropped from L2 without being written back
    {
      const uintptr_t row0 = ((uintptr_t)stage + 127) & ~(uintptr_t)127;
      const uintptr_t lo = max(row0, (uintptr_t)(stage + rs) & ~(uintptr_t)127);
      const uintptr_t hi = (uintptr_t)(stage + rs + cnt) & ~(uintptr_t)127;
      for (uintptr_t a = lo + (uintptr_t)threadIdx.x * 128; a < hi; a += (uintptr_t)blockDim.x * 128)
        asm volatile("discard.global.L2 [%0], 128;" ::"l"(a) : "memory");
    }
    // (b) ranks: the entry of sorted position p and original sample i puts
    //     i, clamped so that a malformed input can never address outside the
    //     curve, at ord[p].  Buckets of more than kSmallBucketSm entries are
    //     listed and ranked by whole warps (unless the list overflows); every
    //     other slot by its own thread.
    for (int b = b0 + (int)threadIdx.x; b < b1; b += blockDim.x) {
      const int k = H(b) - (b == 0 ? 0 : H(b - 1));
      if (k > kSmallBucketSm) {
        const int q = atomicAdd(nbig, 1);
        if (q < kBigBuckets) big[q] = b;
      }
    }
    __syncthreads();
    const int nbg = *nbig;
    const bool warp_ranked = nbg <= kBigBuckets;
    auto emit = [&](int q, int i) { ord[rs + q] = min(max(i, 0), n - 1); };
    if (warp_ranked)
      for (int q = wid; q < nbg; q += nwarp) {
        const int b = big[q];
        sort_bucket_warp(slots, (b == 0 ? 0 : H(b - 1)) - rs, H(b) - rs, b, nb_log2, ib, (unsigned)b << ib, t, P, emit);
      }
    if (warp_ranked && nbg > 0) __syncthreads();   // the sorted slots' index words are back
    for (int j0 = threadIdx.x; j0 < cnt; j0 += stride) {
      int pos[kB], idx[kB];
#pragma unroll
      for (int u = 0; u < kB; ++u) {
        const int j = j0 + u * blockDim.x;
        pos[u] = -1;
        idx[u] = 0;
        if (j < cnt) {
          const uint2 sj = slots[j];
          const int b = bucket_of(sj.y, b0);
          const int s = (b == 0 ? 0 : H(b - 1)) - rs;
          const int e = H(b) - rs;
          idx[u] = (int)(sj.y & imask);
          if (e - s == 1) {
            pos[u] = j;
          } else if (e - s <= kSmallBucketSm || !warp_ranked) {
            // entries of smaller key, and of equal key (itself included);
            // equal keys, rare, are then ordered on the exact phases
            const unsigned kj = sj.x;
            int lt = 0, eq = 0;
#pragma unroll 4
            for (int m = s; m < e; ++m) {
              const unsigned km = slots[m].x;
              lt += km < kj;
              eq += km == kj;
            }
            if (eq > 1)
              for (int m = s; m < e; ++m)
                if (m != j && slots[m].x == kj) lt += slot_less(slots[m], sj, t, P, imask);
            pos[u] = s + lt;
          }
        }
      }
#pragma unroll
      for (int u = 0; u < kB; ++u)
        if (pos[u] >= 0) emit(pos[u], idx[u]);
    }
    __syncthreads();
  }
  return true;
}

// The stable fold order of each period: order[slot_off + local * n + p] = the
// original index of sorted position p.  kThreads: kPrepThreads (one CTA per
// SM), or kPrepThreadsSmall for curves of at most kPrepSmallMaxN samples
// (two CTAs per SM, each with half the shared memory: the barriers of one
// overlap the other's work, which pays on short curves).
template <typename Real, int kThreads = kPrepThreads>
__global__ void __launch_bounds__(kThreads, kPrepThreads / kThreads)
prepare_kernel(const CurveDev<Real>* __restrict__ cds, const Run* __restrict__ runs, int nruns,
               uint2* __restrict__ scr_slot, int* __restrict__ order, int* __restrict__ tau = nullptr,
               bool late = false) {
  extern __shared__ int hist[];
  __shared__ int wtmp_i[32];
  __shared__ int big[kBigBuckets];
  __shared__ int nbig;
  const int item = blockIdx.x;
  if (tau && threadIdx.x == 0) tau[item] = 0x7f800000;   // infinity: the chi2 kernel's first bound
  const int ri = upper_find(0, nruns, item, [&](int i) { return (long long)runs[i].item0; });
  const Run& R = runs[ri];
  const CurveDev<Real>& C = cds[R.curve];
  const int local = item - R.item0;
  if (late && !C.late[R.pidx0 + local]) return;   // only the periods whose lists ran over
  if (tau && !late && threadIdx.x == 0) C.late[R.pidx0 + local] = 0;
  const double* __restrict__ t = C.t;
  const int n = C.n;
  const int nb_log2 = C.nb_log2;
  const int nb = 1 << nb_log2;
  const bool packed = n <= kPackedMaxN && nb_log2 <= 32 - kPackedShift;
  const unsigned imask = packed ? (unsigned)(kPackedMaxN - 1) : 0xffffffffu;
  const double P = C.periods[R.pidx0 + local];
  uint2* slot = scr_slot + R.slot_off - runs[0].slot_off + (size_t)local * n;
  int* ord = order + R.slot_off + (size_t)local * n;
  constexpr int kB = 3;   // elements per thread in flight in each pass (2 and 4: 5% slower, short curves 8%)
  const int stride = blockDim.x * kB;
  __shared__ RoundTables rt;
  if (C.rnb_log2 > 0) {
    const bool done =
        n <= kPackedMaxN
            ? prepare_rounds<kPackedShift>(hist, wtmp_i, big, &nbig, rt, t, n, P, C.rnb_log2, C.rcap, slot, ord)
            : prepare_rounds<0>(hist, wtmp_i, big, &nbig, rt, t, n, P, C.rnb_log2, C.rcap, slot, ord);
    if (done) return;
  }
  // global path: buckets scattered through the scratch row

  for (int b = threadIdx.x; b < nb; b += blockDim.x) hist[b] = 0;
  if (threadIdx.x == 0) nbig = 0;
  const FoldKey fold(P, nb_log2);
  __syncthreads();
  // (1) fold and histogram of buckets
  for (int i0 = threadIdx.x; i0 < n; i0 += stride) {
    double tv[kB];
#pragma unroll
    for (int u = 0; u < kB; ++u) {
      const int i = i0 + u * blockDim.x;
      tv[u] = i < n ? t[i] : P;   // (a padding of 0 would take the divide)
    }
    uint2 wd[kB];
    fold(tv, wd);
#pragma unroll
    for (int u = 0; u < kB; ++u) {
      const int i = i0 + u * blockDim.x;
      if (i < n) atomicAdd(&hist[wd[u].y], 1);
    }
  }
  __syncthreads();
  block_exclusive_scan_smem(hist, nb, wtmp_i);
  // (2) scatter (in-bucket key, index) into bucket slots; afterwards hist[b]
  //     is the end of bucket b and hist[b-1] its start
  for (int i0 = threadIdx.x; i0 < n; i0 += stride) {
    double tv[kB];
#pragma unroll
    for (int u = 0; u < kB; ++u) {
      const int i = i0 + u * blockDim.x;
      tv[u] = i < n ? t[i] : P;   // (a padding of 0 would take the divide)
    }
    uint2 wd[kB];
    fold(tv, wd);
#pragma unroll
    for (int u = 0; u < kB; ++u) {
      const int i = i0 + u * blockDim.x;
      if (i < n) {
        const uint2 at = wd[u];
        const int b = (int)at.y;
        const int s = atomicAdd(&hist[b], 1);
        slot[s] = make_uint2(at.x, (unsigned)i | (packed ? (unsigned)b << kPackedShift : 0u));
      }
    }
  }
  __syncthreads();
  // (3) ranking within buckets: the entry of sorted position p and original
  //     sample i puts i, clamped as above, at ord[p].
  auto emit = [&](int p, int i) { ord[p] = min(max(i, 0), n - 1); };
  //     (a) buckets of more than kSmallBucket entries (clustered phases, as
  //         when the period is close to a multiple of a regular cadence) are
  //         listed, from the shared-memory counts alone;
  for (int b = threadIdx.x; b < nb; b += blockDim.x) {
    const int k = hist[b] - (b == 0 ? 0 : hist[b - 1]);
    if (k > kSmallBucket) {
      const int q = atomicAdd(&nbig, 1);
      if (q < kBigBuckets) big[q] = b;
    }
  }
  __syncthreads();
  //     (b) whole warps rank the listed buckets (unless the list overflowed);
  const bool warp_ranked = nbig <= kBigBuckets;
  if (warp_ranked)
    for (int q = (int)(threadIdx.x >> 5); q < nbig; q += (int)(blockDim.x >> 5)) {
      const int b = big[q];
      rank_bucket_warp(slot, b == 0 ? 0 : hist[b - 1], hist[b], t, P, imask, emit);
    }
  //     (c) every other entry is ranked by its own thread: coalesced over the
  //         slots, its bucket read from the slot word (packed) or found by
  //         binary search of the bucket ends (the emitted positions are then
  //         close to the slot index, so the record writes stay nearly
  //         coalesced).
  for (int i0 = threadIdx.x; i0 < n; i0 += stride) {
#pragma unroll
    for (int u = 0; u < kB; ++u) {
      const int j = i0 + u * blockDim.x;
      if (j < n) {
        const uint2 sj = slot[j];
        int lo;
        if (packed) {
          lo = (int)(sj.y >> kPackedShift);
        } else {
          lo = 0;
          int hi = nb - 1;
          while (lo < hi) {
            const int mid = (lo + hi) >> 1;
            if (hist[mid] > j) hi = mid;
            else lo = mid + 1;
          }
        }
        const int s = lo == 0 ? 0 : hist[lo - 1];
        const int e = hist[lo];
        if (e - s == 1) {
          emit(j, (int)(sj.y & imask));
        } else if (e - s <= kSmallBucket || !warp_ranked) {
          int r = 0;
          for (int m = s; m < e; ++m)
            if (m != j) r += slot_less(slot[m], sj, t, P, imask);
          emit(s + r, (int)(sj.y & imask));
        }
      }
    }
  }
}

}  // namespace gtls

#include "chi2.cuh"

namespace gtls {

template <typename Real>
__global__ void finish_kernel(const CurveDev<Real>* __restrict__ cds, const Run* __restrict__ runs, int nruns,
                              int count, const double* __restrict__ part_v, const long long* __restrict__ part_loc,
                              bool late) {
  const int item = blockIdx.x * blockDim.x + threadIdx.x;
  if (item >= count) return;
  const int ri = upper_find(0, nruns, item, [&](int i) { return (long long)runs[i].item0; });
  const Run& R = runs[ri];
  const CurveDev<Real>& C = cds[R.curve];
  if (C.ntiles == 1) return;   // written by the chi2 kernel
  const int local = item - R.item0;
  const long long pg = R.pidx0 + local;
  if (late && !C.late[pg]) return;
  Best b{INFINITY, 0x7fffffffffffffffLL};
  if (C.union_cnt[pg / C.batch] == 0) {
    b.v = NAN;
    b.loc = -1;
  } else {
    const long long c0 = (long long)R.tile0 + (long long)local * C.ntiles;
    for (int i = 0; i < C.ntiles; ++i) best_update(b, part_v[c0 + i], part_loc[c0 + i]);
  }
  C.chi2_out[pg] = b.v;
  if (C.loc_out) C.loc_out[pg] = b.loc;
}

// ------------------------------------------------- durations, unions, rows
// durationsGrid (GPUFun.py:47-86) with the same operation order.
__device__ __forceinline__ void duration_range(double period_days, float span, int n, int* wmin, int* wmax) {
  const double kSecondsPerDay = 86400;
  const double kRsMin = 695508000 * 0.05, kRsMax = 695508000 * 4.0;
  const double kRjup = 69911000;
  float length = span;
  double nt = length / period_days;
  double corr = (nt + 1.0) / nt;
  double ps = period_days * kSecondsPerDay;
  double fmin = (4.0 * ps) / (20848 * 1000000000000000.0);
  double fmax = (4.0 * ps) / (416970 * 1000000000000000.0);
  double t14min = kRsMin * pow(fmin, 1.0 / 3.0);
  double t14max = (kRsMax + kRjup * 2.0) * pow(fmax, 1.0 / 3.0);
  double dmin = t14min / ps;
  double dmax = t14max / ps;
  dmin = dmin > 0.15 ? 0.15 : dmin;
  dmax = dmax > 0.15 ? 0.15 : dmax;
  *wmin = (int)floor(dmin * n);
  *wmax = (int)ceil(dmax * n * corr);
}

__global__ void duration_range_kernel(const double* __restrict__ periods, long long np, float span, int n,
                                      int* __restrict__ wmin, int* __restrict__ wmax) {
  long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  if (i >= np) return;
  duration_range(periods[i], span, n, &wmin[i], &wmax[i]);
}

// The ascending list of durations valid for at least one period of union
// batch b of the curve (durationsGrid and durationBool GPUFun.py:47-105,
// OR-ed as core.py:704-716).  Widths ascend, so a period's valid ones are a run:
// its ends are counted up and down, and a duration is in the union where the
// running count is not 0.
template <typename Real>
__device__ void duration_union(const CurveDev<Real>& C, long long b, int all_durations) {
  __shared__ int edge[GTLS_MAX_DURATIONS + 1];
  const int D = C.D;
  const long long p0 = b * C.batch;
  const long long p1 = min(C.np, p0 + C.batch);
  for (int d = threadIdx.x; d <= D; d += blockDim.x) edge[d] = 0;
  __syncthreads();
  const int* __restrict__ widths = C.widths;
  auto first_from = [&](int w) {   // first duration of at least w samples
    int lo = 0, hi = D;
    while (lo < hi) {
      const int mid = (lo + hi) >> 1;
      if (widths[mid] >= w) hi = mid;
      else lo = mid + 1;
    }
    return lo;
  };
  for (long long p = p0 + threadIdx.x; p < p1; p += blockDim.x) {
    int wmin = 0, wmax = INT32_MAX - 1;
    if (!all_durations) duration_range(C.periods[p], C.span, C.n, &wmin, &wmax);
    const int lo = first_from(wmin), hi = wmax == INT32_MAX ? D : first_from(wmax + 1);
    if (lo < hi) {
      atomicAdd(&edge[lo], 1);
      atomicAdd(&edge[hi], -1);
    }
  }
  __syncthreads();
  if (threadIdx.x < 32) {
    const int lane = threadIdx.x;
    int* ulist = C.union_list + b * D;
    int cnt = 0, open = 0;
    for (int d0 = 0; d0 < D; d0 += 32) {
      int run = d0 + lane < D ? edge[d0 + lane] : 0;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int y = __shfl_up_sync(0xffffffffu, run, o);
        if (lane >= o) run += y;
      }
      run += open;
      const bool in = d0 + lane < D && run > 0;
      const unsigned m = __ballot_sync(0xffffffffu, in);
      if (in) ulist[cnt + __popc(m & ((1u << lane) - 1u))] = d0 + lane;
      cnt += __popc(m);
      open = __shfl_sync(0xffffffffu, run, 31);
    }
    if (lane == 0) C.union_cnt[b] = cnt;
  }
}

// Template rows as the exact sums read them, (s_i, s_i^2) for i < w_d, and the
// cells of the bounds (screen.cuh): a warp per cell, kTemplateParts CTAs per
// (duration, table).  A row's sums over its cells are added up in memory
// (their last bits depend on the order; the bounds leave room for more).
constexpr int kTemplateParts = 4;
template <typename Real>
__device__ void template_part(const CurveDev<Real>& C, int d, int table, int part) {
  const int w = C.widths[d];
  const double* __restrict__ T = C.templates + (size_t)d * C.max_width;
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, nwarp = blockDim.x >> 5;
  if (table == 0) {
    typename Tr<Real>::R2* row = C.trows + C.trow_off[d];
    for (int i = part * blockDim.x + threadIdx.x; i < w; i += kTemplateParts * blockDim.x) {
      const double sv = T[i];
      typename Tr<Real>::R2 o;
      o.x = (Real)sv;
      o.y = (Real)(sv * sv);
      row[i] = o;
    }
  }
  ScreenRow& row = C.srows[2 * d + table];
  const int first = row.first, m = row.m;   // set by the host, the sums to 0
  const int g = w <= kRingMaxW ? 1 : C.coarse;
  const int* __restrict__ ends = C.sends + first;
  auto at = [&](int i) { return i >= 0 && i < w ? T[i] : 0.0; };
  auto sum_over = [&](double x) { return warp_sum(x); };
  for (int q = part * nwarp + wid; q < m; q += kTemplateParts * nwarp) {
    const int e0 = (q > 0 ? ends[q - 1] : 0) * g, e1 = ends[q] * g, l = e1 - e0;
    // mean of the template over the cell for a window that starts with the
    // cells, and g - 1 samples after them (coarse rows): the line between is a + b offset
    double s0 = 0.0, s1 = 0.0;
#pragma unroll 4
    for (int x = e0 + lane; x < e1; x += 32) {
      s0 += at(x);
      s1 += at(x - (g - 1));
    }
    const double mean0 = sum_over(s0) / l, mean1 = sum_over(s1) / l;
    const float a = (float)mean0, b = g > 1 ? (float)((mean0 - mean1) / (g - 1)) : 0.f;
    double rc2 = 0.0, rb = 0.0, mn = INFINITY, mx = 0.0;
    if (g == 1) {
      double s2 = 0.0;
      for (int x = e0 + lane; x < e1; x += 32) {
        const double r = at(x) - (double)a, sq = at(x) * at(x);
        s2 += r * r;
        mn = fmin(mn, sq);
        mx = fmax(mx, sq);
      }
      rc2 = sum_over(s2);                    // about a, so at least the centred square
      rb = fabs(mean0 - (double)a);          // the mean's rounding
    } else {
      for (int off = lane; off < g; off += 32) {   // a lane per offset of the window's start in its first step
        const double ae = (double)a - (double)b * off;
        double r1 = 0.0, r2 = 0.0;
#pragma unroll 8
        for (int x = e0 - off; x < e1 - off; ++x) {
          const double s = at(x), r = s - ae, sq = s * s;
          r1 += r;
          r2 += r * r;
          mn = fmin(mn, sq);
          mx = fmax(mx, sq);
        }
        rc2 = fmax(rc2, fmax(r2 - r1 * r1 / l, 0.0) + 1e-14 * r2);
        rb = fmax(rb, fabs(r1 / l));
      }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      rc2 = fmax(rc2, __shfl_xor_sync(0xffffffffu, rc2, o));
      rb = fmax(rb, __shfl_xor_sync(0xffffffffu, rb, o));
      mn = fmin(mn, __shfl_xor_sync(0xffffffffu, mn, o));
      mx = fmax(mx, __shfl_xor_sync(0xffffffffu, mx, o));
    }
    if (lane == 0) {
      ScreenCell cell;
      cell.a = a;
      cell.b = b;
      cell.rc = (float)(sqrt(rc2) * 1.000001);
      cell.rb = (float)(rb * 1.000001);
      cell.mn = (float)mn;
      cell.mx = table == 0 ? __int_as_float(ends[q]) : (float)mx;   // the first table has no use for it
      cell.l = (float)l;
      cell.inv_l = (float)(1.0 / l * (1.0 - 0x1p-10));
      C.scells[first + q] = cell;
      atomicAdd(&row.asum, (float)((fabs((double)a) + fabs((double)b) * (g - 1) + rb) * 1.0001));
      atomicAdd(&row.smn, (float)mn);
      atomicAdd(&row.smx, (float)(mx * 1.0001));
      atomicAdd(&row.lmn, (float)(mn * l));
      atomicAdd(&row.lmx, (float)(mx * l));
    }
  }
  if (part == 0 && wid == 0) {
    double t2 = 0.0;
#pragma unroll 8
    for (int i = lane; i < w; i += 32) t2 += T[i] * T[i];
    t2 = sum_over(t2);
    if (lane == 0) {
      row.inv_w = (float)(1.0 / w);
      row.os2 = (float)(2.0 * C.overshoot[d]);
      row.tn = (float)(sqrt(t2) * 1.000001);
      row.t2 = (float)t2;
    }
  }
}

// Everything a search prepares before its periods, in one launch: the CTAs of
// the curves' set-up, of the unions, and of the templates (five launches one
// after the other took 36 us on a 1,499-sample curve).
struct SetupArgs {
  const int* blk_off;        // [n_curves + 1] set-up CTAs of the curves
  const long long* b_off;    // [n_curves + 1] union batches
  const long long* d_off;    // [n_curves + 1] durations
  int n_curves, n_blk, all_durations;
  long long n_batch;
};
template <typename Real>
__global__ void __launch_bounds__(kSetupThreads) setup_kernel(const CurveDev<Real>* __restrict__ cds, SetupArgs a) {
  long long i = blockIdx.x;
  if (i < a.n_blk) {
    const int c = upper_find(0, a.n_curves, i, [&](int k) { return (long long)a.blk_off[k]; });
    curve_setup(cds[c], (int)i - a.blk_off[c], a.blk_off[c + 1] - a.blk_off[c]);
    return;
  }
  i -= a.n_blk;
  if (i < a.n_batch) {
    const int c = upper_find(0, a.n_curves, i, [&](int k) { return a.b_off[k]; });
    duration_union(cds[c], i - a.b_off[c], a.all_durations);
    return;
  }
  i -= a.n_batch;
  const int part = (int)(i % kTemplateParts), table = (int)(i / kTemplateParts & 1);
  i /= 2 * kTemplateParts;
  const int c = upper_find(0, a.n_curves, i, [&](int k) { return a.d_off[k]; });
  template_part(cds[c], (int)(i - a.d_off[c]), table, part);
}

// ------------------------------------------------------------------ host
static int nb_log2_for(int n, int shift) {
  int k = 1;
  while ((1 << k) < n) ++k;
  // at most 32768 buckets (128 KB of counters), 16384 in the two-per-SM shape
  k = std::min(n <= kPrepSmallMaxN ? 14 : 15, k + shift);
  return std::max(1, k);
}

// Shared-memory prepare path of a curve of n samples: NB = 2^(ceil(log2 n) -
// 2) buckets (at most 2^14, about four samples a bucket), and the largest
// round capacity that fits the CTA's shared memory next to them (8 bytes a
// sample: the slot word).  Off (0) for curves beyond kRoundMaxN (the words'
// scatter through global memory, 6.6 us a period of 160,000 samples, takes 2.9
// in rounds) or when fewer than 1,024 samples fit a round.
template <typename Real>
static void rounds_params(CurveDev<Real>& C, int smem_optin) {
  C.rnb_log2 = 0;
  C.rcap = 0;
  const int n = C.n;
  if (n < 1 || n > kRoundMaxN) return;
  int k = 1;
  while ((1 << k) < n) ++k;
  const int nbl = std::max(1, std::min(14, k - 2));
  // two CTAs per SM for short curves: each gets half the shared memory
  const long long budget = (n <= kPrepSmallMaxN ? smem_optin / 2 : smem_optin) - kPrepStaticSmem;
  const long long c = std::min<long long>((budget - (4LL << nbl)) / 8, n);
  if (c < 1024 && c < n) return;
  C.rnb_log2 = nbl;
  C.rcap = (int)c;
}
// Dynamic shared memory of prepare_kernel for a curve: the larger of the
// two paths' needs (a period falls back to the global path when its
// buckets do not fit the rounds).
template <typename Real>
static size_t prep_smem_bytes(const CurveDev<Real>& C) {
  size_t b = sizeof(int) << C.nb_log2;
  if (C.rnb_log2 > 0) b = std::max(b, (sizeof(int) << C.rnb_log2) + sizeof(uint2) * (size_t)C.rcap);
  return b;
}

// One light curve of a search, as the host sees it.
struct CurveHost {
  const double *t, *y, *dy, *periods;
  double* chi2_out;
  int64_t* loc_out;
  const int* widths;
  const double* overshoot;
  const double* templates;
  long long np;
  int n, D, max_width, batch;
  float span;
};

// Dynamic shared memory the kernels may ask for, set once per context.
template <typename Real>
static cudaError_t allow_smem(int optin) {
  const int chi = (int)kChiSmemMax;
  cudaError_t e = cudaSuccess;
  auto set = [&](auto* k, int bytes) {
    if (e == cudaSuccess) e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
  };
  set(prepare_kernel<Real>, optin - kPrepStaticSmem);
  set(prepare_kernel<Real, kPrepThreadsSmall>, optin - kPrepStaticSmem);
  set(chi2_kernel<Real, false>, chi);
  set(chi2_kernel<Real, false, true>, chi);
  set(chi2_kernel<Real, true>, chi);
  return e;
}

// Host copies of small arrays, gathered so that one copy takes them all to the
// start of the arena (each pageable copy costs the host 5 to 10 us).
struct Upload {
  std::vector<char> host;
  template <typename T>
  size_t add(const T* src, size_t count) {
    const size_t at = align_up(host.size(), 256);
    host.resize(at + count * sizeof(T));
    if (count) std::memcpy(host.data() + at, src, count * sizeof(T));
    return at;
  }
};

// Scratch of one period: slots and fold order, and per CTA a row of the prefix
// of v (curves with a coarse prefix), its list and its result; and the row.
static size_t v_stride(int tile, int max_width) {
  const int coarse = coarse_step(tile, max_width);
  return coarse > 0 ? ((size_t)tile + max_width + 2 * coarse + 8) / 8 * 8 : 0;
}
static size_t period_bytes(int n, int max_width, int tile, bool all) {
  const size_t ctas = ((size_t)n + tile - 1) / tile;
  return (size_t)n * (sizeof(uint2) + sizeof(int)) +
         ctas * (sizeof(float) * v_stride(tile, max_width) + list_entries(all) * sizeof(Waiting) + 16) + 4;
}

template <typename Real>
static int run_search(gtls_ctx* ctx, const CurveHost* ch, int n_curves, int precision_pass, int skip_point,
                      double depth_min, int flags, gtls_timing* tm, cudaStream_t st) {
  using R2 = typename Tr<Real>::R2;
  const bool all = precision_pass == GTLS_PASS_ALL;
  const size_t list_cap = list_entries(all);
  bool& allowed = sizeof(Real) == 8 ? ctx->smem_set_fp64 : ctx->smem_set_fp32;
  if (!allowed) {
    GTLS_TRY_CUDA(ctx, allow_smem<Real>(ctx->smem_optin));
    allowed = true;
  }

  // ---- the curves' widths
  std::vector<CurveDev<Real>> cd(n_curves);
  std::vector<long long> p_off(n_curves + 1, 0), b_off(n_curves + 1, 0), d_off(n_curves + 1, 0);
  std::vector<int> blk_off(n_curves + 1, 0);
  for (int c = 0; c < n_curves; ++c) d_off[c + 1] = d_off[c] + ch[c].D;
  const size_t d_total = (size_t)d_off[n_curves];
  std::vector<int> widths(d_total);
  for (int c = 0, c1; c < n_curves; c = c1) {   // runs of curves whose arrays follow one another: one copy
    for (c1 = c + 1; c1 < n_curves && ch[c1].widths == ch[c].widths + (d_off[c1] - d_off[c]); ++c1) {}
    GTLS_TRY_CUDA(ctx, cudaMemcpyAsync(widths.data() + d_off[c], ch[c].widths, sizeof(int) * (d_off[c1] - d_off[c]),
                                       cudaMemcpyDeviceToHost, st));
  }
  GTLS_TRY_CUDA(ctx, cudaStreamSynchronize(st));

  // ---- ranges of starts per chi2 CTA.  The whole period, unless widths that
  // the ring does not hold would make the coarse prefix coarser than
  // kCoarseStep samples, or the caller set a cap.
  const int cap_default = sizeof(Real) == 4 ? kTileCapFp32 : kTileCapFp64;
  const int cap = sizeof(Real) == 4 ? ctx->tile_cap_fp32 : ctx->tile_cap_fp64;
  long long ctas = 0, np_total = 0;
  for (int c = 0; c < n_curves; ++c) {
    const CurveHost& h = ch[c];
    long long tile = std::min(h.n, 1 << 26);   // the blocks of the all-starts pass are numbered in 31 bits
    if (h.max_width > kRingMaxW)
      tile = std::max<long long>(kCoarseStep * (kCoarseCap - 8) - h.max_width, 4LL * h.max_width);
    // the all-starts pass screens 8 or more times as many starts: shorter
    // ranges even out its CTAs (600 of a whole period's third each, two to an SM, are three rounds)
    if (all) tile = std::min<long long>(tile, std::max(8192, h.max_width));
    if (cap != cap_default) tile = std::min<long long>(tile, cap);
    cd[c].ntiles = (int)((h.n + tile - 1) / tile);
    ctas += h.np * cd[c].ntiles;
    np_total += h.np;
  }
  // small searches (the candidates, the harmonics, the best period): narrower
  // ranges, so that the launch still fills the SMs (two CTAs each; aiming at two
  // waves took 30% longer on 350 periods of 1,499 samples; a start's value does
  // not depend on the range it is in)
  const long long want = 2LL * ctx->num_sms;
  // Rounded down, a few CTAs past one wave being a second one (59 periods of
  // 20,658 samples at every start 2.33 -> 2.01 ms, 129 of 2,684 0.216 -> 0.191); up for every start of long
  // curves in FP32, whose time is that of the range around the peak (22 periods of
  // 108,452 samples 24.9 ms, rounded down 30.2).
  bool peaked = false;
  for (int c = 0; c < n_curves; ++c) peaked = peaked || (all && sizeof(Real) == 4 && ch[c].max_width > kRingMaxW);
  const long long per = np_total > 0 && ctas < want ? std::max<long long>(1, (want + (peaked ? np_total - 1 : 0)) / np_total) : 1;
  for (int c = 0; c < n_curves; ++c) {
    const long long tiles = std::max<long long>(cd[c].ntiles, std::min<long long>(per, (ch[c].n + 511) / 512));
    long long tile = ((ch[c].n + tiles - 1) / tiles + 31) / 32 * 32;
    // A period that does not fit the scratch budget so is cut into fewer
    // ranges; as one range it takes less than the budget it is refused under (below).
    const long long widest = std::min<long long>(((long long)ch[c].n + 31) / 32 * 32, all ? kBlockTable * kBlockStarts : 1 << 26);
    while (tile < widest && period_bytes(ch[c].n, ch[c].max_width, (int)tile, all) > ctx->chunk_budget)
      tile = std::min(widest, 2 * tile);
    cd[c].tile = (int)tile;
    cd[c].ntiles = (int)((ch[c].n + tile - 1) / tile);
  }

  // ---- per-curve layout on the host
  std::vector<int> skips(d_total), trow_off(d_total), ends;
  std::vector<ScreenRow> srows(2 * d_total);
  std::vector<size_t> cell_off(n_curves + 1, 0), row_off(n_curves + 1, 0);
  for (int c = 0; c < n_curves; ++c) {
    const CurveHost& h = ch[c];
    const int n = h.n, D = h.D, maxd = h.max_width;
    CurveDev<Real>& C = cd[c];
    const int* hw = widths.data() + d_off[c];
    size_t rows = 0, cells = (size_t)D * kLaneCells;
    C.coarse = coarse_step(C.tile, maxd);
    for (int i = 0; i < D; ++i) {
      const int w = hw[i];
      if (w < 1 || w > maxd || (i > 0 && w <= hw[i - 1]))
        return fail(ctx, GTLS_E_INVALID, "widths must be ascending, >= 1 and <= max_width");
      skips[d_off[c] + i] = (!all && w > skip_point) ? w / skip_point : 1;
      trow_off[d_off[c] + i] = (int)rows;
      rows += w;
      const int g = w <= kRingMaxW ? 1 : C.coarse;
      // the two tables of cells: the first kLaneCells apart, the second after them
      for (int k = 0; k < 2; ++k) {
        std::vector<int> e;
        screen_cells(w, g, k == 0, e);
        ScreenRow r = {};
        r.first = k == 0 ? i * kLaneCells : (int)cells;
        r.m = (int)e.size();
        srows[2 * (d_off[c] + i) + k] = r;
        if (k == 1) cells += e.size();
        ends.resize(cell_off[c] + cells);
        std::copy(e.begin(), e.end(), ends.begin() + cell_off[c] + r.first);
      }
    }
    if (maxd > 0xffff) return fail(ctx, GTLS_E_RANGE, "max_width above 65535");
    cell_off[c + 1] = ends.size();
    row_off[c + 1] = row_off[c] + rows;
    C.t = h.t;
    C.y = h.y;
    C.dy = h.dy;
    C.periods = h.periods;
    C.chi2_out = h.chi2_out;
    C.loc_out = h.loc_out;
    C.widths = h.widths;
    C.overshoot = h.overshoot;
    C.templates = h.templates;
    C.np = h.np;
    C.n = n;
    C.maxd = maxd;
    C.D = D;
    C.max_width = maxd;
    C.batch = h.batch;
    C.nbatch = (int)((h.np + h.batch - 1) / h.batch);
    C.vstride = (int)v_stride(C.tile, maxd);
    C.nb_log2 = nb_log2_for(n, ctx->bucket_shift);
    rounds_params(C, ctx->smem_optin);
    C.span = h.span;
    p_off[c + 1] = p_off[c] + h.np;
    b_off[c + 1] = b_off[c] + C.nbatch;
    blk_off[c + 1] = blk_off[c] + (n + kSetupItems - 1) / kSetupItems;
  }

  // ---- chunks of the period list (curve after curve) and their runs
  const size_t budget = ctx->chunk_budget;
  std::vector<Run> runs;
  std::vector<int> chunk_r0, chunk_items, chunk_tiles;
  std::vector<size_t> chunk_smem_prep, chunk_smem_chi;
  std::vector<int> chunk_small;    // per chunk: all its curves take the two-per-SM prepare shape
  size_t max_slot = 0, max_v = 0, max_part = 0, max_items = 0;
  {
    size_t slot = 0, vs = 0, bytes = 0;
    int items = 0, tiles = 0;
    size_t sm_prep = 0, sm_chi = 0;
    int mode = -1;
    chunk_r0.push_back(0);
    auto close_chunk = [&]() {
      if (items == 0) return;
      chunk_small.push_back(mode);
      chunk_items.push_back(items);
      chunk_tiles.push_back(tiles);
      chunk_smem_prep.push_back(sm_prep);
      chunk_smem_chi.push_back(sm_chi);
      max_slot = std::max(max_slot, slot);
      max_v = std::max(max_v, vs);
      max_part = std::max(max_part, (size_t)tiles);
      max_items = std::max(max_items, (size_t)items);
      chunk_r0.push_back((int)runs.size());
      slot = vs = bytes = 0;
      items = tiles = 0;
      sm_prep = sm_chi = 0;
      mode = -1;
    };
    for (int c = 0; c < n_curves; ++c) {
      const CurveDev<Real>& C = cd[c];
      const size_t per = period_bytes(C.n, C.maxd, C.tile, all);
      // the smallest budget a period is accepted with (as documented)
      const size_t least = (size_t)C.n * 8 + (size_t)(C.n + C.maxd + 1) * (sizeof(R2) + 8);
      long long p = 0;
      // one prepare shape per chunk
      const int cmode = C.n <= kPrepSmallMaxN ? 1 : 0;
      if (C.np > 0 && mode != -1 && mode != cmode) close_chunk();
      while (p < C.np) {
        long long fit = (long long)((budget > bytes ? budget - bytes : 0) / per);
        if (budget < least) fit = 0;
        fit = std::min<long long>(fit, (long long)INT32_MAX - items);
        fit = std::min<long long>(fit, ((1LL << 31) - 1 - tiles) / C.ntiles);
        if (fit <= 0) {
          if (items == 0) return fail(ctx, GTLS_E_RANGE, "one period does not fit the scratch budget");
          close_chunk();
          continue;
        }
        const long long take = std::min<long long>(fit, C.np - p);
        Run r;
        r.curve = c;
        r.item0 = items;
        r.count = (int)take;
        r.tile0 = tiles;
        r.pidx0 = p;
        r.slot_off = (long long)slot;
        r.v_off = (long long)vs;
        runs.push_back(r);
        slot += (size_t)take * C.n;
        vs += (size_t)take * C.ntiles * C.vstride;
        bytes += (size_t)take * per;
        items += (int)take;
        tiles += (int)(take * C.ntiles);
        sm_prep = std::max(sm_prep, prep_smem_bytes(C));
        sm_chi = std::max(sm_chi, chi2_smem_bytes(C.coarse > 0, C.D));
        mode = cmode;
        p += take;
      }
    }
    close_chunk();
  }
  const int nchunks = (int)chunk_items.size();

  // ---- arena: the uploaded arrays, per-curve buffers, and one chunk of scratch
  Upload up;
  const size_t at_cd = up.add((const CurveDev<Real>*)cd.data(), n_curves);   // filled in below
  const size_t at_runs = up.add(runs.data(), runs.size());
  const size_t at_boff = up.add(b_off.data(), b_off.size());
  const size_t at_doff = up.add(d_off.data(), d_off.size());
  const size_t at_blk = up.add(blk_off.data(), blk_off.size());
  const size_t at_skips = up.add(skips.data(), skips.size());
  const size_t at_trow = up.add(trow_off.data(), trow_off.size());
  const size_t at_ends = up.add(ends.data(), ends.size());
  const size_t at_srows = up.add(srows.data(), srows.size());
  const std::vector<int> zeros(n_curves, 0);
  const size_t at_arrived = up.add(zeros.data(), zeros.size());
  size_t total = up.host.size();
  for (int c = 0; c < n_curves; ++c) {
    const CurveDev<Real>& C = cd[c];
    carve_size<double2>(total, C.n);
    carve_size<CurveConst>(total, 1);
    carve_size<double>(total, (size_t)(blk_off[c + 1] - blk_off[c]) * kSetupSums);
    carve_size<int>(total, (size_t)C.nbatch);
    carve_size<int>(total, (size_t)C.nbatch * C.D);
    carve_size<int>(total, (size_t)C.np);
  }
  carve_size<R2>(total, row_off[n_curves]);
  carve_size<ScreenCell>(total, ends.size());
  carve_size<uint2>(total, max_slot);
  carve_size<int>(total, max_slot);
  carve_size<float>(total, max_v);
  carve_size<double>(total, max_part);
  carve_size<long long>(total, max_part);
  carve_size<Waiting>(total, max_part * list_cap);
  carve_size<int>(total, max_items);
  carve_size<unsigned long long>(total, 2);
  total += 32 * 256;
  void* mem = arena(ctx, total);
  if (!mem) return fail(ctx, GTLS_E_NOMEM, "scratch allocation failed");
  char* base = static_cast<char*>(mem);
  Carver cv(mem);
  cv.take<char>(up.host.size());
  for (int c = 0; c < n_curves; ++c) {
    CurveDev<Real>& C = cd[c];
    C.vw = cv.take<double2>(C.n);
    C.cst = cv.take<CurveConst>(1);
    C.sums = cv.take<double>((size_t)(blk_off[c + 1] - blk_off[c]) * kSetupSums);
    C.arrived = reinterpret_cast<int*>(base + at_arrived) + c;
    C.union_cnt = cv.take<int>(C.nbatch);
    C.union_list = cv.take<int>((size_t)C.nbatch * C.D);
    C.late = cv.take<int>((size_t)C.np);
    C.skips = reinterpret_cast<const int*>(base + at_skips) + d_off[c];
    C.trow_off = reinterpret_cast<const int*>(base + at_trow) + d_off[c];
    C.sends = reinterpret_cast<const int*>(base + at_ends) + cell_off[c];
    C.srows = reinterpret_cast<ScreenRow*>(base + at_srows) + 2 * d_off[c];
  }
  R2* trows = cv.take<R2>(row_off[n_curves]);
  ScreenCell* scells = cv.take<ScreenCell>(ends.size());
  for (int c = 0; c < n_curves; ++c) {
    cd[c].trows = trows + row_off[c];
    cd[c].scells = scells + cell_off[c];
  }
  uint2* scr_slot = cv.take<uint2>(max_slot);
  int* order = cv.take<int>(max_slot);
  float* vpre = cv.take<float>(max_v);
  double* part_v = cv.take<double>(max_part);
  long long* part_loc = cv.take<long long>(max_part);
  Waiting* list = cv.take<Waiting>(max_part * list_cap);
  int* tau = cv.take<int>(max_items);
  unsigned long long* work = cv.take<unsigned long long>(2);
  std::memcpy(up.host.data() + at_cd, cd.data(), sizeof(CurveDev<Real>) * n_curves);
  GTLS_TRY_CUDA(ctx, cudaMemcpyAsync(base, up.host.data(), up.host.size(), cudaMemcpyHostToDevice, st));
  const CurveDev<Real>* d_cd = reinterpret_cast<const CurveDev<Real>*>(base + at_cd);
  const Run* d_runs = reinterpret_cast<const Run*>(base + at_runs);
  // ---- optional stage timing with CUDA events on the call's stream
  cudaEvent_t ev[2] = {nullptr, nullptr};
  std::vector<cudaEvent_t> evc;
  if (tm) {
    std::memset(tm, 0, sizeof(*tm));
    for (auto& e : ev) GTLS_TRY_CUDA(ctx, cudaEventCreate(&e));
    GTLS_TRY_CUDA(ctx, cudaEventRecord(ev[0], st));
    GTLS_TRY_CUDA(ctx, cudaMemsetAsync(work, 0, 2 * sizeof(unsigned long long), st));
  }
  SetupArgs sa;
  sa.blk_off = reinterpret_cast<const int*>(base + at_blk);
  sa.b_off = reinterpret_cast<const long long*>(base + at_boff);
  sa.d_off = reinterpret_cast<const long long*>(base + at_doff);
  sa.n_curves = n_curves;
  sa.n_blk = blk_off[n_curves];
  sa.all_durations = (flags & GTLS_SEARCH_ALL_DURATIONS) ? 1 : 0;
  sa.n_batch = b_off[n_curves];
  const long long setup_ctas = sa.n_blk + sa.n_batch + 2LL * kTemplateParts * d_off[n_curves];
  if (setup_ctas > INT32_MAX) return fail(ctx, GTLS_E_RANGE, "too many periods, samples and durations in one call");
  setup_kernel<Real><<<(unsigned)setup_ctas, kSetupThreads, 0, st>>>(d_cd, sa);
  ctx->launches += 1;
  GTLS_TRY_CUDA(ctx, cudaGetLastError());
  if (tm) GTLS_TRY_CUDA(ctx, cudaEventRecord(ev[1], st));

  Chi2Args ca;
  ca.depth_min = depth_min;
  ca.vpre = vpre;
  ca.list = list;
  ca.tau = tau;
  ca.part_v = part_v;
  ca.part_loc = part_loc;
  ca.work = tm ? work : nullptr;
  ca.any_late = ctx->any_late;
  *ctx->any_late = 0;
  auto run_chunks = [&](bool late) -> int {
    for (int k = 0; k < nchunks; ++k) {
      const int r0 = chunk_r0[k], nr = chunk_r0[k + 1] - r0;
      const int items = chunk_items[k], tiles = chunk_tiles[k];
      cudaEvent_t e3[4];
      if (tm) {
        for (auto& e : e3) GTLS_TRY_CUDA(ctx, cudaEventCreate(&e));
        GTLS_TRY_CUDA(ctx, cudaEventRecord(e3[0], st));
      }
      if (chunk_small[k])
        prepare_kernel<Real, kPrepThreadsSmall><<<items, kPrepThreadsSmall, chunk_smem_prep[k], st>>>(
            d_cd, d_runs + r0, nr, scr_slot, order, tau, late);
      else
        prepare_kernel<Real><<<items, kPrepThreads, chunk_smem_prep[k], st>>>(d_cd, d_runs + r0, nr, scr_slot, order,
                                                                               tau, late);
      if (tm) GTLS_TRY_CUDA(ctx, cudaEventRecord(e3[1], st));
      ca.nruns = nr;
      if (all)
        chi2_kernel<Real, true><<<tiles, kChiThreads, chunk_smem_chi[k], st>>>(d_cd, d_runs + r0, order, ca);
      else if (late)
        chi2_kernel<Real, false, true><<<tiles, kChiThreads, chunk_smem_chi[k], st>>>(d_cd, d_runs + r0, order, ca);
      else
        chi2_kernel<Real, false><<<tiles, kChiThreads, chunk_smem_chi[k], st>>>(d_cd, d_runs + r0, order, ca);
      if (tm) GTLS_TRY_CUDA(ctx, cudaEventRecord(e3[2], st));
      if (tiles > items) {   // some periods are split
        finish_kernel<Real><<<(items + 127) / 128, 128, 0, st>>>(d_cd, d_runs + r0, nr, items, part_v, part_loc,
                                                                late);
        ctx->launches += 1;
      }
      if (tm) {
        GTLS_TRY_CUDA(ctx, cudaEventRecord(e3[3], st));
        for (auto& e : e3) evc.push_back(e);
      }
      ctx->launches += 2;
      GTLS_TRY_CUDA(ctx, cudaGetLastError());
    }
    GTLS_TRY_CUDA(ctx, cudaStreamSynchronize(st));
    return GTLS_OK;
  };
  int rc = run_chunks(false);
  if (rc == GTLS_OK && *static_cast<volatile int*>(ctx->any_late)) rc = run_chunks(true);   // the marked periods alone
  if (rc != GTLS_OK) return rc;
  if (tm) {
    float ms = 0;
    GTLS_TRY_CUDA(ctx, cudaEventElapsedTime(&ms, ev[0], ev[1]));
    tm->setup_ms = ms;
    for (size_t i = 0; i < evc.size(); i += 4) {
      GTLS_TRY_CUDA(ctx, cudaEventElapsedTime(&ms, evc[i], evc[i + 1]));
      tm->prepare_ms += ms;
      GTLS_TRY_CUDA(ctx, cudaEventElapsedTime(&ms, evc[i + 1], evc[i + 2]));
      tm->chi2_ms += ms;
      GTLS_TRY_CUDA(ctx, cudaEventElapsedTime(&ms, evc[i + 2], evc[i + 3]));
      tm->finish_ms += ms;
    }
    tm->chunks = nchunks;
    for (auto e : evc) cudaEventDestroy(e);
    for (auto e : ev) cudaEventDestroy(e);
    // work counters of the chi2 kernel, from the unions the kernel used
    long long starts = 0, fma = 0;
    for (int c = 0; c < n_curves; ++c) {
      const CurveDev<Real>& C = cd[c];
      std::vector<int> hc(C.nbatch), hl((size_t)C.nbatch * C.D);
      GTLS_TRY_CUDA(ctx, cudaMemcpy(hc.data(), C.union_cnt, sizeof(int) * C.nbatch, cudaMemcpyDeviceToHost));
      GTLS_TRY_CUDA(ctx, cudaMemcpy(hl.data(), C.union_list, sizeof(int) * hl.size(), cudaMemcpyDeviceToHost));
      for (long long b = 0; b < C.nbatch; ++b) {
        long long np_b = std::min<long long>(C.batch, C.np - b * C.batch);
        for (int u = 0; u < hc[b]; ++u) {
          const size_t dd = d_off[c] + hl[(size_t)b * C.D + u];
          long long sk = skips[dd];
          long long js = (C.n + sk - 1) / sk;
          starts += np_b * js;
          fma += np_b * js * 2LL * widths[dd];
        }
      }
    }
    tm->chi2_starts = starts;
    tm->chi2_fma = fma;
    unsigned long long hwk[2] = {0, 0};
    GTLS_TRY_CUDA(ctx, cudaMemcpy(hwk, work, sizeof(hwk), cudaMemcpyDeviceToHost));
    tm->chi2_active_fma = (long long)hwk[0];
    tm->chi2_issued_fma = (long long)hwk[1];
  }
  return GTLS_OK;
}

static int check_curve(gtls_ctx* ctx, const CurveHost& h) {
  if (h.n < 2 || !h.t || !h.y || !h.dy || (h.np > 0 && !h.periods) || !h.widths || !h.overshoot || !h.templates ||
      (h.np > 0 && !h.chi2_out))
    return fail(ctx, GTLS_E_INVALID, "null pointer or fewer than 2 samples");
  if (h.np < 0 || h.D < 1 || h.D > GTLS_MAX_DURATIONS)
    return fail(ctx, GTLS_E_INVALID, "n_periods >= 0 and 1 <= n_durations <= GTLS_MAX_DURATIONS required");
  if (h.max_width < 1 || h.max_width > h.n) return fail(ctx, GTLS_E_INVALID, "max_width must be in [1, n]");
  if (h.batch < 1) return fail(ctx, GTLS_E_INVALID, "batch must be >= 1");
  return GTLS_OK;
}

}  // namespace gtls

using namespace gtls;

extern "C" int gtls_search(gtls_ctx* ctx, const gtls_search_desc* d, void* stream) {
  if (!ctx) return GTLS_E_INVALID;
  if (!d || d->abi_version != GTLS_ABI_VERSION) return fail(ctx, GTLS_E_INVALID, "bad descriptor or ABI version");
  if (d->n_periods < 1) return fail(ctx, GTLS_E_INVALID, "n_periods >= 1 required");
  if (d->skip_point < 1) return fail(ctx, GTLS_E_INVALID, "skip_point must be >= 1");
  if (d->pass != GTLS_PASS_MAIN && d->pass != GTLS_PASS_ALL) return fail(ctx, GTLS_E_INVALID, "unknown pass");
  if (d->flags & ~GTLS_SEARCH_ALL_DURATIONS) return fail(ctx, GTLS_E_INVALID, "unknown flags");
  CurveHost h;
  h.t = d->t;
  h.y = d->y;
  h.dy = d->dy;
  h.periods = d->periods;
  h.chi2_out = d->chi2_out;
  h.loc_out = d->loc_out;
  h.widths = d->widths;
  h.overshoot = d->overshoot;
  h.templates = d->templates;
  h.np = d->n_periods;
  h.n = d->n;
  h.D = d->n_durations;
  h.max_width = d->max_width;
  h.batch = d->batch;
  h.span = d->span;
  int rc = check_curve(ctx, h);
  if (rc) return rc;
  GTLS_TRY_CUDA(ctx, cudaSetDevice(ctx->device));
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  if (d->precision == GTLS_FP64)
    return run_search<double>(ctx, &h, 1, d->pass, d->skip_point, d->depth_min, d->flags, d->timing, st);
  if (d->precision == GTLS_FP32)
    return run_search<float>(ctx, &h, 1, d->pass, d->skip_point, d->depth_min, d->flags, d->timing, st);
  return fail(ctx, GTLS_E_INVALID, "unknown precision");
}

extern "C" int gtls_search_batch(gtls_ctx* ctx, const gtls_batch_desc* d, void* stream) {
  if (!ctx) return GTLS_E_INVALID;
  if (!d || d->abi_version != GTLS_ABI_VERSION) return fail(ctx, GTLS_E_INVALID, "bad descriptor or ABI version");
  if (d->n_curves < 1 || !d->sample_off || !d->period_off || !d->dur_off || !d->tmpl_off || !d->max_width ||
      !d->batch || !d->span)
    return fail(ctx, GTLS_E_INVALID, "null host array or no curves");
  // device bases first: a NULL base plus a curve's offset would not be NULL
  const bool any_period = d->period_off[d->n_curves] != d->period_off[0];
  if (!d->t || !d->y || !d->dy || !d->widths || !d->overshoot || !d->templates ||
      (any_period && (!d->periods || !d->chi2_out)))
    return fail(ctx, GTLS_E_INVALID, "null device array");
  if (d->skip_point < 1) return fail(ctx, GTLS_E_INVALID, "skip_point must be >= 1");
  if (d->pass != GTLS_PASS_MAIN && d->pass != GTLS_PASS_ALL) return fail(ctx, GTLS_E_INVALID, "unknown pass");
  if (d->flags & ~GTLS_SEARCH_ALL_DURATIONS) return fail(ctx, GTLS_E_INVALID, "unknown flags");
  std::vector<CurveHost> hs(d->n_curves);
  for (int c = 0; c < d->n_curves; ++c) {
    CurveHost& h = hs[c];
    const long long s0 = d->sample_off[c], s1 = d->sample_off[c + 1];
    const long long p0 = d->period_off[c], p1 = d->period_off[c + 1];
    const long long q0 = d->dur_off[c], q1 = d->dur_off[c + 1];
    if (s1 - s0 > (1LL << 30) || s1 < s0 || p1 < p0 || q1 <= q0)
      return fail(ctx, GTLS_E_INVALID, "offsets must be non-decreasing (every curve needs a duration)");
    h.t = d->t + s0;
    h.y = d->y + s0;
    h.dy = d->dy + s0;
    h.periods = d->periods + p0;
    h.chi2_out = d->chi2_out + p0;
    h.loc_out = d->loc_out ? d->loc_out + p0 : nullptr;
    h.widths = d->widths + q0;
    h.overshoot = d->overshoot + q0;
    h.templates = d->templates + d->tmpl_off[c];
    h.np = p1 - p0;
    h.n = (int)(s1 - s0);
    h.D = (int)(q1 - q0);
    h.max_width = d->max_width[c];
    h.batch = d->batch[c];
    h.span = d->span[c];
    int rc = check_curve(ctx, h);
    if (rc) return rc;
  }
  GTLS_TRY_CUDA(ctx, cudaSetDevice(ctx->device));
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  if (d->precision == GTLS_FP64)
    return run_search<double>(ctx, hs.data(), d->n_curves, d->pass, d->skip_point, d->depth_min, d->flags,
                              d->timing, st);
  if (d->precision == GTLS_FP32)
    return run_search<float>(ctx, hs.data(), d->n_curves, d->pass, d->skip_point, d->depth_min, d->flags,
                             d->timing, st);
  return fail(ctx, GTLS_E_INVALID, "unknown precision");
}

extern "C" int gtls_fold_order(gtls_ctx* ctx, const double* t, int32_t n, const double* periods, int64_t n_periods,
                               int32_t* order_out, void* stream) {
  if (!ctx) return GTLS_E_INVALID;
  if (!t || n < 1 || n_periods < 0 || (n_periods > 0 && (!periods || !order_out)))
    return fail(ctx, GTLS_E_INVALID, "bad arguments to gtls_fold_order");
  if (n_periods == 0) return GTLS_OK;
  GTLS_TRY_CUDA(ctx, cudaSetDevice(ctx->device));
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  CurveDev<double> C;
  std::memset(&C, 0, sizeof(C));
  C.t = t;
  C.periods = periods;
  C.np = n_periods;
  C.n = n;
  C.nb_log2 = nb_log2_for(n, ctx->bucket_shift);
  rounds_params(C, ctx->smem_optin);
  // chunks of periods sized to the scratch budget (8 bytes of slots per sample and period)
  const long long per_chunk = std::max<long long>(
      1, std::min<long long>((long long)(ctx->chunk_budget / (8 * (size_t)n)), (long long)INT32_MAX));
  std::vector<Run> runs;
  for (long long p0 = 0; p0 < n_periods; p0 += per_chunk) {
    Run r;
    std::memset(&r, 0, sizeof(r));
    r.count = (int)std::min<long long>(per_chunk, n_periods - p0);
    r.pidx0 = p0;
    r.slot_off = p0 * n;   // offset of the run's rows in order_out
    runs.push_back(r);
  }
  size_t total = 0;
  carve_size<CurveDev<double>>(total, 1);
  carve_size<Run>(total, runs.size());
  carve_size<uint2>(total, (size_t)std::min<long long>(per_chunk, n_periods) * n);
  void* mem = arena(ctx, total);
  if (!mem) return fail(ctx, GTLS_E_NOMEM, "scratch allocation failed");
  Carver cv(mem);
  CurveDev<double>* d_cd = cv.take<CurveDev<double>>(1);
  Run* d_runs = cv.take<Run>(runs.size());
  uint2* slots = cv.take<uint2>((size_t)std::min<long long>(per_chunk, n_periods) * n);
  GTLS_TRY_CUDA(ctx, cudaMemcpyAsync(d_cd, &C, sizeof(C), cudaMemcpyHostToDevice, st));
  GTLS_TRY_CUDA(ctx, cudaMemcpyAsync(d_runs, runs.data(), sizeof(Run) * runs.size(), cudaMemcpyHostToDevice, st));
  const size_t smem = prep_smem_bytes(C);
  if (!ctx->smem_set_fp64) {
    GTLS_TRY_CUDA(ctx, allow_smem<double>(ctx->smem_optin));
    ctx->smem_set_fp64 = true;
  }
  for (size_t k = 0; k < runs.size(); ++k) {
    if (n <= kPrepSmallMaxN)
      prepare_kernel<double, kPrepThreadsSmall><<<runs[k].count, kPrepThreadsSmall, smem, st>>>(d_cd, d_runs + k, 1,
                                                                                                slots, order_out);
    else
      prepare_kernel<double><<<runs[k].count, kPrepThreads, smem, st>>>(d_cd, d_runs + k, 1, slots, order_out);
    ctx->launches += 1;
    GTLS_TRY_CUDA(ctx, cudaGetLastError());
  }
  // the host copies above read C and runs: wait for them before they go out of scope
  GTLS_TRY_CUDA(ctx, cudaStreamSynchronize(st));
  return GTLS_OK;
}

extern "C" int gtls_duration_ranges(gtls_ctx* ctx, const double* periods, int64_t n_periods, float span,
                                    int32_t n_samples, int32_t* wmin, int32_t* wmax, void* stream) {
  if (!ctx) return GTLS_E_INVALID;
  if (!periods || !wmin || !wmax || n_periods < 0 || n_samples < 1)
    return fail(ctx, GTLS_E_INVALID, "bad arguments to gtls_duration_ranges");
  if (n_periods == 0) return GTLS_OK;
  GTLS_TRY_CUDA(ctx, cudaSetDevice(ctx->device));
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  duration_range_kernel<<<(unsigned)((n_periods + 255) / 256), 256, 0, st>>>(periods, n_periods, span, n_samples,
                                                                             wmin, wmax);
  ctx->launches += 1;
  GTLS_TRY_CUDA(ctx, cudaGetLastError());
  return GTLS_OK;
}
