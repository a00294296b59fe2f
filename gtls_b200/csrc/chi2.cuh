// chi2 of every period: bounds for all starts, sums for the few that remain.
// Included by search.cu after the descriptors.
#pragma once
#include <type_traits>

namespace gtls {

constexpr int kChiThreads = 384;
constexpr int kChiWarps = kChiThreads / 32;
constexpr int kItems = 7;                        // samples a thread brings in per batch (odd: no bank conflicts)
constexpr int kBatch = kChiThreads * kItems;     // samples of a batch, and starts screened after it
constexpr int kRing = 4096;                      // prefix values kept at every sample
constexpr int kRingMaxW = kRing - kBatch - 1;    // widths screened from the ring
constexpr int kCoarseCap = 2240;                 // prefix values kept at every g-th sample of the CTA's range
constexpr int kCoarseStep = 24;                  // g wanted when the range may be split
constexpr int kTaskGroupsMain = 4, kTaskGroupsAll = 8;   // groups of 32 starts of one task (its queue entries fit a byte)
constexpr int kSplitW = 1024;                    // wider windows are summed by the whole CTA
constexpr int kTogether = 4;                     // overlapping ones summed together, FP64
constexpr int kStage = 4096;                     // samples of theirs in shared memory at a time
constexpr int kProbe = 16;                       // all-starts pass: first sweep over every (width / kProbe)-th start
constexpr int kList = 4096;                      // starts of a CTA that wait for their sums, main pass
constexpr int kListAll = 8192;                   // and all-starts pass, whose starts come from blocks:
constexpr int kBlockTable = 24576;               // blocks of a CTA's starts and durations (a multiple of three)
constexpr int kBlockStarts = 64;                 // all-starts pass: consecutive starts bounded together from their samples
constexpr int kBlockSamples = 2048;              // samples of their windows in shared memory at a time
constexpr int kBlockSlots = 2048;                // blocks of a CTA taken up at a time

// Arrays of prefix values are skewed by one word per 32, so that starts a
// power of two apart fall into different banks.
__host__ __device__ __forceinline__ int skew(int p) { return p + (p >> 5); }
constexpr int kRingWords = kRing + kRing / 32;
constexpr int kCoarseWords = kCoarseCap + kCoarseCap / 32;
constexpr int kPartWords = kTogether * (kChiThreads / 32) * 6;   // words of their warps' sums, before the samples
static_assert(kPartWords % 4 == 0 && kPartWords + 4 * kStage <= 4 * kRingWords, "");
constexpr size_t kChiSmemRing = 4 * sizeof(float) * kRingWords;
constexpr size_t kChiSmemCoarse = 3 * sizeof(float) * kCoarseWords;
// Dynamic shared memory: the rings, the coarse arrays, and per duration of the
// union its first task, width and skip, and index.
inline size_t chi2_smem_bytes(bool with_coarse, int durations) {
  return kChiSmemRing + (with_coarse ? kChiSmemCoarse : 0) + 8 + (size_t)durations * (2 * sizeof(int) + sizeof(short));
}
constexpr size_t kChiSmemMax = kChiSmemRing + kChiSmemCoarse + 8 + (size_t)GTLS_MAX_DURATIONS * 10;

// Steps of the coarse prefix of a CTA's range of `starts` starts (0: no width
// needs it).
inline int coarse_step(int starts, int max_width) {
  if (max_width <= kRingMaxW) return 0;
  const long long span = (long long)starts + max_width;
  return (int)std::max<long long>(8, (span + kCoarseCap - 8) / (kCoarseCap - 8));
}

struct Best {
  double v;
  long long loc;
};
__device__ __forceinline__ void best_update(Best& b, double v, long long loc) {
  if (v < b.v || (v == b.v && loc < b.loc)) {
    b.v = v;
    b.loc = loc;
  }
}

// A start that waits for its exact sums.
struct Waiting {
  float lb;
  int k, u;
};

// A spike (search.cu) among the samples of a CTA's range: its place in the range.
struct Spike {
  int q;
  float u, w;
};

// Spikes of part of the range, and the rounding of sums over them.
struct NearSpikes {
  const Spike* at;
  int n, uniform;
  float err;
};
__device__ __forceinline__ NearSpikes near_spikes(const Spike* spikes, int from, int end, int uniform) {
  NearSpikes s;
  s.at = spikes + from;
  s.n = min(end, kSpikes) - from;
  s.uniform = uniform;
  s.err = end > kSpikes ? INFINITY : spike_err(s.n);   // (there are no more, by their choice)
  return s;
}
// One spike that a window holds, where the template is t = (s, s^2).
template <typename R2>
__device__ __forceinline__ void add_spike(CellSums& cs, const NearSpikes& s, const R2& t, float u, float w) {
  add_spike(cs, (float)t.x, (float)t.y, u, s.uniform ? 0.f : w, s.err);
}
// v of a spike, to 3 half ulps; infinite where FP32 does not hold its w (starts
// whose windows hold it are summed).
__device__ __forceinline__ float spike_v(const Spike& x) { return x.w > 1e-30f ? x.u / x.w : INFINITY; }
// Those of the lanes' windows of w samples, which start at q (ascending); returns
// their sums of v, |v| and u^2.
struct SpikeSums {
  float v, av, sq;
};
template <typename R2>
__device__ __forceinline__ SpikeSums add_spikes(CellSums& cs, const NearSpikes& s, const R2* __restrict__ trow, int q,
                                                int w) {
  const int lane = threadIdx.x & 31;
  const int from = __shfl_sync(0xffffffffu, q, 0), to = __shfl_sync(0xffffffffu, q, 31) + w;
  SpikeSums o{0.f, 0.f, 0.f};
  for (int i0 = 0; i0 < s.n; i0 += 32) {
    Spike x{-1, 0.f, 0.f};
    if (i0 + lane < s.n) x = s.at[i0 + lane];
    const float xv = spike_v(x);
    __syncwarp();
    for (unsigned m = __ballot_sync(0xffffffffu, x.q >= from && x.q < to); m; m &= m - 1) {
      const int src = __ffs(m) - 1;
      const int i = __shfl_sync(0xffffffffu, x.q, src) - q;
      const float u = __shfl_sync(0xffffffffu, x.u, src), wt = __shfl_sync(0xffffffffu, x.w, src),
                  v = __shfl_sync(0xffffffffu, xv, src);
      if (i >= 0 && i < w) {
        add_spike(cs, s, trow[i], u, wt);
        o.v += v;
        o.av += fabsf(v);
        o.sq = fmaf(u, u, o.sq);
      }
      __syncwarp();
    }
  }
  if (s.err == INFINITY) {
    cs.er = INFINITY;
    o.av = INFINITY;
  }
  return o;
}

// Per CTA, in units of list entries: the list, (all starts) the blocks, and the spikes.
constexpr int list_entries(bool all) { return (all ? kListAll + kBlockTable / 3 : kList) + kSpikes; }
static_assert(sizeof(Waiting) == 3 * sizeof(int) && sizeof(Spike) == sizeof(Waiting), "");

struct Chi2Args {
  int nruns;
  double depth_min;
  float* vpre;              // rows of the prefix of v (CTAs of curves with a coarse prefix)
  Waiting* list;            // [chunk CTAs * list_entries(all)]
  int* tau;                 // [chunk periods] smallest upper bound so far, shared by a period's CTAs
  double* part_v;           // [chunk CTAs]
  long long* part_loc;      // [chunk CTAs]
  unsigned long long* work; // NULL, or [2]: multiply-adds of the starts passing the depth test, and executed
  int* any_late;            // set where a list ran over (host memory)
};

// Order-preserving map of a float to an int (for atomicMin).
__device__ __forceinline__ int float_key(float x) {
  const int b = __float_as_int(x);
  return b ^ ((b >> 31) & 0x7fffffff);
}
__device__ __forceinline__ float key_float(int k) { return __int_as_float(k ^ ((k >> 31) & 0x7fffffff)); }

// Sorted position -> original sample: positions past n wrap to the first ones
// (patchData, GPUFun.py:110-129).
__device__ __forceinline__ int wrap_pos(int p, int n) {
  if (p >= n) p -= n;
  return p < n ? p : p % n;
}

// (u, w) record of a sample from its (v, w), in the form's precision.
__device__ __forceinline__ double2 record_of(double2 g, double) { return make_double2(g.x * g.y, g.y); }
__device__ __forceinline__ float2 record_of(double2 g, float) { return make_float2((float)(g.x * g.y), (float)g.y); }

__device__ __forceinline__ double mul_rn(double a, double b) { return __dmul_rn(a, b); }
__device__ __forceinline__ float mul_rn(float a, float b) { return __fmul_rn(a, b); }

// Chi2 of a start from its window mean and sums; a mean that fails the depth
// test (GPUFun.py:407,437) gives n.  Returns delta (infinite when it fails).
// c C + 2 B is one fused multiply-add; which product it rounds is part of the
// FP32 form's summation order (skips of 32 and more round c C, others 2 B),
// so it is written out.
template <typename Real>
__device__ __forceinline__ double eval_mean(Best& best, Real mean, Real os, Real B, Real C, int skip,
                                            double depth_min, double ebase, double sentinel, long long loc) {
  if ((double)mean > depth_min) {
    const Real c = mean * os * (Real)2;
    const Real delta = c * (sizeof(Real) == 4 && skip >= 32 ? fma((Real)2, B, mul_rn(c, C)) : fma(c, C, (Real)2 * B));
    best_update(best, ebase + (double)delta, loc);
    return (double)delta;
  }
  best_update(best, sentinel, loc);
  return INFINITY;
}

// Sum of x over the warp: the butterfly of xor distances 16, 8, 4, 2, 1.
template <typename T>
__device__ __forceinline__ T warp_sum(T x) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
  return x;
}

// A curve and a period as the exact sums read them.
struct Folded {
  const int* order;      // [n] original sample of each sorted position
  const double2* vw;     // (v, w) per original sample
  int n;
};
__device__ __forceinline__ double2 folded_at(const Folded& f, int p) {
  const int i = f.order[wrap_pos(p, f.n)];
  return f.vw[min(max(i, 0), f.n - 1)];
}

// Sums of a window: S = sum v, B = sum s u, C = sum s^2 w.
template <typename Real>
struct Sums {
  double S;
  Real B, C;
};

// Part of the window sums of one start, over the samples first + lane, + step, ... of [k, k + w), by a warp (FP64).
// Eight samples are in flight and the indices of the next eight loaded ahead:
// a window is a chain of two L2 latencies per step (four in flight and none
// ahead took 2.5 times as long).  Not inlined: its registers stay apart from the
// screening's.
__device__ __noinline__ Sums<double> part_sums(const Folded& f, int k, int w, const double2* __restrict__ trow,
                                               int first, int step) {
  constexpr int kDeep = 8;
  const int lane = threadIdx.x & 31;
  const int n = f.n;
  const int* __restrict__ order = f.order;
  const double2* __restrict__ vw = f.vw;
  double S = 0.0, B = 0.0, C = 0.0;
  int next[kDeep];
#pragma unroll
  for (int q = 0; q < kDeep; ++q) {
    const int i = first + lane + step * q;
    next[q] = i < w ? order[wrap_pos(k + i, n)] : -1;
  }
  for (int i0 = first + lane; i0 < w; i0 += step * kDeep) {
    double2 g[kDeep];
#pragma unroll
    for (int q = 0; q < kDeep; ++q) g[q] = next[q] >= 0 ? vw[min(next[q], n - 1)] : make_double2(0.0, 0.0);
#pragma unroll
    for (int q = 0; q < kDeep; ++q) {
      const int i = i0 + step * (q + kDeep);
      next[q] = i < w ? order[wrap_pos(k + i, n)] : -1;
    }
#pragma unroll
    for (int q = 0; q < kDeep; ++q) {
      const int i = i0 + step * q;
      if (i < w) {
        const double2 t = trow[i];
        S += g[q].x;
        B = fma(t.x, g[q].x * g[q].y, B);
        C = fma(t.y, g[q].y, C);
      }
    }
  }
  return Sums<double>{warp_sum(S), warp_sum(B), warp_sum(C)};
}

// The whole window by one warp.  Windows above kSplitW are the sum of
// kChiWarps parts, as the CTA forms them, so that a start's value does not
// depend on who sums it.  (In FP32 B and C do not; S, in FP64, is added up in
// another order by the CTA, which the FP32 mean it is rounded to has not
// been seen to notice.)
__device__ __forceinline__ Sums<double> window_sums(const Folded& f, int k, int w, int,
                                                    const double2* __restrict__ trow) {
  if (w <= kSplitW) return part_sums(f, k, w, trow, 0, 32);
  Sums<double> t{0.0, 0.0, 0.0};
  for (int p = 0; p < kChiWarps; ++p) {
    const Sums<double> x = part_sums(f, k, w, trow, 32 * p, kChiThreads);
    t.S += x.S;
    t.B += x.B;
    t.C += x.C;
  }
  return t;
}

// FP32: the sums keep one order per (width, skip s), two-level: the products
// of each offset rho = 0..s-1 of a skip block run up (i = rho, rho + s, ...),
// then the offsets' sums are added, for s >= 32 within each lane (rho = lane,
// lane + 32, ...) and across the lanes by the butterfly, below that in
// ascending rho.  The order fixes a start's rounding, whatever else is
// evaluated with it.  (B, C) pairs are packed two-lane FMAs.
__device__ __forceinline__ float2 offset_sum(const Folded& f, int k, int w, int s, int rho,
                                             const float2* __restrict__ trow, double& S) {
  float2 pr = make_float2(0.f, 0.f);
#pragma unroll 4
  for (int i = rho; i < w; i += s) {
    const double2 g = folded_at(f, k + i);
    S += g.x;
    fma_pair(trow[i], record_of(g, 0.f), pr);
  }
  return pr;
}
__device__ __noinline__ Sums<float> window_sums(const Folded& f, int k, int w, int s,
                                                const float2* __restrict__ trow) {
  const int lane = threadIdx.x & 31;
  double S = 0.0;
  float2 acc = make_float2(0.f, 0.f);
  for (int r0 = 0; r0 < s; r0 += 32) {
    const int rho = r0 + lane;
    const float2 pr = rho < s ? offset_sum(f, k, w, s, rho, trow, S) : make_float2(0.f, 0.f);
    if (s >= 32) {
      if (rho < s) add_pair(acc, pr);
    } else {
      for (int q = 0; q < s; ++q) {
        float2 o;
        o.x = __shfl_sync(0xffffffffu, pr.x, q);
        o.y = __shfl_sync(0xffffffffu, pr.y, q);
        add_pair(acc, o);
      }
    }
  }
  S = warp_sum(S);
  if (s >= 32) {
    acc.x = warp_sum(acc.x);
    acc.y = warp_sum(acc.y);
  }
  return Sums<float>{S, acc.x, acc.y};
}

// FP32, skip 1: one chain over the window, by one thread; indices and samples
// are loaded eight ahead of it.
__device__ __noinline__ Sums<float> chain_sums(const Folded& f, int k, int w, const float2* __restrict__ trow) {
  constexpr int kDeep = 8;
  double S = 0.0;
  float2 pr = make_float2(0.f, 0.f);
  int next[kDeep];
#pragma unroll
  for (int q = 0; q < kDeep; ++q) next[q] = q < w ? f.order[wrap_pos(k + q, f.n)] : 0;
  for (int i0 = 0; i0 < w; i0 += kDeep) {
    double2 g[kDeep];
#pragma unroll
    for (int q = 0; q < kDeep; ++q) g[q] = f.vw[min(max(next[q], 0), f.n - 1)];
#pragma unroll
    for (int q = 0; q < kDeep; ++q) next[q] = i0 + kDeep + q < w ? f.order[wrap_pos(k + i0 + kDeep + q, f.n)] : 0;
#pragma unroll
    for (int q = 0; q < kDeep; ++q)
      if (i0 + q < w) {
        S += g[q].x;
        fma_pair(trow[i0 + q], record_of(g[q], 0.f), pr);
      }
  }
  return Sums<float>{S, pr.x, pr.y};
}

// What the exact value of a start needs, in shared memory: its functions are
// kept out of the screening's registers.
template <typename Real>
struct Exact {
  Folded fold;
  const typename Tr<Real>::R2* trows;
  const int* trow_off;
  const double* overshoot;
  const unsigned* wsk;   // per union position, width | skip << 16
  const short* dur;      // and duration
  Best* best;            // per warp
  int* tau_key;
  unsigned long long* work;   // executed multiply-adds, or NULL
  double depth_min, ebase, dscale;
};

// The value of start k of union position u from its window sums, by a whole warp.
template <typename Real>
__device__ __noinline__ void settle(const Exact<Real>& x, int u, int k, Sums<Real> s) {
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const int d = x.dur[u], w = (int)(x.wsk[u] & 0xffff);
  const Real inv_w = (Real)1 / (Real)w;
  Best b = x.best[wid];
  __syncwarp();
  const double delta = eval_mean<Real>(b, -(Real)s.S * inv_w, (Real)x.overshoot[d], s.B, s.C, (int)(x.wsk[u] >> 16),
                                       x.depth_min, x.ebase,
                                       (double)x.fold.n, (long long)u * x.fold.n + k);
  if (lane == 0) {
    x.best[wid] = b;
    if (delta < INFINITY) atomicMin(x.tau_key, float_key(__double2float_ru(delta * x.dscale)));
    if (x.work) atomicAdd(x.work, 2ULL * (unsigned)w);
  }
  __syncwarp();
}

// The same with the sums, by one warp.
template <typename Real>
__device__ __noinline__ void evaluate(const Exact<Real>& x, int u, int k) {
  settle<Real>(x, u, k, window_sums(x.fold, k, (int)(x.wsk[u] & 0xffff), (int)(x.wsk[u] >> 16),
                                    x.trows + x.trow_off[x.dur[u]]));
}

// The parts, one a warp, of the sums of up to kTogether wide windows (>
// kSplitW) by the CTA, each in part_sums' order.  What bounds a wide window is
// its scattered (v, w) reads, a sector each (24,000 clocks for 8,000 samples with two
// CTAs on the SM); the waiting starts lie around the same few dips, so the
// samples go through shared memory once for all.
__device__ __noinline__ void group_sums(const Exact<double>& x, const int2* which, int cnt, double2* stage,
                                        Sums<double>* parts) {
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  int k[kTogether], w[kTogether], lo = 0x7fffffff, hi = 0;
  const double2* trow[kTogether];
  Sums<double> sum[kTogether];
#pragma unroll
  for (int q = 0; q < kTogether; ++q) {
    const int u = q < cnt ? which[q].x : -1;
    k[q] = u >= 0 ? which[q].y : 0;
    w[q] = u >= 0 ? (int)(x.wsk[u] & 0xffff) : 0;
    trow[q] = x.trows + (u >= 0 ? x.trow_off[x.dur[u]] : 0);
    sum[q] = Sums<double>{0.0, 0.0, 0.0};
    if (u >= 0) {
      lo = min(lo, k[q]);
      hi = max(hi, k[q] + w[q]);
    }
  }
  for (int c0 = lo; c0 < hi; c0 += kStage) {
    const int len = min(kStage, hi - c0);
    constexpr int kDeep = 6;
    __syncthreads();
    for (int i0 = threadIdx.x; i0 < len; i0 += kDeep * kChiThreads) {
      int idx[kDeep];
#pragma unroll
      for (int q = 0; q < kDeep; ++q) {
        const int i = i0 + q * kChiThreads;
        idx[q] = i < len ? x.fold.order[wrap_pos(c0 + i, x.fold.n)] : 0;
      }
      double2 g[kDeep];
#pragma unroll
      for (int q = 0; q < kDeep; ++q) g[q] = x.fold.vw[min(max(idx[q], 0), x.fold.n - 1)];
#pragma unroll
      for (int q = 0; q < kDeep; ++q) {
        const int i = i0 + q * kChiThreads;
        if (i < len) stage[i] = g[q];
      }
    }
    __syncthreads();
#pragma unroll
    for (int q = 0; q < kTogether; ++q) {
      const int from = c0 - k[q], to = min(w[q], from + len);
      int i = threadIdx.x;
      if (from > i) i += (from - i + kChiThreads - 1) / kChiThreads * kChiThreads;
#pragma unroll 4
      for (; i < to; i += kChiThreads) {
        const double2 g = stage[i - from], t = trow[q][i];
        sum[q].S += g.x;
        sum[q].B = fma(t.x, g.x * g.y, sum[q].B);
        sum[q].C = fma(t.y, g.y, sum[q].C);
      }
    }
  }
#pragma unroll
  for (int q = 0; q < kTogether; ++q) {
    if (q >= cnt) break;
    const Sums<double> t{warp_sum(sum[q].S), warp_sum(sum[q].B), warp_sum(sum[q].C)};
    if (lane == 0) parts[q * kChiWarps + wid] = t;
  }
}

// One CTA per (period, range of starts).
//
// What bounds the stage: with every passing start summed it was the FMA pipe
// and the latency of the records' reads (6.0 us a period on a 70,000-sample
// curve with 66 durations); with the bounds first (screen.cuh) it is issue
// slots and barriers (2.7 us).
//
//  * The CTA walks its range in batches of 2,688 samples: every thread takes
//    seven folded samples (order, then the (v, w) pair: no records are written
//    to memory), the block scans v, u, w - wbar and u^2 - qbar, and the prefix
//    values go into a ring of 4,096 samples in shared memory (and u, w, u^2 at
//    every g-th sample into a coarse array, and v into a row in memory, for
//    widths the ring does not hold).
//  * After each batch the warps screen the 2,688 starts it completes, for every
//    duration of the union of at most kRingMaxW samples: the depth test of 128
//    starts, the passing ones packed 32 to a group, a lower bound each, and
//    both bounds from more cells for those not ruled out.  The smallest upper
//    bound so far (tau) rules out most; the rest are listed (all starts: their
//    blocks are marked, and those bounded again).  Wider durations
//    follow at the end from the coarse array.
//  * The listed starts still at or below tau get their exact sums, a warp each
//    (windows of more than 1,024 samples the CTA), the most promising first
//    (each result lowers tau).
//
// 384 threads of 80 registers, two CTAs to an SM (their shared memory, 105 KB and 10
// bytes a duration, allows for it up to 980 durations, 830 in the all-starts pass), so that
// one's barriers and scans overlap the other's screening (512 threads of
// 64 registers spill in the screening: 5.9 us).
//
// A list that runs over (main pass) marks its period; what it found is not the
// minimum then.  Such periods are searched again, by the kLate form, which works
// the list off as it goes: after each batch and as many durations as the list holds
// the starts of, from the former minimum as the first tau.  (With all starts of
// the tasks that found the list full summed instead, whatever their depth and
// bounds, 300 periods of 19,728 samples whose bounds were wide took 18.5 ms, 19 times the
// dense sums.)
template <typename Real, bool kAll, bool kLate = false>
__global__ void __launch_bounds__(kChiThreads, 2)
chi2_kernel(const CurveDev<Real>* __restrict__ cds, const Run* __restrict__ runs, const int* __restrict__ order,
            Chi2Args a) {
  using R2 = typename Tr<Real>::R2;
  extern __shared__ __align__(16) float dyn_f[];
  float* const ringV = dyn_f;
  float* const ringU = ringV + kRingWords;   // then W and Q
  constexpr int kTaskGroups = kAll ? kTaskGroupsAll : kTaskGroupsMain, kTaskStarts = 32 * kTaskGroups;
  __shared__ unsigned char queue[kChiWarps][kTaskStarts];
  __shared__ float4 cells_sm[kChiWarps][2 * kLaneCells];
  __shared__ ScreenRow row_sm[kChiWarps][2];
  __shared__ int list_n, tau_key, next_task, nring_sm, low_key, go_sm, picked[2];
  __shared__ short pick[kChiThreads];
  __shared__ double part_s[kChiWarps];
  __shared__ int2 together[kTogether];          // union position (-1: ruled out) and start
  __shared__ unsigned maxbits[4];
  __shared__ double carry[4], wtot[kChiWarps][4];   // of v, u, w, u^2
  __shared__ Best red[kChiWarps];
  __shared__ long long sent_sm;                 // first start of the range known to fail the depth test
  __shared__ unsigned long long work_sm[2];
  __shared__ int spike_end[4], spike_tot[kChiWarps];   // spikes up to the end of batch b: in [b & 3]

  const int cta = blockIdx.x;
  const int ri = upper_find(0, a.nruns, cta, [&](int i) { return (long long)runs[i].tile0; });
  const Run& R = runs[ri];
  const CurveDev<Real>& C = cds[R.curve];
  const int ntiles = C.ntiles;
  const int local = (cta - R.tile0) / ntiles;
  const int tix = (cta - R.tile0) - local * ntiles;
  if (kLate && !C.late[R.pidx0 + local]) return;
  const int bidx = (int)((R.pidx0 + local) / C.batch);   // union batch of the period
  const int n = C.n;
  const int ucnt = C.union_cnt[bidx];
  const int k0 = tix * C.tile;
  const int k1 = min(n, k0 + C.tile);
  __shared__ Exact<Real> ex;
  __shared__ CurveConst cc;
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const int g = C.coarse;
  // U, W, Q at every g-th sample, and v's prefix at every sample, for the widths the ring does not hold
  float* const coarse = ringV + 4 * kRingWords;
  float* const vrow = g > 0 ? a.vpre + R.v_off + (size_t)(cta - R.tile0) * C.vstride : nullptr;
  int* const task_pre = reinterpret_cast<int*>(coarse + (g > 0 ? 3 * kCoarseWords : 0));   // [ucnt + 1]
  unsigned* const wsk = reinterpret_cast<unsigned*>(task_pre + ucnt + 1);                 // [ucnt] width | skip << 16
  short* const dur = reinterpret_cast<short*>(wsk + ucnt);                                // [ucnt]
  if (threadIdx.x == 0) {
    ex.fold = Folded{order + R.slot_off + (size_t)local * n, C.vw, n};
    ex.trows = C.trows;
    ex.trow_off = C.trow_off;
    ex.overshoot = C.overshoot;
    ex.wsk = wsk;
    ex.dur = dur;
    ex.best = red;
    ex.tau_key = &tau_key;
    ex.work = a.work ? &work_sm[1] : nullptr;
    ex.depth_min = a.depth_min;
    ex.ebase = C.cst->ebase;
    ex.dscale = C.cst->dscale;
  }
  const ScreenRow* __restrict__ srows = C.srows;
  const ScreenCell* __restrict__ scells = C.scells;
  const int* __restrict__ sends = C.sends;
  constexpr int kCap = kAll ? kListAll : kList;
  Waiting* const list = a.list + (size_t)cta * list_entries(kAll);
  // all starts: the smallest lower bound (as float_key) of every block, kBlockStarts
  // starts of 2^bgroup neighbouring union positions
  int* const btable = reinterpret_cast<int*>(list + kCap);
  const int nblk = (k1 - k0 + kBlockStarts - 1) / kBlockStarts;
  int bgroup = 0;
  if constexpr (kAll) {
    while ((long long)nblk * (((ucnt - 1) >> bgroup) + 1) > kBlockTable) ++bgroup;
  }
  const int bpos = ((ucnt - 1) >> bgroup) + 1;   // groups of positions
  constexpr int kNoBlock = 0x7fffffff;
  auto to_block = [&](int u, int k, float lb) {   // a NaN's key may be the empty block's
    atomicMin(&btable[(k - k0) / kBlockStarts * bpos + (u >> bgroup)], float_key(lb == lb ? lb : -INFINITY));
  };
  if constexpr (kAll) {
    for (int i = threadIdx.x; i < nblk * bpos; i += kChiThreads) btable[i] = kNoBlock;
  }
  Spike* const spikes = reinterpret_cast<Spike*>(list + list_entries(kAll) - kSpikes);
  int* const tau_all = a.tau + (R.item0 + local);
  // FP32 exact sums: a term takes part in as many roundings, of half an ulp of the
  // absolute sum each, as its offset's run has terms, the offsets' sums are added up
  // in steps and its factors were rounded (window_sums; every start: one run)
  auto gamma_of = [&](int w, int s) {
    if (sizeof(Real) == 8) return kGammaF;
    const int steps = s >= 32 ? (s + 31) / 32 + 5 : s;
    return kGammaF + (float)((w + s - 1) / s + steps + 6) * 6e-8f;
  };
  constexpr long long kNone = 0x7fffffffffffffffLL;

  // tasks of one batch (of the whole range for the coarse widths) per union
  // position, an upper bound: a range of `starts` samples holds at most
  // starts / skip + 1 starts
  auto count_tasks = [&](int u_lo, int u_hi, int starts, bool probe) {   // warp 0; task_pre[0..u_hi-u_lo]
    int c = 0;
    for (int b = u_lo; b < u_hi; b += 32) {
      const int u = b + lane;
      int nt = 0;
      if (u < u_hi) {
        const int s = probe ? max(1, (int)(wsk[u] & 0xffff) / kProbe) : (int)(wsk[u] >> 16);
        nt = (starts / s + kTaskStarts) / kTaskStarts;
      }
      int inc = nt;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int yv = __shfl_up_sync(0xffffffffu, inc, o);
        if (lane >= o) inc += yv;
      }
      if (u < u_hi) task_pre[u - u_lo] = c + inc - nt;
      c += __shfl_sync(0xffffffffu, inc, 31);
    }
    if (lane == 0) task_pre[u_hi - u_lo] = c;
  };
  if (wid == 0) {
    const int* __restrict__ ulist = C.union_list + (size_t)bidx * C.D;
    int nr = 0;
    for (int b = 0; b < ucnt; b += 32) {
      const int u = b + lane;
      int w = kRingMaxW + 1;
      if (u < ucnt) {
        const int d = ulist[u];
        w = C.widths[d];
        wsk[u] = (unsigned)w | ((unsigned)C.skips[d] << 16);
        dur[u] = (short)d;
      }
      nr += __popc(__ballot_sync(0xffffffffu, u < ucnt && w <= kRingMaxW));
    }
    __syncwarp();
    count_tasks(0, nr, kBatch, false);
    if (lane == 0) {
      nring_sm = nr;
      list_n = 0;
      low_key = 0x7f800000;
      tau_key = 0x7f800000;   // infinity
      sent_sm = kNone;
      work_sm[0] = work_sm[1] = 0;
    }
    if (lane < 4) maxbits[lane] = spike_end[lane] = 0;
    if (lane < 4) carry[lane] = 0.0;
  } else if (wid == 4 && lane < (int)(sizeof(CurveConst) / 4)) {
    reinterpret_cast<int*>(&cc)[lane] = reinterpret_cast<const int*>(C.cst)[lane];
  } else if (wid == 1 && lane < 4) {
    ringV[lane * kRingWords] = 0.f;                       // prefix at the range's first start
    if (g > 0 && lane < 3) coarse[lane * kCoarseWords] = 0.f;
    if (g > 0 && lane == 3) vrow[0] = 0.f;
  } else if (wid == 2 && lane < kChiWarps) {
    red[lane] = Best{INFINITY, kNone};
  }
  __syncthreads();
  const int nring = nring_sm;
  const float dthr = (float)(a.depth_min * cc.vscale);
  // E + delta and n are rounded to doubles: starts that close to tau stay
  // (Without a finite E no start that passes has a finite value: none is listed,
  // and n, where a start fails, is the minimum.)
  const bool no_value = cc.kind >= kNoValue;
  const float margin = no_value ? 0.f : (float)((fabs(cc.ebase) + (double)n) * cc.dscale * 0x1p-44);
  if (no_value && threadIdx.x == 0) tau_key = 0;   // (read after the next barriers)
  const bool spiky = cc.spike_u < INFINITY || cc.spike_w < INFINITY;
  if constexpr (kLate) {
    if (threadIdx.x == 0) {   // (read after the next barriers)
      const double x = (C.chi2_out[R.pidx0 + local] - cc.ebase) * cc.dscale;
      if (x < INFINITY) tau_key = float_key(__double2float_ru(x));
    }
  }
  auto over_tau = [&](float lb) { return lb > key_float(*(volatile int*)&tau_key) + margin; };

  // (the warp's best exact value lives in red[wid]: few starts get one)

  // union position and part of task tk of the first cnt positions of task_pre
  auto find_task = [&](int tk, int cnt, int& u, int& sub) {
    int below = 0;   // positions whose tasks start at or before tk
    for (int b = 0; b < cnt; b += 32) {
      const unsigned m = __ballot_sync(0xffffffffu, b + lane < cnt && task_pre[min(b + lane, cnt)] <= tk);
      below += __popc(m);
      if (m != 0xffffffffu) break;
    }
    u = below - 1;
    sub = tk - task_pre[u];
  };

  // The next samples of the range, at most kBatch: fetch() reads them into
  // registers (before the barrier that ends the screening of the batch
  // before, so that a warp that waits there waits for its loads as well),
  // store() adds their prefix values.
  auto is_spike = [&](const double2& g) {
    const double w = g.y * cc.wscale;
    return fabs(g.x * cc.vscale * w) >= cc.spike_u || w > cc.spike_w;
  };
  int batches = 0;           // stored so far
  int ld = 0, fetched = 0;   // samples whose prefix values are stored, samples fetched
  double2 gq[kItems];
  auto fetch = [&](int cnt) {
    fetched = cnt;
    const int q0 = ld + (int)threadIdx.x * kItems;
    const int have = min(kItems, cnt - (int)threadIdx.x * kItems);
    const int* __restrict__ ord = ex.fold.order;
    const double2* __restrict__ vw = ex.fold.vw;
    if (k0 + q0 + kBatch < n)   // the next batch's indices: into L2
      asm volatile("prefetch.global.L2 [%0];" ::"l"(ord + k0 + q0 + kBatch));
    int idx[kItems];
#pragma unroll
    for (int i = 0; i < kItems; ++i) idx[i] = i < have ? ord[wrap_pos(k0 + q0 + i, n)] : -1;
#pragma unroll
    for (int i = 0; i < kItems; ++i)
      gq[i] = i < have ? vw[min(max(idx[i], 0), n - 1)] : make_double2(0.0, 0.0);
  };
  auto store = [&]() {
    const int cnt = fetched;
    const int q0 = ld + (int)threadIdx.x * kItems;   // item i is prefix value q0 + i + 1
    const int have = min(kItems, cnt - (int)threadIdx.x * kItems);
    ++batches;
    if (spiky) {   // listed in order; they are 0 in what follows
      int mine = 0;
#pragma unroll
      for (int i = 0; i < kItems; ++i) mine += i < have && is_spike(gq[i]);
      int upto = mine;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int y = __shfl_up_sync(0xffffffffu, upto, o);
        if (lane >= o) upto += y;
      }
      if (lane == 31) spike_tot[wid] = upto;
      __syncthreads();
      int at = spike_end[(batches - 1) & 3] + upto - mine;
      for (int q = 0; q < wid; ++q) at += spike_tot[q];
#pragma unroll
      for (int i = 0; i < kItems; ++i)
        if (i < have && is_spike(gq[i])) {
          const double w = gq[i].y * cc.wscale, u = gq[i].x * cc.vscale * w;
          if (at < kSpikes) spikes[at] = Spike{q0 + i, (float)u, (float)w};
          ++at;
          gq[i] = make_double2(0.0, 0.0);
        }
      if (threadIdx.x == kChiThreads - 1) spike_end[batches & 3] = at;
    }
    // v, u and w of an item, scaled in FP64 (a weight itself may be beyond FP32); 0 past the end
    auto item = [&](int i, double& v, double& u, double& w) {
      v = gq[i].x * cc.vscale;
      w = gq[i].y * cc.wscale;
      u = v * w;
    };
    const double qbar = cc.qbar, wbar = cc.wbar;
    double sv = 0.0, su = 0.0, sw = 0.0, sq = 0.0;
#pragma unroll
    for (int i = 0; i < kItems; ++i) {
      double v, u, w;
      item(i, v, u, w);
      sv += v;
      su += u;
      sw += w;
      sq = fma(u, u, sq);
    }
    sw = fma((double)-max(have, 0), wbar, sw);
    sq = fma((double)-max(have, 0), qbar, sq);
    double xv = sv, xu = su, xw = sw, xq = sq;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const double yv = __shfl_up_sync(0xffffffffu, xv, o), yu = __shfl_up_sync(0xffffffffu, xu, o),
                   yw = __shfl_up_sync(0xffffffffu, xw, o), yq = __shfl_up_sync(0xffffffffu, xq, o);
      if (lane >= o) {
        xv += yv;
        xu += yu;
        xw += yw;
        xq += yq;
      }
    }
    if (lane == 31) {
      wtot[wid][0] = xv;
      wtot[wid][1] = xu;
      wtot[wid][2] = xw;
      wtot[wid][3] = xq;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
      next_task = 0;
      if (ntiles > 1) atomicMin(&tau_key, atomicMin(tau_all, *(volatile int*)&tau_key));
    }
    // lane 8 f + j adds up field f of warps j and j + 8 before this one; three steps and a broadcast for all four
    static_assert(kChiWarps <= 16, "");
    double sum = ((lane & 7) < wid ? wtot[lane & 7][lane >> 3] : 0.0) +
                 ((lane & 7) + 8 < wid ? wtot[(lane & 7) + 8][lane >> 3] : 0.0);
#pragma unroll
    for (int o = 4; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
    double rv = carry[0] + __shfl_sync(0xffffffffu, sum, 0) + (xv - sv);
    double ru = carry[1] + __shfl_sync(0xffffffffu, sum, 8) + (xu - su);
    double rw = carry[2] + __shfl_sync(0xffffffffu, sum, 16) + (xw - sw);
    double rq = carry[3] + __shfl_sync(0xffffffffu, sum, 24) + (xq - sq);
    float mv = 0.f, mu = 0.f, mw = 0.f, mq = 0.f;
    int cq = 0, cr = 1;   // next coarse step and the items up to it
    if (g > 0) {
      cq = q0 / g + 1;
      cr = cq * g - q0;
    }
#pragma unroll
    for (int i = 0; i < kItems; ++i) {
      if (i < have) {
        double v, u, w;
        item(i, v, u, w);
        rv += v;
        ru += u;
        rw += w - wbar;
        rq += fma(u, u, -qbar);
        const float fv = (float)rv, fu = (float)ru, fw = (float)rw, fq = (float)rq;
        mv = fmaxf(mv, fabsf(fv));
        mu = fmaxf(mu, fabsf(fu));
        mw = fmaxf(mw, fabsf(fw));
        mq = fmaxf(mq, fabsf(fq));
        float* const to = ringV + skew((q0 + i + 1) & (kRing - 1));
        to[0] = fv;
        to[kRingWords] = fu;
        to[2 * kRingWords] = fw;
        to[3 * kRingWords] = fq;
        if (g > 0) {
          vrow[q0 + i + 1] = fv;
          if (i + 1 == cr && cq < kCoarseCap) {   // g >= 8 > kItems: at most one
            float* const tc = coarse + skew(cq);
            tc[0] = fu;
            tc[kCoarseWords] = fw;
            tc[2 * kCoarseWords] = fq;
          }
        }
      }
    }
    // largest magnitude of each prefix so far (their rounding)
    const unsigned r0 = __reduce_max_sync(0xffffffffu, __float_as_uint(mv)),
                   r1 = __reduce_max_sync(0xffffffffu, __float_as_uint(mu)),
                   r2 = __reduce_max_sync(0xffffffffu, __float_as_uint(mw)),
                   r3 = __reduce_max_sync(0xffffffffu, __float_as_uint(mq));
    if (lane < 4) atomicMax(&maxbits[lane], lane == 0 ? r0 : (lane == 1 ? r1 : (lane == 2 ? r2 : r3)));
    __syncthreads();   // the carry has been read by all
    if (threadIdx.x == kChiThreads - 1) {   // the last thread's end is the batch's
      carry[0] = rv;
      carry[1] = ru;
      carry[2] = rw;
      carry[3] = rq;
    }
    ld += cnt;
  };

  // prefix value of v at q samples from the range's start
  auto v_at = [&](auto coarse_tag, int q) {
    if constexpr (decltype(coarse_tag)::value) return vrow[q];
    else return ringV[skew(q & (kRing - 1))];
  };

  // a duration's rows and first table of cells, on their way to the warp's
  // buffers row_sm and cells_sm (.w of a cell's first half is its end)
  int row_part = 0;
  float4 cell_part = make_float4(0.f, 0.f, 0.f, 0.f);
  auto fetch_rows = [&](int d) {
    if (lane < 2 * (int)(sizeof(ScreenRow) / 4)) row_part = reinterpret_cast<const int*>(srows + 2 * d)[lane];
    cell_part = reinterpret_cast<const float4*>(scells + (size_t)d * kLaneCells)[lane];
  };
  auto store_rows = [&]() {
    if (lane < 2 * (int)(sizeof(ScreenRow) / 4)) reinterpret_cast<int*>(row_sm[wid])[lane] = row_part;
    cells_sm[wid][lane] = cell_part;
    __syncwarp();
  };

  // screen starts j0 s .. (j1 - 1) s (at most kTaskStarts) of union position u,
  // whose rows are in the warp's buffers; probe: only lower tau
  auto screen = [&](auto coarse_tag, auto spiky_tag, int u, int s, int j0, int j1, bool probe) {
    constexpr bool kCoarse = decltype(coarse_tag)::value, kSpiky = decltype(spiky_tag)::value;
    const float* const xU = kCoarse ? coarse : ringU;
    constexpr int kWords = kCoarse ? kCoarseWords : kRingWords;
    auto at = [&](int p) { return xU + skew(kCoarse ? p : p & (kRing - 1)); };
    const int d = dur[u];
    const int w = (int)(wsk[u] & 0xffff);
    const float inv_w = row_sm[wid][0].inv_w;
    const ScreenErr e = screen_err(__uint_as_float(maxbits[0]) * kPrefixErr, __uint_as_float(maxbits[1]) * kPrefixErr,
                                   __uint_as_float(maxbits[2]) * kPrefixErr,
                                   __uint_as_float(maxbits[3]) * kPrefixErr);
    const float em0 = e.v * inv_w + 2e-7f * fabsf(dthr);
    // depth test on the sum: fails for certain where V(k) - V(k + w) is below this
    const float vmin = (dthr - em0 - 4e-7f * fabsf(dthr)) / inv_w;
    const float vthr = vmin - 1e-6f * fabsf(vmin);
    float dv[kTaskGroups];
#pragma unroll
    for (int i = 0; i < kTaskGroups; ++i) {
      const int j = j0 + 32 * i + lane;
      const int q = j * s - k0;   // start within the range
      dv[i] = j < j1 ? v_at(coarse_tag, q) - v_at(coarse_tag, q + w) : -INFINITY;
    }
    // the spikes that the windows may hold (the ring has samples of the last two batches)
    NearSpikes near;
    if constexpr (kSpiky) {
      const int from = kCoarse ? 0 : spike_end[(batches - 2) & 3];
      near = near_spikes(spikes, from, spike_end[batches & 3], cc.kind & kUniform);
    }
    if constexpr (kSpiky) {   // less their v, with the rounding in the start's favour
      const int q_lo = j0 * s - k0, q_hi = (j1 - 1) * s - k0 + w;
      float sv[kTaskGroups] = {};
      for (int i0 = 0; i0 < near.n; i0 += 32) {
        Spike x{-1, 0.f, 0.f};
        if (i0 + lane < near.n) x = near.at[i0 + lane];
        const float xv = spike_v(x);
        __syncwarp();
        for (unsigned m = __ballot_sync(0xffffffffu, x.q >= q_lo && x.q < q_hi); m; m &= m - 1) {
          const int at_q = __shfl_sync(0xffffffffu, x.q, __ffs(m) - 1);
          const float v = __shfl_sync(0xffffffffu, xv, __ffs(m) - 1), less = v - fabsf(v) * near.err;
#pragma unroll
          for (int i = 0; i < kTaskGroups; ++i) {
            const int off = at_q - ((j0 + 32 * i + lane) * s - k0);
            if (off >= 0 && off < w) sv[i] += less;
          }
        }
      }
#pragma unroll
      for (int i = 0; i < kTaskGroups; ++i)
        if (j0 + 32 * i + lane < j1) dv[i] = near.err < INFINITY && fabsf(sv[i]) < INFINITY ? dv[i] - sv[i] : INFINITY;
    }
    // a failing start's value n matters at the first one only
    const long long loc0 = (long long)u * n + (long long)j0 * s;
    const bool track = !probe && loc0 < *(volatile long long*)&sent_sm;
    int cnt = 0;
#pragma unroll
    for (int i = 0; i < kTaskGroups; ++i) {
      const bool pass = dv[i] > vthr;
      const unsigned mask = __ballot_sync(0xffffffffu, pass);
      if (pass) queue[wid][cnt + __popc(mask & ((1u << lane) - 1u))] = (unsigned char)(32 * i + lane);
      cnt += __popc(mask);
      if (track) {
        const unsigned fail = __ballot_sync(0xffffffffu, j0 + 32 * i + lane < j1 && !pass);
        if (fail && lane == 0) atomicMin(&sent_sm, loc0 + (long long)(32 * i + __ffs(fail) - 1) * s);
      }
    }
    __syncwarp();
    if (a.work && lane == 0 && !probe && !kLate) atomicAdd(&work_sm[0], (unsigned long long)cnt * 2 * (unsigned)w);
    const float gamma = gamma_of(w, kAll ? 1 : (int)(wsk[u] >> 16));
    for (int b = 0; b < cnt; b += 32) {
      const int k = (j0 + queue[wid][min(b + lane, cnt - 1)]) * s;
      const int q = k - k0;
      // the window's first prefix values, and (coarse) how far it starts before them
      const int q1 = kCoarse ? q / g : q;
      const float kappa = kCoarse ? (float)(q1 * g - q) : 0.f;
      CellSums cs;
      const float* p = at(q1);
      float pu = p[0], pw = p[kWords], pq = p[2 * kWords];
      const float q00 = pq;
      int end = 0;
      const int rm = row_sm[wid][0].m;
#pragma unroll 2
      for (int i = 0; i < rm; ++i) {
        const float4 c0 = cells_sm[wid][2 * i], c1 = cells_sm[wid][2 * i + 1];
        const ScreenCell c{c0.x, c0.y, c0.z, 0.f, c1.x, c1.y, c1.z, c1.w};
        end = __float_as_int(c0.w);
        p = at(q1 + end);
        const float nu = p[0], nw = p[kWords], nq = p[2 * kWords];
        add_cell<kCoarse, false>(cs, c, nu - pu, nw - pw, nq - pq, kappa, cc.qbar, e);
        pu = nu;
        pw = nw;
        pq = nq;
      }
      float m = (v_at(coarse_tag, q) - v_at(coarse_tag, q + w)) * inv_w;
      float em = fmaf(3e-7f, fabsf(m), em0);
      float qwin = (pq - q00) + (float)(kCoarse ? end * g : w) * cc.qbar + 4.f * e.n2;
      if constexpr (kSpiky) {
        const SpikeSums o = add_spikes(cs, near, ex.trows + ex.trow_off[d], q, w);
        m -= o.v * inv_w;
        em = fmaf(o.av * inv_w, near.err, em) + 3e-7f * fabsf(m);
        qwin += o.sq;
      }
      float lb = start_bounds<false>(cs, row_sm[wid][0], m, em, qwin, cc.wbar, cc.kind & kUniform, gamma, e).lb;
      // too close to the depth threshold to tell: such a start needs its exact value (n, if it fails)
      const bool certain = m - em > dthr;
      if (cc.kind >= kNoValue && certain) lb = INFINITY;
      unsigned left = __ballot_sync(0xffffffffu, b + lane < cnt && (!certain || !over_tau(lb)));
      // the starts that are left.  Many (the neighbours of a peak in the
      // all-starts pass, the first ones of a range): the second table for all
      // lanes at once, kLaneCells cells at a time; few: one by one, lowest bound
      // first, a cell per lane.
      const int m2 = row_sm[wid][1].m;
      while (left) {
        if (12 * __popc(left) > m2) {
          CellSums s2;
          p = at(q1);
          pu = p[0], pw = p[kWords], pq = p[2 * kWords];
          for (int c0 = 0; c0 < m2; c0 += kLaneCells) {
            __syncwarp();
            if (lane < 2 * min(kLaneCells, m2 - c0))
              cells_sm[wid][lane] = reinterpret_cast<const float4*>(scells + row_sm[wid][1].first + c0)[lane];
            __syncwarp();
            const int* __restrict__ ends = sends + row_sm[wid][1].first + c0;
            for (int i = 0; i < min(kLaneCells, m2 - c0); ++i) {
              const float4 x0 = cells_sm[wid][2 * i], x1 = cells_sm[wid][2 * i + 1];
              const ScreenCell c{x0.x, x0.y, x0.z, x0.w, x1.x, x1.y, x1.z, x1.w};
              p = at(q1 + ends[i]);
              const float nu = p[0], nw = p[kWords], nq = p[2 * kWords];
              add_cell<kCoarse, true>(s2, c, nu - pu, nw - pw, nq - pq, kappa, cc.qbar, e);
              pu = nu;
              pw = nw;
              pq = nq;
            }
          }
          __syncwarp();
          cells_sm[wid][lane] = reinterpret_cast<const float4*>(scells + (size_t)d * kLaneCells)[lane];
          __syncwarp();
          if constexpr (kSpiky) add_spikes(s2, near, ex.trows + ex.trow_off[d], q, w);
          const StartBounds sb = start_bounds<true>(s2, row_sm[wid][1], m, em, qwin, cc.wbar, cc.kind & kUniform, gamma, e);
          lb = sb.lb;
          const bool on = left >> lane & 1;
          const int ub = __reduce_min_sync(0xffffffffu, on && certain && sb.ub < INFINITY ? float_key(sb.ub) : 0x7f800000);
          if (lane == 0 && ub < *(volatile int*)&tau_key) atomicMin(&tau_key, ub);
          __syncwarp();
          left = __ballot_sync(0xffffffffu, on && (probe ? certain : true) && (!certain || !over_tau(lb)));
          if (kAll && !probe) {
            if (left >> lane & 1) to_block(u, k, certain ? lb : -INFINITY);
          } else if (left) {
            int base = 0;
            if (lane == 0) base = atomicAdd(&list_n, __popc(left));
            const int pos = __shfl_sync(0xffffffffu, base, 0) + __popc(left & ((1u << lane) - 1u));
            const bool keep = left >> lane & 1;
            if (keep && pos < kCap) list[pos] = Waiting{certain ? lb : -INFINITY, k, u};
          }
          break;
        }
        const bool mine = left >> lane & 1;
        const int key = mine ? (certain && lb == lb ? float_key(lb) : (int)0x80000000) : 0x7fffffff;
        const int low = __reduce_min_sync(0xffffffffu, key);
        const int src = __ffs(__ballot_sync(0xffffffffu, mine && key == low)) - 1;
        left &= ~(1u << src);
        const int ks = __shfl_sync(0xffffffffu, k, src);
        const float ms = __shfl_sync(0xffffffffu, m, src), ems = __shfl_sync(0xffffffffu, em, src);
        const bool cert = __shfl_sync(0xffffffffu, (int)certain, src);
        int out = 0;
        if (lane == src) out = cert && over_tau(lb);   // tau may have fallen
        if (__shfl_sync(0xffffffffu, out, src)) break;   // and the others lie higher
        const ScreenRow& row2 = row_sm[wid][1];
        const int qs = ks - k0, qs1 = kCoarse ? qs / g : qs;
        const float kap = kCoarse ? (float)(qs1 * g - qs) : 0.f;
        CellSums s2;
        for (int i = lane; i < m2; i += 32) {
          const ScreenCell c = scells[row2.first + i];
          const float* const x0 = at(qs1 + (i ? sends[row2.first + i - 1] : 0));
          const float* const x1 = at(qs1 + sends[row2.first + i]);
          add_cell<kCoarse, true>(s2, c, x1[0] - x0[0], x1[kWords] - x0[kWords], x1[2 * kWords] - x0[2 * kWords], kap,
                                  cc.qbar, e);
        }
        if constexpr (kSpiky) {
          const R2* const trow = ex.trows + ex.trow_off[d];
          if (near.err == INFINITY) s2.er = INFINITY;
          for (int i = lane; i < near.n; i += 32) {
            const Spike x = near.at[i];
            if (x.q >= qs && x.q < qs + w) add_spike(s2, near, trow[x.q - qs], x.u, x.w);
          }
        }
        s2.B = warp_sum(s2.B);
        s2.er = warp_sum(s2.er);
        s2.cl = warp_sum(s2.cl);
        s2.cu = warp_sum(s2.cu);
        const StartBounds sb = start_bounds<true>(s2, row2, ms, ems, __shfl_sync(0xffffffffu, qwin, src), cc.wbar,
                                                  cc.kind & kUniform, gamma, e);
        if (lane == 0) {   // (it makes all of it)
          if (cert && sb.ub < INFINITY && float_key(sb.ub) < *(volatile int*)&tau_key)
            atomicMin(&tau_key, float_key(sb.ub));
          if (!(cert ? !over_tau(sb.lb) : !probe)) {
          } else if (kAll && !probe) {
            to_block(u, ks, cert ? sb.lb : -INFINITY);
          } else {
            const int pos = atomicAdd(&list_n, 1);
            if (pos < kCap) list[pos] = Waiting{cert ? sb.lb : -INFINITY, ks, u};
          }
        }
        left &= __ballot_sync(0xffffffffu, !certain || !over_tau(lb));
      }
    }
    __syncwarp();
  };

  // the range, batch by batch.  The all-starts pass sweeps it twice, first over a
  // few starts per width: with tau near its end the second sweep rules
  // out all but the neighbours of the best peak.
  const int max_ring_w = nring > 0 ? (int)(wsk[nring - 1] & 0xffff) : 0;
  const int need = (k1 - k0) + (nring < ucnt ? (int)(wsk[ucnt - 1] & 0xffff) + 2 * g : max_ring_w);
  auto claim = [&]() {
    int tk = 0;
    if (lane == 0) tk = atomicAdd(&next_task, 1);
    return __shfl_sync(0xffffffffu, tk, 0);
  };
  // all tasks of starts in [t0, t1) for the union positions u_lo .. u_lo + cnt - 1
  auto run_tasks_of = [&](auto coarse_tag, auto spiky_tag, int u_lo, int cnt, int t0, int t1, bool probe) {
    const int ntask = task_pre[cnt];
    int u = 0, sub = 0;
    auto next = [&]() {   // claims a task and sends for its rows
      const int tk = claim();
      if (tk >= ntask) return false;
      // The coarse widths go widest first, so that no long task is left for the
      // end (4% of the stage on 160,000 samples); the ring's narrowest first: their
      // tau spares the wide ones more than that.
      find_task(decltype(coarse_tag)::value ? ntask - 1 - tk : tk, cnt, u, sub);
      u += u_lo;
      fetch_rows(dur[u]);
      return true;
    };
    for (bool more = next(); more;) {
      const int cu = u, csub = sub;
      store_rows();
      more = next();
      const int s = probe ? max(1, (int)(wsk[cu] & 0xffff) / kProbe) : (kAll ? 1 : (int)(wsk[cu] >> 16));
      const int j0 = (t0 + s - 1) / s + csub * kTaskStarts, j1 = min((t1 + s - 1) / s, j0 + kTaskStarts);
      if (j0 < j1) screen(coarse_tag, spiky_tag, cu, s, j0, j1, probe);
      __syncwarp();
    }
  };
  auto run_tasks = [&](auto coarse_tag, int u_lo, int cnt, int t0, int t1, bool probe) {
    if (spiky) run_tasks_of(coarse_tag, std::true_type{}, u_lo, cnt, t0, t1, probe);
    else run_tasks_of(coarse_tag, std::false_type{}, u_lo, cnt, t0, t1, probe);
  };
  // The listed starts that can still be the minimum, the most promising first:
  // those of the lowest quarter between the smallest lower bound and tau;
  // their values then rule out most others.  The CTA's wide windows go through
  // the rings' memory, unless that is in use.
  auto work_off = [&](bool probe, bool ring_live) {
    const int total = min(list_n, kCap);
    float lo = INFINITY;
    for (int i = threadIdx.x; i < total; i += kChiThreads)
      if (list[i].k >= 0) lo = fminf(lo, list[i].lb);
    const int low = __reduce_min_sync(0xffffffffu, float_key(lo));
    if (lane == 0) atomicMin(&low_key, low);
    __syncthreads();
    const float first = key_float(low_key);
    const float cut = first + 0.25f * (key_float(tau_key) - first);   // NaN or infinite: nothing is put off
    for (int turn = 0; turn < (probe ? 1 : 2); ++turn)   // (the probe: the lowest quarter only)
      for (int c0 = 0; c0 < total; c0 += kChiThreads) {
        // this turn's entries of the next kChiThreads: narrow windows from the front of pick, wide from its end
        __syncthreads();
        if (threadIdx.x < 2) picked[threadIdx.x] = 0;
        if (threadIdx.x == 0 && ntiles > 1) atomicMin(&tau_key, atomicMin(tau_all, *(volatile int*)&tau_key));
        __syncthreads();
        const int i = c0 + threadIdx.x;
        if (i < total) {
          const Waiting x = list[i];
          if (x.k >= 0 && (x.lb > cut) == (turn == 1) && !over_tau(x.lb)) {
            const bool wide = (int)(wsk[x.u] & 0xffff) > kSplitW && !(kAll && sizeof(Real) == 4) && !ring_live;
            const int at = atomicAdd(&picked[wide], 1);
            pick[wide ? kChiThreads - 1 - at : at] = (short)threadIdx.x;
          }
        }
        __syncthreads();
        const int nn = picked[0], nw = picked[1];
        if constexpr (kAll && sizeof(Real) == 4) {
          // every start's sum is one chain over its window: a lane each
          Best best = red[wid];
          __syncwarp();
          const int j = threadIdx.x;
          if (j < nn) {
            const Waiting x = list[c0 + pick[j]];
            const int d = dur[x.u], w = (int)(wsk[x.u] & 0xffff);
            const Sums<float> t = chain_sums(ex.fold, x.k, w, ex.trows + ex.trow_off[d]);
            const float inv_w = 1.f / (float)w;
            const double delta = eval_mean<float>(best, -(float)t.S * inv_w, (float)ex.overshoot[d], t.B, t.C, 1, a.depth_min,
                                                  cc.ebase, (double)n, (long long)x.u * n + x.k);
            if (delta < INFINITY) atomicMin(&tau_key, float_key(__double2float_ru(delta * cc.dscale)));
            if (a.work) atomicAdd(&work_sm[1], 2ULL * (unsigned)w);
          }
          __syncwarp();
#pragma unroll
          for (int o = 16; o > 0; o >>= 1) {
            const double v = __shfl_xor_sync(0xffffffffu, best.v, o);
            const long long l = __shfl_xor_sync(0xffffffffu, best.loc, o);
            best_update(best, v, l);
          }
          if (lane == 0) red[wid] = best;
        } else {
          for (int j = wid; j < nn; j += kChiWarps) {   // a warp each
            const Waiting x = list[c0 + pick[j]];
            int go = 0;
            if (lane == 0) go = !over_tau(x.lb);   // one lane's view of tau for the warp
            if (__shfl_sync(0xffffffffu, go, 0)) evaluate<Real>(ex, x.u, x.k);
          }
          // the CTA together (a warp alone: 100,000 clocks for 10,000 samples)
          auto entry = [&](int j) { return list[c0 + pick[kChiThreads - 1 - j]]; };
          if constexpr (sizeof(Real) == 8) {
            // in order of their starts, up to kTogether whose windows overlap at a time
            if (nw > 1) {
              int* const keys = reinterpret_cast<int*>(dyn_f);   // the rings are free by now
              const int j = threadIdx.x;
              const short at = pick[kChiThreads - 1 - min(j, nw - 1)];
              __syncthreads();
              if (j < nw) keys[j] = list[c0 + at].k;
              __syncthreads();
              if (j < nw) {
                int rank = 0;
                for (int q = 0; q < nw; ++q) rank += keys[q] < keys[j] || (keys[q] == keys[j] && q < j);
                pick[kChiThreads - 1 - rank] = at;
              }
            }
            for (int j = 0; j < nw;) {
              __syncthreads();
              if (wid == 0) {
                Waiting x{0.f, 0, 0};
                int w = 0, go = 0;
                if (lane < kTogether && j + lane < nw) {
                  x = entry(j + lane);
                  w = (int)(wsk[x.u] & 0xffff);
                  go = !over_tau(x.lb);
                }
                int cnt = 1, end = __shfl_sync(0xffffffffu, x.k + w, 0);
                for (; cnt < min(kTogether, nw - j); ++cnt) {
                  if (__shfl_sync(0xffffffffu, x.k, cnt) >= end) break;
                  end = max(end, __shfl_sync(0xffffffffu, x.k + w, cnt));
                }
                if (lane < cnt) together[lane] = make_int2(go ? x.u : -1, x.k);
                if (lane == 0) go_sm = cnt;
              }
              __syncthreads();
              const int cnt = go_sm;
              Sums<double>* const parts = reinterpret_cast<Sums<double>*>(dyn_f);
              group_sums(ex, together, cnt, reinterpret_cast<double2*>(dyn_f + kPartWords), parts);
              __syncthreads();
              if (wid < cnt && together[wid].x >= 0) {
                Sums<double> t{0.0, 0.0, 0.0};
                for (int p = 0; p < kChiWarps; ++p) {
                  t.S += parts[wid * kChiWarps + p].S;
                  t.B += parts[wid * kChiWarps + p].B;
                  t.C += parts[wid * kChiWarps + p].C;
                }
                settle<Real>(ex, together[wid].x, together[wid].y, t);
              }
              j += cnt;
            }
          } else {
            for (int j = 0; j < nw; ++j) {
              const Waiting x = entry(j);
              const int w = (int)(wsk[x.u] & 0xffff), s = (int)(wsk[x.u] >> 16);
              __syncthreads();
              if (threadIdx.x == 0) go_sm = !over_tau(x.lb);
              __syncthreads();
              if (!go_sm) continue;
              if (s < 32 || s > kRingWords * 2) {
                if (wid == 0) evaluate<Real>(ex, x.u, x.k);
                continue;
              }
              const R2* __restrict__ trow = ex.trows + ex.trow_off[dur[x.u]];
              float2* const prs = reinterpret_cast<float2*>(dyn_f);
              double S = 0.0;
              for (int rho = threadIdx.x; rho < s; rho += kChiThreads) prs[rho] = offset_sum(ex.fold, x.k, w, s, rho, trow, S);
              S = warp_sum(S);
              if (lane == 0) part_s[wid] = S;
              __syncthreads();
              if (wid == 0) {
                float2 acc = make_float2(0.f, 0.f);
                for (int rho = lane; rho < s; rho += 32) add_pair(acc, prs[rho]);
                S = 0.0;
                for (int p = 0; p < kChiWarps; ++p) S += part_s[p];
                settle<Real>(ex, x.u, x.k, Sums<Real>{S, (Real)warp_sum(acc.x), (Real)warp_sum(acc.y)});
              }
            }
          }
        }
      }
  };
  // kLate: the end of the durations from u0 on of whose starts, one in skip of `starts` samples, the list holds all
  auto listable = [&](int u0, int end, int starts) {
    int u1 = u0;
    for (int room = kCap; u1 < end; ++u1) {
      room -= starts / (int)(wsk[u1] >> 16) + 1;
      if (room < 0 && u1 > u0) break;
    }
    return u1;
  };
  auto run_and_work_off = [&](auto coarse_tag, int u0, int u1, int t0, int t1) {
    __syncthreads();   // task_pre and the list are free
    if (wid == 0) count_tasks(u0, u1, t1 - t0, false);
    if (threadIdx.x == 0) {
      next_task = 0;
      list_n = 0;
      low_key = 0x7f800000;
    }
    __syncthreads();
    run_tasks(coarse_tag, u0, u1 - u0, t0, t1, false);
    __syncthreads();
    work_off(false, !decltype(coarse_tag)::value);
  };
  for (int sweep = kAll ? 0 : 1; sweep < 2; ++sweep) {
    const bool probe = sweep == 0;
    if (kAll) {
      ld = 0;
      if (threadIdx.x == 0) {
        carry[0] = carry[1] = carry[2] = carry[3] = 0.0;
        spike_end[0] = spike_end[1] = spike_end[2] = spike_end[3] = 0;
      } else if (threadIdx.x >= 32 && threadIdx.x < 36) {
        ringV[lane * kRingWords] = 0.f;
      }
      if (wid == 0) count_tasks(0, nring, kBatch, probe);
      __syncthreads();
    }
    fetch(min(max_ring_w, kBatch));
    store();
    fetch(min(kBatch, need - ld));
    for (int t0 = k0; t0 < k1; t0 += kBatch) {
      store();
      const int t1 = min(k1, t0 + kBatch);
      if constexpr (kLate) {
        for (int u0 = 0, u1; u0 < nring; u0 = u1) {
          u1 = listable(u0, nring, kBatch);
          run_and_work_off(std::false_type{}, u0, u1, t0, t1);
        }
      } else {
        run_tasks(std::false_type{}, 0, nring, t0, t1, probe);
      }
      fetch(min(kBatch, need - ld));
      __syncthreads();
    }
    if (nring < ucnt) {
      while (fetched > 0) {
        store();
        fetch(min(kBatch, need - ld));
      }
      if constexpr (kLate) {
        for (int u0 = nring, u1; u0 < ucnt; u0 = u1) {
          u1 = listable(u0, ucnt, k1 - k0);
          // (a single duration's starts may be more than the list holds)
          const long long part = u1 > u0 + 1 ? k1 - k0 : (long long)(kCap - 1) * (int)(wsk[u0] >> 16);
          for (long long t0 = k0; t0 < k1; t0 += part)
            run_and_work_off(std::true_type{}, u0, u1, (int)t0, (int)min((long long)k1, t0 + part));
        }
      } else {
        __syncthreads();   // next_task is 0, and task_pre free
        if (wid == 0) count_tasks(nring, ucnt, k1 - k0, probe);
        if (threadIdx.x == 0) next_task = 0;
        __syncthreads();
        run_tasks(std::true_type{}, nring, ucnt - nring, k0, k1, probe);
        __syncthreads();
      }
    }
    if constexpr (!kAll && !kLate) {
      if (threadIdx.x == 0 && list_n > kCap) {   // C.late was 0
        C.late[R.pidx0 + local] = 1;
        *a.any_late = 1;
      }
    }
    if (threadIdx.x == 0 && !probe) {
      long long sent = sent_sm;
      // starts skipped by k % skip != 0 carry the value n (GPUFun.py:407,409); the first is 1
      if (!kAll && k0 == 0 && n > 1)
        for (int u = 0; u < ucnt; ++u)
          if (wsk[u] >> 16 > 1) {
            sent = min(sent, (long long)u * n + 1);
            break;
          }
      sent_sm = sent;
      const double x = ((double)n - cc.ebase) * cc.dscale;
      if (sent != kNone && x < INFINITY) atomicMin(&tau_key, float_key(__double2float_ru(x)));
    }
    __syncthreads();

    if (kAll && !probe) {
      // Around a broad peak thousands of neighbouring starts stay (up to 22,000
      // in one CTA of a 70,000-sample curve, and on some curves ten times that).
      // The screening marks their blocks, 64 consecutive starts of a width, in a table
      // that cannot overflow; a block's starts are bounded together from
      // their samples themselves, in FP32, so closely that few are left.  (As a
      // list of starts, of which a full one left all starts of the CTA to be summed, some
      // curves took 0.1 to 1.5 s for 200 periods.)
      int* const block_at = reinterpret_cast<int*>(dyn_f);            // the rings are free by now
      int* const block_lb = block_at + kBlockSlots;
      float* const bv = reinterpret_cast<float*>(block_lb + kBlockSlots);                     // v, (u, w) and (s, s^2)
      float2* const buw = reinterpret_cast<float2*>(bv + kBlockSamples + kBlockStarts);
      float2* const bt = buw + kBlockSamples + kBlockStarts;
      float* const bpart = bv;                                        // [warp][5][kBlockStarts], after the samples
      static_assert(kBlockSlots * 8 + (kBlockSamples + kBlockStarts) * 12 + kBlockSamples * 8 <= 4 * 4 * kRingWords, "");
      static_assert(kChiWarps * 5 * kBlockStarts <= 3 * (kBlockSamples + kBlockStarts) + 2 * kBlockSamples, "");
      if (threadIdx.x == 0) list_n = 0;
      for (bool more = true; more;) {
        if (threadIdx.x == 0) picked[0] = 0;
        __syncthreads();
        float lo = INFINITY;
        for (int i = threadIdx.x; i < nblk * bpos; i += kChiThreads) {
          const int key = __ldcg(btable + i);
          if (key == kNoBlock || over_tau(key_float(key))) continue;
          const int pos = atomicAdd(&picked[0], 1);
          if (pos >= kBlockSlots) continue;
          block_at[pos] = i;
          block_lb[pos] = key;
          btable[i] = kNoBlock;
          if (key_float(key) > -INFINITY) lo = fminf(lo, key_float(key));
        }
        const int low = __reduce_min_sync(0xffffffffu, float_key(lo));
        if (lane == 0) atomicMin(&low_key, low);
        __syncthreads();
        more = picked[0] > kBlockSlots;
        const int nblocks = min(picked[0], kBlockSlots);
        const float cut = key_float(low_key) + 0.25f * (key_float(tau_key) - key_float(low_key));
        __syncthreads();
        if (threadIdx.x == 0) low_key = 0x7f800000;
        for (int j = 0; j < 2 * nblocks; ++j) {   // the lowest quarter first, then the others
          const int h = j < nblocks ? j : j - nblocks;
          const float blb = key_float(block_lb[h]);
          if ((blb > cut) != (j >= nblocks)) continue;
          const int u0 = block_at[h] % bpos << bgroup, kb = k0 + block_at[h] / bpos * kBlockStarts;
          for (int u = u0; u < min(ucnt, u0 + (1 << bgroup)); ++u) {
            __syncthreads();
            if (threadIdx.x == 0) go_sm = !over_tau(blb);
            __syncthreads();
            if (!go_sm) break;
            const int d = dur[u], w = (int)(wsk[u] & 0xffff);
            const R2* __restrict__ trow = ex.trows + ex.trow_off[d];
            // lane's starts kb + lane and kb + 32 + lane, each warp a slice of the window
            float2 bc[2] = {make_float2(0.f, 0.f), make_float2(0.f, 0.f)};
            float sv[2] = {0.f, 0.f}, av[2] = {0.f, 0.f}, qu[2] = {0.f, 0.f};
            for (int c = 0; c < w; c += kBlockSamples) {
              const int len = min(kBlockSamples, w - c);
              __syncthreads();
              {
                constexpr int kPer = (kBlockSamples + kBlockStarts + kChiThreads - 1) / kChiThreads;
                int idx[kPer];
#pragma unroll
                for (int q = 0; q < kPer; ++q) {
                  const int i = threadIdx.x + q * kChiThreads;
                  idx[q] = i < len + kBlockStarts ? ex.fold.order[wrap_pos(kb + c + i, n)] : -1;
                }
#pragma unroll
                for (int q = 0; q < kPer; ++q) {
                  const int i = threadIdx.x + q * kChiThreads;
                  if (idx[q] < 0) continue;
                  const double2 x = ex.fold.vw[min(idx[q], n - 1)];
                  const double v = x.x * cc.vscale, sw = x.y * cc.wscale;
                  bv[i] = (float)v;
                  buw[i] = make_float2((float)(v * sw), (float)sw);
                }
              }
              for (int i = threadIdx.x; i < len; i += kChiThreads) bt[i] = make_float2((float)trow[c + i].x, (float)trow[c + i].y);
              __syncthreads();
              const int slice = (len + kChiWarps - 1) / kChiWarps;
              const int i1 = min(len, (wid + 1) * slice);
#pragma unroll 4
              for (int i = wid * slice; i < i1; ++i) {
                const float2 t = bt[i];
#pragma unroll
                for (int b = 0; b < 2; ++b) {
                  const float2 x = buw[i + lane + 32 * b];
                  const float v = bv[i + lane + 32 * b];
                  fma_pair(t, x, bc[b]);
                  qu[b] = fmaf(x.x, x.x, qu[b]);
                  sv[b] += v;
                  av[b] += fabsf(v);
                }
              }
            }
            __syncthreads();
#pragma unroll
            for (int b = 0; b < 2; ++b) {
              float* const to = bpart + wid * 5 * kBlockStarts + lane + 32 * b;
              to[0] = bc[b].x;
              to[kBlockStarts] = bc[b].y;
              to[2 * kBlockStarts] = qu[b];
              to[3 * kBlockStarts] = sv[b];
              to[4 * kBlockStarts] = av[b];
            }
            __syncthreads();
            bool stays = false;
            if (threadIdx.x < kBlockStarts) {   // two whole warps
              float x[5] = {0.f, 0.f, 0.f, 0.f, 0.f};
              for (int p = 0; p < kChiWarps; ++p)
#pragma unroll
                for (int f = 0; f < 5; ++f) x[f] += bpart[(p * 5 + f) * kBlockStarts + threadIdx.x];
              const int k = kb + (int)threadIdx.x;
              // a sum of at most (w / kBlockSamples + 1) * 171 terms per warp, then of the warps
              const float roundf = (float)((w / kBlockSamples + 1) * (kBlockSamples / kChiWarps + 1) + kChiWarps + 8) * 1.2e-7f;
              ScreenRow row = srows[2 * d];
              row.asum = row.smn = row.smx = row.lmn = row.lmx = 0.f;
              CellSums cs;
              cs.B = x[0];
              cs.cl = cs.cu = x[1];
              const float m = -x[3] * row.inv_w;
              const float em = (roundf * x[4]) * row.inv_w + 4e-7f * fabsf(m) + 2e-7f * fabsf(dthr);
              const StartBounds sb = start_bounds<true>(cs, row, m, em, x[2] * (1.f + 2.f * roundf), 0.f, false,
                                                        gamma_of(w, 1) + roundf, ScreenErr{0.f, 0.f, 0.f, 0.f});
              // (a start that only its samples settle carries n like those that the screening settles)
              const bool fails = m + em <= dthr, mine = k < k1 && !fails, certain = m - em > dthr;
              if (k < k1 && fails) atomicMin(&sent_sm, (long long)u * n + k);
              if (mine && certain && sb.ub < INFINITY) atomicMin(&tau_key, float_key(sb.ub));
              __syncwarp();
              stays = mine && (!certain || !over_tau(sb.lb));
              if constexpr (sizeof(Real) == 8) {
                int pos = 0;
                if (stays) {
                  pos = atomicAdd(&list_n, 1);
                  if (pos < kCap) list[pos] = Waiting{certain ? sb.lb : -INFINITY, k, u};
                }
                unsigned over = __ballot_sync(0xffffffffu, stays && pos >= kCap);
                for (; over; over &= over - 1) evaluate<Real>(ex, u, __shfl_sync(0xffffffffu, k, __ffs(over) - 1));
              }
            }
            if constexpr (sizeof(Real) == 4) {
              // FP32 bounds carry the chains' own rounding, 0.3% at 24,000 samples, and
              // whole blocks stay (15 s for 161 periods of 163,000 samples when
              // they went through the list): their chains run here,
              // a lane each, over the samples in shared memory.
              if (!__syncthreads_or(stays)) continue;
              double* const cv = reinterpret_cast<double*>(bv);
              float2* const cuw = reinterpret_cast<float2*>(cv + kBlockSamples + kBlockStarts);
              float2* const ct = cuw + kBlockSamples + kBlockStarts;
              static_assert(kBlockSlots * 8 + (kBlockSamples + kBlockStarts) * 16 + kBlockSamples * 8 <= 4 * 4 * kRingWords, "");
              double S = 0.0;
              float2 pr = make_float2(0.f, 0.f);
              for (int c = 0; c < w; c += kBlockSamples) {
                const int len = min(kBlockSamples, w - c);
                __syncthreads();
#pragma unroll 6
                for (int i = threadIdx.x; i < len + kBlockStarts; i += kChiThreads) {
                  const double2 x = folded_at(ex.fold, kb + c + i);
                  cv[i] = x.x;
                  cuw[i] = record_of(x, 0.f);
                }
                for (int i = threadIdx.x; i < len; i += kChiThreads) ct[i] = make_float2((float)trow[c + i].x, (float)trow[c + i].y);
                __syncthreads();
                if (threadIdx.x < kBlockStarts) {
#pragma unroll 8
                  for (int i = 0; i < len; ++i) {
                    S += cv[i + threadIdx.x];
                    fma_pair(ct[i], cuw[i + threadIdx.x], pr);
                  }
                }
              }
              if (threadIdx.x < kBlockStarts) {
                Best best = red[wid];
                __syncwarp();
                if (stays) {
                  const float inv_w = 1.f / (float)w;
                  const int k = kb + (int)threadIdx.x;
                  const double delta = eval_mean<float>(best, -(float)S * inv_w, (float)ex.overshoot[d], pr.x, pr.y, 1,
                                                        a.depth_min, cc.ebase, (double)n, (long long)u * n + k);
                  if (delta < INFINITY) atomicMin(&tau_key, float_key(__double2float_ru(delta * cc.dscale)));
                  if (a.work) atomicAdd(&work_sm[1], 2ULL * (unsigned)w);
                }
#pragma unroll
                for (int o = 16; o > 0; o >>= 1) {
                  const double v = __shfl_xor_sync(0xffffffffu, best.v, o);
                  const long long l = __shfl_xor_sync(0xffffffffu, best.loc, o);
                  best_update(best, v, l);
                }
                if (lane == 0) red[wid] = best;
              }
            }
          }
        }
        __syncthreads();
      }
    }
    if constexpr (!kLate) {
      work_off(probe, false);
    }
    if (kAll && probe) {
      __syncthreads();
      if (threadIdx.x == 0) {
        list_n = 0;
        low_key = 0x7f800000;
      }
    }
  }
  __syncthreads();
  if (no_value && cc.ebase > 0.0 && sent_sm == kNone) {
    // E is infinite and all starts pass: the first whose sums are finite is
    // infinite.  Where the narrowest windows have none, with an infinite weight in
    // each, those that hold one of them whole have none either.
    const int w0 = (int)(wsk[0] & 0xffff), s0 = kAll ? 1 : (int)(wsk[0] >> 16);
    for (int u = 0; u < ucnt && (int)(wsk[u] & 0xffff) < w0 + s0; ++u) {
      const int s = kAll ? 1 : (int)(wsk[u] >> 16);
      for (int k = (k0 + s - 1) / s * s + wid * s; k < k1 && red[wid].loc == kNone; k += kChiWarps * s)
        evaluate<Real>(ex, u, k);
      int found = red[wid].loc != kNone;
      if (__syncthreads_or(found)) break;
    }
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    Best b = red[0];
    for (int i = 1; i < kChiWarps; ++i) best_update(b, red[i].v, red[i].loc);
    if (sent_sm != kNone) best_update(b, (double)n, sent_sm);
    if (ntiles > 1) {
      a.part_v[cta] = b.v;
      a.part_loc[cta] = b.loc;
    } else {   // the whole period: no duration of its batch is valid, no value
      const long long pg = R.pidx0 + local;
      C.chi2_out[pg] = ucnt > 0 ? b.v : NAN;
      if (C.loc_out) C.loc_out[pg] = ucnt > 0 ? b.loc : -1;
    }
    if (a.work) {
      atomicAdd(a.work, work_sm[0]);
      atomicAdd(a.work + 1, work_sm[1]);
    }
  }
}

}  // namespace gtls
