// SDE spectra: stats.spectra (stats.py:95-122) and its running median
// (helpers.py:91-106) with numpy.ma semantics for masked entries, for
// gtls_spectra and gtls_spectra_noalloc.
//
// Every quantity is a reduction over the spectrum that the next step needs
// whole (minimum, mean, variance, then the same of the detrended power), so
// the steps are launches: each writes one partial result per CTA, and every CTA
// of the next adds those up for itself, in one order.  A call on 187,850 periods
// with the former single-CTA passes and an all-pairs median per window took 1.28
// ms (160 us on 2,592); it takes 94 (68), of which the kernels are 55 (35).
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstdint>

#include "spectra.cuh"

namespace gtls {

constexpr int kSpecThreads = 256;

__device__ __forceinline__ bool unmasked(const uint8_t* mask, long long i) { return !mask || !mask[i]; }

struct OpAdd { __device__ double operator()(double a, double b) const { return a + b; } };
// NaN-propagating like numpy's min/max
struct OpMin {
  __device__ double operator()(double a, double b) const { return (a != a) ? a : ((b != b) ? b : fmin(a, b)); }
};
struct OpMax {
  __device__ double operator()(double a, double b) const { return (a != a) ? a : ((b != b) ? b : fmax(a, b)); }
};

// Deterministic block reduction (fixed tree), the result in every thread; sh: 32 doubles.
template <typename Op>
__device__ double block_reduce(double v, Op op, double* sh) {
  const int lane = threadIdx.x & 31, nw = blockDim.x >> 5;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v = op(v, __shfl_xor_sync(0xffffffffu, v, o));
  __syncthreads();
  if (lane == 0) sh[threadIdx.x >> 5] = v;
  __syncthreads();
  double r = sh[0];
  for (int w = 1; w < nw; ++w) r = op(r, sh[w]);
  return r;
}
// The same over the n partial results of the launch before.
template <typename Op>
__device__ double reduce_parts(const double* __restrict__ part, int n, double none, Op op, double* sh) {
  double v = none;
  for (int i = threadIdx.x; i < n; i += blockDim.x) v = op(v, part[i]);
  return block_reduce(v, op, sh);
}

// 1: minimum of chi2 and number of unmasked periods
__global__ void __launch_bounds__(kSpecThreads) spec_min_kernel(const double* __restrict__ chi2,
                                                                const uint8_t* __restrict__ mask, long long n,
                                                                SpecScratch s) {
  __shared__ double sh[32];
  double mn = INFINITY, cnt = 0;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x)
    if (unmasked(mask, i)) {
      mn = OpMin()(mn, chi2[i]);
      cnt += 1;
    }
  mn = block_reduce(mn, OpMin(), sh);
  cnt = block_reduce(cnt, OpAdd(), sh);
  if (threadIdx.x == 0) {
    s.part[blockIdx.x] = mn;
    s.part[kSpecCtas + blockIdx.x] = cnt;
  }
}

// 2: SR = min / chi2 and its sum
__global__ void __launch_bounds__(kSpecThreads) spec_sr_kernel(const double* chi2,
                                                               const uint8_t* __restrict__ mask, long long n,
                                                               double* sr, SpecScratch s) {
  __shared__ double sh[32];
  const double mn = reduce_parts(s.part, gridDim.x, INFINITY, OpMin(), sh);
  double sum = 0;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
    const double v = mn / chi2[i];
    sr[i] = v;
    if (unmasked(mask, i)) sum += v;
  }
  sum = block_reduce(sum, OpAdd(), sh);
  if (threadIdx.x == 0) s.part[2 * kSpecCtas + blockIdx.x] = sum;
}

// 3: squares and largest of SR - mean
__global__ void __launch_bounds__(kSpecThreads) spec_var_kernel(const double* __restrict__ sr,
                                                                const uint8_t* __restrict__ mask, long long n,
                                                                SpecScratch s) {
  __shared__ double sh[32];
  const double cnt = reduce_parts(s.part + kSpecCtas, gridDim.x, 0.0, OpAdd(), sh);
  const double mean = reduce_parts(s.part + 2 * kSpecCtas, gridDim.x, 0.0, OpAdd(), sh) / cnt;
  double q = 0, mx = -INFINITY;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x)
    if (unmasked(mask, i)) {
      const double dv = sr[i] - mean;
      q += dv * dv;
      mx = OpMax()(mx, dv);
    }
  q = block_reduce(q, OpAdd(), sh);
  mx = block_reduce(mx, OpMax(), sh);
  if (threadIdx.x == 0) {
    s.part[3 * kSpecCtas + blockIdx.x] = q;
    s.part[4 * kSpecCtas + blockIdx.x] = mx;
    if (blockIdx.x == 0) {
      s.state->count = cnt;
      s.state->mean_sr = mean;
    }
  }
}

// Scale of the raw power from the parts of launch 3: power_raw = (SR - mean) * scale.
__device__ double raw_scale(const SpecScratch& s, int parts, double* sde_raw, double* sh) {
  const double sd = sqrt(reduce_parts(s.part + 3 * kSpecCtas, parts, 0.0, OpAdd(), sh) / s.state->count);
  const double mx = reduce_parts(s.part + 4 * kSpecCtas, parts, -INFINITY, OpMax(), sh);
  *sde_raw = (1 - s.state->mean_sr) / sd;
  return *sde_raw / mx;
}

// 4: raw power, for spectra too short for a running median, with a window too
// wide for the tiles of spec_median_kernel, or with outputs that share an array
__global__ void __launch_bounds__(kSpecThreads) spec_raw_kernel(const double* sr, long long n, double* praw,
                                                                double* power, SpecScratch s) {
  __shared__ double sh[32];
  double sde_raw;
  const double scale = raw_scale(s, gridDim.x, &sde_raw, sh), mean = s.state->mean_sr;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
    const double p = (sr[i] - mean) * scale;
    praw[i] = p;
    power[i] = p;
  }
  if (blockIdx.x == 0 && threadIdx.x == 0) s.state->sde_raw = sde_raw;
}

// Bit position of the r-th set bit (from 0) of a word that has it.
__device__ __forceinline__ int nth_bit(unsigned w, int r) {
  int at = 0;
#pragma unroll
  for (int sh = 16; sh > 0; sh >>= 1) {
    const int c = __popc(w & ((1u << sh) - 1u));
    if (r >= c) {
      r -= c;
      w >>= sh;
      at += sh;
    }
  }
  return at;
}

// 4: raw power, its running median over windows of k periods, and the
// difference, with its sum.  Window rows i = 0..n-k take the median of the
// unmasked values of [i, i + k) as numpy.ma.median does ((lo + hi) / 2 of the
// middle pair); the first and last rows' are repeated to the ends.
//
// A CTA sorts a tile of M consecutive values once (bitonic, a value per
// thread) and then slides the window as a bit set over the sorted places. M / 32
// lanes hold it (32 places each, so 32 runs of rows at once); a row moves two
// bits and finds the middle one by counting, some 70 instructions of a few
// lanes where ranking the window by all pairs took k^2 steps of one.  M is
// the smallest tile of at least twice the window.
template <int M>
__global__ void __launch_bounds__(M) spec_median_kernel(const double* __restrict__ sr, const uint8_t* __restrict__ mask,
                                                        long long n, int k, int raw_parts, double* __restrict__ praw,
                                                        double* __restrict__ power, SpecScratch s) {
  constexpr int kWords = M / 32;   // words and lanes of a bit set
  __shared__ double sh[32];
  __shared__ double key_sm[M];               // while sorting, then the sorted values
  __shared__ unsigned short idx_sm[M];       // and their places in the tile (0xffff: not in any window)
  __shared__ unsigned short rank_sm[M];      // sorted place of each place (0xffff likewise)
  __shared__ double raw_sm[M], med_sm[M];
  const int tid = threadIdx.x, lane = tid & 31;
  double sde_raw;
  const double scale = raw_scale(s, raw_parts, &sde_raw, sh), mean = s.state->mean_sr;
  const long long rows = n - k + 1, front = (n - rows) / 2;
  const int rpt = M - k + 1;   // rows of a tile
  const long long tiles = (rows + rpt - 1) / rpt;
  double sum = 0;
  for (long long tile = blockIdx.x; tile < tiles; tile += gridDim.x) {
    const long long r0 = tile * rpt;
    const int nrow = (int)min((long long)rpt, rows - r0);
    const bool end = tile == tiles - 1;
    const long long e = r0 + tid;
    const bool in = e < n;
    double raw = 0;
    bool use = false;
    if (in) {
      raw = (sr[e] - mean) * scale;
      use = unmasked(mask, e);
      if (tid < rpt || end) praw[e] = raw;   // the tile's own places
    }
    __syncthreads();
    raw_sm[tid] = raw;
    rank_sm[tid] = 0xffff;
    // sort (value, place); values outside every window go last
    double key = use ? raw : INFINITY;
    int idx = use ? tid : 0xffff;
    for (int size = 2; size <= M; size <<= 1)
      for (int step = size >> 1; step > 0; step >>= 1) {
        double ok;
        int oi;
        if (step >= 32) {
          __syncthreads();
          key_sm[tid] = key;
          idx_sm[tid] = (unsigned short)idx;
          __syncthreads();
          ok = key_sm[tid ^ step];
          oi = idx_sm[tid ^ step];
        } else {
          ok = __shfl_xor_sync(0xffffffffu, key, step);
          oi = __shfl_xor_sync(0xffffffffu, idx, step);
        }
        // equal values by place: the same order on both sides of a pair
        const bool less = ok < key || (ok == key && oi < idx);
        const bool low = (tid & step) == 0, up = (tid & size) == 0;
        if (less == (low == up)) {
          key = ok;
          idx = oi;
        }
      }
    __syncthreads();
    key_sm[tid] = key;
    idx_sm[tid] = (unsigned short)idx;
    if (idx != 0xffff) rank_sm[idx] = (unsigned short)tid;
    __syncthreads();
    // rows a..b-1 of the tile by this lane's group of kWords lanes
    const int gl = tid % kWords, per = (nrow + 31) / 32;   // 32 groups
    const int a = min(nrow, tid / kWords * per), b = min(nrow, a + per);
    const unsigned group = (kWords == 32 ? 0xffffffffu : ((1u << kWords) - 1u)) << (lane - gl);
    unsigned word = 0;
#pragma unroll 4
    for (int q = 0; q < 32; ++q) {
      const int place = idx_sm[32 * gl + q];
      if (place != 0xffff && place >= a && place < a + k) word |= 1u << q;
    }
    for (int row = a; row < a + per; ++row) {   // the whole warp keeps step
      if (row > a && row < b) {   // the window moves on
        const int out = rank_sm[row - 1], inn = rank_sm[row + k - 1];
        if (out != 0xffff && gl == out >> 5) word &= ~(1u << (out & 31));
        if (inn != 0xffff && gl == inn >> 5) word |= 1u << (inn & 31);
      }
      const int pc = __popc(word);
      int inc = pc;
#pragma unroll
      for (int o = 1; o < kWords; o <<= 1) {
        const int y = __shfl_up_sync(0xffffffffu, inc, o, kWords);
        if (gl >= o) inc += y;
      }
      const int before = inc - pc, cnt = __shfl_sync(0xffffffffu, inc, kWords - 1, kWords);
      const int hi_r = cnt / 2, lo_r = (cnt & 1) ? hi_r : hi_r - 1;
      // the middle one or two of the window, from the lanes that hold them
      const bool has_lo = lo_r >= before && lo_r < inc, has_hi = hi_r >= before && hi_r < inc;
      double lo = 0, hi = 0;
      if (has_lo) lo = key_sm[32 * gl + nth_bit(word, lo_r - before)];
      if (has_hi) hi = hi_r == lo_r ? lo : key_sm[32 * gl + nth_bit(word, hi_r - before)];
      const unsigned lo_at = __ballot_sync(0xffffffffu, has_lo) & group, hi_at = __ballot_sync(0xffffffffu, has_hi) & group;
      lo = __shfl_sync(0xffffffffu, lo, lo_at ? __ffs(lo_at) - 1 : lane);
      hi = __shfl_sync(0xffffffffu, hi, hi_at ? __ffs(hi_at) - 1 : lane);
      if (gl == 0 && row < b) med_sm[row] = cnt > 0 ? (lo + hi) * 0.5 : NAN;
    }
    __syncthreads();
    // a thread per place: its row is the one that it is the middle of, or the nearest
    if (in) {
      const long long row = e - front;   // global
      const long long near = row < 0 ? 0 : (row >= rows ? rows - 1 : row);
      if (near >= r0 && near < r0 + nrow) {
        const double p = raw_sm[tid] - med_sm[near - r0];
        power[e] = p;
        if (use) sum += p;
      }
    }
  }
  sum = block_reduce(sum, OpAdd(), sh);
  if (tid == 0) {
    s.part[5 * kSpecCtas + blockIdx.x] = sum;
    if (blockIdx.x == 0) s.state->sde_raw = sde_raw;
  }
}

// The running median where the tiles are not used: a thread per row ranks its
// window by all pairs.
__global__ void running_median_kernel(const double* __restrict__ praw, const uint8_t* __restrict__ mask,
                                      long long n, int k, double* __restrict__ med) {
  long long rows = n - k + 1;
  long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  if (i >= rows) return;
  int cnt = 0;
  for (int j = 0; j < k; ++j) cnt += unmasked(mask, i + j);
  double out = NAN;
  if (cnt > 0) {
    int h = cnt / 2;
    int lo_r = (cnt & 1) ? h : h - 1;
    int hi_r = h;
    double lo = NAN, hi = NAN;
    // rank of element j among the unmasked window values, ties broken by position
    for (int j = 0; j < k; ++j) {
      if (!unmasked(mask, i + j)) continue;
      double v = praw[i + j];
      int r = 0;
      for (int m = 0; m < k; ++m) {
        if (!unmasked(mask, i + m)) continue;
        double x = praw[i + m];
        r += (x < v) || (x == v && m < j);
      }
      if (r == lo_r) lo = v;
      if (r == hi_r) hi = v;
    }
    out = (lo + hi) / 2.0;
  }
  med[i] = out;
}

// power = power_raw - median (rows as above) and its sum
__global__ void __launch_bounds__(kSpecThreads) spec_detrend_kernel(const double* praw,
                                                                    const uint8_t* __restrict__ mask, long long n,
                                                                    int k, const double* __restrict__ med,
                                                                    double* power, SpecScratch s) {
  __shared__ double sh[32];
  const long long rows = n - k + 1, front = (n - rows) / 2;
  double sum = 0;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
    const double p = praw[i] - med[min(max(i - front, 0LL), rows - 1)];
    power[i] = p;
    if (unmasked(mask, i)) sum += p;
  }
  sum = block_reduce(sum, OpAdd(), sh);
  if (threadIdx.x == 0) s.part[5 * kSpecCtas + blockIdx.x] = sum;
}

// 5: squares and largest of power - mean (parts: CTAs of launch 4)
__global__ void __launch_bounds__(kSpecThreads) spec_power_var_kernel(const double* __restrict__ power,
                                                                      const uint8_t* __restrict__ mask, long long n,
                                                                      int parts, SpecScratch s) {
  __shared__ double sh[32];
  const double mean = reduce_parts(s.part + 5 * kSpecCtas, parts, 0.0, OpAdd(), sh) / s.state->count;
  double q = 0, mx = -INFINITY;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x)
    if (unmasked(mask, i)) {
      const double p = power[i] - mean;
      q += p * p;
      mx = OpMax()(mx, p);
    }
  q = block_reduce(q, OpAdd(), sh);
  mx = block_reduce(mx, OpMax(), sh);
  if (threadIdx.x == 0) {
    s.part[blockIdx.x] = q;
    s.part[kSpecCtas + blockIdx.x] = mx;
    if (blockIdx.x == 0) s.state->mean_power = mean;
  }
}

// 6: power scaled so that its largest value is the SDE
__global__ void __launch_bounds__(kSpecThreads) spec_scale_kernel(long long n, double* __restrict__ power,
                                                                  SpecScratch s) {
  __shared__ double sh[32];
  const double sd = sqrt(reduce_parts(s.part, gridDim.x, 0.0, OpAdd(), sh) / s.state->count);
  const double mx = reduce_parts(s.part + kSpecCtas, gridDim.x, -INFINITY, OpMax(), sh);
  const double sde = mx / sd, scale = sde / mx, mean = s.state->mean_power;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x)
    power[i] = (power[i] - mean) * scale;
  if (blockIdx.x == 0 && threadIdx.x == 0) s.state->sde = sde;
}

int spectra_launch(const double* chi2, const uint8_t* mask, long long n, int k, double* sr, double* praw,
                   double* power, SpecScratch s, cudaStream_t st) {
  // two values a thread, at most kSpecCtas CTAs
  const int ctas = (int)std::min<long long>(kSpecCtas, (n + 2 * kSpecThreads - 1) / (2 * kSpecThreads));
  int launches = 3;
  spec_min_kernel<<<ctas, kSpecThreads, 0, st>>>(chi2, mask, n, s);
  spec_sr_kernel<<<ctas, kSpecThreads, 0, st>>>(chi2, mask, n, sr, s);
  spec_var_kernel<<<ctas, kSpecThreads, 0, st>>>(sr, mask, n, s);
  if (n <= 2LL * k) {
    spec_raw_kernel<<<ctas, kSpecThreads, 0, st>>>(sr, n, praw, power, s);
    return launches + 1;
  }
  const long long rows = n - k + 1;
  int parts = ctas;
  // A caller that wants only some of the outputs may pass one array for several.
  // The tiles read sr beyond their own places and write both powers, so
  // they need three; the passes over whole arrays below read and write one place each.
  const bool apart = sr != praw && sr != power && praw != power;
  auto tiles = [&](int m) { return (int)std::min<long long>(kSpecCtas, (rows + m - k) / (m - k + 1)); };
  if (apart && k <= 128) {
    parts = tiles(256);
    spec_median_kernel<256><<<parts, 256, 0, st>>>(sr, mask, n, k, ctas, praw, power, s);
  } else if (apart && k <= 256) {
    parts = tiles(512);
    spec_median_kernel<512><<<parts, 512, 0, st>>>(sr, mask, n, k, ctas, praw, power, s);
  } else if (apart && k <= 512) {
    parts = tiles(1024);
    spec_median_kernel<1024><<<parts, 1024, 0, st>>>(sr, mask, n, k, ctas, praw, power, s);
  } else {
    spec_raw_kernel<<<ctas, kSpecThreads, 0, st>>>(sr, n, praw, power, s);
    running_median_kernel<<<(unsigned)((rows + 127) / 128), 128, 0, st>>>(praw, mask, n, k, s.med);
    spec_detrend_kernel<<<ctas, kSpecThreads, 0, st>>>(praw, mask, n, k, s.med, power, s);
    launches += 2;
  }
  spec_power_var_kernel<<<ctas, kSpecThreads, 0, st>>>(power, mask, n, parts, s);
  spec_scale_kernel<<<ctas, kSpecThreads, 0, st>>>(n, power, s);
  return launches + 3;
}

}  // namespace gtls
