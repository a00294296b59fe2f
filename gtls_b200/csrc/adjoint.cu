// Chi2 of an unfolded limb-darkened transit model and its adjoint (gradient
// with respect to the six shape parameters), for many light curves at once.
// An addition with no counterpart in the reference: it refines a search
// peak below the period/duration grid resolution.
//
// The model is the search's own template model (gtls_b200/ldmodel.py, which
// stands in for the batman light curve of src/gputls/transit.py:8-42): a
// central (impact parameter 0) transit on a circular orbit of an opaque disk
// of radius p (stellar radii) across a star with quadratic limb darkening
// I(r) = 1 - u1 (1 - mu) - u2 (1 - mu)^2, mu = sqrt(1 - r^2).  For one light
// curve with parameters (P, T0, D, depth, u1, u2):
//   K   = 1 - u1/3 - u2/6,  p = sqrt(depth K)     (depth = central depth)
//   a   = (1 + p) / sin(pi D / P)                 (D = first-to-fourth contact)
//   phi = 2 pi ((t - T0)/P - n),  n = round((t - T0)/P)
//   z   = a |sin phi|            (no occultation when cos phi < 0)
//   m   = 1 - lambda(z, p, u1, u2),
// lambda = [int_0^{p-z} 2 pi r I dr + int_{|z-p|}^{min(1,z+p)} 2 r acos(c) I dr] / (pi K),
// c = (r^2 + z^2 - p^2) / (2 r z), both integrals by 96-node Gauss-Legendre
// quadrature after r = m + h sin(theta), exactly as ldmodel does.  Written as
// lambda = (M0 - u1 M1 - u2 M2) / (pi K) with the moments Mk of (1 - mu)^k,
// the u-derivatives are closed-form; the (z, p)-derivatives are those of the
// discrete quadrature itself (through the nodes, the limits and c), so the
// gradient is exact for the model the forward pass evaluates.
// chi2 = sum_i w_i (y_i - m(t_i))^2, w_i = 1/dy_i^2.  n is locally constant,
// so dphi/dP = -2 pi (t - T0) / P^2.  The backward pass recomputes the model
// per sample instead of storing it.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstdint>

#include "common.cuh"
#include "occultation.cuh"

namespace gtls {

constexpr int kAdjThreads = 256;
constexpr int kAdjWarps = kAdjThreads / 32;
constexpr int kAdjItems = 4;                     // samples a lane looks at together
constexpr int kAdjRound = 12288;                 // samples a CTA looks at before it evaluates those in transit
constexpr int kAdjSeg = kAdjRound / kAdjWarps;   // of them, a warp's
constexpr int kAdjGroup = 4;                     // lanes that share a sample's quadrature nodes
constexpr int kAdjCtas = 16 * 148;               // CTAs wanted: curves are split until there are as many
constexpr int kAdjSplits = 64;                   // CTAs of a curve, at most

// A curve's parameters and what follows from them alone.
struct TransitCurve {
  double P, T0, depth, u1, u2;
  double K, p, a, ang, sD;
  double inv_P, reach;   // samples further than `reach` periods from a transit's centre are out of it
};

__device__ __forceinline__ TransitCurve transit_curve(const double* __restrict__ th) {
  TransitCurve c;
  c.P = th[0];
  c.T0 = th[1];
  c.depth = th[3];
  c.u1 = th[4];
  c.u2 = th[5];
  c.K = 1.0 - c.u1 / 3.0 - c.u2 / 6.0;
  const double dk = c.depth * c.K;
  c.p = sqrt(dk);
  c.ang = kPi * th[2] / c.P;
  c.sD = sin(c.ang);
  c.a = (1.0 + c.p) / c.sD;
  c.inv_P = 1.0 / c.P;
  // z < 1 + p is |sin phi| < sD where 0 < sD < 1 (elsewhere every sample is
  // looked at); the distance below is rounded, and the exact test follows
  c.reach = !(dk > 0.0) ? -1.0 : (c.sD > 0.0 && c.sD < 1.0 ? asin(c.sD) * (0.5 / kPi) * (1.0 + 1e-9) + 1e-9 : 1.0);
  return c;
}

// Whether the sample at t may be in transit.
__device__ __forceinline__ bool may_transit(const TransitCurve& c, double t) {
  const double q = (t - c.T0) * c.inv_P;
  return fabs(q - rint(q)) <= c.reach + 1e-15 * fabs(q);
}

// Sum over the kAdjGroup lanes of a group.
__device__ __forceinline__ double group_sum(double x) {
#pragma unroll
  for (int o = kAdjGroup / 2; o > 0; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
  return x;
}

// Model flux at time t, and with kGrad its derivatives in (P, T0, D, depth, u1,
// u2) into d, by a group of lanes (all lanes of the warp take part; `on`: the
// group has a sample).
template <bool kGrad>
__device__ __forceinline__ double transit_flux(bool on, double t, const TransitCurve& c, double D, const GLTable& g,
                                               double (&d)[6]) {
  const int gl = threadIdx.x % kAdjGroup;
#pragma unroll
  for (int k = 0; k < 6; ++k) d[k] = 0.0;
  const double x = t - c.T0;
  const double q = x / c.P;
  const double phi = 2.0 * kPi * (q - rint(q));
  double sphi, cphi;
  sincos(phi, &sphi, &cphi);
  const double S = fabs(sphi);
  const double z = c.a * S;
  // (the far side of the orbit never occults)
  const bool hit = on && !(cphi < 0.0) && z < 1.0 + c.p;
  const double norm = kPi * c.K;
  if (!kGrad) {
    double M[3] = {0.0, 0.0, 0.0};
    if (hit) occultation_moments(z, c.p, g, M, gl, kAdjGroup);
    return 1.0 - (group_sum(M[0]) - c.u1 * group_sum(M[1]) - c.u2 * group_sum(M[2])) / norm;
  }
  OccultationGrad o{0.0, 0.0, 0.0, 0.0, 0.0};
  if (hit) o = occultation_grad(z, c.p, c.u1, c.u2, g, gl, kAdjGroup);
  o.N = group_sum(o.N);
  o.Nz = group_sum(o.Nz);
  o.Np = group_sum(o.Np);
  o.M1 = group_sum(o.M1);
  o.M2 = group_sum(o.M2);
  if (!hit) return 1.0;
  const double lz = o.Nz / norm, lp = o.Np / norm;
  const double lu1 = (-o.M1 + o.N / (3.0 * c.K)) / norm;
  const double lu2 = (-o.M2 + o.N / (6.0 * c.K)) / norm;
  // chain rule to the parameters
  const double P = c.P, sD = c.sD, cD = cos(c.ang);
  const double dp_depth = c.K / (2.0 * c.p), dp_u1 = -c.depth / (6.0 * c.p), dp_u2 = -c.depth / (12.0 * c.p);
  const double da_p = 1.0 / sD;
  const double da_D = -(1.0 + c.p) * cD * (kPi / P) / (sD * sD);
  const double da_P = (1.0 + c.p) * cD * (kPi * D / (P * P)) / (sD * sD);
  const double dS_phi = (sphi > 0.0 ? 1.0 : (sphi < 0.0 ? -1.0 : 0.0)) * cphi;
  const double dphi_P = -2.0 * kPi * x / (P * P), dphi_T0 = -2.0 * kPi / P;
  const double dz_P = S * da_P + c.a * dS_phi * dphi_P;
  const double dz_T0 = c.a * dS_phi * dphi_T0;
  const double dz_D = S * da_D;
  const double dz_p = S * da_p;
  d[0] = -(lz * dz_P);
  d[1] = -(lz * dz_T0);
  d[2] = -(lz * dz_D);
  d[3] = -((lz * dz_p + lp) * dp_depth);
  d[4] = -((lz * dz_p + lp) * dp_u1 + lu1);
  d[5] = -((lz * dz_p + lp) * dp_u2 + lu2);
  return 1.0 - o.N / norm;
}

// Deterministic block sum of K values per thread.
template <int K>
__device__ void block_sum(double (&v)[K], double* sh) {
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
#pragma unroll
  for (int k = 0; k < K; ++k) {
    double x = v[k];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
    if (lane == 0) sh[k * 32 + wid] = x;
  }
  __syncthreads();
  if (threadIdx.x < K) {
    double x = 0.0;
    for (int w = 0; w < (int)(blockDim.x >> 5); ++w) x += sh[threadIdx.x * 32 + w];
    sh[K * 32 + threadIdx.x] = x;
  }
  __syncthreads();
#pragma unroll
  for (int k = 0; k < K; ++k) v[k] = sh[K * 32 + k];
}

// chi2 of the curves (kGrad false: one value each) or its gradient (six).
//
// Some 2% of the samples are in transit and cost 96 quadrature nodes each, the
// others nothing but their residual (in the gradient a look whether it is finite:
// 3% of the time).  A CTA therefore
// looks at up to kAdjRound samples with one multiply-add each, lists those that
// may be in transit, and then evaluates the list, four lanes to a sample, so
// that a transit's neighbouring samples are spread over all its lanes.  On 1,024
// curves of 20,000 samples: evaluated where they lie 1.32 and 3.01 ms (chi2,
// gradient; most of a warp waits); queued by warp, a lane each, 0.99 and 1.68 ms
// (the warps with a transit keep the others at the end).  The FP64 pipe bounds
// what is left: acos, two square roots and a reciprocal per node.  `splits` CTAs
// share a curve, so that few curves fill the GPU too; their sums go to part and
// are added in order by model_sum_kernel.  (As the CTAs of a cluster, adding up
// from each other's shared memory, they wait for one another and for a place of
// their size: 148 curves of 20,000 samples 153 -> 203 us in clusters of 8, 350 in 16.)
template <bool kGrad>
__global__ void __launch_bounds__(kAdjThreads) model_kernel(const double* __restrict__ t, const double* __restrict__ y,
                                                            const double* __restrict__ w,
                                                            const int64_t* __restrict__ off,
                                                            const double* __restrict__ params, int splits,
                                                            double* __restrict__ part, const GLTable table) {
  constexpr int kOut = kGrad ? 6 : 1;
  __shared__ GLTable g;   // the lanes of a group read different nodes at once
  __shared__ double sh[(kOut + 1) * 32];
  __shared__ unsigned short list[kAdjRound];   // a segment per warp: offsets within it
  __shared__ int found[kAdjWarps];
  const int c = blockIdx.x / splits, lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  for (int j = threadIdx.x; j < kGLN; j += kAdjThreads) {
    g.s[j] = table.s[j];
    g.jw[j] = table.jw[j];
  }
  const long long n = off[c + 1] - off[c];
  const long long len = ((n + splits - 1) / splits + 31) / 32 * 32;   // samples of a CTA
  const long long first = min(n, (blockIdx.x % splits) * len), count = min(n - first, len);
  const double* __restrict__ tc = t + off[c] + first;
  const double* __restrict__ yc = y + off[c] + first;
  const double* __restrict__ wc = w + off[c] + first;
  const TransitCurve tr = transit_curve(params + 6 * (size_t)c);
  const double D = params[6 * (size_t)c + 2];
  double acc[kOut];
#pragma unroll
  for (int k = 0; k < kOut; ++k) acc[k] = 0.0;
  for (long long r0 = 0; r0 < count; r0 += kAdjRound) {
    // the warp's segment of the round: a whole number of steps, so that rounds end alike
    const int size = (int)min((long long)kAdjRound, count - r0);
    constexpr int kStep = 32 * kAdjItems;
    const int seg = min(kAdjSeg, ((size + kAdjWarps - 1) / kAdjWarps + kStep - 1) / kStep * kStep);
    const int s0 = min(size, wid * seg), s1 = min(size, s0 + seg);
    int hits = 0;
    for (int i0 = s0; i0 < s1; i0 += kStep) {
      double tv[kAdjItems], yv[kAdjItems], wv[kAdjItems];
#pragma unroll
      for (int u = 0; u < kAdjItems; ++u) {
        const int i = i0 + 32 * u + lane;
        tv[u] = i < s1 ? tc[r0 + i] : 0.0;
        yv[u] = i < s1 ? yc[r0 + i] : 1.0;
        wv[u] = i < s1 ? wc[r0 + i] : 0.0;
      }
#pragma unroll
      for (int u = 0; u < kAdjItems; ++u) {
        const int i = i0 + 32 * u + lane;
        const bool in = i < s1 && may_transit(tr, tv[u]);
        const unsigned m = __ballot_sync(0xffffffffu, in);
        if (in) list[wid * kAdjSeg + hits + __popc(m & ((1u << lane) - 1u))] = (unsigned short)(i - s0);
        hits += __popc(m);
        if (i < s1 && !in) {   // (the gradient: 0, or NaN where the residual is not finite)
          const double res = yv[u] - 1.0;
          acc[0] += wv[u] * res * (kGrad ? 0.0 : res);
        }
      }
    }
    if (lane == 0) found[wid] = hits;
    __syncthreads();
    int total = 0;
#pragma unroll
    for (int q = 0; q < kAdjWarps; ++q) total += found[q];
    constexpr int kGroups = kAdjThreads / kAdjGroup;
    for (int e0 = 0; e0 < total; e0 += kGroups) {   // the whole warp keeps step
      const int e = e0 + (int)threadIdx.x / kAdjGroup;
      const bool on = e < total;
      int q = 0, rest = on ? e : 0;
      while (q < kAdjWarps - 1 && rest >= found[q]) rest -= found[q++];
      const long long i = on ? r0 + min(size, q * seg) + list[q * kAdjSeg + rest] : 0;
      double d[6];
      const double m = transit_flux<kGrad>(on, tc[i], tr, D, g, d);
      if (on && threadIdx.x % kAdjGroup == 0) {
        const double res = yc[i] - m;
        if constexpr (kGrad) {
          const double f = -2.0 * wc[i] * res;
#pragma unroll
          for (int k = 0; k < 6; ++k) acc[k] += f * d[k];
        } else {
          acc[0] += wc[i] * res * res;
        }
      }
    }
    __syncthreads();
  }
  if constexpr (kGrad) {
    const double bad = acc[0] - acc[0];   // NaN if anything was
#pragma unroll
    for (int k = 1; k < 6; ++k) acc[k] += bad;
  }
  block_sum<kOut>(acc, sh);
  if (threadIdx.x < kOut) part[(size_t)blockIdx.x * kOut + threadIdx.x] = sh[kOut * 32 + threadIdx.x];
}

// The curves' values from the parts of their CTAs (times grad_out, if given).
template <int K>
__global__ void model_sum_kernel(const double* __restrict__ part, int n_curves, int splits,
                                 const double* __restrict__ grad_out, double* __restrict__ out) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n_curves * K) return;
  const int c = i / K, k = i % K;
  double x = 0.0;
#pragma unroll 4
  for (int s = 0; s < splits; ++s) x += part[((size_t)c * splits + s) * K + k];
  out[i] = grad_out ? grad_out[c] * x : x;
}

template <bool kGrad>
static int model_launch(gtls_ctx* ctx, const double* t, const double* y, const double* w, const int64_t* off,
                        int n_curves, const double* params, const double* grad_out, double* out, cudaStream_t st) {
  constexpr int kOut = kGrad ? 6 : 1;
  GTLS_TRY_CUDA(ctx, cudaSetDevice(ctx->device));
  const int splits = std::min(kAdjSplits, std::max(1, kAdjCtas / n_curves));
  const size_t ctas = (size_t)n_curves * splits;
  // The call is asynchronous, so its scratch is its own, in stream order: calls may
  // overlap on several streams, and a captured one takes its scratch with it.
  // (The arena may go to the next search while this call still runs, and may be
  // freed while a graph holds its address.)
  double* part = nullptr;
  GTLS_TRY_CUDA(ctx, cudaMallocFromPoolAsync(reinterpret_cast<void**>(&part), sizeof(double) * kOut * ctas,
                                             ctx->pool, st));
  model_kernel<kGrad><<<(unsigned)ctas, kAdjThreads, 0, st>>>(t, y, w, off, params, splits, part, gl_table());
  const long long values = (long long)n_curves * kOut;
  model_sum_kernel<kOut><<<(unsigned)((values + 127) / 128), 128, 0, st>>>(part, n_curves, splits, grad_out, out);
  ctx->launches += 2;
  const cudaError_t launched = cudaGetLastError();
  GTLS_TRY_CUDA(ctx, cudaFreeAsync(part, st));
  GTLS_TRY_CUDA(ctx, launched);
  return GTLS_OK;
}

}  // namespace gtls

using namespace gtls;

extern "C" int gtls_model_chi2(gtls_ctx* ctx, const double* t, const double* y, const double* w,
                               const int64_t* curve_off, int32_t n_curves, const double* params, double* chi2_out,
                               void* stream) {
  if (!ctx) return GTLS_E_INVALID;
  if (!t || !y || !w || !curve_off || !params || !chi2_out || n_curves < 1)
    return fail(ctx, GTLS_E_INVALID, "bad arguments to gtls_model_chi2");
  return model_launch<false>(ctx, t, y, w, curve_off, n_curves, params, nullptr, chi2_out,
                             static_cast<cudaStream_t>(stream));
}

extern "C" int gtls_model_chi2_grad(gtls_ctx* ctx, const double* t, const double* y, const double* w,
                                    const int64_t* curve_off, int32_t n_curves, const double* params,
                                    const double* grad_chi2, double* grad_params, void* stream) {
  if (!ctx) return GTLS_E_INVALID;
  if (!t || !y || !w || !curve_off || !params || !grad_chi2 || !grad_params || n_curves < 1)
    return fail(ctx, GTLS_E_INVALID, "bad arguments to gtls_model_chi2_grad");
  return model_launch<true>(ctx, t, y, w, curve_off, n_curves, params, grad_chi2, grad_params,
                            static_cast<cudaStream_t>(stream));
}
