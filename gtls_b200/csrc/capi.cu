// C-ABI entry points of gtls_b200: context, period grid, spectra.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstdint>
#include <cstring>
#include <string>

#include "common.cuh"
#include "spectra.cuh"

namespace gtls {

static thread_local std::string g_create_error;

constexpr size_t kPoolKeep = (size_t)64 << 20;   // bytes of a context's pool kept between calls (it grows by 32 MB at a time)

int fail(gtls_ctx* ctx, int code, const std::string& msg) {
  if (ctx) ctx->err = msg;
  else g_create_error = msg;
  return code;
}

void* arena(gtls_ctx* ctx, size_t bytes) {
  if (bytes <= ctx->arena_bytes) return ctx->arena;
  if (ctx->arena) {
    cudaDeviceSynchronize();
    cudaFree(ctx->arena);
    ctx->arena = nullptr;
    ctx->arena_bytes = 0;
  }
  size_t want = align_up(bytes + bytes / 8, (size_t)1 << 21);
  if (cudaMalloc(&ctx->arena, want) != cudaSuccess) {
    cudaGetLastError();
    ctx->arena = nullptr;
    return nullptr;
  }
  ctx->arena_bytes = want;
  return ctx->arena;
}

// ------------------------------------------------------------ period grid
// x^3 correctly rounded: x*x = h + l and h*x = p + e exactly (FMA), then one
// rounding of p + (e + l*x).
__device__ __forceinline__ double cube_rn(double x) {
  double h = x * x;
  double l = fma(x, x, -h);
  double p = h * x;
  double e = fma(h, x, -p);
  return p + fma(l, x, e);
}

// P(X) = 1 / (a3 * X + c)^3 / 86400 with numpy's operation order
// (grid.py:128-132): no contraction of a3*X + c.
__global__ void period_eval_kernel(double a3, double c, long long npts, double pmin, double pmax,
                                   double* __restrict__ tmp, int* __restrict__ bounds) {
  long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  if (i >= npts) return;
  double X = (double)(i + 1);
  double f = __dadd_rn(__dmul_rn(a3, X), c);
  double fx = cube_rn(f);
  double P = __ddiv_rn(__ddiv_rn(1.0, fx), 86400.0);
  tmp[i] = P;
  if (P > pmin && P <= pmax) {
    atomicMin(&bounds[0], (int)i);
    atomicMax(&bounds[1], (int)i);
  }
}

__global__ void period_reverse_kernel(const double* __restrict__ tmp, const int* __restrict__ bounds,
                                      double* __restrict__ out) {
  int lo = bounds[0], hi = bounds[1];
  long long cnt = hi >= lo ? (long long)(hi - lo + 1) : 0;
  long long j = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  if (j < cnt) out[j] = tmp[hi - j];
}

}  // namespace gtls

using namespace gtls;

extern "C" {

int gtls_abi_version(void) { return GTLS_ABI_VERSION; }

int64_t gtls_launch_count(const gtls_ctx* ctx) { return ctx ? ctx->launches : 0; }

int gtls_set_tuning(gtls_ctx* ctx, const gtls_tuning* t) {
  if (!ctx) return GTLS_E_INVALID;
  if (!t) return fail(ctx, GTLS_E_INVALID, "null tuning");
  auto cap_ok = [](int c) { return c == 0 || (c >= 256 && c <= 65536 && c % 256 == 0); };
  if (!cap_ok(t->tile_cap_fp32) || !cap_ok(t->tile_cap_fp64))
    return fail(ctx, GTLS_E_INVALID, "tile caps must be 0 or multiples of 256 in [256, 65536]");
  if (t->bucket_shift < -3 || t->bucket_shift > 0) return fail(ctx, GTLS_E_INVALID, "bucket_shift must be in [-3, 0]");
  if (t->records_global != 0 && t->records_global != 1) return fail(ctx, GTLS_E_INVALID, "records_global must be 0 or 1");
  ctx->tile_cap_fp32 = t->tile_cap_fp32 ? t->tile_cap_fp32 : kTileCapFp32;
  ctx->tile_cap_fp64 = t->tile_cap_fp64 ? t->tile_cap_fp64 : kTileCapFp64;
  ctx->bucket_shift = t->bucket_shift;
  ctx->records_global = t->records_global;
  return GTLS_OK;
}

int gtls_get_tuning(const gtls_ctx* ctx, gtls_tuning* t) {
  if (!ctx || !t) return GTLS_E_INVALID;
  t->tile_cap_fp32 = ctx->tile_cap_fp32;
  t->tile_cap_fp64 = ctx->tile_cap_fp64;
  t->bucket_shift = ctx->bucket_shift;
  t->records_global = ctx->records_global;
  return GTLS_OK;
}

int gtls_set_chunk_budget(gtls_ctx* ctx, uint64_t bytes) {
  if (!ctx) return GTLS_E_INVALID;
  if (bytes < ((uint64_t)1 << 20)) return fail(ctx, GTLS_E_INVALID, "chunk budget must be >= 1 MiB");
  ctx->chunk_budget = (size_t)bytes;
  return GTLS_OK;
}

int gtls_decode_status(int32_t word, char* msg, size_t cap) {
  std::string m;
  if (word == 0) m = "ok";
  if (word & 1) m += "chi2 kernel: shared-memory tile copy did not complete within its bounded wait";
  if (word & ~1) m += (m.empty() ? "" : "; ") + std::string("unknown device status bits ") + std::to_string(word & ~1);
  if (msg && cap > 0) {
    const size_t k = std::min(cap - 1, m.size());
    std::memcpy(msg, m.data(), k);
    msg[k] = 0;
  }
  return word == 0 ? GTLS_OK : GTLS_E_DEVICE;
}

const char* gtls_last_error(const gtls_ctx* ctx) {
  return ctx ? ctx->err.c_str() : g_create_error.c_str();
}

int gtls_ctx_create(int device, gtls_ctx** out) {
  if (!out) return fail(nullptr, GTLS_E_INVALID, "out is NULL");
  *out = nullptr;
  int ndev = 0;
  cudaError_t e = cudaGetDeviceCount(&ndev);
  if (e != cudaSuccess) return fail(nullptr, GTLS_E_CUDA, std::string("cudaGetDeviceCount: ") + cudaGetErrorString(e));
  if (device < 0 || device >= ndev) return fail(nullptr, GTLS_E_INVALID, "no such CUDA device");
  e = cudaSetDevice(device);
  if (e != cudaSuccess) return fail(nullptr, GTLS_E_CUDA, std::string("cudaSetDevice: ") + cudaGetErrorString(e));
  cudaDeviceProp prop;
  e = cudaGetDeviceProperties(&prop, device);
  if (e != cudaSuccess) return fail(nullptr, GTLS_E_CUDA, cudaGetErrorString(e));
  if (prop.major < 10) return fail(nullptr, GTLS_E_DEVICE, "gtls_b200 is built for sm_100a (B200)");
  // keeps what its calls gave back, up to kPoolKeep, for the next ones
  cudaMemPoolProps pp = {};
  pp.allocType = cudaMemAllocationTypePinned;
  pp.location.type = cudaMemLocationTypeDevice;
  pp.location.id = device;
  cudaMemPool_t pool = nullptr;
  unsigned long long keep = kPoolKeep;
  e = cudaMemPoolCreate(&pool, &pp);
  if (e == cudaSuccess) e = cudaMemPoolSetAttribute(pool, cudaMemPoolAttrReleaseThreshold, &keep);
  int* any_late = nullptr;
  if (e == cudaSuccess) e = cudaHostAlloc(&any_late, sizeof(int), cudaHostAllocMapped);
  if (e != cudaSuccess) {
    if (pool) cudaMemPoolDestroy(pool);
    return fail(nullptr, GTLS_E_CUDA, std::string("memory of a context: ") + cudaGetErrorString(e));
  }
  gtls_ctx* c = new gtls_ctx();
  c->device = device;
  c->pool = pool;
  c->any_late = any_late;
  c->num_sms = prop.multiProcessorCount;
  c->smem_optin = (int)prop.sharedMemPerBlockOptin;
  *out = c;
  return GTLS_OK;
}

int gtls_ctx_destroy(gtls_ctx* ctx) {
  if (!ctx) return GTLS_OK;
  cudaSetDevice(ctx->device);
  cudaDeviceSynchronize();
  if (ctx->arena) cudaFree(ctx->arena);
  if (ctx->pool) cudaMemPoolDestroy(ctx->pool);
  if (ctx->any_late) cudaFreeHost(ctx->any_late);
  delete ctx;
  return GTLS_OK;
}

int gtls_period_grid(gtls_ctx* ctx, double a_over_3, double c, int64_t n_points, double period_min,
                     double period_max, double* periods_out, int64_t* count_out, void* stream) {
  if (!ctx) return GTLS_E_INVALID;
  if (!periods_out || !count_out || n_points < 0 || n_points >= (1LL << 31))
    return fail(ctx, GTLS_E_INVALID, "bad arguments to gtls_period_grid");
  *count_out = 0;
  if (n_points == 0) return GTLS_OK;
  GTLS_TRY_CUDA(ctx, cudaSetDevice(ctx->device));
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  size_t bytes = align_up(sizeof(double) * n_points, 256) + 256;
  void* mem = arena(ctx, bytes);
  if (!mem) return fail(ctx, GTLS_E_NOMEM, "scratch allocation failed");
  Carver cv(mem);
  double* tmp = cv.take<double>(n_points);
  int* bounds = cv.take<int>(2);
  int init[2] = {0x7fffffff, -1};
  GTLS_TRY_CUDA(ctx, cudaMemcpyAsync(bounds, init, sizeof(init), cudaMemcpyHostToDevice, st));
  unsigned g = (unsigned)((n_points + 255) / 256);
  period_eval_kernel<<<g, 256, 0, st>>>(a_over_3, c, n_points, period_min, period_max, tmp, bounds);
  period_reverse_kernel<<<g, 256, 0, st>>>(tmp, bounds, periods_out);
  ctx->launches += 2;
  GTLS_TRY_CUDA(ctx, cudaGetLastError());
  int hb[2];
  GTLS_TRY_CUDA(ctx, cudaMemcpyAsync(hb, bounds, sizeof(hb), cudaMemcpyDeviceToHost, st));
  GTLS_TRY_CUDA(ctx, cudaStreamSynchronize(st));
  *count_out = hb[1] >= hb[0] ? (int64_t)(hb[1] - hb[0] + 1) : 0;
  return GTLS_OK;
}

int gtls_spectra(gtls_ctx* ctx, const double* chi2, const uint8_t* mask, int64_t n, double oversampling_factor,
                 double* sr, double* power_raw, double* power, double* sde_raw, double* sde, void* stream) {
  if (!ctx) return GTLS_E_INVALID;
  if (!chi2 || !sr || !power_raw || !power || !sde_raw || !sde || n < 1)
    return fail(ctx, GTLS_E_INVALID, "bad arguments to gtls_spectra");
  const long long k = spectra_window(oversampling_factor);
  if (k == 0) return fail(ctx, GTLS_E_INVALID, "oversampling_factor * 30 must be an integer");
  GTLS_TRY_CUDA(ctx, cudaSetDevice(ctx->device));
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  size_t bytes = 0;
  carve_size<double>(bytes, kSpecParts);
  carve_size<SpecState>(bytes, 1);
  carve_size<double>(bytes, n);
  void* mem = arena(ctx, bytes + 256);
  if (!mem) return fail(ctx, GTLS_E_NOMEM, "scratch allocation failed");
  Carver cv(mem);
  SpecScratch s;
  s.part = cv.take<double>(kSpecParts);
  s.state = cv.take<SpecState>(1);
  s.med = cv.take<double>(n);
  // (a window of more than n / 2 periods is never taken)
  ctx->launches += spectra_launch(chi2, mask, n, (int)std::min<long long>(k, n), sr, power_raw, power, s, st);
  GTLS_TRY_CUDA(ctx, cudaGetLastError());
  SpecState hs;
  GTLS_TRY_CUDA(ctx, cudaMemcpyAsync(&hs, s.state, sizeof(hs), cudaMemcpyDeviceToHost, st));
  GTLS_TRY_CUDA(ctx, cudaStreamSynchronize(st));
  *sde = n > 2 * k ? hs.sde : hs.sde_raw;
  *sde_raw = hs.sde_raw;
  return GTLS_OK;
}

}  // extern "C"
