// Component-level device entry points mirroring the reference's component
// kernels and the tests that drive them:
//   * map_idx gather                   (src/permcheck.cu:4-19)
//   * RuizClass on explicit arrays     (src/RuizClass.cpp:54-88, kernels
//                                       src/matrix_vector_ops.cu:146-266)
// The Cholesky and Schur-CG components run on the Engine (engine.cu).
#include <algorithm>
#include <climits>
#include <cstring>
#include <mutex>
#include <stdexcept>
#include <string>
#include <unordered_map>
#include <vector>

#include "components.hpp"
#include "engine.hpp"

namespace hykkt {

__global__ void k_map_idx(int n, const int* __restrict__ map, const double* __restrict__ oldv, double* __restrict__ newv) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) newv[i] = oldv[map[i]];
}

void map_index(int n, const int* d_map, const double* d_old, double* d_new, cudaStream_t st) {
  if (n <= 0) return;
  k_map_idx<<<(n + 255) / 256, 256, 0, st>>>(n, d_map, d_old, d_new);
  HYKKT_CUDA(cudaGetLastError());
}

// Ruiz sweeps on [A B^T; B 0], eight lanes per row (the rows of power-grid
// blocks hold 2 to 16 entries: a warp each left most lanes idle); the same
// operation order as the product path (1/sqrt of the row max, v *= s_i*s_j).
// Bounded by latency and launches, not by the 10 MB that a 10,000-bus system
// moves.
constexpr int kRuizLanes = 8;

struct RuizArrays {
  int n, m;
  double* a_v;
  const int *a_i, *a_j;
  double* bt_v;
  const int *bt_i, *bt_j;
  double* b_v;
  const int *b_i, *b_j;
  double *rhs1, *rhs2, *max_d;
};

// 1/sqrt of the row's largest magnitude, from the lanes' own maxima (a NaN
// never compares greater, as in the reference's kernel)
__device__ __forceinline__ double ruiz_row_scale(double ml, double mu, bool top) {
#pragma unroll
  for (int o = kRuizLanes / 2; o > 0; o >>= 1) {
    const double a = __shfl_xor_sync(0xffffffffu, ml, o), b = __shfl_xor_sync(0xffffffffu, mu, o);
    if (a > ml) ml = a;
    if (b > mu) mu = b;
  }
  return 1.0 / sqrt(top ? (ml > mu ? ml : mu) : ml);
}

__global__ void k_ruizc_rowmax(RuizArrays r, double* scale) {
  const int lane = threadIdx.x & (kRuizLanes - 1);
  const int row = (int)((blockIdx.x * (int64_t)blockDim.x + threadIdx.x) / kRuizLanes);
  const bool in = row < r.n + r.m, top = row < r.n;
  double ml = 0.0, mu = 0.0;
  if (in) {
    const double* v = top ? r.a_v : r.b_v;
    const int* rp = top ? r.a_i + row : r.b_i + (row - r.n);
    for (int p = rp[0] + lane; p < rp[1]; p += kRuizLanes) { const double e = fabs(v[p]); if (e > ml) ml = e; }
    if (top)
      for (int p = r.bt_i[row] + lane; p < r.bt_i[row + 1]; p += kRuizLanes) { const double e = fabs(r.bt_v[p]); if (e > mu) mu = e; }
  }
  const double s = ruiz_row_scale(ml, mu, top);
  if (in && lane == 0) scale[row] = s;
}

// One sweep's scaling.  first: max_d starts from it (reset_scaling,
// RuizClass.cpp:95-98, sets 1).  next (optional): the row scales of the sweep
// that follows, from the values just written, which saves that sweep's own
// pass and launch.
__global__ void k_ruizc_scale(RuizArrays r, const double* __restrict__ scale, double* next, int first) {
  const int lane = threadIdx.x & (kRuizLanes - 1);
  const int row = (int)((blockIdx.x * (int64_t)blockDim.x + threadIdx.x) / kRuizLanes);
  const bool in = row < r.n + r.m, top = row < r.n;
  double ml = 0.0, mu = 0.0;
  if (in) {
    const double si = scale[row];
    double* v = top ? r.a_v : r.b_v;
    const int* ci = top ? r.a_j : r.b_j;
    const int* rp = top ? r.a_i + row : r.b_i + (row - r.n);
    for (int p = rp[0] + lane; p < rp[1]; p += kRuizLanes) {
      const double x = __dmul_rn(v[p], __dmul_rn(si, scale[ci[p]])), e = fabs(x);
      v[p] = x;
      if (e > ml) ml = e;
    }
    if (top)
      for (int p = r.bt_i[row] + lane; p < r.bt_i[row + 1]; p += kRuizLanes) {
        const double x = __dmul_rn(r.bt_v[p], __dmul_rn(si, scale[r.n + r.bt_j[p]])), e = fabs(x);
        r.bt_v[p] = x;
        if (e > mu) mu = e;
      }
    if (lane == 0) {
      double* rhs = top ? r.rhs1 + row : r.rhs2 + (row - r.n);
      *rhs = __dmul_rn(*rhs, si);
      r.max_d[row] = first ? si : __dmul_rn(r.max_d[row], si);
    }
  }
  if (!next) return;
  const double s = ruiz_row_scale(ml, mu, top);
  if (in && lane == 0) next[row] = s;
}

__global__ void k_fill(int n, double v, double* x) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) x[i] = v;
}

// scale1 (optional): a second scale vector, for the fused sweeps
static void ruiz_sweeps(int its, const RuizArrays& r, double* scale0, double* scale1, cudaStream_t st) {
  const int tot = r.n + r.m;
  if (its == 0) {
    k_fill<<<(tot + 255) / 256, 256, 0, st>>>(tot, 1.0, r.max_d);
  }
  const int grid = (int)(((int64_t)tot * kRuizLanes + 255) / 256);
  for (int s = 0; s < its; ++s) {
    if (s == 0 || !scale1) k_ruizc_rowmax<<<grid, 256, 0, st>>>(r, scale0);
    k_ruizc_scale<<<grid, 256, 0, st>>>(r, scale0, scale1 && s + 1 < its ? scale1 : nullptr, s == 0);
    if (scale1) std::swap(scale0, scale1);
  }
  HYKKT_CUDA(cudaGetLastError());
}

// A pool of the library's own for the component's scratch, one per device:
// with the default pool every call that is followed by a synchronisation gives
// the memory back to the device and takes it again (300 us of a 340 us call on
// the 10,000-bus system).  It keeps at most kRuizPoolKeep bytes between calls;
// allocations are stream-ordered, so calls on several streams and threads each
// have their own.
constexpr uint64_t kRuizPoolKeep = 32ull << 20;
static cudaMemPool_t ruiz_pool_on_current_device() {
  static std::mutex mu;
  static std::unordered_map<int, cudaMemPool_t> pools;
  int dev = 0;
  HYKKT_CUDA(cudaGetDevice(&dev));
  std::lock_guard<std::mutex> lock(mu);
  auto it = pools.find(dev);
  if (it != pools.end()) return it->second;
  cudaMemPoolProps props{};
  props.allocType = cudaMemAllocationTypePinned;
  props.location.type = cudaMemLocationTypeDevice;
  props.location.id = dev;
  cudaMemPool_t pool = nullptr;
  HYKKT_CUDA(cudaMemPoolCreate(&pool, &props));
  uint64_t keep = kRuizPoolKeep;
  HYKKT_CUDA(cudaMemPoolSetAttribute(pool, cudaMemPoolAttrReleaseThreshold, &keep));
  pools[dev] = pool;
  return pool;
}

void ruiz_scale(int its, int n, int m, double* a_v, const int* a_i, const int* a_j, double* bt_v, const int* bt_i,
                const int* bt_j, double* b_v, const int* b_i, const int* b_j, double* rhs1, double* rhs2, double* max_d,
                cudaStream_t st) {
  if (its < 0 || n < 0 || m < 0) throw std::invalid_argument("ruiz_scale: negative size or sweep count");
  const int tot = n + m;
  if (tot <= 0) return;
  double* scale = nullptr;
  HYKKT_CUDA(cudaMallocFromPoolAsync(reinterpret_cast<void**>(&scale), 2 * (size_t)tot * sizeof(double),
                                     ruiz_pool_on_current_device(), st));
  ruiz_sweeps(its, RuizArrays{n, m, a_v, a_i, a_j, bt_v, bt_i, bt_j, b_v, b_i, b_j, rhs1, rhs2, max_d}, scale,
              scale + tot, st);
  HYKKT_CUDA(cudaFreeAsync(scale, st));
}

// ---------------------------------------------------------------------------
// Ruiz scaling that allocates nothing.
//
// ruiz_scale() above takes its n+m scale vector from the stream-ordered pool
// on every call.  Some callers cannot allocate where they scale: an
// interior-point loop that reserves all of its device memory before the
// first iteration and must not touch the allocator inside it (a pool
// allocation there can fail under a fixed memory budget, or wait on other
// streams' frees).  This variant takes the scale vector from a fixed array
// compiled into the library.
//   * limit: n + m <= kRuizNoAllocMaxRows (1,048,576 rows, 8 MiB of
//     doubles); larger systems are rejected before anything is enqueued;
//   * set-up: the first call on a device resolves the array's address on
//     that device (cudaGetSymbolAddress, with that device current) and
//     caches it; make that first call before any stream capture.  The cache
//     lives as long as the process's context on the device: after
//     cudaDeviceReset the module is loaded again at another address, so a
//     process that resets a device must not call this entry point after it;
//   * nothing has to start at zero: each sweep's row-max kernel writes all
//     n+m entries before the scaling kernel of the sweep reads them;
//   * all calls on one device share the one array, so calls that overlap in
//     time (from other host threads, or on other streams whose work is still
//     in flight) race on it: the caller serialises them, e.g. on one stream.
// ---------------------------------------------------------------------------
constexpr int kRuizNoAllocMaxRows = 1 << 20;
static __device__ __align__(256) double g_ruiz_scale_scratch[kRuizNoAllocMaxRows];

static double* ruiz_scratch_on_current_device() {
  static std::mutex mu;
  static std::unordered_map<int, double*> addr;
  int dev = 0;
  HYKKT_CUDA(cudaGetDevice(&dev));
  std::lock_guard<std::mutex> lock(mu);
  auto it = addr.find(dev);
  if (it != addr.end()) return it->second;
  void* p = nullptr;
  HYKKT_CUDA(cudaGetSymbolAddress(&p, g_ruiz_scale_scratch));
  addr[dev] = static_cast<double*>(p);
  return static_cast<double*>(p);
}

int ruiz_noalloc_max_rows() { return kRuizNoAllocMaxRows; }

void ruiz_scale_noalloc(int its, int n, int m, double* a_v, const int* a_i, const int* a_j, double* bt_v,
                        const int* bt_i, const int* bt_j, double* b_v, const int* b_i, const int* b_j, double* rhs1,
                        double* rhs2, double* max_d, cudaStream_t st) {
  if (its < 0 || n < 0 || m < 0) throw std::invalid_argument("ruiz_scale_noalloc: negative size or sweep count");
  const int64_t tot = (int64_t)n + m;
  if (tot > kRuizNoAllocMaxRows)
    throw std::invalid_argument("ruiz_scale_noalloc: n + m = " + std::to_string(tot) +
                                " exceeds the fixed scratch of " + std::to_string(kRuizNoAllocMaxRows) + " rows");
  double* scale = ruiz_scratch_on_current_device();
  if (tot == 0) return;
  ruiz_sweeps(its, RuizArrays{n, m, a_v, a_i, a_j, bt_v, bt_i, bt_j, b_v, b_i, b_j, rhs1, rhs2, max_d}, scale,
              nullptr, st);
}

// FP64 throughput probe: 8 independent FMA chains per thread.
__global__ void k_dfma_peak(double* out, int iters, double a, double b) {
  double x0 = threadIdx.x, x1 = x0 + 1, x2 = x0 + 2, x3 = x0 + 3, x4 = x0 + 4, x5 = x0 + 5, x6 = x0 + 6, x7 = x0 + 7;
  for (int i = 0; i < iters; ++i) {
    x0 = fma(x0, a, b); x1 = fma(x1, a, b); x2 = fma(x2, a, b); x3 = fma(x3, a, b);
    x4 = fma(x4, a, b); x5 = fma(x5, a, b); x6 = fma(x6, a, b); x7 = fma(x7, a, b);
  }
  const double s = ((x0 + x1) + (x2 + x3)) + ((x4 + x5) + (x6 + x7));
  if (s == 12345.678) out[0] = s;  // keeps the chains live
}

// FP64 tensor-pipe probe: eight independent accumulator chains per warp of
// mma.sync m8n8k4 (FP64 operands and accumulators; 512 flops per warp
// instruction).  mode 1: every warp issues mma; mode 2: even warps mma, odd
// warps the DFMA chains of k_dfma_peak (do the two share one pipe?).
__global__ void k_fp64_probe(double* out, int iters, double a, double b, int mode) {
  const int warp = threadIdx.x >> 5;
  double s = 0.0;
  if (mode == 1 || (mode == 2 && (warp & 1) == 0)) {
    double c[8][2];
#pragma unroll
    for (int k = 0; k < 8; ++k) c[k][0] = c[k][1] = threadIdx.x + k;
    const double av = a + 1e-9 * threadIdx.x, bv = b;
    for (int i = 0; i < iters; ++i) {
#pragma unroll
      for (int k = 0; k < 8; ++k)
        asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};"
                     : "+d"(c[k][0]), "+d"(c[k][1])
                     : "d"(av), "d"(bv));
    }
#pragma unroll
    for (int k = 0; k < 8; ++k) s += c[k][0] + c[k][1];
  } else {
    double x0 = threadIdx.x, x1 = x0 + 1, x2 = x0 + 2, x3 = x0 + 3, x4 = x0 + 4, x5 = x0 + 5, x6 = x0 + 6, x7 = x0 + 7;
    // 4x the chain steps of an mma warp's loop: a DFMA warp instruction does
    // 64 flops, an m8n8k4 one 512, so both kinds issue about equal work
    for (int i = 0; i < 4 * iters; ++i) {
      x0 = fma(x0, a, b); x1 = fma(x1, a, b); x2 = fma(x2, a, b); x3 = fma(x3, a, b);
      x4 = fma(x4, a, b); x5 = fma(x5, a, b); x6 = fma(x6, a, b); x7 = fma(x7, a, b);
    }
    s = ((x0 + x1) + (x2 + x3)) + ((x4 + x5) + (x6 + x7));
  }
  if (s == 12345.678) out[0] = s;
}

double fp64_probe_tflops(int mode) {
  if (mode < 0 || mode > 2) throw std::invalid_argument("fp64 probe mode must be 0, 1 or 2");
  if (mode == 0) return fp64_peak_tflops();
  int dev = 0, sms = 0;
  HYKKT_CUDA(cudaGetDevice(&dev));
  HYKKT_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
  double* out = nullptr;
  HYKKT_CUDA(cudaMalloc(&out, sizeof(double)));
  const int blocks = sms * 8, threads = 256, iters = 1024;
  cudaEvent_t a, b;
  HYKKT_CUDA(cudaEventCreate(&a));
  HYKKT_CUDA(cudaEventCreate(&b));
  k_fp64_probe<<<blocks, threads>>>(out, iters, 0.999999, 1e-7, mode);  // warm-up
  HYKKT_CUDA(cudaGetLastError());
  float best = 1e30f;
  for (int r = 0; r < 5; ++r) {
    HYKKT_CUDA(cudaEventRecord(a));
    k_fp64_probe<<<blocks, threads>>>(out, iters, 0.999999, 1e-7, mode);
    HYKKT_CUDA(cudaEventRecord(b));
    HYKKT_CUDA(cudaEventSynchronize(b));
    float ms = 0;
    HYKKT_CUDA(cudaEventElapsedTime(&ms, a, b));
    best = std::min(best, ms);
  }
  cudaEventDestroy(a);
  cudaEventDestroy(b);
  cudaFree(out);
  const double warps = (double)blocks * threads / 32;
  // mma warps: 8 chains x iters x 512 flops; DFMA warps: 32 lanes x 8 chains x 4 iters x 2 flops
  const double per_mma_warp = 8.0 * iters * 512.0, per_dfma_warp = 32.0 * 8.0 * 4.0 * iters * 2.0;
  const double flops = mode == 1 ? warps * per_mma_warp : warps / 2 * (per_mma_warp + per_dfma_warp);
  return flops / (best * 1e-3) / 1e12;
}

double fp64_peak_tflops() {
  int dev = 0, sms = 0;
  HYKKT_CUDA(cudaGetDevice(&dev));
  HYKKT_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
  double* out = nullptr;
  HYKKT_CUDA(cudaMalloc(&out, sizeof(double)));
  const int blocks = sms * 8, threads = 256, iters = 4096;
  cudaEvent_t a, b;
  HYKKT_CUDA(cudaEventCreate(&a));
  HYKKT_CUDA(cudaEventCreate(&b));
  k_dfma_peak<<<blocks, threads>>>(out, iters, 0.999999, 1e-7);  // warm-up
  float best = 1e30f;
  for (int r = 0; r < 5; ++r) {
    HYKKT_CUDA(cudaEventRecord(a));
    k_dfma_peak<<<blocks, threads>>>(out, iters, 0.999999, 1e-7);
    HYKKT_CUDA(cudaEventRecord(b));
    HYKKT_CUDA(cudaEventSynchronize(b));
    float ms = 0;
    HYKKT_CUDA(cudaEventElapsedTime(&ms, a, b));
    best = std::min(best, ms);
  }
  cudaEventDestroy(a);
  cudaEventDestroy(b);
  cudaFree(out);
  const double flops = 2.0 * 8.0 * iters * (double)blocks * threads;
  return flops / (best * 1e-3) / 1e12;
}

}  // namespace hykkt
