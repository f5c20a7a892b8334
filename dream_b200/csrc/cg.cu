// cg.cu -- vector updates of the conjugate-gradient reconstruction
// (min ||DAS_w^T x - Y||^2 + lam ||x||^2 on the normal equations), fused around
// its two reductions: three launches per iteration beside the operator's two.
//
// The vectors are one image long (65536 points: 256 KB), so a launch is bound by
// its latency, not by memory, and their number is what costs: with 32x32
// elements, 256x256 points and 10 iterations a solve takes 1.50 ms against
// 1.90 ms with the twelve element-wise and reduction launches of an iteration
// in torch. Every element-wise operation rounds as those did (product and sum
// apart); the dot products are summed in FP64 (FP32 there), over the blocks in a
// fixed order.
#include <cuda_runtime.h>
#include <stdint.h>

#include <algorithm>
#include <string>

#include "das_kernels.h"
#include "dream_das.h"

namespace dream {
namespace {

// One point per thread up to 262144 points (7 blocks an SM); strided beyond.
constexpr int CG_THREADS = 256, CG_BLOCKS = 1024;

// One solve's scalars and the partial sums of a launch's blocks.
struct CgScratch {
  float rs, alpha, beta;
  unsigned int done;  // blocks of the current launch that have stored their sum
  double part[CG_BLOCKS];
};
static_assert(sizeof(CgScratch) <= DREAM_CG_SCRATCH_BYTES, "scratch size in the header");

// Sum of v over the grid, in every thread of the block that finishes last; the
// others return false.
__device__ bool grid_sum(double v, CgScratch *s, double &sum) {
  __shared__ double warps[CG_THREADS / 32];
  __shared__ bool last;
  for (int o = 16; o; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  if ((threadIdx.x & 31) == 0) warps[threadIdx.x >> 5] = v;
  __syncthreads();
  if (threadIdx.x == 0) {
    double b = 0.0;
    for (int w = 0; w < CG_THREADS / 32; w++) b += warps[w];
    s->part[blockIdx.x] = b;
    __threadfence();
    last = atomicAdd(&s->done, 1u) == gridDim.x - 1;
  }
  __syncthreads();
  if (!last) return false;
  __threadfence();
  double b = 0.0;
  for (unsigned i = threadIdx.x; i < gridDim.x; i += CG_THREADS) b += __ldcg(&s->part[i]);
  for (int o = 16; o; o >>= 1) b += __shfl_xor_sync(0xffffffffu, b, o);
  if ((threadIdx.x & 31) == 0) warps[threadIdx.x >> 5] = b;
  __syncthreads();
  sum = 0.0;
  for (int w = 0; w < CG_THREADS / 32; w++) sum += warps[w];
  if (threadIdx.x == 0) s->done = 0;
  return true;
}

__global__ void __launch_bounds__(CG_THREADS) cg_start_kernel(const float *__restrict__ r, int64_t n, CgScratch *s) {
  double v = 0.0, sum;
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
    v += (double)r[i] * r[i];
  if (grid_sum(v, s, sum) && threadIdx.x == 0) s->rs = (float)sum;
}

// Ap += lam * p; alpha = rs / <p, Ap>
__global__ void __launch_bounds__(CG_THREADS) cg_alpha_kernel(float *__restrict__ Ap, const float *__restrict__ p,
                                                              int64_t n, float lam, CgScratch *s) {
  double v = 0.0, sum;
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    const float pi = p[i], a = __fadd_rn(Ap[i], __fmul_rn(lam, pi));
    Ap[i] = a;
    v += (double)pi * a;
  }
  if (grid_sum(v, s, sum) && threadIdx.x == 0) s->alpha = __fdiv_rn(s->rs, (float)sum);
}

// x += alpha * p, r -= alpha * Ap; rs = <r, r>, beta its ratio to the last one
__global__ void __launch_bounds__(CG_THREADS) cg_update_kernel(float *__restrict__ x, float *__restrict__ r,
                                                               const float *__restrict__ p,
                                                               const float *__restrict__ Ap, int64_t n,
                                                               float *__restrict__ rs_out, CgScratch *s) {
  const float alpha = s->alpha;
  double v = 0.0, sum;
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    x[i] = __fadd_rn(x[i], __fmul_rn(alpha, p[i]));
    const float ri = __fsub_rn(r[i], __fmul_rn(alpha, Ap[i]));
    r[i] = ri;
    v += (double)ri * ri;
  }
  if (grid_sum(v, s, sum) && threadIdx.x == 0) {
    const float rs = (float)sum;
    s->beta = __fdiv_rn(rs, s->rs);
    s->rs = rs;
    *rs_out = rs;
  }
}

// p = r + beta * p
__global__ void __launch_bounds__(CG_THREADS) cg_next_kernel(float *__restrict__ p, const float *__restrict__ r,
                                                             int64_t n, const CgScratch *s) {
  const float beta = s->beta;
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
    p[i] = __fadd_rn(r[i], __fmul_rn(beta, p[i]));
}

unsigned cg_grid(int64_t n) {
  return (unsigned)std::max<int64_t>(1, std::min<int64_t>(CG_BLOCKS, (n + CG_THREADS - 1) / CG_THREADS));
}

struct OnDevice {
  int prev = -1;
  bool ok = true;
  explicit OnDevice(int dev) {
    if (cudaGetDevice(&prev) != cudaSuccess) prev = -1;
    if (prev != dev) ok = cudaSetDevice(dev) == cudaSuccess;
  }
  ~OnDevice() {
    int cur = -1;
    if (prev >= 0 && cudaGetDevice(&cur) == cudaSuccess && cur != prev) cudaSetDevice(prev);
  }
};

int cg_status(cudaError_t e, const char *what) {
  if (e != cudaSuccess) return set_last_error(DREAM_ERR_CUDA, std::string(what) + ": " + cudaGetErrorString(e));
  return 0;
}

}  // namespace
}  // namespace dream

using namespace dream;

extern "C" {

int dream_das_cg_start(const float *d_r, int64_t n, void *d_scratch, int device, void *stream) {
  DREAM_API_TRY
  if (n < 0 || d_scratch == nullptr || (n > 0 && d_r == nullptr))
    return set_last_error(DREAM_ERR_ARGUMENT, "cg: NULL pointer or negative size");
  OnDevice on(device);
  if (!on.ok) return set_last_error(DREAM_ERR_CUDA, "cudaSetDevice failed");
  const cudaStream_t st = (cudaStream_t)stream;
  const cudaError_t e = cudaMemsetAsync(d_scratch, 0, sizeof(CgScratch), st);
  if (e != cudaSuccess) return cg_status(e, "cg start");
  cg_start_kernel<<<cg_grid(n), CG_THREADS, 0, st>>>(d_r, n, (CgScratch *)d_scratch);
  return cg_status(cudaGetLastError(), "cg start");
  DREAM_API_CATCH
}

int dream_das_cg_step(float *d_x, float *d_r, float *d_p, float *d_Ap, int64_t n, float lam, float *d_rs,
                      void *d_scratch, int device, void *stream) {
  DREAM_API_TRY
  if (n < 0 || d_scratch == nullptr || d_rs == nullptr ||
      (n > 0 && (d_x == nullptr || d_r == nullptr || d_p == nullptr || d_Ap == nullptr)))
    return set_last_error(DREAM_ERR_ARGUMENT, "cg: NULL pointer or negative size");
  OnDevice on(device);
  if (!on.ok) return set_last_error(DREAM_ERR_CUDA, "cudaSetDevice failed");
  const cudaStream_t st = (cudaStream_t)stream;
  CgScratch *s = (CgScratch *)d_scratch;
  cg_alpha_kernel<<<cg_grid(n), CG_THREADS, 0, st>>>(d_Ap, d_p, n, lam, s);
  cg_update_kernel<<<cg_grid(n), CG_THREADS, 0, st>>>(d_x, d_r, d_p, d_Ap, n, d_rs, s);
  cg_next_kernel<<<cg_grid(n), CG_THREADS, 0, st>>>(d_p, d_r, n, s);
  return cg_status(cudaGetLastError(), "cg step");
  DREAM_API_CATCH
}

}  // extern "C"
