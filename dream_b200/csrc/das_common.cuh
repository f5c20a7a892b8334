// das_common.cuh -- device helpers shared by the DAS kernels (sm_100a).
//
// Exact arithmetic: every product, sum and square root that feeds a sample
// index goes through the round-to-nearest intrinsics, so nvcc never fuses a
// multiply and an add (an FMA would change the rounding and hence, at times,
// the selected sample). Square roots are the IEEE correctly rounded ones,
// which is what std::sqrt gives the reference CPU code.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include <map>
#include <mutex>
#include <utility>

namespace dream {

enum Method : int { SAFT = 0, TFM = 1, RCA_COLTX = 2, RCA_ROWTX = 3 };

template <class T>
struct Ar;

template <>
struct Ar<double> {
  static __device__ __forceinline__ double add(double a, double b) { return __dadd_rn(a, b); }
  static __device__ __forceinline__ double sub(double a, double b) { return __dsub_rn(a, b); }
  static __device__ __forceinline__ double mul(double a, double b) { return __dmul_rn(a, b); }
  static __device__ __forceinline__ double sqrt(double a) { return __dsqrt_rn(a); }
};

template <>
struct Ar<float> {
  static __device__ __forceinline__ float add(float a, float b) { return __fadd_rn(a, b); }
  static __device__ __forceinline__ float sub(float a, float b) { return __fsub_rn(a, b); }
  static __device__ __forceinline__ float mul(float a, float b) { return __fmul_rn(a, b); }
  static __device__ __forceinline__ float sqrt(float a) { return __fsqrt_rn(a); }
};

// |g - r| / cp with the reference association ((dx*dx + dy*dy) + dz*dz).
template <class T>
__device__ __forceinline__ T leg_time(T gx, T gy, T gz, T one_over_cp) {
  using A = Ar<T>;
  T ss = A::add(A::add(A::mul(gx, gx), A::mul(gy, gy)), A::mul(gz, gz));
  return A::mul(A::sqrt(ss), one_over_cp);
}

// Truncation toward zero of p, for p already known to lie in (-1, K):
// that is floor(max(p, 0)). Adding 2^52 (2^23 for float) with round-toward-
// zero leaves floor(x) in the low mantissa bits for 0 <= x < 2^52 (2^23),
// which avoids the slow float->int conversion unit.
__device__ __forceinline__ int trunc_index(double p) {
  double v = __dadd_rz(fmax(p, 0.0), 4503599627370496.0);  // 2^52
  return __double2loint(v);
}
__device__ __forceinline__ int trunc_index(float p) {
  float v = __fadd_rz(fmaxf(p, 0.0f), 8388608.0f);  // 2^23
  return __float_as_int(v) - 0x4B000000;
}

// Bounds-checked builds (nvcc -DDREAM_DAS_CHECKED, `python -m dream_b200.build
// --checked`): every A-scan gather verifies its element index against the
// buffer's extent; a violation is counted in *bad and the load is skipped.
// The normal build compiles this to the plain load.
template <class T>
__device__ __forceinline__ bool gather_ok(int64_t i, int64_t n, unsigned long long *bad) {
#ifdef DREAM_DAS_CHECKED
  if (i < 0 || i >= n) {
    if (bad) atomicAdd(bad, 1ull);
    return false;
  }
#endif
  return true;
}

// Warp-aggregated add of a per-thread count to a global counter. Must be
// called by all 32 lanes of the warp.
__device__ __forceinline__ void add_count(unsigned long long *ctr, unsigned int v) {
  unsigned int s = __reduce_add_sync(0xffffffffu, v);
  if (ctr != nullptr && (threadIdx.x & 31) == 0 && s) atomicAdd(ctr, (unsigned long long)s);
}

// Image volumes. The slow axis of a hinted grid, n_slow lines of n_fast points,
// is often a plane of lines: rows of lines that share x (or y). Tiles of
// neighbours in both directions read fewer sectors of an A-scan than tiles along
// one row: 8 x 4 x 4 points of a 128 x 128 x 256 volume 8.4 sectors against 12.8
// for 8 x 16, their warps' 4 x 2 x 4 patches 4.8 against 6.3. 128x128 elements,
// 64x64x128 points, FP32 storage: gather 4.47 -> 3.60 ms, adjoint 18.7 -> 8.7
// (its windows are as long as a tile's span of samples); 32x32x128 points in
// FP64 3.10 -> 2.80, FP32 1.79 -> 1.41. Bands of 2 rows: 3.64, of 8: 4.19.
//
// volume_row: lines of a row of the volume (0: none found), by the whole block
// from the coordinates, at most VOLUME_SCAN of them: one load per line, 1 - 2 us
// a block, the same answer in every block, nothing kept. A call of its own, which
// costs the kernels around it no registers.
constexpr int VOLUME_ROWS = 4, VOLUME_SCAN = 1024;
// fewest terms per point for which the search is worth its time (576 terms, 16x16x32 points, FP64: 0.0324 against
// 0.0305 ms; 4096 terms, 40x40x100 points: 0.70 against 0.82)
constexpr int VOLUME_TERMS = 1024;
template <class T>
__device__ __noinline__ uint32_t volume_row(const T *Ro, int64_t No, int64_t n_fast, int64_t n_slow) {
  __shared__ uint32_t s_row;
  if (n_slow < 2 * VOLUME_ROWS || n_slow >= (int64_t(1) << 31)) return 0;
  const T *y = Ro + No;
  const bool xm = Ro[n_fast] != Ro[0], ym = y[n_fast] != y[0];
  if (xm == ym) return 0;
  const T *fixed = xm ? y : Ro;  // the coordinate that a row shares
  const T v = fixed[0];
  if (fixed[(n_slow - 1) * n_fast] == v) return 0;  // one row: a plane
  if (threadIdx.x == 0) s_row = 0;
  const int64_t end = min(n_slow, (int64_t)VOLUME_SCAN + 1);
  for (int64_t q = 2; q < end; q += blockDim.x) {
    const int64_t s = q + threadIdx.x;
    const bool hit = s < end && fixed[s * n_fast] != v;
    if (__syncthreads_or(hit)) {
      if (hit) atomicMax(&s_row, 0xffffffffu - (uint32_t)s);
      __syncthreads();
      const uint32_t row = 0xffffffffu - s_row;
      return n_slow % row == 0 ? row : 0;
    }
  }
  return 0;
}

// Line at place q of the tiles' order: VOLUME_ROWS rows at a time (fewer at the
// end), across them first; row 0: the lines' own order. A permutation of
// [0, n_slow).
__device__ __forceinline__ int64_t volume_line(int64_t q, uint32_t row, int64_t n_slow) {
  if (row == 0 || q >= n_slow) return q;
  const uint32_t u = (uint32_t)q, band = VOLUME_ROWS * row, b = u / band, r = u - b * band;
  const uint32_t rows = min((uint32_t)VOLUME_ROWS, (uint32_t)n_slow / row - b * VOLUME_ROWS);
  return (int64_t)(b * VOLUME_ROWS + r % rows) * row + r / rows;
}

// Raises a kernel's dynamic shared-memory limit once per (kernel, device):
// later launches (including ones being captured into a CUDA graph) then issue
// no attribute call.
template <class F>
inline cudaError_t ensure_smem(F *kernel, size_t bytes) {
  static std::mutex mu;
  static std::map<std::pair<const void *, int>, size_t> done;
  if (bytes <= 32 * 1024) return cudaSuccess;  // 48 KB hold without it, a kernel's static arrays included
  int dev = 0;
  cudaGetDevice(&dev);
  std::lock_guard<std::mutex> lk(mu);
  auto key = std::make_pair(reinterpret_cast<const void *>(kernel), dev);
  auto it = done.find(key);
  if (it != done.end() && it->second >= bytes) return cudaSuccess;
  cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
  if (e == cudaSuccess) done[key] = bytes;
  return e;
}

}  // namespace dream
