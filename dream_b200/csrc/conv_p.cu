// conv_p.cu -- column-wise full linear convolution on the GPU: the conv_p /
// fftconv_p step of DREAM that turns spatial impulse responses into A-scans
// (extra_src/conv.cc:34-78, extra_src/fftconv_p.cc, extra_src/oct_conv_p.cc).
//
//   Y[:, n] (=|+=|-=) A[:, n] * B[:, n or 0]     Y has A_M + B_M - 1 rows
//
// Exactness. The reference's direct form adds zr[i+j] += xr[i]*yr[j] with i
// outer, so output k receives its products in ascending i (= descending j),
// each product rounded, then added. The kernels keep that order per output
// and never fuse the product into the add, so they reproduce conv()
// bit for bit; FFTW's fftconv_p differs from it by rounding only.
//
// Layout. A CTA owns 4 warps x 32 lanes x R consecutive outputs of one
// column; its window of A (outputs + B_M - 1 samples, zero outside the column)
// and B, reversed, are staged in shared memory. Lane l of warp w holds outputs
// k = k_w + R*l + r. Stepping j downwards, lane l needs A[k_w + R*l + r - j]: a
// window of R samples that slides by one per step, so a step is one new A
// sample, one B sample (a broadcast) and R products and adds. R is odd, which
// puts the 32 lanes' samples in distinct banks with no padding, so every
// shared-memory read has a constant offset. The samples live in a ring of P
// registers, refilled P - R steps ahead of their use; P steps make one trip,
// after which every ring position has its old role. A warp skips the steps in
// which all its outputs would only meet samples outside the column (the
// triangle ends of a long-by-long convolution).
//
// Bound: the FP64 pipe, a product and an add per term (they must not fuse), at
// 0.86 of its rate. Full-matrix-capture synthesis of 101 elements (10201 columns
// 2000 * 2000, then * 150; 4.7e10 terms) 6.2 ms against 5.3 at the pipe's rate;
// with 64-bit clamped indices, a padded window and three rotating buffers (226
// registers) it took 12.3.
//
// '+=' / '-=' add into existing values; out-of-column terms then contribute
// the exact neutral element (-0 for +=, +0 for -=), so a stored -0 stays -0
// exactly as in the reference, which never visits those terms. For '=' their
// products are zeros, which leave a sum that starts from +0 as it is, unless a
// sample of B is infinite or NaN. That product is NaN, and so is the sum, so a
// lane whose sums are not all finite forms them again from the terms inside the
// column. (A test in the trips at a column's ends: 4000 columns of 300 * 300 0.168
// against 0.084 ms; a vote on B with both forms of a trip 0.089.)
#include <cuda_runtime.h>
#include <stdint.h>

#include <algorithm>
#include <mutex>
#include <string>
#include <vector>

#include "das_common.cuh"
#include "das_kernels.h"
#include "dream_conv.h"

namespace dream {
namespace {

constexpr int CONV_WARPS = 4;         // small CTAs: long pulses leave few tiles per column
constexpr int64_t CONV_LMAX = 8192;   // B samples staged in shared memory
// R outputs per lane (odd); ring of P A samples = steps per trip; B samples read ahead (divides P)
constexpr int conv_p(int R) { return R + 3; }
constexpr int conv_y(int R) { return conv_p(R) / 2; }
constexpr int conv_t(int R) { return CONV_WARPS * 32 * R; }  // outputs per CTA

// B slots (L samples, then those read ahead by the last trip) and A-window slots.
constexpr int64_t conv_b_slots(int R, int64_t L) { return L + conv_p(R) + conv_y(R); }
constexpr int64_t conv_window(int R, int64_t L) { return conv_t(R) + L + 2 * conv_p(R); }

constexpr size_t conv_smem_bytes(int R, int64_t L) {
  return (size_t)(conv_b_slots(R, L) + conv_window(R, L)) * sizeof(double);
}

template <int MODE>
__device__ __forceinline__ double conv_acc(double acc, double prod) {
  return MODE == 2 ? __dsub_rn(acc, prod) : __dadd_rn(acc, prod);
}

// One trip: steps 0 .. P - 1 (PART: the first n of them) from the lane's A
// samples xp and the B samples yp; X holds samples 0 .. P - 1, Y the first
// B samples. TEST: sample t of the trip is A[i0 + t]; products of samples
// outside [0, M) become `neutral`.
template <int MODE, int R, bool PART, bool TEST>
__device__ __forceinline__ void conv_trip(double (&acc)[R], double (&X)[conv_p(R)], double (&Y)[conv_y(R)],
                                          const double *xp, const double *yp, int n, int64_t i0, int64_t M,
                                          double neutral) {
  constexpr int CP = conv_p(R), CY = conv_y(R);
#pragma unroll
  for (int u = 0; u < CP; u++) {
    if (PART && u >= n) break;  // uniform across the warp
    const double y = Y[u % CY];
    Y[u % CY] = yp[u + CY];
#pragma unroll
    for (int r = 0; r < R; r++) {
      double prod = __dmul_rn(X[(u + r) % CP], y);
      if (TEST && (i0 + u + r < 0 || i0 + u + r >= M)) prod = neutral;
      acc[r] = conv_acc<MODE>(acc[r], prod);
    }
    X[u] = xp[u + CP];
  }
}

// Outputs k = k0 .. k0 + R - 1 of a '=' tile from its staged samples, only the terms inside the column; xp: the
// lane's first A sample. Out of line: the trips lose no registers to it.
template <int R>
__device__ __noinline__ void conv_inside(const double *xp, const double *ys, int64_t M, int64_t L, int64_t k0,
                                         int64_t NY, double *z) {
  for (int r = 0; r < R && k0 + r < NY; r++) {
    const int64_t k = k0 + r;
    const int s0 = (int)std::max<int64_t>(0, L - 1 - k), s1 = (int)std::min<int64_t>(L - 1, M - 1 - k + L - 1);
    double acc = 0.0;
    for (int s = s0; s <= s1; s++) acc = __dadd_rn(acc, __dmul_rn(xp[r + s], ys[s]));
    z[k] = acc;
  }
}

// Tile launched at grid position y, centre-out: the middle tiles, whose
// outputs have the longest sums, first (mid, mid+1, mid-1, mid+2, ...), so
// the block scheduler spreads them over all SMs before the short ones.
__device__ __forceinline__ int64_t centre_out_tile(int64_t y, int64_t n) {
  const int64_t m = n / 2, hi = n - 1 - m;  // tiles above the middle (hi <= m)
  if (y == 0) return m;
  if (y <= 2 * hi) return (y & 1) ? m + (y + 1) / 2 : m - y / 2;
  return m - (y - hi);
}

// Column n of the output convolves A column n % na with B column n / nb
// (na = N, nb = 1 for fftconv_p / conv_p; the full-matrix-capture synthesis
// pairs every receive column with every transmit column).
template <int MODE, int R>
__global__ void __launch_bounds__(CONV_WARPS * 32) conv_p_kernel(const double *__restrict__ A, int64_t M, int64_t N,
                                                                  const double *__restrict__ B, int64_t L,
                                                                  int64_t ldb, double *__restrict__ Y, int64_t NY,
                                                                  int64_t tiles, int64_t na, int64_t nb) {
  constexpr int CP = conv_p(R), CY = conv_y(R);
  extern __shared__ __align__(16) double conv_sm[];
  double *ys = conv_sm;                    // ys[s] = B[L - 1 - s]
  double *xs = conv_sm + conv_b_slots(R, L);  // xs[q] = A[k_cta - (L - 1) + q] (0 outside the column)
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int W = (int)conv_window(R, L), Li = (int)L;
  const double neutral = MODE == 2 ? 0.0 : -0.0;
  for (int64_t tile = blockIdx.y; tile < tiles; tile += gridDim.y) {
    const int64_t k_cta = centre_out_tile(tile, tiles) * conv_t(R);
    const int64_t base = k_cta - (L - 1);
    // Step s takes sample base + q0 + r + s for output r. Steps where the warp's
    // samples, base + w0 + s .. base + w0 + 32R - 1 + s, all fall outside the
    // column contribute nothing and are skipped.
    const int w0 = warp * 32 * R, q0 = w0 + R * lane;
    const int64_t k_w = k_cta + w0;
    const int s_begin = (int)std::max<int64_t>(0, (L - 1) - (k_w + 32 * R - 1));
    const int s_end = (int)std::max<int64_t>(s_begin, std::min<int64_t>(L, M + (L - 1) - k_w));
    for (int64_t n = blockIdx.x; n < N; n += gridDim.x) {
      const double *x = A + (n % na) * M;
      const double *y = B + (n / nb) * ldb;
      double *z = Y + n * NY;
      __syncthreads();  // the previous column's window is no longer read
      for (int q = tid; q < (int)conv_b_slots(R, L); q += CONV_WARPS * 32) ys[q] = q < Li ? y[Li - 1 - q] : 0.0;
      for (int q = tid; q < W; q += CONV_WARPS * 32) {
        const int64_t i = base + q;
        xs[q] = (i >= 0 && i < M) ? x[i] : 0.0;
      }
      __syncthreads();
      const double *xp = xs + q0 + s_begin, *yp = ys + s_begin;
      double acc[R], X[CP], Yb[CY];
#pragma unroll
      for (int r = 0; r < R; r++) acc[r] = (MODE != 0 && k_cta + q0 + r < NY) ? z[k_cta + q0 + r] : 0.0;
#pragma unroll
      for (int t = 0; t < CP; t++) X[t] = xp[t];
#pragma unroll
      for (int t = 0; t < CY; t++) Yb[t] = yp[t];
      int left = s_end - s_begin;
      int64_t i_w = base + w0 + s_begin;  // the warp's first sample of the trip
      for (; left >= CP; left -= CP, xp += CP, yp += CP, i_w += CP) {
        if (MODE != 0 && (i_w < 0 || i_w + 32 * R + CP > M))
          conv_trip<MODE, R, false, true>(acc, X, Yb, xp, yp, CP, i_w + R * lane, M, neutral);
        else
          conv_trip<MODE, R, false, false>(acc, X, Yb, xp, yp, CP, 0, M, neutral);
      }
      conv_trip<MODE, R, true, MODE != 0>(acc, X, Yb, xp, yp, left, i_w + R * lane, M, neutral);
#pragma unroll
      for (int r = 0; r < R; r++) {
        const int64_t k = k_cta + q0 + r;
        if (k < NY) z[k] = acc[r];
      }
      if (MODE == 0) {
        int top = 0;  // high word of the largest |sum|, infinity and NaN above all
#pragma unroll
        for (int r = 0; r < R; r++) top = max(top, __double2hiint(acc[r]) & 0x7fffffff);
        if (top >= 0x7ff00000) conv_inside<R>(xs + q0, ys, M, L, k_cta + q0, NY, z);
      }
    }
  }
}

// Pulses longer than the shared-memory budget: one output per thread, the
// same order of operations, operands from global memory (L1/L2).
template <int MODE>
__global__ void __launch_bounds__(256) conv_p_global_kernel(const double *__restrict__ A, int64_t M, int64_t N,
                                                             const double *__restrict__ B, int64_t L, int64_t ldb,
                                                             double *__restrict__ Y, int64_t NY, int64_t na,
                                                             int64_t nb) {
  const int64_t k = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  for (int64_t n = blockIdx.y; n < N; n += gridDim.y) {
    if (k >= NY) continue;
    const double *x = A + (n % na) * M;
    const double *y = B + (n / nb) * ldb;
    double acc = MODE == 0 ? 0.0 : Y[n * NY + k];
    const int64_t i_lo = std::max<int64_t>(0, k - (L - 1)), i_hi = std::min<int64_t>(M - 1, k);
    for (int64_t i = i_lo; i <= i_hi; i++) acc = conv_acc<MODE>(acc, __dmul_rn(__ldg(x + i), __ldg(y + (k - i))));
    Y[n * NY + k] = acc;
  }
}

template <int MODE>
cudaError_t launch_mode(const double *A, int64_t M, int64_t N, const double *B, int64_t L, int64_t ldb, double *Y,
                        int64_t NY, cudaStream_t st, int64_t na, int64_t nb) {
  const unsigned gy = (unsigned)std::min<int64_t>(N, 65535);
  // 7 outputs per lane; 5 where that leaves few tiles per SM (2000-sample columns * 2000: 101 columns 0.083 against
  // 0.099 ms, 1024 and more columns alike) and B is short enough that shared memory does not decide (8000 samples
  // x 16 columns of 20000: 0.50 against 0.40)
  const int64_t tiles7 = N * ((NY + conv_t(7) - 1) / conv_t(7));
  const int R = (tiles7 < 4096 && L <= 4096) ? 5 : 7;
  const int64_t gt = (NY + conv_t(R) - 1) / conv_t(R);
  if (L <= CONV_LMAX) {
    const size_t smem = conv_smem_bytes(R, L);
    auto kern = R == 5 ? conv_p_kernel<MODE, 5> : conv_p_kernel<MODE, 7>;
    cudaError_t e = ensure_smem(kern, smem);
    if (e != cudaSuccess) return e;
    // x: columns (fastest, so every column's middle tile launches before any
    // column's edge tiles), y: tiles in centre-out order
    dim3 grid((unsigned)std::min<int64_t>(N, 1 << 30), (unsigned)std::min<int64_t>(gt, 65535));
    kern<<<grid, CONV_WARPS * 32, smem, st>>>(A, M, N, B, L, ldb, Y, NY, gt, na, nb);
  } else {
    dim3 grid((unsigned)((NY + 255) / 256), gy);
    conv_p_global_kernel<MODE><<<grid, 256, 0, st>>>(A, M, N, B, L, ldb, Y, NY, na, nb);
  }
  return cudaGetLastError();
}

// Shapes after the reference's rules (python/include/py_fftconv_p.hpp:70-77,
// extra_src/oct_conv_p.cc:225-236): B a vector (either orientation) for every
// column, or a matrix with A_N columns.
int conv_shapes(int64_t A_M, int64_t A_N, int64_t &B_M, int64_t &B_N, int mode) {
  if (A_M < 0 || A_N < 0 || B_M < 0 || B_N < 0) return set_last_error(DREAM_ERR_ARGUMENT, "negative dimension");
  if (mode != DREAM_CONV_EQU && mode != DREAM_CONV_SUM && mode != DREAM_CONV_NEG)
    return set_last_error(DREAM_ERR_ARGUMENT, "Non-valid string in arg 4!");
  if (B_M != 1 && B_N != 1 && B_N != A_N)
    return set_last_error(DREAM_ERR_ARGUMENT,
                          "Argument 2 must be a vector or a matrix with the same number of columns as arg 1!");
  if (B_M == 1 || B_N == 1) {
    B_M = B_M * B_N;
    B_N = 1;
  }
  return 0;
}

int conv_device(const double *dA, int64_t A_M, int64_t A_N, const double *dB, int64_t B_M, int64_t B_N, double *dY,
                int mode, cudaStream_t st) {
  const int64_t NY = A_M + B_M - 1;
  if (A_N == 0 || NY <= 0) return 0;
  if (dY == nullptr) return set_last_error(DREAM_ERR_ARGUMENT, "NULL output pointer");
  if (A_M == 0 || B_M == 0) {  // no products: '=' clears, '+=' and '-=' leave Y as it is
    if (mode == DREAM_CONV_EQU) {
      cudaError_t e = cudaMemsetAsync(dY, 0, (size_t)NY * A_N * sizeof(double), st);
      if (e != cudaSuccess) return set_last_error(DREAM_ERR_CUDA, cudaGetErrorString(e));
    }
    return 0;
  }
  if (dA == nullptr || dB == nullptr) return set_last_error(DREAM_ERR_ARGUMENT, "NULL input pointer");
  const int64_t ldb = B_N > 1 ? B_M : 0;
  cudaError_t e = mode == DREAM_CONV_EQU   ? launch_mode<0>(dA, A_M, A_N, dB, B_M, ldb, dY, NY, st, A_N, 1)
                  : mode == DREAM_CONV_SUM ? launch_mode<1>(dA, A_M, A_N, dB, B_M, ldb, dY, NY, st, A_N, 1)
                                           : launch_mode<2>(dA, A_M, A_N, dB, B_M, ldb, dY, NY, st, A_N, 1);
  if (e != cudaSuccess) return set_last_error(DREAM_ERR_CUDA, std::string("conv_p launch: ") + cudaGetErrorString(e));
  return 0;
}

// Device buffers of the host-pointer entry, kept per device and grown on demand.
struct ConvBuffers {
  std::mutex mu;
  double *A = nullptr, *B = nullptr, *Y = nullptr;
  size_t cap_a = 0, cap_b = 0, cap_y = 0;
  cudaStream_t st = nullptr;
};

int grow(double *&p, size_t &cap, size_t bytes) {
  if (bytes <= cap) return 0;
  if (p) cudaFree(p);
  p = nullptr;
  cap = 0;
  cudaError_t e = cudaMalloc(&p, bytes);
  if (e != cudaSuccess) {
    cudaGetLastError();
    return set_last_error(DREAM_ERR_ALLOC, "conv_p: device allocation failed");
  }
  cap = bytes;
  return 0;
}

}  // namespace
}  // namespace dream

using namespace dream;

extern "C" {

int dream_conv_p_run_device(const double *dA, int64_t A_M, int64_t A_N, const double *dB, int64_t B_M, int64_t B_N,
                            double *dY, int mode, void *stream) {
  DREAM_API_TRY
  int r = conv_shapes(A_M, A_N, B_M, B_N, mode);
  if (r) return r;
  return conv_device(dA, A_M, A_N, dB, B_M, B_N, dY, mode, (cudaStream_t)stream);
  DREAM_API_CATCH
}

int dream_conv_p_run(const double *A, int64_t A_M, int64_t A_N, const double *B, int64_t B_M, int64_t B_N, double *Y,
                     int mode, int device) {
  DREAM_API_TRY
  int r = conv_shapes(A_M, A_N, B_M, B_N, mode);
  if (r) return r;
  const int64_t NY = A_M + B_M - 1;
  if (A_N == 0 || NY <= 0) return 0;
  if (Y == nullptr || (A_M > 0 && A == nullptr) || (B_M > 0 && B == nullptr))
    return set_last_error(DREAM_ERR_ARGUMENT, "NULL host pointer");
  int ndev = 0;
  if (cudaGetDeviceCount(&ndev) != cudaSuccess || device < 0 || device >= ndev)
    return set_last_error(DREAM_ERR_ARGUMENT, "invalid CUDA device ordinal");
  static std::vector<ConvBuffers> bufs(64);
  if (device >= (int)bufs.size()) return set_last_error(DREAM_ERR_ARGUMENT, "invalid CUDA device ordinal");
  ConvBuffers &cb = bufs[device];
  std::lock_guard<std::mutex> lk(cb.mu);
  int prev = -1;
  cudaGetDevice(&prev);
  if (prev != device) cudaSetDevice(device);
  auto done = [&](int code) {
    if (prev >= 0 && prev != device) cudaSetDevice(prev);
    return code;
  };
  cudaError_t e = cudaSuccess;
  if (cb.st == nullptr && (e = cudaStreamCreateWithFlags(&cb.st, cudaStreamNonBlocking)) != cudaSuccess)
    return done(set_last_error(DREAM_ERR_CUDA, cudaGetErrorString(e)));
  const size_t na = (size_t)A_M * A_N, nb = (size_t)B_M * B_N, ny = (size_t)NY * A_N;
  if ((r = grow(cb.A, cb.cap_a, std::max<size_t>(na, 1) * 8)) || (r = grow(cb.B, cb.cap_b, std::max<size_t>(nb, 1) * 8)) ||
      (r = grow(cb.Y, cb.cap_y, ny * 8)))
    return done(r);
  if (na) e = cudaMemcpyAsync(cb.A, A, na * 8, cudaMemcpyHostToDevice, cb.st);
  if (e == cudaSuccess && nb) e = cudaMemcpyAsync(cb.B, B, nb * 8, cudaMemcpyHostToDevice, cb.st);
  if (e == cudaSuccess && mode != DREAM_CONV_EQU) e = cudaMemcpyAsync(cb.Y, Y, ny * 8, cudaMemcpyHostToDevice, cb.st);
  if (e != cudaSuccess) return done(set_last_error(DREAM_ERR_CUDA, cudaGetErrorString(e)));
  if ((r = conv_device(cb.A, A_M, A_N, cb.B, B_M, B_N, cb.Y, mode, cb.st))) return done(r);
  e = cudaMemcpyAsync(Y, cb.Y, ny * 8, cudaMemcpyDeviceToHost, cb.st);
  if (e == cudaSuccess) e = cudaStreamSynchronize(cb.st);
  if (e != cudaSuccess) return done(set_last_error(DREAM_ERR_CUDA, cudaGetErrorString(e)));
  return done(0);
  DREAM_API_CATCH
}

int dream_conv_p_fmc_device(const double *dHt, int64_t M, int64_t L_t, const double *dHr, int64_t L_r,
                            const double *dP, int64_t P_M, double *dDP, double *dY, void *stream) {
  DREAM_API_TRY
  if (M <= 0 || L_t < 0 || L_r < 0 || P_M <= 0)
    return set_last_error(DREAM_ERR_ARGUMENT, "fmc synthesis: M and the pulse length must be positive");
  const int64_t N = L_t * L_r;
  if (N == 0) return 0;
  if (dHt == nullptr || dHr == nullptr || dP == nullptr || dDP == nullptr || dY == nullptr)
    return set_last_error(DREAM_ERR_ARGUMENT, "NULL pointer");
  const cudaStream_t st = (cudaStream_t)stream;
  const int64_t NY1 = 2 * M - 1, NY2 = NY1 + P_M - 1;
  // double path: column t*L_r + r = Hr[:, r] (*) Ht[:, t]; then every column (*) the pulse
  cudaError_t e = launch_mode<0>(dHr, M, N, dHt, M, M, dDP, NY1, st, L_r, L_r);
  if (e == cudaSuccess) e = launch_mode<0>(dDP, NY1, N, dP, P_M, 0, dY, NY2, st, N, 1);
  if (e != cudaSuccess) return set_last_error(DREAM_ERR_CUDA, std::string("fmc synthesis launch: ") + cudaGetErrorString(e));
  return 0;
  DREAM_API_CATCH
}

}  // extern "C"
