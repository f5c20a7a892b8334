// das_kernels.h -- launch descriptors shared by the C ABI (das_capi.cu) and
// the kernel translation units. Host-side only types.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include <string>

namespace dream {

// Per-call constants, computed on the host exactly as the restated reference
// source computes them (see das_capi.cu: constants_*).
struct Consts64 {
  double Fs, ocp, delay_ms;
};
struct Consts32 {
  float Fs, ocp, delay_ms;
};

// Warp patch of the plain TFM / RCA kernel on a hinted grid: points along the
// fast axis (depth, on the usual grids), the rest of the 32 along the slow one.
// The fewer different samples a patch reads from one A-scan, the fewer
// wavefronts its gather takes: in depth a point moves by the sum of both legs'
// cosines, across by sines of opposite signs, so TFM patches are 4 deep and 8
// wide (64x64 elements, 512x512 points, FP64: 0.69 ms; 8 x 4: 0.80). Both
// sideways axes of an RCA volume move its legs alike: 8 x 4 (128x128 elements,
// 131072 points, FP64 3.1 ms; 4 x 8: 3.6, 2 x 16: 4.9).
constexpr int plain_patch_f(int method) { return method == 1 /* TFM */ ? 4 : 8; }

// Terms whose gathers are issued together.
constexpr int PLAIN_U = 16;

// Leg table of a block of the plain TFM / RCA kernel: n_in legs per thread, in
// whole pairs of gather groups.
constexpr size_t plain_table_bytes(int64_t n_in, size_t elem, int threads) {
  return (size_t)((n_in + 2 * PLAIN_U - 1) / (2 * PLAIN_U) * (2 * PLAIN_U)) * elem * threads;
}
// Threads per block: the largest block whose table leaves room for three on
// an SM; a table that does not fit one warp in shared memory: 0 (no table).
constexpr int plain_tile_threads(int64_t n_in, size_t elem) {
  int bd = 128;
  while (bd > 32 && plain_table_bytes(n_in, elem, bd) > 72 * 1024) bd >>= 1;
  return plain_table_bytes(n_in, elem, bd) <= 200 * 1024 ? bd : 0;
}
// Tile of image points of such a block on a hinted grid.
constexpr int plain_tile_f(int method, int threads) { return threads >= 128 ? 8 : plain_patch_f(method); }
constexpr int plain_tile_s(int method, int threads) { return threads / plain_tile_f(method, threads); }

struct PlainLaunch {
  int method;  // 0 SAFT, 1 TFM, 2 RCA col-tx, 3 RCA row-tx
  bool uni;
  const void *Y;
  int64_t K;
  const void *Ro;
  int64_t No;
  int64_t no0, no1;  // pixel range of this launch (tile-row range when n_fast > 0)
  int64_t n_fast;    // grid hint: points along the grid's fast axis (0: none)
  const void *Gt;
  int64_t Nt;
  const void *Gr;
  int64_t Nr;
  const void *delay_vec;  // device delays (us): 1 value, or No values when delay_multi
  bool delay_multi;
  Consts64 c64;
  Consts32 c32;
  double tri64[15];
  float tri32[15];
  int64_t Nx, Ny, Nz;
  void *Im;
  unsigned long long *oob;
  int64_t ny;               // elements in Y
  unsigned long long *bad;  // gather index violations (bounds-checked builds)
  int64_t *idx;             // non-NULL: write the sample indices instead of the image
};

cudaError_t launch_plain_f64(const PlainLaunch &L, cudaStream_t st);

// Records msg as this host thread's last error (dream_das_last_error) and
// returns code.
int set_last_error(int code, const std::string &msg);

// The status of the C++ exception being handled (call only inside a catch
// block): DREAM_ERR_ALLOC for std::bad_alloc, DREAM_ERR_ARGUMENT otherwise,
// with its message recorded. Every int-returning C ABI entry wraps its body in
// DREAM_API_TRY ... DREAM_API_CATCH, so no exception crosses the C boundary.
int api_exception() noexcept;
#define DREAM_API_TRY try {
#define DREAM_API_CATCH \
  }                     \
  catch (...) {         \
    return ::dream::api_exception(); \
  }
cudaError_t launch_plain_f32(const PlainLaunch &L, cudaStream_t st);

}  // namespace dream
