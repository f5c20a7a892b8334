// das_fast.h -- launch descriptor of the FP32/BF16-storage DAS kernels.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

namespace dream {

struct FastParams {
  int method;  // 0 SAFT, 1 TFM, 2 RCA col-tx, 3 RCA row-tx
  const void *Y;  // float or bf16, K x (Nt*Nr) column-major
  int64_t K;
  const double *Ro;
  int64_t No;
  const double *Gt;
  int Nt;
  const double *Gr;
  int Nr;
  const double *delay;  // us; 1 value or No values
  int delay_multi;
  double Fs, ocp;  // (1/dt)*1000 and 1/cp in FP64, as DAS<double>
  const float *w;  // per A-scan column weights, or nullptr
  float *Im;
  unsigned long long *oob;
  // image tiling: point n = s*n_fast + f
  int64_t n_fast, n_slow;
  int tile_f, tile_s, wf;  // tile extents; warp lanes along the fast axis
  int out_block;           // outer elements whose legs are tabled at a time
  int64_t slow_tile0, slow_tile1;  // slow-tile range of this launch
  int64_t no0, no1;                // point range (SAFT launches)
  // inner-element range [in_lo, in_hi) of this launch (in_hi == 0: all inner
  // elements) and whether to add into Im instead of writing it
  int in_lo, in_hi;
  int accumulate;
  // A-scan columns present in Y: column (o, i) is o * ycol_o + i - ycol_i0
  // (ycol_o == 0: o * n_in + i, the full layout)
  int64_t ycol_o;
  int ycol_i0;
  int64_t ny;               // elements in Y (bounds-checked builds; 0: K * columns)
  unsigned long long *bad;  // gather index violations (bounds-checked builds)
};

// Points along the fast axis (depth, on the usual grids) of a gather warp's patch
// of the image: 4 x 8 on a hinted grid, for the reason given at plain_patch_f;
// unlike the plain FP64 kernel's, an RCA volume's 4-byte samples fare best in them
// too (128x128 elements, 64x64x128 points 4.48 ms, 8 x 4 5.00, 2 x 16 5.7).
inline int gather_patch_f(bool hint, int tile_s) { return !hint ? 32 : (tile_s % 8 == 0 ? 4 : 8); }
// Outer elements tabled at a time, in even blocks. Every block recomputes the
// inner legs; 52 x 128 threads x 8 bytes leave room for four tiles on an SM. One
// block of up to 64 pays for the fourth (64x64 elements: 0.417 against 0.425 ms,
// 61x47: 0.173 against 0.192), two of 64 do not (128 outer elements: 1.02
// against 0.91 ms with three of 44), nor do tiles of the persistent batch or
// weighted ones, whose weights share the table's space (0.544 against 0.521).
inline int gather_out_block(int n_out, bool single) {
  if (single && n_out <= 64) return n_out > 0 ? n_out : 1;
  const int n = (n_out + 51) / 52;
  return n > 0 ? ((n_out + n - 1) / n + 3) / 4 * 4 : 4;
}
// Frames with more elements than this limit allows on a tile of nthr points are
// refused by every storage-precision entry (gather and scatter alike).
inline bool too_many_elements(int n_out, int n_in, int nthr) {
  const size_t head = ((size_t)(3 * n_out + 2 * n_in) * 4 + 15) & ~(size_t)15;
  return head + (((size_t)(n_out + 16) * nthr * 4 + 15) & ~(size_t)15) > 220 * 1024;
}
size_t gather_smem_bytes(const FastParams &P, int nthr);  // leg table of the gather (P.out_block)
cudaError_t launch_fast(const FastParams &P, bool bf16, cudaStream_t st);
// Adjoint on the forward's tiles: Ya[k(n,c), c] += w[c] * X[n] (FP32 A-scans;
// P.w may be NULL). Adds into Ya, which the caller zeroes first. square: 8 x 32-point
// tiles of a TFM grid become 16 x 16 where its spacing asks for it.
cudaError_t launch_scatter(const FastParams &P, bool square, const float *X, float *Ya, cudaStream_t st);
// Per column c of K x ncol arrays: dW[c] = sum_k Y[k,c] * S[k,c] (when Y and dW
// are given), then S[:, c] *= w[c] (when w is given).
cudaError_t launch_column_dot_scale(const float *Y, float *S, const float *w, float *dW, int64_t K, int64_t ncol,
                                    cudaStream_t st);
cudaError_t convert_f32_to_bf16(const float *x, void *y, int64_t n, cudaStream_t st);
// rows x row_elems block of a row-pitched array (same offsets in x and y)
cudaError_t convert_f32_to_bf16_2d(const float *x, void *y, int64_t rows, int64_t row_elems, int64_t pitch,
                                   cudaStream_t st);

// Persistent batch launch over (frame, tile_f index, tile_s index) items
// (int4: frame, tfi, tsi, unused); resets the queue counter *ctr first.
cudaError_t launch_batch(const FastParams *frames, const int4 *items, int n_items, int *ctr, size_t smem, bool bf16,
                         int grid, cudaStream_t st);
int batch_prepare(size_t smem, bool bf16);

}  // namespace dream

struct dream_das_frame;

namespace dream {
// Validates one batch frame and fills its launch descriptor (oob left NULL);
// returns 0 or a DREAM_ERR_* status with the message recorded. Used by
// dream_das_batch_create and dream_das_batch_run_noalloc alike.
int batch_frame_params(const ::dream_das_frame &d, FastParams &F);
}  // namespace dream
