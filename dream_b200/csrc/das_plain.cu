// das_plain.cu -- the plain DAS kernels: FP64 (DAS<double>) and FP32
// (DAS<float>) on arbitrary geometry (`das`) and on uniform grids (`das_uni`).
//
// These kernels are the drop-in replacement of the reference's per-pixel
// loops and keep their arithmetic exactly:
//   SAFT        extra_src/das.cc:306-357, opencl/das_uni_double.cl:9-77
//   TFM         extra_src/das.cc:365-427, opencl/das_uni_double.cl:79-167
//   RCA col-tx  extra_src/das.cc:437-529, opencl/das_uni_double.cl:169-281
//   RCA row-tx  extra_src/das.cc:533-626, opencl/das_uni_double.cl:283-394
// Each thread owns one image point and sums its terms in the reference order
// (outer element loop, inner element loop), so the image is bit-identical to
// the reference CPU code, not merely close to it. With a grid hint TFM and RCA
// blocks take 2-D tiles of the image grid instead of consecutive points, which
// changes only which thread owns which point.
//
// What differs from the reference is where the work goes. The inner-loop
// element leg (receive leg for TFM/col-tx, column leg for row-tx) depends
// only on (pixel, inner element), so it is computed once per pixel into a
// per-thread shared-memory table instead of once per term. Hoisting is exact:
// the leg is the same rounded value. So is the bounds test: rounding is
// monotone, so the extreme legs decide it for all terms of an outer element.
#include "das_common.cuh"
#include "das_kernels.h"

namespace dream {

template <class T>
struct PlainParams {
  const T *Y;
  int64_t K;
  const T *Ro;
  int64_t No;
  const T *Gt;
  int Nt;
  const T *Gr;
  int Nr;
  int64_t no0, no1;  // pixel range [no0, no1) of this launch, or tile-row range when n_fast > 0
  int64_t n_fast, n_slow;  // grid hint: warps take patches of (fast, slow) points
  const T *delay;  // das: device delays in us (1 value, or No when delay_multi)
  int delay_multi;
  T delay_ms;      // das_uni: the scalar delay in ms
  T Fs, ocp, Kf;
  T *Im;
  unsigned long long *oob;
  int64_t ny;               // elements in Y (bounds-checked builds)
  unsigned long long *bad;  // gather index violations (bounds-checked builds)
  int64_t *idx;             // index mode: idx[col * No + no] = sample index or -1
  int bigk;  // K >= 2^22 (FP32: truncation needs the conversion unit) or 2^28 (FP64): no grouped sample numbers
  // uniform grids
  T tri[15];
  int64_t Nx, Ny, Nz;
};

// Truncation of p in (-1, K). Long A-scans (FP32, K >= 2^22) need the
// conversion unit; every other case uses the exact add-based form.
template <class T, bool BIGK>
__device__ __forceinline__ int to_index(T p) {
  if constexpr (BIGK && sizeof(T) == 4) return __float2int_rz(p);
  return trunc_index(p);
}

// delay / 1000 the way each reference form computes it: DAS<double> in
// double, DAS<float> in double rounded to float (extra_src/das.cc:318).
__device__ __forceinline__ double delay_to_ms(double d) { return d / 1000.0; }
__device__ __forceinline__ float delay_to_ms(float d) {
  return __double2float_rn((double)d / 1000.0);
}

// Sample ycol[off] of Y. The bounds-checked build tests the element index
// against the extent of Y first (a violation is counted and reads 0); the
// normal build is the plain load.
template <class T>
__device__ __forceinline__ T load_y(const PlainParams<T> &P, const T *ycol, int64_t off) {
#ifdef DREAM_DAS_CHECKED
  const int64_t gi = (ycol - P.Y) + off;
  return gather_ok<T>(gi, P.ny, P.bad) ? __ldg(P.Y + gi) : (T)0;
#else
  return __ldg(ycol + off);
#endif
}

// The sample k places after y, for a 32-bit k.
template <class T>
__device__ __forceinline__ T load_at(const PlainParams<T> &P, const T *y, uint32_t k) {
  const T *a;  // one multiply-add of the 32-bit number: as y + k it takes two more instructions
  asm("mad.wide.u32 %0, %1, %2, %3;" : "=l"(a) : "r"(k), "n"((int)sizeof(T)), "l"(y));
  return gather_ok<T>((y - P.Y) + k, P.ny, P.bad) ? __ldg(a) : (T)0;
}

// The image point of one thread and its legs, for method M on arbitrary
// (UNI = false) or uniform geometry. TFM: outer = transmit, inner = receive;
// col-tx: columns, rows; row-tx: rows, columns.
template <class T, int M, bool UNI>
struct PlainPoint {
  using A = Ar<T>;
  T xo, yo, zo, delay_ms, gy_c, gx_r;

  __device__ __forceinline__ void init(const PlainParams<T> &P, int64_t no) {
    if (UNI) {
      // linear index -> (ny fastest, nz, nx)   (opencl/das_uni_double.cl:32-43)
      int64_t yq = no / P.Ny, ny = no - yq * P.Ny;
      int64_t zq = yq / P.Nz, nz = yq - zq * P.Nz;
      int64_t xq = zq / P.Nx, nx = zq - xq * P.Nx;
      xo = A::add(P.tri[6], A::mul((T)nx, P.tri[7]));
      yo = A::add(P.tri[9], A::mul((T)ny, P.tri[10]));
      zo = A::add(P.tri[12], A::mul((T)nz, P.tri[13]));
    } else {
      xo = P.Ro[no];
      yo = P.Ro[no + P.No];
      zo = P.Ro[no + 2 * P.No];
    }
    delay_ms = UNI ? P.delay_ms : delay_to_ms(P.delay[P.delay_multi ? no : 0]);
    // RCA stripe clamps (extra_src/das.cc:464-467,475-486,493-503)
    gy_c = (T)0;
    gx_r = (T)0;
    if (M == RCA_COLTX || M == RCA_ROWTX) {
      T gc_y_min, gc_y_max, gr_x_min, gr_x_max;
      if (UNI) {  // opencl/das_uni_double.cl:213-216
        gc_y_min = P.tri[3]; gc_y_max = P.tri[5];
        gr_x_min = P.tri[0]; gr_x_max = P.tri[2];
      } else {  // literal (num_cols/num_rows mixed) reads of the reference
        gc_y_min = P.Gr[0 + 1 * P.Nt];
        gc_y_max = P.Gr[P.Nt - 1 + 1 * P.Nt];
        gr_x_min = P.Gt[0];
        gr_x_max = P.Gt[P.Nr - 1];
      }
      if (yo >= gc_y_min && yo <= gc_y_max) gy_c = (T)0;
      else if (yo < gc_y_min) gy_c = A::sub(gc_y_min, yo);
      else gy_c = A::sub(gc_y_max, yo);
      if (UNI) {
        if (xo < gr_x_min || xo > gr_x_max) gx_r = (xo < gr_x_min) ? A::sub(gr_x_min, xo) : A::sub(gr_x_max, xo);
      } else {
        if (xo >= gr_x_min && xo <= gr_x_max) gx_r = (T)0;
        else if (xo < gr_x_min) gx_r = A::sub(gr_x_min, xo);
        else gx_r = A::sub(gr_x_max, xo);
      }
    }
  }

  // transmit / column elements
  __device__ __forceinline__ void elem_t(const PlainParams<T> &P, int n, T &ex, T &ey, T &ez) const {
    if (UNI) {
      ex = A::add(P.tri[0], A::mul((T)n, P.tri[1]));
      ey = (T)0;
      ez = (T)0;
    } else {
      ex = P.Gt[n];
      ey = P.Gt[n + P.Nt];
      ez = P.Gt[n + 2 * P.Nt];
    }
  }
  // receive / row elements (uniform RCA rows lie along y)
  __device__ __forceinline__ void elem_r(const PlainParams<T> &P, int n, T &ex, T &ey, T &ez) const {
    if (UNI) {
      T c = A::add(P.tri[3], A::mul((T)n, P.tri[4]));
      if (M == RCA_COLTX || M == RCA_ROWTX) {
        ex = (T)0; ey = c;
      } else {
        ex = c; ey = (T)0;
      }
      ez = (T)0;
    } else {
      ex = P.Gr[n];
      ey = P.Gr[n + P.Nr];
      ez = P.Gr[n + 2 * P.Nr];
    }
  }
  // leg of a transmit (TFM, SAFT) or column (RCA) element, of a receive or row element
  __device__ __forceinline__ T leg_t(const PlainParams<T> &P, int n) const {
    T ex, ey, ez;
    elem_t(P, n, ex, ey, ez);
    return leg_time(A::sub(ex, xo), (M == TFM || M == SAFT) ? A::sub(ey, yo) : gy_c, A::sub(ez, zo), P.ocp);
  }
  __device__ __forceinline__ T leg_r(const PlainParams<T> &P, int n) const {
    T ex, ey, ez;
    elem_r(P, n, ex, ey, ez);
    return leg_time((M == TFM || M == SAFT) ? A::sub(ex, xo) : gx_r, A::sub(ey, yo), A::sub(ez, zo), P.ocp);
  }
  // das row-tx: delay on the (inner) column leg; das_uni row-tx: on the
  // (outer) row leg (opencl/das_uni_double.cl:358-360).
  static constexpr bool DELAY_OUTER = (M != RCA_ROWTX) || UNI;
  __device__ __forceinline__ T outer_leg(const PlainParams<T> &P, int o) const {
    const T l = (M == RCA_ROWTX) ? leg_r(P, o) : leg_t(P, o);
    return DELAY_OUTER ? A::add(l, delay_ms) : l;
  }
  __device__ __forceinline__ T inner_leg(const PlainParams<T> &P, int i) const {
    const T l = (M == RCA_ROWTX) ? leg_t(P, i) : leg_r(P, i);
    return DELAY_OUTER ? l : A::add(l, delay_ms);
  }
};

// One thread per point, every term tested on its own: SAFT images (IDX =
// false), the index table of any method (IDX = true: every term's sample
// index, -1 out of bounds, goes to P.idx instead of being gathered), and
// TFM / RCA images whose inner elements are too many for the leg table of
// das_plain_tile_kernel, with the gathers of eight terms in flight (2x801
// elements, 200x200 points, FP64: 0.62 ms, one at a time 0.89).
template <class T, int M, bool UNI, bool BIGK, bool IDX>
__global__ void __launch_bounds__(256) das_plain_kernel(const PlainParams<T> P) {
  using A = Ar<T>;
  const int64_t no_raw = P.no0 + (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const bool active = no_raw < P.no1;
  const int64_t no = active ? no_raw : P.no0;  // inactive lanes read a valid point and write nothing
  PlainPoint<T, M, UNI> pt;
  pt.init(P, no);
  T im = (T)0;
  unsigned int oob = 0;
  const T *ycol = P.Y;
  const int n_out = (M == RCA_ROWTX) ? P.Nr : P.Nt;
  const int n_in = (M == SAFT) ? 1 : (M == RCA_ROWTX ? P.Nt : P.Nr);
  // G terms at a time: the gathers of a group are issued before its adds, which keep the reference's order
  constexpr int G = M == SAFT ? 1 : 8;
  for (int o = 0; o < n_out; o++) {
    T lo = (M == SAFT) ? (T)0 : pt.outer_leg(P, o);
    auto group = [&](int i, int n) {
      T y[G];
      bool v[G];
#pragma unroll
      for (int u = 0; u < G; u++) {
        v[u] = false;
        if (u >= n) continue;
        const T t = (M == SAFT) ? A::mul((T)2, pt.outer_leg(P, o)) : A::add(lo, pt.inner_leg(P, i + u));
        const T p = A::mul(t, P.Fs);
        v[u] = p > (T)-1 && p < P.Kf;
        oob += v[u] ? 0 : 1;
        if constexpr (IDX) {
          if (active) P.idx[((int64_t)o * n_in + i + u) * P.No + no] = v[u] ? (int64_t)to_index<T, BIGK>(p) : -1;
        } else {
          y[u] = v[u] ? load_y(P, ycol, (int64_t)u * P.K + to_index<T, BIGK>(p)) : (T)0;
        }
      }
      if (!IDX) {
#pragma unroll
        for (int u = 0; u < G; u++)
          if (v[u]) im = A::add(im, y[u]);
      }
      ycol += n * P.K;
    };
    int i = 0;
    for (; i + G <= n_in; i += G) group(i, G);
    if (G > 1 && i < n_in) group(i, n_in - i);
  }
  if (!IDX && active) P.Im[no] = im;
  add_count(P.oob, active ? oob : 0u);
}

// Sample numbers of U terms with in-bounds times p = RN(RN(lo + li) * Fs) >= 0,
// plus u * K for the u-th column of the group. FP64 adds 2^52 + u * K toward
// zero, which leaves u * K + floor(p) in the low mantissa word; FP32 adds 2^23
// and takes the bits from there (cofs = u * K - bits(2^23)).
template <int U>
__device__ __forceinline__ void sample_numbers(double lo, const double (&li)[U], double Fs, const double (&mag)[U],
                                               uint32_t (&k)[U]) {
#pragma unroll
  for (int u = 0; u < U; u++)
    k[u] = (uint32_t)__double2loint(__dadd_rz(__dmul_rn(__dadd_rn(lo, li[u]), Fs), mag[u]));
}
__device__ __forceinline__ uint64_t pair(float a, float b) {
  uint64_t r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
  return r;
}
template <int U>
__device__ __forceinline__ void sample_numbers(float lo, const float (&li)[U], float Fs, const uint32_t (&cofs)[U],
                                               uint32_t (&k)[U]) {
  // two terms per instruction (each half rounds as the scalar operation)
  const uint64_t lo2 = pair(lo, lo), fs2 = pair(Fs, Fs), mag2 = pair(8388608.0f, 8388608.0f);
#pragma unroll
  for (int u = 0; u < U; u += 2) {
    uint64_t v = pair(li[u], li[u + 1]);
    asm("add.rn.f32x2 %0, %1, %0;" : "+l"(v) : "l"(lo2));
    asm("mul.rn.f32x2 %0, %0, %1;" : "+l"(v) : "l"(fs2));
    asm("add.rz.f32x2 %0, %0, %1;" : "+l"(v) : "l"(mag2));
    k[u] = (uint32_t)v + cofs[u];
    k[u + 1] = (uint32_t)(v >> 32) + cofs[u + 1];
  }
}
template <class T>
struct ColStep;
template <>
struct ColStep<double> {
  using type = double;
  static __device__ __forceinline__ double of(int u, int64_t K) { return 4503599627370496.0 + (double)(u * K); }
};
template <>
struct ColStep<float> {
  using type = uint32_t;
  static __device__ __forceinline__ uint32_t of(int u, int64_t K) { return (uint32_t)(u * K) - 0x4B000000u; }
};

// TFM and RCA images (or, IDX, their index tables) with the inner legs of
// every thread in shared memory.
//
// Bound and layout (64x64 elements, K = 3000, 512x512 points on B200; the same
// frame with one branch per term and warps of 32 consecutive points took 2.43
// ms in FP64 and 0.98 in FP32). FP64: 0.69 ms, 0.77 of the shared-memory / L1
// data pipe (2 wavefronts per term for the leg, 2.3 for the 8-byte sample),
// the FP64 pipe (two-leg add, scale, truncation, accumulate) at 0.42. FP32:
// 0.36 ms, 8.6 instructions per 32 terms, 0.74 of the issue slots. What got it there:
//  - no test per term. The shortest and the longest inner leg bound every time
//    of an outer element exactly (rounded sums and products are monotone), so
//    one vote per outer element shows that all its terms are in bounds.
//  - sample numbers by adding a power of two toward zero, the column offset
//    inside a group in the same addend (FP64) or one 32-bit add (FP32, whose
//    leg sum, scale and truncation run two terms per instruction).
//  - addresses by one 32x32+64-bit multiply-add (three moves per term fewer
//    than pointer + index).
//  - U = 16 gathers issued before the adds of the 16 before them: with 3 or 4
//    blocks of 4 warps on an SM the gathers' latency is what is left (U = 8:
//    0.82 and 0.42 ms).
// MINB: resident blocks the registers must allow; 3 (170 registers), or 4
// where the table lets a fourth in (32x32 elements, 256x256 points, FP64: less
// than one wave of blocks, 0.065 against 0.094 ms).
template <class T, int M, bool UNI, bool BIGK, bool IDX, int BD, int MINB>
__global__ void __launch_bounds__(BD, MINB * 128 / BD) das_plain_tile_kernel(const PlainParams<T> P) {
  using A = Ar<T>;
  constexpr int U = MINB == 4 ? PLAIN_U / 2 : PLAIN_U;  // 16 FP64 samples, twice, do not fit 128 registers
  constexpr int V = 16 / sizeof(T);  // legs per 16-byte table read
  // Blocks that a long leg table cuts to one warp have too few to hide a test per term: outer elements wholly
  // out of bounds are skipped, the others tested in a loop of their own (64x300 elements, 200x200 points, FP64, K = 300
  // 0.82 against 5.10 ms, K = 1500 6.87 against 7.15). Larger blocks keep the pipelined groups: with both forms they are
  // up to 16 % slower in bounds (RCA 64x64, FP32 0.256 and 0.297 ms).
  constexpr bool FEW = BD == 32;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  T *tab = reinterpret_cast<T *>(smem_raw);  // leg i of thread t: tab[(i / V) * V * BD + t * V + i % V]
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  int64_t no_raw, first;
  bool active;
  if (P.n_fast > 0) {
    constexpr int TF = plain_tile_f(M, BD), TS = plain_tile_s(M, BD);
    // patches of 8 x 4 points become 4 x 8 where a volume's lines are neighbours in two directions
    const uint32_t row =
        !UNI && M != TFM && (int64_t)P.Nt * P.Nr >= VOLUME_TERMS ? volume_row(P.Ro, P.No, P.n_fast, P.n_slow) : 0;
    const int pf = TS % 8 == 0 && row ? 4 : plain_patch_f(M), wf = TF / pf;  // lanes and warps along the fast axis
    const int64_t f0 = (int64_t)blockIdx.x * TF, s0 = (P.no0 + blockIdx.y) * TS;
    const int64_t f = f0 + (warp % wf) * pf + lane % pf;
    const int64_t s = s0 + (warp / wf) * (32 / pf) + lane / pf;
    active = f < P.n_fast && s < P.n_slow;
    no_raw = volume_line(s, row, P.n_slow) * P.n_fast + f;
    first = volume_line(s0, row, P.n_slow) * P.n_fast + f0;
  } else {
    no_raw = P.no0 + (int64_t)blockIdx.x * BD + tid;
    active = no_raw < P.no1;
    first = P.no0 + (int64_t)blockIdx.x * BD;
  }
  const int64_t no = active ? no_raw : first;  // inactive lanes repeat the tile's first point and write nothing
  PlainPoint<T, M, UNI> pt;
  pt.init(P, no);
  const int n_out = (M == RCA_ROWTX) ? P.Nr : P.Nt;
  const int n_in = (M == RCA_ROWTX) ? P.Nt : P.Nr;
  T mn = (T)INFINITY, mx = -(T)INFINITY;
  bool fin = P.Fs > (T)0;
  for (int i = 0; i < n_in; i++) {
    const T l = pt.inner_leg(P, i);
    tab[(i / V) * V * BD + tid * V + i % V] = l;
    mn = l < mn ? l : mn;
    mx = l > mx ? l : mx;
    fin = fin && l == l;  // a NaN leg leaves every group to the tested form
  }
  typename ColStep<T>::type step[U];
#pragma unroll
  for (int u = 0; u < U; u++) step[u] = ColStep<T>::of(u, P.K);

  T im = (T)0;
  unsigned int oob = 0;
  const T *ycol = P.Y;
  int64_t *idx = IDX ? P.idx + no : nullptr;
  auto legs = [&](int i, T(&li)[U]) {
#pragma unroll
    for (int v = 0; v < U / V; v++)
#pragma unroll
      for (int q = 0; q < V; q++) li[v * V + q] = tab[(i / V + v) * V * BD + tid * V + q];
  };
  // samples of terms (o, i .. i+U-1); terms past n_in and out-of-bounds ones
  // are +0, which the sum (never -0: it starts from +0) takes unchanged
  auto gather = [&](T lo, int i, T(&y)[U], bool full) {
    T li[U];
    uint32_t k[U];
    legs(i, li);
    sample_numbers<U>(lo, li, P.Fs, step, k);
    const T *yb = ycol + (int64_t)i * P.K;
#pragma unroll
    for (int u = 0; u < U; u++) {
      y[u] = (T)0;
      if (full || i + u < n_in) y[u] = load_at(P, yb, k[u]);
    }
  };
  auto gather_tested = [&](T lo, int i, T(&y)[U]) {
    T li[U];
    legs(i, li);
#pragma unroll
    for (int u = 0; u < U; u++) {
      y[u] = (T)0;
      if (i + u < n_in) {
        const T p = A::mul(A::add(lo, li[u]), P.Fs);
        const bool v = p > (T)-1 && p < P.Kf;
        if constexpr (IDX) {
          if (active) *idx = v ? (int64_t)to_index<T, BIGK>(p) : -1;
          idx += P.No;
        } else if (v) {
          const int k = to_index<T, BIGK>(p);
          y[u] = BIGK ? load_y(P, ycol + (int64_t)(i + u) * P.K, k)
                      : load_at(P, ycol + (int64_t)i * P.K, (uint32_t)u * (uint32_t)P.K + (uint32_t)k);
        }
        oob += v ? 0 : 1;
      }
    }
  };
  // FEW warps: the terms of one outer element, tested one by one, G at a time; a group
  // without a term in bounds for any point of the warp is skipped
  auto add_tested = [&](T lo) {
    constexpr int G = 8;
    for (int i = 0; i < n_in; i += G) {
      T p[G], y[G];
      uint32_t in = 0;
#pragma unroll
      for (int u = 0; u < G; u++) {
        p[u] = A::mul(A::add(lo, tab[(i / V + u / V) * V * BD + tid * V + u % V]), P.Fs);
        if (i + u < n_in && p[u] > (T)-1 && p[u] < P.Kf) in |= 1u << u;
      }
      oob += min(G, n_in - i) - __popc(in);
      if (!IDX && !__any_sync(0xffffffffu, in)) continue;
#pragma unroll
      for (int u = 0; u < G; u++) {
        const bool v = in >> u & 1;
        y[u] = (T)0;
        if constexpr (IDX) {
          if (i + u < n_in) {
            if (active) *idx = v ? (int64_t)to_index<T, BIGK>(p[u]) : -1;
            idx += P.No;
          }
        } else if (v) {
          const int k = to_index<T, BIGK>(p[u]);
          y[u] = BIGK ? load_y(P, ycol + (int64_t)(i + u) * P.K, k)
                      : load_at(P, ycol + (int64_t)i * P.K, (uint32_t)u * (uint32_t)P.K + (uint32_t)k);
        }
      }
#pragma unroll
      for (int u = 0; u < G; u++) im = A::add(im, y[u]);
    }
  };
  auto accumulate = [&](const T(&y)[U]) {
#pragma unroll
    for (int u = 0; u < U; u++) im = A::add(im, y[u]);
  };
  // Two groups alternate: the gathers of one are issued before the in-order
  // adds of the other, so the sum's serial adds overlap the gathers' latency.
  T ya[U], yb[U];
#pragma unroll
  for (int u = 0; u < U; u++) yb[u] = (T)0;
  for (int o = 0; o < n_out; o++) {
    const T lo = pt.outer_leg(P, o);
    // Rounded sums and products are monotone, so every time of this outer
    // element lies between those of the shortest and the longest inner leg.
    const T first_p = A::mul(A::add(lo, mn), P.Fs), last_p = A::mul(A::add(lo, mx), P.Fs);
    const bool in = fin && first_p >= (T)0 && last_p < P.Kf;
    if (!BIGK && !IDX && __all_sync(0xffffffffu, in)) {
      int i = 0;
      for (; i + 2 * U <= n_in; i += 2 * U) {
        gather(lo, i, ya, true);
        accumulate(yb);
        gather(lo, i + U, yb, true);
        accumulate(ya);
      }
      if (i < n_in) {
        gather(lo, i, ya, false);
        accumulate(yb);
        gather(lo, i + U, yb, false);
        accumulate(ya);
      }
    } else if (FEW && !IDX && __all_sync(0xffffffffu, fin && (first_p >= P.Kf || last_p <= (T)-1))) {
      oob += n_in;
    } else if (FEW) {
      accumulate(yb);
#pragma unroll
      for (int u = 0; u < U; u++) yb[u] = (T)0;
      add_tested(lo);
    } else {
      for (int i = 0; i < n_in; i += 2 * U) {
        gather_tested(lo, i, ya);
        accumulate(yb);
        gather_tested(lo, i + U, yb);
        accumulate(ya);
      }
    }
    ycol += (int64_t)n_in * P.K;
  }
  accumulate(yb);
  if (!IDX && active) P.Im[no] = im;
  add_count(P.oob, active ? oob : 0u);
}

// ---------------------------------------------------------------------------
// launcher
// ---------------------------------------------------------------------------

template <class T, int M, bool UNI, bool IDX>
static cudaError_t launch_terms(const PlainParams<T> &P, cudaStream_t st) {
  const bool bigk = sizeof(T) == 4 && P.bigk;
  auto kern = bigk ? das_plain_kernel<T, M, UNI, true, IDX> : das_plain_kernel<T, M, UNI, false, IDX>;
  constexpr int bd = M == SAFT ? 256 : 128;
  kern<<<(unsigned)((P.no1 - P.no0 + bd - 1) / bd), bd, 0, st>>>(P);
  return cudaGetLastError();
}

template <class T, int M, bool UNI, bool IDX, int BD, int MINB = 3>
static cudaError_t launch_tile(const PlainParams<T> &P, int n_in, cudaStream_t st) {
  const size_t smem = plain_table_bytes(n_in, sizeof(T), BD);
  auto kern = P.bigk ? das_plain_tile_kernel<T, M, UNI, true, IDX, BD, MINB>
                     : das_plain_tile_kernel<T, M, UNI, false, IDX, BD, MINB>;
  cudaError_t e = ensure_smem(kern, smem);
  if (e != cudaSuccess) return e;
  dim3 grid;
  if (P.n_fast > 0) {  // [no0, no1) are tile rows
    constexpr int tf = plain_tile_f(M, BD);
    grid = dim3((unsigned)((P.n_fast + tf - 1) / tf), (unsigned)(P.no1 - P.no0));
  } else {
    grid = dim3((unsigned)((P.no1 - P.no0 + BD - 1) / BD));
  }
  kern<<<grid, BD, smem, st>>>(P);
  return cudaGetLastError();
}

template <class T, int M, bool UNI, bool IDX>
static cudaError_t launch_method(const PlainParams<T> &P, cudaStream_t st) {
  if constexpr (M == SAFT) {
    return launch_terms<T, M, UNI, IDX>(P, st);
  } else {
    const int n_in = M == RCA_ROWTX ? P.Nt : P.Nr;
    switch (plain_tile_threads(n_in, sizeof(T))) {
      case 128:
        if constexpr (sizeof(T) == 8 && !IDX)  // FP32 blocks need few enough registers for a fourth anyway
          if (plain_table_bytes(n_in, sizeof(T), 128) <= 54 * 1024) return launch_tile<T, M, UNI, IDX, 128, 4>(P, n_in, st);
        return launch_tile<T, M, UNI, IDX, 128>(P, n_in, st);
      case 64: return launch_tile<T, M, UNI, IDX, 64>(P, n_in, st);
      case 32: return launch_tile<T, M, UNI, IDX, 32>(P, n_in, st);
      default: return launch_terms<T, M, UNI, IDX>(P, st);
    }
  }
}

template <class T, bool UNI, bool IDX = false>
static cudaError_t launch_any(int method, const PlainParams<T> &P, cudaStream_t st) {
  switch (method) {
    case SAFT: return launch_method<T, SAFT, UNI, IDX>(P, st);
    case TFM: return launch_method<T, TFM, UNI, IDX>(P, st);
    case RCA_COLTX: return launch_method<T, RCA_COLTX, UNI, IDX>(P, st);
    case RCA_ROWTX: return launch_method<T, RCA_ROWTX, UNI, IDX>(P, st);
  }
  return cudaErrorInvalidValue;
}

template <class T>
static PlainParams<T> make_params(const PlainLaunch &L) {
  PlainParams<T> P{};
  P.Y = (const T *)L.Y;
  P.K = L.K;
  P.Ro = (const T *)L.Ro;
  P.No = L.No;
  P.no0 = L.no0;
  P.no1 = L.no1;
  P.n_fast = L.n_fast;
  P.n_slow = L.n_fast > 0 ? L.No / L.n_fast : 0;
  P.Gt = (const T *)L.Gt;
  P.Nt = (int)L.Nt;
  P.Gr = (const T *)L.Gr;
  P.Nr = (int)L.Nr;
  P.delay = (const T *)L.delay_vec;
  P.delay_multi = L.delay_multi ? 1 : 0;
  P.Im = (T *)L.Im;
  P.oob = L.oob;
  P.ny = L.ny;
  P.bad = L.bad;
  P.idx = L.idx;
  P.bigk = L.K >= (int64_t(1) << (sizeof(T) == 4 ? 22 : 28));
  P.Nx = L.Nx;
  P.Ny = L.Ny;
  P.Nz = L.Nz;
  return P;
}

cudaError_t launch_plain_f64(const PlainLaunch &L, cudaStream_t st) {
  PlainParams<double> P = make_params<double>(L);
  P.Fs = L.c64.Fs;
  P.ocp = L.c64.ocp;
  P.delay_ms = L.c64.delay_ms;
  P.Kf = (double)L.K;
  for (int i = 0; i < 15; i++) P.tri[i] = L.tri64[i];
  if (L.idx)
    return L.uni ? launch_any<double, true, true>(L.method, P, st)
                 : launch_any<double, false, true>(L.method, P, st);
  return L.uni ? launch_any<double, true>(L.method, P, st) : launch_any<double, false>(L.method, P, st);
}

cudaError_t launch_plain_f32(const PlainLaunch &L, cudaStream_t st) {
  PlainParams<float> P = make_params<float>(L);
  P.Fs = L.c32.Fs;
  P.ocp = L.c32.ocp;
  P.delay_ms = L.c32.delay_ms;
  P.Kf = (float)L.K;
  for (int i = 0; i < 15; i++) P.tri[i] = L.tri32[i];
  if (L.idx)
    return L.uni ? launch_any<float, true, true>(L.method, P, st)
                 : launch_any<float, false, true>(L.method, P, st);
  return L.uni ? launch_any<float, true>(L.method, P, st) : launch_any<float, false>(L.method, P, st);
}

}  // namespace dream
