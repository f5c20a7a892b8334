// das_fast.cu -- DAS with FP32- or BF16-stored A-scans, FP32 compensated
// accumulation and FP64-exact sample indices (precision upgrade of the
// reference's das_double/das_float forms; optional per-column weights for
// the differentiable operator), and the operator's adjoint.
//
// Gather: every index by the reference's own FP64 chain (below, at
// gather_issue). Tiles: a CTA owns a 2-D tile of image points (tile_f along the
// fastest grid axis x tile_s along the next one, when the caller gives the
// grid's fastest extent n_fast; otherwise consecutive points), so the 32
// gathers of one warp fall on one or two 128-byte lines of the A-scan.
//
// Scatter (adjoint): the same indices, added into shared-memory windows of the
// tile's columns (below, at scatter_windows).
#include <cuda_bf16.h>

#include <algorithm>

#include "das_common.cuh"
#include "das_fast.h"

namespace dream {

namespace {

template <class YT>
__device__ __forceinline__ float load_sample(const YT *p);
template <>
__device__ __forceinline__ float load_sample<float>(const float *p) {
  return __ldg(p);
}
template <>
__device__ __forceinline__ float load_sample<__nv_bfloat16>(const __nv_bfloat16 *p) {
  unsigned short u = __ldg(reinterpret_cast<const unsigned short *>(p));
  return __uint_as_float(((unsigned int)u) << 16);
}

// base (bytes) + off elements as one 32x32+64-bit multiply-add: as pointer + index it takes three moves more.
template <class YT>
__device__ __forceinline__ const YT *elem_addr(const char *base, uint32_t off) {
  const YT *r;
  asm("mad.wide.u32 %0, %1, %2, %3;" : "=l"(r) : "r"(off), "n"((int)sizeof(YT)), "l"(base));
  return r;
}

// Packed FP32 pairs (add.rn.f32x2 / fma.rn.f32x2, sm_100).
__device__ __forceinline__ uint64_t pack_f32x2(float a, float b) {
  uint64_t r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
  return r;
}
__device__ __forceinline__ uint64_t add_f32x2(uint64_t a, uint64_t b) {
  uint64_t r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ uint64_t fma_f32x2(uint64_t a, uint64_t b, uint64_t c) {
  uint64_t r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
  return r;
}
__device__ __forceinline__ uint64_t mul_f32x2(uint64_t a, uint64_t b) {
  uint64_t r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ float lo_f32(uint64_t v) { return __uint_as_float((uint32_t)v); }
__device__ __forceinline__ float hi_f32(uint64_t v) { return __uint_as_float((uint32_t)(v >> 32)); }

// Neumaier compensated add of x into (s, c).
__device__ __forceinline__ void neumaier(float &s, float &c, float x) {
  float t = s + x;
  float e = (fabsf(s) >= fabsf(x)) ? ((s - t) + x) : ((x - t) + s);
  c += e;
  s = t;
}

struct Pixel {
  double xo, yo, zo, delay_ms, gy_c, gx_r;
};


// Elements in Y: K times the A-scan columns (Nt for SAFT, Nt*Nr otherwise).
__device__ __forceinline__ int64_t y_count(const FastParams &P) {
  return P.ny ? P.ny : P.K * (int64_t)P.Nt * (P.method == SAFT ? 1 : P.Nr);
}

__device__ __forceinline__ void pixel_of(const FastParams &P, int64_t no, Pixel &px) {
  using A = Ar<double>;
  px.xo = P.Ro[no];
  px.yo = P.Ro[no + P.No];
  px.zo = P.Ro[no + 2 * P.No];
  px.delay_ms = P.delay[P.delay_multi ? no : 0] / 1000.0;
  px.gy_c = 0.0;
  px.gx_r = 0.0;
  if (P.method == RCA_COLTX || P.method == RCA_ROWTX) {
    // literal stripe-edge reads of extra_src/das.cc:464-467
    const double gc_y_min = P.Gr[0 + 1 * P.Nt], gc_y_max = P.Gr[P.Nt - 1 + 1 * P.Nt];
    const double gr_x_min = P.Gt[0], gr_x_max = P.Gt[P.Nr - 1];
    if (px.yo >= gc_y_min && px.yo <= gc_y_max) px.gy_c = 0.0;
    else if (px.yo < gc_y_min) px.gy_c = A::sub(gc_y_min, px.yo);
    else px.gy_c = A::sub(gc_y_max, px.yo);
    if (px.xo >= gr_x_min && px.xo <= gr_x_max) px.gx_r = 0.0;
    else if (px.xo < gr_x_min) px.gx_r = A::sub(gr_x_min, px.xo);
    else px.gx_r = A::sub(gr_x_max, px.xo);
  }
}

// Coordinate differences between image point px and element e (outer or
// inner), as the reference forms them for each method: TFM uses the element's
// position; an RCA column (Gt) its x and z with the clamped y offset of the
// column stripe, an RCA row (Gr) its y and z with the clamped x offset.
__device__ __forceinline__ void leg_diffs(const FastParams &P, const Pixel &px, bool outer, int e, double &dx,
                                          double &dy, double &dz) {
  if (P.method == TFM) {
    const double *G = outer ? P.Gt : P.Gr;
    const int N = outer ? P.Nt : P.Nr;
    dx = __dsub_rn(__ldg(G + e), px.xo);
    dy = __dsub_rn(__ldg(G + e + N), px.yo);
    dz = __dsub_rn(__ldg(G + e + 2 * N), px.zo);
  } else if ((P.method == RCA_COLTX) == outer) {  // a column
    dx = __dsub_rn(__ldg(P.Gt + e), px.xo);
    dy = px.gy_c;
    dz = __dsub_rn(__ldg(P.Gt + e + 2 * P.Nt), px.zo);
  } else {  // a row
    dx = px.gx_r;
    dy = __dsub_rn(__ldg(P.Gr + e + P.Nr), px.yo);
    dz = __dsub_rn(__ldg(P.Gr + e + 2 * P.Nr), px.zo);
  }
}

// Exact FP64 leg of outer or inner element e, including the delay on the leg
// that carries it (TFM and col-tx: outer; row-tx: inner, the column).
__device__ __forceinline__ double exact_leg(const FastParams &P, const Pixel &px, bool outer, int e) {
  double dx, dy, dz;
  leg_diffs(P, px, outer, e, dx, dy, dz);
  const double l = leg_time(dx, dy, dz, P.ocp);
  return (P.method == RCA_ROWTX) != outer ? __dadd_rn(l, px.delay_ms) : l;
}

// The reference's exact index of term (o, i): returns false when out of bounds.
__device__ __noinline__ bool exact_index(const FastParams &P, const Pixel &px, int o, int i, int &k) {
  using A = Ar<double>;
  double p = A::mul(A::add(exact_leg(P, px, true, o), exact_leg(P, px, false, i)), P.Fs);
  if (P.K > 0 && p > -1.0 && p < (double)P.K) {
    k = trunc_index(p);
    return true;
  }
  return false;
}

// A-scan column of term (outer o, inner i): o * n_in + i for a full Y. A Y
// holding only the columns of inner elements [ycol_i0, ycol_i0 + ycol_o) (an
// inner-element shard) has ycol_o columns per outer element.
__device__ __forceinline__ int64_t ycol_outer(const FastParams &P, int n_in, int o) {
  return (int64_t)o * (P.ycol_o > 0 ? P.ycol_o : n_in);
}
__device__ __forceinline__ int64_t ycol_inner(const FastParams &P, int i) { return (int64_t)i - P.ycol_i0; }
__device__ __forceinline__ int64_t ycol(const FastParams &P, int n_in, int o, int i) {
  return ycol_outer(P, n_in, o) + ycol_inner(P, i);
}

constexpr double LEG_LIMIT = 8388608.0;  // 2^23 samples: window bases and extents stay below it

// Range of |g - c| for c in [c0, c1].
__device__ __forceinline__ void offset_range(double g, double c0, double c1, double &lo, double &hi) {
  lo = g < c0 ? c0 - g : (g > c1 ? g - c1 : 0.0);
  hi = fmax(fabs(g - c0), fabs(g - c1));
}

// Range of |s(c)| for c in [c0, c1], s the reference's stripe offset: 0 on
// [e0, e1], e0 - c below, e1 - c above (extra_src/das.cc:470-480).
__device__ __forceinline__ void stripe_range(double e0, double e1, double c0, double c1, double &lo, double &hi) {
  auto s = [&](double c) { return (c >= e0 && c <= e1) ? 0.0 : (c < e0 ? e0 - c : e1 - c); };
  hi = fmax(fabs(s(c0)), fabs(s(c1)));
  lo = (e0 <= e1) ? fmax(0.0, fmax(e0 - c1, c0 - e1)) : 0.0;
}

// Bounding box of a tile's image points and delays: x, y, z, delay (ms).
struct TileBox {
  double lo[4], hi[4];
};

// Leg range [Lmin, Lmax] in samples of element e over the tile box.
__device__ __forceinline__ void leg_range(const FastParams &P, const TileBox &B, bool outer, int e, double &Lmin,
                                          double &Lmax) {
  double lx, hx, ly, hy, lz, hz;
  if (P.method == TFM) {
    const double *G = outer ? P.Gt : P.Gr;
    const int N = outer ? P.Nt : P.Nr;
    offset_range(G[e], B.lo[0], B.hi[0], lx, hx);
    offset_range(G[e + N], B.lo[1], B.hi[1], ly, hy);
    offset_range(G[e + 2 * N], B.lo[2], B.hi[2], lz, hz);
  } else if ((P.method == RCA_COLTX) == outer) {  // a column; stripe edges as pixel_of reads them
    offset_range(P.Gt[e], B.lo[0], B.hi[0], lx, hx);
    stripe_range(P.Gr[0 + P.Nt], P.Gr[P.Nt - 1 + P.Nt], B.lo[1], B.hi[1], ly, hy);
    offset_range(P.Gt[e + 2 * P.Nt], B.lo[2], B.hi[2], lz, hz);
  } else {  // a row
    stripe_range(P.Gt[0], P.Gt[P.Nr - 1], B.lo[0], B.hi[0], lx, hx);
    offset_range(P.Gr[e + P.Nr], B.lo[1], B.hi[1], ly, hy);
    offset_range(P.Gr[e + 2 * P.Nr], B.lo[2], B.hi[2], lz, hz);
  }
  const bool dl = (P.method == RCA_ROWTX) ? !outer : outer;  // the leg that carries the delay
  Lmin = (sqrt(lx * lx + ly * ly + lz * lz) * P.ocp + (dl ? B.lo[3] : 0.0)) * P.Fs;
  Lmax = (sqrt(hx * hx + hy * hy + hz * hz) * P.ocp + (dl ? B.hi[3] : 0.0)) * P.Fs;
}

// ---------------------------------------------------------------------------
// Gather: one tile of image points, every sample index by the reference's own
// FP64 chain.
//
// trunc(RN(RN(a + b) * Fs)) costs three FP64 instructions per term (leg sum,
// scale, truncation by adding 2^52 toward zero), which the FP64 pipe executes
// beside the integer unit's addresses; in the low mantissa word the last one
// leaves the sample number plus the column offset j * K inside the chunk. The
// bounds test is one vote per chunk: rounded sums and products are monotone, so
// the shortest and the longest legs decide exactly whether every term of the
// chunk is in bounds.
//
// Bound (64x64 elements, K = 3000, 512x512 points, FP32 storage): 0.42 ms at 9.3
// instructions per 32 terms and 0.67 of the issue slots; 6.5 of them are the three
// FP64 operations, the 64-bit address, the load and half a packed add, about 2.5
// the legs. The FP64 pipe is at 0.52 (its own limit for the terms alone would be
// 0.17 ms), the L1 data pipe at 0.43. Fixed-point legs with an ambiguity test
// and an FP64 fallback, the form this replaces, took 0.505 ms there, 0.069
// against 0.037 for 32x32 elements and 256x256 points (no per-tile set-up with
// block barriers here), 38.0 against 25.6 for the 128x128-element RCA volume.
//
// Layout: 8 inner legs and the 8 addends of the truncation in registers, the
// outer legs in shared memory (a thread reads only its own: no barrier), two
// groups of 4 outer x 8 inner gathers alternating. 16 inner legs with one or two
// outer elements per group: 0.47 - 0.57 ms; 2 outer elements per group 0.48; one
// group at a time 0.55; 96 registers (five blocks) 0.47 - 0.51.
// ---------------------------------------------------------------------------

constexpr int GATHER_JC = 8;  // inner elements per register chunk
constexpr int GATHER_NO = 4;  // outer elements whose gathers are issued together

// Raw bits of a gathered sample, and their value: the conversion waits for the
// sample, so it belongs to the sum.
__device__ __forceinline__ uint32_t load_bits(const float *p) { return __float_as_uint(__ldg(p)); }
__device__ __forceinline__ uint32_t load_bits(const __nv_bfloat16 *p) {
  return __ldg(reinterpret_cast<const unsigned short *>(p));
}
template <class YT>
__device__ __forceinline__ float sample_of(uint32_t bits) {
  return __uint_as_float(sizeof(YT) == 2 ? bits << 16 : bits);
}

// Issues the gathers of NO outer elements (legs a) x the chunk's inner elements
// (FULL: all of them, else the first jn), all in bounds. yc: address of the
// first term's column; the next outer element's is ystep bytes further.
template <class YT, bool FULL, int NO>
__device__ __forceinline__ void gather_issue(const FastParams &P, const double (&a)[NO], const double (&B)[GATHER_JC],
                                             const double (&mag)[GATHER_JC], double Fs, const char *yc, int64_t ystep,
                                             int jn, uint32_t (&y)[NO][GATHER_JC]) {
#pragma unroll
  for (int q = 0; q < NO; q++, yc += ystep) {
#pragma unroll
    for (int j = 0; j < GATHER_JC; j++) {
      y[q][j] = 0;
      const uint32_t k = (uint32_t)__double2loint(__dadd_rz(__dmul_rn(__dadd_rn(a[q], B[j]), Fs), mag[j]));
      if ((FULL || j < jn) && gather_ok<float>(elem_addr<YT>(yc, k) - reinterpret_cast<const YT *>(P.Y), y_count(P), P.bad))
        y[q][j] = load_bits(elem_addr<YT>(yc, k));
    }
  }
}

// Their sum, as a tree of packed pairs; weighted, w holds the chunk's
// weights of the first outer element (shared memory, GATHER_JC per element).
template <class YT, bool WEIGHTED, int NO>
__device__ __forceinline__ float gather_sum(const uint32_t (&y)[NO][GATHER_JC], const float *w) {
  constexpr int JP = GATHER_JC / 2;
  uint64_t v[NO * JP];
  auto pair = [&](int q, int j) { return pack_f32x2(sample_of<YT>(y[q][2 * j]), sample_of<YT>(y[q][2 * j + 1])); };
#pragma unroll
  for (int q = 0; q < NO; q++)
#pragma unroll
    for (int j = 0; j < JP; j += 2) {
      uint64_t w0 = 0, w1 = 0;
      if (WEIGHTED) {
        const float4 w4 = *reinterpret_cast<const float4 *>(w + q * GATHER_JC + 2 * j);
        w0 = pack_f32x2(w4.x, w4.y);
        w1 = pack_f32x2(w4.z, w4.w);
      }
      if (!WEIGHTED) {
        v[q * JP + j] = pair(q, j);
        v[q * JP + j + 1] = pair(q, j + 1);
      } else if (q == 0) {
        v[j] = mul_f32x2(pair(q, j), w0);
        v[j + 1] = mul_f32x2(pair(q, j + 1), w1);
      } else {
        v[j] = fma_f32x2(pair(q, j), w0, v[j]);
        v[j + 1] = fma_f32x2(pair(q, j + 1), w1, v[j + 1]);
      }
    }
#pragma unroll
  for (int n = (WEIGHTED ? JP : NO * JP) / 2; n >= 1; n /= 2)
#pragma unroll
    for (int j = 0; j < n; j++) v[j] = add_f32x2(v[j], v[j + n]);
  return lo_f32(v[0]) + hi_f32(v[0]);
}

// One outer element against a chunk, every term tested.
template <class YT, bool WEIGHTED>
__device__ __forceinline__ float gather_tested(const FastParams &P, double a, const double (&B)[GATHER_JC], double Fs,
                                               double Kf, const char *yc, const float *w, int jn, unsigned int &oob) {
  float part = 0.0f;
#pragma unroll
  for (int j = 0; j < GATHER_JC; j++) {
    if (j >= jn) break;
    const double p = __dmul_rn(__dadd_rn(a, B[j]), Fs);
    if (p > -1.0 && p < Kf) {
      const YT *e = reinterpret_cast<const YT *>(yc) + (j * P.K + trunc_index(p));
      const float y = gather_ok<float>(e - reinterpret_cast<const YT *>(P.Y), y_count(P), P.bad) ? load_sample(e) : 0.0f;
      part = WEIGHTED ? fmaf(w[j], y, part) : part + y;
    } else {
      oob++;
    }
  }
  return part;
}

// Bounds of a set of legs from their high words: the words as integers in the
// legs' order (NaN above everything), widened to whole high words, so a set
// costs four integer instructions per leg instead of FP64 comparisons.
struct LegBounds {
  int lo = INT_MAX, hi = INT_MIN;
  __device__ __forceinline__ void add(double l) {
    const int h = __double2hiint(l), key = h ^ ((h >> 31) & 0x7fffffff);
    lo = min(lo, key);
    hi = max(hi, key);
  }
  __device__ __forceinline__ bool finite() const { return hi < 0x7ff00000 && lo > (int)0x800fffff; }
  static __device__ __forceinline__ int word(int key) { return key ^ ((key >> 31) & 0x7fffffff); }
  __device__ __forceinline__ double min_leg() const { return __hiloint2double(word(lo), lo < 0 ? -1 : 0); }
  __device__ __forceinline__ double max_leg() const { return __hiloint2double(word(hi), hi < 0 ? 0 : -1); }
};

// The image point of this thread (inactive lanes repeat the tile's first point)
// in tile (tfi, tsi) of T.tile_f x T.tile_s points (P's own, for the gathers); lines
// in the order of volume_line.
template <class Tile>
__device__ __forceinline__ int64_t tile_point(const FastParams &P, const Tile &T, int64_t tfi, int64_t tsi, uint32_t row,
                                              bool &active) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int lf = lane % P.wf, ls = lane / P.wf;
  const int warps_f = T.tile_f / P.wf;
  const int wfi = warp % warps_f, wsi = warp / warps_f;
  const int64_t f = tfi * T.tile_f + wfi * P.wf + lf;
  const int64_t s = tsi * T.tile_s + wsi * (32 / P.wf) + ls;
  active = f < P.n_fast && s < P.n_slow;
  return active ? volume_line(s, row, P.n_slow) * P.n_fast + f
                : volume_line(tsi * T.tile_s, row, P.n_slow) * P.n_fast + tfi * T.tile_f;
}

// Whether a block looks for rows of lines: RCAs, which image volumes, with terms
// enough to pay for the search.
template <int METHOD>
__device__ __forceinline__ bool volume_tiles(const FastParams &P) {
  return METHOD != TFM && (int64_t)P.Nt * P.Nr >= VOLUME_TERMS;
}

// The legs of one side of a method's term: a point element (TFM), a column or a
// row of an RCA, read through its coordinate columns.
enum LegKind : int { POINT, COLUMN, ROW };
__host__ __device__ constexpr LegKind leg_kind(int method, bool outer) {
  return method == TFM ? POINT : ((method == RCA_COLTX) == outer ? COLUMN : ROW);
}
template <int METHOD, bool OUTER>
struct Legs {
  static constexpr LegKind KIND = leg_kind(METHOD, OUTER);
  static constexpr bool DELAYED = (METHOD == RCA_ROWTX) != OUTER;
  const double *x, *y, *z;
  __device__ __forceinline__ explicit Legs(const FastParams &P) {
    const bool tx = KIND == COLUMN || (KIND == POINT && OUTER);
    const int N = tx ? P.Nt : P.Nr;
    x = tx ? P.Gt : P.Gr;
    y = x + N;
    z = y + N;
  }
  // The exact FP64 leg of element e (as exact_leg).
  __device__ __forceinline__ double operator()(const FastParams &P, const Pixel &px, int e) const {
    const double l = leg_time(KIND == ROW ? px.gx_r : __dsub_rn(__ldg(x + e), px.xo),
                              KIND == COLUMN ? px.gy_c : __dsub_rn(__ldg(y + e), px.yo),
                              __dsub_rn(__ldg(z + e), px.zo), P.ocp);
    return DELAYED ? __dadd_rn(l, px.delay_ms) : l;
  }
};

// One tile of image points (tile indices tfi along the fast axis, tsi along the
// slow axis) with the frame described by P; smem_raw holds the legs of
// P.out_block outer elements per thread. No thread reads another's legs, so
// there is no barrier. Called by the one-frame kernel and by the persistent
// batch kernel.
template <class YT, bool WEIGHTED, int METHOD>
__device__ __forceinline__ void gather_tile(const FastParams &P, int64_t tfi, int64_t tsi, unsigned char *smem_raw) {
  __shared__ double s_mag[GATHER_JC];
  if (threadIdx.x < GATHER_JC) s_mag[threadIdx.x] = 4503599627370496.0 + (double)(threadIdx.x * P.K);
  __syncthreads();
  const int nthr = blockDim.x;
  double *tab = reinterpret_cast<double *>(smem_raw) + threadIdx.x;  // leg of outer element o0 + o: tab[o * nthr]
  float *ws = reinterpret_cast<float *>(smem_raw + (size_t)P.out_block * nthr * sizeof(double));  // weights [o][GATHER_JC]
  const int n_out = METHOD == RCA_ROWTX ? P.Nr : P.Nt, n_in = METHOD == RCA_ROWTX ? P.Nt : P.Nr;
  const Legs<METHOD, true> outer(P);
  const Legs<METHOD, false> inner(P);
  const int i_lo = P.in_lo, i_hi = P.in_hi > 0 ? P.in_hi : n_in;
  const int64_t ostride = P.ycol_o > 0 ? P.ycol_o : n_in;  // columns per outer element
  bool active;
  __shared__ uint32_t s_row;
  if (METHOD != TFM) {
    const uint32_t row = volume_tiles<METHOD>(P) ? volume_row(P.Ro, P.No, P.n_fast, P.n_slow) : 0;
    if (threadIdx.x == 0) s_row = row;
    __syncthreads();
  }
  auto point = [&]() { return tile_point(P, P, tfi, tsi, METHOD != TFM ? *(volatile uint32_t *)&s_row : 0, active); };
  Pixel px;
  pixel_of(P, point(), px);
  // 2^52 + j * K, read from shared memory: as uniform values each use would move them to a register first
  double mag[GATHER_JC];
#pragma unroll
  for (int j = 0; j < GATHER_JC; j++) mag[j] = s_mag[j];
  const YT *Y = reinterpret_cast<const YT *>(P.Y);
  const int64_t ystep = ostride * P.K * (int64_t)sizeof(YT);  // bytes between the columns of neighbouring outer elements
  const double Kf = (double)P.K, Fs = P.Fs;
  float acc_s = 0.0f, acc_c = 0.0f;
  unsigned int oob = 0;
  for (int o0 = 0; o0 < n_out; o0 += P.out_block) {
    const int on = min(P.out_block, n_out - o0);
    LegBounds bA;
#pragma unroll 4
    for (int o = 0; o < on; o++) {
      const double l = outer(P, px, o0 + o);
      tab[o * nthr] = l;
      bA.add(l);
    }
    // no vote for a NaN leg, a negative Fs, or sample numbers beyond 32 bits
    const bool fin = bA.finite() && P.Fs > 0.0 && P.K < (int64_t(1) << 28);
    const double mnA = bA.min_leg(), mxA = bA.max_leg();
    for (int i0 = i_lo; i0 < i_hi; i0 += GATHER_JC) {
      const int jn = min(GATHER_JC, i_hi - i0);
      double B[GATHER_JC];
      LegBounds bB;
#pragma unroll
      for (int j = 0; j < GATHER_JC; j++) {
        if (j >= jn) {
          B[j] = B[0];  // past the last inner element: never gathered
          continue;
        }
        B[j] = inner(P, px, i0 + j);
        bB.add(B[j]);
      }
      const bool ok = fin && bB.finite();
      const double mnB = bB.min_leg(), mxB = bB.max_leg();
      const int64_t col = o0 * ostride + ycol_inner(P, i0);
      const char *yc = reinterpret_cast<const char *>(Y + col * P.K);  // the chunk's first column, outer element o
      const float *w = ws;                                            // and its weights
      if (WEIGHTED) {
        __syncthreads();  // the last chunk's weights are read
        for (int e = threadIdx.x; e < on * GATHER_JC; e += nthr) {
          const int j = e % GATHER_JC;
          ws[e] = j < jn ? __ldg(P.w + col + e / GATHER_JC * ostride + j) : 0.0f;
        }
        __syncthreads();
      }
      const bool in = ok && __dmul_rn(__dadd_rn(mnA, mnB), Fs) >= 0.0 && __dmul_rn(__dadd_rn(mxA, mxB), Fs) < Kf;
      int o = 0;
      if (__all_sync(0xffffffffu, in)) {
        constexpr int NO = GATHER_NO;
        auto outer_legs = [&](int g, double(&a)[NO]) {
#pragma unroll
          for (int q = 0; q < NO; q++) a[q] = tab[(g + q) * nthr];
        };
        if (jn == GATHER_JC && on >= 2 * NO) {
          // two groups alternate: the gathers of one are issued before the other is summed
          uint32_t y0[NO][GATHER_JC], y1[NO][GATHER_JC];
          auto issue = [&](int g, const char *c, uint32_t(&y)[NO][GATHER_JC]) {
            double a[NO];
            outer_legs(g, a);
            gather_issue<YT, true, NO>(P, a, B, mag, Fs, c, ystep, jn, y);
          };
          issue(0, yc, y0);
          for (; o + 2 * NO <= on; o += 2 * NO, w += 2 * NO * GATHER_JC) {
            issue(o + NO, yc + NO * ystep, y1);
            // FP32 storage compensates every 32 terms (whole-image error against FP64 3.2e-8 on the 64x64-element
            // frame; 64 terms: 3.5e-8); BF16's own rounding is 10^4 times larger, so 64 do there (0.439 against 0.478 ms)
            float p0 = gather_sum<YT, WEIGHTED, NO>(y0, w);
            if (sizeof(YT) == 4) neumaier(acc_s, acc_c, p0);
            yc += 2 * NO * ystep;
            if (o + 4 * NO <= on) issue(o + 2 * NO, yc, y0);
            const float p1 = gather_sum<YT, WEIGHTED, NO>(y1, w + NO * GATHER_JC);
            neumaier(acc_s, acc_c, sizeof(YT) == 4 ? p1 : p0 + p1);
          }
        }
        for (; o + NO <= on; o += NO, yc += NO * ystep, w += NO * GATHER_JC) {  // the last, partly filled chunk
          double a[NO];
          outer_legs(o, a);
          uint32_t y[NO][GATHER_JC];
          gather_issue<YT, false, NO>(P, a, B, mag, Fs, yc, ystep, jn, y);
          neumaier(acc_s, acc_c, gather_sum<YT, WEIGHTED, NO>(y, w));
        }
        for (; o < on; o++, yc += ystep, w += GATHER_JC) {
          const double a0[1] = {tab[o * nthr]};
          uint32_t y[1][GATHER_JC];
          gather_issue<YT, false, 1>(P, a0, B, mag, Fs, yc, ystep, jn, y);
          neumaier(acc_s, acc_c, gather_sum<YT, WEIGHTED, 1>(y, w));
        }
      } else {
        for (; o < on; o++, yc += ystep, w += GATHER_JC) {
          const double a0[1] = {tab[o * nthr]};
          const double lo = __dmul_rn(__dadd_rn(a0[0], mnB), Fs), hi = __dmul_rn(__dadd_rn(a0[0], mxB), Fs);
          if (__all_sync(0xffffffffu, ok && lo >= 0.0 && hi < Kf)) {
            uint32_t y[1][GATHER_JC];
            gather_issue<YT, false, 1>(P, a0, B, mag, Fs, yc, ystep, jn, y);
            neumaier(acc_s, acc_c, gather_sum<YT, WEIGHTED, 1>(y, w));
          } else if (__all_sync(0xffffffffu, ok && (lo >= Kf || hi <= -1.0))) {
            oob += jn;
          } else {
            neumaier(acc_s, acc_c, gather_tested<YT, WEIGHTED>(P, a0[0], B, Fs, Kf, yc, w, jn, oob));
          }
        }
      }
    }
  }
  const int64_t no = point();  // worked out again: the loop has no register for it
  if (active) P.Im[no] = P.accumulate ? P.Im[no] + (acc_s + acc_c) : acc_s + acc_c;
  add_count(P.oob, active ? oob : 0u);
}

template <class YT, bool WEIGHTED, int METHOD>
__global__ void __launch_bounds__(256, 2) das_fast_kernel(const FastParams P) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  gather_tile<YT, WEIGHTED, METHOD>(P, blockIdx.x, (int64_t)blockIdx.y + P.slow_tile0, smem_raw);
}

}  // namespace

// Persistent batch kernel: CTAs take (frame, tile) work items from a queue
// (items sorted by decreasing cost on the host) until it is empty. The frame
// descriptor is staged in shared memory; every frame's tile has blockDim.x
// points. ctr must be zero at launch (the batch run resets it).
template <class YT>
__global__ void __launch_bounds__(128, 3) das_batch_kernel(const FastParams *__restrict__ frames,
                                                        const int4 *__restrict__ items, int n_items,
                                                        int *__restrict__ ctr) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ FastParams sP;
  __shared__ int s_item;
  for (;;) {
    if (threadIdx.x == 0) s_item = atomicAdd(ctr, 1);
    __syncthreads();
    const int it = s_item;
    if (it >= n_items) break;
    const int4 w = items[it];
    if (threadIdx.x == 0) sP = frames[w.x];
    __syncthreads();
    if (sP.method == TFM) gather_tile<YT, false, TFM>(sP, w.y, w.z, smem_raw);
    else if (sP.method == RCA_COLTX) gather_tile<YT, false, RCA_COLTX>(sP, w.y, w.z, smem_raw);
    else gather_tile<YT, false, RCA_ROWTX>(sP, w.y, w.z, smem_raw);
    __syncthreads();
  }
}

// SAFT: one leg per term, t_dp = 2*(leg + delay); the FP64 index is computed
// per term (each term has its own element), samples from FP32/BF16 storage.
template <class YT, bool WEIGHTED>
__global__ void __launch_bounds__(256) das_fast_saft_kernel(const FastParams P) {
  using A = Ar<double>;
  const int64_t no_raw = P.no0 + (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const bool active = no_raw < P.no1;
  const int64_t no = active ? no_raw : P.no0;
  Pixel px;
  pixel_of(P, no, px);
  const YT *__restrict__ Y = reinterpret_cast<const YT *>(P.Y);
  float acc_s = 0.0f, acc_c = 0.0f, part = 0.0f;
  unsigned int oob = 0;
  for (int n = 0; n < P.Nt; n++) {
    double l = leg_time(A::sub(P.Gt[n], px.xo), A::sub(P.Gt[n + P.Nt], px.yo), A::sub(P.Gt[n + 2 * P.Nt], px.zo),
                        P.ocp);
    double p = A::mul(A::mul(2.0, A::add(l, px.delay_ms)), P.Fs);
    if (P.K > 0 && p > -1.0 && p < (double)P.K) {
      const int64_t gi = (int64_t)n * P.K + trunc_index(p);
      float y = gather_ok<float>(gi, y_count(P), P.bad) ? load_sample(Y + gi) : 0.0f;
      part = WEIGHTED ? fmaf(__ldg(P.w + n), y, part) : part + y;
    } else {
      oob++;
    }
    if ((n & 15) == 15) {
      neumaier(acc_s, acc_c, part);
      part = 0.0f;
    }
  }
  neumaier(acc_s, acc_c, part);
  if (active) P.Im[no] = acc_s + acc_c;
  add_count(P.oob, active ? oob : 0u);
}

__global__ void f32_to_bf16_kernel(const float *__restrict__ x, __nv_bfloat16 *__restrict__ y, int64_t n) {
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
    y[i] = __float2bfloat16_rn(x[i]);
}

// ---------------------------------------------------------------------------
// host side
// ---------------------------------------------------------------------------

size_t gather_smem_bytes(const FastParams &P, int nthr) {
  return (size_t)P.out_block * (nthr * sizeof(double) + (P.w ? GATHER_JC * sizeof(float) : 0));
}

template <class YT, bool W>
static cudaError_t launch_fast_t(const FastParams &P, cudaStream_t st) {
  if (P.method == SAFT) {
    int64_t n = P.no1 - P.no0;
    if (n <= 0) return cudaSuccess;
    das_fast_saft_kernel<YT, W><<<(unsigned)((n + 255) / 256), 256, 0, st>>>(P);
    return cudaGetLastError();
  }
  const int nthr = P.tile_f * P.tile_s;
  const size_t smem = gather_smem_bytes(P, nthr);
  auto kern = P.method == TFM         ? das_fast_kernel<YT, W, TFM>
              : P.method == RCA_COLTX ? das_fast_kernel<YT, W, RCA_COLTX>
                                      : das_fast_kernel<YT, W, RCA_ROWTX>;
  cudaError_t e = ensure_smem(kern, smem);
  if (e != cudaSuccess) return e;
  const int64_t gx = (P.n_fast + P.tile_f - 1) / P.tile_f;
  const int64_t gy = P.slow_tile1 - P.slow_tile0;
  if (gx <= 0 || gy <= 0) return cudaSuccess;
  dim3 grid((unsigned)gx, (unsigned)gy);
  kern<<<grid, nthr, smem, st>>>(P);
  return cudaGetLastError();
}

cudaError_t launch_fast(const FastParams &P, bool bf16, cudaStream_t st) {
  const bool W = P.w != nullptr;
  if (bf16) return W ? launch_fast_t<__nv_bfloat16, true>(P, st) : launch_fast_t<__nv_bfloat16, false>(P, st);
  return W ? launch_fast_t<float, true>(P, st) : launch_fast_t<float, false>(P, st);
}

// Stream operations only (memset + launch), so a batch run can be captured
// in a CUDA graph; the kernel attribute is set once by batch_prepare.
cudaError_t launch_batch(const FastParams *frames, const int4 *items, int n_items, int *ctr, size_t smem, bool bf16,
                         int grid, cudaStream_t st) {
  cudaError_t e = cudaMemsetAsync(ctr, 0, sizeof(int), st);
  if (e != cudaSuccess || n_items == 0) return e;
  if (bf16) das_batch_kernel<__nv_bfloat16><<<grid, 128, smem, st>>>(frames, items, n_items, ctr);
  else das_batch_kernel<float><<<grid, 128, smem, st>>>(frames, items, n_items, ctr);
  return cudaGetLastError();
}

// Raises the dynamic shared-memory limit where needed (never lowers it: an older
// batch may need more); returns resident CTAs per SM (0 on error).
int batch_prepare(size_t smem, bool bf16) {
  auto kern = bf16 ? das_batch_kernel<__nv_bfloat16> : das_batch_kernel<float>;
  if (ensure_smem(kern, smem) != cudaSuccess) return 0;
  int n = 0;
  cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, kern, 128, smem);
  return n;
}

__global__ void f32_to_bf16_2d_kernel(const float *__restrict__ x, __nv_bfloat16 *__restrict__ y, int64_t rows,
                                      int64_t row_elems, int64_t pitch) {
  const int64_t n = rows * row_elems;
  for (int64_t q = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; q < n; q += (int64_t)gridDim.x * blockDim.x) {
    const int64_t r = q / row_elems, e = q - r * row_elems;
    y[r * pitch + e] = __float2bfloat16_rn(x[r * pitch + e]);
  }
}

cudaError_t convert_f32_to_bf16_2d(const float *x, void *y, int64_t rows, int64_t row_elems, int64_t pitch,
                                   cudaStream_t st) {
  const int64_t n = rows * row_elems;
  if (n <= 0) return cudaSuccess;
  int blocks = (int)std::min<int64_t>((n + 255) / 256, 148 * 16);
  f32_to_bf16_2d_kernel<<<blocks, 256, 0, st>>>(x, reinterpret_cast<__nv_bfloat16 *>(y), rows, row_elems, pitch);
  return cudaGetLastError();
}

cudaError_t convert_f32_to_bf16(const float *x, void *y, int64_t n, cudaStream_t st) {
  if (n <= 0) return cudaSuccess;
  int blocks = (int)std::min<int64_t>((n + 255) / 256, 148 * 16);
  f32_to_bf16_kernel<<<blocks, 256, 0, st>>>(x, reinterpret_cast<__nv_bfloat16 *>(y), n);
  return cudaGetLastError();
}


// ===========================================================================
// Adjoint (scatter) on pixel tiles: Ya[k(n,c), c] += w[c] * x[n] for the
// tile's image points n and every A-scan column c, at the forward's indices.
// Ya must be zeroed (or hold the partial sum to add to) before the launch.
//
// The box bounding the tile's points and delays gives every element's leg range
// (leg_range), hence an integer base (a multiple of 4) and extent per leg; a
// column's samples then lie in the window [base_o + base_i, + ext_o + ext_i +
// 2). Per batch of 2 outer x 8 inner elements every term is added into its
// column's window in shared memory (the addition of the truncation carries the
// window row and the inner base, the row address the outer base), then a fixed
// group of threads per row adds the row to the A-scan with 4-wide vector
// reductions, the weight applied once per sample, and clears it. Two window
// buffers alternate, so one block barrier per batch suffices (between its adds
// and its flush).
//
// Bound: instruction issue (0.59 of the slots; 15.5 instructions per 32 terms, of
// which the index chain, the cell's address and the shared addition are 5, the
// legs of two blocks of outer elements about 2) and the shared-memory / L1 data
// pipe (0.72: a warp's additions to one cell take a wavefront each, 2.7 per
// instruction with 8 x 4 points per warp). 64x64 elements, K = 3000, 512x512
// points: 0.82 ms, weighted 0.85; with fixed-point legs, an ambiguity test and
// batches of one outer x 16 inner elements 0.83 and 0.99 (37x53 elements 0.33
// against 0.55, 32x32 and 256x256 points 0.077 against 0.085). The adds carry no
// guard and the flush no test for zeros: either costs a branch per term (1.2 and
// 0.97 ms).
// ===========================================================================

namespace {

constexpr int SCATTER_JC = 8, SCATTER_NO = 2, SCATTER_ROWS = SCATTER_NO * SCATTER_JC;
// Samples per window row; tiles of wider windows add every term with a global reduction.
constexpr int SCATTER_WCAP = 192;
// Smallest largest |x| of a tile of windows: its scale 2^(22 - E) and the inverse are normal FP32 numbers.
constexpr float SCATTER_X_MIN = 0x1p-104f;

// be of every element, then (16-byte aligned) the two window buffers, then the outer legs.
__host__ __device__ constexpr size_t scatter_head_bytes(int n_out, int n_in) {
  return ((size_t)2 * (n_out + n_in) * sizeof(int) + 15) & ~(size_t)15;
}
constexpr size_t SCATTER_WIN_BYTES = 2 * (size_t)SCATTER_ROWS * SCATTER_WCAP * sizeof(int);

__device__ __forceinline__ void red_add_v4(float *p, float4 v) {
  asm volatile("red.global.add.v4.f32 [%0], {%1, %2, %3, %4};" ::"l"(p), "f"(v.x), "f"(v.y), "f"(v.z), "f"(v.w)
               : "memory");
}
__device__ __forceinline__ void red_add(const float *p, float v) {
  asm volatile("red.global.add.f32 [%0], %1;" ::"l"(p), "f"(v) : "memory");
}
__device__ __forceinline__ void red_add_shared(uint32_t a, int v) {
  asm volatile("red.shared.add.u32 [%0], %1;" ::"r"(a), "r"(v) : "memory");
}

// Scatter of terms (o, i0 .. i0+jn-1) of one image point, straight into Ya.
template <bool WEIGHTED>
__device__ __noinline__ void exact_scatter(const FastParams &P, const Pixel &px, int o, int i0, int jn, int n_in,
                                           float xn, float *Ya) {
  for (int j = 0; j < jn; j++) {
    int k;
    const int64_t col = ycol(P, n_in, o, i0 + j);
    if (exact_index(P, px, o, i0 + j, k)) atomicAdd(Ya + col * P.K + k, WEIGHTED ? __ldg(P.w + col) * xn : xn);
  }
}

struct ScatterTile {
  int2 *be;                  // [n_out + n_in]: integer base of each leg over the tile, bound of floor(leg) - base
  bool usable;               // every base and extent is valid
  bool low;                  // some term may lie before sample 0
  bool in_bounds;            // every term of the tile is in bounds
  int ext_outer, ext_inner;  // largest extents
  float x_max, w_max;        // largest |x| and |weight|, NaN above all
  bool x_scales;             // the windows' fixed-point scale of x_max and its inverse are normal FP32 numbers
};

// Leg bounds and value range of the tile; `scratch`: (blockDim.x / 32) * 8 doubles and 9 ints.
template <bool WEIGHTED>
__device__ __forceinline__ void scatter_setup(const FastParams &P, const Pixel &px, float xn, int w_mx, unsigned char *smem,
                                              double *scratch, int n_out, int n_in, int i_lo, int i_hi, ScatterTile &T) {
  const int tid = threadIdx.x, nthr = blockDim.x, lane = tid & 31, warp = tid >> 5, nwarps = nthr >> 5;
  T.be = reinterpret_cast<int2 *>(smem);
  double *red = scratch;
  int *stat = reinterpret_cast<int *>(red + nwarps * 8);
  constexpr int STAT = WEIGHTED ? 9 : 8;
  {
    double mn[4] = {px.xo, px.yo, px.zo, px.delay_ms}, mx[4] = {px.xo, px.yo, px.zo, px.delay_ms};
#pragma unroll
    for (int off = 16; off > 0; off >>= 1)
#pragma unroll
      for (int q = 0; q < 4; q++) {
        mn[q] = fmin(mn[q], __shfl_xor_sync(0xffffffffu, mn[q], off));
        mx[q] = fmax(mx[q], __shfl_xor_sync(0xffffffffu, mx[q], off));
      }
    if (lane == 0)
#pragma unroll
      for (int q = 0; q < 4; q++) {
        red[warp * 8 + q] = mn[q];
        red[warp * 8 + 4 + q] = mx[q];
      }
  }
  __syncthreads();
  TileBox box;
#pragma unroll
  for (int q = 0; q < 4; q++) {
    box.lo[q] = red[q];
    box.hi[q] = red[4 + q];
  }
  for (int w = 1; w < nwarps; w++)
#pragma unroll
    for (int q = 0; q < 4; q++) {
      box.lo[q] = fmin(box.lo[q], red[w * 8 + q]);
      box.hi[q] = fmax(box.hi[q], red[w * 8 + 4 + q]);
    }
  int bad = !(P.Fs > 0.0), extA = 0, extB = 0, loA = INT_MAX, hiA = INT_MIN, loB = INT_MAX, hiB = INT_MIN;
  for (int e = tid; e < n_out + n_in; e += nthr) {
    const bool outer = e < n_out;
    const int el = outer ? e : e - n_out;
    int b = 0, t = 0;
    if (outer || (el >= i_lo && el < i_hi)) {
      double Lmin, Lmax;
      leg_range(P, box, outer, el, Lmin, Lmax);
      if (Lmin > -LEG_LIMIT && Lmax < LEG_LIMIT && Lmin <= Lmax) {
        b = ((int)floor(Lmin) - 1) & ~3;  // a multiple of 4: windows start 16-byte aligned
        t = (int)floor(Lmax) + 1;
      } else {
        bad = 1;
      }
      if (outer) {
        extA = max(extA, t - b);
        loA = min(loA, b);
        hiA = max(hiA, t);
      } else {
        extB = max(extB, t - b);
        loB = min(loB, b);
        hiB = max(hiB, t);
      }
    }
    T.be[e] = make_int2(b, t - b);
  }
  bad = __reduce_or_sync(0xffffffffu, bad);
  extA = __reduce_max_sync(0xffffffffu, extA);
  extB = __reduce_max_sync(0xffffffffu, extB);
  loA = __reduce_min_sync(0xffffffffu, loA);
  hiA = __reduce_max_sync(0xffffffffu, hiA);
  loB = __reduce_min_sync(0xffffffffu, loB);
  hiB = __reduce_max_sync(0xffffffffu, hiB);
  int x_mx = __reduce_max_sync(0xffffffffu, __float_as_int(fabsf(xn)));  // bits: in the values' order, NaN above all
  if (WEIGHTED) w_mx = __reduce_max_sync(0xffffffffu, w_mx);
  if (lane == 0) {
    int *s = stat + warp * STAT;
    s[0] = bad, s[1] = extA, s[2] = extB, s[3] = loA, s[4] = hiA, s[5] = loB, s[6] = hiB, s[7] = x_mx;
    if (WEIGHTED) s[8] = w_mx;
  }
  __syncthreads();
  for (int w = 0; w < nwarps; w++) {
    const int *s = stat + w * STAT;
    bad |= s[0];
    extA = max(extA, s[1]);
    extB = max(extB, s[2]);
    loA = min(loA, s[3]);
    hiA = max(hiA, s[4]);
    loB = min(loB, s[5]);
    hiB = max(hiB, s[6]);
    x_mx = max(x_mx, s[7]);
    if (WEIGHTED) w_mx = max(w_mx, s[8]);
  }
  __syncthreads();  // the scratch is read
  T.usable = !bad && loA <= hiA && loB <= hiB;
  T.low = (int64_t)loA + loB < 0;
  T.in_bounds = !T.low && (int64_t)hiA + hiB + 2 < P.K;
  T.ext_outer = extA;
  T.ext_inner = extB;
  T.x_max = __int_as_float(x_mx);
  T.w_max = __int_as_float(w_mx);
  T.x_scales = T.x_max >= SCATTER_X_MIN && T.x_max < INFINITY;
}

// Whether a leg (ms) lies inside its window range (bases and extents leave a
// sample on each side), so that the sum of two such legs, whatever its
// rounding, falls on a cell of the row.
__device__ __forceinline__ bool leg_inside(double l, double Fs, int2 be) {
  const double t = l * Fs - (double)be.x;
  return t >= 0.5 && t < (double)be.y + 0.5;
}

// The windows hold fixed-point integers, x scaled by 2^(22 - E) with max |x|
// over the tile below 2^E, so the shared-memory additions are native integer
// atomics, exact and independent of their order (a slot receives at most one
// term per thread per batch, at most 256 terms of magnitude up to 2^22); each
// value is rounded once, to within 2^-22 of the tile's largest |x|. Every leg
// inside its bound puts its terms on cells of the row, so the adds need no guard;
// the flush drops the cells outside the A-scan. Only where times may be negative
// are terms tested one by one (p in (-1, 0) belongs to sample 0, p = -1 does not).
template <bool WEIGHTED, int METHOD>
__device__ __forceinline__ void scatter_windows(const FastParams &P, const ScatterTile &T, const Pixel &px, bool active,
                                                float xn_f, float *Ya, int *win, double *legs, int n_out, int n_in,
                                                int i_lo, int i_hi) {
  constexpr int JC = SCATTER_JC, NO = SCATTER_NO, ROWS = SCATTER_ROWS;
  const int tid = threadIdx.x, nthr = blockDim.x;
  const int64_t K = P.K;
  const int WS = (T.ext_outer + T.ext_inner + 4 + 3) & ~3;  // window samples per row
  const Legs<METHOD, true> outer(P);
  const Legs<METHOD, false> inner(P);
  const double Fs = P.Fs, Kf = (double)K;
  bool vectors = (K & 3) == 0 && (reinterpret_cast<uintptr_t>(Ya) & 15) == 0;  // rows start on 16 bytes
  double *tab = legs + tid;  // leg of outer element o0 + o: tab[o * nthr]
  for (int e = tid; e < 2 * ROWS * WS; e += nthr) win[e] = 0;
  __syncthreads();
  // fixed-point scale of the tile: max |x| < 2^E, values scaled by 2^(22 - E)
  int E;
  frexpf(T.x_max, &E);
  const float qscale = ldexpf(1.0f, 22 - E), iS = ldexpf(1.0f, E - 22);
  const int xn = __float2int_rn(xn_f * qscale);
  // A row flushed in vectors adds 0 * (scale * weight) to its cells without a term: only where that is 0.
  if (WEIGHTED) vectors = vectors && isfinite(iS * T.w_max);
  // flush: a fixed group of nthr / ROWS threads per window row (q, j)
  const int tpr = nthr / ROWS, fr = tid / tpr, fq = tid - fr * tpr, fro = fr / JC, fri = fr % JC;
  const int64_t ostride = P.ycol_o > 0 ? P.ycol_o : n_in;  // columns per outer element
  const int64_t ystep = SCATTER_NO * ostride * K;
  const uint32_t win_a = (uint32_t)__cvta_generic_to_shared(win);
  uint32_t buf = 0;  // byte offset of the batch's buffer
  for (int o0 = 0; o0 < n_out; o0 += P.out_block) {
    const int on = min(P.out_block, n_out - o0);
    bool bad = false;
#pragma unroll 4
    for (int o = 0; o < on; o++) {
      const double l = outer(P, px, o0 + o);
      bad = bad || !leg_inside(l, Fs, T.be[o0 + o]);
      tab[o * nthr] = l;
    }
    const bool outer_bad = __syncthreads_or(bad) != 0;
    for (int i0 = i_lo; i0 < i_hi; i0 += JC) {
      const int jn = min(JC, i_hi - i0);
      double B[JC], mag[JC];
      bad = false;
#pragma unroll
      for (int j = 0; j < JC; j++) {
        if (j >= jn) {  // past the last inner element: never added
          B[j] = B[0];
          mag[j] = mag[0];
          continue;
        }
        const int2 be = T.be[n_out + i0 + j];
        B[j] = inner(P, px, i0 + j);
        bad = bad || !leg_inside(B[j], Fs, be);
        mag[j] = 6755399441055744.0 + (double)(j * WS - be.x);  // 1.5 * 2^52: row j, less the inner base
      }
      if (__syncthreads_or(bad) || outer_bad) {
        // a leg outside the tile's bound (not expected): straight to Ya
        const Pixel c = px;  // a copy for the call by reference: px stays in registers
        if (active)
          for (int o = 0; o < on; o++) exact_scatter<WEIGHTED>(P, c, o0 + o, i0, jn, n_in, xn_f, Ya);
        continue;
      }
      // this thread's flush row: the inner element's column, base and extent
      const bool my_row = fri < jn;
      const int col_r = i0 + (my_row ? fri : 0);
      const int2 be_r = T.be[n_out + col_r];
      const int64_t fcol = (o0 + fro) * ostride + ycol_inner(P, col_r);
      float *yrow = Ya + fcol * K + be_r.x;
      const float *wrow = WEIGHTED ? P.w + fcol : nullptr;
      float w_next = WEIGHTED && my_row && fro < on ? __ldg(wrow) : 0.0f;  // read a batch ahead
      for (int o = 0; o < on; o += NO, yrow += ystep) {
        const bool flush = my_row && o + fro < on;
        const float sc = WEIGHTED ? iS * w_next : iS;  // a power of two: the weight's product rounds once either way
        if (WEIGHTED && my_row && o + NO + fro < on) w_next = __ldg(wrow += NO * ostride);
        const int2 be_o = T.be[o0 + (flush ? o + fro : o)];
        if (!T.low && jn == JC && o + NO <= on) {
          uint32_t cell[NO][JC];
#pragma unroll
          for (int q = 0; q < NO; q++) {
            const double a = tab[(o + q) * nthr];
            const uint32_t row = win_a + buf + (uint32_t)(q * JC * WS - T.be[o0 + o + q].x) * 4u;
#pragma unroll
            for (int j = 0; j < JC; j++)
              cell[q][j] = row + 4u * (uint32_t)__double2loint(__dadd_rz(__dmul_rn(__dadd_rn(a, B[j]), Fs), mag[j]));
          }
#pragma unroll
          for (int q = 0; q < NO; q++)
#pragma unroll
            for (int j = 0; j < JC; j++) red_add_shared(cell[q][j], xn);
        } else {
#pragma unroll
          for (int q = 0; q < NO; q++) {
            if (o + q >= on) break;
            const double a = tab[(o + q) * nthr];
            const uint32_t row = win_a + buf + (uint32_t)(q * JC * WS - T.be[o0 + o + q].x) * 4u;
#pragma unroll
            for (int j = 0; j < JC; j++) {
              const double p = __dmul_rn(__dadd_rn(a, B[j]), Fs);
              if (j < jn && p > -1.0) red_add_shared(row + 4u * (uint32_t)__double2loint(__dadd_rz(p, mag[j])), xn);
            }
          }
        }
        __syncthreads();
        // samples kb + t of the row; its terms lie in the first ext_o + ext_i + 3 cells
        const int wr = flush ? be_o.y + be_r.y + 4 : 0;
        const int64_t kb = (int64_t)be_o.x + be_r.x;  // a multiple of 4
        if (vectors && kb >= 0 && kb + ((wr + 3) & ~3) <= K) {
          int4 *wp = reinterpret_cast<int4 *>(reinterpret_cast<char *>(win) + buf) + (fr * WS >> 2) + fq;
          float *y = yrow + be_o.x + fq * 4;
          for (int t = fq * 4; t < wr; t += tpr * 4, wp += tpr, y += tpr * 4) {
            const int4 vi = *wp;
            *wp = make_int4(0, 0, 0, 0);
            red_add_v4(y, make_float4((float)vi.x * sc, (float)vi.y * sc, (float)vi.z * sc, (float)vi.w * sc));
          }
        } else {
          int *cells = win + buf / 4 + fr * WS;
          for (int t = fq; t < wr; t += tpr) {
            const int vi = cells[t];
            if (vi != 0) {
              cells[t] = 0;
              int64_t k = kb + t;
              if (k == -1) k = 0;  // p in (-1, 0): sample 0 after truncation toward zero
              if (k >= 0 && k < K) atomicAdd(yrow + (k - be_r.x), (float)vi * sc);
            }
          }
        }
        buf ^= (uint32_t)(ROWS * WS) * 4u;
      }
    }
  }
}

struct TileShape {
  int tile_f, tile_s;
};

// Whether a TFM grid's 256-point tiles are 16 x 16 rather than 8 deep and 32 wide.
// A leg spans at most the tile's diagonal, and windows beyond their capacity cost
// two to three times as much: the shorter diagonal, 16 x 16 where lines are further
// apart than half the spacing in depth. 64x64 elements, 1024 lines 0.03 mm apart of
// 40 points 0.64 mm apart: 8 x 32 0.30 ms, 16 x 16 0.82; 37x53 elements, 301 lines
// of 203 points 0.13 and 0.18 mm apart 0.46 and 0.33; 512x512 points 0.79 and 0.82.
// The first points decide, alike in every block.
__device__ __forceinline__ bool square_tile(const FastParams &P) {
  const double *R = P.Ro + (P.n_slow > 1 ? P.n_fast : 0);
  const double x = R[0] - P.Ro[0], y = R[P.No] - P.Ro[P.No], z = R[2 * P.No] - P.Ro[2 * P.No];
  const double d = P.Ro[2 * P.No + 1] - P.Ro[2 * P.No];
  return !(d * d > 4.0 * (x * x + y * y + z * z));
}

template <bool WEIGHTED, int METHOD>
__global__ void __launch_bounds__(256, 2) das_scatter_kernel(const FastParams P, bool square,
                                                             const float *__restrict__ X, float *__restrict__ Ya) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int n_out = METHOD == RCA_ROWTX ? P.Nr : P.Nt, n_in = METHOD == RCA_ROWTX ? P.Nt : P.Nr;
  const int i_lo = P.in_lo, i_hi = P.in_hi > 0 ? P.in_hi : n_in;
  int *win = reinterpret_cast<int *>(smem_raw + scatter_head_bytes(n_out, n_in));
  double *legs = reinterpret_cast<double *>(smem_raw + scatter_head_bytes(n_out, n_in) + SCATTER_WIN_BYTES);
  int w_mx = 0;  // bits of the largest |weight| that this thread reads; here, beside the reads that place the tile
  if (WEIGHTED) {
    const int64_t columns = n_out * (int64_t)(P.ycol_o > 0 ? P.ycol_o : n_in);
#pragma unroll 8
    for (int64_t c = threadIdx.x; c < columns; c += blockDim.x) w_mx = max(w_mx, __float_as_int(fabsf(__ldg(P.w + c))));
  }
  bool active;
  const uint32_t row = volume_tiles<METHOD>(P) ? volume_row(P.Ro, P.No, P.n_fast, P.n_slow) : 0;
  TileShape tile = {P.tile_f, P.tile_s};
  int64_t tfi = blockIdx.x, tsi = (int64_t)blockIdx.y + P.slow_tile0;
  if (METHOD == TFM && square) {  // a launch row holds 32 lines: the blocks of one row of 8 x 32, or two of 16 x 16
    if (square_tile(P)) {
      const int64_t cols = (P.n_fast + 15) / 16, lower = tfi >= cols;
      tile.tile_f = tile.tile_s = 16;
      tsi = 2 * tsi + lower;
      tfi -= lower * cols;
    }
    if (tfi * tile.tile_f >= P.n_fast || tsi * tile.tile_s >= P.n_slow) return;
  }
  const int64_t no = tile_point(P, tile, tfi, tsi, row, active);
  Pixel px;
  pixel_of(P, no, px);
  const float xn = active ? __ldg(X + no) : 0.0f;
  ScatterTile T;
  scatter_setup<WEIGHTED>(P, px, xn, w_mx, smem_raw, reinterpret_cast<double *>(win), n_out, n_in, i_lo, i_hi, T);
  if (T.usable && T.ext_outer + T.ext_inner + 7 <= SCATTER_WCAP && (T.x_max == 0.0f || T.x_scales)) {
    if (T.x_max > 0.0f)
      scatter_windows<WEIGHTED, METHOD>(P, T, px, active, xn, Ya, win, legs, n_out, n_in, i_lo, i_hi);
    return;
  }
  // windows wider than the shared-memory rows, legs outside the integer range, or values outside the windows'
  // fixed-point range: every term added on its own
  if (!active) return;
  const Legs<METHOD, true> outer(P);
  const Legs<METHOD, false> inner(P);
  const int64_t ostride = P.ycol_o > 0 ? P.ycol_o : n_in;
  const double Kf = (double)P.K;
  double *tab = legs + threadIdx.x;
  // Terms without a test: sample numbers of a chunk fit 32 bits, the tile's leg ranges lie inside the A-scan, and this
  // point's own legs inside those ranges (a NaN point's are not, and the box of the tile's points does not show it).
  const bool plain = T.usable && T.in_bounds && P.K < (int64_t(1) << 28);
  for (int o0 = 0; o0 < n_out; o0 += P.out_block) {
    const int on = min(P.out_block, n_out - o0);
    bool outer_in = plain;
    for (int o = 0; o < on; o++) {
      const double l = outer(P, px, o0 + o);
      outer_in = outer_in && leg_inside(l, P.Fs, T.be[o0 + o]);
      tab[o * blockDim.x] = l;
    }
    for (int i0 = i_lo; i0 < i_hi; i0 += SCATTER_JC) {
      const int jn = min(SCATTER_JC, i_hi - i0);
      double B[SCATTER_JC];
      bool in = outer_in && jn == SCATTER_JC;
#pragma unroll
      for (int j = 0; j < SCATTER_JC; j++) {
        B[j] = j < jn ? inner(P, px, i0 + j) : 0.0;
        in = in && leg_inside(B[j], P.Fs, T.be[n_out + (j < jn ? i0 + j : i0)]);
      }
      for (int o = 0; o < on; o++) {
        const double a = tab[o * blockDim.x];
        const int64_t col = (o0 + o) * ostride + ycol_inner(P, i0);
        float *y = Ya + col * P.K;
        if (in) {
#pragma unroll
          for (int j = 0; j < SCATTER_JC; j++) {
            const double p = __dmul_rn(__dadd_rn(a, B[j]), P.Fs);
            const uint32_t k = (uint32_t)__double2loint(__dadd_rz(p, 4503599627370496.0 + (double)(j * P.K)));
            red_add(elem_addr<float>(reinterpret_cast<const char *>(y), k), WEIGHTED ? __ldg(P.w + col + j) * xn : xn);
          }
        } else {
#pragma unroll
          for (int j = 0; j < SCATTER_JC; j++) {
            const double p = __dmul_rn(__dadd_rn(a, B[j]), P.Fs);
            if (j < jn && p > -1.0 && p < Kf)
              atomicAdd(y + j * P.K + trunc_index(p), WEIGHTED ? __ldg(P.w + col + j) * xn : xn);
          }
        }
      }
    }
  }
}

}  // namespace

// Tile scatter over the slow-tile range of P (P.w optional). Ya is not zeroed here.
cudaError_t launch_scatter(const FastParams &P0, bool square, const float *X, float *Ya, cudaStream_t st) {
  FastParams P = P0;
  const int nthr = P.tile_f * P.tile_s;
  const int n_out = P.method == RCA_ROWTX ? P.Nr : P.Nt, n_in = P.method == RCA_ROWTX ? P.Nt : P.Nr;
  // even blocks of at most 40 outer elements, fewer where thousands of elements' bounds take the space
  const size_t fixed = scatter_head_bytes(n_out, n_in) + SCATTER_WIN_BYTES;
  const int64_t room = ((int64_t)220 * 1024 - (int64_t)fixed) / (int64_t)(nthr * sizeof(double));
  const int most = (int)std::max<int64_t>(2, std::min<int64_t>(40, room));
  const int blocks = (n_out + most - 1) / most;
  P.out_block = std::min(most, ((n_out + blocks - 1) / blocks + 1) & ~1);
  const size_t smem = fixed + std::max<size_t>((size_t)P.out_block * nthr * sizeof(double), 1024);
#define SCATTER_KERNEL(W)                                         \
  (P.method == TFM         ? das_scatter_kernel<W, TFM>           \
   : P.method == RCA_COLTX ? das_scatter_kernel<W, RCA_COLTX>     \
                           : das_scatter_kernel<W, RCA_ROWTX>)
  auto kern = P.w ? SCATTER_KERNEL(true) : SCATTER_KERNEL(false);
#undef SCATTER_KERNEL
  cudaError_t e = ensure_smem(kern, smem);
  if (e != cudaSuccess) return e;
  const int64_t gx = square ? (P.n_fast + 15) / 16 * 2 : (P.n_fast + P.tile_f - 1) / P.tile_f;  // square: of either tile
  const int64_t gy = P.slow_tile1 - P.slow_tile0;
  if (gx <= 0 || gy <= 0) return cudaSuccess;
  kern<<<dim3((unsigned)gx, (unsigned)gy), nthr, smem, st>>>(P, square, X, Ya);
  return cudaGetLastError();
}

// Column pass after an unweighted scatter S = DAS^T g: dW[c] = sum_k Y[k, c] *
// S[k, c] (the weight gradient: each term g[n] * Y[k(n,c), c] regrouped by
// sample), and, when w is given, S[:, c] *= w[c] in place (the weighted
// adjoint). One CTA per column; columns are K apart in both arrays.
__global__ void __launch_bounds__(256) column_dot_scale_kernel(const float *__restrict__ Y, float *__restrict__ S,
                                                               const float *__restrict__ w, float *__restrict__ dW,
                                                               int64_t K) {
  const int64_t c = blockIdx.x;
  const float *y = Y ? Y + c * K : nullptr;
  float *sc = S + c * K;
  const float wc = w ? __ldg(w + c) : 1.0f;
  float acc = 0.0f;
  for (int64_t k = threadIdx.x; k < K; k += blockDim.x) {
    const float v = sc[k];
    if (y) acc = fmaf(__ldg(y + k), v, acc);
    if (w) sc[k] = v * wc;
  }
  if (dW == nullptr) return;
  __shared__ float red[8];
  for (int off = 16; off > 0; off >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, off);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = acc;
  __syncthreads();
  if (threadIdx.x == 0) {
    float t = 0.0f;
    for (int q = 0; q < (int)(blockDim.x >> 5); q++) t += red[q];
    dW[c] = t;
  }
}

cudaError_t launch_column_dot_scale(const float *Y, float *S, const float *w, float *dW, int64_t K, int64_t ncol,
                                    cudaStream_t st) {
  if (ncol <= 0 || (K <= 0 && dW == nullptr)) return cudaSuccess;
  for (int64_t c0 = 0; c0 < ncol; c0 += 2147483647) {
    const int64_t n = std::min<int64_t>(ncol - c0, 2147483647);
    column_dot_scale_kernel<<<(unsigned)n, 256, 0, st>>>(Y ? Y + c0 * K : nullptr, S + c0 * K, w ? w + c0 : nullptr,
                                                         dW ? dW + c0 : nullptr, K);
  }
  return cudaGetLastError();
}

}  // namespace dream
