// dreamrect.cu -- spatial impulse responses (SIR) of a rectangular
// transducer and of arrays of rectangular elements on the GPU: DREAM's
// dreamrect (src/dreamrect.cc:248-302, opencl/dreamrect.cl) and
// dream_arr_rect (src/dream_arr_rect.cc:192-244, src/arr_functions.cc)
// without attenuation, the models that produce the responses from which
// A-scans are synthesised.
//
// Array element m (one for dreamrect, at the origin) sees observation point
// n at Ro[n] - G[m] with the delay (delay - foc_m) - steer_m. Its
// a x b aperture is cut into dx x dy surface elements whose centres advance
// by repeated addition (ys += dy outer, xs += dx inner). Surface element e
// contributes
//   ai = (((w_m*v)*ds)/(2*pi*r)) / dt * 1000   to sample   it = rint((t - delay_m)/dt),
// t = (r*1000)/cp, r its distance to the point, and h[it] += ai in (m, e)
// order. Centres, focusing / steering delays and weights are computed on the
// host with the reference's own operations (libm for sin, cos, exp); every
// device operation is the correctly rounded IEEE one, unfused.
//
// Layout. One warp per observation point. An array element's terms lie
// between the travel times to the nearest and the farthest point of its
// rectangle (+-2 samples for the rounding of r and t); an element whose
// window misses [0, nt) has no in-bounds term and is skipped (its terms are
// counted out of bounds without being evaluated). The union of the live
// elements' windows sits in shared memory (sized on the host by the
// diameter of the array and the spread of its delays, up to 8 warps per
// CTA); longer windows are accumulated in the output column itself. The warp
// takes 32 consecutive terms of one live element per step (of several, where
// elements have few: packed_terms): lanes that hit
// the same sample are grouped (__match_any_sync) and the lowest lane of each
// group adds the group's amplitudes in lane order (as many shuffle steps as
// the largest group has members), so every sample receives its terms in the
// reference's order and the SIR equals the reference's bit for bit. Windows
// are only trusted where the rounding bound holds (sample magnitudes below
// 2^36); a term that still lands in [0, nt) outside its point's window is
// counted, and the launch is then repeated with every element live and
// every window [0, nt). Large fields of a single element take one point per
// lane instead (rect_lane_kernel).
#include <cuda_runtime.h>
#include <stdint.h>

#include <algorithm>
#include <cmath>
#include <mutex>
#include <string>
#include <vector>

#include "das_common.cuh"
#include "das_kernels.h"
#include "dream_sir.h"

namespace dream {
namespace {

constexpr double RECT_TWO_PI = 2 * 3.14159265358979323846;  // 2*M_PI as the reference evaluates it
constexpr int RECT_WARPS = 8;                     // observation points per CTA
constexpr int64_t RECT_SMEM_MAX = 192 * 1024;     // shared memory for the CTA's SIR windows
constexpr double RECT_WIN_TRUST = 68719476736.0;  // 2^36: sample magnitudes whose +-2 window margin is proven
// A sample-index estimate farther than this from a half-integer rounds like
// the exact chain: with sample magnitudes below RECT_WIN_TRUST the two differ
// by at most 10 * 2^-53 * 2^36 < 2^-13 samples.
constexpr double RECT_Q_SAFE = 0.5 - 1.0 / 1024.0;
constexpr unsigned RECT_MISS = 1u;      // a term fell in [0, nt) outside its point's window
constexpr unsigned RECT_LAST_OOB = 2u;  // a term of the array's last element was out of bounds

// One array element: centre, focusing and steering delays (us) and
// (weight*v)*ds, the numerator of its terms.
struct ArrElem {
  double gx, gy, gz, foc, steer, wvds;
};

struct RectParams {
  const double *Ro;
  int64_t No;
  const double *xs, *ys;  // surface-element centres (nx, ny)
  int nx, ny;
  const ArrElem *el;      // array elements (M)
  int64_t M;
  double dt, cp;
  double c1, inv_dt;      // 1000/cp and 1/dt, for the sample-index estimate
  double k1;              // c1 * inv_dt
  int plain_range;        // dt and cp lie where the branch-free operations below hold
  int row_steps;          // steps of 32 terms end with the rows
  double ab;              // |a| + |b|
  double half_a, half_b;  // a/2, b/2
  int64_t win;            // samples of a point's SIR window in shared memory (0: none)
  int64_t nt;
  const double *delay;
  int delay_multi;
  int full;               // every element live, windows [0, nt) in the output columns
  int64_t *rest;          // points whose window one lane has no room for (in any order), and their number; rect_kernel
  int64_t n_rest;         // takes these instead of all points when n_rest > 0
  double *H;
  unsigned long long *oob;        // out-of-bounds terms
  unsigned int *flags;            // RECT_MISS | RECT_LAST_OOB
  unsigned long long *rest_count;
};

// The observation point as array element m sees it; `fast`: its sample
// magnitudes are below RECT_WIN_TRUST (windows and index estimates hold).
struct ElemView {
  double xo, yo, zo, rz2, dl, w, bound;
  bool fast;
};

// Point n (reloaded from global memory: kept out of the term loop's registers).
__device__ __forceinline__ void elem_view(const RectParams &P, int64_t m, int64_t n, ElemView &V) {
  const double xo = __ldg(P.Ro + n), yo = __ldg(P.Ro + n + P.No), zo = __ldg(P.Ro + n + 2 * P.No);
  const double dlay = __ldg(P.delay + (P.delay_multi ? n : 0));
  const ArrElem *E = P.el + m;
  V.xo = __dsub_rn(xo, __ldg(&E->gx));
  V.yo = __dsub_rn(yo, __ldg(&E->gy));
  V.zo = __dsub_rn(zo, __ldg(&E->gz));
  V.rz2 = __dmul_rn(V.zo, V.zo);
  V.dl = __dsub_rn(__dsub_rn(dlay, __ldg(&E->foc)), __ldg(&E->steer));
  V.w = __ldg(&E->wvds);
  V.bound = ((fabs(V.xo) + fabs(V.yo) + fabs(V.zo) + P.ab) * fabs(P.c1) + fabs(V.dl)) * fabs(P.inv_dt);
  V.fast = !P.full && V.bound < RECT_WIN_TRUST;
}

// Sample index of a term at distance r, as the kernel computes it.
__device__ __forceinline__ double rect_q(double r, double dl, const RectParams &P) {
  const double t = __ddiv_rn(__dmul_rn(r, 1000.0), P.cp);
  return __ddiv_rn(__dsub_rn(t, dl), P.dt);
}

// Live test and sample window [lo, hi) of an element's terms: every surface
// element centre lies in the a x b rectangle, so r is between the distances
// to its nearest point and to its farthest corner. Unbounded where the
// margin is not proven (or in the repeated launch).
__device__ __forceinline__ bool elem_window(const RectParams &P, const ElemView &V, int64_t &lo, int64_t &hi) {
  const double ax = fabs(V.xo), ay = fabs(V.yo);
  const double ex = fmax(ax - P.half_a, 0.0), ey = fmax(ay - P.half_b, 0.0);
  const double fx = ax + P.half_a, fy = ay + P.half_b;
  if (!V.fast) {
    lo = 0;
    hi = P.nt;
    return true;
  }
  // sample estimates (within 2^-13 of the exact chain's, see RECT_Q_SAFE)
  const double qa = (sqrt(ex * ex + ey * ey + V.rz2) * P.c1 - V.dl) * P.inv_dt;
  const double qb = (sqrt(fx * fx + fy * fy + V.rz2) * P.c1 - V.dl) * P.inv_dt;
  const int64_t sa = __double2ll_rn(qa), sb = __double2ll_rn(qb);
  lo = min(sa, sb) - 2;
  hi = max(sa, sb) + 3;
  return lo < P.nt && hi > 0;
}

// ---------------------------------------------------------------------------
// Branch-free correctly rounded root and quotients, so that several terms' chains
// run side by side (the IEEE intrinsics branch to a slow path each): Newton steps
// from a 2^-20 reciprocal root and Markstein's final corrections by the exact FMA
// residual (P. Markstein, "Computation of elementary functions on the IBM RISC
// System/6000 processor", 1990; "IA-64 and Elementary Functions", 2000). They
// differed from the IEEE operations in none of 1.2e10 samples, half of them next
// to rounding boundaries; the tests repeat 2.4e6 of them through SIRs of a
// single amplitude. term_plain tells where they hold.
// ---------------------------------------------------------------------------

constexpr int RECT_FB = 14;                          // fraction bits of the sample number in the low mantissa word
constexpr double RECT_MAGIC = 1.5 * 274877906944.0;  // 1.5 * 2^(52 - RECT_FB)
constexpr double RECT_PLAIN_MAX = 65536.0;           // sample magnitudes for which it fits there
constexpr double RECT_MIN_S = 0x1p-120, RECT_MIN_W = 0x1p-300, RECT_MAX_W = 0x1p300;

// Root of s, correctly rounded, and h = 1 / (2 root) to within an ulp or two;
// s in [2^-120, 2^500].
__device__ __forceinline__ double rect_root(double s, double &h) {
  double y;
  asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(s));
  double g = __dmul_rn(s, y);
  h = __dmul_rn(y, 0.5);
  const double e = __fma_rn(-g, h, 0.5);  // 1/sqrt(1 - 2e) = 1 + e + 3/2 e^2 + O(e^3), e < 2^-19
  const double c = __dmul_rn(e, __fma_rn(e, 1.5, 1.0));
  g = __fma_rn(g, c, g);
  h = __fma_rn(h, c, h);
  return __fma_rn(__fma_rn(-g, g, s), h, g);
}
// a / b correctly rounded, y0 = 1 / b to within a few ulp.
__device__ __forceinline__ double rect_quot(double a, double b, double y0) {
  const double y = __fma_rn(y0, __fma_rn(-b, y0, 1.0), y0);
  const double q = __dmul_rn(a, y);
  return __fma_rn(__fma_rn(-q, b, a), y, q);
}
// a / b correctly rounded, y = RN(1 / b).
__device__ __forceinline__ double rect_quot_by(double a, double b, double y) {
  const double q = __dmul_rn(a, y);
  return __fma_rn(__fma_rn(-q, b, a), y, q);
}
// Amplitude of a term at distance r, h = 1 / (2 r).
__device__ __forceinline__ double rect_amplitude(const RectParams &P, double w, double r, double h) {
  const double q = rect_quot(w, __dmul_rn(RECT_TWO_PI, r), __dmul_rn(h, 0.31830988618379067));  // 1/(2 pi r) = h / pi
  return __dmul_rn(rect_quot_by(q, P.dt, P.inv_dt), 1000.0);
}
// Sample number of a term at distance r in units of 2^-RECT_FB, plus one half: c0 = fma(-dl, inv_dt, RECT_MAGIC).
// Two roundings to 2^-15 and less than 2^-34 in the constants separate it from the exact chain's, so it rounds like
// the chain unless its fraction lies within 3 units of an integer (rect_near).
__device__ __forceinline__ int rect_number(const RectParams &P, double r, double c0) {
  return __double2loint(__fma_rn(r, P.k1, c0)) + (1 << (RECT_FB - 1));
}
__device__ __forceinline__ bool rect_near(int q) {
  return (unsigned int)((q & ((1 << RECT_FB) - 1)) - 3) > (1u << RECT_FB) - 7u;
}
// Whether every operand of element V's terms lies where these hold (the nearest
// point of the element's rectangle bounds s from below).
__device__ __forceinline__ bool term_plain(const RectParams &P, const ElemView &V) {
  const double ex = fmax(fabs(V.xo) - P.half_a, 0.0), ey = fmax(fabs(V.yo) - P.half_b, 0.0);
  const double w = fabs(V.w);
  return P.plain_range && V.fast && V.bound < RECT_PLAIN_MAX && ex * ex + ey * ey + V.rz2 >= RECT_MIN_S &&
         (w == 0.0 || (w > RECT_MIN_W && w < RECT_MAX_W));
}

__device__ __forceinline__ unsigned long long warp_sum_u64(unsigned long long v) {
  for (int o = 16; o; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// Adds this step's amplitudes in lane order, lanes with the same key (a sample
// number whose top bit is clear) into the same sample *h.
template <class Key>
__device__ __forceinline__ void ordered_adds(bool in, Key key, double ai, double *h, int lane, double *stage) {
  // lanes adding into the same sample form a group; the others get unique keys
  const unsigned int group = __match_any_sync(0xffffffffu, in ? key : ~(Key)lane);
  const int len = __popc(group);
  const bool leader = in && (group & ((1u << lane) - 1u)) == 0u;  // lowest lane of its group
  // a run: the group's lanes are lane .. lane + len - 1
  const bool run = (group >> lane) == (len == 32 ? 0xffffffffu : (1u << len) - 1u);
  if (__all_sync(0xffffffffu, !leader || run)) {
    stage[lane] = ai;
    __syncwarp();
    if (leader) {
      double acc = __dadd_rn(*h, ai);
      const double *q = stage + lane + 1;
      int k = len - 1;
      for (; k >= 8; k -= 8, q += 8) {
#pragma unroll
        for (int u = 0; u < 8; u++) acc = __dadd_rn(acc, q[u]);
      }
#pragma unroll
      for (int u = 0; u < 7; u++)
        if (u < k) acc = __dadd_rn(acc, q[u]);
      *h = acc;
    }
  } else {
    // each leader walks its group's lanes in ascending order (its own first);
    // the warp takes as many steps as the largest group has members
    const unsigned int steps = __reduce_max_sync(0xffffffffu, leader ? (unsigned)len : 0u);
    double acc = leader ? *h : 0.0;
    unsigned int rem = leader ? group : 0u;
    for (unsigned int k = 0; k < steps; k++) {
      const int src = rem ? __ffs(rem) - 1 : lane;
      const bool add = rem != 0u;
      rem &= rem - 1u;
      const double aj = __shfl_sync(0xffffffffu, ai, src);
      if (add) acc = __dadd_rn(acc, aj);
    }
    if (leader) *h = acc;
  }
  __syncwarp();  // this step's sums (and stage reads) complete before the next step
}

// One warp step: lane's term (if valid) at surface element (ix, iy) of the
// element V is added to its sample, every sample receiving its terms in lane
// order. Lanes that hit the same sample are grouped (__match_any_sync); the
// lowest lane of each group adds the group's amplitudes in lane order. When
// every group is a run of consecutive lanes (the common case: along a row
// the sample index changes monotonically on either side of the point's
// projection) the leaders read their run from the warp's 32 staged
// amplitudes, eight per trip; otherwise they walk their member masks.
// SKIP: steps with no term in the SIR skip the amplitudes and the sums (arrays,
// whose live elements still place most terms outside short windows); without
// it the amplitude divisions overlap the index computation.
template <bool SKIP>
__device__ __forceinline__ void term_step(const RectParams &P, const ElemView &V, bool valid, int ix, int iy,
                                          int lane, int64_t w0, int64_t w1, double *h, double *stage,
                                          unsigned long long &oob, unsigned int &flags, bool last) {
  bool in = false;
  int64_t it = 0;
  double r = 1.0;  // idle lanes: a finite amplitude that is never added
  double ai = 0.0;
  if (valid) {
    const double rx = __dsub_rn(V.xo, __ldg(P.xs + ix));
    const double ry = __dsub_rn(V.yo, __ldg(P.ys + iy));
    r = __dsqrt_rn(__dadd_rn(__dadd_rn(__dmul_rn(rx, rx), __dmul_rn(ry, ry)), V.rz2));
    if (!SKIP) {
      ai = __ddiv_rn(V.w, __dmul_rn(RECT_TWO_PI, r));
      ai = __ddiv_rn(ai, P.dt);
      ai = __dmul_rn(ai, 1000.0);
    }
    // rint((t - dl)/dt), ties to even: the estimate where it is certain, else the exact chain
    const double qa = __dmul_rn(__dsub_rn(__dmul_rn(r, P.c1), V.dl), P.inv_dt);
    const double na = rint(qa);
    if (V.fast && fabs(qa - na) < RECT_Q_SAFE)
      it = (int64_t)na;
    else
      it = __double2ll_rn(rect_q(r, V.dl, P));
    in = it >= 0 && it < P.nt;
    oob += in ? 0u : 1u;
    if (!in && last) flags |= RECT_LAST_OOB;
    const bool inside = it >= w0 && it < w1;  // true whenever the window bound holds
    if (in && !inside) flags |= RECT_MISS;
    in = in && inside;
  }
  if (SKIP) {
    if (!__any_sync(0xffffffffu, in)) return;  // no term of this step lands in the SIR
    ai = __ddiv_rn(V.w, __dmul_rn(RECT_TWO_PI, r));
    ai = __ddiv_rn(ai, P.dt);
    ai = __dmul_rn(ai, 1000.0);
  }
  ordered_adds(in, (unsigned long long)it, ai, h + it, lane, stage);
}

// The same step for an element that is term_plain, at a surface element whose
// centre differs by rx from the point in x and by ry2 squared in y; c0 as for
// rect_number. hits counts the terms added (the others are out of bounds; `last`:
// flagged as such, a term of the array's last element).
template <bool SKIP>
__device__ __forceinline__ void plain_step(const RectParams &P, const ElemView &V, double c0, bool valid, double rx,
                                           double ry2, int lane, int w0, int wn, double *h, double *stage,
                                           unsigned int &hits, unsigned int &flags, bool last = false) {
  double rh;
  const double r = rect_root(__dadd_rn(__dadd_rn(__dmul_rn(rx, rx), ry2), V.rz2), rh);
  double ai = SKIP ? 0.0 : rect_amplitude(P, V.w, r, rh);
  const int q = rect_number(P, r, c0);
  int it = q >> RECT_FB;
  if (rect_near(q)) it = __double2int_rn(rect_q(r, V.dl, P));
  const unsigned int slot = (unsigned int)(it - w0);
  const bool in = valid && slot < (unsigned int)wn;
  hits += in ? 1u : 0u;
  if (last && valid && !in) flags |= RECT_LAST_OOB;
  if (valid && !in && (unsigned int)it < (unsigned int)P.nt) flags |= RECT_MISS;  // not expected
  if (SKIP) {
    if (!__any_sync(0xffffffffu, in)) return;  // no term of this step lands in the SIR
    ai = rect_amplitude(P, V.w, r, rh);
  }
  ordered_adds(in, slot, ai, h + it, lane, stage);
}

// All terms of one element, 32 per step. P.row_steps: a step stays inside a row
// (the sample index is monotone along it on either side of the point's
// projection, so equal samples are neighbours); else steps run on across rows.
template <bool SKIP>
__device__ __forceinline__ void element_terms(const RectParams &P, const ElemView &V, int lane, int64_t w0, int64_t w1,
                                              double *h, double *stage, unsigned long long &oob, unsigned int &flags,
                                              bool last) {
  const int64_t E = (int64_t)P.nx * P.ny;
  const bool plain = term_plain(P, V);
  if (plain) {
    const double c0 = __fma_rn(-V.dl, P.inv_dt, RECT_MAGIC);
    const int lo = (int)w0, wn = (int)(w1 - w0);
    unsigned int hits = 0;
    if (P.row_steps) {
      for (int iy = 0; iy < P.ny; iy++) {
        const double ry = __dsub_rn(V.yo, __ldg(P.ys + iy)), ry2 = __dmul_rn(ry, ry);
        for (int x0 = 0; x0 < P.nx; x0 += 32) {
          const int ix = x0 + lane;
          const double rx = __dsub_rn(V.xo, __ldg(P.xs + min(ix, P.nx - 1)));
          plain_step<SKIP>(P, V, c0, ix < P.nx, rx, ry2, lane, lo, wn, h, stage, hits, flags);
        }
      }
    } else {
      // this lane's surface element e = iy*nx + ix, advanced by 32 per step without a division
      int iy = lane / P.nx, ix = lane - iy * P.nx;
      for (int64_t e0 = 0; e0 < E; e0 += 32) {
        const bool valid = e0 + lane < E;
        const double rx = __dsub_rn(V.xo, __ldg(P.xs + ix)), ry = __dsub_rn(V.yo, __ldg(P.ys + (valid ? iy : 0)));
        plain_step<SKIP>(P, V, c0, valid, rx, __dmul_rn(ry, ry), lane, lo, wn, h, stage, hits, flags);
        for (ix += 32; ix >= P.nx; ix -= P.nx) iy++;  // once for rows of 32 or more elements
      }
    }
    const unsigned long long missed = (unsigned long long)E - warp_sum_u64(hits);
    if (lane == 0 && missed) {
      oob += missed;
      if (last) flags |= RECT_LAST_OOB;
    }
    return;
  }
  int iy = lane / P.nx, ix = lane - iy * P.nx;
  for (int64_t e0 = 0; e0 < E; e0 += 32) {
    term_step<SKIP>(P, V, e0 + lane < E, ix, iy, lane, w0, w1, h, stage, oob, flags, last);
    for (ix += 32; ix >= P.nx; ix -= P.nx) iy++;
  }
}

// Terms of the live elements L (bits) among elements m0 .. m0 + 31, 32 consecutive
// ones per step whatever element they belong to; `plain`: all are term_plain.
__device__ __forceinline__ void packed_terms(const RectParams &P, int64_t m0, int64_t n, unsigned int L, bool plain,
                                             int lane, int64_t w0, int64_t w1, double *h, double *stage,
                                             unsigned long long &oob, unsigned int &flags) {
  const int E = P.nx * P.ny, total = __popc(L) * E;
  // this lane's term: its live element (the lowest bit still set in L) and surface element (ix, iy)
  int iy = lane % E / P.nx, ix = lane % E - iy * P.nx;
  for (int j = lane / E; j > 0; j--) L &= L - 1u;
  ElemView V;
  double c0 = 0.0;
  bool last = false;
  auto view = [&]() {  // of the last element where none is left (never added)
    const int64_t m = L ? m0 + __ffs(L) - 1 : P.M - 1;
    elem_view(P, m, n, V);
    c0 = __fma_rn(-V.dl, P.inv_dt, RECT_MAGIC);
    last = m == P.M - 1;
  };
  view();
  unsigned int hits = 0;
  for (int g0 = 0;;) {
    const bool valid = g0 + lane < total;
    if (plain) {
      const double rx = __dsub_rn(V.xo, __ldg(P.xs + ix)), ry = __dsub_rn(V.yo, __ldg(P.ys + iy));
      plain_step<true>(P, V, c0, valid, rx, __dmul_rn(ry, ry), lane, (int)w0, (int)(w1 - w0), h, stage, hits, flags, last);
    } else {
      term_step<true>(P, V, valid, ix, iy, lane, w0, w1, h, stage, oob, flags, last);
    }
    if ((g0 += 32) >= total) break;
    bool next = false;
    for (ix += 32; ix >= P.nx; ix -= P.nx)
      if (++iy == P.ny) {
        iy = 0;
        L &= L - 1u;
        next = true;
      }
    if (next) view();
  }
  if (plain) oob += (lane == 0 ? (unsigned long long)total : 0ull) - hits;  // summed over the warp at the end
}

// ARR = false: dreamrect (one element at the origin, P.M == 1), ARR = true: arrays;
// PACK: their live elements' terms side by side. MINB: blocks per SM.
template <bool ARR, bool PACK, int MINB = 4>
__global__ void __launch_bounds__(RECT_WARPS * 32, MINB) rect_kernel(const RectParams P) {
  extern __shared__ __align__(16) double rect_dyn[];  // [warps][32] staged amplitudes, then [warps][P.win]
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  double *stage = rect_dyn + warp * 32;
  double *win_sm = rect_dyn + (blockDim.x >> 5) * 32 + (int64_t)warp * P.win;
  int64_t n = (int64_t)blockIdx.x * (blockDim.x >> 5) + warp;
  if (n >= (!ARR && P.n_rest > 0 ? P.n_rest : P.No)) return;  // whole warps only: no block-wide barrier below
  if (!ARR && P.n_rest > 0) n = P.rest[n];
  double *out = P.H + n * P.nt;
  ElemView V;
  // union of the live elements' windows
  int64_t lo = INT64_MAX, hi = INT64_MIN;
  bool live0 = false;  // dreamrect: its element is live
  if (!ARR) {
    elem_view(P, 0, n, V);
    live0 = elem_window(P, V, lo, hi);
  } else {
    for (int64_t m = lane; m < P.M; m += 32) {
      int64_t l, h;
      elem_view(P, m, n, V);
      if (elem_window(P, V, l, h)) {
        lo = min(lo, l);
        hi = max(hi, h);
      }
    }
    for (int o = 16; o; o >>= 1) {
      lo = min(lo, (int64_t)__shfl_xor_sync(0xffffffffu, (long long)lo, o));
      hi = max(hi, (int64_t)__shfl_xor_sync(0xffffffffu, (long long)hi, o));
    }
  }
  int64_t w0 = 0, w1 = 0;
  if ((ARR || live0) && lo < hi) {
    w0 = max((int64_t)0, lo);
    w1 = min(P.nt, hi);
  }
  const bool in_smem = !P.full && w1 - w0 <= P.win;
  // the SIR: shared-memory window (offset w0) or the output column itself
  double *h = in_smem ? win_sm - w0 : out;
  if (in_smem) {
    for (int64_t i = lane; i < P.win; i += 32) win_sm[i] = 0.0;
  } else {
    for (int64_t i = lane; i < P.nt; i += 32) out[i] = 0.0;
  }
  __syncwarp();
  const int64_t E = (int64_t)P.nx * P.ny;  // terms per element (> 0)
  unsigned long long oob = 0;
  unsigned int flags = 0;
  if (!ARR) {
    if (!live0) {  // no term in bounds
      if (lane == 0) {
        oob = (unsigned long long)E;
        flags = RECT_LAST_OOB;
      }
    } else {
      element_terms<false>(P, V, lane, w0, w1, h, stage, oob, flags, true);
    }
  } else {
    for (int64_t c0 = 0; c0 < P.M; c0 += 32) {
      // the next 32 elements: dead ones only add to the out-of-bounds count
      bool live = false;
      if (c0 + lane < P.M) {
        int64_t l, h2;
        elem_view(P, c0 + lane, n, V);
        live = elem_window(P, V, l, h2);
        if (!live) {
          oob += (unsigned long long)E;
          if (c0 + lane == P.M - 1) flags |= RECT_LAST_OOB;
        }
      }
      unsigned int L = __ballot_sync(0xffffffffu, live);
      if (PACK) {
        const bool plain = __all_sync(0xffffffffu, !live || term_plain(P, V));
        if (L) packed_terms(P, c0, n, L, plain, lane, w0, w1, h, stage, oob, flags);
        continue;
      }
      for (; L; L &= L - 1u) {
        const int64_t m = c0 + __ffs(L) - 1;
        elem_view(P, m, n, V);
        element_terms<true>(P, V, lane, w0, w1, h, stage, oob, flags, m == P.M - 1);
      }
    }
  }
  if (in_smem) {
    for (int64_t i = lane; i < P.nt; i += 32) out[i] = (i >= w0 && i < w1) ? win_sm[i - w0] : 0.0;
  }
  oob = warp_sum_u64(oob);
  flags = __reduce_or_sync(0xffffffffu, flags);
  if (lane == 0) {
    if (oob) atomicAdd(P.oob, oob);
    if (flags) atomicOr(P.flags, flags);
  }
}

// ---------------------------------------------------------------------------
// dreamrect with one observation point per lane: large fields.
//
// Every lane sums its own point's terms in order into its own column of a
// shared-memory window (sample i of lane l at win[(i + 1) * 32 + l], free of
// bank conflicts; row 0 takes the terms outside the window), so no term has to
// be matched or ordered across lanes, and the surface-element centres are
// uniform. RECT_U terms' chains run side by side, and the adds of one group are
// issued among the arithmetic of the next.
//
// Bound: 26 FP64 operations and 20 others per term. The reference's 10 x 15 mm
// element of 60000 surface elements, nt = 300, 89304 points: 13.9 ms, against
// 42.1 with one warp per point, IEEE intrinsics and the matching of equal samples
// across lanes (228 instructions per 32 terms, serial chains). The FP64 pipe
// alone would take 7.6; the windows (20 KB a warp here) leave 10 warps on an SM,
// too few to hide the 8-cycle operations of every chain. 4 terms side by side:
// 15.7 ms.
// ---------------------------------------------------------------------------

constexpr int RECT_U = 8;

__device__ __forceinline__ double lds_f64(unsigned int a) {
  double v;
  asm volatile("ld.shared.f64 %0, [%1];" : "=d"(v) : "r"(a));
  return v;
}
__device__ __forceinline__ void sts_f64(unsigned int a, double v) {
  asm volatile("st.shared.f64 [%0], %1;" ::"r"(a), "d"(v) : "memory");
}

// This lane's window: samples [w0, w0 + wn) of its point, 256 bytes apart from
// address `first`; `trash` takes the others.
struct LaneSir {
  unsigned int first, trash, hits;
  int w0, wn;
  __device__ __forceinline__ void add(int it, double ai) {
    const unsigned int slot = (unsigned int)(it - w0);
    const bool ok = slot < (unsigned int)wn;
    const unsigned int a = ok ? first + slot * 256u : trash;
    hits += ok ? 1u : 0u;
    sts_f64(a, __dadd_rn(lds_f64(a), ai));
  }
};

// One warp per CTA.
__global__ void __launch_bounds__(32) rect_lane_kernel(const RectParams P) {
  extern __shared__ __align__(16) double rect_dyn[];  // [P.win + 1][32]
  const int lane = threadIdx.x;
  const int64_t first = (int64_t)blockIdx.x * 32;
  const bool active = first + lane < P.No;
  ElemView V;
  elem_view(P, 0, active ? first + lane : first, V);
  const unsigned long long E = (unsigned long long)P.nx * P.ny;
  unsigned long long oob = 0;
  unsigned int flags = 0;
  for (int64_t i = lane; i < (P.win + 1) * 32; i += 32) rect_dyn[i] = 0.0;
  int64_t lo, hi, w0 = 0, w1 = 0;
  if (elem_window(P, V, lo, hi)) {
    w0 = max((int64_t)0, lo);
    w1 = max(w0, min(P.nt, hi));
  }
  // A point without trusted estimates (not a number, or very far away) has the window [0, nt). It is left to
  // rect_kernel, and its lane adds nothing, whatever the warp computes for it.
  const bool fits = w1 - w0 <= P.win;
  if (!fits) w1 = w0;
  LaneSir S;
  S.trash = (unsigned int)__cvta_generic_to_shared(rect_dyn + lane);
  S.first = S.trash + 256u;
  S.hits = 0;
  S.w0 = (int)w0;
  S.wn = (int)(w1 - w0);
  __syncwarp();
  if (!__any_sync(0xffffffffu, S.wn > 0)) {  // no term in bounds
    oob = E;
  } else if (__all_sync(0xffffffffu, term_plain(P, V) || !fits)) {
    const double c0 = __fma_rn(-V.dl, P.inv_dt, RECT_MAGIC);
    int q_min = INT_MAX, q_max = INT_MIN;
    int iy = 0, left = P.nx;  // row and terms left in it
    const double *xs = P.xs;  // rows padded to whole groups with their last centre
    double ry2 = 0.0;
    auto row = [&]() {
      const double ry = __dsub_rn(V.yo, __ldg(P.ys + iy));
      ry2 = __dmul_rn(ry, ry);
    };
    row();
    // amplitudes and samples of the next group of n terms; false after the last one
    auto compute = [&](double(&ai)[RECT_U], int(&it)[RECT_U], int &n) -> bool {
      double r[RECT_U];
      int q[RECT_U];
      unsigned int near = 0;
#pragma unroll
      for (int u = 0; u < RECT_U; u++) {
        const double rx = __dsub_rn(V.xo, __ldg(xs + u));
        double h;
        r[u] = rect_root(__dadd_rn(__dadd_rn(__dmul_rn(rx, rx), ry2), V.rz2), h);
        ai[u] = rect_amplitude(P, V.w, r[u], h);
        q[u] = rect_number(P, r[u], c0);
        it[u] = q[u] >> RECT_FB;
        near = max(near, ((unsigned int)q[u] - 3u) * (1u << (32 - RECT_FB)));
        q_min = min(q_min, q[u]);
        q_max = max(q_max, q[u]);
      }
      if (__any_sync(0xffffffffu, near > (((1u << RECT_FB) - 7u) << (32 - RECT_FB)))) {
#pragma unroll
        for (int u = 0; u < RECT_U; u++)
          if (rect_near(q[u])) it[u] = __double2int_rn(rect_q(r[u], V.dl, P));
      }
      n = min(RECT_U, left);
      xs += RECT_U;
      left -= RECT_U;
      if (left <= 0) {
        if (++iy == P.ny) return false;
        left = P.nx;
        xs = P.xs;
        row();
      }
      return true;
    };
    auto add = [&](const double(&ai)[RECT_U], const int(&it)[RECT_U], int n) {
      if (n == RECT_U) {
#pragma unroll
        for (int u = 0; u < RECT_U; u++) S.add(it[u], ai[u]);
      } else {
#pragma unroll
        for (int u = 0; u < RECT_U; u++)
          if (u < n) S.add(it[u], ai[u]);
      }
    };
    double a0[RECT_U], a1[RECT_U];
    int i0[RECT_U], i1[RECT_U], n0 = 0, n1 = 0;
    for (bool more = compute(a0, i0, n0);;) {
      if (!more) {
        add(a0, i0, n0);
        break;
      }
      more = compute(a1, i1, n1);
      add(a0, i0, n0);
      if (!more) {
        add(a1, i1, n1);
        break;
      }
      more = compute(a0, i0, n0);
      add(a1, i1, n1);
    }
    oob = E - S.hits;
    // every term inside its window: the exact samples lie within 1 of these
    if ((q_min >> RECT_FB) <= lo || (q_max >> RECT_FB) >= hi - 1) flags |= RECT_MISS;
  } else {
    for (int iy = 0; iy < P.ny; iy++) {
      const double ry = __dsub_rn(V.yo, __ldg(P.ys + iy));
      for (int ix = 0; ix < P.nx; ix++) {
        const double rx = __dsub_rn(V.xo, __ldg(P.xs + ix));
        const double r = __dsqrt_rn(__dadd_rn(__dadd_rn(__dmul_rn(rx, rx), __dmul_rn(ry, ry)), V.rz2));
        const double ai = __dmul_rn(__ddiv_rn(__ddiv_rn(V.w, __dmul_rn(RECT_TWO_PI, r)), P.dt), 1000.0);
        const int64_t it = __double2ll_rn(rect_q(r, V.dl, P));
        const bool in = it >= 0 && it < P.nt;
        if (in && !(it >= w0 && it < w1)) flags |= RECT_MISS;
        S.add(in ? (int)it : -1 - S.wn, ai);
      }
    }
    oob = E - S.hits;
  }
  if (oob) flags |= RECT_LAST_OOB;
  if (active && !fits) P.rest[atomicAdd(P.rest_count, 1ull)] = first + lane;
  if (!active || !fits) {
    oob = 0;
    flags = 0;
  }
  __syncwarp();
  for (int p = 0; p < 32 && first + p < P.No; p++) {
    const int pw0 = __shfl_sync(0xffffffffu, S.w0, p), pwn = __shfl_sync(0xffffffffu, S.wn, p);
    double *out = P.H + (first + p) * P.nt;
    for (int i = lane; i < (int)P.nt; i += 32) {
      const unsigned int slot = (unsigned int)(i - pw0);
      out[i] = slot < (unsigned int)pwn ? rect_dyn[(slot + 1) * 32 + p] : 0.0;
    }
  }
  oob = warp_sum_u64(oob);
  flags = __reduce_or_sync(0xffffffffu, flags);
  if (lane == 0) {
    if (oob) atomicAdd(P.oob, oob);
    if (flags) atomicOr(P.flags, flags);
  }
}

// Element centres exactly as the reference's loops produce them.
int rect_centres(double a, double b, double dx, double dy, std::vector<double> &xs, std::vector<double> &ys) {
  if (!(dx > 0.0) || !(dy > 0.0)) return set_last_error(DREAM_ERR_ARGUMENT, "dreamrect: dx and dy must be positive");
  const double xsmin = -a / 2.0, xsmax = a / 2.0, ysmin = -b / 2.0, ysmax = b / 2.0;
  xs.clear();
  ys.clear();
  for (double x = xsmin + dx / 2.0; x <= xsmax; x += dx) {
    xs.push_back(x);
    if (xs.size() > (size_t(1) << 24)) return set_last_error(DREAM_ERR_ARGUMENT, "dreamrect: too many x elements");
  }
  for (double y = ysmin + dy / 2.0; y <= ysmax; y += dy) {
    ys.push_back(y);
    if (ys.size() > (size_t(1) << 24)) return set_last_error(DREAM_ERR_ARGUMENT, "dreamrect: too many y elements");
  }
  return 0;
}

struct RectBuffers {
  std::mutex mu;
  double *centres = nullptr, *Ro = nullptr, *delay = nullptr, *H = nullptr, *elems = nullptr;
  double *rest = nullptr;  // point numbers (RectParams::rest)
  size_t cap_c = 0, cap_ro = 0, cap_d = 0, cap_h = 0, cap_e = 0, cap_r = 0;
  unsigned long long *ctr = nullptr;  // [0] out-of-bounds terms, [1] RECT_* flags (low word), [2] points in rest
  cudaStream_t st = nullptr;
};

int grow(double *&p, size_t &cap, size_t bytes) {
  if (bytes <= cap) return 0;
  if (p) cudaFree(p);
  p = nullptr;
  cap = 0;
  if (cudaMalloc(&p, bytes) != cudaSuccess) {
    cudaGetLastError();
    return set_last_error(DREAM_ERR_ALLOC, "dreamrect: device allocation failed");
  }
  cap = bytes;
  return 0;
}

RectBuffers &rect_buffers(int device) {
  static std::vector<RectBuffers> bufs(64);
  return bufs[device];
}

int status_of(uint64_t oob, int err_level) {
  if (oob == 0) return 0;
  switch (err_level) {
    case DREAM_ERR_LEVEL_IGNORE: return DREAM_STATUS_IGNORE_OUT_OF_BOUNDS;
    case DREAM_ERR_LEVEL_WARN: return DREAM_STATUS_WARN_OUT_OF_BOUNDS;
    case DREAM_ERR_LEVEL_STOP: return DREAM_STATUS_OUT_OF_BOUNDS;
    default: return DREAM_STATUS_NONE;
  }
}

// Array description: element centres G (M x 3, column-major) and the
// focusing, steering and apodisation settings, all on the host.
struct ArrDesc {
  int64_t M = 1;
  bool single = true;         // dreamrect: one element at the origin (G unused)
  const double *G = nullptr;
  int foc_met = DREAM_FOC_OFF, steer_met = DREAM_STEER_OFF, apod_met = DREAM_APOD_OFF;
  const double *focal = nullptr, *apod = nullptr;
  double theta = 0.0, phi = 0.0, apod_par = 0.0;
};

// Per-element centres, delays and term numerators, with the reference's
// operations in its order (max_dim_arr, focusing, beamsteering and
// apodization of src/arr_functions.cc:60-262, called as
// src/dream_arr_rect.cc:206-234 calls them; weight*v*ds of
// src/dreamrect.cc:306). Host code is compiled without contraction, so each
// product and sum is rounded on its own, and sin / cos / exp are the C
// library's, as in the reference's build.
int arr_elements(const ArrDesc &A, double v, double cp, double ds, std::vector<ArrElem> &out) {
  const int64_t M = A.M;
  out.assign((size_t)M, ArrElem{0.0, 0.0, 0.0, 0.0, 0.0, 0.0});
  if (M == 0) return 0;
  if (A.single) {  // dreamrect: one element at the origin, unit weight
    out[0].wvds = 1.0 * v * ds;
    return 0;
  }
  const double *gx = A.G, *gy = A.G + M, *gz = A.G + 2 * M;
  double x_max = std::fabs(gx[0]), y_max = std::fabs(gy[0]);
  for (int64_t i = 1; i < M; i++)
    if (std::fabs(gx[i]) > x_max) x_max = std::fabs(gx[i]);
  for (int64_t i = 1; i < M; i++)
    if (std::fabs(gy[i]) > y_max) y_max = std::fabs(gy[i]);
  const double r_max = std::sqrt(x_max * x_max + y_max * y_max);
  const double pi = 3.14159265358979323846, deg2rad = pi / 180.0;
  for (int64_t n = 0; n < M; n++) {
    ArrElem &el = out[(size_t)n];
    el.gx = gx[n];
    el.gy = gy[n];
    el.gz = gz[n];
    double foc = 0.0;
    if (A.foc_met == DREAM_FOC_UD) {
      foc = A.focal[n];
    } else if (A.foc_met != DREAM_FOC_OFF) {
      const double f = A.focal[0];
      double diff = 0.0;
      switch (A.foc_met) {
        case DREAM_FOC_X: diff = std::sqrt(x_max * x_max + f * f) - std::sqrt(gx[n] * gx[n] + f * f); break;
        case DREAM_FOC_Y: diff = std::sqrt(y_max * y_max + f * f) - std::sqrt(gy[n] * gy[n] + f * f); break;
        case DREAM_FOC_XY:
          diff = std::sqrt(r_max * r_max + f * f) - std::sqrt(gx[n] * gx[n] + gy[n] * gy[n] + f * f);
          break;
        default: {  // DREAM_FOC_X_Y
          const double rx = std::sqrt(gx[n] * gx[n] + f * f), ry = std::sqrt(gy[n] * gy[n] + f * f);
          diff = std::sqrt(r_max * r_max + f * f) - (rx + ry);
        }
      }
      foc = diff * 1.0e3 / cp;
    }
    double steer = 0.0;
    if (A.steer_met == DREAM_STEER_X || A.steer_met == DREAM_STEER_XY) {
      const double sx = std::sin(A.theta * deg2rad);
      steer = (x_max * sx + gx[n] * sx) * 1.0e3 / cp;
    }
    if (A.steer_met == DREAM_STEER_Y || A.steer_met == DREAM_STEER_XY) {
      const double sy = std::sin(A.phi * deg2rad);
      const double st_y = (y_max * sy + gy[n] * sy) * 1.0e3 / cp;
      steer = A.steer_met == DREAM_STEER_XY ? steer + st_y : st_y;
    }
    double w = 1.0;
    if (A.apod_met != DREAM_APOD_OFF) {
      const double r = std::sqrt(gx[n] * gx[n] + gy[n] * gy[n]);
      const double c = 1.0 - r * r / (r_max * r_max);
      switch (A.apod_met) {
        case DREAM_APOD_UD: w = A.apod[n]; break;
        case DREAM_APOD_TRIANGLE: w = 1.0 - std::fabs(r) / r_max; break;
        case DREAM_APOD_GAUSS: w = std::exp(-(A.apod_par * r * r) / (r_max * r_max)); break;
        case DREAM_APOD_RAISED: w = A.apod_par + std::cos(r * pi / r_max); break;
        case DREAM_APOD_HANN: w = 0.5 * (1.0 - std::cos((r + r_max) * pi / r_max)); break;
        case DREAM_APOD_HAMMING: {
          const double a0 = 25.0 / 46.0;
          w = a0 - (1.0 - a0) * std::cos((r + r_max) * pi / r_max);
        } break;
        case DREAM_APOD_SIMPLY: w = c; break;
        default: w = c * c;  // DREAM_APOD_CLAMPED
      }
    }
    el.foc = foc;
    el.steer = steer;
    el.wvds = w * v * ds;
  }
  return 0;
}

int check_desc(const ArrDesc &A) {
  if (A.M < 0) return set_last_error(DREAM_ERR_ARGUMENT, "dream_arr_rect: negative number of elements");
  if (!A.single && A.M > 0 && A.G == nullptr)
    return set_last_error(DREAM_ERR_ARGUMENT, "dream_arr_rect: NULL element grid");
  if (A.foc_met < DREAM_FOC_OFF || A.foc_met > DREAM_FOC_UD)
    return set_last_error(DREAM_ERR_ARGUMENT, "dream_arr_rect: unknown focusing method");
  if (A.steer_met < DREAM_STEER_OFF || A.steer_met > DREAM_STEER_XY)
    return set_last_error(DREAM_ERR_ARGUMENT, "dream_arr_rect: unknown beam steering method");
  if (A.apod_met < DREAM_APOD_OFF || A.apod_met > DREAM_APOD_UD)
    return set_last_error(DREAM_ERR_ARGUMENT, "dream_arr_rect: unknown apodization method");
  if (A.foc_met != DREAM_FOC_OFF && A.focal == nullptr)
    return set_last_error(DREAM_ERR_ARGUMENT, "dream_arr_rect: NULL focal");
  if (A.apod_met == DREAM_APOD_UD && A.apod == nullptr)
    return set_last_error(DREAM_ERR_ARGUMENT, "dream_arr_rect: NULL apodization weights");
  return 0;
}

// Shared-memory window bound of a launch: no point's union window is wider
// than the travel-time difference across the array's extent (the element
// rectangles around their centres) plus the spread of the element delays,
// +-2 samples per side and rounding.
int64_t window_bound(const std::vector<ArrElem> &el, double a, double b, double dt, double cp, int64_t nt) {
  double x0 = INFINITY, x1 = -INFINITY, y0 = INFINITY, y1 = -INFINITY, z0 = INFINITY, z1 = -INFINITY;
  double d0 = INFINITY, d1 = -INFINITY;
  for (const ArrElem &e : el) {
    x0 = std::min(x0, e.gx), x1 = std::max(x1, e.gx);
    y0 = std::min(y0, e.gy), y1 = std::max(y1, e.gy);
    z0 = std::min(z0, e.gz), z1 = std::max(z1, e.gz);
    d0 = std::min(d0, e.foc + e.steer), d1 = std::max(d1, e.foc + e.steer);
  }
  const double ex = x1 - x0 + std::fabs(a), ey = y1 - y0 + std::fabs(b), ez = z1 - z0;
  const double span =
      (std::sqrt(ex * ex + ey * ey + ez * ez) * 1000.0 / std::fabs(cp) + (d1 - d0)) / std::fabs(dt);
  if (!std::isfinite(span) || span > (double)nt) return nt;
  return std::min<int64_t>(nt, (int64_t)(span * (1.0 + 1e-9)) + 8);
}

// With the device current and the buffers locked: SIRs of the points in dRo
// into dH (device pointers), status from the out-of-bounds count.
int rect_device(RectBuffers &rb, const double *dRo, int64_t No, double a, double b, double dx, double dy, double dt,
                int64_t nt, int delay_type, const double *ddelay, double v, double cp, const ArrDesc &A, double *dH,
                int err_level, int64_t *oob_count, cudaStream_t st) {
  const char *fn = A.single ? "dreamrect" : "dream_arr_rect";
  if (No < 0 || nt < 0) return set_last_error(DREAM_ERR_ARGUMENT, std::string(fn) + ": negative size");
  if (delay_type != DREAM_DELAY_SINGLE && delay_type != DREAM_DELAY_MULTIPLE)
    return set_last_error(DREAM_ERR_ARGUMENT, "unknown delay type");
  int r = check_desc(A);
  if (r) return r;
  std::vector<double> xs, ys;
  if ((r = rect_centres(a, b, dx, dy, xs, ys))) return r;
  std::vector<ArrElem> el;
  if ((r = arr_elements(A, v, cp, dx * dy, el))) return r;
  if (oob_count) *oob_count = 0;
  const size_t nx = xs.size(), ny = ys.size();
  const uint64_t terms = (uint64_t)A.M * nx * ny;
  if (No == 0) return 0;
  if (nt == 0) {  // no sample to land in: every term is out of bounds
    const uint64_t all = (uint64_t)No * terms;
    if (oob_count) *oob_count = (int64_t)all;
    return status_of(all, err_level);  // the last element's terms are out of bounds too
  }
  if (dRo == nullptr || ddelay == nullptr || dH == nullptr) return set_last_error(DREAM_ERR_ARGUMENT, "NULL pointer");
  cudaError_t e = cudaSuccess;
  if (rb.ctr == nullptr && (e = cudaMalloc(&rb.ctr, 3 * sizeof(unsigned long long))) != cudaSuccess)
    return set_last_error(DREAM_ERR_ALLOC, cudaGetErrorString(e));
  if (terms == 0) {  // no surface element: the SIRs are zero
    e = cudaMemsetAsync(dH, 0, (size_t)No * nt * 8, st);
    if (e == cudaSuccess) e = cudaStreamSynchronize(st);
    if (e != cudaSuccess) return set_last_error(DREAM_ERR_CUDA, std::string(fn) + ": " + cudaGetErrorString(e));
    return 0;
  }
  if ((r = grow(rb.centres, rb.cap_c, (nx + RECT_U - 1 + ny) * 8)) || (r = grow(rb.elems, rb.cap_e, el.size() * sizeof(ArrElem))))
    return r;
  std::vector<double> both(xs);
  both.insert(both.end(), (size_t)RECT_U - 1, xs.back());  // read, not used, by the last group of a row
  both.insert(both.end(), ys.begin(), ys.end());
  e = cudaMemcpyAsync(rb.centres, both.data(), both.size() * 8, cudaMemcpyHostToDevice, st);
  if (e == cudaSuccess)
    e = cudaMemcpyAsync(rb.elems, el.data(), el.size() * sizeof(ArrElem), cudaMemcpyHostToDevice, st);
  RectParams P;
  P.Ro = dRo;
  P.No = No;
  P.xs = rb.centres;
  P.ys = rb.centres + nx + RECT_U - 1;
  P.nx = (int)nx;
  P.ny = (int)ny;
  P.el = reinterpret_cast<const ArrElem *>(rb.elems);
  P.M = A.M;
  P.half_a = a / 2.0;
  P.half_b = b / 2.0;
  P.dt = dt;
  P.cp = cp;
  P.c1 = 1000.0 / cp;
  P.inv_dt = 1.0 / dt;
  P.k1 = P.c1 * P.inv_dt;
  const auto ranged = [](double v) { return std::fabs(v) > 0x1p-100 && std::fabs(v) < 0x1p100; };
  P.plain_range = nt <= INT32_MAX && ranged(dt) && ranged(cp) && ranged(P.c1) && ranged(P.inv_dt);
  P.ab = std::fabs(a) + std::fabs(b);
  P.nt = nt;
  P.delay = ddelay;
  P.delay_multi = delay_type == DREAM_DELAY_MULTIPLE;
  P.H = dH;
  P.oob = rb.ctr;
  P.flags = reinterpret_cast<unsigned int *>(rb.ctr + 1);
  P.rest_count = rb.ctr + 2;
  P.n_rest = 0;
  unsigned long long h_ctr[3] = {0, 0, 0};
  int dev = 0, sms = 148;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  // Steps that end with the rows where the lanes this leaves idle cost less than the steps that straddle two rows (and
  // whose equal samples are then no neighbours): 30-element rows of arrays 10.1 against 14.4 ms, 200-element rows of
  // one element 38.0 against 36.4, 8-element rows 0.77 against 0.30 (IEEE root and 64-bit samples in all of these).
  P.row_steps = nx >= 20 && (nx % 32 == 0 || nx % 32 > 10);
  // Arrays without such rows: steps that run on from one live element to the next, where a last step of its own would
  // leave a fifth of an element's lanes idle (441 elements, 60000 points, nt = 400, of 1 surface element each 0.86
  // against 12.5 ms, of 4 2.0 against 11.0; of 64 they cost 2 % more). They keep a view per lane, which 64 registers
  // do not hold without spilling: less than a wave of blocks takes 80 (81 elements of 36, 500 points 0.19 ms, 0.23 with
  // 64, 0.27 by element; of 100 0.34 against 0.42 by element; 60000 points 0.83 with 80, 0.76 with 64).
  const uint64_t E = (uint64_t)nx * ny;
  const bool small = (No + RECT_WARPS - 1) / RECT_WARPS <= 4 * (int64_t)sms;
  const bool pack = !P.row_steps && E <= 1024 && (small || (E + 31) / 32 * 32 * 5 > E * 6);
  const auto kernel = A.single ? rect_kernel<false, false>
                      : !pack  ? rect_kernel<true, false>
                      : small  ? rect_kernel<true, true, 3>
                               : rect_kernel<true, true>;
  if (e == cudaSuccess) e = ensure_smem(kernel, RECT_SMEM_MAX);
  // dreamrect: one point per lane where that is the faster form. With c windows on an SM a round takes about 1 + c/50
  // times a lone warp's 71 ns per term; one warp per point takes 6.4 ps per term and point (both on the 60000-element
  // field above: 8000 points 4.25 against 3.51 ms, 16000 4.28 against 6.3).
  const int64_t lane_win = A.single ? window_bound(el, a, b, dt, cp, nt) : 0, lane_smem = (lane_win + 1) * 32 * 8;
  bool lanes = false;
  if (A.single && nt <= INT32_MAX && lane_smem <= RECT_SMEM_MAX) {
    const int64_t c = std::min<int64_t>(16, (227 * 1024) / (lane_smem + 1024));
    const int64_t rounds = (No + 32 * c * sms - 1) / (32 * c * sms);
    lanes = (double)rounds * (1.0 + 0.02 * c) * 11100.0 < (double)No;
  }
  if (lanes && e == cudaSuccess) e = ensure_smem(rect_lane_kernel, RECT_SMEM_MAX);
  if (lanes && (r = grow(rb.rest, rb.cap_r, (size_t)No * sizeof(int64_t)))) return r;
  P.rest = reinterpret_cast<int64_t *>(rb.rest);
  for (int full = 0; full < 2 && e == cudaSuccess; full++) {
    int64_t win = full ? 0 : window_bound(el, a, b, dt, cp, nt);
    int warps = RECT_WARPS;
    while (warps > 1 && (int64_t)warps * (win + 32) * 8 > RECT_SMEM_MAX) warps >>= 1;
    if ((int64_t)warps * (win + 32) * 8 > RECT_SMEM_MAX) {  // very long windows: accumulate in the output columns
      win = 0;
      warps = RECT_WARPS;
    }
    P.win = win;
    P.full = full;
    const size_t smem = (size_t)warps * (win + 32) * sizeof(double);
    const auto read_counters = [&]() {
      cudaError_t c = cudaGetLastError();
      if (c == cudaSuccess) c = cudaMemcpyAsync(h_ctr, rb.ctr, sizeof(h_ctr), cudaMemcpyDeviceToHost, st);
      return c == cudaSuccess ? cudaStreamSynchronize(st) : c;
    };
    e = cudaMemsetAsync(rb.ctr, 0, sizeof(h_ctr), st);
    if (e != cudaSuccess) break;
    if (lanes && !full) {
      P.win = lane_win;
      rect_lane_kernel<<<(unsigned)((No + 31) / 32), 32, lane_smem, st>>>(P);
      e = read_counters();
      if (e == cudaSuccess && h_ctr[2] > 0 && !(h_ctr[1] & RECT_MISS)) {
        P.win = win;
        P.n_rest = (int64_t)h_ctr[2];
        kernel<<<(unsigned)((P.n_rest + warps - 1) / warps), warps * 32, smem, st>>>(P);
        P.n_rest = 0;
        e = read_counters();
      }
    } else {
      kernel<<<(unsigned)((No + warps - 1) / warps), warps * 32, smem, st>>>(P);
      e = read_counters();
    }
    if (!(h_ctr[1] & RECT_MISS)) break;  // every term fell in its point's window
  }
  if (e != cudaSuccess) return set_last_error(DREAM_ERR_CUDA, std::string(fn) + ": " + cudaGetErrorString(e));
  if (oob_count) *oob_count = (int64_t)h_ctr[0];
  // the reference keeps, per point, the status of the array's last element
  // (src/dream_arr_rect.cc:209-243); 'stop' ends at the first out-of-bounds term
  return status_of(err_level == DREAM_ERR_LEVEL_STOP ? h_ctr[0] : (h_ctr[1] & RECT_LAST_OOB), err_level);
}

struct DeviceScope {
  int prev = -1;
  bool ok = true;
  explicit DeviceScope(int dev) {
    cudaGetDevice(&prev);
    if (prev != dev) ok = cudaSetDevice(dev) == cudaSuccess;
  }
  ~DeviceScope() {
    int cur = -1;
    if (prev >= 0 && cudaGetDevice(&cur) == cudaSuccess && cur != prev) cudaSetDevice(prev);
  }
};

int check_device(int device) {
  int ndev = 0;
  if (cudaGetDeviceCount(&ndev) != cudaSuccess || device < 0 || device >= ndev || device >= 64)
    return set_last_error(DREAM_ERR_ARGUMENT, "invalid CUDA device ordinal");
  return 0;
}

}  // namespace
}  // namespace dream

using namespace dream;

extern "C" {

namespace {

int rect_entry_device(const double *dRo, int64_t No, double a, double b, double dx, double dy, double dt,
                      int64_t nt, int delay_type, const double *ddelay, double v, double cp, const ArrDesc &A,
                      double *dH, int err_level, int64_t *oob_count, int device, void *stream) {
  int r = check_device(device);
  if (r) return r;
  RectBuffers &rb = rect_buffers(device);
  std::lock_guard<std::mutex> lk(rb.mu);
  DeviceScope ds(device);
  if (!ds.ok) return set_last_error(DREAM_ERR_CUDA, "cudaSetDevice failed");
  return rect_device(rb, dRo, No, a, b, dx, dy, dt, nt, delay_type, ddelay, v, cp, A, dH, err_level, oob_count,
                     (cudaStream_t)stream);
}

int rect_entry_host(const double *Ro, int64_t No, double a, double b, double dx, double dy, double dt, int64_t nt,
                    int delay_type, const double *delay, double v, double cp, const ArrDesc &A, double *H,
                    int err_level, int64_t *oob_count, int device) {
  int r = check_device(device);
  if (r) return r;
  if (No < 0 || nt < 0) return set_last_error(DREAM_ERR_ARGUMENT, "dreamrect: negative size");
  if (No > 0 && (Ro == nullptr || delay == nullptr || (nt > 0 && H == nullptr)))
    return set_last_error(DREAM_ERR_ARGUMENT, "NULL host pointer");
  RectBuffers &rb = rect_buffers(device);
  std::lock_guard<std::mutex> lk(rb.mu);
  DeviceScope ds(device);
  if (!ds.ok) return set_last_error(DREAM_ERR_CUDA, "cudaSetDevice failed");
  cudaError_t e = cudaSuccess;
  if (rb.st == nullptr && (e = cudaStreamCreateWithFlags(&rb.st, cudaStreamNonBlocking)) != cudaSuccess)
    return set_last_error(DREAM_ERR_CUDA, cudaGetErrorString(e));
  const size_t nd = delay_type == DREAM_DELAY_MULTIPLE ? (size_t)No : 1;
  if ((r = grow(rb.Ro, rb.cap_ro, std::max<size_t>(1, (size_t)No * 3) * 8)) ||
      (r = grow(rb.delay, rb.cap_d, std::max<size_t>(1, nd) * 8)) ||
      (r = grow(rb.H, rb.cap_h, std::max<size_t>(1, (size_t)No * nt) * 8)))
    return r;
  if (No > 0) {
    e = cudaMemcpyAsync(rb.Ro, Ro, (size_t)No * 3 * 8, cudaMemcpyHostToDevice, rb.st);
    if (e == cudaSuccess) e = cudaMemcpyAsync(rb.delay, delay, nd * 8, cudaMemcpyHostToDevice, rb.st);
    if (e != cudaSuccess) return set_last_error(DREAM_ERR_CUDA, cudaGetErrorString(e));
  }
  int st = rect_device(rb, rb.Ro, No, a, b, dx, dy, dt, nt, delay_type, rb.delay, v, cp, A, rb.H, err_level,
                       oob_count, rb.st);
  if (st < 0) return st;
  if (No > 0 && nt > 0) {
    e = cudaMemcpyAsync(H, rb.H, (size_t)No * nt * 8, cudaMemcpyDeviceToHost, rb.st);
    if (e == cudaSuccess) e = cudaStreamSynchronize(rb.st);
    if (e != cudaSuccess) return set_last_error(DREAM_ERR_CUDA, cudaGetErrorString(e));
  }
  return st;
}

ArrDesc arr_desc(int64_t num_elements, const double *G, int foc_met, const double *focal, int steer_met,
                 double theta, double phi, int apod_met, const double *apod, double apod_par) {
  ArrDesc A;
  A.single = false;
  A.M = num_elements;
  A.G = G;
  A.foc_met = foc_met;
  A.focal = focal;
  A.steer_met = steer_met;
  A.theta = theta;
  A.phi = phi;
  A.apod_met = apod_met;
  A.apod = apod;
  A.apod_par = apod_par;
  return A;
}

}  // namespace

int dream_rect_run_device(const double *dRo, int64_t No, double a, double b, double dx, double dy, double dt,
                          int64_t nt, int delay_type, const double *ddelay, double v, double cp, double *dH,
                          int err_level, int64_t *oob_count, int device, void *stream) {
  DREAM_API_TRY
  return rect_entry_device(dRo, No, a, b, dx, dy, dt, nt, delay_type, ddelay, v, cp, ArrDesc(), dH, err_level,
                           oob_count, device, stream);
  DREAM_API_CATCH
}

int dream_rect_run(const double *Ro, int64_t No, double a, double b, double dx, double dy, double dt, int64_t nt,
                   int delay_type, const double *delay, double v, double cp, double *H, int err_level,
                   int64_t *oob_count, int device) {
  DREAM_API_TRY
  return rect_entry_host(Ro, No, a, b, dx, dy, dt, nt, delay_type, delay, v, cp, ArrDesc(), H, err_level, oob_count,
                         device);
  DREAM_API_CATCH
}

int dream_arr_rect_run_device(const double *dRo, int64_t No, double a, double b, double dx, double dy, double dt,
                              int64_t nt, int delay_type, const double *ddelay, double v, double cp,
                              int64_t num_elements, const double *G, int foc_met, const double *focal,
                              int steer_met, double theta, double phi, int apod_met, const double *apod,
                              double apod_par, double *dH, int err_level, int64_t *oob_count, int device,
                              void *stream) {
  DREAM_API_TRY
  if (num_elements > 0 && G == nullptr) return set_last_error(DREAM_ERR_ARGUMENT, "dream_arr_rect: NULL element grid");
  return rect_entry_device(dRo, No, a, b, dx, dy, dt, nt, delay_type, ddelay, v, cp,
                           arr_desc(num_elements, G, foc_met, focal, steer_met, theta, phi, apod_met, apod, apod_par),
                           dH, err_level, oob_count, device, stream);
  DREAM_API_CATCH
}

int dream_arr_rect_run(const double *Ro, int64_t No, double a, double b, double dx, double dy, double dt,
                       int64_t nt, int delay_type, const double *delay, double v, double cp, int64_t num_elements,
                       const double *G, int foc_met, const double *focal, int steer_met, double theta, double phi,
                       int apod_met, const double *apod, double apod_par, double *H, int err_level,
                       int64_t *oob_count, int device) {
  DREAM_API_TRY
  if (num_elements > 0 && G == nullptr) return set_last_error(DREAM_ERR_ARGUMENT, "dream_arr_rect: NULL element grid");
  return rect_entry_host(Ro, No, a, b, dx, dy, dt, nt, delay_type, delay, v, cp,
                         arr_desc(num_elements, G, foc_met, focal, steer_met, theta, phi, apod_met, apod, apod_par),
                         H, err_level, oob_count, device);
  DREAM_API_CATCH
}

}  // extern "C"
