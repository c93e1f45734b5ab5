// p2p_sym.cuh -- velocity of a particle set on itself, each unordered pair evaluated once.
//
// points_affect_points with one set as sources and targets (src/Influence.h:56-416): the core
// K(d^2) of a pair is the same for both particles, so one evaluation serves the two interactions
//   row a <- column b:  u_a += G_b K (y_b - y_a),  v_a -= G_b K (x_b - x_a)
//   column b <- row a:  u_b -= G_a K (y_b - y_a),  v_b += G_a K (x_b - x_a)
// which is 10 f32x2 operations and one reciprocal (or square root) per two interactions, where
// the one-sided kernel (p2p_packed.cuh) spends 14 and two.  Bound: the registers' read ports.  An
// f32x2 operation takes 2.1 SM clocks per scheduler with one or two distinct register operands
// and 3.1 with three (measured; two scalar FMAs in its place take as long), so the four
// accumulations of a pair of pairs cost half of its 24 clocks; MUFU is at 50 %, the FMA pipe at
// 67 %.  Other orders and groupings of the same operations and the accumulations as scalars came
// within 3 % of one another.  Measured (compensated, one-sided -> here): 1M Gaussian patch 249 -> 185.6
// ms (5.4e12 interactions/s), 131,072 Vatistas-2 plain 4.29 -> 3.26 ms, 33,001 Vatistas-2 with varying
// radii 415 -> 274 us, ten Euler steps of 20,000 Rosenhead-Moore 1.65 -> 1.06 ms.
//
// Layout: a row block is 1024 (or 2048) particles, eight (or sixteen) per thread of a 128-thread
// CTA in f32x2 register pairs (a warp owns 256 or 512 consecutive ones); columns are taken 32 at a
// time, one per lane: in step s of 32 lane l meets column l ^ s (a conflict-free shared-memory read)
// with its rows, and the column's running sum (the step's terms added first) moves to the lane that
// meets it next by shuffle, so after 32 steps every lane holds its own column's sum over the warp's
// rows (half of the rows apart from the other half, sym_group).  The four warps' sums are added in
// shared memory and leave as one pair per (row block, column), (hi, lo) of each when compensated; a row's
// own sums stay in registers over a whole run of columns (folded into two-sum pairs every 32 columns when
// compensated, every 256 otherwise).  Rows against their own block are one-sided.
//
// Work: row block k meets every 32-column group from its own first one on; these (block, group)
// units in order form a line of `total` units cut into equal ranges that the CTAs take from a
// counter.  A range may cross blocks; each (range, block) piece writes one row partial at slot
// range + block (strictly increasing along the line, so unique).  sym_reduce_kernel adds a
// particle's row partials and column partials in a fixed order: results do not depend on timing.
// Column partials take 16 bytes (8 when plain) per row block and later particle; large sets run in passes over
// the row blocks that keep them within a fixed scratch size.
#pragma once

#include <type_traits>

#include "p2p_kernel.cuh"

namespace obs {

constexpr int SYM_THREADS = 128;
constexpr int SYM_GRP = 32;                        // columns per group
constexpr int SYM_TG = 8;                          // groups per staged tile
constexpr int SYM_TILE = SYM_GRP * SYM_TG;
// NP f32x2 row pairs per thread: rows and groups per row block
constexpr int sym_gpb(int np) { return SYM_THREADS / 32 * 2 * np; }
constexpr int sym_rows(int np) { return sym_gpb(np) * SYM_GRP; }
constexpr float SYM_FAR = 1.0e18f;                 // padding coordinate: K there is finite and tiny

// A group's 32 columns as staged, every value twice for the packed operands: a warp's reads of
// column (lane ^ s) touch each bank once.
struct __align__(128) SymGroup {
  float4 xy[SYM_GRP];      // (x, x, y, y)
  float2 g[SYM_GRP];       // strength
  float2 z[SYM_GRP];       // radius term
};
static_assert(sizeof(SymGroup) == 1024, "group record");

struct SymArgs {
  const SymGroup* grp;     // the particles in groups of 32, padded to whole row blocks
  int n;                 // particles
  int npad;              // particles padded to whole row blocks
  int ngrp;              // 32-column groups holding a particle
  int gpb;               // groups per row block
  int blk0, nblk;        // row blocks of this pass
  int total;             // (block, group) units of this pass
  int nrange;
  int least;             // units of a range, where a CTA gets several
  int many;              // units of a CTA from which it gets sixteen ranges
  int* counter;
  const unsigned* meta;  // radius extrema (~min, max bits)
  int* status;
  void* colpart;         // per row block, its later columns: (sum G K dy, sum G K dx) as float4, each (hi, lo),
                         // when compensated, else float2
  float2* rowpart;       // [nrange + nblk][2][rows of a block] (hi, lo)
  float4* run;           // [npad] running sums (u hi, u lo, v hi, v lo) over the passes
  int first, last;       // first / last pass
};

// units of the pass before row block k (of the pass)
__device__ __forceinline__ int sym_prefix(const SymArgs& a, int k) {
  return k * (a.ngrp - a.gpb * a.blk0) - (a.gpb / 2) * k * (k - 1);
}
__device__ __forceinline__ int sym_range_begin(const SymArgs& a, int r) {
  return (int)((long long)a.total * r / a.nrange);
}

// the row block (of the pass) that unit pos belongs to
__device__ __forceinline__ int sym_block_of(const SymArgs& a, int pos) {
  int k = 0, hi = a.nblk - 1;
  while (k < hi) {
    const int m = (k + hi + 1) >> 1;
    if (sym_prefix(a, m) <= pos) k = m;
    else hi = m - 1;
  }
  return k;
}

// the ranges r0 .. r1 that hold row block k's units
__device__ __forceinline__ void sym_ranges_of(const SymArgs& a, int k, int& r0, int& r1) {
  const int p0 = sym_prefix(a, k), p1 = sym_prefix(a, k + 1) - 1;
  r0 = (int)((long long)p0 * a.nrange / a.total);
  r1 = (int)((long long)p1 * a.nrange / a.total);
  while (sym_range_begin(a, r0 + 1) <= p0) ++r0;
  while (sym_range_begin(a, r0) > p0) --r0;
  while (sym_range_begin(a, r1 + 1) <= p1) ++r1;
  while (sym_range_begin(a, r1) > p1) --r1;
}

// Column partials are kept for the columns after a row block only: row block k (of the pass) has sym_width
// of them, from column sym_first on, after those of the blocks before it (sym_base).
__host__ __device__ __forceinline__ int sym_first(const SymArgs& a, int k) { return (a.blk0 + k + 1) * a.gpb * SYM_GRP; }
__host__ __device__ __forceinline__ int sym_width(const SymArgs& a, int k) { return a.npad - sym_first(a, k); }
__host__ __device__ __forceinline__ size_t sym_base(const SymArgs& a, int k) {
  return (size_t)k * a.npad - (size_t)a.gpb * SYM_GRP * ((size_t)k * a.blk0 + (size_t)k * (k + 1) / 2);
}

// total and nrange of a pass whose blk0 and nblk are set
inline void sym_plan_pass(SymArgs& a, int slots) {
  a.total = a.nblk * (a.ngrp - a.gpb * a.blk0) - (a.gpb / 2) * a.nblk * (a.nblk - 1);
  // one range per resident CTA for small sets; up to sixteen (a.least units or more each) for large
  // ones, whose units differ in cost (near and far column groups; eight: the 1M patch takes 186.8 instead of 185.5 ms)
  const int per = a.total / slots, ranges = slots * (per < 2 * a.least ? 1 : per >= a.many ? 16 : per >= 8 * a.least ? 8 : per / a.least);
  a.nrange = a.total < ranges ? a.total : ranges;
}

// a pass from row block a.blk0 of nblk on: as many row blocks as have their column partials within cap columns, one
// at least
inline void sym_next_pass(SymArgs& a, int nblk, int slots, size_t cap) {
  a.nblk = 1;
  while (a.blk0 + a.nblk < nblk && sym_base(a, a.nblk + 1) <= cap) ++a.nblk;
  a.first = a.blk0 == 0;
  a.last = a.blk0 + a.nblk == nblk;
  sym_plan_pass(a, slots);
}
// most columns and row partials of any pass
struct SymScratch {
  size_t cols = 0, rows = 0;
  int passes = 0;
};
inline SymScratch sym_scratch(SymArgs a, int nblk, int slots, size_t cap) {
  SymScratch m;
  for (a.blk0 = 0; a.blk0 < nblk; a.blk0 += a.nblk, ++m.passes) {
    sym_next_pass(a, nblk, slots, cap);
    const size_t c = sym_base(a, a.nblk), r = (size_t)a.nrange + a.nblk;
    m.cols = c > m.cols ? c : m.cols;
    m.rows = r > m.rows ? r : m.rows;
  }
  return m;
}

struct SymUni {
  float us2, ucf, cfl, lim;
};

// K of two pairs from d^2 (Rosenhead-Moore: from d^2 + s^2); zz: the pairs' radius terms summed (uniform radii: one constant).  FORM 0: the
// far form 1/d^2 of the Gaussian and compact exponential cores; 1: the core with one radius for
// all; 2: the core with every particle's own radius.
template <int CORE, int FORM>
__device__ __forceinline__ float2 sym_core(float2 d2, float2 zz, const SymUni& q) {
  const float2 one = f2(1.0f, 1.0f), m1 = f2(-1.0f, -1.0f);
  if constexpr (FORM == 0) {
    return f2(rcp_a(d2.x), rcp_a(d2.y));
  } else if constexpr (CORE == CORE_RM) {
    return f2(rcp_a(d2.x), rcp_a(d2.y));
  } else if constexpr (CORE == CORE_V2) {
    const float2 w = __ffma2_rn(d2, d2, zz);
    return f2(rsqrt_a(w.x), rsqrt_a(w.y));
  } else if constexpr (CORE == CORE_WL) {
    const float2 dd = __fadd2_rn(d2, zz);
    const float2 w = __fmul2_rn(dd, dd);
    return __fmul2_rn(__fadd2_rn(dd, zz), f2(rcp_a(w.x), rcp_a(w.y)));
  } else if constexpr (CORE == CORE_V3) {
    const float2 w = __ffma2_rn(__fmul2_rn(d2, d2), d2, zz);
    return f2(ex2_a(lg2_a(w.x) * (-1.0f / 3.0f)), ex2_a(lg2_a(w.y) * (-1.0f / 3.0f)));
  } else if constexpr (CORE == CORE_SING) {
    return f2(d2.x > 0.0f ? rcp_a(d2.x) : 0.0f, d2.y > 0.0f ? rcp_a(d2.y) : 0.0f);
  } else {
    const float2 cf = (FORM == 1) ? f2(q.ucf, q.ucf) : f2(rcp_a(zz.x), rcp_a(zz.y));
    const float2 ood2 = f2(rcp_a(d2.x), rcp_a(d2.y));
    if constexpr (CORE == CORE_GAUSS) {
      // x = d^2/s^2 > 16: 1/d^2; x < 0.001: 1/s^2; else (1 - e^-x)/d^2, on t = -x log2(e)
      const float2 t = (FORM == 1) ? __fmul2_rn(d2, f2(q.cfl, q.cfl)) : __fmul2_rn(__fmul2_rn(d2, cf), f2(-kLog2e, -kLog2e));
      const float2 e = f2(ex2_a(t.x), ex2_a(t.y));
      float2 k = __fmul2_rn(ood2, __ffma2_rn(e, m1, one));
      k.x = (t.x < -16.0f * kLog2e) ? ood2.x : ((t.x > -0.001f * kLog2e) ? cf.x : k.x);
      k.y = (t.y < -16.0f * kLog2e) ? ood2.y : ((t.y > -0.001f * kLog2e) ? cf.y : k.y);
      return k;
    } else {
      // compact exponential, y = (d/s)^3 > 16: 1/d^2; y < 0.001: (d/s^3)(1 - y/2); else (1 - e^-y)/d^2
      const float2 x = __fmul2_rn(d2, cf);
      const float2 sq = f2(sqrt_a(x.x), sqrt_a(x.y));
      const float2 y = __fmul2_rn(x, sq);
      const float2 t = __fmul2_rn(y, f2(-kLog2e, -kLog2e));
      const float2 e = f2(ex2_a(t.x), ex2_a(t.y));
      float2 k = __fmul2_rn(ood2, __ffma2_rn(e, m1, one));
      k.x = (y.x > 16.0f) ? ood2.x : k.x;
      k.y = (y.y > 16.0f) ? ood2.y : k.y;
      k.x = (y.x < 0.001f) ? sq.x * cf.x * fmaf(-0.5f, y.x, 1.0f) : k.x;
      k.y = (y.y < 0.001f) ? sq.y * cf.y * fmaf(-0.5f, y.y, 1.0f) : k.y;
      return k;
    }
  }
}

// one 32-column group against the warp's rows; csum: the warp's sums of the columns (COLS; a row block's own
// columns take none), two sums of half the rows in turn: kept apart in the two planes of csum when compensated
// (the tile's end adds all halves and warps in two-sums), added up otherwise.  Errors of v against FP64, one FP32
// number per row block and column -> this (one-sided): 33,001 Vatistas-2 1.25e-7 -> 1.20e-7 (1.23e-7), 131,072
// Gaussian patch 2.77e-8 -> 2.64e-8 (2.60e-8); time of the 1M patch 183.3 -> 185.6 ms.  Four sums of eight steps
// each: 1.14e-7 and 2.60e-8, 189.6 ms.
// zrow: this thread's rows' radius terms in shared memory (FORM 2).
template <int CORE, int FORM, bool COLS, bool COMP, int NP>
__device__ __forceinline__ void sym_group(const SymGroup& grp, int lane, const SymUni& q,
                                          const float2 (&nx)[NP], const float2 (&ny)[NP], const float2 (&g)[NP],
                                          const float* __restrict__ zrow, float2 (&u)[NP], float2 (&vn)[NP],
                                          float2* csum) {
  float cu = 0.0f, cv = 0.0f;
#pragma unroll 1
  for (int s0 = 0; s0 < SYM_GRP; s0 += SYM_GRP / 2) {
    if (COLS && s0) {                              // the first half's sums, at the lanes half a group away
      csum[lane ^ (SYM_GRP / 2)] = make_float2(cu, cv);
      cu = cv = 0.0f;
    }
#pragma unroll 4
    for (int s = s0; s < s0 + SYM_GRP / 2; ++s) {
      float2 su = f2(0.0f, 0.0f), sv = f2(0.0f, 0.0f);   // this step's rows
      const int col = lane ^ s;
      const float4 c = grp.xy[col];
      const float2 cx = f2(c.x, c.y), cy = f2(c.z, c.w), cg = grp.g[col];
      float2 cz = f2(0.0f, 0.0f);
      if constexpr (FORM == 2) cz = grp.z[col];
#pragma unroll
      for (int p = 0; p < NP; ++p) {
        const float2 dx = __fadd2_rn(cx, nx[p]);
        const float2 dy = __fadd2_rn(cy, ny[p]);
        float2 zz = f2(q.us2, q.us2);
        if constexpr (FORM == 2)
          zz = __fadd2_rn(cz, f2(zrow[(2 * p) * SYM_THREADS], zrow[(2 * p + 1) * SYM_THREADS]));
        // Rosenhead-Moore takes d^2 + s^2 in the same two operations
        const float2 d2 = __ffma2_rn(dx, dx, CORE == CORE_RM ? __ffma2_rn(dy, dy, zz) : __fmul2_rn(dy, dy));
        const float2 k = sym_core<CORE, FORM>(d2, zz, q);
        const float2 rr = __fmul2_rn(cg, k);
        u[p] = __ffma2_rn(rr, dy, u[p]);
        vn[p] = __ffma2_rn(rr, dx, vn[p]);
        if constexpr (!COLS) continue;
        const float2 rc = __fmul2_rn(g[p], k);
        su = (p == 0) ? __fmul2_rn(rc, dy) : __ffma2_rn(rc, dy, su);
        sv = (p == 0) ? __fmul2_rn(rc, dx) : __ffma2_rn(rc, dx, sv);
      }
      if constexpr (!COLS) continue;
      // hand the column's sums to the lane that meets it next (after the last step: to its own)
      const int m = (s ^ (s + 1)) & 31;
      cu = __shfl_xor_sync(0xffffffffu, cu + (su.x + su.y), m);
      cv = __shfl_xor_sync(0xffffffffu, cv + (sv.x + sv.y), m);
    }
  }
  if constexpr (COLS && COMP) {
    csum[SYM_TILE + lane] = make_float2(cu, cv);
  } else if constexpr (COLS) {
    __syncwarp();
    const float2 h = csum[lane];
    csum[lane] = make_float2(h.x + cu, h.y + cv);
  }
}

// CTAs per SM: 128 registers a thread for four row pairs, 255 for eight
constexpr int sym_occ(int np) { return np == 8 ? 2 : 4; }

template <int CORE, bool COMP, int NP>
__global__ void __launch_bounds__(SYM_THREADS, sym_occ(NP)) p2p_sym_kernel(const SymArgs a) {
  constexpr int GPB = sym_gpb(NP), ROWS = sym_rows(NP);
  constexpr bool MASKED = CORE == CORE_GAUSS || CORE == CORE_CEXP;
  wait_for_previous();
  __shared__ SymGroup tile[NSTAGE][SYM_TG];
  constexpr int PLANES = COMP ? 2 : 1;
  __shared__ float2 csum[SYM_THREADS / 32][PLANES * SYM_TILE];   // per-warp column sums of the tile
  __shared__ float zrow[2 * NP * SYM_THREADS];
  __shared__ __align__(8) uint64_t bar[NSTAGE];
  __shared__ int s_range;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  if (tid == 0) {
    for (int s = 0; s < NSTAGE; ++s) mbar_init(&bar[s], 1);
    fence_mbar_init();
  }
  __syncthreads();
  const bool unif = CORE == CORE_SING || ~a.meta[0] == a.meta[1];
  SymUni q;
  q.us2 = unif ? 2.0f * radius_term(CORE, __uint_as_float(a.meta[1])) : 0.0f;
  q.ucf = __frcp_rn(q.us2);
  q.cfl = -q.ucf * kLog2e;
  // far when every pair has d^2/s^2 > 16 (Gaussian) or (d/s)^3 > 16 (compact exponential), 1 % margin, with the largest
  // radius for both: every pair's own limit lies below, where its core gives the same bits.  Sets of varying radii then
  // gain from their order too (Gaussian 30,001 in order, radii 0.6 to 1.4 times the mean: 405 us near only, 289 so, 352
  // unsorted; 131,072 5841 -> 3555)
  q.lim = (CORE == CORE_CEXP ? 6.4131f : 16.16f) * (unif ? q.us2 : 2.0f * max_radius_term(CORE, a.meta[1]));

  uint32_t kt = 0;                                 // tiles consumed: barrier phase
  for (;;) {
    if (tid == 0) s_range = atomicAdd(a.counter, 1);
    __syncthreads();
    const int range = *static_cast<volatile int*>(&s_range);
    if (range >= a.nrange) break;
    int pos = sym_range_begin(a, range);
    const int end = sym_range_begin(a, range + 1);
    int k = sym_block_of(a, pos);
    for (; pos < end; ++k) {
      const int kbeg = sym_prefix(a, k), kend = min(end, sym_prefix(a, k + 1));
      const int blk = a.blk0 + k;
      const int g0 = GPB * blk + (pos - kbeg);          // first column group of this piece
      const int ng = kend - pos;
      const int gdiag = GPB * (blk + 1);                // groups below this are the block's own
      const int ntile = (ng + SYM_TG - 1) / SYM_TG;
      pos = kend;
      auto fetch = [&](int t, int st) {                     // thread 0
        const int cnt = min(SYM_TG, ng - t * SYM_TG);
        const uint32_t bytes = (uint32_t)(cnt * sizeof(SymGroup));
        mbar_arrive_expect_tx(&bar[st], bytes);
        bulk_g2s(&tile[st][0], a.grp + (g0 + t * SYM_TG), bytes, &bar[st]);
      };
      if (tid == 0) {
        fence_proxy_async_smem();
        for (int s = 0; s < NSTAGE && s < ntile; ++s) fetch(s, (kt + s) % NSTAGE);
      }
      float2 nx[NP], ny[NP], g[NP], u[NP], vn[NP], hu[NP], lu[NP], hv[NP], lv[NP];
      float bx0 = 3.0e38f, bx1 = -3.0e38f, by0 = 3.0e38f, by1 = -3.0e38f;
      const int row0 = blk * ROWS + warp * 64 * NP + lane;
#pragma unroll
      for (int p = 0; p < NP; ++p) {
        float4 w[2];
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          // the 32 rows of (p, h) are one group
          const SymGroup& r = a.grp[blk * GPB + warp * 2 * NP + 2 * p + h];
          const float4 xy = r.xy[lane];
          w[h] = make_float4(xy.x, xy.z, r.g[lane].x, r.z[lane].x);
          if (row0 + (2 * p + h) * 32 < a.n) {
            bx0 = fminf(bx0, w[h].x); bx1 = fmaxf(bx1, w[h].x);
            by0 = fminf(by0, w[h].y); by1 = fmaxf(by1, w[h].y);
          }
          if (!unif) zrow[(2 * p + h) * SYM_THREADS + tid] = w[h].w;   // read by this thread alone
        }
        nx[p] = f2(-w[0].x, -w[1].x);
        ny[p] = f2(-w[0].y, -w[1].y);
        g[p] = f2(w[0].z, w[1].z);
        u[p] = vn[p] = hu[p] = lu[p] = hv[p] = lv[p] = f2(0.0f, 0.0f);
      }
      if (MASKED) {
        for (int o = 16; o > 0; o >>= 1) {
          bx0 = fminf(bx0, __shfl_xor_sync(0xffffffffu, bx0, o));
          bx1 = fmaxf(bx1, __shfl_xor_sync(0xffffffffu, bx1, o));
          by0 = fminf(by0, __shfl_xor_sync(0xffffffffu, by0, o));
          by1 = fmaxf(by1, __shfl_xor_sync(0xffffffffu, by1, o));
        }
      }
      for (int t = 0; t < ntile; ++t, ++kt) {
        const int st = kt % NSTAGE;
        const bool ok = mbar_wait_bounded(&bar[st], (kt / NSTAGE) & 1u, WAIT_TRIES);
        if (__syncthreads_or(!ok)) {
          if (tid == 0) {
            record_failure(a.status, DEV_ERR_TIMEOUT, 240 + st, (int)kt, range);
            for (int s = 0; s < NSTAGE; ++s) (void)mbar_wait_bounded(&bar[(kt + s) % NSTAGE], ((kt + s) / NSTAGE) & 1u, WAIT_TRIES);
          }
          return;
        }
        const int cnt = min(SYM_TG, ng - t * SYM_TG);
        for (int b = 0; b < cnt; ++b) {
          const SymGroup& grp = tile[st][b];
          bool far = false;
          if constexpr (MASKED) {
            const float4 c = grp.xy[lane];
            const float ex = fmaxf(0.0f, fmaxf(bx0 - c.x, c.x - bx1));
            const float ey = fmaxf(0.0f, fmaxf(by0 - c.z, c.z - by1));
            // a NaN coordinate takes the near form
            far = __all_sync(0xffffffffu, fmaf(ex, ex, ey * ey) > q.lim);
          }
          auto run = [&](auto cols) {
            constexpr bool COLS = decltype(cols)::value;
            if (MASKED && far) sym_group<CORE, MASKED ? 0 : 1, COLS, COMP, NP>(grp, lane, q, nx, ny, g, zrow + tid, u, vn, csum[warp] + b * SYM_GRP);
            else if (!unif) sym_group<CORE, 2, COLS, COMP, NP>(grp, lane, q, nx, ny, g, zrow + tid, u, vn, csum[warp] + b * SYM_GRP);
            else sym_group<CORE, 1, COLS, COMP, NP>(grp, lane, q, nx, ny, g, zrow + tid, u, vn, csum[warp] + b * SYM_GRP);
          };
          if (g0 + t * SYM_TG + b < gdiag) run(std::false_type{});
          else run(std::true_type{});
          if (COMP || b == cnt - 1) {              // plain sums fold once per tile
#pragma unroll
            for (int p = 0; p < NP; ++p) {
              two_sum2(hu[p], lu[p], u[p]);
              two_sum2(hv[p], lv[p], vn[p]);
              u[p] = vn[p] = f2(0.0f, 0.0f);
            }
          }
        }
        __syncthreads();                           // the tile is consumed, its column sums are complete
        if (tid == 0 && t + NSTAGE < ntile) {
          fence_proxy_async_smem();
          fetch(t + NSTAGE, st);
        }
        // the next tile's sums are written after the barrier that opens it
        const int c0 = (g0 + t * SYM_TG) * SYM_GRP;
        for (int c = tid; c < cnt * SYM_GRP; c += SYM_THREADS) {
          if (c0 + c < gdiag * SYM_GRP || c0 + c >= a.n) continue;
          const size_t at = sym_base(a, k) + (c0 + c - sym_first(a, k));
          if constexpr (COMP) {
            float2 hi = csum[0][c], lo = f2(0.0f, 0.0f);
#pragma unroll
            for (int w = 0; w < SYM_THREADS / 32; ++w)
#pragma unroll
              for (int h = w ? 0 : 1; h < PLANES; ++h) two_sum2(hi, lo, csum[w][h * SYM_TILE + c]);
            static_cast<float4*>(a.colpart)[at] = make_float4(hi.x, lo.x, hi.y, lo.y);
          } else {
            const float2 s0 = csum[0][c], s1 = csum[1][c], s2 = csum[2][c], s3 = csum[3][c];
            static_cast<float2*>(a.colpart)[at] = make_float2((s0.x + s1.x) + (s2.x + s3.x), (s0.y + s1.y) + (s2.y + s3.y));
          }
        }
      }
      float2* rp = a.rowpart + (size_t)(range + k) * 2 * ROWS;
#pragma unroll
      for (int p = 0; p < NP; ++p) {
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const int i = warp * 64 * NP + (2 * p + h) * 32 + lane;
          rp[i] = h ? make_float2(hu[p].y, lu[p].y) : make_float2(hu[p].x, lu[p].x);
          rp[ROWS + i] = h ? make_float2(hv[p].y, lv[p].y) : make_float2(hv[p].x, lv[p].x);
        }
      }
    }
    __syncthreads();
  }
}

}  // namespace obs
