// tree.cu -- O(N log N) velocity of vortex particles: a treecode over Hilbert-ordered sources.
//
// The reference's execution environment names a Barnes-Hut summation (summation_t barneshut,
// src/ExecEnv.h:26-31) that it never runs internally; an external build reaches onbody's
// treecode through external_vel_solver_* (src/Influence.h:31-38, 74-98).  This is that
// summation on the GPU, for the velocity (results_t velonly) of every core:
//
//   * sources are put in Hilbert order (bin_order.cu); a leaf is a run of 32 consecutive sources
//     (one warp), a node at level L+1 groups 4 consecutive nodes of level L, up to one root;
//   * each node keeps its bounding box, a centre c (the box centre), a radius rho bounding
//     |z_j - c| over its sources, the largest radius term of its sources, and P multipole
//     coefficients b_k = sum_j G_j ((z_j - c)/rho)^k (complex; normalised by rho so that every
//     power lies in the unit disc) -- formed by warp reductions at the leaves and shifted up the
//     levels with the binomial theorem ((z - c')/rho' = s (z - c)/rho + t, |s| + |t| <= 1);
//   * one warp takes 64 Hilbert-consecutive targets, two per lane in f32x2 register pairs, and
//     walks the tree with a stack, up to 32 nodes (one per lane) at a time: a node is evaluated
//     through its expansion,
//        sum_j G_j / (z - z_j) = (1/(z - c)) sum_k b_k w^k,   w = rho/(z - c),
//     when rho <= theta (|z - c| - r) for the warp's target box (r its half diagonal), so |w|
//     <= theta and the truncation after P terms is below theta^P/(1 - theta) of the node's
//     sum |G_j|/|z - z_j| (a node farther away stops at the first term count whose |w|^p is below
//     both theta^P / 4 and 2^-26: about half of 24 terms on average; the second one keeps distant nodes at
//     FP32's precision where a caller asks for few terms); and only when every (target, source) pair of the
//     node lies in the core's far regime, where the core is 1/d^2: for the Gaussian and the compact exponential
//     that is the reference's own cut-off (d^2/s^2 > 16, (d/s)^3 > 16: the far branch IS 1/d^2,
//     src/CoreFunc.h:119-131), for the singular core always, and for Rosenhead-Moore,
//     Winckelmans-Leonard and the Vatistas cores where the core differs from 1/d^2 by less
//     than 2^-24 relative.  Other nodes open; at a leaf the pairs are summed directly with the
//     core (core_eval, as the direct kernels).
//
// With u + i v = i conj(F), F = sum_j G_j / (z - z_j): u = Im F, v = Re F (unscaled, as the
// direct sums; finalize_vels semantics optional).  Per-node contributions are accumulated with
// two-sums.  The last groups, all of a small set, split their nodes over two or four warps, every
// one of them walking the same tree and taking its share in turn.  Results are deterministic: the traversal
// order is a function of the inputs.
//
// 1M Gaussian patch, self interaction: 4.1 ms (44 ms in Morton order with 32 targets per warp and
// every node at full order).  Most of the 44 ms was a tail: a run of targets or sources across one
// of the Morton curve's jumps has a box the size of the domain, and its warp opened nearly every
// leaf (twenty times the mean cost in a sample of such groups, more at worst); along the Hilbert
// curve the worst group costs 1.7 times the mean and the mean group accepts half as many nodes.
// What is left is the near leaves (about 170 per group, three quarters of the instructions): issue
// active 60 %, FMA pipe 64 %, MUFU 50 %.  Sorting, tree and extrema take 0.3 ms.
#include <algorithm>
#include <cmath>
#include <cstring>
#include <vector>

#include "obs_context.h"
#include "obs_device.cuh"

namespace obs {

namespace {

constexpr int TREE_LEAF = 32;        // sources per leaf: one warp
constexpr int TREE_FAN = 4;          // children per node
constexpr int TREE_PMAX = 32;        // coefficient stride per node (largest order)
constexpr int TREE_MAXLEV = 16;      // 32 * 4^15 sources
constexpr int TREE_WARPS = 4;        // warps per block (leaf, up and evaluation kernels)
constexpr int TREE_STACK = 576;      // traversal stack entries per warp
constexpr int TREE_RESERVE = 64;     // of these, kept for taking nodes one at a time: > 1 + 3 * TREE_MAXLEV
constexpr int TREE_FINE = 32768;     // more points than this are sorted on the 4096 x 4096 grid
constexpr int TREE_LEVBITS = 26;     // stack entry: level << 26 | index within the level
constexpr double kTreeInv2Pi = 0.15915494309189535;   // 0.5/pi, finalize_vels (src/ElementBase.h:216)

// binomial coefficients for the upward shifts (exact in double, rounded once)
struct Binomials {
  float v[TREE_PMAX][TREE_PMAX];
  constexpr Binomials() : v() {
    for (int k = 0; k < TREE_PMAX; ++k) {
      double c = 1.0;
      for (int m = 0; m < TREE_PMAX; ++m) {
        v[k][m] = m <= k ? (float)c : 0.0f;
        c = c * (double)(k - m) / (double)(m + 1);
      }
    }
  }
};
__constant__ constexpr Binomials c_binom;

struct TreeNodes {
  float4* geo;       // (cx, cy, rho, zmax)
  float4* box;       // (xmin, ymin, xmax, ymax)
  float4* coef;      // [node][TREE_PMAX] (re, re, im, im): twice for the packed evaluation
};

struct TreeArgs {
  const float4* sp4; // sources in Hilbert order: (x, y, radius term, strength)
  int ns;
  const float* tx;   // targets in Hilbert order (tr: radius, null for field points)
  const float* ty;
  const float* tr;
  const int* tperm;  // caller's index of the k-th sorted target
  int nt;
  float* tu;
  float* tv;
  TreeNodes nodes;
  int nlev;
  int lev_off[TREE_MAXLEV];
  int lev_cnt[TREE_MAXLEV];
  int P;
  float theta;
  float lterm;       // log2 of the smaller of theta^P / 4 and 2^-26: a node stops at the first p with p log2|w| below it
  int one, two;      // blocks with a warp per target group, then blocks with two, then four
  int finalize;
  double fsx, fsy;
  int* status;
  const unsigned* meta;   // radius extrema: [2] ~min, [3] max of the sources; [4], [5] of the targets
};

__device__ __forceinline__ float warp_min(float v) {
  for (int o = 16; o > 0; o >>= 1) v = fminf(v, __shfl_xor_sync(0xffffffffu, v, o));
  return v;
}
__device__ __forceinline__ float warp_max(float v) {
  for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
  return v;
}
__device__ __forceinline__ float warp_add(float v) {
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// leaves: one warp per 32 sorted sources; also packs each source as (x, y, radius term, G)
__global__ void __launch_bounds__(TREE_WARPS * 32) tree_leaf_kernel(const float* sx, const float* sy, const float* sr,
                                                                    const float* sg, int ns, int core, float4* sp4,
                                                                    TreeNodes nd, int nleaf, int P) {
  wait_for_previous();
  const int leaf = (int)((blockIdx.x * blockDim.x + threadIdx.x) >> 5);
  const int lane = threadIdx.x & 31;
  if (leaf >= nleaf) return;                        // warp-uniform
  const int i = leaf * TREE_LEAF + lane;
  const bool v = i < ns;
  const float inf = __int_as_float(0x7f800000);
  const float x = v ? sx[i] : 0.0f, y = v ? sy[i] : 0.0f;
  const float z = (v && sr) ? radius_term(core, sr[i]) : 0.0f;
  const float g = v ? sg[i] : 0.0f;
  if (v) sp4[i] = make_float4(x, y, z, g);
  const float x0 = warp_min(v ? x : inf), x1 = warp_max(v ? x : -inf);
  const float y0 = warp_min(v ? y : inf), y1 = warp_max(v ? y : -inf);
  const float zmax = warp_max(z);
  const float cx = 0.5f * (x0 + x1), cy = 0.5f * (y0 + y1);
  const float dx = x - cx, dy = y - cy;
  const float rho = warp_max(v ? sqrtf(dx * dx + dy * dy) : 0.0f);
  const float rn = rho > 0.0f ? rho : 1.0f;
  const float wr = v ? dx / rn : 0.0f, wi = v ? dy / rn : 0.0f;
  float pr = g, pi = 0.0f;                          // G w^k
  float4* cf = nd.coef + (size_t)leaf * TREE_PMAX;
  for (int k = 0; k < P; ++k) {
    const float sr_ = warp_add(pr), si_ = warp_add(pi);
    if (lane == 0) cf[k] = make_float4(sr_, sr_, si_, si_);
    const float t = pr * wr - pi * wi;
    pi = pr * wi + pi * wr;
    pr = t;
  }
  if (lane == 0) {
    nd.geo[leaf] = make_float4(cx, cy, rho, zmax);
    nd.box[leaf] = make_float4(x0, y0, x1, y1);
  }
}

// One level up: a block per parent, a warp per child (children 4q .. 4q+3 of the level below); the
// children's shifted coefficients are added in two-sums, in child order (in plain sums the v of a 200,000-particle
// patch is 3.4e-8 off FP64, not 3.2e-8).  The levels above the leaves are small
// and wait on latency: with one warp per parent going through its children in turn, and the powers
// by repeated multiplication, a level took 25 us (eight of them 240 us of the 1M patch).
static_assert(TREE_WARPS == TREE_FAN, "a warp per child");
__global__ void __launch_bounds__(TREE_WARPS * 32) tree_up_kernel(TreeNodes nd, int off_c, int cnt_c, int off_p, int P) {
  __shared__ float sp[TREE_WARPS][TREE_PMAX];
  __shared__ float2 tp[TREE_WARPS][TREE_PMAX];
  __shared__ float2 cc[TREE_WARPS][TREE_PMAX];
  __shared__ float2 sum[TREE_WARPS][TREE_PMAX];
  const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
  wait_for_previous();
  const int q = blockIdx.x;
  const int c0 = q * TREE_FAN, nc = min(TREE_FAN, cnt_c - c0);
  const bool have = w < nc;                         // warp-uniform
  if (have && lane < P) {
    const float4 b = nd.coef[(size_t)(off_c + c0 + w) * TREE_PMAX + lane];
    cc[w][lane] = make_float2(b.x, b.z);
  }
  float x0 = __int_as_float(0x7f800000), y0 = x0, x1 = -x0, y1 = -x0, zmax = 0.0f;
  for (int c = 0; c < nc; ++c) {
    const float4 b = nd.box[off_c + c0 + c];
    x0 = fminf(x0, b.x); y0 = fminf(y0, b.y); x1 = fmaxf(x1, b.z); y1 = fmaxf(y1, b.w);
    zmax = fmaxf(zmax, nd.geo[off_c + c0 + c].w);
  }
  const float cx = 0.5f * (x0 + x1), cy = 0.5f * (y0 + y1);
  float rho = 0.0f;
  for (int c = 0; c < nc; ++c) {
    const float4 gc = nd.geo[off_c + c0 + c];
    const float ex = gc.x - cx, ey = gc.y - cy;
    rho = fmaxf(rho, sqrtf(ex * ex + ey * ey) + gc.z);
  }
  const float rn = rho > 0.0f ? rho : 1.0f;
  float ar = 0.0f, ai = 0.0f, lr = 0.0f, li = 0.0f;
  if (have) {
    const float4 gc = nd.geo[off_c + c0 + w];
    // (z - c)/rn = s (z - c_child)/rho_child + t, |s| + |t| <= 1; lane m: s^m and t^m by squaring.  A child of
    // radius 0 (one source, or coincident ones) has no coefficient but the first, so s = 0 does for it; taken
    // as radius 1 its s^m = rn^-m left FP32's range in small parents, and inf times those zeros was NaN
    float s = gc.z / rn, tr = (gc.x - cx) / rn, ti = (gc.y - cy) / rn;
    float pws = 1.0f, pwr = 1.0f, pwi = 0.0f;
#pragma unroll
    for (int b = 0; b < 5; ++b) {
      if ((lane >> b) & 1) {
        pws *= s;
        const float t = pwr * tr - pwi * ti;
        pwi = pwr * ti + pwi * tr;
        pwr = t;
      }
      s *= s;
      const float t = tr * tr - ti * ti;
      ti = 2.0f * tr * ti;
      tr = t;
    }
    sp[w][lane] = pws;
    tp[w][lane] = make_float2(pwr, pwi);
  }
  __syncwarp();
  if (have && lane < P) {
#pragma unroll 4
    for (int m = 0; m <= lane; ++m) {
      const float2 b = cc[w][m];
      const float2 t = tp[w][lane - m];
      const float f = c_binom.v[lane][m] * sp[w][m];
      two_sum_acc(ar, lr, f * (b.x * t.x - b.y * t.y));
      two_sum_acc(ai, li, f * (b.x * t.y + b.y * t.x));
    }
  }
  sum[w][lane] = make_float2(ar + lr, ai + li);
  __syncthreads();
  if (w != 0) return;
  const int node = off_p + q;
  if (lane < P) {
    for (int c = 1; c < nc; ++c) {
      two_sum_acc(ar, lr, sum[c][lane].x);
      two_sum_acc(ai, li, sum[c][lane].y);
    }
    nd.coef[(size_t)node * TREE_PMAX + lane] = make_float4(ar + lr, ar + lr, ai + li, ai + li);
  }
  if (lane == 0) {
    nd.geo[node] = make_float4(cx, cy, rho, zmax);
    nd.box[node] = make_float4(x0, y0, x1, y1);
  }
}

// Every (target, source) pair with squared distance >= d2 and radius terms summing to at most
// zsum lies where the core is 1/d^2: exactly (the reference's far branches of the Gaussian and
// compact exponential cores, the singular core), or within 2^-24 relative.
template <int CORE>
__device__ __forceinline__ bool tree_far(float d2, float zsum) {
  if constexpr (CORE == CORE_SING) return d2 > 0.0f;
  else if constexpr (CORE == CORE_GAUSS) return d2 > 0.0f && d2 > 16.05f * zsum;          // d^2/s^2 > 16
  else if constexpr (CORE == CORE_CEXP) return d2 > 0.0f && d2 > 6.36f * zsum;            // (d/s)^3 > 16
  else if constexpr (CORE == CORE_RM) return d2 > 0.0f && d2 > 16777216.0f * zsum;        // s^2/d^2 < 2^-24
  else if constexpr (CORE == CORE_WL) return d2 > 0.0f && d2 > 4096.0f * zsum;            // (s^2/d^2)^2 < 2^-24
  else if constexpr (CORE == CORE_V2) return d2 > 0.0f && d2 * d2 > 8388608.0f * zsum;    // s^4/(2 d^4) < 2^-24
  else return d2 > 0.0f && d2 * d2 * d2 > 8388608.0f * zsum;                              // s^6/(3 d^6) < 2^-24
}

// a leaf's sources in shared memory, every value twice for the packed operands
struct TreeLeaf {
  float4 xy[TREE_LEAF];    // (-x, -x, -y, -y)
  float4 gz[TREE_LEAF];    // (-G, -G, z, z)
};

// sums of -G K dy (= u) and -G K dx (= -v) of a leaf's cnt sources at the lane's two targets
// FORM 0: every pair in the core's far regime; 1: any pair; 2: unif, and no pair inside x < 0.001 (most near
// leaves: without the select a million-particle patch takes 4.1 instead of 4.35 ms)
template <int CORE, bool THICK, int FORM>
__device__ __forceinline__ void tree_leaf_sum(const TreeLeaf& lf, int cnt, float2 tx, float2 ty, float2 tz, bool unif,
                                              float cf, float cfl, float2& au, float2& av) {
  float2 su[2] = {au, au}, sv[2] = {av, av};       // the odd and the even sources apart: half the rounding
  constexpr bool FAR = FORM == 0;
  if (!FAR && CORE == CORE_GAUSS && (FORM == 2 || unif)) {
    // (1 - e^-x)/d^2; x < 0.001 -> 1/s^2 (src/CoreFunc.h:111-181).  The reference's 1/d^2 for
    // x > 16 is within 1.2e-7 of this form, one ulp, so it needs no select here
    const float thr_small = -0.001f * kLog2e;
    const float2 cfl2 = f2(cfl, cfl), m1 = f2(-1.0f, -1.0f), one = f2(1.0f, 1.0f);
#pragma unroll 4
    for (int k0 = 0; k0 < cnt; k0 += 2)
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const float4 P = lf.xy[k0 + h], Q = lf.gz[k0 + h];
        const float2 dx = __fadd2_rn(tx, f2(P.x, P.y)), dy = __fadd2_rn(ty, f2(P.z, P.w));
        const float2 d2 = __ffma2_rn(dx, dx, __fmul2_rn(dy, dy));
        const float2 t = __fmul2_rn(d2, cfl2);
        const float2 ood2 = f2(rcp_a(d2.x), rcp_a(d2.y));
        const float2 ome = __ffma2_rn(f2(ex2_a(t.x), ex2_a(t.y)), m1, one);
        float2 K = __fmul2_rn(ood2, ome);
        if constexpr (FORM != 2) {
          K.x = (t.x > thr_small) ? cf : K.x;
          K.y = (t.y > thr_small) ? cf : K.y;
        }
        const float2 fn = __fmul2_rn(f2(Q.x, Q.y), K);
        su[h] = __ffma2_rn(fn, dy, su[h]);
        sv[h] = __ffma2_rn(fn, dx, sv[h]);
      }
  } else {
#pragma unroll 2
    for (int k0 = 0; k0 < cnt; k0 += 2)
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const float4 P = lf.xy[k0 + h], Q = lf.gz[k0 + h];
        const float2 dx = __fadd2_rn(tx, f2(P.x, P.y)), dy = __fadd2_rn(ty, f2(P.z, P.w));
        const float2 d2 = __ffma2_rn(dx, dx, __fmul2_rn(dy, dy));
        float K0, K1, B;
        if constexpr (FAR) {
          K0 = rcp_a(d2.x);
          K1 = rcp_a(d2.y);
        } else {
          core_eval<CORE, THICK, false, false>(d2.x, Q.z, tz.x, 0.0f, 0.0f, K0, B);
          core_eval<CORE, THICK, false, false>(d2.y, Q.z, tz.y, 0.0f, 0.0f, K1, B);
        }
        const float2 fn = __fmul2_rn(f2(Q.x, Q.y), f2(K0, K1));
        su[h] = __ffma2_rn(fn, dy, su[h]);
        sv[h] = __ffma2_rn(fn, dx, sv[h]);
      }
  }
  au = __fadd2_rn(su[0], su[1]);
  av = __fadd2_rn(sv[0], sv[1]);
}

template <int CORE, bool THICK>
__global__ void __launch_bounds__(TREE_WARPS * 32, 6) tree_eval_kernel(const TreeArgs a) {
  constexpr unsigned FULL = 0xffffffffu;
  __shared__ int stk_all[TREE_WARPS][TREE_STACK];
  __shared__ TreeLeaf leafs[TREE_WARPS];
  __shared__ float4 red[TREE_WARPS][64];
  const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
  wait_for_previous();
  int* stk = stk_all[w];
  TreeLeaf& lf = leafs[w];
  const int blk = blockIdx.x;
  const int split = blk < a.one ? 1 : (blk < a.one + a.two ? 2 : 4);
  const int part = w % split;
  const int grp = blk * 4 / split + w / split + (split > 1 ? 2 * a.one : 0) + (split > 2 ? a.one + a.two : 0);
  const bool live = grp * 64 < a.nt;                // warp-uniform
  const int i0 = grp * 64 + lane, i1 = i0 + 32;
  const bool v0 = live && i0 < a.nt, v1 = live && i1 < a.nt;
  const float inf = __int_as_float(0x7f800000);
  // a lane without a second (or first) target repeats a real one
  const int j0 = v0 ? i0 : a.nt - 1, j1 = v1 ? i1 : j0;
  const float2 tx = f2(a.tx[j0], a.tx[j1]), ty = f2(a.ty[j0], a.ty[j1]);
  const float2 tz = THICK ? f2(radius_term(CORE, a.tr[j0]), radius_term(CORE, a.tr[j1])) : f2(0.0f, 0.0f);
  // Gaussian with one radius for every source (and every target): the packed near leaf sums, with
  // the core's cut-offs on t = -x log2(e), x = d^2 / s^2
  bool gunif = false;
  float gcf = 0.0f, gcfl = 0.0f;
  if constexpr (CORE == CORE_GAUSS) {
    gunif = (~a.meta[2] == a.meta[3]) && (!THICK || ~a.meta[4] == a.meta[5]);
    if (gunif) {
      const float us2 = radius_term(CORE, __uint_as_float(a.meta[3])) +
                        (THICK ? radius_term(CORE, __uint_as_float(a.meta[5])) : 0.0f);
      gcf = __frcp_rn(us2);
      gcfl = -gcf * kLog2e;
    }
  }
  const float bx0 = warp_min(v0 ? fminf(tx.x, tx.y) : inf), bx1 = warp_max(v0 ? fmaxf(tx.x, tx.y) : -inf);
  const float by0 = warp_min(v0 ? fminf(ty.x, ty.y) : inf), by1 = warp_max(v0 ? fmaxf(ty.x, ty.y) : -inf);
  const float ztmax = warp_max(fmaxf(tz.x, tz.y));
  const float ctx_ = 0.5f * (bx0 + bx1), cty = 0.5f * (by0 + by1);
  const float rt = 0.5f * sqrtf((bx1 - bx0) * (bx1 - bx0) + (by1 - by0) * (by1 - by0));
  float2 hu = f2(0.0f, 0.0f), lu = hu, hv = hu, lv = hu;
  const int top = a.nlev - 1;
  if (lane == 0) stk[0] = top << TREE_LEVBITS;      // the root: one node by construction
  int sp = live ? 1 : 0;
  int turn = 0;                                     // nodes and leaves met so far, shared out in turn
  __syncwarp();
  while (sp > 0) {
    // up to 32 nodes off the stack, fewer when their children might not fit above the reserve
    const int take = max(1, min(min(sp, 32), (TREE_STACK - TREE_RESERVE - sp) / 3));
    const bool have = lane < take;
    const int e = have ? stk[sp - 1 - lane] : 0;
    sp -= take;
    const int lev = e >> TREE_LEVBITS, q = e & ((1 << TREE_LEVBITS) - 1);
    const int node = a.lev_off[lev] + q;
    const float4 gn = a.nodes.geo[node];
    const float4 bn = a.nodes.box[node];
    const float gx = fmaxf(0.0f, fmaxf(bn.x - bx1, bx0 - bn.z));
    const float gy = fmaxf(0.0f, fmaxf(bn.y - by1, by0 - bn.w));
    const float dmin2 = gx * gx + gy * gy;
    const float ex = gn.x - ctx_, ey = gn.y - cty;
    const float sep = sqrtf(ex * ex + ey * ey) - rt;
    const bool far = tree_far<CORE>(dmin2, gn.w + ztmax);
    const bool accept = have && sep > 0.0f && gn.z <= a.theta * sep && far;
    const bool leaf = have && !accept && lev == 0;
    const bool open = have && !accept && lev > 0;
    // terms: |w| <= gn.z / sep for every target of the warp
    const float lw = lg2_a(gn.z * rcp_a(sep));      // <= log2(theta) where accepted; -inf for a point node
    const int terms = max(1, min(a.P, (int)ceilf(a.lterm * rcp_a(fminf(lw, -1.0e-3f)))));
    // children onto the stack, first child of the first node on top
    const int c0 = q * TREE_FAN;
    const int nc = open ? min(c0 + TREE_FAN, a.lev_cnt[lev - 1]) - c0 : 0;
    int incl = nc;
    for (int o = 1; o < 32; o <<= 1) {
      const int t = __shfl_up_sync(FULL, incl, o);
      if (lane >= o) incl += t;
    }
    const int total = __shfl_sync(FULL, incl, 31);
    if (sp + total > TREE_STACK) {                  // cannot happen (take); recorded, not taken
      if (lane == 0) record_failure(a.status, DEV_ERR_BOUNDS, 1100, grp, sp);
      break;
    }
    __syncwarp();                                   // every lane has read its entry
    for (int c = 0; c < nc; ++c) stk[sp + total - (incl - nc) - 1 - c] = ((lev - 1) << TREE_LEVBITS) | (c0 + c);
    sp += total;
    __syncwarp();
    for (unsigned m = __ballot_sync(FULL, accept); m; m &= m - 1) {
      if (turn++ % split != part) continue;
      // F = (1/(z - c)) sum_k b_k w^k, w = rn/(z - c); u += Im F, v += Re F
      const int b = __ffs(m) - 1;
      const float4* cf = a.nodes.coef + (size_t)__shfl_sync(FULL, node, b) * TREE_PMAX;
      const float rho = __shfl_sync(FULL, gn.z, b);
      const float rn = rho > 0.0f ? rho : 1.0f;
      const float cx = -__shfl_sync(FULL, gn.x, b), cy = -__shfl_sync(FULL, gn.y, b);
      const int p = __shfl_sync(FULL, terms, b);
      const float2 dx = __fadd2_rn(tx, f2(cx, cx)), dy = __fadd2_rn(ty, f2(cy, cy));
      const float2 d2 = __ffma2_rn(dx, dx, __fmul2_rn(dy, dy));
      const float2 inv = f2(rcp_a(d2.x), rcp_a(d2.y));
      const float2 ri = __fmul2_rn(f2(rn, rn), inv);
      const float2 wr = __fmul2_rn(ri, dx), nwi = __fmul2_rn(ri, dy);
      const float2 wi = f2(-nwi.x, -nwi.y);
      float2 hr = f2(0.0f, 0.0f), hi = hr;
#pragma unroll 4
      for (int k = p - 1; k >= 0; --k) {
        const float4 c = cf[k];
        const float2 t = __ffma2_rn(hr, wr, __ffma2_rn(hi, nwi, f2(c.x, c.y)));
        hi = __ffma2_rn(hr, wi, __ffma2_rn(hi, wr, f2(c.z, c.w)));
        hr = t;
      }
      // (dx - i dy) h / d^2
      const float2 fr = __fmul2_rn(__ffma2_rn(dx, hr, __fmul2_rn(dy, hi)), inv);
      const float2 dyn = f2(-dy.x, -dy.y);
      const float2 fi = __fmul2_rn(__ffma2_rn(dx, hi, __fmul2_rn(dyn, hr)), inv);
      two_sum2(hu, lu, fi);
      two_sum2(hv, lv, fr);
    }
    // leaves: direct sums, with the core or -- when every pair lies in the core's far regime, the
    // leaf being too close for its expansion -- with the far form 1/d^2 the core takes there
    const unsigned farm = __ballot_sync(FULL, far), outm = __ballot_sync(FULL, gunif && dmin2 * gcf > 0.00101f);
    for (unsigned m = __ballot_sync(FULL, leaf); m; m &= m - 1) {
      if (turn++ % split != part) continue;
      const int b = __ffs(m) - 1;
      const int s0 = __shfl_sync(FULL, q, b) * TREE_LEAF;
      const int cnt = min(TREE_LEAF, a.ns - s0);
      __syncwarp();
      {
        const float4 s = a.sp4[s0 + min(lane, cnt - 1)];
        const float g = lane < cnt ? -s.w : 0.0f;   // an odd count: the last source again, without strength
        lf.xy[lane] = make_float4(-s.x, -s.x, -s.y, -s.y);
        lf.gz[lane] = make_float4(g, g, s.z, s.z);
      }
      __syncwarp();
      float2 au = f2(0.0f, 0.0f), av = au;
      if ((farm >> b) & 1u) tree_leaf_sum<CORE, THICK, 0>(lf, cnt, tx, ty, tz, gunif, gcf, gcfl, au, av);
      else if (CORE == CORE_GAUSS && ((outm >> b) & 1u))
        tree_leaf_sum<CORE, THICK, 2>(lf, cnt, tx, ty, tz, true, gcf, gcfl, au, av);
      else tree_leaf_sum<CORE, THICK, 1>(lf, cnt, tx, ty, tz, gunif, gcf, gcfl, au, av);
      two_sum2(hu, lu, au);
      two_sum2(hv, lv, f2(-av.x, -av.y));
    }
  }
  if (split > 1) {                                  // the group's warps, added in order by the first
    red[w][lane] = make_float4(hu.x, lu.x, hv.x, lv.x);
    red[w][32 + lane] = make_float4(hu.y, lu.y, hv.y, lv.y);
    __syncthreads();
    if (part != 0) return;
    for (int k = 1; k < split; ++k) {
      const float4 p = red[w + k][lane], r = red[w + k][32 + lane];
      two_sum2(hu, lu, f2(p.x, r.x));
      two_sum2(hv, lv, f2(p.z, r.z));
      lu = __fadd2_rn(lu, f2(p.y, r.y));
      lv = __fadd2_rn(lv, f2(p.w, r.w));
    }
  }
  const double f = a.finalize ? kTreeInv2Pi : 1.0;
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    if (!(h ? v1 : v0)) continue;
    const int i = h ? i1 : i0;
    const int o = a.tperm ? a.tperm[i] : i;
    if ((unsigned)o >= (unsigned)a.nt) continue;    // never taken: tperm is a permutation
    const double su = (double)(h ? hu.y : hu.x) + (double)(h ? lu.y : lu.x);
    const double sv = (double)(h ? hv.y : hv.x) + (double)(h ? lv.y : lv.x);
    a.tu[o] = (float)(((double)a.tu[o] + su) * f + (a.finalize ? a.fsx : 0.0));
    a.tv[o] = (float)(((double)a.tv[o] + sv) * f + (a.finalize ? a.fsy : 0.0));
  }
}

template <int CORE>
cudaError_t tree_eval_core(bool thick, const TreeArgs& a, int grid, cudaStream_t st) {
  if (thick) launch_early(tree_eval_kernel<CORE, true>, grid, TREE_WARPS * 32, st, a);
  else launch_early(tree_eval_kernel<CORE, false>, grid, TREE_WARPS * 32, st, a);
  return cudaGetLastError();
}

cudaError_t tree_eval(int core, bool thick, const TreeArgs& a, int grid, cudaStream_t st) {
  switch (core) {
    case CORE_RM: return tree_eval_core<CORE_RM>(thick, a, grid, st);
    case CORE_GAUSS: return tree_eval_core<CORE_GAUSS>(thick, a, grid, st);
    case CORE_V2: return tree_eval_core<CORE_V2>(thick, a, grid, st);
    case CORE_WL: return tree_eval_core<CORE_WL>(thick, a, grid, st);
    case CORE_V3: return tree_eval_core<CORE_V3>(thick, a, grid, st);
    case CORE_SING: return tree_eval_core<CORE_SING>(thick, a, grid, st);
    default: return tree_eval_core<CORE_CEXP>(thick, a, grid, st);
  }
}

size_t al256(size_t b) { return (b + 255) & ~(size_t)255; }

BinCurve tree_curve(int n) { return n > TREE_FINE ? BIN_HILBERT12 : BIN_HILBERT8; }

}  // namespace

// Device arrays in; accumulates into tu, tv (finalize_vels semantics with OBS_FLAG_FINALIZE).
int run_tree(obs_context* ctx, int core, int flags, double fsx, double fsy, double theta, int order, int ns,
             const float* sx, const float* sy, const float* sr, const float* ss, int nt, const float* tx,
             const float* ty, const float* tr, float* tu, float* tv) {
  if (ns == 0 || nt == 0) return OBS_OK;
  const int P = std::min(order, TREE_PMAX);
  // levels: leaves, then groups of four up to one root
  int lev_cnt[TREE_MAXLEV], lev_off[TREE_MAXLEV], nlev = 0, total = 0;
  int cnt = (ns + TREE_LEAF - 1) / TREE_LEAF;
  for (;;) {
    if (nlev == TREE_MAXLEV) return OBS_ERR_UNSUPPORTED;
    lev_cnt[nlev] = cnt;
    lev_off[nlev] = total;
    total += cnt;
    ++nlev;
    if (cnt == 1) break;
    cnt = (cnt + TREE_FAN - 1) / TREE_FAN;
  }
  const bool same = (tx == sx && ty == sy && tr == sr);
  const int nmax = std::max(ns, nt);
  const size_t S = (size_t)ns, T = (size_t)nt;
  const size_t o_bin = 0;
  const size_t o_sperm = o_bin + al256(bin_scratch_bytes(nmax));
  const size_t o_s = o_sperm + al256(S * 4);               // x y r g (4 S floats), then (x, y, z, g)
  const size_t o_p4 = o_s + 4 * al256(S * 4);
  const size_t o_tperm = o_p4 + al256(S * 16);
  const size_t o_t = o_tperm + al256(T * 4);               // x y r (3 T floats)
  const size_t o_geo = o_t + 3 * al256(T * 4);
  const size_t o_box = o_geo + al256((size_t)total * sizeof(float4));
  const size_t o_coef = o_box + al256((size_t)total * sizeof(float4));
  const size_t o_meta = o_coef + al256((size_t)total * TREE_PMAX * sizeof(float4));
  const size_t bytes = o_meta + 256;
  int s = ctx->work.ensure(bytes, ctx->stream);
  if (s) return s;
  char* W = ctx->work.as<char>();
  int* sperm = reinterpret_cast<int*>(W + o_sperm);
  float* bs[4];
  for (int k = 0; k < 4; ++k) bs[k] = reinterpret_cast<float*>(W + o_s + k * al256(S * 4));
  float4* sp4 = reinterpret_cast<float4*>(W + o_p4);
  int* tperm = reinterpret_cast<int*>(W + o_tperm);
  float* bt[3];
  for (int k = 0; k < 3; ++k) bt[k] = reinterpret_cast<float*>(W + o_t + k * al256(T * 4));
  TreeNodes nd{reinterpret_cast<float4*>(W + o_geo), reinterpret_cast<float4*>(W + o_box),
               reinterpret_cast<float4*>(W + o_coef)};
  cudaStream_t st = ctx->stream;
  cudaError_t e = cudaSuccess;
  int launches = 0;
  // radius extrema for the Gaussian's uniform-radius leaf sums (zeroed: "not uniform"), before the sort so that
  // the kernels from there to the evaluation follow one another directly
  unsigned* meta = reinterpret_cast<unsigned*>(W + o_meta);
  if ((e = cudaMemsetAsync(meta, 0, 6 * sizeof(unsigned), st)) != cudaSuccess) return cuda_status(e);
  if (core == CORE_GAUSS && sr) {
    if ((e = p2p_launch_target_meta(sr, ns, meta, st)) != cudaSuccess) return cuda_status(e);
    ++launches;
    if (tr && tr == sr && nt == ns) {
      e = cudaMemcpyAsync(meta + 4, meta + 2, 2 * sizeof(unsigned), cudaMemcpyDeviceToDevice, st);
      if (e != cudaSuccess) return cuda_status(e);
    } else if (tr) {
      if ((e = p2p_launch_target_meta(tr, nt, meta + 2, st)) != cudaSuccess) return cuda_status(e);
      ++launches;
    }
  }
  if (e == cudaSuccess) e = bin_order(sx, sy, ns, W + o_bin, sperm, st, &launches, tree_curve(ns));
  if (e == cudaSuccess) e = bin_gather(sperm, sx, sy, sr, ss, ns, bs[0], bs[1], sr ? bs[2] : nullptr, bs[3], st,
                                       &launches);
  if (e != cudaSuccess) return cuda_status(e);
  const float *ttx = bs[0], *tty = bs[1], *ttr = tr ? bs[2] : nullptr;
  const int* tp = sperm;
  if (!same) {
    e = bin_order(tx, ty, nt, W + o_bin, tperm, st, &launches, tree_curve(nt));
    if (e == cudaSuccess) e = bin_gather(tperm, tx, ty, tr, nullptr, nt, bt[0], bt[1], tr ? bt[2] : nullptr, nullptr, st,
                                         &launches);
    if (e != cudaSuccess) return cuda_status(e);
    ttx = bt[0]; tty = bt[1]; ttr = tr ? bt[2] : nullptr;
    tp = tperm;
  }
  const int tb = TREE_WARPS * 32;
  launch_early(tree_leaf_kernel, (lev_cnt[0] + TREE_WARPS - 1) / TREE_WARPS, tb, st, bs[0], bs[1], sr ? bs[2] : nullptr,
               bs[3], ns, core, sp4, nd, lev_cnt[0], P);
  ++launches;
  for (int l = 0; l + 1 < nlev; ++l) {
    launch_early(tree_up_kernel, lev_cnt[l + 1], tb, st, nd, lev_off[l], lev_cnt[l], lev_off[l + 1], P);
    ++launches;
  }
  if ((e = cudaGetLastError()) != cudaSuccess) return cuda_status(e);
  TreeArgs a;
  std::memset(&a, 0, sizeof(a));
  a.sp4 = sp4; a.ns = ns;
  a.tx = ttx; a.ty = tty; a.tr = ttr; a.tperm = tp; a.nt = nt;
  a.tu = tu; a.tv = tv;
  a.nodes = nd;
  a.nlev = nlev;
  for (int l = 0; l < nlev; ++l) { a.lev_off[l] = lev_off[l]; a.lev_cnt[l] = lev_cnt[l]; }
  a.P = P;
  a.theta = (float)theta;
  a.lterm = (float)std::min((double)P * std::log2(theta) - 2.0, -26.0);
  a.finalize = (flags & OBS_FLAG_FINALIZE) ? 1 : 0;
  a.fsx = fsx; a.fsy = fsy;
  a.status = ctx->d_status;
  a.meta = meta;
  // A warp per 64 targets, but four for the last 6 groups per SM (one resident wave of blocks) and two for the 6
  // per SM before them: whole groups started last would leave most of the chip idle at the end.  Every split warp
  // walks the tree again: measured with four for the last 0, 6, 12, 24, 48 per SM, 1,000,000 targets take 4.35, 4.31,
  // 4.34, 4.44, 4.68 ms and 300,000 1.44, 0.97, 1.04, 1.11, 1.15 ms; with none of two, 60,000 take 0.44 ms, not 0.33.
  const int groups = (nt + 63) / 64;
  constexpr int FOUR = 6, TWO = 6;
  const int four = std::min(groups, FOUR * ctx->num_sms), two = std::min(groups - four, TWO * ctx->num_sms);
  a.one = (groups - four - two) / 4;
  a.two = (groups - four - 4 * a.one) / 2;
  e = tree_eval(core, tr != nullptr, a, groups - 3 * a.one - a.two, st);
  ++launches;
  ctx->launches += launches;
  return cuda_status(e);
}

}  // namespace obs
