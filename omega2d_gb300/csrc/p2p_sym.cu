// p2p_sym.cu -- launch planning of the self-interaction sums that evaluate each unordered pair
// once (p2p_sym.cuh), their packing and the reduction of their partials.
#include <algorithm>
#include <cstring>

#include "obs_context.h"
#include "p2p_sym.cuh"

namespace obs {

namespace {

// Particles in groups of 32 in processing order, padded to whole row blocks with far particles of
// zero strength, and the radius extrema (meta[0] = ~min, meta[1] = max bits).
__global__ void sym_pack_kernel(const float* x, const float* y, const float* r, const float* g, const int* perm, int n,
                                int npad, int core, SymGroup* out, unsigned* meta) {
  wait_for_previous();
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  int j = (i < n && perm) ? perm[i] : i;
  if ((unsigned)j >= (unsigned)n) j = 0;          // never taken for i < n: perm is a permutation
  const float rr = (i < n && r) ? r[j] : 0.0f;
  if (i < npad) {
    const bool real = i < n;
    const float X = real ? x[j] : SYM_FAR, Y = real ? y[j] : SYM_FAR;
    const float G = real ? g[j] : 0.0f, z = real ? radius_term(core, rr) : 1.0f;
    SymGroup& o = out[i / SYM_GRP];
    o.xy[i % SYM_GRP] = make_float4(X, X, Y, Y);
    o.g[i % SYM_GRP] = make_float2(G, G);
    o.z[i % SYM_GRP] = make_float2(z, z);
  }
  fold_extrema_block(i < n ? __float_as_uint(rr) : ~0u, i < n ? __float_as_uint(rr) : 0u, meta);
}

__device__ __forceinline__ void df_add(float& hi, float& lo, float bh, float bl) {
  two_sum_acc(hi, lo, bh);
  lo += bl;
}

// Adds a particle's partials of this pass (its row block's pieces, then the row blocks before its
// own, each in order) to its running sum; the last pass stores the result.  A block takes 64
// particles; eight threads share one, each every eighth partial, added up in thread order (with four ten
// steps of 20,000 particles take 20 us longer, with sixteen as long as with four).
constexpr int SYM_RED_T = 64, SYM_RED_SUB = 8;
template <bool COMP, int NP>
__global__ void __launch_bounds__(SYM_RED_T * SYM_RED_SUB) sym_reduce_kernel(const SymArgs a, const P2PArgs o) {
  constexpr int SYM_ROWS = sym_rows(NP);
  wait_for_previous();
  __shared__ float4 red[SYM_RED_SUB][SYM_RED_T];
  const int l = threadIdx.x % SYM_RED_T, sub = threadIdx.x / SYM_RED_T;
  const int j = blockIdx.x * SYM_RED_T + l;
  const int jb = j / SYM_ROWS;                     // the particle's row block (the same for all of a block)
  float4 s = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
  if (j < a.n) {
    const int k = jb - a.blk0;
    if (k >= 0 && k < a.nblk) {
      int r0, r1;
      sym_ranges_of(a, k, r0, r1);
      const float2* rp = a.rowpart + (size_t)k * 2 * SYM_ROWS + (j - jb * SYM_ROWS);
#pragma unroll 4
      for (int r = r0 + sub; r <= r1; r += SYM_RED_SUB) {
        const float2 u = __ldcg(rp + (size_t)r * 2 * SYM_ROWS), v = __ldcg(rp + (size_t)r * 2 * SYM_ROWS + SYM_ROWS);
        df_add(s.x, s.y, u.x, u.y);
        df_add(s.z, s.w, -v.x, -v.y);
      }
    }
    const int kc = min(a.nblk, jb - a.blk0);       // row blocks of this pass before the particle's own
#pragma unroll 8
    for (int m = sub; m < kc; m += SYM_RED_SUB) {
      const size_t at = sym_base(a, m) + (j - sym_first(a, m));
      if constexpr (COMP) {
        const float4 c = __ldcg(static_cast<const float4*>(a.colpart) + at);
        df_add(s.x, s.y, -c.x, -c.y);
        df_add(s.z, s.w, c.z, c.w);
      } else {
        const float2 c = __ldcg(static_cast<const float2*>(a.colpart) + at);
        two_sum_acc(s.x, s.y, -c.x);
        two_sum_acc(s.z, s.w, c.y);
      }
    }
  }
  red[sub][l] = s;
  __syncthreads();
  if (sub != 0 || j >= a.n) return;
  for (int q = 1; q < SYM_RED_SUB; ++q) {
    const float4 t = red[q][l];
    df_add(s.x, s.y, t.x, t.y);
    df_add(s.z, s.w, t.z, t.w);
  }
  if (!a.first) {
    const float4 t = a.run[j];
    df_add(s.x, s.y, t.x, t.y);
    df_add(s.z, s.w, t.z, t.w);
  }
  if (!a.last) {
    a.run[j] = s;
    return;
  }
  const double c[2] = {(double)s.x + (double)s.y, (double)s.z + (double)s.w};
  store_target<RES_VEL>(o, j, c);
}

// one pass: the sums, then their reduction
template <int CORE, int NP>
cudaError_t sym_launch(bool comp, const SymArgs& a, const P2PArgs& o, int grid, cudaStream_t st) {
  launch_early(comp ? p2p_sym_kernel<CORE, true, NP> : p2p_sym_kernel<CORE, false, NP>, grid, SYM_THREADS, st, a);
  launch_early(comp ? sym_reduce_kernel<true, NP> : sym_reduce_kernel<false, NP>, (a.n + SYM_RED_T - 1) / SYM_RED_T,
               SYM_RED_T * SYM_RED_SUB, st, a, o);
  return cudaGetLastError();
}

template <int NP>
cudaError_t sym_dispatch(int core, bool comp, const SymArgs& a, const P2PArgs& o, int grid, cudaStream_t st) {
  switch (core) {
    case CORE_RM: return sym_launch<CORE_RM, NP>(comp, a, o, grid, st);
    case CORE_GAUSS: return sym_launch<CORE_GAUSS, NP>(comp, a, o, grid, st);
    case CORE_V2: return sym_launch<CORE_V2, NP>(comp, a, o, grid, st);
    case CORE_WL: return sym_launch<CORE_WL, NP>(comp, a, o, grid, st);
    case CORE_V3: return sym_launch<CORE_V3, NP>(comp, a, o, grid, st);
    case CORE_SING: return sym_launch<CORE_SING, NP>(comp, a, o, grid, st);
    case CORE_CEXP: return sym_launch<CORE_CEXP, NP>(comp, a, o, grid, st);
    default: return cudaErrorInvalidValue;
  }
}

// Row pairs per thread: eight pass a column's sums on half as often per pair as four, but their row
// blocks are twice as large (8 vs 4: 20,000 Rosenhead-Moore, ten steps 1220 vs 1204 us; 30,000 Gaussian 297 vs 300,
// Vatistas-2 225 vs 231, with varying radii 237 vs 254; 33,001 of those 284 vs 306; 131,072 plain 3.23 vs 3.49 ms;
// 400,000 Gaussian 29.8 vs 31.2; the 1M patch 182 vs 194; 200,000 with varying Gaussian radii 13.2 vs 12.9)
int sym_np(int n) { return n >= 30000 ? 8 : 4; }

// Units of a range, not sorted or a large Gaussian set (4, 8 or 16: 0 to 8 % slower up to 80,000 particles); four where
// sorting put near and far units into runs (32 -> 4: Gaussian 36,000 352 -> 347 us, 50,000 682 -> 587, 60,000 954 ->
// 805, but 64,000 883 -> 905; compact exponential 30,001 354 -> 287, 64,000 1072 -> 961, 100,000 2118 -> 2124).  Sixteen ranges a CTA, not eight, balance the
// cores whose units differ from 256 units a CTA on (131,072 Gaussian 3568 -> 3464 us, 178,513 6514 -> 6269), the others
// from 1024 on (131,072 Vatistas-2 would take 3475, not 3411): their row partials are written and read twice as often.
constexpr int SYM_LEAST = 32;
constexpr size_t SYM_COL_BYTES = (size_t)1 << 30;     // column partials held at once

}  // namespace

// One set as sources and targets (the same arrays) with two-radius cores, from 6,709 particles (smaller sets take
// p2p_small.cu).  Measured against the one-sided kernels (compensated, calls back to back): 8,000 Vatistas-2 43 vs 58
// us, 10,000 Gaussian 61 vs 100, 20,000 Rosenhead-Moore 113 vs 164, 60,000 Vatistas-2 753 vs 1042, with varying radii
// 795 vs 1220; the 1M Gaussian patch 185.4 vs 249 ms.  An order or kernel variant asked for by name
// keeps the one-sided kernels.
bool p2p_sym_applies(const obs_context* ctx, const P2PRequest& rq) {
  if (rq.result != RES_VEL || ctx->kernel_variant != OBS_VARIANT_AUTO || ctx->target_order != OBS_ORDER_AUTO) return false;
  if (rq.ns != rq.nt || rq.sx != rq.tx || rq.sy != rq.ty) return false;
  if (rq.core != CORE_SING && (!rq.tr || rq.tr != rq.sr)) return false;
  return true;
}

int run_p2p_sym(obs_context* ctx, const P2PRequest& rq) {
  const int n = rq.nt;
  const bool comp = rq.accum == OBS_COMPENSATED;
  cudaStream_t st = ctx->stream;
  const int np = sym_np(n), rows = sym_rows(np);
  const int nblk = (n + rows - 1) / rows;
  const int npad = nblk * rows;
  const int ngrp = (n + SYM_GRP - 1) / SYM_GRP;
  const int slots = sym_occ(np) * ctx->num_sms;
  // The sort (eight launches, 60 us) pays once its ranges are fine enough to even out near and far units: at four units
  // a range, compensated with one radius, sorted vs not in us: Gaussian 16,000 110 vs 95, 22,000 166 vs 164, 25,000 192
  // vs 209, 36,000 347 vs 395, 50,000 587 vs 731, 60,000 805 vs 1033; compact exponential, whose near form costs twice
  // the Gaussian's, 16,000 126 vs 127, 20,000 160 vs 190, 36,000 377 vs 565, 60,000 859 vs 1491
  const bool gauss = rq.core == CORE_GAUSS, masked = gauss || rq.core == CORE_CEXP;
  const double pairs = (double)n * n;
  const bool binned = masked && pairs >= (gauss ? 6.25e8 : 3.24e8);
  SymArgs a;
  std::memset(&a, 0, sizeof(a));
  a.n = n; a.npad = npad; a.ngrp = ngrp; a.gpb = sym_gpb(np);
  a.least = !binned || (gauss && pairs >= 4e9) ? SYM_LEAST : 4;
  a.many = masked ? 8 * SYM_LEAST : 32 * SYM_LEAST;
  const size_t col = comp ? sizeof(float4) : sizeof(float2);
  auto al = [](size_t b) { return (b + 255) & ~(size_t)255; };
  const size_t o_pts = 256, o_run = o_pts + (size_t)(npad / SYM_GRP) * sizeof(SymGroup);
  size_t o_col, o_row, o_perm, o_sort, cap = SYM_COL_BYTES / col;
  // column partials of at most a pass's share; of half as much, down to one row block at a time, where the device has
  // no room
  for (;; cap /= 2) {
    const SymScratch m = sym_scratch(a, nblk, slots, cap);
    o_col = o_run + (m.passes > 1 ? al((size_t)npad * sizeof(float4)) : 0);
    o_row = o_col + al(m.cols * col);
    o_perm = o_row + m.rows * 2 * rows * sizeof(float2);
    o_sort = o_perm + (binned ? al((size_t)n * sizeof(int)) : 0);
    const int s = ctx->work.grow(o_sort + (binned ? bin_scratch_bytes(n) : 0), ctx->pair_scratch, st);
    if (s == OBS_OK) break;
    if (m.passes == nblk) return s;
  }
  WorkHeader* h = ctx->work.as<WorkHeader>(0);
  int* perm = binned ? ctx->work.as<int>(o_perm) : nullptr;

  timing_begin(ctx);
  cudaError_t e = cudaMemsetAsync(h, 0, sizeof(WorkHeader), st);
  int nl = 0;
  if (e == cudaSuccess && binned) e = bin_order(rq.sx, rq.sy, n, ctx->work.as<char>(o_sort), perm, st, &nl, BIN_HILBERT8);
  if (e != cudaSuccess) return cuda_status(e);
  launch_early(sym_pack_kernel, (npad + 255) / 256, 256, st, rq.sx, rq.sy, rq.sr, rq.ss, perm, n, npad, rq.core,
               ctx->work.as<SymGroup>(o_pts), h->meta);
  ctx->launches += nl + 1;
  if ((e = cudaGetLastError()) != cudaSuccess) return cuda_status(e);

  a.grp = ctx->work.as<SymGroup>(o_pts);
  a.counter = &h->counter;
  a.meta = h->meta;
  a.status = ctx->d_status;
  a.colpart = ctx->work.as<char>(o_col);
  a.rowpart = ctx->work.as<float2>(o_row);
  a.run = ctx->work.as<float4>(o_run);
  P2PArgs o;
  std::memset(&o, 0, sizeof(o));
  o.nt = n;
  o.perm = perm;
  o.out[0] = rq.tu; o.out[1] = rq.tv;
  o.finalize = (rq.flags & OBS_FLAG_FINALIZE) ? 1 : 0;
  o.fsx = rq.fsx; o.fsy = rq.fsy;
  o.overwrite = rq.overwrite;

  timing_main_begin(ctx);
  for (; a.blk0 < nblk; a.blk0 += a.nblk) {
    sym_next_pass(a, nblk, slots, cap);
    if (!a.first && (e = cudaMemsetAsync(&h->counter, 0, sizeof(int), st)) != cudaSuccess) return cuda_status(e);
    const int grid = std::min(a.nrange, slots);
    e = np == 8 ? sym_dispatch<8>(rq.core, comp, a, o, grid, st) : sym_dispatch<4>(rq.core, comp, a, o, grid, st);
    ctx->launches += 2;
    if (e != cudaSuccess) return cuda_status(e);
  }
  timing_main_end(ctx);
  timing_end(ctx);
  return OBS_OK;
}

}  // namespace obs
