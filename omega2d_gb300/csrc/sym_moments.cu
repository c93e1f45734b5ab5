// sym_moments.cu -- launch planning of the gradient, vorticity, shear and self-VJP sums that evaluate
// each unordered pair once (sym_moments.cuh), their packing and the reduction of their partials.
#include <algorithm>
#include <cstring>

#include "adjoint.h"
#include "obs_context.h"
#include "sym_moments.cuh"

namespace obs {

namespace {

template <bool VJP>
__global__ void mom_pack_kernel(const float* x, const float* y, const float* r, const float* g, const float* lu,
                                const float* lv, const int* perm, int n, int npad, MomGroup<VJP>* out, unsigned* meta) {
  wait_for_previous();
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  int j = (i < n && perm) ? perm[i] : i;
  if ((unsigned)j >= (unsigned)n) j = 0;          // never taken for i < n: perm is a permutation
  const float rr = i < n ? r[j] : 0.0f;
  if (i < npad) {
    const bool real = i < n;
    const float X = real ? x[j] : SYM_FAR, Y = real ? y[j] : SYM_FAR;
    const float G = real ? g[j] : 0.0f, z = real ? radius_term(CORE_GAUSS, rr) : 1.0f;
    MomGroup<VJP>& o = out[i / SYM_GRP];
    const int l = i % SYM_GRP;
    o.xy[l] = make_float4(X, X, Y, Y);
    o.g[l] = make_float2(G, G);
    o.z[l] = make_float2(z, z);
    if constexpr (VJP) {
      const float U = real ? lu[j] : 0.0f, V = real ? lv[j] : 0.0f;
      o.l[l] = make_float4(-U, -U, V, V);
    }
  }
  fold_extrema_block(i < n ? __float_as_uint(rr) : ~0u, i < n ? __float_as_uint(rr) : 0u, meta);
}

__device__ __forceinline__ void df_add(float2& a, float2 b) {
  two_sum_acc(a.x, a.y, b.x);
  a.y += b.y;
}

struct MomOut {
  P2PArgs p;               // gradient-type results
  const int* perm;         // VJP: gradients of position and strength, accumulated (any may be null)
  float* gx; float* gy; float* gg;
};

// As sym_reduce_kernel: a particle's pieces of its own row block, then the row blocks before it, four
// threads each every fourth, then the passes before; the last pass forms and stores the results.
constexpr int MOM_RED_T = 64, MOM_RED_SUB = 4;
template <class OP, int RES, bool COMP>
__global__ void __launch_bounds__(MOM_RED_T * MOM_RED_SUB) mom_reduce_kernel(const MomArgs m, const MomOut o) {
  constexpr int NC = OP::NF + OP::NN, ROWS = mom_rows<OP>();
  wait_for_previous();
  __shared__ float2 red[MOM_RED_SUB][NC][MOM_RED_T];
  const SymArgs& a = m.s;
  const int l = threadIdx.x % MOM_RED_T, sub = threadIdx.x / MOM_RED_T;
  const int j = blockIdx.x * MOM_RED_T + l;
  const int jb = j / ROWS;
  float2 s[NC];
#pragma unroll
  for (int c = 0; c < NC; ++c) s[c] = f2(0.0f, 0.0f);
  if (j < a.n) {
    const int k = jb - a.blk0;
    const int kc = min(a.nblk, k);                 // row blocks of this pass before the particle's own
#pragma unroll 4
    for (int q = sub; q < kc; q += MOM_RED_SUB)
#pragma unroll
      for (int c = 0; c < NC; ++c) {
        const size_t at = NC * sym_base(a, q) + (size_t)c * sym_width(a, q) + (j - sym_first(a, q));
        if constexpr (COMP) df_add(s[c], __ldcg(static_cast<const float2*>(m.colpart) + at));
        else two_sum_acc(s[c].x, s[c].y, __ldcg(static_cast<const float*>(m.colpart) + at));
      }
    // the column sees velocity, X, Y and the strength term with the other sign
#pragma unroll
    for (int c = 0; c < NC; ++c)
      if (OP::VJP || c < 2) s[c] = f2(-s[c].x, -s[c].y);
    if (k >= 0 && k < a.nblk) {
      int r0, r1;
      sym_ranges_of(a, k, r0, r1);
      const float2* rp = m.rowpart + (size_t)k * NC * ROWS + (j - jb * ROWS);
#pragma unroll 2
      for (int r = r0 + sub; r <= r1; r += MOM_RED_SUB)
#pragma unroll
        for (int c = 0; c < NC; ++c) df_add(s[c], __ldcg(rp + ((size_t)r * NC + c) * ROWS));
    }
  }
#pragma unroll
  for (int c = 0; c < NC; ++c) red[sub][c][l] = s[c];
  __syncthreads();
  if (sub != 0 || j >= a.n) return;
#pragma unroll
  for (int c = 0; c < NC; ++c) {
    for (int q = 1; q < MOM_RED_SUB; ++q) df_add(s[c], red[q][c][l]);
    if (!a.first) df_add(s[c], m.run[(size_t)c * a.npad + j]);
    if (!a.last) m.run[(size_t)c * a.npad + j] = s[c];
  }
  if (!a.last) return;
  double v[NC];
#pragma unroll
  for (int c = 0; c < NC; ++c) v[c] = (double)s[c].x + (double)s[c].y;
  if constexpr (OP::VJP) {
    const int i = o.perm ? o.perm[j] : j;
    if ((unsigned)i >= (unsigned)a.n) return;      // never taken: perm is a permutation
    if (o.gx) o.gx[i] = (float)((double)o.gx[i] - 2.0 * v[0] * kInv2Pi);
    if (o.gy) o.gy[i] = (float)((double)o.gy[i] - 2.0 * v[1] * kInv2Pi);
    if (o.gg) o.gg[i] = (float)((double)o.gg[i] + v[2] * kInv2Pi);
  } else {
    double c[NComp<RES>::v];
    c[0] = v[0];
    c[1] = -v[1];
    if constexpr (RES == RES_GRAD) {
      c[2] = -2.0 * v[2];
      c[3] = v[4] + 2.0 * v[3];
      c[4] = 2.0 * v[3] - v[4];
    } else if constexpr (RES == RES_VORT) {
      c[2] = 2.0 * v[2];
    } else {
      c[2] = v[2];
    }
    store_target<RES>(o.p, j, c);
  }
}

constexpr int MOM_OCC = 4;                            // CTAs per SM (__launch_bounds__: 128 registers)
constexpr size_t MOM_COL_BYTES = (size_t)1 << 30;     // column partials held at once

// the set x, y, r, g (and cotangents) on itself; out.p (but perm and nt) or out.gx.. set by the caller
template <class OP, int RES>
int run_moments(obs_context* ctx, bool comp, int n, const float* x, const float* y, const float* r, const float* g,
                const float* lu, const float* lv, MomOut out, size_t off) {
  constexpr int NC = OP::NF + OP::NN, ROWS = mom_rows<OP>();
  using Group = MomGroup<OP::VJP>;
  cudaStream_t st = ctx->stream;
  const int nblk = (n + ROWS - 1) / ROWS;
  const int npad = nblk * ROWS;
  const int ngrp = (n + SYM_GRP - 1) / SYM_GRP;
  const int slots = MOM_OCC * ctx->num_sms;
  // Binned vs not, us (narrow to wide cores): 11,500 gradient 155-176 vs 149-156, VJP 151-168 vs 137-144; 17,000 every
  // one of them faster, gradient 236 vs 272, vorticity 164 vs 205, shear 175 vs 203, VJP 241 vs 270.  The order brings a
  // particle's near ones into the same FP32 sums (17,001 of a patch, du/dx 1.0e-7 off FP64 instead of 5.2e-8), so the
  // line is no lower than the one-sided kernels' 3e8; the VJP's is 7e8 (25,000 of a patch, dL/dy 1.40e-7 instead of
  // 1.29e-7; 437 vs 559 us).  Near units of a binned set cost three times the far ones and come
  // together: in ranges of two or more units, not 32, 28,544 take 498-505 us, not 760 (gradient, wide core), 45,000
  // 1029, not 1191
  const bool binned = (double)n * n >= (OP::VJP ? 7e8 : 3e8);
  MomArgs m;
  std::memset(&m, 0, sizeof(m));
  m.s.n = n; m.s.npad = npad; m.s.ngrp = ngrp; m.s.gpb = mom_gpb<OP>(); m.s.least = binned ? 2 : 32;
  m.s.many = 1024;
  const size_t col = NC * (comp ? sizeof(float2) : sizeof(float));
  auto al = [](size_t b) { return (b + 255) & ~(size_t)255; };
  const size_t o_grp = off + 256, o_run = o_grp + (size_t)(npad / SYM_GRP) * sizeof(Group);
  size_t o_col, o_row, o_perm, o_sort, cap = MOM_COL_BYTES / col;
  for (;; cap /= 2) {                              // as run_p2p_sym
    const SymScratch need = sym_scratch(m.s, nblk, slots, cap);
    o_col = o_run + (need.passes > 1 ? al((size_t)npad * NC * sizeof(float2)) : 0);
    o_row = o_col + al(need.cols * col);
    o_perm = o_row + need.rows * NC * ROWS * sizeof(float2);
    o_sort = o_perm + (binned ? al((size_t)n * sizeof(int)) : 0);
    const int s = ctx->work.grow(o_sort + (binned ? bin_scratch_bytes(n) : 0), ctx->pair_scratch, st);
    if (s == OBS_OK) break;
    if (need.passes == nblk) return s;
  }
  WorkHeader* h = ctx->work.as<WorkHeader>(off);
  int* perm = binned ? ctx->work.as<int>(o_perm) : nullptr;
  Group* grp = ctx->work.as<Group>(o_grp);

  timing_begin(ctx);
  cudaError_t e = cudaMemsetAsync(h, 0, sizeof(WorkHeader), st);
  int nl = 0;
  if (e == cudaSuccess && binned) e = bin_order(x, y, n, ctx->work.as<char>(o_sort), perm, st, &nl, BIN_HILBERT8);
  if (e != cudaSuccess) return cuda_status(e);
  launch_early(mom_pack_kernel<OP::VJP>, (npad + 255) / 256, 256, st, x, y, r, g, lu, lv, perm, n, npad, grp, h->meta);
  ctx->launches += nl + 1;
  if ((e = cudaGetLastError()) != cudaSuccess) return cuda_status(e);

  m.s.counter = &h->counter;
  m.s.meta = h->meta;
  m.s.status = ctx->d_status;
  m.grp = grp;
  m.colpart = ctx->work.as<char>(o_col);
  m.rowpart = ctx->work.as<float2>(o_row);
  m.run = ctx->work.as<float2>(o_run);
  out.p.nt = n;
  out.p.perm = perm;
  out.perm = perm;

  timing_main_begin(ctx);
  for (; m.s.blk0 < nblk; m.s.blk0 += m.s.nblk) {
    sym_next_pass(m.s, nblk, slots, cap);
    if (!m.s.first && (e = cudaMemsetAsync(&h->counter, 0, sizeof(int), st)) != cudaSuccess) return cuda_status(e);
    const int grid = std::min(m.s.nrange, slots);
    if (comp) launch_early(sym_moments_kernel<OP, true>, grid, SYM_THREADS, st, m);
    else launch_early(sym_moments_kernel<OP, false>, grid, SYM_THREADS, st, m);
    if (m.s.last) timing_main_end(ctx);
    launch_early(comp ? mom_reduce_kernel<OP, RES, true> : mom_reduce_kernel<OP, RES, false>, (n + MOM_RED_T - 1) / MOM_RED_T,
                 MOM_RED_T * MOM_RED_SUB, st, m, out);
    ctx->launches += 2;
    if ((e = cudaGetLastError()) != cudaSuccess) return cuda_status(e);
  }
  timing_end(ctx);
  return OBS_OK;
}

}  // namespace

bool p2p_sym_res_applies(const obs_context* ctx, const P2PRequest& rq) {
  if (rq.result != RES_GRAD && rq.result != RES_VORT && rq.result != RES_SHEAR) return false;
  if (rq.core != CORE_GAUSS || ctx->kernel_variant != OBS_VARIANT_AUTO || ctx->target_order != OBS_ORDER_AUTO) return false;
  return rq.ns == rq.nt && rq.sx == rq.tx && rq.sy == rq.ty && rq.tr && rq.tr == rq.sr;
}

int run_p2p_sym_res(obs_context* ctx, const P2PRequest& rq) {
  MomOut o;
  std::memset(&o, 0, sizeof(o));
  o.p.out[0] = rq.tu; o.p.out[1] = rq.tv;
  for (int k = 0; k < 4; ++k) o.p.out[2 + k] = rq.extra[k];
  o.p.finalize = (rq.flags & OBS_FLAG_FINALIZE) ? 1 : 0;
  o.p.fsx = rq.fsx; o.p.fsy = rq.fsy;
  o.p.overwrite = rq.overwrite;
  const bool comp = rq.accum == OBS_COMPENSATED;
  if (rq.result == RES_GRAD) return run_moments<MomGrad, RES_GRAD>(ctx, comp, rq.nt, rq.sx, rq.sy, rq.sr, rq.ss, nullptr, nullptr, o, 0);
  if (rq.result == RES_VORT) return run_moments<MomVort, RES_VORT>(ctx, comp, rq.nt, rq.sx, rq.sy, rq.sr, rq.ss, nullptr, nullptr, o, 0);
  return run_moments<MomShear, RES_SHEAR>(ctx, comp, rq.nt, rq.sx, rq.sy, rq.sr, rq.ss, nullptr, nullptr, o, 0);
}

int run_adjoint_self_sym(obs_context* ctx, int accum, int n, const float* x, const float* y, const float* r,
                         const float* g, const float* lu, const float* lv, float* gx, float* gy, float* gg, size_t off) {
  MomOut o;
  std::memset(&o, 0, sizeof(o));
  o.gx = gx; o.gy = gy; o.gg = gg;
  return run_moments<MomVjp, RES_VEL>(ctx, accum == OBS_COMPENSATED, n, x, y, r, g, lu, lv, o, off);
}

}  // namespace obs
