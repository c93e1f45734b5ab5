// adjoint_small.cu -- VJP gathers of small sets in one launch: the sums of adjoint.cu, organised like
// p2p_small.cu with four owners per block, every pair with its own radii.
#include <cfloat>

#include "adjoint.h"
#include "obs_context.h"
#include "p2p_kernel.cuh"
#include "small_sum.cuh"

namespace obs {

namespace {

constexpr int SMA_T = 4;                    // owners per block

struct SmallAdjArgs {
  int no;
  const float* ox; const float* oy; const float* orad; const float* og;
  int ne;
  const float* ex; const float* ey; const float* er; const float* eg; const float* elu; const float* elv;
  float* gx; float* gy; float* gg;
};

// SELF: owners and elements are one set (owner k, element j, d = x_k - x_j); otherwise the owners are
// sources and the elements targets with cotangents (d = x_target - x_source)
template <int CORE, bool SELF, bool THICK, bool COMP>
__global__ void __launch_bounds__(SML_THREADS) adj_small_kernel(const SmallAdjArgs a) {
  __shared__ float2 red[SML_WARPS][3 * SMA_T];
  __shared__ float2 tot[3 * SMA_T];
  const int o0 = blockIdx.x * SMA_T;
  float ox[SMA_T], oy[SMA_T], oz[SMA_T], og[SMA_T], olu[SMA_T], olv[SMA_T], acc[3][SMA_T];
  float2 r[3][SMA_T];
#pragma unroll
  for (int t = 0; t < SMA_T; ++t) {
    const int i = min(o0 + t, a.no - 1);
    ox[t] = a.ox[i];
    oy[t] = a.oy[i];
    oz[t] = a.orad ? radius_term(CORE, a.orad[i]) : 0.0f;
    // a radius of 0 would make the Gaussian's derivative 1/s^2 times e^-x = inf times 0 at any distance
    if (CORE == CORE_GAUSS && oz[t] == 0.0f) oz[t] = FLT_MIN;
    og[t] = SELF ? a.og[i] : 0.0f;
    olu[t] = SELF ? a.elu[i] : 0.0f;
    olv[t] = SELF ? a.elv[i] : 0.0f;
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      acc[c][t] = 0.0f;
      r[c][t] = make_float2(0.0f, 0.0f);
    }
  }
  int k = 0;
  for (int j = threadIdx.x; j < a.ne; j += SML_THREADS, ++k) {
    if (COMP && k == COMP_BLOCK) {
#pragma unroll
      for (int c = 0; c < 3; ++c)
#pragma unroll
        for (int t = 0; t < SMA_T; ++t) {
          two_sum_acc(r[c][t].x, r[c][t].y, acc[c][t]);
          acc[c][t] = 0.0f;
        }
      k = 0;
    }
    const float x = a.ex[j], y = a.ey[j], lu = a.elu[j], lv = a.elv[j];
    const float z = a.er ? radius_term(CORE, a.er[j]) : 0.0f;
    const float g = SELF ? a.eg[j] : 0.0f;
#pragma unroll
    for (int t = 0; t < SMA_T; ++t) {
      const float dx = SELF ? ox[t] - x : x - ox[t], dy = SELF ? oy[t] - y : y - oy[t];
      const float d2 = fmaf(dx, dx, dy * dy);
      float K, B;
      if constexpr (SELF) core_eval<CORE, true, true, false>(d2, z, oz[t], 0.0f, 0.0f, K, B);
      else core_eval<CORE, THICK, true, false>(d2, oz[t], z, 0.0f, 0.0f, K, B);
      const float qe = fmaf(lv, dx, -lu * dy);
      const float wu = SELF ? fmaf(g, olu[t], -og[t] * lu) : lu;
      const float wv = SELF ? fmaf(g, olv[t], -og[t] * lv) : lv;
      const float q = SELF ? fmaf(dx, wv, -dy * wu) : qe;
      const float bq = B * q;
      acc[0][t] += fmaf(K, wv, bq * dx);
      acc[1][t] += fmaf(-K, wu, bq * dy);
      acc[2][t] = fmaf(SELF ? -qe : qe, K, acc[2][t]);
    }
  }
#pragma unroll
  for (int c = 0; c < 3; ++c)
#pragma unroll
    for (int t = 0; t < SMA_T; ++t) two_sum_acc(r[c][t].x, r[c][t].y, acc[c][t]);
  sml_block_sum<3, SMA_T>(r, red, tot);
  const int i = o0 + threadIdx.x;
  if (threadIdx.x >= SMA_T || i >= a.no) return;
  // scale by 1/(2 pi); the source side also by -G_j
  double s[3];
#pragma unroll
  for (int c = 0; c < 3; ++c) {
    const float2 v = tot[c * SMA_T + threadIdx.x];
    s[c] = ((double)v.x + (double)v.y) * kInv2Pi;
  }
  const double f = SELF ? 1.0 : -(double)a.og[i];
  if (a.gx) a.gx[i] = (float)((double)a.gx[i] + s[0] * f);
  if (a.gy) a.gy[i] = (float)((double)a.gy[i] + s[1] * f);
  if (a.gg) a.gg[i] = (float)((double)a.gg[i] + s[2]);
}

template <int CORE>
void adj_core(bool self, bool thick, bool comp, const SmallAdjArgs& a, int grid, cudaStream_t st) {
  auto k = self ? (comp ? adj_small_kernel<CORE, true, true, true> : adj_small_kernel<CORE, true, true, false>)
           : thick ? (comp ? adj_small_kernel<CORE, false, true, true> : adj_small_kernel<CORE, false, true, false>)
                   : (comp ? adj_small_kernel<CORE, false, false, true> : adj_small_kernel<CORE, false, false, false>);
  k<<<grid, SML_THREADS, 0, st>>>(a);
}

}  // namespace

// Where one launch beats the tiled gathers (compensated, this / those, us).  A block walks all the elements for its
// four owners, so few owners with many elements leave most of the chip idle, where the tiled gathers split the
// elements; and many owners with few elements end in one block sum for every four.
//   Gaussian: 1 owner x 32,768 57 / 92, x 100,000 164 / 115; 8 owners x 20,000 37 / 103, x 100,000 161 / 221, x
//     300,000 475 / 341, x 1,000,000 1566 / 1001; 26,000 owners x 1,000 66 / 67, 30,000 x 400 58 / 62, 32,768 x
//     1,000 81 / 72, x 3,000 147 / 163; self 3,000 40 / 211, 9,000 175 / 246.
//   Vatistas-2 (cheaper pairs): 8 x 32,768 65 / 85, x 100,000 190 / 116, x 1,000,000 1850 / 523; 2,000 x 20,000
//     82 / 90, x 32,768 134 / 127; 4,000 x 20,000 123 / 118; 14,000 x 1,800 43 / 45, 18,000 x 200 32 / 29, 20,000 x
//     1,500 51.7 / 53.6, 26,000 x 1,000 58 / 44, 32,768 x 200 56 / 31; self 9,000 128 / 153.
//   Vatistas-2, plain (half the registers): 8 x 50,000 54 / 94, 4,000 x 20,000 70 / 116, 22,000 x 200 31 / 33, x 1,500
//     46 / 54, 26,000 x 200 35 / 34, 32,768 x 1,000 56 / 52.
bool adjoint_small_applies(const obs_context* ctx, int core, int accum, int no, int ne) {
  if (ctx->kernel_variant != OBS_VARIANT_AUTO || ctx->target_order != OBS_ORDER_AUTO) return false;
  const double pairs = (double)no * ne;
  if (core == CORE_GAUSS) return pairs <= 1.0e8 && ne <= (no < 4 ? 65536 : 131072) && no <= (ne < 1200 ? 30720 : 32768);
  if (accum != OBS_COMPENSATED) return pairs <= 1.0e8 && ne <= (no < 4 ? 65536 : 131072) && no <= 24576;
  return no <= (ne < 1200 ? 16384 : 20480) && (ne <= 16384 ? pairs <= 1.0e8 : ne <= 40960 && pairs <= 6.0e7);
}

int run_adjoint_small(obs_context* ctx, int core, int accum, int mode, int no, const float* ox, const float* oy,
                      const float* orad, const float* og, int ne, const float* ex, const float* ey, const float* er,
                      const float* eg, const float* elu, const float* elv, float* gx, float* gy, float* gg) {
  const SmallAdjArgs a{no, ox, oy, orad, og, ne, ex, ey, er, eg, elu, elv, gx, gy, gg};
  const bool self = mode == 1, thick = self || er != nullptr, comp = accum == OBS_COMPENSATED;
  const int grid = (no + SMA_T - 1) / SMA_T;
  timing_main_begin(ctx);
  switch (core) {
    case CORE_RM: adj_core<CORE_RM>(self, thick, comp, a, grid, ctx->stream); break;
    case CORE_GAUSS: adj_core<CORE_GAUSS>(self, thick, comp, a, grid, ctx->stream); break;
    case CORE_V2: adj_core<CORE_V2>(self, thick, comp, a, grid, ctx->stream); break;
    case CORE_WL: adj_core<CORE_WL>(self, thick, comp, a, grid, ctx->stream); break;
    case CORE_V3: adj_core<CORE_V3>(self, thick, comp, a, grid, ctx->stream); break;
    case CORE_SING: adj_core<CORE_SING>(self, thick, comp, a, grid, ctx->stream); break;
    default: adj_core<CORE_CEXP>(self, thick, comp, a, grid, ctx->stream); break;
  }
  ctx->launches++;
  timing_main_end(ctx);
  return cuda_status(cudaGetLastError());
}

}  // namespace obs
