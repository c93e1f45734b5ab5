// p2p_small_res.cu -- velocity with gradient, vorticity or shear of small sets in one launch: the
// organisation of p2p_small.cu with four targets per block and the pair forms of p2p_kernel.cuh
// (kernelug / kerneluw / kernelue, src/Kernels.h:112-231), every pair with its own radii.
#include <cfloat>
#include <cstring>

#include "obs_context.h"
#include "p2p_kernel.cuh"
#include "small_sum.cuh"

namespace obs {

namespace {

constexpr int SMR_T = 4;                    // targets per block

struct SmallResArgs {
  const float* sx; const float* sy; const float* sr; const float* ss;
  int ns;
  const float* tx; const float* ty; const float* tr;
};

template <int CORE, bool THICK, bool COMP, int RES>
__global__ void __launch_bounds__(SML_THREADS) p2p_small_res_kernel(const SmallResArgs a, const P2PArgs o) {
  constexpr int NC = NComp<RES>::v;
  __shared__ float2 red[SML_WARPS][NC * SMR_T];
  __shared__ float2 tot[NC * SMR_T];
  const int t0 = blockIdx.x * SMR_T;
  float tx[SMR_T], ty[SMR_T], tz[SMR_T], acc[NC][SMR_T];
  float2 r[NC][SMR_T];
#pragma unroll
  for (int t = 0; t < SMR_T; ++t) {
    const int i = min(t0 + t, o.nt - 1);
    tx[t] = a.tx[i];
    ty[t] = a.ty[i];
    tz[t] = THICK ? radius_term(CORE, a.tr[i]) : 0.0f;
#pragma unroll
    for (int c = 0; c < NC; ++c) {
      acc[c][t] = 0.0f;
      r[c][t] = make_float2(0.0f, 0.0f);
    }
  }
  int k = 0;
  for (int j = threadIdx.x; j < a.ns; j += SML_THREADS, ++k) {
    if (COMP && k == COMP_BLOCK) {
#pragma unroll
      for (int c = 0; c < NC; ++c)
#pragma unroll
        for (int t = 0; t < SMR_T; ++t) {
          two_sum_acc(r[c][t].x, r[c][t].y, acc[c][t]);
          acc[c][t] = 0.0f;
        }
      k = 0;
    }
    const float x = a.sx[j], y = a.sy[j], g = a.ss[j];
    float z = a.sr ? radius_term(CORE, a.sr[j]) : 0.0f;
    // a radius of 0 would make the Gaussian's derivative 1/s^2 times e^-x = inf times 0 at any distance
    if (CORE == CORE_GAUSS && z == 0.0f) z = FLT_MIN;
#pragma unroll
    for (int t = 0; t < SMR_T; ++t) {
      const float ndx = x - tx[t], ndy = y - ty[t];
      const float d2 = fmaf(ndx, ndx, ndy * ndy);
      float K, B = 0.0f;
      core_eval<CORE, THICK, true, false>(d2, z, tz[t], 0.0f, 0.0f, K, B);
      const float r2 = g * K, bb = g * B;
      acc[0][t] = fmaf(r2, ndy, acc[0][t]);
      acc[1][t] = fmaf(-r2, ndx, acc[1][t]);
      if constexpr (RES == RES_GRAD) {
        const float bx = bb * ndx;
        acc[2][t] = fmaf(bx, ndy, acc[2][t]);
        acc[3][t] += fmaf(bx, ndx, r2);
        acc[4][t] -= fmaf(bb * ndy, ndy, r2);
      } else if constexpr (RES == RES_VORT) {
        acc[2][t] += fmaf(bb, d2, 2.0f * r2);
      } else {
        acc[2][t] = fmaf(0.5f * fabsf(bb), d2, acc[2][t]);
      }
    }
  }
#pragma unroll
  for (int c = 0; c < NC; ++c)
#pragma unroll
    for (int t = 0; t < SMR_T; ++t) two_sum_acc(r[c][t].x, r[c][t].y, acc[c][t]);
  sml_block_sum<NC, SMR_T>(r, red, tot);
  const int i = t0 + threadIdx.x;
  if (threadIdx.x < SMR_T && i < o.nt) {
    double c[NC];
#pragma unroll
    for (int q = 0; q < NC; ++q) {
      const float2 s = tot[q * SMR_T + threadIdx.x];
      c[q] = (double)s.x + (double)s.y;
    }
    store_target<RES>(o, i, c);
  }
}

template <int CORE, int RES>
void res_launch(bool thick, bool comp, const SmallResArgs& a, const P2PArgs& o, int grid, cudaStream_t st) {
  auto k = thick ? (comp ? p2p_small_res_kernel<CORE, true, true, RES> : p2p_small_res_kernel<CORE, true, false, RES>)
                 : (comp ? p2p_small_res_kernel<CORE, false, true, RES> : p2p_small_res_kernel<CORE, false, false, RES>);
  k<<<grid, SML_THREADS, 0, st>>>(a, o);
}

template <int CORE>
void res_core(int res, bool thick, bool comp, const SmallResArgs& a, const P2PArgs& o, int grid, cudaStream_t st) {
  if (res == RES_GRAD) res_launch<CORE, RES_GRAD>(thick, comp, a, o, grid, st);
  else if (res == RES_VORT) res_launch<CORE, RES_VORT>(thick, comp, a, o, grid, st);
  else res_launch<CORE, RES_SHEAR>(thick, comp, a, o, grid, st);
}

}  // namespace

// Against the tiled kernels (compensated, this -> those, us): Gaussian gradient 1,000 52 -> 141, 5,000
// 85 -> 134, 9,000 177 -> 228, shear 9,000 124 -> 202; Vatistas-2 gradient 5,000 68 -> 84, 7,000 99 -> 96,
// 9,000 137 -> 127.  The compensated gradient's 128 registers leave two blocks per SM, so past the first wave and the second
// its sources count two and three times (sources x targets): Gaussian 26,000 x 1,800 107 -> 110, 32,768 x 1,217 131 ->
// 119, 18,000 x 3,000 108 -> 120, 22,000 x 2,433 140 -> 119, and 2,000 x 20,000 113 -> 103; Vatistas-2 18,000 x 1,800
// 62 -> 77, 22,000 x 1,217 78 -> 71, 14,000 x 3,000 63 -> 68, 18,000 x 2,433 92 -> 84, 500 x 9,000 42 -> 50,
// 1,000 x 20,000 83 -> 60.
bool p2p_small_res_applies(const obs_context* ctx, const P2PRequest& rq) {
  if (rq.result != RES_GRAD && rq.result != RES_VORT && rq.result != RES_SHEAR) return false;
  if (ctx->kernel_variant != OBS_VARIANT_AUTO || ctx->target_order != OBS_ORDER_AUTO) return false;
  const double limit = rq.core == CORE_GAUSS ? 8.2e7 : 4.5e7;
  int most_s = 32768, most_t = 20480;
  if (rq.result == RES_GRAD && rq.accum == OBS_COMPENSATED) {
    const int wave = 2 * SMR_T * ctx->num_sms;
    const bool gauss = rq.core == CORE_GAUSS;
    if (rq.nt > wave) most_s = rq.nt <= 2 * wave ? (gauss ? 28000 : 20000) : (gauss ? 20000 : 16384);
    most_t = gauss ? 16384 : 9728;
  }
  return (double)rq.ns * rq.nt <= limit && rq.ns <= most_s && rq.nt <= most_t;
}

int run_p2p_small_res(obs_context* ctx, const P2PRequest& rq) {
  const SmallResArgs a{rq.sx, rq.sy, rq.sr, rq.ss, rq.ns, rq.tx, rq.ty, rq.tr};
  P2PArgs o;
  std::memset(&o, 0, sizeof(o));
  o.nt = rq.nt;
  o.out[0] = rq.tu; o.out[1] = rq.tv;
  for (int k = 0; k < 4; ++k) o.out[2 + k] = rq.extra[k];
  o.finalize = (rq.flags & OBS_FLAG_FINALIZE) ? 1 : 0;
  o.fsx = rq.fsx; o.fsy = rq.fsy;
  o.overwrite = rq.overwrite;
  const bool thick = rq.tr != nullptr, comp = rq.accum == OBS_COMPENSATED;
  const int grid = (rq.nt + SMR_T - 1) / SMR_T;
  timing_begin(ctx);
  timing_main_begin(ctx);
  switch (rq.core) {
    case CORE_RM: res_core<CORE_RM>(rq.result, thick, comp, a, o, grid, ctx->stream); break;
    case CORE_GAUSS: res_core<CORE_GAUSS>(rq.result, thick, comp, a, o, grid, ctx->stream); break;
    case CORE_V2: res_core<CORE_V2>(rq.result, thick, comp, a, o, grid, ctx->stream); break;
    case CORE_WL: res_core<CORE_WL>(rq.result, thick, comp, a, o, grid, ctx->stream); break;
    case CORE_V3: res_core<CORE_V3>(rq.result, thick, comp, a, o, grid, ctx->stream); break;
    case CORE_SING: res_core<CORE_SING>(rq.result, thick, comp, a, o, grid, ctx->stream); break;
    default: res_core<CORE_CEXP>(rq.result, thick, comp, a, o, grid, ctx->stream); break;
  }
  ctx->launches++;
  timing_main_end(ctx);
  timing_end(ctx);
  return cuda_status(cudaGetLastError());
}

}  // namespace obs
