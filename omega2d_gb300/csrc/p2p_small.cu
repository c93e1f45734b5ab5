// p2p_small.cu -- velocity sums of small sets in one launch (points_affect_points,
// src/Influence.h:56-416, every core, thick targets or field points).
//
// The tiled kernels take four or five launches (clear, pack, extrema, sum, reduction) of about 4 us
// each, which is all the time a thousand particles need.  Here a block owns eight targets, in four
// f32x2 register pairs of every thread, and its threads stride over the sources, read straight from
// the caller's arrays (coalesced); the 256 threads' sums are added over lanes and warps
// (small_sum.cuh) and stored.  Nothing is staged, cleared or left
// for a second launch.  Every pair is evaluated one-sided with its own radii.
#include <cstring>

#include "obs_context.h"
#include "p2p_sym.cuh"
#include "small_sum.cuh"

namespace obs {

namespace {

constexpr int SML_T = 8;                    // targets per block

struct SmallArgs {
  const float* sx; const float* sy; const float* sr; const float* ss;
  int ns;
  const float* tx; const float* ty; const float* tr;
};

template <int CORE, bool THICK, bool COMP>
__global__ void __launch_bounds__(SML_THREADS) p2p_small_kernel(const SmallArgs a, const P2PArgs o) {
  constexpr int NP = SML_T / 2;
  __shared__ float2 red[SML_WARPS][2 * SML_T];
  __shared__ float2 tot[2 * SML_T];
  const int t0 = blockIdx.x * SML_T;
  float2 nx[NP], ny[NP], zt[NP], u[NP], vn[NP], hu[NP], lu[NP], hv[NP], lv[NP];
#pragma unroll
  for (int p = 0; p < NP; ++p) {
    const int i0 = min(t0 + 2 * p, o.nt - 1), i1 = min(t0 + 2 * p + 1, o.nt - 1);
    nx[p] = f2(-a.tx[i0], -a.tx[i1]);
    ny[p] = f2(-a.ty[i0], -a.ty[i1]);
    zt[p] = THICK ? f2(radius_term(CORE, a.tr[i0]), radius_term(CORE, a.tr[i1])) : f2(0.0f, 0.0f);
    u[p] = vn[p] = hu[p] = lu[p] = hv[p] = lv[p] = f2(0.0f, 0.0f);
  }
  const SymUni q{};
  int k = 0;
  for (int j = threadIdx.x; j < a.ns; j += SML_THREADS, ++k) {
    if (COMP && k == COMP_BLOCK) {
#pragma unroll
      for (int p = 0; p < NP; ++p) {
        two_sum2(hu[p], lu[p], u[p]);
        two_sum2(hv[p], lv[p], vn[p]);
        u[p] = vn[p] = f2(0.0f, 0.0f);
      }
      k = 0;
    }
    const float x = a.sx[j], y = a.sy[j], g = a.ss[j];
    const float z = a.sr ? radius_term(CORE, a.sr[j]) : 0.0f;
    const float2 cx = f2(x, x), cy = f2(y, y), cg = f2(g, g);
#pragma unroll
    for (int p = 0; p < NP; ++p) {
      const float2 dx = __fadd2_rn(cx, nx[p]), dy = __fadd2_rn(cy, ny[p]);
      const float2 zz = THICK ? __fadd2_rn(f2(z, z), zt[p]) : f2(z, z);
      const float2 d2 = __ffma2_rn(dx, dx, CORE == CORE_RM ? __ffma2_rn(dy, dy, zz) : __fmul2_rn(dy, dy));
      const float2 r = __fmul2_rn(cg, sym_core<CORE, 2>(d2, zz, q));
      u[p] = __ffma2_rn(r, dy, u[p]);
      vn[p] = __ffma2_rn(r, dx, vn[p]);
    }
  }
  float2 r[2][SML_T];                              // u, v of the eight targets
#pragma unroll
  for (int p = 0; p < NP; ++p) {
    two_sum2(hu[p], lu[p], u[p]);
    two_sum2(hv[p], lv[p], vn[p]);
    r[0][2 * p] = f2(hu[p].x, lu[p].x);
    r[0][2 * p + 1] = f2(hu[p].y, lu[p].y);
    r[1][2 * p] = f2(-hv[p].x, -lv[p].x);
    r[1][2 * p + 1] = f2(-hv[p].y, -lv[p].y);
  }
  sml_block_sum<2, SML_T>(r, red, tot);
  const int i = t0 + threadIdx.x;
  if (threadIdx.x < SML_T && i < o.nt) {
    const float2 su = tot[threadIdx.x], sv = tot[SML_T + threadIdx.x];
    const double c[2] = {(double)su.x + (double)su.y, (double)sv.x + (double)sv.y};
    store_target<RES_VEL>(o, i, c);
  }
}

template <int CORE>
void small_launch(bool thick, bool comp, const SmallArgs& a, const P2PArgs& o, int grid, cudaStream_t st) {
  auto k = thick ? (comp ? p2p_small_kernel<CORE, true, true> : p2p_small_kernel<CORE, true, false>)
                 : (comp ? p2p_small_kernel<CORE, false, true> : p2p_small_kernel<CORE, false, false>);
  k<<<grid, SML_THREADS, 0, st>>>(a, o);
}

}  // namespace

// Where one launch beats the tiled kernels (compensated, calls back to back, this -> those, us; 26
// is the rate at which Python issues the call and two clears).  One set on itself, against
// p2p_sym.cuh: 1,000 26 -> 32, 4,096 26 -> 39-44, 6,000 33-42 -> 51-57, 8,192 47-66 -> 52-61.
// Field points, against the packed kernels: 1,000 x 1,000 26 -> 48-65, 16,000 x 4,000 49-62 ->
// 73-99, 16,000 x 6,000 64-82 -> 71-97, 16,000 x 10,000 99-129 -> 87-120, 30,000 x 1,000 45-58 ->
// 50-67, 65,536 x 200 80-107 -> 52-69 (too few blocks), 2,000 x 50,000 82-103 -> 80-107 and
// 500 x 200,000 197 -> 74 (a block's reduction outweighs its sources).  Two compensated blocks run
// per SM; past the first wave of them a block's walk counts twice or more: 18,000 x 3,000 60 -> 76, 22,000 x 3,000
// 82 -> 76, 26,000 x 2,432 47 -> 69 but x 2,433 81 -> 69, 32,768 x 3,000 106 -> 83 (Vatistas-2 78 -> 60).  Plain sums
// have three or four blocks per SM and stay ahead up to the limit of pairs (Vatistas-2 30,000 x 2,500 50 -> 57).
bool p2p_small_applies(const obs_context* ctx, const P2PRequest& rq) {
  if (rq.result != RES_VEL || ctx->kernel_variant != OBS_VARIANT_AUTO || ctx->target_order != OBS_ORDER_AUTO) return false;
  const double pairs = (double)rq.ns * rq.nt;
  if (p2p_sym_applies(ctx, rq)) return pairs <= 4.5e7;
  const bool one_wave = rq.accum != OBS_COMPENSATED || rq.nt <= 2 * SML_T * ctx->num_sms;
  return pairs <= 9.0e7 && rq.ns <= (one_wave ? 32768 : 20000) && rq.nt <= 20480;
}

int run_p2p_small(obs_context* ctx, const P2PRequest& rq) {
  SmallArgs a{rq.sx, rq.sy, rq.sr, rq.ss, rq.ns, rq.tx, rq.ty, rq.tr};
  P2PArgs o;
  std::memset(&o, 0, sizeof(o));
  o.nt = rq.nt;
  o.out[0] = rq.tu; o.out[1] = rq.tv;
  o.finalize = (rq.flags & OBS_FLAG_FINALIZE) ? 1 : 0;
  o.fsx = rq.fsx; o.fsy = rq.fsy;
  o.overwrite = rq.overwrite;
  const bool thick = rq.tr != nullptr, comp = rq.accum == OBS_COMPENSATED;
  const int grid = (rq.nt + SML_T - 1) / SML_T;
  timing_begin(ctx);
  timing_main_begin(ctx);
  switch (rq.core) {
    case CORE_RM: small_launch<CORE_RM>(thick, comp, a, o, grid, ctx->stream); break;
    case CORE_GAUSS: small_launch<CORE_GAUSS>(thick, comp, a, o, grid, ctx->stream); break;
    case CORE_V2: small_launch<CORE_V2>(thick, comp, a, o, grid, ctx->stream); break;
    case CORE_WL: small_launch<CORE_WL>(thick, comp, a, o, grid, ctx->stream); break;
    case CORE_V3: small_launch<CORE_V3>(thick, comp, a, o, grid, ctx->stream); break;
    case CORE_SING: small_launch<CORE_SING>(thick, comp, a, o, grid, ctx->stream); break;
    default: small_launch<CORE_CEXP>(thick, comp, a, o, grid, ctx->stream); break;
  }
  ctx->launches++;
  timing_main_end(ctx);
  timing_end(ctx);
  return cuda_status(cudaGetLastError());
}

}  // namespace obs
