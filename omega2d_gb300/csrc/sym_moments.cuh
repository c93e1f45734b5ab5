// sym_moments.cuh -- gradient, vorticity and shear of a particle set on itself, and its self VJP, for
// the Gaussian core, each unordered pair evaluated once (p2p_sym.cuh's rows, columns, ranges and
// partials; src/Kernels.h:112-231 for the results, adjoint.cu for the VJP).
//
// With d = x_column - x_row, K the core, B = 2 dK/d(d^2), a = K dx, b = K dy, the pair's numbers are
//   velocity   a, b                                       (change sign between the two particles)
//   gradient   n = B (dx^2 - dy^2) / 4, h = -B dx dy / 2, e = B d^2 / 2 + K    (the same for both):
//              P = sum G h, N = sum G n, E = sum G e:  S1 = -2 P, S2 = E + 2 N, S3 = 2 N - E
//   vorticity  2 e;   shear  |B| d^2 / 2 with |G|
//   self VJP   with wu = G_c lu_r - G_r lu_c, wv = G_c lv_r - G_r lv_c (changing sign as well),
//              X = K wv + B (dx wv - dy wu) dx and Y = -K wu + B (dx wv - dy wu) dy go to the row and, with
//              the other sign, to the column, and a lv - b lu of the other particle to dL/dG
// Beyond the core's far radius K = 1/d^2 and B = -2 K^2, so n = b^2 - K/2, h = a b, e = 0,
// X / 2 = n wv + h wu, Y / 2 = n wu - h wv: far groups need no exponential and drop the sums of e.  A pair
// of pairs takes 17 f32x2 operations for two gradient interactions (one-sided: 24) and 28 for two VJP
// interactions (one-sided: 34); bound by the registers' read ports like the velocity sum.
// Measured, 131,072-particle patch, compensated (one-sided -> here): gradient 8.66 -> 7.0 ms, vorticity 5.66
// -> 4.5, shear 6.2 -> 5.3, self VJP 12.1 -> 8.8 (11.3 in Hilbert order); 3 and 4 row pairs per thread take
// 2 to 20 % longer (fewer, larger row blocks; 128 registers either way), 5 and 6 CTAs per SM as long.
#pragma once

#include "p2p_sym.cuh"

namespace obs {

constexpr int MOM_TG = 4;                            // groups per staged tile
constexpr int MOM_TILE = SYM_GRP * MOM_TG;

// NP: f32x2 row pairs per thread.  NF sums per particle from every pair, NN more from near pairs only.
// FAR: d^2 / s^2 beyond which a pair is far (1 % margin in the kernel): the reference's
// gradient factor equals -2 K^2 to 4e-10 beyond 25, the VJP's far branch begins at the core's own 16.
struct MomGrad { static constexpr int NP = 2, NF = 4, NN = 1; static constexpr bool VJP = false; static constexpr float FAR = 25.0f; };
struct MomVort { static constexpr int NP = 2, NF = 2, NN = 1; static constexpr bool VJP = false; static constexpr float FAR = 25.0f; };
struct MomShear { static constexpr int NP = 2, NF = 3, NN = 0; static constexpr bool VJP = false; static constexpr float FAR = 25.0f; };
struct MomVjp { static constexpr int NP = 2, NF = 3, NN = 0; static constexpr bool VJP = true; static constexpr float FAR = 16.0f; };
template <class OP> constexpr int mom_gpb() { return SYM_THREADS / 32 * 2 * OP::NP; }   // groups per row block
template <class OP> constexpr int mom_rows() { return mom_gpb<OP>() * SYM_GRP; }
// planes of a warp's column sums: the compensated gradient keeps the two halves of the rows apart and adds all
// halves and warps in two-sums (131,072-particle patch: du/dx 8.3e-8 off FP64; 8.6e-8 with the halves added up
// first, 9.4e-8 with one FP32 sum per row block, 8.5e-8 one-sided; 7.09, 6.93 and 6.80 ms).  The others' errors are
// within 1 % of the one-sided ones or below with the halves added up
template <class OP> constexpr int mom_planes(bool comp) { return comp && OP::NF == 4 ? 2 : 1; }

// 32 columns as staged (SymGroup with the VJP's cotangents)
template <bool VJP> struct MomGroup;
template <> struct __align__(128) MomGroup<false> {
  float4 xy[SYM_GRP];
  float2 g[SYM_GRP], z[SYM_GRP];
};
template <> struct __align__(128) MomGroup<true> {
  float4 xy[SYM_GRP];
  float2 g[SYM_GRP], z[SYM_GRP];
  float4 l[SYM_GRP];       // (-lu, -lu, lv, lv): the strength term is then two fused operations
};

struct MomArgs {
  SymArgs s;               // grp, colpart, rowpart and run of SymArgs unused
  const void* grp;
  void* colpart;           // per row block, [NF + NN][its later columns]: float2 (hi, lo) when compensated, else float
  float2* rowpart;         // [nrange + nblk][NF + NN][rows] (hi, lo)
  float2* run;             // [NF + NN][npad] running sums over the passes
};

// a particle's weights: strength (negated for the VJP) and, for the VJP, cotangents (the first one negated)
struct MomW {
  float2 g, mlu, lv;
};

__device__ __forceinline__ float2 abs2(float2 v) { return f2(fabsf(v.x), fabsf(v.y)); }
__device__ __forceinline__ float2 mul2(float2 a, float2 b) { return __fmul2_rn(a, b); }
__device__ __forceinline__ float2 nfma2(float2 a, float2 b, float2 c) {   // c - a b, two roundings
  return __ffma2_rn(__fmul2_rn(a, b), f2(-1.0f, -1.0f), c);
}

// one group against the warp's rows; FORM as sym_core's; csum: the warp's sums of the columns, as in sym_group
// (velocity, X, Y and the dL/dG term as the row sees them: the reduction turns the signs)
// OWN: columns of the rows' own block; the VJP's weights are then formed with both products rounded, so that a particle
// with itself (and any with equal strength and cotangent) has none.
template <class OP, int FORM, bool COMP, bool OWN>
__device__ __forceinline__ void mom_group(const MomGroup<OP::VJP>& grp, int lane, float us2, float ucf,
                                          const float2 (&nx)[OP::NP], const float2 (&ny)[OP::NP], const MomW (&w)[OP::NP],
                                          const float* __restrict__ zrow, float2 (&acc)[OP::NP][OP::NF + OP::NN],
                                          float (*csum)[mom_planes<OP>(COMP) * MOM_TILE], float2* nsum) {
  constexpr bool FAR = FORM == 0;
  constexpr int NC = OP::NF + (FAR ? 0 : OP::NN);
  const float2 half = f2(0.5f, 0.5f), mhalf = f2(-0.5f, -0.5f);
  float cs[OP::NF + OP::NN];
#pragma unroll
  for (int c = 0; c < OP::NF + OP::NN; ++c) cs[c] = 0.0f;
#pragma unroll 1
  for (int s0 = 0; s0 < SYM_GRP; s0 += SYM_GRP / 2) {
    if (s0) {                                      // the first half's sums, at the lanes half a group away
#pragma unroll
      for (int c = 0; c < OP::NF + OP::NN; ++c) {
        csum[c][lane ^ (SYM_GRP / 2)] = cs[c];
        cs[c] = 0.0f;
      }
    }
#pragma unroll 4
    for (int s = s0; s < s0 + SYM_GRP / 2; ++s) {
      const int col = lane ^ s;
      const float4 c4 = grp.xy[col];
      const float2 cx = f2(c4.x, c4.y), cy = f2(c4.z, c4.w), cg = grp.g[col];
      float2 cmlu = f2(0.0f, 0.0f), clv = cmlu;
      if constexpr (OP::VJP) {
        const float4 l = grp.l[col];
        cmlu = f2(l.x, l.y);
        clv = f2(l.z, l.w);
      }
      float2 t[OP::NF + OP::NN];                     // this step's rows for the column
#pragma unroll
      for (int c = 0; c < OP::NF + OP::NN; ++c) t[c] = f2(0.0f, 0.0f);
      // to both particles of a pair, value v times the other one's weight
      auto both = [&](int p, int c, float2 v, float2 wc, float2 wr) {
        acc[p][c] = __ffma2_rn(wc, v, acc[p][c]);
        t[c] = (p == 0) ? __fmul2_rn(wr, v) : __ffma2_rn(wr, v, t[c]);
      };
#pragma unroll
      for (int p = 0; p < OP::NP; ++p) {
        const float2 dx = __fadd2_rn(cx, nx[p]), dy = __fadd2_rn(cy, ny[p]);
        const float2 d2 = __ffma2_rn(dx, dx, __fmul2_rn(dy, dy));
        float2 k, B = f2(0.0f, 0.0f);
        if constexpr (FAR) {
          k = f2(rcp_a(d2.x), rcp_a(d2.y));
        } else {
          const float2 cz = (FORM == 2) ? grp.z[col] : f2(0.0f, 0.0f);
          const float z0 = (FORM == 2) ? zrow[(2 * p) * SYM_THREADS] : 0.0f;
          const float z1 = (FORM == 2) ? zrow[(2 * p + 1) * SYM_THREADS] : 0.0f;
          core_eval<CORE_GAUSS, true, true, FORM == 1>(d2.x, cz.x, z0, us2, ucf, k.x, B.x);
          core_eval<CORE_GAUSS, true, true, FORM == 1>(d2.y, cz.y, z1, us2, ucf, k.y, B.y);
          if constexpr (OP::VJP && FORM == 1) {
            // the exact derivative of the forward's far branch
            B.x = (d2.x * ucf > 16.0f) ? -2.0f * k.x * k.x : B.x;
            B.y = (d2.y * ucf > 16.0f) ? -2.0f * k.y * k.y : B.y;
          }
        }
        if constexpr (OP::VJP) {
          // -wu and wv from the row's negated strength (w.g here)
          const float2 gu = mul2(cg, w[p].mlu), gv = mul2(cg, w[p].lv);
          float2 mwu, wv;
          if constexpr (OWN) {
            const float2 g = mul2(w[p].g, f2(-1.0f, -1.0f));
            mwu = nfma2(g, cmlu, gu);
            wv = nfma2(g, clv, gv);
          } else {
            mwu = __ffma2_rn(w[p].g, cmlu, gu);
            wv = __ffma2_rn(w[p].g, clv, gv);
          }
          float2 X, Y;                               // halved and negated
          if constexpr (FAR) {
            const float2 b = mul2(k, dy), n = __ffma2_rn(b, b, mul2(k, mhalf)), h = mul2(mul2(k, dx), b);
            X = nfma2(n, wv, mul2(h, mwu));
            Y = __ffma2_rn(n, mwu, mul2(h, wv));
          } else {
            const float2 q = __ffma2_rn(dy, mwu, mul2(dx, wv)), bq = mul2(mul2(B, mhalf), q), kh = mul2(k, mhalf);
            X = __ffma2_rn(bq, dx, mul2(kh, wv));
            Y = __ffma2_rn(bq, dy, mul2(kh, mwu));
          }
          acc[p][0] = __fadd2_rn(acc[p][0], X);
          acc[p][1] = __fadd2_rn(acc[p][1], Y);
          t[0] = (p == 0) ? X : __fadd2_rn(t[0], X);
          t[1] = (p == 0) ? Y : __fadd2_rn(t[1], Y);
          // lv dx - lu dy first: it cancels, and K (lv dx) and K (lu dy) added one by one have 20 % more error
          const float2 er = __ffma2_rn(dy, cmlu, mul2(dx, clv)), ec = __ffma2_rn(dy, w[p].mlu, mul2(dx, w[p].lv));
          acc[p][2] = __ffma2_rn(k, er, acc[p][2]);
          t[2] = (p == 0) ? mul2(k, ec) : __ffma2_rn(k, ec, t[2]);
        } else {
          const float2 a = mul2(k, dx), b = mul2(k, dy);
          both(p, 0, b, cg, w[p].g);
          both(p, 1, a, cg, w[p].g);
          const float2 q = mul2(B, half);            // near: B / 2
          if constexpr (OP::NF == 4) {
            float2 n, h;
            if constexpr (FAR) {
              n = __ffma2_rn(b, b, mul2(k, mhalf));
              h = mul2(a, b);
            } else {
              n = mul2(q, __ffma2_rn(dx, dx, mul2(d2, mhalf)));
              h = mul2(mul2(B, mhalf), mul2(dx, dy));
              both(p, 4, __ffma2_rn(q, d2, k), cg, w[p].g);
            }
            both(p, 2, h, cg, w[p].g);
            both(p, 3, n, cg, w[p].g);
          } else if constexpr (OP::NF == 3) {
            both(p, 2, FAR ? k : mul2(abs2(q), d2), abs2(cg), abs2(w[p].g));
          } else if constexpr (!FAR) {
            both(p, 2, __ffma2_rn(q, d2, k), cg, w[p].g);
          }
        }
      }
      const int m = (s ^ (s + 1)) & 31;
#pragma unroll
      for (int c = 0; c < NC; ++c) cs[c] = __shfl_xor_sync(0xffffffffu, cs[c] + (t[c].x + t[c].y), m);
    }
    if constexpr (!FAR && OP::NN > 0) {
      // fold the near-only row sums, compensated in both modes and 16 columns at a time: in spatial order a
      // particle's near ones come together (vorticity of 60,000: 1.4e-7 off FP64 with 32 at a time)
#pragma unroll
      for (int c = 0; c < OP::NN; ++c)
#pragma unroll
        for (int p = 0; p < OP::NP; ++p)
#pragma unroll
          for (int h = 0; h < 2; ++h) {
            float2& n = nsum[(c * 2 * OP::NP + 2 * p + h) * SYM_THREADS];
            float2 s = n;
            two_sum_acc(s.x, s.y, h ? acc[p][OP::NF + c].y : acc[p][OP::NF + c].x);
            n = s;
            if (h) acc[p][OP::NF + c] = f2(0.0f, 0.0f);
          }
    }
  }
  if constexpr (mom_planes<OP>(COMP) == 2) {
#pragma unroll
    for (int c = 0; c < OP::NF + OP::NN; ++c) csum[c][MOM_TILE + lane] = cs[c];
  } else {
    __syncwarp();
#pragma unroll
    for (int c = 0; c < OP::NF + OP::NN; ++c) csum[c][lane] += cs[c];
  }
}

template <class OP, bool COMP>
__global__ void __launch_bounds__(SYM_THREADS, 4) sym_moments_kernel(const MomArgs m) {
  constexpr int NP = OP::NP, NF = OP::NF, NN = OP::NN, NC = NF + NN;
  constexpr int GPB = mom_gpb<OP>(), ROWS = mom_rows<OP>();
  using Group = MomGroup<OP::VJP>;
  wait_for_previous();
  const SymArgs& a = m.s;
  __shared__ Group tile[NSTAGE][MOM_TG];
  constexpr int PLANES = mom_planes<OP>(COMP);
  __shared__ float csum[SYM_THREADS / 32][NC][PLANES * MOM_TILE];
  __shared__ float2 nsum[NN > 0 ? NN : 1][2 * NP][SYM_THREADS];   // near-only row sums (hi, lo), each thread its own
  __shared__ float zrow[2 * NP * SYM_THREADS];
  __shared__ __align__(8) uint64_t bar[NSTAGE];
  __shared__ int s_range;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const Group* groups = static_cast<const Group*>(m.grp);
  if (tid == 0) {
    for (int s = 0; s < NSTAGE; ++s) mbar_init(&bar[s], 1);
    fence_mbar_init();
  }
  __syncthreads();
  const bool unif = ~a.meta[0] == a.meta[1];
  const float us2 = unif ? 2.0f * radius_term(CORE_GAUSS, __uint_as_float(a.meta[1])) : 0.0f;
  const float ucf = __frcp_rn(us2);
  // own radii: with the largest for both, from 25 on, where both forms agree to 4e-10; as in the velocity's kernel
  const float lim = 1.01f * (unif ? OP::FAR * us2 : 50.0f * max_radius_term(CORE_GAUSS, a.meta[1]));

  uint32_t kt = 0;
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
      const int g0 = GPB * blk + (pos - kbeg);
      const int ng = kend - pos;
      const int gdiag = GPB * (blk + 1);
      const int ntile = (ng + MOM_TG - 1) / MOM_TG;
      pos = kend;
      auto fetch = [&](int t, int st) {
        const int cnt = min(MOM_TG, ng - t * MOM_TG);
        const uint32_t bytes = (uint32_t)(cnt * sizeof(Group));
        mbar_arrive_expect_tx(&bar[st], bytes);
        bulk_g2s(&tile[st][0], groups + (g0 + t * MOM_TG), bytes, &bar[st]);
      };
      if (tid == 0) {
        fence_proxy_async_smem();
        for (int s = 0; s < NSTAGE && s < ntile; ++s) fetch(s, (kt + s) % NSTAGE);
      }
      float2 nx[NP], ny[NP];
      MomW w[NP];
      float2 acc[NP][NC], hi[NP][NF], lo[NP][NF];
      float bx0 = 3.0e38f, bx1 = -3.0e38f, by0 = 3.0e38f, by1 = -3.0e38f;
      const int row0 = blk * ROWS + warp * 64 * NP + lane;
#pragma unroll
      for (int p = 0; p < NP; ++p) {
        const Group& r0 = groups[blk * GPB + warp * 2 * NP + 2 * p];
        const Group& r1 = groups[blk * GPB + warp * 2 * NP + 2 * p + 1];
        const float4 q0 = r0.xy[lane], q1 = r1.xy[lane];
        if (row0 + 2 * p * 32 < a.n) {
          bx0 = fminf(bx0, q0.x); bx1 = fmaxf(bx1, q0.x);
          by0 = fminf(by0, q0.z); by1 = fmaxf(by1, q0.z);
        }
        if (row0 + (2 * p + 1) * 32 < a.n) {
          bx0 = fminf(bx0, q1.x); bx1 = fmaxf(bx1, q1.x);
          by0 = fminf(by0, q1.z); by1 = fmaxf(by1, q1.z);
        }
        nx[p] = f2(-q0.x, -q1.x);
        ny[p] = f2(-q0.z, -q1.z);
        w[p].g = OP::VJP ? f2(-r0.g[lane].x, -r1.g[lane].x) : f2(r0.g[lane].x, r1.g[lane].x);
        if (!unif) {                               // read by this thread alone
          zrow[(2 * p) * SYM_THREADS + tid] = r0.z[lane].x;
          zrow[(2 * p + 1) * SYM_THREADS + tid] = r1.z[lane].x;
        }
        if constexpr (OP::VJP) {
          w[p].mlu = f2(r0.l[lane].x, r1.l[lane].x);
          w[p].lv = f2(r0.l[lane].z, r1.l[lane].z);
        }
#pragma unroll
        for (int c = 0; c < NC; ++c) acc[p][c] = f2(0.0f, 0.0f);
#pragma unroll
        for (int c = 0; c < NF; ++c) hi[p][c] = lo[p][c] = f2(0.0f, 0.0f);
      }
      for (int o = 16; o > 0; o >>= 1) {
        bx0 = fminf(bx0, __shfl_xor_sync(0xffffffffu, bx0, o));
        bx1 = fmaxf(bx1, __shfl_xor_sync(0xffffffffu, bx1, o));
        by0 = fminf(by0, __shfl_xor_sync(0xffffffffu, by0, o));
        by1 = fmaxf(by1, __shfl_xor_sync(0xffffffffu, by1, o));
      }
#pragma unroll
      for (int c = 0; c < NN; ++c)
#pragma unroll
        for (int r = 0; r < 2 * NP; ++r) nsum[c][r][tid] = f2(0.0f, 0.0f);
      for (int t = 0; t < ntile; ++t, ++kt) {
        const int st = kt % NSTAGE;
        const bool ok = mbar_wait_bounded(&bar[st], (kt / NSTAGE) & 1u, WAIT_TRIES);
        if (__syncthreads_or(!ok)) {
          if (tid == 0) {
            record_failure(a.status, DEV_ERR_TIMEOUT, 250 + st, (int)kt, range);
            for (int s = 0; s < NSTAGE; ++s) (void)mbar_wait_bounded(&bar[(kt + s) % NSTAGE], ((kt + s) / NSTAGE) & 1u, WAIT_TRIES);
          }
          return;
        }
        const int cnt = min(MOM_TG, ng - t * MOM_TG);
        for (int b = 0; b < cnt; ++b) {
          const Group& grp = tile[st][b];
          float (*cw)[PLANES * MOM_TILE] = reinterpret_cast<float (*)[PLANES * MOM_TILE]>(&csum[warp][0][b * SYM_GRP]);
          bool near = true;
          if (lim < 3.0e38f) {                     // some group may be far
            const float4 c = grp.xy[lane];
            const float ex = fmaxf(0.0f, fmaxf(bx0 - c.x, c.x - bx1));
            const float ey = fmaxf(0.0f, fmaxf(by0 - c.z, c.z - by1));
            near = __any_sync(0xffffffffu, !(fmaf(ex, ex, ey * ey) > lim));   // a NaN coordinate is near
          }
          auto run = [&](auto own) {
            constexpr bool OWN = OP::VJP && decltype(own)::value;
            // the order of the forms moves registers: 131,072 gradient 6.89-6.92 ms with the far form last, 7.00-7.06 first;
            // VJP 8.81 and 8.75
            auto form = [&](auto f) {
              constexpr int FORM = decltype(f)::value;
              mom_group<OP, FORM, COMP, FORM != 0 && OWN>(grp, lane, us2, ucf, nx, ny, w, zrow + tid, acc, cw, &nsum[0][0][tid]);
            };
            if constexpr (OP::VJP) {
              if (!near) form(std::integral_constant<int, 0>{});
              else if (unif) form(std::integral_constant<int, 1>{});
              else form(std::integral_constant<int, 2>{});
            } else {
              if (near && !unif) form(std::integral_constant<int, 2>{});
              else if (near) form(std::integral_constant<int, 1>{});
              else form(std::integral_constant<int, 0>{});
            }
          };
          if (OP::VJP && g0 + t * MOM_TG + b < gdiag) run(std::true_type{});
          else run(std::false_type{});
          if (COMP || b == cnt - 1) {              // plain sums fold once per tile
#pragma unroll
            for (int p = 0; p < NP; ++p)
#pragma unroll
              for (int c = 0; c < NF; ++c) {
                two_sum2(hi[p][c], lo[p][c], acc[p][c]);
                acc[p][c] = f2(0.0f, 0.0f);
              }
          }
        }
        __syncthreads();
        if (tid == 0 && t + NSTAGE < ntile) {
          fence_proxy_async_smem();
          fetch(t + NSTAGE, st);
        }
        const int c0 = (g0 + t * MOM_TG) * SYM_GRP;
        for (int c = tid; c < cnt * SYM_GRP; c += SYM_THREADS) {
          const int j = c0 + c;
          if (j < gdiag * SYM_GRP || j >= a.n) continue;
          const int wd = sym_width(a, k);
          const size_t at = NC * sym_base(a, k) + (j - sym_first(a, k));
          if constexpr (COMP) {
#pragma unroll
            for (int q = 0; q < NC; q += 2) {      // two components at a time
              const int r = q + 1 < NC ? q + 1 : q;
              float2 hi = f2(csum[0][q][c], csum[0][r][c]), lo = f2(0.0f, 0.0f);
#pragma unroll
              for (int w = 0; w < SYM_THREADS / 32; ++w)
#pragma unroll
                for (int g = w ? 0 : 1; g < PLANES; ++g)
                  two_sum2(hi, lo, f2(csum[w][q][g * MOM_TILE + c], csum[w][r][g * MOM_TILE + c]));
              float2* cp = static_cast<float2*>(m.colpart) + at;
              cp[(size_t)q * wd] = f2(hi.x, lo.x);
              if (r > q) cp[(size_t)r * wd] = f2(hi.y, lo.y);
            }
          } else {
#pragma unroll
            for (int q = 0; q < NC; ++q)
              static_cast<float*>(m.colpart)[at + (size_t)q * wd] = (csum[0][q][c] + csum[1][q][c]) + (csum[2][q][c] + csum[3][q][c]);
          }
        }
      }
      float2* rp = m.rowpart + (size_t)(range + k) * NC * ROWS;
#pragma unroll
      for (int p = 0; p < NP; ++p)
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const int i = warp * 64 * NP + (2 * p + h) * 32 + lane;
#pragma unroll
          for (int c = 0; c < NF; ++c)
            rp[(size_t)c * ROWS + i] = h ? f2(hi[p][c].y, lo[p][c].y) : f2(hi[p][c].x, lo[p][c].x);
#pragma unroll
          for (int c = 0; c < NN; ++c) rp[(size_t)(NF + c) * ROWS + i] = nsum[c][2 * p + h][tid];
        }
    }
    __syncthreads();
  }
}

}  // namespace obs
