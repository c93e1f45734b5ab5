// clear_inner.cu -- clear_inner_layer on the GPU (src/Reflect.h:733-760 over clear_inner_panp2,
// :491-729): the particles (or field points) that lie inside a body's cutoff layer are cropped
// with the cut tables or pushed onto the layer.
//
// Layout: a parallel prep forms each panel's normal (Surfaces::compute_bases), a 32-byte record
// (nodes, 1/length^2, normal) and the box of every 32 consecutive panels, and sums the node
// normals.  Then one warp takes up to 32 points.  For each of them in turn the warp searches
// together, one box per lane and then one panel per lane of the boxes that may hold the closest
// panel (clear::box_beyond, seg_bounds, beyond: FP32 bounds on the reference's own arithmetic), and
// lists the panels that may be the closest or tie it, in panel order; consecutive panels of a
// body lie together, so that is a few boxes and one or two panels.  Then every lane evaluates its
// own point's list exactly (the reference's float/double arithmetic) and crops or pushes it; points
// that moved are searched again.  The listed exact evaluations are the only FP64 work (this GPU
// issues about 2 FP64 lane-operations per SM-clock), and they run 32 points at a time.
// 200,000 points against 2048 panels: 0.16 ms (the call 0.23 ms), with the panels in random order
// 1.25 ms; one thread per point against every panel took 3.9 ms in either order, and more than this with few
// panels too (the call, 3, 32 and 256 panels: 200,000 points 147, 157 and 165 us instead of 381, 612 and 959; 1,000
// points 71, 82 and 80 instead of 96, 160 and 301).  It is bound by
// instruction issue (0.6 per clock and scheduler, about 500 warp instructions a point) and, at
// 38 %, FP64.  The removed circulation is summed in FP64 in a
// fixed order: per warp, per block, and over the blocks by the last one to finish.  clear_inner.cuh
// compiles for the host too, where the CPU tests check these steps against the oracle.  This file
// is compiled without fused multiply-adds (-fmad=false), like the oracle.
#include <cmath>
#include <cstring>
#include <mutex>
#include <vector>

#include "clear_inner.cuh"
#include "obs_context.h"
#include "obs_device.cuh"

namespace obs {
namespace {

constexpr int kClearWarps = 4;            // warps per block of the point kernel
constexpr int kClearThreads = 32 * kClearWarps;
constexpr int kMaxSweeps = 64;
constexpr int kClearList = 12;            // panels listed per point; a longer list: every panel is evaluated

struct CutTable {
  float v[3 * clear::CUT_N];              // positions, strengths kept, shifts
};

// one thread per panel: index and length checks, the panel normal (clear::normals' formula),
// the panel's record for the point kernel, its group's box (a group is a warp), and the node
// normals (atomic sums; exact for nodes of one or two panels, since 0 + a + b rounds the same in
// either order).  bad: npan minus the first panel with a bad index or no length (0: none).
__global__ void clear_panels_kernel(int nnodes, const float* __restrict__ nx, const float* __restrict__ ny, int npan,
                                    const unsigned* __restrict__ idx, float* pnx, float* pny, float4* geo,
                                    float4* nrm, float4* box, float* nnx, float* nny, int* deg, int* bad) {
  const int j = blockIdx.x * blockDim.x + threadIdx.x;
  const float inf = INFINITY;
  float4 b4 = make_float4(inf, inf, -inf, -inf);
  if (j < npan) {
    const unsigned a = idx[2 * j], b = idx[2 * j + 1];
    if (a >= (unsigned)nnodes || b >= (unsigned)nnodes) {
      atomicMax(bad, npan - j);
    } else {
      const float x0 = nx[a], y0 = ny[a], x1 = nx[b], y1 = ny[b];
      b4 = make_float4(fminf(x0, x1), fminf(y0, y1), fmaxf(x0, x1), fmaxf(y0, y1));
      float tx = x1 - x0, ty = y1 - y0;
      const float blensq = tx * tx + ty * ty;
      const float base = sqrtf(blensq);
      if (!(base > 0.0f)) {
        atomicMax(bad, npan - j);
      } else {
        tx = (float)((double)tx * (1.0 / (double)base));
        ty = (float)((double)ty * (1.0 / (double)base));
        pnx[j] = -ty;
        pny[j] = tx;
        geo[j] = make_float4(x0, y0, x1, y1);
        nrm[j] = make_float4(1.0f / blensq, -ty, tx, __uint_as_float(a));
        atomicAdd(&nnx[a], -ty); atomicAdd(&nny[a], tx);
        atomicAdd(&nnx[b], -ty); atomicAdd(&nny[b], tx);
        atomicAdd(&deg[a], 1);
        atomicAdd(&deg[b], 1);
      }
    }
  }
  for (int o = 16; o > 0; o >>= 1) {
    b4.x = fminf(b4.x, __shfl_xor_sync(0xffffffffu, b4.x, o));
    b4.y = fminf(b4.y, __shfl_xor_sync(0xffffffffu, b4.y, o));
    b4.z = fmaxf(b4.z, __shfl_xor_sync(0xffffffffu, b4.z, o));
    b4.w = fmaxf(b4.w, __shfl_xor_sync(0xffffffffu, b4.w, o));
  }
  if ((threadIdx.x & 31) == 0 && j < npan) box[j / clear::GROUP] = b4;
}

// a node shared by three or more panels: its normal summed again in panel order (the
// reference's order, src/Reflect.h:521-533); also records a bad panel
__global__ void clear_nodes_kernel(int nnodes, int npan, const unsigned* __restrict__ idx, const float* __restrict__ pnx,
                                   const float* __restrict__ pny, float* nnx, float* nny, const int* __restrict__ deg,
                                   const int* __restrict__ bad, int* status) {
  const int k = blockIdx.x * blockDim.x + threadIdx.x;
  const int fb = *bad;
  if (k == 0 && fb) record_failure(status, DEV_ERR_BOUNDS, 900, npan - fb, 0);   // bad node index or zero-length panel
  if (k >= nnodes || deg[k] <= 2 || fb) return;
  float sx = 0.0f, sy = 0.0f;
  for (int j = 0; j < npan; ++j) {
    const unsigned a = idx[2 * j], b = idx[2 * j + 1];
    if (a == (unsigned)k) { sx += pnx[j]; sy += pny[j]; }
    if (b == (unsigned)k) { sx += pnx[j]; sy += pny[j]; }
  }
  nnx[k] = sx;
  nny[k] = sy;
}

// per-block sums of the point kernel, and the call's results: circulation removed, modifications,
// points out of sweeps, the context's device status word
struct ClearSums {
  double lost, crops, fails;
};

__global__ void __launch_bounds__(kClearThreads) clear_points_kernel(clear::Geo g, const CutTable cut,
                                                                     const float4* __restrict__ geo,
                                                                     const float4* __restrict__ nrm,
                                                                     const float4* __restrict__ box,
                                                                     const int* __restrict__ bad, int method,
                                                                     float cutoff_mult, float ips, int ppw, int n,
                                                                     float* x, float* y, float* s,
                                                                     const float* __restrict__ r, ClearSums* part,
                                                                     int* done, const int* __restrict__ status,
                                                                     double* out) {
  constexpr unsigned FULL = 0xffffffffu;
  __shared__ float tab[3 * clear::CUT_N];
  __shared__ int list[kClearWarps][32][kClearList + 1];
  __shared__ ClearSums red[kClearThreads];
  __shared__ bool s_last;
  for (int k = threadIdx.x; k < 3 * clear::CUT_N; k += kClearThreads) tab[k] = cut.v[k];
  g.cpos = tab;
  g.ckeep = tab + clear::CUT_N;
  g.cshift = tab + 2 * clear::CUT_N;
  __syncthreads();
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int i = (blockIdx.x * kClearWarps + w) * ppw + lane;
  const bool mine = lane < ppw && i < n && !*bad;
  float xi = mine ? x[i] : 0.0f, yi = mine ? y[i] : 0.0f, si = (mine && s) ? s[i] : 0.0f;
  const float rad = (mine && r) ? r[i] : ips;
  double l = 0.0;
  int c = 0;
  bool active = mine;
  const int ng = (g.npan + clear::GROUP - 1) / clear::GROUP;
  const unsigned kInf = 0x7f800000u;
  auto box_at = [&](int k) {
    const float4 b = box[k];
    return clear::Box{b.x, b.y, b.z, b.w};
  };
  for (unsigned todo; (todo = __ballot_sync(FULL, active)) != 0u;) {
    int cnt = 0;                                   // panels listed for this lane's point
    float bound = INFINITY;                        // and its bound on the squared minimum
    for (; todo; todo &= todo - 1) {
      const int q = __ffs(todo) - 1;
      const float px = __shfl_sync(FULL, xi, q), py = __shfl_sync(FULL, yi, q);
      // the nearest box; squared distances compare as their bits (NaN above inf)
      unsigned dmin = 0xffffffffu;
      int kmin = 0;
      for (int k = lane; k < ng; k += 32) {
        const unsigned d = __float_as_uint(clear::box_dist2(box_at(k), px, py));
        if (d < dmin) { dmin = d; kmin = k; }
      }
      const unsigned best = __reduce_min_sync(FULL, dmin);
      const int k0 = __shfl_sync(FULL, kmin, __ffs(__ballot_sync(FULL, dmin == best)) - 1);
      unsigned T = kInf;
      auto bounds = [&](int j, unsigned& ub) {     // past the last panel: never the closest
        ub = kInf;
        if (j >= g.npan) return INFINITY;
        const float4 p = geo[j];
        float u;
        const float lb = clear::seg_bounds(p.x, p.y, p.z, p.w, nrm[j].x, px, py, u);
        ub = __float_as_uint(u);
        return lb;
      };
      unsigned ub;
      (void)bounds(k0 * clear::GROUP + lane, ub);
      T = min(T, __reduce_min_sync(FULL, ub));
      int m = 0;
      for (int kb = 0; kb < ng; kb += 32) {
        const int k = kb + lane;
        unsigned enter = __ballot_sync(FULL, k < ng && !clear::box_beyond(box_at(min(k, ng - 1)), px, py,
                                                                          sqrtf(__uint_as_float(T))));
        for (; enter; enter &= enter - 1) {
          const int j = (kb + __ffs(enter) - 1) * clear::GROUP + lane;
          const float lb = bounds(j, ub);
          T = min(T, __reduce_min_sync(FULL, ub));
          const bool hit = j < g.npan && !clear::beyond(lb, __uint_as_float(T));
          const unsigned hits = __ballot_sync(FULL, hit);
          const int at = m + __popc(hits & ((1u << lane) - 1u));
          if (hit && at < kClearList) list[w][q][at] = j;
          m += __popc(hits);
        }
      }
      if (lane == q) {
        cnt = m;
        bound = __uint_as_float(T);
      }
    }
    __syncwarp();
    if (active) {
      clear::Closest cl;
      clear::closest_init(cl);
      const bool all = cnt > kClearList;           // more panels than the list holds: go through all of them
      const int steps = all ? g.npan : cnt;
      for (int k = 0; k < steps; ++k) {
        const int j = all ? k : list[w][lane][k];
        const float4 pg = geo[j], pn = nrm[j];
        float ub;
        if (all && clear::beyond(clear::seg_bounds(pg.x, pg.y, pg.z, pg.w, pn.x, xi, yi, ub), bound)) continue;
        clear::closest_add(g, cl, __float_as_uint(pn.w), g.idx[2 * j + 1], pg.x, pg.y, pg.z, pg.w, pn.y, pn.z, xi, yi);
      }
      const int rc = clear::clear_apply(g, cl, method, cutoff_mult, ips, rad, xi, yi, si, l);
      if (rc == 1) {
        if (++c >= kMaxSweeps) {      // sweep limit: reported as no convergence
          c = -1;
          active = false;
        }
      } else {
        active = false;
      }
    }
    __syncwarp();
  }
  if (mine) {
    x[i] = xi;
    y[i] = yi;
    if (s) s[i] = si;
  }
  // fixed-order sums: lanes by a shuffle tree (skipped where no lane lost anything), warps, blocks
  const int crops = __reduce_add_sync(FULL, c > 0 ? c : 0), fails = __popc(__ballot_sync(FULL, c < 0));
  if (__any_sync(FULL, l != 0.0))
    for (int o = 16; o > 0; o >>= 1) l += __shfl_xor_sync(FULL, l, o);
  if (lane == 0) red[w] = ClearSums{l, (double)crops, (double)fails};
  __syncthreads();
  if (threadIdx.x == 0) {
    ClearSums t = red[0];
    for (int k = 1; k < kClearWarps; ++k) { t.lost += red[k].lost; t.crops += red[k].crops; t.fails += red[k].fails; }
    part[blockIdx.x] = t;
    __threadfence();
    s_last = atomicAdd(done, 1) == (int)gridDim.x - 1;
  }
  __syncthreads();
  if (!s_last) return;
  __threadfence();
  ClearSums t{0.0, 0.0, 0.0};
  for (int k = threadIdx.x; k < (int)gridDim.x; k += kClearThreads) {
    t.lost += __ldcg(&part[k].lost);
    t.crops += __ldcg(&part[k].crops);
    t.fails += __ldcg(&part[k].fails);
  }
  red[threadIdx.x] = t;
  __syncthreads();
  for (int o = kClearThreads / 2; o > 0; o >>= 1) {
    if (threadIdx.x < o) {
      red[threadIdx.x].lost += red[threadIdx.x + o].lost;
      red[threadIdx.x].crops += red[threadIdx.x + o].crops;
      red[threadIdx.x].fails += red[threadIdx.x + o].fails;
    }
    __syncthreads();
  }
  if (threadIdx.x == 0) {
    out[0] = red[0].lost;
    out[1] = red[0].crops;
    out[2] = red[0].fails;
    out[3] = (double)*status;
  }
}

size_t al256(size_t b) { return (b + 255) & ~(size_t)255; }

}  // namespace

// Device arrays in, updated in place; results (circulation removed, modifications) to the host.
int run_clear_inner(obs_context* ctx, int method, float cutoff_mult, float ips, int nnodes, const float* nx,
                    const float* ny, int npan, const unsigned* idx, int n, float* x, float* y, float* s,
                    const float* r, double* circ_removed, long long* ncropped) {
  static CutTable table;
  static std::once_flag table_once;       // callers on several host threads share the table
  std::call_once(table_once, [] { clear::cut_table(table.v, table.v + clear::CUT_N, table.v + 2 * clear::CUT_N); });
  const size_t P = (size_t)npan, M = (size_t)nnodes;
  // points per warp: 32 where that fills the GPU, fewer for small sets (the warp takes its points
  // in turn), so that there are about eight warps per scheduler
  int ppw = 32;
  while (ppw > 1 && (long long)n < (long long)ppw * 32 * ctx->num_sms) ppw /= 2;
  const int blocks = (int)(((long long)n + (long long)ppw * kClearWarps - 1) / ((long long)ppw * kClearWarps));
  const int ngrp = (npan + clear::GROUP - 1) / clear::GROUP;
  const size_t off_pn = 0;
  const size_t off_geo = off_pn + al256(2 * P * sizeof(float));
  const size_t off_nrm = off_geo + al256(P * sizeof(float4));
  const size_t off_box = off_nrm + al256(P * sizeof(float4));
  const size_t off_nn = off_box + al256((size_t)ngrp * sizeof(float4));   // node normals, degrees, bad, done: cleared
  const size_t zbytes = (3 * M + 2) * sizeof(float);
  const size_t off_part = off_nn + al256(zbytes);
  const size_t off_out = off_part + al256((size_t)blocks * sizeof(ClearSums));
  int st = ctx->work.ensure(off_out + 256, ctx->stream);
  if (st) return st;
  float* pn = ctx->work.as<float>(off_pn);
  float4* geo = ctx->work.as<float4>(off_geo);
  float4* nrm = ctx->work.as<float4>(off_nrm);
  float4* box = ctx->work.as<float4>(off_box);
  float* nn = ctx->work.as<float>(off_nn);
  int* deg = reinterpret_cast<int*>(nn + 2 * M);
  int* bad = deg + M;
  int* done = bad + 1;
  double* out = ctx->work.as<double>(off_out);
  cudaStream_t strm = ctx->stream;
  cudaError_t e = cudaMemsetAsync(nn, 0, zbytes, strm);
  if (e != cudaSuccess) return cuda_status(e);
  clear_panels_kernel<<<(npan + 255) / 256, 256, 0, strm>>>(nnodes, nx, ny, npan, idx, pn, pn + npan, geo, nrm, box, nn,
                                                            nn + nnodes, deg, bad);
  clear_nodes_kernel<<<(nnodes + 255) / 256, 256, 0, strm>>>(nnodes, npan, idx, pn, pn + npan, nn, nn + nnodes, deg, bad,
                                                             ctx->d_status);
  const clear::Geo g{nx, ny, idx, npan, pn, pn + npan, nn, nn + nnodes, nullptr, nullptr, nullptr};
  clear_points_kernel<<<blocks, kClearThreads, 0, strm>>>(g, table, geo, nrm, box, bad, method, cutoff_mult, ips, ppw, n,
                                                          x, y, s, r, ctx->work.as<ClearSums>(off_part), done,
                                                          ctx->d_status, out);
  ctx->launches += 3;
  if ((e = cudaGetLastError()) != cudaSuccess) return cuda_status(e);
  double h[4] = {0.0, 0.0, 0.0, 0.0};
  e = cudaMemcpyAsync(h, out, sizeof(h), cudaMemcpyDeviceToHost, strm);
  if (e == cudaSuccess) e = cudaStreamSynchronize(strm);
  if (e != cudaSuccess) return cuda_status(e);
  if (h[3] != 0.0 && (st = take_device_status(ctx))) return st;
  if (circ_removed) *circ_removed = h[0];
  if (ncropped) *ncropped = (long long)h[1];
  return h[2] > 0.0 ? OBS_ERR_NO_CONVERGENCE : OBS_OK;
}

}  // namespace obs

namespace {

int check_clear(obs_context* ctx, int method, float cutoff_mult, float ips, int nnodes, const float* nx,
                const float* ny, int npan, const unsigned* idx, int n, const float* x, const float* y,
                const float* s, const float* r) {
  if (!ctx || (method != 0 && method != 1) || nnodes < 0 || npan < 0 || n < 0) return OBS_ERR_ARG;
  if (!(ips > 0.0f) || !std::isfinite(ips) || !std::isfinite(cutoff_mult)) return OBS_ERR_ARG;
  if (npan > 0 && (!nx || !ny || !idx || nnodes < 2)) return OBS_ERR_ARG;
  if (n > 0 && (!x || !y)) return OBS_ERR_ARG;
  if (method == 0 && n > 0 && (!s || !r)) return OBS_ERR_ARG;   // cropping needs particles
  return OBS_OK;
}

}  // namespace

extern "C" {

int obs_clear_inner_layer_dev(obs_context* ctx, int method, float cutoff_mult, float ips, int nnodes,
                              const float* nx, const float* ny, int npan, const unsigned* idx, int n, float* x,
                              float* y, float* s, const float* r, double* circ_removed, long long* ncropped) {
  int st = check_clear(ctx, method, cutoff_mult, ips, nnodes, nx, ny, npan, idx, n, x, y, s, r);
  if (st) return st;
  if (circ_removed) *circ_removed = 0.0;
  if (ncropped) *ncropped = 0;
  if (n == 0 || npan == 0) return OBS_OK;
  if ((st = obs::bind(ctx))) return st;
  return obs::run_clear_inner(ctx, method, cutoff_mult, ips, nnodes, nx, ny, npan, idx, n, x, y,
                              method == 0 ? s : nullptr, r, circ_removed, ncropped);
}

int obs_clear_inner_layer(obs_context* ctx, int method, float cutoff_mult, float ips, int nnodes, const float* nx,
                          const float* ny, int npan, const unsigned* idx, int n, float* x, float* y, float* s,
                          const float* r, double* circ_removed, long long* ncropped) {
  int st = check_clear(ctx, method, cutoff_mult, ips, nnodes, nx, ny, npan, idx, n, x, y, s, r);
  if (st) return st;
  if (circ_removed) *circ_removed = 0.0;
  if (ncropped) *ncropped = 0;
  if (n == 0 || npan == 0) return OBS_OK;
  for (size_t k = 0; k < 2 * (size_t)npan; ++k)
    if (idx[k] >= (unsigned)nnodes) return OBS_ERR_ARG;
  if ((st = obs::bind(ctx))) return st;
  const size_t N = (size_t)n, P = (size_t)npan, M = (size_t)nnodes;
  auto al = [](size_t b) { return (b + 255) & ~(size_t)255; };
  const size_t o_nx = 0, o_ny = o_nx + al(M * 4), o_idx = o_ny + al(M * 4), o_x = o_idx + al(P * 8);
  const size_t o_y = o_x + al(N * 4), o_s = o_y + al(N * 4), o_r = o_s + al(N * 4), tot = o_r + al(N * 4);
  if ((st = ctx->io.ensure(tot, ctx->stream))) return st;
  float* dnx = ctx->io.as<float>(o_nx);
  float* dny = ctx->io.as<float>(o_ny);
  unsigned* didx = ctx->io.as<unsigned>(o_idx);
  float* dx = ctx->io.as<float>(o_x);
  float* dy = ctx->io.as<float>(o_y);
  float* ds = (method == 0) ? ctx->io.as<float>(o_s) : nullptr;
  float* dr = r ? ctx->io.as<float>(o_r) : nullptr;
  cudaStream_t strm = ctx->stream;
  cudaError_t e = cudaMemcpyAsync(dnx, nx, M * 4, cudaMemcpyHostToDevice, strm);
  if (e == cudaSuccess) e = cudaMemcpyAsync(dny, ny, M * 4, cudaMemcpyHostToDevice, strm);
  if (e == cudaSuccess) e = cudaMemcpyAsync(didx, idx, P * 8, cudaMemcpyHostToDevice, strm);
  if (e == cudaSuccess) e = cudaMemcpyAsync(dx, x, N * 4, cudaMemcpyHostToDevice, strm);
  if (e == cudaSuccess) e = cudaMemcpyAsync(dy, y, N * 4, cudaMemcpyHostToDevice, strm);
  if (e == cudaSuccess && ds) e = cudaMemcpyAsync(ds, s, N * 4, cudaMemcpyHostToDevice, strm);
  if (e == cudaSuccess && dr) e = cudaMemcpyAsync(dr, r, N * 4, cudaMemcpyHostToDevice, strm);
  if (e != cudaSuccess) return obs::cuda_status(e);
  double circ = 0.0;
  long long nc = 0;
  st = obs::run_clear_inner(ctx, method, cutoff_mult, ips, nnodes, dnx, dny, npan, didx, n, dx, dy, ds, dr, &circ,
                            &nc);
  if (st && st != OBS_ERR_NO_CONVERGENCE) return st;
  // device -> temporaries -> caller, so a failed copy leaves the caller's arrays untouched
  std::vector<float> hx(N), hy(N), hs(ds ? N : 0);
  e = cudaMemcpyAsync(hx.data(), dx, N * 4, cudaMemcpyDeviceToHost, strm);
  if (e == cudaSuccess) e = cudaMemcpyAsync(hy.data(), dy, N * 4, cudaMemcpyDeviceToHost, strm);
  if (e == cudaSuccess && ds) e = cudaMemcpyAsync(hs.data(), ds, N * 4, cudaMemcpyDeviceToHost, strm);
  if (e == cudaSuccess) e = cudaStreamSynchronize(strm);
  if (e != cudaSuccess) return obs::cuda_status(e);
  std::memcpy(x, hx.data(), N * 4);
  std::memcpy(y, hy.data(), N * 4);
  if (ds) std::memcpy(s, hs.data(), N * 4);
  if (circ_removed) *circ_removed = circ;
  if (ncropped) *ncropped = nc;
  return st;
}

}  // extern "C"
