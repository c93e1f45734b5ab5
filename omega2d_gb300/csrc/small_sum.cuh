// small_sum.cuh -- the end of a one-launch sum (p2p_small.cu, p2p_small_res.cu, adjoint_small.cu): a
// block of 256 threads holds C values of partial sums, every thread a (hi, lo) pair of each; they are
// halved over the lanes, added over the warps and left in shared memory.
#pragma once

#include "obs_device.cuh"

namespace obs {

constexpr int SML_THREADS = 256;
constexpr int SML_WARPS = SML_THREADS / 32;

// (hi, lo) += (bh, bl)
__device__ __forceinline__ void sml_add(float2& a, float2 b) {
  two_sum_acc(a.x, a.y, b.x);
  a.y += b.y;
}

__device__ __forceinline__ float2 sml_xor(float2 v, int bit) {
  return make_float2(__shfl_xor_sync(0xffffffffu, v.x, bit), __shfl_xor_sync(0xffffffffu, v.y, bit));
}

// r[G][T] (T a power of two up to 16) over the block; tot[g * T + t] afterwards, for every thread.
// While values are left to halve, a step keeps the half that the lane's bit names and adds the other
// lane's part of it (T - 1 shuffles a group instead of 5 T); the remaining bits are summed in full.
template <int G, int T>
__device__ __forceinline__ void sml_block_sum(float2 (&r)[G][T], float2 (*red)[G * T], float2* tot) {
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  int t = 0;                                       // the value this lane ends with
  int bit = 16;
#pragma unroll
  for (int h = T / 2; h >= 1; h >>= 1, bit >>= 1) {
    const bool up = (lane & bit) != 0;
    if (up) t += h;
#pragma unroll
    for (int g = 0; g < G; ++g)
#pragma unroll
      for (int c = 0; c < h; ++c) {
        const float2 send = up ? r[g][c] : r[g][c + h];
        r[g][c] = up ? r[g][c + h] : r[g][c];
        sml_add(r[g][c], sml_xor(send, bit));
      }
  }
  const int rest = bit;                            // the lane bits below the halved ones
  for (; bit >= 1; bit >>= 1)
#pragma unroll
    for (int g = 0; g < G; ++g) sml_add(r[g][0], sml_xor(r[g][0], bit));
  if ((lane & (2 * rest - 1)) == 0)
#pragma unroll
    for (int g = 0; g < G; ++g) red[w][g * T + t] = r[g][0];
  __syncthreads();
  if (threadIdx.x < G * T) {
    float2 s = red[0][threadIdx.x];
    for (int q = 1; q < SML_WARPS; ++q) sml_add(s, red[q][threadIdx.x]);
    tot[threadIdx.x] = s;
  }
  __syncthreads();
}

}  // namespace obs
