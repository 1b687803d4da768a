// A warp's ids in registers, E per lane: bitonic sort and removal of repetitions.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

// The smaller of both where `lower`, else the larger.  Written as two predicated instructions in networks of 128 ids and more: no
// fewer instructions than the choice between two results (341 M for 262,144 samples, 25 x 10), but 4.8 instead of 5.4 of the 18
// cycles between two of a warp's are spent on fetching the next one, 488 -> 475 us; no gain in networks of 64 and 32 ids.
template <int E>
__device__ __forceinline__ int32_t smaller_if(bool lower, int32_t a, int32_t b) {
  if (E < 4) return lower ? min(a, b) : max(a, b);
  asm("{.reg .pred p; setp.ne.s32 p, %2, 0; @p min.s32 %0, %0, %1; @!p max.s32 %0, %0, %1;}" : "+r"(a) : "r"(b), "r"((int)lower));
  return a;
}

// Ascending over the positions lane * E + e: bitonic merges whose first stage pairs position i with its mirror
// image in the block, so that every exchange puts the smaller id at the lower position.
template <int E>
__device__ __forceinline__ void warp_sort(int32_t (&v)[E]) {
  constexpr int P = 32 * E;
  const int lane = threadIdx.x & 31;
#pragma unroll
  for (int size = 2; size <= P; size <<= 1) {
    if (size <= E) {   // mirror inside a lane
#pragma unroll
      for (int e = 0; e < E; e++) {
        const int o = e ^ (size - 1);
        if (e < o) {
          const int32_t a = v[e], b = v[o];
          v[e] = min(a, b); v[o] = max(a, b);
        }
      }
    } else {           // position p with p ^ (size - 1): lane ^ (size / E - 1), element E - 1 - e
      const int mask = size / E - 1;
      const bool lower = (lane & (size / E / 2)) == 0;
      int32_t w[E];
#pragma unroll
      for (int e = 0; e < E; e++) w[e] = __shfl_xor_sync(0xffffffffu, v[E - 1 - e], mask);
#pragma unroll
      for (int e = 0; e < E; e++) v[e] = smaller_if<E>(lower, v[e], w[e]);
    }
#pragma unroll
    for (int stride = size >> 2; stride > 0; stride >>= 1) {
      if (stride >= E) {
        const bool lower = (lane & (stride / E)) == 0;
#pragma unroll
        for (int e = 0; e < E; e++) {
          const int32_t o = __shfl_xor_sync(0xffffffffu, v[e], stride / E);
          v[e] = smaller_if<E>(lower, v[e], o);
        }
      } else {
#pragma unroll
        for (int e = 0; e < E; e++) {
          if ((e & stride) == 0) {
            const int32_t a = v[e], b = v[e + stride];
            v[e] = min(a, b); v[e + stride] = max(a, b);
          }
        }
      }
    }
  }
}

// The distinct ids of a sorted warp (0x7fffffff: no id) to `to`, in order; their number.
template <int E>
__device__ __forceinline__ int warp_unique_store(const int32_t (&v)[E], int32_t *to) {
  const int lane = threadIdx.x & 31;
  const int32_t before = __shfl_up_sync(0xffffffffu, v[E - 1], 1);  // last id of the lane to the left
  bool head[E];
  int cnt = 0;
#pragma unroll
  for (int e = 0; e < E; e++) {
    const int32_t prev = e == 0 ? before : v[e == 0 ? 0 : e - 1];
    head[e] = v[e] != 0x7fffffff && ((lane == 0 && e == 0) || v[e] != prev);
    cnt += head[e] ? 1 : 0;
  }
  int inc = cnt;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int t = __shfl_up_sync(0xffffffffu, inc, o);
    if (lane >= o) inc += t;
  }
  int pos = inc - cnt;
#pragma unroll
  for (int e = 0; e < E; e++)
    if (head[e]) to[pos++] = v[e];
  return __shfl_sync(0xffffffffu, inc, 31);
}
