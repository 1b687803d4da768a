// What the collective applications' kernels share.
#pragma once

#include "nd_common.cuh"
#include "nd_entries.cuh"
#include "nd_philox.cuh"

struct CollParams {
  uint64_t seed;
  int64_t first_sample;
  int32_t V, fs, L, B, stride, step, ntr;
  int app;
};

__device__ __forceinline__ const int32_t *transits_of(const CollParams &cp, const int32_t *initial, const int32_t *out, int64_t s) {
  return cp.step == 0 ? initial + s * cp.B : out + s * cp.fs + (int64_t)(cp.step - 1) * cp.L;
}

__device__ __forceinline__ bool has_edge_logn(const NdGraphView &g, int32_t src, int32_t dst) {
  int32_t l = __ldg(g.row_ptr + src), r = __ldg(g.row_ptr + src + 1) - 1;
  while (l <= r) {
    const int32_t m = l + (r - l) / 2;
    const int32_t e = __ldg(g.col + m);
    if (e == dst) return true;
    if (e < dst) l = m + 1; else r = m - 1;
  }
  return false;
}

// adjacency entries of one layer of one sample: (row,col) = (i,j) where transit i -- vertex j is an edge.  A transit
// with a bitmap of its neighbours (hub_slot, null: none have one) is asked by a bit test.
__device__ __forceinline__ void emit_adjacency(const NdGraphView &g, const CollParams &cp, const int32_t *tr,
                                               const int32_t *layer, int32_t *arow, int32_t *acol, const int32_t *hub_slot = nullptr,
                                               const uint32_t *hub_bits = nullptr, int words = 0) {
  for (int e = threadIdx.x; e < cp.stride; e += blockDim.x) {
    const int i = e / cp.L, j = e - i * cp.L;
    int32_t ri = -1, cj = -1;
    if (i < cp.ntr) {
      const int32_t t = tr[i], v = layer[j];
      if (t >= 0 && t < cp.V && v >= 0 && v < cp.V) {
        const int32_t slot = hub_slot ? __ldg(hub_slot + t) : -1;
        const bool edge = slot >= 0 ? (__ldg(hub_bits + (size_t)slot * words + ((uint32_t)v >> 5)) >> (v & 31)) & 1u : has_edge_logn(g, t, v);
        if (edge) { ri = i; cj = j; }
      }
    }
    arow[e] = ri;
    acol[e] = cj;
  }
}

int nd_coll_bitmap_alloc(nd_sampler *s);
int nd_coll_bitmap_launch(nd_sampler *s, const CollParams &cp, unsigned long long pairs);
