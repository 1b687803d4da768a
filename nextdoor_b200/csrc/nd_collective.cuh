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

// The adjacency of a layer of a sample is a bit per entry (entry i * L + j: transit i -- vertex j is an edge) in whole
// words; nd_sampler_aux hands it out as (row, col) = (i, j) or (-1, -1).
__host__ __device__ inline int adj_words(int stride) { return (stride + 31) / 32; }

// the adjacency of one layer of one sample, by the whole CTA (whole warps).  A transit
// with a bitmap of its neighbours (hub_slot, null: none have one) is asked by a bit test, the others' lists are bisected, a
// few entries at a time side by side: every step of a search waits for the one before.
__device__ __forceinline__ void emit_adjacency(const NdGraphView &g, const CollParams &cp, const int32_t *tr,
                                               const int32_t *layer, uint32_t *adj, const int32_t *hub_slot = nullptr,
                                               const uint32_t *hub_bits = nullptr, int words = 0) {
  constexpr int SIDE = 4;
  const int lane = threadIdx.x & 31;
  for (int e0 = threadIdx.x; e0 - lane < cp.stride; e0 += SIDE * blockDim.x) {
    int32_t v[SIDE], l[SIDE], r[SIDE];   // searched for in [l, r)
    bool edge[SIDE];
#pragma unroll
    for (int k = 0; k < SIDE; k++) {
      const int e = e0 + k * (int)blockDim.x, i = e / cp.L, j = e - i * cp.L;
      l[k] = r[k] = 0; v[k] = -1; edge[k] = false;
      if (e >= cp.stride || i >= cp.ntr) continue;
      const int32_t t = tr[i];
      v[k] = layer[j];
      if (t < 0 || t >= cp.V || v[k] < 0 || v[k] >= cp.V) continue;
      const int32_t slot = hub_slot ? __ldg(hub_slot + t) : -1;
      if (slot >= 0) {
        edge[k] = (__ldg(hub_bits + (size_t)slot * words + ((uint32_t)v[k] >> 5)) >> (v[k] & 31)) & 1u;
      } else {
        l[k] = __ldg(g.row_ptr + t);
        r[k] = __ldg(g.row_ptr + t + 1);
      }
    }
    for (bool more = true; more;) {
      more = false;
      int32_t m[SIDE], c[SIDE];
#pragma unroll
      for (int k = 0; k < SIDE; k++) {
        m[k] = l[k] + (r[k] - l[k]) / 2;
        c[k] = l[k] < r[k] ? __ldg(g.col + m[k]) : 0;
      }
#pragma unroll
      for (int k = 0; k < SIDE; k++) {
        if (l[k] >= r[k]) continue;
        if (c[k] == v[k]) { edge[k] = true; l[k] = r[k]; }
        else if (c[k] < v[k]) l[k] = m[k] + 1;
        else r[k] = m[k];
        more |= l[k] < r[k];
      }
    }
#pragma unroll
    for (int k = 0; k < SIDE; k++) {
      const int e = e0 + k * (int)blockDim.x;
      const uint32_t word = __ballot_sync(0xffffffffu, edge[k]);
      if (lane == 0 && e < cp.stride) adj[e / 32] = word;
    }
  }
}

int nd_coll_bitmap_alloc(nd_sampler *s);
int nd_coll_bitmap_launch(nd_sampler *s, const CollParams &cp, unsigned long long pairs);
