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

// The adjacency of a layer of a sample is a bit per entry (entry i * L + j: transit i -- vertex j is an edge) in whole
// words; nd_sampler_aux hands it out as (row, col) = (i, j) or (-1, -1).
__host__ __device__ inline int adj_words(int stride) { return (stride + 31) / 32; }

// n pairs (list, vertex), by the whole CTA (whole warps): bit e of `bits`: the vertex of pair e is in its list.  pair(e, list, v)
// gives them, false: there is none.  A list with a bitmap (slot >= 0) is asked by a bit test, the others are bisected, a
// few pairs side by side: every step of a search waits for the one before.
struct PairList { int32_t rs, deg, slot; };
template <class Pair>
__device__ __forceinline__ void probe_pairs(const int32_t *__restrict__ col, const uint32_t *__restrict__ hub_bits, int words, int n, uint32_t *bits, Pair pair) {
  constexpr int SIDE = 4;
  const int lane = threadIdx.x & 31;
  for (int e0 = threadIdx.x; e0 - lane < n; e0 += SIDE * blockDim.x) {
    int32_t v[SIDE], l[SIDE], r[SIDE];   // searched for in [l, r)
    bool edge[SIDE];
#pragma unroll
    for (int k = 0; k < SIDE; k++) {
      const int e = e0 + k * (int)blockDim.x;
      PairList list;
      l[k] = r[k] = 0; v[k] = -1; edge[k] = false;
      if (e >= n || !pair(e, list, v[k])) continue;
      if (list.slot >= 0) {
        edge[k] = (__ldg(hub_bits + (size_t)list.slot * words + ((uint32_t)v[k] >> 5)) >> (v[k] & 31)) & 1u;
      } else {
        l[k] = list.rs;
        r[k] = list.rs + list.deg;
      }
    }
    for (bool more = true; more;) {
      more = false;
      int32_t m[SIDE], c[SIDE];
#pragma unroll
      for (int k = 0; k < SIDE; k++) {
        m[k] = l[k] + (r[k] - l[k]) / 2;
        c[k] = l[k] < r[k] ? __ldg(col + m[k]) : 0;
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
      if (lane == 0 && e < n) bits[e / 32] = word;
    }
  }
}

// the adjacency of one layer of one sample
__device__ __forceinline__ void emit_adjacency(const NdGraphView &g, const CollParams &cp, const int32_t *tr, const int32_t *layer, uint32_t *adj) {
  probe_pairs(g.col, nullptr, 0, cp.stride, adj, [&](int e, PairList &list, int32_t &v) {
    const int i = e / cp.L, j = e - i * cp.L;
    if (i >= cp.ntr) return false;
    const int32_t t = tr[i];
    v = layer[j];
    if (t < 0 || t >= cp.V || v < 0 || v >= cp.V) return false;
    list.rs = __ldg(g.row_ptr + t);
    list.deg = __ldg(g.row_ptr + t + 1) - list.rs;
    list.slot = -1;
    return true;
  });
}

int nd_coll_bitmap_alloc(nd_sampler *s);
int nd_coll_bitmap_launch(nd_sampler *s, const CollParams &cp, unsigned long long pairs);
