// Graph side of the path on the device: CSR construction from edge records, the synthetic R-MAT
// generator, per-vertex max weight, and the byte-budget range partitioner.
//
// Replaces Graph::load_from_edge_list_binary + csr_from_graph (src/graph.hpp:106-159,
// src/csr.hpp:399-424: per-vertex std::vector, OpenMP std::sort, serial fill), transferCSRToGPUs
// (src/nextdoor.cu:1893-1911) and create_csr_partitions (src/graph_partitioner.cuh:1-173).
// The records are sorted by (src, dst, weight) with stable LSD sorts of the in-house radix sort (dst,
// then src; weights inside runs of equal edges), row offsets come from the boundaries of the sorted src array.
#include <fcntl.h>
#include <stdio.h>
#include <stdlib.h>
#include <string.h>
#include <sys/stat.h>
#include <unistd.h>

#include <algorithm>
#include <atomic>
#include <string>
#include <vector>

#include "nd_common.cuh"
#include "nd_host.h"
#include "nd_philox.cuh"

namespace {

// order-preserving map of fp32 onto uint32 (negative weights sort below positive ones)
__device__ __forceinline__ uint32_t float_to_key(float f) {
  const uint32_t b = __float_as_uint(f);
  return (b & 0x80000000u) ? ~b : (b | 0x80000000u);
}
__device__ __forceinline__ float key_to_float(uint32_t k) {
  return __uint_as_float((k & 0x80000000u) ? (k & 0x7fffffffu) : ~k);
}

struct Rec12 { int32_t s, d; float w; };

// What the build needs to know of the records: largest id, whether one is negative, and which bits of the
// weight keys differ between records (all others need no sorting).
struct RecordFacts {
  int32_t max_id;
  int32_t bad;
  uint32_t key_and, key_or;
};

__device__ __forceinline__ void facts_out(RecordFacts *facts, int32_t m, bool bad, uint32_t ka, uint32_t ko) {
  for (int o = 16; o > 0; o >>= 1) {
    m = max(m, __shfl_xor_sync(0xffffffffu, m, o));
    ka &= __shfl_xor_sync(0xffffffffu, ka, o);
    ko |= __shfl_xor_sync(0xffffffffu, ko, o);
  }
  bad = __any_sync(0xffffffffu, bad);
  if ((threadIdx.x & 31) == 0) {
    // (thousands of warps come to the same words: only what changes one goes on to the atomic; 8.4M records 58 -> 42 us)
    if (m > __ldcg(&facts->max_id)) atomicMax(&facts->max_id, m);
    if (bad) atomicOr(&facts->bad, 1);
    if (__ldcg(&facts->key_and) & ~ka) atomicAnd(&facts->key_and, ka);
    if (ko & ~__ldcg(&facts->key_or)) atomicOr(&facts->key_or, ko);
  }
}

__global__ void unpack_records_kernel(const Rec12 *__restrict__ rec, int64_t n, uint32_t *__restrict__ src,
                                      uint32_t *__restrict__ dst, uint32_t *__restrict__ wk, RecordFacts *__restrict__ facts) {
  int32_t m = -1;
  bool bad = false;
  uint32_t ka = 0xffffffffu, ko = 0u;
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    const Rec12 r = rec[i];
    const uint32_t k = float_to_key(r.w);
    src[i] = (uint32_t)r.s; dst[i] = (uint32_t)r.d; wk[i] = k;
    bad |= r.s < 0 || r.d < 0;
    m = max(m, max(r.s, r.d));
    ka &= k; ko |= k;
  }
  facts_out(facts, m, bad, ka, ko);
}

// the same for records that arrive as three arrays: the weights become their keys in place
__global__ void unpack_arrays_kernel(int64_t n, const uint32_t *__restrict__ src, const uint32_t *__restrict__ dst,
                                     uint32_t *__restrict__ wk, RecordFacts *__restrict__ facts) {
  int32_t m = -1;
  bool bad = false;
  uint32_t ka = 0xffffffffu, ko = 0u;
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    const int32_t s = (int32_t)src[i], d = (int32_t)dst[i];
    const uint32_t k = float_to_key(__uint_as_float(wk[i]));
    wk[i] = k;
    bad |= s < 0 || d < 0;
    m = max(m, max(s, d));
    ka &= k; ko |= k;
  }
  facts_out(facts, m, bad, ka, ko);
}

// Records whose weights are still on the way: what their ids say, and their places in the order of arrival.
__global__ void id_facts_kernel(int64_t n, const uint32_t *__restrict__ src, const uint32_t *__restrict__ dst, uint32_t *__restrict__ place,
                                RecordFacts *__restrict__ facts) {
  int32_t m = -1;
  bool bad = false;
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    const int32_t s = (int32_t)src[i], d = (int32_t)dst[i];
    place[i] = (uint32_t)i;
    bad |= s < 0 || d < 0;
    m = max(m, max(s, d));
  }
  facts_out(facts, m, bad, 0xffffffffu, 0u);
}

// ... and the weights' keys once these are there and the places sorted
__global__ void place_weights_kernel(int64_t n, const uint32_t *__restrict__ place, const float *__restrict__ w, uint32_t *__restrict__ wk,
                                     RecordFacts *__restrict__ facts) {
  uint32_t ka = 0xffffffffu, ko = 0u;
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    const uint32_t k = float_to_key(__ldg(w + place[i]));
    wk[i] = k;
    ka &= k; ko |= k;
  }
  facts_out(facts, -1, false, ka, ko);
}

// R-MAT (a,b,c,d) = (.57,.19,.19,.05).  Undirected edge e, attempt t: Philox counter
// (e_lo, e_hi, t, level/4), key = seed ^ "RMAT"; level l consumes draw l with integer quadrant
// thresholds; an attempt with an endpoint >= V or src == dst is retried; the weight is draw
// `scale` of the accepted attempt, 1 + 4 * (x>>8) * 2^-24.  Both directions are emitted.
__global__ void rmat_kernel(int32_t V, int scale, int64_t M, uint64_t seed, uint32_t *__restrict__ src,
                            uint32_t *__restrict__ dst, uint32_t *__restrict__ wk) {
  const uint32_t T1 = 2448131358u, T2 = 3264175144u, T3 = 4080218931u;
  const uint32_t k0 = (uint32_t)seed ^ 0x524D4154u, k1 = (uint32_t)(seed >> 32);
  for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < M; e += (int64_t)gridDim.x * blockDim.x) {
    int32_t s = 0, d = 0;
    float w = 0.f;
    for (uint32_t attempt = 0; attempt < (1u << 20); attempt++) {
      uint32_t o[4];
      s = 0; d = 0;
      bool ok = false;
      for (int l = 0; l <= scale; l++) {
        if ((l & 3) == 0) ndrng::philox4x32_10((uint32_t)e, (uint32_t)((uint64_t)e >> 32), attempt, (uint32_t)(l >> 2), k0, k1, o);
        const uint32_t x = (l & 3) == 0 ? o[0] : ((l & 3) == 1 ? o[1] : ((l & 3) == 2 ? o[2] : o[3]));
        if (l == scale) {
          if (s < V && d < V && s != d) {
            ok = true;
            w = __fadd_rn(1.0f, __fmul_rn(4.0f, __fmul_rn(__uint2float_rn(x >> 8), 5.9604644775390625e-08f)));
          }
          break;
        }
        int sb, db;
        if (x < T1) { sb = 0; db = 0; }
        else if (x < T2) { sb = 0; db = 1; }
        else if (x < T3) { sb = 1; db = 0; }
        else { sb = 1; db = 1; }
        s = (s << 1) | sb;
        d = (d << 1) | db;
      }
      if (ok) break;
    }
    const uint32_t key = float_to_key(w);
    src[2 * e] = s; dst[2 * e] = d; wk[2 * e] = key;
    src[2 * e + 1] = d; dst[2 * e + 1] = s; wk[2 * e + 1] = key;
  }
}

// Records sorted by (src, dst) in their order of arrival: the weights of records with the same pair are brought into
// order where they lie, by the thread that finds the first of them.  Almost all runs are of two or three; those longer
// than RUN_THREAD (an R-MAT graph's hub pairs) go on a list for a CTA each, and runs longer than RUN_CTA set *too_long.
constexpr int RUN_THREAD = 32, RUN_CTA = 4096;
struct RunList {
  int32_t too_long, count;
};
__global__ void sort_runs_kernel(const uint32_t *__restrict__ src, const uint32_t *__restrict__ dst, uint32_t *__restrict__ wk, int64_t n,
                                 RunList *__restrict__ runs, uint32_t *__restrict__ list, const RecordFacts *__restrict__ facts) {
  if (facts->key_and == facts->key_or) return;   // all weights are the same
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i + 1 < n; i += (int64_t)gridDim.x * blockDim.x) {
    const uint32_t s = src[i], d = dst[i], s1 = src[i + 1], d1 = dst[i + 1];   // (loads that do not wait for one another)
    if (s1 != s || d1 != d || (i > 0 && src[i - 1] == s && dst[i - 1] == d)) continue;
    int m = 2;
    while (m <= RUN_THREAD && i + m < n && src[i + m] == s && dst[i + m] == d) m++;
    if (m > RUN_THREAD) { list[atomicAdd(&runs->count, 1)] = (uint32_t)i; continue; }
    for (int k = 1; k < m; k++) {
      const uint32_t x = wk[i + k];
      int j = k;
      for (; j > 0 && wk[i + j - 1] > x; j--) wk[i + j] = wk[i + j - 1];
      wk[i + j] = x;
    }
  }
}

// a CTA per listed run: bitonic sort in shared memory (16 KB)
__global__ void __launch_bounds__(256) sort_long_runs_kernel(const uint32_t *__restrict__ src, const uint32_t *__restrict__ dst, uint32_t *__restrict__ wk,
                                                             int64_t n, RunList *__restrict__ runs, const uint32_t *__restrict__ list) {
  __shared__ uint32_t key[RUN_CTA];
  __shared__ int end;
  const int count = runs->count;
  for (int r = blockIdx.x; r < count; r += gridDim.x) {
    const int64_t at = list[r];
    const uint32_t s = src[at], d = dst[at];
    __syncthreads();
    if (threadIdx.x == 0) {   // past the last record of the run, which lie together: bisection over the window
      int64_t lo = at, hi = n - at > RUN_CTA ? at + RUN_CTA + 1 : n;
      while (hi - lo > 1) {
        const int64_t mid = (lo + hi) >> 1;
        if (src[mid] == s && dst[mid] == d) lo = mid;
        else hi = mid;
      }
      end = (int)(hi - at);
    }
    __syncthreads();
    const int m = end;
    if (m > RUN_CTA) {
      if (threadIdx.x == 0) runs->too_long = 1;
      continue;
    }
    int size = 64;
    while (size < m) size *= 2;
    for (int k = threadIdx.x; k < size; k += blockDim.x) key[k] = k < m ? wk[at + k] : 0xffffffffu;
    for (int width = 2; width <= size; width *= 2)
      for (int step = width / 2; step > 0; step /= 2) {
        __syncthreads();
        for (int k = threadIdx.x; k < size / 2; k += blockDim.x) {
          const int x = (k / step) * 2 * step + k % step, y = x + step;
          const uint32_t kx = key[x], ky = key[y];
          if ((kx > ky) == ((x & width) == 0)) { key[x] = ky; key[y] = kx; }
        }
      }
    __syncthreads();
    for (int k = threadIdx.x; k < m; k += blockDim.x) wk[at + k] = key[k];
  }
}

// The sorted records become the CSR: row_ptr (element i closes the rows (src[i-1], src[i]]) and col.
__global__ void csr_from_sorted_kernel(const uint32_t *__restrict__ src, const uint32_t *__restrict__ dst, int64_t n, int32_t V,
                                       int32_t *__restrict__ row_ptr, int32_t *__restrict__ col) {
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i <= n; i += (int64_t)gridDim.x * blockDim.x) {
    const int64_t lo = i == 0 ? 0 : (int64_t)src[i - 1] + 1;
    const int64_t hi = i == n ? V : (int64_t)src[i];
    for (int64_t v = lo; v <= hi; v++) row_ptr[v] = (int32_t)i;
    if (i < n) col[i] = (int32_t)dst[i];
  }
}

// Vertex::max_weight (src/graph.hpp:71-80) starts from 0, so only positive weights can raise it
// and their bit patterns order like ints.  Thread per edge; the owner row comes from the sorted
// src array when the CSR was just built here, else from a bisection of row_ptr; a warp whose 32
// edges share one row reduces first and issues a single atomic.  With wk, the sorted weights' keys, it makes the weights, too.
__global__ void max_weight_kernel(const int32_t *__restrict__ row_ptr, const uint32_t *__restrict__ src, const uint32_t *__restrict__ wk,
                                  float *__restrict__ w, int32_t V, int64_t E, int32_t *__restrict__ max_w_bits) {
  for (int64_t base = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) & ~31ll; base < E;
       base += (int64_t)gridDim.x * blockDim.x) {
    const int64_t i = base + (threadIdx.x & 31);
    const bool in = i < E;
    const float x = !in ? 0.f : wk ? key_to_float(wk[i]) : w[i];
    if (in && wk) w[i] = x;
    int32_t v = -1;
    if (in) {
      if (src) {
        v = (int32_t)src[i];
      } else {  // largest v with row_ptr[v] <= i
        int32_t lo = 0, hi = V;
        while (hi - lo > 1) {
          const int32_t mid = lo + (hi - lo) / 2;
          if ((int64_t)row_ptr[mid] <= i) lo = mid; else hi = mid;
        }
        v = lo;
      }
    }
    const uint32_t peers = __match_any_sync(0xffffffffu, v);
    float m = x;
    if (peers == 0xffffffffu) {
      for (int o = 16; o > 0; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
      if ((threadIdx.x & 31) == 0 && in && m > 0.f) atomicMax(max_w_bits + v, __float_as_int(m));
    } else if (in && m > 0.f) {
      atomicMax(max_w_bits + v, __float_as_int(m));
    }
  }
}

__global__ void max_degree_kernel(const int32_t *__restrict__ row_ptr, int32_t V, int32_t *__restrict__ out) {
  int32_t m = 0;
  for (int64_t v = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; v < V; v += (int64_t)gridDim.x * blockDim.x)
    m = max(m, row_ptr[v + 1] - row_ptr[v]);
  for (int o = 16; o > 0; o >>= 1) m = max(m, __shfl_xor_sync(0xffffffffu, m, o));
  if ((threadIdx.x & 31) == 0) atomicMax(out, m);
}

// Greedy byte-budget partitioner.  Partition k starts at (u, e_start); with
// G(v) = 4*(row_ptr[v+1] - max(e_start,row_ptr[u])) + 16*(v-u+1) (strictly increasing in v) it is
// closed at the first v with G(v) >= budget, found by bisection.  One thread: the work is
// n_parts * log2(V) dependent loads.
__global__ void partition_kernel(const int32_t *__restrict__ row_ptr, int32_t V, long long budget, int max_parts,
                                 int32_t *__restrict__ first_v, int32_t *__restrict__ last_v,
                                 long long *__restrict__ first_e, long long *__restrict__ last_e,
                                 int32_t *__restrict__ n_parts) {
  if (blockIdx.x != 0 || threadIdx.x != 0) return;
  int np = 0;
  int32_t u = 0;
  long long e_start = 0;
  const long long E = row_ptr[V];
  while (u < V && np < max_parts) {
    const long long es = e_start > row_ptr[u] ? e_start : (long long)row_ptr[u];
    // first v in [u, V) with G(v) >= budget
    int32_t lo = u, hi = V;  // answer in [lo, hi]; hi == V means none
    while (lo < hi) {
      const int32_t mid = lo + (hi - lo) / 2;
      const long long G = 4 * ((long long)row_ptr[mid + 1] - es) + 16 * (long long)(mid - u + 1);
      if (G >= budget) hi = mid; else lo = mid + 1;
    }
    int32_t u_end;
    long long e_end;
    bool closed = lo < V;
    if (!closed) {
      u_end = V - 1; e_end = E - 1;
    } else {
      const int32_t v = lo;
      const long long s = v == u ? es : (long long)row_ptr[v];
      const long long edges = (long long)row_ptr[v + 1] - s;
      const long long n_edges = s - es;
      const long long nv = v - u + 1;
      long long room = (budget - nv * 16) / 4 - n_edges;
      if (room < 0) room = 0;
      if (room >= edges) { u_end = v; e_end = s + edges - 1; }
      else if (v > u) { u_end = v - 1; e_end = s - 1; }
      else { if (room == 0) room = 1; u_end = v; e_end = s + room - 1; }
    }
    first_v[np] = u; last_v[np] = u_end; first_e[np] = e_start; last_e[np] = e_end;
    np++;
    if (!closed) break;
    e_start = e_end + 1;
    u = e_start >= row_ptr[u_end + 1] ? u_end + 1 : u_end;
  }
  *n_parts = np;
}

int grid_for(int64_t n, int threads, int sms) {
  int64_t b = (n + threads - 1) / threads;
  const int64_t cap = (int64_t)sms * 16;
  if (b > cap) b = cap;
  return (int)(b > 0 ? b : 1);
}

// Device memory of a build in one allocation:
// the records twice -- (src, dst, weight key) and the sort's other side --, the sort's histograms, small words.
// 32 bytes of padding behind every array.
struct BuildScratch {
  unsigned char *base = nullptr;
  uint32_t *a[3], *b[3];
  Rec12 *rec;                // over b: 12-byte records before they are unpacked into a
  NdRadixScratch radix;
  RecordFacts *facts;
  int32_t *d_n, *d_max_degree;
  RunList *runs;
  int device = 0;
  size_t bytes = 0;
  ~BuildScratch() { nd_block_free(device, base, bytes); }
};

int build_scratch(BuildScratch *s, int device, int64_t n) {
  s->device = device;
  const size_t words = ((size_t)(n > 0 ? n : 1) + 8 + 63) & ~(size_t)63;
  const NdRadixPlan pl = nd_radix_plan(32, n);
  const size_t radix = nd_radix_scratch_bytes(n);
  s->bytes = 24 * words + radix + 256;
  ND_TRY(nd_block_alloc(device, (void **)&s->base, &s->bytes));
  for (int w = 0; w < 3; w++) { s->a[w] = (uint32_t *)s->base + w * words; s->b[w] = (uint32_t *)s->base + (3 + w) * words; }
  s->rec = (Rec12 *)s->b[0];
  unsigned char *p = s->base + 24 * words;
  s->facts = (RecordFacts *)p;
  s->d_n = (int32_t *)(p + 64);
  s->d_max_degree = (int32_t *)(p + 128);
  s->runs = (RunList *)(p + 192);
  nd_radix_scratch_place(&s->radix, pl, p + 256);
  const RecordFacts none{-1, 0, 0xffffffffu, 0u};
  const int32_t n32 = (int32_t)n;
  ND_CUDA(cudaMemset(p + 128, 0, radix + 128));
  ND_CUDA(cudaMemcpy(s->facts, &none, sizeof(none), cudaMemcpyHostToDevice));
  ND_CUDA(cudaMemcpy(s->d_n, &n32, sizeof(n32), cudaMemcpyHostToDevice));
  return ND_OK;
}

// records in bs->a (weights as keys) -> graph; key bits outside [lo_bit, hi_bit) are the same in all records.  They are
// sorted by dst, then src, and the few that share both by weight where they lie: 6 passes instead of 10 over random edges
// with random weights (8.4M records on the host to a graph, copies included: 6.1 ms -> 4.9; 2.8 since the scatter of
// nd_radix.cu, 0.11 a pass, and with the ids sorted while the weights are on the wire).  A graph that repeats one edge thousands of times goes
// on to the full sort.
struct Build {
  const NdDeviceInfo &dev;
  const int64_t n;
  const int32_t V;
  BuildScratch *bs;
  const int vbits;
  uint32_t *cur[3], *oth[3];
  nd_graph *g = nullptr;

  Build(const NdDeviceInfo &dev_, int64_t n_, int32_t V_, BuildScratch *bs_)
      : dev(dev_), n(n_), V(V_), bs(bs_), vbits(nd_bit_length((uint32_t)(V_ > 1 ? V_ - 1 : 1))) {
    for (int w = 0; w < 3; w++) { cur[w] = bs->a[w]; oth[w] = bs->b[w]; }
  }
  ~Build() {   // a build that fails gives the graph's memory back
    if (!g) return;
    nd_block_free(dev.device, g->block, g->block_bytes);
    delete g;
  }

  int sort_by(int word, int bits, int lo) {
    if (n < 2 || bits <= 0) return ND_OK;
    NdSortArrays arr;
    arr.nwords = 3;
    for (int w = 0; w < 3; w++) { arr.a[w] = cur[w]; arr.b[w] = oth[w]; }
    bool in_b = false;
    NdRadixPlan pl = nd_radix_plan(bits, n);
    for (int p = 0; p < pl.passes; p++) pl.shift[p] += lo;
    ND_TRY(nd_radix_sort(dev, nullptr, &bs->radix, pl, arr, word, bs->d_n, nullptr, false, 0u, false, &in_b));
    if (in_b) for (int w = 0; w < 3; w++) { uint32_t *t = cur[w]; cur[w] = oth[w]; oth[w] = t; }
    return ND_OK;
  }
  int sort_by_ids() {
    ND_TRY(sort_by(1, vbits, 0));
    return sort_by(0, vbits, 0);
  }

  // cur[2] (weight keys) of records that share both ids, brought into order
  int sort_weights(int lo_bit, int hi_bit) {
    if (hi_bit <= lo_bit || n <= 1) return ND_OK;
    RunList runs;
    sort_runs_kernel<<<grid_for(n, 256, dev.sms), 256>>>(cur[0], cur[1], cur[2], n, bs->runs, oth[0], bs->facts);
    sort_long_runs_kernel<<<dev.sms * 4, 256>>>(cur[0], cur[1], cur[2], n, bs->runs, oth[0]);
    nd_count_launches(2);
    ND_CUDA(cudaMemcpy(&runs, bs->runs, sizeof(runs), cudaMemcpyDeviceToHost));
    if (!runs.too_long) return ND_OK;
    ND_TRY(sort_by(2, hi_bit - lo_bit, lo_bit));
    return sort_by_ids();
  }

  // the graph's arrays, from the sorted ids
  int csr() {
    // one block: row offsets, ids and weights (32 bytes of padding for the 16-byte staging windows), maximum weights
    auto round = [](size_t b) { return (b + 255) & ~(size_t)255; };
    const size_t o_col = round(4 * ((size_t)V + 1)), o_w = o_col + round(4 * ((size_t)n + 8)), o_max = o_w + round(4 * ((size_t)n + 8));
    size_t all = o_max + round(4 * (size_t)V);
    unsigned char *block = nullptr;
    ND_TRY(nd_block_alloc(dev.device, (void **)&block, &all));
    g = new nd_graph();
    g->device = dev.device; g->V = V; g->E = n; g->block = block; g->block_bytes = all;
    g->row_ptr = (int32_t *)block; g->col = (int32_t *)(block + o_col); g->w = (float *)(block + o_w); g->max_w = (float *)(block + o_max);
    ND_CUDA(cudaMemsetAsync(g->col + n, 0, sizeof(int32_t) * 8));
    ND_CUDA(cudaMemsetAsync(g->w + n, 0, sizeof(float) * 8));
    ND_CUDA(cudaMemsetAsync(g->max_w, 0, sizeof(float) * (size_t)V));
    csr_from_sorted_kernel<<<grid_for(n + 1, 256, dev.sms), 256>>>(cur[0], cur[1], n, V, g->row_ptr, g->col);
    max_degree_kernel<<<grid_for(V, 256, dev.sms), 256>>>(g->row_ptr, V, bs->d_max_degree);
    nd_count_launches(2);
    ND_CUDA(cudaGetLastError());
    return ND_OK;
  }

  // ... and the weights, from their sorted keys
  int finish(nd_graph **out) {
    if (n > 0) max_weight_kernel<<<grid_for(n, 256, dev.sms), 256>>>(g->row_ptr, cur[0], cur[2], g->w, V, n, (int32_t *)g->max_w);
    nd_count_launches(1);
    ND_CUDA(cudaGetLastError());
    ND_CUDA(cudaMemcpy(&g->max_degree, bs->d_max_degree, sizeof(int32_t), cudaMemcpyDeviceToHost));
    nd_objects_add(1);
    *out = g;
    g = nullptr;
    return ND_OK;
  }
};

int build_from_soa(const NdDeviceInfo &dev, int64_t n, int32_t V, BuildScratch *bs, int lo_bit, int hi_bit, nd_graph **out) {
  ND_REQUIRE(n < ((int64_t)1 << 31), ND_ERR_RANGE, "%lld edges do not fit the int32 edge index of the CSR", (long long)n);
  Build b(dev, n, V, bs);
  ND_TRY(b.sort_by_ids());
  ND_TRY(b.sort_weights(lo_bit, hi_bit));
  ND_TRY(b.csr());
  return b.finish(out);
}

}  // namespace

int nd_graph_finish(nd_graph *g, cudaStream_t st) {
  NdDeviceInfo dev;
  ND_TRY(nd_device_info(g->device, &dev));
  if (!g->max_w) {
    ND_CUDA(nd_malloc(&g->max_w, sizeof(float) * (size_t)(g->V > 0 ? g->V : 1)));
    ND_CUDA(cudaMemsetAsync(g->max_w, 0, sizeof(float) * (size_t)g->V, st));
    if (g->E > 0)
      max_weight_kernel<<<grid_for(g->E, 256, dev.sms), 256, 0, st>>>(g->row_ptr, nullptr, nullptr, g->w, g->V, g->E, (int32_t *)g->max_w);
  }
  NdDevMem<int32_t> m;
  ND_TRY(m.alloc(1));
  ND_CUDA(cudaMemsetAsync(m.p, 0, sizeof(int32_t), st));
  max_degree_kernel<<<grid_for(g->V, 256, dev.sms), 256, 0, st>>>(g->row_ptr, g->V, m.p);
  ND_CUDA(cudaMemcpyAsync(&g->max_degree, m.p, sizeof(int32_t), cudaMemcpyDeviceToHost, st));
  ND_CUDA(cudaStreamSynchronize(st));
  return ND_OK;
}

static void free_graph(nd_graph *g) {
  if (g->block) nd_block_free(g->device, g->block, g->block_bytes);
  else { cudaFree(g->row_ptr); cudaFree(g->col); cudaFree(g->w); cudaFree(g->max_w); }
  cudaFree(g->colw); cudaFree(g->vrec); cudaFree(g->vrow); cudaFree(g->erec); cudaFree(g->pack); cudaFree(g->codes); cudaFree(g->col3); cudaFree(g->adjset); cudaFree(g->adjsign);
  cudaFree(g->deg_codes); cudaFree(g->term); cudaFree(g->hub_slot); cudaFree(g->hub_bits); cudaFree(g->hubs); cudaFree(g->hub_ids); cudaFree(g->hub_terms); cudaFree(g->hub_offs);
  for (const NdHubTable &t : g->hub_tables) { cudaFree(t.sums); cudaFree(t.starts); }
  delete g;
}

extern "C" {

int nd_graph_from_csr(int device, int32_t V, int64_t E, const int32_t *row_ptr, const int32_t *col,
                      const float *w, const float *max_w, nd_graph **out) {
  ND_REQUIRE(out && row_ptr && (E == 0 || (col && w)) && V >= 1 && E >= 0, ND_ERR_ARG, "nd_graph_from_csr: bad argument");
  ND_REQUIRE(E < ((int64_t)1 << 31), ND_ERR_RANGE, "%lld edges do not fit the int32 edge index of the CSR", (long long)E);
  ND_REQUIRE(row_ptr[0] == 0 && row_ptr[V] == E, ND_ERR_ARG, "row_ptr must run from 0 to E");
  ND_CUDA(cudaSetDevice(device));
  nd_graph *g = new nd_graph();
  g->device = device; g->V = V; g->E = E;
  auto build = [&]() -> int {
    ND_CUDA(nd_malloc(&g->row_ptr, sizeof(int32_t) * ((size_t)V + 1)));
    // 32 bytes of padding: staging copies read whole 16-byte windows around a list
    ND_CUDA(nd_malloc(&g->col, sizeof(int32_t) * ((size_t)E + 8)));
    ND_CUDA(nd_malloc(&g->w, sizeof(float) * ((size_t)E + 8)));
    ND_CUDA(cudaMemset(g->col + E, 0, sizeof(int32_t) * 8));
    ND_CUDA(cudaMemset(g->w + E, 0, sizeof(float) * 8));
    ND_CUDA(cudaMemcpy(g->row_ptr, row_ptr, sizeof(int32_t) * ((size_t)V + 1), cudaMemcpyHostToDevice));
    if (E > 0) {
      void *const to[2] = {g->col, g->w};
      const void *const from[2] = {col, w};
      const size_t bytes[2] = {sizeof(int32_t) * (size_t)E, sizeof(float) * (size_t)E};
      ND_TRY(nd_copies_to_device(device, 2, to, from, bytes));
    }
    if (max_w) {
      ND_CUDA(nd_malloc(&g->max_w, sizeof(float) * (size_t)V));
      ND_CUDA(cudaMemcpy(g->max_w, max_w, sizeof(float) * (size_t)V, cudaMemcpyHostToDevice));
    }
    return nd_graph_finish(g, nullptr);
  };
  const int rc = build();
  if (rc != ND_OK) { free_graph(g); return rc; }
  nd_objects_add(1);
  *out = g;
  return ND_OK;
}

static int from_edge_records_min_v(int device, int64_t n, const void *records, int32_t min_v, nd_graph **out);

int nd_graph_from_edge_records(int device, int64_t n, const void *records, nd_graph **out) {
  return from_edge_records_min_v(device, n, records, 0, out);
}

// the vertex count that the ids ask for; min_v: its lower bound (the adjacency-list format numbers vertices by line,
// including lines without edges)
static int vertices_of(const RecordFacts &f, int32_t min_v, int32_t *V) {
  ND_REQUIRE(f.bad == 0 && f.max_id != 0x7fffffff, ND_ERR_RANGE, "edge records hold a negative or out-of-range vertex id");
  *V = f.max_id + 1 > 0 ? f.max_id + 1 : 1;  // vertex count = max id + 1 (src/graph.hpp:131-142)
  if (*V < min_v) *V = min_v;
  return ND_OK;
}

// the facts of the unpacked records decide the rest of the build
static int build_from_facts(const NdDeviceInfo &dev, int64_t n, int32_t min_v, BuildScratch *bs, nd_graph **out) {
  RecordFacts f;
  int32_t V;
  ND_CUDA(cudaGetLastError());
  ND_CUDA(cudaMemcpy(&f, bs->facts, sizeof(f), cudaMemcpyDeviceToHost));
  ND_TRY(vertices_of(f, min_v, &V));
  const uint32_t differ = f.key_and ^ f.key_or;
  int lo = 0, hi = nd_bit_length(differ);
  while (lo < hi && !((differ >> lo) & 1u)) lo++;
  return build_from_soa(dev, n, V, bs, n > 0 ? lo : 0, n > 0 ? hi : 0, out);
}

static int from_edge_records_min_v(int device, int64_t n, const void *records, int32_t min_v, nd_graph **out) {
  ND_REQUIRE(out && (records || n == 0) && n >= 0, ND_ERR_ARG, "nd_graph_from_edge_records: bad argument");
  ND_REQUIRE(n < ((int64_t)1 << 31), ND_ERR_RANGE, "%lld edges do not fit the int32 edge index of the CSR", (long long)n);
  ND_CUDA(cudaSetDevice(device));
  NdDeviceInfo dev;
  ND_TRY(nd_device_info(device, &dev));
  BuildScratch bs;
  ND_TRY(build_scratch(&bs, device, n));
  ND_TRY(nd_copy_to_device(device, bs.rec, records, sizeof(Rec12) * (size_t)n));
  unpack_records_kernel<<<grid_for(n, 256, dev.sms), 256>>>(bs.rec, n, bs.a[0], bs.a[1], bs.a[2], bs.facts);
  nd_count_launches(1);
  return build_from_facts(dev, n, min_v, &bs, out);
}

// From this many records on the ids are sorted, with their places as the third word, while the weights are on the wire
// (8.4 M records 3.07 -> 2.63 ms, 4.2 M 1.76 -> 1.47, 2.1 M 1.03 -> 0.95; 1 M 0.64 -> 0.60 to 0.69, 260 K 0.35 -> 0.42: the
// ids' facts are waited for in between).
static constexpr int64_t WEIGHTS_LATER = (int64_t)1 << 21;

int nd_graph_from_edges(int device, int64_t n, const int32_t *src, const int32_t *dst, const float *w, nd_graph **out) {
  ND_REQUIRE(out && ((src && dst && w) || n == 0) && n >= 0, ND_ERR_ARG, "nd_graph_from_edges: bad argument");
  ND_REQUIRE(n < ((int64_t)1 << 31), ND_ERR_RANGE, "%lld edges do not fit the int32 edge index of the CSR", (long long)n);
  ND_CUDA(cudaSetDevice(device));
  NdDeviceInfo dev;
  ND_TRY(nd_device_info(device, &dev));
  BuildScratch bs;
  ND_TRY(build_scratch(&bs, device, n));
  void *const to[3] = {bs.a[0], bs.a[1], bs.a[2]};
  const void *const from[3] = {src, dst, w};
  const size_t bytes[3] = {4 * (size_t)n, 4 * (size_t)n, 4 * (size_t)n};
  if (n < WEIGHTS_LATER) {
    ND_TRY(nd_copies_to_device(device, 3, to, from, bytes));
    unpack_arrays_kernel<<<grid_for(n, 256, dev.sms), 256>>>(n, bs.a[0], bs.a[1], bs.a[2], bs.facts);
    nd_count_launches(1);
    return build_from_facts(dev, n, 0, &bs, out);
  }
  ND_TRY(nd_copies_to_device(device, 2, to, from, bytes));
  id_facts_kernel<<<grid_for(n, 256, dev.sms), 256>>>(n, bs.a[0], bs.a[1], bs.a[2], bs.facts);
  nd_count_launches(1);
  RecordFacts f;
  int32_t V;
  ND_CUDA(cudaGetLastError());
  ND_CUDA(cudaMemcpy(&f, bs.facts, sizeof(f), cudaMemcpyDeviceToHost));
  ND_TRY(vertices_of(f, 0, &V));
  Build b(dev, n, V, &bs);
  ND_TRY(b.sort_by_ids());
  ND_TRY(b.csr());
  // they arrive in the graph's own array, which the sorts do not touch, and go from there to the sorted places as keys
  ND_TRY(nd_copy_to_device(device, b.g->w, w, bytes[2]));
  place_weights_kernel<<<grid_for(n, 256, dev.sms), 256>>>(n, b.cur[2], b.g->w, b.oth[2], bs.facts);
  std::swap(b.cur[2], b.oth[2]);
  nd_count_launches(1);
  ND_TRY(b.sort_weights(0, 32));
  return b.finish(out);
}

int nd_graph_load_edge_list_binary(int device, const char *path, nd_graph **out) {
  ND_REQUIRE(path && out, ND_ERR_ARG, "nd_graph_load_edge_list_binary: bad argument");
  const int fd = open(path, O_RDONLY);
  if (fd < 0) { nd_set_error("File '%s' not found", path); return ND_ERR_IO; }
  struct stat st;
  const int64_t n = fstat(fd, &st) == 0 ? (int64_t)st.st_size / 12 : -1;
  char *buf = n >= 0 ? (char *)malloc((size_t)(n * 12 > 0 ? n * 12 : 1)) : nullptr;
  std::atomic<bool> ok{buf != nullptr};
  if (buf)   // the workers read (and first touch) a range each
    nd_host_ranges(n * 12, nd_host_threads(), [&](int, int64_t at, int64_t end) {
      while (at < end) {
        const ssize_t got = pread(fd, buf + at, (size_t)(end - at), (off_t)at);
        if (got <= 0) { ok = false; return; }
        at += got;
      }
    });
  close(fd);
  if (!ok) { free(buf); nd_set_error("short read on '%s'", path); return ND_ERR_IO; }
  const int rc = nd_graph_from_edge_records(device, n, buf, out);
  free(buf);
  return rc;
}

// Text edge list (Graph::load_from_edge_list_txt, src/graph.hpp:162-254): whitespace-separated
// "src dst weight" triples, reading stops at the first zero (or missing) weight, and -- as the
// reference does (:210) -- every edge is stored with weight 0: this format carries topology only.
static int load_edge_list_text(int device, const char *path, nd_graph **out) {
  FILE *fp = fopen(path, "r");
  if (!fp) { nd_set_error("File '%s' not found", path); return ND_ERR_IO; }
  std::vector<Rec12> recs;
  long long a = 0, b = 0;
  double w = 0;
  while (fscanf(fp, "%lld %lld %lf", &a, &b, &w) == 3) {
    if (w == 0.0) break;
    if (a < 0 || b < 0 || a > 0x7ffffffe || b > 0x7ffffffe) { fclose(fp); nd_set_error("vertex id out of range in '%s'", path); return ND_ERR_RANGE; }
    recs.push_back(Rec12{(int32_t)a, (int32_t)b, 0.0f});
  }
  fclose(fp);
  return from_edge_records_min_v(device, (int64_t)recs.size(), recs.data(), 0, out);
}

// Text adjacency list (Graph::load_from_adjacency_list, src/graph.hpp:256-326): one vertex per
// line, "id nbr weight nbr weight ..."; vertices are renumbered by line order and neighbour ids
// are translated through that numbering (an id that never heads a line maps to 0, as the
// reference's unordered_map lookup does).
static int load_adjacency_list_text(int device, const char *path, nd_graph **out) {
  FILE *fp = fopen(path, "r");
  if (!fp) { nd_set_error("File '%s' cannot open", path); return ND_ERR_IO; }
  std::vector<Rec12> recs;
  std::vector<long long> ids;
  std::string line;
  std::vector<char> buf(1 << 20);
  while (fgets(buf.data(), (int)buf.size(), fp)) {
    line.assign(buf.data());
    while (!line.empty() && line.back() != '\n' && fgets(buf.data(), (int)buf.size(), fp)) line += buf.data();
    const char *p = line.c_str();
    char *end = nullptr;
    const long long id = strtoll(p, &end, 10);
    if (end == p) continue;  // blank line
    const int32_t row = (int32_t)ids.size();
    ids.push_back(id);
    p = end;
    for (;;) {
      const long long nb = strtoll(p, &end, 10);
      if (end == p) break;
      p = end;
      const float wt = strtof(p, &end);
      if (end == p) break;
      p = end;
      recs.push_back(Rec12{row, (int32_t)nb, wt});  // dst still holds the file's id
    }
  }
  fclose(fp);
  std::vector<std::pair<long long, int32_t>> order(ids.size());
  for (size_t i = 0; i < ids.size(); i++) order[i] = {ids[i], (int32_t)i};
  std::sort(order.begin(), order.end());
  for (Rec12 &r : recs) {
    auto it = std::lower_bound(order.begin(), order.end(), std::make_pair((long long)r.d, (int32_t)-1));
    // several lines with one id: the last one wins, like repeated assignment into the reference's map
    int32_t to = 0;
    while (it != order.end() && it->first == r.d) { to = it->second; ++it; }
    r.d = to;
  }
  return from_edge_records_min_v(device, (int64_t)recs.size(), recs.data(), (int32_t)ids.size(), out);
}

int nd_graph_load(int device, const char *path, const char *graph_type, const char *graph_format, nd_graph **out) {
  ND_REQUIRE(path && graph_type && graph_format && out, ND_ERR_ARG, "nd_graph_load: null argument");
  const bool edge_list = strcmp(graph_type, "edge-list") == 0, adj_list = strcmp(graph_type, "adj-list") == 0;
  ND_REQUIRE(edge_list || adj_list, ND_ERR_ARG, "Incorrect graph file type '%s'", graph_type);
  if (edge_list && strcmp(graph_format, "binary") == 0) return nd_graph_load_edge_list_binary(device, path, out);
  if (edge_list && strcmp(graph_format, "text") == 0) return load_edge_list_text(device, path, out);
  if (adj_list && strcmp(graph_format, "text") == 0) return load_adjacency_list_text(device, path, out);
  nd_set_error("graph_format '%s' not supported for graph_type '%s'", graph_format, graph_type);
  return ND_ERR_ARG;
}

int nd_graph_rmat(int device, int32_t V, int64_t M, uint64_t seed, nd_graph **out) {
  ND_REQUIRE(out && V >= 2 && M >= 1, ND_ERR_ARG, "nd_graph_rmat: bad argument");
  ND_REQUIRE(2 * M < ((int64_t)1 << 31), ND_ERR_RANGE, "%lld CSR entries do not fit the int32 edge index", (long long)(2 * M));
  ND_CUDA(cudaSetDevice(device));
  NdDeviceInfo dev;
  ND_TRY(nd_device_info(device, &dev));
  BuildScratch bs;
  ND_TRY(build_scratch(&bs, device, 2 * M));
  int scale = 0;
  while (((int64_t)1 << scale) < V) scale++;
  rmat_kernel<<<grid_for(M, 256, dev.sms), 256>>>(V, scale, M, seed, bs.a[0], bs.a[1], bs.a[2]);
  ND_CUDA(cudaGetLastError());
  return build_from_soa(dev, 2 * M, V, &bs, 0, 32, out);
}

int nd_graph_info(const nd_graph *g, int32_t *V, int64_t *E, int32_t *max_degree, int *device) {
  ND_REQUIRE(g, ND_ERR_ARG, "null graph");
  if (V) *V = g->V;
  if (E) *E = g->E;
  if (max_degree) *max_degree = g->max_degree;
  if (device) *device = g->device;
  return ND_OK;
}

int nd_graph_to_host(const nd_graph *g, int32_t *row_ptr, int32_t *col, float *w, float *max_w) {
  ND_REQUIRE(g, ND_ERR_ARG, "null graph");
  ND_CUDA(cudaSetDevice(g->device));
  void *const dst[4] = {row_ptr, col, w, max_w};
  const void *const src[4] = {g->row_ptr, g->col, g->w, g->max_w};
  const size_t bytes[4] = {row_ptr ? sizeof(int32_t) * ((size_t)g->V + 1) : 0, col ? sizeof(int32_t) * (size_t)g->E : 0,
                           w ? sizeof(float) * (size_t)g->E : 0, max_w ? sizeof(float) * (size_t)g->V : 0};
  ND_TRY(nd_copies_to_host(g->device, 4, dst, src, bytes));
  return ND_OK;
}

int nd_graph_device_ptrs(const nd_graph *g, const int32_t **row_ptr, const int32_t **col, const float **w,
                         const float **max_w) {
  ND_REQUIRE(g, ND_ERR_ARG, "null graph");
  if (row_ptr) *row_ptr = g->row_ptr;
  if (col) *col = g->col;
  if (w) *w = g->w;
  if (max_w) *max_w = g->max_w;
  return ND_OK;
}

int nd_graph_destroy(nd_graph *g) {
  if (!g) return ND_OK;
  cudaSetDevice(g->device);
  free_graph(g);
  nd_objects_add(-1);
  return ND_OK;
}

int nd_graph_partition(const nd_graph *g, int64_t budget_bytes, int32_t max_parts, int32_t *first_v,
                       int32_t *last_v, int64_t *first_e, int64_t *last_e, int32_t *n_parts) {
  ND_REQUIRE(g && first_v && last_v && first_e && last_e && n_parts && max_parts >= 1, ND_ERR_ARG, "nd_graph_partition: bad argument");
  ND_REQUIRE(budget_bytes >= 20, ND_ERR_ARG, "partition budget of %lld bytes cannot hold one vertex and one edge", (long long)budget_bytes);
  ND_CUDA(cudaSetDevice(g->device));
  NdDevMem<int32_t> fv, lv, parts;
  NdDevMem<long long> fe, le;
  ND_TRY(fv.alloc((size_t)max_parts));
  ND_TRY(lv.alloc((size_t)max_parts));
  ND_TRY(fe.alloc((size_t)max_parts));
  ND_TRY(le.alloc((size_t)max_parts));
  ND_TRY(parts.alloc(1));
  partition_kernel<<<1, 32>>>(g->row_ptr, g->V, budget_bytes, max_parts, fv.p, lv.p, fe.p, le.p, parts.p);
  ND_CUDA(cudaMemcpy(n_parts, parts.p, 4, cudaMemcpyDeviceToHost));
  const size_t k = (size_t)*n_parts;
  ND_CUDA(cudaMemcpy(first_v, fv.p, 4 * k, cudaMemcpyDeviceToHost));
  ND_CUDA(cudaMemcpy(last_v, lv.p, 4 * k, cudaMemcpyDeviceToHost));
  ND_CUDA(cudaMemcpy(first_e, fe.p, 8 * k, cudaMemcpyDeviceToHost));
  ND_CUDA(cudaMemcpy(last_e, le.p, 8 * k, cudaMemcpyDeviceToHost));
  return ND_OK;
}

}  // extern "C"
