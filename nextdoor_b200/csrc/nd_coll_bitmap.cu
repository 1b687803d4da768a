// Importance-sampled layers (FastGCN, LADIES): a CTA per sample, all layers of all samples in one launch.
//
// The union of a sample's neighbour lists is a bitmap with a bit per vertex; the rank of a set bit is the
// candidate's index in the sorted unique union, so nothing is sorted.  Candidate weights are summed per group (FastGCN:
// of 512 vertices, LADIES: of 512 candidates) in fp64 and scanned; a draw bisects the group sums and finds its candidate
// inside one group with a warp.  Sums are fp64, so they agree with the sorted sequential order to ~1e-16 (FastGCN's
// integer weights sum exactly).
//
// What bounds it, and what is done about it (2^20 vertices, 1024 batches of 64, 2 layers of 64: FastGCN
// 4.8 -> 0.98 ms, LADIES 5.7 -> 2.44 ms).  One CTA fills an SM, and neither memory nor issue slots are full: FastGCN issues
// in 58 % of the cycles (612 M warp instructions; 5.6 GB out of the L2 at 24 % of its rate), LADIES in 46 % (1.09 G
// instructions for 131 M list entries, the distinct ones of 313 M); the warps wait for barriers between the phases, for
// shared memory and for loads:
//  * The second layer's transits are hubs (FastGCN draws them with the square of their degree), many of them the
//    same one: repeated transits of a batch are taken once (LADIES with their multiplicity).
//  * A hub's list (up to 140 K ids; FastGCN's second layer has 28 distinct hubs a sample) costs a shared-memory test per id.  Vertices with at least V/128 neighbours
//    have their neighbourhood as a bitmap, built once per graph: V/8 bytes that are ORed in registers, word by
//    word, and stored to the union once; and an adjacency probe of such a transit is a bit test.
//  * FastGCN's weights are summed without a list of candidates (writing that and fetching deg^2 one by one took more
//    than half of the time): the degrees lie in vertex order as two planes of bytes, a lane takes eight vertices with one
//    16-byte load, masks them with its byte of the bitmap and squares and sums them with dp4a.  Vertices with 2048
//    neighbours or more, whose squares would overflow the 32-bit group sums, are a short list per graph.
//  * LADIES' terms (w / rowsum)^2 depend on the edge alone: an array, built once per graph, instead of a pass over
//    the weights and a division per entry and sample.  They are added up in shared memory, in tiles of
//    consecutive candidates (lists are sorted, so a tile is a range of every list, all of them searched for at
//    once), not with atomics on global memory.  CSR arrays of a caller may hold rows in any order: those lists are gone
//    through whole for every tile.
#include <algorithm>
#include <cstdlib>
#include <mutex>
#include <vector>

#include "nd_collective.cuh"

namespace {

using ndrng::Rng;

constexpr int GROUP_WORDS = 16;   // words whose candidates are counted together
constexpr int GROUP = 512;        // candidates (FastGCN: vertices, GROUP_WORDS words) whose weights are summed together
constexpr int BIG_DEGREE = 2048;  // from here a vertex is on the list of big ones and its code is 0: 512 * 2047^2 < 2^31
constexpr int FLIGHT = 4;         // groups a warp sums at a time
constexpr int HUB = 128, LADIES_HUB = 64;   // a vertex with at least V / HUB neighbours has a bitmap of them, and is ORed from V / LADIES_HUB on
constexpr int BIG_LIST = 4096;    // lists at least this long are streamed by the whole CTA
constexpr int VEC = 4;            // 16-byte loads in flight per thread
constexpr int CHUNK = 128;        // list entries a warp takes at a time (LADIES)
constexpr int CHUNK_LOADS = CHUNK / 32;

// The bitmap, the counts of groups and quads of words and the CDF make the "big" part (V/8 + 5V/128 bytes).  It lives in
// shared memory when the whole layout fits the CTA's opt-in shared memory (graphs up to about 1.2 M vertices) and
// otherwise in a per-CTA slice of a global scratch array (glob_bytes > 0), where the same code runs on L2-resident
// words.  The rest is always in shared memory.
struct Layout {
  int words, groups;
  uint32_t off_gcdf, off_gpref, off_qpre;              // inside the big part (the bitmap is at 0)
  uint32_t off_red, off_tr, off_layer, off_ut, off_mult, off_pre, off_tile;   // inside shared memory
  uint32_t tile;                                       // accumulators in shared memory (LADIES)
  uint32_t bytes;                                      // dynamic shared memory of the launch
  uint32_t glob_bytes;                                 // per-CTA slice of the global scratch, 0 = big part in shared memory
};

struct Args {
  NdGraphView g;
  CollParams cp;
  int steps;
  int64_t S;
  Layout lay;
  unsigned char *gscratch;
  const int32_t *initial;
  int32_t *out;
  float *wts_all;                          // LADIES: [CTAs][V] the candidates' weights, in order
  int32_t *pos_all;                        // LADIES: [CTAs][tiles + 1][transits] where the tiles begin in the lists
  int pos_stride;                          // ... entries per CTA
  int sorted;                              // LADIES: the lists ascend, so that a tile is a range of each
  int32_t *adj_row, *adj_col;
  float *prob;
  const uint4 *__restrict__ deg;           // FastGCN: the degrees of eight vertices, low bytes (x, y), high bytes (z, w)
  const NdBigVertex *__restrict__ big;     // FastGCN: vertices with degrees from BIG_DEGREE, in order
  int n_big;
  const float *__restrict__ term;          // LADIES: (w / rowsum)^2 per entry
  const int32_t *__restrict__ hub_slot;    // [V] slot of the vertex's bitmap, -1: none
  const uint32_t *__restrict__ hub_bits;   // [slots][words]
  unsigned long long *acc;                 // counters of the running job: [0] draws, [5] ids, [6] candidates, [8] next sample, [10] CTAs done; zero between jobs
  unsigned long long *stats;               // published by the last CTA
  unsigned long long pairs;
};

// a transit of the batch: row start, degree, how often it occurs, bitmap slot
struct Transit { int32_t rs, deg, mult, slot; };

__device__ __forceinline__ void mark(uint32_t *bm, int32_t v) {
  const uint32_t bit = 1u << (v & 31);
  uint32_t *wp = bm + ((uint32_t)v >> 5);
  if (!(*(volatile uint32_t *)wp & bit)) atomicOr(wp, bit);  // lists overlap: most bits are set already
}

// Streams one neighbour list with `stride` cooperating threads and sets the neighbours' bits.  The body of the list is
// read as 16-byte vectors (the arrays are 256-byte aligned, so entry rs + head is 16-byte aligned for
// head = (4 - rs % 4) % 4), VEC vectors in flight per thread; head and tail entries one by one.
__device__ __forceinline__ void stream_list(const NdGraphView &g, uint32_t *bm, int32_t rs, int32_t deg, int me, int stride) {
  const int32_t *__restrict__ col = g.col + rs;
  int head = (4 - (rs & 3)) & 3;
  if (head > deg) head = deg;
  if (me < head) mark(bm, __ldg(col + me));
  const int n4 = (deg - head) >> 2;
  const int4 *__restrict__ col4 = reinterpret_cast<const int4 *>(col + head);
  for (int e0 = me; e0 < n4; e0 += stride * VEC) {
    int4 v[VEC];
#pragma unroll
    for (int k = 0; k < VEC; k++) v[k] = e0 + k * stride < n4 ? __ldg(col4 + e0 + k * stride) : make_int4(-1, -1, -1, -1);
#pragma unroll
    for (int k = 0; k < VEC; k++)
      if (v[k].x >= 0) { mark(bm, v[k].x); mark(bm, v[k].y); mark(bm, v[k].z); mark(bm, v[k].w); }
  }
  for (int e = head + (n4 << 2) + me; e < deg; e += stride) mark(bm, __ldg(col + e));
}

// exclusive (uint32) or inclusive (double) scan of an array by the whole CTA: every thread owns a contiguous
// chunk, the chunk totals are scanned through warp shuffles
__device__ __forceinline__ uint32_t scan_u32(uint32_t *a, int n, uint32_t *red) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, warps = blockDim.x >> 5;
  const int per = (n + blockDim.x - 1) / blockDim.x;
  const int b = min((int)threadIdx.x * per, n), e = min(b + per, n);
  uint32_t sum = 0;
  for (int i = b; i < e; i++) sum += a[i];
  uint32_t inc = sum;
  for (int o = 1; o < 32; o <<= 1) {
    const uint32_t t = __shfl_up_sync(0xffffffffu, inc, o);
    if (lane >= o) inc += t;
  }
  if (lane == 31) red[warp] = inc;
  __syncthreads();
  uint32_t base = inc - sum, total = 0;
  for (int w = 0; w < warps; w++) {
    if (w < warp) base += red[w];
    total += red[w];
  }
  for (int i = b; i < e; i++) { const uint32_t c = a[i]; a[i] = base; base += c; }
  __syncthreads();
  return total;
}

__device__ __forceinline__ void scan_f64(double *a, int n, double *red) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int per = (n + blockDim.x - 1) / blockDim.x;
  const int b = min((int)threadIdx.x * per, n), e = min(b + per, n);
  double sum = 0.0;
  for (int i = b; i < e; i++) sum += a[i];
  double inc = sum;
  for (int o = 1; o < 32; o <<= 1) {
    const double t = __shfl_up_sync(0xffffffffu, inc, o);
    if (lane >= o) inc += t;
  }
  if (lane == 31) red[warp] = inc;
  __syncthreads();
  double base = inc - sum;
  for (int w = 0; w < warp; w++) base += red[w];
  for (int i = b; i < e; i++) { base += a[i]; a[i] = base; }
  __syncthreads();
}

// vertex of rank r (r < number of candidates)
__device__ __forceinline__ int32_t vertex_of_rank(const uint32_t *bm, const uint32_t *gpref, int groups, uint32_t r) {
  int lo = 0, hi = groups - 1;   // last group with gpref <= r
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (gpref[mid] <= r) lo = mid; else hi = mid - 1;
  }
  uint32_t left = r - gpref[lo];
  for (int w = lo * GROUP_WORDS;; w++) {
    uint32_t bits = bm[w];
    const uint32_t c = __popc(bits);
    if (left >= c) { left -= c; continue; }
    while (left--) bits &= bits - 1;
    return (w << 5) + __ffs(bits) - 1;
  }
}

// first entry of the sorted list [e0, e1) that is at least v
__device__ __forceinline__ int32_t lower_bound(const int32_t *__restrict__ col, int32_t e0, int32_t e1, int32_t v) {
  while (e0 < e1) {
    const int32_t m = e0 + ((e1 - e0) >> 1);
    if (__ldg(col + m) < v) e0 = m + 1; else e1 = m;
  }
  return e0;
}

// bits 0..3 -> 0xff in bytes 0..3
__device__ __forceinline__ uint32_t byte_mask(uint32_t bits) { return (((bits & 15u) * 0x204081u) & 0x01010101u) * 255u; }

// sum of deg^2 over the vertices of `bits` (eight vertices, degrees as in Args::deg)
__device__ __forceinline__ uint32_t sum_squares(uint32_t bits, const uint4 &d) {
  const uint32_t m0 = byte_mask(bits), m1 = byte_mask(bits >> 4);
  const uint32_t l0 = d.x & m0, l1 = d.y & m1, h0 = d.z & m0, h1 = d.w & m1;
  const uint32_t ll = __dp4a(l1, l1, __dp4a(l0, l0, 0u)), lh = __dp4a(l1, h1, __dp4a(l0, h0, 0u)), hh = __dp4a(h1, h1, __dp4a(h0, h0, 0u));
  return ll + (lh << 9) + (hh << 16);
}

template <bool LADIES>
__global__ void __launch_bounds__(1024, 1)
coll_bitmap_kernel(const __grid_constant__ Args a) {
  extern __shared__ __align__(16) unsigned char smem[];
  __shared__ long long sh_sample;
  __shared__ int sh_hubs, sh_rest;
  const Layout &lay = a.lay;
  CollParams cp = a.cp;
  unsigned char *big = lay.glob_bytes ? a.gscratch + (size_t)blockIdx.x * lay.glob_bytes : smem;
  uint32_t *bm = reinterpret_cast<uint32_t *>(big);
  double *gcdf = reinterpret_cast<double *>(big + lay.off_gcdf);
  uint32_t *gpref = reinterpret_cast<uint32_t *>(big + lay.off_gpref);
  uint16_t *qpre = reinterpret_cast<uint16_t *>(big + lay.off_qpre);
  double *red = reinterpret_cast<double *>(smem + lay.off_red);   // 32 doubles, 32 words
  uint32_t *red_u = reinterpret_cast<uint32_t *>(red + 32);
  int32_t *sh_tr = reinterpret_cast<int32_t *>(smem + lay.off_tr);
  int32_t *sh_layer = reinterpret_cast<int32_t *>(smem + lay.off_layer);
  Transit *ut = reinterpret_cast<Transit *>(smem + lay.off_ut);
  int32_t *sh_mult = reinterpret_cast<int32_t *>(smem + lay.off_mult);   // how often a transit occurs; 0: an earlier one is the same
  uint32_t *pre = reinterpret_cast<uint32_t *>(smem + lay.off_pre);
  double *tile = reinterpret_cast<double *>(smem + lay.off_tile);
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, warps = blockDim.x >> 5;
  float *wts = LADIES ? a.wts_all + (size_t)blockIdx.x * (size_t)cp.V : nullptr;
  int32_t *pos_tab = LADIES ? a.pos_all + (size_t)blockIdx.x * (size_t)a.pos_stride : nullptr;
  unsigned long long ids_sum = 0, uniq_sum = 0, draws = 0;   // thread 0
  for (int64_t s = blockIdx.x; s < a.S;) {
    for (int step = 0; step < a.steps; step++) {
      cp.step = step;
      cp.ntr = step == 0 ? cp.B : cp.L;
      const int32_t *tr = transits_of(cp, a.initial, a.out, s);
      if (tid == 0) { sh_hubs = 0; sh_rest = 0; }
      for (int i = tid; i < cp.ntr; i += blockDim.x) {
        sh_tr[i] = step == 0 ? tr[i] : sh_layer[i];
        sh_mult[i] = 1;
      }
      __syncthreads();
      // ---- the batch's transits, each once: the hubs from the front of the list, the others from its end
      for (int q = tid; q < cp.ntr * cp.ntr; q += blockDim.x) {
        const int i = q / cp.ntr, j = q - i * cp.ntr;
        if (j > i && sh_tr[i] == sh_tr[j]) {   // the first of a kind counts the others, which are struck out (negative)
          atomicAdd(sh_mult + i, 1);
          atomicOr(sh_mult + j, (int)0x80000000);
        }
      }
      __syncthreads();
      unsigned long long ids = 0;
      for (int i = tid; i < cp.ntr; i += blockDim.x) {
        const int32_t t = sh_tr[i];
        if (t < 0 || t >= cp.V) continue;
        const int32_t rs = __ldg(a.g.row_ptr + t), deg = __ldg(a.g.row_ptr + t + 1) - rs, slot = __ldg(a.hub_slot + t);
        ids += (unsigned long long)deg;
        if (sh_mult[i] > 0) {
          // (LADIES goes through the lists again, so that a hub's bitmap saves it less)
          ut[slot >= 0 && (!LADIES || deg >= cp.V / LADIES_HUB) ? atomicAdd(&sh_hubs, 1) : cp.ntr - 1 - atomicAdd(&sh_rest, 1)] = Transit{rs, deg, sh_mult[i], slot};
        }
      }
      for (int o = 16; o > 0; o >>= 1) ids += __shfl_xor_sync(0xffffffffu, ids, o);
      if (lane == 0) reinterpret_cast<unsigned long long *>(red)[warp] = ids;
      __syncthreads();
      const int nh = sh_hubs, nu = nh + sh_rest;
      if (tid == 0) for (int w = 0; w < warps; w++) ids_sum += reinterpret_cast<unsigned long long *>(red)[w];
      // ---- the union: hubs' bitmaps, then the other lists
      for (int w4 = tid; w4 < lay.words / 4; w4 += blockDim.x) {
        uint4 u = make_uint4(0u, 0u, 0u, 0u);
#pragma unroll 8
        for (int i = 0; i < nh; i++) {
          const uint4 h = __ldg(reinterpret_cast<const uint4 *>(a.hub_bits + (size_t)ut[i].slot * lay.words) + w4);
          u.x |= h.x; u.y |= h.y; u.z |= h.z; u.w |= h.w;
        }
        reinterpret_cast<uint4 *>(bm)[w4] = u;
      }
      __syncthreads();
      const Transit *rest = ut + cp.ntr - (nu - nh);
      for (int i = warp; i < nu - nh; i += warps)   // short lists: a warp each
        if (rest[i].deg < BIG_LIST) stream_list(a.g, bm, rest[i].rs, rest[i].deg, lane, 32);
      for (int i = 0; i < nu - nh; i++)             // long lists: the whole CTA
        if (rest[i].deg >= BIG_LIST) stream_list(a.g, bm, rest[i].rs, rest[i].deg, tid, blockDim.x);
      __syncthreads();
      uint32_t U;
      int groups;
      if (!LADIES) {
        // ---- the groups' weights, and the number of candidates
        const uint8_t *bytes = reinterpret_cast<const uint8_t *>(bm);
        uint32_t seen = 0;
        groups = lay.groups;
        for (int g0 = warp * FLIGHT; g0 < groups; g0 += warps * FLIGHT) {
          uint32_t bits[2 * FLIGHT];
          uint4 d[2 * FLIGHT];
#pragma unroll
          for (int k = 0; k < 2 * FLIGHT; k++) {
            const int at = g0 * (GROUP / 8) + k * 32 + lane;
            bits[k] = at < groups * (GROUP / 8) ? bytes[at] : 0u;
            d[k] = bits[k] ? __ldg(a.deg + at) : make_uint4(0u, 0u, 0u, 0u);
          }
#pragma unroll
          for (int k = 0; k < FLIGHT; k++) {
            seen += __popc(bits[2 * k] | bits[2 * k + 1] << 8);
            const uint32_t sum = __reduce_add_sync(0xffffffffu, sum_squares(bits[2 * k], d[2 * k]) + sum_squares(bits[2 * k + 1], d[2 * k + 1]));
            if (lane == 0 && g0 + k < groups) gcdf[g0 + k] = (double)sum;
          }
        }
        seen = __reduce_add_sync(0xffffffffu, seen);
        if (lane == 0) red_u[warp] = seen;
        __syncthreads();
        U = 0;
        for (int w = 0; w < warps; w++) U += red_u[w];
        for (int i0 = warp * 32; i0 < a.n_big; i0 += warps * 32) {   // the big ones; neighbours on the list mostly share a group
          const NdBigVertex v = i0 + lane < a.n_big ? a.big[i0 + lane] : NdBigVertex{-1, 0.f};
          const bool in = v.v >= 0 && ((bm[v.v >> 5] >> (v.v & 31)) & 1u);
          double x = in ? (double)v.weight : 0.0;
          int same;
          __match_all_sync(0xffffffffu, v.v / GROUP, &same);
          if (same) {
            for (int o = 16; o > 0; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
            if (lane == 0) atomicAdd(gcdf + v.v / GROUP, x);
          } else if (in) {
            atomicAdd(gcdf + v.v / GROUP, x);
          }
        }
      } else {
        // ---- candidates per group (and per quad of words inside it): half a warp takes the 16 words of a group
        for (int w0 = warp * 32; w0 < lay.words; w0 += warps * 32) {
          const int w = w0 + lane;
          const uint32_t bits = w < lay.words ? bm[w] : 0u;
          const uint32_t c = __popc(bits);
          uint32_t inc = c;
          for (int o = 1; o < GROUP_WORDS; o <<= 1) {
            const uint32_t t = __shfl_up_sync(0xffffffffu, inc, o, GROUP_WORDS);
            if ((lane & (GROUP_WORDS - 1)) >= o) inc += t;
          }
          if (w < lay.words) {
            if ((lane & (GROUP_WORDS - 1)) == GROUP_WORDS - 1) gpref[w / GROUP_WORDS] = inc;
            if ((lane & 3) == 0) qpre[w >> 2] = (uint16_t)(inc - c);
          }
        }
        __syncthreads();
        U = scan_u32(gpref, lay.groups, red_u);
        groups = (int)((U + GROUP - 1) / GROUP);   // of candidates
        // ---- the terms of every list entry, added up per candidate in tiles of consecutive candidates
        auto transit = [&](int i) -> const Transit & { return ut[i < nh ? i : cp.ntr - nu + i]; };
        int32_t *sh_pos = sh_mult;   // not needed any more
        const int tiles = (int)((U + lay.tile - 1) / lay.tile);
        for (int q = tid; a.sorted && q < (tiles + 1) * nu; q += blockDim.x) {   // where every tile begins in every list
          const int k = q / nu, i = q - k * nu;
          const Transit t = transit(i);
          int32_t e = t.rs;
          if (k == tiles) e = t.rs + t.deg;
          else if (k > 0) e = lower_bound(a.g.col, t.rs, t.rs + t.deg, vertex_of_rank(bm, gpref, lay.groups, (uint32_t)k * lay.tile));
          pos_tab[q] = e;
        }
        for (int k = 0; k < tiles; k++) {
          const uint32_t r0 = (uint32_t)k * lay.tile, n = min(lay.tile, U - r0);
          const int32_t *pos = pos_tab + k * nu;
          __syncthreads();
          for (uint32_t r = tid; r < n; r += blockDim.x) tile[r] = 0.0;
          for (int i = tid; i < nu; i += blockDim.x) {
            // (lists in another order are gone through whole for every tile)
            const int32_t at = a.sorted ? __ldcg(pos + i) : transit(i).rs;
            sh_pos[i] = at;
            pre[i] = a.sorted ? (uint32_t)(__ldcg(pos + nu + i) - at) : (uint32_t)transit(i).deg;
          }
          __syncthreads();
          const uint32_t total = scan_u32(pre, nu, red_u);
          for (uint32_t c0 = (uint32_t)warp * CHUNK; c0 < total; c0 += (uint32_t)warps * CHUNK) {
            int lo = 0, hi = nu - 1;   // transit of the chunk's first entry: the last with pre <= c0
            while (lo < hi) {
              const int mid = (lo + hi + 1) >> 1;
              if (pre[mid] <= c0) lo = mid; else hi = mid - 1;
            }
            int32_t v[CHUNK_LOADS];
            float x[CHUNK_LOADS];
            int m[CHUNK_LOADS];
#pragma unroll
            for (int j = 0; j < CHUNK_LOADS; j++) {
              const uint32_t f = c0 + (uint32_t)(j * 32 + lane);
              v[j] = -1; x[j] = 0.f; m[j] = 0;
              if (f < total) {
                while (lo + 1 < nu && pre[lo + 1] <= f) lo++;
                const int32_t e = sh_pos[lo] + (int32_t)(f - pre[lo]);
                v[j] = __ldg(a.g.col + e);
                x[j] = __ldg(a.term + e);
                m[j] = transit(lo).mult;
              }
            }
#pragma unroll
            for (int j = 0; j < CHUNK_LOADS; j++)
              if (v[j] >= 0) {
                const uint32_t word = (uint32_t)v[j] >> 5, quad = word >> 2, in_quad = word & 3u;
                const uint4 q = *reinterpret_cast<const uint4 *>(bm + 4 * quad);
                uint32_t r = gpref[word / GROUP_WORDS] + qpre[quad];
                r += in_quad > 0 ? __popc(q.x) : 0;
                r += in_quad > 1 ? __popc(q.y) : 0;
                r += in_quad > 2 ? __popc(q.z) : 0;
                const uint32_t own = in_quad == 0 ? q.x : in_quad == 1 ? q.y : in_quad == 2 ? q.z : q.w;
                r += __popc(own & ((1u << (v[j] & 31)) - 1u));
                if (r - r0 < n) atomicAdd(tile + (r - r0), (double)x[j] * (double)m[j]);
              }
          }
          __syncthreads();
          for (uint32_t g0 = (uint32_t)warp * GROUP; g0 < n; g0 += (uint32_t)warps * GROUP) {   // weights out, and the groups' sums
            double sum = 0.0;
            for (uint32_t r = g0 + lane; r < g0 + GROUP && r < n; r += 32) {
              const float x = (float)tile[r];
              wts[r0 + r] = x;
              sum += (double)x;
            }
            for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
            if (lane == 0) gcdf[(r0 + g0) / GROUP] = sum;
          }
        }
      }
      __syncthreads();
      if (tid == 0) uniq_sum += U;
      scan_f64(gcdf, groups, red);
      const double total = groups > 0 ? gcdf[groups - 1] : 0.0;
      // ---- the layer's draws, a warp each
      for (int j = warp; j < cp.L; j += warps) {
        int32_t pick = cp.V;
        float pr = 0.f;
        if (U > 0 && total > 0.0) {
          Rng rng(cp.seed, (uint32_t)(cp.first_sample + s), (uint32_t)cp.step, (uint32_t)j);
          const double target = (double)rng.uniform() * total;
          int lo = 0, hi = groups - 1;  // first group whose prefix reaches the target (rounding: the last one takes what is above all)
          while (lo < hi) {
            const int mid = lo + (hi - lo) / 2;
            if (gcdf[mid] >= target) hi = mid; else lo = mid + 1;
          }
          // (a target of zero takes the first candidate of all, whatever its weight)
          if (!LADIES && target <= 0.0) while (!__any_sync(0xffffffffu, bm[lo * GROUP_WORDS + (lane & (GROUP_WORDS - 1))])) lo++;
          const double before = lo > 0 ? gcdf[lo - 1] : 0.0;
          // the group in four blocks of 128 candidates (FastGCN: vertices), a lane holding four of each: the first (block,
          // lane) that reaches the target, then the first of its candidates that does
          float x[4][4];
          uint32_t there = 0;   // which of the lane's sixteen are candidates
#pragma unroll
          for (int q = 0; q < 4; q++) {
            const uint32_t r = (uint32_t)(lo * GROUP + q * 128 + lane * 4);
            if (LADIES) {
#pragma unroll
              for (int k = 0; k < 4; k++) {
                x[q][k] = r + k < U ? __ldcg(wts + r + k) : 0.f;
                there |= r + k < U ? 1u << (4 * q + k) : 0u;
              }
            } else {
              const uint32_t bits = (bm[r >> 5] >> (r & 31)) & 15u;
              const uint32_t *codes = reinterpret_cast<const uint32_t *>(a.deg + (r >> 3)) + ((r >> 2) & 1u);
              const uint32_t low = bits ? __ldg(codes) : 0u, high = bits ? __ldg(codes + 2) : 0u;
              there |= bits << (4 * q);
#pragma unroll
              for (int k = 0; k < 4; k++) {
                int32_t d = (int32_t)((low >> (8 * k) & 255u) | (high >> (8 * k) & 255u) << 8);
                if (((bits >> k) & 1u) == 0) d = 0;
                else if (d == 0) d = __ldg(a.g.row_ptr + r + k + 1) - __ldg(a.g.row_ptr + r + k);
                x[q][k] = __fmul_rn(__int2float_rn(d), __int2float_rn(d));
              }
            }
          }
          double at_block = before, lane_before = 0.0;
          bool found = false;
          int bq = -1, bl = 0;
#pragma unroll
          for (int q = 0; q < 4; q++) {
            const double mine = ((double)x[q][0] + (double)x[q][1]) + ((double)x[q][2] + (double)x[q][3]);
            double run = mine;
            for (int o = 1; o < 32; o <<= 1) {
              const double t = __shfl_up_sync(0xffffffffu, run, o);
              if (lane >= o) run += t;
            }
            const bool some = (there >> (4 * q)) & 15u;
            const uint32_t reach = __ballot_sync(0xffffffffu, some && at_block + run >= target), any = __ballot_sync(0xffffffffu, some);
            // (nobody reaches it, by rounding: the last candidates of the group)
            if (bq < 0 || !found) {
              if (reach || any) {
                bq = q;
                bl = reach ? __ffs(reach) - 1 : 31 - __clz(any);
                lane_before = at_block + __shfl_sync(0xffffffffu, run - mine, bl);
                found = reach != 0u;
              }
            }
            at_block += __shfl_sync(0xffffffffu, run, 31);
          }
          const uint32_t first = (uint32_t)(lo * GROUP + bq * 128 + bl * 4);
          uint32_t rank = first;
          float wt = 0.f;
          double run = lane_before;
          bool hit = false;
          const uint32_t its = __shfl_sync(0xffffffffu, there, bl) >> (4 * bq);
#pragma unroll
          for (int k = 0; k < 4; k++) {
            const float own = bq == 0 ? x[0][k] : bq == 1 ? x[1][k] : bq == 2 ? x[2][k] : x[3][k];
            const float t = __shfl_sync(0xffffffffu, own, bl);
            run += (double)t;
            if (!hit && ((its >> k) & 1u)) {
              rank = first + k;
              wt = t;
              hit = run >= target;
            }
          }
          pick = LADIES ? vertex_of_rank(bm, gpref, lay.groups, rank) : (int32_t)rank;
          pr = (float)((double)wt / total);
        }
        if (lane == 0) {
          sh_layer[j] = pick;
          a.out[s * cp.fs + (int64_t)cp.step * cp.L + j] = pick;
          a.prob[s * cp.fs + (int64_t)cp.step * cp.L + j] = pr;
        }
      }
      if (tid == 0) { if (U > 0 && total > 0.0) draws += (unsigned long long)cp.L; }
      __syncthreads();
      const int64_t at = (s * a.steps + cp.step) * (int64_t)cp.stride;
      emit_adjacency(a.g, cp, sh_tr, sh_layer, a.adj_row + at, a.adj_col + at, a.hub_slot, a.hub_bits, lay.words);
      __syncthreads();
    }
    if (tid == 0) sh_sample = a.S > gridDim.x ? (long long)gridDim.x + (long long)atomicAdd(&a.acc[8], 1ull) : (long long)a.S;
    __syncthreads();
    s = sh_sample;
  }
  if (tid == 0) {
    atomicAdd(&a.acc[0], draws);
    atomicAdd(&a.acc[5], ids_sum);
    atomicAdd(&a.acc[6], uniq_sum);
    __threadfence();
    if (atomicAdd(&a.acc[10], 1ull) == (unsigned long long)gridDim.x - 1ull) {   // the last CTA
      __threadfence();
      for (int i = 0; i < 8; i++) { a.stats[i] = i == 1 ? a.pairs : __ldcg(&a.acc[i]); a.acc[i] = 0ull; }
      a.acc[8] = a.acc[10] = 0ull;
    }
  }
}

// ---------------------------------------------------------------- arrays built once per graph

// a thread per eight vertices; the big ones go on the list (of `cap`), in any order
__global__ void deg_build_kernel(const int32_t *__restrict__ row_ptr, int32_t V, int64_t units, uint4 *__restrict__ deg, NdBigVertex *__restrict__ big,
                                 int32_t *__restrict__ n_big, int cap) {
  for (int64_t u = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; u < units; u += (int64_t)gridDim.x * blockDim.x) {
    uint32_t low[2] = {0u, 0u}, high[2] = {0u, 0u};
    for (int k = 0; k < 8; k++) {
      const int64_t v = 8 * u + k;
      if (v >= V) break;
      const int32_t d = row_ptr[v + 1] - row_ptr[v];
      if (d >= BIG_DEGREE) {
        const int at = atomicAdd(n_big, 1);
        if (at < cap) big[at] = NdBigVertex{(int32_t)v, __fmul_rn(__int2float_rn(d), __int2float_rn(d))};
        continue;
      }
      low[k >> 2] |= (uint32_t)(d & 255) << (8 * (k & 3));
      high[k >> 2] |= (uint32_t)(d >> 8) << (8 * (k & 3));
    }
    deg[u] = make_uint4(low[0], low[1], high[0], high[1]);
  }
}

// fp64 sums of the rows' weights (the order of the adds does not matter)
__global__ void __launch_bounds__(BUILD_THREADS)
rowsum_build_kernel(const int32_t *__restrict__ row_ptr, const float *__restrict__ w, int32_t V, int64_t E, double *__restrict__ sum) {
  for_entry_spans(row_ptr, V, E, [&](int64_t e0, int64_t e1, int32_t lo, int32_t hi) {
    for (int64_t b = e0; b < e1; b += BUILD_THREADS) {
      const int64_t e = b + threadIdx.x;
      const int32_t v = e < e1 ? row_of_entry(row_ptr, lo, hi, e) : -1;
      double x = e < e1 ? (double)w[e] : 0.0;
      if (__match_any_sync(0xffffffffu, v) == 0xffffffffu) {   // a warp inside one row
        for (int o = 16; o > 0; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
        if ((threadIdx.x & 31) == 0 && v >= 0) atomicAdd(sum + v, x);
      } else if (v >= 0) {
        atomicAdd(sum + v, x);
      }
    }
  });
}

__global__ void __launch_bounds__(BUILD_THREADS)
unsorted_kernel(const int32_t *__restrict__ row_ptr, const int32_t *__restrict__ col, int32_t V, int64_t E, int *__restrict__ unsorted) {
  for_entries(row_ptr, V, E, [&](int64_t e, int32_t v) {
    if (e + 1 < (int64_t)row_ptr[v + 1] && col[e] > col[e + 1]) *unsorted = 1;
  });
}

__global__ void __launch_bounds__(BUILD_THREADS)
term_build_kernel(const int32_t *__restrict__ row_ptr, const float *__restrict__ w, const double *__restrict__ sum, int32_t V, int64_t E,
                  float *__restrict__ term) {
  for_entries(row_ptr, V, E, [&](int64_t e, int32_t v) {
    const float r = __fdiv_rn(w[e], (float)sum[v]);
    term[e] = __fmul_rn(r, r);
  });
}

// Vertices in the order in which they get a bitmap: more neighbours first, of equally many the lower id; no two the same.
__host__ __device__ __forceinline__ uint64_t hub_rank(int32_t deg, uint32_t v) { return (uint64_t)(uint32_t)deg << 32 | (0xffffffffu - v); }

__global__ void __launch_bounds__(256) hub_count_kernel(const int32_t *__restrict__ row_ptr, int32_t V, uint64_t least, int32_t *__restrict__ count) {
  int32_t n = 0;
  for (int64_t v = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; v < V; v += (int64_t)gridDim.x * blockDim.x)
    n += hub_rank(row_ptr[v + 1] - row_ptr[v], (uint32_t)v) >= least ? 1 : 0;
  n = __reduce_add_sync(0xffffffffu, n);
  if ((threadIdx.x & 31) == 0 && n) atomicAdd(count, n);
}

__global__ void hub_slots_kernel(const int32_t *__restrict__ row_ptr, int32_t V, uint64_t least, int cap, int32_t *__restrict__ slot,
                                 int32_t *__restrict__ hubs, int32_t *__restrict__ count) {
  for (int64_t v = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; v < V; v += (int64_t)gridDim.x * blockDim.x) {
    int32_t at = -1;
    if (hub_rank(row_ptr[v + 1] - row_ptr[v], (uint32_t)v) >= least) {
      at = atomicAdd(count, 1);
      if (at < cap) hubs[at] = (int32_t)v; else at = -1;
    }
    slot[v] = at;
  }
}

// a CTA row per hub, `gridDim.y` CTAs share its list
__global__ void hub_bits_kernel(const int32_t *__restrict__ row_ptr, const int32_t *__restrict__ col, const int32_t *__restrict__ hubs, int words,
                                uint32_t *__restrict__ bits) {
  const int32_t v = hubs[blockIdx.x];
  uint32_t *b = bits + (size_t)blockIdx.x * words;
  for (int32_t e = row_ptr[v] + blockIdx.y * blockDim.x + threadIdx.x; e < row_ptr[v + 1]; e += gridDim.y * blockDim.x) {
    const uint32_t u = (uint32_t)col[e];
    atomicOr(b + (u >> 5), 1u << (u & 31u));
  }
}

int words_of(int32_t V) { return (int)((((int64_t)V + 31) / 32 + GROUP_WORDS - 1) / GROUP_WORDS * GROUP_WORDS); }

// A bitmap pays against the list it replaces from about V/128 neighbours: four times the list's bytes, but ORed a word
// at a time (FastGCN from V/64, V/128, V/192: 1.14, 0.98, 0.99 ms with 1024 batches on 2^20 vertices, 0.83, 0.59, 0.59
// with 256 on 2^21).
// At most HUBS of them, those with the most neighbours: a graph can hold 128 E / V such vertices.  (1024 batches on 233 K
// vertices and 114 M entries: FastGCN 4.1 ms with the 1024 that came first, 0.79 with the largest; LADIES, which goes
// through the lists again, 22.6 and 21.7.  Finding the rank adds 1.2 ms to the first sampler of such a graph.)
constexpr int HUBS = 1024;
std::mutex g_layers_mutex;

// bitmaps of the hubs' neighbourhoods
int ensure_hubs(const nd_graph *g, int grid) {
  if (g->hub_slot) return ND_OK;
  NdDevMem<int32_t> slot, hubs;
  NdDevMem<uint32_t> bits;
  ND_TRY(slot.alloc((size_t)g->V));
  ND_TRY(hubs.alloc(HUBS + 1));
  int32_t *const count = hubs.p + HUBS;
  int32_t n = 0;
  auto slots = [&](uint64_t least) -> int {
    ND_CUDA(cudaMemset(count, 0, sizeof(int32_t)));
    hub_slots_kernel<<<grid, 256>>>(g->row_ptr, g->V, least, HUBS, slot.p, hubs.p, count);
    ND_CUDA(cudaMemcpy(&n, count, sizeof(n), cudaMemcpyDeviceToHost));
    return ND_OK;
  };
  uint64_t least = (uint64_t)std::max<int32_t>(g->V / HUB, 256) << 32;
  ND_TRY(slots(least));
  if (n > HUBS) {   // the rank that HUBS vertices reach, by bisection: at most 63 passes over the row offsets
    for (uint64_t lo = least, hi = (uint64_t)1 << 63; n != HUBS;) {
      least = lo + (hi - lo) / 2;
      ND_CUDA(cudaMemset(count, 0, sizeof(int32_t)));
      hub_count_kernel<<<grid, 256>>>(g->row_ptr, g->V, least, count);
      ND_CUDA(cudaMemcpy(&n, count, sizeof(n), cudaMemcpyDeviceToHost));
      if (n > HUBS) lo = least; else hi = least;
    }
    ND_TRY(slots(least));
  }
  const size_t words = (size_t)words_of(g->V) * (size_t)std::max(n, 1);
  ND_TRY(bits.alloc(words));
  ND_CUDA(cudaMemset(bits.p, 0, sizeof(uint32_t) * words));
  if (n > 0) hub_bits_kernel<<<dim3((unsigned)n, 8), 256>>>(g->row_ptr, g->col, hubs.p, words_of(g->V), bits.p);
  ND_CUDA(cudaDeviceSynchronize());
  g->hub_bits = bits.release();
  g->hub_slot = slot.release();
  return ND_OK;
}

// FastGCN: the packed degrees and the list of big vertices
int ensure_degrees(const nd_graph *g, int grid) {
  if (g->deg_codes) return ND_OK;
  const int64_t units = 4 * (int64_t)words_of(g->V);
  const int cap = (int)(g->E / BIG_DEGREE) + 1;
  NdDevMem<uint4> deg;
  NdDevMem<NdBigVertex> big;
  NdDevMem<int32_t> count;
  int32_t n = 0;
  ND_TRY(deg.alloc((size_t)std::max<int64_t>(units, 1)));
  ND_TRY(big.alloc((size_t)cap));
  ND_TRY(count.alloc(1));
  ND_CUDA(cudaMemset(count.p, 0, sizeof(int32_t)));
  deg_build_kernel<<<grid, 256>>>(g->row_ptr, g->V, units, deg.p, big.p, count.p, cap);
  ND_CUDA(cudaMemcpy(&n, count.p, sizeof(n), cudaMemcpyDeviceToHost));
  std::vector<NdBigVertex> list((size_t)n);
  ND_CUDA(cudaMemcpy(list.data(), big.p, sizeof(NdBigVertex) * (size_t)n, cudaMemcpyDeviceToHost));
  std::sort(list.begin(), list.end(), [](const NdBigVertex &x, const NdBigVertex &y) { return x.v < y.v; });
  ND_CUDA(cudaMemcpy(big.p, list.data(), sizeof(NdBigVertex) * (size_t)n, cudaMemcpyHostToDevice));
  g->n_big = n;
  g->big = big.release();
  g->deg_codes = deg.release();
  return ND_OK;
}

// LADIES: the terms of the entries, and whether the rows ascend
int ensure_terms(const nd_graph *g, int grid) {
  if (g->term) return ND_OK;
  if (g->rows_sorted < 0) {
    NdDevMem<int> flag;
    int unsorted = 0;
    ND_TRY(flag.alloc(1));
    ND_CUDA(cudaMemset(flag.p, 0, sizeof(int)));
    unsorted_kernel<<<grid, BUILD_THREADS>>>(g->row_ptr, g->col, g->V, g->E, flag.p);
    ND_CUDA(cudaMemcpy(&unsorted, flag.p, sizeof(int), cudaMemcpyDeviceToHost));
    g->rows_sorted = unsorted ? 0 : 1;
  }
  NdDevMem<float> term;
  NdDevMem<double> sum;
  ND_TRY(term.alloc((size_t)(g->E > 0 ? g->E : 1)));
  ND_TRY(sum.alloc((size_t)g->V));
  ND_CUDA(cudaMemset(sum.p, 0, sizeof(double) * (size_t)g->V));
  rowsum_build_kernel<<<grid, BUILD_THREADS>>>(g->row_ptr, g->w, g->V, g->E, sum.p);
  term_build_kernel<<<grid, BUILD_THREADS>>>(g->row_ptr, g->w, sum.p, g->V, g->E, term.p);
  ND_CUDA(cudaDeviceSynchronize());
  g->term = term.release();
  return ND_OK;
}

// What a graph's first sampler builds goes to the graph when all of it is there: a build that runs out of memory
// leaves nothing behind.
int ensure_layers(const nd_graph *g, int sms, bool ladies) {
  std::lock_guard<std::mutex> lock(g_layers_mutex);
  const int grid = sms * 16;
  ND_TRY(ensure_hubs(g, grid));
  return ladies ? ensure_terms(g, grid) : ensure_degrees(g, grid);
}

// ND_COLLECTIVE_BITMAP_GLOBAL=1 puts the big part into global scratch whatever the graph's size (the tests use it to
// cover that path on small graphs).  Asked once per sampler: its buffers are sized by the answer.
bool force_global() {
  const char *e = getenv("ND_COLLECTIVE_BITMAP_GLOBAL");
  return e && e[0] == '1';
}

struct Plan {
  Layout lay;
  int threads, per_sm;
};

// Two CTAs of 512 threads per SM where both layouts fit, else one of 1024.
Plan plan_of(const nd_sampler *s) {
  const int32_t V = s->g->V;
  const int L = s->p.fanout[0], B = s->p.batch, ntr = B > L ? B : L;
  const bool ladies = s->p.app == ND_APP_LADIES_IS;
  Layout l;
  l.words = words_of(V);
  l.groups = l.words / GROUP_WORDS;
  uint32_t big = 4u * (uint32_t)l.words;       // a multiple of 64
  l.off_gcdf = big; big += 8u * (uint32_t)l.groups;
  l.off_gpref = big; big += ladies ? 4u * (uint32_t)(l.groups + 1) : 0u;
  l.off_qpre = big; big += ladies ? 2u * (uint32_t)(l.words / 4) : 0u;
  big = (big + 255u) & ~255u;
  auto place = [&](uint32_t off) {
    l.off_red = off; off += 8u * 32u + 4u * 32u;
    l.off_ut = off; off += (uint32_t)sizeof(Transit) * (uint32_t)ntr;
    l.off_tr = off; off += 4u * (uint32_t)ntr;
    l.off_layer = off; off += 4u * (uint32_t)L;
    l.off_mult = off; off += 4u * (uint32_t)ntr;
    l.off_pre = off; off += ladies ? 4u * (uint32_t)ntr : 0u;
    return (off + 15u) & ~15u;
  };
  const uint32_t tile_least = ladies ? 8u * 4096u : 0u, tile_most = ladies ? 8u * 16384u : 0u;   // whole groups
  const uint32_t optin = (uint32_t)(s->dev.smem_optin - ND_SMEM_STATIC), half = optin / 2u - 1024u;
  const uint32_t need = place(big) + tile_least;
  Plan p;
  const bool global = s->coll_global || need > optin;
  const uint32_t base = place(global ? 0u : big);
  const bool two = !global && need <= half;
  const uint32_t room = (two ? half : optin) - base;
  l.off_tile = base;
  l.tile = std::min(room, tile_most) / (8u * GROUP) * GROUP;
  l.bytes = base + 8u * l.tile;
  l.glob_bytes = global ? big : 0u;
  p.lay = l;
  p.threads = two ? 512 : 1024;
  p.per_sm = two ? 2 : 1;
  return p;
}

// LADIES: where the tiles begin in the transits' lists
int pos_entries(const nd_sampler *s, const Layout &lay) {
  const int L = s->p.fanout[0], B = s->p.batch;
  return (int)((s->g->V + lay.tile - 1) / lay.tile + 1) * (B > L ? B : L);
}

}  // namespace

extern "C" int nd_graph_hub_slots(const nd_graph *g, const int32_t **slot) {
  ND_REQUIRE(g && slot, ND_ERR_ARG, "nd_graph_hub_slots: null argument");
  std::lock_guard<std::mutex> lock(g_layers_mutex);
  *slot = g->hub_slot;
  return ND_OK;
}

int nd_coll_bitmap_alloc(nd_sampler *s) {
  const bool ladies = s->p.app == ND_APP_LADIES_IS;
  s->coll_global = force_global();
  const Plan p = plan_of(s);
  ND_TRY(ensure_layers(s->g, s->dev.sms, ladies));
  ND_CUDA(ladies ? nd_smem_most(coll_bitmap_kernel<true>, s->dev) : nd_smem_most(coll_bitmap_kernel<false>, s->dev));
  s->coll_grid = (int)std::min<int64_t>(s->S > 0 ? s->S : 1, (int64_t)s->dev.sms * p.per_sm);
  if (p.lay.glob_bytes) ND_CUDA(nd_malloc(&s->d_bm, (size_t)p.lay.glob_bytes * (size_t)s->coll_grid));
  if (ladies) ND_CUDA(nd_malloc(&s->d_cand_w, sizeof(float) * (size_t)s->coll_grid * (size_t)s->g->V));
  if (ladies) ND_CUDA(nd_malloc(&s->d_runs, sizeof(int32_t) * (size_t)s->coll_grid * (size_t)pos_entries(s, p.lay)));
  ND_CUDA(nd_malloc(&s->d_rows_acc, 16 * sizeof(unsigned long long)));
  ND_CUDA(cudaMemset(s->d_rows_acc, 0, 16 * sizeof(unsigned long long)));
  return ND_OK;
}

int nd_coll_bitmap_launch(nd_sampler *s, const CollParams &cp, unsigned long long pairs) {
  const bool ladies = s->p.app == ND_APP_LADIES_IS;
  const Plan p = plan_of(s);
  const nd_graph *g = s->g;
  const Args a{nd_view(g), cp, s->p.steps, s->S, p.lay, s->d_bm, s->d_initial, s->d_out, s->d_cand_w,
               s->d_runs, ladies ? pos_entries(s, p.lay) : 0, g->rows_sorted, s->d_adj_row, s->d_adj_col, s->d_prob,
               g->deg_codes, g->big, g->n_big, g->term, g->hub_slot, g->hub_bits, s->d_rows_acc, s->d_stats, pairs};
  if (ladies) coll_bitmap_kernel<true><<<s->coll_grid, p.threads, p.lay.bytes, s->stream>>>(a);
  else coll_bitmap_kernel<false><<<s->coll_grid, p.threads, p.lay.bytes, s->stream>>>(a);
  nd_count_launches(1);
  ND_CUDA(cudaGetLastError());
  return ND_OK;
}
