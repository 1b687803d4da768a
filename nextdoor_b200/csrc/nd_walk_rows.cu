// Random walks, a lane per walk: the kernels of the sample-parallel mode (sampleParallelKernel,
// src/nextdoor.cu:1348-1518) and of the load-balanced mode.  The draws are keyed by (sample, step), so every
// organisation of a job gives the same samples, and on B200 a lane that keeps its walk in registers beats a
// step-by-step pass over a transit-sorted map at every number of walks (measured, transit-parallel loop with
// counting inversion -> this file: uniform walk on 57 K vertices 1.10 -> 0.07 ms, DeepWalk on 2^20 vertices
// 5.2 -> 1.4 ms, node2vec 7.6 -> 2.1 ms, PPR on 2^24 vertices 5.4 -> 2.4 ms).
//
// What bounds it.  Large graphs: the rate of random DRAM reads.  A walker picks every CSR entry with the same
// probability, and a gather that misses the L2 reads a whole line of 128 bytes (11.1 GB for 91 M gathers of 4 bytes from
// 2 GB); the GPU serves 40-45 G of those a second, and as many of 64 bytes (the loads' L2::64B): not the bytes are the
// bound.  Independent gathers run at 285 G/s from up to 75 MB, 195 from 90, 139 from 110, 117 from 134, 88 from
// 200, 55 from 400, 40 from 2 GB and more.  So what counts is the number of gathers, and the size of what they go to,
// hence: one try per round for the weighted apps (no speculation), the id and its weight in one word, the first stop draw
// of a step made before the vertex is fetched, a filter in front of node2vec's sets, rows written once, in
// 32-byte sectors.  Small graphs: the chain of a walk, two dependent L2 reads per step, one where the entries carry the
// neighbour's row, and the instructions between them (57 K vertices: a step is 0.5 us, 111 instructions of a warp at 8.9
// cycles each, 45 % of them waiting for the read).
#include <mutex>

#include "nd_common.cuh"
#include "nd_entries.cuh"
#include "nd_nbrset.cuh"
#include "nd_philox.cuh"
#include "nd_walk_rows.cuh"

namespace {

constexpr int ROWS_THREADS = 128;
// CTAs per SM: 1536 lanes at 40 registers.  Measured on DeepWalk, 2^20 vertices: 8 -> 1.95, 12 -> 1.63,
// 14 -> 1.81, 16 -> 1.90 ms; two walks per lane at half the lanes 2.0 ms (fewer L1 hits, longer tail).
constexpr int ROWS_CTAS = 12;
constexpr int RETRY_CAP = 1 << 16;
constexpr int32_t AGAIN = -2;   // the round ended without an accepted vertex

struct RowsArgs {
  int32_t V;
  const int32_t *__restrict__ row_ptr;
  const int32_t *__restrict__ col;
  const float *__restrict__ w;
  const float *__restrict__ max_w;
  const int2 *__restrict__ vrow;     // [V] (row start, degree)
  const int4 *__restrict__ erec;     // [E] (neighbour, its row start, its degree, weight as 256ths of the row's maximum, rounded down)
  const int2 *__restrict__ colw;     // [E] (neighbour, weight bits)
  const int2 *__restrict__ vrec;     // [V+1] (row start, max weight bits)
  const uint32_t *__restrict__ pack; // [E] neighbour << 8 | weight as 256ths of the row's maximum, rounded down (CODES: a byte each, the weight)
  const uint2 *__restrict__ col3;    // [E/3] three neighbours of 21 bits each
  const int32_t *__restrict__ adjset;
  const uint32_t *__restrict__ adjsign;
  ndrng::RoundKeys keys;
  float p, q, stop_prob;
  int n2v_compat, steps;
  int64_t first_sample, S;
  const int32_t *__restrict__ initial;
  int32_t *__restrict__ out;
  int32_t *__restrict__ plen;
  int4 *__restrict__ list;                  // walks that can start: (sample, row start, degree, max weight bits or vertex); null: all walks, in order
  // Counters of the running job, zero between jobs: [0..7] as published, [8] walks handed out beyond the first
  // round, [9] entries of the list, [10] CTAs that are done; the last CTA publishes them and clears them again,
  // so a job needs no launch for that and can be replayed from a graph.
  unsigned long long *__restrict__ acc;
  uint32_t *__restrict__ ended;             // [steps] walks that ended after k vertices, or null
  unsigned long long *__restrict__ stats;   // published counters [8]
  uint32_t *__restrict__ ended_out;         // published histogram
  int *__restrict__ status;
};

template <int APP>
__host__ __device__ constexpr bool weighted() { return APP == ND_APP_DEEPWALK || APP == ND_APP_PPR; }

// Layouts of the entries.  ALT (weighted walks): id and weight in a word.  FAT (uniform, weighted walks): they carry the
// neighbour's row, and the weight.  DENSE (uniform walk, node2vec): three ids of 21 bits in 8 bytes.  FAR: weighted walks as
// ALT, node2vec as PLAIN, rows from the offsets.  CODES (weighted walks): a byte of weight beside the ids, rows from the
// offsets: what needs the least memory.
enum : int { LAYOUT_PLAIN = 0, LAYOUT_ALT = 1, LAYOUT_DENSE = 2, LAYOUT_FAR = 3, LAYOUT_FAT = 4, LAYOUT_CODES = 5 };

// ---- loads.  The small per-vertex and per-entry arrays ask to stay in the L2; the (id, weight) records, an array far
// larger than the L2, bypass the L1.
struct Hot {
  uint64_t pol;
  __device__ __forceinline__ Hot() { asm("createpolicy.fractional.L2::evict_last.b64 %0, 1.0;" : "=l"(pol)); }
  __device__ __forceinline__ int32_t ld(const int32_t *p) const { int32_t v; asm("ld.global.nc.L2::cache_hint.s32 %0, [%1], %2;" : "=r"(v) : "l"(p), "l"(pol)); return v; }
  __device__ __forceinline__ int2 ld(const int2 *p) const { int2 v; asm("ld.global.nc.L2::cache_hint.v2.s32 {%0, %1}, [%2], %3;" : "=r"(v.x), "=r"(v.y) : "l"(p), "l"(pol)); return v; }
  __device__ __forceinline__ int4 ld(const int4 *p) const { int4 v; asm("ld.global.nc.L2::cache_hint.v4.s32 {%0, %1, %2, %3}, [%4], %5;" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p), "l"(pol)); return v; }
};
__device__ __forceinline__ int2 ld_once(const int2 *p) { int2 v; asm("ld.global.nc.L1::no_allocate.v2.s32 {%0, %1}, [%2];" : "=r"(v.x), "=r"(v.y) : "l"(p)); return v; }

// ---- ids without their unused bits
//
// Between 64 MB and a few times the L2, a smaller array is fewer misses: three ids of 21 bits in 8 bytes, 2.67 bytes an
// entry (2^20 vertices, 33.5 M entries, 134 -> 89 MB: uniform walk 0.91 -> 0.78 ms, node2vec 2.26 -> 2.14; 2^21
// vertices, 50 M entries: 1.57 -> 1.37, 3.88 -> 3.61; 600 K, 14.4 M: 0.34 -> 0.32, 0.98 -> 1.00; 300 K, 7.2 M, inside the
// L2 either way: 0.17 -> 0.18, 0.21 -> 0.22).
constexpr int DENSE_IDS = 3, DENSE_ID_BITS = 21;
constexpr int32_t DENSE_V = 1 << DENSE_ID_BITS;
constexpr int64_t DENSE_ENTRIES = (int64_t)1 << 24;

// neighbour of entry e
template <int LAYOUT>
__device__ __forceinline__ int32_t id_of(const RowsArgs &a, int32_t e) {
  if (LAYOUT != LAYOUT_DENSE) return __ldg(a.col + e);
  const uint32_t group = (uint32_t)e / DENSE_IDS, off = ((uint32_t)e - DENSE_IDS * group) * DENSE_ID_BITS;
  const uint2 q = __ldg(a.col3 + group);
  return (int32_t)((uint32_t)(((unsigned long long)q.y << 32 | q.x) >> off) & ((1u << DENSE_ID_BITS) - 1u));
}

// ---- rows of the result
//
// Vertices are collected in shared memory and go out in aligned pieces: slot j of thread t at [j * threads + t],
// so every access of a warp is free of bank conflicts.  64-byte pieces for the walks that run their full
// length (a dirty half of a 64-byte DRAM unit costs as much as the whole: DeepWalk 1.84 -> 1.77 ms against
// 32-byte pieces), 32-byte pieces for PPR, whose rows hold a few vertices.
template <int APP>
__host__ __device__ constexpr int piece() { return APP == ND_APP_PPR ? 8 : 16; }   // vertices
template <int PIECE>
__device__ __forceinline__ int piece_slot(const RowsArgs &a, uint32_t s, int step) { return (int)(((int64_t)s * a.steps + step) & (PIECE - 1)); }

// The piece that holds the p vertices before slot n of the row goes out.  Slots behind the walk hold the
// invalid id, so a sector that lies inside the row is written whole (one that is written in part costs the
// memory a read of it).  Returns the first slot behind those written.
template <int PIECE>
__device__ __forceinline__ int piece_out(const RowsArgs &a, const int32_t *buf, uint32_t s, int n, int p) {
  int32_t *row = a.out + (int64_t)s * a.steps;
  int written = n;
#pragma unroll
  for (int q = 0; q < PIECE; q += 8) {
    const int at = n - p + q;   // slot of the row the sector begins at
    if (q < p) {
      if (at >= 0 && at + 8 <= a.steps) {
        int32_t v[8];
#pragma unroll
        for (int j = 0; j < 8; j++) v[j] = q + j < p ? buf[(q + j) * ROWS_THREADS + threadIdx.x] : a.V;
        asm volatile("st.global.L2::evict_first.v8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"l"(row + at), "r"(v[0]), "r"(v[1]), "r"(v[2]),
                     "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7])
                     : "memory");
        written = at + 8 > written ? at + 8 : written;
      } else {
        for (int j = at < 0 ? -at : 0; j < 8 && q + j < p; j++) row[at + j] = buf[(q + j) * ROWS_THREADS + threadIdx.x];
      }
    }
  }
  return written;
}

// What the CTA's walks add up to, and how a walk ends.
template <int PIECE>
struct Rows {
  int32_t *buf;
  uint32_t *ended;     // histogram of the CTA's walks that ended early, by their vertices
  unsigned int *sum;   // [0] vertices, [1] walks that ended early
  __device__ __forceinline__ Rows(const RowsArgs &a, unsigned int *sums) {
    extern __shared__ int32_t sh_dyn[];
    buf = sh_dyn;
    ended = reinterpret_cast<uint32_t *>(sh_dyn + PIECE * ROWS_THREADS);
    sum = sums;
    if (threadIdx.x < 2) sum[threadIdx.x] = 0u;
    if (a.ended) for (int k = threadIdx.x; k < a.steps; k += ROWS_THREADS) ended[k] = 0u;
    __syncthreads();
  }
  __device__ __forceinline__ void put(const RowsArgs &a, uint32_t s, int step, int32_t v) {
    const int p = piece_slot<PIECE>(a, s, step);
    buf[p * ROWS_THREADS + threadIdx.x] = v;
    if (p == PIECE - 1) piece_out<PIECE>(a, buf, s, step + 1, PIECE);
  }
  // the walk has ended with n vertices: its open piece, and the slots the row's previous walk filled beyond them
  __device__ __forceinline__ void end(const RowsArgs &a, uint32_t s, int n, bool counts) {
    const int p = piece_slot<PIECE>(a, s, n);
    const int written = p ? piece_out<PIECE>(a, buf, s, n, p) : n;
    const int32_t had = a.plen[s];
    for (int j = written; j < had; j++) a.out[(int64_t)s * a.steps + j] = a.V;
    if (had != n) a.plen[s] = n;
    if (n) atomicAdd(&sum[0], (unsigned int)n);
    if (counts && n < a.steps) {
      atomicAdd(&sum[1], 1u);
      if (a.ended) atomicAdd(&ended[n], 1u);
    }
  }
  // the whole CTA, at its end; `tries` and `words` of every thread go to counters `tries_at` and 4
  __device__ __forceinline__ void out(const RowsArgs &a, uint32_t tries, int tries_at, uint32_t words) {
    __shared__ int last;
    for (int o = 16; o > 0; o >>= 1) {
      tries += __shfl_xor_sync(0xffffffffu, tries, o);
      words += __shfl_xor_sync(0xffffffffu, words, o);
    }
    if ((threadIdx.x & 31) == 0) {
      if (tries) atomicAdd(&a.acc[tries_at], (unsigned long long)tries);
      if (words) atomicAdd(&a.acc[4], (unsigned long long)words);
    }
    __syncthreads();
    if (threadIdx.x == 0 && sum[0] + sum[1]) {
      atomicAdd(&a.acc[0], (unsigned long long)sum[0]);
      atomicAdd(&a.acc[1], (unsigned long long)sum[0] + sum[1]);
    }
    if (a.ended)
      for (int k = threadIdx.x; k < a.steps; k += ROWS_THREADS)
        if (ended[k]) atomicAdd(&a.ended[k], ended[k]);
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) last = atomicAdd(&a.acc[10], 1ull) == (unsigned long long)gridDim.x - 1ull;
    __syncthreads();
    if (!last) return;
    __threadfence();
    if (threadIdx.x < 8) a.stats[threadIdx.x] = __ldcg(&a.acc[threadIdx.x]);
    if (a.ended)
      for (int k = threadIdx.x; k < a.steps; k += ROWS_THREADS) {
        a.ended_out[k] = __ldcg(&a.ended[k]);
        a.ended[k] = 0u;
      }
    __syncthreads();
    if (threadIdx.x < 11) a.acc[threadIdx.x] = 0ull;
  }
};

__device__ __forceinline__ void draw_block(const RowsArgs &a, uint32_t s, int step, uint32_t block, uint32_t (&o)[4]) {
  ndrng::philox4x32_10((uint32_t)(a.first_sample + s), (uint32_t)step, 0u, block, a.keys, o);
}
__device__ __forceinline__ int32_t draw_index(uint32_t u, int32_t n) { return ndrng::rand_int_from(ndrng::u32_to_uniform(u), n); }

// ---- which walks a lane takes
//
// A job with more walks than there are lanes starts from a list of the walks that can start (on the R-MAT
// graphs 40-47 % of the vertices have no neighbours, and a lane without a walk reads nothing); the first
// walks of a lane follow from its place, the next ones are handed out to its warp 64 at a time.  A job whose
// walks all have a lane takes them in order, without the pass that makes the list.
constexpr int START_PER_THREAD = 4;
template <int APP, int LAYOUT>
__global__ void __launch_bounds__(256) walk_start_kernel(const __grid_constant__ RowsArgs a) {
  __shared__ uint32_t sh_n, sh_dead;
  __shared__ unsigned long long sh_base;
  if (threadIdx.x == 0) { sh_n = 0u; sh_dead = 0u; }
  __syncthreads();
  const int lane = threadIdx.x & 31;
  const int64_t first = (int64_t)blockIdx.x * 256 * START_PER_THREAD + threadIdx.x;
  int4 e[START_PER_THREAD];
  int32_t t[START_PER_THREAD], had[START_PER_THREAD];
#pragma unroll
  for (int j = 0; j < START_PER_THREAD; j++) {
    const int64_t s = first + j * 256;
    t[j] = s < a.S ? a.initial[s] : -1;
    had[j] = s < a.S ? a.plen[s] : 0;
  }
  uint32_t at[START_PER_THREAD], dead = 0;
#pragma unroll
  for (int j = 0; j < START_PER_THREAD; j++) {
    const int64_t s = first + j * 256;
    const bool valid = t[j] >= 0 && t[j] < a.V;
    const int32_t rs = valid ? __ldg(a.row_ptr + t[j]) : 0, deg = valid ? __ldg(a.row_ptr + t[j] + 1) - rs : 0;
    bool active = deg > 0;
    if (APP == ND_APP_PPR && active) {   // the stop draw does not depend on the vertex
      uint32_t o[4];
      draw_block(a, (uint32_t)s, 0, 0u, o);
      active = !(ndrng::u32_to_uniform(o[0]) < a.stop_prob);
    }
    e[j] = make_int4((int)(uint32_t)s, rs, active ? deg : 0, weighted<APP>() && LAYOUT == LAYOUT_PLAIN ? (active ? __float_as_int(__ldg(a.max_w + t[j])) : 0) : t[j]);
    if (!active) {
      for (int k = 0; k < had[j]; k++) a.out[s * a.steps + k] = a.V;
      if (had[j]) a.plen[s] = 0;
    }
    const unsigned m = __ballot_sync(0xffffffffu, active);
    dead += __popc(__ballot_sync(0xffffffffu, valid && !active));
    uint32_t base = 0;
    if (lane == 0 && m) base = atomicAdd(&sh_n, (uint32_t)__popc(m));
    at[j] = __shfl_sync(0xffffffffu, base, 0) + __popc(m & ((1u << lane) - 1u));
  }
  if (lane == 0 && dead) atomicAdd(&sh_dead, dead);
  __syncthreads();
  if (threadIdx.x == 0) {   // one atomic per CTA and counter: with one per warp this pass took 0.43 instead of 0.13 ms on 2^24 walks
    sh_base = sh_n ? atomicAdd(&a.acc[9], (unsigned long long)sh_n) : 0ull;
    if (sh_dead) {
      atomicAdd(&a.acc[1], (unsigned long long)sh_dead);
      if (a.ended) atomicAdd(&a.ended[0], sh_dead);
    }
  }
  __syncthreads();
#pragma unroll
  for (int j = 0; j < START_PER_THREAD; j++)
    if (e[j].z > 0) a.list[sh_base + at[j]] = e[j];
}

// Row start and degree of a vertex.  Two row offsets lie in one sector seven times out of eight and take half of the room
// of a record of both, which is one load: FAR, from FAR_V vertices on, where the records do not fit the L2 beside what
// else a walk reads (PPR on 2^24 vertices 2.47 -> 2.38 ms, node2vec on 2^22 15.4 -> 15.0, DeepWalk on 2^22 the same;
// DeepWalk on 2^20 1.41 with the records, 1.52 with the offsets; uniform walk on 2^22 3.26 and 3.35: keeps the records).
constexpr int32_t FAR_V = 1 << 22;
template <int LAYOUT>
__device__ __forceinline__ int2 row_of(const RowsArgs &a, const Hot &hot, int32_t v) {
  if (LAYOUT != LAYOUT_FAR && LAYOUT != LAYOUT_CODES) return hot.ld(a.vrow + v);
  const int32_t at = hot.ld(a.row_ptr + v), end = hot.ld(a.row_ptr + v + 1);
  return make_int2(at, end - at);
}

// (row start, degree, max weight bits or vertex) of a vertex
template <int APP, int LAYOUT>
__device__ __forceinline__ int4 vertex_of(const RowsArgs &a, const Hot &hot, int32_t v) {
  if (weighted<APP>() && LAYOUT == LAYOUT_PLAIN) {
    const int2 r = hot.ld(a.vrec + v), n = hot.ld(a.vrec + v + 1);
    return make_int4(r.x, n.x - r.x, r.y, 0);
  }
  const int2 r = row_of<LAYOUT>(a, hot, v);
  return make_int4(r.x, r.y, v, 0);
}

// walk i of the job as (sample, row start, degree, max weight bits or vertex); degree -1: the seed is not a vertex
template <int APP, int LAYOUT>
__device__ __forceinline__ int4 walk_of(const RowsArgs &a, const Hot &hot, int64_t i) {
  if (a.list) return a.list[i];
  const int32_t t = a.initial[i];
  if (t < 0 || t >= a.V) return make_int4((int)(uint32_t)i, 0, -1, 0);
  const int4 v = vertex_of<APP, LAYOUT>(a, hot, t);
  return make_int4((int)(uint32_t)i, v.x, v.y, v.z);
}

// Walks that run their full length (EQUAL) take equal rounds: with w rounds of lanes every round takes n / w walks, or the
// last one would run a fraction of the lanes for as long as the others; and a warp gets 32 at a time.  (Without and with,
// one walk per vertex: node2vec on 400 K vertices 1.20 -> 0.95 ms, 600 K 1.34 -> 1.21, 2^20 2.08 -> 2.11, 1.5 M 3.15 -> 2.87,
// 2^21 4.89 -> 4.59; DeepWalk 0.68 -> 0.60, 0.80 -> 0.74, 1.37 -> 1.40, 2.02 -> 1.91, 3.13 -> 2.96: what it gives is the part of
// a round that the last one lacks, and 2^20 with few of them empty lacks little.)
template <bool EQUAL>
struct Taker {
  static constexpr int GRANT = EQUAL ? 32 : 64;
  int64_t n, lanes, cur, end;
  __device__ __forceinline__ explicit Taker(const RowsArgs &a)
      : n(a.list ? (int64_t)a.acc[9] : a.S), lanes((int64_t)gridDim.x * ROWS_THREADS), cur(0), end(0) {
    if (EQUAL && n > lanes) {
      const int64_t rounds = (n + lanes - 1) / lanes;
      lanes = ((n + rounds - 1) / rounds + 31) / 32 * 32;
    }
  }
  // the lane's first walk (n or more: none)
  __device__ __forceinline__ int64_t first() const {
    const int64_t i = (int64_t)blockIdx.x * ROWS_THREADS + threadIdx.x;
    return i < lanes ? i : n;
  }
  // the next walk of every lane that wants one (n or more: none left); the whole warp calls it
  __device__ __forceinline__ int64_t next(const RowsArgs &a, unsigned want) {
    const int lane = threadIdx.x & 31;
    const int need = __popc(want), my = __popc(want & ((1u << lane) - 1u));
    const int64_t avail = end - cur;
    int64_t i = cur + my;
    if (need <= avail) {
      cur += need;
    } else {
      unsigned long long nb = (unsigned long long)n;
      if (n > lanes) {
        if (lane == 0) nb = (unsigned long long)lanes + atomicAdd(&a.acc[8], (unsigned long long)GRANT);
        nb = __shfl_sync(0xffffffffu, nb, 0);
      }
      if (my >= avail) i = (int64_t)nb + (my - avail);
      cur = (int64_t)nb + (need - avail);
      end = (int64_t)nb + GRANT;
    }
    return i;
  }
};

// ---------------------------------------------------------------- uniform walk (example/uniformRandWalk.cu:27-37)
//
// The lanes of a warp go in step.  The draw of the next step does not depend on the vertex: it is made while
// the gather is in flight, so that a step is its dependent reads and little else.  Equal rounds, as in Taker.
template <int LAYOUT>
__device__ __forceinline__ void uniform_walks(const RowsArgs &a) {
  constexpr bool FAT = LAYOUT == LAYOUT_FAT;
  constexpr int PIECE = piece<ND_APP_UNIFORM_WALK>();
  __shared__ unsigned int sums[2];
  Rows<PIECE> rows(a, sums);
  const Hot hot;
  const int64_t all = a.list ? (int64_t)a.acc[9] : a.S, lanes = (int64_t)gridDim.x * ROWS_THREADS, me = (int64_t)blockIdx.x * ROWS_THREADS + threadIdx.x;
  const int64_t rounds = (all + lanes - 1) / lanes, per = rounds ? (all + rounds - 1) / rounds : 0;
  for (int64_t round = 0; round < rounds; round++) {
    const int64_t w0 = round * per, wn = all - w0 < per ? all - w0 : per;
    if (me >= wn) continue;
    const int4 e = walk_of<ND_APP_UNIFORM_WALK, LAYOUT>(a, hot, w0 + me);
    const uint32_t s = (uint32_t)e.x;
    int32_t rs = e.y, deg = e.z;
    uint32_t u[4];
    draw_block(a, s, 0, 0u, u);
    if (deg <= 0) rows.end(a, s, 0, deg == 0);
    for (int step = 0; deg > 0; step++) {
      const int32_t x = draw_index(u[0], deg);
      int32_t v;
      int2 r = make_int2(0, 0);
      if (FAT) {
        const int4 f = hot.ld(a.erec + rs + x);
        draw_block(a, s, step + 1, 0u, u);
        v = f.x; r = make_int2(f.y, f.z);
      } else {
        v = id_of<LAYOUT>(a, rs + x);
        draw_block(a, s, step + 1, 0u, u);
        if (step + 1 < a.steps) r = row_of<LAYOUT>(a, hot, v);
      }
      rows.put(a, s, step, v);
      rs = r.x;
      deg = step + 1 < a.steps ? r.y : 0;
      if (deg <= 0) rows.end(a, s, step + 1, true);
    }
  }
  rows.out(a, 0u, 2, 0u);
}

// ---------------------------------------------------------------- weighted walks (randomWalks.cu:65-124)
//
// A lane is a state machine: a trip of the loop is one try {x = rand_int(n); y = u * max_w; accept unless
// y > w[x]} wherever the lane's walk stands, a lane whose try was rejected stays on its step, a lane whose
// walk ended takes the next one, and the vote at the loop head is where the warp meets again.  Draws of a
// step: PPR's stop draw, then two per try; a block of four is made once and kept (k0..k2).
// PPR makes the stop draw of a step before it fetches the vertex, which a walk that stops never needs.
//
// Weights.  PLAIN: (id, weight) records.  ALT: the id and the weight as whole 256ths of the row's maximum, rounded down, in
// one word: b/256 <= w/max < (b+1)/256 decides all but one try in 256 without the weight or the maximum -- u <= b/256
// accepts and u >= (b+1)/256 rejects, and both follow for u * max against w because b * (max/256) and
// (b+1) * (max/256), rounded as the kernel rounds u * max, were compared with w when b was chosen.  One gather per try
// where there were a byte per try, then the id: DeepWalk on 2^20 vertices 1.57 -> 1.40 ms, on 600 K 0.93 -> 0.61, on 40 K
// 0.20 -> 0.15; PPR on 2^21 0.46 -> 0.38.  The words go through the L1 like any other load: ld.global.nc with
// L1::no_allocate leaves them the first to go in the L2 as well, three of four tries on 134 MB of them then miss instead of
// two of five (DeepWalk 1.93 ms), and only arrays far larger than the L2 (PLAIN) lose nothing by it.
template <int APP, int LAYOUT>
__device__ __forceinline__ void weighted_walks(const RowsArgs &a) {
  constexpr bool PPR = APP == ND_APP_PPR;
  __shared__ unsigned int sums[2];
  Rows<piece<APP>()> rows(a, sums);
  const Hot hot;
  Taker<!PPR> take(a);
  uint32_t s = 0, k0 = 0, k1 = 0, k2 = 0, tries = 0;
  // cur: the vertex the walk has moved to, its record not fetched yet; -1: (rs, deg, mw) are those of the walk's vertex
  int32_t rs = 0, deg = 0, mw = 0, cur = -1;
  int step = -1, t = 0;   // step -1: no walk; t: tries of this step so far
  if (take.first() < take.n) {
    const int4 e = walk_of<APP, LAYOUT>(a, hot, take.first());
    s = (uint32_t)e.x; rs = e.y; deg = e.z; mw = e.w; step = 0;
  }
  while (__any_sync(0xffffffffu, step >= 0)) {
    const bool odd = (t & 1) != 0;
    uint32_t dx = PPR && odd ? k2 : k0, dy = k1;
    bool over = step == a.steps || (cur < 0 && deg <= 0);
    if (PPR ? (odd || t == 0) : !odd) {
      uint32_t o[4];
      draw_block(a, s, step, (uint32_t)(PPR ? (t + 1) >> 1 : t >> 1), o);
      if (PPR) {
        if (odd) { dy = o[0]; } else { dx = o[1]; dy = o[2]; over |= ndrng::u32_to_uniform(o[0]) < a.stop_prob; }
        k0 = o[1]; k1 = o[2]; k2 = o[3];
      } else {
        dx = o[0]; dy = o[1]; k0 = o[2]; k1 = o[3];
      }
    }
    over = over && step >= 0;
    if (cur >= 0 && !over) {
      const int4 r = vertex_of<APP, LAYOUT>(a, hot, cur);
      rs = r.x; deg = r.y; mw = r.z;
      cur = -1;
    }
    const unsigned want = __ballot_sync(0xffffffffu, over);
    if (want) {
      const int64_t i = take.next(a, want);
      if (over) {
        rows.end(a, s, step, deg >= 0);
        step = -1; deg = 0; cur = -1; t = 0;
        if (i < take.n) {
          const int4 e = walk_of<APP, LAYOUT>(a, hot, i);
          s = (uint32_t)e.x; rs = e.y; deg = e.z; mw = e.w; step = 0;
        }
      }
    }
    if (deg <= 0 || over) continue;   // no walk, a vertex without neighbours, or a walk just taken: it starts in the next trip
    const int32_t x = draw_index(dx, deg);
    const float u = ndrng::u32_to_uniform(dy);
    int32_t nbr = AGAIN;
    int2 row = make_int2(0, 0);   // FAT: the neighbour's
    if (LAYOUT != LAYOUT_PLAIN) {
      uint32_t id, b;
      if (LAYOUT == LAYOUT_FAT) {
        const int4 r = hot.ld(a.erec + rs + x);
        id = (uint32_t)r.x; b = (uint32_t)r.w; row = make_int2(r.y, r.z);
      } else if (LAYOUT == LAYOUT_CODES) {
        id = 0u; b = __ldg(reinterpret_cast<const uint8_t *>(a.pack) + rs + x);
      } else {
        const uint32_t r = __ldg(a.pack + rs + x);
        id = r >> 8; b = r & 255u;
      }
      bool accept = deg == 1 || u <= (float)b * 0.00390625f;
      if (!accept && (b == 255u || u < (float)(b + 1u) * 0.00390625f))
        accept = !(__fmul_rn(u, __ldg(a.max_w + mw)) > __ldg(a.w + rs + x));
      if (accept) nbr = LAYOUT == LAYOUT_CODES ? __ldg(a.col + rs + x) : (int32_t)id;
    } else {
      const int2 r = ld_once(a.colw + rs + x);
      if (deg == 1 || !(__fmul_rn(u, __int_as_float(mw)) > __int_as_float(r.y))) nbr = r.x;
    }
    tries += deg > 1 ? 1u : 0u;
    if (nbr == AGAIN && ++t > RETRY_CAP) {
      atomicOr(a.status, ND_DEV_RETRY_LIMIT);
      nbr = __ldg(a.col + rs);
      if (LAYOUT == LAYOUT_FAT) row = row_of<LAYOUT>(a, hot, nbr);
    }
    if (nbr >= 0) {
      rows.put(a, s, step, nbr);
      step++;
      t = 0;
      if (LAYOUT == LAYOUT_FAT) { rs = row.x; deg = row.y; mw = nbr; } else { cur = nbr; }
    }
  }
  rows.out(a, tries, 2, 0u);
}

// ---------------------------------------------------------------- node2vec (randomWalks.cu:141-172)
//
// A candidate that is not the previous vertex t is accepted when y < 1/q (neighbour of t) or y < 1 (not a
// neighbour): below `lo` the membership does not matter, at or above `hi` neither; below `sure` nothing
// about the candidate matters.
struct N2vConsts {
  float inv_q, bound, lo, hi, sure;
  __device__ __forceinline__ N2vConsts(float p, float q) {
    inv_q = __fdiv_rn(1.0f, q);
    bound = p > inv_q ? p : inv_q;
    if (bound < 1.0f) bound = 1.0f;
    lo = inv_q < 1.0f ? inv_q : 1.0f;
    hi = inv_q < 1.0f ? 1.0f : inv_q;
    sure = lo < p ? lo : p;
  }
};

// v in the list [ts, ts + tn), exactly; `words` counts the 4-byte words read
__device__ __forceinline__ bool member_exact(const RowsArgs &a, int32_t ts, int32_t tn, int32_t v, uint32_t hash, uint32_t &words) {
  if (tn < SET_MIN_DEG) {
    bool found = false;
#pragma unroll
    for (int k = 0; k < SET_MIN_DEG - 1; k++) found |= (k < tn ? __ldg(a.col + ts + k) : -1) == v;
    words += tn;
    return found;
  }
  const uint32_t n_buckets = ((uint32_t)(ts + tn) >> 2) - ((uint32_t)ts >> 2);
  const int4 *region = reinterpret_cast<const int4 *>(a.adjset) + 2 * (size_t)((uint32_t)ts >> 2);
  uint32_t b = set_bucket_of_hash(hash, n_buckets);
  for (uint32_t it = 0; it < n_buckets; it++) {
    const int4 c = __ldg(region + 2 * (size_t)b), d = __ldg(region + 2 * (size_t)b + 1);
    words += 8;
    if (c.x == v || c.y == v || c.z == v || c.w == v || d.x == v || d.y == v || d.z == v || d.w == v) return true;
    if (d.w == SET_EMPTY) return false;   // slots fill front to back inside a bucket
    b = b + 1 < n_buckets ? b + 1 : 0;
  }
  return false;
}

// The same state machine; a trip is a round of two tries (one block of draws).  The round ends at the first
// try that is sure to accept, so the second candidate is fetched for nothing only when the first one's
// membership accepts it (one try per round: 2.32 -> 2.6 ms).  A membership test asks the filter first: a word
// of 8 bits per neighbour answers about 95 % of the tests that fail (88 % of all), the rest read the set
// (without the filter 2.9 ms).
template <int LAYOUT>
__device__ __forceinline__ void n2v_walks(const RowsArgs &a) {
  constexpr int APP = ND_APP_NODE2VEC;
  constexpr int TRIES = 2;
  __shared__ unsigned int sums[2];
  Rows<piece<APP>()> rows(a, sums);
  const Hot hot;
  const N2vConsts c(a.p, a.q);
  Taker<true> take(a);
  uint32_t s = 0, tries = 0, words = 0;
  int32_t rs = 0, deg = 0, cur = 0, prev = 0, ts = 0, tn = 0;   // [ts, ts + tn): the row of the previous vertex
  int step = -1, round = 0;
  if (take.first() < take.n) {
    const int4 e = walk_of<APP, LAYOUT>(a, hot, take.first());
    s = (uint32_t)e.x; rs = e.y; deg = e.z; cur = e.w; step = 0;
  }
  while (__any_sync(0xffffffffu, step >= 0)) {
    int32_t nbr = AGAIN;
    const bool over0 = step >= 0 && deg <= 0;
    if (step >= 0 && !over0) {
      uint32_t o[4];
      draw_block(a, s, step, (uint32_t)round, o);
      int32_t x[TRIES], v[TRIES];
      float y[TRIES];
      int n_try = TRIES;
#pragma unroll
      for (int j = 0; j < TRIES; j++) {
        x[j] = draw_index(o[2 * j], deg);
        y[j] = __fmul_rn(ndrng::u32_to_uniform(o[2 * j + 1]), c.bound);
      }
      const bool simple = deg == 1 || step == 0;
      if (simple) x[0] = 0;
#pragma unroll
      for (int j = TRIES - 1; j >= 0; j--) if (y[j] < c.sure) n_try = j + 1;
      if (simple) n_try = 1;
#pragma unroll
      for (int j = 0; j < TRIES; j++) v[j] = j < n_try ? id_of<LAYOUT>(a, rs + x[j]) : -1;
      const uint32_t w0 = (uint32_t)ts >> 2, n_words = ((uint32_t)(ts + tn) >> 2) - w0;
      bool is_ret[TRIES], need[TRIES];
      uint32_t h[TRIES], word[TRIES];
#pragma unroll
      for (int j = 0; j < TRIES; j++) {
        is_ret[j] = a.n2v_compat ? (x[j] == prev) : (v[j] == prev);   // randomWalks.cu:159 compares the index
        need[j] = !simple && j < n_try && !is_ret[j] && y[j] >= c.lo && y[j] < c.hi;
        h[j] = set_mix((uint32_t)v[j]);
        word[j] = 0xffffffffu;
        if (need[j] && tn >= SET_MIN_DEG) word[j] = (uint32_t)hot.ld(reinterpret_cast<const int32_t *>(a.adjsign) + w0 + set_bucket_of_hash(h[j], n_words));
      }
      if (simple) {
        nbr = v[0];
      } else {
#pragma unroll
        for (int j = 0; j < TRIES; j++) {
          if (nbr == AGAIN && j < n_try) {
            tries++;
            bool accept;
            if (is_ret[j]) {
              accept = y[j] < a.p;
            } else if (!need[j]) {
              accept = y[j] < c.lo;
            } else {
              const uint32_t sign = set_sign(h[j]);
              words += tn >= SET_MIN_DEG ? 1u : 0u;
              const bool found = (word[j] & sign) == sign && member_exact(a, ts, tn, v[j], h[j], words);
              accept = y[j] < (found ? c.inv_q : 1.0f);
            }
            if (accept) nbr = v[j];
          }
        }
        round++;
        if (nbr == AGAIN && TRIES * round > RETRY_CAP) {
          atomicOr(a.status, ND_DEV_RETRY_LIMIT);
          nbr = __ldg(a.col + rs);
        }
      }
    }
    const bool moved = nbr >= 0, over = over0 || (moved && step + 1 == a.steps);
    int4 next = make_int4(0, 0, 0, 0);   // the new vertex, or the next walk (w: there is one)
    uint32_t s_next = 0;
    if (moved && !over) next = vertex_of<APP, LAYOUT>(a, hot, nbr);
    const unsigned want = __ballot_sync(0xffffffffu, over);
    if (want) {
      const int64_t i = take.next(a, want);
      if (over && i < take.n) {
        const int4 e = walk_of<APP, LAYOUT>(a, hot, i);
        next = make_int4(e.y, e.z, e.w, 1);
        s_next = (uint32_t)e.x;
      }
    }
    if (moved) {
      rows.put(a, s, step, nbr);
      step++;
    }
    if (over) {
      rows.end(a, s, step, deg >= 0);
      s = s_next;
      step = next.w ? 0 : -1;
    }
    if (moved || over) {
      prev = cur; ts = rs; tn = deg;
      rs = next.x; deg = next.y; cur = next.z;
      round = 0;
    }
  }
  rows.out(a, tries, 3, words);
}

template <int APP, int LAYOUT>
__device__ __forceinline__ void walks(const RowsArgs &a) {
  if (APP == ND_APP_UNIFORM_WALK) uniform_walks<LAYOUT>(a);
  else if (APP == ND_APP_NODE2VEC) n2v_walks<LAYOUT>(a);
  else weighted_walks<APP, LAYOUT>(a);
}

// Both modes; the load-balanced one also counts the walks that are alive at every step (RowsArgs::ended).
template <int APP, int LAYOUT>
__global__ void __launch_bounds__(ROWS_THREADS, ROWS_CTAS) walk_next_count_kernel(const __grid_constant__ RowsArgs a) { walks<APP, LAYOUT>(a); }

// ---------------------------------------------------------------- layouts, built by a graph's first sampler that reads them

__global__ void vrow_build_kernel(const int32_t *__restrict__ row_ptr, int32_t V, int2 *__restrict__ vrow) {
  for (int64_t v = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; v < V; v += (int64_t)gridDim.x * blockDim.x)
    vrow[v] = make_int2(row_ptr[v], row_ptr[v + 1] - row_ptr[v]);
}

__global__ void colw_build_kernel(const int32_t *__restrict__ col, const float *__restrict__ w, int64_t E, int2 *__restrict__ colw) {
  for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < E; e += (int64_t)gridDim.x * blockDim.x)
    colw[e] = make_int2(col[e], __float_as_int(w[e]));
}

__global__ void vrec_build_kernel(const int32_t *__restrict__ row_ptr, const float *__restrict__ max_w, int32_t V, int2 *__restrict__ vrec) {
  for (int64_t v = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; v <= V; v += (int64_t)gridDim.x * blockDim.x)
    vrec[v] = make_int2(row_ptr[v], v < V ? __float_as_int(max_w[v]) : 0);
}

// A row whose maximum is negative, not a number or so small that its 256th is not exact: the comparisons that the packed
// weights replace do not follow from one another there.
__global__ void odd_max_kernel(const int32_t *__restrict__ row_ptr, const float *__restrict__ max_w, int32_t V, int *__restrict__ odd) {
  for (int64_t v = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; v < V; v += (int64_t)gridDim.x * blockDim.x)
    if (row_ptr[v + 1] - row_ptr[v] > 1 && !(max_w[v] == 0.f || max_w[v] >= 7.8886090522101181e-31f)) *odd = 1;   // 2^-100
}

// a weight as 256ths of its row's maximum, rounded down
__device__ __forceinline__ uint32_t weight_code(float w, float max_w) {
  const float unit = __fmul_rn(max_w, 0.00390625f);
  int b = 255;   // a weight that is not a number accepts every draw: decided by comparing with it
  if (w == w) {
    const float r = __fdiv_rn(w, unit);
    b = r > 0.f ? (r < 255.f ? (int)r : 255) : 0;
    while (b > 0 && !(__fmul_rn((float)b, unit) <= w)) b--;
    while (b < 255 && __fmul_rn((float)(b + 1), unit) <= w) b++;
  }
  return (uint32_t)b;
}

__global__ void __launch_bounds__(BUILD_THREADS)
pack_build_kernel(const int32_t *__restrict__ row_ptr, const int32_t *__restrict__ col, const float *__restrict__ max_w, const float *__restrict__ w,
                  int32_t V, int64_t E, uint32_t *__restrict__ pack) {
  for_entries(row_ptr, V, E, [&](int64_t e, int32_t v) { pack[e] = (uint32_t)col[e] << 8 | weight_code(w[e], max_w[v]); });
}

__global__ void __launch_bounds__(BUILD_THREADS)
codes_build_kernel(const int32_t *__restrict__ row_ptr, const float *__restrict__ max_w, const float *__restrict__ w, int32_t V, int64_t E,
                   uint8_t *__restrict__ codes) {
  for_entries(row_ptr, V, E, [&](int64_t e, int32_t v) { codes[e] = (uint8_t)weight_code(w[e], max_w[v]); });
}

__global__ void __launch_bounds__(BUILD_THREADS)
erec_build_kernel(const int32_t *__restrict__ row_ptr, const int32_t *__restrict__ col, const float *__restrict__ max_w, const float *__restrict__ w,
                  int32_t V, int64_t E, int4 *__restrict__ erec) {
  for_entries(row_ptr, V, E, [&](int64_t e, int32_t v) {
    const int32_t to = col[e], rs = row_ptr[to];
    erec[e] = make_int4(to, rs, row_ptr[to + 1] - rs, (int)weight_code(w[e], max_w[v]));
  });
}

__global__ void col3_build_kernel(const int32_t *__restrict__ col, int64_t E, uint2 *__restrict__ col3) {
  const int64_t n = (E + DENSE_IDS - 1) / DENSE_IDS;
  for (int64_t g = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; g < n; g += (int64_t)gridDim.x * blockDim.x) {
    unsigned long long q = 0;
    for (int k = 0; k < DENSE_IDS; k++)
      if (DENSE_IDS * g + k < E) q |= (unsigned long long)(uint32_t)col[DENSE_IDS * g + k] << (k * DENSE_ID_BITS);
    col3[g] = make_uint2((uint32_t)q, (uint32_t)(q >> 32));
  }
}

__global__ void __launch_bounds__(BUILD_THREADS)
adjsign_build_kernel(const int32_t *__restrict__ row_ptr, const int32_t *__restrict__ col, int32_t V, int64_t E, uint32_t *__restrict__ sign) {
  for_entries(row_ptr, V, E, [&](int64_t e, int32_t t) {
    const int32_t rs = row_ptr[t], deg = row_ptr[t + 1] - rs;
    if (deg < SET_MIN_DEG) return;
    const uint32_t w0 = (uint32_t)rs >> 2, n = ((uint32_t)(rs + deg) >> 2) - w0, h = set_mix((uint32_t)col[e]);
    atomicOr(sign + w0 + set_bucket_of_hash(h, n), set_sign(h));
  });
}

// insert every neighbour id into its row's set: first free slot at or after the home bucket
__global__ void __launch_bounds__(BUILD_THREADS)
adjset_build_kernel(const int32_t *__restrict__ row_ptr, const int32_t *__restrict__ col, int32_t V, int64_t E, int32_t *__restrict__ adjset,
                    int *__restrict__ status) {
  for_entries(row_ptr, V, E, [&](int64_t e, int32_t t) {
    const int32_t rs = row_ptr[t], deg = row_ptr[t + 1] - rs;
    if (deg < SET_MIN_DEG) return;
    const uint32_t n_buckets = ((uint32_t)(rs + deg) >> 2) - ((uint32_t)rs >> 2);
    int32_t *region = adjset + 8 * (size_t)((uint32_t)rs >> 2);
    const int32_t v = col[e];
    uint32_t b = set_bucket(v, n_buckets);
    bool done = false;
    for (uint32_t it = 0; it < n_buckets && !done; it++) {
      for (int i = 0; i < 8 && !done; i++) {
        int32_t *slot = region + 8 * (size_t)b + i;
        int32_t at = *(volatile int32_t *)slot;
        if (at == SET_EMPTY) at = atomicCAS(slot, SET_EMPTY, v);
        done = at == SET_EMPTY || at == v;  // placed, or the id is in the set already (repeated edge)
      }
      b = b + 1 < n_buckets ? b + 1 : 0;
    }
    if (!done) atomicOr(status, ND_DEV_RETRY_LIMIT);  // cannot happen: a region has at least deg slots
  });
}

// Entries that carry the neighbour's row (16 bytes each) shorten a step by a dependent read; they pay while the array, here
// 64 MB, stays in the L2 (130 K vertices, 2.8 M entries, without and with: uniform walk 95 -> 83 us, PPR 115 -> 106, DeepWalk
// 203 -> 198; 60 K, 1.2 M: PPR 117 -> 104; 200 K, 4.8 M: 131 -> 120, 142 -> 132, 293 -> 291; 300 K, 7.2 M: uniform walk
// 171 -> 197, DeepWalk 329 -> 350).  Built by the first sampler of a graph: 0.4 ms at 2.8 M entries.  node2vec fetches two candidates a round and waits for the filter anyway: 298 -> 326.
constexpr int64_t ERECS = (int64_t)1 << 22;
// Ids that leave a byte of a word to the weight.
constexpr int32_t PACK_V = 1 << 24;

template <int APP, int LAYOUT>
void launch(nd_sampler *s, RowsArgs &a, bool count) {
  const int64_t ctas = (s->S + ROWS_THREADS - 1) / ROWS_THREADS, cap = (int64_t)s->dev.sms * ROWS_CTAS;
  const int grid = (int)(ctas < cap ? ctas : cap);
  const int smem = 4 * piece<APP>() * ROWS_THREADS + (count ? 4 * a.steps : 0);
  if (ctas > cap) {   // more walks than lanes: start from the list
    constexpr int per_cta = 256 * START_PER_THREAD;
    walk_start_kernel<APP, LAYOUT><<<(int)((s->S + per_cta - 1) / per_cta), 256, 0, s->stream>>>(a);
    nd_count_launches(1);
  } else {
    a.list = nullptr;
  }
  walk_next_count_kernel<APP, LAYOUT><<<grid, ROWS_THREADS, smem, s->stream>>>(a);
  nd_count_launches(1);
}

template <int APP>
void launch_as(nd_sampler *s, RowsArgs &a, bool count) {
  constexpr bool w = weighted<APP>(), n2v = APP == ND_APP_NODE2VEC;
  switch (s->layout) {   // (the others are not layouts of the app)
    case LAYOUT_FAT: return launch<APP, n2v ? LAYOUT_PLAIN : LAYOUT_FAT>(s, a, count);
    case LAYOUT_ALT: return launch<APP, w ? LAYOUT_ALT : LAYOUT_PLAIN>(s, a, count);
    case LAYOUT_DENSE: return launch<APP, w ? LAYOUT_PLAIN : LAYOUT_DENSE>(s, a, count);
    case LAYOUT_CODES: return launch<APP, w ? LAYOUT_CODES : LAYOUT_PLAIN>(s, a, count);
    case LAYOUT_FAR: return launch<APP, w || n2v ? LAYOUT_FAR : LAYOUT_PLAIN>(s, a, count);
    default: return launch<APP, LAYOUT_PLAIN>(s, a, count);
  }
}

// The derived layouts of a graph are built by the first sampler that needs them; samplers of one
// graph may be created from several host threads, so the builds are serialised, and a sampler keeps the layout that it
// found room for: another's may come to the graph later.  What belongs together goes to the graph together, when all of
// it is there: a build that runs out of memory leaves nothing behind.
std::mutex g_derived_mutex;

template <class T>
int make(T *&p, size_t n) {
  NdDevMem<T> m;
  ND_TRY(m.alloc(n));
  p = m.release();
  return ND_OK;
}

// (neighbour id, weight) records and per-vertex (row start, maximum weight) records
int ensure_colw(const nd_graph *g, int sms) {
  if (g->colw || g->E == 0) return ND_OK;
  NdDevMem<int2> colw, vrec;
  ND_TRY(colw.alloc((size_t)g->E));
  ND_TRY(vrec.alloc((size_t)g->V + 1));
  colw_build_kernel<<<sms * 16, 256>>>(g->col, g->w, g->E, colw.p);
  vrec_build_kernel<<<sms * 16, 256>>>(g->row_ptr, g->max_w, g->V, vrec.p);
  ND_CUDA(cudaDeviceSynchronize());
  g->colw = colw.release();
  g->vrec = vrec.release();
  return ND_OK;
}

int ensure_vrow(const nd_graph *g, int sms) {
  if (g->vrow) return ND_OK;
  NdDevMem<int2> vrow;
  ND_TRY(vrow.alloc((size_t)g->V));
  vrow_build_kernel<<<sms * 16, 256>>>(g->row_ptr, g->V, vrow.p);
  ND_CUDA(cudaGetLastError());
  g->vrow = vrow.release();
  return ND_OK;
}

// `there`: there was room for it
int ensure_erec(const nd_graph *g, int sms, bool *there) {
  *there = g->erec != nullptr;
  if (g->erec) return ND_OK;
  NdDevMem<int4> erec;
  if (erec.alloc((size_t)(g->E > 0 ? g->E : 1)) != ND_OK) return ND_OK;
  erec_build_kernel<<<sms * 16, BUILD_THREADS>>>(g->row_ptr, g->col, g->max_w, g->w, g->V, g->E, erec.p);
  ND_CUDA(cudaGetLastError());
  g->erec = erec.release();
  *there = true;
  return ND_OK;
}

int ensure_pack(const nd_graph *g, int sms, bool *there) {
  *there = g->pack != nullptr;
  if (g->pack) return ND_OK;
  NdDevMem<uint32_t> pack;
  if (pack.alloc((size_t)(g->E > 0 ? g->E : 1)) != ND_OK) return ND_OK;
  pack_build_kernel<<<sms * 16, BUILD_THREADS>>>(g->row_ptr, g->col, g->max_w, g->w, g->V, g->E, pack.p);
  ND_CUDA(cudaGetLastError());
  g->pack = pack.release();
  *there = true;
  return ND_OK;
}

int ensure_codes(const nd_graph *g, int sms) {
  if (g->codes) return ND_OK;
  NdDevMem<uint8_t> codes;
  ND_TRY(codes.alloc((size_t)(g->E > 0 ? g->E : 1)));
  codes_build_kernel<<<sms * 16, BUILD_THREADS>>>(g->row_ptr, g->max_w, g->w, g->V, g->E, codes.p);
  ND_CUDA(cudaGetLastError());
  g->codes = codes.release();
  return ND_OK;
}

// Entries with rows, ids and weights in one word, or the records of ensure_colw where a word does not hold the ids; a byte of
// weight per entry where there is no room for those.  Rows whose weights are no codes have the records.
int ensure_weighted(const nd_graph *g, int sms, int *layout) {
  if (g->odd_max < 0) {
    NdDevMem<int> flag;
    int odd = 0;
    ND_TRY(flag.alloc(1));
    ND_CUDA(cudaMemset(flag.p, 0, sizeof(int)));
    odd_max_kernel<<<sms * 16, 256>>>(g->row_ptr, g->max_w, g->V, flag.p);
    ND_CUDA(cudaMemcpy(&odd, flag.p, sizeof(int), cudaMemcpyDeviceToHost));
    g->odd_max = odd;
  }
  *layout = LAYOUT_PLAIN;
  if (g->odd_max == 1) return ensure_colw(g, sms);
  const bool near = g->V < FAR_V;
  bool there = false;
  const bool rows = (near || g->E <= ERECS) && ensure_vrow(g, sms) == ND_OK;
  if (rows && g->E <= ERECS) ND_TRY(ensure_erec(g, sms, &there));
  if (there) { *layout = LAYOUT_FAT; return ND_OK; }
  if (g->V <= PACK_V) ND_TRY(ensure_pack(g, sms, &there));
  if (there) { *layout = rows && near ? LAYOUT_ALT : LAYOUT_FAR; return ND_OK; }
  if (g->V > PACK_V && ensure_colw(g, sms) == ND_OK) return ND_OK;
  *layout = LAYOUT_CODES;
  return ensure_codes(g, sms);
}

int ensure_col3(const nd_graph *g, int sms, bool *there) {
  *there = g->col3 != nullptr;
  if (g->col3) return ND_OK;
  NdDevMem<uint2> col3;
  if (col3.alloc((size_t)(g->E / DENSE_IDS + 1)) != ND_OK) return ND_OK;
  col3_build_kernel<<<sms * 16, 256>>>(g->col, g->E, col3.p);
  ND_CUDA(cudaGetLastError());
  g->col3 = col3.release();
  *there = true;
  return ND_OK;
}

// the neighbour sets (8 bytes per CSR entry) and the filter in front of them (one byte); `d_status` / `h_status`: the
// status word the build reports to
int ensure_adjset(const nd_graph *g, int sms, int *d_status, const int *h_status) {
  if (g->adjset) return ND_OK;
  const size_t words = (size_t)(g->E > 0 ? g->E : 1) / 4 + 2, slots = 8 * words;
  NdDevMem<uint32_t> sign;
  NdDevMem<int32_t> set;
  ND_TRY(sign.alloc(words));
  ND_TRY(set.alloc(slots));
  ND_CUDA(cudaMemset(sign.p, 0, 4 * words));
  ND_CUDA(cudaMemset(set.p, 0xff, sizeof(int32_t) * slots));
  adjsign_build_kernel<<<sms * 16, BUILD_THREADS>>>(g->row_ptr, g->col, g->V, g->E, sign.p);
  adjset_build_kernel<<<sms * 16, BUILD_THREADS>>>(g->row_ptr, g->col, g->V, g->E, set.p, d_status);
  ND_CUDA(cudaDeviceSynchronize());
  const int st = *(const volatile int *)h_status;
  ND_REQUIRE(st == 0, ND_ERR_DEVICE, "neighbour-set construction failed (status %d)", st);
  g->adjsign = sign.release();
  g->adjset = set.release();
  return ND_OK;
}

}  // namespace

int nd_graph_ensure_vrow(const nd_graph *g, int sms) {
  std::lock_guard<std::mutex> lock(g_derived_mutex);
  return ensure_vrow(g, sms);
}

int nd_graph_ensure_colw(const nd_graph *g, int sms) {
  std::lock_guard<std::mutex> lock(g_derived_mutex);
  return ensure_colw(g, sms);
}

int nd_walk_rows_alloc(nd_sampler *s) {
  const nd_graph *g = s->g;
  const int sms = s->dev.sms, app = s->p.app;
  if (s->S > (int64_t)sms * ROWS_CTAS * ROWS_THREADS) ND_TRY(make(s->d_list, (size_t)s->S));
  const size_t acc = 16 + ((size_t)s->p.steps + 1) / 2;
  ND_TRY(make(s->d_rows_acc, acc));
  ND_CUDA(cudaMemset(s->d_rows_acc, 0, 8 * acc));
  std::lock_guard<std::mutex> lock(g_derived_mutex);
  if (app == ND_APP_DEEPWALK || app == ND_APP_PPR) return ensure_weighted(g, sms, &s->layout);
  const bool n2v = app == ND_APP_NODE2VEC, far = n2v && g->V >= FAR_V;
  if (!far) ND_TRY(ensure_vrow(g, sms));
  if (n2v) ND_TRY(ensure_adjset(g, sms, s->d_status, s->h_status));
  bool fat = !n2v && g->E <= ERECS, dense = !far && g->V <= DENSE_V && g->E >= DENSE_ENTRIES;
  if (fat) ND_TRY(ensure_erec(g, sms, &fat));
  if (dense) ND_TRY(ensure_col3(g, sms, &dense));
  s->layout = far ? LAYOUT_FAR : fat ? LAYOUT_FAT : dense ? LAYOUT_DENSE : LAYOUT_PLAIN;
  return ND_OK;
}

int nd_walk_rows_launch(nd_sampler *s, bool count) {
  const nd_graph *g = s->g;
  uint32_t *ended = count ? reinterpret_cast<uint32_t *>(s->d_rows_acc + 16) : nullptr;
  RowsArgs a{g->V, g->row_ptr, g->col, g->w, g->max_w, g->vrow, g->erec, g->colw, g->vrec,
             s->layout == LAYOUT_CODES ? reinterpret_cast<const uint32_t *>(g->codes) : g->pack, g->col3, g->adjset, g->adjsign,
             ndrng::RoundKeys(s->p.seed), s->p.p, s->p.q, s->p.stop_prob, s->p.n2v_ref_compat, s->p.steps, s->first, s->S, s->d_initial, s->d_out,
             s->d_plen, s->d_list, s->d_rows_acc, ended, s->d_stats, (uint32_t *)s->d_nlive, s->d_status};
  switch (s->p.app) {
    case ND_APP_UNIFORM_WALK: launch_as<ND_APP_UNIFORM_WALK>(s, a, count); break;
    case ND_APP_DEEPWALK: launch_as<ND_APP_DEEPWALK>(s, a, count); break;
    case ND_APP_PPR: launch_as<ND_APP_PPR>(s, a, count); break;
    default: launch_as<ND_APP_NODE2VEC>(s, a, count); break;
  }
  ND_CUDA(cudaGetLastError());
  return ND_OK;
}
