// Random-walk applications (stepSize == 1): uniform walk, DeepWalk, PPR, node2vec.
//
// Transit-parallel path (doTransitParallelSampling, src/nextdoor.cu:2191-3006): every step runs
// one next() kernel over the transit-sorted (transit, sample) map -- the role of samplingKernel /
// identityKernel (src/nextdoor.cu:212-336, 338-504) -- and then inverts the freshly written
// sample->transit pairs with the in-house radix sort.  The next() kernel already counts the first
// radix digit of the keys it writes, so the inversion starts at its scan.
// The other two modes run a lane per walk (nd_walk_rows.cu); what the transit-parallel path needs beyond
// that -- maps, sort scratch, staged output -- is made when it is first asked for.
//
// The transit-parallel kernels write the walk step-major (tmp[step][sample], 4-byte stores that the L2
// merges into full sectors) and a last kernel transposes that into the reference's sample-major layout
// finalSamples[sample*steps + step] (src/nextdoor.cu:2041, 293-334) with coalesced row stores.
#include "nd_cache.cuh"
#include "nd_common.cuh"
#include "nd_nbrset.cuh"
#include "nd_philox.cuh"
#include "nd_walk_rows.cuh"

namespace {

using ndrng::Rng;

struct WalkParams {
  uint64_t seed;
  float p, q, stop_prob;
  int n2v_compat;
  int steps;
  const int32_t *adjset;  // node2vec: per-vertex hash sets of the neighbour ids
  const int2 *colw;       // DeepWalk / PPR: (neighbour id, weight bits) records
  const int2 *vrec = nullptr;  // DeepWalk / PPR: (row start, max weight bits) per vertex, V + 1 entries
  int keep_all_step = -1; // PPR, load-balanced loop: the step whose map goes to the tail launch keeps every pair (see walk_next_ticket_kernel)
};

constexpr int RETRY_CAP = 1 << 16;

// events the algorithmic-bytes model is evaluated from (stats[2..4]); kept per thread and
// flushed once per warp when the kernel ends
struct Events {
  uint32_t weight_tries = 0, n2v_tries = 0, n2v_probes = 0;
  uint32_t not_entered = 0;  // PPR: pairs left out of the next map because the walk is known to stop there (stats[7])
  __device__ __forceinline__ void flush(unsigned long long *stats) {
    uint32_t a = weight_tries, b = n2v_tries, c = n2v_probes, d = not_entered;
    for (int o = 16; o > 0; o >>= 1) {
      a += __shfl_xor_sync(0xffffffffu, a, o);
      b += __shfl_xor_sync(0xffffffffu, b, o);
      c += __shfl_xor_sync(0xffffffffu, c, o);
      d += __shfl_xor_sync(0xffffffffu, d, o);
    }
    if ((threadIdx.x & 31) == 0) {
      if (a) atomicAdd(&stats[2], (unsigned long long)a);
      if (b) atomicAdd(&stats[3], (unsigned long long)b);
      if (c) atomicAdd(&stats[4], (unsigned long long)c);
      if (d) atomicAdd(&stats[7], (unsigned long long)d);
    }
  }
  // The same for a kernel whose CTAs are short-lived (a tile each): the warps' sums meet in shared
  // memory and the CTA adds them once -- with one atomic per warp the half a million warps of a large
  // step queue up on the four counters (measured: 0.4 ms per pass and counter on the 2^24-vertex job).
  // Every thread of the CTA must call it.
  __device__ __forceinline__ void flush_cta(unsigned long long *stats) {
    __shared__ uint32_t sums[4];
    uint32_t a = weight_tries, b = n2v_tries, c = n2v_probes, d = not_entered;
    for (int o = 16; o > 0; o >>= 1) {
      a += __shfl_xor_sync(0xffffffffu, a, o);
      b += __shfl_xor_sync(0xffffffffu, b, o);
      c += __shfl_xor_sync(0xffffffffu, c, o);
      d += __shfl_xor_sync(0xffffffffu, d, o);
    }
    __syncthreads();
    if (threadIdx.x < 4) sums[threadIdx.x] = 0u;
    __syncthreads();
    if ((threadIdx.x & 31) == 0) {
      if (a) atomicAdd(&sums[0], a);
      if (b) atomicAdd(&sums[1], b);
      if (c) atomicAdd(&sums[2], c);
      if (d) atomicAdd(&sums[3], d);
    }
    __syncthreads();
    if (threadIdx.x < 4 && sums[threadIdx.x]) atomicAdd(&stats[threadIdx.x < 3 ? 2 + threadIdx.x : 7], (unsigned long long)sums[threadIdx.x]);
  }
};

// Gathers from the big graph arrays (neighbour ids, weight records, set buckets) are used once per
// launch in the transit-parallel kernels: there they are loaded with the streaming policy
// (evict-first) so that they do not push the small per-sample and per-vertex arrays (maps,
// counters, staged output row, row offsets) out of L2.
template <bool STREAM, typename T>
__device__ __forceinline__ T ld_graph(const T *p) { return STREAM ? __ldcs(p) : __ldg(p); }

// Exact membership of v in the neighbour list [ts, ts+tn) of t.  `probes` counts the 4-byte words read.
template <bool STREAM>
__device__ __forceinline__ bool n2v_member_slow(const NdGraphView &g, const int32_t *adjset, int32_t ts, int32_t tn,
                                                int32_t v, uint32_t bucket, uint32_t n_buckets, uint32_t &probes) {
  if (tn < SET_MIN_DEG) {  // short list: read it
    bool found = false;
#pragma unroll
    for (int k = 0; k < SET_MIN_DEG - 1; k++) {
      const int32_t e = k < tn ? ld_graph<STREAM>(g.col + ts + k) : -1;
      found |= e == v;
    }
    probes += tn;
    return found;
  }
  const int4 *region = reinterpret_cast<const int4 *>(adjset) + 2 * (size_t)((uint32_t)ts >> 2);
  for (uint32_t it = 0; it < n_buckets; it++) {  // the home bucket was full: walk on
    bucket = bucket + 1 < n_buckets ? bucket + 1 : 0;
    const int4 a = ld_graph<STREAM>(region + 2 * (size_t)bucket), b = ld_graph<STREAM>(region + 2 * (size_t)bucket + 1);
    probes += 8;
    if (a.x == v || a.y == v || a.z == v || a.w == v || b.x == v || b.y == v || b.z == v || b.w == v) return true;
    if (b.w == SET_EMPTY) return false;  // slots fill front to back inside a bucket
  }
  return false;
}

constexpr int N2V_BATCH = 4;      // node2vec tries whose gathers are issued together
constexpr int WEIGHT_BATCH = 2;   // weighted tries per round: a larger batch buys latency with gathers that a 60 % acceptance rate wastes

constexpr int32_t ROUND_AGAIN = -2;   // a round of tries ended without an accepted vertex

// The rejection loops of DeepWalk / PPR / node2vec draw their tries from the keyed stream in
// order, so try k of an invocation is a pure function of (sample, step, k).  A ROUND evaluates a
// batch of tries: the gathers of the whole round are issued together (one memory latency instead
// of one per try) and the first try that accepts, in draw order, wins -- the same vertex the
// one-try-at-a-time loop returns.  Only the tries up to the winner are counted.  `rng` carries the
// draw position from round to round.

// weighted rejection (randomWalks.cu:81-89): {x = rand_int(n); y = u * max_w} until !(y > w[x])
template <bool STREAM, int BATCH>
__device__ __forceinline__ int32_t weighted_round(const WalkParams &wp, int32_t rs, int32_t n, float max_w, Rng &rng,
                                                  Events &ev) {
  const int2 *__restrict__ recs = wp.colw + rs;
  float y[BATCH];
  int2 rec[BATCH];
#pragma unroll
  for (int k = 0; k < BATCH; k++) {
    const int32_t x = rng.rand_int(n);
    y[k] = __fmul_rn(rng.uniform(), max_w);
    rec[k] = ld_graph<STREAM>(recs + x);
  }
#pragma unroll
  for (int k = 0; k < BATCH; k++) {
    ev.weight_tries++;
    if (!(y[k] > __int_as_float(rec[k].y))) return rec[k].x;
  }
  return ROUND_AGAIN;
}

// node2vec (randomWalks.cu:151-171).  A candidate that is not the previous vertex t is accepted
// when y < 1/q (neighbour of t) or y < 1 (not a neighbour): below `lo` the membership does not
// matter, at or above `hi` neither; below `sure` nothing about the candidate matters.
struct N2vConsts {
  float inv_q, bound, lo, hi, sure;
  __device__ __forceinline__ explicit N2vConsts(const WalkParams &wp) {
    inv_q = __fdiv_rn(1.0f, wp.q);
    bound = wp.p > inv_q ? wp.p : inv_q;
    if (bound < 1.0f) bound = 1.0f;
    lo = inv_q < 1.0f ? inv_q : 1.0f;
    hi = inv_q < 1.0f ? 1.0f : inv_q;
    sure = lo < wp.p ? lo : wp.p;
  }
};

// t = previous vertex, [ts, ts + tn) its row
template <bool STREAM, int BATCH>
__device__ __forceinline__ int32_t n2v_round(const NdGraphView &g, const WalkParams &wp, const N2vConsts &c, int32_t rs,
                                             int32_t n, int32_t t, int32_t ts, int32_t tn, Rng &rng, Events &ev) {
  const int32_t *__restrict__ edges = g.col + rs;
  const uint32_t n_buckets = ((uint32_t)(ts + tn) >> 2) - ((uint32_t)ts >> 2);
  const int4 *__restrict__ region = reinterpret_cast<const int4 *>(wp.adjset) + 2 * (size_t)((uint32_t)ts >> 2);
  const bool use_set = tn >= SET_MIN_DEG;
  int32_t x[BATCH], v[BATCH];
  float y[BATCH];
  int n_try = BATCH;  // the round ends at the first try that is sure to accept
#pragma unroll
  for (int k = 0; k < BATCH; k++) {
    if (k < n_try) {
      x[k] = rng.rand_int(n);
      y[k] = __fmul_rn(rng.uniform(), c.bound);
      if (y[k] < c.sure) n_try = k + 1;
    }
  }
#pragma unroll
  for (int k = 0; k < BATCH; k++) v[k] = k < n_try ? ld_graph<STREAM>(edges + x[k]) : -1;
  // membership gathers of the tries that need one, issued together
  bool is_ret[BATCH], need[BATCH];
  uint32_t bucket[BATCH];
  int4 ba[BATCH], bb[BATCH];
#pragma unroll
  for (int k = 0; k < BATCH; k++) {
    is_ret[k] = wp.n2v_compat ? (x[k] == t) : (v[k] == t);  // randomWalks.cu:159 compares the index
    need[k] = k < n_try && !is_ret[k] && y[k] >= c.lo && y[k] < c.hi;
    bucket[k] = set_bucket(v[k], n_buckets);
    if (need[k] && use_set) {
      ba[k] = ld_graph<STREAM>(region + 2 * (size_t)bucket[k]);
      bb[k] = ld_graph<STREAM>(region + 2 * (size_t)bucket[k] + 1);
    } else {
      ba[k] = make_int4(SET_EMPTY, SET_EMPTY, SET_EMPTY, SET_EMPTY);
      bb[k] = ba[k];
    }
  }
#pragma unroll
  for (int k = 0; k < BATCH; k++) {
    if (k < n_try) {
      ev.n2v_tries++;
      bool accept;
      if (is_ret[k]) {
        accept = y[k] < wp.p;
      } else if (!need[k]) {
        accept = y[k] < c.lo;
      } else {
        bool found = ba[k].x == v[k] || ba[k].y == v[k] || ba[k].z == v[k] || ba[k].w == v[k] ||
                     bb[k].x == v[k] || bb[k].y == v[k] || bb[k].z == v[k] || bb[k].w == v[k];
        if (use_set) ev.n2v_probes += 8;
        if (!found && (!use_set || bb[k].w != SET_EMPTY))
          found = n2v_member_slow<STREAM>(g, wp.adjset, ts, tn, v[k], bucket[k], n_buckets, ev.n2v_probes);
        accept = y[k] < (found ? c.inv_q : 1.0f);
      }
      if (accept) return v[k];
    }
  }
  return ROUND_AGAIN;
}

// node2vec next() on a transit with n > 1 neighbours at a step > 0 when the row [ts, ts + tn) of the
// previous vertex t is known already
template <bool STREAM>
__device__ __forceinline__ int32_t n2v_next_known(const NdGraphView &g, const WalkParams &wp, int32_t rs, int32_t n,
                                                  int32_t t, int32_t ts, int32_t tn, Rng &rng, int *status, Events &ev) {
  const N2vConsts c(wp);
  for (int it = 0; it <= RETRY_CAP; it += N2V_BATCH) {
    const int32_t r = n2v_round<STREAM, N2V_BATCH>(g, wp, c, rs, n, t, ts, tn, rng, ev);
    if (r != ROUND_AGAIN) return r;
  }
  atomicOr(status, ND_DEV_RETRY_LIMIT);
  return ld_graph<STREAM>(g.col + rs);
}

// One next() of the app on a transit with n > 0 neighbours; -1 = no vertex.
template <int APP, bool STREAM = true>
__device__ __forceinline__ int32_t app_next(const NdGraphView &g, const WalkParams &wp, int step,
                                            int32_t transit, int32_t rs, int32_t n, int32_t &state_t,
                                            Rng &rng, int *status, Events &ev, bool have_max_w = false,
                                            float max_w_in = 0.f) {  // weighted apps: the transit's maximum weight, if the caller fetched it beside the row offsets
  const int32_t *__restrict__ edges = g.col + rs;
  if (APP == ND_APP_UNIFORM_WALK) {  // example/uniformRandWalk.cu:35-36
    return ld_graph<STREAM>(edges + rng.rand_int(n));
  }
  if (APP == ND_APP_DEEPWALK || APP == ND_APP_PPR) {  // randomWalks.cu:74-90, 102-124
    if (APP == ND_APP_PPR) {
      const float pr = rng.uniform();
      if (pr < wp.stop_prob) return -1;
    }
    if (n == 1) return ld_graph<STREAM>(edges);
    const float max_w = have_max_w ? max_w_in : __ldg(g.max_w + transit);
    for (int it = 0; it <= RETRY_CAP; it += WEIGHT_BATCH) {
      const int32_t r = weighted_round<STREAM, WEIGHT_BATCH>(wp, rs, n, max_w, rng, ev);
      if (r != ROUND_AGAIN) return r;
    }
    atomicOr(status, ND_DEV_RETRY_LIMIT);
    return ld_graph<STREAM>(edges);
  }
  if (APP == ND_APP_NODE2VEC) {  // randomWalks.cu:141-172
    if (n == 1 || step == 0) { state_t = transit; return ld_graph<STREAM>(edges); }
    const int32_t t = state_t;
    const int32_t ts = __ldg(g.row_ptr + t);
    const int32_t tn = __ldg(g.row_ptr + t + 1) - ts;
    state_t = transit;
    return n2v_next_known<STREAM>(g, wp, rs, n, t, ts, tn, rng, status, ev);
  }
  return -1;
}

// ---------------------------------------------------------------- set-up kernels

__global__ void walk_reset_kernel(const int32_t *__restrict__ initial, int32_t V, int64_t S, int steps,
                                  int32_t *__restrict__ len, int32_t *__restrict__ state,
                                  unsigned long long *__restrict__ stats, int32_t *__restrict__ tail_ctr,
                                  const int32_t *__restrict__ init_n, int32_t *__restrict__ nlive) {
  const int64_t s = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (s < 8) stats[s] = 0ull;
  if (s == 0) { *tail_ctr = 0; nlive[0] = *init_n; }
  if (s >= S) return;
  const int32_t t = initial[s];
  len[s] = (t >= 0 && t < V) ? steps : -1;
  if (state) state[s] = 0;
}

// walks whose start vertex is valid and has neighbours
__global__ void count_active_kernel(const int32_t *__restrict__ initial, int64_t n, int32_t V,
                                    const int32_t *__restrict__ row_ptr, int32_t *__restrict__ out) {
  int c = 0;
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    const int32_t t = initial[i];
    if (t >= 0 && t < V && row_ptr[t + 1] > row_ptr[t]) c++;
  }
  for (int o = 16; o > 0; o >>= 1) c += __shfl_xor_sync(0xffffffffu, c, o);
  if ((threadIdx.x & 31) == 0 && c) atomicAdd(out, c);
}

__global__ void init_map_kernel(const int32_t *__restrict__ initial, int32_t V, int64_t n,
                                int32_t *__restrict__ keys, int32_t *__restrict__ vals) {
  const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (i >= n) return;
  const int32_t t = initial[i];
  keys[i] = (t >= 0 && t < V) ? t : V;
  vals[i] = (int32_t)i;
}

// ---------------------------------------------------------------- transit-parallel next()

constexpr int NEXT_THREADS = 256;

// One CTA per radix tile of the transit->sample map.  HIST: also count the first radix digit of the
// new keys (layout and digit as the radix scatter of pass 0 expects them).
template <int APP, bool HIST>
__global__ void __launch_bounds__(NEXT_THREADS, APP == ND_APP_NODE2VEC ? 3 : 1)
walk_next_tp_kernel(NdGraphView g, WalkParams wp, int step, int64_t first_sample, int tile_size,
                    const int32_t *__restrict__ in_key, const int32_t *__restrict__ in_val,
                    const int32_t *__restrict__ d_n, int32_t *__restrict__ out_key,
                    int32_t *__restrict__ out_val, int32_t *__restrict__ tmp_step,
                    int32_t *__restrict__ len, int32_t *__restrict__ state, int shift, int bins,
                    uint32_t *__restrict__ tile_hist, int64_t max_tiles, uint32_t *__restrict__ ghist,
                    int *__restrict__ status, unsigned long long *__restrict__ stats) {
  extern __shared__ uint32_t sh_hist[];
  Events ev;
  const int n = *d_n;
  const int tiles = (n + tile_size - 1) / tile_size;
  const uint32_t mask = bins - 1;
  if (HIST) for (int b = threadIdx.x; b < bins; b += NEXT_THREADS) sh_hist[bins + b] = 0;
  for (int tile = blockIdx.x; tile < tiles; tile += gridDim.x) {
    if (HIST) {
      for (int b = threadIdx.x; b < bins; b += NEXT_THREADS) sh_hist[b] = 0;
      __syncthreads();
    }
    const int base = tile * tile_size;
    for (int i = base + threadIdx.x; i < base + tile_size && i < n; i += NEXT_THREADS) {
      const int32_t t = in_key[i];
      const int32_t s = in_val[i];
      int32_t nbr = -1;
      if (t < 0 || t >= g.V) {
        atomicOr(status, ND_DEV_BAD_TRANSIT);
      } else {
        const int32_t rs = __ldg(g.row_ptr + t);
        const int32_t deg = __ldg(g.row_ptr + t + 1) - rs;
        if (deg > 0) {  // next() runs only on transits with edges (src/nextdoor.cu:255,412)
          Rng rng(wp.seed, (uint32_t)(first_sample + s), (uint32_t)step, 0u);
          int32_t st = 0;
          if (APP == ND_APP_NODE2VEC && step > 0) st = state[s];
          nbr = app_next<APP>(g, wp, step, t, rs, deg, st, rng, status, ev);
          if (APP == ND_APP_NODE2VEC && nbr >= 0) state[s] = st;
        }
      }
      if (nbr >= 0) tmp_step[s] = nbr; else len[s] = step;
      if (HIST) {
        out_key[i] = nbr >= 0 ? nbr : g.V;
        out_val[i] = s;
        if (nbr >= 0) atomicAdd(&sh_hist[((uint32_t)nbr >> shift) & mask], 1u);
      }
    }
    if (HIST) {
      __syncthreads();
      for (int b = threadIdx.x; b < bins; b += NEXT_THREADS) {  // a bin is always handled by the same thread
        const uint32_t c = sh_hist[b];
        tile_hist[(int64_t)b * max_tiles + tile] = c;
        sh_hist[bins + b] += c;
      }
      __syncthreads();
    }
  }
  if (HIST)  // one global atomic per bin and CTA
    for (int b = threadIdx.x; b < bins; b += NEXT_THREADS)
      if (sh_hist[bins + b]) atomicAdd(&ghist[b], sh_hist[bins + b]);
  if (APP != ND_APP_UNIFORM_WALK) ev.flush(stats);
}

// ---------------------------------------------------------------- next() + counting inversion (opt-in step loop)
//
// The load-balanced mode's step loop, kept behind its switches for the uniform walk (ND_WALK_STAGING) and PPR
// (ND_WALK_NO_TAIL, ND_WALK_TAIL_PAIRS): a lane per walk is faster at every size (nd_walk_rows.cu).
//
// The transit ids are a dense key space (< V) and the map holds at most one pair per walk, so
// the inversion does not need a multi-pass sort: next() takes a ticket on its new transit
// (atomicAdd on cnt[transit], the ticket is the pair's rank inside the transit's run) and counts
// the pair in a coarse histogram (one bin per CNT_SUPER vertices, kept in shared memory and
// flushed once per CTA); one kernel turns the counters into run offsets (a CTA per bin: the bins
// before it give its base, then an exclusive scan of its own counters, which also clears them and
// publishes the live count); one kernel moves every pair to offs[transit] + rank.  Three launches
// and 16 B read + 8 B written per pair beside the counter traffic, against 2-3 radix passes of
// three launches each.  The order of the pairs inside one transit's run depends on the order the
// tickets were drawn; results do not, because every draw is keyed by the sample.

constexpr int CNT_SUPER = 4096;                             // counters per scan CTA = vertices per coarse bin
constexpr int CNT_SUPER_SHIFT = 12;
constexpr int SCAN_THREADS = 512;
constexpr int SCAN_PER_THREAD = CNT_SUPER / SCAN_THREADS;   // 32 consecutive counters per thread
constexpr int MAX_SMEM_BINS = 8192;                         // coarse bins kept in shared memory (V <= 2^25)

// ---- opt-in: the reference's grid bin for walks (staged adjacency list shared by all samples on a hub)
//
// A tile of HUB_TILE consecutive pairs of the sorted map whose pairs all stand on ONE transit is a
// hub tile; the consecutive hub tiles of a transit form its run.  The CTA that finds the first
// tile of a run streams the transit's adjacency list through shared memory once per pass of
// HUB_PASS tiles and serves all their draws from it (uniform walk: the index is drawn first, the
// pair picks its neighbour when the chunk that holds the index is staged).  The pairs outside
// whole hub tiles stay with the thread-per-pair kernel.  Measured slower than plain gathers (a
// transit of degree d holds d * S / E walkers, so 128 bytes of list are streamed per gather of one
// sector that is saved), hence off unless ND_WALK_STAGING=1; the weighted apps and node2vec probe
// several random positions per try and cannot be served from a streamed chunk at all.
constexpr int HUB_TILE = 256;
constexpr int HUB_PASS = 8;        // tiles whose pairs a CTA serves per sweep of the list
constexpr int HUB_CHUNK = 8192;    // neighbour ids staged at once (32 KB)

// transit of hub tile `tau` of the 8-byte-record map, or -1 if the tile is not one
__device__ __forceinline__ int32_t hub_tile(const int2 *rec, int n, int tau) {
  const int base = tau * HUB_TILE;
  if (tau < 0 || base + HUB_TILE > n) return -1;
  const int32_t a = rec[base].x, b = rec[base + HUB_TILE - 1].x;
  return a == b ? a : -1;
}

constexpr int COUNT_THREADS = 256;

// what the kernel writes for one pair
template <bool COUNT>
__device__ __forceinline__ void count_emit(const ndmem::Keep &keep, int i, int32_t s, int32_t nbr, int32_t V, int step,
                                           bool smem_bins, uint32_t *sh_bins, int32_t *__restrict__ out_key,
                                           int32_t *__restrict__ out_val, int32_t *__restrict__ out_rank,
                                           uint32_t *__restrict__ cnt, uint32_t *__restrict__ bsum,
                                           int32_t *__restrict__ tmp_step, int32_t *__restrict__ len,
                                           bool ends_next = false) {  // the walk takes this vertex and is known to stop at the next step
  if (nbr >= 0) keep.st(tmp_step + s, nbr); else len[s] = step;
  if (ends_next) len[s] = step + 1;
  if (COUNT) {
    const bool in_map = nbr >= 0 && !ends_next;
    keep.st(out_key + i, in_map ? nbr : V);
    if (in_map) {
      keep.st(out_val + i, s);
      keep.st(out_rank + i, (int32_t)keep.atom_add(cnt + nbr, 1u));
      if (smem_bins) atomicAdd(&sh_bins[nbr >> CNT_SUPER_SHIFT], 1u);
      else atomicAdd(&bsum[nbr >> CNT_SUPER_SHIFT], 1u);
    }
  }
}

// A CTA takes tiles of 256 pairs of the sorted map, records {transit, sample}: one record lies in one 32-byte
// sector, so the scatter kernel places a pair with one random sector write.
template <int APP, bool COUNT>
__global__ void __launch_bounds__(COUNT_THREADS, APP == ND_APP_UNIFORM_WALK ? 4 : 5)
walk_next_ticket_kernel(NdGraphView g, WalkParams wp, int step, int64_t first_sample, const int2 *__restrict__ in_rec,
                        const int32_t *__restrict__ d_n, int32_t *__restrict__ out_key, int32_t *__restrict__ out_val,
                        int32_t *__restrict__ out_rank, uint32_t *__restrict__ cnt, uint32_t *__restrict__ bsum, int bins,
                        int32_t *__restrict__ tmp_step, int32_t *__restrict__ len, int *__restrict__ status,
                        unsigned long long *__restrict__ stats, int skip_hub_tiles) {
  static_assert(APP == ND_APP_UNIFORM_WALK || APP == ND_APP_PPR, "the apps with a step loop");
  extern __shared__ uint32_t sh_bins[];
  Events ev;
  const int n = *d_n;
  if ((int64_t)blockIdx.x * COUNT_THREADS >= n) return;  // no pair for this CTA
  const bool smem_bins = COUNT && bins <= MAX_SMEM_BINS;
  if (smem_bins) {
    for (int b = threadIdx.x; b < bins; b += COUNT_THREADS) sh_bins[b] = 0u;
    __syncthreads();
  }
  const ndmem::Keep keep;
  for (int base = blockIdx.x * COUNT_THREADS; base < n; base += gridDim.x * COUNT_THREADS) {
    // staged hub lists (uniform walk): a tile whose 256 pairs all stand on one transit belongs to walk_next_hub_kernel
    if (APP == ND_APP_UNIFORM_WALK && skip_hub_tiles && hub_tile(in_rec, n, base / HUB_TILE) >= 0) continue;
    const int i = base + threadIdx.x;
    if (i >= n) continue;
    const int2 r = keep.ld(in_rec + i);
    const int32_t t = r.x, s = r.y;
    int32_t nbr = -1;
    if (t < 0 || t >= g.V) {
      atomicOr(status, ND_DEV_BAD_TRANSIT);
    } else {
      const int32_t rs = keep.ld_const(g.row_ptr + t);
      const int32_t deg = keep.ld_const(g.row_ptr + t + 1) - rs;
      const float mw = APP == ND_APP_PPR ? __ldg(g.max_w + t) : 0.f;   // independent of the row offsets: one latency, not two
      if (deg > 0) {  // next() runs only on transits with edges (src/nextdoor.cu:255,412)
        Rng rng(wp.seed, (uint32_t)(first_sample + s), (uint32_t)step, 0u);
        int32_t st = 0;
        nbr = app_next<APP>(g, wp, step, t, rs, deg, st, rng, status, ev, true, mw);
      }
    }
    // PPR: whether a walk stops at a step is the first draw of that step's keyed sequence and does
    // not depend on where the walk stands, so the next step's verdict is known now: a pair that
    // would only enter the next map to be dropped from it takes no ticket and is not scattered.
    // (Not in the step that feeds the tail launch: the result update that runs beside the tail
    // tells the tail's walks from the others by their length, and a walk ended here would have
    // the length of one that the tail is about to continue.)
    bool ends_next = false;
    if (APP == ND_APP_PPR && COUNT && nbr >= 0 && step != wp.keep_all_step) {
      Rng ahead(wp.seed, (uint32_t)(first_sample + s), (uint32_t)(step + 1), 0u);
      ends_next = ahead.uniform() < wp.stop_prob;
      ev.not_entered += ends_next ? 1u : 0u;
    }
    count_emit<COUNT>(keep, i, s, nbr, g.V, step, smem_bins, sh_bins, out_key, out_val, out_rank, cnt, bsum, tmp_step, len, ends_next);
  }
  if (smem_bins) {
    __syncthreads();
    for (int b = threadIdx.x; b < bins; b += COUNT_THREADS) {
      const uint32_t cb = sh_bins[b];
      if (cb) atomicAdd(&bsum[b], cb);
    }
  }
  if (APP != ND_APP_UNIFORM_WALK) ev.flush_cta(stats);
}

template <bool COUNT>
__global__ void __launch_bounds__(HUB_TILE)
walk_next_hub_kernel(NdGraphView g, WalkParams wp, int step, int64_t first_sample, const int2 *__restrict__ in_rec,
                     const int32_t *__restrict__ d_n, int32_t *__restrict__ out_key, int32_t *__restrict__ out_val,
                     int32_t *__restrict__ out_rank, uint32_t *__restrict__ cnt, uint32_t *__restrict__ bsum,
                     int32_t *__restrict__ tmp_step, int32_t *__restrict__ len) {
  __shared__ int32_t sh_list[HUB_CHUNK];
  const ndmem::Keep keep;
  const int n = *d_n;
  const int tiles = n / HUB_TILE;
  for (int tau = blockIdx.x; tau < tiles; tau += gridDim.x) {
    const int32_t t = hub_tile(in_rec, n, tau);
    if (t < 0 || hub_tile(in_rec, n, tau - 1) == t) continue;       // not the first tile of a run
    int nt = 1;
    while (hub_tile(in_rec, n, tau + nt) == t) nt++;
    const bool ok = t < g.V;
    const int32_t rs = ok ? __ldg(g.row_ptr + t) : 0;
    const int32_t deg = ok ? __ldg(g.row_ptr + t + 1) - rs : 0;
    for (int j0 = 0; j0 < nt; j0 += HUB_PASS) {
      const int m = nt - j0 < HUB_PASS ? nt - j0 : HUB_PASS;
      int32_t smp[HUB_PASS], x[HUB_PASS], nbr[HUB_PASS];
#pragma unroll
      for (int j = 0; j < HUB_PASS; j++) {
        smp[j] = 0; x[j] = -1; nbr[j] = -1;
        if (j < m) {
          smp[j] = in_rec[(tau + j0 + j) * HUB_TILE + threadIdx.x].y;
          Rng rng(wp.seed, (uint32_t)(first_sample + smp[j]), (uint32_t)step, 0u);
          if (deg > 0) x[j] = rng.rand_int(deg);
        }
      }
      for (int c0 = 0; c0 < deg; c0 += HUB_CHUNK) {
        const int cn = deg - c0 < HUB_CHUNK ? deg - c0 : HUB_CHUNK;
        for (int i = threadIdx.x; i < cn; i += HUB_TILE) sh_list[i] = __ldg(g.col + rs + c0 + i);
        __syncthreads();
#pragma unroll
        for (int j = 0; j < HUB_PASS; j++)
          if (x[j] >= c0 && x[j] < c0 + cn) nbr[j] = sh_list[x[j] - c0];
        __syncthreads();
      }
#pragma unroll
      for (int j = 0; j < HUB_PASS; j++)
        if (j < m)
          count_emit<COUNT>(keep, (int)((tau + j0 + j) * HUB_TILE + threadIdx.x), smp[j], nbr[j], g.V, step, false, nullptr, out_key,
                            out_val, out_rank, cnt, bsum, tmp_step, len);
    }
  }
}

// CTA b owns the counters of coarse bin b: its base is the sum of the bins before it; exclusive
// scan of its counters into offs; counters cleared for the next step; the last CTA publishes the
// number of live pairs.  A bin nobody drew a ticket in holds no transit of the next step: its
// offsets are never read and its counters are zero already.
__global__ void __launch_bounds__(SCAN_THREADS)
cnt_scan_kernel(uint32_t *__restrict__ cnt, const uint32_t *__restrict__ bsum, uint32_t *__restrict__ offs,
                int32_t *__restrict__ d_n_out) {
  __shared__ uint32_t wsum[SCAN_THREADS / 32];
  __shared__ uint32_t base_sh;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const bool is_last = blockIdx.x == gridDim.x - 1;
  const uint32_t own = bsum[blockIdx.x];
  if (own == 0u && !is_last) return;
  uint32_t part = 0;
  for (int i = threadIdx.x; i < (int)blockIdx.x; i += SCAN_THREADS) part += bsum[i];
  for (int o = 16; o > 0; o >>= 1) part += __shfl_xor_sync(0xffffffffu, part, o);
  if (lane == 0) wsum[warp] = part;
  __syncthreads();
  if (threadIdx.x == 0) {
    uint32_t t = 0;
    for (int w = 0; w < SCAN_THREADS / 32; w++) t += wsum[w];
    base_sh = t;
  }
  __syncthreads();
  if (own == 0u) {  // last CTA, empty bin
    if (threadIdx.x == 0) *d_n_out = (int32_t)base_sh;
    return;
  }
  // each thread owns SCAN_PER_THREAD consecutive counters (the arrays are padded to whole bins)
  const size_t first = (size_t)blockIdx.x * CNT_SUPER + (size_t)threadIdx.x * SCAN_PER_THREAD;
  uint32_t c[SCAN_PER_THREAD];
  uint32_t tsum = 0;
#pragma unroll
  for (int r = 0; r < SCAN_PER_THREAD / 4; r++) {
    const uint4 a = *reinterpret_cast<const uint4 *>(cnt + first + 4 * r);
    c[4 * r] = a.x; c[4 * r + 1] = a.y; c[4 * r + 2] = a.z; c[4 * r + 3] = a.w;
    tsum += a.x + a.y + a.z + a.w;
  }
  uint32_t inc = tsum;
  for (int o = 1; o < 32; o <<= 1) {
    const uint32_t t = __shfl_up_sync(0xffffffffu, inc, o);
    if (lane >= o) inc += t;
  }
  __syncthreads();  // wsum reuse
  if (lane == 31) wsum[warp] = inc;
  __syncthreads();
  uint32_t run = base_sh + inc - tsum;
  for (int w = 0; w < warp; w++) run += wsum[w];
  if (tsum != 0u) {  // a thread without tickets has nothing to publish or clear
#pragma unroll
    for (int r = 0; r < SCAN_PER_THREAD / 4; r++) {
      uint4 o;
      o.x = run; run += c[4 * r];
      o.y = run; run += c[4 * r + 1];
      o.z = run; run += c[4 * r + 2];
      o.w = run; run += c[4 * r + 3];
      *reinterpret_cast<uint4 *>(offs + first + 4 * r) = o;
      *reinterpret_cast<uint4 *>(cnt + first + 4 * r) = make_uint4(0u, 0u, 0u, 0u);
    }
  }
  if (is_last && threadIdx.x == SCAN_THREADS - 1) *d_n_out = (int32_t)run;
}

// Moves every live pair to its place in the sorted map of the next step -- one record, one random
// sector write -- and clears the coarse bins (the scan before it was their last reader).
constexpr int SCATTER_PPT = 2;
__global__ void __launch_bounds__(256)
walk_scatter_kernel(const int32_t *__restrict__ d_n, int32_t V, const int32_t *__restrict__ ukey,
                    const int32_t *__restrict__ uval, const int32_t *__restrict__ urank,
                    const uint32_t *__restrict__ offs, int2 *__restrict__ out_rec, uint32_t *__restrict__ bsum, int bins) {
  const int n = *d_n;
  const ndmem::Keep keep;
  for (int b = blockIdx.x * blockDim.x + threadIdx.x; b < bins; b += gridDim.x * blockDim.x) bsum[b] = 0u;
  constexpr int TILE = 256 * SCATTER_PPT;
  for (int base = blockIdx.x * TILE; base < n; base += gridDim.x * TILE) {
    int32_t k[SCATTER_PPT], v[SCATTER_PPT], r[SCATTER_PPT];
    uint32_t pos[SCATTER_PPT];
#pragma unroll
    for (int j = 0; j < SCATTER_PPT; j++) {
      const int i = base + j * 256 + threadIdx.x;
      k[j] = i < n ? keep.ld(ukey + i) : V;
      const bool ok = k[j] != V;
      v[j] = ok ? keep.ld(uval + i) : 0;
      r[j] = ok ? keep.ld(urank + i) : 0;
    }
#pragma unroll
    for (int j = 0; j < SCATTER_PPT; j++) pos[j] = k[j] != V ? keep.ld(offs + k[j]) + (uint32_t)r[j] : 0u;
#pragma unroll
    for (int j = 0; j < SCATTER_PPT; j++)
      if (k[j] != V) keep.st(out_rec + pos[j], make_int2(k[j], v[j]));
  }
}

// the transit-sorted initial map (key, value arrays) as records
__global__ void __launch_bounds__(256)
pack_map_kernel(const int32_t *__restrict__ d_n, const int32_t *__restrict__ key, const int32_t *__restrict__ val,
                int2 *__restrict__ rec) {
  const int n = *d_n;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) rec[i] = make_int2(key[i], val[i]);
}

// Row start, degree and maximum weight of a vertex for a kernel that reaches it by a random id: the
// two neighbouring 8-byte records share a 32-byte sector three times out of four, where the row
// offsets and the maximum weights are two arrays and two sectors.
__device__ __forceinline__ void vertex_of(const WalkParams &wp, int32_t v, int32_t &rs, int32_t &deg, float &max_w) {
  const int2 a = __ldg(wp.vrec + v), b = __ldg(wp.vrec + v + 1);
  rs = a.x;
  deg = b.x - rs;
  max_w = __int_as_float(a.y);
}

// The tail of a job whose walks end early (PPR): once few walks are still alive, a step of the
// transit-parallel loop is three launches whose fixed cost outweighs the per-pair work.  From
// there on one launch finishes the job, a lane per walk: a lane takes a pair of the sorted map
// (a batch of indices per warp from a device counter, so that the lanes end together) and walks its sample to
// the end; a warp makes one round of tries per trip, and a lane
// whose walk ended takes the next pair.  The draws are keyed by (sample, step), so the samples are
// the ones the step-by-step loop would have produced.
// DIRECT: the launch lasts at least as long as the longest surviving walk's chain of dependent
// loads and leaves most of the memory system idle, so it runs on a second stream beside the result
// update of the walks that ended in the step loop (walk_finalize_sparse_kernel with tail_from =
// first_step).  The two kernels split the result rows between them: a survivor's slots from
// first_step on, its entry of plen and its share of the counters belong to this kernel, everything
// else to the other.
constexpr int TAIL_CTAS = 6;
template <int APP, bool DIRECT>
__global__ void __launch_bounds__(256, TAIL_CTAS)
walk_tail_kernel(NdGraphView g, WalkParams wp, int first_step, int64_t first_sample, const int2 *__restrict__ in_rec,
                 const int32_t *__restrict__ d_n, int32_t *__restrict__ next_pair, int64_t S, int32_t *__restrict__ tmp,
                 int32_t *__restrict__ len, int32_t *__restrict__ plen, int32_t *__restrict__ out, int *__restrict__ status,
                 unsigned long long *__restrict__ stats) {
  static_assert(APP == ND_APP_DEEPWALK || APP == ND_APP_PPR, "weighted walks only");
  Events ev;
  const ndmem::Keep keep;
  const int n = *d_n;
  const int lane = threadIdx.x & 31;
  constexpr int TAIL_BATCH = 64;   // at least the 32 indices one trip can ask for
  bool have = false, fresh = true, done = false;
  int32_t s = 0, cur = 0, rs = 0, deg = 0, had = 0;
  int step = 0, rounds = 0;
  int w_cur = 0, w_end = 0;
  float max_w = 0.f;
  int32_t *row = nullptr;
  unsigned int edges = 0, live = 0;
  Rng rng(wp.seed, 0u, 0u, 0u);
  while (true) {
    // The lanes without a walk take the next pair indices of the warp's batch; the warp draws a
    // batch of TAIL_BATCH indices from the device counter when the batch runs out.  (Some lane's
    // walk ends in almost every trip, and an atomic with its round trip to the L2 in every trip
    // doubled the trip: the 1 M-pair tail of the 2^24-vertex job took 0.75 ms with one atomic per
    // trip.)  w_cur / w_end are the same in all lanes.
    const unsigned want = __ballot_sync(0xffffffffu, !done && !have);
    if (want) {
      const int need = __popc(want), avail = w_end - w_cur;
      const int my = __popc(want & ((1u << lane) - 1u));
      int i = w_cur + my;
      if (need <= avail) {
        w_cur += need;
      } else {
        int nb = 0;
        if (lane == 0) nb = atomicAdd(next_pair, TAIL_BATCH);
        nb = __shfl_sync(0xffffffffu, nb, 0);
        if (my >= avail) i = nb + (my - avail);
        w_cur = nb + (need - avail);
        w_end = nb + TAIL_BATCH;
      }
      if (!done && !have) {
        if (i >= n) {
          done = true;
        } else {
          const int2 r = keep.ld(in_rec + i);
          s = r.y;
          cur = r.x;
          step = first_step;
          have = true;
          fresh = true;
          if (cur >= 0 && cur < g.V) {
            vertex_of(wp, cur, rs, deg, max_w);
          } else {
            deg = 0;
          }
          if (DIRECT) {
            row = out + (int64_t)s * wp.steps;
            had = plen[s];
          }
        }
      }
    }
    if (!__any_sync(0xffffffffu, have)) break;   // no lane holds a walk, so every lane found the map exhausted
    if (have) {
      int32_t nbr = ROUND_AGAIN;
      if (deg == 0) {
        nbr = -1;
      } else if (fresh) {  // first trip of a step: the draws of the step start, the cases without a rejection loop
        rng = Rng(wp.seed, (uint32_t)(first_sample + s), (uint32_t)step, 0u);
        rounds = 0;
        fresh = false;
        if (APP == ND_APP_PPR) {
          const float pr = rng.uniform();
          if (pr < wp.stop_prob) nbr = -1;
        }
        if (nbr == ROUND_AGAIN && deg == 1) nbr = __ldg(g.col + rs);
      }
      if (nbr == ROUND_AGAIN) {
        nbr = weighted_round<false, 2>(wp, rs, deg, max_w, rng, ev);
        if (nbr == ROUND_AGAIN && ++rounds > RETRY_CAP) {
          atomicOr(status, ND_DEV_RETRY_LIMIT);
          nbr = __ldg(g.col + rs);
        }
      }
      if (nbr >= 0) {
        if (DIRECT) row[step] = nbr;
        else tmp[(int64_t)step * S + s] = nbr;
        cur = nbr;
        if (++step < wp.steps) {
          vertex_of(wp, cur, rs, deg, max_w);
          fresh = true;
        }
      }
      if (nbr == -1 || step == wp.steps) {  // the walk ends here, after `step` vertices
        if (step < wp.steps) len[s] = step;
        if (DIRECT) {
          for (int k = step; k < had; k++) row[k] = g.V;   // slots the previous pass filled beyond this walk's end
          if (had != step) plen[s] = step;
          edges += step - first_step;
          live += (step < wp.steps ? step + 1 : wp.steps) - first_step;
        }
        have = false;
      }  // ROUND_AGAIN: the lane stays on its step
    }
  }
  if (DIRECT) {
    for (int o = 16; o > 0; o >>= 1) {
      edges += __shfl_xor_sync(0xffffffffu, edges, o);
      live += __shfl_xor_sync(0xffffffffu, live, o);
    }
    if (lane == 0) {
      if (edges) atomicAdd(&stats[0], (unsigned long long)edges);
      if (live) atomicAdd(&stats[1], (unsigned long long)live);
    }
  }
  ev.flush(stats);
}

// ---------------------------------------------------------------- finalize: step-major -> sample-major

constexpr int FIN_SAMPLES = 32;   // samples per CTA
constexpr int FIN_THREADS = 256;

// Step-major staging -> the reference's sample-major rows, every row written whole: a CTA takes 32
// samples, transposes through shared memory and stores 16 bytes per thread.  The kernel of the
// apps whose walks run their full length (uniform walk, DeepWalk, node2vec).
constexpr int FIN_MAX_STEPS = 128;  // steps per smem chunk
__global__ void __launch_bounds__(FIN_THREADS)
walk_finalize_kernel(const int32_t *__restrict__ tmp, const int32_t *__restrict__ len, int32_t *__restrict__ plen, int64_t S,
                     int steps, int32_t invalid, int32_t *__restrict__ out,
                     unsigned long long *__restrict__ stats) {
  __shared__ int32_t tile[FIN_MAX_STEPS][FIN_SAMPLES + 1];
  __shared__ int32_t sh_len[FIN_SAMPLES];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int64_t groups = (S + FIN_SAMPLES - 1) / FIN_SAMPLES;
  unsigned long long edges = 0, live = 0;
  for (int64_t grp = blockIdx.x; grp < groups; grp += gridDim.x) {
    const int64_t s0 = grp * FIN_SAMPLES;
    const int ns = (int)(S - s0 < FIN_SAMPLES ? S - s0 : FIN_SAMPLES);
    if (threadIdx.x < FIN_SAMPLES) {
      const int32_t l = threadIdx.x < ns ? len[s0 + threadIdx.x] : -1;
      sh_len[threadIdx.x] = l;
      if (threadIdx.x < ns) {
        plen[s0 + threadIdx.x] = l > 0 ? l : 0;   // every row is written whole: its slots beyond the walk hold the invalid id
        edges += l > 0 ? l : 0;
        live += l < 0 ? 0 : (l < steps ? l + 1 : steps);
      }
    }
    __syncthreads();
    for (int k0 = 0; k0 < steps; k0 += FIN_MAX_STEPS) {
      const int kc = steps - k0 < FIN_MAX_STEPS ? steps - k0 : FIN_MAX_STEPS;
      const int32_t mylen = sh_len[lane];
      for (int k = warp; k < kc; k += FIN_THREADS / 32) {
        int32_t v = invalid;
        if (lane < ns && k0 + k < mylen) v = tmp[(int64_t)(k0 + k) * S + s0 + lane];
        tile[k][lane] = v;
      }
      __syncthreads();
      // rows of `steps` ints, ns of them back to back
      if (kc == steps) {  // the group's rows are one contiguous, 128-byte aligned piece: 16-byte stores
        int32_t *dst = out + s0 * steps;
        const int total = ns * steps, quads = total >> 2;
        for (int q = threadIdx.x; q < quads; q += FIN_THREADS) {
          int i = (4 * q) / steps, k = 4 * q - i * steps;
          int32_t e[4];
#pragma unroll
          for (int c = 0; c < 4; c++) {
            e[c] = tile[k][i];
            if (++k == steps) { k = 0; i++; }
          }
          __stcs(reinterpret_cast<int4 *>(dst) + q, make_int4(e[0], e[1], e[2], e[3]));
        }
        for (int j = (quads << 2) + threadIdx.x; j < total; j += FIN_THREADS) dst[j] = tile[j % steps][j / steps];
      } else {
        for (int j = threadIdx.x; j < ns * kc; j += FIN_THREADS) {
          const int i = j / kc, k = j % kc;
          out[(s0 + i) * steps + k0 + k] = tile[k][i];
        }
      }
      __syncthreads();
    }
  }
  // CTA-level reduction of the counters, one atomic each
  for (int o = 16; o > 0; o >>= 1) {
    edges += __shfl_xor_sync(0xffffffffu, edges, o);
    live += __shfl_xor_sync(0xffffffffu, live, o);
  }
  if (threadIdx.x == 0 && stats) {  // only warp 0 accumulated
    if (edges) atomicAdd(&stats[0], edges);
    if (live) atomicAdd(&stats[1], live);
  }
}


// The result array keeps its contents from pass to pass, and the kernel keeps the invariant that
// out[s][k] holds the invalid id for every k >= plen[s]: a pass therefore only has to write the
// slots a walk fills now or filled last time.  For walks that end early (PPR: 3 valid steps on
// average in rows of 100) that is a few per cent of the array, where writing every row in full is
// 6.7 GB per pass on the 2^24-vertex job and as long as a quarter of the sampling itself.  Groups
// of 32 samples whose rows need more than FIN_SPARSE slots on average (a scattered 4-byte store
// costs the memory system a sector, so beyond that writing the rows whole is cheaper) go through
// the shared-memory transpose and are written whole, with 16-byte stores.
constexpr int FIN_SPARSE = 8;
constexpr int FIN_BATCH = 8;    // staged rows a lane reads at once
constexpr float FIN_SPARSE_STOP = 0.04f;  // PPR stop probability from which the result update takes this kernel

__global__ void __launch_bounds__(FIN_THREADS)
walk_finalize_sparse_kernel(const int32_t *__restrict__ tmp, const int32_t *__restrict__ len, int32_t *__restrict__ plen, int64_t S,
                     int steps, int32_t invalid, int32_t *__restrict__ out,
                     unsigned long long *__restrict__ stats, int tail_from) {
  // a warp owns a group of 32 samples (lane = sample) from start to end: no block barrier anywhere
  __shared__ int32_t tiles[FIN_THREADS / 32][32][FIN_SAMPLES + 1];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  int32_t (*tile)[FIN_SAMPLES + 1] = tiles[warp];
  const int64_t groups = (S + FIN_SAMPLES - 1) / FIN_SAMPLES;
  const int64_t warps = (int64_t)gridDim.x * (FIN_THREADS / 32);
  unsigned long long edges = 0, live = 0;
  for (int64_t grp = (int64_t)blockIdx.x * (FIN_THREADS / 32) + warp; grp < groups; grp += warps) {
    const int64_t s0 = grp * FIN_SAMPLES;
    const int ns = (int)(S - s0 < FIN_SAMPLES ? S - s0 : FIN_SAMPLES);
    const int32_t l = lane < ns ? len[s0 + lane] : -1;
    // A walk that was alive after step tail_from - 1 is being finished by the tail kernel while this
    // kernel runs (tail_from > steps: no such kernel).  Its length entry reads as `steps` or as its
    // final length, at least tail_from either way; this kernel writes its slots below tail_from and
    // leaves the rest of the row, the row's plen entry and the rest of its counts to the tail kernel.
    const bool surv = l >= tail_from;
    const int32_t had = lane < ns && !surv ? plen[s0 + lane] : 0;
    const int32_t now = surv ? tail_from : (l > 0 ? l : 0);
    const int32_t need = now > had ? now : had;
    if (lane < ns) {
      edges += now;
      live += surv ? tail_from : (l < 0 ? 0 : (l < steps ? l + 1 : steps));
      if (!surv && now != had) plen[s0 + lane] = now;
    }
    const int width = __reduce_max_sync(0xffffffffu, need);   // slots the widest row of the group has to (re)write
    const int total = __reduce_add_sync(0xffffffffu, need);   // ... and all its rows together
    // (a group with a survivor never takes the whole-row path: that one would write the tail kernel's slots)
    if (total <= FIN_SPARSE * FIN_SAMPLES || (steps & 3) != 0 || __any_sync(0xffffffffu, surv)) {
      // the staged row k is read coalesced, each sample's row gets only its few slots
      int32_t *row = out + (s0 + lane) * steps;
      for (int k0 = 0; k0 < width; k0 += FIN_BATCH) {   // the loads of a batch are in flight together
        int32_t v[FIN_BATCH];
#pragma unroll
        for (int j = 0; j < FIN_BATCH; j++) v[j] = k0 + j < now ? tmp[(int64_t)(k0 + j) * S + s0 + lane] : invalid;
#pragma unroll
        for (int j = 0; j < FIN_BATCH; j++)
          if (k0 + j < need) row[k0 + j] = v[j];
      }
      continue;
    }
    // rows written whole, 32 steps at a time through the warp's tile, 16-byte stores
    for (int k0 = 0; k0 < steps; k0 += 32) {
      const int kc = steps - k0 < 32 ? steps - k0 : 32;   // a multiple of 4
      for (int kb = 0; kb < kc; kb += FIN_BATCH) {
        int32_t v[FIN_BATCH];
#pragma unroll
        for (int j = 0; j < FIN_BATCH; j++) {
          const int k = k0 + kb + j;
          v[j] = (lane < ns && kb + j < kc && k < now) ? tmp[(int64_t)k * S + s0 + lane] : invalid;
        }
#pragma unroll
        for (int j = 0; j < FIN_BATCH; j++)
          if (kb + j < kc) tile[kb + j][lane] = v[j];
      }
      __syncwarp();
      const int qn = kc >> 2;                              // 16-byte pieces per sample in this chunk
      for (int q = lane; q < ns * qn; q += 32) {
        const int i = q / qn, c = q - i * qn;
        const int4 v = make_int4(tile[4 * c][i], tile[4 * c + 1][i], tile[4 * c + 2][i], tile[4 * c + 3][i]);
        __stcs(reinterpret_cast<int4 *>(out + (s0 + i) * steps + k0) + c, v);
      }
      __syncwarp();
    }
  }
  // CTA-level reduction of the counters, one atomic per warp
  for (int o = 16; o > 0; o >>= 1) {
    edges += __shfl_xor_sync(0xffffffffu, edges, o);
    live += __shfl_xor_sync(0xffffffffu, live, o);
  }
  if (lane == 0 && stats) {
    if (edges) atomicAdd(&stats[0], edges);
    if (live) atomicAdd(&stats[1], live);
  }
}

// fills the result array with the invalid id once, when the sampler is made (see walk_finalize_kernel)
__global__ void walk_fill_kernel(int32_t *__restrict__ out, int64_t n4, int64_t n, int32_t v) {
  const int4 q = make_int4(v, v, v, v);
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n4; i += (int64_t)gridDim.x * blockDim.x)
    reinterpret_cast<int4 *>(out)[i] = q;
  for (int64_t i = 4 * n4 + blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) out[i] = v;
}

template <int APP>
int launch_next_tp(nd_sampler *s, const WalkParams &wp, int step, bool hist, int grid, const int32_t *in_key,
                   const int32_t *in_val, const int32_t *d_n, int32_t *out_key, int32_t *out_val) {
  const NdRadixPlan &pl = s->radix.plan;
  const int bins = 1 << pl.bits[0];
  NdGraphView gv = nd_view(s->g);
  int32_t *tmp_step = s->d_tmp + (int64_t)step * s->S;
  if (hist) {
    walk_next_tp_kernel<APP, true><<<grid, NEXT_THREADS, 2 * bins * sizeof(uint32_t), s->stream>>>(
        gv, wp, step, s->first, pl.tile, in_key, in_val, d_n, out_key, out_val, tmp_step, s->d_len,
        s->d_state, pl.shift[0], bins, s->radix.tile_hist, pl.max_tiles, s->radix.ghist, s->d_status, s->d_stats);
  } else {
    walk_next_tp_kernel<APP, false><<<grid, NEXT_THREADS, 0, s->stream>>>(
        gv, wp, step, s->first, pl.tile, in_key, in_val, d_n, out_key, out_val, tmp_step, s->d_len,
        s->d_state, 0, 1, nullptr, 0, nullptr, s->d_status, s->d_stats);
  }
  return ND_OK;
}

// next() of one step of the ticket loop: up to 16 CTAs per SM, a tile each
template <int APP>
int launch_ticket(nd_sampler *s, const WalkParams &wp, int step, bool last, int bins, const int2 *in_rec, const int32_t *d_n,
                  int32_t *ukey, int32_t *uval, int32_t *tmp_step) {
  const size_t smem = sizeof(uint32_t) * (bins <= MAX_SMEM_BINS && !last ? (size_t)bins : 0);
  const int64_t tiles = (s->S + COUNT_THREADS - 1) / COUNT_THREADS, cap = (int64_t)s->dev.sms * 16;
  const int grid = (int)(tiles < cap ? (tiles > 0 ? tiles : 1) : cap);
  NdGraphView gv = nd_view(s->g);
  const char *staging_env = getenv("ND_WALK_STAGING");   // hub tiles of the uniform walk through walk_next_hub_kernel
  const int staging = APP == ND_APP_UNIFORM_WALK && staging_env && staging_env[0] == '1' ? 1 : 0;
  if (last)
    walk_next_ticket_kernel<APP, false><<<grid, COUNT_THREADS, smem, s->stream>>>(
        gv, wp, step, s->first, in_rec, d_n, ukey, uval, s->d_rank, s->d_cnt, s->d_bsum, bins, tmp_step, s->d_len, s->d_status, s->d_stats, staging);
  else
    walk_next_ticket_kernel<APP, true><<<grid, COUNT_THREADS, smem, s->stream>>>(
        gv, wp, step, s->first, in_rec, d_n, ukey, uval, s->d_rank, s->d_cnt, s->d_bsum, bins, tmp_step, s->d_len, s->d_status, s->d_stats, staging);
  if (staging) {  // the hub tiles the kernel above left out
    const int hgrid = (int)(tiles < (int64_t)s->dev.sms * 8 ? (tiles > 0 ? tiles : 1) : (int64_t)s->dev.sms * 8);
    if (last)
      walk_next_hub_kernel<false><<<hgrid, HUB_TILE, 0, s->stream>>>(gv, wp, step, s->first, in_rec, d_n, ukey, uval, s->d_rank,
                                                                     s->d_cnt, s->d_bsum, tmp_step, s->d_len);
    else
      walk_next_hub_kernel<true><<<hgrid, HUB_TILE, 0, s->stream>>>(gv, wp, step, s->first, in_rec, d_n, ukey, uval, s->d_rank,
                                                                    s->d_cnt, s->d_bsum, tmp_step, s->d_len);
    nd_count_launches(1);
  }
  return ND_OK;
}

// whether mode 1 takes the step loop over sorted maps for this sampler (its switches are set)
bool step_loop(const nd_sampler *s) {
  const char *st = getenv("ND_WALK_STAGING");
  if (s->p.app == ND_APP_UNIFORM_WALK) return st && st[0] == '1';
  return s->p.app == ND_APP_PPR && (getenv("ND_WALK_NO_TAIL") || getenv("ND_WALK_TAIL_PAIRS"));
}

}  // namespace

bool nd_walk_step_loop(const nd_sampler *s) { return step_loop(s); }

bool nd_walk_lane_per_walk(const nd_sampler *s, int mode) {
  return mode == ND_MODE_SAMPLE_PARALLEL || (mode == ND_MODE_TRANSIT_PARALLEL_LB && !step_loop(s));
}

namespace {
__device__ int g_step_status;                       // device status word of nd_walk_step

// One next() per explicit (transit, sample) pair; the sample id is the global one the draws are keyed by.
template <int APP>
__global__ void __launch_bounds__(256)
walk_step_kernel(NdGraphView g, WalkParams wp, int step, int64_t n, const int32_t *__restrict__ transit,
                 const int64_t *__restrict__ sample, int32_t *__restrict__ next) {
  Events ev;
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    const int32_t t = transit[i];
    int32_t nbr = -1;
    if (t >= 0 && t < g.V) {
      const int32_t rs = __ldg(g.row_ptr + t);
      const int32_t deg = __ldg(g.row_ptr + t + 1) - rs;
      if (deg > 0) {
        Rng rng(wp.seed, (uint32_t)sample[i], (uint32_t)step, 0u);
        int32_t st = 0;
        nbr = app_next<APP, false>(g, wp, step, t, rs, deg, st, rng, &g_step_status, ev);
      }
    }
    next[i] = nbr;
  }
}
// The same for walkers packed as (global sample id << 32) | vertex; an ended walk becomes all ones.
template <int APP>
__global__ void __launch_bounds__(256)
walk_step_packed_kernel(NdGraphView g, WalkParams wp, int step, int64_t n, const unsigned long long *__restrict__ in,
                        unsigned long long *__restrict__ out) {
  Events ev;
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    const unsigned long long x = in[i];
    const int32_t t = (int32_t)(uint32_t)x;
    const uint32_t sample = (uint32_t)(x >> 32);
    int32_t nbr = -1;
    if (x != ~0ull && t >= 0 && t < g.V) {
      const int32_t rs = __ldg(g.row_ptr + t);
      const int32_t deg = __ldg(g.row_ptr + t + 1) - rs;
      if (deg > 0) {
        Rng rng(wp.seed, sample, (uint32_t)step, 0u);
        int32_t st = 0;
        nbr = app_next<APP, false>(g, wp, step, t, rs, deg, st, rng, &g_step_status, ev);
      }
    }
    out[i] = nbr >= 0 ? (((unsigned long long)sample << 32) | (uint32_t)nbr) : ~0ull;
  }
}
}  // namespace

// reads and clears the status word of the two step operators on the current device, after `st` drained
int nd_walk_step_status_read(cudaStream_t st, int *status) {
  ND_CUDA(cudaStreamSynchronize(st));
  int h = 0;
  ND_CUDA(cudaMemcpyFromSymbol(&h, g_step_status, sizeof(int)));
  if (h != 0) {
    const int zero = 0;
    ND_CUDA(cudaMemcpyToSymbol(g_step_status, &zero, sizeof(int)));
  }
  *status = h;
  return ND_OK;
}

int nd_walk_step_packed_launch(const nd_graph *g, const nd_app_params *p, int step, int64_t n, const uint64_t *d_in,
                               uint64_t *d_out, cudaStream_t st) {
  NdDeviceInfo dev;
  ND_TRY(nd_device_info(g->device, &dev));
  if (p->app == ND_APP_DEEPWALK || p->app == ND_APP_PPR) ND_TRY(nd_graph_ensure_colw(g, dev.sms));
  WalkParams wp{p->seed, p->p, p->q, p->stop_prob, p->n2v_ref_compat, p->steps, nullptr, g->colw};
  const int64_t blocks = (n + 255) / 256;
  const int grid = (int)(blocks < (int64_t)dev.sms * 16 ? blocks : (int64_t)dev.sms * 16);
  NdGraphView gv = nd_view(g);
  const unsigned long long *in = (const unsigned long long *)d_in;
  unsigned long long *out = (unsigned long long *)d_out;
  switch (p->app) {
    case ND_APP_UNIFORM_WALK: walk_step_packed_kernel<ND_APP_UNIFORM_WALK><<<grid, 256, 0, st>>>(gv, wp, step, n, in, out); break;
    case ND_APP_DEEPWALK: walk_step_packed_kernel<ND_APP_DEEPWALK><<<grid, 256, 0, st>>>(gv, wp, step, n, in, out); break;
    default: walk_step_packed_kernel<ND_APP_PPR><<<grid, 256, 0, st>>>(gv, wp, step, n, in, out); break;
  }
  nd_count_launches(1);
  ND_CUDA(cudaGetLastError());
  return ND_OK;
}

int nd_walk_step_launch(const nd_graph *g, const nd_app_params *p, int step, int64_t n, const int32_t *d_transits,
                        const int64_t *d_samples, int32_t *d_next, cudaStream_t st) {
  NdDeviceInfo dev;
  ND_TRY(nd_device_info(g->device, &dev));
  if (p->app == ND_APP_DEEPWALK || p->app == ND_APP_PPR) ND_TRY(nd_graph_ensure_colw(g, dev.sms));
  WalkParams wp{p->seed, p->p, p->q, p->stop_prob, p->n2v_ref_compat, p->steps, nullptr, g->colw};
  const int64_t blocks = (n + 255) / 256;
  const int grid = (int)(blocks < (int64_t)dev.sms * 16 ? blocks : (int64_t)dev.sms * 16);
  NdGraphView gv = nd_view(g);
  switch (p->app) {
    case ND_APP_UNIFORM_WALK: walk_step_kernel<ND_APP_UNIFORM_WALK><<<grid, 256, 0, st>>>(gv, wp, step, n, d_transits, d_samples, d_next); break;
    case ND_APP_DEEPWALK: walk_step_kernel<ND_APP_DEEPWALK><<<grid, 256, 0, st>>>(gv, wp, step, n, d_transits, d_samples, d_next); break;
    default: walk_step_kernel<ND_APP_PPR><<<grid, 256, 0, st>>>(gv, wp, step, n, d_transits, d_samples, d_next); break;
  }
  nd_count_launches(1);
  ND_CUDA(cudaGetLastError());
  return ND_OK;
}

int nd_walk_ensure_tmp(nd_sampler *s) {
  if (!s->d_tmp) ND_CUDA(nd_malloc(&s->d_tmp, sizeof(int32_t) * (size_t)(s->S > 0 ? s->S : 1) * s->p.steps));
  return ND_OK;
}

int nd_walk_alloc(nd_sampler *s) {
  const int64_t S = s->S;
  const int steps = s->p.steps;
  ND_REQUIRE(steps >= 1 && steps <= 4096, ND_ERR_ARG, "walk length %d out of range [1,4096]", steps);
  // the result array starts out all-invalid with no slot in use (every kernel that writes rows keeps it that way)
  ND_CUDA(nd_malloc(&s->d_plen, sizeof(int32_t) * (size_t)(S > 0 ? S : 1)));
  ND_CUDA(cudaMemset(s->d_plen, 0, sizeof(int32_t) * (size_t)(S > 0 ? S : 1)));
  if (S > 0) walk_fill_kernel<<<s->dev.sms * 8, 256>>>(s->d_out, S * steps / 4, S * steps, s->g->V);
  ND_CUDA(nd_malloc(&s->d_nlive, sizeof(int32_t) * (size_t)(steps + 5)));  // live pairs per step, a spare slot, the tail launch's work counter, walks that can start, pairs of the initial map
  s->d_init_n = s->d_nlive + steps + 4;
  s->map_stale = true;
  return nd_walk_rows_alloc(s);
}

// What the transit-parallel modes need beyond a lane per walk, made by the first job that runs in one.
static int tp_alloc(nd_sampler *s) {
  const int64_t S = s->S;
  const size_t S1 = (size_t)(S > 0 ? S : 1);
  ND_TRY(nd_walk_ensure_tmp(s));
  if (s->p.app == ND_APP_DEEPWALK || s->p.app == ND_APP_PPR) ND_TRY(nd_graph_ensure_colw(s->g, s->dev.sms));
  if (!s->d_len) ND_CUDA(nd_malloc(&s->d_len, sizeof(int32_t) * S1));
  if (s->p.app == ND_APP_NODE2VEC && !s->d_state) ND_CUDA(nd_malloc(&s->d_state, sizeof(int32_t) * S1));
  s->map_cap = S;
  for (int i = 0; i < 2; i++) {
    if (!s->d_map_key[i]) ND_CUDA(nd_malloc(&s->d_map_key[i], sizeof(int32_t) * S1));
    if (!s->d_map_val[i]) ND_CUDA(nd_malloc(&s->d_map_val[i], sizeof(int32_t) * S1));
  }
  if (!s->d_init_key) ND_CUDA(nd_malloc(&s->d_init_key, sizeof(int32_t) * S1));
  if (!s->d_init_val) ND_CUDA(nd_malloc(&s->d_init_val, sizeof(int32_t) * S1));
  const int key_bits = nd_bit_length((uint32_t)(s->g->V > 1 ? s->g->V - 1 : 1));
  if (!s->radix.tile_hist) ND_TRY(nd_radix_scratch_alloc(&s->radix, key_bits, S));
  return ND_OK;
}

// ... and the step loop of the load-balanced mode
static int loop_alloc(nd_sampler *s) {
  if (s->loop_ready) return ND_OK;
  const size_t V = (size_t)s->g->V, S1 = (size_t)(s->S > 0 ? s->S : 1);
  const size_t bins = (V + CNT_SUPER - 1) / CNT_SUPER;
  if (!s->d_cnt) ND_CUDA(nd_malloc(&s->d_cnt, sizeof(uint32_t) * bins * CNT_SUPER));   // padded to whole bins
  if (!s->d_offs) ND_CUDA(nd_malloc(&s->d_offs, sizeof(uint32_t) * bins * CNT_SUPER));
  if (!s->d_bsum) ND_CUDA(nd_malloc(&s->d_bsum, sizeof(uint32_t) * bins));
  if (!s->d_rank) ND_CUDA(nd_malloc(&s->d_rank, sizeof(int32_t) * S1));
  ND_CUDA(cudaMemset(s->d_cnt, 0, sizeof(uint32_t) * bins * CNT_SUPER));
  ND_CUDA(cudaMemset(s->d_bsum, 0, sizeof(uint32_t) * bins));
  for (int i = 0; i < 2; i++) if (!s->d_srec[i]) ND_CUDA(nd_malloc(&s->d_srec[i], sizeof(int2) * S1));
  if (!s->d_init_rec) ND_CUDA(nd_malloc(&s->d_init_rec, sizeof(int2) * S1));
  if (s->p.app == ND_APP_PPR && s->p.stop_prob > 0.f && !s->h_active) {  // the tail launch runs beside the result update
    ND_CUDA(cudaStreamCreateWithFlags(&s->side, cudaStreamNonBlocking));
    ND_CUDA(cudaEventCreateWithFlags(&s->side_fork, cudaEventDisableTiming));
    ND_CUDA(cudaEventCreateWithFlags(&s->side_join, cudaEventDisableTiming));
    ND_CUDA(cudaEventCreateWithFlags(&s->active_done, cudaEventDisableTiming));
    ND_CUDA(cudaMallocHost(&s->h_active, sizeof(int32_t)));
    *s->h_active = -1;
  }
  s->map_stale = true;   // the records are made with the map
  ND_CUDA(cudaDeviceSynchronize());   // the clears above ran on the default stream
  s->loop_ready = true;
  return ND_OK;
}

// Sort the initial transit->sample map once (the reference uploads it unsorted in the prologue of
// doTransitParallelSampling, src/nextdoor.cu:2207-2231, and never balances step 0, :2400).
int nd_sampler_build_initial_map(nd_sampler *s) {
  const int64_t n = s->S * s->isz;
  ND_REQUIRE(n < ((int64_t)1 << 31), ND_ERR_RANGE, "initial map of %lld pairs does not fit int32", (long long)n);
  const int32_t n32 = (int32_t)n;
  int32_t *d_n_in = s->d_nlive + s->p.steps + 1;  // spare slot
  ND_CUDA(cudaMemcpyAsync(d_n_in, &n32, sizeof(int32_t), cudaMemcpyHostToDevice, s->stream));
  const int blocks = (int)((n + 255) / 256);
  init_map_kernel<<<blocks > 0 ? blocks : 1, 256, 0, s->stream>>>(s->d_initial, s->g->V, n, s->d_map_key[0], s->d_map_val[0]);
  NdSortArrays arr;
  arr.nwords = 2;
  arr.a[0] = (uint32_t *)s->d_map_key[0]; arr.a[1] = (uint32_t *)s->d_map_val[0]; arr.a[2] = nullptr;
  arr.b[0] = (uint32_t *)s->d_map_key[1]; arr.b[1] = (uint32_t *)s->d_map_val[1]; arr.b[2] = nullptr;
  bool in_b = false;
  ND_TRY(nd_radix_sort(s->dev, s->stream, &s->radix, s->radix.plan, arr, 0, d_n_in, s->d_init_n, true, (uint32_t)s->g->V, false, &in_b));
  const int src = in_b ? 1 : 0;
  ND_CUDA(cudaMemcpyAsync(s->d_init_key, s->d_map_key[src], sizeof(int32_t) * n, cudaMemcpyDeviceToDevice, s->stream));
  ND_CUDA(cudaMemcpyAsync(s->d_init_val, s->d_map_val[src], sizeof(int32_t) * n, cudaMemcpyDeviceToDevice, s->stream));
  if (s->d_init_rec) {  // the records the step loop starts from
    const int pg = (int)(blocks < s->dev.sms * 16 ? (blocks > 0 ? blocks : 1) : s->dev.sms * 16);
    pack_map_kernel<<<pg, 256, 0, s->stream>>>(s->d_init_n, s->d_map_key[src], s->d_map_val[src], (int2 *)s->d_init_rec);
  }
  if (s->h_active) {  // PPR: how many walks can start (read when the step loop is laid out, not waited for here)
    s->active_starts = -1;
    *s->h_active = -1;
    int32_t *d_active = s->d_nlive + s->p.steps + 3;
    ND_CUDA(cudaMemsetAsync(d_active, 0, sizeof(int32_t), s->stream));
    count_active_kernel<<<s->dev.sms * 4, 256, 0, s->stream>>>(s->d_initial, n, s->g->V, s->g->row_ptr, d_active);
    ND_CUDA(cudaMemcpyAsync(s->h_active, d_active, sizeof(int32_t), cudaMemcpyDeviceToHost, s->stream));
    ND_CUDA(cudaEventRecord(s->active_done, s->stream));
  }
  s->map_stale = false;
  return ND_OK;  // stream-ordered: no host synchronisation, so chunks on different streams overlap
}

// Enqueues one whole job on the sampler's stream: no host synchronisation, no allocation, every
// size that changes from step to step is read from device memory -- so the sequence can be
// captured into a CUDA graph once and replayed.
static int walk_enqueue(nd_sampler *s, int mode) {
  const int64_t S = s->S;
  const int steps = s->p.steps;
  const int app = s->p.app;
  cudaStream_t st = s->stream;
  WalkParams wp{s->p.seed, s->p.p, s->p.q, s->p.stop_prob, s->p.n2v_ref_compat, steps, s->g->adjset, s->g->colw, s->g->vrec};
  bool tail_direct = false, join = false;   // PPR tail launch: writes the result rows itself / runs on the side stream
  int tail_from = 0x7fffffff;               // first step of that launch
  const int rblocks = (int)((S + 255) / 256);
  walk_reset_kernel<<<rblocks > 1 ? rblocks : 1, 256, 0, st>>>(s->d_initial, s->g->V, S, steps, s->d_len, s->d_state, s->d_stats,
                                                                s->d_nlive + steps + 2, s->d_init_n, s->d_nlive);
  nd_count_launches(1);
  if (mode == ND_MODE_TRANSIT_PARALLEL) {
    // plain transit-parallel: sort-based inversion, first digit histogram fused into next()
    const NdRadixPlan &pl = s->radix.plan;
    const int64_t tiles = pl.max_tiles;
    const int grid = (int)(tiles < (int64_t)s->dev.sms * 8 ? tiles : (int64_t)s->dev.sms * 8);
    const int32_t *in_key = s->d_init_key, *in_val = s->d_init_val;
    int cur = 0;  // buffer the next kernel writes into
    for (int step = 0; step < steps; step++) {
      const bool last = step == steps - 1;
      int32_t *ok = s->d_map_key[cur], *ov = s->d_map_val[cur];
      const int32_t *d_n = s->d_nlive + step;
      nd_phase_begin(s, ND_PHASE_NEXT);
      switch (app) {
        case ND_APP_UNIFORM_WALK: launch_next_tp<ND_APP_UNIFORM_WALK>(s, wp, step, !last, grid, in_key, in_val, d_n, ok, ov); break;
        case ND_APP_DEEPWALK: launch_next_tp<ND_APP_DEEPWALK>(s, wp, step, !last, grid, in_key, in_val, d_n, ok, ov); break;
        case ND_APP_PPR: launch_next_tp<ND_APP_PPR>(s, wp, step, !last, grid, in_key, in_val, d_n, ok, ov); break;
        default: launch_next_tp<ND_APP_NODE2VEC>(s, wp, step, !last, grid, in_key, in_val, d_n, ok, ov); break;
      }
      nd_phase_end(s);
      nd_count_launches(1);
      if (last) break;
      nd_phase_begin(s, ND_PHASE_INVERT);
      NdSortArrays arr;
      arr.nwords = 2;
      arr.a[0] = (uint32_t *)s->d_map_key[cur]; arr.a[1] = (uint32_t *)s->d_map_val[cur]; arr.a[2] = nullptr;
      arr.b[0] = (uint32_t *)s->d_map_key[cur ^ 1]; arr.b[1] = (uint32_t *)s->d_map_val[cur ^ 1]; arr.b[2] = nullptr;
      bool in_b = false;
      ND_TRY(nd_radix_sort(s->dev, st, &s->radix, s->radix.plan, arr, 0, d_n, s->d_nlive + step + 1, true,
                           (uint32_t)s->g->V, true, &in_b));
      nd_phase_end(s);
      const int res = in_b ? (cur ^ 1) : cur;
      in_key = s->d_map_key[res];
      in_val = s->d_map_val[res];
      cur = res ^ 1;
    }
  } else {
    // the step loop of the load-balanced mode: next() draws tickets, counting inversion
    const int V = s->g->V;
    const int bins = (V + CNT_SUPER - 1) / CNT_SUPER;
    // unsorted pairs written by next(): key/val in d_map_*[0], rank; the sorted maps are records that ping-pong between d_srec[0] and d_srec[1]
    int32_t *ukey = s->d_map_key[0], *uval = s->d_map_val[0];
    const int2 *in_rec = (const int2 *)s->d_init_rec;
    const int64_t sblocks = (S + 256 * SCATTER_PPT - 1) / (256 * SCATTER_PPT);
    const int sgrid = (int)(sblocks < (int64_t)s->dev.sms * 16 ? (sblocks > 0 ? sblocks : 1) : (int64_t)s->dev.sms * 16);
    // PPR: a step of the loop costs about 40 us of launches and of the scan over the per-vertex
    // counters whatever the number of pairs, which is what a million pairs cost on top of it.  The
    // map of step k >= 1 holds the walks that can start and pass the stop draws of steps 1..k
    // (pairs known to stop are not entered): active * (1 - stop probability)^(k+1).  The loop runs
    // while that is above a million, one tail launch finishes the rest (ND_WALK_TAIL_PAIRS moves the
    // hand-over, for tests and A/B runs).  `active` was counted when the seeds were set; the layout
    // is fixed when the loop is first captured and kept for later seeds.
    int tp_steps = steps;
    if (app == ND_APP_PPR && s->p.stop_prob > 0.f && !getenv("ND_WALK_NO_TAIL")) {
      const char *e = getenv("ND_WALK_TAIL_PAIRS");
      const double floor_pairs = e ? atof(e) : 1048576.0;
      const double active = s->active_starts >= 0 ? (double)s->active_starts : (double)S;
      const double keep = 1.0 - (double)s->p.stop_prob;
      double in_map = active * keep * keep;   // step 1
      int k = 1;
      while (k < steps && in_map > floor_pairs) { in_map *= keep; k++; }
      tp_steps = k;
    }
    wp.keep_all_step = tp_steps < steps ? tp_steps - 1 : -1;
    int cur = 0;  // sorted map the scatter of this step writes
    for (int step = 0; step < tp_steps; step++) {
      const bool last = step == steps - 1;
      const int32_t *d_n = s->d_nlive + step;
      int32_t *tmp_step = s->d_tmp + (int64_t)step * S;
      nd_phase_begin(s, ND_PHASE_NEXT);
      if (app == ND_APP_PPR) ND_TRY(launch_ticket<ND_APP_PPR>(s, wp, step, last, bins, in_rec, d_n, ukey, uval, tmp_step));
      else ND_TRY(launch_ticket<ND_APP_UNIFORM_WALK>(s, wp, step, last, bins, in_rec, d_n, ukey, uval, tmp_step));
      nd_phase_end(s);
      nd_count_launches(1);
      if (last) break;
      nd_phase_begin(s, ND_PHASE_INVERT);
      cnt_scan_kernel<<<bins, SCAN_THREADS, 0, st>>>(s->d_cnt, s->d_bsum, s->d_offs, s->d_nlive + step + 1);
      walk_scatter_kernel<<<sgrid, 256, 0, st>>>(d_n, V, ukey, uval, s->d_rank, s->d_offs, (int2 *)s->d_srec[cur], s->d_bsum, bins);
      nd_phase_end(s);
      nd_count_launches(2);
      in_rec = (const int2 *)s->d_srec[cur];
      cur ^= 1;
    }
    if (tp_steps < steps) {
      // with the sparse result update the tail writes its walks' slots itself and runs beside that
      // update on the side stream (one after the other on the main stream when the phases are timed)
      tail_direct = s->p.stop_prob >= FIN_SPARSE_STOP && s->side != nullptr;
      const char *ti = getenv("ND_WALK_TAIL_INLINE");   // A/B switch: anything but empty or 0 keeps the tail on the main stream
      const bool forked = tail_direct && !s->timer.on && !(ti && ti[0] && ti[0] != '0');
      cudaStream_t ts = st;
      if (forked) {
        ND_CUDA(cudaEventRecord(s->side_fork, st));
        ND_CUDA(cudaStreamWaitEvent(s->side, s->side_fork, 0));
        ts = s->side;
      }
      nd_phase_begin(s, ND_PHASE_TAIL);
      const int tgrid = s->dev.sms * TAIL_CTAS;   // resident CTAs; the lanes draw their pairs from a counter
      int32_t *next_pair = s->d_nlive + steps + 2;
      if (tail_direct)
        walk_tail_kernel<ND_APP_PPR, true><<<tgrid, 256, 0, ts>>>(nd_view(s->g), wp, tp_steps, s->first, in_rec, s->d_nlive + tp_steps, next_pair,
                                                                 S, s->d_tmp, s->d_len, s->d_plen, s->d_out, s->d_status, s->d_stats);
      else
        walk_tail_kernel<ND_APP_PPR, false><<<tgrid, 256, 0, ts>>>(nd_view(s->g), wp, tp_steps, s->first, in_rec, s->d_nlive + tp_steps, next_pair,
                                                                  S, s->d_tmp, s->d_len, s->d_plen, s->d_out, s->d_status, s->d_stats);
      nd_phase_end(s);
      nd_count_launches(1);
      if (forked) {
        ND_CUDA(cudaEventRecord(s->side_join, s->side));
        join = true;
      }
      tail_from = tail_direct ? tp_steps : tail_from;
    }
  }
  nd_phase_begin(s, ND_PHASE_FINALIZE);
  const int64_t groups = (S + FIN_SAMPLES - 1) / FIN_SAMPLES, fblocks = (groups + FIN_THREADS / 32 - 1) / (FIN_THREADS / 32);
  const int fgrid = (int)(fblocks < (int64_t)s->dev.sms * 16 ? fblocks : (int64_t)s->dev.sms * 16);
  const int dgrid = (int)(groups < (int64_t)s->dev.sms * 16 ? groups : (int64_t)s->dev.sms * 16);
  // walks that end early leave most of a row invalid: the sparse kernel; full-length walks: whole rows
  if (app == ND_APP_PPR && s->p.stop_prob >= FIN_SPARSE_STOP)
    walk_finalize_sparse_kernel<<<fgrid > 0 ? fgrid : 1, FIN_THREADS, 0, st>>>(s->d_tmp, s->d_len, s->d_plen, S, steps, s->g->V, s->d_out, s->d_stats, tail_from);
  else
    walk_finalize_kernel<<<dgrid > 0 ? dgrid : 1, FIN_THREADS, 0, st>>>(s->d_tmp, s->d_len, s->d_plen, S, steps, s->g->V, s->d_out, s->d_stats);
  nd_phase_end(s);
  nd_count_launches(1);
  if (join) ND_CUDA(cudaStreamWaitEvent(st, s->side_join, 0));
  ND_CUDA(cudaGetLastError());
  return ND_OK;
}

int nd_walk_sample(nd_sampler *s, int mode) {
  const bool rows = nd_walk_lane_per_walk(s, mode), loop = mode == ND_MODE_TRANSIT_PARALLEL_LB && !rows;
  s->live_is_ended = mode == ND_MODE_TRANSIT_PARALLEL_LB && rows;
  if (rows) {   // a lane per walk: one or two launches, nothing to capture
    nd_phase_begin(s, ND_PHASE_NEXT);
    const int rc = nd_walk_rows_launch(s, mode == ND_MODE_TRANSIT_PARALLEL_LB);
    nd_phase_end(s);
    return rc;
  }
  ND_TRY(tp_alloc(s));
  if (loop) ND_TRY(loop_alloc(s));
  if (s->map_stale) ND_TRY(nd_sampler_build_initial_map(s));
  // the count of walks that can start is waited for here, outside any stream capture, the first
  // time a step loop is laid out after the seeds were set
  if (s->h_active && s->active_starts < 0 && s->active_done) {
    const bool lays_out = s->stream != nullptr && s->stream != cudaStreamLegacy && s->stream != cudaStreamPerThread &&
                          !s->timer.on && !s->graph_off && !s->graph_exec[mode];   // about to capture this mode's loop
    const cudaError_t ready = lays_out ? cudaEventSynchronize(s->active_done) : cudaEventQuery(s->active_done);
    if (ready == cudaSuccess) s->active_starts = *s->h_active;
    else cudaGetLastError();   // not there yet: this (uncaptured) run is laid out by the number of samples
  }
  // Graph replay needs a capturable stream (not the legacy default stream) and no phase timers.
  const bool capturable = s->stream != nullptr && s->stream != cudaStreamLegacy && s->stream != cudaStreamPerThread;
  if (!capturable || s->timer.on || s->graph_off) return walk_enqueue(s, mode);
  if (!s->graph_exec[mode]) {
    const long long before = nd_launch_count();
    cudaGraph_t graph = nullptr;
    if (cudaStreamBeginCapture(s->stream, cudaStreamCaptureModeThreadLocal) != cudaSuccess) {
      cudaGetLastError();
      s->graph_off = true;
      return walk_enqueue(s, mode);
    }
    const int rc = walk_enqueue(s, mode);
    const cudaError_t ec = cudaStreamEndCapture(s->stream, &graph);
    s->graph_launches[mode] = (int)(nd_launch_count() - before);
    nd_count_launches(-s->graph_launches[mode]);  // nothing ran yet
    if (rc != ND_OK || ec != cudaSuccess || !graph ||
        cudaGraphInstantiate(&s->graph_exec[mode], graph, 0) != cudaSuccess) {
      cudaGetLastError();
      if (graph) cudaGraphDestroy(graph);
      s->graph_exec[mode] = nullptr;
      s->graph_off = true;
      return walk_enqueue(s, mode);
    }
    cudaGraphDestroy(graph);
  }
  ND_CUDA(cudaGraphLaunch(s->graph_exec[mode], s->stream));
  nd_count_launches(s->graph_launches[mode]);
  return ND_OK;
}
