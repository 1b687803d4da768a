// Importance-sampled layers (FastGCN, LADIES): a CTA per sample, all layers of all samples in one launch.
//
// The union of a sample's neighbour lists is a bitmap with a bit per vertex; the rank of a set bit is the
// candidate's place in the sorted unique union, so nothing is sorted.  Candidate weights are summed per group (FastGCN:
// of 512 vertices, LADIES: of 128) in fp64 and scanned; a draw bisects the group sums and finds its candidate
// inside one group with a warp.  Sums are fp64, so they agree with the sorted sequential order to ~1e-16 (FastGCN's
// integer weights sum exactly).
//
// What bounds it, and what is done about it (2^20 vertices, 1024 batches of 64, 2 layers of 64: FastGCN
// 4.8 -> 0.58 ms, LADIES 5.7 -> 0.67 ms).  One CTA fills an SM there, and neither memory nor issue slots are full:
// FastGCN issues in 45 % of the cycles (270 M instructions, 5.1 GB out of the L2), LADIES in 44 % (303 M instructions for 131 M
// list entries, the distinct ones of 313 M); the warps wait for barriers between the phases, for loads and for shared memory:
//  * The second layer's transits are hubs (FastGCN draws them with the square of their degree), many of them the
//    same one: repeated transits of a batch are taken once (LADIES with their multiplicity).
//  * A hub's list (up to 140 K ids; FastGCN's second layer has 28 distinct hubs a sample) costs a shared-memory test per id.  Vertices with at least V/128 neighbours
//    have their neighbourhood as a bitmap, built once per graph: V/8 bytes that are ORed in registers, word by
//    word, and stored to the union once; and an adjacency probe of such a transit is a bit test.
//  * FastGCN's weights are summed without a list of candidates (writing that and fetching deg^2 one by one took more
//    than half of the time).  The degrees lie in the order of the bitmap, a byte each: a lane takes the 32 vertices of a word with one load,
//    masks them with it and squares and sums them with dp4a (byte b of code word j is vertex j + 8 b: a mask is a shift and a
//    byte permutation; sixteen vertices a lane in their own order, with a multiplication a mask, 0.622 ms, now 0.588).  The two bytes that hold degrees up to 2047 take three times as many, so that from 256 on, where few vertices have
//    as many, they are a list (20 K of 2^20, 65 against 160 thousand cycles an SM); where they are not few the codes have a
//    second byte, for the groups that need it.  Groups without a candidate are passed over, and the lists beside the hubs',
//    where they are short (a first layer's: 2 K entries), are weighed entry by entry as they come into the union, one or an eight of
//    entries to a thread, instead of looking through 2^20 vertices for them (390 -> 100 thousand cycles an SM with the lists
//    a warp each before; V / FEW: 64 0.755, 16 0.79 ms).  Groups' sums are two 32-bit words until they are scanned: a 64-bit
//    add in shared memory is a loop.  0.89 -> 0.74 ms, 256 batches on 2^21 0.56 -> 0.46, 700 of 100 on 100 K 0.50 -> 0.46.
//  * FastGCN's draws: the groups are found a thread a draw (a warp each took as long twice, for two draws); then a warp sums the
//    group's weights, sixteen vertices a lane, and goes to the vertices of the one lane that reaches the target, one scan each
//    instead of one for every 128 vertices.  0.74 -> 0.70 ms, 0.46 -> 0.45, 0.46 -> 0.41.  (Weights as whole numbers: 0.75, the
//    few of them that are not below 2^24 diverge.)
//  * LADIES' terms (w / rowsum)^2 depend on the edge alone: an array, built once per graph, instead of a pass over
//    the weights and a division per entry and sample.  One pass over the lists sets the union's bits and adds the terms
//    up per group; then the groups that the draws fall into get an accumulator per vertex, where the union was,
//    and a second pass adds up the terms of their candidates alone (131 K entries, 37 of 8192 groups, 9 % of the entries).
//    (Until then the candidates' weights were added up by rank, in tiles of shared memory: the rank of every entry, a
//    double added per entry, a few barriers per tile; 1024 batches on 2^20 vertices 2.50 -> 1.07 ms, 256 on 2^21 1.37 ->
//    0.64, 700 batches of 100 and 3 layers of 100 on 100 K 1.52 -> 0.88.)  A thread takes eight entries, 32 bytes of ids and
//    of terms; what neighbouring entries add to one group is added up in registers and across the lanes first, as a 64-bit
//    add in shared memory costs 18 cycles a warp.  Groups of 128: with larger ones the second pass adds more, with smaller
//    ones the first (64: 1.08, 256: 1.05 ms, but 0.29 instead of 0.25 with 300 batches on 500 K).
//  * Hubs hold two thirds of the entries of a second layer (2.7 of 27 lists).  Both passes leave them out: their sums per
//    group are a table per graph, 64 KB a hub, and a group's candidates are a range of the hub's neighbours, each kept
//    once with the sum of its terms (graphs repeat edges between hubs hundreds of times: the plain range, with all its adds
//    to one candidate, took longer than the pass it replaced).  1.07 -> 0.80, 0.64 -> 0.51, 0.88 -> 0.72, 0.25 -> 0.19 ms.
//    Where the tables would be larger than HUB_TABLES, or a hub's list does not ascend, hubs are lists like the others.
#include <algorithm>
#include <cstdlib>
#include <mutex>
#include <vector>

#include "nd_collective.cuh"

namespace {

using ndrng::Rng;

constexpr int GROUP_WORDS = 16;   // words of a FastGCN group; bitmaps are whole ones
constexpr int GROUP = 512;        // FastGCN: vertices (GROUP_WORDS words) whose weights are summed together
constexpr int LADIES_GROUP_BITS = 7;   // LADIES: 2^7 vertices, more where the sums of the groups would not fit shared memory
constexpr int RUN = 4;            // listed vertices a thread takes at a time
constexpr int BIG_DEGREE = 2048;  // from here a vertex is listed and its code is 0: 512 * 2047^2 < 2^31
constexpr int LISTED = 32;        // degrees are codes of a byte where no more than V / LISTED vertices do not fit one
constexpr int FLIGHT = 4;         // pairs of groups a warp sums at a time (2^20 vertices 2: 0.595, 3: 0.589, 4: 0.588 ms; 600 K, 100 batches 77.7, 76.7, 76.3 us)
constexpr int HUB = 128;          // a vertex with at least V / HUB neighbours has a bitmap of them
constexpr int32_t SHARED_V = 1 << 18;   // see plan_of()
constexpr int FEW = 64;           // lists with fewer than V / FEW entries in all are weighed entry by entry
// Entries a thread, up to which lists that are weighed entry by entry are taken an entry at a time, and not eight (148 batches of 4, layers
// of 4, 30 K vertices: 29.9 us, one 26.3, two 26.2, four 26.3; 125 K: 33.7, 33.1, 30.9, 30.9; 1000 of 64 on 1 M: 527, 523, 521, 521, without a
// limit 533; 148 of 16, 40 edges a vertex, 106, 106, 106, 106, 115).
constexpr int ENTRIES = 4;
constexpr int PAIRS = 8, PAIR_ROWS = 8;   // longest layer and fewest lists that are probed pair by pair, see the kernel's adjacency
constexpr int SUB = 16;           // LADIES: lanes that add up a group of a hub (100 K vertices: 32 0.62, 16 0.595, 8 0.595, 4 0.60 ms; 2^20: 0.77, 0.77, 0.78, 0.80)
constexpr int OCT = 8;            // list entries a thread takes at a time: 32 aligned bytes

// The bitmap and FastGCN's CDF make the "big" part (V/8 + V/64 bytes).  It lives in shared memory when the whole layout
// fits the CTA's opt-in shared memory (graphs up to about 1.2 M vertices) and otherwise in a per-CTA slice of a global
// scratch array (glob_bytes > 0), where the same code runs on L2-resident words.  The rest is always in shared memory.
struct Layout {
  int words, groups;
  int group_bits;                                      // LADIES: vertices of a group, as a power of two
  int slots;                                           // LADIES: groups with accumulators at a time
  uint32_t off_gcdf;                                   // FastGCN: inside the big part (the bitmap is at 0); LADIES: inside shared memory, unless sums_far
  bool sums_far;
  uint32_t off_red, off_tr, off_layer, off_ut, off_mult, off_same, off_pre;   // inside shared memory
  uint32_t off_draw, off_acc;                           // the same; LADIES' accumulators, which may be where the bitmap is
  uint32_t off_slot;                                   // LADIES: with the groups' sums
  uint32_t bytes;                                      // dynamic shared memory of the launch
  uint32_t glob_bytes;                                 // per-CTA slice of the global scratch, 0 = big part in shared memory
};

// vertices there is room for on a list of n
__host__ __device__ inline int64_t listed_room(int64_t n) { return (n + 7) / 8 * 8 + 8; }

// The degrees, FastGCN.  Codes: the low bytes of 32 vertices' each in two (squares() says in which order), then the high ones if
// there are any; a listed vertex's is zero.
struct Degrees {
  const uint4 *__restrict__ codes;
  const uint32_t *__restrict__ wide;        // a bit per group: it has high bytes that are not zero; null: none has
  const int32_t *__restrict__ listed;       // [listed_room(n_listed)] vertices in order, read in whole runs, beyond n_listed 0 without a weight
  const uint2 *__restrict__ weights;        // ... their weights as the words of a Sum
  int n_listed;
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
  uint32_t *adj;
  float *prob;
  Degrees deg;                             // FastGCN
  const NdBigVertex *__restrict__ huge;    // ... vertices with at least HUGE_DEGREE neighbours
  int n_huge;
  const float *__restrict__ term;          // LADIES: (w / rowsum)^2 per entry
  const int32_t *__restrict__ hub_slot;    // [V] slot of the vertex's bitmap, -1: none
  const uint32_t *__restrict__ hub_bits;   // [slots][words]
  const double *__restrict__ hub_sums;     // LADIES: [slots][groups] the terms of a hub's list per group, or null
  const int32_t *__restrict__ hub_starts;  // ... [slots][groups + 1] where each group of it begins in
  const int32_t *__restrict__ hub_ids;     // ... the hubs' neighbours, each once
  const double *__restrict__ hub_terms;    // ... and the sums of their terms
  unsigned long long *acc;                 // counters of the running job: [0] draws, [5] ids, [6] candidates, [8] next sample, [10] CTAs done; zero between jobs
  unsigned long long *stats;               // published by the last CTA
  unsigned long long pairs;
};

// a transit of the batch: row start, degree, how often it occurs, bitmap slot
struct Transit { int32_t rs, deg, mult, slot; };

constexpr uint32_t NO_SLOT = 255u;

// exclusive scan of an array by the whole CTA; its sum.  A few words are one warp's (every thread adding up all warps' sums takes a
// thousand cycles); else every thread owns a contiguous chunk and the chunks' sums are scanned through shuffles.
__device__ __forceinline__ uint32_t scan_u32(uint32_t *a, int n, uint32_t *red) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, warps = blockDim.x >> 5;
  if (n <= 128) {
    if (warp == 0) {
      uint32_t carry = 0;
      for (int i0 = 0; i0 < n; i0 += 32) {
        const uint32_t own = i0 + lane < n ? a[i0 + lane] : 0u;
        uint32_t inc = own;
        for (int o = 1; o < 32; o <<= 1) {
          const uint32_t t = __shfl_up_sync(0xffffffffu, inc, o);
          if (lane >= o) inc += t;
        }
        if (i0 + lane < n) a[i0 + lane] = carry + inc - own;
        carry += __shfl_sync(0xffffffffu, inc, 31);
      }
      if (lane == 0) red[0] = carry;
    }
    __syncthreads();
    return red[0];
  }
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

// Inclusive scan of n doubles by the whole CTA, get(i) gives the i-th to be added (in place is fine).  A thread owns P neighbouring
// ones, read and written two at a time; of eight each second thread starts at another pair, or the accesses of a quarter
// of a warp would meet in two banks' places (rows of 32 scanned by shuffles and every warp's base added up from memory, with the
// counts' sums and the lists' scan done likewise by all threads: 1024 batches on 2^20 vertices FastGCN 0.69 -> 0.665 ms, LADIES
// 0.775 -> 0.725; 600 of 32, layers of 100, on 900 K 0.43 -> 0.40).  The adds that lead to two neighbouring sums come in different orders,
// so the sums may differ by a rounding where nothing lies between them: an element of zero takes over the sum before it,
// and the first sum to reach a target is never one of those.  (Values are made relative to the warp first; the warps' bases are
// added up in order from what their last elements become, so what is equal stays equal.)
template <int P, class Get>
__device__ __forceinline__ void scan_f64(double *a, int n, double *red, Get get) {
  constexpr int PAIRS = P / 2;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, warps = blockDim.x >> 5;
  const int turn = PAIRS == 4 ? (threadIdx.x >> 1) & 3 : 0;
  double start = 0.0;   // the sum before the block
  for (int b0 = 0; b0 < n; b0 += P * (int)blockDim.x) {
    const int b = b0 + P * (int)threadIdx.x;
    double2 d[PAIRS];
#pragma unroll
    for (int k = 0; k < PAIRS; k++) {
      const int i = b + 2 * ((k + turn) & (PAIRS - 1));
      d[k] = i + 1 < n ? get.two(i) : make_double2(i < n ? get.one(i) : 0.0, 0.0);
    }
    if (PAIRS == 4) {   // pair k is at (k - turn) & 3
      if (turn & 1) { const double2 x = d[3]; d[3] = d[2]; d[2] = d[1]; d[1] = d[0]; d[0] = x; }
      if (turn & 2) { double2 x = d[0]; d[0] = d[2]; d[2] = x; x = d[1]; d[1] = d[3]; d[3] = x; }
    }
    double sum = 0.0;
#pragma unroll
    for (int k = 0; k < PAIRS; k++) { sum += d[k].x; sum += d[k].y; }
    double before = sum;
    for (int o = 1; o < 32; o <<= 1) {
      const double t = __shfl_up_sync(0xffffffffu, before, o);
      if (lane >= o) before += t;
    }
    before = __shfl_up_sync(0xffffffffu, before, 1);
    if (lane == 0) before = 0.0;
    const bool some = sum != 0.0;
    double last = before;
#pragma unroll
    for (int k = 0; k < PAIRS; k++) { last += d[k].x; last += d[k].y; }
    const uint32_t those = __ballot_sync(0xffffffffu, some), left = those & ((1u << lane) - 1u);
    const double taken = __shfl_sync(0xffffffffu, last, left ? 31 - __clz(left) : 0);   // what elements of zero take over
    double take = left ? taken : 0.0;
    const double end = __shfl_sync(0xffffffffu, last, those ? 31 - __clz(those) : 0);
    if (lane == 0) red[warp] = those ? end : 0.0;
    __syncthreads();
    double base = start, next = start;
#pragma unroll 8
    for (int w = 0; w < warps; w++) {
      next += red[w];
      if (w + 1 == warp) base = next;
    }
    start = next;
    double run = before;
#pragma unroll
    for (int k = 0; k < PAIRS; k++) {
      run += d[k].x;
      if (d[k].x != 0.0) take = run;
      d[k].x = base + take;
      run += d[k].y;
      if (d[k].y != 0.0) take = run;
      d[k].y = base + take;
    }
    if (PAIRS == 4) {
      if (turn & 1) { const double2 x = d[0]; d[0] = d[1]; d[1] = d[2]; d[2] = d[3]; d[3] = x; }
      if (turn & 2) { double2 x = d[0]; d[0] = d[2]; d[2] = x; x = d[1]; d[1] = d[3]; d[3] = x; }
    }
#pragma unroll
    for (int k = 0; k < PAIRS; k++) {
      const int i = b + 2 * ((k + turn) & (PAIRS - 1));
      if (i + 1 < n) *reinterpret_cast<double2 *>(a + i) = d[k];
      else if (i < n) a[i] = d[k].x;
    }
    __syncthreads();
  }
}

// The threads' sum, for all of them.  (Added up in memory from every warp's first lane instead, with a fence behind, the end of a call cost
// 1 to 3 us: 148 batches of 8, layers of 8, 3000 vertices 26.7 -> 24.9 us, of 1 24.6 -> 21.7, of 16 28.9 -> 26.9; LADIES, of 1, 33.0 -> 31.0.)
__device__ __forceinline__ unsigned long long sum_of_all(unsigned long long x, double *red) {
  unsigned long long *const sums = reinterpret_cast<unsigned long long *>(red);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, warps = blockDim.x >> 5;
  for (int o = 16; o > 0; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
  __syncthreads();
  if (lane == 0) sums[warp] = x;
  __syncthreads();
  x = lane < warps ? sums[lane] : 0ull;
  for (int o = 16; o > 0; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
  return x;
}

// eight consecutive words at an address that is a multiple of 32
__device__ __forceinline__ void load8(const int32_t *p, int32_t (&v)[OCT]) {
  asm("ld.global.nc.v8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
      : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]) : "l"(p));
}

// Octs: the aligned groups of eight entries that a list touches.
__device__ __forceinline__ uint32_t octs_of(int32_t rs, int32_t deg) { return deg > 0 ? (((uint32_t)rs + (uint32_t)deg + OCT - 1u) / OCT) - (uint32_t)rs / OCT : 0u; }

// the list of oct o of all: the last with pre <= o
__device__ __forceinline__ int list_of_oct(const uint32_t *pre, int nu, uint32_t o) {
  int lo = 0;
  for (int hi = nu - 1; lo < hi;) {
    const int mid = (lo + hi + 1) >> 1;
    if (pre[mid] <= o) lo = mid; else hi = mid - 1;
  }
  return lo;
}

// the entries of an oct that belong to the list, as bits
__device__ __forceinline__ uint32_t oct_mask(int64_t e, const Transit &t) {
  const int64_t lo = (int64_t)t.rs - e, hi = (int64_t)t.rs + t.deg - e;
  return (hi >= OCT ? 0xffu : (1u << (int)hi) - 1u) & (lo <= 0 ? 0xffu : 0xffu << (int)lo);
}

__device__ __forceinline__ float square(int32_t deg) {
  const float d = __int2float_rn(deg);
  return __fmul_rn(d, d);
}

// ... as a whole number, which it is
__device__ __forceinline__ unsigned long long weight_of(int32_t deg) { return deg <= 4096 ? (unsigned long long)((uint32_t)deg * (uint32_t)deg) : (unsigned long long)square(deg); }

// FastGCN: a group's sum is two words while it is added up (64-bit adds in shared memory are loops): low SUM_BITS bits of the
// weights below, the rest above.  A group's 512 weights fit them up to HUGE_DEGREE neighbours.
constexpr int SUM_BITS = 22, HUGE_DEGREE = 1 << 22;
struct Sum {
  uint32_t low = 0, high = 0;
  __device__ __forceinline__ void add(int32_t deg) {
    if (deg < BIG_DEGREE) {
      low += (uint32_t)(deg * deg);
    } else if (deg < HUGE_DEGREE) {
      const unsigned long long w = weight_of(deg);
      low += (uint32_t)w & ((1u << SUM_BITS) - 1u);
      high += (uint32_t)(w >> SUM_BITS);
    }
  }
  __device__ __forceinline__ void to(uint2 *sums, int group) const {
    if (low) atomicAdd(&sums[group].x, low);
    if (high) atomicAdd(&sums[group].y, high);
  }
  static __device__ __forceinline__ double value(const uint2 &s) { return (double)s.x + (double)(1 << SUM_BITS) * (double)s.y; }
};

struct Doubles {
  const double *a;
  __device__ __forceinline__ double one(int i) const { return a[i]; }
  __device__ __forceinline__ double2 two(int i) const { return *reinterpret_cast<const double2 *>(a + i); }
};
struct Sums {
  const uint2 *a;
  __device__ __forceinline__ double one(int i) const { return Sum::value(a[i]); }
  __device__ __forceinline__ double2 two(int i) const {
    const uint4 s = *reinterpret_cast<const uint4 *>(a + i);
    return make_double2(Sum::value(make_uint2(s.x, s.y)), Sum::value(make_uint2(s.z, s.w)));
  }
};
// few elements: two a thread
template <class Get>
__device__ __forceinline__ void scan_groups(double *a, int n, double *red, Get get) {
  if (n <= 2 * (int)blockDim.x) scan_f64<2>(a, n, red, get);
  else scan_f64<8>(a, n, red, get);
}

// FastGCN: the entries of the lists without bitmaps into the union; with WEIGHTS what they add to it goes to the groups' sums
// and is counted (the number the thread has added).
template <bool WEIGHTS>
__device__ __forceinline__ uint32_t add_lists(const NdGraphView &g, const Transit *rest, int n, const uint32_t *pre, uint32_t total, uint32_t *bm, uint2 *sums) {
  uint32_t added = 0;
  int i = 0;
  for (uint32_t o = threadIdx.x; o < total; o += blockDim.x) {
    if (i + 1 < n && pre[i + 1] <= o) i = list_of_oct(pre, n, o);
    const Transit t = rest[i];
    const int64_t e = ((int64_t)((uint32_t)t.rs / OCT) + (int64_t)(o - pre[i])) * OCT;
    int32_t v[OCT];
    load8(g.col + e, v);
    uint32_t fresh = oct_mask(e, t);
    {
      uint32_t word[OCT];
#pragma unroll
      for (int j = 0; j < OCT; j++) word[j] = (fresh >> j) & 1u ? bm[(uint32_t)v[j] >> 5] : ~0u;
#pragma unroll
      for (int j = 0; j < OCT; j++) {   // (most ids of a hub's neighbours are there already)
        const uint32_t bit = 1u << (v[j] & 31);
        if ((word[j] & bit) || (atomicOr(bm + ((uint32_t)v[j] >> 5), bit) & bit)) fresh &= ~(1u << j);
      }
    }
    if (!WEIGHTS || !fresh) continue;
    added += __popc(fresh);
    int32_t deg[OCT];
#pragma unroll
    for (int j = 0; j < OCT; j++) deg[j] = (fresh >> j) & 1u ? __ldg(g.row_ptr + v[j] + 1) - __ldg(g.row_ptr + v[j]) : 0;
    int at = -1;
    Sum sum;
#pragma unroll
    for (int j = 0; j < OCT; j++) {
      if (!((fresh >> j) & 1u)) continue;
      if (v[j] / GROUP != at) {
        if (at >= 0) sum.to(sums, at);
        at = v[j] / GROUP;
        sum = Sum();
      }
      sum.add(deg[j]);
    }
    sum.to(sums, at);
  }
  return added;
}

// ... with WEIGHTS, an entry to a thread: eight are one after another, which lists that leave most of the CTA idle need not wait for.
__device__ __forceinline__ uint32_t add_entries(const NdGraphView &g, const Transit *rest, int n, const uint32_t *pre, uint32_t total, uint32_t *bm, uint2 *sums) {
  uint32_t added = 0;
  for (uint32_t x = threadIdx.x; x < total * OCT; x += blockDim.x) {
    const uint32_t o = x / OCT;
    const int i = list_of_oct(pre, n, o);
    const Transit t = rest[i];
    const int64_t e = ((int64_t)((uint32_t)t.rs / OCT) + (int64_t)(o - pre[i])) * OCT + x % OCT;
    if (e < t.rs || e >= (int64_t)t.rs + t.deg) continue;
    const int32_t v = __ldg(g.col + e);
    const uint32_t bit = 1u << (v & 31);
    if (bm[(uint32_t)v >> 5] & bit) continue;
    const int32_t from = __ldg(g.row_ptr + v), to = __ldg(g.row_ptr + v + 1);
    if (atomicOr(bm + ((uint32_t)v >> 5), bit) & bit) continue;
    added++;
    Sum sum;
    sum.add(to - from);
    sum.to(sums, v / GROUP);
  }
  return added;
}

// LADIES: the terms of the entries of lists without tables into the sums of their groups, and the entries into the
// union (hubs have no octs).  A lane takes an oct and adds up what follows in one group; what the last entries of a lane's and the first of the
// next one's share is passed on, so that neighbouring entries of a long list cost one atomic and the lanes' atomics do not
// meet.
__device__ __forceinline__ void add_terms(const NdGraphView &g, const float *__restrict__ term, const Transit *ut, int ntr, int nh, int nu,
                                          const uint32_t *pre, uint32_t total, uint32_t *bm, double *sums, int group_bits) {
  const int lane = threadIdx.x & 31;
  int i = 0;
  for (uint32_t o0 = threadIdx.x - lane; o0 < total; o0 += blockDim.x) {
    const uint32_t o = o0 + lane;
    int first = -1, at = -1;    // the groups of the lane's first and last entries
    double sum = 0.0, sum_first = 0.0;
    double mult = 0.0;
    bool several = false;
    if (o < total) {
      if (i + 1 < nu && pre[i + 1] <= o) i = list_of_oct(pre, nu, o);
      const Transit t = ut[i < nh ? i : ntr - nu + i];
      const int64_t e = ((int64_t)((uint32_t)t.rs / OCT) + (int64_t)(o - pre[i])) * OCT;
      int32_t v[OCT], x[OCT];
      load8(g.col + e, v);
      load8(reinterpret_cast<const int32_t *>(term) + e, x);
      const uint32_t in = oct_mask(e, t);
      mult = (double)t.mult;
      {
        uint32_t word[OCT];
#pragma unroll
        for (int j = 0; j < OCT; j++) word[j] = (in >> j) & 1u ? bm[(uint32_t)v[j] >> 5] : ~0u;
#pragma unroll
        for (int j = 0; j < OCT; j++)
          if (!((word[j] >> (v[j] & 31)) & 1u)) atomicOr(bm + ((uint32_t)v[j] >> 5), 1u << (v[j] & 31));
      }
#pragma unroll
      for (int j = 0; j < OCT; j++) {
        if (!((in >> j) & 1u)) continue;
        const int group = v[j] >> group_bits;
        if (group != at) {
          if (at < 0) first = group;
          else if (!several) { sum_first = sum; several = true; }
          else atomicAdd(sums + at, sum * mult);
          at = group;
          sum = 0.0;
        }
        sum += (double)__int_as_float(x[j]);
      }
    }
    const int at_before = __shfl_up_sync(0xffffffffu, at, 1), i_before = __shfl_up_sync(0xffffffffu, i, 1);
    const bool joins = lane > 0 && first >= 0 && first == at_before && i == i_before;
    const uint32_t joined = __ballot_sync(0xffffffffu, joins);
    double before = 0.0;
    if (joined) {
      const uint32_t heads = __ballot_sync(0xffffffffu, several || !joins);
      const int head = 31 - __clz(heads & (0xffffffffu >> (31 - lane)));
      for (int step = 1; step < 32; step <<= 1) {
        const double t = __shfl_up_sync(0xffffffffu, sum, step);
        if (lane - step >= head) sum += t;
      }
      before = __shfl_up_sync(0xffffffffu, sum, 1);
    }
    if (several) atomicAdd(sums + first, (joins ? sum_first + before : sum_first) * mult);
    if (at >= 0 && !((joined >> 1 >> lane) & 1u)) atomicAdd(sums + at, sum * mult);
  }
}

// LADIES: the weights of the candidates of the groups that slot[] gives an accumulator for each vertex (NO_SLOT: none)
__device__ __forceinline__ void add_candidates(const NdGraphView &g, const float *__restrict__ term, const Transit *ut, int ntr, int nh, int nu,
                                               const uint32_t *pre, uint32_t total, const uint8_t *slot, double *acc, int group_bits) {
  int i = 0;
  for (uint32_t o = threadIdx.x; o < total; o += blockDim.x) {
    if (i + 1 < nu && pre[i + 1] <= o) i = list_of_oct(pre, nu, o);
    const Transit t = ut[i < nh ? i : ntr - nu + i];
    const int64_t e = ((int64_t)((uint32_t)t.rs / OCT) + (int64_t)(o - pre[i])) * OCT;
    int32_t v[OCT], x[OCT];
    load8(g.col + e, v);
    load8(reinterpret_cast<const int32_t *>(term) + e, x);
    const uint32_t in = oct_mask(e, t);
    uint32_t k[OCT];
#pragma unroll
    for (int j = 0; j < OCT; j++) k[j] = (in >> j) & 1u ? slot[v[j] >> group_bits] : NO_SLOT;
#pragma unroll
    for (int j = 0; j < OCT; j++)
      if (k[j] != NO_SLOT) atomicAdd(acc + ((size_t)k[j] << group_bits) + (v[j] & ((1 << group_bits) - 1)), (double)__int_as_float(x[j]) * (double)t.mult);
  }
}

// first group whose prefix reaches the target (rounding: the last one takes what is above all)
__device__ __forceinline__ int first_reaching(const double *cdf, int n, double target) {
  int lo = 0, hi = n - 1;
  while (lo < hi) {
    const int mid = lo + (hi - lo) / 2;
    if (cdf[mid] >= target) hi = mid; else lo = mid + 1;
  }
  return lo;
}

// LADIES: the draw's candidate in its group, by a warp: the first whose running sum reaches the target, or by rounding the
// last there is.  Blocks of 128 candidates, a lane holding four.  One with a weight of zero is none (its running sum is
// the one before it, which another order of the adds may leave a rounding below the target); a group that is drawn from
// has one that is not.
__device__ __forceinline__ void pick_in_group(const double *acc, int n, double before, double target, int &pick, double &wt) {
  const int lane = threadIdx.x & 31;
  double at_block = before, run = before;
  int first = 0;
  bool found = false;
  for (int q = 0; q < n && !found; q += 128) {
    const int r = q + lane * 4;
    const double *x = acc + r;
    const double mine = (x[0] + x[1]) + (x[2] + x[3]);
    double upto = mine;
    for (int o = 1; o < 32; o <<= 1) {
      const double t = __shfl_up_sync(0xffffffffu, upto, o);
      if (lane >= o) upto += t;
    }
    const uint32_t reach = __ballot_sync(0xffffffffu, mine > 0.0 && at_block + upto >= target), any = __ballot_sync(0xffffffffu, mine > 0.0);
    if (any) {
      found = reach != 0u;
      const int l = found ? __ffs(reach) - 1 : 31 - __clz(any);
      first = q + l * 4;
      run = at_block + __shfl_sync(0xffffffffu, upto - mine, l);
    }
    at_block += __shfl_sync(0xffffffffu, upto, 31);
  }
  bool hit = false;
#pragma unroll
  for (int k = 0; k < 4; k++) {
    const double t = acc[first + k];
    run += t;
    if (!hit && t > 0.0) {
      pick = first + k;
      wt = t;
      hit = run >= target;
    }
  }
}

// The sum of deg^2 over the vertices of a bitmap's word (32, low and high bytes of their degrees as in Degrees::codes), in products
// of low, low and high, and high bytes.  Byte b of code word j is vertex j + 8 b, so that a shift brings its bit to the top of the
// byte, which is then filled with it.
template <bool WIDE>
__device__ __forceinline__ uint32_t squares(uint32_t bits, const int32_t (&low)[8], const int32_t (&high)[8]) {
  uint32_t ll = 0, lh = 0, hh = 0;
#pragma unroll
  for (int j = 0; j < 8; j++) {
    uint32_t m;
    asm("prmt.b32 %0, %1, 0, 0xba98;" : "=r"(m) : "r"(bits << (7 - j)));
    const uint32_t l = (uint32_t)low[j] & m;
    ll = __dp4a(l, l, ll);
    if (WIDE) {
      lh = __dp4a(l, (uint32_t)high[j], lh);
      hh = __dp4a((uint32_t)high[j] & m, (uint32_t)high[j], hh);
    }
  }
  return WIDE ? ll + (lh << 9) + (hh << 16) : ll;
}

// FastGCN: the groups' weights, without the listed and the huge vertices' (their codes are zero); the candidates the thread has seen.  A warp takes FLIGHT times two
// groups at a time, a lane a word of the bitmap and its 32 bytes of codes.  WIDE: the codes have high bytes.
template <bool WIDE>
__device__ __forceinline__ uint32_t sum_groups(const uint32_t *bm, const Degrees &d, int words, int groups, uint2 *sums) {
  constexpr int AT_ONCE = WIDE ? FLIGHT / 2 : FLIGHT;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, warps = blockDim.x >> 5;
  const int32_t *__restrict__ low_bytes = reinterpret_cast<const int32_t *>(d.codes), *__restrict__ high_bytes = low_bytes + (int64_t)words * 8;
  uint32_t seen = 0;
  for (int w0 = warp * AT_ONCE * 32; w0 < words; w0 += warps * AT_ONCE * 32) {
    uint32_t bits[AT_ONCE], some = 0u;
    bool wide[AT_ONCE];
    int32_t lo[AT_ONCE][8], hi[AT_ONCE][8];
#pragma unroll
    for (int k = 0; k < AT_ONCE; k++) {
      const int w = w0 + 32 * k + lane, g = w / GROUP_WORDS;
      bits[k] = w < words ? bm[w] : 0u;
      wide[k] = WIDE && w < words && ((__ldg(d.wide + g / 32) >> (g & 31)) & 1u);
      some |= bits[k];
    }
    if (!__any_sync(0xffffffffu, some)) continue;   // (a first layer's thousand candidates leave most groups empty)
#pragma unroll
    for (int k = 0; k < AT_ONCE; k++) {
      const int w = w0 + 32 * k + lane;
#pragma unroll
      for (int j = 0; j < 8; j++) lo[k][j] = hi[k][j] = 0;
      if (bits[k]) load8(low_bytes + 8 * (int64_t)w, lo[k]);
      if (WIDE && wide[k] && bits[k]) load8(high_bytes + 8 * (int64_t)w, hi[k]);
    }
#pragma unroll
    for (int k = 0; k < AT_ONCE; k++) {
      seen += __popc(bits[k]);
      const uint32_t sum = squares<WIDE>(bits[k], lo[k], hi[k]);
      const uint32_t first = __reduce_add_sync(0xffffffffu, lane < GROUP_WORDS ? sum : 0u), second = __reduce_add_sync(0xffffffffu, sum) - first;
      const uint32_t low = lane == 0 ? first : second;
      if (lane < 2 && low) atomicAdd(&sums[w0 / GROUP_WORDS + 2 * k + lane].x, low);
    }
  }
  return seen;
}

// ... and over the listed vertices; neighbours on the list mostly share a group.  Their weights come as the two words that are added
// (from degrees, with a case for each size and 64-bit conversions for the large: 1024 batches on 2^20 vertices 0.631 ms, so 0.622;
// 100 of 100 on 600 K 84.4 and 82.6 us).
__device__ __forceinline__ void sum_listed(const uint32_t *bm, const Degrees &d, uint2 *sums) {
  for (int i0 = threadIdx.x * RUN; i0 < d.n_listed; i0 += blockDim.x * RUN) {
    const int4 four = __ldg(reinterpret_cast<const int4 *>(d.listed + i0));
    const int32_t v[RUN] = {four.x, four.y, four.z, four.w};
    int32_t weight[2 * RUN];
    load8(reinterpret_cast<const int32_t *>(d.weights + i0), weight);
    uint32_t word[RUN];
#pragma unroll
    for (int k = 0; k < RUN; k++) word[k] = bm[v[k] >> 5];
    int at = v[0] / GROUP;
    Sum sum;
#pragma unroll
    for (int k = 0; k < RUN; k++) {
      if (v[k] / GROUP != at) {
        sum.to(sums, at);
        at = v[k] / GROUP;
        sum = Sum();
      }
      const bool in = (word[k] >> (v[k] & 31)) & 1u;
      sum.low += in ? (uint32_t)weight[2 * k] : 0u;
      sum.high += in ? (uint32_t)weight[2 * k + 1] : 0u;
    }
    sum.to(sums, at);
  }
}

// The adjacency of a batch's lists, a row of bits each: bit j of row i, the layer's vertex j is in list i.  A list with a bitmap is
// asked by a bit test.  Of the others the warp, which has a row or a few side by side, first gets 32 entries, the last ones of as
// many parts of the list, from which a lane finds the part of its vertex without a read, and then bisects that: of 32, 64, 1024 and 8191
// entries (the longest list without a bitmap on 2^20 vertices) 1, 2, 6 and 9 reads that wait for one another instead of up to 6, 7, 11 and 13 (FastGCN 2^20 vertices 0.644 -> 0.636 ms, LADIES 0.689 -> 0.68).
// WORDS: the words of a row that are side by side, which share the list and its 32 entries (a word of any row each, with a division
// to find it, before: layers of 100 on 100 K, 700 batches, FastGCN 360 -> 323 us, LADIES 592 -> 549; of 64 on 70 K, 1024:
// 190 -> 180).  (Three places a step instead of one take half of the steps and more time; going through short lists once more with a
// filter of the layer's vertices too: a layer holds a hub many times, and graphs repeat edges.)  `apart`: the places between the
// hubs in ut and the other lists.
template <int ROWS, int WORDS>
__device__ __forceinline__ void probe_rows_as(const int32_t *__restrict__ col, const uint32_t *__restrict__ hub_bits, int words, int32_t V, const Transit *ut,
                                              int apart, int nh, int rows, const int32_t *layer, int L, uint32_t *out) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, warps = blockDim.x >> 5, row_words = (L + 31) / 32;
  for (int row0 = warp; row0 < rows; row0 += ROWS * warps) {
    int32_t rs[ROWS], deg[ROWS], slot[ROWS], last[ROWS];   // last: the last entry of the lane's part of the list
#pragma unroll
    for (int q = 0; q < ROWS; q++) {
      const int row = row0 + q * warps;
      const Transit t = ut[row < rows ? row < nh ? row : row + apart : row0 < nh ? row0 : row0 + apart];
      rs[q] = t.rs; deg[q] = t.deg; slot[q] = t.slot;
      const int part = (t.deg + 31) / 32;
      last[q] = 0x7fffffff;
      if (t.slot < 0 && lane * part < t.deg) last[q] = __ldg(col + t.rs + min((lane + 1) * part, t.deg) - 1);
    }
    for (int j0 = 0; j0 < L; j0 += 32 * WORDS) {
      int32_t v[WORDS], l[ROWS][WORDS], r[ROWS][WORDS];   // searched for in [l, r)
      uint32_t word[ROWS][WORDS];
      bool edge[ROWS][WORDS], more = false;
#pragma unroll
      for (int w = 0; w < WORDS; w++) {
        const int j = j0 + 32 * w + lane;
        v[w] = j < L ? layer[j] : V;
        if (v[w] < 0 || v[w] >= V) v[w] = -1;   // in no list
      }
#pragma unroll
      for (int q = 0; q < ROWS; q++)
#pragma unroll
        for (int w = 0; w < WORDS; w++) word[q][w] = slot[q] >= 0 && v[w] >= 0 ? __ldg(hub_bits + (size_t)slot[q] * words + ((uint32_t)v[w] >> 5)) : 0u;
#pragma unroll
      for (int q = 0; q < ROWS; q++) {
        const int part = (deg[q] + 31) / 32;
#pragma unroll
        for (int w = 0; w < WORDS; w++) {
          l[q][w] = r[q][w] = 0;
          if (slot[q] >= 0) {   // (the warp is of one mind: a list is the warp's)
            edge[q][w] = v[w] >= 0 && ((word[q][w] >> (v[w] & 31)) & 1u);
            continue;
          }
          int at = 0;           // the first part whose last entry is not below the vertex
#pragma unroll
          for (int step = 16; step > 0; step >>= 1)
            if (__shfl_sync(0xffffffffu, last[q], at + step - 1) < v[w]) at += step;
          const int32_t its = __shfl_sync(0xffffffffu, last[q], at);
          edge[q][w] = its == v[w];
          if (its > v[w] && v[w] >= 0) {
            l[q][w] = rs[q] + at * part;
            r[q][w] = min(rs[q] + deg[q], l[q][w] + part) - 1;   // (the last one has been compared with)
            more |= l[q][w] < r[q][w];
          }
        }
      }
      while (__any_sync(0xffffffffu, more)) {
        more = false;
        int32_t m[ROWS][WORDS], c[ROWS][WORDS];
#pragma unroll
        for (int q = 0; q < ROWS; q++)
#pragma unroll
          for (int w = 0; w < WORDS; w++) {
            m[q][w] = l[q][w] + (r[q][w] - l[q][w]) / 2;
            c[q][w] = l[q][w] < r[q][w] ? __ldg(col + m[q][w]) : 0;
          }
#pragma unroll
        for (int q = 0; q < ROWS; q++)
#pragma unroll
          for (int w = 0; w < WORDS; w++) {
            if (l[q][w] >= r[q][w]) continue;
            if (c[q][w] == v[w]) { edge[q][w] = true; l[q][w] = r[q][w]; }
            else if (c[q][w] < v[w]) l[q][w] = m[q][w] + 1;
            else r[q][w] = m[q][w];
            more |= l[q][w] < r[q][w];
          }
      }
#pragma unroll
      for (int q = 0; q < ROWS; q++)
#pragma unroll
        for (int w = 0; w < WORDS; w++) {
          const uint32_t answers = __ballot_sync(0xffffffffu, edge[q][w]);
          if (lane == 0 && row0 + q * warps < rows && j0 + 32 * w < L) out[(row0 + q * warps) * row_words + j0 / 32 + w] = answers;
        }
    }
  }
}
__device__ __forceinline__ void probe_rows(const int32_t *__restrict__ col, const uint32_t *__restrict__ hub_bits, int words, int32_t V, const Transit *ut,
                                           int apart, int nh, int rows, const int32_t *layer, int L, uint32_t *out) {
  // (as many warps as rows, or half as many: four rows a warp are 1 us a layer more, 148 batches of 8, 2 layers of 8, LADIES on 3000 vertices 36.3 ->
  // 34.4 us, on 500 K 61.7 -> 58.5, FastGCN of 16 on 125 K 37.1 -> 33.3; with four times as many rows as warps 76 -> 78)
  if (L <= 32 && rows <= 2 * (int)(blockDim.x >> 5)) probe_rows_as<1, 1>(col, hub_bits, words, V, ut, apart, nh, rows, layer, L, out);
  else if (L <= 32) probe_rows_as<4, 1>(col, hub_bits, words, V, ut, apart, nh, rows, layer, L, out);
  else if (L <= 64) probe_rows_as<2, 2>(col, hub_bits, words, V, ut, apart, nh, rows, layer, L, out);
  else probe_rows_as<1, 4>(col, hub_bits, words, V, ut, apart, nh, rows, layer, L, out);
}

// SUMS_FAR: LADIES' group sums are in the big part.
// 64 registers a thread.  Counters that only one thread needs are in shared memory: in registers they had FastGCN store 48 bytes a
// thread in local memory and load 32 (-Xptxas -v; now none), LADIES 36 and 24 (now 24 and 16, which scan_f64's eight elements take;
// two a thread take none, but leave more to add up).  1024 batches on 2^20 vertices FastGCN 718 -> 705 us, LADIES 1184 -> 1170 (edges 32 a vertex);
// on 70 K FastGCN 165 -> 163.
template <bool LADIES, bool SUMS_FAR>
__global__ void __launch_bounds__(1024, 1)
coll_bitmap_kernel(const __grid_constant__ Args a) {
  extern __shared__ __align__(16) unsigned char smem[];
  __shared__ long long sh_sample;
  __shared__ int sh_hubs, sh_rest;
  __shared__ uint32_t sh_drawn;   // layers with draws; thread 0's
  const Layout &lay = a.lay;
  CollParams cp = a.cp;
  unsigned char *big = lay.glob_bytes ? a.gscratch + (size_t)blockIdx.x * lay.glob_bytes : smem;
  uint32_t *bm = reinterpret_cast<uint32_t *>(big);
  double *gcdf = reinterpret_cast<double *>((LADIES && !SUMS_FAR ? smem : big) + lay.off_gcdf);
  uint2 *gsum = reinterpret_cast<uint2 *>(gcdf);                         // FastGCN: its weights while they are added up
  double *red = reinterpret_cast<double *>(smem + lay.off_red);   // 32 doubles, 32 words
  uint32_t *red_u = reinterpret_cast<uint32_t *>(red + 32);
  int32_t *sh_tr = reinterpret_cast<int32_t *>(smem + lay.off_tr);
  int32_t *sh_layer = reinterpret_cast<int32_t *>(smem + lay.off_layer);
  Transit *ut = reinterpret_cast<Transit *>(smem + lay.off_ut);
  int32_t *sh_mult = reinterpret_cast<int32_t *>(smem + lay.off_mult);   // how often a transit occurs (the first of a kind counts); then its place in ut, -1: not a vertex
  int32_t *sh_same = reinterpret_cast<int32_t *>(smem + lay.off_same);   // the first transit that is the same
  uint32_t *pre = reinterpret_cast<uint32_t *>(smem + lay.off_pre);
  double *sh_target = reinterpret_cast<double *>(smem + lay.off_draw);   // of a draw: the point of the CDF, its group, LADIES: the first draw of the group
  double *acc = reinterpret_cast<double *>(smem + lay.off_acc);          // LADIES from here on
  int32_t *sh_group = reinterpret_cast<int32_t *>(sh_target + cp.L), *sh_first = sh_group + cp.L;
  int32_t *sh_slot_group = sh_first + cp.L;
  uint32_t *sh_firsts = reinterpret_cast<uint32_t *>(sh_slot_group + cp.L);   // draws that are the first of their group, as bits
  uint8_t *slot = (LADIES && !SUMS_FAR ? smem : big) + lay.off_slot;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, warps = blockDim.x >> 5;
  unsigned long long ids_sum = 0, uniq_sum = 0;   // the thread's
  if (tid == 0) sh_drawn = 0;
  for (int64_t s = blockIdx.x; s < a.S;) {
    for (int step = 0; step < a.steps; step++) {
      cp.step = step;
      cp.ntr = step == 0 ? cp.B : cp.L;
      const int32_t *tr = transits_of(cp, a.initial, a.out, s);
      if (tid == 0) { sh_hubs = 0; sh_rest = 0; }
      int32_t rs0 = 0, end0 = 0, slot0 = -1;   // row and slot of the thread's first transit, asked for before the repeated ones are found
      for (int i = tid; i < cp.ntr; i += blockDim.x) {
        const int32_t t = step == 0 ? tr[i] : sh_layer[i];
        sh_tr[i] = t;
        sh_mult[i] = 1;
        if (i == tid && t >= 0 && t < cp.V) {
          rs0 = __ldg(a.g.row_ptr + t);
          end0 = __ldg(a.g.row_ptr + t + 1);
          slot0 = __ldg(a.hub_slot + t);
        }
      }
      __syncthreads();
      // ---- the batch's transits, each once: the hubs from the front of the list, the others from its end
      for (int j = tid; j < cp.ntr; j += blockDim.x) {
        const int32_t t = sh_tr[j];
        int first = j;
#pragma unroll 8
        for (int k = 0; k < j; k++) first = sh_tr[k] == t && k < first ? k : first;
        sh_same[j] = first;
        if (first != j) atomicAdd(sh_mult + first, 1);
      }
      __syncthreads();
      for (int i = tid; i < cp.ntr; i += blockDim.x) {
        const int32_t t = sh_tr[i];
        const bool valid = t >= 0 && t < cp.V, first = sh_same[i] == i;
        int place = -1;
        if (valid) {
          const int32_t rs = i == tid ? rs0 : __ldg(a.g.row_ptr + t), deg = (i == tid ? end0 : __ldg(a.g.row_ptr + t + 1)) - rs;
          ids_sum += (unsigned long long)deg;
          if (first) {
            const int32_t slot = i == tid ? slot0 : __ldg(a.hub_slot + t);
            place = slot >= 0 && (!LADIES || a.hub_sums) ? atomicAdd(&sh_hubs, 1) : cp.ntr - 1 - atomicAdd(&sh_rest, 1);
            ut[place] = Transit{rs, deg, sh_mult[i], slot};
          }
        }
        if (first) sh_mult[i] = place;
      }
      __syncthreads();
      const int nh = sh_hubs, nu = nh + sh_rest;
      // ---- the union: hubs' bitmaps, then the other lists
      // (32 bytes a load: with 16, eight of them in flight, FastGCN 0.661 ms and not 0.642, LADIES 0.725 and 0.71; lanes that know from
      // flags that their 16 bytes are zero, as half of them are, and do not ask for them: 0.744)
      for (int w8 = tid; w8 < lay.words / 8; w8 += blockDim.x) {
        uint32_t u[8] = {0u, 0u, 0u, 0u, 0u, 0u, 0u, 0u};
#pragma unroll 4
        for (int i = 0; i < nh; i++) {
          int32_t h[8];
          load8(reinterpret_cast<const int32_t *>(a.hub_bits + (size_t)ut[i].slot * lay.words) + 8 * w8, h);
#pragma unroll
          for (int k = 0; k < 8; k++) u[k] |= (uint32_t)h[k];
        }
        reinterpret_cast<uint4 *>(bm)[2 * w8] = make_uint4(u[0], u[1], u[2], u[3]);
        reinterpret_cast<uint4 *>(bm)[2 * w8 + 1] = make_uint4(u[4], u[5], u[6], u[7]);
      }
      const int groups = lay.groups;
      uint32_t seen = 0, octs = 0;
      if (!LADIES) {
        const Transit *rest = ut + cp.ntr - (nu - nh);
        for (int i = tid; i < nu - nh; i += blockDim.x) pre[i] = octs_of(rest[i].rs, rest[i].deg);
        for (int k = tid; k < groups; k += blockDim.x) gsum[k] = make_uint2(0u, 0u);
        __syncthreads();
        octs = scan_u32(pre, nu - nh, red_u);
        // Few entries beside the hubs': what they add is weighed one by one, else the whole union is gone through.
        const bool few = (int64_t)octs * OCT * FEW <= cp.V;
        if (!few) {
          add_lists<false>(a.g, rest, nu - nh, pre, octs, bm, gsum);
          __syncthreads();
        }
        if (!few || nh > 0) {
          seen += a.deg.wide ? sum_groups<true>(bm, a.deg, lay.words, groups, gsum) : sum_groups<false>(bm, a.deg, lay.words, groups, gsum);
          sum_listed(bm, a.deg, gsum);
        }
        if (few) {
          if (nh > 0) __syncthreads();
          seen += octs * OCT <= ENTRIES * blockDim.x ? add_entries(a.g, rest, nu - nh, pre, octs, bm, gsum) : add_lists<true>(a.g, rest, nu - nh, pre, octs, bm, gsum);
        }
      } else {
        // ---- the groups' weights and the rest of the union, then the number of candidates
        constexpr int AT_ONCE = 4;   // groups a thread has in flight (one at a time: LADIES 0.71 ms, four 0.69)
        for (int k = tid; k < groups; k += AT_ONCE * blockDim.x) {
          double sum[AT_ONCE] = {0.0, 0.0, 0.0, 0.0};
#pragma unroll 2
          for (int i = 0; i < nh; i++) {
            const double *from = a.hub_sums + (size_t)ut[i].slot * groups + k;
            const double mult = (double)ut[i].mult;
#pragma unroll
            for (int q = 0; q < AT_ONCE; q++) sum[q] += (k + q * (int)blockDim.x < groups ? __ldg(from + q * blockDim.x) : 0.0) * mult;
          }
#pragma unroll
          for (int q = 0; q < AT_ONCE; q++)
            if (k + q * (int)blockDim.x < groups) gcdf[k + q * blockDim.x] = sum[q];
        }
        for (int i = tid; i < nu; i += blockDim.x) {
          const Transit &t = ut[i < nh ? i : cp.ntr - nu + i];
          pre[i] = i < nh ? 0u : octs_of(t.rs, t.deg);
        }
        __syncthreads();
        octs = scan_u32(pre, nu, red_u);
        add_terms(a.g, a.term, ut, cp.ntr, nh, nu, pre, octs, bm, gcdf, lay.group_bits);
        __syncthreads();
        for (int w4 = tid; w4 < lay.words / 4; w4 += blockDim.x) {
          const uint4 u = reinterpret_cast<const uint4 *>(bm)[w4];
          seen += __popc(u.x) + __popc(u.y) + __popc(u.z) + __popc(u.w);
        }
      }
      uniq_sum += seen;
      const bool candidates = __syncthreads_or(seen != 0u);
      if (LADIES) {
        scan_groups(gcdf, groups, red, Doubles{gcdf});
      } else if (!a.n_huge) {
        scan_groups(gcdf, groups, red, Sums{gsum});
      } else {
        for (int k = tid; k < groups; k += blockDim.x) gcdf[k] = Sum::value(gsum[k]);   // (in its place)
        __syncthreads();
        {
          for (int i = tid; i < a.n_huge; i += blockDim.x) {
            const NdBigVertex v = a.huge[i];
            if ((bm[v.v >> 5] >> (v.v & 31)) & 1u) atomicAdd(gcdf + v.v / GROUP, (double)v.weight);
          }
          __syncthreads();
        }
        scan_groups(gcdf, groups, red, Doubles{gcdf});
      }
      const double total = groups > 0 ? gcdf[groups - 1] : 0.0;
      // ---- the layer's draws
      if (LADIES) {
        const bool any = candidates && total > 0.0;
        const int n = 1 << lay.group_bits;
        for (int j = tid; j < cp.L; j += blockDim.x) {
          if (!any) {
            sh_layer[j] = cp.V;
            a.out[s * cp.fs + (int64_t)cp.step * cp.L + j] = cp.V;
            a.prob[s * cp.fs + (int64_t)cp.step * cp.L + j] = 0.f;
            continue;
          }
          Rng rng(cp.seed, (uint32_t)(cp.first_sample + s), (uint32_t)cp.step, (uint32_t)j);
          const double target = (double)rng.uniform() * total;
          sh_target[j] = target;
          sh_group[j] = first_reaching(gcdf, groups, target);
        }
        if (any) {
          // the groups drawn from, each once, in the order of their first draws
          __syncthreads();
          for (int j0 = tid - lane; j0 < cp.L; j0 += blockDim.x) {
            const int j = j0 + lane, group = j < cp.L ? sh_group[j] : -1;
            int first = j;
#pragma unroll 8
            for (int k = 0; k < j0 + 32 && k < cp.L; k++) first = sh_group[k] == group && k < first ? k : first;
            if (j < cp.L) sh_first[j] = first;
            const uint32_t firsts = __ballot_sync(0xffffffffu, j < cp.L && first == j);
            if (lane == 0) sh_firsts[j0 / 32] = firsts;
          }
          __syncthreads();
          auto slot_of = [&](int j) {
            const int first = sh_first[j];
            int before = __popc(sh_firsts[first / 32] & ((1u << (first & 31)) - 1u));
            for (int k = 0; k < first / 32; k++) before += __popc(sh_firsts[k]);
            return before;
          };
          int drawn = 0;
          for (int k = 0; k < (cp.L + 31) / 32; k++) drawn += __popc(sh_firsts[k]);
          for (int s0 = 0; s0 < drawn; s0 += lay.slots) {
            const int here = min(drawn - s0, lay.slots);
            __syncthreads();
            for (int k = tid; k < here * n; k += blockDim.x) acc[k] = 0.0;
            for (int k = tid; k < groups; k += blockDim.x) slot[k] = (uint8_t)NO_SLOT;
            __syncthreads();
            for (int j = tid; j < cp.L; j += blockDim.x) {
              const int k = sh_first[j] == j ? slot_of(j) - s0 : -1;
              if (k >= 0 && k < here) {
                slot[sh_group[j]] = (uint8_t)k;
                sh_slot_group[k] = sh_group[j];
              }
            }
            __syncthreads();
            add_candidates(a.g, a.term, ut, cp.ntr, nh, nu, pre, octs, slot, acc, lay.group_bits);
            for (int q = tid / SUB; q < here * nh; q += blockDim.x / SUB) {   // hubs: a few lanes go to a group of one
              const int k = q / nh;
              const Transit t = ut[q - k * nh];
              const int32_t *at = a.hub_starts + (size_t)t.slot * (groups + 1) + sh_slot_group[k];
              const int32_t end = __ldg(at + 1);
              for (int32_t e = __ldg(at) + tid % SUB; e < end; e += SUB)
                atomicAdd(acc + ((size_t)k << lay.group_bits) + (__ldg(a.hub_ids + e) & (n - 1)), __ldg(a.hub_terms + e) * (double)t.mult);
            }
            __syncthreads();
            for (int j = warp; j < cp.L; j += warps) {
              const int k = slot_of(j) - s0, group = sh_group[j];
              if (k < 0 || k >= here) continue;
              int pick = 0;
              double wt = 0.0;
              pick_in_group(acc + (size_t)k * n, n, group > 0 ? gcdf[group - 1] : 0.0, sh_target[j], pick, wt);
              if (lane == 0) {
                sh_layer[j] = group * n + pick;
                a.out[s * cp.fs + (int64_t)cp.step * cp.L + j] = group * n + pick;
                a.prob[s * cp.fs + (int64_t)cp.step * cp.L + j] = (float)(wt / total);
              }
            }
          }
        }
      }
      if (!LADIES) {
        for (int j = tid; j < cp.L; j += blockDim.x) {
          Rng rng(cp.seed, (uint32_t)(cp.first_sample + s), (uint32_t)cp.step, (uint32_t)j);
          const double target = (double)rng.uniform() * total;
          sh_target[j] = target;
          sh_group[j] = first_reaching(gcdf, groups, target);
        }
        __syncthreads();
      }
      for (int j = LADIES ? cp.L : warp; j < cp.L; j += warps) {   // FastGCN: a warp each
        int32_t pick = cp.V;
        float pr = 0.f;
        if (candidates && total > 0.0) {
          const double target = sh_target[j];
          int lo = sh_group[j];
          // (a target of zero takes the first candidate of all, whatever its weight)
          if (target <= 0.0) while (!__any_sync(0xffffffffu, bm[lo * GROUP_WORDS + (lane & (GROUP_WORDS - 1))])) lo++;
          const double before = lo > 0 ? gcdf[lo - 1] : 0.0;
          // the first lane, of sixteen vertices each, in which a candidate reaches the target, then the candidate; by rounding
          // nobody reaches it: the last ones
          const int64_t r = (int64_t)lo * GROUP + lane * 16;
          const uint32_t mine = reinterpret_cast<const uint16_t *>(bm)[lo * 32 + lane];
          double sum = 0.0;
          if (mine) {
            int32_t at[17];
            if (r + 16 <= cp.V) {
#pragma unroll
              for (int q = 0; q < 4; q++) {
                const int4 f = __ldg(reinterpret_cast<const int4 *>(a.g.row_ptr + r) + q);
                at[4 * q] = f.x; at[4 * q + 1] = f.y; at[4 * q + 2] = f.z; at[4 * q + 3] = f.w;
              }
              at[16] = __ldg(a.g.row_ptr + r + 16);
            } else {
#pragma unroll
              for (int k = 0; k < 17; k++) at[k] = __ldg(a.g.row_ptr + (r + k < cp.V ? r + k : (int64_t)cp.V));
            }
            double part[4] = {0.0, 0.0, 0.0, 0.0};
#pragma unroll
            for (int k = 0; k < 16; k++) part[k & 3] += (mine >> k) & 1u ? (double)square(at[k + 1] - at[k]) : 0.0;
            sum = (part[0] + part[1]) + (part[2] + part[3]);
          }
          double run = sum;
          for (int o = 1; o < 32; o <<= 1) {
            const double t = __shfl_up_sync(0xffffffffu, run, o);
            if (lane >= o) run += t;
          }
          const uint32_t reach = __ballot_sync(0xffffffffu, mine && before + run >= target), any = __ballot_sync(0xffffffffu, mine != 0u);
          const int l = reach ? __ffs(reach) - 1 : 31 - __clz(any | 1u);
          const double at_lane = before + __shfl_sync(0xffffffffu, run - sum, l);
          const uint32_t its = __shfl_sync(0xffffffffu, mine, l);
          const int32_t v = lo * GROUP + l * 16 + (lane & 15);
          const bool there = (its >> (lane & 15)) & 1u;
          const float own = there ? square(__ldg(a.g.row_ptr + v + 1) - __ldg(a.g.row_ptr + v)) : 0.f;
          run = (double)own;
          for (int o = 1; o < 16; o <<= 1) {
            const double t = __shfl_up_sync(0xffffffffu, run, o, 16);
            if ((lane & 15) >= o) run += t;
          }
          const uint32_t hits = __ballot_sync(0xffffffffu, there && at_lane + run >= target) & 0xffffu;
          const int k = hits ? __ffs(hits) - 1 : 31 - __clz(its | 1u);
          const float wt = __shfl_sync(0xffffffffu, own, k);
          const int32_t rank = lo * GROUP + l * 16 + k;
          pick = (int32_t)rank;
          pr = (float)((double)wt / total);
        }
        if (lane == 0) {
          sh_layer[j] = pick;
          a.out[s * cp.fs + (int64_t)cp.step * cp.L + j] = pick;
          a.prob[s * cp.fs + (int64_t)cp.step * cp.L + j] = pr;
        }
      }
      if (tid == 0) { if (candidates && total > 0.0) sh_drawn++; }
      __syncthreads();
      uint32_t *adj = a.adj + (s * a.steps + cp.step) * (int64_t)adj_words(cp.stride);
      const int row_words = (cp.L + 31) / 32;
      if ((int64_t)nu * row_words > lay.words || (nu > PAIR_ROWS && cp.L <= (nu > 2 * warps ? PAIRS : PAIRS / 2))) {
        // A thread a pair: where the rows do not fit, and for layers so short that a warp to a row leaves most of its lanes idle (167 batches
        // of 250, layers of 1, 20 K vertices: rows, as below, FastGCN 47.5 us, LADIES 77, pairs 35.6 and 67; 1 M, FastGCN 174, 162; of 4 20 K LADIES 87, 80.6;
        // of 8 49.4, 43.2.  Of 4 or 8 lists rows are faster, 0.885 to 0.91 in units of either, of 30 lists from layers of 8 on).
        probe_pairs(a.g.col, a.hub_bits, lay.words, cp.stride, adj, [&](int e, PairList &list, int32_t &v) {
          const int i = e / cp.L, place = i < cp.ntr ? sh_mult[sh_same[i]] : -1;
          if (place < 0) return false;
          const Transit &t = ut[place];
          list = PairList{t.rs, t.deg, t.slot};
          v = sh_layer[e - i * cp.L];
          return v >= 0 && v < cp.V;
        });
      } else {
        // a row of answers for every list, where the union was; repeated transits have the same
        probe_rows(a.g.col, a.hub_bits, lay.words, cp.V, ut, cp.ntr - nu, nh, nu, sh_layer, cp.L, bm);
        __syncthreads();
        for (int w = tid; w < adj_words(cp.stride); w += blockDim.x) {
          uint32_t word = 0;
          for (int e = 32 * w, end = min(e + 32, cp.ntr * cp.L); e < end;) {
            const int i = e / cp.L, j = e - i * cp.L, n = min(cp.L - j, end - e), place = sh_mult[sh_same[i]];
            if (place >= 0) {
              const uint32_t *at = bm + (place < nh ? place : place - (cp.ntr - nu)) * row_words + j / 32;
              uint32_t bits = at[0] >> (j & 31);
              if ((j & 31) + n > 32) bits |= at[1] << (32 - (j & 31));
              word |= (n < 32 ? bits & ((1u << n) - 1u) : bits) << (e & 31);
            }
            e += n;
          }
          adj[w] = word;
        }
      }
      __syncthreads();
    }
    if (tid == 0) sh_sample = a.S > gridDim.x ? (long long)gridDim.x + (long long)atomicAdd(&a.acc[8], 1ull) : (long long)a.S;
    __syncthreads();
    s = sh_sample;
  }
  ids_sum = sum_of_all(ids_sum, red);
  uniq_sum = sum_of_all(uniq_sum, red);
  if (tid == 0) {
    atomicAdd(&a.acc[5], ids_sum);
    atomicAdd(&a.acc[6], uniq_sum);
    atomicAdd(&a.acc[0], (unsigned long long)sh_drawn * (unsigned long long)cp.L);
    __threadfence();
    if (atomicAdd(&a.acc[10], 1ull) == (unsigned long long)gridDim.x - 1ull) {   // the last CTA
      __threadfence();
      for (int i = 0; i < 8; i++) { a.stats[i] = i == 1 ? a.pairs : __ldcg(&a.acc[i]); a.acc[i] = 0ull; }
      a.acc[8] = a.acc[10] = 0ull;
    }
  }
}

// ---------------------------------------------------------------- arrays built once per graph

// The degrees of a lane's sixteen vertices, a warp per group: f(group, u, d).
template <class F>
__device__ __forceinline__ void for_groups(const int32_t *__restrict__ row_ptr, int32_t V, int64_t units, F f) {
  for (int64_t u = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; u < units; u += (int64_t)gridDim.x * blockDim.x) {   // (whole warps)
    int32_t d[16];
#pragma unroll
    for (int k = 0; k < 16; k++) {
      const int64_t v = 16 * u + k;
      d[k] = v < V ? row_ptr[v + 1] - row_ptr[v] : 0;
    }
    f(16 * u / GROUP, u, d);
  }
}

// Vertices with at least 256, BIG_DEGREE, HUGE_DEGREE neighbours; of a group, those of the first two kinds that are not of the third,
// in the low and the high half of a word.
__global__ void __launch_bounds__(256) deg_count_kernel(const int32_t *__restrict__ row_ptr, int32_t V, int64_t units, int32_t *__restrict__ count,
                                                        uint32_t *__restrict__ of_group) {
  int32_t all[3] = {0, 0, 0};
  for_groups(row_ptr, V, units, [&](int64_t group, int64_t, const int32_t (&d)[16]) {
    int32_t n[3] = {0, 0, 0};
#pragma unroll
    for (int k = 0; k < 16; k++) {
      n[0] += d[k] >= 256 ? 1 : 0; n[1] += d[k] >= BIG_DEGREE ? 1 : 0; n[2] += d[k] >= HUGE_DEGREE ? 1 : 0;
    }
    const uint32_t both = __reduce_add_sync(0xffffffffu, (uint32_t)(n[0] - n[2]) | (uint32_t)(n[1] - n[2]) << 16);
    if ((threadIdx.x & 31) == 0) of_group[group] = both;
    for (int k = 0; k < 3; k++) all[k] += n[k];
  });
  for (int k = 0; k < 3; k++) {
    all[k] = __reduce_add_sync(0xffffffffu, all[k]);
    if ((threadIdx.x & 31) == 0 && all[k]) atomicAdd(count + k, all[k]);
  }
}

// where a group's vertices begin on the list, in the place of its counts (the half `shift` says), by one CTA
constexpr int STARTS_THREADS = 1024;
__global__ void __launch_bounds__(STARTS_THREADS) deg_starts_kernel(uint32_t *__restrict__ of_group, int groups, int shift) {
  __shared__ uint32_t sums[STARTS_THREADS / 32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  uint32_t before = 0;
  for (int g0 = 0; g0 < groups; g0 += STARTS_THREADS) {
    const int g = g0 + (int)threadIdx.x;
    const uint32_t own = g < groups ? (of_group[g] >> shift) & 0xffffu : 0u;
    uint32_t upto = own;
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t t = __shfl_up_sync(0xffffffffu, upto, o);
      if (lane >= o) upto += t;
    }
    if (lane == 31) sums[warp] = upto;
    __syncthreads();
    uint32_t start = before + upto - own;
    for (int w = 0; w < STARTS_THREADS / 32; w++) {
      if (w < warp) start += sums[w];
      before += sums[w];
    }
    if (g < groups) of_group[g] = start;
    __syncthreads();
  }
}

// Codes, with `high` the high bytes and a flag per group, and the vertices with `least` neighbours and more: onto the list, or onto
// the one of the huge ones, in any order.
__global__ void __launch_bounds__(256)
deg_build_kernel(const int32_t *__restrict__ row_ptr, int32_t V, int64_t units, int32_t least, uint4 *__restrict__ low_bytes, uint4 *__restrict__ high_bytes,
                 uint32_t *__restrict__ wide, const uint32_t *__restrict__ starts, int32_t *__restrict__ listed, uint2 *__restrict__ weights,
                 NdBigVertex *__restrict__ huge, int32_t *__restrict__ n_huge) {
  const int lane = threadIdx.x & 31;
  for_groups(row_ptr, V, units, [&](int64_t group, int64_t u, const int32_t (&d)[16]) {
    uint32_t low[8] = {0u, 0u, 0u, 0u, 0u, 0u, 0u, 0u}, high[8] = {0u, 0u, 0u, 0u, 0u, 0u, 0u, 0u}, any = 0u;   // two bytes of each of eight words
    int mine = 0;
#pragma unroll
    for (int k = 0; k < 16; k++) {
      if (d[k] >= least) { mine += d[k] < HUGE_DEGREE ? 1 : 0; continue; }
      low[k & 7] |= (uint32_t)(d[k] & 255) << (8 * (k >> 3));
      high[k & 7] |= (uint32_t)(d[k] >> 8) << (8 * (k >> 3));
      any |= (uint32_t)(d[k] >> 8);
    }
    uint16_t *to = reinterpret_cast<uint16_t *>(low_bytes + (u & ~(int64_t)1)) + (u & 1);   // (see squares())
#pragma unroll
    for (int j = 0; j < 8; j++) to[2 * j] = (uint16_t)low[j];
    if (high_bytes) {
      to = reinterpret_cast<uint16_t *>(high_bytes + (u & ~(int64_t)1)) + (u & 1);
#pragma unroll
      for (int j = 0; j < 8; j++) to[2 * j] = (uint16_t)high[j];
      if (__any_sync(0xffffffffu, any != 0u) && lane == 0) atomicOr(wide + group / 32, 1u << (group & 31));
    }
    int upto = mine;
    for (int o = 1; o < 32; o <<= 1) {
      const int t = __shfl_up_sync(0xffffffffu, upto, o);
      if (lane >= o) upto += t;
    }
    uint32_t at = starts[group] + (uint32_t)(upto - mine);
#pragma unroll
    for (int k = 0; k < 16; k++) {
      if (d[k] < least) continue;
      if (d[k] < HUGE_DEGREE) {
        Sum sum;
        sum.add(d[k]);
        weights[at] = make_uint2(sum.low, sum.high);
        listed[at++] = (int32_t)(16 * u + k);
      } else {
        huge[atomicAdd(n_huge, 1)] = NdBigVertex{(int32_t)(16 * u + k), square(d[k])};
      }
    }
  });
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

__global__ void hub_degrees_kernel(const int32_t *__restrict__ row_ptr, const int32_t *__restrict__ hubs, int n, int32_t *__restrict__ deg) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) deg[i] = row_ptr[hubs[i] + 1] - row_ptr[hubs[i]];
}

// LADIES: a hub's neighbours, each once, and the sums of their terms, a CTA per hub (graphs repeat edges between hubs hundreds
// of times: what a warp has of one neighbour is added up first); hub i's go to ids[offs[i]] and on, terms zero before,
// their number to count[i].  *odd: a list does not ascend.
constexpr int HUB_THREADS = 1024;
__global__ void __launch_bounds__(HUB_THREADS) hub_unique_kernel(const int32_t *__restrict__ row_ptr, const int32_t *__restrict__ col,
                                                                 const float *__restrict__ term, const int32_t *__restrict__ hubs,
                                                                 const int32_t *__restrict__ offs, int32_t *__restrict__ ids, double *__restrict__ terms,
                                                                 int32_t *__restrict__ count, int *__restrict__ odd) {
  __shared__ int32_t heads_of[HUB_THREADS / 32];
  const int32_t v = hubs[blockIdx.x], rs = row_ptr[v], end = row_ptr[v + 1];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  int32_t at = offs[blockIdx.x];
  for (int32_t e0 = rs; e0 < end; e0 += HUB_THREADS) {
    const int32_t e = e0 + (int32_t)threadIdx.x;
    const int32_t c = e < end ? col[e] : 0, before = e < end && e > rs ? col[e - 1] : -1;
    if (e < end && before > c) *odd = 1;
    const uint32_t heads = __ballot_sync(0xffffffffu, e < end && c != before);
    __syncthreads();
    if (lane == 0) heads_of[warp] = __popc(heads);
    __syncthreads();
    int32_t to = at + __popc(heads & (0xffffffffu >> (31 - lane))) - 1;   // the neighbour's place: of the last head up to here
    for (int w = 0; w < HUB_THREADS / 32; w++) {
      if (w < warp) to += heads_of[w];
      at += heads_of[w];
    }
    double sum = e < end ? (double)term[e] : 0.0;
    const int head = 31 - __clz((heads | 1u) & (0xffffffffu >> (31 - lane)));
    for (int step = 1; step < 32; step <<= 1) {
      const double t = __shfl_up_sync(0xffffffffu, sum, step);
      if (lane - step >= head) sum += t;
    }
    if (e >= end) continue;
    if ((heads >> lane) & 1u) ids[to] = c;
    if (lane == 31 || e + 1 == end || ((heads >> (lane + 1)) & 1u)) atomicAdd(terms + to, sum);
  }
  if (threadIdx.x == 0) count[blockIdx.x] = at - offs[blockIdx.x];
}

// ... and its groups: where each begins there, and its sum
__global__ void __launch_bounds__(HUB_THREADS) hub_table_kernel(const int32_t *__restrict__ ids, const double *__restrict__ terms, const int32_t *__restrict__ offs,
                                                        const int32_t *__restrict__ count, int groups, int group_bits, double *__restrict__ sums,
                                                        int32_t *__restrict__ starts) {
  const int32_t first = offs[blockIdx.x], end = first + count[blockIdx.x];
  for (int k = threadIdx.x; k <= groups; k += blockDim.x) {
    int32_t lo = first, hi = end;   // first neighbour of group k or a later one
    while (lo < hi) {
      const int32_t mid = lo + ((hi - lo) >> 1);
      if ((int64_t)ids[mid] < (int64_t)k << group_bits) lo = mid + 1; else hi = mid;
    }
    starts[(size_t)blockIdx.x * (groups + 1) + k] = lo;
    double sum = 0.0;
    for (; k < groups && lo < end && ids[lo] >> group_bits == k; lo++) sum += terms[lo];
    if (k < groups) sums[(size_t)blockIdx.x * groups + k] = sum;
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
  g->n_hubs = n;
  g->hubs = hubs.release();
  g->hub_bits = bits.release();
  g->hub_slot = slot.release();
  return ND_OK;
}

// FastGCN: the packed degrees and the vertices whose degrees they do not hold, listed: from 256 on where those are few, else
// from BIG_DEGREE on, with a second byte per vertex.  In one allocation: low bytes, high bytes and flags, the listed ones' weights
// and ids, the huge ones.
int ensure_degrees(const nd_graph *g, int grid) {
  if (g->deg_codes) return ND_OK;
  const int64_t words = words_of(g->V), units = 2 * words;
  const int groups = (int)(words / GROUP_WORDS);
  NdDevMem<int32_t> counts;   // of n, of the huge ones that are listed, of the groups
  ND_TRY(counts.alloc((size_t)groups + 4));
  uint32_t *const of_group = reinterpret_cast<uint32_t *>(counts.p + 4);
  ND_CUDA(cudaMemset(counts.p, 0, sizeof(int32_t) * 4));
  deg_count_kernel<<<grid, 256>>>(g->row_ptr, g->V, units, counts.p, of_group);
  int32_t n[3] = {0, 0, 0};   // vertices with at least 256, BIG_DEGREE, HUGE_DEGREE neighbours
  ND_CUDA(cudaMemcpy(n, counts.p, sizeof(n), cudaMemcpyDeviceToHost));
  const bool few = (int64_t)n[0] * LISTED <= g->V;
  const size_t plane = 32 * (size_t)words, high = few ? 0 : plane, flags = few ? 0 : ((size_t)groups + 255) / 256 * 32;
  const size_t n_listed = (size_t)(n[few ? 0 : 1] - n[2]), room = (size_t)listed_room((int64_t)n_listed), lists = 12 * room;
  NdDevMem<unsigned char> deg;
  ND_TRY(deg.alloc(plane + high + flags + lists + sizeof(NdBigVertex) * ((size_t)n[2] + 1)));
  unsigned char *const at_high = deg.p + plane, *const at_flags = at_high + high, *const at_lists = at_flags + flags;
  uint2 *const weights = reinterpret_cast<uint2 *>(at_lists);
  NdBigVertex *const huge = reinterpret_cast<NdBigVertex *>(at_lists + lists);
  ND_CUDA(cudaMemset(at_flags, 0, flags + lists));
  deg_starts_kernel<<<1, STARTS_THREADS>>>(of_group, groups, few ? 0 : 16);
  deg_build_kernel<<<grid, 256>>>(g->row_ptr, g->V, units, few ? 256 : BIG_DEGREE, reinterpret_cast<uint4 *>(deg.p), few ? nullptr : reinterpret_cast<uint4 *>(at_high),
                                  reinterpret_cast<uint32_t *>(at_flags), of_group, reinterpret_cast<int32_t *>(weights + room), weights, huge, counts.p + 3);
  ND_CUDA(cudaDeviceSynchronize());
  g->n_huge = n[2];
  g->deg_wide = !few;
  g->huge = huge;
  g->listed = weights;
  g->n_listed = (int)n_listed;
  g->deg_codes = reinterpret_cast<uint4 *>(deg.release());
  return ND_OK;
}

// LADIES: the terms of the entries
int ensure_terms(const nd_graph *g, int grid) {
  if (g->term) return ND_OK;
  NdDevMem<float> term;
  NdDevMem<double> sum;
  ND_TRY(term.alloc((size_t)g->E + OCT));
  ND_TRY(sum.alloc((size_t)g->V));
  ND_CUDA(cudaMemset(sum.p, 0, sizeof(double) * (size_t)g->V));
  rowsum_build_kernel<<<grid, BUILD_THREADS>>>(g->row_ptr, g->w, g->V, g->E, sum.p);
  term_build_kernel<<<grid, BUILD_THREADS>>>(g->row_ptr, g->w, sum.p, g->V, g->E, term.p);
  ND_CUDA(cudaDeviceSynchronize());
  g->term = term.release();
  return ND_OK;
}

// LADIES: the hubs' neighbours and groups of 2^bits vertices, unless they would take more than HUB_TABLES bytes, the
// device has no room for them or a list does not ascend
constexpr size_t HUB_TABLES = (size_t)256 << 20;
int ensure_hub_tables(const nd_graph *g, const Layout &lay) {
  NdHubTable &t = g->hub_tables[lay.group_bits - LADIES_GROUP_BITS];
  const size_t n = (size_t)g->n_hubs, groups = (size_t)lay.groups;
  if (t.sums || n == 0 || g->hub_lists == 0 || n * (12 * groups + 4) > HUB_TABLES) return ND_OK;
  if (g->hub_lists < 0) {
    NdDevMem<int32_t> ids, d_offs;
    if (d_offs.alloc(2 * n) != ND_OK) return ND_OK;
    std::vector<int32_t> offs(n);
    hub_degrees_kernel<<<(unsigned)(n + 255) / 256, 256>>>(g->row_ptr, g->hubs, (int)n, d_offs.p);
    ND_CUDA(cudaMemcpy(offs.data(), d_offs.p, sizeof(int32_t) * n, cudaMemcpyDeviceToHost));
    int64_t all = 0;
    for (size_t i = 0; i < n; i++) {
      const int32_t deg = offs[i];
      offs[i] = (int32_t)all;
      all += deg;
    }
    if (12 * (size_t)all > HUB_TABLES) { g->hub_lists = 0; return ND_OK; }
    NdDevMem<double> terms;
    NdDevMem<int> flag;
    int odd = 0;
    if (ids.alloc((size_t)all) != ND_OK || terms.alloc((size_t)all) != ND_OK || flag.alloc(1) != ND_OK) return ND_OK;
    ND_CUDA(cudaMemset(flag.p, 0, sizeof(int)));
    ND_CUDA(cudaMemcpy(d_offs.p, offs.data(), sizeof(int32_t) * n, cudaMemcpyHostToDevice));
    ND_CUDA(cudaMemset(terms.p, 0, sizeof(double) * (size_t)all));
    hub_unique_kernel<<<(unsigned)n, HUB_THREADS>>>(g->row_ptr, g->col, g->term, g->hubs, d_offs.p, ids.p, terms.p, d_offs.p + n, flag.p);
    ND_CUDA(cudaMemcpy(&odd, flag.p, sizeof(int), cudaMemcpyDeviceToHost));
    g->hub_lists = odd ? 0 : 1;
    if (odd) return ND_OK;
    g->hub_ids = ids.release();
    g->hub_terms = terms.release();
    g->hub_offs = d_offs.release();
  }
  NdDevMem<double> sums;
  NdDevMem<int32_t> starts;
  if (sums.alloc(n * groups) != ND_OK || starts.alloc(n * (groups + 1)) != ND_OK) return ND_OK;
  hub_table_kernel<<<(unsigned)n, HUB_THREADS>>>(g->hub_ids, g->hub_terms, g->hub_offs, g->hub_offs + n, lay.groups, lay.group_bits, sums.p, starts.p);
  ND_CUDA(cudaDeviceSynchronize());
  t.starts = starts.release();
  t.sums = sums.release();
  return ND_OK;
}

// What a graph's first sampler builds goes to the graph when all of it is there: a build that runs out of memory
// leaves nothing behind.
int ensure_layers(const nd_graph *g, int sms, bool ladies, const Layout &lay, NdHubTable *table) {
  std::lock_guard<std::mutex> lock(g_layers_mutex);
  const int grid = sms * 16;
  ND_TRY(ensure_hubs(g, grid));
  if (!ladies) return ensure_degrees(g, grid);
  ND_TRY(ensure_terms(g, grid));
  if (lay.sums_far) return ND_OK;
  ND_TRY(ensure_hub_tables(g, lay));
  *table = g->hub_tables[lay.group_bits - LADIES_GROUP_BITS];
  return ND_OK;
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

// Two CTAs of 512 threads per SM where both layouts fit, or one, three or four by the number of samples, else one of 1024.
Plan plan_of(const nd_sampler *s) {
  const int32_t V = s->g->V;
  const int L = s->p.fanout[0], B = s->p.batch, ntr = B > L ? B : L;
  const bool ladies = s->p.app == ND_APP_LADIES_IS;
  const uint32_t optin = (uint32_t)(s->dev.smem_optin - ND_SMEM_STATIC), half = optin / 2u - 1024u;
  Layout l;
  l.words = words_of(V);
  l.sums_far = false;
  // The layout with `group_bits`, the big part in shared memory or not; its bytes without accumulators of their own.
  auto place = [&](int group_bits, bool global) {
    l.group_bits = group_bits;
    l.groups = ladies ? (int)(((int64_t)l.words * 32 + (1 << group_bits) - 1) >> group_bits) : l.words / GROUP_WORDS;
    const uint32_t sums = 8u * (uint32_t)l.groups, slots = ladies ? ((uint32_t)l.groups + 15u) & ~15u : 0u;
    uint32_t big = 4u * (uint32_t)l.words;       // a multiple of 64
    if (!ladies || l.sums_far) { l.off_gcdf = big; l.off_slot = big + sums; big += sums + slots; }
    big = (big + 255u) & ~255u;
    l.glob_bytes = global ? big : 0u;
    uint32_t off = global ? 0u : big;
    if (ladies && !l.sums_far) { l.off_gcdf = off; l.off_slot = off + sums; off += sums + slots; }
    l.off_draw = off; off += ((ladies ? 20u * (uint32_t)L + 4u * (((uint32_t)L + 31u) / 32u) : 12u * (uint32_t)L) + 7u) & ~7u;
    l.off_red = off; off += 8u * 32u + 4u * 32u;
    l.off_ut = off; off += (uint32_t)sizeof(Transit) * (uint32_t)ntr;
    l.off_tr = off; off += 4u * (uint32_t)ntr;
    l.off_layer = off; off += 4u * (uint32_t)L;
    l.off_mult = off; off += 4u * (uint32_t)ntr;
    l.off_same = off; off += 4u * (uint32_t)ntr;
    l.off_pre = off; off += 4u * (uint32_t)ntr;
    return (off + 15u) & ~15u;
  };
  // Accumulators of a group that is drawn from: in the bitmap's place where that holds SLOTS of them or one for every
  // draw, else in what is left of `room`.
  constexpr uint32_t SLOTS = 16;
  auto fits = [&](int bits, bool global, uint32_t room) {
    const uint32_t used = place(bits, global), slot = 8u << bits, wanted = std::min<uint32_t>((uint32_t)L, NO_SLOT);
    l.bytes = used;
    if (!ladies) return used <= room;
    const uint32_t over = global ? 0u : 4u * (uint32_t)l.words / slot, beside = used < room ? (room - used) / slot : 0u;
    l.off_acc = over >= std::min(wanted, std::max(SLOTS, beside)) ? 0u : used;
    l.slots = (int)std::min(wanted, l.off_acc ? beside : over);
    if (l.off_acc) l.bytes += slot * (uint32_t)l.slots;
    return used <= room && (uint32_t)l.slots >= std::min(wanted, SLOTS);
  };
  bool two = false, placed = false;
  const int most = ladies ? LADIES_GROUP_BITS + 2 : LADIES_GROUP_BITS;
  for (int bits = LADIES_GROUP_BITS; bits <= most && !placed && !s->coll_global; bits++) placed = two = fits(bits, false, half);
  for (int bits = LADIES_GROUP_BITS; bits <= most && !placed && !s->coll_global; bits++) placed = fits(bits, false, optin);
  for (int bits = LADIES_GROUP_BITS; !placed && bits <= LADIES_GROUP_BITS + 5; bits++) placed = fits(bits, true, optin);
  if (!placed) {   // (LADIES from about 12 M vertices on, or thousands of transits)
    l.sums_far = true;
    fits(LADIES_GROUP_BITS, true, optin);
    if (ladies && l.slots < 1) { l.slots = 1; l.bytes += 8u << LADIES_GROUP_BITS; }
  }
  // Where two fit an SM: with no more samples than SMs a sample has one for itself (140 batches of 64, 2 layers of 64: 70 K
  // vertices, FastGCN 67 -> 63 us, LADIES 95 -> 82; 330 K: 91 -> 82, 120 -> 94), except where batch, layer and graph are so small that
  // 32 warps wait for one another longer than 16 work (up to 131 K vertices, 20 and 148 batches; FastGCN on 3, 30, 70, 125 K vertices of 8: 33 -> 27,
  // 34.7 -> 30.9, 38.7 -> 35.3, 38.3 -> 36.9, of 40 40.2 -> 35.1, 41.3 -> 39.2, 47.0 -> 45.5, 47.1 -> 47.3, but of 64 43.4, 45.2, 52 and 54 us instead of
  // 43.3, 43.4, 51.5 and 51.6; LADIES on 3, 30, 70, 125 K of 8 41 -> 37, 39.2 -> 37.1, 41.9 -> 40.7, 41.6 -> 39.1, on 5 to 30 K of 12 39.2 .. 46.3 -> 37.5 .. 45,
  // of 16 on 3 and 8 K 44.7 -> 41.5, 43.2 -> 41.4, but 53.5 -> 55.6 on 70 K).  With many samples, three or four smaller CTAs
  // overlap better while the graph is small (70 K, 1024 batches, two, three, four an SM: 215, 206, 187; 322, 314, 290; 500 K,
  // 640: 412, 448 with three), unless their last round would be nearly empty (700: 166, 155, 158) or, LADIES, there were not
  // accumulators for half of the draws at a time (batches and layers of 100, 100 K, 520: 475, 533), for three quarters on larger
  // graphs (200 K, 64, 1024: 348, 356; but layers of 32 on 250 K 289, 251).  The groups stay: tables of
  // the graph go by them.
  Plan p;
  p.per_sm = two ? 2 : 1;
  const bool small = V <= SHARED_V / 2;
  if (two && s->S <= s->dev.sms) {
    if (!small || ntr > (!ladies ? 40 : V <= SHARED_V / 32 ? 16 : 12)) p.per_sm = 1;
  }
  if (two && p.per_sm == 1) {
    fits(l.group_bits, false, optin);
  } else if (two && s->S > 2 * s->dev.sms && V <= SHARED_V) {
    for (int k = 4; k > 2 && p.per_sm == 2; k--) {
      const int64_t round = (int64_t)k * s->dev.sms, rounds = (s->S + round - 1) / round;
      if (10 * s->S < 7 * rounds * round) continue;
      const Layout with_two = l;
      if (fits(l.group_bits, false, optin / (uint32_t)k - 1024u) && (!ladies || 4 * l.slots >= (small ? 2 * L : 3 * L))) p.per_sm = k;
      else l = with_two;
    }
  }
  p.threads = 1024 / p.per_sm / 32 * 32;
  p.lay = l;
  return p;
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
  ND_CUDA(ladies ? (p.lay.sums_far ? nd_smem_most(coll_bitmap_kernel<true, true>, s->dev) : nd_smem_most(coll_bitmap_kernel<true, false>, s->dev))
                 : nd_smem_most(coll_bitmap_kernel<false, false>, s->dev));
  s->coll_grid = (int)std::min<int64_t>(s->S > 0 ? s->S : 1, (int64_t)s->dev.sms * p.per_sm);
  if (p.lay.glob_bytes) ND_CUDA(nd_malloc(&s->d_bm, (size_t)p.lay.glob_bytes * (size_t)s->coll_grid));
  ND_CUDA(nd_malloc(&s->d_rows_acc, 16 * sizeof(unsigned long long)));
  ND_CUDA(cudaMemset(s->d_rows_acc, 0, 16 * sizeof(unsigned long long)));
  return ensure_layers(s->g, s->dev.sms, ladies, p.lay, &s->hub_table);   // last: what is optional there leaves the sampler its room
}

int nd_coll_bitmap_launch(nd_sampler *s, const CollParams &cp, unsigned long long pairs) {
  const bool ladies = s->p.app == ND_APP_LADIES_IS;
  const Plan p = plan_of(s);
  const nd_graph *g = s->g;
  const Args a{nd_view(g), cp, s->p.steps, s->S, p.lay, s->d_bm, s->d_initial, s->d_out, s->d_adj, s->d_prob,
               Degrees{g->deg_codes, g->deg_wide ? reinterpret_cast<const uint32_t *>(g->deg_codes + 4 * (int64_t)p.lay.words) : nullptr,
                       reinterpret_cast<const int32_t *>(g->listed + listed_room(g->n_listed)), g->listed, g->n_listed},
               g->huge, g->n_huge, g->term, g->hub_slot, g->hub_bits, s->hub_table.sums, s->hub_table.starts, g->hub_ids, g->hub_terms, s->d_rows_acc, s->d_stats, pairs};
  if (ladies && p.lay.sums_far) coll_bitmap_kernel<true, true><<<s->coll_grid, p.threads, p.lay.bytes, s->stream>>>(a);
  else if (ladies) coll_bitmap_kernel<true, false><<<s->coll_grid, p.threads, p.lay.bytes, s->stream>>>(a);
  else coll_bitmap_kernel<false, false><<<s->coll_grid, p.threads, p.lay.bytes, s->stream>>>(a);
  nd_count_launches(1);
  ND_CUDA(cudaGetLastError());
  return ND_OK;
}
