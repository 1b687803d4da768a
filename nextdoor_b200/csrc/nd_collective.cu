// Collective-neighbourhood layer sampling: one sample is a batch of transits and every layer draws
// stepSize vertices for the whole batch.
//
// ND_APP_FASTGCN_REF / ND_APP_LADIES_REF follow the reference's shipped next()
// (src/apps/fastgcn/fastgcnSampling.cu:23-47, src/apps/ladies/ladiessampling.cu:23-47): a vertex
// drawn uniformly from the whole graph, then one probe of the list (src/csr.hpp:343-359) per
// transit to fill the layer's adjacency (row, col) entries.
//
// ND_APP_FASTGCN_IS / ND_APP_LADIES_IS are the importance samplers the reference does not have:
// the candidates of a layer are the sorted unique union of the transits' neighbours, weighted by
// degree^2 (FastGCN) or by the sum over transits of (w(i,v)/rowsum_i)^2 (LADIES); the weights are
// prefix-summed in candidate order and every slot inverts the CDF at u * total.  Pipeline per
// layer, the collective-neighbourhood construction of the reference made useful
// (collectiveNeighbrsSize / collectiveNeighborhood, src/nextdoor.cu:1206-1283, whose copied
// neighbourhood the shipped next() never reads):
//   sizes   : sum of degrees per sample                        (one warp per sample)
//   gather  : every neighbour id, its sample and its LADIES term into one flat array
//   sort    : by id, then stably by sample, with the in-house radix sort (3 words per element)
//   weigh   : the first element of every (sample, id) run carries the candidate's weight, the
//             rest carry 0, so no compaction pass is needed and the CDF is unchanged
//   sample  : one CTA per sample: block-wide prefix sum built from warp-shuffle scans, the
//             stepSize inverse-CDF draws, and the adjacency probes
// The per-layer sizes come back to the host once (the reference does the same before its
// per-step cudaMalloc, src/nextdoor.cu:2413-2429) so that samples can be processed in chunks that
// fit the candidate buffers whatever the hub sizes are.
#include <algorithm>
#include <cstdlib>
#include <vector>

#include "nd_collective.cuh"

namespace {

using ndrng::Rng;
constexpr int CTHREADS = 256;

// ---------------------------------------------------------------- reference semantics: uniform over V
//
// A layer's vertices are drawn from the whole graph, whatever the transits are, so all layers of a pass are drawn
// first and all their (transit, layer) pairs are probed together: the transits' lists are flattened over the
// CTA, every entry asks a filter of the layer's ids in shared memory, and the few that pass look for the id.
// A list longer than PROBE_RATIO times the layer is bisected for every id instead.  (One bisection per
// (transit, slot) pair, 205 M of them for 10,000 samples of 5 x 64 x 64 on 57 K vertices: 1.04 ms, the kernel now 0.20.)
// The flags of the edges that were found are the adjacency as it is kept: a bit per entry (the two arrays of the
// reference's form, 1.6 GB for those samples, took 0.1 ms of 0.54).
constexpr int FILTER_WORDS = 256;   // 8192 bits per layer
constexpr int PROBE_RATIO = 8;

struct RefLayout {
  int per_pass;                                                        // layers drawn and probed together
  uint32_t off_red, off_rec, off_ids, off_pre, off_filter, off_flags;           // bytes
  uint32_t bytes;
  int flag_words;                                                      // per transit
  int words;                                                           // of a layer's adjacency
  uint32_t inv_L, inv_words;                                           // 2^32 / L, rounded up: x / L is the high half of x * inv_L below 2^16
};

static RefLayout ref_layout(int steps, int B, int L) {
  RefLayout r;
  const int ntr = B > L ? B : L;
  r.flag_words = (L + 31) / 32;
  r.words = adj_words(ntr * L);
  r.inv_L = (uint32_t)((((uint64_t)1 << 32) + (uint32_t)L - 1) / (uint32_t)L);
  r.inv_words = (uint32_t)((((uint64_t)1 << 32) + (uint32_t)r.words - 1) / (uint32_t)r.words);
  // (a layer's filter is a kilobyte: no more than 24 of them fit, and the sums below stay in 32 bits)
  for (r.per_pass = std::min(steps, 24);; r.per_pass--) {
    const uint32_t k = (uint32_t)r.per_pass, nt = k * (uint32_t)ntr;
    uint32_t off = 0;
    r.off_red = off; off += 8u * (CTHREADS / 32);
    r.off_rec = off; off += 8u * (nt + 1u);
    r.off_ids = off; off += 4u * (k + 1u) * (uint32_t)L;   // the layer before the pass too: its transits
    r.off_pre = off; off += 4u * (nt + 1u);
    r.off_filter = off; off += 4u * k * FILTER_WORDS;
    r.off_flags = off; off += 4u * nt * (uint32_t)r.flag_words;
    r.bytes = off;
    if (r.per_pass == 1 || off <= 24u * 1024u) return r;
  }
}

// x / n of a kernel's RefLayout, inv = 2^32 / n rounded up (0: n is 1): x below 2^16, or 0 is the only quotient
__device__ __forceinline__ int quotient(int x, uint32_t inv) { return inv ? (int)__umulhi((uint32_t)x, inv) : x; }

// the last i of [lo, hi] with pre[i] <= f, lo if there is none
__device__ __forceinline__ int last_at_most(const uint32_t *pre, int lo, int hi, uint32_t f) {
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (pre[mid] <= f) lo = mid; else hi = mid - 1;
  }
  return lo;
}

__global__ void __launch_bounds__(CTHREADS)
coll_ref_kernel(NdGraphView g, CollParams cp, const __grid_constant__ ndrng::RoundKeys keys, RefLayout lay, int steps, int64_t S, const int32_t *__restrict__ initial, int32_t *__restrict__ out,
                uint32_t *__restrict__ adj, unsigned long long *__restrict__ stats) {
  extern __shared__ __align__(16) unsigned char sm[];
  uint2 *red = reinterpret_cast<uint2 *>(sm + lay.off_red);
  // The transits whose lists are streamed, those without neighbours left out: pre[l] entries come before the list, and entry f
  // of all of them is rec[l].x + f of the graph's, of transit rec[l].y & 0xffff and layer rec[l].y >> 16.  Those whose lists are
  // bisected come from the arrays' ends: rec (row start, as above), pre the length.
  int2 *rec = reinterpret_cast<int2 *>(sm + lay.off_rec);
  int32_t *ids = reinterpret_cast<int32_t *>(sm + lay.off_ids);
  __shared__ int heavy;
  uint32_t *pre = reinterpret_cast<uint32_t *>(sm + lay.off_pre);
  uint32_t *filter = reinterpret_cast<uint32_t *>(sm + lay.off_filter), *flags = reinterpret_cast<uint32_t *>(sm + lay.off_flags);
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, L = cp.L;
  for (int64_t s = blockIdx.x; s < S; s += gridDim.x) {
    for (int k0 = 0; k0 < steps; k0 += lay.per_pass) {
      const int kn = min(lay.per_pass, steps - k0);
      // transits of the pass, back to back: the batch (first layer of the sample), then the layers before
      const int n0 = k0 == 0 ? cp.B : L, nt = n0 + (kn - 1) * L;
      __syncthreads();   // the pass before has written its entries
      if (tid == 0) heavy = 0;
      if (k0 > 0) for (int j = tid; j < L; j += CTHREADS) ids[j] = ids[lay.per_pass * L + j];
      for (int i = tid; i < kn * FILTER_WORDS; i += CTHREADS) filter[i] = 0u;
      for (int i = tid; i < nt * lay.flag_words; i += CTHREADS) flags[i] = 0u;
      __syncthreads();
      for (int q = tid; q < kn * L; q += CTHREADS) {
        const int k = quotient(q, lay.inv_L), j = q - k * L;
        uint32_t o[4];
        ndrng::philox4x32_10((uint32_t)(cp.first_sample + s), (uint32_t)(k0 + k), (uint32_t)j, 0u, keys, o);
        const int32_t id = ndrng::rand_int_from(ndrng::u32_to_uniform(o[0]), cp.V);
        ids[L + q] = id;
        out[s * cp.fs + (int64_t)k0 * L + q] = id;
        atomicOr(filter + k * FILTER_WORDS + (((uint32_t)id >> 5) & (FILTER_WORDS - 1)), 1u << (id & 31));
      }
      __syncthreads();
      // rows of the transits; their places in the list, and how many entries come before them
      uint32_t carry = 0;
      int n_live = 0;
      for (int i0 = 0; i0 < nt; i0 += CTHREADS) {
        const int i = i0 + tid;
        uint32_t n = 0;
        int2 r = make_int2(0, i);
        if (i < nt) {
          const int32_t t = i < n0 ? (k0 == 0 ? initial[s * cp.B + i] : ids[i]) : ids[L + (i - n0)];
          int32_t deg = 0;
          if (t >= 0 && t < cp.V) { r.x = __ldg(g.row_ptr + t); deg = __ldg(g.row_ptr + t + 1) - r.x; }
          if (i >= n0) r.y |= (1 + quotient(i - n0, lay.inv_L)) << 16;
          if (deg > PROBE_RATIO * L) {   // bisected
            const int h = nt - atomicAdd(&heavy, 1);
            rec[h] = r;
            pre[h] = (uint32_t)deg;
          } else {
            n = (uint32_t)deg;
          }
        }
        uint32_t inc = n;
        for (int o = 1; o < 32; o <<= 1) {
          const uint32_t t = __shfl_up_sync(0xffffffffu, inc, o);
          if (lane >= o) inc += t;
        }
        const uint32_t live = __ballot_sync(0xffffffffu, n > 0);
        if (lane == 31) red[warp] = make_uint2(inc, __popc(live));
        __syncthreads();
        uint32_t before = carry + inc - n;
        int at = n_live + __popc(live & ((1u << lane) - 1u));
        for (int w = 0; w < CTHREADS / 32; w++) {
          const uint2 x = red[w];
          if (w < warp) { before += x.x; at += (int)x.y; }
          carry += x.x;
          n_live += (int)x.y;
        }
        if (n > 0) {
          pre[at] = before;
          rec[at] = make_int2(r.x - (int32_t)before, r.y);
        }
        if (i0 + CTHREADS >= nt && tid == 0) pre[n_live] = carry;
        __syncthreads();
      }
      // the entries of the short lists: a warp takes a run of them, a lane four neighbouring ones at a time
      constexpr int LOADS = 4;
      const uint32_t chunks = (carry + 32 * LOADS - 1) / (32 * LOADS), each = (chunks + CTHREADS / 32 - 1) / (CTHREADS / 32) * (32 * LOADS);
      const uint32_t run_end = min(((uint32_t)warp + 1u) * each, carry);
      int from = 0;   // list of the chunk's first entry: the last with pre <= c0
      if (warp * each < run_end) from = last_at_most(pre, 0, n_live - 1, warp * each);
      for (uint32_t c0 = warp * each; c0 < run_end; c0 += 32 * LOADS) {
        int32_t v[LOADS], who[LOADS];
        const uint32_t c1 = min(c0 + 32 * LOADS, run_end) - 1;
        int to;   // list of its last entry: seldom 32 further on
        const uint32_t within = __ballot_sync(0xffffffffu, from + 1 + lane < n_live && pre[from + 1 + lane] <= c1);
        if (within == 0xffffffffu) to = last_at_most(pre, from + 32, n_live - 1, c1);
        else to = from + __popc(within);
        const uint32_t f0 = c0 + (uint32_t)(LOADS * lane);
        int lo = f0 <= c1 ? last_at_most(pre, from, to, f0) : to;
        int2 r = rec[lo];
        uint32_t end = pre[lo + 1];
#pragma unroll
        for (int j = 0; j < LOADS; j++) {
          const uint32_t f = f0 + j;
          v[j] = -1;
          if (f <= c1) {
            if (f == end) { lo++; r = rec[lo]; end = pre[lo + 1]; }
            v[j] = __ldg(g.col + (r.x + (int32_t)f));
          }
          who[j] = r.y;
        }
        from = to;
#pragma unroll
        for (int j = 0; j < LOADS; j++) {
          const bool may = v[j] >= 0 && ((filter[(who[j] >> 16) * FILTER_WORDS + (((uint32_t)v[j] >> 5) & (FILTER_WORDS - 1))] >> (v[j] & 31)) & 1u);
          for (uint32_t left = __ballot_sync(0xffffffffu, may); left; left &= left - 1) {   // the warp looks for each of them
            const int src = __ffs(left) - 1;
            const int32_t id = __shfl_sync(0xffffffffu, v[j], src);
            const int w_i = __shfl_sync(0xffffffffu, who[j], src), i = w_i & 0xffff, layer = w_i >> 16;
            for (int w = 0; w < lay.flag_words; w++) {
              const int q = 32 * w + lane;
              const uint32_t found = __ballot_sync(0xffffffffu, q < L && ids[L + layer * L + q] == id);
              if (found && lane == 0) atomicOr(flags + i * lay.flag_words + w, found);
            }
          }
        }
      }
      const int nheavy = heavy;
      for (int q = tid; q < nheavy * L; q += CTHREADS) {
        const int h = nt - q / L, j = q % L;
        const int2 r = rec[h];
        const int i = r.y & 0xffff;
        const int32_t id = ids[L + (r.y >> 16) * L + j], end = r.x + (int32_t)pre[h];
        int32_t lo = r.x, hi = end;
        while (lo < hi) {
          const int32_t m = lo + ((hi - lo) >> 1);
          if (__ldg(g.col + m) < id) lo = m + 1; else hi = m;
        }
        if (lo < end && __ldg(g.col + lo) == id) atomicOr(flags + i * lay.flag_words + (j >> 5), 1u << (j & 31));
      }
      __syncthreads();
      // the layers' adjacency: the flags are the bits where a transit's are whole words
      const int words = lay.words;
      for (int q = tid; q < kn * words; q += CTHREADS) {
        const int k = kn == 1 ? 0 : quotient(q, lay.inv_words), w = q - k * words;
        const int first = k == 0 ? 0 : n0 + (k - 1) * L, n = k == 0 ? n0 : L;
        uint32_t bits = 0u;
        if ((L & 31) == 0) {
          if (w < n * lay.flag_words) bits = flags[first * lay.flag_words + w];
        } else {
          for (int e = 32 * w; e < 32 * w + 32;) {   // up to the end of the word, of the transit's flags' word or of its row
            const int i = e / L, j = e - i * L, len = min(min(32 * w + 32 - e, L - j), 32 - (j & 31));
            if (i >= n) break;
            bits |= (flags[(first + i) * lay.flag_words + (j >> 5)] >> (j & 31) & (0xffffffffu >> (32 - len))) << (e & 31);
            e += len;
          }
        }
        __stcs(adj + (s * steps + k0) * (int64_t)words + q, bits);
      }
    }
  }
  if (blockIdx.x == 0 && tid < 8)
    stats[tid] = tid == 0 ? (unsigned long long)S * steps * cp.L
                 : tid == 1 ? (unsigned long long)S * (cp.B + (unsigned long long)(steps - 1) * cp.L) : 0ull;
}

// ---------------------------------------------------------------- importance sampling pipeline

// one warp per sample: sum of the transits' degrees
__global__ void __launch_bounds__(CTHREADS)
coll_sizes_kernel(NdGraphView g, CollParams cp, int64_t S, const int32_t *__restrict__ initial,
                  const int32_t *__restrict__ out, int32_t *__restrict__ sizes) {
  const int64_t s = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5;
  if (s >= S) return;
  const int lane = threadIdx.x & 31;
  const int32_t *tr = transits_of(cp, initial, out, s);
  int64_t sum = 0;
  for (int i = lane; i < cp.ntr; i += 32) {
    const int32_t t = tr[i];
    if (t >= 0 && t < cp.V) sum += __ldg(g.row_ptr + t + 1) - __ldg(g.row_ptr + t);
  }
  for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
  if (lane == 0) sizes[s] = (int32_t)(sum > 0x7fffffff ? 0x7fffffff : sum);
}

// one CTA per sample of the chunk: copy every transit's neighbours into the flat candidate arrays.
// Warp w takes transits w, w+8, ...; the start of transit i inside the sample's region is the
// running sum of the degrees before it (shared-memory scan by thread 0: ntr <= 1024).
__global__ void __launch_bounds__(CTHREADS)
coll_gather_kernel(NdGraphView g, CollParams cp, int64_t s0, int64_t s1, const int32_t *__restrict__ initial,
                   const int32_t *__restrict__ out, const int64_t *__restrict__ offs, uint32_t *__restrict__ c_id,
                   uint32_t *__restrict__ c_seg, uint32_t *__restrict__ c_w) {
  __shared__ int32_t sh_start[1025];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  for (int64_t s = s0 + blockIdx.x; s < s1; s += gridDim.x) {
    const int32_t *tr = transits_of(cp, initial, out, s);
    if (threadIdx.x == 0) {
      int32_t run = 0;
      for (int i = 0; i < cp.ntr; i++) {
        sh_start[i] = run;
        const int32_t t = tr[i];
        if (t >= 0 && t < cp.V) run += __ldg(g.row_ptr + t + 1) - __ldg(g.row_ptr + t);
      }
      sh_start[cp.ntr] = run;
    }
    __syncthreads();
    const int64_t base = offs[s] - offs[s0];
    for (int i = warp; i < cp.ntr; i += CTHREADS / 32) {
      const int32_t t = tr[i];
      if (t < 0 || t >= cp.V) continue;
      const int32_t rs = __ldg(g.row_ptr + t), deg = __ldg(g.row_ptr + t + 1) - rs;
      float rowsum = 0.f;
      if (cp.app == ND_APP_LADIES_IS) {  // fp64 partial sums: the order of the adds does not matter
        double part = 0.0;
        for (int e = lane; e < deg; e += 32) part += (double)__ldg(g.w + rs + e);
        for (int o = 16; o > 0; o >>= 1) part += __shfl_xor_sync(0xffffffffu, part, o);
        rowsum = (float)part;
      }
      const int64_t dst = base + sh_start[i];
      for (int e = lane; e < deg; e += 32) {
        c_id[dst + e] = (uint32_t)__ldg(g.col + rs + e);
        c_seg[dst + e] = (uint32_t)(s - s0);
        float term = 0.f;
        if (cp.app == ND_APP_LADIES_IS) {
          const float r = __fdiv_rn(__ldg(g.w + rs + e), rowsum);
          term = __fmul_rn(r, r);
        }
        c_w[dst + e] = __float_as_uint(term);
      }
    }
    __syncthreads();
  }
}

// thread per element: the first element of a (sample, id) run gets the candidate's weight (for
// LADIES the run's terms summed in their stable order), the others get 0
__global__ void __launch_bounds__(CTHREADS)
coll_weigh_kernel(NdGraphView g, int app, int64_t n, const uint32_t *__restrict__ c_id, const uint32_t *__restrict__ c_seg,
                  const uint32_t *__restrict__ c_w, float *__restrict__ wt, unsigned long long *__restrict__ stats) {
  uint32_t heads = 0;
  for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < n; e += (int64_t)gridDim.x * blockDim.x) {
    const uint32_t id = c_id[e], seg = c_seg[e];
    const bool head = e == 0 || c_id[e - 1] != id || c_seg[e - 1] != seg;
    float w = 0.f;
    if (head) {
      heads++;
      if (app == ND_APP_FASTGCN_IS) {
        const float d = __int2float_rn(__ldg(g.row_ptr + id + 1) - __ldg(g.row_ptr + id));
        w = __fmul_rn(d, d);
      } else {
        for (int64_t k = e; k < n && c_id[k] == id && c_seg[k] == seg; k++) w = __fadd_rn(w, __uint_as_float(c_w[k]));
      }
    }
    wt[e] = w;
  }
  for (int o = 16; o > 0; o >>= 1) heads += __shfl_xor_sync(0xffffffffu, heads, o);
  if ((threadIdx.x & 31) == 0 && heads) atomicAdd(&stats[6], (unsigned long long)heads);
}

// one CTA per sample: inclusive prefix sum of the weights over the sample's region (warp-shuffle
// scans + carry), then the layer's draws and the adjacency entries
__global__ void __launch_bounds__(CTHREADS)
coll_sample_kernel(NdGraphView g, CollParams cp, int steps, int64_t s0, int64_t s1, const int32_t *__restrict__ initial,
                   int32_t *out, const int64_t *__restrict__ offs, const uint32_t *__restrict__ c_id,
                   const float *__restrict__ wt, double *__restrict__ cdf, uint32_t *__restrict__ adj,
                   float *__restrict__ prob, unsigned long long *__restrict__ stats) {
  __shared__ double warp_tot[CTHREADS / 32];
  __shared__ double carry_sh;
  __shared__ int32_t sh_tr[1024];
  __shared__ int32_t sh_layer[1024];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  for (int64_t s = s0 + blockIdx.x; s < s1; s += gridDim.x) {
    const int64_t base = offs[s] - offs[s0];
    const int64_t n = offs[s + 1] - offs[s];
    // fp64 accumulation of the fp32 weights (sums agree with any other order of addition to
    // ~1e-16; FastGCN's integer weights sum exactly)
    if (threadIdx.x == 0) carry_sh = 0.0;
    __syncthreads();
    for (int64_t c0 = 0; c0 < n; c0 += CTHREADS) {
      const int64_t i = c0 + threadIdx.x;
      double inc = i < n ? (double)wt[base + i] : 0.0;
      for (int o = 1; o < 32; o <<= 1) {
        const double t = __shfl_up_sync(0xffffffffu, inc, o);
        if (lane >= o) inc += t;
      }
      if (lane == 31) warp_tot[warp] = inc;
      __syncthreads();
      double woff = carry_sh;
      for (int w = 0; w < warp; w++) woff += warp_tot[w];
      if (i < n) cdf[base + i] = woff + inc;
      __syncthreads();
      if (threadIdx.x == CTHREADS - 1) carry_sh = woff + inc;
      __syncthreads();
    }
    const double total = carry_sh;
    const int32_t *tr = transits_of(cp, initial, out, s);
    for (int i = threadIdx.x; i < cp.ntr; i += CTHREADS) sh_tr[i] = tr[i];
    uint32_t valid = 0;
    for (int j = threadIdx.x; j < cp.L; j += CTHREADS) {
      int32_t pick = cp.V;
      float pr = 0.f;
      if (n > 0 && total > 0.0) {
        Rng rng(cp.seed, (uint32_t)(cp.first_sample + s), (uint32_t)cp.step, (uint32_t)j);
        const double target = (double)rng.uniform() * total;
        int64_t lo = 0, hi = n - 1;  // first index whose cdf reaches the target
        while (lo < hi) {
          const int64_t mid = lo + (hi - lo) / 2;
          if (cdf[base + mid] >= target) hi = mid; else lo = mid + 1;
        }
        // (by rounding one behind a candidate, of weight zero or the candidate's id again)
        while (lo > 0 && !(wt[base + lo] > 0.f)) lo--;
        pick = (int32_t)c_id[base + lo];
        pr = (float)((double)wt[base + lo] / total);
        valid++;
      }
      sh_layer[j] = pick;
      out[s * cp.fs + (int64_t)cp.step * cp.L + j] = pick;
      prob[s * cp.fs + (int64_t)cp.step * cp.L + j] = pr;
    }
    __syncthreads();
    emit_adjacency(g, cp, sh_tr, sh_layer, adj + (s * steps + cp.step) * (int64_t)adj_words(cp.stride));
    for (int o = 16; o > 0; o >>= 1) valid += __shfl_xor_sync(0xffffffffu, valid, o);
    if (lane == 0 && valid) atomicAdd(&stats[0], (unsigned long long)valid);
    __syncthreads();
  }
}

// clears the counters; stats[1] (live pairs) is known up front for these apps
__global__ void coll_reset_kernel(unsigned long long *stats, unsigned long long pairs) {
  if (threadIdx.x < 8) stats[threadIdx.x] = threadIdx.x == 1 ? pairs : 0ull;
}

}  // namespace

// candidate buffers: three 32-bit words per element (id, sample, LADIES term), double-buffered for
// the sort, plus weight and CDF
static int ensure_cand(nd_sampler *s, int64_t need) {
  if (need <= s->cand_cap) return ND_OK;
  int64_t cap = std::max<int64_t>(need, (int64_t)1 << 22);
  cudaFree(s->d_cand); cudaFree(s->d_cand_w);
  nd_radix_scratch_free(&s->radix);
  s->d_cand = nullptr; s->d_cand_w = nullptr; s->cand_cap = 0;
  ND_CUDA(nd_malloc(&s->d_cand, sizeof(uint32_t) * 6 * (size_t)cap));
  ND_CUDA(nd_malloc(&s->d_cand_w, (sizeof(float) + sizeof(double)) * (size_t)cap));  // cdf (fp64) first, then weights
  ND_TRY(nd_radix_scratch_alloc(&s->radix, 32, cap));
  s->cand_cap = cap;
  return ND_OK;
}

int nd_collective_alloc(nd_sampler *s) {
  const nd_app_params &p = s->p;
  const int L = p.fanout[0], B = p.batch;
  const size_t S1 = (size_t)(s->S > 0 ? s->S : 1);
  ND_CUDA(nd_malloc(&s->d_adj, sizeof(uint32_t) * S1 * p.steps * (size_t)adj_words((B > L ? B : L) * L)));
  ND_CUDA(nd_malloc(&s->d_prob, sizeof(float) * S1 * s->fs));
  ND_CUDA(cudaMemset(s->d_prob, 0, sizeof(float) * S1 * s->fs));
  ND_CUDA(nd_malloc(&s->d_len, sizeof(int32_t) * (S1 + 1)));        // per-sample sizes of the layer
  ND_CUDA(nd_malloc(&s->d_tmp, sizeof(int64_t) * (S1 + 1)));        // per-sample region offsets
  ND_CUDA(nd_malloc(&s->d_nlive, sizeof(int32_t) * 4));
  ND_CUDA(nd_smem_most(coll_ref_kernel, s->dev));
  if (p.app == ND_APP_FASTGCN_IS || p.app == ND_APP_LADIES_IS) {
    // the union is built as a bitmap with a bit per vertex (nd_coll_bitmap.cu); ND_COLLECTIVE_SORT=1 selects
    // the sort pipeline instead (kept for the tests, which compare the two)
    const char *force = getenv("ND_COLLECTIVE_SORT");
    if (B <= 1024 && L <= 1024 && !(force && force[0] == '1')) {
      s->coll_bitmap = true;
      ND_TRY(nd_coll_bitmap_alloc(s));
    } else {
      ND_TRY(ensure_cand(s, (int64_t)1 << 22));
    }
  }
  return ND_OK;
}

const char *nd_collective_kernel_name(const nd_sampler *s) {
  if (!s->coll_bitmap) return "coll_sizes/gather/weigh/sample kernels + radix sort";
  return s->d_bm ? "coll_bitmap_kernel (bitmap in global scratch)" : "coll_bitmap_kernel (bitmap in shared memory)";
}

int nd_collective_sample(nd_sampler *s, int mode) {
  (void)mode;  // the reference runs next() of collective apps through sampleParallelKernel in every mode (src/nextdoor.cu:2900-2916)
  const nd_app_params &p = s->p;
  const int64_t S = s->S;
  cudaStream_t st = s->stream;
  NdGraphView gv = nd_view(s->g);
  CollParams cp;
  cp.seed = p.seed; cp.first_sample = s->first; cp.V = s->g->V; cp.fs = s->fs; cp.L = p.fanout[0]; cp.B = p.batch;
  cp.stride = (cp.B > cp.L ? cp.B : cp.L) * cp.L; cp.step = 0; cp.ntr = cp.B; cp.app = p.app;
  const bool ref_app = p.app == ND_APP_FASTGCN_REF || p.app == ND_APP_LADIES_REF;
  const unsigned long long pairs = (unsigned long long)(S * (cp.B + (int64_t)(p.steps - 1) * cp.L));
  if (s->coll_bitmap && !ref_app) {  // one launch, nothing comes back to the host: asynchronous like the walk and k-hop jobs
    nd_phase_begin(s, ND_PHASE_NEXT);
    const int rc = nd_coll_bitmap_launch(s, cp, pairs);
    nd_phase_end(s);
    return rc;
  }
  if (ref_app) {
    const RefLayout lay = ref_layout(p.steps, cp.B, cp.L);
    const int per_sm = lay.bytes <= 24u * 1024u ? 8 : 1;
    nd_phase_begin(s, ND_PHASE_NEXT);
    coll_ref_kernel<<<(int)std::min<int64_t>(S, (int64_t)s->dev.sms * per_sm), CTHREADS, lay.bytes, st>>>(
        gv, cp, ndrng::RoundKeys(p.seed), lay, p.steps, S, s->d_initial, s->d_out, s->d_adj, s->d_stats);
    nd_phase_end(s);
    nd_count_launches(1);
    ND_CUDA(cudaGetLastError());
    return ND_OK;
  }
  coll_reset_kernel<<<1, 32, 0, st>>>(s->d_stats, 0ull);
  nd_count_launches(1);
  std::vector<int32_t> sizes((size_t)S);
  std::vector<int64_t> offs((size_t)S + 1);
  int64_t union_ids = 0;
  int64_t *d_offs = (int64_t *)s->d_tmp;
  for (int step = 0; step < p.steps; step++) {
    cp.step = step;
    cp.ntr = step == 0 ? cp.B : cp.L;
    nd_phase_begin(s, ND_PHASE_COLLECT);
    coll_sizes_kernel<<<(int)((S * 32 + CTHREADS - 1) / CTHREADS), CTHREADS, 0, st>>>(gv, cp, S, s->d_initial, s->d_out, s->d_len);
    nd_count_launches(1);
    ND_CUDA(cudaMemcpyAsync(sizes.data(), s->d_len, sizeof(int32_t) * (size_t)S, cudaMemcpyDeviceToHost, st));
    ND_CUDA(cudaStreamSynchronize(st));
    offs[0] = 0;
    int64_t biggest = 0;
    for (int64_t i = 0; i < S; i++) { offs[i + 1] = offs[i] + sizes[i]; biggest = std::max<int64_t>(biggest, sizes[i]); }
    union_ids += offs[S];
    ND_REQUIRE(biggest < ((int64_t)1 << 30), ND_ERR_RANGE, "a collective neighbourhood of %lld ids does not fit", (long long)biggest);
    ND_TRY(ensure_cand(s, biggest));
    ND_CUDA(cudaMemcpyAsync(d_offs, offs.data(), sizeof(int64_t) * ((size_t)S + 1), cudaMemcpyHostToDevice, st));
    nd_phase_end(s);
    const int64_t cap = s->cand_cap;
    uint32_t *c_a[3] = {(uint32_t *)s->d_cand, (uint32_t *)s->d_cand + cap, (uint32_t *)s->d_cand + 2 * cap};
    uint32_t *c_b[3] = {(uint32_t *)s->d_cand + 3 * cap, (uint32_t *)s->d_cand + 4 * cap, (uint32_t *)s->d_cand + 5 * cap};
    double *cdf = (double *)s->d_cand_w;
    float *wt = (float *)(cdf + cap);
    int64_t s0 = 0;
    while (s0 < S) {  // chunk of samples whose neighbourhoods fit the buffers together
      int64_t s1 = s0 + 1;
      while (s1 < S && offs[s1 + 1] - offs[s0] <= cap) s1++;
      const int64_t n = offs[s1] - offs[s0];
      const int cgrid = (int)std::min<int64_t>(s1 - s0, (int64_t)s->dev.sms * 8);
      if (n > 0) {
        nd_phase_begin(s, ND_PHASE_COLLECT);
        const int32_t n32 = (int32_t)n;
        ND_CUDA(cudaMemcpyAsync(s->d_nlive, &n32, sizeof(int32_t), cudaMemcpyHostToDevice, st));
        coll_gather_kernel<<<cgrid, CTHREADS, 0, st>>>(gv, cp, s0, s1, s->d_initial, s->d_out, d_offs, c_a[0], c_a[1], c_a[2]);
        nd_count_launches(1);
        uint32_t *cur[3] = {c_a[0], c_a[1], c_a[2]}, *oth[3] = {c_b[0], c_b[1], c_b[2]};
        const int key_word[2] = {0, 1};
        const int key_bits[2] = {nd_bit_length((uint32_t)(cp.V > 1 ? cp.V - 1 : 1)), nd_bit_length((uint32_t)(s1 - s0 > 1 ? s1 - s0 - 1 : 1))};
        for (int k = 0; k < 2; k++) {
          NdSortArrays arr;
          arr.nwords = 3;
          for (int w = 0; w < 3; w++) { arr.a[w] = cur[w]; arr.b[w] = oth[w]; }
          NdRadixPlan pl = nd_radix_plan(key_bits[k], cap);
          bool in_b = false;
          ND_TRY(nd_radix_sort(s->dev, st, &s->radix, pl, arr, key_word[k], s->d_nlive, nullptr, false, 0u, false, &in_b));
          if (in_b) for (int w = 0; w < 3; w++) std::swap(cur[w], oth[w]);
        }
        const int wgrid = (int)std::min<int64_t>((n + CTHREADS - 1) / CTHREADS, (int64_t)s->dev.sms * 16);
        coll_weigh_kernel<<<wgrid, CTHREADS, 0, st>>>(gv, p.app, n, cur[0], cur[1], cur[2], wt, s->d_stats);
        nd_count_launches(1);
        nd_phase_end(s);
        nd_phase_begin(s, ND_PHASE_NEXT);
        coll_sample_kernel<<<cgrid, CTHREADS, 0, st>>>(gv, cp, p.steps, s0, s1, s->d_initial, s->d_out, d_offs, cur[0], wt, cdf,
                                                     s->d_adj, s->d_prob, s->d_stats);
        nd_count_launches(1);
        nd_phase_end(s);
        // the next chunk reuses the buffers and the host copy of its size
        ND_CUDA(cudaStreamSynchronize(st));
      } else {
        coll_sample_kernel<<<cgrid, CTHREADS, 0, st>>>(gv, cp, p.steps, s0, s1, s->d_initial, s->d_out, d_offs, c_a[0], wt, cdf,
                                                     s->d_adj, s->d_prob, s->d_stats);
        nd_count_launches(1);
      }
      s0 = s1;
    }
  }
  const unsigned long long h[2] = {(unsigned long long)(S * (cp.B + (int64_t)(p.steps - 1) * cp.L)), (unsigned long long)union_ids};
  ND_CUDA(cudaMemcpyAsync(s->d_stats + 1, &h[0], sizeof(unsigned long long), cudaMemcpyHostToDevice, st));
  ND_CUDA(cudaMemcpyAsync(s->d_stats + 5, &h[1], sizeof(unsigned long long), cudaMemcpyHostToDevice, st));
  ND_CUDA(cudaStreamSynchronize(st));
  ND_CUDA(cudaGetLastError());
  return ND_OK;
}
