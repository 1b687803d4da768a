// k-hop neighbourhoods, a warp per sample: the whole job in one launch (sample-parallel and load-balanced modes).
//
// A sample's row -- all its hops -- lives in shared memory from its seed to its last hop, so nothing of it
// passes through device memory between hops: no transit maps, no sort, no second pass for the distinct ids.
// Per hop: the parents that are vertices with neighbours are listed, every slot of theirs draws an entry of
// the adjacency array (phase one: draws and, without replacement, Floyd's resolution), then all entries are
// gathered with GATHERS loads in flight per lane (phase two).  ND_APP_KHOP draws as KHopApp::next
// (src/apps/khop/khop.cu:10-23); ND_APP_KHOP_DISTINCT without replacement, every hop sorted and made unique at
// the end (src/distinct.cuh:1-111).  A warp writes its row at the end.
// What bounds it: with replacement, gathers of 4 bytes from the adjacency array at the rate of random DRAM
// reads (262,144 seeds, 25 x 10, 2^21 vertices: 0.89 ms transit-parallel -> 0.36); without (1.15 -> 0.475 ms), the
// instructions: 341 M of a warp, 0.29 ms at one per cycle and scheduler, and of the 18 cycles from one to the next 4.8 are
// spent waiting for the next instruction to be fetched, 2.5 for memory and 2.4 for shared memory (DRAM 35 %); without its sorts
// 0.375 ms, without the resolution of picks taken twice 0.43, without the gathers 0.46, with a cheap hash for the draws 0.46; a mini-batch
// of 1024 (74 -> 12 us with the seeds' copy), the hand-over from the copy to the kernel and the caller (100 seeds take 12.4 us too), and of the
// kernel's 10 us one warp's instructions: a thousand for a sample, 15.7 cycles each, 4.6 of them for memory and 4.6 at barriers, 10 % of the warps in use.
#include "nd_common.cuh"
#include "nd_khop_rows.cuh"
#include "nd_philox.cuh"
#include "nd_warp_sort.cuh"

namespace {

constexpr int GATHERS = 8;
constexpr int SORT_MAX = 256;        // longest hop a warp sorts in registers
constexpr int ROW_MAX = 4096;        // longest row that is kept in shared memory

// CTAs of 256 per SM (registers): measured 4 / 5 / 6 / 8 on 262,144 seeds, 25 x 10, 2^21 vertices: with
// replacement 0.403 / 0.396 / 0.428 / 0.526 ms, without 0.548 / 0.524 / 0.500 / 0.498
constexpr int CTAS = 5;
constexpr int CTAS_DISTINCT = 6;
__host__ __device__ constexpr int khop_ctas(bool distinct) { return distinct ? CTAS_DISTINCT : CTAS; }

struct KhopRows {
  ndrng::RoundKeys keys;
  int64_t first_sample, S;
  int32_t V, fs;
  int steps;
  int fan[ND_MAX_STEPS_FANOUT];
  int parents_max;
  int batch;                               // samples handed to a warp at a time
  const int2 *__restrict__ vrow;
  const int32_t *__restrict__ col;
  const int32_t *__restrict__ initial;
  int32_t *__restrict__ out;
  int32_t *__restrict__ hop_counts;        // [S][steps], distinct only
  unsigned long long *__restrict__ acc;    // counters of the running job: [0] edges, [1] pairs, [8] samples handed out, [10] CTAs that are done; zero between jobs
  unsigned long long *__restrict__ stats;  // published by the last CTA
};

// the first draw of a slot, below n
__device__ __forceinline__ int32_t draw(const KhopRows &a, uint32_t sample, int hop, int slot, int32_t n) {
  uint32_t o[4];
  ndrng::philox4x32_10(sample, (uint32_t)hop, (uint32_t)slot, 0u, a.keys, o);
  return ndrng::rand_int_from(ndrng::u32_to_uniform(o[0]), n);
}

// Entry (relative to the list) that slot j of a parent with `deg` > f neighbours picks without replacement:
// Floyd, slot after slot -- a candidate that is taken is replaced by m_j = deg - f + j.  Slot j's candidate is
// taken when an earlier slot had the same one (whoever holds it now), or when it equals the m_i of an earlier
// slot i that was replaced; the second can only spread from lower to higher slots, so a few votes settle it.
__device__ __forceinline__ int32_t floyd(int32_t cand, int32_t deg, int f, int j, int base, uint32_t group, bool active) {
  const int lane = threadIdx.x & 31;
  const uint32_t earlier = __match_any_sync(0xffffffffu, cand) & group & ((1u << lane) - 1u);
  const int32_t q = cand - (deg - f);   // the slot whose m equals the candidate
  bool taken = active && earlier != 0u;
  uint32_t r = __ballot_sync(0xffffffffu, taken);
  while (r != 0u) {
    taken = taken || (active && q >= 0 && q < j && ((r >> (base + q)) & 1u));
    const uint32_t r2 = __ballot_sync(0xffffffffu, taken);
    if (r2 == r) break;
    r = r2;
  }
  return taken ? deg - f + j : cand;
}

// The ids of one hop in shared memory, sorted, without repetitions, padded with the invalid id; their number.
template <int E>
__device__ __forceinline__ int sort_unique(int32_t *seg, int m, int len, int32_t V) {
  const int lane = threadIdx.x & 31;
  int32_t v[E];
#pragma unroll
  for (int e = 0; e < E; e++) v[e] = e * 32 + lane < m ? seg[e * 32 + lane] : 0x7fffffff;
  warp_sort<E>(v);
  __syncwarp();
  const int uniq = warp_unique_store<E>(v, seg);
  for (int i = uniq + lane; i < len; i += 32) seg[i] = V;
  return uniq;
}

template <bool DISTINCT>
__global__ void __launch_bounds__(256, khop_ctas(DISTINCT))
khop_rows_kernel(const __grid_constant__ KhopRows a) {
  extern __shared__ __align__(16) int32_t sh[];
  __shared__ unsigned int sh_sum[2];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, warps = blockDim.x >> 5;
  int32_t *row = sh + warp * a.fs;
  int32_t *live_p = sh + warps * a.fs + warp * 3 * a.parents_max, *live_rs = live_p + a.parents_max, *live_deg = live_rs + a.parents_max;
  if (threadIdx.x < 2) sh_sum[threadIdx.x] = 0u;
  __syncthreads();
  uint32_t edges = 0, pairs = 0;
  // the first sample of a warp follows from its place, the next ones are handed out a few at a time: samples
  // differ in work (half of an R-MAT graph's vertices have no neighbours), and warps must not wait for warps
  const int64_t all_warps = (int64_t)gridDim.x * warps;
  int64_t s = (int64_t)blockIdx.x * warps + warp, s_end = s + 1;
  while (s < a.S) {
    {
      int n_prev = 1, prefix_prev = 0, prefix = 0, n_last = 0, empty_from = a.steps;
      const uint32_t gs = (uint32_t)(a.first_sample + s);
      for (int k = 0; k < a.steps; k++) {
        const int f = a.fan[k], n = n_prev * f;
        // the parents that are vertices with neighbours
        int n_live = 0;
        for (int p0 = 0; p0 < n_prev; p0 += 32) {
          const int p = p0 + lane;
          const int32_t t = p < n_prev ? (k == 0 ? a.initial[s] : row[prefix_prev + p]) : -1;
          const bool valid = t >= 0 && t < a.V;
          const int2 r = valid ? __ldg(a.vrow + t) : make_int2(0, 0);
          const uint32_t m = __ballot_sync(0xffffffffu, r.y > 0);
          if (r.y > 0) {
            const int at = n_live + __popc(m & ((1u << lane) - 1u));
            live_p[at] = p; live_rs[at] = r.x; live_deg[at] = r.y;
          }
          n_live += __popc(m);
          pairs += valid ? 1u : 0u;
        }
        // no hop has vertices from here on (half of the seeds of an R-MAT graph): the rest of the row is empty
        if (n_live == 0) {
          for (int i = prefix + lane; i < a.fs; i += 32) row[i] = a.V;
          empty_from = k;
          break;
        }
        // the last hop of a row whose hops are sorted anyway is gathered without its empty slots
        const bool dense = DISTINCT && k == a.steps - 1 && n <= SORT_MAX;
        int m = 0;
        if (!dense) for (int i = lane; i < n; i += 32) row[prefix + i] = -1;
        __syncwarp();
        // phase one: the slots' entries of the adjacency array
        if (!DISTINCT) {
          for (int c = lane; c < n_live * f; c += 32) {
            const int l = c / f, slot = live_p[l] * f + (c - l * f);
            row[prefix + slot] = live_rs[l] + draw(a, gs, k, slot, live_deg[l]);
          }
        } else {
          const int per = 32 / f, sub = lane / f, j = lane - sub * f, base = sub * f;
          const uint32_t group = (f == 32 ? 0xffffffffu : (1u << f) - 1u) << (base & 31);
          for (int l0 = 0; l0 < n_live; l0 += per) {
            const int l = l0 + sub;
            const bool on = sub < per && l < n_live;
            const int32_t deg = on ? live_deg[l] : 0;
            const int slot = on ? live_p[l] * f + j : 0;
            int32_t idx = deg <= f ? (j < deg ? j : -1) : 0;
            if (deg > f) {
              idx = draw(a, gs, k, slot, deg - f + j + 1);
            }
            const int32_t pick = floyd(deg > f ? idx : -1 - lane, deg, f, j, base, group, deg > f);
            if (deg > f) idx = pick;
            const bool takes = on && idx >= 0;
            int at = slot;
            if (dense) {
              const uint32_t b = __ballot_sync(0xffffffffu, takes);
              at = m + __popc(b & ((1u << lane) - 1u));
              m += __popc(b);
            }
            if (takes) row[prefix + at] = live_rs[l] + idx;
          }
        }
        __syncwarp();
        // phase two: the neighbours
        const int slots = dense ? m : n;
        if (slots <= 32) {   // (the unrolled loop costs its eight turns whatever the hop's length)
          const int32_t e = lane < slots ? row[prefix + lane] : -1;
          if (lane < slots) row[prefix + lane] = e >= 0 ? __ldg(a.col + e) : a.V;
          edges += e >= 0 ? 1u : 0u;
        } else for (int c0 = lane; c0 < slots; c0 += 32 * GATHERS) {
          int32_t v[GATHERS];
#pragma unroll
          for (int j = 0; j < GATHERS; j++) {
            const int c = c0 + j * 32;
            const int32_t e = c < slots ? row[prefix + c] : -1;
            v[j] = a.V;
            if (e >= 0) { v[j] = __ldg(a.col + e); edges++; }
          }
#pragma unroll
          for (int j = 0; j < GATHERS; j++)
            if (c0 + j * 32 < slots) row[prefix + c0 + j * 32] = v[j];
        }
        __syncwarp();
        n_last = m;
        prefix_prev = prefix;
        prefix += n;
        n_prev = n;
      }
      if (DISTINCT) {
        int off = 0, n = 1;
        for (int k = 0; k < a.steps; k++) {
          n *= a.fan[k];
          int32_t *seg = row + off;
          if (k >= empty_from) {
            if (n <= SORT_MAX && lane == 0) a.hop_counts[s * a.steps + k] = 0;
          } else if (n <= SORT_MAX) {
            int m = k == a.steps - 1 ? n_last : 0;   // the vertices to the front, so that the network is no longer than they are
            if (m == 0 && k == a.steps - 1) for (int i = lane; i < n; i += 32) seg[i] = a.V;
            for (int i0 = 0; k < a.steps - 1 && i0 < n; i0 += 32) {
              const int32_t v = i0 + lane < n ? seg[i0 + lane] : a.V;
              const uint32_t b = __ballot_sync(0xffffffffu, v != a.V);
              if (v != a.V) seg[m + __popc(b & ((1u << lane) - 1u))] = v;
              m += __popc(b);
              __syncwarp();
            }
            const int uniq = m == 0 ? 0
                             : m <= 32 ? sort_unique<1>(seg, m, n, a.V)
                             : m <= 64 ? sort_unique<2>(seg, m, n, a.V)
                             : m <= 128 ? sort_unique<4>(seg, m, n, a.V)
                             : sort_unique<8>(seg, m, n, a.V);
            if (lane == 0) a.hop_counts[s * a.steps + k] = uniq;
          }
          off += n;
        }
      }
    }
    __syncwarp();
    int32_t *dst = a.out + s * a.fs;
    for (int i = lane; i < a.fs; i += 32) __stcs(dst + i, row[i]);
    __syncwarp();
    if (++s >= s_end) {
      s = a.S;
      if (a.S > all_warps) {
        unsigned long long nb = 0;
        if (lane == 0) nb = atomicAdd(&a.acc[8], (unsigned long long)a.batch);
        s = all_warps + (int64_t)__shfl_sync(0xffffffffu, nb, 0);
        s_end = s + a.batch;
      }
    }
  }
  for (int o = 16; o > 0; o >>= 1) {
    edges += __shfl_xor_sync(0xffffffffu, edges, o);
    pairs += __shfl_xor_sync(0xffffffffu, pairs, o);
  }
  if (lane == 0) {
    atomicAdd(&sh_sum[0], edges);
    atomicAdd(&sh_sum[1], pairs);
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    atomicAdd(&a.acc[0], (unsigned long long)sh_sum[0]);
    atomicAdd(&a.acc[1], (unsigned long long)sh_sum[1]);
    __threadfence();
    if (atomicAdd(&a.acc[10], 1ull) == (unsigned long long)gridDim.x - 1ull) {   // the last CTA
      __threadfence();
      for (int i = 0; i < 8; i++) a.stats[i] = i < 2 ? __ldcg(&a.acc[i]) : 0ull;
      a.acc[0] = a.acc[1] = a.acc[8] = a.acc[10] = 0ull;
    }
  }
}

}  // namespace

bool nd_khop_rows_fits(const nd_sampler *s) { return s->fs <= ROW_MAX; }

int nd_khop_rows_alloc(nd_sampler *s) {
  ND_TRY(nd_graph_ensure_vrow(s->g, s->dev.sms));
  ND_CUDA(s->p.app == ND_APP_KHOP_DISTINCT ? nd_smem_most(khop_rows_kernel<true>, s->dev) : nd_smem_most(khop_rows_kernel<false>, s->dev));
  ND_CUDA(nd_malloc(&s->d_rows_acc, 16 * sizeof(unsigned long long)));
  ND_CUDA(cudaMemset(s->d_rows_acc, 0, 16 * sizeof(unsigned long long)));
  return ND_OK;
}

int nd_khop_rows_launch(nd_sampler *s) {
  const nd_app_params &p = s->p;
  const bool distinct = p.app == ND_APP_KHOP_DISTINCT;
  KhopRows a;
  a.keys = ndrng::RoundKeys(p.seed); a.first_sample = s->first; a.S = s->S; a.V = s->g->V; a.fs = s->fs; a.steps = p.steps;
  int n = 1;
  a.parents_max = 1;
  for (int k = 0; k < p.steps; k++) {
    a.fan[k] = p.fanout[k];
    a.parents_max = n > a.parents_max ? n : a.parents_max;
    n *= p.fanout[k];
  }
  a.vrow = s->g->vrow; a.col = s->g->col; a.initial = s->d_initial; a.out = s->d_out; a.hop_counts = s->d_hop_counts;
  a.acc = s->d_rows_acc; a.stats = s->d_stats;
  // Eight samples per CTA; four where the rows are long or a mini-batch would leave SMs without a CTA.
  const size_t per_warp = sizeof(int32_t) * ((size_t)a.fs + 3 * (size_t)a.parents_max);
  const int warps = per_warp * 8 <= 48 * 1024 && s->S > (int64_t)s->dev.sms * 8 ? 8 : 4;
  const size_t smem = per_warp * warps;
  const int64_t groups = (s->S + warps - 1) / warps, cap = (int64_t)s->dev.sms * khop_ctas(distinct) * 8 / warps;
  const int grid = (int)(groups < cap ? groups : cap);
  a.batch = s->S > (int64_t)grid * warps * 16 ? 4 : 1;   // one by one where four would leave warps idle at the end
  if (distinct) khop_rows_kernel<true><<<grid, warps * 32, smem, s->stream>>>(a);
  else khop_rows_kernel<false><<<grid, warps * 32, smem, s->stream>>>(a);
  nd_count_launches(1);
  if (distinct) {   // hops too long for a warp's registers
    int off = 0;
    n = 1;
    for (int k = 0; k < p.steps; k++) {
      n *= p.fanout[k];
      if (n > SORT_MAX) {
        ND_TRY(nd_distinct_launch(s->stream, s->d_out + off, s->S, n, s->fs, s->g->V, s->d_hop_counts + k, p.steps));
        nd_count_launches(1);
      }
      off += n;
    }
  }
  ND_CUDA(cudaGetLastError());
  return ND_OK;
}
