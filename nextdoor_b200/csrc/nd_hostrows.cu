// Walk results into a caller's dense host array without moving the empty slots.
//
// getFinalSamples (src/nextdoor.cu:3211-3237) hands the caller a dense [samples, steps] array.
// For walks that end early almost all of it is the invalid id (PPR with a stop probability of
// 0.15: 3 vertices on average in rows of 100), and copying it over PCIe takes twenty times longer
// than sampling it.  A walk's vertices are a prefix of its row, and the sampler knows each row's
// length (d_plen), so this path moves only the prefixes: the rows are packed on the device, the
// lengths and the packed vertices are copied, and host threads write them into the caller's
// array.  The caller's array keeps its contents from call to call like the device array does:
// `row_len` holds for every row how many leading slots may hold a vertex (everything behind is
// the invalid id), so an update rewrites only the slots a walk fills now or filled in the
// previous update of that array.  Three calls, so that the caller can overlap them with the next
// job's sampling: begin (enqueue) -> fetch (lengths have landed: enqueue the vertices) -> finish
// (vertices have landed: write the rows).
//
// Where the GPU can reach the caller's array and lengths (pinned memory) it writes a share of the rows itself, while the
// host threads write the others: the threads are bound by a cache line of the array or two per row, the GPU by the wire,
// and neither takes the other's time (2^21 rows of PPR: 2.3 ms by 16 threads, 2.2 by the GPU).
//
// An update lives on what begin has packed: from then on the sampler's result may change, and its next job neither
// waits for the host nor is waited for.  (Except where the job writes the staging array that the packed rows lie in, as the
// transit-parallel modes do: nd_hostrows_next_job.)
#include <algorithm>

#include <cuda.h>

#include "nd_common.cuh"
#include "nd_host.h"

struct NdHostRows {
  int32_t *h_len = nullptr;     // pinned [S]: the rows' lengths of the job being copied
  int32_t *h_vals = nullptr;    // pinned: packed vertices
  size_t vals_cap = 0;
  uint32_t *d_chunk = nullptr;  // per chunk of PACK_CHUNK rows: sum of lengths, then exclusive prefix
  int n_chunks = 0;
  cudaEvent_t packed = nullptr, len_done = nullptr, vals_done = nullptr, total_done = nullptr;
  uint32_t *h_total = nullptr;  // pinned: number of packed vertices (nd_sampler_pack_rows)
  cudaStream_t cs = nullptr;
  cudaStream_t vs = nullptr;    // the vertices': on the caller's copy stream they would wait for the lengths of all chunks begun since
  int32_t *out = nullptr, *row_len = nullptr;
  int64_t total = 0;
  uint32_t *h_chunk = nullptr;  // pinned: d_chunk of the job being copied
  bool moved = false;           // the sampler's result may be another job's by now
  bool ahead = false;           // fetched by the sampler's next job, the caller's fetch is still to come
  bool dense = false;           // most slots are in use: the dense array is copied as it is
  int stage = 0;                // 0 idle, 1 begun, 2 fetched
  int64_t direct = 0;           // rows from the front that the GPU writes
  uint32_t *d_pos = nullptr;    // ... [direct + 1]: where each of them begins in the packed array
  int32_t *dev_out = nullptr, *dev_row_len = nullptr;   // ... where it finds the caller's arrays
  cudaStream_t ds = nullptr;    // ... and the stream it does it on
  int threads = 1;
};

namespace {

constexpr int PACK_CHUNK = 4096;   // rows whose lengths are summed together
constexpr int PACK_ROWS = 256;     // rows of a CTA, one per thread

// Where a warp's rows lie in the packed array.  A row is three or four vertices in a line of its own, so the kernels are
// bound by how many of those lines are asked for at a time: a lane per row for the lengths, then a lane per vertex,
// which finds its row by bisecting the warp's prefix sums, so that packed vertices are read and written coalesced
// whatever the lengths (512k rows of PPR: 51 -> 12 us).
struct WarpRows {
  uint32_t len, inc;    // the lane's row: length, inclusive prefix in the warp
  uint32_t total;       // of the warp
  size_t pos;           // of the warp's first vertex

  __device__ __forceinline__ WarpRows(const int32_t *__restrict__ lens, int64_t row, int64_t S, const uint32_t *__restrict__ chunk_base, uint32_t *wsum) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    len = row < S ? (uint32_t)lens[row] : 0u;
    inc = len;
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t u = __shfl_up_sync(0xffffffffu, inc, o);
      if (lane >= o) inc += u;
    }
    total = __shfl_sync(0xffffffffu, inc, 31);
    // the rows of the chunk before the CTA's: a few loads that neighbouring CTAs share
    uint32_t before = 0;
    for (int64_t r = (int64_t)(blockIdx.x / (PACK_CHUNK / PACK_ROWS)) * PACK_CHUNK + threadIdx.x; r < (int64_t)blockIdx.x * PACK_ROWS; r += PACK_ROWS)
      before += (uint32_t)lens[r];
    before = __reduce_add_sync(0xffffffffu, before);
    if (lane == 0) { wsum[warp] = total; wsum[PACK_ROWS / 32 + warp] = before; }
    __syncthreads();
    pos = chunk_base[blockIdx.x / (PACK_CHUNK / PACK_ROWS)];
    for (int w = 0; w < PACK_ROWS / 32; w++) pos += wsum[PACK_ROWS / 32 + w] + (w < warp ? wsum[w] : 0u);
  }
  // fn(lane of the row, slot in the row, place in the warp's packed vertices)
  template <typename F>
  __device__ __forceinline__ void each(F fn) const {
    for (uint32_t base = 0; base < total; base += 32) {
      const uint32_t k = base + (threadIdx.x & 31);
      int r = 0;
#pragma unroll
      for (int step = 16; step > 0; step >>= 1)
        if (__shfl_sync(0xffffffffu, inc, r + step - 1) <= k) r += step;
      const uint32_t first = __shfl_sync(0xffffffffu, inc - len, r);
      if (k < total) fn(r, k - first, k);
    }
  }
};

__global__ void __launch_bounds__(PACK_ROWS)
pack_sum_kernel(const int32_t *__restrict__ plen, int64_t S, uint32_t *__restrict__ chunk) {
  __shared__ uint32_t wsum[PACK_ROWS / 32];
  const int64_t first = (int64_t)blockIdx.x * PACK_CHUNK;
  uint32_t t = 0;
#pragma unroll
  for (int r = threadIdx.x; r < PACK_CHUNK; r += PACK_ROWS) t += first + r < S ? (uint32_t)plen[first + r] : 0u;
  for (int o = 16; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
  if ((threadIdx.x & 31) == 0) wsum[threadIdx.x >> 5] = t;
  __syncthreads();
  if (threadIdx.x == 0) {
    uint32_t a = 0;
    for (int w = 0; w < PACK_ROWS / 32; w++) a += wsum[w];
    chunk[blockIdx.x] = a;
  }
}

// one CTA: chunk sums -> exclusive prefix in place, the grand total in chunk[n]
__global__ void __launch_bounds__(1024) pack_scan_kernel(uint32_t *__restrict__ chunk, int n) {
  __shared__ uint32_t wsum[32];
  __shared__ uint32_t carry_sh;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if (threadIdx.x == 0) carry_sh = 0;
  __syncthreads();
  for (int base = 0; base < n; base += 1024) {
    const int i = base + threadIdx.x;
    const uint32_t v = i < n ? chunk[i] : 0u;
    uint32_t inc = v;
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t t = __shfl_up_sync(0xffffffffu, inc, o);
      if (lane >= o) inc += t;
    }
    if (lane == 31) wsum[warp] = inc;
    __syncthreads();
    uint32_t before = carry_sh;
    for (int w = 0; w < warp; w++) before += wsum[w];
    if (i < n) chunk[i] = before + inc - v;
    __syncthreads();
    if (threadIdx.x == 1023) carry_sh = before + inc;
    __syncthreads();
  }
  if (threadIdx.x == 0) chunk[n] = carry_sh;
}

// the inverse of pack_rows_kernel on the receiving side: row r of `out` takes its len[r] vertices
// from vals, the slots it held before beyond that (row_len[r]) go back to the invalid id
__global__ void __launch_bounds__(PACK_ROWS)
unpack_rows_kernel(const int32_t *__restrict__ len, const int32_t *__restrict__ vals, const uint32_t *__restrict__ chunk_base,
                   int64_t S, int steps, int32_t invalid, int32_t *__restrict__ out, int32_t *__restrict__ row_len) {
  __shared__ uint32_t wsum[PACK_ROWS / 16];
  const int64_t mine = (int64_t)blockIdx.x * PACK_ROWS + threadIdx.x, first = mine - (threadIdx.x & 31);
  const WarpRows rows(len, mine, S, chunk_base, wsum);
  rows.each([&](int r, uint32_t slot, uint32_t k) { out[(first + r) * steps + slot] = vals[rows.pos + k]; });
  if (mine >= S) return;
  const int32_t had = row_len[mine];
  for (int k = (int)rows.len; k < had; k++) out[mine * steps + k] = invalid;
  if (had != (int)rows.len) row_len[mine] = (int32_t)rows.len;
}

// the prefixes of the rows to vals, back to back, and where the first `placed` rows and the one behind them begin there
__global__ void __launch_bounds__(PACK_ROWS)
pack_rows_kernel(const int32_t *__restrict__ plen, const int32_t *__restrict__ out, int64_t S, int steps,
                 const uint32_t *__restrict__ chunk_base, int64_t placed, uint32_t *__restrict__ place, int32_t *__restrict__ vals) {
  __shared__ uint32_t wsum[PACK_ROWS / 16];
  const int64_t mine = (int64_t)blockIdx.x * PACK_ROWS + threadIdx.x, first = mine - (threadIdx.x & 31);
  const WarpRows rows(plen, mine, S, chunk_base, wsum);
  if (placed > 0 && mine <= placed) place[mine] = (uint32_t)rows.pos + rows.inc - rows.len;
  rows.each([&](int r, uint32_t slot, uint32_t k) { vals[rows.pos + k] = out[(first + r) * steps + slot]; });
}

// The first `n` rows of the packed array into the caller's: the 64-byte lines of every row that hold a slot a walk fills
// now or filled at the array's previous update, whole (what lies behind a row's vertices is the invalid id, in the
// neighbouring rows of a line as well).  Bound by the wire: 1.1 M rows of 2^21 are 1.8 M lines, 2.2 ms at 52 GB/s; the
// vertices alone are 1.5 M writes of 4 to 32 bytes and take 2.9, their 32-byte sectors 2.4.  Two lanes to a line; 128
// threads of 32 registers find room beside the kernel that samples the next chunk.
constexpr int DIRECT_THREADS = 128;
__global__ void __launch_bounds__(DIRECT_THREADS, 16)
direct_rows_kernel(const uint32_t *__restrict__ pos, const int32_t *__restrict__ vals, uint32_t n, uint32_t steps, int32_t invalid, int32_t *out,
                   int32_t *row_len) {
  const int lane = threadIdx.x & 31;
  // places are counted from the line that the array begins in (32-bit: n * steps is at most 16/17 of 2^32, see direct_rows)
  const uint32_t begin = (uint32_t)((uintptr_t)out / 4 % 16), end = begin + n * steps;
  for (uint32_t first = blockIdx.x * DIRECT_THREADS + threadIdx.x - lane; first < n; first += gridDim.x * DIRECT_THREADS) {
    const uint32_t mine = first + lane;
    const int32_t now = mine < n ? (int32_t)(pos[mine + 1] - pos[mine]) : 0, had = mine < n ? row_len[mine] : 0;
    const uint32_t len = min((uint32_t)max(now, had), steps);
    if (__any_sync(0xffffffffu, now != had) && mine < n) row_len[mine] = now;
    const uint32_t line0 = (begin + mine * steps) / 16;
    const uint32_t lines = len > 0 ? (begin + mine * steps + len - 1) / 16 - line0 + 1u : 0u;
    uint32_t inc = lines;
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t u = __shfl_up_sync(0xffffffffu, inc, o);
      if (lane >= o) inc += u;
    }
    const uint32_t total = __shfl_sync(0xffffffffu, inc, 31);
    for (uint32_t base = 0; base < total; base += 16) {
      const uint32_t k = base + lane / 2;
      int r = 0;
#pragma unroll
      for (int step = 16; step > 0; step >>= 1)
        if (__shfl_sync(0xffffffffu, inc, r + step - 1) <= k) r += step;
      const uint32_t line = __shfl_sync(0xffffffffu, line0 - (inc - lines), r & 31) + k;
      const uint32_t at = line * 16 + lane % 2 * 8;   // eight places, of rows that may begin and end anywhere in them
      if (k >= total || at >= end || at + 8 <= begin) continue;
      const uint32_t slot0 = at > begin ? at - begin : 0u;
      uint32_t row = slot0 / steps, slot = slot0 - row * steps, p = pos[row], behind = pos[row + 1];
      int32_t v[8];
#pragma unroll
      for (int j = 0; j < 8; j++) {
        v[j] = invalid;
        if (at + j < begin || at + j >= end) continue;
        if (slot < behind - p) v[j] = vals[p + slot];
        if (++slot == steps) {
          slot = 0u;
          p = behind;
          if (++row < n) behind = pos[row + 1];
        }
      }
      int32_t *const to = out - begin + at;
      if (at >= begin && at + 8 <= end) {
        asm volatile("st.global.v8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"l"(to), "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]),
                     "r"(v[5]), "r"(v[6]), "r"(v[7])
                     : "memory");
      } else {
#pragma unroll
        for (int j = 0; j < 8; j++)
          if (at + j >= begin && at + j < end) to[j] = v[j];
      }
    }
  }
}

// Where the GPU finds `bytes` of host memory at `p`: inside one pinned allocation or registration, or null.
void *reachable(const void *p, size_t bytes) {
  static const auto range = []() -> CUresult (*)(unsigned int, CUpointer_attribute *, void **, CUdeviceptr) {
    void *f = nullptr;
    cudaDriverEntryPointQueryResult found;
    if (cudaGetDriverEntryPoint("cuPointerGetAttributes", &f, cudaEnableDefault, &found) != cudaSuccess || found != cudaDriverEntryPointSuccess) f = nullptr;
    cudaGetLastError();
    return (CUresult(*)(unsigned int, CUpointer_attribute *, void **, CUdeviceptr))f;
  }();
  cudaPointerAttributes at;
  if (!range || cudaPointerGetAttributes(&at, p) != cudaSuccess) { cudaGetLastError(); return nullptr; }
  if (at.type != cudaMemoryTypeHost || !at.devicePointer || at.devicePointer != p) return nullptr;
  CUdeviceptr start = 0;
  size_t size = 0;
  CUpointer_attribute what[2] = {CU_POINTER_ATTRIBUTE_RANGE_START_ADDR, CU_POINTER_ATTRIBUTE_RANGE_SIZE};
  void *into[2] = {&start, &size};
  if (range(2, what, into, (CUdeviceptr)p) != CUDA_SUCCESS) return nullptr;
  const uintptr_t a = (uintptr_t)p, s0 = (uintptr_t)start;
  return a >= s0 && a - s0 <= size && bytes <= size - (a - s0) ? at.devicePointer : nullptr;
}

// positions in the packed array are 32-bit
bool packable(const nd_sampler *s) { return s->S * (int64_t)s->fs < ((int64_t)1 << 32); }

// staging state of a sampler, made at the first use
int hostrows_init(nd_sampler *s) {
  if (s->hostrows) return ND_OK;
  s->hostrows = new NdHostRows();   // a creation that fails half way is taken down again, so the next call starts over
  NdHostRows *h = s->hostrows;
  const size_t S1 = (size_t)(s->S > 0 ? s->S : 1);
  h->n_chunks = (int)((S1 + PACK_CHUNK - 1) / PACK_CHUNK);
  h->threads = nd_host_threads();
  cudaError_t e = cudaMallocHost(&h->h_len, sizeof(int32_t) * S1);
  if (e == cudaSuccess) e = cudaMallocHost(&h->h_chunk, sizeof(uint32_t) * ((size_t)h->n_chunks + 1));
  if (e == cudaSuccess) e = cudaMallocHost(&h->h_total, sizeof(uint32_t));
  if (e == cudaSuccess) e = nd_malloc(&h->d_chunk, sizeof(uint32_t) * ((size_t)h->n_chunks + 1));
  if (e == cudaSuccess) e = cudaStreamCreateWithFlags(&h->vs, cudaStreamNonBlocking);
  if (e == cudaSuccess) e = cudaEventCreateWithFlags(&h->packed, cudaEventDisableTiming);
  if (e == cudaSuccess) e = cudaEventCreateWithFlags(&h->len_done, cudaEventDisableTiming);
  if (e == cudaSuccess) e = cudaEventCreateWithFlags(&h->vals_done, cudaEventDisableTiming);
  if (e == cudaSuccess) e = cudaEventCreateWithFlags(&h->total_done, cudaEventDisableTiming);
  if (e != cudaSuccess) {
    nd_hostrows_free(s);
    nd_set_error("staging buffers of the packed result: %s", cudaGetErrorString(e));
    cudaGetLastError();
    return ND_ERR_CUDA;
  }
  return ND_OK;
}

bool find_rows(nd_sampler *s) {
  NdHostRows *h = s->hostrows;
  h->dev_out = (int32_t *)reachable(h->out, sizeof(int32_t) * (size_t)s->S * s->fs);
  h->dev_row_len = (int32_t *)reachable(h->row_len, sizeof(int32_t) * (size_t)s->S);
  return h->dev_out && h->dev_row_len;
}

// The rows that the GPU writes itself, whole chunks from the front: as fast as 16 host threads (above).  The host's memory
// serves both, so that they are not twice as fast together.  Jobs of 2^21 rows on a host of 16 hardware threads, no share, a
// third, half, two thirds, four fifths: by 4 threads 9.1, 6.1, 4.6, 3.2, 2.6 ms; by 8 5.0, 3.9, 3.1, 2.5, 2.7; by 16 3.5, 2.5,
// 2.4, 2.6, 2.8; by 32, two to a hardware thread, 4.0, 2.8, 2.4, 2.5, 2.8.  (Threads that the host does not have, or that
// other processes use, count all the same: ND_HOST_THREADS says how many there are.)  None where a caller has captured a job, whose replays may come at any time.
int64_t direct_rows(nd_sampler *s, int32_t *out, int32_t *row_len) {
  NdHostRows *h = s->hostrows;
  if (s->S < 4 * PACK_CHUNK || s->in_graph || (uintptr_t)out % 4 || (uintptr_t)row_len % 4) return 0;
  if (!find_rows(s)) return 0;
  const int64_t n = s->S * 16 / (16 + h->threads) / PACK_CHUNK * PACK_CHUNK;
  if (n == 0) return 0;
  if (!h->ds && cudaStreamCreateWithFlags(&h->ds, cudaStreamNonBlocking) != cudaSuccess) { cudaGetLastError(); h->ds = nullptr; return 0; }
  if (!h->d_pos && nd_malloc(&h->d_pos, sizeof(uint32_t) * ((size_t)n + 1)) != cudaSuccess) { cudaGetLastError(); h->d_pos = nullptr; return 0; }
  return n;
}

// the prefixes of the rows packed into the staging array of the walk (free between two passes), on the sampler's stream
int pack_enqueue(nd_sampler *s, int64_t placed) {
  NdHostRows *h = s->hostrows;
  ND_TRY(nd_walk_ensure_tmp(s));
  pack_sum_kernel<<<h->n_chunks, PACK_ROWS, 0, s->stream>>>(s->d_plen, s->S, h->d_chunk);
  pack_scan_kernel<<<1, 1024, 0, s->stream>>>(h->d_chunk, h->n_chunks);
  pack_rows_kernel<<<(unsigned)((s->S + PACK_ROWS - 1) / PACK_ROWS), PACK_ROWS, 0, s->stream>>>(s->d_plen, s->d_out, s->S, s->fs, h->d_chunk, placed, h->d_pos,
                                                                                               s->d_tmp);
  nd_count_launches(3);
  ND_CUDA(cudaGetLastError());
  return ND_OK;
}

// the packed vertices to the host, once the chunks' sums are there
int fetch_vals(nd_sampler *s, cudaStream_t st) {
  NdHostRows *h = s->hostrows;
  const size_t first = h->h_chunk[h->direct / PACK_CHUNK], n = (size_t)h->total - first;
  if (n > h->vals_cap) {
    if (h->h_vals) ND_CUDA(cudaFreeHost(h->h_vals));
    h->h_vals = nullptr;
    h->vals_cap = 0;
    const size_t cap = n + n / 4 + 4096;
    ND_CUDA(cudaMallocHost(&h->h_vals, sizeof(int32_t) * cap));
    h->vals_cap = cap;
  }
  if (n > 0) ND_CUDA(cudaMemcpyAsync(h->h_vals, s->d_tmp + first, sizeof(int32_t) * n, cudaMemcpyDeviceToHost, st));
  return ND_OK;
}

// The rows of a fetched update that the GPU was to write go to the host threads, too.
int rows_to_host(nd_sampler *s) {
  NdHostRows *h = s->hostrows;
  const int64_t n = h->direct;
  const bool ahead = h->ahead;
  h->stage = 0;   // an error below abandons the update
  h->ahead = false;
  ND_CUDA(cudaEventSynchronize(h->vals_done));
  h->direct = 0;
  ND_TRY(fetch_vals(s, h->vs));
  ND_CUDA(cudaMemcpyAsync(h->h_len, h->d_pos, sizeof(uint32_t) * (size_t)n, cudaMemcpyDeviceToHost, h->vs));
  ND_CUDA(cudaStreamSynchronize(h->vs));
  uint32_t end = h->h_chunk[n / PACK_CHUNK];
  for (int64_t i = n - 1; i >= 0; i--) {
    const uint32_t pos = (uint32_t)h->h_len[i];
    h->h_len[i] = (int32_t)(end - pos);
    end = pos;
  }
  h->stage = 2;
  h->ahead = ahead;
  return ND_OK;
}

}  // namespace

// The sampler's next job is about to be enqueued.  An update in between only has to know, unless the job writes the array
// that the packed rows lie in (`staging`) or there are none (a result too large for them): then what is not on its way
// to the host yet is sent there first.
int nd_hostrows_next_job(nd_sampler *s, bool staging) {
  NdHostRows *h = s->hostrows;
  if (!h || h->stage == 0) return ND_OK;
  if (h->stage == 1 && (staging || !packable(s))) {
    ND_TRY(nd_sampler_host_update_fetch(s));
    h->ahead = true;
  }
  if (staging && h->direct) ND_TRY(rows_to_host(s));
  h->moved = true;
  return ND_OK;
}

void nd_hostrows_free(nd_sampler *s) {
  NdHostRows *h = s->hostrows;
  if (!h) return;
  if (h->h_len) cudaFreeHost(h->h_len);
  if (h->h_vals) cudaFreeHost(h->h_vals);
  if (h->h_chunk) cudaFreeHost(h->h_chunk);
  cudaFree(h->d_chunk);
  cudaFree(h->d_pos);
  if (h->vs) cudaStreamDestroy(h->vs);
  if (h->ds) cudaStreamDestroy(h->ds);
  if (h->packed) cudaEventDestroy(h->packed);
  if (h->len_done) cudaEventDestroy(h->len_done);
  if (h->vals_done) cudaEventDestroy(h->vals_done);
  if (h->total_done) cudaEventDestroy(h->total_done);
  if (h->h_total) cudaFreeHost(h->h_total);
  delete h;
  s->hostrows = nullptr;
}

extern "C" {

int nd_host_fill_int32(int32_t *dst, int64_t n, int32_t value) {
  ND_REQUIRE(dst || n == 0, ND_ERR_ARG, "nd_host_fill_int32: null destination");
  ND_REQUIRE(n >= 0, ND_ERR_ARG, "nd_host_fill_int32: negative length");
  nd_host_ranges(n, nd_host_threads(), [=](int, int64_t a, int64_t b) {
    nd_fill_past_caches(dst + a, b - a, value);
  });
  return ND_OK;
}

int nd_sampler_host_update_begin(nd_sampler *s, int32_t *out, int32_t *row_len, void *copy_stream) {
  ND_REQUIRE(s && ((out && row_len) || s->S == 0), ND_ERR_ARG, "nd_sampler_host_update_begin: null argument");
  ND_REQUIRE(nd_is_walk(s->p.app), ND_ERR_ARG, "host row updates exist for the walk apps (their rows are prefixes)");
  ND_REQUIRE(s->sampled, ND_ERR_STATE, "host update requested before sample()");
  ND_CUDA(cudaSetDevice(s->g->device));
  ND_TRY(hostrows_init(s));
  NdHostRows *h = s->hostrows;
  ND_REQUIRE(h->stage == 0, ND_ERR_STATE, "the previous host update of this sampler was not finished");
  h->out = out;
  h->row_len = row_len;
  h->cs = copy_stream ? (cudaStream_t)copy_stream : s->stream;
  if (s->S == 0) { h->stage = 1; return ND_OK; }
  // (an error below leaves stage 0: nothing was begun as far as the caller is concerned)
  h->moved = s->in_graph;
  h->direct = packable(s) ? direct_rows(s, out, row_len) : 0;
  if (packable(s)) ND_TRY(pack_enqueue(s, h->direct));   // (larger arrays take the dense copy in fetch)
  if (h->cs != s->stream) {
    ND_CUDA(cudaEventRecord(h->packed, s->stream));
    ND_CUDA(cudaStreamWaitEvent(h->cs, h->packed, 0));
  }
  ND_CUDA(cudaMemcpyAsync(h->h_len + h->direct, s->d_plen + h->direct, sizeof(int32_t) * (size_t)(s->S - h->direct), cudaMemcpyDeviceToHost, h->cs));
  if (packable(s))
    ND_CUDA(cudaMemcpyAsync(h->h_chunk, h->d_chunk, sizeof(uint32_t) * ((size_t)h->n_chunks + 1), cudaMemcpyDeviceToHost, h->cs));
  ND_CUDA(cudaEventRecord(h->len_done, h->cs));
  if (h->cs != s->stream) {  // the next sampling of this sampler waits for the copies that read its buffers
    if (!s->copy_done) ND_CUDA(cudaEventCreateWithFlags(&s->copy_done, cudaEventDisableTiming));
    if (s->copy_pending) ND_CUDA(cudaStreamWaitEvent(h->cs, s->copy_done, 0));
    ND_CUDA(cudaEventRecord(s->copy_done, h->cs));
    s->copy_pending = true;
  }
  h->stage = 1;
  return ND_OK;
}

int nd_sampler_host_update_fetch(nd_sampler *s) {
  ND_REQUIRE(s && s->hostrows && (s->hostrows->stage == 1 || s->hostrows->ahead), ND_ERR_STATE, "nd_sampler_host_update_fetch without a begun update");
  NdHostRows *h = s->hostrows;
  if (h->ahead) { h->ahead = false; return ND_OK; }
  h->stage = 0;   // an error below abandons the update; stage 2 is set once the copy is enqueued
  h->total = 0;
  h->dense = false;
  if (s->S == 0) { h->stage = 2; return ND_OK; }
  ND_CUDA(cudaSetDevice(s->g->device));
  ND_CUDA(cudaEventSynchronize(h->len_done));
  if (packable(s)) h->total = (int64_t)h->h_chunk[h->n_chunks];
  h->dense = (2 * h->total > s->S * (int64_t)s->fs && !h->moved) || !packable(s);
  if (h->dense) {
    ND_CUDA(cudaMemcpyAsync(h->out, s->d_out, sizeof(int32_t) * (size_t)s->S * s->fs, cudaMemcpyDeviceToHost, h->vs));
    if (h->direct) ND_CUDA(cudaMemcpyAsync(h->h_len, s->d_plen, sizeof(int32_t) * (size_t)h->direct, cudaMemcpyDeviceToHost, h->vs));
    h->direct = 0;
  } else if (h->total > 0) {
    ND_TRY(fetch_vals(s, h->vs));
  }
  ND_CUDA(cudaEventRecord(h->vals_done, h->vs));
  if (!s->copy_done) ND_CUDA(cudaEventCreateWithFlags(&s->copy_done, cudaEventDisableTiming));
  if (s->copy_pending) ND_CUDA(cudaStreamWaitEvent(h->vs, s->copy_done, 0));   // the event stands for all copies of the job
  ND_CUDA(cudaEventRecord(s->copy_done, h->vs));
  s->copy_pending = true;
  h->stage = 2;
  return ND_OK;
}

int nd_sampler_host_update_finish(nd_sampler *s, int64_t *values_copied) {
  ND_REQUIRE(s && s->hostrows && s->hostrows->stage >= 1, ND_ERR_STATE, "nd_sampler_host_update_finish without a begun update");
  NdHostRows *h = s->hostrows;
  if (h->stage == 1) ND_TRY(nd_sampler_host_update_fetch(s));
  if (h->direct && !find_rows(s)) ND_TRY(rows_to_host(s));   // (unregistered since the update was begun)
  ND_REQUIRE(h->stage == 2, ND_ERR_STATE, "nd_sampler_host_update_finish: the update was abandoned after an error");
  h->stage = 0;
  h->ahead = false;
  if (values_copied) *values_copied = h->dense ? s->S * (int64_t)s->fs : h->total;
  if (s->S == 0) return ND_OK;
  ND_CUDA(cudaSetDevice(s->g->device));
  ND_CUDA(cudaEventSynchronize(h->vals_done));
  const int32_t *len = h->h_len, *vals = h->h_vals;
  int32_t *out = h->out, *row_len = h->row_len;
  const int steps = s->fs;
  const int32_t invalid = s->g->V;
  if (h->dense) {  // the whole array came over as it is: only the lengths are left to note
    nd_host_ranges(s->S, h->threads, [=](int, int64_t a, int64_t b) {
      for (int64_t i = a; i < b; i++) row_len[i] = len[i];
    });
    return ND_OK;
  }
  const uint32_t *chunk = h->h_chunk;
  const int64_t direct = h->direct;
  const cudaStream_t ds = h->ds;
  if (direct) {
    const int grid = (int)std::min<int64_t>((direct + DIRECT_THREADS - 1) / DIRECT_THREADS, (int64_t)s->dev.sms * 4);
    direct_rows_kernel<<<grid, DIRECT_THREADS, 0, ds>>>(h->d_pos, s->d_tmp, (uint32_t)direct, (uint32_t)steps, invalid, h->dev_out, h->dev_row_len);
    nd_count_launches(1);
    ND_CUDA(cudaGetLastError());
  }
  nd_host_ranges(s->S - direct, h->threads, [=](int, int64_t a, int64_t b) {
    a += direct; b += direct;
    const int32_t *src = vals + (chunk[a / PACK_CHUNK] - chunk[direct / PACK_CHUNK]);   // the position of the range's first row in the packed array
    for (int64_t i = a - a % PACK_CHUNK; i < a; i++) src += len[i];
    constexpr int AHEAD = 24;   // rows lie apart and are not in any cache: ask for them before they are written
    for (int64_t i = a; i < b; i++) {
      if (i + AHEAD < b && (len[i + AHEAD] | row_len[i + AHEAD])) __builtin_prefetch(out + (i + AHEAD) * steps, 1);
      const int32_t now = len[i], had = row_len[i];
      int32_t *row = out + i * steps;
      for (int k = 0; k < now; k++) row[k] = src[k];
      for (int k = now; k < had; k++) row[k] = invalid;
      src += now;
      if (now != had) row_len[i] = now;
    }
  });
  if (direct) ND_CUDA(cudaStreamSynchronize(ds));
  return ND_OK;
}

// ---- the same packing between GPUs: the sender packs, the receiver unpacks into its dense array

int nd_sampler_pack_rows(nd_sampler *s, const int32_t **d_row_len, const int32_t **d_vals) {
  ND_REQUIRE(s && d_row_len && d_vals, ND_ERR_ARG, "nd_sampler_pack_rows: null argument");
  ND_REQUIRE(nd_is_walk(s->p.app), ND_ERR_ARG, "packed rows exist for the walk apps (their rows are prefixes)");
  ND_REQUIRE(s->sampled, ND_ERR_STATE, "packed rows requested before sample()");
  ND_REQUIRE(packable(s), ND_ERR_RANGE, "result array too large for 32-bit positions in the packed form");
  ND_CUDA(cudaSetDevice(s->g->device));
  ND_TRY(hostrows_init(s));
  NdHostRows *h = s->hostrows;
  ND_REQUIRE(h->stage == 0, ND_ERR_STATE, "a host update of this sampler is using the staging array");
  ND_TRY(nd_walk_ensure_tmp(s));
  *d_row_len = s->d_plen;
  *d_vals = s->d_tmp;
  *h->h_total = 0;
  if (s->S > 0) {
    ND_TRY(pack_enqueue(s, 0));
    ND_CUDA(cudaMemcpyAsync(h->h_total, h->d_chunk + h->n_chunks, sizeof(uint32_t), cudaMemcpyDeviceToHost, s->stream));
  }
  ND_CUDA(cudaEventRecord(h->total_done, s->stream));
  return ND_OK;
}

int nd_sampler_pack_rows_total(nd_sampler *s, int64_t *total) {
  ND_REQUIRE(s && total && s->hostrows && s->hostrows->total_done, ND_ERR_STATE, "nd_sampler_pack_rows_total before nd_sampler_pack_rows");
  ND_CUDA(cudaSetDevice(s->g->device));
  ND_CUDA(cudaEventSynchronize(s->hostrows->total_done));
  *total = (int64_t)*s->hostrows->h_total;
  return ND_OK;
}

int64_t nd_rows_scratch_words(int64_t n_rows) { return (n_rows + PACK_CHUNK - 1) / PACK_CHUNK + 1; }

int nd_rows_unpack(int device, void *stream, int64_t n_rows, int steps, int32_t invalid, const int32_t *d_len,
                   const int32_t *d_vals, int32_t *d_out, int32_t *d_row_len, uint32_t *d_scratch) {
  ND_REQUIRE(n_rows >= 0 && steps >= 1, ND_ERR_ARG, "nd_rows_unpack: bad size");
  if (n_rows == 0) return ND_OK;
  ND_REQUIRE(d_len && d_out && d_row_len && d_scratch, ND_ERR_ARG, "nd_rows_unpack: null argument");
  ND_REQUIRE(n_rows * (int64_t)steps < ((int64_t)1 << 32), ND_ERR_RANGE, "nd_rows_unpack: array too large for 32-bit positions");
  ND_CUDA(cudaSetDevice(device));
  cudaStream_t st = (cudaStream_t)stream;
  const int n_chunks = (int)((n_rows + PACK_CHUNK - 1) / PACK_CHUNK);
  pack_sum_kernel<<<n_chunks, PACK_ROWS, 0, st>>>(d_len, n_rows, d_scratch);
  pack_scan_kernel<<<1, 1024, 0, st>>>(d_scratch, n_chunks);
  unpack_rows_kernel<<<(unsigned)((n_rows + PACK_ROWS - 1) / PACK_ROWS), PACK_ROWS, 0, st>>>(d_len, d_vals, d_scratch, n_rows, steps, invalid, d_out, d_row_len);
  nd_count_launches(3);
  ND_CUDA(cudaGetLastError());
  return ND_OK;
}

}  // extern "C"
