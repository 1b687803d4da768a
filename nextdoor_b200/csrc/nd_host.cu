// Worker threads and staged host <-> device copies.
//
// A copy between the device and pageable memory runs at 10 GB/s up and 19 GB/s down on this box (one driver
// thread copies to or from its own pinned buffer, and faults in a fresh destination page by page); PCIe moves
// 53-55.  Here the pieces of a large copy go through a ring of pinned buffers that several workers fill or empty
// at once: 31-36 GB/s up and into memory that is there, 15-20 into fresh pages (pieces of 512 KB 27, of 1 MB 31;
// non-temporal stores and a second stream gain nothing).  One copy at a time uses the ring; a second one, and small
// ones, take the plain call.
#include "nd_host.h"

#include <stdlib.h>
#include <string.h>
#include <sys/mman.h>
#include <unistd.h>

#include <algorithm>
#include <atomic>
#include <chrono>
#include <condition_variable>
#include <deque>
#include <memory>
#include <mutex>
#include <new>
#include <thread>
#include <vector>

#ifdef __SSE2__
#include <emmintrin.h>
#endif

#include "nd_common.cuh"

// ---------------------------------------------------------------- workers

static void nd_host_idle();

namespace {

struct Job {
  const std::function<void(int)> *task;
  int n;
  std::atomic<int> next{0}, done{0};
};

struct Pool {
  std::mutex m;
  std::condition_variable work, finished;
  std::deque<Job *> jobs;      // with tasks nobody has taken
  int workers = 0, idle = 0;
  pid_t pid = 0;               // threads do not survive a fork
};
Pool *g_pool = nullptr;        // never destroyed: a worker may outlive the static objects
std::mutex g_pool_mutex;

Pool *pool() {
  std::lock_guard<std::mutex> lock(g_pool_mutex);
  if (!g_pool || g_pool->pid != getpid()) {
    g_pool = new Pool();
    g_pool->pid = getpid();
  }
  return g_pool;
}

void worker(Pool *p) {
  std::unique_lock<std::mutex> lock(p->m);
  for (;;) {
    if (p->jobs.empty()) {
      p->idle++;
      const bool woken = p->work.wait_for(lock, std::chrono::seconds(1), [&] { return !p->jobs.empty(); });
      p->idle--;
      if (!woken) {
        const bool last = --p->workers == 0;
        lock.unlock();
        if (last) nd_host_idle();
        return;
      }
    }
    Job *job = p->jobs.front();
    const int i = job->next.fetch_add(1, std::memory_order_relaxed);   // under the lock: the job is alive while it is in the queue
    if (i >= job->n - 1) p->jobs.pop_front();
    if (i >= job->n) continue;
    const int n = job->n;
    lock.unlock();
    (*job->task)(i);
    const bool last = job->done.fetch_add(1, std::memory_order_acq_rel) + 1 == n;   // after this the job may be gone
    lock.lock();
    if (last) p->finished.notify_all();
  }
}

}  // namespace

int nd_host_threads() {
  if (const char *e = getenv("ND_HOST_THREADS")) {
    const int n = atoi(e);
    if (n >= 1) return n < 256 ? n : 256;
  }
  const unsigned hc = std::thread::hardware_concurrency();
  return hc == 0 ? 4 : (hc > 32 ? 32 : (int)hc);
}

void nd_host_run(int n, const std::function<void(int)> &task, const std::function<void()> &own) {
  if (n <= 0 || (n == 1 && !own)) {
    if (own) own();
    if (n == 1) task(0);
    return;
  }
  Pool *p = pool();
  Job job;
  job.task = &task;
  job.n = n;
  {
    std::lock_guard<std::mutex> lock(p->m);
    p->jobs.push_back(&job);
    const int want = std::min(own ? n : n - 1, nd_host_threads() - 1) - p->idle;
    for (int k = 0; k < want && p->workers < 256; k++) {
      try {
        std::thread(worker, p).detach();
        p->workers++;
      } catch (...) {   // out of threads: the caller does it
        break;
      }
    }
  }
  p->work.notify_all();
  if (own) own();
  for (;;) {   // the caller's share
    const int i = job.next.fetch_add(1, std::memory_order_relaxed);
    if (i >= n) break;
    task(i);
    job.done.fetch_add(1, std::memory_order_acq_rel);
  }
  std::unique_lock<std::mutex> lock(p->m);
  p->jobs.erase(std::remove(p->jobs.begin(), p->jobs.end(), &job), p->jobs.end());
  p->finished.wait(lock, [&] { return job.done.load(std::memory_order_acquire) == n; });
}

// ---------------------------------------------------------------- staged copies

namespace {

constexpr size_t PIECE = (size_t)2 << 20;   // forty microseconds on the wire
constexpr int RING = 8;                    // pinned pieces
constexpr size_t FRESH = (size_t)48 << 20;       // see staged()
constexpr size_t STAGED_MIN = (size_t)2 << 20;   // below this the plain call is as fast

struct Ring {
  std::mutex m;                 // one copy at a time
  unsigned char *pinned = nullptr;
  int device = -1;              // of the stream and the events
  cudaStream_t stream = nullptr;
  cudaEvent_t done[RING] = {};  // the piece's transfer
};
Ring g_ring;
std::mutex g_objects_mutex;
int g_objects = 0;
std::atomic<bool> g_exiting{false};   // the process is on its way out: leave the driver alone

void ring_device_free() {
  if (g_ring.stream) cudaStreamDestroy(g_ring.stream);
  g_ring.stream = nullptr;
  for (cudaEvent_t &e : g_ring.done) { if (e) cudaEventDestroy(e); e = nullptr; }
  g_ring.device = -1;
}

// under g_ring.m, with `device` current
bool ring_ready(int device) {
  if (!g_ring.pinned && cudaHostAlloc(&g_ring.pinned, PIECE * RING, cudaHostAllocPortable) != cudaSuccess) {
    cudaGetLastError();
    g_ring.pinned = nullptr;
    return false;
  }
  static const int once = atexit([] { g_exiting.store(true); });
  (void)once;
  if (g_ring.device == device) return true;
  ring_device_free();
  bool ok = cudaStreamCreateWithFlags(&g_ring.stream, cudaStreamNonBlocking) == cudaSuccess;
  for (int i = 0; i < RING && ok; i++) ok = cudaEventCreateWithFlags(&g_ring.done[i], cudaEventDisableTiming) == cudaSuccess;
  if (!ok) { cudaGetLastError(); ring_device_free(); return false; }
  g_ring.device = device;
  return true;
}

bool pageable(const void *p) {
  cudaPointerAttributes at;
  if (cudaPointerGetAttributes(&at, p) != cudaSuccess) { cudaGetLastError(); return true; }
  return at.type == cudaMemoryTypeUnregistered;
}

// What the caller writes for someone else to read -- the wire, another thread much later -- goes past the caches: a store
// through them reads the line first (839 MB filled: 13.0 ms, 4.4 past them).  The stores of a thread are behind it after
// stores_done().
void store_past_caches(void *to, const void *from, size_t bytes) {
#ifdef __SSE2__
  unsigned char *t = (unsigned char *)to;
  const unsigned char *f = (const unsigned char *)from;
  const size_t head = std::min(bytes, (size_t)(-(uintptr_t)t & 15));
  if (head) memcpy(t, f, head);
  t += head; f += head; bytes -= head;
  for (; bytes >= 64; bytes -= 64, t += 64, f += 64) {
    const __m128i a = _mm_loadu_si128((const __m128i *)f), b = _mm_loadu_si128((const __m128i *)f + 1);
    const __m128i c = _mm_loadu_si128((const __m128i *)f + 2), d = _mm_loadu_si128((const __m128i *)f + 3);
    _mm_stream_si128((__m128i *)t, a);
    _mm_stream_si128((__m128i *)t + 1, b);
    _mm_stream_si128((__m128i *)t + 2, c);
    _mm_stream_si128((__m128i *)t + 3, d);
  }
  if (bytes) memcpy(t, f, bytes);
#else
  memcpy(to, from, bytes);
#endif
}
void stores_done() {
#ifdef __SSE2__
  _mm_sfence();
#endif
}

struct Segment {
  unsigned char *host, *dev;
  size_t bytes;
};

// Piece k of the copy uses slot k % RING.  The caller alone talks to the driver (threads that wait for
// events get in each other's way): it enqueues the pieces in order and publishes how many
// transfers are over.  The workers move pieces between the slots and the user's memory; the caller does so when
// none of them has got on for a while, so the copy ends without them too.
int staged(const std::vector<Segment> &segments, size_t bytes, bool up) {
  struct Piece { unsigned char *host, *dev; size_t size; };
  std::vector<Piece> piece;
  size_t most = PIECE / 8;   // small ones first, so that the wire and the workers are busy early
  for (const Segment &g : segments)
    for (size_t at = 0; at < g.bytes;) {
      const size_t n = std::min(most, g.bytes - at);
      piece.push_back(Piece{g.host + at, g.dev + at, n});
      at += n;
      if (most < PIECE && piece.size() % 4 == 0) most *= 2;
    }
  const size_t pieces = piece.size();
  std::vector<std::atomic<char>> moved(pieces);   // the host side of the piece is done
  std::atomic<size_t> over{0};                    // transfers that are complete
  std::atomic<size_t> next{0};                    // next piece to move
  std::atomic<bool> stop{false};
  // up: the slot's last transfer is over; down: the piece's own is
  auto movable = [&](size_t k) { return up ? k < over.load(std::memory_order_acquire) + RING : k < over.load(std::memory_order_acquire); };
  auto move = [&](size_t k) {
    unsigned char *slot = g_ring.pinned + (k % RING) * PIECE;
    if (up) { store_past_caches(slot, piece[k].host, piece[k].size); stores_done(); }
    else memcpy(piece[k].host, slot, piece[k].size);
    moved[k].store(1, std::memory_order_release);
  };
  std::atomic<int> helpers{0};                    // workers at it
  auto mover = [&] {
    helpers.fetch_add(1);
    for (;;) {
      const size_t k = next.fetch_add(1);
      if (k >= pieces) return;
      for (int spins = 0; !movable(k); spins++) {
        if (stop.load(std::memory_order_relaxed)) return;
        if (spins > 500) std::this_thread::yield();
      }
      move(k);
    }
  };
  cudaError_t err = cudaSuccess;
  auto driver = [&] {
    size_t sent = 0, done = 0;
    auto last = std::chrono::steady_clock::now();
    while (done < pieces) {
      if (sent < pieces && sent < done + RING && (up ? moved[sent].load(std::memory_order_acquire) != 0 : sent < RING || moved[sent - RING].load(std::memory_order_acquire) != 0)) {
        unsigned char *slot = g_ring.pinned + (sent % RING) * PIECE;
        err = up ? cudaMemcpyAsync(piece[sent].dev, slot, piece[sent].size, cudaMemcpyHostToDevice, g_ring.stream)
                 : cudaMemcpyAsync(slot, piece[sent].dev, piece[sent].size, cudaMemcpyDeviceToHost, g_ring.stream);
        if (err == cudaSuccess) err = cudaEventRecord(g_ring.done[sent % RING], g_ring.stream);
        if (err != cudaSuccess) return;
        sent++;
        last = std::chrono::steady_clock::now();
        continue;
      }
      if (done < sent) {
        const cudaError_t q = cudaEventQuery(g_ring.done[done % RING]);
        if (q == cudaSuccess) {
          over.store(++done, std::memory_order_release);
          last = std::chrono::steady_clock::now();
          continue;
        }
        if (q != cudaErrorNotReady) { err = q; return; }
      }
      // (waking a worker takes as long as moving a piece or two: until one is there the caller moves)
      if (helpers.load(std::memory_order_relaxed) > 0 && std::chrono::steady_clock::now() - last < std::chrono::microseconds(200)) continue;
      size_t k = next.load();
      if (k < pieces && movable(k) && next.compare_exchange_strong(k, k + 1)) move(k);
    }
  };
  // Up, eight keep up with the wire (100 MB: 2.05 ms, 49 GB/s; 2.3 with four; through the caches 2.8 with four, 3.2 with
  // six).  A large destination is likely to be fresh memory, where more of them share the page faults (15 -> 25 GB/s), but
  // take longer to wake.
  const size_t want = up ? 8 : bytes >= FRESH ? 12 : 4;
  const int movers = (int)std::min<size_t>(std::min<size_t>(pieces, want), (size_t)std::max(1, nd_host_threads() - 1));
  nd_host_run(movers, [&](int) { mover(); }, [&] {
    driver();
    stop.store(err != cudaSuccess);
  });
  cudaError_t e = cudaStreamSynchronize(g_ring.stream);   // nothing of the ring is in flight, whatever happened
  if (err != cudaSuccess) e = err;
  cudaGetLastError();   // a query that was not ready counts as an error of the thread
  ND_REQUIRE(e == cudaSuccess, ND_ERR_CUDA, "staged copy of %zu bytes failed: %s", bytes, cudaGetErrorString(e));
  return ND_OK;
}

int copy(int device, int n, void *const *dst, const void *const *src, const size_t *bytes, bool up) {
  ND_CUDA(cudaSetDevice(device));
  std::vector<Segment> plain, stage;   // pinned memory needs no staging
  size_t all = 0;
  for (int k = 0; k < n; k++) {
    if (!bytes[k]) continue;
    unsigned char *d = (unsigned char *)dst[k], *s = (unsigned char *)const_cast<void *>(src[k]);
    const Segment g = up ? Segment{s, d, bytes[k]} : Segment{d, s, bytes[k]};
    if (nd_host_threads() > 2 && pageable(g.host)) { stage.push_back(g); all += bytes[k]; }
    else plain.push_back(g);
  }
  if (all >= STAGED_MIN) {
    std::unique_lock<std::mutex> lock(g_ring.m, std::try_to_lock);
    if (lock.owns_lock() && ring_ready(device)) {
      ND_TRY(staged(stage, all, up));
      stage.clear();
    }
  }
  plain.insert(plain.end(), stage.begin(), stage.end());
  for (const Segment &g : plain)
    ND_CUDA(cudaMemcpy(up ? g.dev : g.host, up ? g.host : g.dev, g.bytes, up ? cudaMemcpyHostToDevice : cudaMemcpyDeviceToHost));
  return ND_OK;
}

}  // namespace

void nd_fill_past_caches(int32_t *to, int64_t n, int32_t value) {
#ifdef __SSE2__
  for (; n > 0 && ((uintptr_t)to & 15); n--) *to++ = value;
  const __m128i v = _mm_set1_epi32(value);
  for (; n >= 4; n -= 4, to += 4) _mm_stream_si128((__m128i *)to, v);
  stores_done();
#endif
  for (; n > 0; n--) *to++ = value;
}

// Adjacencies are a bit per entry on the device and on the way, 1/64 of the bytes of the two arrays that the workers write
// here (67 MB: 2.6 ms copied into memory that is there, 0.8 written; no faster past the caches, which hold memory that is
// lent again).
constexpr int64_t SMALL_ADJACENCY = 1 << 13;   // words (2 MB in two arrays) that the caller's thread writes by itself
int nd_adjacency_to_host(int device, const uint32_t *bits, int64_t layers, int stride, int L, int32_t *row, int32_t *col) {
  if (layers <= 0 || !(row || col)) return ND_OK;
  ND_CUDA(cudaSetDevice(device));
  const int per = (stride + 31) / 32;
  const int64_t words = layers * per;
  auto expand = [&](const uint32_t *in, int64_t w0, int64_t n) {
    nd_host_ranges(n, n < SMALL_ADJACENCY ? 1 : nd_host_threads(), [=](int, int64_t a, int64_t b) {
      for (int64_t w = a; w < b; w++) {
        const int64_t layer = (w0 + w) / per;
        const int at = (int)((w0 + w) - layer * per) * 32;
        const int64_t e0 = layer * stride + at;
        const size_t len = (size_t)std::min(32, stride - at);
        if (len == 32) {
          if (row) memset(row + e0, 0xff, 128);
          if (col) memset(col + e0, 0xff, 128);
        } else {
          if (row) memset(row + e0, 0xff, 4 * len);
          if (col) memset(col + e0, 0xff, 4 * len);
        }
        for (uint32_t left = in[w]; left; left &= left - 1) {
          const int k = __builtin_ctz(left);   // in the layer: transit (at + k) / L, vertex (at + k) % L
          if (row) row[e0 + k] = (at + k) / L;
          if (col) col[e0 + k] = (at + k) % L;
        }
      }
    });
  };
  std::unique_lock<std::mutex> lock(g_ring.m, std::defer_lock);
  if (words >= SMALL_ADJACENCY && lock.try_lock() && ring_ready(device)) {
    const int64_t most = (int64_t)(PIECE * RING / 4);
    for (int64_t w0 = 0; w0 < words; w0 += most) {
      const int64_t n = std::min(most, words - w0);
      ND_CUDA(cudaMemcpyAsync(g_ring.pinned, bits + w0, 4 * (size_t)n, cudaMemcpyDeviceToHost, g_ring.stream));
      ND_CUDA(cudaStreamSynchronize(g_ring.stream));
      expand((const uint32_t *)g_ring.pinned, w0, n);
    }
    return ND_OK;
  }
  if (lock.owns_lock()) lock.unlock();
  const int64_t most = std::min<int64_t>(words, 1 << 20);
  const std::unique_ptr<uint32_t[]> in(new (std::nothrow) uint32_t[(size_t)most]);
  ND_REQUIRE(in, ND_ERR_RANGE, "no memory for the adjacency's bits");
  for (int64_t w0 = 0; w0 < words; w0 += most) {
    const int64_t n = std::min(most, words - w0);
    ND_TRY(nd_copy_to_host(device, in.get(), bits + w0, 4 * (size_t)n));
    expand(in.get(), w0, n);
  }
  return ND_OK;
}

int nd_copies_to_host(int device, int n, void *const *dst, const void *const *src, const size_t *bytes) { return copy(device, n, dst, src, bytes, false); }
int nd_copies_to_device(int device, int n, void *const *dst, const void *const *src, const size_t *bytes) { return copy(device, n, dst, src, bytes, true); }
int nd_copy_to_host(int device, void *dst, const void *src, size_t bytes) { return copy(device, 1, &dst, &src, &bytes, false); }
int nd_copy_to_device(int device, void *dst, const void *src, size_t bytes) { return copy(device, 1, &dst, &src, &bytes, true); }

// ---------------------------------------------------------------- device memory that is kept

namespace {
constexpr size_t KEEP_BLOCK = (size_t)384 << 20, KEEP_ALL = (size_t)1 << 30;
struct Block {
  int device;
  void *p;
  size_t bytes;
};
std::mutex g_blocks_mutex;
std::vector<Block> g_kept;   // free blocks, oldest first
size_t g_kept_bytes = 0;

void drop_oldest() {   // under the lock
  cudaSetDevice(g_kept.front().device);
  cudaFree(g_kept.front().p);
  g_kept_bytes -= g_kept.front().bytes;
  g_kept.erase(g_kept.begin());
}
}  // namespace

cudaError_t nd_malloc_bytes(void **p, size_t bytes) {
  const cudaError_t e = cudaMalloc(p, bytes);
  if (e != cudaErrorMemoryAllocation) return e;
  cudaGetLastError();
  {   // what is kept may be what is missing
    std::lock_guard<std::mutex> lock(g_blocks_mutex);
    if (g_kept.empty()) return e;
    int now = 0;
    cudaGetDevice(&now);
    while (!g_kept.empty()) drop_oldest();
    cudaSetDevice(now);
  }
  return cudaMalloc(p, bytes);
}

int nd_block_alloc(int device, void **p, size_t *bytes) {
  {
    std::lock_guard<std::mutex> lock(g_blocks_mutex);
    size_t best = g_kept.size();
    for (size_t k = 0; k < g_kept.size(); k++)
      if (g_kept[k].device == device && g_kept[k].bytes >= *bytes && g_kept[k].bytes / 2 <= *bytes && (best == g_kept.size() || g_kept[k].bytes < g_kept[best].bytes))
        best = k;
    if (best < g_kept.size()) {
      *p = g_kept[best].p;
      *bytes = g_kept[best].bytes;
      g_kept_bytes -= g_kept[best].bytes;
      g_kept.erase(g_kept.begin() + (long)best);
      return ND_OK;
    }
  }
  ND_CUDA(nd_malloc_bytes(p, *bytes));
  return ND_OK;
}

void nd_block_free(int device, void *p, size_t bytes) {
  if (!p) return;
  cudaSetDevice(device);
  if (bytes > KEEP_BLOCK) { cudaFree(p); return; }
  cudaDeviceSynchronize();   // as cudaFree does: no stream uses it any more
  std::lock_guard<std::mutex> lock(g_blocks_mutex);
  g_kept.push_back(Block{device, p, bytes});
  g_kept_bytes += bytes;
  while (g_kept_bytes > KEEP_ALL) drop_oldest();
  cudaSetDevice(device);
}

// ---------------------------------------------------------------- host memory of results that is kept

namespace {
constexpr size_t KEEP_RESULT = (size_t)128 << 20, HUGE_PAGE = (size_t)2 << 20, SMALL_STEP = (size_t)64 << 10;
struct HostBlock {
  void *p;
  size_t bytes;
  bool pinned;
};
// Blocks of less than a huge page are kept and pinned on an account of their own: a queue of small results, held and dropped,
// neither pushes the large blocks out nor takes the pinned memory that they are to get.
struct ResultPool {
  size_t most;                           // of `bytes`, and of `pinned`
  std::vector<HostBlock> free;           // oldest first
  size_t bytes = 0, pinned = 0;          // of the free ones; of all that are pinned, lent ones too
};
std::mutex g_results_mutex;
ResultPool g_large{(size_t)256 << 20, {}}, g_small{(size_t)64 << 20, {}};
std::vector<HostBlock> g_lent;           // blocks that callers have

ResultPool &pool_of(size_t bytes) { return bytes < HUGE_PAGE ? g_small : g_large; }

void unmap(const HostBlock &b) {   // under the lock
  if (b.pinned) {
    if (!g_exiting.load()) cudaHostUnregister(b.p);
    pool_of(b.bytes).pinned -= b.bytes;
  }
  munmap(b.p, b.bytes);
}
void drop_results(ResultPool &pool, size_t keep) {   // under the lock
  while (pool.bytes > keep) {
    pool.bytes -= pool.free.front().bytes;
    unmap(pool.free.front());
    pool.free.erase(pool.free.begin());
  }
}
}  // namespace

// Memory for a result array of a caller that makes a new one for every call: faulting 23 MB in takes as long as copying
// them, and a copy into pageable memory 0.64 ms (35 GB/s, through the ring) instead of 0.44 (52).  So what is freed is
// kept, and pinned when it is lent again -- a caller that keeps its results never gets there.  From 2 MB on blocks are whole
// huge pages; below, where a caller may hold hundreds, steps of 64 KB whose pages are asked for at once, and one that is lent
// again is a quarter larger at most (300 results of 256 KB held: 73 MB and 106 us each; a huge page each 582 MB and 275 us; faulted
// in one by one 142 us, as in malloc's memory; of 1 MB 345, 370 and 490 us).  Contents undefined.
extern "C" int nd_result_alloc(int device, int64_t bytes, void **p) {
  ND_REQUIRE(p && bytes > 0, ND_ERR_ARG, "nd_result_alloc: bad argument");
  size_t n = ((size_t)bytes + SMALL_STEP - 1) / SMALL_STEP * SMALL_STEP;
  if (n >= HUGE_PAGE) n = (n + HUGE_PAGE - 1) / HUGE_PAGE * HUGE_PAGE;
  const size_t largest = n < HUGE_PAGE ? n + n / 4 : 2 * n;
  std::unique_lock<std::mutex> lock(g_results_mutex);
  ResultPool &pool = pool_of(n);
  size_t best = pool.free.size();
  for (size_t k = 0; k < pool.free.size(); k++)   // (the last one freed of the smallest that fit)
    if (pool.free[k].bytes >= n && pool.free[k].bytes <= largest && (best == pool.free.size() || pool.free[k].bytes <= pool.free[best].bytes)) best = k;
  HostBlock b{nullptr, n, false};
  if (best < pool.free.size()) {
    b = pool.free[best];
    pool.bytes -= b.bytes;
    pool.free.erase(pool.free.begin() + (long)best);
    if (!b.pinned && pool.pinned + b.bytes <= pool.most && !g_exiting.load()) {
      b.pinned = cudaSetDevice(device) == cudaSuccess && cudaHostRegister(b.p, b.bytes, cudaHostRegisterPortable) == cudaSuccess;
      if (b.pinned) pool.pinned += b.bytes;
      else cudaGetLastError();
    }
  } else {
    lock.unlock();
    b.p = mmap(nullptr, n, PROT_READ | PROT_WRITE, MAP_PRIVATE | MAP_ANONYMOUS | (n < HUGE_PAGE ? MAP_POPULATE : 0), -1, 0);
    ND_REQUIRE(b.p != MAP_FAILED, ND_ERR_RANGE, "no memory for a result of %lld bytes", (long long)bytes);
    if (n >= HUGE_PAGE) madvise(b.p, n, MADV_HUGEPAGE);
    lock.lock();
  }
  g_lent.push_back(b);
  *p = b.p;
  return ND_OK;
}

// kept for the next result while graphs or samplers are alive, 256 MB in all and 64 MB of small ones
extern "C" int nd_result_free(void *p) {
  std::lock_guard<std::mutex> objects(g_objects_mutex);
  std::lock_guard<std::mutex> lock(g_results_mutex);
  for (size_t k = 0; k < g_lent.size(); k++) {
    if (g_lent[k].p != p) continue;
    const HostBlock b = g_lent[k];
    g_lent.erase(g_lent.begin() + (long)k);
    if (b.bytes > KEEP_RESULT || g_objects <= 0) { unmap(b); return ND_OK; }
    ResultPool &pool = pool_of(b.bytes);
    pool.free.push_back(b);
    pool.bytes += b.bytes;
    drop_results(pool, pool.most);
    return ND_OK;
  }
  ND_REQUIRE(!p, ND_ERR_ARG, "nd_result_free: not a result's memory");
  return ND_OK;
}

extern "C" int nd_pinned_alloc(int device, int64_t bytes, void **p) {
  ND_REQUIRE(p && bytes > 0, ND_ERR_ARG, "nd_pinned_alloc: bad argument");
  ND_CUDA(cudaSetDevice(device));
  void *q = nullptr;
  ND_CUDA(cudaHostAlloc(&q, (size_t)bytes, cudaHostAllocPortable));
  memset(q, 0, (size_t)bytes);
  *p = q;
  return ND_OK;
}

extern "C" int nd_pinned_free(void *p) {
  if (p) ND_CUDA(cudaFreeHost(p));
  return ND_OK;
}

void nd_objects_add(int n) {
  std::lock_guard<std::mutex> lock(g_objects_mutex);
  g_objects += n;
  if (g_objects > 0) return;
  {
    std::lock_guard<std::mutex> results(g_results_mutex);
    drop_results(g_large, 0);
    drop_results(g_small, 0);
  }
  std::lock_guard<std::mutex> blocks(g_blocks_mutex);
  int now = 0;
  cudaGetDevice(&now);
  while (!g_kept.empty()) drop_oldest();
  cudaSetDevice(now);
}

// The last worker ends, a second after the last work: without graphs and samplers the ring goes too.
static void nd_host_idle() {
  {
    std::lock_guard<std::mutex> lock(g_objects_mutex);
    if (g_objects > 0) return;
  }
  std::unique_lock<std::mutex> ring(g_ring.m, std::try_to_lock);
  if (!ring.owns_lock() || g_exiting.load()) return;
  ring_device_free();
  if (g_ring.pinned) cudaFreeHost(g_ring.pinned);
  g_ring.pinned = nullptr;
}
