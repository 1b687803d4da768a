// Host side of the library: worker threads and staged transfers between pageable memory and the device.
#pragma once

#include <stddef.h>
#include <stdint.h>

#include <functional>

// Host threads of the library's own work (ND_HOST_THREADS, default the hardware threads, at most 32).
int nd_host_threads();

// Runs task(0) .. task(n - 1) on the caller and the library's workers and returns when all are done; the caller runs
// `own` first, while workers may be at the tasks already.  Tasks must not wait for one another.  Workers are
// started when there is work for them, at most nd_host_threads() - 1, and end after a second without any; a
// worker that cannot be started is done without.  Several threads may call it at the same time.
void nd_host_run(int n, const std::function<void(int)> &task, const std::function<void()> &own = nullptr);

// fn(range, first, end) on `threads` contiguous ranges of [0, count)
template <class F>
void nd_host_ranges(int64_t count, int threads, F fn) {
  if (threads > count) threads = count > 0 ? (int)count : 1;
  nd_host_run(threads, [&](int t) { fn(t, count * t / threads, count * (t + 1) / threads); });
}

// `n` words, written past the caches.
void nd_fill_past_caches(int32_t *to, int64_t n, int32_t value);

// Blocking copies on a stream of their own: everything the copy depends on has to be complete.
int nd_copy_to_host(int device, void *dst, const void *src, size_t bytes);
int nd_copy_to_device(int device, void *dst, const void *src, size_t bytes);
int nd_copies_to_host(int device, int n, void *const *dst, const void *const *src, const size_t *bytes);     // several as one
int nd_copies_to_device(int device, int n, void *const *dst, const void *const *src, const size_t *bytes);

// Adjacency entries (row, col) = (i, j) or (-1, -1), entry i * L + j of a layer of `stride`, from a bit each, a layer in whole
// words; row or col may be null.
int nd_adjacency_to_host(int device, const uint32_t *bits, int64_t layers, int stride, int L, int32_t *row, int32_t *col);

// Device memory for building graphs.  Blocks of up to 384 MB are kept for the next build when they are freed, 1 GB of
// them in all, while graphs or samplers are alive (a cudaMalloc / cudaFree pair costs 0.5 to 30 ms, by the box); an
// allocation of the library that would fail gives all of them back first.  `bytes`: in: at least, out: what the block
// has.  The release waits for the device, as cudaFree does.
int nd_block_alloc(int device, void **p, size_t *bytes);
void nd_block_free(int device, void *p, size_t bytes);

// Graphs and samplers alive: without any, no block is kept, and the staging memory of the
// copies is returned when the workers end.
void nd_objects_add(int n);
