// Loops over the CSR entries of a graph together with the rows they belong to.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

// source row of the CSR entry e, which lies in the rows [lo, hi)
__device__ __forceinline__ int32_t row_of_entry(const int32_t *__restrict__ row_ptr, int32_t lo, int32_t hi, int64_t e) {
  while (hi - lo > 1) {
    const int32_t mid = lo + ((hi - lo) >> 1);
    if ((int64_t)row_ptr[mid] <= e) lo = mid; else hi = mid;
  }
  return lo;
}

// f(first entry, end, first row, row behind the last) for spans of BUILD_SPAN consecutive entries, a CTA each: the rows
// of a span's first and last entry bound the search of all others.
constexpr int BUILD_THREADS = 256, BUILD_SPAN = 2048;
template <class F>
__device__ __forceinline__ void for_entry_spans(const int32_t *__restrict__ row_ptr, int32_t V, int64_t E, F f) {
  __shared__ int32_t sh[2];
  for (int64_t e0 = (int64_t)blockIdx.x * BUILD_SPAN; e0 < E; e0 += (int64_t)gridDim.x * BUILD_SPAN) {
    const int64_t e1 = e0 + BUILD_SPAN < E ? e0 + BUILD_SPAN : E;
    __syncthreads();
    if (threadIdx.x < 2) sh[threadIdx.x] = row_of_entry(row_ptr, 0, V, threadIdx.x ? e1 - 1 : e0);
    __syncthreads();
    f(e0, e1, sh[0], sh[1] + 1);
  }
}

// f(entry, its row) for every entry
template <class F>
__device__ __forceinline__ void for_entries(const int32_t *__restrict__ row_ptr, int32_t V, int64_t E, F f) {
  for_entry_spans(row_ptr, V, E, [&](int64_t e0, int64_t e1, int32_t lo, int32_t hi) {
    for (int64_t e = e0 + threadIdx.x; e < e1; e += BUILD_THREADS) f(e, row_of_entry(row_ptr, lo, hi, e));
  });
}
