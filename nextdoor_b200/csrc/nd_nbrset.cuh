// Exact membership of a vertex in a neighbour list (node2vec), by per-vertex hash sets.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

// node2vec asks "is v a neighbour of the previous vertex t?" for its candidates, and t is usually a
// hub (a 17-probe bisection of dependent loads).  Every vertex with at least SET_MIN_DEG
// neighbours gets an open-addressing hash set of its neighbour ids instead: buckets of 8 ids (one
// 32-byte sector), the buckets [row_ptr[t]/4, (row_ptr[t]+deg)/4) of one array (regions of
// consecutive vertices cannot overlap; at least deg slots each, load factor about 1/2).  An id
// lives in the first free slot at or after its home bucket, so a lookup reads the home bucket and
// is done unless that bucket is full and does not hold the id (about 5 % of the lookups).  The
// answer is exact, i.e. the answer of utils::binarySearch (src/utils.hpp:30-48).
constexpr int SET_MIN_DEG = 8;
constexpr int32_t SET_EMPTY = -1;

__device__ __forceinline__ uint32_t set_mix(uint32_t x) {
  x ^= x >> 16; x *= 0x7feb352du; x ^= x >> 15; x *= 0x846ca68bu; x ^= x >> 16;
  return x;
}
__device__ __forceinline__ uint32_t set_bucket_of_hash(uint32_t h, uint32_t n_buckets) {
  return (uint32_t)(((unsigned long long)h * n_buckets) >> 32);
}
__device__ __forceinline__ uint32_t set_bucket(int32_t v, uint32_t n_buckets) {
  return set_bucket_of_hash(set_mix((uint32_t)v), n_buckets);
}

// In front of the sets: one 32-bit word per bucket with SET_SIGN_BITS bits for every id of the list whose
// home bucket it is (8 bits of filter per neighbour, a quarter of the ids' own size and an eighth of the
// sets').  A missing bit proves that the id is not in the list.
__device__ __forceinline__ uint32_t set_sign(uint32_t h) {
  // the low bits of the hash: the bucket comes from the high ones
  return (1u << (h & 31u)) | (1u << ((h >> 5) & 31u)) | (1u << ((h >> 10) & 31u));
}
