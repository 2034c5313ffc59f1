// Where a build row of a join goes in its group: the slot of its key, and how many rows came to the slot before.
// In one word, of which the slot has 58 bits: a table of 2^32 slots, for 2^30 rows and more, has one beyond
// them for the key 0, which 32 bits cut down to slot 0.
#pragma once
#include <cstdint>

#ifdef __CUDACC__
#define XLB_PLACE_FN __host__ __device__ __forceinline__
#else
#define XLB_PLACE_FN inline
#endif

constexpr int PLACE_NUMBER_BITS = 6;

XLB_PLACE_FN uint64_t place_of(uint64_t slot, unsigned number) { return (slot << PLACE_NUMBER_BITS) | number; }
XLB_PLACE_FN uint64_t place_slot(uint64_t place) { return place >> PLACE_NUMBER_BITS; }
XLB_PLACE_FN unsigned place_number(uint64_t place) { return (unsigned)(place & ((1u << PLACE_NUMBER_BITS) - 1)); }
