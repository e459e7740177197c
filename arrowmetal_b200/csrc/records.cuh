// Device helpers shared by the digit passes (radix_sort.cu) and the bucket sort (bucket_sort.cu): how a
// sorted key leaves as its column's value, and the payload records that ride with the rows.
#pragma once

#include <stdint.h>

#include "am_internal.h"
#include "radix_sort.cuh"

namespace am {
namespace rs {

// Inverse of the integer and totalOrder key maps (SortSource.swift:131-190 read backwards): the value
// bits of a key, at the key's width.
template <typename KeyT>
__device__ __forceinline__ uint64_t unkey_bits(KeyT k, int pt, int desc) {
  if (desc) k = KeyT(~k);
  if constexpr (sizeof(KeyT) == 8) {
    const uint64_t S = 0x8000000000000000ull;
    if (pt == PT_I64) return k ^ S;
    if (pt == PT_F64) return (k & S) ? (k ^ S) : ~k;
    return k;
  } else {
    const uint32_t S = 0x80000000u;
    if (pt == PT_U32) return k;
    if (pt == PT_F32) return (k & S) ? (k ^ S) : uint32_t(~k);
    return uint32_t(k ^ S);          // int32 and the narrow types widened to it (truncated on store)
  }
}

__device__ __forceinline__ void store_width(void* base, uint64_t i, int width, uint64_t v) {
  switch (width) {
    case 8: static_cast<uint64_t*>(base)[i] = v; break;
    case 4: static_cast<uint32_t*>(base)[i] = uint32_t(v); break;
    case 2: static_cast<uint16_t*>(base)[i] = uint16_t(v); break;
    default: static_cast<uint8_t*>(base)[i] = uint8_t(v); break;
  }
}
// ---- payload records (RecLayout)

__device__ __forceinline__ uint64_t load_width(const void* base, uint64_t i, int width) {
  switch (width) {
    case 8: return static_cast<const uint64_t*>(base)[i];
    case 4: return static_cast<const uint32_t*>(base)[i];
    case 2: return static_cast<const uint16_t*>(base)[i];
    default: return static_cast<const uint8_t*>(base)[i];
  }
}

// Row `row`'s record: its id and its payload fields read from the columns.
__device__ __forceinline__ uint4 build_record(const RecLayout& L, uint32_t row) {
  if (L.pair) {
    const uint64_t w = static_cast<const uint64_t*>(L.src[L.wide])[row];
    return make_uint4(row, uint32_t(w), uint32_t(w >> 32), static_cast<const uint32_t*>(L.src[L.narrow])[row]);
  }
  uint64_t lo = 0;           // payload bytes 0-7
  uint32_t hi = 0;           // payload bytes 8-11
  for (int c = 0; c < L.ncols; c++) {
    const uint64_t v = load_width(L.src[c], row, L.width[c]);
    const int o = L.off[c];
    if (o < 8) lo |= v << (8 * o);
    else hi |= uint32_t(v) << (8 * (o - 8));
  }
  return make_uint4(row, uint32_t(lo), uint32_t(lo >> 32), hi);
}

// A record's payload fields, written to row `dst` of the sorted payload columns.
__device__ __forceinline__ void unpack_record(const RecLayout& L, const uint4& r, uint64_t dst) {
  const uint64_t lo = uint64_t(r.y) | (uint64_t(r.z) << 32);
  if (L.pair) {
    static_cast<uint64_t*>(L.dst[L.wide])[dst] = lo;
    static_cast<uint32_t*>(L.dst[L.narrow])[dst] = r.w;
    return;
  }
  for (int c = 0; c < L.ncols; c++) {
    const int o = L.off[c];
    const uint64_t v = o < 8 ? (lo >> (8 * o)) : uint64_t(r.w >> (8 * (o - 8)));
    store_width(L.dst[c], dst, L.width[c], v);
  }
}

}  // namespace rs
}  // namespace am
