// The bucket sort of one key (bucket_sort.cu): what the radix sort's host side (radix_sort.cu) hands it.
#pragma once

#include <stdint.h>

#include "radix_sort.cuh"

namespace am {
namespace bs {

constexpr uint32_t MODE_BUCKETS = 1, MODE_FALLBACK = 2;
constexpr int FREQUENT = 4;              // keys with too many rows for a bucket that a sort can set apart

// What the sampling, the histogram and the scan decide, read by the kernels after them. All zero when a
// sort starts (or cleared by it, Sort::clear).
struct State {
  unsigned long long lo, span;           // smallest sampled key, and the largest's distance from it
  unsigned long long diff;               // bits in which some value key differs from lo
  uint32_t mode;
  uint32_t up;                           // (key - lo) << up: the sampled range fills the word
  uint32_t linear;                       // not 0: the range is cut into this many equal buckets
  uint32_t buckets, s2, bins1;           // buckets; level 1 sorts by bucket >> s2 into bins1 bins
  uint32_t n_value, n_null, n_nan;
  uint32_t max_bucket;
  uint32_t later;                        // buckets that the fast form put off
  uint32_t counted;                      // the count's CTAs that are done
  // Keys too frequent for a bucket (Sort::frequent), ascending: their rows leave in row order, as null rows
  // do, to the places from `key_at` on among the values.
  uint32_t nkeys;
  unsigned long long key[FREQUENT];
  uint32_t key_rows[FREQUENT], key_at[FREQUENT];
};

// Strings behind 8-byte keys of their leading characters (strings.cu): rows of equal keys order by the rest
// of their strings, then by row id.
struct StringTies {
  const void* offsets;                   // row 0's offset; NULL: no strings
  const uint8_t* bytes;
  const uint32_t* chars;                 // device memory: the characters a key holds
  int32_t wide;                          // 64-bit offsets
  int32_t desc;
};

// Ranks instead of an order: out[row] = 1 + the first position of the row's equal keys (RANK_FIRST_OF), the
// last one's (RANK_LAST_OF), or its own position's (RANK_OWN); null and NaN rows are equal rows each, or
// (merge) all of them together.
constexpr int RANK_FIRST_OF = 1, RANK_LAST_OF = 2, RANK_OWN = 3;
struct RankOut {
  uint32_t* out;                         // NULL: no ranks
  int32_t mode;
  int32_t merge;
};

// The first rows' selection: keys below `limit` are kept, and those at it of the first `rows` rows, `count` of them.
struct FirstState {
  unsigned long long limit, rows;
  uint32_t count, pad;
};

// One bucket sort. `rec` (may be NULL): the payload columns that ride with the rows.
struct Sort {
  rs::ColView col;
  int key_bytes;
  uint64_t n;
  const void* src_keys;                  // not NULL: at most MAX_PAIRS rows given as keys and row ids, no column
  const uint32_t* src_ids;
  char* scratch;                         // `scratch_bytes(n)` bytes, the first `zeroed_bytes(n)` zero
  char* zeroed;                          // not NULL: those zero bytes are here instead
  void* clear;                           // not NULL: `clear_bytes` (a multiple of 16) that the sort itself clears first
  size_t clear_bytes;
  void* keys[2];                         // n keys each
  char* ids[2];                          // n x 4 bytes, or n x 16 with a payload; NULL: the sorted key column alone is wanted
  StringTies ties;
  RankOut ranks;
  bool payload;
  rs::RecLayout rec;
  void* out;                             // the order (NULL: not wanted)
  bool wide;
  void* key_out;                         // the sorted key column (NULL: not wanted)
  int key_pt;
  bool key_source;                       // a float order that ties values: null rows, zeros and NaNs keep their own bits
  bool key_desc, nulls_first;
  bool frequent;                         // set frequent keys apart (an order alone: no payload, key column, ranks or ties)
  uint32_t* err;
  rs::SortSummary* summary;
};

// Rows a bucket sort takes: up to what MAX_BUCKETS buckets hold.
constexpr uint64_t MAX_ROWS = uint64_t(60) << 20;

constexpr uint64_t MAX_PAIRS = 65536;

size_t scratch_bytes(uint64_t n);
size_t zeroed_bytes(uint64_t n);
// Enqueues the sort; afterwards State::mode says whether it ran (MODE_BUCKETS) or its rows are as they
// were (MODE_FALLBACK: the digit passes must run). Returns the State on the device.
State* enqueue(const Sort& b, cudaStream_t s);
// A batch of sorts of one key width in one launch a step: an item a sort, filled on the host, read by the
// kernels from device memory (no payload, no strings). `prepare_batch` before a stream is captured.
size_t batch_item_bytes();
void fill_batch_item(const Sort& b, void* item);
void prepare_batch(int key_bytes);
void enqueue_batch(const void* items, const void* host_items, uint32_t count, int key_bytes, bool timed, cudaStream_t s);
// Enqueues the choice of a key limit that at least the k smallest value keys are almost surely within, and
// one read of the column that appends the rows within it, as (key, row id) pairs in no order, to arrays
// of MAX_PAIRS; fs->count says how many there are. n is at least MAX_PAIRS.
void enqueue_first(const rs::ColView& col, int key_bytes, uint64_t n, uint64_t k, FirstState* fs, void* keys, uint32_t* rows,
                   cudaStream_t s);

}  // namespace bs
}  // namespace am
