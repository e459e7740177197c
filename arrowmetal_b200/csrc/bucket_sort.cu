// Single-key sort by buckets: each row moves once or twice through HBM to its bucket of a few thousand
// rows, and every bucket is then ordered inside one CTA's shared memory.
//
//   1. buckets_kernel: up to 65,536 keys, evenly spread over the column, give the key
//      distribution. The sampled key range is cut into 512 equal coarse cells, a coarse cell into up to
//      2^11 equal fine cells by its share of the sample, a fine cell into equal sub-buckets by its
//      estimated rows (light neighbours share a bucket): a monotone map key -> bucket of two table reads
//      and one multiply, whose buckets hold about TARGET (CELL_TARGET) rows whatever the distribution.
//   2. bucket_histogram_kernel reads the column once: exact rows of every bucket, and of every level-1
//      bin of every chunk (a contiguous range of rows). bucket_starts_kernel turns them into starts, and
//      decides: when a bucket is larger than one CTA should sort (large_rows; a key repeated very often),
//      nothing has moved yet and the digit passes sort the column instead.
//   3. level1_kernel, one CTA a chunk, scatters the chunk's rows to their level-1 bins (the bucket
//      itself up to BINS1 buckets, else 256 buckets a bin), level2_kernel each bin's rows to their
//      buckets. A row's place among its tile's rows of a bin comes from one shared-memory atomic, in no
//      particular order: the row id that moves with it orders equal keys at the end. Rows are staged in
//      shared memory by bin, so a bin's rows leave as one run. The null and NaN rows go straight to
//      their final places, in row order (ballots, and the chunks' counts).
//   4. bucket_sort_kernel orders each bucket by (key, row id): a counting step over 2,048 bins that
//      divide the bucket's key range, then comparisons of (position, row id) within the bin (a row or two), and
//      writes ids, rebuilt keys and payload to their final rows. Buckets of keys that repeat more often than
//      a bin may hold, and those of more than CAP rows, are left to bucket_later_kernel: a second counting step, over
//      row ids, orders the rows of one key, and larger buckets are cut into parts first.
//
// Keys that repeat, the order of 16M int64 rows in us (digit passes and two-level sort; buckets with a bitonic sort of
// crowded ones; this): 10 rows a value 880, 1,454, 689; 50: 1,057, 2,640, 777; 500: 1,608, 1,242, 880; 3,000: 1,193,
// 1,245, 1,047.
//
// The order is the stable sort's: (key, row id) is what a stable sort orders by. What it replaces moved
// rows stably (nine ballots a row and a look-back over the tiles before it, 8.4 and 5.8 warp
// instructions a row in two passes bound by instruction issue); no step here needs the rows before a
// tile, so there is no look-back and no ordering between tiles.
#include <cooperative_groups.h>

#include <algorithm>
#include <cstring>
#include <memory>
#include <type_traits>

#include "am_internal.h"
#include "bucket_sort.cuh"
#include "key_encode.cuh"
#include "radix_sort.cuh"
#include "records.cuh"

namespace am {
namespace bs {

using namespace rs;

constexpr int COARSE_BITS = 9, COARSE = 1 << COARSE_BITS;
constexpr int FINE_BITS = 11;                     // a coarse cell has at most 2^11 fine cells
constexpr int FINE_GOAL = 512;                    // sum of 2^bits <= 2 x goal + COARSE
constexpr int FINE = 2 * FINE_GOAL + COARSE;
constexpr uint32_t MAX_BUCKETS = 40960;
constexpr int BINS1 = 1024;                       // level-1 bins
constexpr int S2 = 8, BINS2 = 1 << S2;            // buckets a level-1 bin of a two-level sort
static_assert(MAX_BUCKETS / BINS2 <= 256, "level-1 bins of a two-level sort");
constexpr int CAP = 2048;                         // rows the shared-memory sort of a bucket (or a part of one) takes
constexpr int BIG = 4096;                         // rows of one key whose strings differ that a bucket may hold
constexpr uint32_t LARGE = 16384;                 // rows a bucket may hold at most: it is split by its CTA
constexpr uint32_t TARGET = 1300;                 // rows a bucket of evenly spread keys is meant to hold
// With cells, whose densities are estimates: four columns of 5.5M normally distributed float64 keys had
// their largest bucket at 1,710-2,205 rows with 1,300, and one of more than CAP rows costs 100 us.
constexpr uint32_t CELL_TARGET = 1100;
constexpr uint32_t SAMPLES = 65536;               // keys looked at (every key of a shorter column)
constexpr int CLUSTER = 8;                        // CTAs of the one-cluster kernels
constexpr uint32_t FUSED_BUCKETS = 8192;          // buckets whose starts the count's last CTA finds
constexpr uint32_t ONE_CAP = 1024;                // buckets of a column of at most SAMPLES rows
constexpr int BINS = 2048, BINS_LOG = 11;         // bins of the shared-memory sort
constexpr uint32_t CATS = 2 + FREQUENT;           // a chunk's rows apart from the buckets: null, NaN, each frequent key
// Rows a bin may hold for the comparisons. 16M int64 keys with 10 rows a value, the order: 676 us where such bins are
// compared, 843 where later_body takes most of them (24); with 50 rows a value 776 in later_body, 1,113 compared (64).
constexpr uint32_t MAX_BIN = 40;
constexpr uint32_t META_SPLIT = 0x80000000u;
// From so many rows on, keys that differ in their two low bytes alone take the digit passes, of which they need two:
// 16M int64 keys of 2,500 values 471 us by passes, 958 by buckets; 4.5M 231 and 304; 1M 115 and 114.
constexpr uint64_t FEW_DIGITS_ROWS = uint64_t(1) << 20, FEW_DIGITS_SPAN = uint64_t(1) << 16;
// Four passes of a 4-byte key beat its buckets where keys repeat more than about 16 times (16M int32 rows: 645 us by
// passes; by buckets 621 with 10 rows a value, 698 with 50, 902 with 3,000; keys that do not repeat 408). Of the
// sample's 8 x 8,192 keys, about 1.6e8 x (rows a value) / rows meet an equal one.
constexpr uint64_t PAIRS_ROWS = uint64_t(1) << 22;
constexpr float PAIRS_LIMIT = 1.6e8f * 16.0f;
constexpr uint64_t WHOLE_SAMPLE_ROWS = uint64_t(1) << 22;
constexpr int CUR_PAD = 8;                        // cursors 32 bytes apart: same-sector atomics queue
constexpr int THREADS = 512, ITEMS = 7, TILE = THREADS * ITEMS, WARPS = THREADS / 32;
constexpr int HTHREADS = 1024, HITEMS = 8;
constexpr int LTHREADS = 256, LITEMS = CAP / LTHREADS, LBLOCKS = 4;
constexpr int NTHREADS = 256, NITEMS = CAP / NTHREADS, NBLOCKS = 4;      // the buckets that they put off

struct Args {
  State* st;
  uint32_t *coarse, *fine, *bfirst, *bmeta, *bcount, *bpos, *later, *cursor1, *cursor2, *chunk_bins, *chunk_cats;
  uint32_t nsamples, nchunks, chunk_rows, bucket_cap, bins1_cap;
  uint32_t large;                                 // rows a bucket may hold
  uint32_t hist_grid, level2_grid, sort_grid, later_grid;     // CTAs that take part in those steps
  uint64_t n;
  void* keys[2];
  uint32_t* ids[2];                               // NULL: no row ids (a sorted copy of an invertible key alone)
  uint4* rec[2];                                  // with a payload: row id and payload fields (RecLayout), instead of ids
  void *out, *key_out;
  uint4* clear;                                   // not NULL: memory that the plan's launch clears, the state among it
  uint64_t clear16;                               // in 16-byte units
  const void* src_keys;                           // not NULL: the rows are these keys, with these ids, and no column
  const uint32_t* src_ids;
  const void* key_src;                            // not NULL: keys that stand for several values are read here
  unsigned long long twin0, twin1;                // those keys: a zero's, a NaN's
  int32_t wide, key_pt, key_desc, nulls_first, has_payload;
  int32_t frequent;                               // set frequent keys apart
  int32_t one_launch;                             // the plan's launch counts and moves the rows too
  uint32_t* err;
  SortSummary* sum;
  StringTies ties;
  RankOut ranks;
  RecLayout pay;
};

// ---- the map key -> (bucket, fine cell, position in the fine cell)
//
// x = key - lo, shifted so that the sampled range fills the word: the top 9 bits are the coarse cell, the
// bits below lead the position within it.
template <typename KeyT>
struct Map {
  KeyT lo, span;
  uint32_t up, last, linear;
};
template <typename KeyT>
__device__ __forceinline__ Map<KeyT> load_map(const State* st) {
  return {KeyT(st->lo), KeyT(st->span), st->up, st->buckets - 1, st->linear};
}
// Fine cell `f` and the 32 bits below it, of x <= span.
template <typename KeyT>
__device__ __forceinline__ void cell_of(const Map<KeyT>& m, const uint32_t* coarse, KeyT x, uint32_t& f, uint32_t& frac) {
  const KeyT y = KeyT(x << m.up);
  constexpr int TOP = int(sizeof(KeyT)) * 8 - COARSE_BITS;
  const uint32_t e = coarse[uint32_t(y >> TOP)], fb = e >> 16;
  const KeyT z = KeyT(y << COARSE_BITS);
  uint32_t hi;
  if constexpr (sizeof(KeyT) == 8) {
    hi = uint32_t(z >> 32);
    frac = __funnelshift_l(uint32_t(z), hi, fb);
  } else {
    hi = z;
    frac = z << fb;
  }
  f = (e & 0xFFFFu) + ((hi >> 1) >> (31u - fb));
}
template <typename KeyT>
__device__ __forceinline__ uint32_t bucket_of(const Map<KeyT>& m, const uint32_t* coarse, const uint32_t* fine, KeyT key) {
  const KeyT x = KeyT(key - m.lo);                 // a key below lo wraps past the span
  if (x > m.span) return key < m.lo ? 0u : m.last;
  if (m.linear) return 1u + __umulhi(uint32_t(KeyT(x << m.up) >> (8 * sizeof(KeyT) - 32)), m.linear);
  uint32_t f, frac;
  cell_of(m, coarse, x, f, frac);
  const uint32_t e = fine[f];
  return (e & 0xFFFFu) + __umulhi(frac, e >> 16);
}

__device__ __forceinline__ void load_tables(const Args& a, uint32_t* coarse, uint32_t* fine) {
  if (a.st->linear) return;
  for (int i = threadIdx.x; i < COARSE; i += blockDim.x) coarse[i] = a.coarse[i];
  for (int i = threadIdx.x; i < FINE; i += blockDim.x) fine[i] = a.fine[i];
}

// A warp's NI x 32 rows from row w0 (item i of a lane: row w0 + 32 i + lane), rows before `end`, as
// loaded: raw key bits, and lane i's word of the validity bitmap is item i's 32 rows.
template <typename KeyT, int NI>
struct RawTile {
  KeyT key[NI];
  uint32_t word;
};
template <int NI>
__device__ __forceinline__ bool whole_words(const ColView& col, uint64_t w0, uint64_t end) {
  return w0 + NI * 32 <= end && (col.valid_off & 31) == 0 && (reinterpret_cast<uintptr_t>(col.valid) & 3u) == 0;
}
template <typename KeyT, int NI>
__device__ __forceinline__ void load_tile(const ColView& col, uint64_t w0, uint64_t end, RawTile<KeyT, NI>& r) {
  const uint32_t lane = threadIdx.x & 31u;
  const bool plain = sizeof(KeyT) == 8 || col.pt == PT_I32 || col.pt == PT_U32 || col.pt == PT_F32;
  if (w0 + NI * 32 <= end && plain) {
    const KeyT* v = static_cast<const KeyT*>(col.values) + w0 + lane;
#pragma unroll
    for (int i = 0; i < NI; i++) r.key[i] = v[i * 32];
  } else {
    uint32_t row[NI], ok = 0;
#pragma unroll
    for (int i = 0; i < NI; i++) {
      const uint64_t g = w0 + uint64_t(i) * 32 + lane;
      row[i] = uint32_t(g);
      if (g < end) ok |= 1u << i;
    }
    load_raw_rows<KeyT, NI>(col, row, ok, r.key);
  }
  r.word = 0;
  if (col.valid && lane < uint32_t(NI) && whole_words<NI>(col, w0, end))
    r.word = reinterpret_cast<const uint32_t*>(col.valid)[((uint64_t(col.valid_off) + w0) >> 5) + lane];
}
// Raw bits into keys; bit i of `values`, `nulls`, `nans` says what item i is. Keys of rows that are not
// values mean nothing.
template <typename KeyT, int NI>
__device__ __forceinline__ void encode_tile(const ColView& col, uint64_t w0, uint64_t end, RawTile<KeyT, NI>& t,
                                            uint32_t& values, uint32_t& nulls, uint32_t& nans) {
  const uint32_t lane = threadIdx.x & 31u;
  uint32_t ok = (1u << NI) - 1u;
  if (w0 + NI * 32 > end) {
    ok = 0;
#pragma unroll
    for (int i = 0; i < NI; i++)
      if (w0 + uint64_t(i) * 32 + lane < end) ok |= 1u << i;
  }
  values = ok;
  if (col.valid) {
    if (whole_words<NI>(col, w0, end)) {
      values = 0;
#pragma unroll
      for (int i = 0; i < NI; i++) values |= ((__shfl_sync(0xffffffffu, t.word, i) >> lane) & 1u) << i;
    } else {
      values = striped_validity<NI>(col, w0, end, ok);
    }
  }
  nulls = ok & ~values;
  nans = 0;
  constexpr KeyT SIGN = KeyT(KeyT(1) << (8 * sizeof(KeyT) - 1));
  const KeyT flip = col.desc ? KeyT(~KeyT(0)) : KeyT(0);
  if (sizeof(KeyT) == 8 ? col.pt == PT_F64 : (col.pt == PT_F32 || col.pt == PT_F16)) {
    constexpr KeyT INF = sizeof(KeyT) == 8 ? KeyT(0x7FF0000000000000ull) : KeyT(0x7F800000u);
    const bool total = col.float_order == FO_TOTAL;
#pragma unroll
    for (int i = 0; i < NI; i++) {
      KeyT r = t.key[i];
      if constexpr (sizeof(KeyT) == 4)
        if (col.pt == PT_F16) r = f16_to_f32_bits(uint32_t(r));
      const KeyT mag = KeyT(r & ~SIGN);
      if (!total) {
        if (mag > INF) {
          if (col.nan_cat) nans |= 1u << i;
          r = KeyT(INF | 1u);
        }
        if (mag == 0) r = 0;
      }
      t.key[i] = KeyT(r ^ (((r & SIGN) ? KeyT(~KeyT(0)) : SIGN) ^ flip));
    }
    nans &= values;
    values &= ~nans;
  } else {
    const KeyT x = KeyT((sizeof(KeyT) == 8 ? (col.pt == PT_I64 ? SIGN : KeyT(0)) : (col.pt == PT_U32 ? KeyT(0) : SIGN)) ^ flip);
#pragma unroll
    for (int i = 0; i < NI; i++) t.key[i] ^= x;
  }
}

// Exclusive scan of one value a thread over the block; `total` to every thread. Two barriers.
template <int NT>
__device__ __forceinline__ uint32_t block_scan(uint32_t v, uint32_t* s_warp, uint32_t& total) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  uint32_t x = v;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
    if (lane >= o) x += y;
  }
  __syncthreads();
  if (lane == 31) s_warp[warp] = x;
  __syncthreads();
  const uint32_t c = lane < NT / 32 ? s_warp[lane] : 0u;
  total = __reduce_add_sync(0xffffffffu, c);
  return x - v + __reduce_add_sync(0xffffffffu, lane < warp ? c : 0u);
}

__device__ __forceinline__ void store_id(const Args& a, uint64_t dst, uint32_t id) {
  if (!a.out) return;
  if (a.wide) static_cast<uint64_t*>(a.out)[dst] = id;
  else static_cast<uint32_t*>(a.out)[dst] = id;
}

// The rank of a null or NaN row at position `dst` of the order, beside nv values.
__device__ __forceinline__ void store_category_rank(const Args& a, uint32_t row, uint32_t dst, bool is_null, uint32_t nv,
                                                    uint32_t nn, uint32_t nx) {
  if (!a.ranks.out) return;
  uint32_t lo, hi;                       // the row's equals: positions [lo, hi)
  if (a.ranks.merge) {
    lo = a.nulls_first ? 0u : nv;
    hi = lo + nn + nx;
  } else if (is_null) {
    lo = a.nulls_first ? 0u : nv + nx;
    hi = lo + nn;
  } else {
    lo = a.nulls_first ? nn : nv;
    hi = lo + nx;
  }
  a.ranks.out[row] = a.ranks.mode == RANK_FIRST_OF ? lo + 1 : a.ranks.mode == RANK_LAST_OF ? hi : dst + 1;
}

// The key column's bits at a row, where a row's key does not give them (0 where null rows are written as 0).
__device__ __forceinline__ uint64_t source_bits(const Args& a, uint32_t row) {
  return a.key_src ? load_width(a.key_src, row, pt_bytes(a.key_pt)) : 0ull;
}

// ---- bulk copies between shared and global memory (addresses and sizes multiples of 16 bytes)

__device__ __forceinline__ uint32_t smem_addr(const void* p) { return uint32_t(__cvta_generic_to_shared(p)); }
// Shared memory written by this thread becomes visible to bulk copies issued after the next barrier.
__device__ __forceinline__ void fence_bulk() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }
__device__ __forceinline__ void bulk_store(void* dst, const void* src, uint32_t bytes) {
  asm volatile("cp.async.bulk.global.shared::cta.bulk_group [%0], [%1], %2;" ::"l"(dst), "r"(smem_addr(src)), "r"(bytes) : "memory");
}
__device__ __forceinline__ void bulk_commit() { asm volatile("cp.async.bulk.commit_group;" ::: "memory"); }
// Until this thread's bulk stores have read their shared memory; until they are complete.
__device__ __forceinline__ void bulk_wait_read() { asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory"); }
__device__ __forceinline__ void bulk_wait_all() { asm volatile("cp.async.bulk.wait_group 0;" ::: "memory"); }
__device__ __forceinline__ void mbar_init(uint64_t* bar) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_addr(bar)) : "memory");
  asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}
__device__ __forceinline__ void bulk_load(void* dst, const void* src, uint32_t bytes, uint64_t* bar) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_addr(bar)), "r"(bytes) : "memory");
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(smem_addr(dst)),
               "l"(src), "r"(bytes), "r"(smem_addr(bar))
               : "memory");
}
// Waits for the phase of `parity`: at most about a second, then false.
__device__ __forceinline__ bool mbar_wait(uint64_t* bar, uint32_t parity) {
  for (uint32_t polls = 0; polls < (1u << 20); polls++) {
    uint32_t done;
    asm volatile("{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}"
                 : "=r"(done) : "r"(smem_addr(bar)), "r"(parity) : "memory");
    if (done) return true;
  }
  return false;
}

// ---- 1. the sample and the bucket map

// One cluster of CTAs; each holds its share of the sample in registers, and sums counts over the
// cluster's shared memories. (One CTA alone, its samples read twice from L2, took 60 us for 65,536.)
struct PlanShared {
  uint32_t coarse_cnt[COARSE];
  union {
    uint32_t part_cnt[4 * FINE];         // the quarters of the fine cells, up to the plan
    struct {
      uint32_t bins[ONE_CAP], start[ONE_CAP];      // then (one launch) the CTA's rows of each bucket, where they go
    };
  };
  uint32_t coarse[COARSE];
  uint32_t warp[32];
  uint32_t group[1024];
  unsigned long long smax[CLUSTER], smin[CLUSTER], scnt[CLUSTER];
  unsigned long long wmax[32], wmin[32];
  uint32_t pairs[CLUSTER];               // the CTAs' pairs of equal keys, then their most frequent keys
  uint32_t mode, buckets, linear;        // the plan, from the first CTA
  // One launch for the counts and the moves too (columns of at most SAMPLES rows): the fine cells, the
  // CTA's null and NaN rows by item and warp, and their sums.
  uint32_t fine[FINE];
  uint32_t cats[2][SAMPLES / (1024 * CLUSTER) * 32];
  uint32_t ncats[2];
  unsigned long long diff;
};

__device__ __forceinline__ void tell_plan(const Args& a, unsigned long long lo, unsigned long long span, uint32_t up,
                                          uint32_t buckets, uint32_t linear) {
  State* st = a.st;
  st->lo = lo;
  st->span = span;
  st->up = up;
  st->linear = linear;
  st->buckets = buckets;
  st->s2 = buckets <= a.bins1_cap ? 0u : uint32_t(S2);
  st->bins1 = buckets <= a.bins1_cap ? buckets : (buckets + BINS2 - 1) >> S2;
  st->mode = MODE_BUCKETS;
}

// The first CTA, with the cluster's counts of the quarter cells: buckets from the fine cells' rows.
template <typename KeyT>
__device__ void plan_cells(const Args& a, PlanShared& sm, const Map<KeyT>& map, unsigned long long lo, unsigned long long span,
                           uint32_t shc, uint32_t sv, uint32_t nfine, bool full) {
  const int t = threadIdx.x;
  State* st = a.st;
  const uint32_t* coarse = sm.coarse;
  // Rows of each fine cell, at the upper end of what the sample says; single-key cells (nothing left to
  // split) that surely exceed a bucket end the attempt here.
  constexpr int PER = (FINE + 1023) / 1024;
  const float scale = float(a.n) / float(a.nsamples);
  uint32_t rows[PER], dense[PER], room[PER], below[PER];     // below: what shifts a key's distance from lo to its place in the cell
  uint32_t bad = 0;
#pragma unroll
  for (int q = 0; q < PER; q++) {
    const uint32_t f = uint32_t(t) * PER + q;
    rows[q] = 0;
    dense[q] = 0;
    room[q] = 1;
    below[q] = 0;
    if (f >= nfine) continue;
    const uint4 part = *reinterpret_cast<const uint4*>(&sm.part_cnt[4 * f]);
    const uint32_t h0 = part.x + part.y, h1 = part.z + part.w, most = max(max(part.x, part.y), max(part.z, part.w));
    const float c = float(h0 + h1), h = float(max(h0, h1));
    // (At 50M rows a sampled key stands for 763: a cell of 5,000 rows shows one sample once in a hundred columns.)
    rows[q] = full ? h0 + h1 : uint32_t((c + 1.5f * sqrtf(c) + 2.5f) * scale);
    // Split by the fuller half, or by the fullest quarter where the rows of a wide cell crowd there (a
    // float's cell of eight octaves has half its rows in the last): by the halves alone, two buckets of 6M
    // normally distributed float64 keys held over CAP rows, and their slow form was the sort's last 100 us
    // (the buckets' sort 172 us, 66 so).
    const float e = float(most);
    dense[q] = full ? max(2u * max(h0, h1), 4u * most)
                    : uint32_t(max(2.0f * (h + sqrtf(h) + 2.0f), 4.0f * (e + 0.5f * sqrtf(e))) * scale);
    // The fine cell's coarse cell: the last one starting at or before it.
    uint32_t l = 0, r = COARSE;
    while (r - l > 1) {
      const uint32_t mid = (l + r) >> 1;
      if ((coarse[mid] & 0xFFFFu) <= f) l = mid;
      else r = mid;
    }
    const uint32_t left = shc - (coarse[l] >> 16);           // key bits below the fine cell
    room[q] = left >= 16 ? 65535u : 1u << left;
    below[q] = uint32_t(sizeof(KeyT)) * 8u - left;
    if (room[q] == 1u && (c - 4.0f * sqrtf(c)) * scale > float(a.large)) bad = 1;
  }
  bad = __syncthreads_or(bad);
  // Buckets: a heavy cell (over half a target) is split into equal parts; light neighbours share one.
  // With more buckets than fit, larger targets.
  uint32_t target = CELL_TARGET, total = 0, base[PER], m[PER];
  bool start[PER];
  for (int attempt = 0; attempt < 8 && !bad; attempt++) {
    const uint32_t half = target / 2;
    uint32_t light = 0;
#pragma unroll
    for (int q = 0; q < PER; q++)
      if (rows[q] <= half) light += rows[q];
    uint32_t all;
    uint32_t before = block_scan<1024>(light, sm.warp, all);
    // The group of the cell before this thread's first one.
    uint32_t group[PER];
#pragma unroll
    for (int q = 0; q < PER; q++) {
      const bool heavy = rows[q] > half;
      group[q] = heavy ? 0xFFFFFFFFu : before / half;
      if (!heavy) before += rows[q];
    }
    sm.group[t] = group[PER - 1];
    __syncthreads();
    uint32_t prev = t ? sm.group[t - 1] : 0xFFFFFFFFu, add = 0;
#pragma unroll
    for (int q = 0; q < PER; q++) {
      const uint32_t f = uint32_t(t) * PER + q;
      m[q] = 1;
      start[q] = group[q] == 0xFFFFFFFFu || group[q] != prev;
      if (group[q] == 0xFFFFFFFFu) m[q] = min((dense[q] + target - 1) / target, room[q]);
      prev = group[q];
      base[q] = add;
      if (f < nfine && start[q]) add += m[q];
    }
    const uint32_t off = block_scan<1024>(add, sm.warp, total);
#pragma unroll
    for (int q = 0; q < PER; q++) base[q] += off;
    if (total + 2 <= a.bucket_cap) break;
    target += target / 8;
  }
  if (bad || total + 2 > a.bucket_cap || sv == 0) {
    if (t == 0) {
      st->mode = MODE_FALLBACK;
      sm.mode = MODE_FALLBACK;
    }
    return;
  }
  // The tables. Bucket 0 and the last take the keys outside the sampled range.
#pragma unroll
  for (int q = 0; q < PER; q++) {
    const uint32_t f = uint32_t(t) * PER + q;
    if (f >= nfine) continue;
    const uint32_t b = 1u + base[q] - (start[q] ? 0u : 1u);
    a.fine[f] = b | (m[q] << 16);
    sm.fine[f] = b | (m[q] << 16);
    if (rows[q] > target / 2) {
      for (uint32_t k = 0; k < m[q]; k++) {
        a.bfirst[b + k] = below[q] << 16;
        a.bmeta[b + k] = META_SPLIT | m[q];
      }
    } else {
      if (start[q]) a.bfirst[b] = f;
      atomicMax(&a.bmeta[b], f);               // the last cell of the bucket (bmeta starts at zero)
    }
  }
  if (t == 0) {
    const uint32_t nb = total + 2;
    a.bmeta[0] = META_SPLIT;
    a.bmeta[nb - 1] = META_SPLIT;
    a.bfirst[0] = 0xFFFF0000u;
    a.bfirst[nb - 1] = 0xFFFF0000u;
    sm.buckets = nb;
    sm.mode = MODE_BUCKETS;
    tell_plan(a, lo, span, map.up, nb, 0u);
  }
}

// Sets frequent keys apart: up to FREQUENT that hold at least 1/512 of the sample and more rows than half
// of BIG. The sample's keys are counted by a hash into 2,048 counters (about 32 each); in a counter four
// times that one key has the majority, so each of its bits is the majority's bit. A wrong guess is a key of
// another counter, or a key of few rows: nothing depends on either. Returns which of this thread's keys
// they are. (key2 of a 16M-row lexsort, a float with 80 K rows each of zero and both infinities: without,
// no bucket holds those rows and eight digit passes run, 1,300 us.)
constexpr int COUNTERS_LOG = 11, COUNTERS = 1 << COUNTERS_LOG;
template <typename KeyT, int U>
__device__ uint32_t take_frequent(const Args& a, PlanShared& sm, const KeyT (&key)[U], uint32_t live) {
  namespace cg = cooperative_groups;
  cg::cluster_group cl = cg::this_cluster();
  static_assert(COUNTERS <= 4 * FINE && FREQUENT * 64 + FREQUENT + FREQUENT * 2 <= 1024, "they borrow the plan's arrays");
  constexpr uint32_t NONE = 0xFFFFFFFFu;
  const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
  uint32_t* counter = sm.part_cnt;
  uint32_t* votes = sm.group;                      // by key and bit, then the voters, then the keys' words
  uint32_t* voters = votes + FREQUENT * 64;
  uint32_t* words = voters + FREQUENT;
  auto counter_of = [](KeyT k) { return uint32_t((uint64_t(k) * 0x9E3779B97F4A7C15ull) >> (64 - COUNTERS_LOG)); };
  for (int i = t; i < COUNTERS; i += 1024) counter[i] = 0;
  if (t < FREQUENT * 64 + FREQUENT) votes[t] = 0;
  __syncthreads();
#pragma unroll
  for (int u = 0; u < U; u++)
    if ((live >> u) & 1u) atomicAdd(&counter[counter_of(key[u])], 1u);
  cl.sync();
  uint32_t best[COUNTERS / 1024];                  // count << COUNTERS_LOG | counter
#pragma unroll
  for (int q = 0; q < COUNTERS / 1024; q++) {
    uint32_t c = 0;
#pragma unroll
    for (int r = 0; r < CLUSTER; r++) c += cl.map_shared_rank(&sm, r)->part_cnt[q * 1024 + t];
    best[q] = (c << COUNTERS_LOG) | uint32_t(q * 1024 + t);
  }
  const uint32_t least = max(4 * SAMPLES / COUNTERS, uint32_t(float(BIG / 2) * float(a.nsamples) / float(a.n)));
  uint32_t at[FREQUENT];
#pragma unroll
  for (int h = 0; h < FREQUENT; h++) {
    uint32_t m = 0;
#pragma unroll
    for (int q = 0; q < COUNTERS / 1024; q++) m = max(m, best[q]);
    m = __reduce_max_sync(0xffffffffu, m);
    if (lane == 0) sm.warp[warp] = m;
    __syncthreads();
    m = __reduce_max_sync(0xffffffffu, sm.warp[lane]);
    __syncthreads();
    at[h] = (m >> COUNTERS_LOG) >= least ? m & uint32_t(COUNTERS - 1) : NONE;
#pragma unroll
    for (int q = 0; q < COUNTERS / 1024; q++)
      if (best[q] == m) best[q] = 0;
  }
  // A quarter of the sample votes.
  constexpr int BITS = int(sizeof(KeyT)) * 8;
#pragma unroll
  for (int u = 0; u < (U + 3) / 4; u++) {
    const uint32_t mine = (live >> u) & 1u ? counter_of(key[u]) : NONE - 1;
#pragma unroll
    for (int h = 0; h < FREQUENT; h++) {
      const uint32_t who = __ballot_sync(0xffffffffu, mine == at[h]);
      if (!who) continue;
      if (lane == 0) atomicAdd(&voters[h], uint32_t(__popc(who)));
      for (int bit = 0; bit < BITS; bit++) {
        const uint32_t ones = who & __ballot_sync(0xffffffffu, (key[u] >> bit) & 1);
        if (lane == (bit & 31) && ones) atomicAdd(&votes[h * 64 + bit], uint32_t(__popc(ones)));
      }
    }
  }
  cl.sync();
  if (t < FREQUENT * 64) {
    uint32_t yes = 0, all = 0;
#pragma unroll
    for (int r = 0; r < CLUSTER; r++) {
      const PlanShared* o = cl.map_shared_rank(&sm, r);
      yes += o->group[t];
      all += o->group[FREQUENT * 64 + (t >> 6)];
    }
    const uint32_t w = __ballot_sync(0xffffffffu, 2 * yes > all);
    if (lane == 0) words[t >> 5] = w;
  }
  __syncthreads();
  // Ascending; keys of different counters differ.
  KeyT found[FREQUENT];
  uint32_t n = 0, hit = 0;
#pragma unroll
  for (int h = 0; h < FREQUENT; h++) {
    const KeyT k = KeyT(uint64_t(words[2 * h]) | (uint64_t(words[2 * h + 1]) << 32));
    found[h] = k;
    if (at[h] == NONE || counter_of(k) != at[h]) continue;
    uint32_t before = 0;
#pragma unroll
    for (int g = 0; g < FREQUENT; g++) {
      const KeyT o = KeyT(uint64_t(words[2 * g]) | (uint64_t(words[2 * g + 1]) << 32));
      if (g != h && at[g] != NONE && counter_of(o) == at[g] && o < k) before++;
    }
    if (t == 0 && cl.block_rank() == 0) a.st->key[before] = k;
    n++;
#pragma unroll
    for (int u = 0; u < U; u++)
      if (((live >> u) & 1u) && key[u] == k) hit |= 1u << u;
  }
  if (t == 0 && cl.block_rank() == 0) a.st->nkeys = n;
  __syncthreads();                                 // the borrowed arrays are free
  return hit;
}

template <typename KeyT, bool FREQ = false>
__device__ __forceinline__ void buckets_body(const ColView& col, const Args& a) {
  namespace cg = cooperative_groups;
  cg::cluster_group cl = cg::this_cluster();
  __shared__ PlanShared sm;
  const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
  const uint32_t rank = cl.block_rank();
  State* st = a.st;
  if (a.clear)
    for (uint64_t i = rank * 1024 + t; i < a.clear16; i += 1024 * CLUSTER) a.clear[i] = make_uint4(0, 0, 0, 0);
  cl.sync();                             // every CTA runs before its shared memory is written; the state is clear
  // The sample: one row of each nsamples-th part of the column, at a mixed offset (no period of the data
  // lines up), or every row. nsamples is SAMPLES or the rows.
  constexpr int U = SAMPLES / (1024 * CLUSTER);
  KeyT key[U];
  uint32_t live = 0, nulls = 0, nans = 0;
  const bool full = a.nsamples == a.n;
#pragma unroll
  for (int u = 0; u < U; u++) {
    const uint32_t j = (rank * U + u) * 1024 + t;
    key[u] = 0;
    if (j < a.nsamples) {
      uint64_t row = j;
      if (!full) {
        const uint64_t lo = uint64_t(j) * a.n / SAMPLES, hi = uint64_t(j + 1) * a.n / SAMPLES;
        uint32_t h = j * 2654435761u;
        h ^= h >> 15;
        h *= 2246822519u;
        h ^= h >> 13;
        row = lo + __umulhi(h, uint32_t(hi - lo));
      }
      int cat = 0;
      if (a.src_ids) {
        key[u] = static_cast<const KeyT*>(a.src_keys)[row];
      } else {
        const bool valid = !col.valid || bit_at(col.valid, col.valid_off + int64_t(row));
        key[u] = key_from_raw<KeyT>(col, load_raw<KeyT>(col, row), valid, cat);
      }
      if (cat == 0) live |= 1u << u;
      else if (cat == 1) nans |= 1u << u;
      else nulls |= 1u << u;
    }
  }
  if constexpr (FREQ) live &= ~take_frequent<KeyT, U>(a, sm, key, live);
  for (int i = t; i < COARSE; i += 1024) sm.coarse_cnt[i] = 0;
  for (int i = t; i < 4 * FINE; i += 1024) sm.part_cnt[i] = 0;
  // The sampled range, over the cluster.
  {
    uint64_t mx = 0, mn = 0;
#pragma unroll
    for (int u = 0; u < U; u++)
      if ((live >> u) & 1u) {
        mx = max(mx, uint64_t(key[u]));
        mn = max(mn, ~uint64_t(key[u]));
      }
    mx = warp_max_u64(mx);
    mn = warp_max_u64(mn);
    const uint32_t c = __reduce_add_sync(0xffffffffu, __popc(live));
    if (lane == 0) {
      sm.wmax[warp] = mx;
      sm.wmin[warp] = mn;
      sm.warp[warp] = c;
    }
    __syncthreads();
    if (warp == 0) {
      const uint64_t bx = warp_max_u64(sm.wmax[lane]), bn = warp_max_u64(sm.wmin[lane]);
      const uint32_t bc = __reduce_add_sync(0xffffffffu, sm.warp[lane]);
      if (lane < CLUSTER) {
        PlanShared* o = cl.map_shared_rank(&sm, lane);
        o->smax[rank] = bx;
        o->smin[rank] = bn;
        o->scnt[rank] = bc;
      }
    }
  }
  cl.sync();
  uint64_t vmax = 0, vmin_inv = 0;
  uint32_t sv = 0;
#pragma unroll
  for (int r = 0; r < CLUSTER; r++) {
    vmax = max(vmax, uint64_t(sm.smax[r]));
    vmin_inv = max(vmin_inv, uint64_t(sm.smin[r]));
    sv += uint32_t(sm.scnt[r]);
  }
  const unsigned long long lo = sv ? ~vmin_inv : 0ull, span = sv ? vmax - lo : 0ull;
  auto give_up = [&] {
    if (rank == 0 && t == 0) {
      st->mode = MODE_FALLBACK;
      sm.mode = MODE_FALLBACK;
    }
  };
  if (!a.one_launch && a.n >= FEW_DIGITS_ROWS && sv && span < FEW_DIGITS_SPAN) {
    give_up();
    return;
  }
  const int bits = max(COARSE_BITS, span ? 64 - __clzll((long long)span) : 0);
  const uint32_t shc = uint32_t(bits - COARSE_BITS);        // key bits below a coarse cell
  const Map<KeyT> map{KeyT(lo), KeyT(span), uint32_t(sizeof(KeyT)) * 8u - uint32_t(bits), 0u, 0u};
#pragma unroll
  for (int u = 0; u < U; u++)
    if ((live >> u) & 1u) atomicAdd(&sm.coarse_cnt[uint32_t(KeyT(key[u] - map.lo) >> shc)], 1u);
  const bool count_pairs = sizeof(KeyT) == 4 && a.n >= PAIRS_ROWS;
  if (count_pairs) {
    // Sampled keys that meet an equal one of the CTA's, in a table of the last key at each place.
    uint32_t pairs = 0;
#pragma unroll
    for (int u = 0; u < U; u++)
      if ((live >> u) & 1u) {
        const uint32_t k = uint32_t(key[u]);
        pairs += atomicExch(&sm.part_cnt[__umulhi(k * 2654435761u, uint32_t(4 * FINE))], k) == k ? 1u : 0u;
      }
    pairs = __reduce_add_sync(0xffffffffu, pairs);
    if (lane == 0) sm.warp[warp] = pairs;
    __syncthreads();
    pairs = __reduce_add_sync(0xffffffffu, sm.warp[lane]);
    if (t < CLUSTER) cl.map_shared_rank(&sm, t)->pairs[rank] = pairs;
  }
  cl.sync();
  if (count_pairs) {
    uint32_t pairs = 0;
#pragma unroll
    for (int r = 0; r < CLUSTER; r++) pairs += sm.pairs[r];
    if (float(pairs) * float(a.n) > PAIRS_LIMIT) {
      give_up();
      return;
    }
    for (int i = t; i < 4 * FINE; i += 1024) sm.part_cnt[i] = 0;
  }
  uint32_t in_cell = 0;                  // the sample's keys in coarse cell t
  if (t < COARSE) {
#pragma unroll
    for (int r = 0; r < CLUSTER; r++) in_cell += cl.map_shared_rank(&sm, r)->coarse_cnt[t];
  }
  bool planned = false;
  if (t == 0) sm.linear = 0;
  // Evenly spread keys (every coarse cell's count within 4.5 deviations of its width's share) need no
  // tables: equal cuts of the range, filled to TARGET rows (a deviation the test cannot see still
  // fits CAP).
  {
    uint32_t off = 0;
    if (t < COARSE) {
      const unsigned long long c0 = (unsigned long long)t << shc, w = 1ull << shc;
      const float keys_in = c0 > span ? 0.0f : span - c0 >= w ? float(w) : float(span - c0) + 1.0f;
      const float e = float(sv) * keys_in / (float(span) + 1.0f);
      off = fabsf(float(in_cell) - e) > 4.5f * sqrtf(e) + 3.0f ? 1u : 0u;
    }
    const bool even = !__syncthreads_or(int(off)) && sv >= 16u * COARSE && shc > 0;
    if (even) {
      const float est = float(a.n) * float(sv) / float(a.nsamples);
      const float range = bits == 64 ? 18446744073709551616.0f : float(1ull << bits);
      const uint32_t cuts = uint32_t(ceilf(est / float(TARGET) * (range / (float(span) + 1.0f))));
      const uint32_t top = uint32_t(KeyT(KeyT(span) << map.up) >> (8 * sizeof(KeyT) - 32));
      const uint32_t nb = __umulhi(top, cuts) + 3u;
      if (nb <= a.bucket_cap) {
        for (uint32_t b = rank * 1024 + t; b < nb; b += 1024 * CLUSTER) {
          const bool outer = b == 0 || b == nb - 1;
          a.bmeta[b] = META_SPLIT | (outer ? 0u : cuts);
          a.bfirst[b] = (outer ? 0xFFFFu : map.up) << 16;
        }
        if (t == 0 && rank == 0) {
          sm.linear = cuts;
          sm.buckets = nb;
          sm.mode = MODE_BUCKETS;
          tell_plan(a, lo, span, map.up, nb, cuts);
        }
        planned = true;
      }
    }
  }
  if (!planned && !a.one_launch) {
    // A key with more rows than a bucket may hold ends the attempt here: the sample's keys counted by a hash.
    constexpr int COUNTERS = 2048;
    static_assert(COUNTERS <= 4 * FINE && COUNTERS % 1024 == 0, "they borrow the quarters' counters");
    __syncthreads();
#pragma unroll
    for (int u = 0; u < U; u++)
      if ((live >> u) & 1u) atomicAdd(&sm.part_cnt[uint32_t((uint64_t(key[u]) * 0x9E3779B97F4A7C15ull) >> 53)], 1u);
    // Over the cluster where a bucket may hold few of the sample's keys; of a shorter column each CTA's own
    // keys tell (two cluster barriers and the remote counts less: 5 us of a 1M-row sort).
    const bool whole = a.n >= WHOLE_SAMPLE_ROWS;
    if (whole) cl.sync();
    else __syncthreads();
    uint32_t most = 0;
#pragma unroll
    for (int q = 0; q < COUNTERS / 1024; q++) {
      uint32_t c = 0;
      if (whole) {
#pragma unroll
        for (int r = 0; r < CLUSTER; r++) c += cl.map_shared_rank(&sm, r)->part_cnt[q * 1024 + t];
      } else {
        c = sm.part_cnt[q * 1024 + t];
      }
      most = max(most, c);
    }
    most = __reduce_max_sync(0xffffffffu, most);
    if (lane == 0) sm.warp[warp] = most;
    __syncthreads();
    most = __reduce_max_sync(0xffffffffu, sm.warp[lane]);
    if (t < CLUSTER) cl.map_shared_rank(&sm, t)->pairs[rank] = most;
    cl.sync();
    most = 0xFFFFFFFFu;                            // what every CTA saw
#pragma unroll
    for (int r = 0; r < CLUSTER; r++) most = min(most, sm.pairs[r]);
    const float c = float(most), seen = whole ? float(a.nsamples) : float(a.nsamples) / CLUSTER;
    const float others = (whole ? float(sv) : float(sv) / CLUSTER) / COUNTERS;
    if ((c - others - 3.0f * sqrtf(c)) * float(a.n) > float(a.large) * seen) {
      give_up();
      return;
    }
    for (int i = t; i < COUNTERS; i += 1024) sm.part_cnt[i] = 0;
    __syncthreads();
  }
  if (!planned) {
    // Fine cells of each coarse cell: 2^fb, from its share of the sample (about FINE_GOAL cells over the
    // column, fewer when the sample is small: at least 24 sampled rows a cell on average).
    const uint32_t goal = min(uint32_t(FINE_GOAL), max(1u, sv / 24u));
    uint32_t fb = 0, width = 0;
    if (t < COARSE) {
      const uint32_t want = sv ? uint32_t(uint64_t(in_cell) * goal / sv) : 0u;
      fb = want > 1u ? 32u - __clz(want - 1u) : 0u;
      fb = min(fb, min(uint32_t(FINE_BITS), shc));
      width = 1u << fb;
    }
    uint32_t nfine;
    const uint32_t fbase = block_scan<1024>(width, sm.warp, nfine);
    if (t < COARSE) {
      sm.coarse[t] = fbase | (fb << 16);
      if (rank == 0) a.coarse[t] = sm.coarse[t];
    }
    __syncthreads();
#pragma unroll
    for (int u = 0; u < U; u++)
      if ((live >> u) & 1u) {
        uint32_t f, frac;
        cell_of(map, sm.coarse, KeyT(key[u] - map.lo), f, frac);
        atomicAdd(&sm.part_cnt[4 * f + (frac >> 30)], 1u);
      }
    cl.sync();
    // Each CTA sums its share of the counts into the first one's.
    constexpr int SHARE = 4 * FINE / CLUSTER;
    static_assert(SHARE <= 1024 && 4 * FINE % CLUSTER == 0, "a count a thread");
    if (t < SHARE) {
      const int i = int(rank) * SHARE + t;
      uint32_t c = 0;
#pragma unroll
      for (int r = 0; r < CLUSTER; r++) c += cl.map_shared_rank(&sm, r)->part_cnt[i];
      cl.map_shared_rank(&sm, 0)->part_cnt[i] = c;
    }
    cl.sync();
    if (rank == 0) plan_cells<KeyT>(a, sm, map, lo, span, shc, sv, nfine, full);
  }
  cl.sync();                             // no CTA leaves, or goes on, before the plan stands
  if (!a.one_launch) return;

  // ---- a column of at most SAMPLES rows, every one of them in the cluster's registers: its counts and
  // moves too, without the launches of steps 2 and 3.
  const PlanShared* p0 = cl.map_shared_rank(&sm, 0);
  const uint32_t nb = p0->buckets, linear = p0->linear;
  bool go = p0->mode == MODE_BUCKETS;
  if (go && !linear)
    for (int i = t; i < FINE; i += 1024) sm.fine[i] = rank == 0 ? sm.fine[i] : p0->fine[i];
  if (t < int(ONE_CAP)) sm.bins[t] = 0;
  if (t == 0) sm.diff = 0;
  __syncthreads();
  const Map<KeyT> all{KeyT(lo), KeyT(span), map.up, nb - 1, linear};
  uint32_t slot[U];                      // bucket << 16 | place among the CTA's rows of it
  KeyT diff = 0;
#pragma unroll
  for (int u = 0; u < U; u++) {
    const bool is = (live >> u) & 1u;
    if (go && is) {
      const uint32_t b = bucket_of(all, sm.coarse, sm.fine, key[u]);
      slot[u] = (b << 16) | atomicAdd(&sm.bins[b], 1u);
      diff |= key[u] ^ KeyT(lo);
    }
    const uint32_t wn = __popc(__ballot_sync(0xffffffffu, (nulls >> u) & 1u));
    const uint32_t wx = __popc(__ballot_sync(0xffffffffu, (nans >> u) & 1u));
    if (lane == 0) {
      sm.cats[0][u * 32 + warp] = wn;
      sm.cats[1][u * 32 + warp] = wx;
    }
  }
  diff = warp_or<KeyT>(diff);
  if (lane == 0 && diff) atomicOr(&sm.diff, (unsigned long long)diff);
  __syncthreads();
  // Null and NaN rows before each (item, warp) of the CTA: rows in order, items first.
  uint32_t n_null, n_nan;
  const uint32_t mine_null = t < U * 32 ? sm.cats[0][t] : 0u, mine_nan = t < U * 32 ? sm.cats[1][t] : 0u;
  const uint32_t before_null = block_scan<1024>(mine_null, sm.warp, n_null);
  const uint32_t before_nan = block_scan<1024>(mine_nan, sm.warp, n_nan);
  if (t < U * 32) {
    sm.cats[0][t] = before_null;
    sm.cats[1][t] = before_nan;
  }
  if (t == 0) {
    sm.ncats[0] = n_null;
    sm.ncats[1] = n_nan;
  }
  cl.sync();
  uint32_t rows = 0, ahead = 0, null_at = 0, nan_at = 0, nn = 0, nx = 0;
  unsigned long long dall = 0;
  for (int r = 0; r < CLUSTER; r++) {
    const PlanShared* o = cl.map_shared_rank(&sm, r);
    const uint32_t c = t < int(ONE_CAP) ? o->bins[t] : 0u;
    if (uint32_t(r) < rank) ahead += c;
    rows += c;
    const uint32_t cn = o->ncats[0], cx = o->ncats[1];
    if (uint32_t(r) < rank) {
      null_at += cn;
      nan_at += cx;
    }
    nn += cn;
    nx += cx;
    dall |= o->diff;
  }
  uint32_t values;
  const uint32_t at = block_scan<1024>(rows, sm.warp, values);
  sm.start[t] = at + ahead;
  const uint32_t over = __syncthreads_or(int(rows > a.large));
  go = go && !over;
  if (rank == 0) {
    if (go && uint32_t(t) < nb) a.bpos[t] = at;
    if (t == 0) {
      st->n_value = values;
      st->n_null = nn;
      st->n_nan = nx;
      if (go) {
        a.bpos[nb] = values;
        uint32_t active = 0;
        for (uint32_t d = 0; d < sizeof(KeyT); d++) active += (dall >> (8 * d)) & 255u ? 1u : 0u;
        a.sum->value_rows = values;
        a.sum->null_rows = nn;
        a.sum->nan_rows = nx;
        a.sum->passes_run = active;
        a.sum->method = 2;
        a.sum->passes_total = uint32_t(sizeof(KeyT));
      } else {
        st->mode = MODE_FALLBACK;
      }
    }
  }
  if (go) {
    null_at += a.nulls_first ? 0u : values + nx;
    nan_at += a.nulls_first ? nn : values;
    const uint32_t lt = (1u << lane) - 1u;
#pragma unroll
    for (int u = 0; u < U; u++) {
      const uint32_t row = (rank * U + u) * 1024 + t;
      const bool isn = (nulls >> u) & 1u, isx = (nans >> u) & 1u;
      const uint32_t bn = __ballot_sync(0xffffffffu, isn), bx = __ballot_sync(0xffffffffu, isx);
      if ((live >> u) & 1u) {
        const uint32_t dst = sm.start[slot[u] >> 16] + (slot[u] & 0xFFFFu);
        if (dst < values) {
          static_cast<KeyT*>(a.keys[0])[dst] = key[u];
          if (a.has_payload) a.rec[0][dst] = build_record(a.pay, row);
          else if (a.ids[0]) a.ids[0][dst] = a.src_ids ? a.src_ids[row] : row;
        } else {
          atomicOr(a.err, ERR_BOUNDS);
        }
      } else if (isn || isx) {
        const uint32_t dst = isn ? null_at + sm.cats[0][u * 32 + warp] + __popc(bn & lt)
                                 : nan_at + sm.cats[1][u * 32 + warp] + __popc(bx & lt);
        if (dst < a.n) {
          store_id(a, dst, row);
          store_category_rank(a, row, dst, isn, values, nn, nx);
          if (a.has_payload) unpack_record(a.pay, build_record(a.pay, row), dst);
          if (a.key_out) store_width(a.key_out, dst, pt_bytes(a.key_pt), source_bits(a, row));
        } else {
          atomicOr(a.err, ERR_BOUNDS);
        }
      }
    }
  }
  cl.sync();                             // no CTA leaves while another reads its counts
}

// ---- 2. exact counts

// Bucket starts, cursors, the chunks' null and NaN starts, and the decision: by one cluster, or, up to FUSED_BUCKETS
// of them, by the count's last CTA (one launch less).
template <typename KeyT, int CTAS>
__device__ __forceinline__ void starts_body(const Args& a) {
  namespace cg = cooperative_groups;
  cg::cluster_group cl = cg::this_cluster();
  __shared__ uint32_t s_warp[32], s_sum[CLUSTER], s_max[CLUSTER];
  State* st = a.st;
  if (CTAS > 1) {
    if (a.one_launch || a.bucket_cap <= FUSED_BUCKETS || st->mode != MODE_BUCKETS) return;
    cl.sync();                           // every CTA runs before its shared memory is written
  }
  constexpr uint32_t PER = 8;
  static_assert(MAX_BUCKETS <= CLUSTER * 1024 * PER && FUSED_BUCKETS <= 1024 * PER, "one round takes every bucket");
  const uint32_t t = threadIdx.x, lane = t & 31u, warp = t >> 5, rank = CTAS > 1 ? cl.block_rank() : 0u;
  const uint32_t nb = st->buckets, s2 = st->s2;
  // CTA r takes the r-th of equal shares (a multiple of PER), a thread PER buckets in a row.
  const uint32_t share = (nb + CTAS * PER - 1) / (CTAS * PER) * PER;
  const uint32_t b = rank * share + t * PER;
  uint32_t c[PER], sum = 0, big = 0;
#pragma unroll
  for (uint32_t q = 0; q < PER; q++) {
    c[q] = t * PER < share && b + q < nb ? __ldcg(a.bcount + b + q) : 0u;
    sum += c[q];
    big = max(big, c[q]);
  }
  uint32_t tot;
  uint32_t at = block_scan<1024>(sum, s_warp, tot);
  big = __reduce_max_sync(0xffffffffu, big);
  __syncthreads();
  if (lane == 0) s_warp[warp] = big;
  __syncthreads();
  big = __reduce_max_sync(0xffffffffu, s_warp[lane]);
  if (CTAS > 1) {
    if (t < uint32_t(CTAS)) {
      cl.map_shared_rank(s_sum, t)[rank] = tot;
      cl.map_shared_rank(s_max, t)[rank] = big;
    }
    cl.sync();
  } else {
    if (t == 0) {
      s_sum[0] = tot;
      s_max[0] = big;
    }
    __syncthreads();
  }
  uint32_t carry = 0;
  for (uint32_t r = 0; r < uint32_t(CTAS); r++) {
    if (r < rank) at += s_sum[r];
    carry += s_sum[r];
    big = max(big, s_max[r]);
  }
#pragma unroll
  for (uint32_t q = 0; q < PER; q++) {
    if (t * PER < share && b + q < nb) {
      a.bpos[b + q] = at;
      a.cursor2[size_t(b + q) * CUR_PAD] = at;
      if (((b + q) & ((1u << s2) - 1u)) == 0u) a.cursor1[size_t((b + q) >> s2) * CUR_PAD] = at;
      at += c[q];
    }
  }
  if (rank != 0) return;
  uint32_t all;
  const uint32_t nulls = t < a.nchunks ? __ldcg(a.chunk_cats + CATS * t) : 0u;
  const uint32_t nans = t < a.nchunks ? __ldcg(a.chunk_cats + CATS * t + 1) : 0u;
  const uint32_t null0 = block_scan<1024>(nulls, s_warp, all);
  const uint32_t nan0 = block_scan<1024>(nans, s_warp, all);
  if (t < a.nchunks) {
    a.chunk_cats[CATS * t] = null0;
    a.chunk_cats[CATS * t + 1] = nan0;
  }
  uint32_t apart = 0;                    // rows of the frequent keys
  for (uint32_t h = 0; h < st->nkeys; h++) {
    const uint32_t rows = t < a.nchunks ? __ldcg(a.chunk_cats + CATS * t + 2 + h) : 0u;
    const uint32_t before = block_scan<1024>(rows, s_warp, all);
    if (t < a.nchunks) a.chunk_cats[CATS * t + 2 + h] = __ldcg(&st->key_at[h]) + before;
    if (t == 0) st->key_rows[h] = all;
    apart += all;
  }
  if (t == 0) {
    const uint32_t n_value = __ldcg(&st->n_value);
    a.bpos[nb] = carry;
    st->max_bucket = big;
    if (carry + apart != n_value) atomicOr(a.err, ERR_BOUNDS);
    if (big > a.large || carry + apart != n_value) {
      st->mode = MODE_FALLBACK;
    } else {
      // The counters: no digit pass runs; the key's digits that vary stand in for them.
      uint32_t active = 0;
      for (uint32_t d = 0; d < sizeof(KeyT); d++) active += (__ldcg(&st->diff) >> (8 * d)) & 255u ? 1u : 0u;
      a.sum->value_rows = n_value;
      a.sum->null_rows = __ldcg(&st->n_null);
      a.sum->nan_rows = __ldcg(&st->n_nan);
      a.sum->passes_run = active;
      a.sum->method = 2;
      a.sum->passes_total = uint32_t(sizeof(KeyT));
    }
  }
}

// One read of the column (63 us for 45M keys and 16,384 bins on a B200: the HBM copy rate). Each CTA
// takes consecutive chunks; a chunk's level-1 counts are the growth of its bins' sums over the chunk.
template <typename KeyT, bool FREQ = false>
__device__ __forceinline__ void histogram_body(const ColView& col, const Args& a) {
  extern __shared__ __align__(16) unsigned char hsm[];
  State* st = a.st;
  if (blockIdx.x >= a.hist_grid || st->mode != MODE_BUCKETS) return;
  uint32_t* bins = reinterpret_cast<uint32_t*>(hsm);
  __shared__ uint32_t coarse[COARSE], fine[FINE], prev[BINS1];
  __shared__ uint32_t s_null, s_nan, s_rows[FREQUENT];
  __shared__ KeyT s_key[FREQUENT];
  __shared__ unsigned long long s_or;
  const uint32_t nb = st->buckets, s2 = st->s2, nbins = st->bins1, nkeys = FREQ ? st->nkeys : 0u;
  load_tables(a, coarse, fine);
  if (threadIdx.x < uint32_t(FREQUENT)) {
    s_key[threadIdx.x] = KeyT(st->key[threadIdx.x]);
    s_rows[threadIdx.x] = 0;
  }
  for (uint32_t i = threadIdx.x; i < nb; i += HTHREADS) bins[i] = 0;
  for (int i = threadIdx.x; i < BINS1; i += HTHREADS) prev[i] = 0;
  if (threadIdx.x == 0) {
    s_null = 0;
    s_nan = 0;
    s_or = 0;
  }
  __syncthreads();
  const Map<KeyT> map = load_map<KeyT>(st);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  KeyT diff = 0;                        // bits that differ from lo's in some key
  uint32_t values = 0, all_null = 0, all_nan = 0;
  uint32_t below[FREQUENT] = {};        // value rows before each frequent key
  const uint32_t c0 = uint32_t(uint64_t(blockIdx.x) * a.nchunks / a.hist_grid);
  const uint32_t c1 = uint32_t(uint64_t(blockIdx.x + 1) * a.nchunks / a.hist_grid);
  for (uint32_t c = c0; c < c1; c++) {
    const uint64_t first = uint64_t(c) * a.chunk_rows, end = min(a.n, first + a.chunk_rows);
    uint32_t n_null = 0, n_nan = 0, n_key[FREQUENT] = {};
    for (uint64_t w0 = first + uint64_t(warp) * (HITEMS * 32); w0 < end; w0 += HTHREADS * HITEMS) {
      RawTile<KeyT, HITEMS> r;
      uint32_t is_value, is_null, is_nan;
      load_tile(col, w0, end, r);
      encode_tile(col, w0, end, r, is_value, is_null, is_nan);
      values += __popc(is_value);
      n_null += __popc(is_null);
      n_nan += __popc(is_nan);
      if (nkeys) {
        uint32_t apart = 0;
#pragma unroll
        for (int h = 0; h < FREQUENT; h++) {
          if (uint32_t(h) >= nkeys) break;
          const KeyT k = s_key[h];
          uint32_t same = 0, less = 0;
#pragma unroll
          for (int i = 0; i < HITEMS; i++) {
            same |= uint32_t(r.key[i] == k) << i;
            less |= uint32_t(r.key[i] < k) << i;
          }
          same &= is_value;
          below[h] += __popc(less & is_value);
          n_key[h] += __popc(same);
          if (same) diff |= k ^ map.lo;
          apart |= same;
        }
        is_value &= ~apart;
      }
#pragma unroll
      for (int i = 0; i < HITEMS; i++) {
        if (!((is_value >> i) & 1u)) continue;
        diff |= r.key[i] ^ map.lo;
        atomicAdd(bins + bucket_of(map, coarse, fine, r.key[i]), 1u);
      }
    }
    n_null = __reduce_add_sync(0xffffffffu, n_null);
    n_nan = __reduce_add_sync(0xffffffffu, n_nan);
    if (lane == 0) {
      if (n_null) atomicAdd(&s_null, n_null);
      if (n_nan) atomicAdd(&s_nan, n_nan);
    }
#pragma unroll
    for (int h = 0; h < FREQUENT; h++) {
      if (uint32_t(h) >= nkeys) break;
      const uint32_t rows = __reduce_add_sync(0xffffffffu, n_key[h]);
      if (lane == 0 && rows) atomicAdd(&s_rows[h], rows);
    }
    __syncthreads();
    if (s2 == 0) {
      for (uint32_t d = threadIdx.x; d < nbins; d += HTHREADS) {
        a.chunk_bins[size_t(c) * BINS1 + d] = bins[d] - prev[d];
        prev[d] = bins[d];
      }
    } else {
      for (uint32_t d = warp; d < nbins; d += HTHREADS / 32) {
        uint32_t sum = 0;
#pragma unroll
        for (uint32_t q = 0; q < BINS2; q += 32) {
          const uint32_t b = (d << S2) + q + lane;
          sum += b < nb ? bins[b] : 0u;
        }
        sum = __reduce_add_sync(0xffffffffu, sum);
        if (lane == 0) {
          a.chunk_bins[size_t(c) * BINS1 + d] = sum - prev[d];
          prev[d] = sum;
        }
      }
    }
    if (threadIdx.x == 0) {
      a.chunk_cats[CATS * c] = s_null;
      a.chunk_cats[CATS * c + 1] = s_nan;
      for (uint32_t h = 0; h < nkeys; h++) {
        a.chunk_cats[CATS * c + 2 + h] = s_rows[h];
        s_rows[h] = 0;
      }
      all_null += s_null;
      all_nan += s_nan;
      s_null = 0;
      s_nan = 0;
    }
    __syncthreads();
  }
  diff = warp_or<KeyT>(diff);
  values = __reduce_add_sync(0xffffffffu, values);
  if (lane == 0) {
    atomicOr(&s_or, (unsigned long long)diff);
    if (values) atomicAdd(&st->n_value, values);
  }
#pragma unroll
  for (int h = 0; h < FREQUENT; h++) {
    if (uint32_t(h) >= nkeys) break;
    const uint32_t rows = __reduce_add_sync(0xffffffffu, below[h]);
    if (lane == 0 && rows) atomicAdd(&st->key_at[h], rows);
  }
  __syncthreads();
  for (uint32_t i = threadIdx.x; i < nb; i += HTHREADS)
    if (bins[i]) atomicAdd(a.bcount + i, bins[i]);
  if (threadIdx.x == 0) {
    if (all_null) atomicAdd(&st->n_null, all_null);
    if (all_nan) atomicAdd(&st->n_nan, all_nan);
    atomicOr(&st->diff, s_or);
  }
  if (a.bucket_cap <= FUSED_BUCKETS) {
    __shared__ uint32_t s_last;
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) s_last = atomicAdd(&st->counted, 1u) == a.hist_grid - 1 ? 1u : 0u;
    __syncthreads();
    if (!s_last) return;
    __threadfence();
    starts_body<KeyT, 1>(a);
  }
}

// ---- 3. rows to their buckets

template <typename KeyT, int PAY>
struct TileShared {
  static constexpr int NB = PAY ? BINS1 / 2 : BINS1;
  uint32_t coarse[COARSE], fine[FINE];
  // Rows of the tile per bin, then the bins' starts in it; what added to a row's place in the tile gives
  // its destination; the chunk's next destination in each bin.
  uint32_t start[NB], delta[NB], at[NB];
  uint32_t warp[32];
  uint32_t cats[WARPS][2];
  uint32_t key_cats[WARPS][FREQUENT], key_at[FREQUENT];  // the frequent keys' rows by warp; their next places
  KeyT apart[FREQUENT];
  uint4 rec[PAY ? TILE : 1];
  KeyT key[TILE];
  // Per staged row: its bin, and without records (which hold the row id) its place in the tile below it.
  std::conditional_t<PAY != 0, uint16_t, uint32_t> word[TILE];
};

template <typename KeyT, int PAY, bool FREQ = false>
__device__ __forceinline__ void level1_body(const ColView& col, const Args& a) {
  extern __shared__ __align__(16) unsigned char tsm[];
  using SM = TileShared<KeyT, PAY>;
  SM& sm = *reinterpret_cast<SM*>(tsm);
  const State* st = a.st;
  if (blockIdx.x >= a.nchunks || st->mode != MODE_BUCKETS) return;
  const int t = threadIdx.x, warp = t >> 5, lane = t & 31;
  const uint32_t lt = (1u << lane) - 1u;
  const uint32_t s2 = st->s2, nbins = st->bins1;
  const Map<KeyT> map = load_map<KeyT>(st);
  load_tables(a, sm.coarse, sm.fine);
  const uint32_t c = blockIdx.x;
  const uint64_t first = uint64_t(c) * a.chunk_rows, end = min(a.n, first + a.chunk_rows);
  // The chunk's share of every bin, reserved once (chunks reserve in any order).
  for (int d = t; d < SM::NB; d += THREADS) {
    uint32_t at = 0;
    if (uint32_t(d) < nbins) {
      const uint32_t mine = a.chunk_bins[size_t(c) * BINS1 + d];
      if (mine) at = atomicAdd(a.cursor1 + size_t(d) * CUR_PAD, mine);
    }
    sm.at[d] = at;
    sm.start[d] = 0;
  }
  const bool cats = col.valid || col.nan_cat;
  uint32_t null_at = a.chunk_cats[CATS * c], nan_at = a.chunk_cats[CATS * c + 1];
  const uint32_t nkeys = FREQ ? st->nkeys : 0u;
  const uint32_t nv = st->n_value, nn = st->n_null, nx = st->n_nan;
  null_at += a.nulls_first ? 0u : nv + nx;
  nan_at += a.nulls_first ? nn : nv;
  if (uint32_t(t) < nkeys) {
    sm.key_at[t] = a.chunk_cats[CATS * c + 2 + t] + (a.nulls_first ? nn + nx : 0u);
    sm.apart[t] = KeyT(st->key[t]);
  }
  KeyT* __restrict__ kout = static_cast<KeyT*>(a.keys[0]);
  uint32_t* __restrict__ iout = a.ids[0];
  uint4* __restrict__ rout = a.rec[0];
  const uint32_t wofs = uint32_t(warp) * (ITEMS * 32) + uint32_t(lane);
  const bool direct = PAY && a.pay.pair;           // the payload words are two columns as they are
  const uint64_t* wsrc = direct ? static_cast<const uint64_t*>(a.pay.src[a.pay.wide]) : nullptr;
  const uint32_t* hsrc = direct ? static_cast<const uint32_t*>(a.pay.src[a.pay.narrow]) : nullptr;
  RawTile<KeyT, ITEMS> r;
  uint64_t pw[PAY ? ITEMS : 1];
  uint32_t ph[PAY ? ITEMS : 1];
  auto load_rows = [&](uint64_t tile) {
    load_tile(col, tile + (wofs - lane), end, r);
    if constexpr (PAY) {
      if (direct) {
        const uint64_t* w = wsrc + tile + wofs;
        const uint32_t* h = hsrc + tile + wofs;
        const uint64_t left = end - tile;
#pragma unroll
        for (int i = 0; i < ITEMS; i++)
          if (wofs + i * 32 < left) {
            pw[i] = w[i * 32];
            ph[i] = h[i * 32];
          }
      }
    }
  };
  if (first < end) load_rows(first);
  __syncthreads();
  for (uint64_t tile = first; tile < end; tile += TILE) {
    uint32_t values, nulls, nans;
    encode_tile(col, tile + (wofs - lane), end, r, values, nulls, nans);
    uint32_t apart = 0;                 // items of a frequent key
    auto same_as = [&](KeyT k) {
      uint32_t same = 0;
#pragma unroll
      for (int i = 0; i < ITEMS; i++) same |= uint32_t(r.key[i] == k) << i;
      return same;
    };
    if (nkeys) {
      for (uint32_t h = 0; h < nkeys; h++) {
        const uint32_t same = same_as(sm.apart[h]) & values;
        const uint32_t rows = __reduce_add_sync(0xffffffffu, __popc(same));
        if (lane == 0) sm.key_cats[warp][h] = rows;
        apart |= same;
      }
      values &= ~apart;
    }
    uint32_t slot[ITEMS];               // bin << 16 | place among the tile's rows of the bin
#pragma unroll
    for (int i = 0; i < ITEMS; i++) {
      if (!((values >> i) & 1u)) continue;
      const uint32_t d = bucket_of(map, sm.coarse, sm.fine, r.key[i]) >> s2;
      slot[i] = (d << 16) | atomicAdd(&sm.start[d], 1u);
    }
    if (cats) {
      const uint32_t wn = __reduce_add_sync(0xffffffffu, __popc(nulls)), wx = __reduce_add_sync(0xffffffffu, __popc(nans));
      if (lane == 0) {
        sm.cats[warp][0] = wn;
        sm.cats[warp][1] = wx;
      }
    }
    __syncthreads();
    // The last tile's records have left shared memory before this one's are staged.
    if constexpr (PAY) bulk_wait_read();
    // Bin counts into starts: one or two bins a thread.
    constexpr int PER = SM::NB / THREADS;
    static_assert(PER == 1 || PER == 2, "bins a thread");
    const uint32_t c0 = sm.start[PER * t], c1 = PER == 2 ? sm.start[PER * t + PER - 1] : 0u;
    uint32_t tile_n;
    const uint32_t s0 = block_scan<THREADS>(c0 + c1, sm.warp, tile_n);
    const uint32_t at0 = sm.at[PER * t];
    sm.start[PER * t] = s0;
    sm.delta[PER * t] = at0 - s0;
    sm.at[PER * t] = at0 + c0;
    if constexpr (PER == 2) {
      const uint32_t at1 = sm.at[2 * t + 1];
      sm.start[2 * t + 1] = s0 + c0;
      sm.delta[2 * t + 1] = at1 - (s0 + c0);
      sm.at[2 * t + 1] = at1 + c1;
    }
    __syncthreads();
#pragma unroll
    for (int i = 0; i < ITEMS; i++) {
      if (!((values >> i) & 1u)) continue;
      const uint32_t pos = sm.start[slot[i] >> 16] + (slot[i] & 0xFFFFu);
      sm.key[pos] = r.key[i];
      if constexpr (PAY) {
        sm.word[pos] = uint16_t(slot[i] >> 16);
        const uint32_t row = uint32_t(tile) + wofs + uint32_t(i) * 32;
        sm.rec[pos] = direct ? make_uint4(row, uint32_t(pw[i]), uint32_t(pw[i] >> 32), ph[i]) : build_record(a.pay, row);
      } else {
        sm.word[pos] = (slot[i] & 0xFFFF0000u) | (wofs + i * 32);
      }
    }
    // Null and NaN rows wait behind the values, in row order: they go straight to their final places.
    uint32_t tn = 0, tx = 0;
    if (cats) {
      uint32_t wn = 0, wx = 0;
#pragma unroll
      for (int v = 0; v < WARPS; v++) {
        const uint2 q = *reinterpret_cast<const uint2*>(sm.cats[v]);
        if (v < warp) {
          wn += q.x;
          wx += q.y;
        }
        tn += q.x;
        tx += q.y;
      }
      // (A tile's rows are at most TILE: behind the values there is room for the others.) With a payload
      // their records wait there too, from the registers they were loaded to: read again from the columns
      // at the store, each row's 16 bytes cost two more 32-byte sectors (50M rows, 10% nulls: the step
      // 716 us, 682 so).
      auto stage = [&](uint32_t rows, uint32_t p) {
#pragma unroll
        for (int i = 0; i < ITEMS; i++) {
          const bool is = (rows >> i) & 1u;
          const uint32_t m = __ballot_sync(0xffffffffu, is);
          if (is) {
            const uint32_t at = p + __popc(m & lt);
            sm.word[at] = wofs + i * 32;
            if constexpr (PAY) {
              const uint32_t row = uint32_t(tile) + wofs + uint32_t(i) * 32;
              sm.rec[at] = direct ? make_uint4(row, uint32_t(pw[i]), uint32_t(pw[i] >> 32), ph[i]) : build_record(a.pay, row);
            }
          }
          p += __popc(m);
        }
      };
      if (tn) stage(nulls, tile_n + wn);
      if (tx) stage(nans, tile_n + tn + wx);
    }
    // The frequent keys' rows: straight to their places, from here.
    for (uint32_t h = 0; h < nkeys; h++) {
      uint32_t p = sm.key_at[h];
      for (int v = 0; v < warp; v++) p += sm.key_cats[v][h];
      const uint32_t same = same_as(sm.apart[h]) & apart;
#pragma unroll
      for (int i = 0; i < ITEMS; i++) {
        const bool is = (same >> i) & 1u;
        const uint32_t m = __ballot_sync(0xffffffffu, is);
        if (is) {
          const uint32_t dst = p + __popc(m & lt);
          if (dst < a.n) store_id(a, dst, uint32_t(tile) + wofs + uint32_t(i) * 32);
          else atomicOr(a.err, ERR_BOUNDS);
        }
        p += __popc(m);
      }
    }
    // The next tile's rows arrive while this one leaves.
    if (tile + TILE < end) load_rows(tile + TILE);
    if constexpr (PAY) fence_bulk();
    __syncthreads();
    if (uint32_t(t) < nkeys)
      for (int v = 0; v < WARPS; v++) sm.key_at[t] += sm.key_cats[v][t];
    if constexpr (PAY) {
      // Thread d sends bin d's records as one copy; it runs while the next tile is read and ranked.
      static_assert(PER == 1, "one bin a thread");
      if (c0) {
        if (at0 + c0 <= nv) bulk_store(rout + at0, sm.rec + s0, c0 * 16u);
        else atomicOr(a.err, ERR_BOUNDS);
      }
      bulk_commit();
    }
    const int nit = int(tile_n + THREADS - 1 - t) / THREADS;
#pragma unroll
    for (int i = 0; i < ITEMS; i++) {
      if (i >= nit) break;
      const uint32_t j = uint32_t(i) * THREADS + t;
      const uint32_t word = sm.word[j];
      const uint32_t dst = sm.delta[PAY ? word : word >> 16] + j;
      if (dst >= nv) {
        atomicOr(a.err, ERR_BOUNDS);
        continue;
      }
      kout[dst] = sm.key[j];
      if constexpr (!PAY)
        if (iout) iout[dst] = uint32_t(tile) + (word & 0xFFFFu);
    }
    for (uint32_t j = tile_n + t; j < tile_n + tn + tx; j += THREADS) {
      const uint32_t q = j - tile_n, row = uint32_t(tile) + sm.word[j];
      const uint32_t dst = q < tn ? null_at + q : nan_at + (q - tn);
      if (dst >= a.n) {
        atomicOr(a.err, ERR_BOUNDS);
        continue;
      }
      store_id(a, dst, row);
      if constexpr (!PAY) store_category_rank(a, row, dst, q < tn, nv, nn, nx);
      if constexpr (PAY) unpack_record(a.pay, sm.rec[j], dst);
      if (a.key_out) store_width(a.key_out, dst, pt_bytes(a.key_pt), source_bits(a, row));
    }
    null_at += tn;
    nan_at += tx;
    for (int d = t; d < SM::NB; d += THREADS) sm.start[d] = 0;
    __syncthreads();
  }
  if constexpr (PAY) bulk_wait_all();
}

template <typename KeyT, int PAY>
struct Tile2Shared {
  uint32_t coarse[COARSE], fine[FINE];
  uint32_t tiles[MAX_BUCKETS / BINS2 + 1];      // tiles before each level-1 bin
  uint32_t start[BINS2], delta[BINS2];
  uint32_t warp[32];
  std::conditional_t<PAY != 0, uint4, uint32_t> rec[TILE];      // records, or row ids
  KeyT key[TILE];
  uint8_t bin[TILE];
};

// Level 2: tiles of one level-1 bin's rows to its 256 buckets. A tile reserves its rows of a bucket with
// one atomic.
template <typename KeyT, int PAY>
__device__ __forceinline__ void level2_body(const Args& a) {
  extern __shared__ __align__(16) unsigned char tsm[];
  using SM = Tile2Shared<KeyT, PAY>;
  SM& sm = *reinterpret_cast<SM*>(tsm);
  const State* st = a.st;
  if (blockIdx.x >= a.level2_grid || st->mode != MODE_BUCKETS || st->s2 == 0) return;
  const int t = threadIdx.x, warp = t >> 5, lane = t & 31;
  const uint32_t nbins = st->bins1, nb = st->buckets, nv = st->n_value;
  const Map<KeyT> map = load_map<KeyT>(st);
  load_tables(a, sm.coarse, sm.fine);
  auto bin_start = [&](uint32_t d) { return a.bpos[min(d << S2, nb)]; };
  uint32_t ntiles;
  {
    const uint32_t rows = uint32_t(t) < nbins ? bin_start(t + 1) - bin_start(t) : 0u;
    const uint32_t before = block_scan<THREADS>((rows + TILE - 1) / TILE, sm.warp, ntiles);
    if (t <= int(MAX_BUCKETS / BINS2)) sm.tiles[t] = before;
  }
  const KeyT* __restrict__ kin = static_cast<const KeyT*>(a.keys[0]);
  KeyT* __restrict__ kout = static_cast<KeyT*>(a.keys[1]);
  const uint32_t t0 = uint32_t(uint64_t(blockIdx.x) * ntiles / a.level2_grid);
  const uint32_t t1 = uint32_t(uint64_t(blockIdx.x + 1) * ntiles / a.level2_grid);
  if (t < BINS2) sm.start[t] = 0;
  __syncthreads();
  uint32_t d = 0;
  if (t0 < t1) {                         // the bin of the first tile: the last one starting at or before it
    uint32_t l = 0, r = nbins;
    while (r - l > 1) {
      const uint32_t mid = (l + r) >> 1;
      if (sm.tiles[mid] <= t0) l = mid;
      else r = mid;
    }
    d = l;
  }
  using RecT = std::conditional_t<PAY != 0, uint4, uint32_t>;
  const RecT* __restrict__ rin = reinterpret_cast<const RecT*>(PAY ? static_cast<const void*>(a.rec[0]) : a.ids[0]);
  RecT* __restrict__ rout = reinterpret_cast<RecT*>(PAY ? static_cast<void*>(a.rec[1]) : a.ids[1]);
  KeyT key[ITEMS];
  // Tile q's first row and rows; its keys.
  uint32_t first = 0, tile_n = 0;
  int nit = 0;                          // this thread's rows of it: row i x THREADS + t, i < nit
  auto load = [&](uint32_t q) {
    while (d + 1 < nbins && sm.tiles[d + 1] <= q) d++;
    const uint32_t end = bin_start(d + 1);
    first = bin_start(d) + (q - sm.tiles[d]) * TILE;
    tile_n = min(uint32_t(TILE), end - first);
    nit = int((tile_n + THREADS - 1 - t) / THREADS);
    const KeyT* p = kin + first + t;
#pragma unroll
    for (int i = 0; i < ITEMS; i++) {
      if (i >= nit) break;
      key[i] = p[i * THREADS];
    }
  };
  if (t0 < t1) load(t0);
  for (uint32_t q = t0; q < t1; q++) {
    const uint32_t b0 = d << S2, row0 = first;
    const int ni = nit;
    uint32_t slot[ITEMS];
#pragma unroll
    for (int i = 0; i < ITEMS; i++) {
      if (i >= ni) break;
      const uint32_t b = (bucket_of(map, sm.coarse, sm.fine, key[i]) - b0) & uint32_t(BINS2 - 1);
      slot[i] = (b << 16) | atomicAdd(&sm.start[b], 1u);
    }
    RecT rec[ITEMS];
    const RecT* rp = rin + row0 + t;
#pragma unroll
    for (int i = 0; i < ITEMS; i++) {
      if (i >= ni || !rin) break;
      rec[i] = rp[i * THREADS];
    }
    __syncthreads();
    uint32_t run = 0, run_at = 0, run_dst = 0;    // this thread's bucket: rows, where in the tile, where to
    if (warp < BINS2 / 32) {
      // The buckets' starts in the tile: each of these warps its own 32 buckets after the ones before.
      if constexpr (PAY) bulk_wait_read();        // the last tile's records have left
      const uint32_t c = sm.start[t];
      uint32_t x = c, before = 0;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= o) x += y;
      }
      for (int v = 0; v < warp; v++) before += sm.start[v * 32 + lane];
      before = __reduce_add_sync(0xffffffffu, before);
      run = c;
      run_at = before + x - c;
      run_dst = c ? atomicAdd(a.cursor2 + size_t(b0 + t) * CUR_PAD, c) : 0u;
      sm.delta[t] = run_dst - run_at;
      asm volatile("bar.sync 1, %0;" ::"n"(BINS2) : "memory");
      sm.start[t] = run_at;
    }
    __syncthreads();
#pragma unroll
    for (int i = 0; i < ITEMS; i++) {
      if (i >= ni) break;
      const uint32_t b = slot[i] >> 16, pos = sm.start[b] + (slot[i] & 0xFFFFu);
      sm.key[pos] = key[i];
      if (rin) sm.rec[pos] = rec[i];
      sm.bin[pos] = uint8_t(b);
    }
    if (q + 1 < t1) load(q + 1);
    if constexpr (PAY) fence_bulk();
    __syncthreads();
    if constexpr (PAY) {
      if (run) {
        if (run_dst + run <= nv) bulk_store(rout + run_dst, sm.rec + run_at, run * 16u);
        else atomicOr(a.err, ERR_BOUNDS);
      }
      bulk_commit();
    }
    if (t < BINS2) sm.start[t] = 0;
#pragma unroll
    for (int i = 0; i < ITEMS; i++) {
      const uint32_t j = uint32_t(i) * THREADS + t;
      if (i >= ni) break;
      const uint32_t dst = sm.delta[sm.bin[j]] + j;
      if (dst >= nv) {
        atomicOr(a.err, ERR_BOUNDS);
        continue;
      }
      kout[dst] = sm.key[j];
      if constexpr (!PAY)
        if (rin) rout[dst] = sm.rec[j];
    }
    __syncthreads();
  }
  if constexpr (PAY) bulk_wait_all();
}

// ---- 4. each bucket in shared memory

constexpr int TIES_ID = 0, TIES_STRING = 1;

// Row a before row b, their keys being equal: by row id, or first by the strings behind them, eight bytes at a time.
// Of each string the first TIE_BYTES are looked at: where those of both agree and more follow, `far` says that the
// derived keys must order the column (one CTA would compare them for as long as they are: 4,000 rows of a shared
// 100 KB took 6e7 dependent reads a thread).
constexpr uint64_t TIE_BYTES = 512;
__device__ __forceinline__ uint64_t eight_bytes(const uint8_t* p) {          // big-endian, from any address; two aligned words
  const uintptr_t at = reinterpret_cast<uintptr_t>(p);
  const uint64_t* w = reinterpret_cast<const uint64_t*>(at & ~uintptr_t(7));
  const uint32_t sh = uint32_t(at & 7u) * 8u;
  const uint64_t v = sh ? (w[0] >> sh) | (w[1] << (64 - sh)) : w[0];
  return (uint64_t(__byte_perm(uint32_t(v), 0, 0x0123)) << 32) | __byte_perm(uint32_t(v >> 32), 0, 0x0123);
}
template <int TIES>
__device__ __forceinline__ bool tied_before(const StringTies& s, uint32_t a, uint32_t b, bool& far, bool strings_alone = false) {
  if constexpr (TIES == TIES_STRING) {
    uint64_t oa, ob, la, lb;
    if (s.wide) {
      const int64_t* o = static_cast<const int64_t*>(s.offsets);
      oa = uint64_t(o[a]);
      ob = uint64_t(o[b]);
      la = uint64_t(o[a + 1ull]) - oa;
      lb = uint64_t(o[b + 1ull]) - ob;
    } else {
      const int32_t* o = static_cast<const int32_t*>(s.offsets);
      oa = uint64_t(uint32_t(o[a]));
      ob = uint64_t(uint32_t(o[b]));
      la = uint64_t(uint32_t(o[a + 1ull])) - oa;
      lb = uint64_t(uint32_t(o[b + 1ull])) - ob;
    }
    const uint64_t n = la < lb ? la : lb, end = n < TIE_BYTES ? n : TIE_BYTES;
    uint64_t i = *s.chars;
    // Whole eight bytes of both strings, then single ones (a string's last word could end past the column's bytes).
    for (; i + 16 <= end; i += 8) {
      const uint64_t x = eight_bytes(s.bytes + oa + i), y = eight_bytes(s.bytes + ob + i);
      if (x != y) return (x < y) != (s.desc != 0);
    }
    for (; i < end; i++) {
      const uint8_t x = s.bytes[oa + i], y = s.bytes[ob + i];
      if (x != y) return (x < y) != (s.desc != 0);
    }
    if (n > end) far = true;
    if (la != lb) return (la < lb) != (s.desc != 0);
    if (strings_alone) return false;
  }
  return a < b;
}

// Two strings whose keys are equal are equal.
__device__ __forceinline__ bool same_string(const StringTies& s, uint32_t a, uint32_t b, bool& far) {
  return !tied_before<TIES_STRING>(s, a, b, far, true) && !tied_before<TIES_STRING>(s, b, a, far, true);
}

// What a CTA has at hand: a bucket of the map, or a part of a larger one (split_rows): rows whose positions
// come from their own keys' range (KIND_KEY), or rows of one key, placed by their ids (KIND_ID).
constexpr uint32_t KIND_BUCKET = 0, KIND_KEY = 1, KIND_ID = 2;
// Parts waiting, at most. A split of a large bucket leaves 3 x rows / 1,024 + 2 of them or fewer, one of at most CAP
// rows 2 x rows / 33 + 4, and one of those waiting is split at a time, at most nine deep (11 bits of the key's or the
// id's range each).
constexpr uint32_t PARTS = 256;
constexpr uint32_t PART_ROWS = CAP / 2;
static_assert(3 * LARGE / PART_ROWS + 2 * CAP / (MAX_BIN + 1) + 9 * 4 <= PARTS, "the parts of the largest bucket");
constexpr uint32_t MAX_PAIRED = 8;                 // rows a bin may hold for comparisons, of the buckets put off
constexpr uint32_t CROWD = MAX_PAIRED + 1;         // their crowded bins start at least so many rows apart

// A CTA's shared memory.
template <typename KeyT, int PAY, int TIES>
struct FastShared {
  uint64_t full;                        // the bucket's records have arrived
  uint32_t warp[32];
  uint32_t crowded;                     // some bin holds more than MAX_BIN rows
  uint32_t some_fast;                   // some bucket of the CTA was ordered by the fast form
  union {
    struct {
      alignas(16) uint32_t start[BINS / 2 + 4];     // rows per bin, then where each bin starts: 16 bits each
      uint64_t word[CAP];               // by bin: the row's position, and its id (strings: its place in the bucket) below it
    };
    struct {                            // in order:
      KeyT key[CAP];
      uint32_t id[PAY ? 1 : CAP];
      uint16_t place[PAY ? CAP : 2];    // the row's place in the bucket
    };
  };
  uint32_t in_id[TIES == TIES_STRING ? CAP : 1];      // the rows' ids, as they come
  alignas(16) uint4 rec[PAY ? CAP : 1]; // the rows' records, as they come
};
// The same of the buckets put off; and the keys and places of up to BIG strings' rows, in a bitonic sort.
template <typename KeyT>
struct SlowRows {
  KeyT key[BIG];
  uint16_t place[BIG];
};
template <typename KeyT, int PAY, int TIES = TIES_ID>
struct LaterShared {
  uint64_t full;
  uint32_t warp[32];
  unsigned long long red[3][NTHREADS / 32];
  uint32_t mixed[CAP / CROWD + 1];      // by crowded bin: its rows are at several positions
  // The waiting parts: first row; rows, buffers (bit 29) and kind (bits 30 and 31); the rows of their key, where it
  // is one (ranks).
  uint32_t part_at[PARTS], part_n[PARTS];
  uint32_t run_at[PAY ? 1 : PARTS], run_n[PAY ? 1 : PARTS];
  union {
    struct {
      union {
        struct {
          alignas(16) uint32_t start[BINS + 4];   // rows per bin, then where each bin starts
          uint32_t word[CAP];           // by bin: the row's position below its bin, then its place in the bucket
        };
        KeyT key[CAP];                  // in order
      };
      uint32_t id[PAY ? 1 : CAP];       // the rows' ids, as they come; then in order
      uint16_t place[CAP];              // the words' bins; then, in order, the rows' places in the bucket
      alignas(16) uint4 rec[PAY ? CAP : 1];       // the rows' records, as they come
    };
    std::conditional_t<TIES == TIES_STRING, SlowRows<KeyT>, uint32_t> slow;
  };
};

// Read and written as 16-byte vectors, and by bulk copies.
template <typename SM>
constexpr bool vectors_aligned() {
  return offsetof(SM, start) % 16 == 0 && offsetof(SM, rec) % 16 == 0;
}
static_assert(vectors_aligned<FastShared<uint32_t, 0, TIES_ID>>() && vectors_aligned<FastShared<uint64_t, 0, TIES_ID>>() &&
              vectors_aligned<FastShared<uint32_t, 1, TIES_ID>>() && vectors_aligned<FastShared<uint64_t, 1, TIES_ID>>() &&
              vectors_aligned<FastShared<uint64_t, 0, TIES_STRING>>() && vectors_aligned<LaterShared<uint32_t, 0>>() &&
              vectors_aligned<LaterShared<uint64_t, 0>>() && vectors_aligned<LaterShared<uint32_t, 1>>() &&
              vectors_aligned<LaterShared<uint64_t, 1>>() && vectors_aligned<LaterShared<uint64_t, 0, TIES_STRING>>(),
              "shared arrays read as vectors");

// Strings that differ behind many equal keys: bitonic sort of (key, the rest of the string, row id), the ids of
// equal keys read where the rows are.
template <int TIES, typename KeyT, typename IdOf>
__device__ __forceinline__ void bitonic_rows(KeyT* key, uint16_t* place, uint32_t size, const KeyT* in, IdOf&& id_of,
                                             const StringTies& ties, bool& far) {
  uint32_t p = 2;
  while (p < size) p <<= 1;
  for (uint32_t i = threadIdx.x; i < p; i += NTHREADS) {
    key[i] = i < size ? in[i] : KeyT(~KeyT(0));
    place[i] = uint16_t(i);             // places from `size` on come after every row
  }
  __syncthreads();
  for (uint32_t k = 2; k <= p; k <<= 1) {
    if (__syncthreads_or(int(far))) return;          // the order is not used
    for (uint32_t j = k >> 1; j > 0; j >>= 1) {
      for (uint32_t q = threadIdx.x; q < p / 2; q += NTHREADS) {
        const uint32_t i = 2 * q - (q & (j - 1)), l = i + j;
        const KeyT ki = key[i], kl = key[l];
        bool less = kl < ki;
        if (kl == ki) {
          const uint32_t pi = place[i], pl = place[l];
          less = pl >= size ? false : pi >= size ? true : tied_before<TIES>(ties, id_of(pl), id_of(pi), far);
        }
        if (less == ((i & k) == 0)) {
          key[i] = kl;
          key[l] = ki;
          const uint16_t pi = place[i];
          place[i] = place[l];
          place[l] = pi;
        }
      }
      __syncthreads();
    }
  }
}

// Smallest and largest of every thread's (lo, hi) and (lo2, hi2), to every thread.
__device__ __forceinline__ uint64_t warp_least(uint64_t v) {
  const uint32_t h = __reduce_min_sync(0xffffffffu, uint32_t(v >> 32));
  const uint32_t l = __reduce_min_sync(0xffffffffu, uint32_t(v >> 32) == h ? uint32_t(v) : ~0u);
  return (uint64_t(h) << 32) | l;
}
__device__ __forceinline__ uint32_t warp_least(uint32_t v) { return __reduce_min_sync(0xffffffffu, v); }
template <typename SM, typename T>
__device__ __forceinline__ void block_range(SM& sm, T& lo, T& hi, uint32_t& lo2, uint32_t& hi2) {
  lo = warp_least(lo);
  hi = T(~warp_least(T(~hi)));
  lo2 = warp_least(lo2);
  hi2 = ~warp_least(~hi2);
  __syncthreads();
  if ((threadIdx.x & 31) == 0) {
    const int w = threadIdx.x >> 5;
    sm.red[0][w] = lo;
    sm.red[1][w] = hi;
    sm.red[2][w] = (uint64_t(hi2) << 32) | lo2;
  }
  __syncthreads();
#pragma unroll
  for (int w = 0; w < NTHREADS / 32; w++) {
    lo = min(lo, T(sm.red[0][w]));
    hi = max(hi, T(sm.red[1][w]));
    lo2 = min(lo2, uint32_t(sm.red[2][w]));
    hi2 = max(hi2, uint32_t(sm.red[2][w] >> 32));
  }
}
// Shift that brings the top bit of `range` to bit 63 (0 for an empty range).
__device__ __forceinline__ uint32_t range_shift(uint64_t range) { return range ? uint32_t(__clzll((long long)range)) : 0u; }

// Rows per bin into the bins' starts, over all 2,048; true when some bin holds more than MAX_PAIRED rows.
template <typename SM>
__device__ __forceinline__ bool count_scan(SM& sm, uint32_t rows) {
  constexpr int PER = BINS / NTHREADS;
  const uint32_t t = threadIdx.x;
  uint4 c[PER / 4];
  uint32_t sum = 0, mx = 0, all;
#pragma unroll
  for (int q = 0; q < PER / 4; q++) {
    c[q] = *reinterpret_cast<const uint4*>(&sm.start[t * PER + 4 * q]);
    sum += c[q].x + c[q].y + c[q].z + c[q].w;
    mx = max(mx, max(max(c[q].x, c[q].y), max(c[q].z, c[q].w)));
  }
  uint32_t s = block_scan<NTHREADS>(sum, sm.warp, all);
#pragma unroll
  for (int q = 0; q < PER / 4; q++) {
    *reinterpret_cast<uint4*>(&sm.start[t * PER + 4 * q]) = make_uint4(s, s + c[q].x, s + c[q].x + c[q].y, s + c[q].x + c[q].y + c[q].z);
    s += c[q].x + c[q].y + c[q].z + c[q].w;
  }
  if (t == NTHREADS - 1) sm.start[BINS] = rows;
  return __syncthreads_or(int(mx > MAX_PAIRED)) != 0;
}

// A bucket too large for the fast form, cut into parts that fit it: its rows move to the other buffers
// (unused by then) by 2,048 bins over the range of their keys, or, all keys being equal, of their row ids;
// bins of more than `heavy` rows become parts of their own, the others share parts of at most CAP rows. A part that
// is still too large is split again by its own, 2,048 times smaller range, so every split ends. One CTA does
// it: the map's buckets are a thousand rows, and only a key repeated thousands of times makes a larger one.
// Adds the parts to the list; returns their number. Leaves sm.start dirty.
constexpr uint32_t NOT_SPLIT = ~0u;                // strings of one key that differ
template <typename KeyT, int PAY, int TIES, typename SM>
__device__ __forceinline__ uint32_t split_rows(SM& sm, const Args& a, uint32_t first, uint32_t size, uint32_t side, uint32_t kind,
                                            uint32_t heavy, uint32_t run_at, uint32_t run_n, uint32_t parts) {
  const uint32_t t = threadIdx.x;
  const KeyT* kin = static_cast<const KeyT*>(a.keys[side]) + first;
  KeyT* kout = static_cast<KeyT*>(a.keys[side ^ 1u]) + first;
  const bool ids = PAY || a.ids[0];              // else the rows' places stand in for them
  const uint32_t* iin = ids ? a.ids[side] + first : nullptr;
  uint32_t* iout = ids ? a.ids[side ^ 1u] + first : nullptr;
  const uint4* rin = a.rec[side] + first;
  uint4* rout = a.rec[side ^ 1u] + first;
  constexpr uint32_t U = 4, STEP = U * NTHREADS;
  uint64_t lo = ~0ull, hi = 0;
  uint32_t id0 = ~0u, id1 = 0;
  for (uint32_t r0 = t; r0 < size; r0 += STEP) {
#pragma unroll
    for (uint32_t u = 0; u < U; u++)
      if (r0 + u * NTHREADS < size) {
        const uint64_t k = kin[r0 + u * NTHREADS];
        const uint32_t id = PAY ? rin[r0 + u * NTHREADS].x : ids ? iin[r0 + u * NTHREADS] : r0 + u * NTHREADS;
        lo = min(lo, k);
        hi = max(hi, k);
        id0 = min(id0, id);
        id1 = max(id1, id);
      }
  }
  block_range(sm, lo, hi, id0, id1);
  const bool by_id = lo == hi;
  if (by_id) {
    if (kind != KIND_ID) {
      if constexpr (TIES == TIES_STRING) {
        bool differ = false, far = false;
        for (uint32_t r = t; r < size && !far; r += NTHREADS) differ |= !same_string(a.ties, iin[r], iin[0], far);
        if (far) a.st->mode = MODE_FALLBACK;
        if (__syncthreads_or(int(differ || far))) return NOT_SPLIT;
      }
      run_at = first;
      run_n = size;
    }
    lo = id0;
    hi = id1;
  }
  const uint32_t sh = range_shift(hi - lo);
  auto bin_of = [&](uint64_t x) { return uint32_t(((x - lo) << sh) >> (64 - BINS_LOG)); };
  auto axis = [&](uint32_t r) { return by_id ? uint64_t(PAY ? rin[r].x : ids ? iin[r] : r) : uint64_t(kin[r]); };
  for (uint32_t x = t; x < BINS; x += NTHREADS) sm.start[x] = 0;
  __syncthreads();
  for (uint32_t r0 = t; r0 < size; r0 += STEP) {
#pragma unroll
    for (uint32_t u = 0; u < U; u++)
      if (r0 + u * NTHREADS < size) atomicAdd(&sm.start[bin_of(axis(r0 + u * NTHREADS))], 1u);
  }
  __syncthreads();
  constexpr uint32_t PER = BINS / NTHREADS;
  {
    uint32_t c[PER], sum = 0, all;
#pragma unroll
    for (uint32_t q = 0; q < PER; q++) {
      c[q] = sm.start[t * PER + q];
      sum += c[q];
    }
    uint32_t s = block_scan<NTHREADS>(sum, sm.warp, all);
#pragma unroll
    for (uint32_t q = 0; q < PER; q++) {
      sm.start[t * PER + q] = s;
      sm.word[t * PER + q] = s;                    // the scatter's cursors
      s += c[q];
    }
    if (t == NTHREADS - 1) sm.start[BINS] = size;
  }
  __syncthreads();
  // A part starts at a bin of its own, after one, and where a window of PART_ROWS rows starts.
  uint32_t flags = 0, total;
#pragma unroll
  for (uint32_t q = 0; q < PER; q++) {
    const uint32_t b = t * PER + q, s = sm.start[b], e = sm.start[b + 1];
    const uint32_t p = b ? sm.start[b - 1] : 0u;
    if (b == 0 || e - s > heavy || s - p > heavy || s / PART_ROWS != p / PART_ROWS) flags |= 1u << q;
  }
  uint32_t at = parts + block_scan<NTHREADS>(uint32_t(__popc(flags)), sm.warp, total);
  if (parts + total > PARTS) {                     // ruled out by the bound on the parts
    if (t == 0) atomicOr(a.err, ERR_BOUNDS);
    return parts;
  }
#pragma unroll
  for (uint32_t q = 0; q < PER; q++)
    if ((flags >> q) & 1u) sm.part_at[at++] = first + sm.start[t * PER + q];
  __syncthreads();
  for (uint32_t p = t; p < total; p += NTHREADS) {
    const uint32_t end = p + 1 < total ? sm.part_at[parts + p + 1] : first + size;
    sm.part_n[parts + p] = (end - sm.part_at[parts + p]) | ((side ^ 1u) << 29) | ((by_id ? KIND_ID : KIND_KEY) << 30);
    if constexpr (!PAY) {
      sm.run_at[parts + p] = run_at;
      sm.run_n[parts + p] = run_n;
    }
  }
  for (uint32_t r0 = t; r0 < size; r0 += STEP) {
    KeyT k[U];
    uint32_t id[PAY ? 1 : U];
    uint4 rec[PAY ? U : 1];
#pragma unroll
    for (uint32_t u = 0; u < U; u++)
      if (r0 + u * NTHREADS < size) {
        k[u] = kin[r0 + u * NTHREADS];
        if constexpr (PAY) rec[u] = rin[r0 + u * NTHREADS];
        else id[u] = ids ? iin[r0 + u * NTHREADS] : r0 + u * NTHREADS;
      }
#pragma unroll
    for (uint32_t u = 0; u < U; u++)
      if (r0 + u * NTHREADS < size) {
        uint32_t row;
        if constexpr (PAY) row = rec[u].x;
        else row = id[u];
        const uint32_t p = atomicAdd(&sm.word[bin_of(by_id ? uint64_t(row) : uint64_t(k[u]))], 1u);
        kout[p] = k[u];
        if constexpr (PAY) rout[p] = rec[u];
        else if (ids) iout[p] = id[u];
      }
  }
  // The parts' records come by bulk copies.
  if constexpr (PAY) asm volatile("fence.proxy.async;" ::: "memory");
  __syncthreads();
  return parts + total;
}

// The rows of a bucket with many rows at one position, or in one bin: from the words by bin (and sm.place, the
// words' bins), a bin's rows in neighbouring threads, to the bucket's keys and ids (or places) in order.
//   Rows at one position are nearly always one key's: they are ranked by row id, and each one's key is compared
// with that of one of them; only where some differ the ranking is made again by whole keys.
//   A crowded bin (more than MAX_PAIRED rows) at one position cuts its m places into m cells by row id, which hold a
// row or two each: a second counting step. At several positions (two repeated keys that share a bin) its rows are
// compared with one another, up to MAX_MIXED of them; for more the bucket is split by the range of its own keys, every
// crowded bin a part.
constexpr uint32_t MAX_MIXED = 256;
constexpr uint32_t LOW = uint32_t(1 << BINS_LOG) - 1u;       // a word's place
constexpr uint32_t TIED_DONE = 0, TIED_SPLIT = 1, TIED_TIMEOUT = 2;
template <typename KeyT, int PAY, typename SM>
__device__ __forceinline__ uint32_t order_tied(SM& sm, const Args& a, const KeyT* kin, uint32_t rows, bool exact, bool crowded,
                                               uint32_t parity, uint32_t id0, uint32_t idsh) {
  const uint32_t t = threadIdx.x;
  const int ni = int((rows + NTHREADS - 1 - t) / NTHREADS);
  if constexpr (PAY) {
    if (!mbar_wait(&sm.full, parity)) {
      atomicOr(a.err, ERR_LOOKBACK_TIMEOUT);
      return TIED_TIMEOUT;
    }
  }
  auto id_at = [&](uint32_t p) { return PAY ? sm.rec[PAY ? p : 0].x : sm.id[PAY ? 0 : p]; };
  // Item i: the row whose word is the (i x NTHREADS + t)-th. Words and places are kept, all else is read again from
  // shared memory: with ids and bins in registers too they spill (27 local loads a row).
  uint32_t word[NITEMS], at[NITEMS];
  uint32_t crowd = 0;                              // items in crowded bins at one position
  auto bin_of_item = [&](int i, uint32_t& s0, uint32_t& s1) {
    const uint32_t b = sm.place[t + i * NTHREADS];
    s0 = sm.start[b];
    s1 = sm.start[b + 1];
  };
#pragma unroll
  for (int i = 0; i < NITEMS; i++) word[i] = i < ni ? sm.word[t + i * NTHREADS] : 0u;
  if (crowded) {
#pragma unroll
    for (int i = 0; i < NITEMS; i++) {
      if (i >= ni) break;
      uint32_t s0, s1;
      bin_of_item(i, s0, s1);
      if (s1 - s0 > MAX_PAIRED && (sm.word[s0] ^ word[i]) > LOW) sm.mixed[s0 / CROWD] = 1;
    }
    bool split = false;
    __syncthreads();
#pragma unroll
    for (int i = 0; i < NITEMS; i++) {
      if (i >= ni) break;
      uint32_t s0, s1;
      bin_of_item(i, s0, s1);
      if (s1 - s0 <= MAX_PAIRED) continue;
      if (!sm.mixed[s0 / CROWD]) crowd |= 1u << i;
      else split |= s1 - s0 > MAX_MIXED;
    }
    if (__syncthreads_or(int(split))) return TIED_SPLIT;
  }
  bool differ = false;
#pragma unroll
  for (int i = 0; i < NITEMS; i++) {
    if (i >= ni) break;
    uint32_t s0, s1;
    bin_of_item(i, s0, s1);
    const uint32_t me = word[i], mine = id_at(me & LOW);
    uint32_t rank = s0, rep = me;
    if ((crowd >> i) & 1u) {
      rep = sm.word[s0];
      rank = s0 + __umulhi((mine - id0) << idsh, s1 - s0);
    } else if (s1 - s0 > 1) {
#pragma unroll 1
      for (uint32_t q = s0; q < s1; q++) {
        const uint32_t o = sm.word[q];
        if ((o ^ me) <= LOW) {
          rep = min(rep, o);
          rank += id_at(o & LOW) < mine ? 1u : 0u;
        } else {
          rank += o < me ? 1u : 0u;
        }
      }
    }
    at[i] = rank;
    if (!exact && rep != me) differ |= kin[rep & LOW] != kin[me & LOW];
  }
  if (__syncthreads_or(int(differ))) {
    // Few rows are compared with one another; a larger bin becomes a part, whose own range is 2,048 times smaller.
    bool split = false;
#pragma unroll 1
    for (int i = 0; i < ni; i++) {
      const uint32_t q = t + i * NTHREADS, me = sm.word[q], mine = id_at(me & LOW), b = sm.place[q];
      const uint32_t s0 = sm.start[b], s1 = sm.start[b + 1];
      const KeyT k = kin[me & LOW];
      if (s1 - s0 > MAX_BIN && !sm.mixed[s0 / CROWD]) {
        split |= kin[sm.word[s0] & LOW] != k;
        continue;
      }
      uint32_t rank = s0;
      for (uint32_t x = s0; x < s1; x++) {
        const uint32_t o = sm.word[x], p = o & LOW;
        if ((o ^ me) <= LOW) {
          if (o == me) continue;
          const KeyT other = kin[p];
          rank += other < k || (other == k && id_at(p) < mine) ? 1u : 0u;
        } else {
          rank += o < me ? 1u : 0u;
        }
      }
#pragma unroll
      for (int j = 0; j < NITEMS; j++)
        if (j == i) at[j] = rank;
    }
    if (__syncthreads_or(int(split))) return TIED_SPLIT;
  }
  if (crowded) {
    for (uint32_t x = t; x < BINS; x += NTHREADS) sm.start[x] = 0;
    __syncthreads();
    uint32_t in[NITEMS];
#pragma unroll
    for (int i = 0; i < NITEMS; i++) {
      if (i >= ni) break;
      in[i] = atomicAdd(&sm.start[at[i]], 1u);
    }
    __syncthreads();
    count_scan(sm, rows);
#pragma unroll
    for (int i = 0; i < NITEMS; i++) {
      if (i >= ni) break;
      sm.word[sm.start[at[i]] + in[i]] = id_at(word[i] & LOW);
    }
    __syncthreads();
#pragma unroll
    for (int i = 0; i < NITEMS; i++) {
      if (i >= ni) break;
      const uint32_t s0 = sm.start[at[i]], s1 = sm.start[at[i] + 1];
      uint32_t rank = s0;
      if (s1 - s0 > 1) {
        const uint32_t mine = id_at(word[i] & LOW);
#pragma unroll 1
        for (uint32_t q = s0; q < s1; q++) rank += sm.word[q] < mine ? 1u : 0u;
      }
      at[i] = rank;
    }
  }
  // In order: the places, then (the ids of this thread's rows read before others' land there) ids and keys.
  if constexpr (!PAY) {
    uint32_t id[NITEMS];
#pragma unroll
    for (int i = 0; i < NITEMS; i++) id[i] = i < ni ? sm.id[word[i] & LOW] : 0u;
    __syncthreads();
#pragma unroll
    for (int i = 0; i < NITEMS; i++) {
      if (i >= ni) break;
      sm.id[at[i]] = id[i];
    }
  } else {
    __syncthreads();
#pragma unroll
    for (int i = 0; i < NITEMS; i++) {
      if (i >= ni) break;
      sm.place[at[i]] = uint16_t(word[i] & LOW);
    }
  }
#pragma unroll
  for (int i = 0; i < NITEMS; i++) {
    if (i >= ni) break;
    sm.key[at[i]] = kin[word[i] & LOW];
  }
  return TIED_DONE;
}

// Bucket b is left to later_body.
__device__ __forceinline__ void put_off(const Args& a, uint32_t b) {
  const uint32_t at = atomicAdd(&a.st->later, 1u);
  if (at < a.bucket_cap) a.later[at] = b;
  else atomicOr(a.err, ERR_BOUNDS);
}

// A row leaves: its id, its key as the column's value, its payload.
template <typename KeyT>
struct KeyOut {
  bool xored;                           // an integer key of the key's own width leaves by one XOR
  KeyT bits;
  __device__ __forceinline__ explicit KeyOut(const Args& a)
      : xored(a.key_pt == PT_I64 || a.key_pt == PT_U64 || a.key_pt == PT_I32 || a.key_pt == PT_U32),
        bits(KeyT(((a.key_pt == PT_I64 || a.key_pt == PT_I32) ? KeyT(KeyT(1) << (8 * sizeof(KeyT) - 1)) : KeyT(0)) ^
                  (a.key_desc ? KeyT(~KeyT(0)) : KeyT(0)))) {}
};

// A bucket's (or a part's) rows, ordered in shared memory, to their places from `dst0` on. PART: rows [run0, run1)
// of the values all have this part's key, where that is not empty. False when the records did not come.
template <typename KeyT, int PAY, bool FREQ, int LTHREADS, bool PART = false, typename SM>
__device__ __forceinline__ bool write_rows(SM& sm, const Args& a, const KeyOut<KeyT>& ko, uint64_t dst0, uint32_t rows, uint32_t nkeys,
                                           uint32_t parity, uint64_t run0 = 0, uint64_t run1 = 0) {
  const uint32_t t = threadIdx.x;
  constexpr int LITEMS = CAP / LTHREADS;
  const int ni = int((rows + LTHREADS - 1 - t) / LTHREADS);
  // Rows of the frequent keys before key k: they are not in the buckets.
  auto apart_before = [&](KeyT k) {
    uint32_t n = 0;
    for (uint32_t h = 0; h < nkeys; h++) n += k > KeyT(a.st->key[h]) ? a.st->key_rows[h] : 0u;
    return n;
  };
  // Frequent keys between the bucket's rows: row by row. (Not in a sort of ranks, keys or payload.)
  if (FREQ && nkeys) {
    const uint32_t lo = apart_before(sm.key[0]), hi = apart_before(sm.key[rows - 1]);
    if (dst0 + hi + rows > a.n) {                          // the scan rules it out
      if (t == 0) atomicOr(a.err, ERR_BOUNDS);
      return true;
    }
    if constexpr (!PAY)
      if (lo != hi) {
        for (uint32_t r = t; r < rows; r += LTHREADS) store_id(a, dst0 + r + apart_before(sm.key[r]), sm.id[r]);
        return true;
      }
    dst0 += lo;
  }
  if constexpr (!PAY) {
    if (a.ranks.out) {
      // The run of equal keys around a row: by bisection of the ordered keys where a neighbour is equal.
      for (uint32_t r = t; r < rows; r += LTHREADS) {
        const KeyT k = sm.key[r];
        uint32_t p = r;
        if (a.ranks.mode == RANK_FIRST_OF && r > 0 && sm.key[r - 1] == k) {
          uint32_t lo = 0;
          while (lo < p) {
            const uint32_t mid = (lo + p) >> 1;
            if (sm.key[mid] < k) lo = mid + 1;
            else p = mid;
          }
        } else if (a.ranks.mode == RANK_LAST_OF && r + 1 < rows && sm.key[r + 1] == k) {
          uint32_t hi = rows;
          while (p + 1 < hi) {
            const uint32_t mid = (p + hi) >> 1;
            if (sm.key[mid] <= k) p = mid;
            else hi = mid;
          }
        }
        uint64_t rank = dst0 + p + 1;
        if (PART && run0 < run1 && a.ranks.mode == RANK_FIRST_OF) rank = run0 + 1;
        if (PART && run0 < run1 && a.ranks.mode == RANK_LAST_OF) rank = run1;
        const uint32_t row = sm.id[r];
        if (row < a.n) a.ranks.out[row] = uint32_t(rank);
        else atomicOr(a.err, ERR_BOUNDS);
      }
    }
    if (a.out) {
      if (a.wide) {
        uint64_t* o = static_cast<uint64_t*>(a.out) + dst0 + t;
#pragma unroll
        for (int i = 0; i < LITEMS; i++) {
          if (i >= ni) break;
          o[i * LTHREADS] = sm.id[t + i * LTHREADS];
        }
      } else {
        uint32_t* o = static_cast<uint32_t*>(a.out) + dst0 + t;
#pragma unroll
        for (int i = 0; i < LITEMS; i++) {
          if (i >= ni) break;
          o[i * LTHREADS] = sm.id[t + i * LTHREADS];
        }
      }
    }
  }
  if (a.key_out) {
    if (ko.xored) {
      KeyT* o = static_cast<KeyT*>(a.key_out) + dst0 + t;
#pragma unroll
      for (int i = 0; i < LITEMS; i++) {
        if (i >= ni) break;
        o[i * LTHREADS] = sm.key[t + i * LTHREADS] ^ ko.bits;
      }
    }
  }
  if constexpr (PAY) {
    if (!mbar_wait(&sm.full, parity)) {
      atomicOr(a.err, ERR_LOOKBACK_TIMEOUT);
      return false;
    }
  }
  if (a.key_out && !ko.xored) {
    for (uint32_t r = t; r < rows; r += LTHREADS) {
      const KeyT k = sm.key[r];
      uint64_t v = unkey_bits<KeyT>(k, a.key_pt, a.key_desc);
      if (a.key_src && (k == KeyT(a.twin0) || k == KeyT(a.twin1))) {
        uint32_t id;
        if constexpr (PAY) id = sm.rec[sm.place[r]].x;
        else id = sm.id[r];
        v = source_bits(a, id);
      }
      store_width(a.key_out, dst0 + r, pt_bytes(a.key_pt), v);
    }
  }
  if constexpr (PAY) {
    if (a.pay.pair && !a.out) {
      uint64_t* w = static_cast<uint64_t*>(a.pay.dst[a.pay.wide]) + dst0 + t;
      uint32_t* h = static_cast<uint32_t*>(a.pay.dst[a.pay.narrow]) + dst0 + t;
#pragma unroll
      for (int i = 0; i < LITEMS; i++) {
        if (i >= ni) break;
        const uint4 v = sm.rec[sm.place[t + i * LTHREADS]];
        w[i * LTHREADS] = uint64_t(v.y) | (uint64_t(v.z) << 32);
        h[i * LTHREADS] = v.w;
      }
    } else {
      for (uint32_t r = t; r < rows; r += LTHREADS) {
        const uint4 v = sm.rec[sm.place[r]];
        store_id(a, dst0 + r, v.x);
        unpack_record(a.pay, v, dst0 + r);
      }
    }
  }
  return true;
}

// The buckets that sort_body put off: those with bins of repeated keys, or of more rows than its form takes, which are
// cut into parts. A launch of its own: within sort_body its registers cost every bucket (16M int64 keys that do not
// repeat: the buckets' sort 149 us, 193 with this behind its loop, the next bucket's keys waited for to be spilled).
template <typename KeyT, int PAY, bool FREQ = false, int TIES = TIES_ID>
__device__ __forceinline__ void later_body(const Args& a) {
  extern __shared__ __align__(16) unsigned char lsm[];
  using SM = LaterShared<KeyT, PAY, TIES>;
  SM& sm = *reinterpret_cast<SM*>(lsm);
  const State* st = a.st;
  const uint32_t count = st->later;
  if (blockIdx.x >= count || st->mode != MODE_BUCKETS) return;
  const uint32_t t = threadIdx.x, src = st->s2 ? 1u : 0u, nkeys = FREQ ? st->nkeys : 0u;
  const uint64_t vbase = a.nulls_first ? uint64_t(st->n_null) + st->n_nan : 0ull;
  const KeyOut<KeyT> ko(a);
  if (PAY && t == 0) mbar_init(&sm.full);
  uint32_t parts = 0, turn = blockIdx.x, parity = 0;
  // Rows whose strings differ behind equal keys.
  auto by_strings = [&](uint32_t first, uint32_t size, uint32_t side) {
    if constexpr (TIES == TIES_STRING) {
      const uint32_t* iin = a.ids[side] + first;
      bool far = size > uint32_t(BIG);
      if (!far) {
        __syncthreads();
        bitonic_rows<TIES>(sm.slow.key, sm.slow.place, size, static_cast<const KeyT*>(a.keys[side]) + first,
                           [&](uint32_t p) { return iin[p]; }, a.ties, far);
        far = __syncthreads_or(int(far)) != 0;     // (the sort then ended early: its places are in no order)
        for (uint32_t r = t; r < size && !far; r += NTHREADS) store_id(a, vbase + first + r, iin[sm.slow.place[r]]);
      }
      if (far) a.st->mode = MODE_FALLBACK;
    }
  };
  for (;;) {
    __syncthreads();                               // the last part's memory, and its place in the list, are free
    uint32_t first, size, side, kind, run_at = 0, run_n = 0;
    if (parts) {
      parts--;
      first = sm.part_at[parts];
      size = sm.part_n[parts] & 0x1FFFFFFFu;
      side = (sm.part_n[parts] >> 29) & 1u;
      kind = sm.part_n[parts] >> 30;
      if constexpr (!PAY) {
        run_at = sm.run_at[parts];
        run_n = sm.run_n[parts];
      }
    } else {
      if (turn >= count) return;
      const uint32_t b = a.later[turn];
      turn += gridDim.x;
      first = a.bpos[b];
      size = a.bpos[b + 1] - first;
      side = src;
      kind = KIND_KEY;
      if (vbase + first + size > a.n || size > a.large) {         // the scan rules both out
        if (t == 0) atomicOr(a.err, ERR_BOUNDS);
        return;
      }
    }
    if (size == 0) continue;
    __syncthreads();
    uint32_t heavy = PART_ROWS;                    // split, bins of more rows becoming parts
    if (size <= uint32_t(CAP)) {
      if constexpr (PAY) {
        if (t == 0) bulk_load(sm.rec, a.rec[side] + first, size * 16u, &sm.full);
      }
      const KeyT* kin = static_cast<const KeyT*>(a.keys[side]) + first;
      const int ni = int((size + NTHREADS - 1 - t) / NTHREADS);
      KeyT key[NITEMS];
      KeyT klo = KeyT(~KeyT(0)), khi = 0;
      uint32_t id0 = ~0u, id1 = 0;
#pragma unroll
      for (int i = 0; i < NITEMS; i++)
        if (i < ni) key[i] = kin[t + i * NTHREADS];
#pragma unroll
      for (int i = 0; i < NITEMS; i++) {
        if (i >= ni) break;
        const uint32_t id = PAY ? a.rec[side][first + t + i * NTHREADS].x
                                : a.ids[0] ? a.ids[side][first + t + i * NTHREADS] : t + i * NTHREADS;
        if constexpr (!PAY) sm.id[t + i * NTHREADS] = id;
        id0 = min(id0, id);
        id1 = max(id1, id);
      }
      if (!parts && turn < count) {
        // The next bucket's rows come from HBM to L2 meanwhile.
        const uint32_t b = a.later[turn], nf = a.bpos[b], nn = a.bpos[b + 1] - nf;
        const char* k0 = reinterpret_cast<const char*>(static_cast<const KeyT*>(a.keys[src]) + nf);
        const char* i0 = PAY ? reinterpret_cast<const char*>(a.rec[src] + nf) : reinterpret_cast<const char*>(a.ids[src] + nf);
        const uint32_t ib = PAY ? 16u : a.ids[0] ? 4u : 0u;
        for (uint32_t x = t * 128u; x < nn * uint32_t(sizeof(KeyT)); x += NTHREADS * 128u)
          asm volatile("prefetch.global.L2 [%0];" ::"l"(k0 + x));
        for (uint32_t x = t * 128u; x < nn * ib; x += NTHREADS * 128u)
          asm volatile("prefetch.global.L2 [%0];" ::"l"(i0 + x));
      }
      for (uint32_t x = t; x < BINS; x += NTHREADS) sm.start[x] = 0;
      if (t <= CAP / CROWD) sm.mixed[t] = 0;
      // Positions: the top bits of the distance from the part's smallest key, or row id; the ids' own range orders crowded bins.
#pragma unroll
      for (int i = 0; i < NITEMS; i++) {
        if (i >= ni) break;
        klo = min(klo, key[i]);
        khi = max(khi, key[i]);
      }
      block_range(sm, klo, khi, id0, id1);
      const uint32_t idsh = id1 > id0 ? __clz(id1 - id0) : 0u;
      const uint64_t lo = kind == KIND_ID ? uint64_t(id0) : uint64_t(klo), hi = kind == KIND_ID ? uint64_t(id1) : uint64_t(khi);
      const uint32_t sh = range_shift(hi - lo);
      if (PAY && kind == KIND_ID && !mbar_wait(&sm.full, parity)) {
        atomicOr(a.err, ERR_LOOKBACK_TIMEOUT);
        return;
      }
      auto pos_of = [&](int i) {
        uint64_t x = uint64_t(key[i]);
        if (kind == KIND_ID) x = PAY ? sm.rec[PAY ? t + i * NTHREADS : 0].x : sm.id[PAY ? 0 : t + i * NTHREADS];
        return uint32_t(((x - lo) << sh) >> 32);
      };
      uint32_t at[NITEMS];
#pragma unroll
      for (int i = 0; i < NITEMS; i++) {
        if (i >= ni) break;
        at[i] = atomicAdd(&sm.start[pos_of(i) >> (32 - BINS_LOG)], 1u);
      }
      __syncthreads();
      const bool crowded = count_scan(sm, size);
#pragma unroll
      for (int i = 0; i < NITEMS; i++) {
        if (i >= ni) break;
        const uint32_t pos = pos_of(i), bin = pos >> (32 - BINS_LOG), q = sm.start[bin] + at[i];
        sm.word[q] = (pos << BINS_LOG) | (t + i * NTHREADS);
        sm.place[q] = uint16_t(bin);
      }
      __syncthreads();
      const uint32_t tied = order_tied<KeyT, PAY>(sm, a, kin, size, sh >= 32u, crowded, parity, id0, idsh);
      if (tied == TIED_TIMEOUT) return;
      if (PAY) parity ^= 1u;
      if (tied != TIED_SPLIT) {
        __syncthreads();
        if constexpr (TIES == TIES_STRING) {
          // Equal keys are in row order: right where their strings are equal (a part of one key's rows was looked at whole).
          bool differ = false, far = false;
          for (uint32_t r = t + 1; r < size && kind != KIND_ID && !far; r += NTHREADS)
            if (sm.key[r] == sm.key[r - 1]) differ |= !same_string(a.ties, sm.id[r], sm.id[r - 1], far);
          if (far) a.st->mode = MODE_FALLBACK;
          if (__syncthreads_or(int(differ || far))) {
            by_strings(first, size, side);
            continue;
          }
        }
        // A part of one key's rows: where they all are.
        const uint64_t run0 = kind == KIND_ID ? vbase + run_at : 0ull, run1 = kind == KIND_ID ? run0 + run_n : 0ull;
        if (!write_rows<KeyT, PAY, FREQ, NTHREADS, true>(sm, a, ko, vbase + first, size, nkeys, parity ^ (PAY ? 1u : 0u), run0, run1))
          return;
        continue;
      }
      heavy = MAX_BIN;
    }
    const uint32_t split = split_rows<KeyT, PAY, TIES>(sm, a, first, size, side, kind, heavy, run_at, run_n, parts);
    if (TIES == TIES_STRING && split == NOT_SPLIT) by_strings(first, size, side);
    else parts = split;
  }
}

// The 32 bits below the bucket number of (position in the cell, as a fraction of the key's width) x (buckets of the
// cell). The bucket number comes from the top 32 bits alone, so the bits below can carry past it.
__device__ __forceinline__ uint32_t position_in(uint32_t z, uint32_t mul) { return z * mul; }
__device__ __forceinline__ uint32_t position_in(uint64_t z, uint32_t mul) {
  const uint32_t p = uint32_t(z >> 32) * mul, below = __umulhi(uint32_t(z), mul);
  return p + below < p ? ~0u : p + below;
}

template <typename KeyT, int PAY, int TIES, bool FREQ = false>
__device__ __forceinline__ void sort_body(const Args& a) {
  extern __shared__ __align__(16) unsigned char lsm[];
  using SM = FastShared<KeyT, PAY, TIES>;
  SM& sm = *reinterpret_cast<SM*>(lsm);
  const State* st = a.st;
  if (blockIdx.x >= a.sort_grid || st->mode != MODE_BUCKETS) return;
  const uint32_t t = threadIdx.x;
  const uint32_t nb = st->buckets, src = st->s2 ? 1u : 0u;
  const uint64_t vbase = a.nulls_first ? uint64_t(st->n_null) + st->n_nan : 0ull;
  const Map<KeyT> map = load_map<KeyT>(st);
  const KeyOut<KeyT> ko(a);
  const uint32_t nkeys = FREQ ? st->nkeys : 0u;
  constexpr uint32_t SUB = 32 - BINS_LOG;          // position bits below the bin

  // Two bins' rows, and then starts, share a word.
  auto count_in = [&](uint32_t bin) { return (atomicAdd(&sm.start[bin >> 1], 1u << ((bin & 1u) * 16)) >> ((bin & 1u) * 16)) & 0xFFFFu; };
  auto start_of = [&](uint32_t bin) { return uint32_t(reinterpret_cast<const uint16_t*>(sm.start)[bin]); };

  // The bucket at hand: its rows, its part of the map, and this thread's keys of it (item i is the
  // bucket's row i x LTHREADS + t; items below nit).
  uint32_t first = 0, size = 0, meta = 0, f0 = 0;
  int nit = 0;
  KeyT key[LITEMS];
  auto next_bucket = [&](uint32_t b) {             // the next one with rows, from b on
    for (; b < nb; b += a.sort_grid) {
      first = a.bpos[b];
      size = a.bpos[b + 1] - first;
      if (size == 0) continue;
      meta = a.bmeta[b];
      f0 = a.bfirst[b];
      break;
    }
    return b;
  };
  auto load_rows = [&] {
    nit = size <= uint32_t(CAP) ? int((size + LTHREADS - 1 - t) / LTHREADS) : 0;
    const KeyT* kin = static_cast<const KeyT*>(a.keys[src]) + first + t;
#pragma unroll
    for (int i = 0; i < LITEMS; i++) {
      if (i >= nit) break;
      key[i] = kin[i * LTHREADS];
    }
  };
  auto load_records = [&] {                        // by thread 0, into the free buffer
    if constexpr (PAY)
      if (size <= uint32_t(CAP)) bulk_load(sm.rec, a.rec[src] + first, size * 16u, &sm.full);
  };
  if (t == 0) {
    sm.crowded = 0;
    sm.some_fast = 0;
    mbar_init(&sm.full);
  }
  for (int x = t; x < BINS / 2; x += LTHREADS) sm.start[x] = 0;
  __syncthreads();
  uint32_t b = next_bucket(blockIdx.x), parity = 0;
  bool far = false;                                // strings that agree for longer than a tie looks
  if (b < nb) {
    load_rows();
    if (t == 0) load_records();
  }
  while (b < nb) {
    const uint32_t rows = size, row0 = first;
    const int ni = nit;
    const KeyT* kin = static_cast<const KeyT*>(a.keys[src]) + row0;
    const uint32_t* iin = a.ids[src] ? a.ids[src] + row0 : nullptr;        // NULL: places stand in for the ids
    const uint64_t dst0 = vbase + row0;
    if (dst0 + rows > a.n || rows > a.large) {             // the scan rules both out
      if (t == 0) atomicOr(a.err, ERR_BOUNDS);
      if (PAY && rows <= uint32_t(CAP)) (void)mbar_wait(&sm.full, parity);
      break;
    }
    bool fast = rows <= uint32_t(CAP);
    uint32_t at[LITEMS];                           // the row's place among its bin's; by bin; in order
    if (fast) {
      uint32_t pos[LITEMS];
      uint32_t id[PAY ? 1 : LITEMS];
      if constexpr (!PAY) {
#pragma unroll
        for (int i = 0; i < LITEMS; i++) {
          if (i >= ni) break;
          id[i] = iin ? iin[t + i * LTHREADS] : t + i * LTHREADS;
        }
      }
      // A row's position in the bucket's key range, as 32 bits: in a split cell the part of
      // (position in the cell) x (buckets of the cell) below the bucket number; in a bucket of several
      // cells, (cell, position in it). Its top bits are the bin.
      if (meta & META_SPLIT) {
        const uint32_t sh = f0 >> 16, mul = meta & ~META_SPLIT;     // mul 0: keys outside the sampled range
        const uint32_t sh0 = sh == 0xFFFFu ? 0u : sh >> 1, sh1 = sh == 0xFFFFu ? 0u : sh - (sh >> 1);
#pragma unroll
        for (int i = 0; i < LITEMS; i++) {
          if (i >= ni) break;
          const KeyT z = KeyT(KeyT(KeyT(key[i] - map.lo) << sh0) << sh1);      // sh may be the key's width
          pos[i] = position_in(z, mul);
          at[i] = count_in(pos[i] >> SUB);
        }
      } else {
        const uint32_t cells = meta - f0 + 1u, k = cells > 1u ? 32u - __clz(cells - 1u) : 0u;
#pragma unroll
        for (int i = 0; i < LITEMS; i++) {
          if (i >= ni) break;
          uint32_t f, frac;
          cell_of(map, a.coarse, KeyT(key[i] - map.lo), f, frac);
          pos[i] = uint32_t(((uint64_t(f - f0) << 32) | frac) >> k);
          at[i] = count_in(pos[i] >> SUB);
        }
      }
      __syncthreads();
      {
        static_assert(BINS == 8 * LTHREADS, "a vector of bins a thread");
        const uint4 c = *reinterpret_cast<const uint4*>(&sm.start[t * 4]);
        const uint32_t w[4] = {c.x, c.y, c.z, c.w};
        uint32_t sum = 0, mx = 0, all;
#pragma unroll
        for (int q = 0; q < 4; q++) {
          sum += (w[q] & 0xFFFFu) + (w[q] >> 16);
          mx = max(mx, max(w[q] & 0xFFFFu, w[q] >> 16));
        }
        if (mx > MAX_BIN) sm.crowded = 1;
        uint32_t s = block_scan<LTHREADS>(sum, sm.warp, all), o[4];
#pragma unroll
        for (int q = 0; q < 4; q++) {
          const uint32_t next = s + (w[q] & 0xFFFFu);
          o[q] = s | (next << 16);
          s = next + (w[q] >> 16);
        }
        *reinterpret_cast<uint4*>(&sm.start[t * 4]) = make_uint4(o[0], o[1], o[2], o[3]);
        if (t == LTHREADS - 1) sm.start[BINS / 2] = rows;
      }
      if constexpr (PAY)
        if (!mbar_wait(&sm.full, parity)) atomicOr(a.err, ERR_LOOKBACK_TIMEOUT);
      __syncthreads();
      fast = sm.crowded == 0;
      if (fast) {
#pragma unroll
        for (int i = 0; i < LITEMS; i++) {
          if (i >= ni) break;
          const uint32_t s0 = start_of(pos[i] >> SUB), r = t + i * LTHREADS;
          uint32_t below;
          if constexpr (TIES == TIES_STRING) {
            below = r;
            sm.in_id[r] = id[i];
          } else if constexpr (PAY) {
            below = sm.rec[r].x;
          } else {
            below = id[i];
          }
          sm.word[s0 + at[i]] = (uint64_t(pos[i]) << 32) | below;
          at[i] = s0 + at[i];
        }
        __syncthreads();
        // A row's place: the rows of its bin that come before it, by position and, at one position, by row id. Rows at one
        // position are nearly always one key's; the keys in order tell whether they are.
        bool some = false;                         // rows at one position
#pragma unroll
        for (int i = 0; i < LITEMS; i++) {
          if (i >= ni) break;
          const uint32_t s0 = start_of(pos[i] >> SUB), s1 = start_of((pos[i] >> SUB) + 1);
          if (s1 - s0 > 1) {
            const uint64_t me = sm.word[at[i]];
            uint32_t rank = s0;
#pragma unroll 1
            for (uint32_t q = s0; q < s1; q++) {
              const uint64_t o = sm.word[q];
              if constexpr (TIES == TIES_STRING) {
                if (uint32_t(o >> 32) == pos[i] && o != me) {
                  const KeyT k = kin[uint32_t(o)];
                  rank += k < key[i] || (k == key[i] && tied_before<TIES>(a.ties, sm.in_id[uint32_t(o)], id[PAY ? 0 : i], far)) ? 1u : 0u;
                  continue;
                }
              } else {
                some |= uint32_t(o >> 32) == pos[i] && o != me;
              }
              rank += o < me ? 1u : 0u;
            }
            at[i] = rank;
          }
        }
        some = __syncthreads_or(int(some)) != 0;
#pragma unroll
        for (int i = 0; i < LITEMS; i++) {
          if (i >= ni) break;
          sm.key[at[i]] = key[i];
          if constexpr (PAY) sm.place[at[i]] = uint16_t(t + i * LTHREADS);
          else sm.id[at[i]] = id[i];
        }
        if (some) {
          __syncthreads();
          bool wrong = false;
          for (uint32_t r = t + 1; r < rows; r += LTHREADS) wrong |= sm.key[r] < sm.key[r - 1];
          fast = !__syncthreads_or(int(wrong));
        }
      }
    }
    // The next bucket's keys arrive while this one leaves.
    const uint32_t bn = next_bucket(b + a.sort_grid);
    if (bn < nb) load_rows();
    __syncthreads();
    if (fast) {
      if (t == 0) sm.some_fast = 1;
      if (!write_rows<KeyT, PAY, FREQ, LTHREADS>(sm, a, ko, dst0, rows, nkeys, parity)) return;
    } else {
      // Left to later_body; in a column of repeated keys, where neither of the CTA's first two buckets was fast,
      // with all of the CTA's that follow.
      const bool rest = !sm.some_fast && b >= blockIdx.x + a.sort_grid;
      if (t == 0) put_off(a, b);
      if (rest)
        for (uint32_t x = bn + t * a.sort_grid; x < nb; x += LTHREADS * a.sort_grid)
          if (a.bpos[x + 1] != a.bpos[x]) put_off(a, x);
      if constexpr (PAY) {
        if (rows <= uint32_t(CAP) && !mbar_wait(&sm.full, parity)) {
          atomicOr(a.err, ERR_LOOKBACK_TIMEOUT);
          return;
        }
      }
      if (rest) return;
    }
    if (PAY && rows <= uint32_t(CAP)) parity ^= 1u;
    b = bn;
    __syncthreads();
    for (int x = t; x < BINS / 2; x += LTHREADS) sm.start[x] = 0;
    if (t == 0) {
      sm.crowded = 0;
      if (b < nb) load_records();
    }
    __syncthreads();
  }
  if (TIES == TIES_STRING && far) a.st->mode = MODE_FALLBACK;
}

// ---- the launches: of one sort, and of a batch's sorts (one a row of the grid)

template <typename KeyT, bool FREQ>
__global__ void __cluster_dims__(CLUSTER, 1, 1) __launch_bounds__(1024)
buckets_kernel(const __grid_constant__ ColView col, const __grid_constant__ Args a) {
  buckets_body<KeyT, FREQ>(col, a);
}
template <typename KeyT, bool FREQ>
__global__ void __launch_bounds__(HTHREADS)
bucket_histogram_kernel(const __grid_constant__ ColView col, const __grid_constant__ Args a) {
  histogram_body<KeyT, FREQ>(col, a);
}
template <typename KeyT>
__global__ void __cluster_dims__(CLUSTER, 1, 1) __launch_bounds__(1024) bucket_starts_kernel(const __grid_constant__ Args a) {
  starts_body<KeyT, CLUSTER>(a);
}
template <typename KeyT, int PAY, bool FREQ>
__global__ void __launch_bounds__(THREADS, 2) level1_kernel(const __grid_constant__ ColView col, const __grid_constant__ Args a) {
  level1_body<KeyT, PAY, FREQ>(col, a);
}
template <typename KeyT, int PAY>
__global__ void __launch_bounds__(THREADS, 2) level2_kernel(const __grid_constant__ Args a) {
  level2_body<KeyT, PAY>(a);
}
template <typename KeyT, int PAY, int TIES, bool FREQ>
__global__ void __launch_bounds__(LTHREADS, LBLOCKS) bucket_sort_kernel(const __grid_constant__ Args a) {
  sort_body<KeyT, PAY, TIES, FREQ>(a);
}
template <typename KeyT, int PAY, bool FREQ, int TIES>
__global__ void __launch_bounds__(NTHREADS, NBLOCKS) bucket_later_kernel(const __grid_constant__ Args a) {
  later_body<KeyT, PAY, FREQ, TIES>(a);
}

struct alignas(16) BatchItem {
  ColView col;
  Args a;
};
__device__ __forceinline__ const BatchItem& batch_item(const BatchItem* __restrict__ items) {
  __shared__ BatchItem it;
  const uint32_t* src = reinterpret_cast<const uint32_t*>(items + blockIdx.y);
  for (uint32_t i = threadIdx.x; i < sizeof(BatchItem) / 4; i += blockDim.x) reinterpret_cast<uint32_t*>(&it)[i] = src[i];
  __syncthreads();
  return it;
}
template <typename KeyT>
__global__ void __cluster_dims__(CLUSTER, 1, 1) __launch_bounds__(1024) batch_buckets_kernel(const BatchItem* __restrict__ items) {
  const BatchItem& it = batch_item(items);
  buckets_body<KeyT>(it.col, it.a);
}
template <typename KeyT>
__global__ void __launch_bounds__(HTHREADS) batch_histogram_kernel(const BatchItem* __restrict__ items) {
  const BatchItem& it = batch_item(items);
  histogram_body<KeyT>(it.col, it.a);
}
template <typename KeyT>
__global__ void __cluster_dims__(CLUSTER, 1, 1) __launch_bounds__(1024) batch_starts_kernel(const BatchItem* __restrict__ items) {
  starts_body<KeyT, CLUSTER>(batch_item(items).a);
}
template <typename KeyT>
__global__ void __launch_bounds__(THREADS, 2) batch_level1_kernel(const BatchItem* __restrict__ items) {
  const BatchItem& it = batch_item(items);
  level1_body<KeyT, 0>(it.col, it.a);
}
template <typename KeyT>
__global__ void __launch_bounds__(THREADS, 2) batch_level2_kernel(const BatchItem* __restrict__ items) {
  level2_body<KeyT, 0>(batch_item(items).a);
}
template <typename KeyT>
__global__ void __launch_bounds__(LTHREADS, LBLOCKS) batch_sort_kernel(const BatchItem* __restrict__ items) {
  sort_body<KeyT, 0, TIES_ID>(batch_item(items).a);
}
template <typename KeyT>
__global__ void __launch_bounds__(NTHREADS, NBLOCKS) batch_later_kernel(const BatchItem* __restrict__ items) {
  later_body<KeyT, 0>(batch_item(items).a);
}

// ---- 5. the first k rows
//
// A sampled threshold that the k-th smallest key is almost surely at or below, one read of the column
// that keeps the rows at or below it, and the bucket sort of those few (key, row) pairs, whose first k
// row ids are the answer. The pairs are kept in no order: (key, row id) orders them.

// One cluster: the threshold. Selection by 8-bit digits of the sampled keys' distance from the smallest,
// until the digit's keys are few beyond the wanted ones.
struct FirstShared {
  uint32_t cnt[2][256];
  uint32_t warp[32];
  uint32_t pick[3];                      // the digit, the keys before it, its keys
  unsigned long long smax[CLUSTER], smin[CLUSTER], scnt[CLUSTER];
  unsigned long long wmax[32], wmin[32];
};

template <typename KeyT>
__global__ void __cluster_dims__(CLUSTER, 1, 1) __launch_bounds__(1024)
first_threshold_kernel(const __grid_constant__ ColView col, uint64_t n, uint64_t k, FirstState* __restrict__ fs) {
  namespace cg = cooperative_groups;
  cg::cluster_group cl = cg::this_cluster();
  __shared__ FirstShared sm;
  const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
  const uint32_t rank = cl.block_rank();
  cl.sync();                             // every CTA runs before its shared memory is written
  constexpr int U = SAMPLES / (1024 * CLUSTER);
  KeyT key[U];
  uint32_t live = 0;
#pragma unroll
  for (int u = 0; u < U; u++) {
    const uint32_t j = (rank * U + u) * 1024 + t;
    const uint64_t lo = uint64_t(j) * n / SAMPLES, hi = uint64_t(j + 1) * n / SAMPLES;
    uint32_t h = j * 2654435761u;
    h ^= h >> 15;
    h *= 2246822519u;
    h ^= h >> 13;
    const uint64_t row = lo + __umulhi(h, uint32_t(hi - lo));
    const bool valid = !col.valid || bit_at(col.valid, col.valid_off + int64_t(row));
    int cat;
    key[u] = key_from_raw<KeyT>(col, load_raw<KeyT>(col, row), valid, cat);
    if (cat == 0) live |= 1u << u;
  }
  uint64_t mx = 0, mn = 0;
#pragma unroll
  for (int u = 0; u < U; u++)
    if ((live >> u) & 1u) {
      mx = max(mx, uint64_t(key[u]));
      mn = max(mn, ~uint64_t(key[u]));
    }
  mx = warp_max_u64(mx);
  mn = warp_max_u64(mn);
  const uint32_t c = __reduce_add_sync(0xffffffffu, __popc(live));
  if (lane == 0) {
    sm.wmax[warp] = mx;
    sm.wmin[warp] = mn;
    sm.warp[warp] = c;
  }
  __syncthreads();
  if (warp == 0) {
    const uint64_t bx = warp_max_u64(sm.wmax[lane]), bn = warp_max_u64(sm.wmin[lane]);
    const uint32_t bc = __reduce_add_sync(0xffffffffu, sm.warp[lane]);
    if (lane < CLUSTER) {
      FirstShared* o = cl.map_shared_rank(&sm, lane);
      o->smax[rank] = bx;
      o->smin[rank] = bn;
      o->scnt[rank] = bc;
    }
  }
  cl.sync();
  uint64_t vmax = 0, vmin_inv = 0;
  uint32_t sv = 0;
#pragma unroll
  for (int r = 0; r < CLUSTER; r++) {
    vmax = max(vmax, uint64_t(sm.smax[r]));
    vmin_inv = max(vmin_inv, uint64_t(sm.smin[r]));
    sv += uint32_t(sm.scnt[r]);
  }
  // The sampled rank that holds k rows with a margin of four deviations.
  const float mu = float(k) * float(SAMPLES) / float(n);
  const uint32_t want = uint32_t(mu + 4.0f * sqrtf(mu) + 8.0f);
  if (sv < want) {                       // (the same in every CTA)
    if (rank == 0 && t == 0) {
      fs->limit = ~0ull;
      fs->rows = n;
    }
    cl.sync();
    return;
  }
  const uint64_t lo = ~vmin_inv, span = vmax - lo;
  const int bits = span ? 64 - __clzll((long long)span) : 1;
  uint64_t prefix = 0;                   // the digits chosen so far, of (key - lo) in `bits` bits
  int shift = bits;
  uint32_t left = want;
  for (int round = 0; shift > 0; round++) {
    const int step = shift < 8 ? shift : 8, next = shift - step, buf = round & 1;
    if (t < 256) sm.cnt[buf][t] = 0;
    __syncthreads();
#pragma unroll
    for (int u = 0; u < U; u++) {
      const uint64_t x = uint64_t(key[u]) - lo;
      if (((live >> u) & 1u) && (shift >= 64 || (x >> shift) == prefix)) atomicAdd(&sm.cnt[buf][(x >> next) & ((1u << step) - 1u)], 1u);
    }
    cl.sync();
    uint32_t mine = 0;
    if (t < 256)
      for (int r = 0; r < CLUSTER; r++) mine += cl.map_shared_rank(&sm, r)->cnt[buf][t];
    uint32_t all;
    const uint32_t before = block_scan<1024>(mine, sm.warp, all);
    if (t < 256 && before < left && left <= before + mine) {
      sm.pick[0] = t;
      sm.pick[1] = before;
      sm.pick[2] = mine;
    }
    __syncthreads();
    prefix = (shift >= 64 ? 0ull : prefix << step) | sm.pick[0];
    left -= sm.pick[1];
    shift = next;
    if (sm.pick[2] - left <= want / 4 + 8) break;
    __syncthreads();
  }
  if (rank == 0 && t == 0) {
    const uint64_t x = shift ? (prefix << shift) | ((1ull << shift) - 1ull) : prefix;
    fs->limit = lo + (x < span ? x : span);
    // Many rows at the limit itself: the first of them, in row order, are enough (evenly spread over the column, with a
    // margin of four deviations and a quarter).
    const float equal = shift ? 0.0f : float(sm.pick[2]) * float(n) / float(SAMPLES), wanted = float(k);
    fs->rows = n;
    if (equal > 2.0f * wanted + 1024.0f) {
      const float part = 1.25f * (wanted + 4.0f * sqrtf(wanted) + 64.0f) / equal;
      if (part < 1.0f) fs->rows = uint64_t(float(n) * part);
    }
  }
  cl.sync();                             // no CTA leaves while another reads its counts
}

// Rows whose key is below the limit, and those at the limit among the first rows, appended as (key, row) pairs; pairs past `cap` are
// only counted.
template <typename KeyT>
__global__ void __launch_bounds__(256) first_collect_kernel(const __grid_constant__ ColView col, uint64_t n, FirstState* __restrict__ fs,
                                                            uint32_t cap, KeyT* __restrict__ keys, uint32_t* __restrict__ rows) {
  constexpr int NI = 8;
  const KeyT limit = KeyT(fs->limit);
  const uint64_t equal_rows = fs->rows;
  const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5, lt = (1u << lane) - 1u;
  const uint64_t step = uint64_t(gridDim.x) * (256 * NI);
  for (uint64_t w0 = uint64_t(blockIdx.x) * (256 * NI) + warp * (NI * 32); w0 < n; w0 += step) {
    RawTile<KeyT, NI> r;
    uint32_t values, nulls, nans;
    load_tile(col, w0, n, r);
    encode_tile(col, w0, n, r, values, nulls, nans);
    uint32_t hit = 0;
#pragma unroll
    for (int i = 0; i < NI; i++)
      if (((values >> i) & 1u) && (r.key[i] < limit || (r.key[i] == limit && w0 + i * 32 + lane < equal_rows))) hit |= 1u << i;
    if (!__any_sync(0xffffffffu, hit != 0u)) continue;
#pragma unroll
    for (int i = 0; i < NI; i++) {
      const bool is = (hit >> i) & 1u;
      const uint32_t m = __ballot_sync(0xffffffffu, is);
      if (m == 0u) continue;
      uint32_t at = 0;
      if (lane == 0) at = atomicAdd(&fs->count, uint32_t(__popc(m)));
      at = __shfl_sync(0xffffffffu, at, 0) + __popc(m & lt);
      if (is && at < cap) {
        keys[at] = r.key[i];
        rows[at] = uint32_t(w0) + uint32_t(i) * 32 + lane;
      }
    }
  }
}

// ---- host side

static uint32_t bucket_cap(uint64_t n) {
  const uint64_t want = 4 * (n / TARGET) + 256;
  return uint32_t(std::min<uint64_t>(MAX_BUCKETS, (want + 1023) & ~uint64_t(1023)));
}
namespace {
// A chunk a level-1 CTA, two of them an SM; at most as many as the starts have threads.
uint32_t rows_per_chunk(uint64_t n) {
  const uint64_t chunks = std::min<uint64_t>(1024, uint64_t(device().sm_count) * 2);
  const uint64_t per = (n + chunks - 1) / chunks;
  return uint32_t((per + TILE - 1) / TILE * TILE);
}
uint32_t chunks_of(uint64_t n) { return n <= SAMPLES ? 0u : uint32_t((n + rows_per_chunk(n) - 1) / rows_per_chunk(n)); }

// Rows a bucket may hold before the digit passes sort the column instead: one CTA works on it alone.
uint32_t large_rows(uint64_t n) { return uint32_t(std::min<uint64_t>(LARGE, std::max<uint64_t>(BIG, n / 1024))); }

struct Layout {
  size_t state, bcount, bmeta, zeroed, coarse, fine, bfirst, bpos, later, cursor1, cursor2, chunk_bins, chunk_cats, total;
  explicit Layout(uint64_t n) {
    size_t at = 0;
    auto take = [&](size_t bytes) {
      const size_t r = at;
      at = (at + bytes + 255) & ~size_t(255);
      return r;
    };
    const size_t nb = bucket_cap(n);
    state = take(sizeof(State));
    bcount = take(nb * 4);
    bmeta = take(nb * 4);
    zeroed = at;
    coarse = take(COARSE * 4);
    fine = take(FINE * 4);
    bfirst = take(nb * 4);
    bpos = take((nb + 1) * 4);
    later = take(nb * 4);
    cursor1 = take(size_t(BINS1) * CUR_PAD * 4);
    cursor2 = take(nb * CUR_PAD * 4);
    chunk_bins = take(size_t(chunks_of(n)) * BINS1 * 4);
    chunk_cats = take(size_t(chunks_of(n)) * CATS * 4);
    total = at;
  }
};

template <typename F>
void smem_limit(F fn, size_t bytes) {
  AM_CUDA(cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, int(bytes)));
}

template <typename KeyT, int PAY, int TIES, bool FREQ = false>
void launch_moves(const ColView& cv, const Args& a, cudaStream_t s) {
  static std::once_flag once;
  std::call_once(once, [] {
    smem_limit(level1_kernel<KeyT, PAY, FREQ>, sizeof(TileShared<KeyT, PAY>));
    smem_limit(level2_kernel<KeyT, PAY>, sizeof(Tile2Shared<KeyT, PAY>));
    smem_limit(bucket_sort_kernel<KeyT, PAY, TIES, FREQ>, sizeof(FastShared<KeyT, PAY, TIES>));
    smem_limit(bucket_later_kernel<KeyT, PAY, FREQ, TIES>, sizeof(LaterShared<KeyT, PAY, TIES>));
  });
  if (!a.one_launch) {
    {
      KernelTimer kt("bucket_level1", s);
      level1_kernel<KeyT, PAY, FREQ><<<a.nchunks, THREADS, sizeof(TileShared<KeyT, PAY>), s>>>(cv, a);
      AM_CUDA(cudaGetLastError());
    }
    if (a.bucket_cap > a.bins1_cap) {
      KernelTimer kt("bucket_level2", s);
      level2_kernel<KeyT, PAY><<<a.level2_grid, THREADS, sizeof(Tile2Shared<KeyT, PAY>), s>>>(a);
      AM_CUDA(cudaGetLastError());
    }
  }
  {
    KernelTimer kt("bucket_sort", s);
    bucket_sort_kernel<KeyT, PAY, TIES, FREQ><<<a.sort_grid, LTHREADS, sizeof(FastShared<KeyT, PAY, TIES>), s>>>(a);
    AM_CUDA(cudaGetLastError());
  }
  {
    KernelTimer kt("bucket_later", s);
    bucket_later_kernel<KeyT, PAY, FREQ, TIES><<<a.later_grid, NTHREADS, sizeof(LaterShared<KeyT, PAY, TIES>), s>>>(a);
    AM_CUDA(cudaGetLastError());
  }
}

// The plan and the counts. FREQ: frequent keys are set apart (the other sorts' kernels carry none of it).
template <typename KeyT, bool FREQ = false>
void launch_counts(const Sort& b, const Args& a, cudaStream_t s) {
  {
    KernelTimer kt("bucket_plan", s);
    buckets_kernel<KeyT, FREQ><<<CLUSTER, 1024, 0, s>>>(b.col, a);
    AM_CUDA(cudaGetLastError());
  }
  if (a.one_launch) return;
  static std::once_flag once;
  std::call_once(once, [] { smem_limit(bucket_histogram_kernel<KeyT, FREQ>, size_t(MAX_BUCKETS) * 4); });
  {
    KernelTimer kt("bucket_histogram", s);
    bucket_histogram_kernel<KeyT, FREQ><<<a.hist_grid, HTHREADS, size_t(a.bucket_cap) * 4, s>>>(b.col, a);
    AM_CUDA(cudaGetLastError());
  }
  if (a.bucket_cap > FUSED_BUCKETS) {
    KernelTimer kt("bucket_scan", s);
    bucket_starts_kernel<KeyT><<<CLUSTER, 1024, 0, s>>>(a);
    AM_CUDA(cudaGetLastError());
  }
}

template <typename KeyT>
void launch_all(const Sort& b, const Args& a, int pay, cudaStream_t s) {
  if constexpr (sizeof(KeyT) == 8) {
    if (a.frequent) {
      launch_counts<KeyT, true>(b, a, s);
      launch_moves<KeyT, 0, TIES_ID, true>(b.col, a, s);
      return;
    }
  }
  launch_counts<KeyT>(b, a, s);
  if constexpr (sizeof(KeyT) == 8) {
    if (a.ties.offsets) {
      launch_moves<KeyT, 0, TIES_STRING>(b.col, a, s);
      return;
    }
  }
  if (pay) launch_moves<KeyT, 1, TIES_ID>(b.col, a, s);
  else launch_moves<KeyT, 0, TIES_ID>(b.col, a, s);
}
}  // namespace

void enqueue_first(const ColView& col, int key_bytes, uint64_t n, uint64_t k, FirstState* fs, void* keys, uint32_t* rows,
                   cudaStream_t s) {
  AM_CUDA(cudaMemsetAsync(fs, 0, sizeof(FirstState), s));
  const uint64_t tiles = (n + 256 * 8 - 1) / (256 * 8);
  const int grid = int(std::min<uint64_t>(tiles, uint64_t(device().sm_count) * 8));
  auto go = [&](auto tag) {
    using KeyT = decltype(tag);
    {
      KernelTimer kt("topk_threshold", s);
      first_threshold_kernel<KeyT><<<CLUSTER, 1024, 0, s>>>(col, n, k, fs);
      AM_CUDA(cudaGetLastError());
    }
    KernelTimer kt("topk_collect", s);
    first_collect_kernel<KeyT><<<grid, 256, 0, s>>>(col, n, fs, SAMPLES, static_cast<KeyT*>(keys), rows);
    AM_CUDA(cudaGetLastError());
  };
  if (key_bytes == 8) go(uint64_t(0));
  else go(uint32_t(0));
}

size_t scratch_bytes(uint64_t n) { return Layout(n).total; }
size_t zeroed_bytes(uint64_t n) { return Layout(n).zeroed; }

static Args make_args(const Sort& b) {
  const Layout L(b.n);
  auto at = [&](size_t off) {
    return reinterpret_cast<uint32_t*>(off < L.zeroed && b.zeroed ? b.zeroed + off : b.scratch + off);
  };
  Args a{};
  a.st = reinterpret_cast<State*>(at(L.state));
  a.coarse = at(L.coarse);
  a.fine = at(L.fine);
  a.bfirst = at(L.bfirst);
  a.bmeta = at(L.bmeta);
  a.bcount = at(L.bcount);
  a.bpos = at(L.bpos);
  a.later = at(L.later);
  a.cursor1 = at(L.cursor1);
  a.cursor2 = at(L.cursor2);
  a.chunk_bins = at(L.chunk_bins);
  a.chunk_cats = at(L.chunk_cats);
  a.nsamples = uint32_t(std::min<uint64_t>(b.n, SAMPLES));
  a.bucket_cap = bucket_cap(b.n);
  a.chunk_rows = rows_per_chunk(b.n);
  a.nchunks = chunks_of(b.n);
  a.n = b.n;
  for (int i = 0; i < 2; i++) {
    a.keys[i] = b.keys[i];
    a.ids[i] = reinterpret_cast<uint32_t*>(b.ids[i]);
    a.rec[i] = reinterpret_cast<uint4*>(b.ids[i]);
  }
  a.ties = b.ties;
  a.ranks = b.ranks;
  a.clear = static_cast<uint4*>(b.clear);
  a.clear16 = b.clear ? b.clear_bytes / 16 : 0;
  a.src_keys = b.src_keys;
  a.src_ids = b.src_ids;
  a.out = b.out;
  a.wide = b.wide ? 1 : 0;
  a.key_out = b.key_out;
  a.key_pt = b.key_pt;
  if (b.key_source) {
    // Keys of both zeros, and of every NaN: a column's own bits are read back for them.
    const bool wide = b.key_bytes == 8;
    const unsigned long long flip = b.key_desc ? ~0ull : 0ull, sign = wide ? 1ull << 63 : 1ull << 31;
    a.key_src = b.col.values;
    a.twin0 = sign ^ flip;
    a.twin1 = (sign | (wide ? 0x7FF0000000000001ull : 0x7F800001ull)) ^ flip;
  }
  a.key_desc = b.key_desc ? 1 : 0;
  a.nulls_first = b.nulls_first ? 1 : 0;
  a.err = b.err;
  a.sum = b.summary;
  if (b.payload) a.pay = b.rec;
  a.bins1_cap = b.payload ? BINS1 / 2 : BINS1;
  a.large = b.src_ids ? LARGE : large_rows(b.n);
  a.has_payload = b.payload ? 1 : 0;
  a.one_launch = b.n <= SAMPLES ? 1 : 0;
  a.frequent = b.frequent && !a.one_launch && !b.payload && !b.key_out && !b.ranks.out && !b.ties.offsets && !b.src_ids && b.key_bytes == 8 ? 1 : 0;
  if (a.one_launch) {
    a.bucket_cap = std::min(a.bucket_cap, ONE_CAP);
    a.bins1_cap = ONE_CAP;
  }
  const uint32_t sms = uint32_t(device().sm_count);
  a.hist_grid = std::min(a.nchunks, sms);
  a.level2_grid = uint32_t(std::min<uint64_t>((b.n + TILE - 1) / TILE, sms * 2));
  a.sort_grid = uint32_t(std::min<uint64_t>(b.n / (TARGET / 2) + 3, sms * LBLOCKS));
  a.later_grid = std::min(a.sort_grid, sms * NBLOCKS);
  return a;
}

State* enqueue(const Sort& b, cudaStream_t s) {
  const Args a = make_args(b);
  const int pay = b.payload ? 1 : 0;
  if (b.key_bytes == 8) launch_all<uint64_t>(b, a, pay, s);
  else launch_all<uint32_t>(b, a, pay, s);
  return a.st;
}

size_t batch_item_bytes() { return sizeof(BatchItem); }

void fill_batch_item(const Sort& b, void* item) {
  BatchItem it{};
  it.col = b.col;
  it.a = make_args(b);
  std::memcpy(item, &it, sizeof(it));
}

namespace {
template <typename KeyT>
void launch_batch(const BatchItem* items, const BatchItem* host, uint32_t count, bool timed, cudaStream_t s) {
  prepare_batch(int(sizeof(KeyT)));
  uint32_t hist = 0, chunks = 0, level2 = 0, sort = 0, later = 0, cap = 0;
  for (uint32_t i = 0; i < count; i++) {
    const Args& a = host[i].a;
    sort = std::max(sort, a.sort_grid);
    later = std::max(later, a.later_grid);
    if (a.one_launch) continue;
    hist = std::max(hist, a.hist_grid);
    chunks = std::max(chunks, a.nchunks);
    cap = std::max(cap, a.bucket_cap);
    if (a.bucket_cap > a.bins1_cap) level2 = std::max(level2, a.level2_grid);
  }
  // A grid has at most 65,535 rows.
  for (uint32_t at = 0; at < count; at += 65535) {
    const uint32_t rows = std::min<uint32_t>(count - at, 65535);
    const BatchItem* it = items + at;
    auto step = [&](const char* name, auto&& launch) {
      std::unique_ptr<KernelTimer> kt(timed ? new KernelTimer(name, s) : nullptr);
      launch();
      AM_CUDA(cudaGetLastError());
    };
    step("batch_plan", [&] { batch_buckets_kernel<KeyT><<<dim3(CLUSTER, rows), 1024, 0, s>>>(it); });
    if (hist) {
      step("batch_histogram", [&] { batch_histogram_kernel<KeyT><<<dim3(hist, rows), HTHREADS, size_t(cap) * 4, s>>>(it); });
      if (cap > FUSED_BUCKETS) step("batch_scan", [&] { batch_starts_kernel<KeyT><<<dim3(CLUSTER, rows), 1024, 0, s>>>(it); });
      step("batch_level1", [&] {
        batch_level1_kernel<KeyT><<<dim3(chunks, rows), THREADS, sizeof(TileShared<KeyT, 0>), s>>>(it);
      });
    }
    if (level2)
      step("batch_level2", [&] {
        batch_level2_kernel<KeyT><<<dim3(level2, rows), THREADS, sizeof(Tile2Shared<KeyT, 0>), s>>>(it);
      });
    step("batch_sort", [&] {
      batch_sort_kernel<KeyT><<<dim3(sort, rows), LTHREADS, sizeof(FastShared<KeyT, 0, TIES_ID>), s>>>(it);
    });
    // A share of the chip an array (its CTAs take as many buckets as there are): 592 CTAs each of 1,024 arrays,
    // nearly all idle, took 4 ms.
    const uint32_t each = std::max<uint32_t>(1, std::min<uint32_t>(later, 2 * NBLOCKS * uint32_t(device().sm_count) / rows));
    step("batch_later", [&] {
      batch_later_kernel<KeyT><<<dim3(each, rows), NTHREADS, sizeof(LaterShared<KeyT, 0>), s>>>(it);
    });
  }
}
template <typename KeyT>
void prepare() {
  static std::once_flag once;
  std::call_once(once, [] {
    smem_limit(batch_histogram_kernel<KeyT>, size_t(MAX_BUCKETS) * 4);
    smem_limit(batch_level1_kernel<KeyT>, sizeof(TileShared<KeyT, 0>));
    smem_limit(batch_level2_kernel<KeyT>, sizeof(Tile2Shared<KeyT, 0>));
    smem_limit(batch_sort_kernel<KeyT>, sizeof(FastShared<KeyT, 0, TIES_ID>));
    smem_limit(batch_later_kernel<KeyT>, sizeof(LaterShared<KeyT, 0>));
  });
}
}  // namespace

void prepare_batch(int key_bytes) {
  if (key_bytes == 8) prepare<uint64_t>();
  else prepare<uint32_t>();
}

void enqueue_batch(const void* items, const void* host_items, uint32_t count, int key_bytes, bool timed, cudaStream_t s) {
  const BatchItem* it = static_cast<const BatchItem*>(items);
  const BatchItem* h = static_cast<const BatchItem*>(host_items);
  if (key_bytes == 8) launch_batch<uint64_t>(it, h, count, timed, s);
  else launch_batch<uint32_t>(it, h, count, timed, s);
}

}  // namespace bs
}  // namespace am
