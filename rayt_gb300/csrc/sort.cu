// Feedback primitives: sorted unique of int32 feedback words, radix sort, and
// an inclusive scan.
//
// The reference does this with a work-group merge sort plus log2(N/wg) global
// merge passes (rayt/GPU algorithms/kernels/merge_sort.cl:2-73), an
// adjacent-difference flag, a Hillis-Steele scan of log2(N) full passes
// (rayt/GPU algorithms/kernels/scan.cl:2-12) and a scatter
// (rayt/GPU_renderer/kernels/feedback_compression.cl:4-34).  Here:
//
// Feedback unique, up to kSmall words: small_unique_kernel, one CTA.  Above:
//   compact_kernel   drops NO_HIT words, applies NodeToBlock, maps each word
//                    to an unsigned key (x ^ 0x80000000 keeps signed order),
//                    drops most repeats through a per-CTA filter, finds the
//                    key range; its last CTA chooses the path:
//   bitmap           (the keys span at most 2^26 values) a bitmap over [min, max], whose set bits read
//                    in order are the sorted unique set: set straight into
//                    the global bitmap and written out (direct_bitmap: few
//                    keys or a small bitmap), or range by range: range_hist and range_partition
//                    split the keys into 256 ranges (unstable), bucket_bitmap
//                    builds each range's slice in shared memory, emit writes
//                    the set bits in order.
//   radix            (wider ranges; launched once the host has read the
//                    choice) digit_hist, the digit passes, unique_kernel.
// Sort, up to kSmall keys: small_sort_kernel, one CTA.  Above: digit_hist (the
// four digits' counts in one read, and the range), and then
//   few values       counted by split_kernel, written by split_sort_kernel;
//   evenly spread    split_kernel moves the keys to up to 4608 parts of their
//                    range, split_sort_kernel sorts each in shared memory;
//   other keys, or more than 70 million: four digit_kernel passes (persistent
//                    CTAs, tiles of 8192 keys brought into shared memory by
//                    bulk async copies a tile ahead, per-digit decoupled
//                    look-back, scatter staged through shared memory); a pass
//                    whose digit is the same in every key is skipped.
//                    Launched once the host has read that they are needed.
//
// Scan: scan_kernel.
//
// The scan, direct_bitmap and emit kernels are cooperative launches (their CTAs
// wait on one another).  Tiles of the digit and unique kernels are claimed in order from an atomic
// counter by persistent CTAs until they run out, so a tile only waits on tiles
// claimed by running CTAs.  Published words live in a table of their own
// and are tagged with a per-call epoch and the pass, so the table is never
// cleared.  Every wait is bounded and sets an error flag instead of hanging.
#include <algorithm>
#include <cmath>
#include <type_traits>

#include "internal.h"

namespace rayt {
namespace {

constexpr int kThreads = 256;
constexpr int kWarps = kThreads / 32;
constexpr int kItems = 16;
constexpr int kTile = kThreads * kItems;  // 4096 keys
constexpr int kBuckets = 256;
constexpr int kPasses = 4;
// the range partition's per-bucket cursors, one per 128-byte line, so that
// claims on different buckets (every tile claims from most of them) never
// contend for one line
constexpr int kCursorStride = 32;
// the bitmap path keeps one range bucket's bitmap (span / 256 bits) in shared memory
constexpr int kMaxSpanLog2 = 26;
// Inputs of up to kDirectWords words put their keys straight into the bitmap
// (the launches of the partition would cost more than they give).  Of larger
// ones, those that kept up to kDirectKeys keys, or whose bitmap is one slice,
// or a few slices and not many keys for each CTA to read: scattered atomics on
// a wide one take 10 to 100 us per million keys (30 million words, 1.5 million
// kept, 50 million bits: 196 us straight, 160 us partitioned), and every slice
// is another read of the keys (30 million words, 24 million kept, 1.1 million
// bits, two slices: 168 us partitioned, 144 straight).
constexpr int kDirectWords = 1 << 21;
constexpr int kDirectKeys = 1 << 18;
constexpr unsigned long long kDirectFewSlices = 4, kDirectReads = 1ull << 26;
// The straight bitmap is built in shared memory, in slices of up to this many
// words, each by its share of the CTAs (at least kDirectSliceCtas): 1.9 million
// words, 1.6 million kept over 1.1 million bits: 110 us with atomics on the
// bitmap in memory, 58 in two slices.  Fewer than kDirectSliceKeys keys set
// their bits in memory when they span more than one slice.
constexpr int kDirectSliceWords = 1 << 15;
constexpr uint32_t kDirectSliceKeys = 1 << 15;
constexpr int kDirectSliceCtas = 2;
constexpr long long kSpinLimit = 1ll << 26;  // polls, a backstop to the time limit

// Time limit of every wait on another CTA's result (ns): a correct wait ends in
// microseconds, so one that lasts this long sets the call's error flag and
// gives up.
__device__ unsigned long long g_wait_ns = 1000000000ull;

__device__ __forceinline__ unsigned long long global_ns() {
  unsigned long long t;
  asm volatile("mov.u64 %0, %globaltimer;" : "=l"(t));
  return t;
}
// True once a wait that began at `start` has run out of polls or time.
__device__ __forceinline__ bool wait_over(long long& spins, unsigned long long start) {
  return ++spins > kSpinLimit || ((spins & 63) == 0 && global_ns() - start > g_wait_ns);
}
// Sets a call's error flag (device or mapped host memory).
__device__ __forceinline__ void set_error(int* err) { *(volatile int*)err = 1; }

// Programmatic launches: the kernel after this one may take its place while this
// one still runs; what it reads of this one's, it reads after its own
// wait_for_dependency.
__device__ __forceinline__ void dependents_may_start() {
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}
__device__ __forceinline__ void wait_for_dependency() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

// The end of a call's last kernel: the CTA that ends last publishes the call's
// number to the host.  Every thread of every CTA comes here.
__device__ __forceinline__ void publish(const DoneFlag& done) {
  if (!done.flag) return;
  __threadfence();
  __syncthreads();
  if (threadIdx.x == 0 && atomicAdd(done.ctas, 1) == (int)gridDim.x - 1) {
    *done.ctas = 0;
    __threadfence_system();
    *(volatile unsigned int*)done.flag = done.number;
  }
}

__device__ __forceinline__ unsigned long long ld_volatile64(const unsigned long long* p) {
  return *(const volatile unsigned long long*)p;
}
__device__ __forceinline__ void st_volatile64(unsigned long long* p, unsigned long long v) {
  *(volatile unsigned long long*)p = v;
}

// Look-back words: [63:34] tag (the call's 27-bit epoch * 8 + the pass, so words
// of earlier calls and passes never look published), [33:32] 1 = tile aggregate, 2 = inclusive
// prefix, [31:0] value.
__device__ __forceinline__ unsigned long long lb_word(uint32_t tag, uint32_t flag, uint32_t value) {
  return ((unsigned long long)tag << 34) | ((unsigned long long)flag << 32) | value;
}

// Sum of the values published by tiles before `tile` for one lane of a
// look-back table with `stride` words per tile.  Predecessors are read
// kLookAhead at a time (independent loads in flight together), then consumed
// newest first until an inclusive prefix appears; a word not yet published is
// polled (bounded) before the walk goes on.
constexpr int kLookAhead = 4;
__device__ __forceinline__ bool lb_ready(unsigned long long w, uint32_t tag) {
  return (uint32_t)(w >> 34) == tag && ((w >> 32) & 3u) != 0;
}
__device__ uint32_t look_back(const unsigned long long* status, int tile, int stride, int lane, uint32_t tag,
                              int* err) {
  uint32_t excl = 0;
  for (int j = tile - 1; j >= 0; j -= kLookAhead) {
    const int k = min(kLookAhead, j + 1);
    unsigned long long w[kLookAhead];
#pragma unroll
    for (int i = 0; i < kLookAhead; ++i)
      if (i < k) w[i] = ld_volatile64(status + (size_t)(j - i) * stride + lane);
#pragma unroll
    for (int i = 0; i < kLookAhead; ++i) {
      if (i >= k) break;
      long long spins = 0;
      const unsigned long long start = lb_ready(w[i], tag) ? 0 : global_ns();
      while (!lb_ready(w[i], tag)) {
        if (wait_over(spins, start)) {
          set_error(err);
          return excl;
        }
        __nanosleep(32);  // a polling warp yields its issue slots to the SM's other warps
        w[i] = ld_volatile64(status + (size_t)(j - i) * stride + lane);
      }
      excl += (uint32_t)w[i];
      if (((w[i] >> 32) & 3u) == 2u) return excl;
    }
  }
  return excl;
}

// Sum of the values published by tiles before `tile` in a table of one word
// per tile, looked back by a whole warp: lane i reads tile j - i, so one round
// trip covers 32 predecessors.  The ready prefix of lanes up to the first
// inclusive prefix is summed; a round that meets an unpublished word first
// consumes the ready lanes before it and polls again (bounded).  All 32 lanes
// call it and get the same result.
__device__ uint32_t warp_look_back(const unsigned long long* status, int tile, uint32_t tag, int* err) {
  const int lane = threadIdx.x & 31;
  uint32_t excl = 0;
  int j = tile - 1;
  long long spins = 0;
  unsigned long long start = 0;
  while (j >= 0) {
    const int t = j - lane;
    const unsigned long long w = t >= 0 ? ld_volatile64(status + t) : 0ull;
    const bool ready = t < 0 || lb_ready(w, tag);
    const bool incl = t < 0 || (ready && ((w >> 32) & 3u) == 2u);
    const unsigned not_ready = __ballot_sync(0xffffffffu, !ready);
    const unsigned incl_mask = __ballot_sync(0xffffffffu, incl);
    const int first_nr = not_ready ? __ffs(not_ready) - 1 : 32;
    const int first_incl = incl_mask ? __ffs(incl_mask) - 1 : 32;
    const int take = first_nr <= first_incl ? first_nr : first_incl + 1;  // lanes consumed by this read
    uint32_t v = lane < take && t >= 0 ? (uint32_t)w : 0u;
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) v += __shfl_xor_sync(0xffffffffu, v, off);
    excl += v;
    if (first_incl < first_nr) return excl;  // reached an inclusive prefix (or the first tile)
    j -= take;
    if (take == 0) {  // the nearest unpublished word: poll it
      if (start == 0) start = global_ns();
      if (wait_over(spins, start)) {
        if (lane == 0) set_error(err);
        return excl;
      }
    } else {
      spins = 0;
      start = 0;
    }
  }
  return excl;
}

// Called by one warp: turns the per-warp counts s_warp[0..kW) into exclusive
// offsets (s_warp[kW] = the tile's total), publishes the tile's aggregate,
// looks back, publishes the inclusive prefix and returns the tile's exclusive
// prefix.
template <int kW>
__device__ uint32_t tile_prefix(uint32_t* s_warp, unsigned long long* status, int tile, uint32_t tag, int* err) {
  const int lane = threadIdx.x & 31;
  const uint32_t c = lane < kW ? s_warp[lane] : 0u;
  uint32_t incl = c;
  for (int off = 1; off < 32; off <<= 1) {
    const uint32_t t = __shfl_up_sync(0xffffffffu, incl, off);
    if (lane >= off) incl += t;
  }
  const uint32_t run = __shfl_sync(0xffffffffu, incl, 31);
  unsigned long long* st = status + tile;
  if (lane == 0) st_volatile64(st, lb_word(tag, tile == 0 ? 2u : 1u, run));
  __syncwarp();
  if (lane < kW) s_warp[lane] = incl - c;
  if (lane == 0) s_warp[kW] = run;
  if (tile == 0) return 0;
  const uint32_t excl = warp_look_back(status, tile, tag, err);
  if (lane == 0) st_volatile64(st, lb_word(tag, 2u, excl + run));
  return excl;
}

constexpr int kCountValues = 1 << 14;
// Control words of a call, zeroed by one memset before it.
struct Control {
  uint32_t hist[kPasses * kBuckets];  // digit counts
  uint32_t range_counts[kBuckets];    // keys per range bucket
  uint32_t range[2];                  // max of ~key (so the minimum), max key
  int keys;                           // compacted keys
  int no_hit;                         // 1: some input word was NO_HIT
  int done[4];                        // CTAs finished: compaction, range histogram, digit histogram, split
  int barrier[3];                     // CTAs at the barriers of the bitmap's cooperative kernels
  int tiles[kPasses];                 // tile counters: digit passes
  int unique_tiles, bucket_items;
  int split_over;                     // 1: a range of the split got more keys than it holds
};
// Words one kernel of a call leaves for the next; not cleared.
struct Plan {
  int path;               // feedback unique: kPath...
  uint32_t bitmap_words, range_shift;
  int clear;              // the bitmap is wider than what the compaction cleared
  int skip[kPasses];      // digit pass not needed
  int unstable[kPasses];  // first pass: equal digits may leave in any order
  int src[kPasses], dst[kPasses], last;  // buffers of the passes, and where the keys end up
  int counting;           // sort: the keys take this many values from `lowest` on (0: too many), and are counted
  uint32_t lowest;
  uint32_t split;         // sort: factor of the split's linear map (0: the keys take the digit passes)
  uint32_t values[kCountValues];         // keys of each value; or of each range of the split, and their starts
  uint32_t offsets[kPasses * kBuckets];  // global start of each digit
  uint32_t range_offsets[kBuckets];
  uint32_t cursors[kBuckets * kCursorStride];
  uint32_t segment_bits[1 << (kMaxSpanLog2 - 15)];  // set bits per 1024 words of the bitmap
};
constexpr int kPathEmpty = 0, kPathDirect = 1, kPathPartition = 2, kPathRadix = 3;

struct SortScratchLayout {
  uint32_t* keys_a;
  uint32_t* keys_b;
  size_t key_words;  // of both together
  uint32_t* bitmap;
  Control* control;
  Plan* plan;
  size_t bitmap_bits;  // of the bitmap that the compaction clears
  size_t bitmap_cap;   // and that there is room for
  size_t bytes;
};

SortScratchLayout layout(void* base, int n, bool unique = false) {
  auto up = [](size_t v) { return (v + 255) & ~(size_t)255; };
  SortScratchLayout l{};
  size_t off = 0;
  uint8_t* b = static_cast<uint8_t*>(base);
  l.control = reinterpret_cast<Control*>(b + off); off += up(sizeof(Control));
  l.plan = reinterpret_cast<Plan*>(b + off); off += up(sizeof(Plan));
  l.keys_a = reinterpret_cast<uint32_t*>(b + off); off += up((size_t)n * 4 + 16);
  l.keys_b = reinterpret_cast<uint32_t*>(b + off);
  const size_t widest = unique && n <= kDirectWords ? ((size_t)1 << kMaxSpanLog2) / 8 : 0;
  off += up(std::max((size_t)n * 4 + 16, widest));
  l.key_words = (size_t)(b + off - reinterpret_cast<uint8_t*>(l.keys_a)) / 4;
  l.bitmap_bits = std::min<size_t>((((size_t)n * 4 + 16) / 16) * 16 * 8, (size_t)1 << kMaxSpanLog2);
  l.bitmap_cap = std::max(l.bitmap_bits, widest * 8);
  // the direct path leaves keys_b free; larger inputs may be partitioned into it
  if (n <= kDirectWords) l.bitmap = l.keys_b;
  else l.bitmap = reinterpret_cast<uint32_t*>(b + off), off += up(l.bitmap_bits / 8);
  l.bytes = off;
  return l;
}

// Exclusive scan of 256 values, 8 per lane, by one warp: row[i] becomes the sum
// of the values before it; returns the total.
__device__ __forceinline__ uint32_t warp_scan_256(const uint32_t* in, uint32_t* out) {
  const int lane = threadIdx.x & 31;
  uint32_t v[8], sum = 0;
#pragma unroll
  for (int k = 0; k < 8; ++k) { v[k] = in[lane * 8 + k]; sum += v[k]; }
  uint32_t incl = sum;
  for (int off = 1; off < 32; off <<= 1) {
    const uint32_t t = __shfl_up_sync(0xffffffffu, incl, off);
    if (lane >= off) incl += t;
  }
  uint32_t run = incl - sum;
  __syncwarp();
#pragma unroll
  for (int k = 0; k < 8; ++k) { out[lane * 8 + k] = run; run += v[k]; }
  return __shfl_sync(0xffffffffu, incl, 31);
}

// True in every thread of the CTA that finishes last of `ctas` (no CTA waits);
// what the other CTAs wrote before their call is visible to it.
__device__ __forceinline__ bool last_cta(int* done, int ctas) {
  __shared__ bool s_last;
  __threadfence();
  __syncthreads();
  if (threadIdx.x == 0) s_last = atomicAdd(done, 1) == ctas - 1;
  __syncthreads();
  if (s_last) __threadfence();
  return s_last;
}

// ---- compaction ---------------------------------------------------------------
// NodeToBlock's division of a node index (0 <= x < 2^31) by nodes_in_block d
// without a hardware divide: q = floor(x * M / 2^64) with M = ceil(2^64 / d).
// For x < 2^31 and d < 2^32 the product's excess x * (M - 2^64/d) / 2^64 is
// below 1/d, so the floor equals floor(x / d) exactly (Granlund & Montgomery,
// "Division by invariant integers using multiplication", 1994).  d = 1 passes
// x through.
struct Divider {
  unsigned long long m;  // 0: d == 1
};
inline Divider make_divider(uint32_t d) {
  Divider v;
  v.m = d <= 1 ? 0ull : ~0ull / d + 1ull;
  return v;
}
__device__ __forceinline__ uint32_t divide(uint32_t x, Divider v) {
  return v.m ? (uint32_t)__umul64hi((unsigned long long)x, v.m) : x;
}

// Tiles of 4096 words, grid-strided over the resident CTAs.  A thread owns 16
// words of a tile, read as four 16-byte loads when `words` is 16-byte aligned
// (scalar loads otherwise, and for the last, partial tile).  The next tile's
// loads are issued before the current tile is processed, so memory latency
// overlaps the work.  The per-word loop only drops NO_HIT words: each warp
// appends the words it keeps to its own region of shared memory, each thread's
// together (a ballot and two counts per row of 32 words instead: 349 us for the
// unique of 2^28 words, so 341), or row by row where a warp keeps every word
// of a tile (2^26 kept words of 199 values 250 us without that, 156 so; nine
// tenths of them kept 162 and 164).
// NodeToBlock, the key mapping and the filter run when the regions are
// flushed, on the kept words with every lane busy (at 10% kept words, doing
// them per word cost three quarters of the instructions of an issue-bound
// kernel).  The filter is a direct-mapped table of keys the CTA has kept
// before: a key found there is dropped.  Feedback repeats its frequent keys
// (neighbouring pixels hit the same blocks), and every later kernel reads
// what is kept here.  Warps race on the table without order; the worst that
// does is keep a repeat.  The CTA flushes, claiming its output range with one
// atomicAdd, only when a region could not take another tile or after its last
// tile; the regions go out coalesced.  (Regions of 640 words and 4096 filter
// entries leave 5 CTAs per SM; 1024 and 2048 took 403 us for the unique of
// 2^28 words where these take 364.)  Input words are read once, with
// evict-first loads, so they do not push the compacted keys out of L2.  Keys
// leave in any order.  The CTAs also clear the bitmap (they are done before
// the first kernel that sets bits), and the last one chooses the path.
constexpr int kRegion = 640;  // words per warp region; a tile adds at most 512
constexpr int kFilterLog2 = 12;
constexpr int kFlush = 2;  // words in flight per lane of a flush
constexpr uint32_t kNoKey = 0xffffffffu;  // NO_HIT's key: never kept

template <bool kVec>
__device__ __forceinline__ void load_words(int32_t (&w)[kItems], const int32_t* words, uint32_t n, uint32_t first) {
  // thread's words: first + r * 128 + j, r, j = 0..3
  if (kVec && first + (kItems * 32 - 4 * (threadIdx.x & 31)) <= n) {
#pragma unroll
    for (int r = 0; r < 4; ++r) {
      const int4 v = __ldcs(reinterpret_cast<const int4*>(words + first + r * 128));
      w[4 * r] = v.x; w[4 * r + 1] = v.y; w[4 * r + 2] = v.z; w[4 * r + 3] = v.w;
    }
  } else {
#pragma unroll
    for (int r = 0; r < 4; ++r)
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const uint32_t i = first + r * 128 + j;
        w[4 * r + j] = i < n ? __ldcs(words + i) : kNoHit;
      }
  }
}

template <bool kVec>
__global__ void __launch_bounds__(kThreads) compact_kernel(const int32_t* words, int n_words, int nib, Divider div,
                                                           uint32_t* keys, Control* ctl, Plan* plan, uint4* bitmap,
                                                           uint32_t bitmap_units, unsigned long long bitmap_cap,
                                                           int32_t* out, int* result) {
  __shared__ uint32_t s_range[2];  // max of ~key (so the minimum), max key
  __shared__ uint32_t s_keys[kWarps * kRegion];
  __shared__ uint32_t s_filter[1 << kFilterLog2];
  __shared__ uint32_t s_fill[2][kWarps];  // by tile parity: a warp may write the next tile's entry early
  __shared__ uint32_t s_base;
  const uint32_t n = (uint32_t)n_words;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const unsigned lt = (1u << lane) - 1;
  const uint32_t mine = warp * (kItems * 32) + lane * 4;  // offset of the thread's first word in a tile
  uint32_t* region = s_keys + warp * kRegion;
  volatile uint32_t* filter = s_filter;
  const uint32_t stride = gridDim.x * kTile;  // tiles of n < 2^31 words: base + stride stays below 2^32
  int32_t cur[kItems], nxt[kItems];
  uint32_t base = blockIdx.x * kTile;
  load_words<kVec>(cur, words, n, base + mine);
  for (uint32_t i = blockIdx.x * kThreads + threadIdx.x; i < bitmap_units; i += gridDim.x * kThreads)
    bitmap[i] = make_uint4(0u, 0u, 0u, 0u);
  for (int i = threadIdx.x; i < (1 << kFilterLog2); i += kThreads) s_filter[i] = kNoKey;
  if (threadIdx.x < 2) s_range[threadIdx.x] = 0;
  uint32_t not_min = 0, max_key = 0;
  uint32_t fill = 0;  // words in this warp's region
  bool dropped = false;
  for (int parity = 0; base < n; base += stride, parity ^= 1) {
    const uint32_t next = base + stride;
    load_words<kVec>(nxt, words, n, next + mine);
    const uint32_t before = fill;
    {  // each thread's kept words together: one scan for the tile's 16 words
      uint32_t count = 0;
#pragma unroll
      for (int q = 0; q < kItems; ++q) count += cur[q] != kNoHit;  // words past the end were loaded as NO_HIT
      uint32_t incl = count;
#pragma unroll
      for (int off = 1; off < 32; off <<= 1) {
        const uint32_t t = __shfl_up_sync(0xffffffffu, incl, off);
        if (lane >= off) incl += t;
      }
      const uint32_t total = __shfl_sync(0xffffffffu, incl, 31);
      if (total == kItems * 32) {  // all of them: threads' runs of 16 would meet in two banks
#pragma unroll
        for (int q = 0; q < kItems; ++q) region[fill + q * 32 + lane] = (uint32_t)cur[q];
      } else {
        uint32_t* at = region + fill + (incl - count);
#pragma unroll
        for (int q = 0; q < kItems; ++q)
          if (cur[q] != kNoHit) *at++ = (uint32_t)cur[q];
      }
      fill += total;
    }
    {
      const uint32_t first = base + warp * (kItems * 32);
      dropped = dropped || (first < n && fill - before < min(n - first, (uint32_t)kItems * 32));
    }
#pragma unroll
    for (int q = 0; q < kItems; ++q) cur[q] = nxt[q];
    if (lane == 0) s_fill[parity][warp] = fill;
    __syncthreads();
    bool flush = next >= n;
#pragma unroll
    for (int k = 0; k < kWarps; ++k) flush = flush || s_fill[parity][k] > kRegion - kItems * 32;
    if (!flush) continue;
    // words to keys, in place (a round writes at or below what it has read)
    uint32_t kept = 0;
    for (uint32_t j0 = 0; j0 < fill; j0 += 32 * kFlush) {
      uint32_t key[kFlush];
      bool keep[kFlush];
#pragma unroll
      for (int r = 0; r < kFlush; ++r) {
        const uint32_t j = j0 + r * 32 + lane;
        keep[r] = j < fill;
        int32_t v = keep[r] ? (int32_t)region[j] : 0;
        if (v > 0 && nib > 0) v = (int32_t)(((divide((uint32_t)((v >> 1) - 1), div) + 1) << 1) | (v & 1));
        key[r] = (uint32_t)v ^ 0x80000000u;
      }
#pragma unroll
      for (int r = 0; r < kFlush; ++r) {
        const uint32_t h = (key[r] * 0x9e3779b1u) >> (32 - kFilterLog2);
        if (keep[r]) {
          if (filter[h] == key[r]) keep[r] = false;
          else filter[h] = key[r];
        }
      }
      __syncwarp();  // the round's words are read before keys overwrite them
#pragma unroll
      for (int r = 0; r < kFlush; ++r) {
        const unsigned mask = __ballot_sync(0xffffffffu, keep[r]);
        if (keep[r]) {
          region[kept + __popc(mask & lt)] = key[r];
          not_min = max(not_min, ~key[r]);
          max_key = max(max_key, key[r]);
        }
        kept += __popc(mask);
      }
      __syncwarp();
    }
    __syncthreads();  // every warp has read this tile's fills
    if (lane == 0) s_fill[parity][warp] = kept;
    __syncthreads();
    if (threadIdx.x == 0) {
      uint32_t total = 0;
      for (int k = 0; k < kWarps; ++k) total += s_fill[parity][k];
      s_base = total ? (uint32_t)atomicAdd(&ctl->keys, (int)total) : 0u;
    }
    __syncthreads();
    uint32_t at = s_base;
    for (int k = 0; k < warp; ++k) at += s_fill[parity][k];
    for (uint32_t j = lane; j < kept; j += 32) keys[at + j] = region[j];
    fill = 0;
    __syncthreads();  // s_base is reused by the next flush
  }
  not_min = __reduce_max_sync(0xffffffffu, not_min);
  max_key = __reduce_max_sync(0xffffffffu, max_key);
  __syncthreads();  // s_range zeroed
  if (lane == 0) {
    atomicMax(&s_range[0], not_min);
    atomicMax(&s_range[1], max_key);
    if (dropped) ctl->no_hit = 1;
  }
  __syncthreads();
  if (threadIdx.x < 2 && s_range[threadIdx.x]) atomicMax(&ctl->range[threadIdx.x], s_range[threadIdx.x]);
  if (!last_cta(&ctl->done[0], gridDim.x) || threadIdx.x != 0) return;
  // the path: a bitmap when it fits, straight or range by range
  const volatile Control* c = ctl;
  const int m = c->keys;
  const uint32_t lo = ~c->range[0], hi = c->range[1];
  const unsigned long long span = (unsigned long long)hi - (unsigned long long)lo + 1ull;
  constexpr unsigned long long kSlice = kDirectSliceWords * 32ull;
  const unsigned long long slices = (span + kSlice - 1) / kSlice;
  const bool direct = n_words <= kDirectWords || m <= kDirectKeys || slices == 1 ||
                      (slices <= kDirectFewSlices && m * slices <= kDirectReads);
  const int path = m == 0 ? kPathEmpty : span > bitmap_cap ? kPathRadix : direct ? kPathDirect : kPathPartition;
  plan->path = path;
  plan->bitmap_words = (uint32_t)((span + 31) / 32);
  plan->clear = path == kPathDirect && span > bitmap_units * 128ull;
  const int bits = span > 1 ? 64 - __clzll((long long)(span - 1)) : 0;  // bits of the largest key - min
  plan->range_shift = bits > 8 ? (uint32_t)(bits - 8) : 0u;
  if (path == kPathEmpty) {
    if (c->no_hit) out[0] = kNoHit;
    result[0] = c->no_hit ? 1 : 0;
  }
  // the host may be waiting for this to launch the radix passes
  *(volatile int*)&result[1] = path;
}

// Compaction launch: 16-byte loads when `words` allows them.
cudaError_t launch_compact(int grid, const int32_t* words, int n, int nib, const SortScratchLayout& l, int32_t* out,
                           int* result, cudaStream_t s) {
  const Divider div = make_divider((uint32_t)nib);
  uint4* bitmap = reinterpret_cast<uint4*>(l.bitmap);
  const uint32_t units = (uint32_t)(l.bitmap_bits / 128);
  if ((reinterpret_cast<uintptr_t>(words) & 15) == 0)
    compact_kernel<true><<<grid, kThreads, 0, s>>>(words, n, nib, div, l.keys_a, l.control, l.plan, bitmap, units,
                                                  l.bitmap_cap, out, result);
  else
    compact_kernel<false><<<grid, kThreads, 0, s>>>(words, n, nib, div, l.keys_a, l.control, l.plan, bitmap, units,
                                                   l.bitmap_cap, out, result);
  return cudaGetLastError();
}

// ---- digit histograms ----------------------------------------------------------
// All four digits' counts in one read of the keys.  Random digits collide in
// the banks of a 256-entry table (3 to 4 wavefronts per atomic: the counting
// took 139 us on 2^26 keys with a copy of the keys beside it); here each lane
// of a warp counts in its own bank, 256 x 32 counters per digit, so an atomic
// is one wavefront whatever the digits are.  One CTA of 1024 threads per SM
// holds the 128 KB of counters.  The last CTA turns the counts into offsets
// and lays out the passes: a digit that is the same in every key needs none,
// and keys of up to kCountValues different values are not passed over at all.
constexpr int kHistThreads = 1024;
// True if digit p has the value v in about as many of m keys as it would have
// if the keys were spread evenly over [lo, hi]: within what a range of the
// split holds beyond its even share.
__device__ __forceinline__ bool even_digit(uint32_t count, int p, uint32_t v, uint32_t lo, uint32_t hi, uint32_t m) {
  const uint32_t unit = 1u << (8 * p);
  auto below = [&](unsigned long long x) {  // numbers below x whose digit p is v
    const unsigned long long whole = x >> (8 * p + 8);
    const long long rest = (long long)(x - (whole << (8 * p + 8))) - (long long)v * unit;
    return whole * unit + (unsigned long long)(rest < 0 ? 0 : rest > (long long)unit ? (long long)unit : rest);
  };
  const float share = (float)(below((unsigned long long)hi + 1) - below(lo)) * (float)m / ((float)(hi - lo) + 1.f);
  return (float)count <= share * 1.0625f + 8.f * sqrtf(share) + 8.f;
}
constexpr int kHistSmemBytes = kPasses * kBuckets * 32 * 4;
__global__ void __launch_bounds__(kHistThreads, 1) digit_hist_kernel(const uint32_t* keys, int n, const int* count,
                                                                    uint32_t flip, bool in_place, int split_ranges,
                                                                    Control* ctl, Plan* plan) {
  extern __shared__ __align__(128) uint32_t s_hist[];
  __shared__ uint32_t s_max[kPasses];
  uint32_t not_min = 0, max_key = 0;
  dependents_may_start();
  for (int i = threadIdx.x; i < kPasses * kBuckets * 8; i += kHistThreads)
    reinterpret_cast<uint4*>(s_hist)[i] = make_uint4(0, 0, 0, 0);
  wait_for_dependency();
  for (int i = blockIdx.x * kHistThreads + threadIdx.x; i < kCountValues; i += gridDim.x * kHistThreads)
    plan->values[i] = 0;
  const uint32_t m = count ? (uint32_t)*count : (uint32_t)n;
  __syncthreads();
  const int lane = threadIdx.x & 31;
  uint32_t* col = s_hist + lane;
  auto add = [&](uint32_t k) {
    k ^= flip;
    not_min = max(not_min, ~k);
    max_key = max(max_key, k);
#pragma unroll
    for (int p = 0; p < kPasses; ++p) atomicAdd(col + (p * kBuckets + ((k >> (8 * p)) & 255u)) * 32, 1u);
  };
  {  // 16-byte units from the first boundary on, four in flight per thread, and the keys beside them
    const uint32_t head = min(m, (uint32_t)(-(reinterpret_cast<uintptr_t>(keys) >> 2) & 3u));
    const uint32_t units = (m - head) / 4, step = gridDim.x * kHistThreads;
    const uint4* k4 = reinterpret_cast<const uint4*>(keys + head);
    uint32_t i = blockIdx.x * kHistThreads + threadIdx.x;
    for (; i + 3 * step < units; i += 4 * step) {  // below 2^28 + 4 * step
      uint4 v[4];
#pragma unroll
      for (int r = 0; r < 4; ++r) v[r] = __ldg(k4 + i + r * step);
#pragma unroll
      for (int r = 0; r < 4; ++r) add(v[r].x), add(v[r].y), add(v[r].z), add(v[r].w);
    }
    for (; i < units; i += step) {
      const uint4 v = __ldg(k4 + i);
      add(v.x), add(v.y), add(v.z), add(v.w);
    }
    if (blockIdx.x == 0) {
      if (threadIdx.x < head) add(__ldg(keys + threadIdx.x));
      if (threadIdx.x < m - head - units * 4) add(__ldg(keys + head + units * 4 + threadIdx.x));
    }
  }
  __syncthreads();
  {  // thread t: digit value t of the 4 x 256, its 32 columns from its own banks on
    uint32_t sum = 0;
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      const uint4 v = reinterpret_cast<const uint4*>(s_hist)[threadIdx.x * 8 + ((lane + k) & 7)];
      sum += v.x + v.y + v.z + v.w;
    }
    if (sum) atomicAdd(&ctl->hist[threadIdx.x], sum);
  }
  if (in_place) {
    not_min = __reduce_max_sync(0xffffffffu, not_min);
    max_key = __reduce_max_sync(0xffffffffu, max_key);
    if (lane == 0) {
      atomicMax(&ctl->range[0], not_min);
      atomicMax(&ctl->range[1], max_key);
    }
  }
  if (!last_cta(&ctl->done[2], gridDim.x)) return;
  uint32_t* counts = s_hist;  // reused
  __syncthreads();
  counts[threadIdx.x] = *(volatile uint32_t*)&ctl->hist[threadIdx.x];
  if (threadIdx.x < kPasses) s_max[threadIdx.x] = 0;
  __syncthreads();
  {
    const uint32_t most = __reduce_max_sync(0xffffffffu, counts[threadIdx.x]);
    if (lane == 0) atomicMax(&s_max[threadIdx.x >> 8], most);
  }
  __syncthreads();
  if (threadIdx.x < 32 * kPasses) {
    const int p = threadIdx.x >> 5;
    warp_scan_256(counts + p * kBuckets, plan->offsets + p * kBuckets);
  }
  const uint32_t lo = ~*(volatile uint32_t*)&ctl->range[0], hi = *(volatile uint32_t*)&ctl->range[1];
  const bool uneven = __syncthreads_or(
      split_ranges && !even_digit(counts[threadIdx.x], threadIdx.x >> 8, threadIdx.x & 255u, lo, hi, m));
  if (threadIdx.x == 0) {
    plan->split = split_ranges && !uneven && hi - lo >= (uint32_t)kCountValues
                      ? (uint32_t)(((unsigned long long)split_ranges << 32) / ((unsigned long long)(hi - lo) + 1))
                      : 0u;
    plan->counting = in_place && hi - lo < (uint32_t)kCountValues ? (int)(hi - lo) + 1 : 0;
    plan->lowest = lo;
    int active = 0;
    bool skip[kPasses];
    for (int p = 0; p < kPasses; ++p) active += !(skip[p] = s_max[p] == m);
    // in place: buffer 0 is both where the keys come from and where they go,
    // so one pass alone has nowhere to go and another one runs with it
    if (in_place && active == 1) {
      skip[skip[0] ? 0 : 1] = false;
      active = 2;
    }
    int at = 0, j = 0;
    for (int p = 0; p < kPasses; ++p) {
      plan->skip[p] = skip[p];
      if (skip[p]) continue;
      plan->src[p] = at;
      // in place: 0 -> 1 -> 2 -> 1 -> 0 for four passes; else 0 and 1 in turn
      at = in_place ? (j == active - 1 ? 0 : (j & 1) ? 2 : 1) : 1 - at;
      plan->dst[p] = at;
      // the first pass may leave equal digits in any order (no earlier pass
      // has ordered them): worth it where no digit is so frequent that its
      // count is contended
      plan->unstable[p] = j == 0 && s_max[p] <= m / 16;
      ++j;
    }
    plan->last = at;
  }
}

// ---- bulk async copies into shared memory ------------------------------------
// A tile of keys arrives in shared memory by one cp.async.bulk (the copy
// engine moves it; no thread holds it in registers), and its completion is an
// mbarrier phase with a transaction count.
__device__ __forceinline__ uint32_t smem_addr(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void mbar_init(unsigned long long* bar) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_addr(bar)) : "memory");
}
// Makes the barriers' initialisation visible to the copy engine.
__device__ __forceinline__ void mbar_init_fence() {
  asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
}
__device__ __forceinline__ bool mbar_try_wait(unsigned long long* bar, uint32_t parity) {
  uint32_t done;
  asm volatile(
      "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}\n"
      : "=r"(done)
      : "r"(smem_addr(bar)), "r"(parity)
      : "memory");
  return done != 0;
}
// Waits for the phase of `bar` with parity `parity`; false (error flag set)
// when the wait runs out.
__device__ __forceinline__ bool mbar_wait(unsigned long long* bar, uint32_t parity, int* err) {
  if (mbar_try_wait(bar, parity)) return true;
  long long spins = 0;
  const unsigned long long start = global_ns();
  while (!mbar_try_wait(bar, parity)) {
    if (wait_over(spins, start)) {
      set_error(err);
      return false;
    }
  }
  return true;
}
// Copies `bytes` (a multiple of 16, both addresses 16-byte aligned) from
// global to shared memory; the copy completes the current phase of `bar`.
// Shared memory last touched by the threads is handed to the copy engine by
// the proxy fence.
__device__ __forceinline__ void bulk_load(void* dst, const void* src, uint32_t bytes, unsigned long long* bar) {
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_addr(bar)), "r"(bytes) : "memory");
  if (bytes == 0) return;  // the phase is complete already
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                   smem_addr(dst)),
               "l"(src), "r"(bytes), "r"(smem_addr(bar))
               : "memory");
}

// ---- one counting pass over 8 bits ---------------------------------------------
// Persistent CTAs of 512 threads claim tiles of 8192 keys in order from
// the pass's tile counter until the keys run out (the count is read on the
// device: for feedback unique only the compaction knows it).  A CTA claims its
// next tile when it starts the current one, and the next tile's keys come into
// the other half of a double buffer by one bulk async copy while the current
// tile is ranked, looked back and written out.  (A next tile is always above
// its CTA's current one, so the lowest unfinished tile is always some CTA's
// current tile and every look-back ends.)  Per tile:
// - ranking, stable: a warp's 512 keys in 16 rounds of 32: the lanes of a
//   round holding the same digit find one another through a per-warp table of
//   peer masks in shared memory (each lane ORs its bit into its digit's word;
//   one shared atomic instead of eight ballots and the selects between them,
//   which had made the pass issue-bound at 4.9 warp instructions per key); the
//   group's first lane adds the group to the warp's count of that digit with
//   one atomic, clears the mask word and shares the old count; ranks follow
//   lane order inside the group, and rounds apply in order.  The pass is bound
//   by the shared-memory pipe, and these accesses by random digits are most of
//   its wavefronts, so the first pass, which has no earlier order to keep,
//   takes its ranks from one atomic per key on the CTA's counts instead;
// - the per-digit counts over warps become offsets; the tile's count per digit
//   is published at once (the look-back's aggregate); the 256 counts are
//   scanned into the tile-local start of each digit run, which is added into
//   the per-warp offsets;
// - the keys (held in registers since the ranking) are staged in tile-local
//   sorted order in place, in the buffer they came from (one shared load of
//   the warp's offset per key);
// - one thread per digit looks back for the digit run's global position;
// - each digit run goes out contiguously.
// 8192-key tiles halve the look-back's walk per key twice over 4096-key ones:
// half the tiles, and half as many tiles in flight behind a tile's
// predecessors.
constexpr int kDigitThreads = 512;
constexpr int kDigitWarps = kDigitThreads / 32;
constexpr int kDigitTile = kDigitThreads * kItems;  // 8192 keys
static_assert(kCountValues <= 2 * kDigitTile, "the tile buffers hold the value counters");
// shared memory: two tile buffers, per-warp counts and peer masks, the run
// starts and offsets, 8 warp totals, two mbarriers and the next tile's index
constexpr int kDigitSmemBytes = (2 * kDigitTile + 2 * kDigitWarps * kBuckets + 2 * kBuckets + 8) * 4 + 32;

// Bytes copied for tile t of m keys: whole 16-byte units; the up to three keys
// after them are read straight from memory when they are ranked.
__device__ __forceinline__ uint32_t digit_tile_bytes(int t, int m) {
  const int valid = min(kDigitTile, m - t * kDigitTile);
  return (uint32_t)(valid / 4 * 16);
}

// ---- few values ----------------------------------------------------------------
// Keys of few different values need no passes: the first pass's launch counts
// each value and the second's writes the runs (four launches over 2^26 keys of
// 201 values took 1490 us, as every lane's digit met in two words; counted,
// 252).  The counters lie in the CTA's shared memory, one per lane and value
// where there is room for that, so that frequent values do not queue.
__device__ __forceinline__ void count_values(const uint32_t* keys, int n, uint32_t flip, Plan* plan, uint32_t* smem) {
  const int values = plan->counting, lane = threadIdx.x & 31;
  const uint32_t lo = plan->lowest;
  const bool by_lane = values * 32 <= kCountValues;
  const int words = by_lane ? values * 32 : values, scale = by_lane ? 32 : 1, col = by_lane ? lane : 0;
  for (uint32_t i = threadIdx.x; i < (uint32_t)words; i += blockDim.x) smem[i] = 0;
  __syncthreads();
  const uint32_t step = gridDim.x * blockDim.x;
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < (uint32_t)n; i += 4 * step) {  // n < 2^30
    uint32_t k[4];
#pragma unroll
    for (int r = 0; r < 4; ++r) k[r] = i + r * step < (uint32_t)n ? (__ldg(keys + i + r * step) ^ flip) - lo : ~0u;
#pragma unroll
    for (int r = 0; r < 4; ++r)
      if (k[r] != ~0u) atomicAdd(&smem[k[r] * scale + col], 1u);
  }
  __syncthreads();
  for (uint32_t v = threadIdx.x; v < (uint32_t)values; v += blockDim.x) {
    uint32_t sum = 0;
    if (by_lane) {
#pragma unroll 8
      for (int k = 0; k < 32; ++k) sum += smem[v * 32 + ((lane + k) & 31)];
    } else {
      sum = smem[v];
    }
    if (sum) atomicAdd(&plan->values[v], sum);
  }
}

// Every CTA scans the counts and writes its part of the runs, kValues of them at
// most (the scan and the bisection are unrolled over that many: 300 thousand
// keys of 201 values 47 us with 16384 always, 35 with 512; loops over the values
// there are were 25% slower for 16000).
template <int kValues>
__device__ __forceinline__ void write_values_of(uint32_t* out, int n, uint32_t flip, const Plan* plan, uint32_t* smem) {
  __shared__ uint32_t s_warp[kDigitWarps];
  const int values = plan->counting, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const uint32_t lo = plan->lowest;
  // smem[v]: the first position of value v; thread t scans `per` values
  constexpr int kPer = kValues / kDigitThreads;
  for (int v = threadIdx.x; v < kValues; v += kDigitThreads) smem[v] = v < values ? plan->values[v] : 0u;
  __syncthreads();
  uint32_t sum = 0;
  for (int k = 0; k < kPer; ++k) sum += smem[threadIdx.x * kPer + ((k + lane) & (kPer - 1))];
  uint32_t incl = sum;
#pragma unroll
  for (int off = 1; off < 32; off <<= 1) {
    const uint32_t t = __shfl_up_sync(0xffffffffu, incl, off);
    if (lane >= off) incl += t;
  }
  if (lane == 31) s_warp[warp] = incl;
  __syncthreads();
  uint32_t run = incl - sum + __reduce_add_sync(0xffffffffu, lane < warp ? s_warp[lane] : 0u);  // warp < 16
  for (int k = 0; k < kPer; ++k) {
    uint32_t* at = smem + threadIdx.x * kPer + k;
    const uint32_t c = *at;
    *at = run;
    run += c;
  }
  __syncthreads();
  // each thread four neighbouring positions at a time: the value of the first
  // by bisection (the last value that starts at or before it and has keys),
  // the others' by stepping on
  const uint32_t step = gridDim.x * kDigitThreads * 4u;
  const bool whole = (reinterpret_cast<uintptr_t>(out) & 15) == 0;
  for (uint32_t p = (blockIdx.x * kDigitThreads + threadIdx.x) * 4u; p < (uint32_t)n; p += step) {
    int v = 0;
#pragma unroll
    for (int half = kValues / 2; half > 0; half >>= 1)
      if (v + half < values && smem[v + half] <= p) v += half;
    uint32_t q[4];
#pragma unroll
    for (int r = 0; r < 4; ++r) {
      while (v + 1 < values && smem[v + 1] <= p + r) ++v;
      q[r] = (lo + (uint32_t)v) ^ flip;
    }
    if (whole && p + 4 <= (uint32_t)n) {
      *reinterpret_cast<uint4*>(out + p) = make_uint4(q[0], q[1], q[2], q[3]);
    } else {
#pragma unroll
      for (int r = 0; r < 4; ++r)
        if (p + r < (uint32_t)n) out[p + r] = q[r];
    }
  }
}

__device__ __forceinline__ void write_values(uint32_t* out, int n, uint32_t flip, const Plan* plan, uint32_t* smem) {
  if (plan->counting <= kDigitThreads) write_values_of<kDigitThreads>(out, n, flip, plan, smem);
  else write_values_of<kCountValues>(out, n, flip, plan, smem);
}

// Key `li` of a partial tile of `valid` keys: in shared memory, or past the last
// whole 16-byte unit in global memory.
__device__ __forceinline__ uint32_t tail_key(const uint32_t* s_tile_keys, const uint32_t* tile_keys, int li,
                                             int valid) {
  return li < (valid & ~3) ? s_tile_keys[li] : li < valid ? tile_keys[li] : 0u;
}

// Ranks a warp's kRounds * 32 keys (positions w0 + r * 32 + lane of `src`, or
// of the partial tile `tail`) among the warp's keys of the same digit, stable;
// two 16-bit ranks per word.
template <bool kFull, int kRounds>
__device__ __forceinline__ void rank_keys(const uint32_t* src, const uint32_t* tail, uint32_t (&keys)[kRounds],
                                          uint32_t (&ranks)[(kRounds + 1) / 2], uint32_t* s_count, uint32_t* s_peers,
                                          int shift, uint32_t flip, int valid, int w0, int lane) {
#pragma unroll
  for (int r = 0; r < kRounds; ++r) {
    const int li = w0 + r * 32 + lane;
    const bool ok = kFull || li < valid;
    keys[r] = kFull ? src[li] : tail_key(src, tail, li, valid);
    const uint32_t d = ((keys[r] >> shift) & 255u) ^ flip;
    if (ok) atomicOr(&s_peers[d], 1u << lane);
    __syncwarp();
    const unsigned peers = ok ? s_peers[d] : (1u << lane);
    __syncwarp();  // every lane has read its mask before the leader clears it
    const int leader = __ffs(peers) - 1;
    uint32_t before = 0;
    if (ok && lane == leader) {
      s_peers[d] = 0u;
      before = atomicAdd(&s_count[d], (uint32_t)__popc(peers));
    }
    before = __shfl_sync(0xffffffffu, before, leader);
    __syncwarp();  // the cleared mask is in place before the next round's ORs
    const uint32_t rank = before + __popc(peers & ((1u << lane) - 1));
    ranks[r / 2] = (r & 1) ? ranks[r / 2] | (rank << 16) : rank;
  }
}

// Buffers of the passes by the plan's numbers: source 0 may be another memory
// than destination 0 (an unaligned array is sorted from a copy).
struct DigitBuffers {
  const uint32_t* in0;
  uint32_t *out0, *b1, *b2;
};

__device__ __forceinline__ void digit_kernel_cta(const DigitBuffers bufs, int n, const int* count, int pass,
                                                 uint32_t flip, Plan* plan, unsigned long long* status,
                                                 int* tile_counter, uint32_t tag, int* err) {
  extern __shared__ __align__(128) uint32_t smem[];
  uint32_t* s_warp = smem + 2 * kDigitTile;         // [warp][digit] counts, then offsets
  uint32_t* s_peers = s_warp + kDigitWarps * kBuckets;  // [warp][digit] peer masks of a round
  uint32_t* s_start = s_peers + kDigitWarps * kBuckets; // tile-local start of each digit run
  uint32_t* s_off = s_start + kBuckets;                 // global position - tile-local position
  uint32_t* s_wsum = s_off + kBuckets;                  // per digit warp: its digits' counts summed
  unsigned long long* s_bar = reinterpret_cast<unsigned long long*>(s_wsum + 8);
  int* s_next = reinterpret_cast<int*>(s_bar + 2);
  // what does not depend on the kernel before runs beside it
  dependents_may_start();
  for (int i = threadIdx.x; i < 2 * kDigitWarps * kBuckets; i += kDigitThreads) s_warp[i] = 0;
  if (threadIdx.x == 0) {
    mbar_init(&s_bar[0]);
    mbar_init(&s_bar[1]);
    mbar_init_fence();
  }
  wait_for_dependency();
  if (plan->counting) {
    if (pass == 0) count_values(bufs.in0, n, 0x80000000u, plan, smem);
    if (pass == 1) write_values(bufs.out0, n, 0x80000000u, plan, smem);
    return;
  }
  if (plan->skip[pass]) return;
  const int m = count ? *count : n;
  const int shift = 8 * pass;
  const bool unstable = plan->unstable[pass] != 0;
  const int src = plan->src[pass], dst = plan->dst[pass];
  const uint32_t* in = src == 0 ? bufs.in0 : src == 1 ? bufs.b1 : bufs.b2;
  uint32_t* out = dst == 0 ? bufs.out0 : dst == 1 ? bufs.b1 : bufs.b2;
  const uint32_t* digit_base = plan->offsets + pass * kBuckets;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int w0 = warp * (kItems * 32);  // warp `warp` ranks keys [w0, w0 + 512) of a tile
  const int rows = unstable ? 1 : kDigitWarps;  // rows of counts in use
  uint32_t* s_mine = unstable ? s_warp : s_warp + warp * kBuckets;  // this warp's row
  if (threadIdx.x == 0) {
    const int t = atomicAdd(tile_counter, 1);
    *s_next = t;
    if ((long long)t * kDigitTile < m) bulk_load(smem, in + (size_t)t * kDigitTile, digit_tile_bytes(t, m), &s_bar[0]);
  }
  __syncthreads();
  int tile = *s_next;
  __syncthreads();  // every thread has read s_next before it is rewritten
  uint32_t phases = 0u;  // bit b: parity of buffer b's next completion
  int b = 0;
  while ((long long)tile * kDigitTile < m) {
    const int valid = min(kDigitTile, m - tile * kDigitTile);
    uint32_t* s_tile_keys = smem + b * kDigitTile;
    const uint32_t* tile_keys = in + (size_t)tile * kDigitTile;
    if (threadIdx.x == 0) *s_next = atomicAdd(tile_counter, 1);  // read after (A)
    const bool landed = mbar_wait(&s_bar[b], (phases >> b) & 1u, err);
    uint32_t keys[kItems], ranks[kItems / 2];
    if (unstable) {
#pragma unroll
      for (int r = 0; r < kItems; ++r) {
        const int li = w0 + r * 32 + lane;
        keys[r] = valid == kDigitTile ? s_tile_keys[li] : tail_key(s_tile_keys, tile_keys, li, valid);
        uint32_t rank = 0;
        if (li < valid) rank = atomicAdd(&s_warp[((keys[r] >> shift) & 255u) ^ flip], 1u);
        ranks[r / 2] = (r & 1) ? ranks[r / 2] | (rank << 16) : rank;
      }
    } else if (valid == kDigitTile) {
      rank_keys<true>(s_tile_keys, nullptr, keys, ranks, s_mine, s_peers + warp * kBuckets, shift, flip, valid, w0,
                      lane);
    } else {
      rank_keys<false>(s_tile_keys, tile_keys, keys, ranks, s_mine, s_peers + warp * kBuckets, shift, flip, valid, w0,
                       lane);
    }
    // (A) every read of this buffer is done.  A wait that ran out (error flag
    // set) ends the CTA, after its copy has landed (bounded), so that nothing
    // lands in shared memory after the CTA has left.
    if (!__syncthreads_and(landed)) {
      if (threadIdx.x == 0) mbar_wait(&s_bar[b], (phases >> b) & 1u, err);
      return;
    }
    phases ^= 1u << b;
    const int next = *s_next;
    // the other buffer was drained before the last tile ended
    if (threadIdx.x == 0 && (long long)next * kDigitTile < m)
      bulk_load(smem + (b ^ 1) * kDigitTile, in + (size_t)next * kDigitTile, digit_tile_bytes(next, m), &s_bar[b ^ 1]);
    // per digit: exclusive prefix over warps and the tile's count; the count
    // is published at once so later tiles' look-backs can pass this one
    // The 256 digit threads (8 warps) also scan the tile's counts: within the
    // warp by shuffles, across warps through the warp totals after (B).
    uint32_t tile_count = 0, incl = 0;
    if (threadIdx.x < kBuckets) {
      const int d = threadIdx.x;
      uint32_t run = 0;
      if (unstable) {
        run = s_warp[d];
      } else {
#pragma unroll
        for (int w = 0; w < kDigitWarps; ++w) {
          const uint32_t v = s_warp[w * kBuckets + d];
          s_warp[w * kBuckets + d] = run;
          run += v;
        }
      }
      tile_count = run;
      st_volatile64(status + (size_t)tile * kBuckets + d, lb_word(tag, tile == 0 ? 2u : 1u, run));
      incl = run;
#pragma unroll
      for (int off = 1; off < 32; off <<= 1) {
        const uint32_t t = __shfl_up_sync(0xffffffffu, incl, off);
        if (lane >= off) incl += t;
      }
      if (lane == 31) s_wsum[warp] = incl;
    }
    __syncthreads();  // (B)
    // tile-local start of each digit run, folded into the per-warp offsets so
    // that staging reads one word per key
    if (threadIdx.x < kBuckets) {
      const int d = threadIdx.x;
      uint32_t start = incl - tile_count;
      for (int k = 0; k < warp; ++k) start += s_wsum[k];
      s_start[d] = start;
      if (unstable) {
        s_warp[d] = start;
      } else {
#pragma unroll
        for (int w = 0; w < kDigitWarps; ++w) s_warp[w * kBuckets + d] += start;
      }
    }
    __syncthreads();  // (C)
    // stage keys in tile-local sorted order, in place: every read of the buffer finished before (A)
#pragma unroll
    for (int r = 0; r < kItems; ++r) {
      const int li = w0 + r * 32 + lane;
      if (valid == kDigitTile || li < valid) {
        const uint32_t k = keys[r];
        const uint32_t rank = (r & 1) ? ranks[r / 2] >> 16 : ranks[r / 2] & 0xffffu;
        s_tile_keys[s_mine[((k >> shift) & 255u) ^ flip] + rank] = k;
      }
    }
    // global position of each digit run: look-back over earlier tiles
    if (threadIdx.x < kBuckets) {
      const int d = threadIdx.x;
      uint32_t excl = 0;
      if (tile != 0) {
        excl = look_back(status, tile, kBuckets, d, tag, err);
        st_volatile64(status + (size_t)tile * kBuckets + d, lb_word(tag, 2u, excl + tile_count));
      }
      s_off[d] = digit_base[d] + excl - s_start[d];
    }
    __syncthreads();  // (D)
    // contiguous write-out of each digit run; the counts are cleared for the
    // next tile on the way (the write-out does not read them)
    for (int i = threadIdx.x; i < rows * kBuckets; i += kDigitThreads) s_warp[i] = 0;
    if (valid == kDigitTile) {
#pragma unroll
      for (int k = 0; k < kItems; ++k) {
        const int i = threadIdx.x + k * kDigitThreads;
        const uint32_t key = s_tile_keys[i];
        const uint32_t pos = s_off[((key >> shift) & 255u) ^ flip] + (uint32_t)i;
        if (pos < (uint32_t)m) out[pos] = key;  // past m only after a look-back gave up (error flag set)
      }
    } else {
      for (int i = threadIdx.x; i < valid; i += kDigitThreads) {
        const uint32_t key = s_tile_keys[i];
        const uint32_t pos = s_off[((key >> shift) & 255u) ^ flip] + (uint32_t)i;
        if (pos < (uint32_t)m) out[pos] = key;
      }
    }
    __syncthreads();  // (E) the buffer, the run starts and offsets and the counts are reused
    tile = next;
    b ^= 1;
  }
}
__global__ void __launch_bounds__(kDigitThreads, 2) digit_kernel(const DigitBuffers bufs, int n, const int* count,
                                  int pass, uint32_t flip, Plan* plan, unsigned long long* status,
                                  int* tile_counter, uint32_t tag, int* err, const DoneFlag done) {
  digit_kernel_cta(bufs, n, count, pass, flip, plan, status, tile_counter, tag, err);
  publish(done);
}

// ---- evenly spread keys ----------------------------------------------------------
// A sort of keys alone may put equal keys in any order, and keys that are
// spread about evenly over their range need no digit passes: a linear map of
// the range, product = (key - lowest) * factor, has the number of one of up to
// kSplitRanges equal parts of the range in its upper word.
// split_kernel moves each key into its part's region of scratch (regions have
// room for a part's even share and some more, so nothing has to be counted
// first: a tile claims its places with one atomic per part), and
// split_sort_kernel sorts each region in shared memory and writes it where it
// belongs.  Keys are read and written twice instead of four times and no tile
// waits on another (2^26 random keys: four digit passes 1040 us; here 256 +
// 261; 10^6 keys, whole call: 84 us, here 48).
// The histogram kernel before them chooses by the digits' counts (even_digit).
// Keys that pass that test and still overfill a region, or crowd one of
// split_sort_kernel's bins, leave the array a permutation of itself, and the
// host launches the digit passes over it.
constexpr int kMoveThreads = 1024;   // split_kernel
constexpr int kMoveTile = 32768;     // keys of a tile, at most
constexpr int kMoveGroups = kMoveTile / (4 * kMoveThreads);  // 16-byte units per thread
constexpr int kSplitThreads = 512;   // split_sort_kernel
constexpr int kSplitRoom = 16384;    // keys of a region, at most
constexpr int kSplitRanges = 4608;
constexpr int kSplitFill = 15360;    // keys a region gets on average, at most
constexpr int kSplitGroups = kSplitRoom / (4 * kSplitThreads);
constexpr int kSplitSmemBytes = (kMoveTile + 2 * kSplitRanges) * 4;
constexpr int kSplitPer = (kSplitRanges + kMoveThreads - 1) / kMoveThreads;
constexpr int kSortBins = 12288;     // at most; a multiple of kSortBinsUnit, four per thread
constexpr int kSortBinsUnit = 4 * kSplitThreads;
constexpr int kSortSmemBytes = (kSplitRoom + kSortBins) * 4;
constexpr uint32_t kSortRun = 16;    // keys that a thread sorts in registers
constexpr uint32_t kCrowded = 64;    // keys of a bin that are ranked against one another
static_assert(kCountValues <= kMoveTile && kCountValues <= kSplitRoom && kSplitThreads == kDigitThreads,
              "the value counters lie in the tile, and in the region");
static_assert(2 * kSplitRanges + 1 <= kCountValues, "the ranges' counts and starts lie in the plan's value counts");

struct SplitShape {
  int ranges;      // 0: no split
  uint32_t room;   // keys of a region
  int tile;        // keys of a tile, a multiple of 4
  int bins;        // of a region
};

// Brings keys [begin, end) into L2 (begin a multiple of 4, the keys on a 16-byte
// boundary; up to three at the end may be left out).
__device__ __forceinline__ void fetch_keys(const uint32_t* keys, uint32_t begin, uint32_t end) {
  if (begin / 4 < end / 4)
    asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(keys + begin), "r"((end / 4 - begin / 4) * 16)
                 : "memory");
}
// Four keys from position 4 * u on; past the end of n keys whatever.
template <bool kVec>
__device__ __forceinline__ uint4 load_unit(const uint32_t* keys, uint32_t u, uint32_t n) {
  if (kVec && u * 4 + 4 <= n) return __ldg(reinterpret_cast<const uint4*>(keys) + u);
  uint4 v = make_uint4(0, 0, 0, 0);
  if (u * 4 < n) v.x = __ldg(keys + u * 4);
  if (u * 4 + 1 < n) v.y = __ldg(keys + u * 4 + 1);
  if (u * 4 + 2 < n) v.z = __ldg(keys + u * 4 + 2);
  if (u * 4 + 3 < n) v.w = __ldg(keys + u * 4 + 3);
  return v;
}

// Exclusive scan over the CTA of one value per thread.
__device__ __forceinline__ uint32_t cta_exclusive(uint32_t v, uint32_t* s_wsum) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  uint32_t incl = v;
#pragma unroll
  for (int off = 1; off < 32; off <<= 1) {
    const uint32_t t = __shfl_up_sync(0xffffffffu, incl, off);
    if (lane >= off) incl += t;
  }
  if (lane == 31) s_wsum[warp] = incl;
  __syncthreads();
  return incl - v + __reduce_add_sync(0xffffffffu, lane < warp ? s_wsum[lane] : 0u);  // warp < 32
}

// The longer a range's run in a tile, the fewer lines a warp's stores meet:
// tiles of 32768 keys (7 keys a run at 4560 ranges), one per SM, took 250 us
// for 2^26 keys where two per SM of 16384 took 310, 97 of them for the stores
// being scattered.  A tile's keys are read again (from L2) to be staged, as
// registers hold their ranks.  Each CTA has its next tile fetched into L2.
template <bool kVec, int kGroups>
__device__ __forceinline__ void split_cta(const uint32_t* keys, uint32_t n, uint32_t* regions, const SplitShape shape,
                                          Control* ctl, Plan* plan, uint32_t* smem) {
  __shared__ uint32_t s_wsum[kMoveThreads / 32];
  uint32_t* s_tile = smem;
  uint32_t* s_count = smem + kMoveTile;      // keys of the tile per range, then their starts in the tile
  uint32_t* s_off = s_count + kSplitRanges;   // position in the regions - position in the tile
  uint32_t* claimed = plan->values;
  const uint32_t lo = plan->lowest, factor = plan->split, ranges = (uint32_t)shape.ranges, room = shape.room;
  const uint32_t tile = (uint32_t)shape.tile;
  const uint32_t per = ((ranges + kMoveThreads - 1) / kMoveThreads) | 1u;  // odd: a thread's ranges lie in all banks
  const uint32_t tiles = (n + tile - 1) / tile;
  for (uint32_t t = blockIdx.x; t < tiles; t += gridDim.x) {
    const uint32_t begin = t * tile, end = min(n, begin + tile);  // n < 2^27
    for (uint32_t i = threadIdx.x; i < per * kMoveThreads && i < (uint32_t)kSplitRanges; i += kMoveThreads)
      s_count[i] = 0;
    const bool over = *(volatile int*)&ctl->split_over != 0;
    if (__syncthreads_or(over)) return;
    if (kVec && threadIdx.x == 0 && t + gridDim.x < tiles) {  // this CTA's next tile
      const uint32_t next = (t + gridDim.x) * tile;
      fetch_keys(keys, next, min(n, next + tile));
    }
    constexpr int kBatch = kGroups < 4 ? kGroups : 4;
    uint32_t ranks[kGroups * 2];
    auto range_of = [&](uint32_t x) { return __umulhi(x, factor); };
#pragma unroll
    for (int h = 0; h < kGroups; h += kBatch) {
      uint4 v[kBatch];
#pragma unroll
      for (int g = 0; g < kBatch; ++g)
        v[g] = load_unit<kVec>(keys, begin / 4 + (h + g) * kMoveThreads + threadIdx.x, end);
#pragma unroll
      for (int g = 0; g < kBatch; ++g) {
        const uint32_t at = begin + ((h + g) * kMoveThreads + threadIdx.x) * 4;
        const uint32_t k[4] = {v[g].x, v[g].y, v[g].z, v[g].w};
        uint32_t r[4] = {0, 0, 0, 0};
#pragma unroll
        for (int e = 0; e < 4; ++e)
          if (at + e < end) r[e] = atomicAdd(&s_count[range_of((k[e] ^ 0x80000000u) - lo)], 1u);
        ranks[(h + g) * 2] = r[0] | (r[1] << 16);
        ranks[(h + g) * 2 + 1] = r[2] | (r[3] << 16);
      }
    }
    __syncthreads();
    // every claim in flight beside the scan
    uint32_t count[kSplitPer], got[kSplitPer];
#pragma unroll
    for (int j = 0; j < kSplitPer; ++j) {
      const uint32_t d = threadIdx.x + j * kMoveThreads;
      count[j] = d < ranges ? s_count[d] : 0u;
      got[j] = count[j] ? atomicAdd(&claimed[d], count[j]) : 0u;
    }
    __syncthreads();
    {
      const uint32_t first = threadIdx.x * per;
      uint32_t sum = 0;
#pragma unroll
      for (int j = 0; j < kSplitPer; ++j)
        if (j < per && first + j < ranges) sum += s_count[first + j];
      uint32_t run = cta_exclusive(sum, s_wsum);
#pragma unroll
      for (int j = 0; j < kSplitPer; ++j)
        if (j < per && first + j < ranges) {
          const uint32_t c = s_count[first + j];
          s_count[first + j] = run;
          run += c;
        }
    }
    __syncthreads();
    bool full = false;
#pragma unroll
    for (int j = 0; j < kSplitPer; ++j) {
      const uint32_t d = threadIdx.x + j * kMoveThreads;
      full |= got[j] + count[j] > room;
      if (d < ranges) s_off[d] = d * room + got[j] - s_count[d];
    }
    if (full) *(volatile int*)&ctl->split_over = 1;
#pragma unroll
    for (int h = 0; h < kGroups; h += kBatch) {
      uint4 v[kBatch];
#pragma unroll
      for (int g = 0; g < kBatch; ++g)
        v[g] = load_unit<kVec>(keys, begin / 4 + (h + g) * kMoveThreads + threadIdx.x, end);
#pragma unroll
      for (int g = 0; g < kBatch; ++g) {
        const uint32_t at = begin + ((h + g) * kMoveThreads + threadIdx.x) * 4;
        const uint32_t k[4] = {v[g].x, v[g].y, v[g].z, v[g].w};
        const uint32_t r[2] = {ranks[(h + g) * 2], ranks[(h + g) * 2 + 1]};
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const uint32_t x = (k[e] ^ 0x80000000u) - lo;
          if (at + e < end) s_tile[s_count[range_of(x)] + ((r[e >> 1] >> (16 * (e & 1))) & 0xffffu)] = x;
        }
      }
    }
    __syncthreads();
#pragma unroll 8
    for (uint32_t i = threadIdx.x; i < end - begin; i += kMoveThreads) {
      const uint32_t x = s_tile[i], d = range_of(x);
      const uint32_t pos = s_off[d] + i;
      if (pos - d * room < room) regions[pos] = x;  // else split_over is set
    }
    __syncthreads();
  }
}
template <bool kVec, int kGroups>
__global__ void __launch_bounds__(kMoveThreads, 1) split_kernel(const uint32_t* keys, int n, uint32_t* regions,
                                                                 const SplitShape shape, Control* ctl, Plan* plan) {
  extern __shared__ __align__(128) uint32_t smem[];
  __shared__ uint32_t s_wsum[kMoveThreads / 32];
  dependents_may_start();
  wait_for_dependency();
  if (plan->counting) {
    count_values(keys, n, 0x80000000u, plan, smem);
    return;
  }
  if (!plan->split) return;
  split_cta<kVec, kGroups>(keys, (uint32_t)n, regions, shape, ctl, plan, smem);
  if (!last_cta(&ctl->done[3], gridDim.x)) return;
  // where each range's keys begin in the array
  const uint32_t ranges = (uint32_t)shape.ranges, per = (ranges + kMoveThreads - 1) / kMoveThreads;
  const volatile uint32_t* claimed = plan->values;
  uint32_t sum = 0, c[kSplitPer];
#pragma unroll
  for (uint32_t j = 0; j < kSplitPer; ++j) {
    c[j] = j < per && threadIdx.x * per + j < ranges ? claimed[threadIdx.x * per + j] : 0u;
    sum += c[j];
  }
  uint32_t run = cta_exclusive(sum, s_wsum);
#pragma unroll
  for (uint32_t j = 0; j < kSplitPer; ++j) {
    if (j < per && threadIdx.x * per + j < ranges) plan->values[kSplitRanges + threadIdx.x * per + j] = run;
    run += c[j];
  }
}

// One region per CTA and turn.  The lower word of the product is the key's place
// within its range, and that times the number of bins its bin, about one key
// each: a key's rank among its bin's keys is what the atomic that counts it
// returns, the bins' starts are scanned, and the keys go to their bins in
// shared memory.  What is left is to order the few keys of each bin: a thread
// sorts 16 neighbouring keys in registers, and then merges the halves of two
// such runs that meet, which puts every bin of up to 9 keys in order, as it
// lies in two runs at most.  (Ranking each key against the others of its bin
// took 365 us for 2^26 keys, at 157 instructions per 32 of them; this takes 261
// at 79 and is bound by shared memory, 67% of its wavefronts' rate.)  Where
// a bin has more keys they are ranked so; no order is missing where a bin is a
// single value.
__device__ __forceinline__ void order(uint32_t& a, uint32_t& b) {
  const uint32_t lo = min(a, b);
  b = max(a, b);
  a = lo;
}
// The steps of Batcher's odd-even merge sort of 16 keys that merge sorted runs
// of kP keys, from kP = kFrom on.
template <int kFrom>
__device__ __forceinline__ void merge_runs(uint32_t (&k)[kSortRun]) {
#pragma unroll
  for (int p = kFrom; p < (int)kSortRun; p *= 2) {
#pragma unroll
    for (int q = p; q >= 1; q /= 2) {
#pragma unroll
      for (int j = 0; j < (int)kSortRun; ++j)
        if (j >= q % p && (j - q % p) % (2 * q) < q && j + q < (int)kSortRun && j / (2 * p) == (j + q) / (2 * p))
          order(k[j], k[j + q]);
    }
  }
}
// Where position i of a region lies in shared memory: 16-byte units of
// neighbouring runs lie in different banks.
__device__ __forceinline__ uint32_t run_place(uint32_t i) { return i ^ ((i >> 3) & 12u); }
template <int kFrom>
__device__ __forceinline__ void sort_run(uint32_t* s_keys, uint32_t at) {
  uint32_t k[kSortRun];
#pragma unroll
  for (uint32_t u = 0; u < kSortRun; u += 4) {
    const uint4 v = *reinterpret_cast<const uint4*>(s_keys + run_place(at + u));
    k[u] = v.x, k[u + 1] = v.y, k[u + 2] = v.z, k[u + 3] = v.w;
  }
  merge_runs<kFrom>(k);
#pragma unroll
  for (uint32_t u = 0; u < kSortRun; u += 4)
    *reinterpret_cast<uint4*>(s_keys + run_place(at + u)) = make_uint4(k[u], k[u + 1], k[u + 2], k[u + 3]);
}

template <int kGroups>
__device__ __forceinline__ bool split_sort_cta(uint32_t* out, const uint32_t* regions, const SplitShape shape,
                                               const Plan* plan, uint32_t* smem) {
  __shared__ uint32_t s_wsum[kSplitThreads / 32];
  uint32_t* s_keys = smem;
  uint32_t* s_bin = smem + kSplitRoom;  // count, then start | count << 16
  const uint32_t lo = plan->lowest, factor = plan->split, bins = (uint32_t)shape.bins;
  // neighbouring keys are at least a bin apart
  const bool single = (unsigned long long)factor * bins >> 32 != 0;
  auto bin_of = [&](uint32_t x) { return __umulhi(x * factor, bins); };
  bool any_crowded = false;
  for (int q = blockIdx.x; q < shape.ranges; q += gridDim.x) {
    const uint32_t count = plan->values[q], base = plan->values[kSplitRanges + q];
    const uint32_t* keys = regions + (size_t)q * shape.room;
    if (threadIdx.x == 0 && q + (int)gridDim.x < shape.ranges)  // this CTA's next region
      fetch_keys(keys + (size_t)gridDim.x * shape.room, 0, plan->values[q + gridDim.x]);
    for (uint32_t i = threadIdx.x * 4; i < bins; i += kSortBinsUnit)
      *reinterpret_cast<uint4*>(s_bin + i) = make_uint4(0, 0, 0, 0);
    __syncthreads();
    constexpr int kBatch = kGroups < 4 ? kGroups : 4;
    uint32_t ranks[kGroups * 2];
#pragma unroll
    for (int h = 0; h < kGroups; h += kBatch) {
      if (h * kSplitThreads * 4 >= count) break;
      uint4 v[kBatch];
#pragma unroll
      for (int g = 0; g < kBatch; ++g) v[g] = load_unit<true>(keys, (h + g) * kSplitThreads + threadIdx.x, count);
#pragma unroll
      for (int g = 0; g < kBatch; ++g) {
        const uint32_t at = ((h + g) * kSplitThreads + threadIdx.x) * 4;
        const uint32_t k[4] = {v[g].x, v[g].y, v[g].z, v[g].w};
        uint32_t r[4] = {0, 0, 0, 0};
#pragma unroll
        for (int e = 0; e < 4; ++e)
          if (at + e < count) r[e] = atomicAdd(&s_bin[bin_of(k[e])], 1u);
        ranks[(h + g) * 2] = r[0] | (r[1] << 16);
        ranks[(h + g) * 2 + 1] = r[2] | (r[3] << 16);
      }
    }
    __syncthreads();
    uint32_t most = 0;
    {
      const uint32_t per = bins / kSplitThreads, first = threadIdx.x * per;
      uint32_t sum = 0;
      for (uint32_t j = 0; j < per; j += 4) {
        const uint4 v = *reinterpret_cast<const uint4*>(s_bin + first + j);
        sum += v.x + v.y + v.z + v.w;
        most = max(max(most, max(v.x, v.y)), max(v.z, v.w));
      }
      uint32_t run = cta_exclusive(sum, s_wsum);
      for (uint32_t j = 0; j < per; j += 4) {
        uint4* at = reinterpret_cast<uint4*>(s_bin + first + j);
        const uint4 v = *at;
        const uint32_t y = run + v.x, z = y + v.y, w = z + v.z;
        *at = make_uint4(run | (v.x << 16), y | (v.y << 16), z | (v.z << 16), w | (v.w << 16));
        run = w + v.w;
      }
    }
    const bool ranked = __syncthreads_or(most > kSortRun / 2 + 1) && !single;
    const bool crowded = __syncthreads_or(most > kCrowded) && !single;
    any_crowded |= crowded;
#pragma unroll
    for (int h = 0; h < kGroups; h += kBatch) {
      if (h * kSplitThreads * 4 >= count) break;
      uint4 v[kBatch];
#pragma unroll
      for (int g = 0; g < kBatch; ++g) v[g] = load_unit<true>(keys, (h + g) * kSplitThreads + threadIdx.x, count);
#pragma unroll
      for (int g = 0; g < kBatch; ++g) {
        const uint32_t at = ((h + g) * kSplitThreads + threadIdx.x) * 4;
        const uint32_t k[4] = {v[g].x, v[g].y, v[g].z, v[g].w};
        const uint32_t r[2] = {ranks[(h + g) * 2], ranks[(h + g) * 2 + 1]};
#pragma unroll
        for (int e = 0; e < 4; ++e)
          if (at + e < count) {
            const uint32_t rank = (r[e >> 1] >> (16 * (e & 1))) & 0xffffu;
            s_keys[run_place((s_bin[bin_of(k[e])] & 0xffffu) + rank)] = k[e];
          }
      }
    }
    const uint32_t runs = (count + kSortRun - 1) / kSortRun;  // runs * 16 <= kSplitRoom
    if (count + threadIdx.x < runs * kSortRun) s_keys[run_place(count + threadIdx.x)] = ~0u;
    __syncthreads();
    if (!single && !ranked) {
      for (uint32_t r = threadIdx.x; r < runs; r += kSplitThreads) sort_run<1>(s_keys, r * kSortRun);
      __syncthreads();
      for (uint32_t r = threadIdx.x; r + 1 < runs; r += kSplitThreads)
        sort_run<kSortRun / 2>(s_keys, r * kSortRun + kSortRun / 2);
      __syncthreads();
    }
    if (ranked && !crowded) {
      for (uint32_t i = threadIdx.x; i < count; i += kSplitThreads) {
        const uint32_t x = s_keys[run_place(i)];
        const uint32_t w = s_bin[bin_of(x)], first = w & 0xffffu, last = first + (w >> 16);
        uint32_t to = first;
        for (uint32_t j = first; j < last; ++j) {
          const uint32_t y = s_keys[run_place(j)];
          to += y < x || (y == x && j < i);
        }
        out[base + to] = (x + lo) ^ 0x80000000u;
      }
    } else {
#pragma unroll 4
      for (uint32_t i = threadIdx.x; i < count; i += kSplitThreads)
        out[base + i] = (s_keys[run_place(i)] + lo) ^ 0x80000000u;
    }
    __syncthreads();
  }
  return any_crowded;
}
// `again` (mapped host memory): 1 if the keys must take the digit passes.
template <int kGroups>
__global__ void __launch_bounds__(kSplitThreads, 2) split_sort_kernel(uint32_t* out, int n, const uint32_t* regions,
                                                                      const SplitShape shape, Control* ctl,
                                                                      const Plan* plan, int* again,
                                                                      const DoneFlag done) {
  extern __shared__ __align__(128) uint32_t smem[];
  wait_for_dependency();
  bool digits = false;
  if (plan->counting)
    write_values(out, n, 0x80000000u, plan, smem);
  else if (!plan->split || *(volatile int*)&ctl->split_over)
    digits = true;
  else
    digits = split_sort_cta<kGroups>(out, regions, shape, plan, smem);
  if (digits && threadIdx.x == 0) *(volatile int*)again = 1;
  publish(done);
}

// ---- one CTA --------------------------------------------------------------------
// Up to kSmall keys stay in one CTA: a chain of launches costs 40 to 80 us
// whatever the size (2013 keys: 45 us in 7 kernels, and the copy of the error
// flag).  The keys are reduced by their minimum, so only the 8-bit digits that
// their range needs are passed over (one for the reference test's 201
// values), each with the digit pass's ranking; the keys live in shared memory
// between passes.
constexpr int kSmallThreads = 1024;
constexpr int kSmallWarps = kSmallThreads / 32;
constexpr int kSmall = 8192;
template <int kRounds>
constexpr int small_smem_bytes() {
  return (kSmallThreads * kRounds + 2 * kSmallWarps * kBuckets + kBuckets) * 4;
}

// Sorts the kSmallThreads * kRounds keys in s_keys by their low `bits` bits,
// in place.  All threads of the CTA call it.
template <int kRounds>
__device__ void cta_sort(uint32_t* s_keys, int bits) {
  uint32_t* s_warp = s_keys + kSmallThreads * kRounds;       // [warp][digit] counts, then offsets
  uint32_t* s_peers = s_warp + kSmallWarps * kBuckets;       // [warp][digit] peer masks
  uint32_t* s_count = s_peers + kSmallWarps * kBuckets;      // per digit
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  for (int i = threadIdx.x; i < 2 * kSmallWarps * kBuckets; i += kSmallThreads) s_warp[i] = 0;
  __syncthreads();
  for (int shift = 0; shift < bits; shift += 8) {
    uint32_t keys[kRounds], ranks[(kRounds + 1) / 2];
    rank_keys<true>(s_keys, nullptr, keys, ranks, s_warp + warp * kBuckets, s_peers + warp * kBuckets, shift, 0u, 0,
                    warp * kRounds * 32, lane);
    __syncthreads();
    // four threads per digit sum 8 warps each, then the digit's offsets
    const int d = threadIdx.x >> 2, part = threadIdx.x & 3;
    uint32_t* col = s_warp + part * (kSmallWarps / 4) * kBuckets + d;
    uint32_t v[kSmallWarps / 4], sum = 0;
#pragma unroll
    for (int w = 0; w < kSmallWarps / 4; ++w) {
      v[w] = col[w * kBuckets];
      sum += v[w];
    }
    uint32_t incl = sum;
#pragma unroll
    for (int off = 1; off < 4; off <<= 1) {
      const uint32_t t = __shfl_up_sync(0xffffffffu, incl, off);
      if (part >= off) incl += t;
    }
    if (part == 3) s_count[d] = incl;
    __syncthreads();
    if (warp == 0) warp_scan_256(s_count, s_count);
    __syncthreads();
    uint32_t run = s_count[d] + incl - sum;
#pragma unroll
    for (int w = 0; w < kSmallWarps / 4; ++w) {
      col[w * kBuckets] = run;
      run += v[w];
    }
    __syncthreads();
#pragma unroll
    for (int r = 0; r < kRounds; ++r) {
      const uint32_t rank = (r & 1) ? ranks[r / 2] >> 16 : ranks[r / 2] & 0xffffu;
      s_keys[s_warp[warp * kBuckets + ((keys[r] >> shift) & 255u)] + rank] = keys[r];
    }
    __syncthreads();
    if (shift + 8 < bits) {
      for (int i = threadIdx.x; i < kSmallWarps * kBuckets; i += kSmallThreads) s_warp[i] = 0;
      __syncthreads();
    }
  }
}

// Minimum and maximum over the CTA of (lo, hi); all threads get both.
__device__ __forceinline__ void cta_range(uint32_t& lo, uint32_t& hi) {
  __shared__ uint32_t s_lo[kSmallWarps], s_hi[kSmallWarps];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  lo = __reduce_min_sync(0xffffffffu, lo);
  hi = __reduce_max_sync(0xffffffffu, hi);
  if (lane == 0) s_lo[warp] = lo, s_hi[warp] = hi;
  __syncthreads();
  lo = __reduce_min_sync(0xffffffffu, s_lo[lane]);
  hi = __reduce_max_sync(0xffffffffu, s_hi[lane]);
}

template <int kRounds>
__device__ __forceinline__ void small_sort_kernel_cta(int32_t* data, int n) {
  extern __shared__ __align__(128) uint32_t smem[];
  uint32_t k[kRounds], lo = 0xffffffffu, hi = 0;
#pragma unroll
  for (int r = 0; r < kRounds; ++r) {
    const int i = r * kSmallThreads + threadIdx.x;
    if (i < n) {
      k[r] = (uint32_t)data[i] ^ 0x80000000u;
      lo = min(lo, k[r]);
      hi = max(hi, k[r]);
    }
  }
  cta_range(lo, hi);
  // the places past n hold the largest key: they sort to the end
#pragma unroll
  for (int r = 0; r < kRounds; ++r) {
    const int i = r * kSmallThreads + threadIdx.x;
    smem[i] = (i < n ? k[r] : hi) - lo;
  }
  cta_sort<kRounds>(smem, 32 - __clz((int)(hi - lo)));
  for (int i = threadIdx.x; i < n; i += kSmallThreads) data[i] = (int32_t)((smem[i] + lo) ^ 0x80000000u);
}
template <int kRounds>
__global__ void __launch_bounds__(kSmallThreads, 1) small_sort_kernel(int32_t* data, int n, const DoneFlag done) {
  small_sort_kernel_cta<kRounds>(data, n);
  publish(done);
}

// Feedback unique of up to kSmall words: NO_HIT words (and the places past n)
// become a key above every other.  result[0] = the unique count.
template <int kRounds>
__device__ __forceinline__ void small_unique_kernel_cta(const int32_t* words, int n, int nib, Divider div,
                                                        int32_t* out, int* result) {
  extern __shared__ __align__(128) uint32_t smem[];
  __shared__ uint32_t s_warp[kSmallWarps];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  uint32_t k[kRounds], lo = 0xffffffffu, hi = 0;
  bool none = false;  // a NO_HIT word
#pragma unroll
  for (int r = 0; r < kRounds; ++r) {
    const int i = r * kSmallThreads + threadIdx.x;
    int32_t v = i < n ? words[i] : kNoHit;
    none = none || (i < n && v == kNoHit);
    if (v > 0 && v != kNoHit && nib > 0) v = (int32_t)(((divide((uint32_t)((v >> 1) - 1), div) + 1) << 1) | (v & 1));
    k[r] = (uint32_t)v ^ 0x80000000u;
    if (k[r] != kNoKey) {
      lo = min(lo, k[r]);
      hi = max(hi, k[r]);
    }
  }
  cta_range(lo, hi);
  none = __syncthreads_or(none);
  const bool any = lo <= hi;
  const uint32_t top = any ? hi - lo + 1 : 0;  // the dropped words' key; hi < kNoKey, so it does not wrap
#pragma unroll
  for (int r = 0; r < kRounds; ++r) smem[r * kSmallThreads + threadIdx.x] = k[r] == kNoKey ? top : k[r] - lo;
  cta_sort<kRounds>(smem, 32 - __clz((int)top));
  __syncthreads();
  // run starts of the kept keys, kRounds consecutive keys per thread
  uint32_t starts = 0, cnt = 0;
  const int first = threadIdx.x * kRounds;
#pragma unroll
  for (int r = 0; r < kRounds; ++r) {
    const uint32_t v = smem[first + r];
    const bool start = v != top && (first + r == 0 || smem[first + r - 1] != v);
    starts |= (uint32_t)start << r;
    cnt += start;
  }
  uint32_t incl = cnt;
  for (int off = 1; off < 32; off <<= 1) {
    const uint32_t t = __shfl_up_sync(0xffffffffu, incl, off);
    if (lane >= off) incl += t;
  }
  if (lane == 31) s_warp[warp] = incl;
  __syncthreads();
  uint32_t pos = incl - cnt, total = 0;
  {
    const uint32_t w = s_warp[lane];
    pos += __reduce_add_sync(0xffffffffu, lane < warp ? w : 0u);
    total = __reduce_add_sync(0xffffffffu, w);
  }
#pragma unroll
  for (int r = 0; r < kRounds; ++r)
    if ((starts >> r) & 1u) out[pos++] = (int32_t)((smem[first + r] + lo) ^ 0x80000000u);
  if (threadIdx.x == 0) {
    if (none) out[total++] = kNoHit;
    result[0] = (int)total;
    result[1] = kPathEmpty;
  }
}
template <int kRounds>
__global__ void __launch_bounds__(kSmallThreads, 1) small_unique_kernel(const int32_t* words, int n, int nib,
                                  Divider div, int32_t* out, int* result, const DoneFlag done) {
  small_unique_kernel_cta<kRounds>(words, n, nib, div, out, result);
  publish(done);
}

// ---- unique of sorted keys -----------------------------------------------------
// Persistent like digit_kernel, and pipelined the same way: a tile's run-start
// keys are compacted into shared memory (each warp into its own range), the
// next tile (claimed at the start of this one) is loaded, and only then does
// the tile's look-back for its output position run.
__device__ __forceinline__ void unique_kernel_cta(const uint32_t* keys_a, const uint32_t* keys_b, Control* ctl,
                                                  const Plan* plan, int32_t* out, unsigned long long* status,
                                                  int* result, uint32_t tag, int* err) {
  __shared__ int s_tile;
  __shared__ uint32_t s_warp[kWarps + 1];
  __shared__ uint32_t s_excl;
  __shared__ uint32_t s_starts[kTile];
  const uint32_t* keys = plan->last == 0 ? keys_a : keys_b;
  int* tile_counter = &ctl->unique_tiles;
  const int m = ctl->keys;  // at least one
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  // warp `warp` owns keys [w0, w0 + 512) of a tile, 32 per round (coalesced);
  // a key starts a run when it differs from the key before it
  const int w0 = warp * (kItems * 32);
  const unsigned lt = (1u << lane) - 1;
  if (threadIdx.x == 0) s_tile = atomicAdd(tile_counter, 1);
  __syncthreads();
  int tile = s_tile;
  __syncthreads();  // every thread has read s_tile
  if ((long long)tile * kTile >= m) return;
  uint32_t k[kItems];
  uint32_t prev_last = 0;  // the key before this warp's first key
  {
    const long long b = (long long)tile * kTile + w0;
#pragma unroll
    for (int r = 0; r < kItems; ++r) k[r] = b + r * 32 + lane < m ? __ldg(keys + b + r * 32 + lane) : 0u;
    if (lane == 0 && b > 0 && b < m) prev_last = __ldg(keys + b - 1);
  }
  for (;;) {
    const int base = tile * kTile;
    const int valid = min(kTile, m - base);
    if (threadIdx.x == 0) s_tile = atomicAdd(tile_counter, 1);  // the next tile
    uint32_t cnt = 0;
#pragma unroll
    for (int r = 0; r < kItems; ++r) {
      const int li = w0 + r * 32 + lane;
      uint32_t prev = __shfl_up_sync(0xffffffffu, k[r], 1);
      if (lane == 0) prev = prev_last;
      prev_last = __shfl_sync(0xffffffffu, k[r], 31);
      const bool start = li < valid && (base + li == 0 || prev != k[r]);
      const unsigned starts = __ballot_sync(0xffffffffu, start);
      if (start) s_starts[w0 + cnt + __popc(starts & lt)] = k[r];
      cnt += __popc(starts);
    }
    if (lane == 0) s_warp[warp] = cnt;
    __syncthreads();
    const int next = s_tile;
    const long long next_base = (long long)next * kTile;
    {  // the next tile's keys are in flight during the look-back and write-out
      const long long b = next_base + w0;
#pragma unroll
      for (int r = 0; r < kItems; ++r) k[r] = b + r * 32 + lane < m ? __ldg(keys + b + r * 32 + lane) : 0u;
      prev_last = lane == 0 && b > 0 && b < m ? __ldg(keys + b - 1) : 0u;
    }
    if (warp == 0) {
      const uint32_t excl = tile_prefix<kWarps>(s_warp, status, tile, tag, err);
      if (lane == 0 && base + valid == m) {  // last tile: totals and the NO_HIT sentinel
        int u = min((int)(excl + s_warp[kWarps]), m);
        if (ctl->no_hit) out[u++] = kNoHit;
        result[0] = u;
      }
      if (lane == 0) s_excl = excl;
    }
    __syncthreads();
    const uint32_t pos = s_excl + s_warp[warp];
    for (uint32_t j = lane; j < cnt; j += 32)
      if (pos + j < (uint32_t)m) out[pos + j] = (int32_t)(s_starts[w0 + j] ^ 0x80000000u);
    __syncthreads();  // shared state is reused by the next tile
    if (next_base >= m) return;
    tile = next;
  }
}
__global__ void __launch_bounds__(kThreads) unique_kernel(const uint32_t* keys_a, const uint32_t* keys_b,
                                  Control* ctl, const Plan* plan, int32_t* out, unsigned long long* status,
                                  int* result, uint32_t tag, int* err, const DoneFlag done) {
  wait_for_dependency();
  unique_kernel_cta(keys_a, keys_b, ctl, plan, out, status, result, tag, err);
  publish(done);
}

// ---- unique by bitmap ------------------------------------------------------------
// Bit b of the bitmap stands for key min + b.  Each kernel returns at once on
// the paths that do not need it.

// ---- writing a bitmap's values -------------------------------------------------
// By cooperative kernels of 1024-thread CTAs: each CTA writes the values of some
// of the words, and what it needs to know of the words before is their bit
// count.  (Tiles claimed in order with a look-back for the position took
// 35 us on 1.5 million words, and 10 us on 3 thousand.)
constexpr int kShareThreads = 1024;
constexpr int kShareWarps = kShareThreads / 32;

// Waits until `ctas` CTAs have come here; false in every thread when the wait
// runs out.  What they wrote before is visible after it.
__device__ __forceinline__ bool grid_barrier(int* counter, int ctas, int* err) {
  __threadfence();
  __syncthreads();
  bool ok = true;
  if (threadIdx.x == 0) {
    atomicAdd(counter, 1);
    long long spins = 0;
    const unsigned long long start = global_ns();
    while (*(volatile int*)counter < ctas) {
      if (wait_over(spins, start)) {
        set_error(err);
        ok = false;
        break;
      }
    }
    __threadfence();
  }
  return __syncthreads_and(ok) != 0;
}

// Sum of v over the CTA's threads, in all of them.
__device__ __forceinline__ uint32_t share_sum(uint32_t v, uint32_t* s_warp) {
  const uint32_t sum = __reduce_add_sync(0xffffffffu, v);
  __syncthreads();  // an earlier use of s_warp is over
  if ((threadIdx.x & 31) == 0) s_warp[threadIdx.x >> 5] = sum;
  __syncthreads();
  return __reduce_add_sync(0xffffffffu, s_warp[threadIdx.x & 31]);
}

// Set bits of words [w0, w1), w0 a multiple of 4, over the CTA's threads.
__device__ __forceinline__ uint32_t count_bits(const uint32_t* bitmap, int w0, int w1, uint32_t* s_warp) {
  uint32_t bits = 0;
  for (int i = w0 / 4 + threadIdx.x; i < w1 / 4; i += kShareThreads) {
    const uint4 q = __ldcg(reinterpret_cast<const uint4*>(bitmap) + i);
    bits += __popc(q.x) + __popc(q.y) + __popc(q.z) + __popc(q.w);
  }
  const int i = max(w0, w1 & ~3) + (int)threadIdx.x;
  if (i < w1) bits += __popc(__ldcg(bitmap + i));
  return share_sum(bits, s_warp);
}

// A warp's bitmap words (one per lane, the lane's first output position `pos`)
// as signed words.  Dense words go word by word, a lane per bit (one coalesced
// store per word); else each lane walks its own word's bits into the warp's
// stage, which is then written in order (stored as they are found, every value
// is a sector of its own, which bound the kernel).
constexpr int kStage = 512;  // values per warp
__device__ __forceinline__ void emit_words(uint32_t w, uint32_t key0, uint32_t pos, uint32_t* stage, int32_t* out) {
  const int lane = threadIdx.x & 31;
  const uint32_t first = __shfl_sync(0xffffffffu, pos, 0);
  const uint32_t total = __shfl_sync(0xffffffffu, pos + __popc(w), 31) - first;
  if (total > kStage) {
    unsigned nonempty = __ballot_sync(0xffffffffu, w != 0);
    while (nonempty) {
      const int src = __ffs(nonempty) - 1;
      nonempty &= nonempty - 1;
      const uint32_t v = __shfl_sync(0xffffffffu, w, src);
      const uint32_t k = __shfl_sync(0xffffffffu, key0, src);
      const uint32_t at = __shfl_sync(0xffffffffu, pos, src) + __popc(v & ((1u << lane) - 1));
      if ((v >> lane) & 1u) out[at] = (int32_t)((k + (uint32_t)lane) ^ 0x80000000u);
    }
  } else {
    uint32_t at = pos - first;
    while (w) {
      const int b = __ffs(w) - 1;
      w &= w - 1;
      stage[at++] = (key0 + (uint32_t)b) ^ 0x80000000u;
    }
    __syncwarp();
    for (uint32_t i = lane; i < total; i += 32) out[first + i] = (int32_t)stage[i];
    __syncwarp();
  }
}

// Positions of one word per thread over the CTA: `run` plus the bits of the
// threads before; run becomes the total.
__device__ __forceinline__ uint32_t word_positions(uint32_t w, uint32_t& run, uint32_t* s_warp) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t bits = __popc(w);
  uint32_t incl = bits;
#pragma unroll
  for (int off = 1; off < 32; off <<= 1) {
    const uint32_t t = __shfl_up_sync(0xffffffffu, incl, off);
    if (lane >= off) incl += t;
  }
  __syncthreads();  // an earlier use of s_warp is over
  if (lane == 31) s_warp[warp] = incl;
  __syncthreads();
  const uint32_t c = s_warp[lane];
  const uint32_t pos = run + __reduce_add_sync(0xffffffffu, lane < warp ? c : 0u) + incl - bits;
  run += __reduce_add_sync(0xffffffffu, c);
  return pos;
}

// Writes the bitmap's values, complete in global memory; s_words: kEmitSmemBytes
// of shared memory.  A small bitmap is cut into one share
// per CTA, and every CTA counts the bits of the words before its own.  A large
// one is cut into segments of 1024 words, dealt to the CTAs in turn (feedback's
// low block numbers set whole stretches of bits; shares of neighbouring words
// left most CTAs waiting for a few, 97 us instead of 35), which count them,
// meet at a barrier and read each other's counts.  The CTA with the last words
// writes the count and the NO_HIT sentinel when any word was NO_HIT.
constexpr int kCountAllWords = 1 << 15;
constexpr int kEmitSmemBytes = (2 * kShareThreads + kShareWarps * kStage) * 4;
static_assert((1 << kMaxSpanLog2) / 32 / kShareThreads <= 2 * kShareThreads, "two segment counts per thread");
__device__ __forceinline__ void emit_bitmap(const uint32_t* bitmap, Control* ctl, Plan* plan, int ctas,
                                            uint32_t* s_words, uint32_t* s_warp, int32_t* out, int* result, int* err) {
  const uint32_t lo = ~ctl->range[0];
  const int words = (int)plan->bitmap_words;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  uint32_t* stage = s_words + 2 * kShareThreads + warp * kStage;
  uint32_t run = 0;
  bool last;
  if (words <= kCountAllWords) {
    const int share = ((words + ctas - 1) / ctas + 3) & ~3;  // whole 16-byte units
    const int w0 = min(words, (int)blockIdx.x * share), w1 = min(words, w0 + share);
    last = w0 < w1 && w1 == words;
    run = count_bits(bitmap, 0, w0, s_warp);
    for (int r0 = w0; r0 < w1; r0 += kShareThreads) {
      const int k = r0 + threadIdx.x;
      const uint32_t w = k < w1 ? __ldcg(bitmap + k) : 0u;
      const uint32_t pos = word_positions(w, run, s_warp);
      if (share > kShareThreads / 2) {
        emit_words(w, lo + (uint32_t)k * 32u, pos, stage, out);
        continue;
      }
      // a few words: a warp per word, a lane per bit, so that every warp has some
      s_words[threadIdx.x] = w;
      s_words[kShareThreads + threadIdx.x] = pos;
      __syncthreads();
      for (int i = warp; i < w1 - r0; i += kShareWarps) {
        const uint32_t v = s_words[i], at = s_words[kShareThreads + i] + __popc(v & ((1u << lane) - 1));
        if ((v >> lane) & 1u) out[at] = (int32_t)((lo + (uint32_t)(r0 + i) * 32u + (uint32_t)lane) ^ 0x80000000u);
      }
      __syncthreads();  // s_words is over
    }
  } else {
    const int segments = (words + kShareThreads - 1) / kShareThreads;
    last = (int)blockIdx.x == (segments - 1) % ctas;
    for (int g = blockIdx.x; g < segments; g += ctas) {
      const int k = g * kShareThreads + threadIdx.x;
      const uint32_t bits = share_sum(k < words ? __popc(__ldcg(bitmap + k)) : 0u, s_warp);
      if (threadIdx.x == 0) plan->segment_bits[g] = bits;
    }
    if (!grid_barrier(&ctl->barrier[1], ctas, err)) return;
    {  // segment starts: two counts per thread
      const int g = 2 * threadIdx.x;
      const uint32_t c0 = g < segments ? __ldcg(plan->segment_bits + g) : 0u;
      const uint32_t c1 = g + 1 < segments ? __ldcg(plan->segment_bits + g + 1) : 0u;
      const uint32_t sum = c0 + c1;
      uint32_t incl = sum;
#pragma unroll
      for (int off = 1; off < 32; off <<= 1) {
        const uint32_t t = __shfl_up_sync(0xffffffffu, incl, off);
        if (lane >= off) incl += t;
      }
      __syncthreads();
      if (lane == 31) s_warp[warp] = incl;
      __syncthreads();
      const uint32_t at = __reduce_add_sync(0xffffffffu, lane < warp ? s_warp[lane] : 0u) + incl - sum;
      s_words[g] = at;
      s_words[g + 1] = at + c0;
      __syncthreads();
    }
    for (int g = blockIdx.x; g < segments; g += ctas) {
      const int k = g * kShareThreads + threadIdx.x;
      const uint32_t w = k < words ? __ldcg(bitmap + k) : 0u;
      run = s_words[g];
      const uint32_t pos = word_positions(w, run, s_warp);
      emit_words(w, lo + (uint32_t)k * 32u, pos, stage, out);
    }
  }
  if (last && threadIdx.x == 0) {  // run: the bits up to the last word's
    if (ctl->no_hit) out[run++] = kNoHit;
    result[0] = (int)run;
  }
}

__device__ __forceinline__ void emit_kernel_cta(const uint32_t* bitmap, Control* ctl, Plan* plan, int32_t* out,
                                                int* result, int* err) {
  extern __shared__ __align__(128) uint32_t s_words[];
  __shared__ uint32_t s_warp[kShareWarps];
  if (plan->path != kPathPartition) return;
  emit_bitmap(bitmap, ctl, plan, gridDim.x, s_words, s_warp, out, result, err);
}
__global__ void __launch_bounds__(kShareThreads) emit_kernel(const uint32_t* bitmap, Control* ctl, Plan* plan,
                                  int32_t* out, int* result, int* err, const DoneFlag done) {
  emit_kernel_cta(bitmap, ctl, plan, out, result, err);
  publish(done);
}

// Sets the keys' bits straight in the bitmap, then writes its values.  Keys
// that many CTAs of the compaction kept arrive together, and atomics on one
// word queue (450 thousand keys over 3 thousand words: 120 us): each CTA takes
// a slice of up to 2^20 bits and a share of the keys, builds the slice in
// shared memory from those of them that fall in it, and adds its words to the
// global bitmap, starting at a place of its own.  Where few keys span several
// slices each thread looks at a bit in memory before it sets it, one key at a
// time so that the looks see the bits set before.  A range wider than the
// bitmap that the compaction cleared is cleared here first (until ranges of up
// to 2^26 values had a bitmap at every size, 8 thousand to 2 million words
// took the six launches of the radix passes: 73 to 94 us, now 37 to 72).
static_assert(kDirectSliceWords * 4 >= kEmitSmemBytes, "the slice's memory serves the writing too");
__device__ __forceinline__ void direct_bitmap_kernel_cta(const uint32_t* keys, Control* ctl, Plan* plan,
                                                         uint32_t* bitmap, int32_t* out, int* result, int* err) {
  extern __shared__ __align__(128) uint32_t s_slice[];
  __shared__ uint32_t s_warp[kShareWarps];
  if (plan->path != kPathDirect) return;
  const uint32_t m = (uint32_t)ctl->keys, lo = ~ctl->range[0];
  const int words = (int)plan->bitmap_words;
  int ctas = gridDim.x;
  if (plan->clear) {
    uint4* units = reinterpret_cast<uint4*>(bitmap);
    for (int i = blockIdx.x * kShareThreads + threadIdx.x; i < (words + 3) / 4; i += gridDim.x * kShareThreads)
      units[i] = make_uint4(0, 0, 0, 0);
    if (!grid_barrier(&ctl->barrier[2], ctas, err)) return;
  }
  const int slices = (words + kDirectSliceWords - 1) / kDirectSliceWords;
  if (slices > 1 && (m < kDirectSliceKeys || slices > ctas / kDirectSliceCtas)) {
    for (uint32_t i = blockIdx.x * kShareThreads + threadIdx.x; i < m; i += gridDim.x * kShareThreads) {
      const uint32_t bit = __ldg(keys + i) - lo, mask = 1u << (bit & 31);
      if ((__ldcg(bitmap + (bit >> 5)) & mask) == 0) atomicOr(bitmap + (bit >> 5), mask);
    }
  } else {
    // one slice: a CTA per 1024 keys builds, and per 1024 words at least writes
    // (8193 words, 820 keys over a million bits: 62 us with one CTA for both, 40 so)
    int builders = ctas;
    if (slices == 1) {
      builders = (int)min((uint32_t)ctas, (m + kShareThreads - 1) / kShareThreads);
      ctas = min(ctas, max(builders, (words + kShareThreads - 1) / kShareThreads));
      if ((int)blockIdx.x >= ctas) return;
    }
    const int slice = (int)blockIdx.x % slices, part = (int)blockIdx.x / slices;
    const int parts = (builders - 1 - slice) / slices + 1;
    if ((int)blockIdx.x < builders) {
      uint32_t* slice_words = bitmap + slice * kDirectSliceWords;
      const int n = min(kDirectSliceWords, words - slice * kDirectSliceWords);
      for (int i = threadIdx.x; i < n; i += kShareThreads) s_slice[i] = 0;
      __syncthreads();
      const uint32_t low = lo + (uint32_t)slice * (kDirectSliceWords * 32u), bits = (uint32_t)n * 32u;
      const uint32_t step = (uint32_t)parts * kShareThreads;
      auto set = [&](uint32_t key) {
        const uint32_t bit = key - low, mask = 1u << (bit & 31);
        if (bit < bits && (s_slice[bit >> 5] & mask) == 0) atomicOr(s_slice + (bit >> 5), mask);
      };
      // eight keys in flight per thread by 16-byte loads, four by scalar ones where
      // there are too few for that (30 million words, 15 million kept, three
      // slices: the call took 168 us with four scalar ones, 158 so; 16 keys as many)
      const uint32_t units = m / (step * 4) * step;  // 16-byte units that give every thread as many
      const uint4* keys4 = reinterpret_cast<const uint4*>(keys);
      for (uint32_t u = part * kShareThreads + threadIdx.x; u < units; u += step * 2) {
        uint4 v[2];
#pragma unroll
        for (int r = 0; r < 2; ++r) {
          const uint32_t none = low - 1u;  // in no slice
          v[r] = u + r * step < units ? __ldg(keys4 + u + r * step) : make_uint4(none, none, none, none);
        }
#pragma unroll
        for (int r = 0; r < 2; ++r) set(v[r].x), set(v[r].y), set(v[r].z), set(v[r].w);
      }
      for (uint32_t i = units * 4 + part * kShareThreads + threadIdx.x; i < m; i += step * 4) {
        uint32_t key[4];
#pragma unroll
        for (int r = 0; r < 4; ++r) key[r] = i + r * step < m ? __ldg(keys + i + r * step) : low - 1u;
#pragma unroll
        for (int r = 0; r < 4; ++r) set(key[r]);
      }
      __syncthreads();
      const int turn = (int)((unsigned long long)n * part / parts);
      for (int i = threadIdx.x; i < n; i += kShareThreads) {
        const int k = i + turn < n ? i + turn : i + turn - n;
        const uint32_t v = s_slice[k];
        if (v && (__ldcg(slice_words + k) & v) != v) atomicOr(slice_words + k, v);
      }
    }
  }
  if (!grid_barrier(&ctl->barrier[0], ctas, err)) return;
  emit_bitmap(bitmap, ctl, plan, ctas, s_slice, s_warp, out, result, err);
}
__global__ void __launch_bounds__(kShareThreads) direct_bitmap_kernel(const uint32_t* keys, Control* ctl, Plan* plan,
                                  uint32_t* bitmap, int32_t* out, int* result, int* err, const DoneFlag done) {
  direct_bitmap_kernel_cta(keys, ctl, plan, bitmap, out, result, err);
  publish(done);
}

// Histogram of the range buckets (top 8 bits of key - min) of the kept keys,
// each lane counting in its own bank (see digit_hist_kernel); the last CTA
// turns the counts into offsets.
__global__ void __launch_bounds__(kThreads) range_hist_kernel(const uint32_t* keys, Control* ctl, Plan* plan) {
  __shared__ uint32_t sh[kBuckets * 32];
  wait_for_dependency();
  if (plan->path != kPathPartition) return;
  const uint32_t m = (uint32_t)ctl->keys, lo = ~ctl->range[0];
  const int shift = (int)plan->range_shift;
  for (int i = threadIdx.x; i < kBuckets * 32; i += kThreads) sh[i] = 0;
  __syncthreads();
  const int lane = threadIdx.x & 31;
  for (uint32_t i0 = blockIdx.x * kThreads * 8u; i0 < m; i0 += gridDim.x * kThreads * 8u) {
    uint32_t k[8];
#pragma unroll
    for (int r = 0; r < 8; ++r) {
      const uint32_t i = i0 + r * kThreads + threadIdx.x;
      k[r] = i < m ? __ldg(keys + i) : 0u;
    }
#pragma unroll
    for (int r = 0; r < 8; ++r)
      if (i0 + r * kThreads + threadIdx.x < m) atomicAdd(&sh[((k[r] - lo) >> shift) * 32 + lane], 1u);
  }
  __syncthreads();
  {
    uint32_t sum = 0;
#pragma unroll 8
    for (int k = 0; k < 32; ++k) sum += sh[threadIdx.x * 32 + ((lane + k) & 31)];
    if (sum) atomicAdd(&ctl->range_counts[threadIdx.x], sum);
  }
  if (!last_cta(&ctl->done[1], gridDim.x)) return;
  __syncthreads();
  sh[threadIdx.x] = *(volatile uint32_t*)&ctl->range_counts[threadIdx.x];
  __syncthreads();
  if (threadIdx.x < 32) warp_scan_256(sh, sh);
  __syncthreads();
  plan->range_offsets[threadIdx.x] = sh[threadIdx.x];
  plan->cursors[threadIdx.x * kCursorStride] = sh[threadIdx.x];
}

// Range partition of the bitmap path.  Unstable (the bitmap does not care
// about order): tiles of 4096 keys, grid-strided; a key's slot in its range
// bucket comes from a shared per-tile count, the tile claims one range per
// bucket from the bucket's cursor, and the keys are staged in shared memory in
// bucket order so each bucket's run goes out contiguously while the next
// tile's keys load.  A key takes its slot with an atomic of its own, except
// in the bucket of a lane picked each round, whose lanes share one: feedback's
// frequent blocks lie in one bucket, where single atomics would queue.  No CTA
// waits on another.
__global__ void __launch_bounds__(kThreads, 4) range_partition_kernel(const uint32_t* in, uint32_t* out,
                                                                   const Control* ctl, Plan* plan) {
  __shared__ uint32_t s_cnt[kBuckets];    // per-tile count, then the tile-local start of each bucket
  __shared__ uint32_t s_base[kBuckets];   // global start of each bucket's run
  __shared__ uint32_t s_keys[kTile];
  wait_for_dependency();
  if (plan->path != kPathPartition) return;
  const uint32_t m = (uint32_t)ctl->keys, lo = ~ctl->range[0];
  const int shift = (int)plan->range_shift;
  uint32_t* cursors = plan->cursors;
  const int lane = threadIdx.x & 31;
  const unsigned lt = (1u << lane) - 1;
  const uint32_t stride = gridDim.x * (uint32_t)kTile;
  uint32_t k[kItems];
#pragma unroll
  for (int r = 0; r < kItems; ++r) {
    const uint32_t i = blockIdx.x * (uint32_t)kTile + r * kThreads + threadIdx.x;
    k[r] = i < m ? __ldg(in + i) : 0u;
  }
  for (uint32_t base = blockIdx.x * (uint32_t)kTile; base < m; base += stride) {
    const uint32_t valid = min((uint32_t)kTile, m - base);
    s_cnt[threadIdx.x] = 0;
    __syncthreads();
    uint32_t slot[kItems / 2];  // two 16-bit slots (< 4096) per word
#pragma unroll
    for (int r = 0; r < kItems; ++r) {
      const bool ok = r * kThreads + threadIdx.x < valid;
      const uint32_t b = ok ? (k[r] - lo) >> shift : 0x100u;
      const uint32_t shared_b = __shfl_sync(0xffffffffu, b, r);  // lane r's bucket
      const unsigned peers = __ballot_sync(0xffffffffu, b == shared_b);
      uint32_t sl = 0;
      if (ok) {
        const bool sharing = b == shared_b;
        const int leader = __ffs(peers) - 1;
        if (!sharing || lane == leader) sl = atomicAdd(&s_cnt[b], sharing ? (uint32_t)__popc(peers) : 1u);
      }
      const uint32_t first = __shfl_sync(0xffffffffu, sl, __ffs(peers) - 1);
      if (b == shared_b) sl = first + __popc(peers & lt);
      slot[r / 2] = (r & 1) ? slot[r / 2] | (sl << 16) : sl;
    }
    __syncthreads();
    {
      const uint32_t c = s_cnt[threadIdx.x];
      if (c) s_base[threadIdx.x] = atomicAdd(cursors + threadIdx.x * kCursorStride, c);
    }
    __syncthreads();
    if (threadIdx.x < 32) warp_scan_256(s_cnt, s_cnt);  // tile-local bucket starts
    __syncthreads();
#pragma unroll
    for (int r = 0; r < kItems; ++r)
      if (r * kThreads + threadIdx.x < valid)
        s_keys[s_cnt[(k[r] - lo) >> shift] + ((r & 1) ? slot[r / 2] >> 16 : slot[r / 2] & 0xffffu)] = k[r];
    // the next tile's keys are in flight during the write-out
#pragma unroll
    for (int r = 0; r < kItems; ++r) {
      const uint32_t i = base + stride + r * kThreads + threadIdx.x;
      k[r] = i < m ? __ldg(in + i) : 0u;
    }
    __syncthreads();
    for (uint32_t i = threadIdx.x; i < valid; i += kThreads) {
      const uint32_t key = s_keys[i];
      const uint32_t b = (key - lo) >> shift;
      out[s_base[b] + i - s_cnt[b]] = key;
    }
    __syncthreads();  // shared state is reused by the next tile
  }
}

// One range bucket's bitmap slice (at most 2^18 bits) built in shared memory
// from its partitioned keys (a shared atomicOr only for bits not yet set),
// then OR-ed into the global bitmap word by word
// (only words with bits set; a word shared with a neighbouring bucket is
// combined by the atomic).  Work items are chunks of kChunk keys of one
// bucket, claimed from a counter, so a bucket holding most keys (feedback is
// Zipf-like) is spread over many CTAs.
constexpr int kChunk = 16384;
constexpr int kSliceWords = (1 << (kMaxSpanLog2 - 8)) / 32 + 1;
__global__ void __launch_bounds__(kThreads) bucket_bitmap_kernel(const uint32_t* keys, Control* ctl, const Plan* plan,
                                                                 uint32_t* bitmap) {
  __shared__ uint32_t s_bits[kSliceWords];
  __shared__ uint32_t s_first[kBuckets + 1];  // first item of each bucket; [256] = all items
  __shared__ int s_item;
  wait_for_dependency();
  if (plan->path != kPathPartition) return;
  const uint32_t lo = ~ctl->range[0];
  const int shift = (int)plan->range_shift;
  s_first[threadIdx.x] = (ctl->range_counts[threadIdx.x] + kChunk - 1) / kChunk;
  __syncthreads();
  if (threadIdx.x < 32) {
    const uint32_t total = warp_scan_256(s_first, s_first);
    if (threadIdx.x == 0) s_first[kBuckets] = total;
  }
  __syncthreads();
  const uint32_t items = s_first[kBuckets];
  for (;;) {
    if (threadIdx.x == 0) s_item = atomicAdd(&ctl->bucket_items, 1);
    __syncthreads();
    const uint32_t item = (uint32_t)s_item;
    if (item >= items) return;
    int b = 0;  // the bucket: last with s_first[b] <= item
    for (int step = kBuckets / 2; step > 0; step >>= 1)
      if (s_first[b + step] <= item) b += step;
    const uint32_t count = ctl->range_counts[b];
    const uint32_t first = plan->range_offsets[b] + (item - s_first[b]) * kChunk;
    const uint32_t end = plan->range_offsets[b] + min(count, (item - s_first[b] + 1) * kChunk);
    const uint32_t bit0 = (uint32_t)b << shift;  // the bucket's first bit
    const uint32_t w0 = bit0 >> 5;
    const int words = (int)(((bit0 + (1u << shift) - 1) >> 5) - w0 + 1);
    for (int i = threadIdx.x; i < words; i += kThreads) s_bits[i] = 0;
    __syncthreads();
    for (uint32_t r0 = first; r0 < end; r0 += kThreads * 8) {  // the same rounds for every thread
      uint32_t k[8];
#pragma unroll
      for (int r = 0; r < 8; ++r) {
        const uint32_t i = r0 + r * kThreads + threadIdx.x;
        k[r] = i < end ? __ldg(keys + i) : 0u;
      }
#pragma unroll
      for (int r = 0; r < 8; ++r) {
        if (r0 + r * kThreads + threadIdx.x >= end) continue;
        const uint32_t bit = k[r] - lo;
        const uint32_t word = (bit >> 5) - w0, mask = 1u << (bit & 31);
        // a bit already set costs a (broadcast) load, not an atomic: frequent
        // keys stop contending once set; two lanes racing both OR the same bit
        if ((s_bits[word] & mask) == 0) atomicOr(s_bits + word, mask);
      }
    }
    __syncthreads();
    for (int i = threadIdx.x; i < words; i += kThreads)
      if (s_bits[i]) atomicOr(bitmap + w0 + i, s_bits[i]);
    __syncthreads();  // s_bits / s_item are reused by the next item
  }
}

// ---- inclusive scan (wrapping int32) ---------------------------------------------
// One CTA per SM, in rounds: in round k CTA c has tile k * gridDim.x + c, which
// it holds in shared memory from the one read to the one write.  A round's sums
// are published by every CTA and read by every CTA, so a CTA knows the sum of
// all rounds before and needs no walk over its predecessors.  Three buffers
// let the steps overlap: while tile k + 1 is on its way (one bulk async copy),
// tile k is summed and its sum published, and then tile k - 1, whose round has
// had that long to arrive, is scanned and written.  A look-back of tiles in
// claim order, however wide, took 570 to 840 us on 2^28 values where the reads
// and writes alone took 400 (a tile's slot waits for the slowest load before
// it).  The CTAs wait on one another, so the launch is cooperative; each wait
// is bounded.  Sums wrap like the reference's int arithmetic.
//
// The array is taken from the 16-byte boundary at or before it: element i of
// the tiles is data[i - mis], zero before `mis` and from `end` on.  The copies
// move the whole 16-byte units inside the array, the threads the elements
// before and after them.
constexpr int kScanThreads = 512;
constexpr int kScanWarps = kScanThreads / 32;
constexpr int kScanRows = 8;                            // rows of 128 elements per warp, at most
constexpr int kScanTile = kScanWarps * 128 * kScanRows;  // 16384 elements
constexpr int kScanBuffers = 3;
constexpr int kScanBlock = kScanThreads + 32;            // and the warp that collects the rounds' sums
constexpr int kScanSmemBytes = kScanBuffers * kScanTile * 4;

// Thread 0 starts the copy of the tile's whole units; the others fill in the
// array's first and last elements and zeros.
__device__ __forceinline__ void scan_load(uint32_t* buf, const int32_t* base, int first, int rows, int mis, int end,
                                          unsigned long long* bar) {
  const int stop = first + rows * (kScanWarps * 128);
  const int a = max(first, (mis + 3) & ~3), b = max(a, min(stop, end) & ~3);
  if (threadIdx.x == 0) bulk_load(buf + (a - first), base + a, (uint32_t)(b - a) * 4u, bar);
  auto edge = [&](int i) { buf[i - first] = i >= mis && i < end ? (uint32_t)base[i] : 0u; };
  if ((int)threadIdx.x < a - first) edge(first + threadIdx.x);  // the first unit
  for (int i = b + threadIdx.x; i < stop; i += kScanThreads) edge(i);
}

// The scanning warps' barrier (the collecting warp does not take part).
__device__ __forceinline__ void scan_sync() { asm volatile("bar.sync 1, %0;" ::"n"(kScanThreads) : "memory"); }

// The same; true when every one of them passes true.
__device__ __forceinline__ bool scan_sync_and(bool v) {
  uint32_t r;
  asm volatile(
      "{\n .reg .pred p, q;\n setp.ne.u32 p, %1, 0;\n bar.red.and.pred q, 1, %2, p;\n selp.u32 %0, 1, 0, q;\n}\n"
      : "=r"(r)
      : "r"((uint32_t)v), "n"(kScanThreads)
      : "memory");
  return r != 0;
}

__device__ __forceinline__ void mbar_arrive(unsigned long long* bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_addr(bar)) : "memory");
}

__device__ __forceinline__ void scan_kernel_cta(int32_t* data, int n, int rows, unsigned long long* status,
                                                uint32_t tag, int* err) {
  extern __shared__ __align__(128) uint32_t s_tiles[];
  __shared__ unsigned long long s_bar[kScanBuffers];        // a tile has landed
  __shared__ unsigned long long s_collected[2], s_used[2];  // a round's sums are in s_round; they are used
  __shared__ uint32_t s_warp[kScanBuffers][kScanWarps];
  // sum of the round's tiles before this CTA's, of all of them, and whether every one arrived
  __shared__ uint32_t s_round[2][3];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int mis = (int)((reinterpret_cast<uintptr_t>(data) >> 2) & 3u);
  int32_t* base = data - mis;
  const int end = n + mis, tile_size = rows * (kScanWarps * 128);  // n < 2^30
  const int tiles = (end + tile_size - 1) / tile_size, step = gridDim.x;
  if (threadIdx.x == 0) {
    for (int b = 0; b < kScanBuffers; ++b) mbar_init(&s_bar[b]);
    for (int b = 0; b < 2; ++b) mbar_init(&s_collected[b]), mbar_init(&s_used[b]);
    mbar_init_fence();
  }
  __syncthreads();
  if (warp == kScanWarps) {  // collects each round's sums
    for (int k = 0; (int)blockIdx.x + k * step < tiles; ++k) {
      const int row0 = k * step, count = min(step, tiles - row0);
      uint32_t before = 0, all = 0;
      bool ok = true;
      for (int i = lane; tiles > 1 && i < count; i += 32) {
        unsigned long long w = ld_volatile64(status + row0 + i);
        long long spins = 0;
        const unsigned long long start = lb_ready(w, tag) ? 0 : global_ns();
        while (!lb_ready(w, tag)) {
          if (wait_over(spins, start)) {
            set_error(err);
            ok = false;
            break;
          }
          __nanosleep(64);
          w = ld_volatile64(status + row0 + i);
        }
        all += (uint32_t)w;
        if (i < (int)blockIdx.x) before += (uint32_t)w;
      }
      ok = __all_sync(0xffffffffu, ok);
      before = __reduce_add_sync(0xffffffffu, before);
      all = __reduce_add_sync(0xffffffffu, all);
      // the slot's sums of two rounds ago are used
      if (k >= 2 && !mbar_wait(&s_used[k & 1], (uint32_t)(k / 2 - 1) & 1u, err)) ok = false;
      if (lane == 0) {
        s_round[k & 1][0] = before;
        s_round[k & 1][1] = all;
        s_round[k & 1][2] = ok ? 1u : 0u;
        mbar_arrive(&s_collected[k & 1]);
      }
      if (!__all_sync(0xffffffffu, ok)) return;
    }
    return;
  }
  const int seg = warp * rows * 128 + lane * 4;  // the thread's first element in a tile
  int issued = kScanBuffers;                     // rounds whose copies were started
  for (int b = 0; b < kScanBuffers; ++b) {
    const int t = blockIdx.x + b * step;
    if (t < tiles) scan_load(s_tiles + b * kScanTile, base, t * tile_size, rows, mis, end, &s_bar[b]);
  }
  // A wait that ran out (error flag set) ends the CTA once the copies under way
  // have landed (bounded), so that nothing lands after it has left.
  auto leave = [&](int k) {
    if (threadIdx.x == 0)
      for (int q = k; q <= k + 2; ++q)
        if ((int)blockIdx.x + q * step < tiles && q < issued)
          mbar_wait(&s_bar[q % kScanBuffers], (uint32_t)(q / kScanBuffers) & 1u, err);
  };
  uint32_t carry = 0;  // sum of all rounds before
  for (int k = 0;; ++k) {
    const int t = blockIdx.x + k * step;  // below 2^31: at most 2^30 / 2048 tiles
    if (t < tiles) {
      const int b = k % kScanBuffers;
      const bool landed = mbar_wait(&s_bar[b], (uint32_t)(k / kScanBuffers) & 1u, err);
      scan_sync();  // the threads' own elements are in place
      const uint32_t* tile = s_tiles + b * kScanTile;
      uint32_t sum = 0;
#pragma unroll
      for (int r = 0; r < kScanRows; ++r)
        if (r < rows) {
          const uint4 q = *reinterpret_cast<const uint4*>(tile + seg + r * 128);
          sum += q.x + q.y + q.z + q.w;
        }
      sum = __reduce_add_sync(0xffffffffu, sum);
      if (lane == 0) s_warp[b][warp] = sum;
      if (!scan_sync_and(landed)) return leave(k);
      if (warp == 0 && tiles > 1) {
        const uint32_t total = __reduce_add_sync(0xffffffffu, lane < kScanWarps ? s_warp[b][lane] : 0u);
        if (lane == 0) st_volatile64(status + t, lb_word(tag, 2u, total));
      }
    }
    if (k > 0) {  // finish the tile of the round before
      const int p = t - step, b = (k - 1) % kScanBuffers, slot = (k - 1) & 1;
      const bool arrived = mbar_wait(&s_collected[slot], (uint32_t)((k - 1) / 2) & 1u, err) && s_round[slot][2] != 0;
      if (!scan_sync_and(arrived)) return leave(k);
      uint32_t* tile = s_tiles + b * kScanTile;
      uint32_t run = carry + s_round[slot][0];
      run += __reduce_add_sync(0xffffffffu, lane < warp ? s_warp[b][lane] : 0u);  // warp < 16
      carry += s_round[slot][1];
      uint32_t v[kScanRows][4];
#pragma unroll
      for (int r = 0; r < kScanRows; ++r) {
        if (r >= rows) break;
        const uint4 q = *reinterpret_cast<const uint4*>(tile + seg + r * 128);
        v[r][0] = q.x;
        v[r][1] = v[r][0] + q.y;
        v[r][2] = v[r][1] + q.z;
        v[r][3] = v[r][2] + q.w;
      }
      scan_sync();  // the buffer and the slot are read
      if (threadIdx.x == 0) mbar_arrive(&s_used[slot]);
      const int next = p + kScanBuffers * step;
      if (next < tiles) scan_load(tile, base, next * tile_size, rows, mis, end, &s_bar[b]);
      issued = k + 3;
#pragma unroll
      for (int r = 0; r < kScanRows; ++r) {
        if (r >= rows) break;
        uint32_t incl = v[r][3];
#pragma unroll
        for (int off = 1; off < 32; off <<= 1) {
          const uint32_t u = __shfl_up_sync(0xffffffffu, incl, off);
          if (lane >= off) incl += u;
        }
        const uint32_t at = run + incl - v[r][3];
        run += __shfl_sync(0xffffffffu, incl, 31);
        const int i = p * tile_size + seg + r * 128;
        if (i >= mis && i + 4 <= end) {
          *reinterpret_cast<int4*>(base + i) = make_int4((int)(v[r][0] + at), (int)(v[r][1] + at),
                                                         (int)(v[r][2] + at), (int)(v[r][3] + at));
        } else {
#pragma unroll
          for (int j = 0; j < 4; ++j)
            if (i + j >= mis && i + j < end) base[i + j] = (int32_t)(v[r][j] + at);
        }
      }
    }
    if (t >= tiles) return;
  }
}
__global__ void __launch_bounds__(kScanBlock, 1) scan_kernel(int32_t* data, int n, int rows,
                                  unsigned long long* status, uint32_t tag, int* err, const DoneFlag done) {
  scan_kernel_cta(data, n, rows, status, tag, err);
  publish(done);
}

// Copy of an array that does not start on a 16-byte boundary (the digit passes
// bring their tiles in by 16-byte copies), kItems loads in flight per thread.
__global__ void __launch_bounds__(kThreads) copy_keys_kernel(const uint32_t* in, uint32_t* out, int n) {
  for (uint32_t i0 = blockIdx.x * kTile + threadIdx.x; i0 < (uint32_t)n; i0 += gridDim.x * kTile) {
    uint32_t k[kItems];
#pragma unroll
    for (int r = 0; r < kItems; ++r)
      if (i0 + r * kThreads < (uint32_t)n) k[r] = __ldcs(in + i0 + r * kThreads);
#pragma unroll
    for (int r = 0; r < kItems; ++r)
      if (i0 + r * kThreads < (uint32_t)n) out[i0 + r * kThreads] = k[r];
  }
}

int tiles_of(int n, int tile) { return std::max(1, (int)(((long long)n + tile - 1) / tile)); }

// Resident CTAs of kernel K of `threads` threads, at most `tiles`.
template <auto K>
int persistent_grid(int tiles, int threads = kThreads, int smem = 0) {
  static int resident[64] = {};  // by device (the callers hold prims_mutex())
  int dev = 0;
  cudaGetDevice(&dev);
  int& r = resident[dev & 63];
  if (!r) {
    int sms = 0, per_sm = 0;
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    if (smem > 48 * 1024) cudaFuncSetAttribute(K, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, K, threads, smem);
    r = sms * (per_sm > 0 ? per_sm : 1);
  }
  return std::min(r, tiles);
}

// Kernel K behind the one before it on the stream, grid CTAs of `threads`.
template <auto K, class... Args>
cudaError_t launch_behind(int tiles, int threads, int smem, cudaStream_t s, Args... args) {
  cudaLaunchAttribute attr{};
  attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr.val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(persistent_grid<K>(tiles, threads, smem));
  cfg.blockDim = dim3(threads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cfg.attrs = &attr;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, K, args...);
}

// Digit counts, offsets and the plan of the passes over n keys (or *count).
cudaError_t launch_digit_hist(const uint32_t* keys, int n, const int* count, uint32_t flip, bool in_place,
                              int split_ranges, const SortScratchLayout& l, cudaStream_t s) {
  return launch_behind<digit_hist_kernel>(tiles_of(n, kHistThreads * 4), kHistThreads, kHistSmemBytes, s, keys, n, count,
                                          flip, in_place, split_ranges, l.control, l.plan);
}

// The four digit passes.  `sign_flip`: the keys are signed words (the top
// digit's upper bit is flipped as it is read).
cudaError_t launch_digits(const DigitBuffers& bufs, int n, const int* count, bool sign_flip,
                          const SortScratchLayout& l, unsigned long long* status, uint32_t epoch, int* err,
                          const DoneFlag& done, cudaStream_t s) {
  const int grid = persistent_grid<digit_kernel>(tiles_of(n, kDigitTile), kDigitThreads, kDigitSmemBytes);
  for (int p = 0; p < kPasses; ++p) {
    cudaLaunchAttribute attr{};
    attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(grid);
    cfg.blockDim = dim3(kDigitThreads);
    cfg.dynamicSmemBytes = kDigitSmemBytes;
    cfg.stream = s;
    cfg.attrs = &attr;
    cfg.numAttrs = 1;
    const cudaError_t e = cudaLaunchKernelEx(&cfg, digit_kernel, bufs, n, count, p,
                                             sign_flip && p == kPasses - 1 ? 0x80u : 0u, l.plan, status,
                                             &l.control->tiles[p], epoch * 8u + (uint32_t)p, err,
                                             p == kPasses - 1 ? done : DoneFlag{});
    if (e != cudaSuccess) return e;
  }
  return cudaSuccess;
}

// The split of n keys.  Two regions per SM or more, so that every SM sorts, and
// of more keys a multiple of that, so that every CTA sorts as many; regions of
// 512 keys on average or more.
SplitShape split_shape(int n, const SortScratchLayout& l) {
  SplitShape sh{};
  const int resident = persistent_grid<split_sort_kernel<kSplitGroups>>(1 << 30, kSplitThreads, kSortSmemBytes);
  const long long full = ((long long)n + (long long)resident * kSplitFill - 1) / ((long long)resident * kSplitFill);
  const long long ranges = std::min<long long>(resident * full, n / 512);
  if (ranges < 1 || ranges > kSplitRanges) return sh;
  const double share = (double)n / (double)ranges;
  const double room = share * 1.0625 + 8 * std::sqrt(share) + 64;
  sh.room = (uint32_t)std::min<long long>(kSplitRoom, ((long long)room + 3) / 4 * 4);
  if ((size_t)ranges * sh.room > l.key_words) return sh;
  sh.ranges = (int)ranges;
  const int moving = persistent_grid<split_kernel<true, kMoveGroups>>(1 << 30, kMoveThreads, kSplitSmemBytes);
  // tiles: as many for every resident CTA
  const long long turns = ((long long)n + (long long)moving * kMoveTile - 1) / ((long long)moving * kMoveTile);
  const long long tile = ((long long)n + moving * turns - 1) / (moving * turns);
  sh.tile = (int)std::max<long long>(4 * kMoveThreads, (tile + 3) / 4 * 4);
  // about a bin per key, as shared memory allows
  sh.bins = std::min(kSortBins, ((int)sh.room + kSortBinsUnit - 1) / kSortBinsUnit * kSortBinsUnit);
  return sh;
}

// f of the smallest of 1, 2, 4 and 8 units per thread with which `threads`
// threads hold `keys`: small tiles and regions have kernels that are not unrolled
// over eight (a call with eight always and so: 300 thousand keys 38.8 and 34.9 us,
// a million 45.5 and 41.4).
template <class F>
cudaError_t by_units(uint32_t keys, uint32_t threads, const F& f) {
  if (keys <= 4 * threads) return f(std::integral_constant<int, 1>());
  if (keys <= 8 * threads) return f(std::integral_constant<int, 2>());
  if (keys <= 16 * threads) return f(std::integral_constant<int, 4>());
  return f(std::integral_constant<int, 8>());
}

cudaError_t launch_split(uint32_t* keys, int n, const SplitShape& shape, const SortScratchLayout& l, int* again,
                         const DoneFlag& done, cudaStream_t s) {
  static_assert(kMoveGroups == 8 && kSplitGroups == 8, "by_units ends there");
  const int tiles = tiles_of(n, shape.tile);
  const bool whole = (reinterpret_cast<uintptr_t>(keys) & 15) == 0;
  const uint32_t *in = keys, *regions = l.keys_a;
  const Plan* plan = l.plan;
  const cudaError_t e = by_units((uint32_t)shape.tile, kMoveThreads, [&](auto units) {
    constexpr int kGroups = decltype(units)::value;
    return whole ? launch_behind<split_kernel<true, kGroups>>(tiles, kMoveThreads, kSplitSmemBytes, s, in, n, l.keys_a,
                                                              shape, l.control, l.plan)
                 : launch_behind<split_kernel<false, kGroups>>(tiles, kMoveThreads, kSplitSmemBytes, s, in, n,
                                                               l.keys_a, shape, l.control, l.plan);
  });
  if (e != cudaSuccess) return e;
  return by_units(shape.room, kSplitThreads, [&](auto units) {
    constexpr int kGroups = decltype(units)::value;
    return launch_behind<split_sort_kernel<kGroups>>(shape.ranges, kSplitThreads, kSortSmemBytes, s, keys, n, regions,
                                                     shape, l.control, plan, again, done);
  });
}

template <int kRounds>
void launch_small_sort(int32_t* data, int n, const DoneFlag& done, cudaStream_t s) {
  constexpr int bytes = small_smem_bytes<kRounds>();
  const int grid = persistent_grid<small_sort_kernel<kRounds>>(1, kSmallThreads, bytes);
  small_sort_kernel<kRounds><<<grid, kSmallThreads, bytes, s>>>(data, n, done);
}
template <int kRounds>
void launch_small_unique(const int32_t* words, int n, int nib, int32_t* out, int* result, const DoneFlag& done,
                         cudaStream_t s) {
  constexpr int bytes = small_smem_bytes<kRounds>();
  const int grid = persistent_grid<small_unique_kernel<kRounds>>(1, kSmallThreads, bytes);
  small_unique_kernel<kRounds><<<grid, kSmallThreads, bytes, s>>>(words, n, nib, make_divider((uint32_t)nib), out,
                                                                 result, done);
}

// Waits, as a look-back does, on a word that nothing publishes: the wait must
// give up after g_wait_ns, set the error flag and return.
__global__ void bounded_wait_probe_kernel(const unsigned long long* never, int* err) {
  if (threadIdx.x == 0 && blockIdx.x == 0) look_back(never, 1, 1, 0, 1u, err);
}

}  // namespace

cudaError_t bounded_wait_probe(double limit_s, int* err, cudaStream_t s) {
  const unsigned long long limit = (unsigned long long)(limit_s * 1e9), normal = 1000000000ull;
  unsigned long long* never = nullptr;
  cudaError_t e = cudaMalloc(&never, 2 * sizeof(unsigned long long));
  if (e != cudaSuccess) return e;
  if ((e = cudaMemsetAsync(never, 0, 2 * sizeof(unsigned long long), s)) == cudaSuccess &&
      (e = cudaMemcpyToSymbolAsync(g_wait_ns, &limit, sizeof(limit), 0, cudaMemcpyHostToDevice, s)) == cudaSuccess) {
    bounded_wait_probe_kernel<<<1, 32, 0, s>>>(never, err);
    e = cudaGetLastError();
  }
  cudaError_t e2 = cudaMemcpyToSymbolAsync(g_wait_ns, &normal, sizeof(normal), 0, cudaMemcpyHostToDevice, s);
  cudaError_t e3 = cudaStreamSynchronize(s);
  cudaFree(never);
  return e != cudaSuccess ? e : (e2 != cudaSuccess ? e2 : e3);
}

size_t sort_scratch_bytes(int n) { return n <= kSmall ? 0 : layout(nullptr, n).bytes; }
size_t feedback_scratch_bytes(int n) { return n <= kSmall ? 0 : layout(nullptr, n, true).bytes; }
size_t sort_status_bytes(int n) { return n <= kSmall ? 0 : (size_t)tiles_of(n, kDigitTile) * kBuckets * 8; }
// the digit passes' words, or the unique kernel's one per tile of sorted keys
size_t feedback_status_bytes(int n) { return std::max(sort_status_bytes(n), (size_t)tiles_of(n, kTile) * 8); }
size_t scan_status_bytes(int n) { return ((size_t)tiles_of(n, kScanTile) + 1024) * 8; }

cudaError_t feedback_unique_device(const int32_t* words, int n, int nib, int32_t* unique_out, void* scratch,
                                   unsigned long long* status, uint32_t epoch, int* result, int* err,
                                   const DoneFlag& done, cudaStream_t s) {
  if (n <= kSmall) {
    if (n <= 2 * kSmallThreads) launch_small_unique<2>(words, n, nib, unique_out, result, done, s);
    else if (n <= 4 * kSmallThreads) launch_small_unique<4>(words, n, nib, unique_out, result, done, s);
    else launch_small_unique<kSmall / kSmallThreads>(words, n, nib, unique_out, result, done, s);
    return cudaGetLastError();
  }
  const SortScratchLayout l = layout(scratch, n, true);
  cudaError_t e;
  if ((e = cudaMemsetAsync(l.control, 0, sizeof(Control), s)) != cudaSuccess) return e;
  const int tiles = tiles_of(n, kTile);
  if ((e = launch_compact(persistent_grid<compact_kernel<true>>(tiles), words, n, nib, l, unique_out, result, s)) !=
      cudaSuccess)
    return e;
  const uint32_t* keys = l.keys_a;
  Control* control = l.control;
  Plan* plan = l.plan;
  uint32_t* bitmap = l.bitmap;
  {
    const int grid =
        persistent_grid<direct_bitmap_kernel>(1 << 30, kShareThreads, kDirectSliceWords * 4);
    DoneFlag d = n <= kDirectWords ? done : DoneFlag{};
    void* args[] = {&keys, &control, &plan, &bitmap, &unique_out, &result, &err, &d};
    e = cudaLaunchCooperativeKernel(reinterpret_cast<void*>(direct_bitmap_kernel), dim3(grid),
                                    dim3(kShareThreads), args, kDirectSliceWords * 4, s);
    if (e != cudaSuccess || n <= kDirectWords) return e;
  }
  const uint32_t* sorted = l.keys_b;
  const Control* counts = l.control;
  const Plan* chosen = l.plan;
  if ((e = launch_behind<range_hist_kernel>(tiles, kThreads, 0, s, keys, control, plan)) != cudaSuccess) return e;
  if ((e = launch_behind<range_partition_kernel>(tiles, kThreads, 0, s, keys, l.keys_b, counts, plan)) != cudaSuccess)
    return e;
  if ((e = launch_behind<bucket_bitmap_kernel>(tiles, kThreads, 0, s, sorted, control, chosen, bitmap)) != cudaSuccess)
    return e;
  const int grid = persistent_grid<emit_kernel>(tiles_of(n, kShareThreads), kShareThreads, kEmitSmemBytes);
  DoneFlag d = done;
  void* args[] = {&bitmap, &control, &plan, &unique_out, &result, &err, &d};
  return cudaLaunchCooperativeKernel(reinterpret_cast<void*>(emit_kernel), dim3(grid),
                                     dim3(kShareThreads), args, kEmitSmemBytes, s);
}

bool feedback_unique_needs_radix(const int* result) {
  return __atomic_load_n(result + 1, __ATOMIC_ACQUIRE) == kPathRadix;
}

cudaError_t feedback_unique_radix_device(int n, int32_t* unique_out, void* scratch, unsigned long long* status,
                                         uint32_t epoch, int* result, int* err, const DoneFlag& done,
                                         cudaStream_t s) {
  const SortScratchLayout l = layout(scratch, n, true);
  cudaError_t e;
  if ((e = launch_digit_hist(l.keys_a, n, &l.control->keys, 0u, false, 0, l, s)) != cudaSuccess) return e;
  const DigitBuffers bufs = {l.keys_a, l.keys_a, l.keys_b, nullptr};
  if ((e = launch_digits(bufs, n, &l.control->keys, false, l, status, epoch, err, DoneFlag{}, s)) != cudaSuccess)
    return e;
  const uint32_t *keys_a = l.keys_a, *keys_b = l.keys_b;
  const Plan* plan = l.plan;
  return launch_behind<unique_kernel>(tiles_of(n, kTile), kThreads, 0, s, keys_a, keys_b, l.control, plan, unique_out,
                                      status, result, epoch * 8u + 4u, err, done);
}

bool sort_needs_passes(const int* again) { return *again != 0; }

cudaError_t sort_i32_device(int32_t* data, int n, void* scratch, unsigned long long* status, uint32_t epoch,
                            int* again, int* err, const DoneFlag& done, cudaStream_t s) {
  if (n <= 1) return cudaSuccess;
  if (n <= kSmall) {
    if (n <= 2 * kSmallThreads) launch_small_sort<2>(data, n, done, s);
    else if (n <= 4 * kSmallThreads) launch_small_sort<4>(data, n, done, s);
    else launch_small_sort<kSmall / kSmallThreads>(data, n, done, s);
    return cudaGetLastError();
  }
  const SortScratchLayout l = layout(scratch, n);
  const SplitShape shape = split_shape(n, l);
  cudaError_t e;
  if ((e = cudaMemsetAsync(l.control, 0, sizeof(Control), s)) != cudaSuccess) return e;
  uint32_t* keys = reinterpret_cast<uint32_t*>(data);
  if ((e = launch_digit_hist(keys, n, nullptr, 0x80000000u, true, shape.ranges, l, s)) != cudaSuccess) return e;
  if (shape.ranges) return launch_split(keys, n, shape, l, again, done, s);
  return sort_passes_device(data, n, scratch, status, epoch, err, done, s);
}

cudaError_t sort_passes_device(int32_t* data, int n, void* scratch, unsigned long long* status, uint32_t epoch,
                               int* err, const DoneFlag& done, cudaStream_t s) {
  const SortScratchLayout l = layout(scratch, n);
  uint32_t* keys = reinterpret_cast<uint32_t*>(data);
  DigitBuffers bufs = {keys, keys, l.keys_a, l.keys_b};
  if (reinterpret_cast<uintptr_t>(data) & 15) {  // the passes read a copy (keys_b is written by the second pass)
    copy_keys_kernel<<<persistent_grid<copy_keys_kernel>(tiles_of(n, kTile)), kThreads, 0, s>>>(keys, l.keys_b, n);
    const cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return e;
    bufs.in0 = l.keys_b;
  }
  return launch_digits(bufs, n, nullptr, true, l, status, epoch, err, done, s);
}

cudaError_t scan_i32_device(int32_t* data, int n, unsigned long long* status, uint32_t epoch, int* err,
                            const DoneFlag& done, cudaStream_t s) {
  if (n <= 0) return cudaSuccess;
  const int end = n + (int)((reinterpret_cast<uintptr_t>(data) >> 2) & 3u);
  // rows per warp: a full tile per CTA, or what spreads the array over every SM
  const int sms = persistent_grid<scan_kernel>(1 << 30, kScanBlock, kScanSmemBytes);
  constexpr int kRow = kScanWarps * 128;
  int rows = std::min(kScanRows, (int)(((long long)end + (long long)sms * kRow - 1) / ((long long)sms * kRow)));
  uint32_t tag = epoch * 8u + 6u;
  const int grid = std::min(sms, tiles_of(end, rows * kRow));
  if (grid == 1) {
    scan_kernel<<<1, kScanBlock, kScanSmemBytes, s>>>(data, n, rows, status, tag, err, done);
    return cudaGetLastError();
  }
  DoneFlag d = done;
  void* args[] = {&data, &n, &rows, &status, &tag, &err, &d};
  return cudaLaunchCooperativeKernel(reinterpret_cast<void*>(scan_kernel), dim3(grid), dim3(kScanBlock), args,
                                     kScanSmemBytes, s);
}

}  // namespace rayt
