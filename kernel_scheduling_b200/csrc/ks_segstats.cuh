// ks_segstats.cuh -- K4 core: per row (segment of the sorted sample stream) and per value lane, the exact integer
// statistics  sum, min, max and the two middle order statistics  lo = x[(n-1)/2], hi = x[n/2].
//
// A sample is a 16-byte item {sort key, lane 0, lane 1, lane 2}; every kernel loads an item once (one 128-bit load) and
// feeds all three lanes from it.  The stage entry point ks_segment_stats hands in a plain u32 array instead (one lane).
//
// Rows differ in size by six orders of magnitude (most key pairs meet a few times, the hottest pair owns percent of
// all samples), so size classes share the work.  In the table builds k_tile_stats (ks_tilestats.cuh) finishes the rows of up
// to 512 samples; in the stage entry point ks_segment_stats k_seg_classify (1..4 samples), k_seg_small (5..32) and k_seg_mid
// (33..512) do.  Longer rows, in both:
//
//   513 .. 2048   k_seg_lanes: one warp per row and value lane, the values in registers (64 per thread), no barrier anywhere
//                 (table builds; the stage entry point leaves them to k_seg_big).
//   .. 8192       k_seg_big: one CTA per row, staged once in 96 KB of shared memory, the values of one lane at a time in
//                 registers (32 per thread), one barrier per probe.
//   above         k_segL_sample / k_segL_pass / k_segL_finish.  1,024 values of the row (8,192 of a row of 2^17 or more),
//                 one from a hashed place in every 1,024th (8,192nd) of it, give two pivots that enclose the middle ranks
//                 with 5.5 standard deviations to spare; ONE pass over the row (chunks of 4,096 samples that any CTA may
//                 take) adds up sum / min / max, counts the values below, at and above the pivots and collects those
//                 strictly between them (a sixth of the row; a sixteenth); one CTA per row and lane finds the ranks among the
//                 collected values, narrowing them the same way while they are more than 8,192.  A row of 2^19 or more that
//                 collected more than kNarrowMin is narrowed over many CTAs first: the CTA that does the last chunk of its
//                 pass places two more pivots, and k_segL_finish begins with a pass over the collected values.  If the
//                 pivots missed (or the collected values did not fit their quarter of the row), one CTA searches the whole
//                 row instead: slow, and exact.
//
// All of them but the shortest classes find a middle value by COUNTING (narrow_to_rank): false position on the number of
// values below a pivot, which for the durations of one kernel takes 3 to 6 probes of two instructions per 32 samples and
// a reduction; radix selection over shared-memory histograms took two to three rounds of about ten instructions each.
//
// On 84 M samples of a c3 trace (47 M of them in rows above 512): k_seg_lanes 0.17 ms, k_seg_big 0.18 ms, the three kernels of
// the large rows 0.02 + 0.13 + 0.06 ms; all samples of such rows read once at the measured copy rate would take 0.12 ms.
//
// No kernel waits on another CTA.
#pragma once

#include "ks_common.cuh"
#include "ks_strided.h"

namespace ks {

constexpr int kLanes = 3;
constexpr uint32_t kTinyRow = 4;       // rows of up to this many samples carry no RowStats after k_tile_stats (see tiny_row_stats)
constexpr uint32_t kMidMax = 512;      // largest row the warp-per-row kernel takes
constexpr uint32_t kBigMax = 8192;     // largest row the CTA-per-row kernel takes
constexpr uint32_t kLargeChunk = 4096; // samples per work item of a large row
// The pivots of n values are two of a sample's, as many ranks below and above the wanted one as 5.5 standard deviations of a
// rank are (5.5 x sqrt(sample) / 2).  A warp draws 1,024, a whole CTA 8,192: twice the samples' cache lines and block-wide
// instead of warp-wide steps, for a third of the values in between.
constexpr uint32_t kLargeSample = 1024, kLargeSpread = 88;
constexpr uint32_t kWideSample = 8192, kWideSpread = 249;
constexpr uint32_t kWideMin = 1u << 17;    // rows of at least this many samples get the wide sample
// A single CTA narrows about 1,400 values per us: a row of 100 M values, whose sixteenth is 6 M, would keep it at work for
// milliseconds while the chip idles.  Collected values of a row and lane above which many CTAs narrow them, and the shortest
// rows for which that is looked at (a sixteenth of them is as many).
constexpr uint32_t kNarrowMin = 1u << 15, kNarrowRow = 1u << 19;

struct RowStats {
  unsigned long long sum[kLanes];
  uint32_t mn[kLanes], mx[kLanes], lo[kLanes], hi[kLanes];
};

// accumulators of one large row
struct LargeRow {
  uint32_t row, start, cnt, pad;
  unsigned long long sum[kLanes];
  uint32_t mn[kLanes], mx[kLanes];
  uint32_t p1[kLanes], p2[kLanes];  // pivots, p1 <= p2
  uint32_t lt[kLanes], e1[kLanes];  // values below p1, equal to p1
  uint32_t e2[kLanes];              // values equal to p2 (0 if p1 == p2)
  uint32_t n_mid[kLanes];           // values strictly between: in the row's part of SegArgs::cand unless they are too many
  // the same once more among those: pivots, counts, and whether it was done
  uint32_t q1[kLanes], q2[kLanes], q_lt[kLanes], q_e1[kLanes], q_e2[kLanes], q_mid[kLanes];
  uint32_t done, q_done[kLanes];  // chunks of the two passes that are done
  bool narrowed[kLanes];
};
__device__ __forceinline__ void large_row_init(LargeRow* L, uint32_t row, uint32_t start, uint32_t cnt) {
  L->row = row; L->start = start; L->cnt = cnt;
  for (int l = 0; l < kLanes; ++l) { L->sum[l] = 0; L->mn[l] = 0xFFFFFFFFu; L->mx[l] = 0; L->lt[l] = L->e1[l] = L->e2[l] = L->n_mid[l] = 0; L->q_done[l] = 0; L->narrowed[l] = false; }
  L->done = 0;
}

struct SegArgs {
  const uint4* items;      // 16-byte samples (lanes = .y .z .w), or nullptr:
  const uint32_t* plain;   // one lane of plain u32 values
  int n_lanes;             // 3 with items, 1 with plain
  const uint32_t* row_start;
  const uint32_t* row_cnt;   // samples per row, or nullptr: the rows lie one behind the other, a row ends where the next starts
  const uint32_t* n_rows_dev;
  uint32_t max_rows;
  RowStats* stats;
  uint32_t* small_rows;    // [max_rows] rows of 9..32 samples
  uint32_t* small8_rows;   // [max_rows] rows of 5..8 samples
  uint32_t* mid_rows;      // [max_rows]
  uint32_t* big_rows;      // [max_rows] rows of kMidMax+1 .. kBigMax samples
  LargeRow* large;         // [max_large]
  uint32_t* chunk_row;     // [max_chunks] index into large[]
  uint32_t* chunk_idx;     // [max_chunks] chunk number inside the row
  // scratch of the large rows: per lane cand_words words; a row owns a quarter as many as it has samples, and a sixteenth
  // behind all the quarters (for the second narrowing)
  uint32_t* cand;          // [n_lanes][cand_words]
  size_t cand_words;       // n / 4 + n / 16 + 4
  size_t cand_second;      // where the sixteenths begin
  uint32_t* chunk2_job;    // [max_chunks2] chunks of the second narrowing: index into large[] * n_lanes + lane ...
  uint32_t* chunk2_idx;    // ... and chunk number inside the collected values
  uint32_t max_large, max_chunks, max_chunks2;
  Control* ctl;            // pad32 / n_small / n_big = rows of 5..8 / 9..32 / mid rows, low word of pad2[1] = big rows,
                           // ticket = large rows, scratch0 = chunks, chunks2 = chunks of the second narrowing
};

__device__ __forceinline__ uint32_t* big_row_counter(Control* ctl) { return reinterpret_cast<uint32_t*>(&ctl->pad2[1]); }

// Registers a row of more than kBigMax samples and its chunks.  A table that the host throws away (a guessed key count was too
// small, so its samples were not sorted) can have rows whose ends were taken for those of later rows: more chunks than there is room
// for.  Every row below the ticket and every chunk below the counter is written all the same -- a row that does not fit gets no
// samples, its chunks are skipped.
constexpr uint32_t kNoRow = 0xFFFFFFFFu;
__device__ __forceinline__ void register_large_row(const SegArgs& a, uint32_t row, uint32_t start, uint32_t cnt) {
  const uint32_t nch = chunk_count(cnt, kLargeChunk);
  const uint32_t l = atomicAdd(&a.ctl->ticket, 1u);
  const unsigned long long base = atomicAdd(&a.ctl->scratch0, (unsigned long long)nch);  // (64 bits: the chunks of such rows may be many)
  const bool fits = l < a.max_large && base + nch <= a.max_chunks;
  if (!fits) atomicOr(&a.ctl->err, kErrTooLarge);
  if (l < a.max_large) large_row_init(a.large + l, row, start, fits ? cnt : 0u);
  for (uint32_t c = 0; c < nch && base + c < a.max_chunks; ++c) { a.chunk_row[base + c] = fits ? l : kNoRow; a.chunk_idx[base + c] = c; }
}

struct Val3 {
  uint32_t v[kLanes];
};

__device__ __forceinline__ Val3 seg_fetch(const SegArgs& a, size_t i) {
  Val3 r;
  if (a.items) {
    const uint4 it = a.items[i];
    r.v[0] = it.y; r.v[1] = it.z; r.v[2] = it.w;
  } else {
    r.v[0] = a.plain[i]; r.v[1] = 0; r.v[2] = 0;
  }
  return r;
}

// ---------------------------------------------------------------------------------------------------------
// The value of rank k by counting.  [L, H] always encloses it: c_lo = values below L <= k < c_hi = values up to H.  A probe p
// in (L, H] moves one end; the next one is placed by false position on the counts, an end that stays twice loses half its
// weight (the Illinois rule), and after kFalsePos probes plain bisection takes over, so any distribution ends within
// kFalsePos + 32 probes.  It stops when the rank is the smallest value of the bracket (c_lo == k), its largest (c_hi == k +
// 1) or the bracket holds a single value.  count_below(p) is the number of values < p and must be the same in every thread;
// values are compared only, so the result is exact whatever the pivots are.
constexpr int kFalsePos = 12;
struct Bracket {
  uint32_t L, H, c_lo, c_hi;
};
// mn is the smallest value, or below_mn (at most k) values lie below it.
template <class CountBelow>
__device__ __forceinline__ Bracket narrow_to_rank(uint32_t k, uint32_t cnt, uint32_t mn, uint32_t mx, uint32_t guess, CountBelow count_below, uint32_t below_mn = 0u) {
  Bracket b{mn, mx, below_mn, cnt};
  float w_lo = (float)(k - below_mn) + 0.5f, w_hi = (float)(cnt - k) - 0.5f;  // distance of rank k + 1/2 from the counts at the ends, weighted
  bool low_moved = false, high_moved = false;
  uint32_t p = guess;
  for (int probe = 1; b.c_lo != k && b.c_hi != k + 1 && b.L != b.H; ++probe) {
    p = min(max(p, b.L + 1), b.H);
    const uint32_t c = count_below(p);
    if (c <= k) {
      b.L = p; b.c_lo = c;
      w_lo = (float)(k - c) + 0.5f;
      if (low_moved) w_hi *= 0.5f;
      low_moved = true; high_moved = false;
    } else {
      b.H = p - 1; b.c_hi = c;
      w_hi = (float)(c - k) - 0.5f;
      if (high_moved) w_lo *= 0.5f;
      high_moved = true; low_moved = false;
    }
    const uint32_t width = b.H - b.L;
    p = b.L + (probe >= kFalsePos ? (width >> 1) + (width & 1u) : (uint32_t)((float)width * __fdividef(w_lo, w_lo + w_hi)));
  }
  return b;
}

// One warp, up to 32 * R values in registers (positions behind the cnt values: 0xFFFFFFFF): the value of rank k.
template <int R>
__device__ __forceinline__ uint32_t warp_rank(const uint32_t (&x)[R], uint32_t cnt, uint32_t mn, uint32_t mx, uint32_t guess, uint32_t k, uint32_t below_mn = 0u) {
  const Bracket b = narrow_to_rank(k, cnt, mn, mx, guess, [&](uint32_t p) {
    uint32_t c = 0;
#pragma unroll
    for (int i = 0; i < R; ++i) c += x[i] < p ? 1u : 0u;
    return warp_sum(c);
  }, below_mn);
  uint32_t v = b.L;
  if (b.c_lo == k) {  // the smallest value at or above L
    v = 0xFFFFFFFFu;
#pragma unroll
    for (int i = 0; i < R; ++i) v = x[i] >= b.L ? min(v, x[i]) : v;
    v = warp_min(v);
  } else if (b.c_hi == k + 1) {  // the largest up to H (H is below the padding here: some value lies above it)
    v = 0;
#pragma unroll
    for (int i = 0; i < R; ++i) v = x[i] <= b.H ? max(v, x[i]) : v;
    v = warp_max(v);
  }
  return v;
}
// ... and the two middle values
template <int R>
__device__ __forceinline__ void warp_middle(const uint32_t (&x)[R], uint32_t cnt, uint32_t mn, uint32_t mx, unsigned long long sum, uint32_t* lo, uint32_t* hi) {
  const uint32_t k = (cnt - 1) >> 1;
  const uint32_t v = warp_rank<R>(x, cnt, mn, mx, (uint32_t)__fdividef((float)sum, (float)cnt), k);
  *lo = *hi = v;
  if (!(cnt & 1u)) {  // rank k + 1: the same value again if more than k + 1 values are at or below it, else the next larger one
    uint32_t le = 0, next = 0xFFFFFFFFu;
#pragma unroll
    for (int i = 0; i < R; ++i) {
      le += x[i] <= v ? 1u : 0u;
      next = x[i] > v ? min(next, x[i]) : next;
    }
    le = warp_sum(le);
    next = warp_min(next);
    *hi = le > k + 1 ? v : next;
  }
}

// A CTA of kBigThreads threads: block-wide sum / min / max, one barrier each (two sets of partials taken in turns: a set is
// written again only behind the barrier of the other one).
constexpr int kBigThreads = 256;
struct CtaReduce {
  uint32_t (*part)[kBigThreads / 32];  // [2][warps], shared memory
  uint32_t turn;
  template <class Op>
  __device__ __forceinline__ uint32_t run(uint32_t v, uint32_t empty, Op op) {
    v = op(v);
    if (lane_id() == 0) part[turn][threadIdx.x >> 5] = v;
    __syncthreads();
    v = op(lane_id() < kBigThreads / 32 ? part[turn][lane_id()] : empty);
    turn ^= 1u;
    return v;
  }
  __device__ __forceinline__ uint32_t sum(uint32_t v) { return run(v, 0u, [](uint32_t t) { return warp_sum(t); }); }
  __device__ __forceinline__ uint32_t min_of(uint32_t v) { return run(v, 0xFFFFFFFFu, [](uint32_t t) { return warp_min(t); }); }
  __device__ __forceinline__ uint32_t max_of(uint32_t v) { return run(v, 0u, [](uint32_t t) { return warp_max(t); }); }
};
// The value of rank k and, if want_next, of rank k + 1 among cnt values that the CTA's threads visit: each(f) calls f(x) for
// every value of the thread (and may also call it for padding 0xFFFFFFFF).
template <class Each>
__device__ __forceinline__ void cta_ranks(CtaReduce& red, uint32_t cnt, uint32_t mn, uint32_t mx, uint32_t guess, uint32_t k, bool want_next, Each each, uint32_t* lo, uint32_t* hi) {
  const Bracket b = narrow_to_rank(k, cnt, mn, mx, guess, [&](uint32_t p) {
    uint32_t c = 0;
    each([&](uint32_t x) { c += x < p ? 1u : 0u; });
    return red.sum(c);
  });
  uint32_t v = b.L;
  if (b.c_lo == k) {
    uint32_t t = 0xFFFFFFFFu;
    each([&](uint32_t x) { t = x >= b.L ? min(t, x) : t; });
    v = red.min_of(t);
  } else if (b.c_hi == k + 1) {
    uint32_t t = 0;
    each([&](uint32_t x) { t = x <= b.H ? max(t, x) : t; });
    v = red.max_of(t);
  }
  *lo = *hi = v;
  if (want_next) {
    uint32_t le = 0, next = 0xFFFFFFFFu;
    each([&](uint32_t x) { le += x <= v ? 1u : 0u; next = x > v ? min(next, x) : next; });
    le = red.sum(le);
    next = red.min_of(next);
    *hi = le > k + 1 ? v : next;
  }
}

// The statistics of a row of 1..kTinyRow samples straight from its samples: a five-comparator network per value lane.
__device__ __forceinline__ void tiny_row_stats(const uint4* items, uint32_t cnt, RowStats* st) {
  uint32_t x[kTinyRow][kLanes];
#pragma unroll
  for (uint32_t i = 0; i < kTinyRow; ++i) {
    uint4 it = make_uint4(0, 0xFFFFFFFFu, 0xFFFFFFFFu, 0xFFFFFFFFu);
    if (i < cnt) it = items[i];
    x[i][0] = it.y; x[i][1] = it.z; x[i][2] = it.w;
  }
#pragma unroll
  for (int l = 0; l < kLanes; ++l) {
    uint32_t x0 = x[0][l], x1 = x[1][l], x2 = x[2][l], x3 = x[3][l];
    st->sum[l] = (unsigned long long)x0 + (cnt > 1 ? x1 : 0u) + (cnt > 2 ? x2 : 0u) + (cnt > 3 ? x3 : 0u);
    uint32_t t;
#define KS_CSWAP(p, q) t = min(p, q); q = max(p, q); p = t;
    KS_CSWAP(x0, x1) KS_CSWAP(x2, x3) KS_CSWAP(x0, x2) KS_CSWAP(x1, x3) KS_CSWAP(x1, x2)
#undef KS_CSWAP
    auto pick = [&](uint32_t i) { return i == 0 ? x0 : i == 1 ? x1 : i == 2 ? x2 : x3; };
    st->mn[l] = x0;
    st->mx[l] = pick(cnt - 1);
    st->lo[l] = pick((cnt - 1) >> 1);
    st->hi[l] = pick(cnt >> 1);
  }
}

// The statistics of row `row` of a sorted sample stream after k_tile_stats and the kernels of the longer rows.
__device__ __forceinline__ RowStats table_row_stats(const RowStats* stats, const uint32_t* row_start, const uint32_t* row_cnt, const uint4* items, uint32_t n_items, uint32_t row) {
  const uint32_t s = row_start[row], cnt = row_cnt[row];
  if (cnt - 1 >= kTinyRow || s > n_items || cnt > n_items - s) return stats[row];  // the bounds: row offsets of a table the host throws away
  RowStats st;
  tiny_row_stats(items + s, cnt, &st);
  return st;
}

__device__ __forceinline__ int bit_length32(uint32_t v) { return 32 - __clz(v); }

// true if u agrees with prefix on all bits above hi_bit
__device__ __forceinline__ bool matches_prefix(uint32_t u, uint32_t prefix, int hi_bit) {
  return hi_bit >= 31 || (u >> (hi_bit + 1)) == (prefix >> (hi_bit + 1));
}

// One warp, 256 bins in shared memory (8 consecutive bins per lane): the bin that holds rank k and the count below it.
__device__ __forceinline__ void warp_pick_bin(const uint32_t* bins, uint32_t k, uint32_t* digit, uint32_t* below) {
  const uint32_t lane = lane_id();
  uint32_t c[8], tot = 0;
#pragma unroll
  for (int i = 0; i < 8; ++i) { c[i] = bins[lane * 8 + i]; tot += c[i]; }
  const uint32_t inc = warp_incl_scan(tot);
  const uint32_t exc = inc - tot;
  const bool mine = k >= exc && k < inc;
  uint32_t d = 0, b = 0;
  if (mine) {
    uint32_t acc = exc;
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      if (k >= acc && k < acc + c[i]) { d = lane * 8 + i; b = acc; }
      acc += c[i];
    }
  }
  const uint32_t who = __ffs(__ballot_sync(0xFFFFFFFFu, mine)) - 1;
  *digit = __shfl_sync(0xFFFFFFFFu, d, who & 31u);
  *below = __shfl_sync(0xFFFFFFFFu, b, who & 31u);
}

// ---------------------------------------------------------------------------------------------------------
// One thread per row.  Rows of up to four samples are finished right here with a five-comparator sorting network in
// registers; the others go to the work list of their size class.
__device__ __forceinline__ void push_row(uint32_t* list, uint32_t* counter, bool mine, uint32_t row) {
  const uint32_t ballot = __ballot_sync(__activemask(), mine);
  if (!mine) return;
  const uint32_t first = __ffs(ballot) - 1;
  uint32_t base = 0;
  if (lane_id() == first) base = atomicAdd(counter, (uint32_t)__popc(ballot));
  base = __shfl_sync(ballot, base, first);
  list[base + __popc(ballot & lanemask_lt())] = row;
}

// The large rows (more than kBigMax samples) are found by a kernel of their own, so that their chain of launches can
// start while k_seg_classify and the other classes are still at work on other streams: one thread per row registers the
// row and its chunks.
__global__ void __launch_bounds__(256) k_seg_find_large(const SegArgs a) {
  const uint32_t n_rows = min(*a.n_rows_dev, a.max_rows);
  for (uint32_t row = blockIdx.x * blockDim.x + threadIdx.x; row < n_rows; row += gridDim.x * blockDim.x) {
    const uint32_t s = a.row_start[row], cnt = a.row_start[row + 1] - s;
    if (cnt <= kBigMax) continue;
    register_large_row(a, row, s, cnt);
  }
}

__global__ void __launch_bounds__(256) k_seg_classify(const SegArgs a) {
  // the statistics of 256 consecutive rows are 18 KB of consecutive memory: staged here, written with coalesced stores
  constexpr int kWords = sizeof(RowStats) / 4;
  __shared__ uint32_t stage[256 * kWords];
  const uint32_t n_rows = min(*a.n_rows_dev, a.max_rows);
  const uint32_t n_round = (n_rows + 255u) & ~255u;  // whole CTAs take part in the staging and the list pushes
  for (uint32_t row0 = blockIdx.x * blockDim.x; row0 < n_round; row0 += gridDim.x * blockDim.x) {
    const uint32_t row = row0 + threadIdx.x;
    const bool valid = row < n_rows;
    const uint32_t s = valid ? a.row_start[row] : 0, cnt = valid ? a.row_start[row + 1] - s : 0;
    push_row(a.small8_rows, &a.ctl->pad32, valid && cnt > 4 && cnt <= 8, row);
    push_row(a.small_rows, &a.ctl->n_small, valid && cnt > 8 && cnt <= kSmallSegment, row);
    push_row(a.mid_rows, &a.ctl->n_big, valid && cnt > kSmallSegment && cnt <= kMidMax, row);
    push_row(a.big_rows, big_row_counter(a.ctl), valid && cnt > kMidMax && cnt <= kBigMax, row);
    RowStats st;
#pragma unroll
    for (int l = 0; l < kLanes; ++l) { st.sum[l] = 0; st.mn[l] = 0; st.mx[l] = 0; st.lo[l] = 0; st.hi[l] = 0; }
    // empty rows (stage API only) and tiny rows are finished here
    if (valid && cnt > 0 && cnt <= 4) {
      Val3 x[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        if ((uint32_t)i < cnt) x[i] = seg_fetch(a, (size_t)s + i);
        else { x[i].v[0] = x[i].v[1] = x[i].v[2] = 0xFFFFFFFFu; }
      }
      const uint32_t i_max = cnt - 1, i_lo = (cnt - 1) >> 1, i_hi = cnt >> 1;
#pragma unroll
      for (int l = 0; l < kLanes; ++l) {
        uint32_t x0 = x[0].v[l], x1 = x[1].v[l], x2 = x[2].v[l], x3 = x[3].v[l];
        const unsigned long long sum = (unsigned long long)x0 + (cnt > 1 ? x1 : 0u) + (cnt > 2 ? x2 : 0u) + (cnt > 3 ? x3 : 0u);
        uint32_t t;
#define KS_CSWAP(p, q) t = min(p, q); q = max(p, q); p = t;
        KS_CSWAP(x0, x1) KS_CSWAP(x2, x3) KS_CSWAP(x0, x2) KS_CSWAP(x1, x3) KS_CSWAP(x1, x2)
#undef KS_CSWAP
        auto pick = [&](uint32_t i) { return i == 0 ? x0 : i == 1 ? x1 : i == 2 ? x2 : x3; };
        st.sum[l] = sum;
        st.mn[l] = x0;
        st.mx[l] = pick(i_max);
        st.lo[l] = pick(i_lo);
        st.hi[l] = pick(i_hi);
      }
    }
    // rows of the other classes get zeros now and their statistics from the class kernels, which run after this one
    __syncthreads();
    const uint32_t* w = reinterpret_cast<const uint32_t*>(&st);
#pragma unroll
    for (int i = 0; i < kWords; ++i) stage[threadIdx.x * kWords + i] = w[i];
    __syncthreads();
    const uint32_t rows_here = min(256u, n_rows > row0 ? n_rows - row0 : 0u);
    uint32_t* dst = reinterpret_cast<uint32_t*>(a.stats + row0);
    for (uint32_t i = threadIdx.x; i < rows_here * kWords; i += blockDim.x) dst[i] = stage[i];
  }
}

// W lanes per row (W = 8 for rows of 5..8 samples, 32 for 9..32): a warp takes 32 / W rows at a time; shuffle
// reductions and a W-wide bitonic network inside each group
template <int W>
__device__ __forceinline__ uint32_t bitonic_sort_group(uint32_t v) {
  const uint32_t sub = lane_id() & (W - 1);
#pragma unroll
  for (int k = 2; k <= W; k <<= 1) {
#pragma unroll
    for (int j = k >> 1; j > 0; j >>= 1) {
      const uint32_t o = __shfl_xor_sync(0xFFFFFFFFu, v, j);
      const bool up = (sub & k) == 0;
      const bool lower = (sub & j) == 0;
      v = (lower == up) ? min(v, o) : max(v, o);
    }
  }
  return v;
}

template <int W>
__global__ void __launch_bounds__(256) k_seg_small(const SegArgs a) {
  constexpr uint32_t G = 32 / W;
  const uint32_t* list = W == 8 ? a.small8_rows : a.small_rows;
  const uint32_t n_list = min(W == 8 ? a.ctl->pad32 : a.ctl->n_small, a.max_rows);
  const uint32_t lane = lane_id(), sub = lane & (W - 1), gbase = lane & ~(uint32_t)(W - 1);
  const uint32_t warps = gridDim.x * (blockDim.x >> 5);
  const uint32_t n_round = (n_list + G - 1) / G * G;
  for (uint32_t t0 = (blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5)) * G; t0 < n_round; t0 += warps * G) {
    const uint32_t t = t0 + lane / W;
    const bool valid = t < n_list;
    const uint32_t row = valid ? list[t] : 0;
    const uint32_t s = valid ? a.row_start[row] : 0, cnt = valid ? a.row_start[row + 1] - s : 1;
    const bool have = valid && sub < cnt;
    Val3 x;
    if (have) x = seg_fetch(a, (size_t)s + sub);
    else { x.v[0] = x.v[1] = x.v[2] = 0; }
    RowStats* st = a.stats + row;
#pragma unroll
    for (int l = 0; l < kLanes; ++l) {
      if (l >= a.n_lanes) break;
      const uint32_t v = x.v[l];
      unsigned long long sum = v;
#pragma unroll
      for (int o = W / 2; o; o >>= 1) sum += __shfl_xor_sync(0xFFFFFFFFu, sum, o);
      const uint32_t sorted = bitonic_sort_group<W>(have ? v : 0xFFFFFFFFu);
      const uint32_t mn = __shfl_sync(0xFFFFFFFFu, sorted, gbase);
      const uint32_t mx = __shfl_sync(0xFFFFFFFFu, sorted, gbase + cnt - 1);
      const uint32_t lo = __shfl_sync(0xFFFFFFFFu, sorted, gbase + ((cnt - 1) >> 1));
      const uint32_t hi = __shfl_sync(0xFFFFFFFFu, sorted, gbase + (cnt >> 1));
      if (valid && sub == 0) { st->sum[l] = sum; st->mn[l] = mn; st->mx[l] = mx; st->lo[l] = lo; st->hi[l] = hi; }
    }
  }
}

// ---------------------------------------------------------------------------------------------------------
// One warp per row of 33..kMidMax samples.  The row is read from global memory ONCE: its three value lanes are staged in
// the warp's own shared memory while sum/min/max are taken, and the selection rounds (and the pass for the upper middle
// value) run over shared memory.  No block-wide barrier anywhere.
constexpr int kMidWarps = 8;
constexpr size_t seg_mid_smem_bytes() { return (size_t)kMidWarps * kLanes * (kMidMax + 256) * sizeof(uint32_t); }

__global__ void __launch_bounds__(kMidWarps * 32, 3) k_seg_mid(const SegArgs a) {
  extern __shared__ __align__(16) uint32_t mid_smem[];
  const uint32_t warp = threadIdx.x >> 5, lane = lane_id();
  uint32_t* vals = mid_smem + (size_t)warp * kLanes * (kMidMax + 256);  // [kLanes][kMidMax]
  uint32_t* hist = vals + kLanes * kMidMax;                              // [kLanes][256]
  const uint32_t n_mid = min(a.ctl->n_big, a.max_rows);
  const uint32_t warps = gridDim.x * kMidWarps;
  const int nl = a.n_lanes;
  for (uint32_t t = blockIdx.x * kMidWarps + warp; t < n_mid; t += warps) {
    const uint32_t row = a.mid_rows[t];
    const uint32_t s = a.row_start[row], cnt = min(a.row_start[row + 1] - s, kMidMax);
    unsigned long long sum[kLanes] = {0, 0, 0};
    uint32_t mn[kLanes] = {0xFFFFFFFFu, 0xFFFFFFFFu, 0xFFFFFFFFu}, mx[kLanes] = {0, 0, 0};
    __syncwarp();  // the previous row's readers of the staging area are done
    for (uint32_t i0 = lane; i0 < cnt; i0 += 128) {
      Val3 xs[4];
#pragma unroll
      for (int u = 0; u < 4; ++u) if (i0 + 32 * u < cnt) xs[u] = seg_fetch(a, (size_t)s + i0 + 32 * u);
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        if (i0 + 32 * u >= cnt) break;
#pragma unroll
        for (int l = 0; l < kLanes; ++l) {
          const uint32_t v = xs[u].v[l];
          vals[l * kMidMax + i0 + 32 * u] = v;
          sum[l] += v; mn[l] = min(mn[l], v); mx[l] = max(mx[l], v);
        }
      }
    }
#pragma unroll
    for (int l = 0; l < kLanes; ++l) { sum[l] = warp_sum64(sum[l]); mn[l] = warp_min(mn[l]); mx[l] = warp_max(mx[l]); }
    __syncwarp();

    const uint32_t k_lo = (cnt - 1) >> 1, k_hi = cnt >> 1;
    uint32_t prefix[kLanes] = {0, 0, 0}, k[kLanes] = {k_lo, k_lo, k_lo};
    int hi_bit[kLanes];
    bool open = false;
#pragma unroll
    for (int l = 0; l < kLanes; ++l) {
      hi_bit[l] = (l < nl && mn[l] != mx[l]) ? bit_length32(mx[l] - mn[l]) - 1 : -1;
      open = open || hi_bit[l] >= 0;
    }
    while (open) {
      int nb[kLanes], shift[kLanes];
#pragma unroll
      for (int l = 0; l < kLanes; ++l) {
        nb[l] = min(8, hi_bit[l] + 1);
        shift[l] = hi_bit[l] + 1 - nb[l];
        if (hi_bit[l] >= 0) {
#pragma unroll
          for (int i = 0; i < 8; ++i) hist[l * 256 + lane * 8 + i] = 0;
        }
      }
      __syncwarp();
#pragma unroll
      for (int l = 0; l < kLanes; ++l) {
        if (hi_bit[l] < 0) continue;
        for (uint32_t i = lane; i < cnt; i += 32) {
          const uint32_t u = vals[l * kMidMax + i] - mn[l];
          if (matches_prefix(u, prefix[l], hi_bit[l])) atomicAdd(&hist[l * 256 + ((u >> shift[l]) & ((1u << nb[l]) - 1u))], 1u);
        }
      }
      __syncwarp();
      open = false;
#pragma unroll
      for (int l = 0; l < kLanes; ++l) {
        if (hi_bit[l] < 0) continue;
        uint32_t d, below;
        warp_pick_bin(hist + l * 256, k[l], &d, &below);
        prefix[l] |= d << shift[l];
        k[l] -= below;
        hi_bit[l] = shift[l] - 1;
        open = open || hi_bit[l] >= 0;
      }
      __syncwarp();
    }
    uint32_t lo[kLanes], hi[kLanes];
#pragma unroll
    for (int l = 0; l < kLanes; ++l) { lo[l] = mn[l] + prefix[l]; hi[l] = lo[l]; }
    if (k_hi != k_lo) {
      // hi = x[k_lo + 1]: lo again if more than k_hi values are <= lo, else the smallest value above lo
#pragma unroll
      for (int l = 0; l < kLanes; ++l) {
        if (l >= nl) continue;
        uint32_t le = 0, next = 0xFFFFFFFFu;
        for (uint32_t i = lane; i < cnt; i += 32) {
          const uint32_t v = vals[l * kMidMax + i];
          le += v <= lo[l];
          if (v > lo[l]) next = min(next, v);
        }
        const uint32_t le_t = warp_sum(le), nx = warp_min(next);
        hi[l] = (le_t > k_hi) ? lo[l] : nx;
      }
    }
    if (lane == 0) {
      RowStats* st = a.stats + row;
      for (int l = 0; l < nl; ++l) { st->sum[l] = sum[l]; st->mn[l] = mn[l]; st->mx[l] = mx[l]; st->lo[l] = lo[l]; st->hi[l] = hi[l]; }
    }
  }
}

// ---------------------------------------------------------------------------------------------------------
// One warp per row and value lane, rows of kMidMax+1 .. kLanesMax samples: 64 values per thread in registers.  The three
// warps of a row are neighbours, so the 128-byte lines of its samples come from L1 for two of them.
constexpr uint32_t kLanesMax = 2048;
__global__ void __launch_bounds__(256, 2) k_seg_lanes(const SegArgs a) {
  constexpr int R = kLanesMax / 32;
  const uint32_t lane = lane_id();
  const uint32_t n_jobs = kLanes * min(big_row_counter(a.ctl)[1], a.max_rows);
  for (uint32_t j = blockIdx.x * 8 + (threadIdx.x >> 5); j < n_jobs; j += gridDim.x * 8) {
    const uint32_t row = a.mid_rows[j / kLanes], l = j % kLanes;
    const uint32_t cnt = min(a.row_cnt[row], kLanesMax);
    const uint32_t* v = reinterpret_cast<const uint32_t*>(a.items + a.row_start[row]) + 1 + l;
    uint32_t x[R], mn = 0xFFFFFFFFu, mx = 0;
    unsigned long long sum = 0;
#pragma unroll
    for (int i = 0; i < R; ++i) x[i] = lane + 32 * i < cnt ? v[4 * (lane + 32 * i)] : 0xFFFFFFFFu;
#pragma unroll
    for (int i = 0; i < R; ++i) {
      const uint32_t z = lane + 32 * i < cnt ? x[i] : 0u;
      sum += z; mx = max(mx, z); mn = min(mn, x[i]);
    }
    sum = warp_sum48(sum);
    mn = warp_min(mn);
    mx = warp_max(mx);
    uint32_t lo, hi;
    warp_middle<R>(x, cnt, mn, mx, sum, &lo, &hi);
    if (lane == 0) {
      RowStats* st = a.stats + row;
      st->sum[l] = sum; st->mn[l] = mn; st->mx[l] = mx; st->lo[l] = lo; st->hi[l] = hi;
    }
  }
}

// one value lane of the samples: base and stride in words
__device__ __forceinline__ const uint32_t* seg_lane(const SegArgs& a, size_t first, int l, uint32_t* stride) {
  *stride = a.items ? 4u : 1u;
  return a.items ? reinterpret_cast<const uint32_t*>(a.items + first) + 1 + l : a.plain + first;
}
// all values v[i * stride], i < n, of a CTA of kBigThreads threads, four loads in flight per thread
template <class F>
__device__ __forceinline__ void each_of(const uint32_t* v, uint32_t stride, uint32_t n, F f) {
  strided(
      n, threadIdx.x, kBigThreads,
      [&](size_t i) {
        uint32_t x[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) x[u] = v[(i + kBigThreads * u) * stride];
#pragma unroll
        for (int u = 0; u < 4; ++u) f(x[u]);
      },
      [&](size_t i) { f(v[i * stride]); });
}

// One CTA per row of up to kBigMax samples: the row is read once and staged in the CTA's shared memory (96 KB) while sum / min
// / max are taken; then, one value lane after the other, 32 values per thread in registers and the search with block-wide
// counts.  The search state is computed by every thread alike from the shared counts.
constexpr size_t seg_big_smem_bytes() { return (size_t)kLanes * kBigMax * sizeof(uint32_t); }

struct BigShared {
  uint32_t part[2][kBigThreads / 32];
  unsigned long long sum[kBigThreads / 32][kLanes];
  uint32_t mn[kBigThreads / 32][kLanes], mx[kBigThreads / 32][kLanes];
  uint32_t pivot[2], queued;  // seg_long_lane
};
// One CTA, one row of cnt <= kBigMax samples from s on, staged in big_vals ([kLanes][kBigMax]).
__device__ __forceinline__ void seg_big_row(const SegArgs& a, uint32_t row, uint32_t s, uint32_t cnt, uint32_t* big_vals, BigShared& sh, CtaReduce& red) {
  constexpr int R = kBigMax / kBigThreads;
  const uint32_t tid = threadIdx.x, lane = lane_id(), warp = tid >> 5;
  unsigned long long sum[kLanes] = {0, 0, 0};
  uint32_t mn[kLanes] = {0xFFFFFFFFu, 0xFFFFFFFFu, 0xFFFFFFFFu}, mx[kLanes] = {0, 0, 0};
  __syncthreads();  // the previous row's readers of the shared arrays are done
  for (uint32_t i0 = tid; i0 < cnt; i0 += 4 * kBigThreads) {
    Val3 xs[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) if (i0 + kBigThreads * u < cnt) xs[u] = seg_fetch(a, (size_t)s + i0 + kBigThreads * u);
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      if (i0 + kBigThreads * u >= cnt) break;
#pragma unroll
      for (int l = 0; l < kLanes; ++l) {
        const uint32_t v = xs[u].v[l];
        big_vals[l * kBigMax + i0 + kBigThreads * u] = v;
        sum[l] += v; mn[l] = min(mn[l], v); mx[l] = max(mx[l], v);
      }
    }
  }
#pragma unroll
  for (int l = 0; l < kLanes; ++l) {
    const unsigned long long s2 = warp_sum48(sum[l]);
    const uint32_t n2 = warp_min(mn[l]), x2 = warp_max(mx[l]);
    if (lane == 0) { sh.sum[warp][l] = s2; sh.mn[warp][l] = n2; sh.mx[warp][l] = x2; }
  }
  __syncthreads();
  RowStats* st = a.stats + row;
#pragma unroll 1
  for (int l = 0; l < a.n_lanes; ++l) {
    unsigned long long sum_l = 0;
    uint32_t mn_l = 0xFFFFFFFFu, mx_l = 0, lo, hi;
    for (int w = 0; w < kBigThreads / 32; ++w) { sum_l += sh.sum[w][l]; mn_l = min(mn_l, sh.mn[w][l]); mx_l = max(mx_l, sh.mx[w][l]); }
    const uint32_t k = (cnt - 1) >> 1, mean = (uint32_t)__fdividef((float)sum_l, (float)cnt);
    uint32_t x[R];
#pragma unroll
    for (int i = 0; i < R; ++i) x[i] = tid + kBigThreads * i < cnt ? big_vals[l * kBigMax + tid + kBigThreads * i] : 0xFFFFFFFFu;
    cta_ranks(red, cnt, mn_l, mx_l, mean, k, !(cnt & 1u),
              [&](auto f) {
#pragma unroll
                for (int i = 0; i < R; ++i) f(x[i]);
              },
              &lo, &hi);
    if (tid == 0) { st->sum[l] = sum_l; st->mn[l] = mn_l; st->mx[l] = mx_l; st->lo[l] = lo; st->hi[l] = hi; }
  }
}

__global__ void __launch_bounds__(kBigThreads, 2) k_seg_big(const SegArgs a) {
  extern __shared__ __align__(16) uint32_t big_vals[];  // [kLanes][kBigMax]
  __shared__ BigShared sh;
  const uint32_t n_big = min(big_row_counter(a.ctl)[0], a.max_rows);
  CtaReduce red{sh.part, 0u};
  for (uint32_t t = blockIdx.x; t < n_big; t += gridDim.x) {
    const uint32_t row = a.big_rows[t], s = a.row_start[row];
    seg_big_row(a, row, s, min(a.row_cnt ? a.row_cnt[row] : a.row_start[row + 1] - s, kBigMax), big_vals, sh, red);
  }
}

// ---------------------------------------------------------------------------------------------------------
// Large rows.  The i-th of `samples` values drawn from cnt: one from every stretch of cnt / samples, at a place that a hash of
// its number picks.  (Evenly spaced ones see a single phase of a row whose values repeat with a period that divides the
// spacing: a row of 4 M values with a period of 4,096 then took 5 ms instead of 0.16, its middle far from the pivots.)
__device__ __forceinline__ uint32_t sample_place(uint32_t i, uint32_t cnt, uint32_t samples) {
  uint32_t h = i + 1;  // the finalizer of MurmurHash3
  h = (h ^ (h >> 16)) * 0x85EBCA6Bu;
  h = (h ^ (h >> 13)) * 0xC2B2AE35u;
  h ^= h >> 16;
  return (uint32_t)((unsigned long long)i * cnt / samples) + __umulhi(h, cnt / samples);
}
// Pivots around rank k of cnt values v[i * stride], one warp: the ranks kLargeSpread below and above the place of k among
// kLargeSample of them.
__device__ __forceinline__ void sample_pivots(const uint32_t* v, uint32_t stride, uint32_t cnt, uint32_t k, uint32_t* p1, uint32_t* p2) {
  constexpr int R = kLargeSample / 32;
  const uint32_t lane = lane_id();
  uint32_t x[R], mn = 0xFFFFFFFFu, mx = 0;
  unsigned long long sum = 0;
#pragma unroll
  for (int i = 0; i < R; ++i) x[i] = v[(size_t)stride * sample_place((uint32_t)i * 32 + lane, cnt, kLargeSample)];
#pragma unroll
  for (int i = 0; i < R; ++i) { mn = min(mn, x[i]); mx = max(mx, x[i]); sum += x[i]; }
  mn = warp_min(mn);
  mx = warp_max(mx);
  sum = warp_sum48(sum);
  const uint32_t mean = (uint32_t)(sum / kLargeSample), at = (uint32_t)(((unsigned long long)k * kLargeSample) / cnt);
  *p1 = warp_rank<R>(x, kLargeSample, mn, mx, mean, at > kLargeSpread ? at - kLargeSpread : 0u);
  uint32_t below = 0;  // p1 is the lower end of the second search
#pragma unroll
  for (int i = 0; i < R; ++i) below += x[i] < *p1 ? 1u : 0u;
  *p2 = warp_rank<R>(x, kLargeSample, *p1, mx, mean, min(at + kLargeSpread, kLargeSample - 1), warp_sum(below));
}
// ... and a CTA, from kWideSample of them (buf: as many words of shared memory)
__device__ __forceinline__ void wide_pivots(CtaReduce& red, uint32_t* buf, const uint32_t* v, uint32_t stride, uint32_t cnt, uint32_t k, uint32_t* p1, uint32_t* p2) {
  constexpr uint32_t R = kWideSample / kBigThreads;
  uint32_t mn = 0xFFFFFFFFu, mx = 0, mean = 0, next;
#pragma unroll 8
  for (uint32_t i = 0; i < R; ++i) {
    const uint32_t x = v[(size_t)stride * sample_place(i * kBigThreads + threadIdx.x, cnt, kWideSample)];
    buf[i * kBigThreads + threadIdx.x] = x;  // (a thread reads only what it has written)
    mn = min(mn, x); mx = max(mx, x); mean += x / kWideSample;
  }
  mn = red.min_of(mn);
  mx = red.max_of(mx);
  mean = red.sum(mean);
  const uint32_t at = (uint32_t)(((unsigned long long)k * kWideSample) / cnt);
  auto each = [&](auto f) {
#pragma unroll 8
    for (uint32_t i = 0; i < R; ++i) f(buf[i * kBigThreads + threadIdx.x]);
  };
  cta_ranks(red, kWideSample, mn, mx, mean, at > kWideSpread ? at - kWideSpread : 0u, false, each, p1, &next);
  cta_ranks(red, kWideSample, mn, mx, mean, min(at + kWideSpread, kWideSample - 1), false, each, p2, &next);
}
// a row's part of the scratch: [0] the first narrowing, [1] the second
__device__ __forceinline__ uint32_t* cand_part(const SegArgs& a, const LargeRow* L, int l, int which, uint32_t* cap) {
  const size_t unit = which ? 16 : 4, from = L->start / unit, to = ((size_t)L->start + L->cnt) / unit;
  *cap = (uint32_t)(to - from);
  return a.cand + (size_t)l * a.cand_words + (which ? a.cand_second : 0) + from;
}

__global__ void __launch_bounds__(kBigThreads) k_segL_sample(const SegArgs a) {
  __shared__ uint32_t buf[kWideSample];
  __shared__ uint32_t part[2][kBigThreads / 32];
  CtaReduce red{part, 0u};
  const uint32_t n_jobs = a.n_lanes * min(a.ctl->ticket, a.max_large);
  for (uint32_t j = blockIdx.x; j < n_jobs; j += gridDim.x) {
    LargeRow* L = a.large + j / a.n_lanes;
    if (L->cnt < kWideMin) continue;
    const int l = (int)(j % a.n_lanes);
    uint32_t stride, p1, p2;
    const uint32_t* v = seg_lane(a, L->start, l, &stride);
    wide_pivots(red, buf, v, stride, L->cnt, (L->cnt - 1) >> 1, &p1, &p2);
    if (threadIdx.x == 0) { L->p1[l] = p1; L->p2[l] = p2; }
  }
  for (uint32_t j = blockIdx.x * 8 + (threadIdx.x >> 5); j < n_jobs; j += gridDim.x * 8) {
    LargeRow* L = a.large + j / a.n_lanes;
    if (L->cnt >= kWideMin || L->cnt == 0) continue;
    const int l = (int)(j % a.n_lanes);
    uint32_t stride, p1, p2;
    const uint32_t* v = seg_lane(a, L->start, l, &stride);
    sample_pivots(v, stride, L->cnt, (L->cnt - 1) >> 1, &p1, &p2);
    if (lane_id() == 0) { L->p1[l] = p1; L->p2[l] = p2; }
  }
}

// A value against the pivots: counts, and the values strictly between them into a shared-memory queue (one counter update per
// warp; kBounded: those behind the first cap values are counted only).  All lanes of the warp call it.
struct PivotCount {
  uint32_t lt = 0, e1 = 0, e2 = 0;
  template <bool kBounded = false>
  __device__ __forceinline__ void add(bool have, uint32_t x, uint32_t p1, uint32_t p2, uint32_t* queue, uint32_t* queue_len, uint32_t cap = 0u) {
    lt += have && x < p1 ? 1u : 0u;
    e1 += have && x == p1 ? 1u : 0u;
    e2 += have && x == p2 && p1 != p2 ? 1u : 0u;
    const bool mid = have && x > p1 && x < p2;
    const uint32_t ballot = __ballot_sync(0xFFFFFFFFu, mid);
    if (ballot) {
      uint32_t at = 0;
      if (lane_id() == 0) at = atomicAdd(queue_len, (uint32_t)__popc(ballot));
      at = __shfl_sync(0xFFFFFFFFu, at, 0);
      at += __popc(ballot & lanemask_lt());
      if (mid && (!kBounded || at < cap)) queue[at] = x;
    }
  }
};

// Where the ranks k and k2 (k or k + 1) lie among values of which `below` are under p1, e1 equal to it, m strictly between the
// pivots, e2 equal to p2 and the others above.  What lies on a pivot is known at once.
struct MiddlePlace {
  bool missed;          // a rank lies outside the pivots
  bool lo_mid, hi_mid;  // rank k / k2 is among the m values in between
  uint32_t lo, hi;      // ... else its value
  uint32_t r;           // the first of the ranks in between, counted among the m values
  uint32_t guess;       // about its value: they lie strictly between the pivots, about evenly
};
__device__ __forceinline__ MiddlePlace place_middle(uint32_t k, uint32_t k2, uint32_t p1, uint32_t p2, uint32_t below, uint32_t e1, uint32_t m, uint32_t e2) {
  const uint32_t f1 = below + e1, f2 = f1 + m, f3 = f2 + e2;
  MiddlePlace w;
  w.missed = k < below || k2 >= f3;
  w.lo_mid = k >= f1 && k < f2;
  w.hi_mid = k2 >= f1 && k2 < f2;
  w.lo = k < f1 ? p1 : p2;
  w.hi = k2 < f1 ? p1 : p2;
  w.r = w.lo_mid ? k - f1 : k2 - f1;
  w.guess = p1 + (uint32_t)((float)(p2 - p1) * __fdividef((float)w.r + 0.5f, (float)m));
  return w;
}

// True in the CTA that does the last of a row's `chunks` chunks.  It then sees what the others stored and added: their stores
// lie in front of a fence and an atomic, its loads behind the same atomic and a fence.  Nobody waits.
__device__ __forceinline__ bool last_chunk(uint32_t* done, uint32_t chunks, uint32_t* flag) {
  __syncthreads();
  if (threadIdx.x == 0) {
    __threadfence();
    *flag = atomicAdd(done, 1u) + 1 == chunks ? 1u : 0u;
    __threadfence();
  }
  __syncthreads();
  return *flag != 0;
}
__device__ __forceinline__ uint32_t fresh(const uint32_t* p) { return *reinterpret_cast<const volatile uint32_t*>(p); }  // (others add to it in the same launch)

// Pivots and chunks of the second narrowing of a row, one CTA; buf: kWideSample words of shared memory.
__device__ __forceinline__ void narrow_again(const SegArgs& a, uint32_t large, uint32_t* buf, uint32_t (*part)[kBigThreads / 32], uint32_t* s_base) {
  LargeRow* L = a.large + large;
  CtaReduce red{part, 0u};
  for (int l = 0; l < a.n_lanes; ++l) {
    const uint32_t m = fresh(&L->n_mid[l]);
    uint32_t cap, q1, q2;
    const uint32_t* src = cand_part(a, L, l, 0, &cap);
    if (m <= kNarrowMin || m > cap) continue;
    const MiddlePlace w = place_middle((L->cnt - 1) >> 1, L->cnt >> 1, L->p1[l], L->p2[l], fresh(&L->lt[l]), fresh(&L->e1[l]), m, fresh(&L->e2[l]));
    if (w.missed || !(w.lo_mid || w.hi_mid)) continue;
    wide_pivots(red, buf, src, 1u, m, w.r, &q1, &q2);
    const uint32_t nch = chunk_count(m, kLargeChunk);
    __syncthreads();  // the previous lane's readers of s_base are done
    if (threadIdx.x == 0) {
      L->q1[l] = q1; L->q2[l] = q2;
      L->q_lt[l] = L->q_e1[l] = L->q_e2[l] = L->q_mid[l] = 0;
      *s_base = (uint32_t)atomicAdd(&a.ctl->chunks2, (unsigned long long)nch);
      L->narrowed[l] = *s_base + nch <= a.max_chunks2;
    }
    __syncthreads();
    for (uint32_t c = threadIdx.x; c < nch && *s_base + c < a.max_chunks2; c += kBigThreads) {
      a.chunk2_job[*s_base + c] = large * a.n_lanes + l;
      a.chunk2_idx[*s_base + c] = c;
    }
  }
}

constexpr size_t segL_pass_smem_bytes() { return (size_t)kLanes * kLargeChunk * sizeof(uint32_t); }
__global__ void __launch_bounds__(256, 4) k_segL_pass(const SegArgs a) {
  extern __shared__ __align__(16) uint32_t queue[];  // [kLanes][kLargeChunk]
  __shared__ uint32_t q_len[kLanes], q_base[kLanes];
  __shared__ unsigned long long sh_sum[kLanes];
  __shared__ uint32_t sh[kLanes][5];  // min, max, lt, e1, e2
  __shared__ uint32_t part[2][kBigThreads / 32], s_word;
  const uint32_t n_chunks = (uint32_t)min(a.ctl->scratch0, (unsigned long long)a.max_chunks);
  const int nl = a.n_lanes;
  for (uint32_t c = blockIdx.x; c < n_chunks; c += gridDim.x) {
    if (a.chunk_row[c] == kNoRow) continue;
    LargeRow* L = a.large + a.chunk_row[c];
    const uint32_t off = a.chunk_idx[c] * kLargeChunk;
    const uint32_t m = min(kLargeChunk, L->cnt - off);
    const size_t base = (size_t)L->start + off;
    __syncthreads();  // the previous chunk's readers of the shared arrays are done
    if (threadIdx.x < kLanes) {
      const int l = threadIdx.x;
      q_len[l] = 0; sh_sum[l] = 0; sh[l][0] = 0xFFFFFFFFu; sh[l][1] = sh[l][2] = sh[l][3] = sh[l][4] = 0;
    }
    __syncthreads();
    uint32_t p1[kLanes], p2[kLanes], mn[kLanes], mx[kLanes];
    unsigned long long sum[kLanes];
    PivotCount cnt[kLanes];
#pragma unroll
    for (int l = 0; l < kLanes; ++l) { p1[l] = L->p1[l]; p2[l] = L->p2[l]; sum[l] = 0; mn[l] = 0xFFFFFFFFu; mx[l] = 0; }
    for (uint32_t i0 = 0; i0 < m; i0 += 1024) {  // whole warps stay in the loop: the queue pushes are warp-wide
      Val3 xs[4];
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const uint32_t i = i0 + 256 * u + threadIdx.x;
        if (i < m) xs[u] = seg_fetch(a, base + i);
        else xs[u].v[0] = xs[u].v[1] = xs[u].v[2] = 0;
      }
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const bool have = i0 + 256 * u + threadIdx.x < m;
#pragma unroll
        for (int l = 0; l < kLanes; ++l) {
          if (l >= nl) break;
          const uint32_t x = xs[u].v[l];
          sum[l] += x;
          mx[l] = max(mx[l], x);
          mn[l] = min(mn[l], have ? x : 0xFFFFFFFFu);
          cnt[l].add(have, x, p1[l], p2[l], queue + l * kLargeChunk, &q_len[l]);
        }
      }
    }
#pragma unroll
    for (int l = 0; l < kLanes; ++l) {
      const unsigned long long s2 = warp_sum48(sum[l]);
      const uint32_t n2 = warp_min(mn[l]), x2 = warp_max(mx[l]), lt = warp_sum(cnt[l].lt), e1 = warp_sum(cnt[l].e1), e2 = warp_sum(cnt[l].e2);
      if (lane_id() == 0) {
        atomicAdd(&sh_sum[l], s2);
        atomicMin(&sh[l][0], n2);
        atomicMax(&sh[l][1], x2);
        if (lt) atomicAdd(&sh[l][2], lt);
        if (e1) atomicAdd(&sh[l][3], e1);
        if (e2) atomicAdd(&sh[l][4], e2);
      }
    }
    __syncthreads();
    if (threadIdx.x < (uint32_t)nl) {
      const int l = threadIdx.x;
      atomicAdd(&L->sum[l], sh_sum[l]);
      atomicMin(&L->mn[l], sh[l][0]);
      atomicMax(&L->mx[l], sh[l][1]);
      atomicAdd(&L->lt[l], sh[l][2]);
      atomicAdd(&L->e1[l], sh[l][3]);
      atomicAdd(&L->e2[l], sh[l][4]);
      q_base[l] = q_len[l] ? atomicAdd(&L->n_mid[l], q_len[l]) : 0u;
    }
    __syncthreads();
    for (int l = 0; l < nl; ++l) {
      uint32_t cap;
      uint32_t* dst = cand_part(a, L, l, 0, &cap);
      const uint32_t b = q_base[l], n = q_len[l];
      for (uint32_t i = threadIdx.x; i < n; i += 256) if (b + i < cap) dst[b + i] = queue[l * kLargeChunk + i];
    }
    if (L->cnt >= kNarrowRow && last_chunk(&L->done, chunk_count(L->cnt, kLargeChunk), &s_word)) narrow_again(a, a.chunk_row[c], queue, part, &s_word);
  }
}

// One chunk of the second narrowing: the collected values against its pivots.  True in the CTA that does the last one of the row
// and lane.
__device__ __forceinline__ bool narrow_chunk(const SegArgs& a, uint32_t c, uint32_t* queue, CtaReduce& red, uint32_t* q_len, uint32_t* q_base, uint32_t* s_word) {
  const uint32_t j = a.chunk2_job[c], off = a.chunk2_idx[c] * kLargeChunk;
  LargeRow* L = a.large + j / a.n_lanes;
  const int l = (int)(j % a.n_lanes);
  uint32_t cap;
  const uint32_t* src = cand_part(a, L, l, 0, &cap) + off;
  const uint32_t all = L->n_mid[l], m = min(kLargeChunk, all - off), q1 = L->q1[l], q2 = L->q2[l];
  if (threadIdx.x == 0) *q_len = 0;
  __syncthreads();
  PivotCount cn;
#pragma unroll
  for (uint32_t i0 = 0; i0 < kLargeChunk; i0 += 8 * kBigThreads) {  // whole warps: the queue pushes are warp-wide
    uint32_t x[8];
#pragma unroll
    for (int u = 0; u < 8; ++u) { const uint32_t i = i0 + kBigThreads * u + threadIdx.x; x[u] = i < m ? src[i] : 0u; }
#pragma unroll
    for (int u = 0; u < 8; ++u) cn.add(i0 + kBigThreads * u + threadIdx.x < m, x[u], q1, q2, queue, q_len);
  }
  const uint32_t lt = red.sum(cn.lt), e1 = red.sum(cn.e1), e2 = red.sum(cn.e2);  // (barriers: the queue is complete)
  if (threadIdx.x == 0) {
    if (lt) atomicAdd(&L->q_lt[l], lt);
    if (e1) atomicAdd(&L->q_e1[l], e1);
    if (e2) atomicAdd(&L->q_e2[l], e2);
    *q_base = *q_len ? atomicAdd(&L->q_mid[l], *q_len) : 0u;
  }
  __syncthreads();
  uint32_t* dst = cand_part(a, L, l, 1, &cap);
  const uint32_t b = *q_base, n = *q_len;
  for (uint32_t i = threadIdx.x; i < n; i += kBigThreads) if (b + i < cap) dst[b + i] = queue[i];
  return last_chunk(&L->q_done[l], chunk_count(all, kLargeChunk), s_word);
}

// One CTA, one value lane of a row of kBigMax+1 .. kSmallSamples samples: what k_segL_* do over many CTAs, for the small builds that
// finish in one launch.  One pass over the lane (16 loads in flight per thread) adds it up, counts against the pivots and collects
// what lies between them (a sixth) in the queue, all kLanes * kBigMax words of shared memory.
__device__ __forceinline__ void seg_long_lane(const SegArgs& a, uint32_t row, uint32_t s, uint32_t cnt, int l, uint32_t* queue, BigShared& sh, CtaReduce& red) {
  constexpr uint32_t kCap = kLanes * kBigMax;
  constexpr int R = kBigMax / kBigThreads, U = 16;
  const uint32_t tid = threadIdx.x, lane = lane_id(), warp = tid >> 5, k = (cnt - 1) >> 1;
  const bool want_next = !(cnt & 1u);
  uint32_t stride;
  const uint32_t* v = seg_lane(a, s, l, &stride);
  __syncthreads();  // the previous row's readers of the shared arrays are done
  if (warp == 0) {
    uint32_t q1, q2;
    sample_pivots(v, stride, cnt, k, &q1, &q2);
    if (lane == 0) { sh.pivot[0] = q1; sh.pivot[1] = q2; sh.queued = 0; }
  }
  __syncthreads();
  const uint32_t p1 = sh.pivot[0], p2 = sh.pivot[1];
  PivotCount cn;
  unsigned long long sum = 0;
  uint32_t mn = 0xFFFFFFFFu, mx = 0, lo, hi;
  for (uint32_t i0 = 0; i0 < cnt; i0 += kBigThreads * U) {  // whole warps stay in the loop: the queue pushes are warp-wide
    uint32_t x[U];
#pragma unroll
    for (int u = 0; u < U; ++u) { const uint32_t i = i0 + kBigThreads * u + tid; x[u] = i < cnt ? v[(size_t)i * stride] : 0u; }
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const bool have = i0 + kBigThreads * u + tid < cnt;
      sum += x[u];
      mx = max(mx, x[u]);
      mn = min(mn, have ? x[u] : 0xFFFFFFFFu);
      cn.add<true>(have, x[u], p1, p2, queue, &sh.queued, kCap);
    }
  }
  sum = warp_sum48(sum);
  mn = red.min_of(mn);  // (barriers: the queue and its length are settled)
  mx = red.max_of(mx);
  if (lane == 0) sh.sum[warp][0] = sum;
  const uint32_t below = red.sum(cn.lt), e1 = red.sum(cn.e1), e2 = red.sum(cn.e2), m = sh.queued;
  sum = 0;
  for (int w = 0; w < kBigThreads / 32; ++w) sum += sh.sum[w][0];
  const MiddlePlace w = place_middle(k, want_next ? k + 1 : k, p1, p2, below, e1, m, e2);
  if (w.missed || m > kCap) {
    cta_ranks(red, cnt, mn, mx, p1, k, want_next, [&](auto f) { each_of(v, stride, cnt, f); }, &lo, &hi);
  } else {
    lo = w.lo;
    hi = w.hi;
    if (w.lo_mid || w.hi_mid) {
      const bool both = w.lo_mid && w.hi_mid && want_next;
      uint32_t y, z;
      if (m <= kBigMax) {
        uint32_t x[R];
#pragma unroll
        for (int i = 0; i < R; ++i) x[i] = tid + kBigThreads * i < m ? queue[tid + kBigThreads * i] : 0xFFFFFFFFu;
        cta_ranks(red, m, p1 + 1, p2 - 1, w.guess, w.r, both,
                  [&](auto f) {
#pragma unroll
                    for (int i = 0; i < R; ++i) f(x[i]);
                  },
                  &y, &z);
      } else {
        cta_ranks(red, m, p1 + 1, p2 - 1, w.guess, w.r, both, [&](auto f) { each_of(queue, 1u, m, f); }, &y, &z);
      }
      if (w.lo_mid) lo = y;
      if (w.hi_mid) hi = both ? z : y;
    }
  }
  if (tid == 0) {
    RowStats* st = a.stats + row;
    st->sum[l] = sum; st->mn[l] = mn; st->mx[l] = mx; st->lo[l] = lo; st->hi[l] = hi;
  }
}

// One CTA per large row and value lane: the ranks (cnt - 1) / 2 and cnt / 2 among the collected values.  Rows that are narrowed a
// second time come first, chunk by chunk; the CTA that does the last chunk goes on with the ranks.
constexpr int kFinishUnroll = 8;  // values per thread and round of a narrowing
__global__ void __launch_bounds__(kBigThreads) k_segL_finish(const SegArgs a) {
  constexpr int R = kBigMax / kBigThreads;
  static_assert(kBigThreads * kFinishUnroll <= kLargeChunk, "one queue for both");
  __shared__ uint32_t queue[kLargeChunk];
  __shared__ uint32_t part[2][kBigThreads / 32];
  __shared__ uint32_t sh_p[2], q_len, q_base, s_word;
  const uint32_t tid = threadIdx.x;
  const uint32_t n_chunks = (uint32_t)min(a.ctl->chunks2, (unsigned long long)a.max_chunks2);
  const uint32_t n_jobs = a.n_lanes * min(a.ctl->ticket, a.max_large);
  CtaReduce red{part, 0u};
  for (uint32_t item = blockIdx.x; item < n_chunks + n_jobs; item += gridDim.x) {
    if (item < n_chunks && !narrow_chunk(a, item, queue, red, &q_len, &q_base, &s_word)) continue;
    const uint32_t j = item < n_chunks ? a.chunk2_job[item] : item - n_chunks;
    const LargeRow* L = a.large + j / a.n_lanes;
    const int l = (int)(j % a.n_lanes);
    if (L->narrowed[l] != (item < n_chunks) || L->cnt == 0) continue;
    const uint32_t cnt = L->cnt, k = (cnt - 1) >> 1;
    const bool want_next = !(cnt & 1u);
    uint32_t lo = 0, hi = 0, cap;
    const uint32_t* src = cand_part(a, L, l, 0, &cap);
    uint32_t p1 = L->p1[l], p2 = L->p2[l], below = L->lt[l], e1 = L->e1[l], e2 = L->e2[l], m = L->n_mid[l];
    bool found = m <= cap;
    int which = 1;
    if (found && L->narrowed[l]) {  // unless its pivots missed, or its values did not fit: then from the first narrowing on
      const uint32_t inside = below + e1 + fresh(&L->q_lt[l]), qe1 = fresh(&L->q_e1[l]), qe2 = fresh(&L->q_e2[l]), qm = fresh(&L->q_mid[l]);
      uint32_t cap2;
      const uint32_t* narrow = cand_part(a, L, l, 1, &cap2);
      if (qm <= cap2 && !place_middle(k, cnt >> 1, L->q1[l], L->q2[l], inside, qe1, qm, qe2).missed) {
        src = narrow;
        which = 0;
        p1 = L->q1[l]; p2 = L->q2[l]; below = inside; e1 = qe1; e2 = qe2; m = qm;
      }
    }
    for (; found; which ^= 1) {
      const MiddlePlace w = place_middle(k, cnt >> 1, p1, p2, below, e1, m, e2);
      if (w.missed) { found = false; break; }
      if (!w.lo_mid) lo = w.lo;
      if (!w.hi_mid) hi = w.hi;
      if (!w.lo_mid && !w.hi_mid) break;
      const uint32_t r = w.r, guess = w.guess, in_front = below + e1;
      const bool lo_mid = w.lo_mid, hi_mid = w.hi_mid, both = lo_mid && hi_mid && want_next;
      if (m <= kBigMax) {
        uint32_t x[R], u, v;
#pragma unroll
        for (int i = 0; i < R; ++i) x[i] = tid + kBigThreads * i < m ? src[tid + kBigThreads * i] : 0xFFFFFFFFu;
        cta_ranks(red, m, p1 + 1, p2 - 1, guess, r, both,
                  [&](auto f) {
#pragma unroll
                    for (int i = 0; i < R; ++i) f(x[i]);
                  },
                  &u, &v);
        if (lo_mid) lo = u;
        if (hi_mid) hi = both ? v : u;
        break;
      }
      // narrow the collected values the same way, from one part of the scratch into the other
      const uint32_t old_p1 = p1, old_p2 = p2;
      uint32_t* dst = cand_part(a, L, l, which, &cap);
      if (tid < 32) {
        uint32_t q1, q2;
        sample_pivots(src, 1u, m, r, &q1, &q2);
        if (tid == 0) { sh_p[0] = q1; sh_p[1] = q2; q_base = 0; q_len = 0; }
      }
      __syncthreads();
      p1 = sh_p[0]; p2 = sh_p[1];
      PivotCount cn;
      for (uint32_t i0 = 0; i0 < m; i0 += kBigThreads * kFinishUnroll) {
        uint32_t x[kFinishUnroll];
#pragma unroll
        for (int u = 0; u < kFinishUnroll; ++u) { const uint32_t i = i0 + kBigThreads * u + tid; x[u] = i < m ? src[i] : 0u; }
#pragma unroll
        for (int u = 0; u < kFinishUnroll; ++u) cn.add(i0 + kBigThreads * u + tid < m, x[u], p1, p2, queue, &q_len);
        __syncthreads();
        const uint32_t n = q_len, b = q_base;
        for (uint32_t i = tid; i < n; i += kBigThreads) if (b + i < cap) dst[b + i] = queue[i];
        __syncthreads();
        if (tid == 0) { q_base = b + n; q_len = 0; }
        __syncthreads();
      }
      const uint32_t mid = q_base;
      const uint32_t lt = red.sum(cn.lt);
      e1 = red.sum(cn.e1);
      e2 = red.sum(cn.e2);
      __syncthreads();  // q_base and the pivots have been read; the copied values are there for the whole CTA
      if (mid > cap || mid > m / 2) {  // no room, or hardly narrower: search the values as they are
        uint32_t u, v;
        cta_ranks(red, m, old_p1 + 1, old_p2 - 1, guess, r, both, [&](auto f) { each_of(src, 1u, m, f); }, &u, &v);
        if (lo_mid) lo = u;
        if (hi_mid) hi = both ? v : u;
        break;
      }
      below = in_front + lt;
      m = mid;
      src = dst;
    }
    if (!found) {
      uint32_t stride;
      const uint32_t* v = seg_lane(a, L->start, l, &stride);
      cta_ranks(red, cnt, L->mn[l], L->mx[l], p1, k, want_next, [&](auto f) { each_of(v, stride, cnt, f); }, &lo, &hi);
    }
    if (tid == 0) {
      RowStats* st = a.stats + L->row;
      st->sum[l] = L->sum[l]; st->mn[l] = L->mn[l]; st->mx[l] = L->mx[l]; st->lo[l] = lo; st->hi[l] = hi;
    }
    __syncthreads();
  }
}

}  // namespace ks
