// ks_tilestats.cuh -- K4 in one read of the sorted sample stream: row detection and the integer statistics of every row
// of up to kTsRowMax samples, fused.
//
// The sorted stream is cut into tiles of kTsTile samples.  A CTA stages its tile plus kTsOver samples behind it in shared
// memory (structure of arrays: sort key and the three value lanes), marks where the sort key changes, numbers the rows
// that START in its tile (a row number is a run's base from one atomic per tile plus the place in the tile), sorts
// them into classes and computes sum / min / max and the two middle order statistics of every
// such row of at most kTsRowMax samples -- straight from shared memory, by size class:
//     1..kTinyRow      nothing but the row's place: k_finalize_* compute such a row from its samples (16 bytes each), which
//                      moves less than writing and reading 72 bytes of statistics
//     5..8, 9..16      one thread per row: the row's values in registers, a bitonic sorting network (fully unrolled, so
//                      every index is static) -- no lane idles the way it does when a warp sorts one short row
//     17..32           one warp per row: a warp-wide bitonic network, the three value lanes side by side
//     33..kTsRowMax    one warp per row: the values of one lane at a time in registers, the median by counting (warp_middle)
// After the rows of a tile are listed the warps work through the classes on their own (no block-wide barrier until the
// tile is done).  Longer rows, and the rare shorter one that leaves the window, go on the deferred list; k_seg_deferred
// hands them to the kernels of the longer rows (ks_segstats.cuh).
//
// Tiles are taken from a ticket counter; no tile waits for another.  A tile's rows are numbered in one run (one atomic on the
// row counter), the tiles in no order, and k_rows_scan_tiles / k_rows_order put them into the order of the samples.
//
// What bounds it: the instructions of the row classes (without them a pass over 84 M samples takes 0.30 ms, 4.5 TB/s; with
// them 0.76 ms).  On the way from 1.66 ms: rows numbered without a look-back 1.06 (and rows of up to four samples left to the
// table kernels: 40 % less on a trace of 28 M mostly tiny rows), staging by cp.async 0.88, thread classes by value lane and the
// 32-wide network for 17..32 samples 0.76.  Statistics of config c3 at 100 M launches (211 M samples) with the kernels of the
// long rows: 6.45 -> 3.24 ms.
#pragma once

#include "ks_common.cuh"
#include "ks_decode.cuh"
#include "ks_segstats.cuh"
#include "ks_sort.cuh"

namespace ks {

constexpr int kTsThreads = 256;
constexpr int kTsWarps = kTsThreads / 32;
constexpr int kTsTile = 2048;
constexpr int kTsOver = 512;
constexpr int kTsWin = kTsTile + kTsOver;
constexpr uint32_t kTsRowMax = 512;  // largest row finished inside a tile
constexpr uint32_t kOpenRow = 0xFFFFFFFFu;

struct TileStatsArgs {
  const uint4* items;     // sorted samples {sort key, lane 0, lane 1, lane 2}
  const uint32_t* n_dev;  // number of samples in device memory (then n is the bound the buffers were sized for), or nullptr
  uint32_t n;
  uint32_t* tile_rows;    // [tiles] rows that start in the tile ...
  uint32_t* tile_base;    // [tiles] ... and the number the first of them was given
  uint32_t* ticket;       // zeroed
  uint32_t* row_start;    // [max_rows]
  uint32_t* row_cnt;      // [max_rows]; kOpenRow: the row leaves its tile's window, k_seg_deferred finds its end
  uint32_t* row_key;      // [max_rows]
  uint32_t* row_of_kid;   // [kMaxKeys + 1], preset to 0xFFFFFFFF
  RowStats* stats;        // [max_rows]
  uint32_t* deferred;     // [max_deferred] rows not finished here; count in Control::n_small
  uint32_t max_deferred;
  uint32_t max_rows;
  Control* ctl;           // n_rows (zeroed before), ticket2 = rows with a sort key below n_keys (the solo rows)
};

// rows a tile can hold per class (a row of the class has at least 5 / 9 / 17 / 129 samples)
constexpr int kTsCap8 = kTsTile / 5 + 2, kTsCap16 = kTsTile / 9 + 2, kTsCapW = kTsTile / 17 + 2, kTsCapB = kTsTile / 129 + 2;

struct TsShared {
  uint32_t key[kTsWin];
  uint32_t val[kLanes][kTsWin];
  uint16_t rs[kTsTile + 2];  // window position of every row start of the tile, then the end of the last row
  uint16_t list8[kTsCap8], list16[kTsCap16], listw[kTsCapW], listb[kTsCapB];  // local row numbers by class
  uint32_t word_cnt[kTsTile / 32];
  uint32_t n8, n16, nw, nb, qhead;
  uint32_t end_last, tile[2], row_base, rows_here, n_solo_rows;
};

constexpr size_t tile_stats_smem_bytes() { return sizeof(TsShared); }

__device__ __forceinline__ void ts_store(RowStats* st, int l, unsigned long long sum, uint32_t mn, uint32_t mx, uint32_t lo, uint32_t hi) {
  st->sum[l] = sum; st->mn[l] = mn; st->mx[l] = mx; st->lo[l] = lo; st->hi[l] = hi;
}

// Bitonic sorting network over N registers, ascending.  Every loop is unrolled, so every index and direction is static.
template <int N>
__device__ __forceinline__ void net_sort(uint32_t (&x)[N]) {
#pragma unroll
  for (int k = 2; k <= N; k <<= 1) {
#pragma unroll
    for (int j = k >> 1; j > 0; j >>= 1) {
#pragma unroll
      for (int i = 0; i < N; ++i) {
        const int l = i ^ j;
        if (l > i) {
          const bool up = (i & k) == 0;
          const uint32_t p = x[i], q = x[l];
          x[i] = up ? min(p, q) : max(p, q);
          x[l] = up ? max(p, q) : min(p, q);
        }
      }
    }
  }
}
template <int N>
__device__ __forceinline__ uint32_t net_pick(const uint32_t (&x)[N], uint32_t idx) {
  uint32_t r = x[0];
#pragma unroll
  for (int i = 1; i < N; ++i) r = idx == (uint32_t)i ? x[i] : r;
  return r;
}

// One thread, one value lane of a row of 1..N samples.
template <int N>
__device__ __forceinline__ void ts_thread_row(const uint32_t* v, uint32_t cnt, RowStats* st, int l) {
  uint32_t x[N];
  unsigned long long sum = 0;
#pragma unroll
  for (int i = 0; i < N; ++i) {
    const bool have = (uint32_t)i < cnt;
    x[i] = have ? v[i] : 0xFFFFFFFFu;
    sum += have ? x[i] : 0u;
  }
  net_sort<N>(x);
  ts_store(st, l, sum, x[0], net_pick<N>(x, cnt - 1), net_pick<N>(x, (cnt - 1) >> 1), net_pick<N>(x, cnt >> 1));
}

// One warp, a row of 17..32 samples, one per thread: the three value lanes side by side through a bitonic network.
__device__ __forceinline__ void ts_warp_row32(const TsShared& sh, uint32_t s, uint32_t cnt, RowStats* st) {
  const uint32_t lane = lane_id();
  uint32_t x[kLanes];
  unsigned long long sum[kLanes];
#pragma unroll
  for (int l = 0; l < kLanes; ++l) {
    x[l] = lane < cnt ? sh.val[l][s + lane] : 0xFFFFFFFFu;
    sum[l] = warp_sum48(lane < cnt ? x[l] : 0u);
  }
#pragma unroll
  for (int k = 2; k <= 32; k <<= 1) {
#pragma unroll
    for (int j = k >> 1; j > 0; j >>= 1) {
      const bool keep_min = ((lane & j) == 0) == ((lane & k) == 0);
#pragma unroll
      for (int l = 0; l < kLanes; ++l) {
        const uint32_t o = __shfl_xor_sync(0xFFFFFFFFu, x[l], j);
        x[l] = keep_min ? min(x[l], o) : max(x[l], o);
      }
    }
  }
#pragma unroll
  for (int l = 0; l < kLanes; ++l) {
    const uint32_t mx = __shfl_sync(0xFFFFFFFFu, x[l], cnt - 1), lo = __shfl_sync(0xFFFFFFFFu, x[l], (cnt - 1) >> 1), hi = __shfl_sync(0xFFFFFFFFu, x[l], cnt >> 1);
    if (lane == 0) ts_store(st, l, sum[l], x[l], mx, lo, hi);
  }
}

// One warp, one row of up to 32 * R samples in shared memory, one value lane after the other: its values in registers, the
// middle by counting.  (Three lanes side by side hide more latency but issue more: the kernel is bound by issue, it took 1.36
// instead of 0.76 ms on 84 M samples.)
template <int R>
__device__ __forceinline__ void ts_warp_row(const TsShared& sh, uint32_t s, uint32_t cnt, RowStats* st) {
  const uint32_t lane = lane_id();
#pragma unroll 1
  for (int l = 0; l < kLanes; ++l) {
    const uint32_t* v = sh.val[l] + s;
    uint32_t x[R], mn = 0xFFFFFFFFu, mx = 0, lo, hi;
    unsigned long long sum = 0;
#pragma unroll
    for (int i = 0; i < R; ++i) {
      const bool have = lane + 32 * i < cnt;
      x[i] = have ? v[lane + 32 * i] : 0xFFFFFFFFu;
      const uint32_t z = have ? x[i] : 0u;
      sum += z; mx = max(mx, z); mn = min(mn, x[i]);
    }
    sum = warp_sum48(sum);
    mn = warp_min(mn);
    mx = warp_max(mx);
    warp_middle<R>(x, cnt, mn, mx, sum, &lo, &hi);
    if (lane == 0) ts_store(st, l, sum, mn, mx, lo, hi);
  }
}

__device__ __forceinline__ void copy_async4(uint32_t* dst, const uint32_t* src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(smem_u32(dst)), "l"(src) : "memory");
}
__device__ __forceinline__ void l2_prefetch(const void* p, uint32_t bytes) {  // 16-byte aligned, a multiple of 16 bytes
  asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(p), "r"(bytes) : "memory");
}

__global__ void __launch_bounds__(kTsThreads, 4) k_tile_stats(const TileStatsArgs a) {
  extern __shared__ __align__(16) unsigned char ts_raw[];
  TsShared& sh = *reinterpret_cast<TsShared*>(ts_raw);
  const uint32_t tid = threadIdx.x, lane = tid & 31u, warp = tid >> 5;
  const uint32_t n = a.n_dev ? min(*a.n_dev, a.n) : a.n;
  const uint32_t ntiles = (n + kTsTile - 1) / kTsTile;
  const uint32_t nk = key_count(a.ctl);
  if (tid == 0) { sh.tile[0] = atomicAdd(a.ticket, 1u); sh.n_solo_rows = 0; }
  for (uint32_t it = 0;; ++it) {
    __syncthreads();  // the previous tile's readers of the shared arrays are done; sh.tile is settled
    if (tid == 0 && sh.n_solo_rows) { atomicAdd(&a.ctl->ticket2, sh.n_solo_rows); sh.n_solo_rows = 0; }
    const uint32_t tile = sh.tile[it & 1];
    if (tile >= ntiles) break;
    // the next tile is drawn now (no tile waits for another, so nobody is held up by one that is drawn early) and brought
    // into L2 while this one is worked on
    uint32_t next = 0;
    if (tid == kTsThreads - 1) next = atomicAdd(a.ticket, 1u);
    const uint32_t t0 = tile * kTsTile;
    const uint32_t own = min((uint32_t)kTsTile, n - t0);  // samples whose rows this tile numbers
    const uint32_t wn = min((uint32_t)kTsWin, n - t0);    // staged samples
    if (tid == 0) {
      sh.n8 = sh.n16 = sh.nw = sh.nb = 0;
      sh.qhead = 0;
      sh.end_last = wn;
    }

    // ---- stage the window as a structure of arrays: asynchronous 4-byte copies, no registers and no shared-memory stores
    // (with 128-bit loads through registers the kernel took a fifth longer)
    for (uint32_t i = tid; i < wn; i += kTsThreads) {
      const uint32_t* g = reinterpret_cast<const uint32_t*>(a.items + (size_t)t0 + i);
      copy_async4(&sh.key[i], g);
#pragma unroll
      for (int l = 0; l < kLanes; ++l) copy_async4(&sh.val[l][i], g + 1 + l);
    }
    const uint32_t prev_key = t0 ? a.items[(size_t)t0 - 1].x : 0u;
    if (tid == kTsThreads - 1) {
      sh.tile[(it + 1) & 1] = next;
      if (next < ntiles) l2_prefetch(a.items + (size_t)next * kTsTile, min((uint32_t)kTsTile, n - next * kTsTile) * 16u);
    }
    asm volatile("cp.async.wait_all;" ::: "memory");
    __syncthreads();

    // ---- row starts among the tile's own samples (consecutive lanes, consecutive samples; one ballot per 32 samples)
    uint32_t ballot[kTsTile / kTsThreads];
#pragma unroll
    for (int k = 0; k < kTsTile / kTsThreads; ++k) {
      const uint32_t i = k * kTsThreads + tid;
      bool flag = false;
      if (i < own) flag = (i == 0) ? (t0 == 0 || sh.key[0] != prev_key) : (sh.key[i] != sh.key[i - 1]);
      ballot[k] = __ballot_sync(0xFFFFFFFFu, flag);
      if (lane == 0) sh.word_cnt[k * kTsWarps + warp] = __popc(ballot[k]);
    }
    // where the tile's last row ends: the first change of the sort key behind the tile's own samples
    for (uint32_t j = own + tid; j < wn; j += kTsThreads)
      if (sh.key[j] != sh.key[j - 1]) atomicMin(&sh.end_last, j);
    __syncthreads();
    if (warp == 0) {  // exclusive scan over the 64 words; the tile's rows take the next numbers, in no order among the tiles
      const uint32_t c0 = sh.word_cnt[lane], c1 = sh.word_cnt[32 + lane];
      const uint32_t i0 = warp_incl_scan(c0);
      const uint32_t tot0 = __shfl_sync(0xFFFFFFFFu, i0, 31);
      const uint32_t i1 = warp_incl_scan(c1);
      sh.word_cnt[lane] = i0 - c0;
      sh.word_cnt[32 + lane] = tot0 + i1 - c1;
      const uint32_t n_local = tot0 + __shfl_sync(0xFFFFFFFFu, i1, 31);
      if (lane == 0) {
        sh.rows_here = n_local;
        sh.rs[n_local] = (uint16_t)sh.end_last;  // end_last was settled before the barrier above
      }
    }
    __syncthreads();
    // positions of the row starts
#pragma unroll
    for (int k = 0; k < kTsTile / kTsThreads; ++k) {
      if (ballot[k] & (1u << lane)) sh.rs[sh.word_cnt[k * kTsWarps + warp] + __popc(ballot[k] & lanemask_lt())] = (uint16_t)(k * kTsThreads + tid);
    }
    __syncthreads();
    const uint32_t rows_here = sh.rows_here;
    const uint32_t end_last = sh.end_last;
    const bool last_complete = end_last < wn || t0 + wn >= n;
    if (tid == 0) {
      const uint32_t base = rows_here ? atomicAdd(&a.ctl->n_rows, rows_here) : 0u;
      sh.row_base = base;
      a.tile_rows[tile] = rows_here;
      a.tile_base[tile] = base;
    }
    if (warp != 0) {  // the rows by class
      for (uint32_t lr = tid - 32; lr < rows_here; lr += kTsThreads - 32) {
        const uint32_t cnt = sh.rs[lr + 1] - sh.rs[lr];
        if (cnt <= kTinyRow || cnt > kTsRowMax || !(lr + 1 < rows_here || last_complete)) continue;
        if (cnt <= 8) sh.list8[atomicAdd(&sh.n8, 1u)] = (uint16_t)lr;
        else if (cnt <= 16) sh.list16[atomicAdd(&sh.n16, 1u)] = (uint16_t)lr;
        else if (cnt <= 128) sh.listw[atomicAdd(&sh.nw, 1u)] = (uint16_t)lr;
        else sh.listb[atomicAdd(&sh.nb, 1u)] = (uint16_t)lr;
      }
    }
    __syncthreads();
    const uint32_t row_base = sh.row_base;

    // ---- the row arrays; rows of up to kTinyRow samples are complete with them
    for (uint32_t lr = tid; lr < rows_here; lr += kTsThreads) {
      const uint32_t s = sh.rs[lr], cnt = sh.rs[lr + 1] - s;
      const uint32_t g = row_base + lr;
      if (g >= a.max_rows) break;  // more rows than the arrays hold: k_rows_scan_tiles reports it
      const uint32_t key = sh.key[s];
      a.row_start[g] = t0 + s;
      a.row_key[g] = key;
      if (key < nk) { a.row_of_kid[key] = g; atomicAdd(&sh.n_solo_rows, 1u); }
      const bool open = !(lr + 1 < rows_here || last_complete);
      a.row_cnt[g] = open ? kOpenRow : cnt;
      if (cnt > kTsRowMax || open) {
        const uint32_t at = atomicAdd(&a.ctl->n_small, 1u);
        if (at < a.max_deferred) a.deferred[at] = g;
        else atomicOr(&a.ctl->err, kErrTooLarge);
      }
    }
    // ---- the listed rows.  Work items, the longest first: a row of 129..kTsRowMax samples, 32 value lanes of rows of the
    // two smallest classes, a row of 17..128 samples; no warp waits for another until the tile is done.
    {
      const uint32_t nb = sh.nb, m16 = 3 * sh.n16, m8 = 3 * sh.n8;
      const uint32_t j16 = nb, j8 = j16 + ((m16 + 31) >> 5), jw = j8 + ((m8 + 31) >> 5), items_total = jw + sh.nw;
      while (true) {  // the warps draw work items from a counter: a warp with a long row does not hold up its share of the short ones
        uint32_t j = 0;
        if (lane == 0) j = atomicAdd(&sh.qhead, 1u);
        j = __shfl_sync(0xFFFFFFFFu, j, 0);
        if (j >= items_total) break;
        if (j >= j16 && j < jw) {
          const bool is16 = j < j8;
          const uint32_t t = (j - (is16 ? j16 : j8)) * 32 + lane, lr = t >= (is16 ? m16 : m8) ? kTsTile : is16 ? sh.list16[t / 3] : sh.list8[t / 3];
          if (lr < kTsTile && row_base + lr < a.max_rows) {
            const uint32_t s = sh.rs[lr], cnt = sh.rs[lr + 1] - s, l = t % 3;
            if (is16) ts_thread_row<16>(sh.val[l] + s, cnt, a.stats + row_base + lr, l);
            else ts_thread_row<8>(sh.val[l] + s, cnt, a.stats + row_base + lr, l);
          }
        } else {
          const uint32_t lr = j < nb ? sh.listb[j] : sh.listw[j - jw];
          const uint32_t s = sh.rs[lr], cnt = sh.rs[lr + 1] - s;
          RowStats* st = a.stats + row_base + lr;
          if (row_base + lr < a.max_rows) {  // warp-uniform
            if (cnt <= 32) ts_warp_row32(sh, s, cnt, st);
            else if (cnt <= 64) ts_warp_row<2>(sh, s, cnt, st);
            else if (cnt <= 128) ts_warp_row<4>(sh, s, cnt, st);
            else if (cnt <= 256) ts_warp_row<8>(sh, s, cnt, st);
            else ts_warp_row<16>(sh, s, cnt, st);
          }
        }
        __syncwarp();
      }
    }
  }
}

// The rows in the order of the samples.  A tile's rows are numbered in one run, the tiles in no order: k_rows_scan_tiles (one
// CTA) turns the tiles' row counts into their offsets, k_rows_order (one warp per tile) writes row_order[position] = row.
// The look-back that used to hand out the numbers in order was two fifths of the statistics kernel (a tile waited for the
// slowest of the several hundred tiles in flight in front of it); the two launches run beside the kernels of the long rows.
struct RowsOrderArgs {
  uint32_t* tile_rows;        // in: rows per tile; out: rows in all earlier tiles
  const uint32_t* tile_base;
  const uint32_t* n_dev;
  uint32_t n;
  uint32_t* row_order;        // [max_rows]
  uint32_t max_rows;
  Control* ctl;
};
__global__ void __launch_bounds__(1024) k_rows_scan_tiles(const RowsOrderArgs a) {
  __shared__ uint32_t warp_tot[32];
  const uint32_t n = a.n_dev ? min(*a.n_dev, a.n) : a.n;
  const uint32_t ntiles = (n + kTsTile - 1) / kTsTile;
  uint32_t carry = 0;
  for (uint32_t base = 0; base < ntiles; base += 4 * 1024) {  // four consecutive tiles per thread
    const uint32_t i = base + 4 * threadIdx.x;
    uint32_t v[4], sum = 0;
#pragma unroll
    for (int u = 0; u < 4; ++u) { v[u] = i + u < ntiles ? a.tile_rows[i + u] : 0u; sum += v[u]; }
    const uint32_t inc = warp_incl_scan(sum);
    if (lane_id() == 31) warp_tot[threadIdx.x >> 5] = inc;
    __syncthreads();
    const uint32_t w = warp_tot[lane_id()], w_inc = warp_incl_scan(w);
    uint32_t off = carry + inc - sum + __shfl_sync(0xFFFFFFFFu, w_inc - w, threadIdx.x >> 5);
    carry += __shfl_sync(0xFFFFFFFFu, w_inc, 31);
#pragma unroll
    for (int u = 0; u < 4; ++u) { if (i + u < ntiles) a.tile_rows[i + u] = off; off += v[u]; }
    __syncthreads();
  }
  if (threadIdx.x == 0 && carry > a.max_rows) {
    atomicOr(&a.ctl->err, kErrTooLarge);
    a.ctl->n_rows = 0;          // no later kernel walks rows that are not there
    a.ctl->pad2[0] = carry;     // so that the host can size the arrays and run again
  }
}
__global__ void __launch_bounds__(256) k_rows_order(const RowsOrderArgs a) {
  const uint32_t n = a.n_dev ? min(*a.n_dev, a.n) : a.n;
  const uint32_t ntiles = (n + kTsTile - 1) / kTsTile, n_rows = a.ctl->n_rows;  // 0: more rows than the arrays hold
  for (uint32_t t = blockIdx.x * 8 + (threadIdx.x >> 5); t < ntiles; t += gridDim.x * 8) {
    const uint32_t at = a.tile_rows[t], end = t + 1 < ntiles ? a.tile_rows[t + 1] : n_rows, base = a.tile_base[t];
    for (uint32_t i = at + lane_id(); i < end && i < n_rows; i += 32) a.row_order[i] = base + (i - at);
  }
}

// A row that leaves its tile's window ends where its sort key does: galloping search over the sorted samples.
__device__ __forceinline__ uint32_t open_row_count(const uint4* items, uint32_t n, uint32_t st, uint32_t key) {
  uint32_t lo = min(st + kTsOver, n), hi = lo, step = kTsTile;  // samples [st, lo) are the row's
  while (hi < n && items[hi].x == key) { lo = hi + 1; hi += min(step, n - hi); step <<= 1; }
  while (lo < hi) {
    const uint32_t mid = lo + ((hi - lo) >> 1);
    if (items[mid].x == key) lo = mid + 1; else hi = mid;
  }
  return lo - st;
}

// One thread per deferred row: the list of its size class, or a large row and its chunks.
struct DeferredArgs {
  const uint32_t* deferred;
  const uint32_t* row_start;
  uint32_t* row_cnt;
  const uint32_t* row_key;
  const uint4* items;
  const uint32_t* n_dev;
  uint32_t n;
  uint32_t max_deferred;
  SegArgs seg;
};
__global__ void __launch_bounds__(256) k_seg_deferred(const DeferredArgs a) {
  const SegArgs& s = a.seg;
  const uint32_t n_rows = *s.n_rows_dev;
  if (n_rows > s.max_rows) return;  // too many rows for the arrays: the table is thrown away
  const uint32_t n = a.n_dev ? min(*a.n_dev, a.n) : a.n;
  const uint32_t nd = min(s.ctl->n_small, a.max_deferred);
  for (uint32_t t = blockIdx.x * blockDim.x + threadIdx.x; t < nd; t += gridDim.x * blockDim.x) {
    const uint32_t row = a.deferred[t];
    if (row >= n_rows) continue;
    const uint32_t st = a.row_start[row];
    uint32_t cnt = a.row_cnt[row];
    if (cnt == kOpenRow) {
      cnt = open_row_count(a.items, n, st, a.row_key[row]);
      a.row_cnt[row] = cnt;
    }
    if (cnt <= kLanesMax) {
      s.mid_rows[atomicAdd(big_row_counter(s.ctl) + 1, 1u)] = row;  // one warp per value lane
    } else if (cnt <= kBigMax) {
      s.big_rows[atomicAdd(big_row_counter(s.ctl), 1u)] = row;
    } else {
      register_large_row(s, row, st, cnt);
    }
  }
}

// Small builds: everything behind k_tile_stats in one launch.  The last CTA puts the rows in order, the others take the
// deferred rows, one CTA per row whatever its length.  (Eight launches on three streams otherwise: statistics of 10,500
// samples 0.035 ms on the device, 0.031 so, and a dozen calls into the driver less.  The line is where one warp can still add
// up the tiles; at 4 M samples the kernels by row length take 0.155 ms.)
constexpr uint32_t kSmallSamples = 1u << 16;
struct RowsSmallArgs {
  DeferredArgs d;
  RowsOrderArgs o;
};
__global__ void __launch_bounds__(kBigThreads, 2) k_rows_small(const RowsSmallArgs a) {
  extern __shared__ __align__(16) uint32_t big_vals[];  // [kLanes][kBigMax]
  __shared__ BigShared sh;
  __shared__ uint32_t s_cnt;
  const SegArgs& s = a.d.seg;
  const uint32_t n = a.d.n_dev ? min(*a.d.n_dev, a.d.n) : a.d.n;
  const uint32_t n_rows = *s.n_rows_dev;
  if (blockIdx.x == gridDim.x - 1) {
    constexpr uint32_t kTiles = kSmallSamples / kTsTile;
    static_assert(kTiles <= 32, "one warp adds up the tiles");
    const uint32_t ntiles = (n + kTsTile - 1) / kTsTile, lane = lane_id();
    const uint32_t mine = lane < ntiles ? a.o.tile_rows[lane] : 0u, inc = warp_incl_scan(mine), total = __shfl_sync(0xFFFFFFFFu, inc, 31);
    if (total > a.o.max_rows) {
      if (threadIdx.x == 0) {
        atomicOr(&a.o.ctl->err, kErrTooLarge);
        a.o.ctl->pad2[0] = total;  // so that the host can size the arrays and run again
        a.o.ctl->n_rows = 0;       // no later kernel walks rows that are not there
      }
      return;
    }
    for (uint32_t t = threadIdx.x >> 5; t < ntiles; t += kBigThreads / 32) {
      const uint32_t cnt = __shfl_sync(0xFFFFFFFFu, mine, t), at = __shfl_sync(0xFFFFFFFFu, inc, t) - cnt, base = a.o.tile_base[t];
      for (uint32_t i = lane; i < cnt; i += 32) a.o.row_order[at + i] = base + i;
    }
    return;
  }
  if (n_rows > s.max_rows) return;
  const uint32_t nd = min(s.ctl->n_small, a.d.max_deferred);
  CtaReduce red{sh.part, 0u};
  for (uint32_t t = blockIdx.x; t < kLanes * nd; t += gridDim.x - 1) {  // row t % nd; lane t / nd of it if it is long
    const uint32_t row = a.d.deferred[t % nd], l = t / nd;
    if (row >= n_rows) continue;
    const uint32_t st = a.d.row_start[row];
    __syncthreads();  // the previous row's readers of s_cnt are done
    if (threadIdx.x == 0) {
      volatile uint32_t* at = a.d.row_cnt + row;  // the CTAs of the other lanes look at it too: kOpenRow or the count
      uint32_t cnt = *at;
      if (cnt == kOpenRow) { cnt = open_row_count(a.d.items, n, st, a.d.row_key[row]); if (l == 0) *at = cnt; }
      s_cnt = cnt;
    }
    __syncthreads();
    const uint32_t cnt = s_cnt;
    if (cnt > kBigMax) seg_long_lane(s, row, st, cnt, (int)l, big_vals, sh, red);
    else if (l == 0) seg_big_row(s, row, st, cnt, big_vals, sh, red);
  }
}

}  // namespace ks
