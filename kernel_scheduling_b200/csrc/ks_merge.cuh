// ks_merge.cuh -- puts a timeline that consists of a few ordered runs into start order: pairwise merges, all pairs of a pass in
// one launch.
//
// That is what the agents' logs are: every process writes its launches in start order (scheduler/agent.cpp:683-705), and the
// logs come one behind the other.  The decode kernel notes where start_ns falls; with up to kMaxRuns runs the timeline is
// merged in ceil(log2(runs)) passes of 32 bytes per launch, where the radix sort takes one pass per 8 bits of the time range
// (five for ten minutes) and ranks every launch in each.  Equal starts keep the order of the input, as in the radix sort.
//
// A pass: k_merge_cuts finds, one thread per output tile, how many of the tile's predecessors come from the left run (binary
// search along the merge path); k_merge_tiles stages the two stretches of a tile in shared memory, every thread searches the
// start of its eight outputs there and merges them, and the tile leaves coalesced.  Bound by the stream of 32 bytes per
// launch: 20 M launches in four runs take 0.35 ms for both passes (the radix sort: 2.0 ms).
#pragma once

#include "ks_common.cuh"

namespace ks {

constexpr int kMergeThreads = 256;
constexpr int kMergeItems = 8;
constexpr uint32_t kMergeTile = kMergeThreads * kMergeItems;

struct MergeArgs {
  const unsigned long long* kin;
  const unsigned long long* vin;
  unsigned long long* kout;
  unsigned long long* vout;
  uint32_t n_runs;
  uint32_t run[kMaxRuns + 1];              // start of every run, then the end of the last
  uint32_t first_tile[kMaxRuns / 2 + 1];   // output tiles in front of every pair of runs (2p, 2p + 1)
  uint32_t* cuts;                          // [tiles] elements of the left run in front of the tile
};

struct MergePair {
  uint32_t a, na, b, nb, tile;  // left and right run, and the tile's number inside the pair
};
__device__ __forceinline__ MergePair merge_pair(const MergeArgs& m, uint32_t t) {
  uint32_t p = 0;
  while (2 * (p + 1) < m.n_runs && m.first_tile[p + 1] <= t) ++p;
  MergePair r;
  r.a = m.run[2 * p];
  r.na = m.run[2 * p + 1] - r.a;
  r.b = m.run[2 * p + 1];
  r.nb = 2 * p + 1 < m.n_runs ? m.run[2 * p + 2] - r.b : 0u;  // an odd last run has no partner
  r.tile = t - m.first_tile[p];
  return r;
}
// how many of the first d merged elements come from a (ties: a first)
__device__ __forceinline__ uint32_t merge_cut(const unsigned long long* a, uint32_t na, const unsigned long long* b, uint32_t nb, uint32_t d) {
  uint32_t lo = d > nb ? d - nb : 0u, hi = min(d, na);
  while (lo < hi) {
    const uint32_t mid = (lo + hi) >> 1;
    if (a[mid] <= b[d - 1 - mid]) lo = mid + 1; else hi = mid;
  }
  return lo;
}

__global__ void __launch_bounds__(256) k_merge_cuts(const MergeArgs m, uint32_t n_tiles) {
  const uint32_t t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= n_tiles) return;
  const MergePair p = merge_pair(m, t);
  m.cuts[t] = merge_cut(m.kin + p.a, p.na, m.kin + p.b, p.nb, p.tile * kMergeTile);
}

__global__ void __launch_bounds__(kMergeThreads) k_merge_tiles(const MergeArgs m) {
  // padded by one word in eight: the threads' runs of eight outputs start in different banks
  __shared__ unsigned long long s_k[kMergeTile + kMergeTile / 8], s_v[kMergeTile + kMergeTile / 8];
  auto at = [](uint32_t i) { return i + (i >> 3); };
  const uint32_t t = blockIdx.x, tid = threadIdx.x;
  const MergePair p = merge_pair(m, t);
  const uint32_t d0 = p.tile * kMergeTile, d1 = min(d0 + kMergeTile, p.na + p.nb), n = d1 - d0;
  const uint32_t i0 = m.cuts[t], i1 = d1 == p.na + p.nb ? p.na : m.cuts[t + 1];
  const uint32_t ca = i1 - i0, j0 = d0 - i0;
  for (uint32_t i = tid; i < n; i += kMergeThreads) {
    const size_t src = i < ca ? (size_t)p.a + i0 + i : (size_t)p.b + j0 + (i - ca);
    s_k[at(i)] = m.kin[src];
    s_v[at(i)] = m.vin[src];
  }
  __syncthreads();
  const uint32_t d = min(tid * kMergeItems, n), cb = n - ca;
  uint32_t lo = d > cb ? d - cb : 0u, hi = min(d, ca);
  while (lo < hi) {
    const uint32_t mid = (lo + hi) >> 1;
    if (s_k[at(mid)] <= s_k[at(ca + d - 1 - mid)]) lo = mid + 1; else hi = mid;
  }
  uint32_t i = lo, j = ca + d - lo;
  unsigned long long k[kMergeItems], v[kMergeItems];
#pragma unroll
  for (int u = 0; u < kMergeItems; ++u) {
    k[u] = v[u] = 0;
    if (d + u < n) {
      const bool left = j >= n || (i < ca && s_k[at(i)] <= s_k[at(j)]);
      const uint32_t src = at(left ? i : j);
      k[u] = s_k[src];
      v[u] = s_v[src];
      if (left) ++i; else ++j;
    }
  }
  __syncthreads();
#pragma unroll
  for (int u = 0; u < kMergeItems; ++u) {
    if (d + u < n) { s_k[at(d + u)] = k[u]; s_v[at(d + u)] = v[u]; }
  }
  __syncthreads();
  const size_t out = (size_t)p.a + d0;
  for (uint32_t q = tid; q < n; q += kMergeThreads) {
    m.kout[out + q] = s_k[at(q)];
    m.vout[out + q] = s_v[at(q)];
  }
}

// Control::min_start / max_start of an ordered timeline
__global__ void k_range_of_ordered(const unsigned long long* __restrict__ tl_start, uint64_t n, Control* ctl) {
  atomicMin(&ctl->min_start, tl_start[0]);
  atomicMax(&ctl->max_start, tl_start[n - 1]);
}

}  // namespace ks
