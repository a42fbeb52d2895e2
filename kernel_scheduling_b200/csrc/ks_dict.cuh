// ks_dict.cuh -- turns the open-addressing key dictionary into dense key ids.
//
// The decode kernel leaves the distinct keys scattered over kDictSlots slots and lists them as it inserts them (the sharded
// and the online paths, whose dictionaries have several sources, collect them with k_dict_compact).  Here they are ranked by
// key value (kid = number of smaller keys, so kid order = key order and every later table comes out sorted without
// looking at the 64-bit keys again), and the solo launches are turned into the first entries of the sample stream.
#pragma once

#include <cstddef>

#include "ks_common.cuh"

namespace ks {

struct DictArgs {
  const unsigned long long* dict_keys;  // [kDictSlots]
  unsigned long long* dkeys;            // [kMaxKeys + 1] compacted keys (arbitrary order)
  uint32_t* dslot;                      // [kMaxKeys + 1] their slots
  uint32_t* kid_of_slot;                // [kDictSlots]
  uint32_t* slot_of_kid;                // [kMaxKeys + 1]
  unsigned long long* keys_sorted;      // [kMaxKeys + 1]
  Control* ctl;
};

__global__ void __launch_bounds__(256) k_dict_compact(const DictArgs a) {
  const uint32_t slot = blockIdx.x * blockDim.x + threadIdx.x;
  const unsigned long long k = slot < kDictSlots ? a.dict_keys[slot] : 0ull;
  const uint32_t ballot = __ballot_sync(0xFFFFFFFFu, k != 0ull);
  if (!ballot) return;
  uint32_t base = 0;
  const uint32_t first = __ffs(ballot) - 1;
  if (lane_id() == first) base = atomicAdd(&a.ctl->n_keys, (uint32_t)__popc(ballot));
  base = __shfl_sync(0xFFFFFFFFu, base, first);
  if (k != 0ull) {
    const uint32_t i = base + __popc(ballot & lanemask_lt());
    if (i < kMaxKeys) {
      a.dkeys[i] = k;
      a.dslot[i] = slot;
    } else {
      atomicOr(&a.ctl->err, kErrTooManyKeys);
    }
  }
}

// The listed keys (dkeys / dslot, written by the decode kernel) ranked and placed in one launch: a CTA takes 32 * PER keys, PER
// per lane, its 32 warps count the smaller keys in a slice of the list each.
template <int PER>
__device__ __forceinline__ void dict_rank_place(const DictArgs& a, uint32_t nk, uint32_t* s_rank) {
  const uint32_t lane = lane_id(), warp = threadIdx.x >> 5;
  const uint32_t per = ((nk + 31) / 32 + 1) & ~1u, j0 = warp * per, j1 = min(nk, j0 + per);  // (even: keys are read two at a time)
  for (uint32_t i0 = blockIdx.x * 32 * PER; i0 < nk; i0 += gridDim.x * 32 * PER) {
    unsigned long long mine[PER];
    uint32_t cnt[PER];
#pragma unroll
    for (int u = 0; u < PER; ++u) {
      const uint32_t i = i0 + u * 32 + lane;
      mine[u] = i < nk ? a.dkeys[i] : 0ull;
      cnt[u] = 0;
    }
    if (threadIdx.x < 32 * PER) s_rank[threadIdx.x] = 0;
    __syncthreads();
    uint32_t j = j0;
#pragma unroll 4
    for (; j + 1 < j1; j += 2) {
      const ulonglong2 k = *reinterpret_cast<const ulonglong2*>(a.dkeys + j);
#pragma unroll
      for (int u = 0; u < PER; ++u) { cnt[u] += k.x < mine[u] ? 1u : 0u; cnt[u] += k.y < mine[u] ? 1u : 0u; }
    }
    if (j < j1) {
#pragma unroll
      for (int u = 0; u < PER; ++u) cnt[u] += a.dkeys[j] < mine[u] ? 1u : 0u;
    }
#pragma unroll
    for (int u = 0; u < PER; ++u) if (cnt[u]) atomicAdd(&s_rank[u * 32 + lane], cnt[u]);
    __syncthreads();
    if (threadIdx.x < 32 * PER && i0 + threadIdx.x < nk) {
      const uint32_t i = i0 + threadIdx.x, r = s_rank[threadIdx.x], slot = a.dslot[i];
      a.kid_of_slot[slot] = r;
      a.slot_of_kid[r] = slot;
      a.keys_sorted[r] = a.dkeys[i];
    }
    __syncthreads();
  }
}
// One key per lane while that gives every CTA work; two or four (a loaded key is compared with all of them) where there are
// more keys than lanes to go round.
constexpr int kDictPer = 4;
__global__ void __launch_bounds__(1024, 2) k_dict_rank_place(const DictArgs a) {
  __shared__ uint32_t s_rank[32 * kDictPer];
  const uint32_t found = a.ctl->n_keys, nk = min(found, kMaxKeys);
  if (blockIdx.x == 0 && threadIdx.x == 0 && found > kMaxKeys) atomicOr(&a.ctl->err, kErrTooManyKeys);
  if (nk <= gridDim.x * 32) dict_rank_place<1>(a, nk, s_rank);
  else if (nk <= gridDim.x * 64) dict_rank_place<2>(a, nk, s_rank);
  else dict_rank_place<kDictPer>(a, nk, s_rank);
}

// What a run starts from: an empty dictionary, zero counters, no rows.
struct ResetArgs {
  uint4* dict_keys;
  uint4* dict_launches;
  uint4* dict_solo;
  uint4* row_of_kid;
  Control* ctl;
};
__global__ void __launch_bounds__(256) k_reset(const ResetArgs a) {
  const uint32_t t0 = blockIdx.x * blockDim.x + threadIdx.x, step = gridDim.x * blockDim.x;
  const uint4 zero = make_uint4(0, 0, 0, 0), ones = make_uint4(0xFFFFFFFFu, 0xFFFFFFFFu, 0xFFFFFFFFu, 0xFFFFFFFFu);
  for (uint32_t i = t0; i < kDictSlots / 2; i += step) a.dict_keys[i] = zero;
  for (uint32_t i = t0; i < kDictSlots / 4; i += step) { a.dict_launches[i] = zero; a.dict_solo[i] = zero; }
  for (uint32_t i = t0; i < (kMaxKeys + 1) / 4; i += step) a.row_of_kid[i] = ones;
  if (t0 < sizeof(Control) / 4) {
    const uint32_t at = offsetof(Control, min_start) / 4;
    reinterpret_cast<uint32_t*>(a.ctl)[t0] = t0 == at || t0 == at + 1 ? 0xFFFFFFFFu : 0u;
  }
}

// The solo launches become samples [0, n_solo) of the sample stream: sort key = kid, lane 0 = duration.
// Also starts the pair counter behind them.
struct SoloArgs {
  const unsigned long long* solo_stream;
  const uint32_t* kid_of_slot;
  uint4* samples;  // {sort key, lane 0, lane 1, lane 2}
  uint64_t capacity;
  Control* ctl;
};
__global__ void __launch_bounds__(256) k_solo_samples(const SoloArgs a) {
  const uint32_t ns = a.ctl->n_solo;
  if (blockIdx.x == 0 && threadIdx.x == 0) a.ctl->n_pairs = ns;  // pairs are appended behind the solo samples
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < ns && i < a.capacity; i += gridDim.x * blockDim.x) {
    const unsigned long long e = a.solo_stream[i];
    a.samples[i] = make_uint4(a.kid_of_slot[(uint32_t)e & kMetaSlotMask], (uint32_t)(e >> 32), 0u, 0u);
  }
}

}  // namespace ks
