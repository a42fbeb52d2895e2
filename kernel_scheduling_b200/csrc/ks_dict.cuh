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

// The listed keys (dkeys / dslot, written by the decode kernel) ranked and placed in one launch: a CTA takes 32 keys, its 32
// warps count the smaller keys in a slice of the list each.
__global__ void __launch_bounds__(1024) k_dict_rank_place(const DictArgs a) {
  __shared__ uint32_t s_rank[32];
  const uint32_t found = a.ctl->n_keys, nk = min(found, kMaxKeys), lane = lane_id(), warp = threadIdx.x >> 5;
  if (blockIdx.x == 0 && threadIdx.x == 0 && found > kMaxKeys) atomicOr(&a.ctl->err, kErrTooManyKeys);
  const uint32_t per = (nk + 31) / 32, j0 = warp * per, j1 = min(nk, j0 + per);
  for (uint32_t i0 = blockIdx.x * 32; i0 < nk; i0 += gridDim.x * 32) {
    const uint32_t i = i0 + lane;
    const unsigned long long mine = i < nk ? a.dkeys[i] : 0ull;
    if (warp == 0) s_rank[lane] = 0;
    __syncthreads();
    uint32_t cnt = 0;
#pragma unroll 8
    for (uint32_t j = j0; j < j1; ++j) cnt += a.dkeys[j] < mine ? 1u : 0u;
    if (cnt) atomicAdd(&s_rank[lane], cnt);
    __syncthreads();
    if (warp == 0 && i < nk) {
      const uint32_t r = s_rank[lane], slot = a.dslot[i];
      a.kid_of_slot[slot] = r;
      a.slot_of_kid[r] = slot;
      a.keys_sorted[r] = mine;
    }
    __syncthreads();
  }
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
