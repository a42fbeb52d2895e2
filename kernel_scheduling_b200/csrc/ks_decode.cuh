// ks_decode.cuh -- K1: record decode, kernel-key hash and key dictionary in one read of the trace.
//
// A CTA streams tiles of 384 records (18,432 contiguous bytes) into shared memory with bulk asynchronous copies
// (cp.async.bulk, completion on an mbarrier, two tiles in flight), so global memory is read as whole 128-byte
// lines although a record is 48 bytes; each thread then takes its record from shared memory as three 128-bit
// loads (a 48-byte stride is conflict-free for 128-bit shared loads).  Per record it
//   * computes the 64-bit kernel key (ks_common.cuh kernel_key),
//   * finds the key's slot in the open-addressing dictionary (2^18 slots, 2 MB: the probes are L2 hits; keys known to sit in
//     their home slots are answered from shared memory),
//   * writes the compact timeline entry  start_ns (u64) | duration (u32) | meta (u32: slot, solo, tenant),
//   * appends solo launches to the solo stream (slot | duration << 32),
//   * checks the record (end >= start, duration < 2^31 ns so that a pair's span fits 32 bits) and whether start_ns is non-decreasing.
// Per-key launch counts are accumulated in a per-CTA shared-memory cache (sets of four keys) and flushed now and then, so hot
// keys do not turn into a queue of same-address global atomics; solo launches wait in a shared-memory queue, so the counter
// of the solo stream is updated once per few hundred of them.
//
// What bounds it: instructions and latency (hash, dictionary probe, counting), at 3.5 TB/s = half of the copy rate on c3 (20 M
// launches, 64 bytes each: 0.37 ms; 0.32 ms with the counting left out).  Counting through 1,024 linearly probed entries of
// three words cost as much as everything else once a stretch of the trace had more keys than that: 0.59 ms for the mixed
// trace, 0.86 ms for the logs one behind the other; with 4,096 entries in sets of four, one 64-bit load for a set's tags and
// both counts in one word 0.37 and 0.41 ms.  Solo launches scattered through the trace (c5, 4 M): 0.133 -> 0.095 ms.
#pragma once

#include "ks_common.cuh"

namespace ks {

constexpr int kDecodeThreads = 384;  // one record per thread and tile
constexpr int kDecodeStages = 2;
constexpr int kDecodeTile = kDecodeThreads;
constexpr int kDecodeTileBytes = kDecodeTile * 48;
constexpr int kDecodeCtasPerSm = 3;  // 36 warps per SM (256 threads with two records each, 24 warps, were 5 to 10 % slower)
constexpr int kCtaCountBits = 12;
constexpr uint32_t kCtaCountSlots = 1u << kCtaCountBits;  // per-CTA launch-count cache: sets of four, indexed by dictionary slot
constexpr uint32_t kCountFlushTiles = 160;  // it is flushed and emptied after so many tiles of a CTA (the counts are 16 bits wide)
static_assert(kCountFlushTiles * kDecodeTile < 65536, "16-bit counts");
constexpr uint32_t kCountCheckTiles = 8;  // ... or when the keys that found no room became many more: looked at every so many tiles
// Per-CTA cache of keys that sit in their home slots.  Without it the loads of the few hottest dictionary words queue up in L2: c1,
// 4 M launches, 0.091 ms; with it 0.083 (0.079 with loads that L1 may serve, which is no scope to read words at that other CTAs
// change with atomics).
constexpr uint32_t kHomeKeys = 1024;
constexpr uint32_t kSoloQueue = 2 * kDecodeTile;  // solo launches waiting in shared memory; written out when half full

struct DecodeArgs {
  const unsigned char* records;
  uint64_t n;
  int type_mode;
  // dictionary
  unsigned long long* dict_keys;  // [kDictSlots], 0 = empty
  uint4* dict_words;              // [kDictSlots][2] the launch fields behind a key (written by the inserting thread)
  unsigned long long* dkeys;      // optional: the keys in the order of their insertion and their slots, Control::n_keys of them
  uint32_t* dslot;                // [kMaxKeys + 1] each
  uint32_t* dict_launches;        // [kDictSlots]
  uint32_t* dict_solo;            // [kDictSlots]
  // outputs
  unsigned long long* tl_start;   // [n]
  unsigned long long* tl_dm;      // [n] duration | meta << 32
  unsigned long long* solo_stream;  // [n] slot | duration << 32, first Control::n_solo entries valid
  unsigned long long* keys_out;   // optional [n]: the key of every record
  uint32_t* run_starts;           // [kMaxRuns] where start_ns falls, in no order; Control::descents of them
  int halo;                       // 1: records of a neighbouring time window -- keyed and placed on the timeline, but not counted
  Control* ctl;
};

__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

__device__ __forceinline__ void mbar_init(uint64_t* bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_expect_tx(uint64_t* bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes) : "memory");
}
__device__ __forceinline__ void bulk_load(void* dst, const void* src, uint32_t bytes, uint64_t* bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(smem_u32(dst)), "l"(src),
               "r"(bytes), "r"(smem_u32(bar))
               : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(uint64_t* bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(ok)
      : "r"(smem_u32(bar)), "r"(parity)
      : "memory");
  return ok != 0;
}
// Bounded wait; false if the copy never arrived.
__device__ __forceinline__ bool mbar_wait_bounded(uint64_t* bar, uint32_t parity) {
  for (uint32_t spins = 0; spins < kSpinLimit; ++spins) {
    if (mbar_try_wait(bar, parity)) return true;
  }
  return false;
}

// A word that other CTAs change with atomics: read at the scope of those.
__device__ __forceinline__ uint64_t ld_relaxed_gpu_u64(const unsigned long long* p) {
  uint64_t v;
  asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
  return v;
}

// Dictionary lookup / insert of one key; returns the slot, or kDictSlots if the table is full.
__device__ __forceinline__ uint32_t dict_find_or_insert(unsigned long long* dict_keys, uint64_t key, bool* inserted) {
  uint32_t slot = dict_home(key);
  *inserted = false;
  for (uint32_t probe = 0; probe < kDictSlots; ++probe) {
    const uint64_t cur = ld_volatile_u64(reinterpret_cast<const uint64_t*>(dict_keys + slot));
    if (cur == key) return slot;
    if (cur == 0) {
      const unsigned long long old = atomicCAS(dict_keys + slot, 0ull, (unsigned long long)key);
      if (old == 0ull) { *inserted = true; return slot; }
      if (old == key) return slot;
    }
    slot = (slot + 1) & (kDictSlots - 1);
  }
  return kDictSlots;
}

// The count cache: a dictionary slot may sit in any of the four entries of the set its bits 2..11 name; the tag holds the other
// bits, so an entry's slot follows from its place and its tag.
__device__ __forceinline__ uint32_t count_tag(uint32_t slot) { return ((slot >> kCtaCountBits) << 2 | (slot & 3u)) + 1u; }
__device__ __forceinline__ uint32_t count_slot(uint32_t entry, uint32_t tag) { return ((tag - 1u) >> 2) << kCtaCountBits | (entry & ~3u) | ((tag - 1u) & 3u); }
__device__ __forceinline__ bool count_cached(unsigned short* cc_tag, uint32_t* cc_cnt, uint32_t slot, uint32_t add) {
  const uint32_t set = slot & (kCtaCountSlots - 1) & ~3u, tag = count_tag(slot);
  for (int attempt = 0; attempt < 2; ++attempt) {
    const unsigned long long t4 = *reinterpret_cast<const volatile unsigned long long*>(cc_tag + set);
    const uint32_t t[4] = {(uint32_t)t4 & 0xFFFFu, (uint32_t)t4 >> 16, (uint32_t)(t4 >> 32) & 0xFFFFu, (uint32_t)(t4 >> 48)};
    int way = -1;
#pragma unroll
    for (int w = 3; w >= 0; --w) way = t[w] == tag ? w : way;
    if (way < 0) {  // not there: the first free entry
      int spare = -1;
#pragma unroll
      for (int w = 3; w >= 0; --w) spare = t[w] == 0u ? w : spare;
      if (spare < 0) return false;
      const uint32_t old = atomicCAS(cc_tag + set + spare, (unsigned short)0, (unsigned short)tag);
      if (old == 0u || old == tag) way = spare;
    }
    if (way >= 0) { atomicAdd(&cc_cnt[set + way], add); return true; }
  }
  return false;  // lost the entry to other keys twice
}

__global__ void __launch_bounds__(kDecodeThreads, kDecodeCtasPerSm) k_decode_hash(const DecodeArgs a) {
  extern __shared__ __align__(128) unsigned char smem[];
  unsigned char* tiles = smem;                                                           // [stages][tile bytes]
  unsigned long long* solo_q = reinterpret_cast<unsigned long long*>(smem + kDecodeStages * kDecodeTileBytes);  // [kSoloQueue]
  uint64_t* bars = reinterpret_cast<uint64_t*>(solo_q + kSoloQueue);                                             // [stages]
  unsigned long long* home_keys = reinterpret_cast<unsigned long long*>(bars + kDecodeStages);  // [kHomeKeys] 0 = none
  uint32_t* cc_cnt = reinterpret_cast<uint32_t*>(home_keys + kHomeKeys);                   // [kCtaCountSlots] launches | solo launches << 16
  unsigned short* cc_tag = reinterpret_cast<unsigned short*>(cc_cnt + kCtaCountSlots);    // [kCtaCountSlots] 0 = free, see count_tag
  __shared__ uint32_t solo_n, solo_base, crowded;

  const uint32_t tid = threadIdx.x, lane = tid & 31u;
  const uint64_t ntiles = (a.n + kDecodeTile - 1) / kDecodeTile;
  for (uint32_t i = tid; i < kCtaCountSlots; i += kDecodeThreads) { cc_tag[i] = 0; cc_cnt[i] = 0; }
  for (uint32_t i = tid; i < kHomeKeys; i += kDecodeThreads) home_keys[i] = 0;
  if (tid == 0) {
    solo_n = crowded = 0;
    for (int s = 0; s < kDecodeStages; ++s) mbar_init(&bars[s], 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  }
  __syncthreads();

  auto issue = [&](uint64_t tile, int stage) {
    const uint64_t first = tile * kDecodeTile;
    const uint32_t cnt = (uint32_t)min((uint64_t)kDecodeTile, a.n - first);
    const uint32_t bytes = cnt * 48u;
    mbar_expect_tx(&bars[stage], bytes);
    bulk_load(tiles + stage * kDecodeTileBytes, a.records + first * 48ull, bytes, &bars[stage]);
  };
  // prologue: fill the pipeline
  if (tid == 0) {
    for (int s = 0; s < kDecodeStages; ++s) {
      const uint64_t t = blockIdx.x + (uint64_t)s * gridDim.x;
      if (t < ntiles) issue(t, s);
    }
  }

  uint32_t err = 0, max_dur = 0;
  uint32_t it = 0, waiting = 0;
  uint32_t flushed = 0, usual = 0;  // tile behind the last flush of the count cache; records without room in the check after it
  for (uint64_t tile = blockIdx.x; tile < ntiles; tile += gridDim.x, ++it) {
    const int stage = it % kDecodeStages;
    const uint32_t parity = (it / kDecodeStages) & 1u;
    if (!mbar_wait_bounded(&bars[stage], parity)) err |= kErrWait;  // carry on: the CTA still terminates

    const uint64_t r = tile * kDecodeTile + tid;  // consecutive lanes, consecutive records
    const bool valid = r < a.n;
    const unsigned char* rp = tiles + stage * kDecodeTileBytes + tid * 48;
    uint4 w0 = make_uint4(0, 0, 0, 0), w1 = w0, w2 = w0;
    unsigned long long prev = 0;
    if (valid) {
      w0 = *reinterpret_cast<const uint4*>(rp);
      w1 = *reinterpret_cast<const uint4*>(rp + 16);
      w2 = *reinterpret_cast<const uint4*>(rp + 32);
      if (tid > 0) prev = *reinterpret_cast<const unsigned long long*>(rp - 48 + 32);
      else if (r > 0) prev = *reinterpret_cast<const unsigned long long*>(a.records + (r - 1) * 48ull + 32);
    }
    const unsigned long long start = (unsigned long long)w2.x | ((unsigned long long)w2.y << 32);
    const unsigned long long end = (unsigned long long)w2.z | ((unsigned long long)w2.w << 32);
    const unsigned long long key = kernel_key(w0.x, w0.y, w0.z, w0.w, w1.x, w1.y, w1.z, w1.w, a.type_mode != 0);
    const bool solo = (w1.w & kMetaSoloBit) != 0;
    const uint32_t solo_ballot = __ballot_sync(0xFFFFFFFFu, valid && solo && !a.halo);
    uint32_t slot = 0;
    if (valid) {
      // the key's slot (keys of a warp are mostly distinct, so every lane probes for itself; the dictionary is 2 MB and lives
      // in L2)
      bool inserted = false;
      slot = dict_home(key);
      volatile unsigned long long* known = home_keys + (slot & (kHomeKeys - 1));
      if (*known != key) {
        if (ld_relaxed_gpu_u64(a.dict_keys + slot) == key) *known = key;
        else slot = dict_find_or_insert(a.dict_keys, key, &inserted);
      }
      if (slot >= kDictSlots) { err |= kErrTooManyKeys; slot = 0; inserted = false; }
      if (inserted) {
        uint4 k0 = w0, k1 = w1;
        k1.w &= ~kMetaSoloBit;
        if (a.type_mode) { k0.y = k0.z = k0.w = 0; k1.w &= 0xFF000000u; }
        a.dict_words[2 * (size_t)slot] = k0;
        a.dict_words[2 * (size_t)slot + 1] = k1;
        if (a.dkeys) {
          const uint32_t i = atomicAdd(&a.ctl->n_keys, 1u);
          if (i < kMaxKeys) { a.dkeys[i] = key; a.dslot[i] = slot; }
        }
      }
      if (!a.halo && !count_cached(cc_tag, cc_cnt, slot, solo ? 0x10001u : 1u)) {  // a crowded set: global atomics
        atomicAdd(&crowded, 1u);
        atomicAdd(&a.dict_launches[slot], 1u);
        if (solo) atomicAdd(&a.dict_solo[slot], 1u);
      }
      if (end < start || end - start >= 0x80000000ull) err |= kErrRecord;
      if (start < prev && !(a.halo && r == 0)) {
        err |= kErrUnordered;
        if (ld_relaxed_gpu_u64(&a.ctl->descents) < kMaxRuns) {  // (an old answer: one more than needed)
          const unsigned long long at = atomicAdd(&a.ctl->descents, 1ull);
          if (at < kMaxRuns) a.run_starts[at] = (uint32_t)r;
        }
      }
      const uint32_t dur = (uint32_t)(end - start);
      const uint32_t meta = slot | (w1.w & (kMetaSoloBit | 0xFF000000u));
      a.tl_start[r] = start;
      a.tl_dm[r] = (unsigned long long)dur | ((unsigned long long)meta << 32);
      if (a.keys_out) a.keys_out[r] = key;
      max_dur = max(max_dur, dur);
      // Control::min_start / max_start: of an ordered trace they are the first and the last start.  An unordered one
      // gets them from a pass of its own (the host runs it when the order flag comes back set).
      if (r == 0) atomicMin(&a.ctl->min_start, start);
      if (r == a.n - 1) atomicMax(&a.ctl->max_start, start);
    }
    // solo launches join the queue: one counter update per warp
    if (solo_ballot) {
      uint32_t at = 0;
      const uint32_t first = __ffs(solo_ballot) - 1;
      if (lane == first) at = atomicAdd(&solo_n, (uint32_t)__popc(solo_ballot));
      at = __shfl_sync(0xFFFFFFFFu, at, first);
      if (solo_ballot >> lane & 1u) solo_q[at + __popc(solo_ballot & lanemask_lt())] = (unsigned long long)slot | ((end - start) << 32);
    }

    // everyone is done with this stage's tile; every thread counts the queue for itself (the counter in shared memory may
    // already be at work for the next tile when a slow warp gets here)
    waiting += (uint32_t)__syncthreads_count(solo_ballot >> lane & 1u);
    if (tid == 0) {
      const uint64_t next = tile + (uint64_t)kDecodeStages * gridDim.x;
      if (next < ntiles) issue(next, stage);
    }
    const bool last = tile + gridDim.x >= ntiles;
    if (waiting > kSoloQueue - kDecodeTile || (last && waiting)) {  // a tile more might not fit
      if (tid == 0) { solo_base = atomicAdd(&a.ctl->n_solo, waiting); solo_n = 0; }
      __syncthreads();
      const uint32_t base = solo_base;
      for (uint32_t i = tid; i < waiting; i += kDecodeThreads) a.solo_stream[base + i] = solo_q[i];
      __syncthreads();  // the queue may be filled again
      waiting = 0;
    }
    // The count cache takes keys first come, first served.  A trace whose key mix changes (one tenant's solo run, then
    // another's, then all of them together) would leave it full of keys that no longer occur, and the hottest keys of the
    // later mix would all go to the same few global counters.  So it is emptied when clearly more records find no room than
    // did at first, and refills with the keys of the stretch at hand, the frequent ones first.  (Emptying it every 40 tiles
    // instead costs 3 to 5 %, never emptying it doubles the time of logs one behind the other.)
    bool flush = last;
    if (!last && (it + 1) % kCountCheckTiles == 0) {
      __syncthreads();  // (the next tile's records are not counted yet: every thread sees the same number)
      const uint32_t now = crowded;
      __syncthreads();
      if (tid == 0 && now) atomicSub(&crowded, now);
      flush = it + 1 - flushed >= kCountFlushTiles;
      if (it + 1 - flushed <= kCountCheckTiles) usual = now;
      else flush = flush || now > 2 * usual + kDecodeTile;
    }
    if (flush) {
      flushed = it + 1;
      for (uint32_t i = tid; i < kCtaCountSlots; i += kDecodeThreads) {
        const uint32_t tag = cc_tag[i], c = cc_cnt[i];
        if (tag) {
          const uint32_t s = count_slot(i, tag);
          atomicAdd(&a.dict_launches[s], c & 0xFFFFu);
          if (c >> 16) atomicAdd(&a.dict_solo[s], c >> 16);
          cc_tag[i] = 0; cc_cnt[i] = 0;
        }
      }
      __syncthreads();
    }
  }

  // flush per-thread reductions
  err = __reduce_or_sync(0xFFFFFFFFu, err);
  max_dur = warp_max(max_dur);
  if (lane == 0) {
    if (err) atomicOr(&a.ctl->err, err);
    if (max_dur) atomicMax(&a.ctl->max_dur, max_dur);
  }
}

constexpr size_t decode_smem_bytes() { return kDecodeStages * kDecodeTileBytes + kSoloQueue * 8 + kDecodeStages * 8 + kHomeKeys * 8 + kCtaCountSlots * 6; }

}  // namespace ks
