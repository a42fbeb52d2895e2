// ks_strided.h -- index arithmetic of loops over up to 2^32 - 1 values: plain C++, so that its bounds can be checked on the host.
#pragma once

#include <cstddef>
#include <cstdint>

#ifdef __CUDACC__
#define KS_INDEX_FN __device__ __forceinline__
#else
#define KS_INDEX_FN inline
#endif

namespace ks {

// chunks of `chunk` values in a row of cnt values (cnt + chunk - 1 would wrap for the longest rows)
KS_INDEX_FN uint32_t chunk_count(uint32_t cnt, uint32_t chunk) { return cnt / chunk + (cnt % chunk ? 1u : 0u); }

// The values i < n of thread tid out of `threads`: i = tid, tid + threads, ...  four(i) takes i and the next three while all of
// them are below n, one(i) the last ones.  The index has 64 bits: within 4 * threads of 2^32 a 32-bit one would wrap to a
// small number that passes the test again, and the loop would never end.
template <class Four, class One>
KS_INDEX_FN void strided(uint32_t n, uint32_t tid, uint32_t threads, Four four, One one) {
  size_t i = tid;
  for (; i + 3 * (size_t)threads < n; i += 4 * (size_t)threads) four(i);
  for (; i < n; i += threads) one(i);
}

}  // namespace ks
