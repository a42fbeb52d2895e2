// Walks the loops of ks_strided.h at their longest: prints nothing and returns 0 if every index is met once, in order.
#include <cstdio>
#include <cstdlib>
#include <initializer_list>

#include "ks_strided.h"

static const uint32_t kThreads = 256;

static int walk(uint32_t n, uint32_t tid) {
  uint64_t want = tid;  // the next index that has to come
  bool bad = false;
  auto take = [&](size_t i) { bad = bad || i != want || i >= n; want = i + kThreads; };
  auto step = [&](size_t i) {
    take(i);
    if (bad) { std::printf("n %u thread %u: index %zu\n", n, tid, i); std::exit(1); }
  };
  ks::strided(n, tid, kThreads, [&](size_t i) { for (int u = 0; u < 4; ++u) step(i + (size_t)kThreads * u); }, step);
  if (want < n) { std::printf("n %u thread %u: ends before %llu\n", n, tid, (unsigned long long)want); return 1; }
  return 0;
}

int main() {
  const uint32_t sizes[] = {0, 1, 255, 256, 257, 767, 768, 769, 1023, 1024, 1025, 5000, 0x7FFFFFFFu, 0xFFFFFC00u, 0xFFFFFC01u, 0xFFFFFD00u, 0xFFFFFFFFu};
  const uint32_t threads[] = {0, 1, 255};
  for (uint32_t n : sizes)
    for (uint32_t t : threads)
      if (walk(n, t)) return 1;
  const uint32_t chunk = 4096;
  for (uint32_t n : {0u, 1u, 4095u, 4096u, 4097u, 0xFFFFF000u, 0xFFFFF001u, 0xFFFFFFFFu})
    if (ks::chunk_count(n, chunk) != (uint32_t)(((uint64_t)n + chunk - 1) / chunk)) { std::printf("chunks of %u\n", n); return 1; }
  return 0;
}
