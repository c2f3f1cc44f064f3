// CopyPool (copy_pool.h) without a GPU: copies of odd sizes by several threads
// at once give the source's bytes and touch nothing beside them, also when no
// memory can be had for a copy's job, in which case copy() must not throw.
// Prints "ok" and returns 0.
#include <cstdio>
#include <cstdlib>

#include "copy_pool.h"

static thread_local bool no_memory = false;
static std::atomic<unsigned> refused{0};

void *operator new(std::size_t n) {
  if (no_memory) {
    refused++;
    throw std::bad_alloc();
  }
  void *p = std::malloc(n);
  if (p == nullptr) throw std::bad_alloc();
  return p;
}
void operator delete(void *p) noexcept { std::free(p); }
void operator delete(void *p, std::size_t) noexcept { std::free(p); }

static bool copies_right(rfmm::CopyPool &pool, size_t bytes, bool starved) {
  constexpr size_t kRim = 64;
  std::vector<uint8_t> src(bytes), dst(bytes + 2 * kRim, 0xA5);
  for (size_t i = 0; i < bytes; i++) src[i] = (uint8_t)(i * 2654435761u >> 13);
  no_memory = starved;
  bool threw = false;
  try {
    pool.copy(dst.data() + kRim, src.data(), bytes);
  } catch (...) {
    threw = true;
  }
  no_memory = false;
  bool rim = true;
  for (size_t i = 0; i < kRim; i++) rim = rim && dst[i] == 0xA5 && dst[bytes + kRim + i] == 0xA5;
  return !threw && rim && std::memcmp(dst.data() + kRim, src.data(), bytes) == 0;
}

int main() {
  const size_t sizes[] = {0, 1, 32, (1u << 20) - 1, 1u << 20, (1u << 20) + 1, (3u << 20) + 12345, 9000032};
  std::atomic<unsigned> bad{0};
  for (unsigned helpers : {0u, 1u, 3u}) {
    rfmm::CopyPool pool;
    pool.start(helpers);
    std::vector<std::thread> callers;
    for (int t = 0; t < 4; t++)
      callers.emplace_back([&, t] {
        for (int round = 0; round < 6; round++)
          for (size_t bytes : sizes)
            if (!copies_right(pool, bytes, (round + t) % 3 == 0)) bad++;
      });
    for (auto &c : callers) c.join();
  }
  if (bad != 0 || refused == 0) {
    std::printf("%u wrong copies, %u refused allocations\n", bad.load(), refused.load());
    return 1;
  }
  std::printf("ok\n");
  return 0;
}
