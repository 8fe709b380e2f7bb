// Host test of csrc/host_copy.h: concurrent copies are whole, their threads are bounded together,
// thread numbers of one call do not overlap, and a failed piece ends its call only.
#include <chrono>
#include <condition_variable>
#include <cstdint>
#include <cstdio>
#include <cstring>
#include <mutex>
#include <set>

#include "../jpeg2000-decoder_b200/csrc/host_copy.h"

static std::atomic<int> g_bad{0};
#define CHECK(c)                                    \
  do {                                              \
    if (!(c)) {                                     \
      ++g_bad;                                      \
      std::printf("line %d: %s\n", __LINE__, #c);   \
    }                                               \
  } while (0)

// Threads that copy at the same time in `callers` concurrent calls, at most
static int most_at_once(int callers) {
  const size_t bytes = 24 * j2k::COPY_PIECE + 12345;
  std::atomic<int> now{0}, most{0}, started{0};
  std::vector<std::thread> th;
  for (int k = 0; k < callers; ++k)
    th.emplace_back([&, k] {
      std::vector<uint8_t> src(bytes), dst(bytes);
      for (size_t i = 0; i < bytes; ++i) src[i] = (uint8_t)(i * 31 + (i >> 13) + k);
      std::atomic<bool> busy[j2k::COPY_THREADS] = {};
      ++started;
      while (started < callers) std::this_thread::yield();
      const bool ok = j2k::copy_in_pieces(bytes, [&](int t, size_t off, size_t len) {
        CHECK(t >= 0 && t < j2k::COPY_THREADS && !busy[t].exchange(true));
        const int n = ++now;
        for (int m = most; n > m && !most.compare_exchange_weak(m, n);) {}
        std::this_thread::sleep_for(std::chrono::milliseconds(3));
        std::memcpy(&dst[off], &src[off], len);
        --now;
        busy[t] = false;
        return true;
      });
      CHECK(ok && src == dst);
    });
  for (auto &x : th) x.join();
  return most;
}

int main() {
  const int cores = (int)std::max(1u, std::thread::hardware_concurrency());
  const int one = std::min(j2k::COPY_THREADS, cores);
  const int alone = most_at_once(1);
  CHECK(alone <= one && (one == 1 || alone > 1));
  CHECK(most_at_once(12) <= 12 + j2k::COPY_HELPERS);
  // the helpers are back, also after a failed call
  for (int i = 0; i < 5; ++i) {
    std::atomic<int> calls{0};
    CHECK(!j2k::copy_in_pieces(24 * j2k::COPY_PIECE, [&](int, size_t off, size_t) {
      ++calls;
      return off != 0;
    }));
    CHECK(calls >= 1 && calls <= 24);
  }
  j2k::CopyHelpers all(1000);
  CHECK(all.count() == j2k::COPY_HELPERS);
  CHECK(most_at_once(3) <= 3);  // none left: the callers copy alone
  std::printf(g_bad ? "%d BAD\n" : "ALL OK\n", (int)g_bad);
  return g_bad != 0;
}
