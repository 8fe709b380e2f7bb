// Host test of csrc/t1_shape.h: the autotuner's candidates are launches that differ, and the rule
// of the auto form moves with the number of SMs.
#include <cstdio>
#include <set>
#include <utility>

#include "../jpeg2000-decoder_b200/csrc/t1_shape.h"

using namespace j2k;

static int g_bad = 0;
#define CHECK(c)                                    \
  do {                                              \
    if (!(c)) {                                     \
      ++g_bad;                                      \
      std::printf("line %d: %s\n", __LINE__, #c);   \
    }                                               \
  } while (0)

int main() {
  for (int n : {0, 1, 147, 148, 149, 296, 297, 444, 592, 593, 1184, 1185, 4736, 100000}) {
    std::set<std::pair<int, int>> shapes;
    const auto all = t1_candidates(n, 148);
    bool latency = false;
    for (const T1Shape &s : all) {
      CHECK(s.warps == 2 || s.warps == 4 || s.warps == 8);
      shapes.insert({s.form, t1_most_warps(s.form, s.warps, n, 148)});
      latency = latency || s.form == T1_LATENCY;
    }
    CHECK(shapes.size() == all.size());
    CHECK(latency && all.size() >= 2);
  }
  CHECK(t1_candidates(100000, 148).size() == 4);
  for (int asked : {0, 1, 2, 8}) CHECK(t1_most_warps(T1_LATENCY, asked, 100000, 148) == 1);
  CHECK(t1_most_warps(T1_COMPACT, 0, 100000, 148) == 8 && t1_most_warps(T1_COMPACT, 3, 100000, 148) == 3);
  CHECK(t1_most_warps(T1_COMPACT, 100, 100000, 148) == 8 && t1_most_warps(T1_COMPACT, 8, 300, 148) == 3);
  // one block in a short queue; a long queue with a short, then a long chain
  CHECK(t1_auto_form(1, 2, 148, 1000, 1000, 10) == T1_LATENCY);
  CHECK(t1_auto_form(2 * 148 * 32, 2, 148, 1u << 30, 1000, 10) == T1_LATENCY);
  CHECK(t1_auto_form(2 * 148 * 32 + 1, 2, 148, 1u << 30, 1000, 10) == T1_COMPACT);
  // 4 MB take 3077 us; the chains 1070 us (2.2 times: 2354) and 1800 us (3960)
  CHECK(t1_auto_form(2 * 148 * 32 + 1, 2, 148, 4000000, 1000, 10) == T1_COMPACT);
  CHECK(t1_auto_form(2 * 148 * 32 + 1, 2, 148, 4000000, 2000, 10) == T1_LATENCY);
  // half the SMs take a queue twice as long for the same chain: its border lies at half the bytes
  for (uint64_t coded = 1000; coded < 20000000; coded += 997)
    CHECK(t1_auto_form(100000, 1, 148, 2 * coded, 1500, 20) == t1_auto_form(100000, 1, 74, coded, 1500, 20));
  std::printf(g_bad ? "%d BAD\n" : "ALL OK\n", g_bad);
  return g_bad != 0;
}
