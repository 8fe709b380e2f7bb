/*
 * t1_shape.h — launch shapes of the one-block-per-warp Tier-1 forms: which form a queue takes, the
 * warps of a CTA, and what the autotuner times.
 */
#ifndef J2K_T1_SHAPE_H
#define J2K_T1_SHAPE_H

#include <algorithm>
#include <cstdint>
#include <vector>

namespace j2k {

enum { T1_COMPACT = 1, T1_LATENCY = 2 };

// Most warps of a CTA for a queue of n code-blocks, `asked` of them being set by the caller (0: no
// bound of their own).  A queue shorter than the resident warps is spread over all SMs: its time is
// that of its longest blocks, which two warps of one scheduler would lengthen.  The latency form
// always has one: its shared-memory addresses are constants then.
inline int t1_most_warps(int form, int asked, int n, int sms) {
  if (form == T1_LATENCY) return 1;
  const int spread = std::max(1, (n + sms - 1) / sms);
  return std::min(spread, asked > 0 ? std::min(8, asked) : 8);
}

// The auto form without an autotuned choice: the latency form while the queue holds at most
// `waves` blocks per resident warp slot of the GPU, and for longer queues while the serial chain
// of the longest block still dominates: the compact form takes twice as long for it, and that is
// paid back only once the whole queue takes about 2.2 times as long as the chain.  Measured Tier-1
// ms, latency / compact form: 4096x2160 12-bit 9/7 pictures x2 3.95 / 7.27, x4 6.25 / 8.22, x6
// 9.27 / 9.98; 2048x2048 9/7 x8 4.43 / 8.05; 1080p 9/7 frames x8 3.90 / 4.01, x10 4.82 / 4.50,
// x24 11.46 / 9.58; 1080p lossless x6 12.54 / 12.29.  (Chain: 0.73 us a coded byte and 34 us a
// pass; the compact form takes 1.3 MB of coded bytes a ms on 148 SMs.)
inline int t1_auto_form(int64_t n, int waves, int sms, uint64_t coded, uint32_t longest, uint32_t longest_passes) {
  const double chain_us = 0.73 * longest + 34.0 * longest_passes, queue_us = coded / 1300.0 * 148 / sms;
  return n <= (int64_t)waves * sms * 32 || queue_us < 2.2 * chain_us ? T1_LATENCY : T1_COMPACT;
}

// What the autotuner times for a queue of n code-blocks: every launch shape once.  The widths 2, 4
// and 8 of the compact form are the same shape while the queue does not fill them, and the latency
// form has no width (the number beside it means nothing).
struct T1Shape {
  int form, warps;
};
inline std::vector<T1Shape> t1_candidates(int n, int sms) {
  std::vector<T1Shape> out;
  int last = 0;
  for (int warps : {2, 4, 8}) {
    const int most = t1_most_warps(T1_COMPACT, warps, n, sms);
    if (most != last) out.push_back({T1_COMPACT, warps});
    last = most;
  }
  out.push_back({T1_LATENCY, 2});
  return out;
}

}  // namespace j2k
#endif
