// Host build of the one-block-per-warp Tier-1 decoder (jpeg2000-decoder_b200/csrc/
// t1_kernel.cuh) for the CPU tests.  The 32 lanes are fibers: each runs until it reaches a
// warp-wide operation (ballot, any, sync) and waits there for the others, so the lanes'
// shared-memory traffic between two such points is that of the device, in lane order.
// The context slots, which every lane updates alike, are private to each lane here (on the
// device the warp updates them in lock-step).
#include <setjmp.h>
#include <ucontext.h>

#include <algorithm>
#include <cstdint>
#include <cstdlib>
#include <cstring>
#include <vector>

#define __device__
#define __host__
#define __forceinline__ inline
#define __restrict__
using std::max;
using std::min;
struct uint2 { uint32_t x, y; };
struct alignas(16) uint4 { uint32_t x, y, z, w; };
static inline uint4 make_uint4(uint32_t x, uint32_t y, uint32_t z, uint32_t w) { return {x, y, z, w}; }
static inline uint2 make_uint2(uint32_t x, uint32_t y) { return {x, y}; }
static inline int __popc(uint32_t x) { return __builtin_popcount(x); }
static inline int __clz(uint32_t x) { return x ? __builtin_clz(x) : 32; }
static inline int __ffs(uint32_t x) { return __builtin_ffs((int)x); }
static inline uint32_t __brev(uint32_t x) {
  uint32_t r = 0;
  for (int i = 0; i < 32; ++i) r |= ((x >> i) & 1u) << (31 - i);
  return r;
}
static inline uint32_t __funnelshift_r(uint32_t lo, uint32_t hi, uint32_t n) {
  return (uint32_t)(((uint64_t)hi << 32 | lo) >> (n & 31));
}
static inline uint32_t __funnelshift_l(uint32_t lo, uint32_t hi, uint32_t n) {
  return (uint32_t)(((uint64_t)hi << 32 | lo) << (n & 31) >> 32);
}
static inline uint32_t __byte_perm(uint32_t a, uint32_t b, uint32_t s) {
  const uint64_t v = (uint64_t)b << 32 | a;
  uint32_t r = 0;
  for (int i = 0; i < 4; ++i) r |= (uint32_t)(v >> (8 * ((s >> (4 * i)) & 7)) & 0xFF) << (8 * i);
  return r;
}
template <typename T>
static inline T __ldg(const T *p) { return *p; }
static inline void atomicXor(unsigned int *p, unsigned int v) { *p ^= v; }

namespace {
constexpr int LANES = 32;
// started through a context, switched by _setjmp / _longjmp (no signal-mask system calls)
ucontext_t g_main, g_lane[LANES];
jmp_buf g_main_at, g_lane_at[LANES];
bool g_started[LANES];
std::vector<char> g_stack[LANES];
bool g_done[LANES];
int g_cur = 0;
uint32_t g_arg[2][LANES];
unsigned g_phase[LANES];
// one warp-wide operation: leave the argument, let every other lane arrive, read them all
const uint32_t *exchange(uint32_t v) {
  const unsigned ph = g_phase[g_cur]++ & 1;
  g_arg[ph][g_cur] = v;
  if (!_setjmp(g_lane_at[g_cur])) _longjmp(g_main_at, 1);
  return g_arg[ph];
}
void resume(int lane) {
  if (_setjmp(g_main_at)) return;
  if (g_started[lane]) _longjmp(g_lane_at[lane], 1);
  g_started[lane] = true;
  swapcontext(&g_main, &g_lane[lane]);
}
}  // namespace
static inline uint32_t __ballot_sync(uint32_t, uint32_t pred) {
  const uint32_t *a = exchange(pred != 0);
  uint32_t r = 0;
  for (int i = 0; i < LANES; ++i) r |= (a[i] & 1u) << i;
  return r;
}
static inline int __any_sync(uint32_t, uint32_t pred) { return __ballot_sync(0, pred) != 0; }
static inline void __syncwarp() { exchange(0); }
template <typename T>
static inline T __shfl_sync(uint32_t, T v, int from) { return (T)exchange((uint32_t)v)[from & 31]; }

#include "../jpeg2000-decoder_b200/csrc/t1_kernel.cuh"

using namespace j2k_dev;

namespace {
struct Job {
  const j2k_cblk *cb;
  const uint8_t *bytes;
  const uint32_t *seglens;
  Block b[LANES];
  int plane, passes, latency, status[LANES];
} g_job;

void lane_main(int lane) {
  Block &b = g_job.b[lane];
  g_job.status[lane] =
      g_job.latency ? decode_block<true>(*g_job.cb, g_job.bytes, g_job.seglens, b, g_job.plane, g_job.passes)
                    : decode_block<false>(*g_job.cb, g_job.bytes, g_job.seglens, b, g_job.plane, g_job.passes);
  g_done[lane] = true;
  _longjmp(g_main_at, 1);
}
}  // namespace

// Decodes `cb` into out (cb->w * cb->h raw sign-magnitude samples, row-major): the block
// status, or -2 when the lanes end apart from one another.
extern "C" int t1_warp_host_block(const j2k_cblk *cb, const uint8_t *bytes, const uint32_t *seglens, int latency,
                                  int32_t *out) {
  static T1Tables T;
  static bool ready = false;
  if (!ready) {
    build_t1_tables(T);
    ready = true;
  }
  typedef T1Layout<64, 64> Lay;
  // exactly the device's area, filled with garbage, in allocations of their own size
  uint8_t *mem = (uint8_t *)aligned_alloc(16, Lay::PER_WARP);
  std::memset(mem, 0xA5, Lay::PER_WARP);
  uint8_t *slots = (uint8_t *)aligned_alloc(16, (size_t)LANES * (Lay::BITS - Lay::CX));
  std::vector<int32_t> img((size_t)cb->w * cb->h, 0x5A5A5A5A);
  j2k_cblk c = *cb;
  g_job.cb = &c;
  g_job.bytes = bytes;
  g_job.seglens = seglens;
  g_job.latency = latency;
  block_planes(c, g_job.plane, g_job.passes);
  for (int l = 0; l < LANES; ++l) {
    Block &b = g_job.b[l];
    b.lane = l;
    b.w = c.w;
    b.gap = c.w + 3;
    b.stripes = (c.h + 3) >> 2;
    b.cw = reinterpret_cast<uint32_t *>(mem) + b.gap + 1;
    b.rf = reinterpret_cast<uint4 *>(mem + Lay::RF);
    b.cx = slots + (size_t)l * (Lay::BITS - Lay::CX);
    b.bits = reinterpret_cast<uint32_t *>(mem + Lay::BITS);
    b.list = mem + Lay::LIST;
    b.mq = reinterpret_cast<const uint8_t *>(T.mq);
    b.sc = T.sc;
    b.zc = T.zc[c.band == 3 ? 2 : (c.band == 1 ? 1 : 0)];
    b.out = reinterpret_cast<uint32_t *>(img.data());
    b.stride = c.w;
    g_done[l] = g_started[l] = false;
    g_phase[l] = 0;
    g_stack[l].resize(64 << 10);
    getcontext(&g_lane[l]);
    g_lane[l].uc_stack.ss_sp = g_stack[l].data();
    g_lane[l].uc_stack.ss_size = g_stack[l].size();
    g_lane[l].uc_link = &g_main;
    makecontext(&g_lane[l], (void (*)())lane_main, 1, l);
  }
  int rc = 0;
  for (;;) {
    int done = 0;
    for (g_cur = 0; g_cur < LANES; ++g_cur) {
      if (!g_done[g_cur]) resume(g_cur);
      done += g_done[g_cur];
    }
    if (done == LANES) break;
    if (done) {
      rc = -2;
      break;
    }
  }
  for (int l = 1; l < LANES; ++l)
    if (g_phase[l] != g_phase[0] || g_job.status[l] != g_job.status[0]) rc = -2;
  if (!rc) rc = g_job.status[0];
  const Block &b = g_job.b[0];
  for (int y = 0; y < c.h; ++y)
    for (int x = 0; x < c.w; ++x)
      out[y * c.w + x] = (b.cw[(y >> 2) * b.gap + x] >> (SIG_POS + 3 * (y & 3))) & 1 ? img[(size_t)y * c.w + x] : 0;
  free(mem);
  free(slots);
  return rc;
}

// An MQ encoder (T.800 C.2) of seeded symbols in 19 contexts, decoded again as the passes take
// symbols: in pairs (a refill before the first, a level check between the two) or alone.  The
// symbols are steered to bytes of 0xFF and then to carries into the byte after them.  Returns the number of symbols decoded wrongly; *carries the bytes above
// 0x7F after a 0xFF.
extern "C" int t1_warp_host_symbols(uint32_t seed, int n, int cut, int latency, int *carries) {
  static T1Tables T;
  build_t1_tables(T);
  const uint8_t *tab = reinterpret_cast<const uint8_t *>(T.mq);
  alignas(16) uint8_t cx[N_CTX * SLOT];
  auto rnd = [&] {
    seed ^= seed << 13;
    seed ^= seed >> 17;
    return seed ^= seed << 5;
  };
  std::vector<uint8_t> ctx(n), sym(n), code(1, 0);
  init_states(cx, tab);
  uint32_t A = 0x8000, C = 0, CT = 12;
  auto byteout = [&] {
    bool stuff = code.back() == 0xFF && code.size() > 1;
    if (!stuff && C >= 0x8000000) {
      code.back()++;
      if (code.back() == 0xFF) {
        C &= 0x7FFFFFF;
        stuff = true;
      }
    }
    code.push_back((uint8_t)(stuff ? C >> 20 : C >> 19));
    C &= stuff ? 0xFFFFF : 0x7FFFF;
    CT = stuff ? 7 : 8;
  };
  for (int i = 0; i < n; ++i) {
    ctx[i] = rnd() % 4 ? C_UNI : rnd() % N_CTX;
    uint2 &e = *reinterpret_cast<uint2 *>(cx + ctx[i] * SLOT);
    const uint2 *rec = reinterpret_cast<const uint2 *>(tab + (e.y & 0xFFFF));
    const uint32_t q = e.x >> 8, mps = e.y >> 31;
    A -= q;
    // the upper subinterval (C += q) goes to the MPS unless the intervals are exchanged
    const bool exchanged = !(A & 0x8000) && A < q;
    const bool up = rnd() % 8 == 0 ? rnd() & 1 : code.back() == 0xFF || C + q < 0x8000000u >> CT;
    const bool lps = up == exchanged;
    sym[i] = (uint8_t)(mps ^ lps);
    if (!lps) {
      if (A & 0x8000) {
        C += q;
        continue;
      }
      if (A < q) A = q;
      else C += q;
      e = rec[2];
    } else {
      if (A < q) C += q;
      else A = q;
      e = rec[3];
    }
    do {
      A <<= 1;
      C <<= 1;
      if (!--CT) byteout();
    } while (!(A & 0x8000));
  }
  const uint32_t top = C + A;
  C |= 0xFFFF;
  if (C >= top) C -= 0x8000;
  C <<= CT;
  byteout();
  C <<= CT;
  byteout();
  *carries = 0;
  for (size_t i = 1; i + 1 < code.size(); ++i) *carries += code[i] == 0xFF && code[i + 1] > 0x7F;
  const uint32_t len = (uint32_t)code.size() - 1;
  code.resize(len + 32, 0x5A);
  init_states(cx, tab);
  Mq m;
  mq_init(m, code.data() + 1, len);
  int wrong = 0;
  auto one = [&](int i) {
    uint8_t *slot = cx + ctx[i] * SLOT;
    uint2 e = *reinterpret_cast<uint2 *>(slot);
    wrong += is_one(latency ? mq_symbol<true>(m, slot, e, tab) : mq_symbol<false>(m, slot, e, tab)) != sym[i];
  };
  for (int i = 0; i < n;) {
    if (latency) mq_ready<true>(m);
    one(i++);
    if (i % cut == 0 || i >= n) continue;
    if (latency) mq_level<true>(m);
    one(i++);
  }
  return wrong;
}
