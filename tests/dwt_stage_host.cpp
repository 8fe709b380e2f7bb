// Host build of the inverse DWT's window staging (jpeg2000-decoder_b200/csrc/dwt_kernel.cuh) for
// the CPU tests: every copy that a CTA's threads issue for one window is noted instead of made.
#include <algorithm>
#include <cstdint>
#include <cstring>
#include <vector>

#define __device__
#define __host__
#define __global__
#define __shared__
#define __forceinline__ inline
#define __restrict__
#define __align__(n) alignas(n)
#define __launch_bounds__(...)
#define J2K_DWT_LEVELS_ONLY
using std::max;
using std::min;
struct Index { int x; };
static Index threadIdx, blockIdx, blockDim, gridDim;
static inline float __fadd_rn(float a, float b) { return a + b; }
static inline float __fsub_rn(float a, float b) { return a - b; }
static inline float __fmul_rn(float a, float b) { return a * b; }
static inline void __syncthreads() {}
static const char *g_tile;
static inline size_t __cvta_generic_to_shared(const void *p) { return (const char *)p - g_tile; }
static void host_stage_copy(uint32_t to, const void *from);

#include "../jpeg2000-decoder_b200/csrc/dwt_kernel.cuh"

using namespace j2k_dev;

namespace {
// addresses only: nothing is read through them
const uintptr_t QUAD = (uintptr_t)1 << 40, LL = (uintptr_t)1 << 41;
struct Copy {
  uint32_t to;
  uintptr_t from;
};
std::vector<Copy> g_copies;

template <int TILE>
void stage(int w, int h, int stride, int stride_ll, int ox, int oy) {
  static DwtSmem<true, TILE> S;
  g_tile = (const char *)S.tile;
  g_copies.clear();
  const WinSrc<true> src{(const int32_t *)QUAD, stride, (const int32_t *)LL, stride_ll};
  for (threadIdx.x = 0; threadIdx.x < DWT_THREADS; ++threadIdx.x)
    dwt_stage<true, TILE>(&S, 1, &src, w, h, (w + 1) / 2, (h + 1) / 2, ox, oy);
}

// the element a copy reads: bit 30 set in the LL buffer, row in bits 15.., column below; -1 when it
// lies outside the level's w x h samples (LL buffer: its low part)
int element(uintptr_t from, int w, int h, int stride, int stride_ll) {
  const bool ll = from >= LL - (1 << 30);
  const int64_t off = (int64_t)(from - (ll ? LL : QUAD));
  const int st = ll ? stride_ll : stride, nw = ll ? (w + 1) / 2 : w, nh = ll ? (h + 1) / 2 : h;
  if (off < 0 || off % 4) return -1;
  const int64_t y = off / 4 / st, x = off / 4 % st;
  return y < nh && x < nw ? (int)(ll << 30 | y << 15 | x) : -1;
}
}  // namespace

static void host_stage_copy(uint32_t to, const void *from) { g_copies.push_back({to, (uintptr_t)from}); }

// The window of the tile at (ox, oy): N x N elements read, row-major (see element); -2 where
// nothing is staged.  Returns N, or -1 when a copy lands outside the window or twice.
template <int TILE>
static int window(int w, int h, int stride, int stride_ll, int ox, int oy, int32_t *out) {
  constexpr int N = DwtSmem<true, TILE>::N, PITCH = DwtSmem<true, TILE>::PITCH;
  stage<TILE>(w, h, stride, stride_ll, ox, oy);
  std::fill(out, out + N * N, -2);
  for (const Copy &c : g_copies) {
    const uint32_t at = c.to / 4, y = at / PITCH, x = at % PITCH;
    if (c.to % 4 || y >= (uint32_t)N || x >= (uint32_t)N || out[y * N + x] != -2) return -1;
    out[y * N + x] = element(c.from, w, h, stride, stride_ll);
  }
  return N;
}
extern "C" int dwt_stage_host_window(int tile, int w, int h, int stride, int stride_ll, int ox, int oy, int32_t *out) {
  return tile == 64 ? window<64>(w, h, stride, stride_ll, ox, oy, out)
                    : window<32>(w, h, stride, stride_ll, ox, oy, out);
}

// Copies from outside the level over every tile of a w x h level (rows as long as the level)
extern "C" int64_t dwt_stage_host_outside(int tile, int w, int h) {
  int64_t bad = 0;
  for (int oy = 0; oy < h; oy += tile)
    for (int ox = 0; ox < w; ox += tile) {
      if (tile == 64) stage<64>(w, h, w, (w + 1) / 2, ox, oy);
      else stage<32>(w, h, w, (w + 1) / 2, ox, oy);
      for (const Copy &c : g_copies) bad += element(c.from, w, h, w, (w + 1) / 2) < 0;
    }
  return bad;
}
