/*
 * dwt_kernel.cuh — inverse 5/3 and 9/7 DWT levels and the inverse MCT / DC-shift / pack
 * stage for sm_100a.
 *
 * One CTA reconstructs a 64x64 output tile of one resolution level of one
 * tile-component: it stages the 72x72 interleaved window (the four quadrants of the
 * Mallat layout plus a 4-sample whole-sample-symmetric halo) in shared memory with
 * coalesced asynchronous copies, lifts the window's rows and then its columns, a thread
 * lifting eight outputs at a time in registers, and stores the 64x64 result from the column
 * pass.  Every level is one read and one write of the level's samples; all tile-components
 * of a batch at a given level share one launch.
 * The kernels are bound by instruction issue and the latency of a tile's phases (a 4096x2160 level:
 * 67 % of the issue slots of an active SM, DRAM 1.3 TB/s), so the work is cut into short independent
 * chains, the staging walks lines with pointers, and a tile's copies run under the column pass
 * of the tile before it.  Measured on B200 against a thread per 72-sample line streamed through
 * shared memory: a 4096x2160 9/7 plane of five levels 79.8 -> 43.2 us, a 1000x777 5/3 tile
 * 45.1 -> 16.9 us (a programmatic launch per level, 32x32 tiles in the small levels), the DWT +
 * MCT stage of 32 1080p frames 0.955 -> 0.79 ms.
 *
 * Arithmetic follows the reference exactly so that results are bit-identical:
 *   9/7: each lifting update is D = S - c * (L + R) with three separately rounded float
 *        operations (bmi_cpu_dwt_decoder.cpp:2374-2385, vdwt_analyst_line :4975-4993),
 *        constants of bmi_cpu_dwt.h:31-41; the reconstructed LL entering a finer level is
 *        multiplied by K_lo*K_lo (:1599, :1626); band gains are folded in by Tier-1.
 *   5/3: x[2n] -= (x[2n-1] + x[2n+1] + 2) >> 2, x[2n+1] += (x[2n] + x[2n+2]) >> 1 with
 *        symmetric ends (:2609-2659, :3311-3534); with J2K_FLAG_REF_COMPAT the last
 *        column rows are rebuilt the way VDWT_R53_LINES does (:3364-3398).
 * A whole-sample symmetric input extension is preserved by every lifting step, so
 * mirroring the input once and lifting across the halo gives the same values as the
 * reference's per-step mirroring at the region edges.
 */
#pragma once
#include <cstdint>
#include <type_traits>

#include "plan.h"

namespace j2k_dev {

constexpr int DWT_T = 64;          // output tile edge
constexpr int DWT_H = 4;           // halo
constexpr int DWT_PITCH = DWT_T + 2 * DWT_H + 1;  // of a 64x64 tile's window

struct DwtLevel {
  uint64_t base;     // element offset of the tile-component region (same in every buffer)
  int32_t stride;    // tile-component width
  int32_t rw, rh;    // size of the resolution being rebuilt
  int32_t lw, lh;    // size of its low-pass part (resolution r-1)
  int8_t ll_src;     // buffer holding the LL quadrant: 0 coefficients, 1 B, 2 C
  int8_t out_dst;    // buffer receiving the level: 1 B, 2 C
  int8_t ll_gain;    // 9/7: scale the LL quadrant by K_lo^2 (reconstructed LL)
  int8_t refcompat;  // 5/3: reference column-end arithmetic
  int32_t tiles_x;
};

struct DwtTask {
  uint32_t level;  // index into the DwtLevel array
  uint16_t tx, ty;
};

// Output stage: one tile of one image, up to four components.
struct OutGroup {
  uint64_t comp_off[4];  // element offsets of the final component regions
  int8_t comp_buf[4];    // buffer ids (0 coefficients, 1 B, 2 C), -1 = absent
  int32_t stride[4];
  int32_t x0, y0, w, h;  // tile rectangle in the output image
  uint64_t out_off;      // byte offset of the image in the output buffer
  int32_t pitch_px;      // output width in pixels
  int16_t fmt, bitdepth;
  int8_t rev, mct, ncomp, checkout;  // checkout: reference mCheckOutComponent, -1 = all
  int32_t tiles_x;
  // sub-sampled components (SIZ XRsiz / YRsiz > 1): pixel (x0 + xx, y0 + yy) shows sample
  // (floor((ax + xx) / sx[c]) - cx[c], floor((ay + yy) / sy[c]) - cy[c]) of component c's
  // tile-component (clamped to its cw x ch samples), ax / ay being the tile's absolute
  // pixel origin and cx / cy the tile-component's absolute origin on the component's grid
  int32_t ax, ay;
  int32_t cx[4], cy[4], cw[4], ch[4];
  uint8_t sx[4], sy[4];
  int8_t sampled;
};
struct OutTask {
  uint32_t group;
  uint16_t tx, ty;
};

// Source position of window position p on a line of n samples: whole-sample symmetric
// extension, which keeps the parity on lines of two and more samples.  Positions more than four
// past the end feed no output: they are brought back to one that exists.
__device__ __forceinline__ int mirror(int p, int n) {
  if (n == 1) return 0;
  if (p > n + 3) p = n + 3 - ((n + 3 - p) & 1);
  while (p < 0 || p >= n) p = p < 0 ? -p : 2 * (n - 1) - p;
  return p;
}

// Where the part that holds a parity's samples begins on the de-interleaved line, whose low part
// has lo samples: sample mirror(p, n) lies at part_start(p & 1, n, lo) + (mirror(p, n) >> 1).  A
// line of one sample has only its low part, for odd positions as well.
__device__ __forceinline__ int part_start(int odd, int n, int lo) { return odd && n > 1 ? lo : 0; }

__device__ __forceinline__ float lift97(float s, float c, float l, float r) {
  return __fsub_rn(s, __fmul_rn(c, __fadd_rn(l, r)));
}

template <bool REV>
struct DwtTypes;
template <>
struct DwtTypes<true> {
  typedef int32_t T;
};
template <>
struct DwtTypes<false> {
  typedef float T;
};

constexpr int DWT_THREADS = 256;    // threads per CTA of the level kernels
constexpr int FUSED_THREADS = 256;  // threads per CTA of the fused last-level + output kernel

// Inverse lifting of eight outputs of a line from the fifteen samples around them, in
// registers: x[i] is position i - 3 counted from the first output (an even position), y the
// outputs.  Every update has the value of the step-by-step scheme over the whole line.  A
// thread per eight outputs repeats 6 of 22 (9/7) or 1 of 9 (5/3) updates of its neighbours, but
// the chain is four updates long; one thread per line streamed 72 samples through shared
// memory one after the other (a 64x64 tile's two passes took 4 us of latency).
constexpr int SEG = 8, SEG_IN = SEG + 7;
template <bool REV>
__device__ __forceinline__ void lift_segment(const typename DwtTypes<REV>::T *x, typename DwtTypes<REV>::T *y) {
  if constexpr (REV) {
    // x[2n] -= (x[2n-1] + x[2n+1] + 2) >> 2; x[2n+1] += (x[2n] + x[2n+2]) >> 1
    int ev[5];
#pragma unroll
    for (int k = 0; k < 5; ++k) ev[k] = x[2 * k + 3] - ((x[2 * k + 2] + x[2 * k + 4] + 2) >> 2);
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      y[2 * k] = ev[k];
      y[2 * k + 1] = x[2 * k + 4] + ((ev[k] + ev[k + 1]) >> 1);
    }
  } else {
    // steps c0 (evens), c1 (odds), c2 (evens), c3 (odds): x -= c * (left + right), each
    // operation rounded separately
    const float c0 = 0.44350685204397f, c1 = 0.88291107553093f, c2 = -0.05298011857296f, c3 = -1.58613434205992f;
    float e0[7], o1[6], e2[5];
#pragma unroll
    for (int k = 0; k < 7; ++k) e0[k] = lift97(x[2 * k + 1], c0, x[2 * k], x[2 * k + 2]);  // positions -2 .. 10
#pragma unroll
    for (int k = 0; k < 6; ++k) o1[k] = lift97(x[2 * k + 2], c1, e0[k], e0[k + 1]);  // -1 .. 9
#pragma unroll
    for (int k = 0; k < 5; ++k) e2[k] = lift97(e0[k + 1], c2, o1[k], o1[k + 1]);  // 0 .. 8
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      y[2 * k] = e2[k];
      y[2 * k + 1] = lift97(o1[k + 1], c3, e2[k], e2[k + 1]);  // 1 .. 7
    }
  }
}

template <bool REV>
__device__ __forceinline__ typename DwtTypes<REV>::T *dwt_buf(int id, void *a, void *b, void *c) {
  typedef typename DwtTypes<REV>::T T;
  return (T *)(id == 0 ? a : (id == 1 ? b : c));
}

// Shared memory of one window of a TxT output tile: the staged samples and the
// reference-compat column-end inputs.  Odd pitch: conflict-free column access.
template <bool REV, int TILE = DWT_T>
struct DwtSmem {
  static constexpr int N = TILE + 2 * DWT_H, PITCH = N + 1;
  typename DwtTypes<REV>::T tile[N * PITCH];
  typename DwtTypes<REV>::T keep[2][TILE];
};
// The rows of a level kernel's window after the row pass, in a buffer of their own: no thread
// holds its outputs while others still read (41 KB a CTA, five CTAs an SM)
template <bool REV, int TILE = DWT_T>
struct LevelSmem {
  static constexpr int MID_PITCH = TILE + 1;
  DwtSmem<REV, TILE> win;
  typename DwtTypes<REV>::T mid[DwtSmem<REV, TILE>::N * MID_PITCH];
};

// Inputs of one window: the level's Mallat quadrants (`quad`) and the LL quadrant
// (`llsrc`, another buffer for every level but the first)
template <bool REV>
struct WinSrc {
  const typename DwtTypes<REV>::T *quad;
  int stride_q;
  const typename DwtTypes<REV>::T *llsrc;
  int stride_ll;
};

// One asynchronous copy of the staging, `to` a shared-memory address
template <typename T>
__device__ __forceinline__ void stage_copy(uint32_t to, const T *from) {
#ifdef __CUDACC__
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4;\n" ::"r"(to), "l"(from));
#else
  host_stage_copy(to, from);  // of the including file
#endif
}

// Stage the window of the tile at (ox, oy) with asynchronous 4-byte copies: every thread issues
// all of its loads before waiting.  A warp copies a window row: lane l holds positions l,
// l + 32 and l + 64 (as far as the row goes), even ones from the low part and odd ones from the
// high part of the line (64 contiguous bytes of each per copy).  The warps' number is even, so the
// parity of a lane's columns and of a warp's rows never changes: a lane and warp of even parity
// take LL, the others the level's quadrants (a line of one sample has only its low part, which
// odd positions then read as well; no output comes from them), and inside the level a warp's
// pointers advance by whole lines.
enum { STAGE_DETAIL = 1, STAGE_LL = 2 };  // the quadrants to stage
template <bool REV, int TILE, int WHICH = STAGE_DETAIL | STAGE_LL>
__device__ __forceinline__ void dwt_stage(DwtSmem<REV, TILE> *S, int nw, const WinSrc<REV> *src, int rw, int rh, int lw,
                                          int lh, int ox, int oy) {
  typedef typename DwtTypes<REV>::T T;
  constexpr int N = DwtSmem<REV, TILE>::N, PITCH = DwtSmem<REV, TILE>::PITCH, COLS = (N + 31) / 32;
  constexpr int WARPS = DWT_THREADS / 32;
  static_assert(DWT_THREADS == FUSED_THREADS && WARPS % 2 == 0 && N % WARPS == 0, "rows are dealt to an even number of warps");
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int odd = lane & 1, high = warp & 1;
  if (!(WHICH & (odd || high ? STAGE_DETAIL : STAGE_LL))) return;
  int col[COLS];
#pragma unroll
  for (int j = 0; j < COLS; ++j) col[j] = (mirror(ox - DWT_H + lane + 32 * j, rw) >> 1) + part_start(odd, rw, lw);
  const bool last = lane < N - 32 * (COLS - 1);
  const bool inside = oy >= DWT_H && oy + TILE + DWT_H <= rh;
  for (int w = 0; w < nw; ++w) {
    const bool ll = !high && !odd;
    const T *base = ll ? src[w].llsrc : src[w].quad + (size_t)part_start(high, rh, lh) * src[w].stride_q;
    const int stride = ll ? src[w].stride_ll : src[w].stride_q;
    const uint32_t d0 = (uint32_t)__cvta_generic_to_shared(S[w].tile + warp * PITCH + lane);
    auto copy = [&](const T *line, uint32_t d) {
#pragma unroll
      for (int j = 0; j < COLS; ++j)
        if (j < COLS - 1 || last) stage_copy(d + 128 * j, line + col[j]);
    };
    if (inside) {
      const T *line = base + (size_t)((oy - DWT_H + warp) >> 1) * stride;
      const size_t step = (size_t)(WARPS / 2) * stride;
#pragma unroll
      for (int i = 0; i < N / WARPS; ++i, line += step) copy(line, d0 + 4 * PITCH * WARPS * i);
    } else {
#pragma unroll 1
      for (int i = 0; i < N / WARPS; ++i)
        copy(base + (size_t)(mirror(oy - DWT_H + warp + WARPS * i, rh) >> 1) * stride, d0 + 4 * PITCH * WARPS * i);
    }
  }
}

// Rebuild the TILE x TILE output tile at (ox, oy) of one level for `nw` windows of the same
// geometry (the components of one tile at their last level, or one tile-component).  The
// results are left in the centre of each window, S[w].tile[(y + 4) * PITCH + x + 4], or
// (DIRECT: a single window, its rows in `mid`) stored to `out` from the column pass.  `staged`: the
// window is already on its way; `window_free` is called once the window has been read for the
// last time (DIRECT: the next tile's copies then run under the column pass).
template <bool REV, bool DIRECT, int TILE, class F>
__device__ __forceinline__ void dwt_windows(DwtSmem<REV, TILE> *S, int nw, const WinSrc<REV> *src, int rw, int rh, int lw,
                                            int lh, bool ll_gain, float gain, bool refcompat, int ox, int oy,
                                            typename DwtTypes<REV>::T *mid, typename DwtTypes<REV>::T *out,
                                            int stride_out, bool staged, F window_free) {
  typedef typename DwtTypes<REV>::T T;
  constexpr int N = DwtSmem<REV, TILE>::N, PITCH = DwtSmem<REV, TILE>::PITCH, MID_PITCH = TILE + 1;
  if (!staged) dwt_stage<REV, TILE>(S, nw, src, rw, rh, lw, lh, ox, oy);
  asm volatile("cp.async.wait_all;\n" ::: "memory");
  __syncthreads();
  // Rows: a thread lifts eight outputs of a row; consecutive threads take consecutive rows (the
  // odd pitch keeps the banks apart).  The reconstructed LL entering a finer 9/7 level is
  // scaled by K_lo^2 on the way.
  constexpr int SEGS = TILE / SEG, ROW_TASKS = N * SEGS;
  constexpr int RT = (ROW_TASKS + DWT_THREADS - 1) / DWT_THREADS;
  auto row_task = [&](int w, int seg, int r, T *y) {
    const T *p = S[w].tile + r * PITCH + SEG * seg + DWT_H - 3;
    T x[SEG_IN];
#pragma unroll
    for (int k = 0; k < SEG_IN; ++k) x[k] = p[k];
    if constexpr (!REV) {
      if (ll_gain) {
        const float g = !(r & 1) ? gain : 1.f;
#pragma unroll
        for (int k = 1; k < SEG_IN; k += 2) x[k] = __fmul_rn(x[k], g);
      }
    }
    if (rw > 1) {
      lift_segment<REV>(x, y);
    } else {
#pragma unroll
      for (int k = 0; k < SEG; ++k) y[k] = x[k + 3];
    }
  };
  if (DIRECT) {
#pragma unroll 1
    for (int t = threadIdx.x; t < ROW_TASKS; t += DWT_THREADS) {
      const int seg = t / N, r = t - seg * N;
      T y[SEG];
      row_task(0, seg, r, y);
      T *p = mid + r * MID_PITCH + SEG * seg;
#pragma unroll
      for (int k = 0; k < SEG; ++k) p[k] = y[k];
    }
  } else {
    // in place: the outputs wait in registers until the window's inputs have been read
    for (int w = 0; w < nw; ++w) {
      T y[RT][SEG];
#pragma unroll
      for (int i = 0; i < RT; ++i) {
        const int t = threadIdx.x + i * DWT_THREADS;
        if (t < ROW_TASKS) row_task(w, t / N, t % N, y[i]);
      }
      __syncthreads();
#pragma unroll
      for (int i = 0; i < RT; ++i) {
        const int t = threadIdx.x + i * DWT_THREADS;
        if (t < ROW_TASKS) {
          T *p = S[w].tile + (t % N) * PITCH + SEG * (t / N) + DWT_H;
#pragma unroll
          for (int k = 0; k < SEG; ++k) p[k] = y[i][k];
        }
      }
    }
  }
  __syncthreads();
  // reference-compat: keep the horizontally transformed inputs the column end reads
  const int n = rh;
  const bool fix = REV && refcompat && n >= 3 && (oy <= n - 1) && (n - 2 < oy + TILE);
  if (fix) {
    int rowA = n - 3, rowB = -1;  // H[m-2]
    if (n & 1) {
      const int m = (n + 1) / 2;
      rowA = n - 3;                 // L[m-2]
      rowB = (m >= 3) ? n - 4 : 1;  // H[m-3] (H[0] when m == 2)
    }
    for (int e = threadIdx.x; e < nw * TILE; e += blockDim.x) {
      const int w = e / TILE, c = e - w * TILE;
      const T *rows = DIRECT ? mid + c : S[w].tile + DWT_H + c;
      constexpr int pitch = DIRECT ? MID_PITCH : PITCH;
      S[w].keep[0][c] = rows[(rowA - oy + DWT_H) * pitch];
      if (rowB >= 0) S[w].keep[1][c] = rows[(rowB - oy + DWT_H) * pitch];
    }
  }
  // Columns: a thread lifts eight outputs of a column, consecutive threads consecutive columns
  constexpr int COL_TASKS = TILE * SEGS, CT = (COL_TASKS + DWT_THREADS - 1) / DWT_THREADS, STEP = DWT_THREADS / TILE;
  const int ow = min(TILE, rw - ox), oh = min(TILE, rh - oy);
  auto col_task = [&](const T *p, int pitch, T *y) {
    T x[SEG_IN];
#pragma unroll
    for (int k = 0; k < SEG_IN; ++k) x[k] = p[k * pitch];
    if (rh > 1) {
      lift_segment<REV>(x, y);
    } else {
#pragma unroll
      for (int k = 0; k < SEG; ++k) y[k] = x[k + 3];
    }
  };
  const int c = threadIdx.x % TILE;
  if (DIRECT) {
    if (!fix) window_free();
#pragma unroll 1
    for (int seg = threadIdx.x / TILE; seg < SEGS; seg += STEP) {
      T y[SEG];
      col_task(mid + (SEG * seg + DWT_H - 3) * MID_PITCH + c, MID_PITCH, y);
      if (!fix) {
        T *o = out + (size_t)(oy + SEG * seg) * stride_out + ox + c;
        const int rows = c < ow ? oh - SEG * seg : 0;
        if (rows >= SEG) {
#pragma unroll
          for (int k = 0; k < SEG; ++k, o += stride_out) *o = y[k];
        } else {
#pragma unroll
          for (int k = 0; k < SEG; ++k, o += stride_out)
            if (k < rows) *o = y[k];
        }
      } else {
        T *p = S[0].tile + (SEG * seg + DWT_H) * PITCH + DWT_H + c;
#pragma unroll
        for (int k = 0; k < SEG; ++k) p[k * PITCH] = y[k];
      }
    }
    if (!fix) return;
  } else {
    for (int w = 0; w < nw; ++w) {
      T y[CT][SEG];
#pragma unroll
      for (int i = 0; i < CT; ++i)
        col_task(S[w].tile + (SEG * (threadIdx.x / TILE + i * STEP) + DWT_H - 3) * PITCH + DWT_H + c, PITCH, y[i]);
      __syncthreads();
#pragma unroll
      for (int i = 0; i < CT; ++i) {
        T *p = S[w].tile + (SEG * (threadIdx.x / TILE + i * STEP) + DWT_H) * PITCH + DWT_H + c;
#pragma unroll
        for (int k = 0; k < SEG; ++k) p[k * PITCH] = y[i][k];
      }
    }
  }
  __syncthreads();
  if constexpr (REV) {
    if (fix) {
      for (int e = threadIdx.x; e < nw * TILE; e += blockDim.x) {
        const int w = e / TILE, cc = e - w * TILE;
        T *colp = S[w].tile + DWT_H + cc;
        const int r1 = n - 1 - oy + DWT_H, r2 = n - 2 - oy + DWT_H, r3 = n - 3 - oy + DWT_H;
        if (!(n & 1)) {
          colp[r1 * PITCH] = S[w].keep[0][cc] + colp[r2 * PITCH];
        } else {
          const T hx = S[w].keep[1][cc];
          const T x1 = S[w].keep[0][cc] - ((hx + 1) >> 1);
          colp[r1 * PITCH] = x1;
          colp[r2 * PITCH] = hx + ((x1 + colp[r3 * PITCH]) >> 1);
        }
      }
      __syncthreads();
    }
  }
  if (DIRECT) {
    for (int i = threadIdx.x; i < TILE * TILE; i += blockDim.x) {
      const int yy = i / TILE, xx = i % TILE;
      if (yy < oh && xx < ow)
        out[(size_t)(oy + yy) * stride_out + ox + xx] = S[0].tile[(yy + DWT_H) * PITCH + xx + DWT_H];
    }
    __syncthreads();
    window_free();
  }
}

// One level of one tile-component, as a tile's kernel needs it
template <bool REV>
struct LevelArgs {
  WinSrc<REV> src;
  typename DwtTypes<REV>::T *out;
  int stride_out, rw, rh, lw, lh, ox, oy;  // (ox, oy): the tile
  bool ll_gain, refcompat;
};
template <bool REV, int TILE, int WHICH = STAGE_DETAIL | STAGE_LL>
__device__ __forceinline__ void dwt_stage_tile(LevelSmem<REV, TILE> &S, const LevelArgs<REV> &a) {
  dwt_stage<REV, TILE, WHICH>(&S.win, 1, &a.src, a.rw, a.rh, a.lw, a.lh, a.ox, a.oy);
}
// Output tiles of levels, stored to their `out`, one after the other: next(args) sets the next
// tile's arguments or returns false.  The copies of a tile's window run under the column pass of
// the tile before it; the first one's are started by first(args).
template <bool REV, int TILE, class Next, class First>
__device__ __forceinline__ void dwt_tiles(LevelSmem<REV, TILE> &S, float gain, Next next, First first) {
  LevelArgs<REV> cur, ahead;
  bool more = next(cur);
  if (more) first(cur);
  while (more) {
    bool then = false;
    dwt_windows<REV, true, TILE>(&S.win, 1, &cur.src, cur.rw, cur.rh, cur.lw, cur.lh, cur.ll_gain, gain, cur.refcompat,
                                 cur.ox, cur.oy, S.mid, cur.out, cur.stride_out, true, [&] {
                                   then = next(ahead);
                                   if (then) dwt_stage_tile<REV, TILE>(S, ahead);
                                 });
    cur = ahead;
    more = then;
  }
}

template <bool REV>
__global__ void __launch_bounds__(DWT_THREADS) dwt_level_kernel(const DwtLevel *__restrict__ levels,
                                                        const DwtTask *__restrict__ tasks, int ntasks, void *bufA,
                                                        void *bufB, void *bufC, float ll_gain_value) {
  typedef typename DwtTypes<REV>::T T;
  __shared__ LevelSmem<REV> S;
  int task = blockIdx.x;
  dwt_tiles<REV, DWT_T>(S, ll_gain_value, [&](LevelArgs<REV> &a) {
    if (task >= ntasks) return false;
    const DwtTask tk = tasks[task];
    const DwtLevel L = levels[tk.level];
    task += gridDim.x;
    a.src = {dwt_buf<REV>(0, bufA, bufB, bufC) + L.base, L.stride, dwt_buf<REV>(L.ll_src, bufA, bufB, bufC) + L.base, L.stride};
    a.out = dwt_buf<REV>(L.out_dst, bufA, bufB, bufC) + L.base;
    a.stride_out = L.stride;
    a.rw = L.rw;
    a.rh = L.rh;
    a.lw = L.lw;
    a.lh = L.lh;
    a.ox = tk.tx * DWT_T;
    a.oy = tk.ty * DWT_T;
    a.ll_gain = L.ll_gain != 0;
    a.refcompat = L.refcompat != 0;
    return true;
  }, [&](const LevelArgs<REV> &a) { dwt_stage_tile<REV, DWT_T>(S, a); });
}

// ------------------------------------------------------------------ output stage -------
__device__ __forceinline__ int clampi(int v, int hi) { return v < 0 ? 0 : (v > hi ? hi : v); }
__device__ __forceinline__ int lift_depth(int v, int in, int out) { return in >= out ? v >> (in - out) : v << (out - in); }

// bytes per pixel and container depth of a reference OutputFormat
__device__ __host__ __forceinline__ int fmt_bytes(int fmt) {
  switch (fmt) {
    case 0: return 4;
    case 1: return 6;
    case 2: return 3;
    case 3: return 4;
    case 4: return 8;
    case 5: return 6;
    case 6: return 3;
    case 8: return 8;
    default: return 0;
  }
}

__device__ __forceinline__ void put_slot(uint8_t *px, int pxb, int slot, int v) {
  // reference pixel structs store the highest component index first (codec_base.h:51-143)
  if (pxb == 3) px[2 - slot] = (uint8_t)v;
  else if (pxb == 4) px[3 - slot] = (uint8_t)v;
  else if (pxb == 6) ((uint16_t *)px)[2 - slot] = (uint16_t)v;
  else ((uint16_t *)px)[3 - slot] = (uint16_t)v;
}

// Last level of every component of one tile with the output stage fused into its store:
// the components' windows stay in shared memory and the packed pixels are the only write.
struct FusedGroup {
  OutGroup G;
  uint64_t base[3];  // element offset of each component's region (same in every buffer)
  int8_t ll_src[3];  // buffer of each component's LL quadrant: 0 coefficients, 1 B, 2 C
  int8_t ll_gain, refcompat;
  int32_t stride, rw, rh, lw, lh;
};

// Inverse RCT (5/3, int) or ICT (9/7, float) + DC level shift + clamp of one pixel: R, G, B
// (RRct_53 :3936-4130, RICT_97_FLOAT :3570-3643 of bmi_cpu_dwt_decoder.cpp)
template <typename T>
__device__ __forceinline__ void mct_pixel(T y, T u, T w, int dc, int maxv, int *rgb) {
  if constexpr (std::is_integral<T>::value) {
    const int g = (int)y - (((int)u + (int)w) >> 2) + dc;
    rgb[0] = clampi((int)w + g, maxv);
    rgb[1] = clampi(g, maxv);
    rgb[2] = clampi((int)u + g, maxv);
  } else {
    const float sh = (float)dc, fm = (float)maxv;
    float t = __fadd_rn(__fadd_rn(y, __fmul_rn(1.402f, w)), sh);
    rgb[0] = (int)(t < 0.f ? 0.f : (t > fm ? fm : t));
    t = __fadd_rn(__fadd_rn(__fadd_rn(y, __fmul_rn(-0.34413f, u)), __fmul_rn(-0.71414f, w)), sh);
    rgb[1] = (int)(t < 0.f ? 0.f : (t > fm ? fm : t));
    t = __fadd_rn(__fadd_rn(y, __fmul_rn(1.772f, u)), sh);
    rgb[2] = (int)(t < 0.f ? 0.f : (t > fm ? fm : t));
  }
}

// Inverse RCT / ICT + DC level shift + clamp + LIFT + pack of one pixel (bmi_cpu_dwt_decoder.cpp
// RICT_97_FLOAT :3570-3643, RRct_53 :3936-4130, MergeComponents :4283-4598).  `v[c]` is
// component c's reconstructed sample (int32 for 5/3, float for 9/7), `have[c]` whether the
// component is present.
template <typename T>
__device__ __forceinline__ void emit_pixel(const OutGroup &G, uint8_t *out, int yy, int xx, const T *v,
                                           const bool *have) {
  const int pxb = fmt_bytes(G.fmt);
  const int B = G.bitdepth;
  const int outdepth = (pxb == 3 || pxb == 4) ? 8 : 16;
  const int maxv = (1 << B) - 1, dc = 1 << (B - 1);
  const bool rgb = (G.fmt == 0 || G.fmt == 1 || G.fmt == 2 || G.fmt == 8);
  const bool do_mct = rgb && G.mct && G.ncomp >= 3 && have[1] && have[2];
  const int slot0 = (pxb == 4 || pxb == 8) ? 1 : 0;
  uint8_t *px = out + G.out_off + ((size_t)(G.y0 + yy) * G.pitch_px + (G.x0 + xx)) * pxb;
  uint8_t tmp[8] = {0, 0, 0, 0, 0, 0, 0, 0};
  if (do_mct) {
    int c3[3];
    mct_pixel<T>(v[0], v[1], v[2], dc, maxv, c3);
    if (G.checkout >= 0 && G.checkout < 3) {
      // one component replicated into R, G and B (RICT_97_FLOAT / RRct_53 case 0..2)
      const int vv = lift_depth(c3[G.checkout], B, outdepth);
      for (int k = 0; k < 3; ++k) put_slot(tmp, pxb, k + slot0, vv);
    } else {
      for (int k = 0; k < 3; ++k) put_slot(tmp, pxb, k + slot0, lift_depth(c3[k], B, outdepth));
    }
  } else if (G.checkout >= 0 && have[G.checkout]) {
    // MergeComponents with a checked-out component: value in R = G = B, and in the
    // alpha slot only for the 4-component formats (bmi_cpu_dwt_decoder.cpp:4300-4308)
    const int vv = lift_depth(clampi((int)v[G.checkout] + dc, maxv), B, outdepth);
    if (pxb == 3 || pxb == 6) {
      for (int k = 0; k < 3; ++k) put_slot(tmp, pxb, k, vv);
    } else {
      for (int k = 1; k < 4; ++k) put_slot(tmp, pxb, k, vv);
      if (G.fmt == 3 || G.fmt == 4) put_slot(tmp, pxb, 0, vv);
    }
  } else {
    for (int c = 0; c < G.ncomp && c < 4; ++c) {
      if (!have[c]) continue;
      if ((pxb == 3 || pxb == 6) && c > 2) continue;
      put_slot(tmp, pxb, c, lift_depth(clampi((int)v[c] + dc, maxv), B, outdepth));
    }
  }
  for (int k = 0; k < pxb; ++k) px[k] = tmp[k];
}

#ifndef J2K_DWT_LEVELS_ONLY
// Output stage for tiles whose last level was not fused: reads the reconstructed
// components from the level buffers.
__global__ void __launch_bounds__(256) output_kernel(const OutGroup *__restrict__ groups,
                                                     const OutTask *__restrict__ tasks, int ntasks, const void *bufA,
                                                     const void *bufB, const void *bufC, uint8_t *out) {
  for (int task = blockIdx.x; task < ntasks; task += gridDim.x) {
    const OutTask tk = tasks[task];
    const OutGroup G = groups[tk.group];
    const void *cb[4];
    bool have[4];
    for (int c = 0; c < 4; ++c) {
      const void *bb = G.comp_buf[c] == 0 ? bufA : (G.comp_buf[c] == 1 ? bufB : bufC);
      cb[c] = G.comp_buf[c] < 0 ? nullptr : (const void *)((const uint8_t *)bb + G.comp_off[c] * 4);
      have[c] = cb[c] != nullptr;
    }
    const int ox = tk.tx * 64, oy = tk.ty * 64;
    for (int i = threadIdx.x; i < 64 * 64; i += blockDim.x) {
      const int yy = oy + i / 64, xx = ox + i % 64;
      if (yy >= G.h || xx >= G.w) continue;
      size_t at[4];
      for (int c = 0; c < 4; ++c) {
        at[c] = (size_t)yy * G.stride[c] + xx;
        if (G.sampled && have[c]) {  // replicate a sub-sampled component's nearest-left sample
          const int i = min(max((G.ax + xx) / G.sx[c] - G.cx[c], 0), G.cw[c] - 1);
          const int j = min(max((G.ay + yy) / G.sy[c] - G.cy[c], 0), G.ch[c] - 1);
          at[c] = (size_t)j * G.stride[c] + i;
        }
      }
      if (G.rev) {
        int32_t v[4] = {0, 0, 0, 0};
        for (int c = 0; c < 4; ++c)
          if (have[c]) v[c] = ((const int32_t *)cb[c])[at[c]];
        emit_pixel<int32_t>(G, out, yy, xx, v, have);
      } else {
        float v[4] = {0.f, 0.f, 0.f, 0.f};
        for (int c = 0; c < 4; ++c)
          if (have[c]) v[c] = ((const float *)cb[c])[at[c]];
        emit_pixel<float>(G, out, yy, xx, v, have);
      }
    }
  }
}

// Last DWT level of up to three components of one tile fused with the output stage (the
// inverse MCT reads the components' windows in shared memory): one CTA per 64x64 tile.
// Dynamic shared memory: `nwin` DwtSmem windows.
template <bool REV>
__global__ void __launch_bounds__(FUSED_THREADS, 3) last_level_output_kernel(const FusedGroup *__restrict__ groups,
                                                                        const OutTask *__restrict__ tasks, int ntasks,
                                                                        void *bufA, void *bufB, void *bufC,
                                                                        float ll_gain_value, uint8_t *out) {
  typedef typename DwtTypes<REV>::T T;
  extern __shared__ __align__(16) uint8_t dsm[];
  DwtSmem<REV> *S = reinterpret_cast<DwtSmem<REV> *>(dsm);
  for (int task = blockIdx.x; task < ntasks; task += gridDim.x) {
    const OutTask tk = tasks[task];
    const FusedGroup &F = groups[tk.group];
    const OutGroup G = F.G;
    const int nc = min(3, (int)G.ncomp);
    WinSrc<REV> src[3];
    bool have[4] = {false, false, false, false};
    for (int c = 0; c < nc; ++c) {
      const T *A = dwt_buf<REV>(0, bufA, bufB, bufC) + F.base[c];
      src[c] = {A, F.stride, dwt_buf<REV>(F.ll_src[c], bufA, bufB, bufC) + F.base[c], F.stride};
      have[c] = true;
    }
    const int ox = tk.tx * DWT_T, oy = tk.ty * DWT_T;
    dwt_windows<REV, false, DWT_T>(S, nc, src, F.rw, F.rh, F.lw, F.lh, F.ll_gain != 0, ll_gain_value, F.refcompat != 0, ox, oy,
                            nullptr, nullptr, 0, false, [] {});
    const int ow = min(DWT_T, F.rw - ox), oh = min(DWT_T, F.rh - oy);
    if (G.fmt == 2 && G.bitdepth == 8 && G.mct && nc == 3) {
      // 24-bit RGB after the inverse MCT (the common path): sixteen pixels per thread (48
      // bytes, bytes B, G, R per pixel) go out as three 16-byte stores when the run is
      // 16-byte aligned and whole, else as 32-bit words or bytes
      constexpr int RUN = 16;
      for (int i = threadIdx.x; i < DWT_T * (DWT_T / RUN); i += blockDim.x) {
        const int yy = i / (DWT_T / RUN), xx = (i % (DWT_T / RUN)) * RUN;
        if (yy >= oh || xx >= ow) continue;
        uint8_t *px = out + G.out_off + ((size_t)(G.y0 + oy + yy) * G.pitch_px + (G.x0 + ox + xx)) * 3;
        uint32_t words[12];
#pragma unroll
        for (int j = 0; j < 12; ++j) words[j] = 0;
        const int npx = min(RUN, ow - xx);
#pragma unroll
        for (int k = 0; k < RUN; ++k) {
          const int o = (yy + DWT_H) * DWT_PITCH + xx + k + DWT_H;
          int rgb[3];
          mct_pixel<T>(S[0].tile[o], S[1].tile[o], S[2].tile[o], 128, 255, rgb);
#pragma unroll
          for (int j = 0; j < 3; ++j) {
            const int b = k * 3 + j;  // byte j of pixel k: B, G, R
            words[b >> 2] |= (uint32_t)rgb[2 - j] << (8 * (b & 3));
          }
        }
        if (npx == RUN && !((uintptr_t)px & 15)) {
          uint4 *v = reinterpret_cast<uint4 *>(px);
          v[0] = make_uint4(words[0], words[1], words[2], words[3]);
          v[1] = make_uint4(words[4], words[5], words[6], words[7]);
          v[2] = make_uint4(words[8], words[9], words[10], words[11]);
        } else if (npx == RUN && !((uintptr_t)px & 3)) {
#pragma unroll
          for (int j = 0; j < 12; ++j) reinterpret_cast<uint32_t *>(px)[j] = words[j];
        } else {
          // a partial or unaligned run (picture edge, odd widths): pixel by pixel, recomputed
          // so that `words` stays in registers
          for (int k = 0; k < npx; ++k) {
            const int o = (yy + DWT_H) * DWT_PITCH + xx + k + DWT_H;
            int rgb[3];
            mct_pixel<T>(S[0].tile[o], S[1].tile[o], S[2].tile[o], 128, 255, rgb);
            px[3 * k] = (uint8_t)rgb[2];
            px[3 * k + 1] = (uint8_t)rgb[1];
            px[3 * k + 2] = (uint8_t)rgb[0];
          }
        }
      }
    } else {
      for (int i = threadIdx.x; i < DWT_T * DWT_T; i += blockDim.x) {
        const int yy = i / DWT_T, xx = i % DWT_T;
        if (yy >= oh || xx >= ow) continue;
        T v[4] = {0, 0, 0, 0};
        for (int c = 0; c < nc; ++c) v[c] = S[c].tile[(yy + DWT_H) * DWT_PITCH + xx + DWT_H];
        emit_pixel<T>(G, out, oy + yy, ox + xx, v, have);
      }
    }
    __syncthreads();
  }
}

// ------------------------------------------------------------------ coarse levels -------
// The coarsest levels of a tile-component are tiny (a 512x512 tile-component with five
// levels synthesises 32x32 and 64x64 before its first 128x128 level), so one launch per
// level leaves the GPU idle between short grids.  Here one CTA synthesises every level up to
// resolution `rc` of one tile-component in shared memory: the top-left res_w[rc] x res_h[rc]
// block of the tile-component's Mallat region already holds LL and every band up to that
// resolution, so it is staged once, each level is rebuilt in place (rows into a second
// buffer, columns back), and resolution rc is written once to the level buffer the level
// kernels would have left it in.  Arithmetic is the per-level kernels' (and the oracle's):
// whole-sample symmetric lifting over the full line, the same rounded float operations,
// K_lo^2 on a reconstructed 9/7 LL, the reference's 5/3 column end on request.
constexpr int COARSE_MAX = 64;  // largest resolution edge synthesised here
struct CoarseTask {
  uint64_t base;      // element offset of the tile-component region
  int32_t stride;     // tile-component width
  int8_t rc;          // resolutions 1..rc are synthesised here
  int8_t out_dst;     // buffer receiving resolution rc: 1 B, 2 C
  int8_t refcompat;   // 5/3: reference column-end arithmetic
  int8_t pad;
  int16_t res_w[8], res_h[8];  // resolutions 0..rc (rc <= 7: 64 << 7 exceeds any level kept here)
};

// In-place inverse lifting of one interleaved line of n samples (element stride st), the
// oracle's line97 / line53: x[-1] = x[1], x[n] = x[n - 2]
template <bool REV>
__device__ __forceinline__ void lift_full_line(typename DwtTypes<REV>::T *x, int n, int st) {
  if (n < 2) return;
  auto at = [&](int i) -> typename DwtTypes<REV>::T & {
    const int j = i < 0 ? -i : (i >= n ? 2 * (n - 1) - i : i);
    return x[j * st];
  };
  if constexpr (REV) {
    for (int i = 0; i < n; i += 2) at(i) = at(i) - ((at(i - 1) + at(i + 1) + 2) >> 2);
    for (int i = 1; i < n; i += 2) at(i) = at(i) + ((at(i - 1) + at(i + 1)) >> 1);
  } else {
    for (int i = 0; i < n; i += 2) at(i) = lift97(at(i), 0.44350685204397f, at(i - 1), at(i + 1));
    for (int i = 1; i < n; i += 2) at(i) = lift97(at(i), 0.88291107553093f, at(i - 1), at(i + 1));
    for (int i = 0; i < n; i += 2) at(i) = lift97(at(i), -0.05298011857296f, at(i - 1), at(i + 1));
    for (int i = 1; i < n; i += 2) at(i) = lift97(at(i), -1.58613434205992f, at(i - 1), at(i + 1));
  }
}

template <bool REV>
__global__ void __launch_bounds__(128) dwt_coarse_kernel(const CoarseTask *__restrict__ tasks, int ntasks, void *bufA,
                                                          void *bufB, void *bufC, float ll_gain_value) {
  typedef typename DwtTypes<REV>::T T;
  constexpr int P = COARSE_MAX + 1;  // odd pitch
  __shared__ T X[COARSE_MAX * P], Y[COARSE_MAX * P];
  for (int task = blockIdx.x; task < ntasks; task += gridDim.x) {
    const CoarseTask tk = tasks[task];
    const T *A = dwt_buf<REV>(0, bufA, bufB, bufC) + tk.base;
    T *out = dwt_buf<REV>(tk.out_dst, bufA, bufB, bufC) + tk.base;
    const int W = tk.res_w[tk.rc], H = tk.res_h[tk.rc];
    for (int i = threadIdx.x; i < W * H; i += blockDim.x) {
      const int y = i / W, x = i - y * W;
      X[y * P + x] = A[(size_t)y * tk.stride + x];
    }
    __syncthreads();
    for (int r = 1; r <= tk.rc; ++r) {
      const int rw = tk.res_w[r], rh = tk.res_h[r], lw = tk.res_w[r - 1], lh = tk.res_h[r - 1];
      if (!REV && r > 1) {  // the reconstructed LL entering a finer 9/7 level
        for (int i = threadIdx.x; i < lw * lh; i += blockDim.x) {
          const int y = i / lw, x = i - y * lw;
          X[y * P + x] = (T)__fmul_rn((float)X[y * P + x], ll_gain_value);
        }
        __syncthreads();
      }
      // rows: interleave low / high parts into Y, lift
      for (int y = threadIdx.x; y < rh; y += blockDim.x) {
        T *row = Y + y * P;
        for (int i = 0; i < rw; ++i) row[i] = X[y * P + ((i & 1) ? lw + (i >> 1) : (i >> 1))];
        lift_full_line<REV>(row, rw, 1);
      }
      __syncthreads();
      // columns: interleave low / high rows back into X, lift (5/3: the reference's column
      // end on request, from the column's de-interleaved inputs as in the level kernels)
      for (int x = threadIdx.x; x < rw; x += blockDim.x) {
        T *col = X + x;
        for (int i = 0; i < rh; ++i) col[i * P] = Y[((i & 1) ? lh + (i >> 1) : (i >> 1)) * P + x];
        if constexpr (REV) {
          const int n = rh;
          const bool fix = tk.refcompat && n >= 3;
          T a = 0, b = 0;
          if (fix) {
            if (!(n & 1)) {
              a = Y[(lh + n / 2 - 2) * P + x];  // H[m - 2]
            } else {
              const int m = (n + 1) / 2;
              b = Y[(lh + (m >= 3 ? m - 3 : 0)) * P + x];  // H[m - 3] (H[0] when m == 2)
              a = Y[(m - 2) * P + x];                       // L[m - 2]
            }
          }
          lift_full_line<REV>(col, rh, P);
          if (fix) {
            if (!(n & 1)) {
              col[(n - 1) * P] = a + col[(n - 2) * P];
            } else {
              const T x1 = a - ((b + 1) >> 1);
              col[(n - 1) * P] = x1;
              col[(n - 2) * P] = b + ((x1 + col[(n - 3) * P]) >> 1);
            }
          }
        } else {
          lift_full_line<REV>(col, rh, P);
        }
      }
      __syncthreads();
    }
    for (int i = threadIdx.x; i < W * H; i += blockDim.x) {
      const int y = i / W, x = i - y * W;
      out[(size_t)y * tk.stride + x] = X[y * P + x];
    }
    __syncthreads();
  }
}
#endif  // J2K_DWT_LEVELS_ONLY

}  // namespace j2k_dev

namespace j2k_dev {

// One level of one tile-component, all buffers given explicitly (no descriptor tables in device
// memory).  Used by the entry point that runs on a static scratch array (noalloc.cu).
template <bool REV>
struct OneLevel {
  typedef typename DwtTypes<REV>::T T;
  const T *coef, *ll;  // Mallat layout (row stride coef_stride) and the LL quadrant (ll_stride)
  T *out;
  int coef_stride, ll_stride, out_stride, rw, rh, lw, lh;
  int scale_ll, refcompat;
  int first, more;  // the call's first launch; another level follows
  float ll_gain;
};
// A level of at most two 64x64 tiles an SM is cut into 32x32 tiles: more of the chip works on it,
// each CTA for a shorter time (the 1000x777 level, 208 large tiles: a 5/3 tile-component of that
// size, in L2, takes 16.6 us, 19.0 with large ones; 4096x2160 with 560 and 2176 tiles is left as
// it is).
constexpr int SMALL_T = 32, SMALL_MOST = 2 * 148;
// The next level's CTAs may be launched while this one drains (programmatic launch): their first
// detail quadrants, which no level writes, are on their way when they wait for this one's results,
// so a level costs no launch latency.  The first level is launched in the same way behind the
// caller's work, and waits for it before it reads anything.  84x1088, 256x256, 1000x777 and
// 4096x2160 tile-components of three to five levels, calls one behind the other with inputs not in
// L2: 8.3, 12.5, 17.1 and 43.5 us (as one cooperative launch 10.4, 14.5, 18.6 and 46.6; first level
// launched plainly 10.4, 14.4, 18.6 and 45.5); from call to result 22, 26, 31 and 58 us (cooperative
// 22.5, 27, 30.5 and 59; the last three with plain launches 34, 36 and 65).  No CTA waits for one
// that is not yet running, so the levels need no part of the GPU to themselves, as a cooperative
// launch does: that is refused where the caller may use fewer SMs, and waits until work on other
// streams has left every SM room.
template <bool REV, int TILE>
__global__ void __launch_bounds__(DWT_THREADS) dwt_one_level_kernel(const OneLevel<REV> L) {
  __shared__ LevelSmem<REV, TILE> S;
  // the caller's work before the call, before anything is read and before a second level may start
  if (L.first) asm volatile("griddepcontrol.wait;" ::: "memory");
  if (L.more) asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  const int tiles_x = (L.rw + TILE - 1) / TILE, tiles = tiles_x * ((L.rh + TILE - 1) / TILE);
  int t = blockIdx.x;
  dwt_tiles<REV, TILE>(S, L.ll_gain, [&](LevelArgs<REV> &a) {
    if (t >= tiles) return false;
    a = {{L.coef, L.coef_stride, L.ll, L.ll_stride}, L.out, L.out_stride, L.rw, L.rh, L.lw, L.lh, (t % tiles_x) * TILE,
         (t / tiles_x) * TILE, L.scale_ll != 0, L.refcompat != 0};
    t += gridDim.x;
    return true;
  }, [&](const LevelArgs<REV> &a) {
    dwt_stage_tile<REV, TILE, STAGE_DETAIL>(S, a);
    asm volatile("griddepcontrol.wait;" ::: "memory");  // every CTA has a tile, so every CTA waits
    dwt_stage_tile<REV, TILE, STAGE_LL>(S, a);
  });
}

}  // namespace j2k_dev
