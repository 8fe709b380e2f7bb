/*
 * t1_kernel.cuh — EBCOT Tier-1 code-block decoder for sm_100a.
 *
 * One warp per code-block, blocks pulled from a device work queue (atomic counter over a
 * host-sorted order, longest blocks first) by persistent CTAs.
 *
 * The arithmetic decode is a serial chain: every symbol needs the interval the previous one
 * left.  It bounds the kernel twice over: a single picture lasts as long as the chain of its
 * densest block (139 cycles a symbol: 3.2 ms for the 45.3 k symbols of a 2048x2048 RGB 9/7
 * picture's; integer instructions issue every second cycle, a dependent one after 4 to 5, a
 * shared-memory load returns after 23, a branch costs 15 to 25 and one on which the lanes differ
 * 40 and more), and a long queue fills the SMs' issue slots with instructions that all 32 lanes
 * execute alike.  So what counts is instructions and branches per symbol:
 *   - the code register is extended by 32 and more bits of upcoming code, refilled four bytes at
 *     a time, so renormalisation is a shift without a loop, and one check covers two symbols;
 *   - each MQ context slot holds its probability-table entry (Qe, MPS, place in the table), so
 *     a symbol needs one shared-memory load before its decision, and the entries that may
 *     follow lie side by side;
 *   - refinement symbols change no later label: the lanes list a 32-column chunk's labels in
 *     scan order (positions from four ballots), the serial loop only walks the list, and each
 *     lane takes its column's bits from the decoded bit string and issues the sample updates;
 *     bypass (raw) bits of a chunk come byte by byte;
 *   - in significance propagation and cleanup the lanes tell which columns have work; the walk
 *     takes a column's rows from its context word.  A sample that becomes significant updates
 *     the eight words around it by as many lanes at once, without a branch (a tree of lane
 *     conditions there cost 450 cycles a sample);
 *   - stores that only some lanes make are predicated, never branched around;
 *   - in the cleanup pass a run of all-zero columns whose run-length symbols would all
 *     decode as MPS without renormalisation (C >= k*Qe and A - k*Qe >= 0x8000, scaled) is
 *     consumed in one step;
 *   - samples live in the block's own region of the output buffer, not in shared memory:
 *     they are only written while decoding (significance sets sign + 1.5 * 2^p, a
 *     refinement flips bit p and sets the new midpoint bit by a fire-and-forget atomic XOR).
 * Two forms share this code: the throughput form leaves a symbol early when it is an MPS
 * without renormalisation (fewest instructions), the latency form has no branch in a symbol and
 * takes refinement symbols four at a time (shortest chain).
 * Measured against the form with a renormalisation loop, a byte at a time, rows unrolled
 * (B200, Tier-1 ms): one 2048x2048 RGB 9/7 picture 7.22 -> 3.2, one 512x512 gray lossless
 * picture 4.92 -> 2.54, one 256x256 RGB 9/7 picture 1.62 -> 0.90, one 2048x1080 12-bit BYPASS +
 * RESET picture 5.47 -> 2.83, 32 1080p 9/7 frames 14.76 -> 12.54.
 *
 * Semantics follow the reference block decoder exactly (decoder/codec/src/
 * bmi_block_decoder.cpp:10-853, bmi_mq_decoder.h/.cpp, bmi_t1_macro.h): same context-word
 * layout, same scaled MQ registers and 0xFF/marker handling, same midpoint ("one and a
 * half") reconstruction bits, same MSB-plane rule including its plane-0 -> plane-1 case for
 * 9/7 blocks (:708-711), and the same 5/3 placement shift (dec_t1_comp.cpp:341-366).  Raw
 * (bypass) passes, context reset, per-pass termination and segmentation symbols follow
 * ITU-T T.800 Annex D (the reference asserts on them).
 */
#pragma once
#include <cstdint>
#include <cstring>
#include <utility>

#include "plan.h"

namespace j2k_dev {

// ---- context word of a stripe column (bmi_t1_macro.h:14-73): bits 0..17 the significance of
// the 3 x 6 samples around the column's four rows (row group j, columns left / own / right at
// bits 3j, 3j+1, 3j+2; group 0 is the row above, row k's own bit is 4 + 3k), bit 18 the sign
// of the sample above, 19 + 3k / 20 + 3k / 21 + 3k row k's sign (chi; set on rows outside
// the block), mu (significant before this bit-plane) and pi (coded by this plane's
// significance pass), bit 31 the sign of the sample below
constexpr int SIG_POS = 4, CHI_POS = 19, MU_POS = 20, PI_POS = 21;
constexpr uint32_t ROWS = 0x249;  // one bit per row, at 3k: a set of the column's rows
constexpr uint32_t CHI_ALL = ROWS << CHI_POS, MU_ALL = ROWS << MU_POS, PI_ALL = ROWS << PI_POS;

enum { C_SIG = 0, C_RUN = 9, C_SIGN = 10, C_MAG = 15, C_UNI = 18, N_CTX = 19 };
constexpr uint32_t SLOT = 8;  // bytes of a context slot
constexpr uint32_t RUN_OFF = C_RUN * SLOT, UNI_OFF = C_UNI * SLOT;  // byte offsets of context slots

// Read-only tables, copied to shared memory by every CTA (the lanes look labels up at
// different addresses, which constant memory would serialise):
//   mq[94][4]: for state s = idx*2 + mps the entries of the state itself (twice), of the one after
//              an MPS and of the one after an LPS (both in one 16-byte load); an entry is .x = Qe << 8 (the scaled register
//              unit), .y = (mps << 31) | byte offset of the state's first record
//   zc[3][512]: slot offset of the zero-coding context for LL/LH, HL, HH neighbourhoods
//   sc[2048] : slot offset of the sign context | xor bit in bit 7, by sign_index()
struct alignas(16) T1Tables {
  uint2 mq[94][4];
  uint8_t zc[3][512];
  uint8_t sc[2048];
};

// MQ decoder registers: A and C in the reference's scale (0x8000 is 0x800000); the low eight
// bits of C and all of l0, l1 are upcoming code, `T` the number of code bits held there (below
// the scale point).  Code bytes are read as aligned 32-bit words: `cur` holds the byte at
// `ap`, and the word after it is requested as soon as `cur` is entered.
struct Mq {
  int32_t A, C;
  uint32_t l0, l1;
  int32_t T;
  uint32_t last;      // the byte before `ap` (0xFF: the next byte carries seven bits)
  uint32_t ap, aend;  // byte position and segment end, counted from `w`
  const uint32_t *w;  // the segment's first byte rounded down to a 4-byte boundary
  uint32_t cur, nxt;  // the word holding byte ap and the one after it
};
constexpr int32_t A_MIN = 0x800000;
// Enough for two symbols: a renormalisation shifts by 15 at most, only bits above the scale
// point are compared, and bits missing after the second one are added by the next refill
constexpr int T_MIN = 15;

// Append n code bits v at position T of the 72-bit field (C's low eight bits, l0, l1); T may be
// negative: C was shifted further than the bits that were there
__device__ __forceinline__ void mq_append(Mq &m, uint32_t v, int n) {
  const uint64_t x = (uint64_t)v << (40 - n - m.T);  // T < T_MIN: nothing reaches l1
  m.C += (int32_t)(uint32_t)(x >> 32);
  m.l0 += (uint32_t)x;
  m.T += n;
}

// Refill to at least T_MIN bits; false when that many are not to be had yet.  Four plain bytes
// go in at once; around a 0xFF byte and at the segment's end the rules of FILL_LSBS
// (bmi_mq_decoder.h:52-73) hold byte by byte: after a 0xFF the next byte carries 7 bits,
// unless it is a marker (> 0x8F), which is not consumed and reads as eight ones; bytes past the
// segment's end read as 0xFF.  A byte 0x80..0x8F after a 0xFF adds a carry above its seven
// bits.  The reference adds it only once every earlier bit has been shifted into the compared
// part and another shift is due, so it waits here until T is negative: the shifted sum is the
// same, as both are linear, and no comparison sees the carry early.  Until then T stays below
// T_MIN and every single symbol needs a refill before it (mq_level).
__device__ __forceinline__ bool mq_refill(Mq &m) {
  const uint32_t four = __funnelshift_r(m.cur, m.nxt, (m.ap & 3) * 8);
  const uint32_t z = ~((four << 8) | m.last);  // a zero byte: the byte before or one of the first three is 0xFF
  if (!((z - 0x01010101u) & ~z & 0x80808080u) && m.T >= 0 && m.ap + 4 <= m.aend) {
    const uint32_t v = __byte_perm(four, 0, 0x0123);
    const uint64_t x = (uint64_t)v << (40 - m.T);
    m.C += (int32_t)((v >> 8) >> (16 + m.T));
    m.l0 |= (uint32_t)(x >> 32);
    m.l1 = (uint32_t)x;
    m.T += 32;
    m.last = four >> 24;
    m.ap += 4;
    m.cur = m.nxt;
    m.nxt = __ldg(m.w + (m.ap >> 2) + 1);
    return true;
  }
#pragma unroll 1
  while (m.T < T_MIN) {
    const uint32_t b = m.ap < m.aend ? (m.cur >> ((m.ap & 3) * 8)) & 0xFF : 0xFF;
    if (m.last != 0xFF) {
      mq_append(m, b, 8);
      m.last = b;
    } else if (b > 0x8F) {
      mq_append(m, 0xFF, 8);
      continue;
    } else {
      if (b >= 0x80 && m.T >= 0) return false;
      mq_append(m, b, 7);
      m.last = 0;
    }
    m.ap++;
    if (!(m.ap & 3)) {
      m.cur = m.nxt;
      m.nxt = __ldg(m.w + (m.ap >> 2) + 1);
    }
  }
  return true;
}

// Init, bmi_mq_decoder.cpp:186-219: two bytes loaded and shifted up by 15.  The word loads
// may reach up to 9 bytes past the segment; the code byte buffer carries 16 bytes of slack
// after its last segment.
__device__ __forceinline__ void mq_init(Mq &m, const uint8_t *base, uint32_t len) {
  const uint32_t off = (uint32_t)((uintptr_t)base & 3);
  m.w = reinterpret_cast<const uint32_t *>(base - off);
  m.ap = off;
  m.aend = off + len;
  m.cur = __ldg(m.w);
  m.nxt = __ldg(m.w + 1);
  m.last = 0;
  m.C = 0;
  m.l0 = m.l1 = 0;
  m.T = -15;
  m.A = A_MIN;
  mq_refill(m);
}

// One symbol (MQ_DECODE, bmi_mq_decoder.h:86-128) of a context whose slot entry is `e`, T being
// at least 0; returns the symbol in bit 31 (the other bits mean nothing: callers test the sign,
// which takes no instruction to extract) and leaves the entry that follows in `e` and in the
// slot.  The throughput form returns early on an MPS without renormalisation; the latency form has
// no branch: the successor (itself, after an MPS, after an LPS) is one of the state's records.
// All lanes decode the same symbols from the same registers and store the same entry, so a slot's
// load and store need the warp in lock-step between them: no branch from here to the next
// warp-wide operation may depend on the lane.  Stores that only some lanes make are predicated
// (put_sample, flip_sample, put_label), and the passes meet at __syncwarp() for every chunk, every
// sample that becomes significant and every list of refinement symbols.
template <bool LATENCY>
__device__ __forceinline__ uint32_t mq_symbol(Mq &m, uint8_t *slot, uint2 &e, const uint8_t *tab) {
  const int32_t q = (int32_t)e.x;
  const uint32_t mps = e.y;
  const int32_t a1 = m.A - q, d1 = m.C - q;
  const bool ex = m.C < q;
  if (!LATENCY && !ex && a1 >= A_MIN) {  // MPS without renormalisation
    m.A = a1;
    m.C = d1;
    return mps;
  }
  const bool lps = (a1 < q) != ex;
  const int32_t a = ex ? q : a1, c = ex ? m.C : d1;
  uint32_t rec = e.y & 0xFFFF;
  if (!LATENCY || a < A_MIN) rec += 2 * sizeof(uint2);
  if (lps) rec += sizeof(uint2);
  e = *reinterpret_cast<const uint2 *>(tab + rec);
  *reinterpret_cast<uint2 *>(slot) = e;
  const int n = __clz(a) - 8;
  m.A = a << n;
  m.C = (int32_t)__funnelshift_l(m.l0, (uint32_t)c, n);
  m.l0 = __funnelshift_l(m.l1, m.l0, n);
  m.l1 <<= n;
  m.T -= n;
  if (!LATENCY && m.T < T_MIN) mq_refill(m);  // else before the symbol, once for two of them
  return lps ? ~mps : mps;
}
__device__ __forceinline__ bool is_one(uint32_t symbol) { return (int32_t)symbol < 0; }
// Before a pair of symbols / between the two (a refill is due there only while a carry waits).
// The throughput form looks after every renormalisation instead: its common symbol has none.
template <bool LATENCY>
__device__ __forceinline__ void mq_ready(Mq &m) {
  if (LATENCY && m.T < T_MIN) mq_refill(m);
}
template <bool LATENCY>
__device__ __forceinline__ void mq_level(Mq &m) {
  if (LATENCY && m.T < 0) mq_refill(m);
}
// a symbol on its own
template <bool LATENCY>
__device__ __forceinline__ uint32_t mq_decode(Mq &m, uint8_t *cx, uint32_t off, const uint8_t *tab) {
  uint2 e = *reinterpret_cast<const uint2 *>(cx + off);
  mq_ready<LATENCY>(m);
  return mq_symbol<LATENCY>(m, cx + off, e, tab);
}

// Raw (bypass) bits, T.800 D.6: after 0xFF the next byte carries 7 bits; bytes past the end
// read as 0xFF
struct Raw {
  const uint8_t *base;
  uint32_t pos, end;
  uint32_t c;
  int ct;
};
__device__ __forceinline__ void raw_init(Raw &r, const uint8_t *base, uint32_t len) {
  r.base = base;
  r.pos = 0;
  r.end = len;
  r.c = 0;
  r.ct = 0;
}
__device__ __forceinline__ void raw_byte(Raw &r) {
  r.ct = r.c == 0xFF ? 7 : 8;
  r.c = r.pos < r.end ? (uint32_t)__ldg(r.base + r.pos) : 0xFFu;
  r.pos++;
}
__device__ __forceinline__ uint32_t raw_bit(Raw &r) {
  if (r.ct == 0) raw_byte(r);
  r.ct--;
  return r.c << (31 - r.ct);  // bit 31, as a symbol
}
// the next n bits (1 <= n <= 32), first bit in bit 31
__device__ __forceinline__ uint32_t raw_bits(Raw &r, int n) {
  uint32_t x = 0;
  int got = 0;
  while (got < n) {
    if (r.ct == 0) raw_byte(r);
    const int k = min(r.ct, n - got);
    r.ct -= k;
    x = (x << k) | ((r.c >> r.ct) & ((1u << k) - 1u));
    got += k;
  }
  return x << (32 - n);
}

// Shared memory of one warp.  The context words of a block w samples wide lie in rows of
// w + 3 words, one row per stripe with a row of zeros above and below and a column left and
// right, so that a sample's neighbours always exist.
template <int MAXW, int MAXH>
struct T1Layout {
  static constexpr int STRIPES = MAXH / 4, CHUNKS = (MAXW + 31) / 32;
  static constexpr int CWN = (STRIPES + 2) * (MAXW + 3) + 2;
  static constexpr int RF = (CWN * 4 + 15) & ~15;           // refined rows, 16 bytes per chunk
  static constexpr int CX = RF + STRIPES * CHUNKS * 16;     // context slots
  static constexpr int BITS = CX + ((N_CTX * (int)SLOT + 15) & ~15);  // a chunk's refinement bits
  static constexpr int LIST = BITS + 16;                    // a chunk's refinement labels in scan order
  static constexpr int PER_WARP = LIST + 4 * 32 + 16;
};

struct Block {
  uint32_t *cw;    // first context word of stripe 0
  uint4 *rf;       // per stripe and chunk: rows 0..3, bit = column: refined before
  uint8_t *cx;     // context slots
  uint32_t *bits;
  uint8_t *list;
  const uint8_t *mq, *zc, *sc;  // tables (zc: the block's band)
  uint32_t *out;    // the block's first sample in the output buffer
  uint32_t stride;  // elements per row
  int w, gap, stripes, lane;
  // how this lane (0..8) updates a word around a sample that becomes significant
  int spread_off;                      // word offset from the sample's column
  uint32_t spread_bits, spread_sign;   // bits set; where the sign goes (own column only)
  uint32_t spread_rows, spread_shift;  // rows (ROWS set) it applies to; all ones: shifted by the row
};

// Lanes 0..8 hold the 3 x 3 words (stripe above / own / below, column left / own / right; the
// centre, lane 4, is the walk's own).  Row k of the own stripe's words gets its bit shifted by 3k; the words above change for row
// 0 only (not at all with stripe-causal contexts, T.800 D.7: a stripe's last row sees the next
// stripe as insignificant) and the words below for row 3 only (bmi_block_decoder.cpp:53-101).
__device__ __forceinline__ void spread_init(Block &b, bool causal) {
  const int lane = b.lane, r = lane / 3, c = lane - 3 * r;
  const bool on = lane < 9 && lane != 4 && !(r == 0 && causal);
  const uint32_t own = c == 0 ? 0x20u : 0x08u;
  b.spread_off = lane < 9 ? (r - 1) * b.gap + c - 1 : 0;
  b.spread_bits = r == 0 ? (c == 0 ? 0x100u << 9 : (c == 1 ? 0x80u << 9 : 0x40u << 9))
                         : (r == 1 ? own : (c == 0 ? 0x04u : (c == 1 ? 0x02u : 0x01u)));
  b.spread_sign = c != 1 ? 0u : (r == 0 ? 1u << 31 : 1u << 18);
  b.spread_rows = !on ? 0u : (r == 0 ? 1u : (r == 1 ? ROWS : 1u << 9));
  b.spread_shift = r == 1 ? 0xFFFFFFFFu : 0u;
}
// No branch: a lane without a part in it ORs zero (lanes 9 up into the centre, which no lane
// changes; a divergent branch here cost 400 cycles a sample).
__device__ __forceinline__ void spread(const Block &b, uint32_t *wp, uint32_t k3, uint32_t sign) {
  const uint32_t on = 0u - ((b.spread_rows >> k3) & 1u);
  const uint32_t v = (b.spread_bits | (b.spread_sign & (uint32_t)((int32_t)sign >> 31))) << (k3 & b.spread_shift);
  wp[b.spread_off] |= v & on;
}

// Index of a sample's sign context: the significance and sign of its four neighbours (own
// column's word cw, the left word l and the right word r; row k), eight bits gathered into
// eleven without a loop: up / down sigma at bits 1, 7 and chi at 16, 22 of the shifted word,
// left at 4 / 19, right (shifted by 2) at 6 / 21; the chi half folds between the sigma half.
__device__ __host__ __forceinline__ uint32_t sign_fold(uint32_t x) { return ((x | (x >> 11)) >> 1) & 0x7FF; }
__device__ __forceinline__ uint32_t sign_index(uint32_t cw, uint32_t l, uint32_t r, uint32_t k3) {
  uint32_t v = cw >> k3;
  if (k3 == 0) v = (v & ~0x10000u) | ((v >> 2) & 0x10000u);  // row 0: the sign above is bit 18
  constexpr uint32_t UD = (1u << 1) | (1u << 7) | (1u << 16) | (1u << 22), LR = (1u << 4) | (1u << 19);
  const uint32_t x = (v & UD) | ((l >> k3) & LR) | (((r >> k3) & LR) << 2);
  return sign_fold(x);
}

inline void build_t1_tables(T1Tables &T) {
  static const uint16_t QE[47] = {0x5601, 0x3401, 0x1801, 0x0AC1, 0x0521, 0x0221, 0x5601, 0x5401, 0x4801, 0x3801,
                                  0x3001, 0x2401, 0x1C01, 0x1601, 0x5601, 0x5401, 0x5101, 0x4801, 0x3801, 0x3401,
                                  0x3001, 0x2801, 0x2401, 0x2201, 0x1C01, 0x1801, 0x1601, 0x1401, 0x1201, 0x1101,
                                  0x0AC1, 0x09C1, 0x08A1, 0x0521, 0x0441, 0x02A1, 0x0221, 0x0141, 0x0111, 0x0085,
                                  0x0049, 0x0025, 0x0015, 0x0009, 0x0005, 0x0001, 0x5601};
  static const uint8_t NMPS[47] = {1,  2,  3,  4,  5,  38, 7,  8,  9,  10, 11, 12, 13, 29, 15, 16,
                                   17, 18, 19, 20, 21, 22, 23, 24, 25, 26, 27, 28, 29, 30, 31, 32,
                                   33, 34, 35, 36, 37, 38, 39, 40, 41, 42, 43, 44, 45, 45, 46};
  static const uint8_t NLPS[47] = {1,  6,  9,  12, 29, 33, 6,  14, 14, 14, 17, 18, 20, 21, 14, 14,
                                   15, 16, 17, 18, 19, 19, 20, 21, 22, 23, 24, 25, 26, 27, 28, 29,
                                   30, 31, 32, 33, 34, 35, 36, 37, 38, 39, 40, 41, 42, 43, 46};
  std::memset(&T, 0, sizeof(T));
  auto entry = [&](int s) {
    uint2 e;
    e.x = (uint32_t)QE[s >> 1] << 8;
    e.y = ((uint32_t)(s & 1) << 31) | (uint32_t)(s * sizeof(T.mq[0]));
    return e;
  };
  for (int s = 0; s < 94; ++s) {
    const int idx = s >> 1, mps = s & 1;
    const int sw = QE[idx] == 0x5601 && NLPS[idx] != 46;
    T.mq[s][0] = entry(s);
    T.mq[s][1] = entry(s);
    T.mq[s][2] = entry(NMPS[idx] << 1 | mps);
    T.mq[s][3] = entry(NLPS[idx] << 1 | (mps ^ sw));
  }
  for (int band = 0; band < 3; ++band)
    for (int nb = 0; nb < 512; ++nb) {
      int h = ((nb >> 3) & 1) + ((nb >> 5) & 1);
      int v = ((nb >> 1) & 1) + ((nb >> 7) & 1);
      int d = (nb & 1) + ((nb >> 2) & 1) + ((nb >> 6) & 1) + ((nb >> 8) & 1);
      int c;
      if (band == 2) {  // HH
        int hv = h + v;
        if (d >= 3) c = 8;
        else if (d == 2) c = hv >= 1 ? 7 : 6;
        else if (d == 1) c = hv >= 2 ? 5 : (hv == 1 ? 4 : 3);
        else c = hv >= 2 ? 2 : hv;
      } else {
        if (band == 1) std::swap(h, v);  // HL
        if (h == 2) c = 8;
        else if (h == 1) c = v >= 1 ? 7 : (d >= 1 ? 6 : 5);
        else if (v == 2) c = 4;
        else if (v == 1) c = 3;
        else c = d >= 2 ? 2 : d;
      }
      T.zc[band][nb] = (uint8_t)((C_SIG + c) * SLOT);
    }
  for (int i = 0; i < 256; ++i) {
    // bit 0 sigma up, 1 chi up, 2 sigma down, 3 chi down, 4 sigma left, 5 chi left,
    // 6 sigma right, 7 chi right (T.800 Table D.3)
    auto contrib = [&](int sb, int xb) { return ((i >> sb) & 1) ? (((i >> xb) & 1) ? -1 : 1) : 0; };
    int H = contrib(4, 5) + contrib(6, 7);
    int V = contrib(0, 1) + contrib(2, 3);
    H = H < -1 ? -1 : (H > 1 ? 1 : H);
    V = V < -1 ? -1 : (V > 1 ? 1 : V);
    int x = 0;
    if (H < 0 || (H == 0 && V < 0)) {
      H = -H;
      V = -V;
      x = 1;
    }
    const int c = (H == 1) ? (V == 1 ? 4 : (V == 0 ? 3 : 2)) : (V == 1 ? 1 : 0);
    static const int at[8] = {1, 16, 7, 22, 4, 19, 6, 21};  // their places in sign_index()
    uint32_t w = 0;
    for (int k = 0; k < 8; ++k) w |= (uint32_t)((i >> k) & 1) << at[k];
    T.sc[sign_fold(w)] = (uint8_t)((C_SIGN + c) * SLOT | x << 7);
  }
}

enum { P_SIGPROP = 0, P_MAGREF = 1, P_CLEANUP = 2 };

// Rows with a significant sample in their 3 x 3 neighbourhood, the own bit included
__device__ __forceinline__ uint32_t near_rows(uint32_t w) {
  const uint32_t y = w | (w >> 1) | (w >> 2);
  return (y | (y >> 3) | (y >> 6)) & ROWS;
}

// List positions of a chunk: the lanes' row sets x, columns in lane order, rows downwards;
// returns the number of entries, `pos` the lane's first
__device__ __forceinline__ int list_positions(uint32_t x, int lane, int &pos, uint4 &rows) {
  rows.x = __ballot_sync(0xffffffffu, x & 1u);
  rows.y = __ballot_sync(0xffffffffu, x & 8u);
  rows.z = __ballot_sync(0xffffffffu, x & 0x40u);
  rows.w = __ballot_sync(0xffffffffu, x & 0x200u);
  const uint32_t lt = (1u << lane) - 1u;
  pos = __popc(rows.x & lt) + __popc(rows.y & lt) + __popc(rows.z & lt) + __popc(rows.w & lt);
  return __popc(rows.x) + __popc(rows.y) + __popc(rows.z) + __popc(rows.w);
}

// Predicated stores without a branch (a branch on which the lanes differ costs the warp tens
// of cycles): a sample's first value, from the lane that owns its column (the same lane issues
// the sample's refinements, so its updates stay in order), a refinement, and a list label
__device__ __forceinline__ void put_sample(uint32_t *at, uint32_t v, uint32_t on) {
#ifdef __CUDACC__
  asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.u32 p, %2, 0;\n\t@p st.global.u32 [%0], %1;\n\t}" ::"l"(at), "r"(v), "r"(on)
               : "memory");
#else
  if (on) *at = v;
#endif
}
__device__ __forceinline__ void flip_sample(uint32_t *at, uint32_t v, uint32_t on) {
#ifdef __CUDACC__
  asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.u32 p, %2, 0;\n\t@p red.global.xor.b32 [%0], %1;\n\t}" ::"l"(at), "r"(v),
               "r"(on)
               : "memory");
#else
  if (on) *at ^= v;
#endif
}
__device__ __forceinline__ void put_label(uint8_t *at, uint32_t v, uint32_t on) {
#ifdef __CUDACC__
  asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.u32 p, %2, 0;\n\t@p st.shared.u8 [%0], %1;\n\t}" ::"r"(
                   (uint32_t)__cvta_generic_to_shared(at)),
               "r"(v), "r"(on)
               : "memory");
#else
  if (on) *at = (uint8_t)v;
#endif
}

template <int PASS>
__device__ __forceinline__ uint32_t pass_rows(uint32_t word) {
  if (PASS == P_SIGPROP) return near_rows(word) & ~((word >> SIG_POS) | (word >> CHI_POS));
  return ~((word >> SIG_POS) | (word >> CHI_POS) | (word >> PI_POS)) & ROWS;
}

// Significance propagation (bmi_block_decoder.cpp:10-215): samples not yet significant with a
// significant neighbour.  Cleanup (:351-586): every sample not yet coded in this bit-plane; an
// all-zero column is one run-length symbol (if it is 1, two uniform symbols give the row of
// the first significant sample, whose sign follows directly).  A sample that becomes
// significant changes the words around it, so the walk goes column by column from the words
// themselves; the lanes only tell which columns of a chunk have work, and a column right of a
// new significant sample joins them.
// PASS and RAW (a bypass segment: raw bits instead of MQ symbols) are compile-time constants.
template <bool LATENCY, int PASS, bool RAW>
__device__ __forceinline__ void significance_pass(const Block &b, int p, Mq &mq, Raw &raw) {
  const int lane = b.lane;
  for (int s = 0; s < b.stripes; ++s) {
    uint32_t *row = b.cw + s * b.gap;
    uint32_t *out = b.out + (size_t)(4 * s) * b.stride;
    for (int c0 = 0; c0 < b.w; c0 += 32) {
      __syncwarp();
      const bool valid = c0 + lane < b.w;
      const uint32_t word = valid ? row[c0 + lane] : 0u;
      uint32_t *mine = out + c0 + lane;
      uint32_t live = __ballot_sync(0xffffffffu, valid && pass_rows<PASS>(word));
      uint32_t zero = PASS == P_CLEANUP ? __ballot_sync(0xffffffffu, valid && word == 0) : 0u;
      const uint32_t inside = __ballot_sync(0xffffffffu, valid);
      while (live) {
        const int bit = __ffs(live) - 1;
        uint32_t *wp = row + c0 + bit;
        uint32_t W = *wp, x, k3 = 0;
        const uint32_t L = wp[-1], R = wp[1];  // their own bits do not change during the walk of this column
        bool forced = false;
        if (PASS == P_CLEANUP && ((zero >> bit) & 1)) {
          uint2 e = *reinterpret_cast<const uint2 *>(b.cx + RUN_OFF);
          const int32_t q = (int32_t)e.x, room = min(mq.A - A_MIN, mq.C);
          if (!(e.y >> 31) && room >= q) {
            // zero columns from here on: as many as need no renormalisation
            int n = __clz(__brev(~(zero >> bit)));
            if (n * q > room) n = room / q;
            mq.A -= n * q;
            mq.C -= n * q;
            live &= ~((n >= 32 ? 0xffffffffu : (1u << n) - 1u) << bit);
            continue;
          }
          live &= live - 1;
          mq_ready<LATENCY>(mq);
          if (!is_one(mq_symbol<LATENCY>(mq, b.cx + RUN_OFF, e, b.mq))) continue;
          k3 = is_one(mq_decode<LATENCY>(mq, b.cx, UNI_OFF, b.mq)) ? 6 : 0;
          k3 += is_one(mq_decode<LATENCY>(mq, b.cx, UNI_OFF, b.mq)) ? 3 : 0;
          x = ROWS & (0xFFFFFFF8u << k3);
          forced = true;
        } else {
          live &= live - 1;
          x = pass_rows<PASS>(W);
          if (PASS == P_CLEANUP) {
            // a column whose symbols would all be MPS (insignificant) without renormalisation is one
            // step: the labels hold as long as nothing becomes significant (85 % of the symbols of
            // a lossy frame are such; a 1021x677 12-bit 9/7 picture 2.11 -> 1.87 ms, 32 1080p frames
            // 12.94 -> 12.71)
            int32_t sum = 0;
            uint32_t any = 0;
#pragma unroll
            for (int k = 0; k < 4; ++k) {
              const uint2 e = *reinterpret_cast<const uint2 *>(b.cx + b.zc[(W >> (3 * k)) & 0x1EF]);
              if (x & (1u << (3 * k))) {
                sum += (int32_t)e.x;
                any |= e.y;
              }
            }
            if (!is_one(any) && min(mq.A - A_MIN, mq.C) >= sum) {
              mq.A -= sum;
              mq.C -= sum;
              continue;
            }
          }
          if (PASS == P_SIGPROP) W |= x << PI_POS;
        }
        uint32_t hit = 0;
        while (forced || x) {
          if (!forced) {
            k3 = __ffs(x) - 1;
            x &= x - 1;
            uint32_t d;
            if (RAW) {
              d = raw_bit(raw);
            } else {
              mq_ready<LATENCY>(mq);
              const uint32_t off = b.zc[(W >> k3) & 0x1EF];
              uint2 e = *reinterpret_cast<const uint2 *>(b.cx + off);
              d = mq_symbol<LATENCY>(mq, b.cx + off, e, b.mq);
            }
            if (!is_one(d)) continue;
          }
          forced = false;
          // row k3 / 3 becomes significant: sign, neighbours, first value
          uint32_t sign;  // in bit 31
          if (RAW) {
            sign = raw_bit(raw);
          } else {
            const uint32_t sv = b.sc[LATENCY ? sign_index(W, L, R, k3) : sign_index(W, wp[-1], wp[1], k3)], off = sv & 0x7F;
            uint2 e = *reinterpret_cast<const uint2 *>(b.cx + off);
            mq_level<LATENCY>(mq);
            sign = mq_symbol<LATENCY>(mq, b.cx + off, e, b.mq) ^ (sv << 24);
          }
          sign &= 1u << 31;
          hit = 0xffffffffu;
          W |= ((1u << SIG_POS) | (sign >> (31 - CHI_POS))) << k3;
          // (the latency form keeps its lane's column address, the throughput form the registers)
          put_sample((LATENCY ? mine : out + c0 + bit) + (k3 * 11 >> 5) * b.stride, sign + (3u << p >> 1),
                     lane == bit);
          if (PASS == P_SIGPROP) {
            x = pass_rows<PASS>(W) & (0xFFFFFFF8u << k3);
            W |= x << PI_POS;
          }
          __syncwarp();
          spread(b, wp, k3, sign);
          __syncwarp();
        }
        *wp = W;
        const uint32_t right = (2u << bit) & inside & hit;
        if (PASS == P_SIGPROP) live |= right;
        else zero &= ~right;
      }
      if (PASS == P_CLEANUP) {
        // end of the bit-plane for this chunk's columns: mu |= sigma, pi cleared
        // (bmi_block_decoder.cpp:571-573); no later symbol of this pass reads a column's own
        // mu / pi bits
        __syncwarp();
        if (valid) {
          const uint32_t w = row[c0 + lane];
          row[c0 + lane] = (w | ((w << (MU_POS - SIG_POS)) & MU_ALL)) & ~PI_ALL;
        }
      }
    }
  }
  __syncwarp();
}

// A symbol of a context that stays in registers: its entry `e` and the two that may follow, `f`,
// so the next symbol's Qe is one select away instead of a load
__device__ __forceinline__ uint32_t mq_same(Mq &m, uint2 &e, uint4 &f, const uint8_t *tab) {
  const int32_t q = (int32_t)e.x;
  const uint32_t mps = e.y;
  const int32_t a1 = m.A - q, d1 = m.C - q;
  const bool ex = m.C < q;
  const bool lps = (a1 < q) != ex;
  const int32_t a = ex ? q : a1, c = ex ? m.C : d1;
  const bool ren = a < A_MIN;
  const uint32_t nx = lps ? f.z : f.x, ny = lps ? f.w : f.y;
  e.x = ren ? nx : e.x;
  e.y = ren ? ny : e.y;
  f = *reinterpret_cast<const uint4 *>(tab + (e.y & 0xFFFF) + 16);
  const int n = __clz(a) - 8;
  m.A = a << n;
  m.C = (int32_t)__funnelshift_l(m.l0, (uint32_t)c, n);
  m.l0 = __funnelshift_l(m.l1, m.l0, n);
  m.l1 <<= n;
  m.T -= n;
  return lps ? ~mps : mps;
}
// The refinement symbols of a chunk: n labels in scan order, decoded bits to b.bits, first one
// in bit 31.  The
// latency form takes four at a time: their slots are loaded together and entries changed
// within the four passed on in registers, so no symbol waits for a store and a load.
template <bool LATENCY>
__device__ __forceinline__ void refine(const Block &b, const uint8_t *list, int n, Mq &mq) {
  uint8_t *cx = b.cx + C_MAG * SLOT;
  uint32_t bits = 0;  // the last 32, newest in bit 0
  auto push = [](uint32_t bits, uint32_t symbol) { return __funnelshift_l(symbol, bits, 1); };
  int i = 0;
  if (LATENCY) {
    const uint32_t *four = reinterpret_cast<const uint32_t *>(list);
    uint32_t next = four[0];
    constexpr uint32_t ALL2 = 2 * SLOT * 0x01010101u;
    while (i + 4 <= n) {
      if (next == ALL2) {
        // every sample refined before: one context, its entry in registers
        uint2 e = *reinterpret_cast<const uint2 *>(cx + 2 * SLOT);
        uint4 f = *reinterpret_cast<const uint4 *>(b.mq + (e.y & 0xFFFF) + 16);
        bool more;
        do {
          if (mq.T < T_MIN && !mq_refill(mq)) break;
          next = four[(i >> 2) + 1];
          bits = push(bits, mq_same(mq, e, f, b.mq));
          bits = push(bits, mq_same(mq, e, f, b.mq));
          if (mq.T < T_MIN && !mq_refill(mq)) {
            *reinterpret_cast<uint2 *>(cx + 2 * SLOT) = e;  // a carry waits
            i += 2;
            goto singles;
          }
          bits = push(bits, mq_same(mq, e, f, b.mq));
          bits = push(bits, mq_same(mq, e, f, b.mq));
          i += 4;
          if (!(i & 31)) b.bits[(i >> 5) - 1] = bits;
          more = next == ALL2 && i + 4 <= n;
        } while (more);
        *reinterpret_cast<uint2 *>(cx + 2 * SLOT) = e;
        if (mq.T < T_MIN && !mq_refill(mq)) break;
        continue;
      }
      const uint32_t o = next;
      const uint32_t o0 = o & 0xFF, o1 = (o >> 8) & 0xFF, o2 = (o >> 16) & 0xFF, o3 = o >> 24;
      uint2 e0 = *reinterpret_cast<const uint2 *>(cx + o0), e1 = *reinterpret_cast<const uint2 *>(cx + o1),
            e2 = *reinterpret_cast<const uint2 *>(cx + o2), e3 = *reinterpret_cast<const uint2 *>(cx + o3);
      next = four[(i >> 2) + 1];
      if (mq.T < T_MIN && !mq_refill(mq)) break;
      bits = push(bits, mq_symbol<true>(mq, cx + o0, e0, b.mq));
      if (o1 == o0) e1 = e0;
      bits = push(bits, mq_symbol<true>(mq, cx + o1, e1, b.mq));
      i += 2;
      if (mq.T < T_MIN && !mq_refill(mq)) break;
      if (o2 == o0) e2 = e0;
      if (o2 == o1) e2 = e1;
      bits = push(bits, mq_symbol<true>(mq, cx + o2, e2, b.mq));
      if (o3 == o0) e3 = e0;
      if (o3 == o1) e3 = e1;
      if (o3 == o2) e3 = e2;
      bits = push(bits, mq_symbol<true>(mq, cx + o3, e3, b.mq));
      i += 2;
      if (!(i & 31)) b.bits[(i >> 5) - 1] = bits;
    }
  }
singles:
  __syncwarp();  // the ways here differ in length
  // one at a time: the throughput form, a chunk's last three, and while a carry waits
  for (; i < n; ++i) {
    bits = push(bits, mq_decode<LATENCY>(mq, cx, list[i], b.mq));
    if ((i & 31) == 31) b.bits[i >> 5] = bits;
  }
  if (n & 31) b.bits[n >> 5] = bits << (32 - (n & 31));
}

// Magnitude refinement (bmi_block_decoder.cpp:217-349): samples significant before this
// bit-plane.  The reference's "first refinement" test (|v| >> p) < 4 is true exactly on a
// sample's first refinement: a bit per sample in `rf`.
template <bool LATENCY, bool RAW>
__device__ __forceinline__ void refinement_pass(const Block &b, int p, Mq &mq, Raw &raw) {
  const int lane = b.lane;
  uint8_t *list = b.list;
  const int chunks = (b.w + 31) >> 5;
  for (int s = 0; s < b.stripes; ++s) {
    for (int h = 0; h < chunks; ++h) {
      const int c = h * 32 + lane;
      const uint32_t word = c < b.w ? b.cw[s * b.gap + c] : 0u;
      const uint32_t x = (word >> SIG_POS) & (word >> MU_POS) & ROWS;
      if (!__any_sync(0xffffffffu, x)) continue;
      int pos;
      uint4 rows;
      const int n = list_positions(x, lane, pos, rows);
      uint4 rf = b.rf[s * chunks + h];
      int at = pos;
      if (!RAW) {
        // label: 2 once refined, else 1 with a significant neighbour
        const uint32_t y = word | (word >> 1) | (word >> 2);
        const uint32_t near = y | (y >> 6) | (word >> 3) | (word >> 5);
        put_label(list + at, (rf.x >> lane) & 1 ? 2 * SLOT : (near & 1u) * SLOT, x & 1u);
        at += x & 1u;
        put_label(list + at, (rf.y >> lane) & 1 ? 2 * SLOT : ((near >> 3) & 1u) * SLOT, x & 8u);
        at += (x >> 3) & 1u;
        put_label(list + at, (rf.z >> lane) & 1 ? 2 * SLOT : ((near >> 6) & 1u) * SLOT, x & 0x40u);
        at += (x >> 6) & 1u;
        put_label(list + at, (rf.w >> lane) & 1 ? 2 * SLOT : ((near >> 9) & 1u) * SLOT, x & 0x200u);
      }
      __syncwarp();
      rf.x |= rows.x;
      rf.y |= rows.y;
      rf.z |= rows.z;
      rf.w |= rows.w;
      if (lane == 0) b.rf[s * chunks + h] = rf;
      __syncwarp();
      if (RAW) {
        for (int i = 0; i < n; i += 32) b.bits[i >> 5] = raw_bits(raw, min(32, n - i));
      } else {
        refine<LATENCY>(b, list, n, mq);
      }
      __syncwarp();
      // each lane's samples: bit p as decoded, the next midpoint bit
      unsigned int *col = b.out + (size_t)(4 * s) * b.stride + c;
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        const uint32_t on = x & (1u << (3 * k));
        const uint32_t d = (b.bits[(pos >> 5) & 3] << (pos & 31)) >> 31;  // unused (and in bounds) when off
        pos += on ? 1 : 0;
        flip_sample(col + (size_t)k * b.stride, ((1u - d) << p) | ((1u << p) >> 1), on);
      }
      __syncwarp();
    }
  }
}

// (every lane writes the same)
__device__ __forceinline__ void init_states(uint8_t *cx, const uint8_t *tab) {
  // bmi_mq_decoder.cpp:65-79: (state 0, MPS 0) except sig ctx 0 -> state 4, run -> state 3
  const uint2(*t)[4] = reinterpret_cast<const uint2(*)[4]>(tab);
  uint2 *slot = reinterpret_cast<uint2 *>(cx);
  for (int i = 0; i < N_CTX; ++i) slot[i] = t[0][0];
  slot[C_SIG] = t[4 << 1][0];
  slot[C_RUN] = t[3 << 1][0];
  slot[C_UNI] = t[46 << 1][0];
}

__device__ __forceinline__ bool seg_starts(int flags, int j) {
  if (j == 0) return true;
  if (flags & J2K_CB_TERMALL) return true;
  int type = (j - 1) % 3;
  return (flags & J2K_CB_BYPASS) && j >= 10 && type != 1;
}

// MSB plane and pass count of a block (bmi_block_decoder.cpp:603-622, :708-711)
__device__ __forceinline__ void block_planes(const j2k_cblk &cb, int &bit_plane, int &num_passes) {
  const int missing = cb.missing;
  const int p_max = 30 - missing;
  num_passes = 3 * p_max - 2;
  if (num_passes > cb.num_passes) num_passes = cb.num_passes;
  if (cb.flags & J2K_CB_IRREV) {
    bit_plane = (int)cb.mb - 1 - missing;
  } else {
    if (((int)cb.mb - missing) * 3 - 2 <= 0) num_passes = 0;
    bit_plane = -1 - missing;
  }
  if (bit_plane < 0) bit_plane = p_max;
  if (bit_plane == 0) bit_plane = 1;
}

// Decode one code-block with the whole warp: raw sign-magnitude samples in b.out, the
// significance of every sample in the context words.  Returns a status (0 ok).
template <bool LATENCY>
__device__ __forceinline__ int decode_block(const j2k_cblk &cb, const uint8_t *__restrict__ bytes,
                                            const uint32_t *__restrict__ seglens, Block &b, int bit_plane,
                                            int num_passes) {
  const int w = cb.w, h = cb.h, lane = b.lane;
  const int stripes = b.stripes;
  // clear the context words and refinement bits (the samples need no clearing: the final
  // rewrite gives 0 to those that never became significant); mark columns and rows outside
  // the block
  uint32_t *first = b.cw - b.gap - 1;
  const int nwords = (stripes + 2) * b.gap + 2;
  for (int i = lane; i < nwords; i += 32) first[i] = 0;
  for (int i = lane; i < stripes * ((w + 31) >> 5); i += 32) b.rf[i] = make_uint4(0, 0, 0, 0);
  __syncwarp();
  for (int s = lane; s < stripes; s += 32) {
    uint32_t *r = b.cw + s * b.gap + w;
    r[0] = CHI_ALL;
    r[1] = CHI_ALL;
    r[2] = CHI_ALL;
  }
  if (h & 3) {
    const uint32_t m = CHI_ALL & (0xFFFFFFFFu << (CHI_POS + 3 * (h & 3)));
    for (int c = lane; c < w; c += 32) b.cw[(stripes - 1) * b.gap + c] = m;
  }
  init_states(b.cx, b.mq);
  spread_init(b, (cb.flags & J2K_CB_CAUSAL) != 0);
  __syncwarp();
  if (num_passes > 0 && 30 - (int)cb.missing <= 0) return 1;

  const int multi = (cb.flags & (J2K_CB_BYPASS | J2K_CB_TERMALL)) != 0;
  const uint8_t *data = bytes + cb.data_off;
  Mq mq;
  Raw raw;
  mq.A = mq.C = mq.T = 0;
  mq.l0 = mq.l1 = mq.last = mq.ap = mq.aend = mq.cur = mq.nxt = 0;
  mq.w = reinterpret_cast<const uint32_t *>(bytes);
  raw_init(raw, data, 0);
  uint32_t seg_pos = 0;
  int seg_idx = 0;
  bool israw = false;
  int status = 0;
  for (int k = 0, type = 2; k < num_passes; ++k, ++type) {
    if (type == 3) {
      type = 0;
      bit_plane--;
    }
    if (bit_plane < 0) {
      status = 2;
      break;
    }
    if (seg_starts(multi ? cb.flags : 0, k)) {
      uint32_t len;
      if (multi) {
        if (seg_idx >= cb.nseg) {
          status = 3;
          break;
        }
        len = __ldg(seglens + cb.seg_off + seg_idx);
        seg_idx++;
      } else {
        len = cb.data_len;
      }
      if (seg_pos + len > cb.data_len) {
        status = 4;
        break;
      }
      israw = (cb.flags & J2K_CB_BYPASS) && k >= 10 && type != 2;
      if (israw) raw_init(raw, data + seg_pos, len);
      else mq_init(mq, data + seg_pos, len);
      seg_pos += len;
    }
    if (type == P_CLEANUP) significance_pass<LATENCY, P_CLEANUP, false>(b, bit_plane, mq, raw);
    else if (type == P_SIGPROP && israw) significance_pass<LATENCY, P_SIGPROP, true>(b, bit_plane, mq, raw);
    else if (type == P_SIGPROP) significance_pass<LATENCY, P_SIGPROP, false>(b, bit_plane, mq, raw);
    else if (israw) refinement_pass<LATENCY, true>(b, bit_plane, mq, raw);
    else refinement_pass<LATENCY, false>(b, bit_plane, mq, raw);
    if (type == 2 && (cb.flags & J2K_CB_SEGSYM)) {
      // four uniform symbols (the reference's fixed-Qe MQ_DECODE_START, bmi_mq_decoder.h:131-169,
      // is an ordinary symbol of a slot pinned at state 46)
#pragma unroll 1
      for (int i = 0; i < 4; ++i) mq_decode<LATENCY>(mq, b.cx, UNI_OFF, b.mq);
    }
    if (cb.flags & J2K_CB_RESET) {
      __syncwarp();
      init_states(b.cx, b.mq);
      __syncwarp();
    }
  }
  __syncwarp();
  return status;
}

}  // namespace j2k_dev
