// bsw16.cuh -- banded affine Smith-Waterman on packed int16 lanes (two cells per
// 32-bit register), bit-exact with the int32 sweep of bsw.cuh / banded_sw_with
// (src/alignment/mod.rs:1370-1650) whenever the host-side range check passes.
//
// Layout
//   A group of G lanes owns one pair. The row (capacity 2H cells, H = G*K) is cut
//   in two halves: word k of lane g holds cell c = g*K + k in its low 16 bits and
//   cell H + c in its high 16 bits, so every per-row quantity (band start, shift,
//   argmax, x-drop) stays one scalar per pair while the DP arithmetic runs two
//   cells per instruction with the DPX 16x2 forms (__viaddmax_s16x2,
//   __vimax_s16x2_relu, and the three-input __vimax3_u16x2 for the row-max keys).
//
// Biased values
//   Every DP value v is kept as v + B (B = bias >= gof + 2H*ge + mismatch + 1), so
//   all stored halves are non-negative and below 2^13 (checked on the host). That
//   makes plain 32-bit IADD/IADD3 exact on packed words (no carry crosses the
//   half boundary when each half's result stays in [0, 2^16)).
//
// What bounds it, and what follows
//   One lane per pair is bound by the integer pipes (about 830 instructions a row of 34
//   words, 550 of them on the ALU pipe). A row therefore computes H and nothing else:
//   no direction or extend flags. The trace is the low byte of every cell's H, and the
//   traceback finds each move by comparing values (warp_walk_h). With four flags per
//   cell (1268 instructions a row, 163M against 98M on the ALU pipe for 37,888 pairs of
//   150 bp) 300,000 pairs at band 33 took 2.85 ms; this form takes 2.07 ms (1449 G
//   cells/s), bands 64 and 128 at 200 bp 2.76 -> 2.19 and 3.12 -> 2.41 ms.
//   Short lanes (several per pair) are bound by the latency of a row: 16 pairs of 150 bp
//   took 146 us on 4 x 9 words, 57 us on 32 x 2; 6,000 of 1,000 bp at band 256 4.72 ms,
//   now 2.84.
//
// Band edges
//   Cells outside the previous row's band read as "neutral" (H = 0, E = -gof or
//   less): a diagonal predecessor out of band then contributes 0 + s (the reference's
//   scored-restart quirk, mod.rs:1464-1480) and an upper predecessor out of band
//   yields E = -gof instead of i32::MIN/4, which never wins a cell and never ties a
//   nonzero H, so H equals the reference's. The invariant is kept by masking H at and
//   beyond the row length after each row; E there follows from a neutral H above it,
//   except below a row that reached further right (masked in the row whose end moved
//   back).
#pragma once

#include <type_traits>

#include "common.cuh"

namespace kira {

template <int G, int K>
struct Bsw16Shape {
  static constexpr int kHalf = G * K;                  // cells per half row
  static constexpr int kCap = 2 * kHalf;               // cells per row
  static constexpr int kWords = (K + 1) / 2;           // window-byte words per lane
  static constexpr int kSlabs = (K + 1) / 2;           // 4-byte stores per lane per row
  static constexpr int kLaneBytes = 4 * kSlabs;        // a byte per cell
  static constexpr int kRowStride = G * kLaneBytes;
  // Rows interleave in blocks of kInterleave: a block stores slab by slab, and in
  // each slab row by row, so one line holds one slab of kInterleave consecutive rows
  // (the cells a diagonal traceback run reads next). Few lanes per pair interleave 8
  // rows, which keeps the shared-memory staging strip (one block) small.
  static constexpr int kInterleave = G <= 4 ? 8 : G >= 32 ? 1 : 32 / G;
  // Bytes of one interleave block of a group; its shared-memory staging strip is 16
  // bytes longer, which spreads the groups' stores over the banks.
  static constexpr int kStripBytes = kSlabs * kInterleave * G * 4;
  static constexpr int kStripStride = G < 8 ? kStripBytes + 16 : 0;  // wider groups: no strip
  // Bytes of a group's realignment buffer (short lanes).
  static constexpr int kRowBytes = K < 17 ? 8 * G * K : 0;
  // Bits of the word index in a row-max key ((h << kKeyBits) | (max - k) per half).
  static constexpr int kKeyBits =
      K <= 2 ? 1 : K <= 4 ? 2 : K <= 8 ? 3 : K <= 16 ? 4 : K <= 32 ? 5 : 6;
  static_assert(K <= 64, "a row-max key holds 6 bits of word index");
};

__device__ __forceinline__ uint32_t prmt(uint32_t a, uint32_t b, uint32_t sel) {
  uint32_t r;
  asm("prmt.b32 %0, %1, %2, %3;" : "=r"(r) : "r"(a), "r"(b), "r"(sel));
  return r;
}

// Bits of `y` where m is set, bits of `x` elsewhere (one LOP3).
__device__ __forceinline__ uint32_t bsel(uint32_t x, uint32_t y, uint32_t m) {
  return (x & ~m) | (y & m);
}

// Both halves of a packed word as the same 16-bit value (two's complement).
__host__ __device__ __forceinline__ uint32_t pk2(int32_t v) {
  return ((uint32_t)v & 0xFFFFu) * 0x10001u;
}

// (lo, hi) as an integer sum hi * 2^16 + lo: the form that 32-bit IADD adds per
// half when both halves' results stay inside [0, 2^16).
__host__ __device__ __forceinline__ uint32_t isum(int32_t lo, int32_t hi) {
  return (uint32_t)hi * 65536u + (uint32_t)lo;
}

// __shfl_sync within a group of G lanes (a group of one lane reads itself).
template <int G>
__device__ __forceinline__ uint32_t gshfl(uint32_t gmask, uint32_t v, int src) {
  if constexpr (G == 1) return v;
  else return __shfl_sync(gmask, v, src, G);
}

// Base classes. On long lanes the sweep keeps a window byte as a one-hot class: bit 0..3 for A, C,
// G, T, bit 4 for N, no bit for any other byte. A row whose read byte has class c
// shifts its window words left by 7 - c, which puts "equal" into the top bit of every
// byte: one shift per word instead of an XOR and a zero-byte test. A read byte outside
// the five classes compares the raw window bytes (a row of its own, reloaded after).
// Short lanes keep the raw bytes: for their few words the test costs no more than the
// classes of a row's two bytes.
__device__ __forceinline__ int32_t bsw16_class(uint32_t b) {  // -1: no class
  const uint32_t c = ((b >> 1) ^ (b >> 2)) & 3u;
  const uint32_t letter = (0x54474341u >> (8u * c)) & 0xFFu;  // "ACGT"
  return b == letter ? (int32_t)c : b == 0x4Eu ? 4 : -1;
}
__device__ __forceinline__ uint32_t bsw16_onehot(uint32_t b) {
  const int32_t c = bsw16_class(b);
  return c < 0 ? 0u : 1u << c;
}
// Four raw bytes as four one-hot bytes.
__device__ __forceinline__ uint32_t bsw16_onehot4(uint32_t w) {
  const uint32_t y = ((w >> 1) ^ (w >> 2)) & 0x03030303u;  // class of an ACGT byte
  const uint32_t sel = prmt(y | (y >> 4), 0u, 0x4420u);    // the four classes as nibbles
  auto zero = [](uint32_t t) {                             // 0x80 per zero byte
    return ~(((t & 0x7F7F7F7Fu) + 0x7F7F7F7Fu) | t) & 0x80808080u;
  };
  const uint32_t acgt = prmt(zero(w ^ prmt(0x54474341u, 0u, sel)), 0u, 0xBA98u);
  return (prmt(0x08040201u, 0u, sel) & acgt) | (zero(w ^ 0x4E4E4E4Eu) >> 3);
}

// Window bytes of a lane's cells as the sweep keeps them (word j: bytes of cells 2j
// and 2j + 1 of the low half and of the high half, in the order lo 2j, hi 2j,
// lo 2j+1, hi 2j+1), from the two runs of bytes starting at `a` (low-half cells) and
// `b` (high-half cells). Aligned 4-byte loads and funnel shifts: no word loaded
// lies past the one holding the window's last byte `last`, so bytes past the window
// end are whatever that word holds (those cells are never active). Short lanes: the
// bytes; long ones: one-hot classes (`raw` < 0), or 0x80 where the byte equals `raw`.
template <int K, bool CLASSES = (K >= 17)>
__device__ __forceinline__ void bsw16_window_words(uint32_t (&wb)[(K + 1) / 2],
                                                   const uint8_t* a, const uint8_t* b,
                                                   const uint8_t* last, int32_t raw) {
  constexpr int NW = (K + 1) / 2;
  const uintptr_t la = reinterpret_cast<uintptr_t>(last) & ~static_cast<uintptr_t>(3);
  const uintptr_t a0 = reinterpret_cast<uintptr_t>(a) & ~static_cast<uintptr_t>(3);
  const uintptr_t b0 = reinterpret_cast<uintptr_t>(b) & ~static_cast<uintptr_t>(3);
  const uint32_t sa = (static_cast<uint32_t>(reinterpret_cast<uintptr_t>(a)) & 3u) * 8u;
  const uint32_t sb = (static_cast<uint32_t>(reinterpret_cast<uintptr_t>(b)) & 3u) * 8u;
  const uint32_t q4 = static_cast<uint32_t>(raw) * 0x01010101u;
  auto at = [la](uintptr_t x) {
    return __ldg(reinterpret_cast<const uint32_t*>(x < la ? x : la));
  };
  auto enc = [raw, q4](uint32_t w) {
    if constexpr (!CLASSES) return w;
    const uint32_t t = w ^ q4;
    return raw < 0 ? bsw16_onehot4(w)
                   : ~(((t & 0x7F7F7F7Fu) + 0x7F7F7F7Fu) | t) & 0x80808080u;
  };
  // A loop that pushes two words a round through the array, its loads one round ahead.
  // (On long lanes a rolled one: unrolled, the loads in flight took the registers that
  // hold a third block per scheduler.)
  constexpr int kUnroll = K < 17 ? (NW > 1 ? NW / 2 : 1) : 1;
  uint32_t wa = at(a0), wv = at(b0), na = at(a0 + 4u), nb = at(b0 + 4u);
  auto next = [&](int m, uint32_t& ua, uint32_t& ub) {
    const uint32_t xa = at(a0 + 4u * (m + 2)), xb = at(b0 + 4u * (m + 2));
    ua = enc(__funnelshift_r(wa, na, sa));
    ub = enc(__funnelshift_r(wv, nb, sb));
    wa = na, wv = nb;
    na = xa, nb = xb;
  };
  uint32_t ua, ub;
  if constexpr (NW > 1) {
#pragma unroll kUnroll
    for (int m = 0; m < NW / 2; ++m) {
      next(m, ua, ub);
#pragma unroll
      for (int j = 0; j + 2 < NW; ++j) wb[j] = wb[j + 2];
      wb[NW - 2] = prmt(ua, ub, 0x5140u);
      wb[NW - 1] = prmt(ua, ub, 0x7362u);
    }
  }
  if constexpr (NW & 1) {
    next(NW / 2, ua, ub);
#pragma unroll
    for (int j = 0; j + 1 < NW; ++j) wb[j] = wb[j + 1];
    wb[NW - 1] = prmt(ua, ub, 0x5140u);
  }
}

// Moves a group's window words by one cell; `byte`: the new one-hot byte of the row
// capacity's last cell (used by the group's last lane).
template <int G, int K>
__device__ __forceinline__ void bsw16_window_step(uint32_t (&wb)[(K + 1) / 2], uint32_t byte,
                                                  int32_t gi, uint32_t gmask) {
  constexpr int NW = (K + 1) / 2;
  const uint32_t n0 = gshfl<G>(gmask, wb[0], (gi + 1) & (G - 1));
#pragma unroll
  for (int j = 0; j + 1 < NW; ++j) wb[j] = prmt(wb[j], wb[j + 1], 0x5432u);
  // The cell after this lane's last: the next lane's first (for the last lane, cell H
  // in the low half and the new byte in the high half).
  const uint32_t nx = gi == G - 1 ? prmt(n0, byte, 0x0041u) : n0;
  // Odd K: the last word holds cell K - 1 alone; even K: cells K - 2 and K - 1.
  wb[NW - 1] = (K & 1) ? nx : prmt(wb[NW - 1], nx, 0x5432u);
}

// Realignment of the previous row (the band moved other than one column): cell
// c <- old cell c + S, or c - S when DOWN; cells from outside the row capacity become
// neutral (those of the previous row at and beyond its length already are). Word k's
// halves hold cells g*K + k and H + g*K + k, so the S cells that cross a lane's end
// come from the next lane (for the last lane: cell H on = lane 0's high half in the
// low half, nothing in the high half), or the previous one when DOWN.
template <int G, int K, int S, bool DOWN>
__device__ __forceinline__ void bsw16_move(uint32_t (&v)[K], uint32_t neutral, int32_t gi,
                                           uint32_t gmask) {
  static_assert(S < K, "the cells that cross come from one lane");
  uint32_t x[S];
#pragma unroll
  for (int t = 0; t < S; ++t) {
    x[t] = DOWN ? gshfl<G>(gmask, v[K - S + t], (gi + G - 1) & (G - 1))
                : gshfl<G>(gmask, v[t], (gi + 1) & (G - 1));
    if (gi == (DOWN ? 0 : G - 1))
      x[t] = DOWN ? prmt(neutral, x[t], 0x5410u) : prmt(x[t], neutral, 0x5432u);
  }
  if constexpr (DOWN) {
#pragma unroll
    for (int k = K - 1; k >= S; --k) v[k] = v[k - S];
#pragma unroll
    for (int t = 0; t < S; ++t) v[t] = x[t];
  } else {
#pragma unroll
    for (int k = 0; k + S < K; ++k) v[k] = v[k + S];
#pragma unroll
    for (int t = 0; t < S; ++t) v[K - S + t] = x[t];
  }
}

// A realignment by s cells (either way). Long lanes: rolled loops of moves by 16, 4 and
// 1. (One code path per shift, or a round trip through shared memory, kept so many
// values alive at the joins that the one-lane shape took 212-255 registers; it takes 168
// this way, 12 warps per SM instead of 8, and no shared memory beside the trace strips.)
// Short lanes: each group stages the row as 16-bit halves in its own shared-memory strip
// [h: 2H][e: 2H], one pass for any shift.
template <int G, int K>
__device__ __forceinline__ void bsw16_realign(uint32_t (&ph)[K], uint32_t (&pe)[K], int32_t s,
                                              uint32_t b2, int32_t gi, uint32_t gmask,
                                              uint16_t* buf) {
  constexpr int H = G * K;
  if constexpr (K < 17) {
    const int32_t c0 = gi * K;
#pragma unroll
    for (int k = 0; k < K; ++k) {
      buf[c0 + k] = (uint16_t)(ph[k] & 0xFFFFu);
      buf[H + c0 + k] = (uint16_t)(ph[k] >> 16);
      buf[2 * H + c0 + k] = (uint16_t)(pe[k] & 0xFFFFu);
      buf[3 * H + c0 + k] = (uint16_t)(pe[k] >> 16);
    }
    __syncwarp(gmask);
    const uint32_t none = b2 & 0xFFFFu;
#pragma unroll
    for (int k = 0; k < K; ++k) {
      const uint32_t a = (uint32_t)(c0 + k + s), b = (uint32_t)(H + c0 + k + s);
      const bool va = a < 2u * H, vb = b < 2u * H;
      const uint32_t hl = va ? (uint32_t)buf[a] : none, hh = vb ? (uint32_t)buf[b] : none;
      const uint32_t el = va ? (uint32_t)buf[2 * H + a] : 0u, eh = vb ? (uint32_t)buf[2 * H + b] : 0u;
      ph[k] = hl | (hh << 16);
      pe[k] = el | (eh << 16);
    }
    __syncwarp(gmask);
  } else {
    // A shift by the capacity or more leaves neutral cells only.
    int32_t up = min(s, 2 * H), down = min(-s, 2 * H);
#pragma unroll 1
    for (; up >= 16; up -= 16) {
      bsw16_move<G, K, 16, false>(ph, b2, gi, gmask);
      bsw16_move<G, K, 16, false>(pe, 0u, gi, gmask);
    }
#pragma unroll 1
    for (; up >= 4; up -= 4) {
      bsw16_move<G, K, 4, false>(ph, b2, gi, gmask);
      bsw16_move<G, K, 4, false>(pe, 0u, gi, gmask);
    }
#pragma unroll 1
    for (; up > 0; --up) {
      bsw16_move<G, K, 1, false>(ph, b2, gi, gmask);
      bsw16_move<G, K, 1, false>(pe, 0u, gi, gmask);
    }
#pragma unroll 1
    for (; down >= 16; down -= 16) {
      bsw16_move<G, K, 16, true>(ph, b2, gi, gmask);
      bsw16_move<G, K, 16, true>(pe, 0u, gi, gmask);
    }
#pragma unroll 1
    for (; down >= 4; down -= 4) {
      bsw16_move<G, K, 4, true>(ph, b2, gi, gmask);
      bsw16_move<G, K, 4, true>(pe, 0u, gi, gmask);
    }
#pragma unroll 1
    for (; down > 0; --down) {
      bsw16_move<G, K, 1, true>(ph, b2, gi, gmask);
      bsw16_move<G, K, 1, true>(pe, 0u, gi, gmask);
    }
  }
}

// Activity mask of word k (0xFFFF per active half) from d0 = (2^15 + row_len - 1 -
// cell) per half of word 0: bit 15 of a half is set while its cell is inside the
// row, and PRMT replicates it over the half.
__device__ __forceinline__ uint32_t bsw16_act(uint32_t d0, int k) {
  uint32_t r;
  asm("prmt.b32 %0, %1, 0, 0xBB99;" : "=r"(r) : "r"(d0 - (uint32_t)k * 0x10001u));
  return r;
}

// Trace rows go to global memory in whole interleave blocks. A group stages the
// slabs of its current block (kInterleave rows, kStripBytes, laid out exactly
// as in global memory) in its own shared-memory strip and, once the block is complete
// (or the sweep ends), one lane copies the strip out with one bulk asynchronous copy
// (cp.async.bulk shared -> global): every DRAM sector is written whole, once, and the
// per-row stores stay in shared memory. The strip is reused after the copy has read
// it (wait_group.read before the next block's first store).
struct TraceStage {
  uint32_t* strip;    // this group's shared-memory strip (16-byte aligned)
  uint8_t* gtrace;    // the item's trace slot in global memory
  uint32_t bytes;     // kStripBytes: one interleave block
  bool dirty = false;     // rows staged since the last copy
  bool inflight = false;  // a copy of the strip may still be reading it
  int32_t blk = 0;        // block the staged rows belong to

  // Before a store into the strip: the previous copy has finished reading it.
  __device__ __forceinline__ void ready(uint32_t g, uint32_t gmask) {
    if (inflight) {
      if (g == 0) asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");
      __syncwarp(gmask);
      inflight = false;
    }
  }
  // Copies the staged block out (the group's stores are made visible to the async
  // proxy first; lane 0 issues the copy).
  __device__ __forceinline__ void flush(uint32_t g, uint32_t gmask) {
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    __syncwarp(gmask);
    if (g == 0) {
      const uint32_t src = (uint32_t)__cvta_generic_to_shared(strip);
      const uint8_t* dst = gtrace + (size_t)blk * bytes;
      asm volatile("cp.async.bulk.global.shared::cta.bulk_group [%0], [%1], %2;"
                   :: "l"(dst), "r"(src), "r"(bytes) : "memory");
      asm volatile("cp.async.bulk.commit_group;" ::: "memory");
    }
    inflight = true;
    dirty = false;
  }
};

// Waits until every bulk copy this thread issued has completed (end of a kernel).
__device__ __forceinline__ void bulk_copies_done() {
  asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");
}

template <int G, int K>
__device__ __forceinline__ void bsw16_group_sweep(
    const uint8_t* __restrict__ rd, uint32_t q, const uint8_t* __restrict__ wn, uint32_t w,
    int32_t band, int32_t offset, int32_t abort_score, const SwParams& sp, int32_t bias,
    uint16_t* rowbuf, uint32_t* strip, uint8_t* __restrict__ trace, uint32_t* __restrict__ meta,
    uint32_t g, uint32_t gmask, DpEnd& out, uint64_t& cells_out) {
  constexpr int H = G * K;
  constexpr int NW = Bsw16Shape<G, K>::kWords;
  constexpr int NS = Bsw16Shape<G, K>::kSlabs;
  constexpr int R = Bsw16Shape<G, K>::kInterleave;
  // Words at the end of each lane that every row masks; the others only in rows
  // shorter than the capacity by more than kEdge cells (5 for the shapes of 72 cells,
  // so the 67 cells of band 33 count as a full row).
  constexpr int kEdge = K < 4 ? K : K % 9 ? 4 : 5;
  // Short lanes (few words, many lanes): a row is bound by the latency of its chain,
  // not by its instructions. Rows with nothing unusual in any pair of the warp (the
  // band moved one column, a known base) then run as one straight line of code.
  constexpr bool kLatency = K < 17;
  // Groups of 8 lanes and more store whole 32-byte sectors themselves; fewer lanes
  // stage a block of rows (TraceStage).
  constexpr bool kStaged = G < 8;
  constexpr bool kClasses = !kLatency;  // window bytes as one-hot classes
  TraceStage ts{strip, trace, (uint32_t)Bsw16Shape<G, K>::kStripBytes};
  const int32_t gi = (int32_t)g;
  const int32_t c0 = gi * K;
  const int32_t match = sp.match, mism = sp.mismatch, gof = sp.gof, ge = sp.gap_extend;
  // Packed constants (per-half two's complement for DPX, integer sums for IADD). The
  // row keeps H - gof, the operand of both gap openings, so no row computes it twice;
  // the diagonal's scores carry the + gof back.
  const uint32_t B2 = pk2(bias), BG2 = pk2(bias - gof);
  const uint32_t MAT2 = pk2(match + gof), MIS2 = pk2(gof - mism), NGE2 = pk2(-ge);
  const uint32_t GOFS = isum(gof, gof), NGOF2 = pk2(-gof);
  const uint32_t GE65537 = (uint32_t)ge * 65537u, DEC0 = ge ? 65536u : 0u;  // pk2(-k * ge)
  // Per-half cell index of word 0 under 2^15 (the activity masks' d0 less row_len - 1).
  const uint32_t D0B = isum(0x8000 - 1 - c0, 0x8000 - 1 - H - c0);

  int32_t prev_start = 1, prev_len = 0;
  int32_t best = 0, bi = 0, bj = 0, bq = 0, bqj = 0;
  uint32_t early = 0;
  uint32_t cells = 0;  // < 2^32: read_len * row length
  const int32_t drift = sp.adaptive ? sp.max_drift : 0;
  int32_t acenter = 1 + offset;
  const int32_t wl = (int32_t)w;
  uint32_t ph[K], pe[K];  // the previous row's H - gof and E
#pragma unroll
  for (int k = 0; k < K; ++k) {
    ph[k] = BG2;
    pe[k] = 0u;
  }
  // Window bytes (long lanes: classes) of this lane's cells, four per word: word j holds cells 2j (low
  // half, high half) and 2j+1 (low, high) as bytes 0..3.
  uint32_t wb[NW];
#pragma unroll
  for (int j = 0; j < NW; ++j) wb[j] = 0u;
  bool raw_words = false;  // wb holds the last row's raw comparison, not classes

  // The read base of the next row is loaded a row ahead (its latency hides behind
  // the current row's work).
  uint32_t qb_next = q ? ldb(rd, 0) : 0u;
  uint32_t wnext = 0u;
  // Short lanes: the pairs of a warp go through their rows together, until the last of
  // them is done; the votes are also where the warp's groups meet again after rows that
  // took them through different code. (Long lanes have one code path, and the votes cost
  // the one-lane shape 13 %.)
  bool live = q > 0;
  for (uint32_t iu = 1; kLatency || iu <= q; ++iu) {
    const int32_t i = (int32_t)iu;
    const uint32_t qb = qb_next;
    const int32_t sc = i + offset;
    const int32_t center = sp.adaptive ? min(max(acenter, sc - drift), sc + drift) : sc;
    const int32_t js = max(center - band, 1);
    const int32_t je = min(center + band, wl);
    const int32_t row_len = je - js + 1;
    const int32_t sft = js - prev_start - 1;
    const int32_t qc = kClasses ? bsw16_class(qb) : 0;
    const uint32_t qb4 = qb * 0x01010101u;
    const bool plain = prev_len > 0 && sft == 0 && qc >= 0 && !raw_words &&
                       je >= prev_start + prev_len - 1 && js <= je;
    bool all_plain = false;
    if constexpr (kLatency) {
      all_plain = !__any_sync(0xFFFFFFFFu, live && !plain);
      if (!__any_sync(0xFFFFFFFFu, live)) break;
      if (!live) continue;
      live = iu < q;
    }
    if (iu < q) qb_next = ldb(rd, (uint64_t)iu);
    if (js > je) {  // mod.rs:1437-1444: row skipped, no centre / x-drop update
      if (g == 0) meta[i] = (1u << 11);
      if (kStaged && ts.dirty && (i & (R - 1)) == R - 1) ts.flush(g, gmask);
#pragma unroll
      for (int k = 0; k < K; ++k) {
        ph[k] = BG2;
        pe[k] = 0u;
      }
      prev_len = 0;
      prev_start = 1;
      continue;
    }
    cells += (uint32_t)row_len;
    // The row itself (fast: `plain` for every pair of the warp): the group's key of the
    // row maximum and its first cell.
    auto row = [&](auto fast_tag) -> uint32_t {
      constexpr bool fast = decltype(fast_tag)::value;
      if constexpr (!fast) {
        if (sft != 0 && prev_len > 0)
          bsw16_realign<G, K>(ph, pe, sft, BG2, gi, gmask, rowbuf);
        if (je < prev_start + prev_len - 1) {
          // The band's right end moved back: the previous row's columns past it (cells
          // beyond row_len here) are in no row from now on until they read as neutral.
          // Everywhere else a cell outside its row has a neutral H, so its E decays to
          // the opening of a neutral cell by itself and needs no mask.
          const uint32_t d1 = D0B + isum(row_len + 1, row_len + 1);
#pragma unroll
          for (int k = 0; k < K; ++k) {
            const uint32_t m = bsw16_act(d1, k);
            ph[k] = bsel(BG2, ph[k], m);
            pe[k] &= m;
          }
        }
      }
      // Upper neighbours of the last word: the next lane's first word; for the last
      // lane the low half continues into cell H (lane 0's high half) and the high
      // half runs past the capacity (neutral).
      uint32_t nh = gshfl<G>(gmask, ph[0], (gi + 1) & (G - 1));
      uint32_t ne = gshfl<G>(gmask, pe[0], (gi + 1) & (G - 1));
      if (gi == G - 1) {
        nh = prmt(nh, BG2, 0x5432u);
        ne = prmt(ne, 0u, 0x5432u);
      }
      const uint8_t* wrow = wn + (js - 1);
      // The next row's new window byte if its band moves one column (index in
      // [js - 1, wl - 1]); used only by the group's last lane.
      const uint32_t wcur = wnext;
      if (gi == G - 1) wnext = __ldg(wn + js + min(2 * H - 1, wl - js - 1));
      // Window classes: cells past the window end hold any byte (they are never active
      // in this or a later row); cells past the row end hold real window bytes, so a
      // row whose band moved up to three columns takes the previous row's words moved by
      // as many cells (the group's last lane brings the new bytes in: the first, wcur,
      // was loaded during the previous row on the guess that the band moves one column,
      // i.e. wrow[min(2H - 1, wl - js)] for js = prev_start + 1), and a row whose band
      // stayed keeps them.
      if constexpr (fast) {
        bsw16_window_step<G, K>(wb, kClasses ? bsw16_onehot(wcur) : wcur, gi, gmask);
      } else {
        const bool reload = prev_len == 0 || raw_words || qc < 0 || sft < -1 || sft > 2;
        const int32_t steps = reload ? 0 : sft + 1;
        uint32_t nb = wcur;
#pragma unroll 1
        for (int32_t t = 0; t < steps; ++t) {
          bsw16_window_step<G, K>(wb, kClasses ? bsw16_onehot(nb) : nb, gi, gmask);
          const int32_t j = prev_start + 2 + t;  // the band start after the next step
          if (gi == G - 1 && t + 1 < steps) nb = __ldg(wn + (j - 1) + min(2 * H - 1, wl - j));
        }
        if (reload) {
          raw_words = kClasses && qc < 0;
          bsw16_window_words<K>(wb, wrow + c0, wrow + H + c0, wn + (wl - 1),
                                raw_words ? (int32_t)qb : -1);
        }
      }
      const uint32_t qsh = raw_words ? 0u : (uint32_t)(7 - qc);
      // E, then H of every cell without the F that enters the lane (or the half) from
      // before it; the F chain of the lane's own cells runs along. Each word is replaced
      // in place: word k reads only words k and k + 1 of the previous row.
      uint32_t z = 0u, f = 0u;
#pragma unroll
      for (int k = 0; k < K; ++k) {
        if ((k & 1) == 0) {  // top bit of each byte: equal (raw bytes: different)
          if constexpr (kClasses) {
            z = wb[k >> 1] << qsh;
          } else {
            const uint32_t x = wb[k >> 1] ^ qb4;
            z = x | ((x & 0x7F7F7F7Fu) + 0x7F7F7F7Fu);
          }
        }
        const uint32_t uh = k + 1 < K ? ph[k + 1 < K ? k + 1 : 0] : nh;
        const uint32_t ue = k + 1 < K ? pe[k + 1 < K ? k + 1 : 0] : ne;
        const uint32_t e = __viaddmax_s16x2(ue, NGE2, uh);  // max(E_up - ge, H_up - gof)
        // The cell's top bit replicated over its half.
        const uint32_t ms = prmt(z, 0u, (k & 1) ? 0xBBAAu : 0x9988u);
        const uint32_t hm = __viaddmax_s16x2(
            ph[k], kClasses ? bsel(MIS2, MAT2, ms) : bsel(MAT2, MIS2, ms), B2);  // max(Hdiag + s, 0)
        if constexpr (kLatency) {  // one operation a word on the F chain
          const uint32_t t = __vimax_s16x2_relu(hm, e) - GOFS;
          ph[k] = __viaddmax_s16x2(f, NGOF2, t);  // H - gof
          f = __viaddmax_s16x2(f, NGE2, t);       // max(F - ge, max(Hdiag + s, E) - gof)
        } else {  // one operation fewer
          const uint32_t t = __vimax3_s16x2(hm, e, f) - GOFS;  // H - gof
          f = __viaddmax_s16x2(f, NGE2, t);                    // max(F - ge, H - gof)
          ph[k] = t;
        }
        pe[k] = e;
      }
      // F entering each lane's first cell from the cells before it: the decayed maximum
      // over the lanes before it, where the high half also sees every low-half cell.
      // (F is linear in (max, +), so it joins the lane's own chain afterwards.)
      uint32_t excl, tot;
      if constexpr (G == 1) {  // one lane: nothing before it, the total is its own
        excl = 0u;
        tot = f;
      } else if constexpr (G == 2) {  // two lanes: one exchange gives both the prefix and the total
        const uint32_t other = __shfl_xor_sync(gmask, f, 1, G);
        const uint32_t first = gi == 0 ? f : other, last = gi == 0 ? other : f;
        tot = __viaddmax_s16x2(first, pk2(-K * ge), last);
        excl = gi == 0 ? 0u : other;
      } else {
        uint32_t v = f;
#pragma unroll
        for (int off = 1; off < G; off <<= 1) {
          const uint32_t tt = __shfl_up_sync(gmask, v, off, G);
          if (gi >= off) v = __viaddmax_s16x2(tt, pk2(-off * K * ge), v);
        }
        excl = __shfl_up_sync(gmask, v, 1, G);
        if (gi == 0) excl = 0u;
        tot = __shfl_sync(gmask, v, G - 1, G);
      }
      excl = __viaddmax_s16x2(prmt(tot, 0u, 0x1054u), pk2(-c0 * ge) & 0xFFFF0000u, excl);
      excl = __viaddmax_s16x2(excl, NGOF2, 0u);  // F - gof, beside H - gof
      const uint32_t d0 = D0B + isum(row_len, row_len);
#pragma unroll
      for (int k = 0; k < K; ++k) {
        // pk2(-k * ge), as one multiply-add per word and row: hoisted out of the row loop
        // the K constants would take K registers.
        uint32_t dec = 0u;
        if (k) asm volatile("mad.lo.u32 %0, %1, %2, %3;" : "=r"(dec) : "r"(GE65537), "r"(-k), "r"(DEC0));
        ph[k] = __viaddmax_s16x2(excl, dec, ph[k]);
        // Cells at and beyond the row length become neutral: the last words in every
        // row, all of them in a row cut by a window edge (or of a narrower band). The
        // branch is taken by the pairs that need it; rows in the middle of a read skip it.
        if (fast || k >= K - kEdge) ph[k] = bsel(BG2, ph[k], bsw16_act(d0, k));
      }
      if (!fast && row_len < 2 * H - kEdge) {
#pragma unroll
        for (int k = 0; k < K - kEdge; ++k) ph[k] = bsel(BG2, ph[k], bsw16_act(d0, k));
      }
      // The row's trace: the low byte of every cell's H - gof + bias, words 2x and 2x + 1
      // in one 32-bit slab (cells lo 2x, hi 2x, lo 2x+1, hi 2x+1).
      // Layout [row block][slab][row in block][lane] of 4-byte slabs: a group's lanes
      // fill one contiguous G x 4-byte run per slab and row. The block is staged in
      // the group's strip and copied out whole (TraceStage).
      uint32_t* trow;
      if constexpr (kStaged) {
        ts.ready(g, gmask);
        ts.blk = i / R;
        trow = ts.strip + (i & (R - 1)) * G + g;
      } else {
        trow = reinterpret_cast<uint32_t*>(trace + (size_t)(i / R) * Bsw16Shape<G, K>::kStripBytes) +
               (i & (R - 1)) * G + g;
      }
#pragma unroll
      for (int x = 0; x < NS; ++x)
        trow[x * R * G] = prmt(ph[2 * x], 2 * x + 1 < K ? ph[2 * x + 1 < K ? 2 * x + 1 : 0] : 0u,
                               0x6420u);
      if constexpr (kStaged) {
        ts.dirty = true;
        if ((i & (R - 1)) == R - 1) ts.flush(g, gmask);
      }
      if (g == 0) meta[i] = ((uint32_t)js << 11) | (uint32_t)row_len;

      // Row max and its first cell: per half the key (h << KB) | (KM - k), whose
      // unsigned maximum carries the lowest k holding the max; then one 32-bit key per
      // lane (low-half cells precede high-half cells on ties).
      constexpr int KB = Bsw16Shape<G, K>::kKeyBits;
      constexpr uint32_t KM = (1u << KB) - 1u;
      uint32_t mx = 0u, mx1 = 0u;  // two running maxima (alternate word pairs)
#pragma unroll
      for (int k = 0; k < K; k += 2) {
        const uint32_t ka = ph[k] * (1u << KB) + (KM - (uint32_t)k) * 0x10001u;
        const uint32_t kb = k + 1 < K ? ph[k + 1 < K ? k + 1 : 0] * (1u << KB) +
                                            (KM - (uint32_t)(k + 1)) * 0x10001u
                                      : 0u;
        if (k & 2)
          mx1 = __vimax3_u16x2(mx1, ka, kb);
        else
          mx = __vimax3_u16x2(mx, ka, kb);
      }
      mx = __vimax3_u16x2(mx, mx1, 0u);
      const uint32_t vlo = (mx & 0xFFFFu) >> KB, vhi = mx >> (16 + KB);
      const bool lo_first = vlo >= vhi;
      const uint32_t idx = lo_first ? (uint32_t)c0 + (KM - (mx & KM))
                                    : (uint32_t)(H + c0) + (KM - ((mx >> 16) & KM));
      uint32_t key = ((lo_first ? vlo : vhi) << 11) | (2047u - idx);
      if constexpr (G == 32) {
        key = __reduce_max_sync(gmask, key);
      } else {
#pragma unroll
        for (int off = G / 2; off > 0; off >>= 1) key = max(key, __shfl_xor_sync(gmask, key, off, G));
      }
      return key;
    };
    uint32_t key;
    if constexpr (kLatency) key = all_plain ? row(std::true_type{}) : row(std::false_type{});
    else key = row(std::false_type{});
    const int32_t row_best = (int32_t)(key >> 11) - (bias - gof);
    const int32_t row_best_j = row_best > 0 ? js + (2047 - (int32_t)(key & 2047u)) : -1;
    if (row_best > best) {
      best = row_best;
      bi = i;
      bj = row_best_j;
    }
    if (iu == q && row_best > bq) {
      bq = row_best;
      bqj = row_best_j;
    }
    prev_start = js;
    prev_len = row_len;
    if (sp.adaptive) {  // mod.rs:1546-1559
      const int32_t raw = row_best_j >= 0 ? row_best_j + 1 : acenter + 1;
      const int32_t sn = i + 1 + offset;
      acenter = min(max(raw, sn - drift), sn + drift);
    }
    if (sp.dp_xdrop > 0 && best - row_best > sp.dp_xdrop) early = 1;  // mod.rs:1561-1564
    if (abort_score > kAbortOff) {  // mod.rs:1565-1572
      const int32_t remaining = (int32_t)(q - iu);
      if (best + remaining * match < abort_score) early = 1;
    }
    if (early) {
      if constexpr (kLatency) live = false;
      else break;
    }
  }
  // The last (partial) block, then the strip is free for the group's next item.
  if constexpr (kStaged) {
    if (ts.dirty) ts.flush(g, gmask);
    ts.ready(g, gmask);
  }
  if (bq > 0 && sat_add(bq, sp.clip) > best) {  // mod.rs:1575-1579
    best = bq;
    bi = (int32_t)q;
    bj = bqj;
  }
  out.score = best;
  out.end_i = bi;
  out.end_j = bj;
  out.early_abort = early;
  cells_out = cells;
}

// The packed full-window sweep of align_batch_simd (sw_batch_avx2_inner,
// src/alignment/mod.rs:1914-2135): every row covers columns 1 .. w, no band, no x-drop;
// same layout and trace as the banded sweep (row start 1, row length w). The row is
// bound by the latency and issue of its few words: the window stays in registers for
// the whole read, the diagonal predecessor is the word before, nothing moves.
//   Cells past the window (c >= w) never reach a cell inside it, and with their diagonal
// held at 0 their H never passes column w's (E and F decay from it alone), so a row's
// first maximum needs no mask. `rowkeys`: per-row keys for the group abort rule (null:
// no bound is active).
template <int G, int K>
__device__ __forceinline__ void bsw16_full_sweep(
    const uint8_t* __restrict__ rd, uint32_t q, const uint8_t* __restrict__ wn, uint32_t w,
    const SwParams& sp, int32_t bias, uint8_t* __restrict__ trace, uint32_t* __restrict__ meta,
    uint32_t g, uint32_t gmask, DpEnd& out, uint32_t* __restrict__ rowkeys) {
  constexpr int H = G * K;
  constexpr int NW = (K + 1) / 2;
  constexpr int NS = Bsw16Shape<G, K>::kSlabs;
  constexpr int R = Bsw16Shape<G, K>::kInterleave;
  constexpr int KB = Bsw16Shape<G, K>::kKeyBits;
  constexpr uint32_t KM = (1u << KB) - 1u;
  static_assert(G >= 8, "groups that store whole sectors");
  const int32_t gi = (int32_t)g, c0 = gi * K;
  const int32_t gof = sp.gof, ge = sp.gap_extend;
  const uint32_t B2 = pk2(bias), BG2 = pk2(bias - gof);
  const uint32_t MAT2 = pk2(sp.match + gof), MIS2 = pk2(gof - sp.mismatch), NGE2 = pk2(-ge);
  const uint32_t GOFS = isum(gof, gof), NGOF2 = pk2(-gof);
  const uint32_t GE65537 = (uint32_t)ge * 65537u, DEC0 = ge ? 65536u : 0u;  // pk2(-k * ge)
  const uint32_t d0 = isum(0x8000 - 1 - c0 + (int32_t)w, 0x8000 - 1 - H - c0 + (int32_t)w);
  uint32_t ph[K], pe[K], in[K], wb[NW];
#pragma unroll
  for (int k = 0; k < K; ++k) {
    ph[k] = BG2;
    pe[k] = 0u;
    in[k] = bsw16_act(d0, k);  // the cells inside the window
  }
  if (w) bsw16_window_words<K, false>(wb, wn + c0, wn + H + c0, wn + (w - 1), -1);
  int32_t best = 0, bi = 0, bj = 0, bq = 0, bqj = 0;
  uint32_t qb_next = q ? ldb(rd, 0) : 0u;
  for (uint32_t iu = 1; iu <= q; ++iu) {
    const int32_t i = (int32_t)iu;
    if (w == 0) {  // mod.rs:1437-1444
      if (g == 0) {
        meta[i] = (1u << 11);
        if (rowkeys) rowkeys[i] = 0;
      }
      continue;
    }
    const uint32_t qb4 = qb_next * 0x01010101u;
    if (iu < q) qb_next = ldb(rd, (uint64_t)iu);
    // The diagonal predecessor of a lane's first word: the previous lane's last word
    // (lane 0: column 0, H = 0, in the low half; cell H - 1 in the high half).
    uint32_t diag = __shfl_sync(gmask, ph[K - 1], (gi + G - 1) & (G - 1), G);
    if (gi == 0) diag = prmt(BG2, diag, 0x5410u);
    uint32_t z = 0u, f = 0u;
#pragma unroll
    for (int k = 0; k < K; ++k) {
      if ((k & 1) == 0) {  // top bit of each byte: different
        const uint32_t x = wb[k >> 1] ^ qb4;
        z = x | ((x & 0x7F7F7F7Fu) + 0x7F7F7F7Fu);
      }
      const uint32_t uh = ph[k];
      const uint32_t e = __viaddmax_s16x2(pe[k], NGE2, uh);  // max(E_up - ge, H_up - gof)
      const uint32_t ms = prmt(z, 0u, (k & 1) ? 0xBBAAu : 0x9988u);
      const uint32_t hm = bsel(B2, __viaddmax_s16x2(diag, bsel(MAT2, MIS2, ms), B2), in[k]);
      const uint32_t tg = __vimax_s16x2_relu(hm, e) - GOFS;
      ph[k] = __viaddmax_s16x2(f, NGOF2, tg);  // H - gof
      f = __viaddmax_s16x2(f, NGE2, tg);
      pe[k] = e;
      diag = uh;
    }
    uint32_t v = f;
#pragma unroll
    for (int off = 1; off < G; off <<= 1) {
      const uint32_t tt = __shfl_up_sync(gmask, v, off, G);
      if (gi >= off) v = __viaddmax_s16x2(tt, pk2(-off * K * ge), v);
    }
    uint32_t excl = __shfl_up_sync(gmask, v, 1, G);
    if (gi == 0) excl = 0u;
    const uint32_t tot = __shfl_sync(gmask, v, G - 1, G);
    excl = __viaddmax_s16x2(prmt(tot, 0u, 0x1054u), pk2(-c0 * ge) & 0xFFFF0000u, excl);
    excl = __viaddmax_s16x2(excl, NGOF2, 0u);
    uint32_t mx = 0u, mx1 = 0u, ka = 0u;
#pragma unroll
    for (int k = 0; k < K; ++k) {
      uint32_t dec = 0u;
      if (k) asm volatile("mad.lo.u32 %0, %1, %2, %3;" : "=r"(dec) : "r"(GE65537), "r"(-k), "r"(DEC0));
      ph[k] = __viaddmax_s16x2(excl, dec, ph[k]);
      const uint32_t kk = ph[k] * (1u << KB) + (KM - (uint32_t)k) * 0x10001u;
      if (k & 1) {
        if (k & 2) mx1 = __vimax3_u16x2(mx1, ka, kk);
        else mx = __vimax3_u16x2(mx, ka, kk);
      }
      ka = kk;
    }
    if (K & 1) mx = __vimax3_u16x2(mx, ka, 0u);
    mx = __vimax3_u16x2(mx, mx1, 0u);
    uint32_t* trow = reinterpret_cast<uint32_t*>(
                         trace + (size_t)(i / R) * Bsw16Shape<G, K>::kStripBytes) +
                     (i & (R - 1)) * G + g;
#pragma unroll
    for (int x = 0; x < NS; ++x)
      trow[x * R * G] = prmt(ph[2 * x], 2 * x + 1 < K ? ph[2 * x + 1 < K ? 2 * x + 1 : 0] : 0u,
                             0x6420u);
    const uint32_t vlo = (mx & 0xFFFFu) >> KB, vhi = mx >> (16 + KB);
    const bool lo_first = vlo >= vhi;
    const uint32_t idx = lo_first ? (uint32_t)c0 + (KM - (mx & KM))
                                  : (uint32_t)(H + c0) + (KM - ((mx >> 16) & KM));
    uint32_t key = ((lo_first ? vlo : vhi) << 11) | (2047u - idx);
    if constexpr (G == 32) {
      key = __reduce_max_sync(gmask, key);
    } else {
#pragma unroll
      for (int off = G / 2; off > 0; off >>= 1) key = max(key, __shfl_xor_sync(gmask, key, off, G));
    }
    const int32_t row_best = (int32_t)(key >> 11) - (bias - gof);
    const int32_t j = 1 + (2047 - (int32_t)(key & 2047u));
    if (g == 0) {
      meta[i] = (1u << 11) | w;
      if (rowkeys) rowkeys[i] = ((uint32_t)row_best << kKeyIdxBits) | (uint32_t)(1023 - (j - 1));
    }
    if (row_best > best) {
      best = row_best;
      bi = i;
      bj = j;
    }
    if (iu == q && row_best > bq) {
      bq = row_best;
      bqj = j;
    }
  }
  if (bq > 0 && sat_add(bq, sp.clip) > best) {
    best = bq;
    bi = (int32_t)q;
    bj = bqj;
  }
  out.score = best;
  out.end_i = bi;
  out.end_j = bj;
  out.early_abort = 0;
}

// Trace bytes of the packed sweep: hb(i, j) is the low byte of H of cell (i, j), or -1
// outside the row's band (row 0 and column 0 included). The row holds two halves of
// G*K band cells; in each, lane gi keeps cells gi*K .. +K-1, word kk of lane gi in
// slab kk/2, stored as [row block][slab][row in block][lane] of 4-byte slabs
// (Bsw16Shape::kInterleave rows per block).
template <int G, int K, bool STAGED_META = false>
struct Bsw16Trace {
  const uint8_t* __restrict__ trace;
  const uint32_t* __restrict__ meta;  // global, or the walk's shared-memory copy
  uint32_t zero;                      // the stored byte of H = 0 (bias - gof)
  __device__ __forceinline__ int32_t operator()(int32_t i, int32_t j) const {
    constexpr uint32_t H = Bsw16Shape<G, K>::kHalf, S = Bsw16Shape<G, K>::kRowStride;
    constexpr uint32_t R = Bsw16Shape<G, K>::kInterleave;
    if (i <= 0 || j <= 0) return -1;
    const uint32_t m = STAGED_META ? meta[i] : __ldg(meta + i);
    const int32_t rs = (int32_t)(m >> 11), rl = (int32_t)(m & 2047u);
    const int32_t idx = j - rs;
    if (idx < 0 || idx >= rl) return -1;
    const uint32_t hi = (uint32_t)idx >= H ? 1u : 0u;
    const uint32_t c = (uint32_t)idx - hi * H;
    const uint32_t gi = c / (uint32_t)K, kk = c - gi * (uint32_t)K;
    const uint32_t ib = (uint32_t)i & (R - 1u);
    const uint32_t b = __ldg(trace + (size_t)((uint32_t)i - ib) * S +
                             ((kk >> 1) * R + ib) * (G * 4u) + gi * 4u + (kk & 1u) * 2u + hi);
    return (int32_t)((b - zero) & 255u);
  }
};

// The reference's traceback (mod.rs:1581-1627) from H alone. The walk carries the
// exact value v of the H cell it stands on, starting from the end cell's score:
//   * the move is diagonal when H(i-1, j-1) + s(i, j) == v (out of band: 0 + s), which
//     has priority over E and E over F (mod.rs:1504-1516);
//   * else E when some cell g above in the same column, every row between in band,
//     has H == v + gof + (g - 1) * gap_extend: the first such g is where the
//     reference's E opens (it extends only when that is strictly better), and the cells
//     before it hold at most gap_open less;
//   * else F, the same along the row;
//   * a cell with v == 0 stops the walk.
// Stored values are H mod 256. While scores stay below 256 that is H itself. Above,
// a comparison can only be wrong towards a cell whose H is too low by a multiple of
// 256 (every predecessor's H is at most the value the move needs), and from then on v
// stays above the true H of the cell it stands on, which is 0 wherever a walk can end:
// a walk that ends with v != 0 took a wrong move and is reported (`lost`), and one
// that ends with v == 0 is the reference's. (Neighbouring cells rarely differ that
// much: scores per base above 255, or a jump at the band's edge.)
//
// In a diagonal run the 32 lanes take one cell each: a ballot of the matching bases and
// the popcount of the lower lanes' bits give each lane's v, and a ballot finds the
// first cell that is not diagonal. In a gap they take one length each, sixteen up the
// column and sixteen along the row at a time: a walk is a chain of dependent loads, and
// a gap is one of them (20k segments of 1-2 kb at 5-12 % error: 1775 -> 931 us against
// the column first and then the row, 32 lengths each).
template <class Trace>
__device__ __forceinline__ uint32_t warp_walk_h(const Trace& hb, int32_t& i, int32_t& j, int32_t v,
                                                const uint8_t* __restrict__ rd,
                                                const uint8_t* __restrict__ wn, const SwParams& sp,
                                                uint32_t* __restrict__ ops, uint32_t cap,
                                                uint32_t& overflow, bool& lost) {
  constexpr uint32_t kAll = 0xFFFFFFFFu;
  const int32_t lane = (int32_t)(threadIdx.x & 31u);
  uint32_t n = 0, cur_op = 0xFFu, cur_len = 0;
  auto emit = [&]() {
    if (!cur_len) return;
    if (n < cap) {
      if (lane == 0) ops[n] = (cur_len << 4) | cur_op;
    } else {
      overflow = 1;
    }
    ++n;
  };
  auto push = [&](uint32_t op, uint32_t cnt) {
    if (!cnt) return;
    if (op == cur_op) {
      cur_len += cnt;
      return;
    }
    emit();
    cur_op = op;
    cur_len = cnt;
  };
  auto first_of = [](uint32_t m) { return m ? (uint32_t)(__ffs(m) - 1) : 32u; };
  while (i > 0 && j > 0 && v > 0) {
    const int32_t ci = i - lane, cj = j - lane;
    const bool inside = ci > 0 && cj > 0;
    const int32_t p = hb(ci - 1, cj - 1);
    const bool eq = inside && rd[ci - 1] == wn[cj - 1];
    const int32_t step = eq ? sp.match : -sp.mismatch;
    const uint32_t eqm = __ballot_sync(kAll, eq);
    const int32_t before = __popc(eqm & ((1u << lane) - 1u));
    const int32_t vt = v - before * (sp.match + sp.mismatch) + lane * sp.mismatch;
    const bool diag = inside && vt > 0 && (p >= 0 ? ((p + step - vt) & 255) == 0 : vt == step);
    const uint32_t t = first_of(~__ballot_sync(kAll, diag));
    push(0u, t);
    i -= (int32_t)t;
    j -= (int32_t)t;
    v = __shfl_sync(kAll, t < 32u ? vt : vt - step, t < 32u ? (int)t : 31);
    if (t == 32u) continue;
    if (v <= 0 || i <= 0 || j <= 0) break;
    // A gap that ends here: lengths 1..16 up the column and along the row in one round
    // (the column goes first), then 32 lengths a round of the one still open.
    // Every cell the gap extends over holds at least the gap's value there, so H lies
    // in [target - gap_open, target]: the first cell outside that refutes the gap.
    auto gap = [&](int32_t base, int32_t di, int32_t dj) -> uint32_t {
      for (;; base += 32) {
        const int32_t g = base + lane;
        const int32_t h = hb(i - g * di, j - g * dj);
        const int32_t d = (v + sp.gof + (g - 1) * sp.gap_extend - h) & 255;
        const uint32_t out = first_of(__ballot_sync(kAll, h < 0 || d > sp.gap_open));
        const uint32_t at = first_of(__ballot_sync(kAll, h >= 0 && d == 0));
        if (at < out) return (uint32_t)base + at;
        if (out < 32u) return 0u;
      }
    };
    const bool along = lane >= 16;
    const int32_t g = (lane & 15) + 1;
    const int32_t h = hb(i - (along ? 0 : g), j - (along ? g : 0));
    const int32_t d = (v + sp.gof + (g - 1) * sp.gap_extend - h) & 255;
    const uint32_t outs = __ballot_sync(kAll, h < 0 || d > sp.gap_open);
    const uint32_t ats = __ballot_sync(kAll, h >= 0 && d == 0);
    auto first16 = [](uint32_t m) { return m ? (uint32_t)(__ffs(m) - 1) : 16u; };
    auto length = [&](uint32_t out, uint32_t at, int32_t di, int32_t dj) -> uint32_t {
      if (at < out) return at + 1u;
      return out < 16u ? 0u : gap(17, di, dj);
    };
    uint32_t op = 1u, len = length(first16(outs & 0xFFFFu), first16(ats & 0xFFFFu), 1, 0);
    if (!len) {
      op = 2u;
      len = length(first16(outs >> 16), first16(ats >> 16), 0, 1);
    }
    if (!len) break;  // no source: an earlier move was wrong (v != 0)
    push(op, len);
    if (op == 1u) i -= (int32_t)len;
    else j -= (int32_t)len;
    v += sp.gof + ((int32_t)len - 1) * sp.gap_extend;
  }
  lost = v != 0;
  emit();
  return n;
}

}  // namespace kira
