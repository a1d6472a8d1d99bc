// planes.cuh -- 2-bit + valid bit planes of ASCII sequence arenas.
//
// Block b of a plane arena covers bases 32b .. 32b+31 of the byte arena it was
// built from: {x: code bit 0, y: code bit 1, z: ACGT-valid, w: exactly an upper-case
// A, C, G or T}, one bit per base (bit i = base 32b + i). Where w is set, equal codes
// are equal bytes. Codes and validity are encode_base / is_acgt of
// src/alignment/bitpacked.rs:12-20,89-91 (A0 C1 G2 T3, lower case folded, every
// other byte code 0 and invalid). Sieve and Myers need nothing else from a base,
// so both read their sequences as plane words: 32 consecutive bases starting at
// any position are two 16-byte loads and one funnel shift per plane.
#pragma once

#include <type_traits>

#include "common.cuh"

namespace kira {

struct PlaneWord {
  uint32_t b0, b1, v;
};

// 32 bases starting at base position `pos` of the arena (bits beyond the arena's
// end are whatever padding the planes hold; callers mask by length).
__device__ __forceinline__ PlaneWord plane_word_at(const uint4* __restrict__ planes, uint64_t pos) {
  const uint64_t blk = pos >> 5;
  const uint32_t off = (uint32_t)pos & 31u;
  const uint4 a = __ldg(planes + blk);
  const uint4 b = __ldg(planes + blk + 1);
  PlaneWord w;
  w.b0 = __funnelshift_r(a.x, b.x, off);
  w.b1 = __funnelshift_r(a.y, b.y, off);
  w.v = __funnelshift_r(a.z, b.z, off);
  return w;
}

// As plane_word_at; `u`: the upper-case plane of the same bases.
__device__ __forceinline__ PlaneWord plane_word_at(const uint4* __restrict__ planes, uint64_t pos,
                                                   uint32_t& u) {
  const uint64_t blk = pos >> 5;
  const uint32_t off = (uint32_t)pos & 31u;
  const uint4 a = __ldg(planes + blk);
  const uint4 b = __ldg(planes + blk + 1);
  u = __funnelshift_r(a.w, b.w, off);
  return PlaneWord{__funnelshift_r(a.x, b.x, off), __funnelshift_r(a.y, b.y, off),
                   __funnelshift_r(a.z, b.z, off)};
}

__device__ __forceinline__ uint32_t low_mask(uint32_t nbits) {
  return nbits >= 32u ? 0xFFFFFFFFu : ((1u << nbits) - 1u);
}

}  // namespace kira

namespace kira {

// ---------------------------------------------------------------------------
// Lane-per-pair sieve on plane words (scan_best_with_second_raw semantics,
// src/alignment/bitpacked.rs:154-199; checked mode: a non-ACGT base in the read
// or the window gives None, as packed_scan_scratch, src/alignment/mod.rs:594-621).
// Per shift and 32 read bases: 2 funnel shifts, XOR, LOP3, POPC, add.
// ---------------------------------------------------------------------------
struct LaneSieve {
  bool hit;
  uint32_t shift, mism, second;  // second = 0xFFFFFFFF when absent
  // spectral_hit_is_certified (src/alignment/mod.rs:688-762) of the hit: 0 no, 1 yes, 2
  // open (a lower-case base: the caller compares the bytes).
  uint32_t cert;
};

// Bits of word k whose positions lie in [lo, hi).
__device__ __forceinline__ uint32_t span_mask(int k, uint32_t lo, uint32_t hi) {
  const uint32_t base = 32u * (uint32_t)k;
  return (hi > base ? low_mask(hi - base) : 0u) & ~(lo > base ? low_mask(lo - base) : 0u);
}

// spectral_hit_is_certified on plane words: every base involved is an upper-case ACGT,
// so a code mismatch is a byte mismatch. r0 / r1: the read; the window's words at the
// hit are loaded again. Byte loops over the same 150-base reads (one lane a pair, up to
// 600 dependent loads) made the survivor sieve 36 us for 64 pairs.
template <int RW>
__device__ __forceinline__ bool sieve_certified(const uint32_t (&r0)[RW], const uint32_t (&r1)[RW],
                                                uint32_t q, const uint4* __restrict__ wp,
                                                uint64_t at, uint32_t mism, bool strict) {
  uint32_t w0[RW], w1[RW];
  uint32_t pos0 = 0xFFFFFFFFu, pos1 = 0xFFFFFFFFu;
#pragma unroll
  for (int k = 0; k < RW; ++k) {
    PlaneWord pw{0u, 0u, 0u};
    if (32u * k < q) pw = plane_word_at(wp, at + 32u * k);
    w0[k] = pw.b0;
    w1[k] = pw.b1;
    uint32_t x = ((r0[k] ^ w0[k]) | (r1[k] ^ w1[k])) & span_mask(k, 0u, q);
    if (x && pos0 == 0xFFFFFFFFu) {
      pos0 = 32u * k + (uint32_t)(__ffs(x) - 1);
      x &= x - 1u;
    }
    if (x && pos1 == 0xFFFFFFFFu) pos1 = 32u * k + (uint32_t)(__ffs(x) - 1);
  }
  const uint32_t edge = min(q, 8u);
  if (pos0 < edge || pos0 + edge >= q) return false;
  if (mism == 2u && (pos1 < edge || pos1 + edge >= q || pos1 - pos0 <= 4u)) return false;
  const uint32_t p = pos0, suffix = q - (p + 1u);
  if (suffix < (strict ? 4u : 8u)) return true;
  // Mismatches of the read against the window moved by d bases, from the first mismatch
  // on: read[i] against ref[i - d] for i in [p + d, q), and ref[i + d] for i in [p, q - d).
  auto moved = [&](auto d_tag) -> bool {
    constexpr int d = decltype(d_tag)::value;
    uint32_t back = 0, fwd = 0;
#pragma unroll
    for (int k = 0; k < RW; ++k) {
      const uint32_t b0 = __funnelshift_l(k ? w0[k ? k - 1 : 0] : 0u, w0[k], d);
      const uint32_t b1 = __funnelshift_l(k ? w1[k ? k - 1 : 0] : 0u, w1[k], d);
      const uint32_t f0 = __funnelshift_r(w0[k], k + 1 < RW ? w0[k + 1 < RW ? k + 1 : 0] : 0u, d);
      const uint32_t f1 = __funnelshift_r(w1[k], k + 1 < RW ? w1[k + 1 < RW ? k + 1 : 0] : 0u, d);
      back += __popc(((r0[k] ^ b0) | (r1[k] ^ b1)) & span_mask(k, p + d, q));
      fwd += __popc(((r0[k] ^ f0) | (r1[k] ^ f1)) & span_mask(k, p, q - d));
    }
    return back <= 1u || fwd <= 1u;
  };
  if (moved(std::integral_constant<int, 1>{})) return false;
  return !(strict && suffix >= 6u && moved(std::integral_constant<int, 2>{}));
}

// RW: plane words of the read. MIXED: of the longest read among the warp's lanes; a
// lane's shorter read is masked word by word (one more operation a word and shift, where
// one variant per length in the warp ran them one after another).
template <int RW, bool MIXED>
__device__ __forceinline__ LaneSieve sieve_lane_rw(const uint4* __restrict__ rp, uint64_t rpos,
                                                   uint32_t q, const uint4* __restrict__ wp,
                                                   uint64_t wpos, uint32_t w, uint32_t max_mism,
                                                   bool strict) {
  LaneSieve o{false, 0, 0, 0xFFFFFFFFu, 0u};
  uint32_t r0[RW], r1[RW];
  uint32_t bad = 0, lower = 0;  // bases outside ACGT; bases that are not upper-case ACGT
  auto mask = [q](int k) {
    return MIXED ? span_mask(k, 0u, q) : k == RW - 1 ? low_mask(q - 32u * (RW - 1)) : 0xFFFFFFFFu;
  };
#pragma unroll
  for (int k = 0; k < RW; ++k) {
    uint32_t u = 0u;
    PlaneWord pw{0u, 0u, 0u};
    if (!MIXED || 32u * k < q) pw = plane_word_at(rp, rpos + 32u * k, u);
    const uint32_t m = mask(k);
    r0[k] = pw.b0 & m;
    r1[k] = pw.b1 & m;
    bad |= ~pw.v & m;
    lower |= ~u & m;
  }
  uint32_t w0[RW + 1], w1[RW + 1];
  auto window = [&](uint32_t base, uint32_t& b0, uint32_t& b1) {
    b0 = b1 = 0u;
    if (MIXED && base >= w) return;
    uint32_t u;
    const PlaneWord pw = plane_word_at(wp, wpos + base, u);
    b0 = pw.b0;
    b1 = pw.b1;
    if (base < w) {
      bad |= ~pw.v & low_mask(w - base);
      lower |= ~u & low_mask(w - base);
    }
  };
#pragma unroll
  for (int k = 0; k <= RW; ++k) window(32u * k, w0[k], w1[k]);
  uint32_t rm[MIXED ? RW : 1];  // the read's positions
  if constexpr (MIXED) {
#pragma unroll
    for (int k = 0; k < RW; ++k) rm[k] = mask(k);
  }
  const uint32_t tail_mask = mask(RW - 1);
  const uint32_t n_shifts = w - q + 1u;
  uint32_t best = 0xFFFFFFFFu, second = 0xFFFFFFFFu;
  uint32_t t = 0;
  for (uint32_t blk = 0;; ++blk) {
    const uint32_t tend = min(n_shifts, t + 32u);
    for (; t < tend; ++t) {
      const uint32_t sh = t & 31u;
      uint32_t mism = 0;
#pragma unroll
      for (int k = 0; k < RW; ++k) {
        const uint32_t a0 = __funnelshift_r(w0[k], w0[k + 1], sh);
        const uint32_t a1 = __funnelshift_r(w1[k], w1[k + 1], sh);
        uint32_t x = (r0[k] ^ a0) | (r1[k] ^ a1);
        if constexpr (MIXED) x &= rm[k];
        else if (k == RW - 1) x &= tail_mask;
        mism += __popc(x);
      }
      const uint32_t key = (mism << 20) | t;
      if (key < best) {
        second = best;
        best = key;
      } else if (key < second) {
        second = key;
      }
    }
    if (t >= n_shifts) break;
    // slide one word: window words blk+1 .. blk+1+RW
#pragma unroll
    for (int k = 0; k < RW; ++k) {
      w0[k] = w0[k + 1];
      w1[k] = w1[k + 1];
    }
    window(32u * (blk + 1u + RW), w0[RW], w1[RW]);
  }
  if (bad) return o;
  o.hit = true;
  o.shift = best & 0xFFFFFu;
  o.mism = best >> 20;
  o.second = second == 0xFFFFFFFFu ? 0xFFFFFFFFu : (second >> 20);
  if (o.mism <= max_mism && o.second > o.mism + 1u && o.mism <= 2u) {
    if (o.mism == 0u) o.cert = 1u;
    else if (lower) o.cert = 2u;
    else o.cert = sieve_certified<RW>(r0, r1, q, wp, wpos + o.shift, o.mism, strict) ? 1u : 0u;
  }
  return o;
}

template <int RWMAX>
__device__ __forceinline__ LaneSieve sieve_lane(const uint4* rp, uint64_t rpos, uint32_t q,
                                                const uint4* wp, uint64_t wpos, uint32_t w,
                                                uint32_t max_mism, bool strict) {
  LaneSieve none{false, 0, 0, 0xFFFFFFFFu, 0u};
  if (q == 0 || w < q) return none;
  const uint32_t lanes = __activemask();
  const uint32_t rw = (q + 31u) / 32u, top = __reduce_max_sync(lanes, rw);
  const bool mixed = __any_sync(lanes, rw != top);
  switch (top) {
#define KIRA_LSIEVE_CASE(n)                                                                       \
  case n:                                                                                         \
    if (n <= RWMAX)                                                                               \
      return mixed ? sieve_lane_rw<(n <= RWMAX ? n : 1), true>(rp, rpos, q, wp, wpos, w,          \
                                                               max_mism, strict)                  \
                   : sieve_lane_rw<(n <= RWMAX ? n : 1), false>(rp, rpos, q, wp, wpos, w,         \
                                                                max_mism, strict);                \
    break;
    KIRA_LSIEVE_CASE(1) KIRA_LSIEVE_CASE(2) KIRA_LSIEVE_CASE(3) KIRA_LSIEVE_CASE(4)
    KIRA_LSIEVE_CASE(5) KIRA_LSIEVE_CASE(6) KIRA_LSIEVE_CASE(7) KIRA_LSIEVE_CASE(8)
    KIRA_LSIEVE_CASE(9) KIRA_LSIEVE_CASE(10) KIRA_LSIEVE_CASE(11) KIRA_LSIEVE_CASE(12)
    KIRA_LSIEVE_CASE(13) KIRA_LSIEVE_CASE(14) KIRA_LSIEVE_CASE(15) KIRA_LSIEVE_CASE(16)
#undef KIRA_LSIEVE_CASE
    default:
      break;
  }
  return none;
}

}  // namespace kira
