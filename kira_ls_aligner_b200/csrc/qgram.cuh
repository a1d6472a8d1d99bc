// qgram.cuh -- exact block filter in front of the Myers stage.
//
// The Myers stage (bounded_edit_distance, src/alignment/myers.rs:47-70) answers
// None unless the read (m bases) aligns to some substring T' of the window with at
// most k edits. T' has at least m - k bases, so of the window's blocks [5j, 5j + 5) at
// least floor((m - k - 4) / 5) lie inside it, and one edit (a substitution, a window
// base without a partner, or read bases between two window bases) touches at most one
// of them; every untouched block occurs verbatim in the read. So
//
//     ed <= k  implies  #{j : window block j occurs in the read} >= (m - k - 4) / 5 - k.
//
// A pair whose count is below that bound is a Myers None for certain, and the
// filter answers exactly that (the same MYERS_REJECT result and detail). Bases
// outside ACGT match nothing in Myers: each costs an edit of its own, so a block (or a
// read 5-gram) that contains one is left out. The filter only ever removes pairs Myers
// would reject, so every output is unchanged; survivors still run Myers.
//
// Why blocks of 5 and the read's set: the set of a read's 5-grams is 1024 bits, and a
// random window block is in it with probability about 145 / 1024 at 150 bases, 6.6 of
// 50 blocks, against a bound of 19 at k = 8. Only n / 5 look-ups per pair remain (a
// filter on all 4-grams, the window's set against the read's grams, took 247 inserts and
// 147 look-ups), and the candidates of one read, which lie next to each other in a
// batch, share one set: the lanes of a warp that hold the same read build it together.
// 2M pairs of 150 / 250 bp, 8 candidates a read: 0.38 -> 0.19 ms, now bound by the
// load/store pipe (plane loads 20M of 47M wavefronts, look-ups that meet in a bank 17M).
//
// A set is 32 words in shared memory, contiguous, one per distinct read of the warp: a
// 5-gram's code-bit-1 bits choose the word and its code-bit-0 bits the bit in it, both
// straight from the plane words.
#pragma once

#include "common.cuh"
#include "planes.cuh"

namespace kira {

constexpr uint32_t kQgram = 5, kQgramWords = 32;

// The bound above (<= 0: the filter proves nothing).
__device__ __forceinline__ int32_t qgram_need(uint32_t m, uint32_t k) {
  const int32_t inside = (int32_t)m - (int32_t)k - (int32_t)(kQgram - 1u);
  return inside > 0 ? inside / (int32_t)kQgram - (int32_t)k : 0;
}

// Positions whose kQgram bases from there on are all set in v (32 bases).
__device__ __forceinline__ uint32_t qgram_valid(uint32_t v) {
  return v & (v >> 1) & (v >> 2) & (v >> 3) & (v >> 4);
}

// Where the count of this lane's window blocks found in its read falls against two
// bounds lo <= hi: 0 when count >= hi, 1 when lo <= count < hi, 2 when count < lo. All 32
// lanes call; a lane with `active` false or hi <= 0 gets 0 (nothing is proved). `sets`:
// the warp's 32 x kQgramWords words.
__device__ __forceinline__ uint32_t qgram_outcome(bool active, const uint4* __restrict__ rplanes,
                                                  uint64_t rpos, uint32_t m,
                                                  const uint4* __restrict__ wplanes, uint64_t wpos,
                                                  uint32_t n, int32_t lo, int32_t hi,
                                                  uint32_t* sets) {
  constexpr uint32_t kAll = 0xFFFFFFFFu;
  const uint32_t lane = threadIdx.x & 31u;
  active = active && hi > 0 && m >= kQgram;
  if (!__any_sync(kAll, active)) return 0u;
  // Lanes with the same read (an inactive lane is alone: its key is no arena offset).
  const uint32_t same = __match_any_sync(kAll, active ? rpos : ~(uint64_t)lane) &
                        __match_any_sync(kAll, m);
  const uint32_t leader = (uint32_t)(__ffs(same) - 1), size = (uint32_t)__popc(same);
  const uint32_t rank = (uint32_t)__popc(same & ((1u << lane) - 1u));
  uint32_t* set = sets + leader * kQgramWords;
  if (active) {
    for (uint32_t w = rank; w < kQgramWords; w += size) set[w] = 0u;
  }
  __syncwarp();
  if (active) {
    constexpr uint32_t kUnit = 16;  // 5-gram starts a step: one plane word
    const uint32_t grams = m - (kQgram - 1u);
    for (uint32_t s = rank * kUnit; s < grams; s += size * kUnit) {
      const PlaneWord pw = plane_word_at(rplanes, rpos + s);
      const uint32_t ok = qgram_valid(pw.v) & low_mask(min(grams - s, kUnit));
      if (ok == low_mask(kUnit)) {
#pragma unroll
        for (uint32_t t = 0; t < kUnit; ++t)
          atomicOr(&set[(pw.b1 >> t) & 31u], 1u << ((pw.b0 >> t) & 31u));
      } else {
#pragma unroll
        for (uint32_t t = 0; t < kUnit; ++t)
          if ((ok >> t) & 1u) atomicOr(&set[(pw.b1 >> t) & 31u], 1u << ((pw.b0 >> t) & 31u));
      }
    }
  }
  __syncwarp();
  uint32_t count = 0;
  if (active) {
    // 160 bases (5 plane words) hold 32 blocks.
    for (uint32_t base = 0; base + kQgram <= n; base += 160u) {
      uint32_t b0[6], b1[6], all = 0xFFFFFFFFu, v[6];
#pragma unroll
      for (int k = 0; k < 5; ++k) {
        PlaneWord pw{0u, 0u, 0xFFFFFFFFu};  // past the window: no block counts there
        if (base + 32u * k < n) pw = plane_word_at(wplanes, wpos + base + 32u * k);
        b0[k] = pw.b0;
        b1[k] = pw.b1;
        v[k] = pw.v;
        all &= pw.v;
      }
      b0[5] = b1[5] = v[5] = 0u;
      const uint32_t blocks = min((n - base) / kQgram, 32u);
      uint32_t hits = 0;  // block j at bit 31 - j
#pragma unroll
      for (int j8 = 0; j8 < 32; j8 += 8) {
        if ((uint32_t)j8 < blocks) {
#pragma unroll
          for (int j = j8; j < j8 + 8; ++j) {
            const int at = (int)kQgram * j, k = at / 32, o = at % 32;
            const uint32_t x1 = o <= 27 ? b1[k] >> o : __funnelshift_r(b1[k], b1[k + 1], o);
            const uint32_t x0 = o <= 27 ? b0[k] >> o : __funnelshift_r(b0[k], b0[k + 1], o);
            hits = 2u * hits + ((set[x1 & 31u] >> (x0 & 31u)) & 1u);
          }
        } else {
          hits <<= 8;
        }
      }
      if (all != 0xFFFFFFFFu) {  // some base outside ACGT (perhaps past the window)
        uint32_t ok = 0;
#pragma unroll
        for (int j = 0; j < 32; ++j) {
          const int at = (int)kQgram * j, k = at / 32, o = at % 32;
          const uint32_t x = __funnelshift_r(v[k], v[k + 1], o);
          ok = 2u * ok + ((x & 31u) == 31u ? 1u : 0u);
        }
        hits &= ok;
      }
      count += (uint32_t)__popc(hits & ~low_mask(32u - blocks));
    }
  }
  __syncwarp();  // the sets are free for the next pairs
  if (!active) return 0u;
  return (int32_t)count < lo ? 2u : (int32_t)count < hi ? 1u : 0u;
}

}  // namespace kira
