// myers.cuh -- Myers (1999) bit-parallel bounded edit distance, one pair per lane.
//
// Semantics: bounded_edit_distance (src/alignment/myers.rs:47-70) with the
// fixed/heap recurrences of :101-204 / :206-324 (identical results): semi-global
// (free text ends, whole pattern), best = minimum column score with the LAST
// column on ties (`err <= best`), exact early reject when neither the running
// best nor the current column can reach k. Text bytes outside ACGT match
// nothing; pattern bytes outside ACGT set no Peq bit.
//
// B200 mapping: the bit vector is held as L 32-bit limbs in registers (the
// reference uses 64-bit blocks; the limb width does not change any result). One lane
// per pair:
//   * pattern and text come from the 2-bit + valid plane arenas (planes.cuh):
//     one 32-base word is two 16-byte loads and a funnel shift, no cross-lane work;
//   * the pattern ends at the top bit of the top limb, whatever its length: the bits
//     below its first base are rows that match every base and start with no vertical
//     difference, so they stay rows of zeros -- the boundary the first base needs. No
//     limb is masked and the score change of a column is the top limb's top bit, for
//     patterns of different lengths in one warp alike (per-limb masks and a per-limb
//     choice of the top one were a third of the work: the stage took 356 us of 131k pairs
//     of 100-250 bases, now 195; 190 of 2M pairs of 150, now 66);
//   * Peq lives in shared memory as [k][code][lane] with code 4 = "matches
//     nothing" (only the rows below the pattern), so every per-lane read is
//     bank-conflict-free.
//   * Per column and limb: one LDS for Eq (instead of a 4-way select), the
//     (Eq & VP) + VP carry chain on the PTX carry flag (add.cc / addc), and one
//     funnel shift for each of the HP / HN shifts across limbs: ten operations on the
//     ALU pipe, which bounds it.
#pragma once

#include "addchain.cuh"
#include "common.cuh"
#include "planes.cuh"

namespace kira {

// Shared memory of one warp: Peq[k][code][lane], code 4 = "matches nothing".
struct MyersSmem {
  uint32_t* peq;  // [L][5][32]
};

// Rows of limb k below a pattern of m bases that ends at bit 32L - 1.
template <int L>
__device__ __forceinline__ uint32_t myers_below(int k, uint32_t m) {
  const int32_t lo = 32 * k - (int32_t)(32u * L - m);  // pattern position of the limb's bit 0
  return lo <= -32 ? 0xFFFFFFFFu : lo < 0 ? (1u << -lo) - 1u : 0u;
}

// Builds this lane's Peq columns from the pattern's plane words (no cross-lane
// work): eq_A = ~b1 & ~b0 & valid, ... and the rows below the pattern everywhere.
template <int L>
__device__ __forceinline__ void myers_build_peq(const uint4* __restrict__ planes, uint64_t pos,
                                                uint32_t m, uint32_t lane, MyersSmem sm) {
#pragma unroll
  for (int k = 0; k < L; ++k) {
    const int32_t lo = 32 * k - (int32_t)(32u * L - m);
    PlaneWord pw{0u, 0u, 0u};
    if (lo > -32) {
      pw = plane_word_at(planes, pos + (uint32_t)max(lo, 0));
      if (lo < 0) {
        pw.b0 <<= -lo;
        pw.b1 <<= -lo;
        pw.v <<= -lo;
      }
    }
    const uint32_t below = myers_below<L>(k, m);
    uint32_t* col = sm.peq + (uint32_t)k * 160u + lane;
    col[0] = (~pw.b1 & ~pw.b0 & pw.v) | below;
    col[32] = (~pw.b1 & pw.b0 & pw.v) | below;
    col[64] = (pw.b1 & ~pw.b0 & pw.v) | below;
    col[96] = (pw.b1 & pw.b0 & pw.v) | below;
    col[128] = below;
  }
}

// Runs the recurrence for this lane's pair (m <= 32 L). Returns true on a hit <= max_k;
// with WHERE, (dist, end) of the best column, else as soon as one column is a hit.
template <int L, bool WHERE>
__device__ __forceinline__ bool myers_lane(uint32_t m, uint32_t n, uint32_t max_k,
                                           MyersSmem sm, const uint4* __restrict__ tplanes,
                                           uint64_t tpos, uint32_t lane, uint32_t& dist,
                                           uint32_t& end_pos) {
  if (m == 0) {  // myers.rs:50-54
    dist = 0;
    end_pos = 0;
    return true;
  }
  if (n == 0) {  // myers.rs:55-58
    dist = m;
    end_pos = 0;
    return m <= max_k;
  }
  uint32_t vp[L], vn[L];
#pragma unroll
  for (int k = 0; k < L; ++k) {
    vp[k] = ~myers_below<L>(k, m);
    vn[k] = 0u;
  }
  const uint32_t* peq = sm.peq + lane;
  uint32_t err = m, best = m, pos = 0;
  if (!WHERE && m <= max_k) return true;
  // Column code: 0-3 for ACGT, 4 (the rows below the pattern alone) for any other base.
  auto load = [&](uint32_t b0, uint32_t b1, uint32_t v, uint32_t (&eq)[L]) {
    const uint32_t* pc = peq + ((v & 1u) ? ((b0 & 1u) | ((b1 & 1u) << 1)) : 4u) * 32u;
#pragma unroll
    for (int k = 0; k < L; ++k) eq[k] = pc[k * 160];
  };
  uint32_t j = 0;  // columns done
  auto column = [&](const uint32_t (&eq)[L]) {
    uint32_t av[L], sum[L];
#pragma unroll
    for (int k = 0; k < L; ++k) av[k] = eq[k] & vp[k];
    add_chain<L>(av, vp, sum);
    uint32_t hp_prev = 0, hn_prev = 0;
#pragma unroll
    for (int k = 0; k < L; ++k) {
      const uint32_t vpk = vp[k], vnk = vn[k];
      const uint32_t d0 = (sum[k] ^ vpk) | eq[k] | vnk;
      const uint32_t hp = vnk | ~(d0 | vpk);
      const uint32_t hn = d0 & vpk;
      const uint32_t hps = k ? __funnelshift_l(hp_prev, hp, 1) : (hp << 1);
      const uint32_t hns = k ? __funnelshift_l(hn_prev, hn, 1) : (hn << 1);
      hp_prev = hp;
      hn_prev = hn;
      vp[k] = hns | ~(d0 | hps);
      vn[k] = d0 & hps;
    }
    err = err + (hp_prev >> 31) - (hn_prev >> 31);
    ++j;
    if (WHERE) {
      if (err <= best) {
        best = err;
        pos = j;
      }
    } else {
      best = min(best, err);
    }
  };
  // Four columns a step: their Peq words are loaded together, ahead of the chain from
  // column to column, and the exits are tested once. The text plane word of the next 32
  // columns is loaded a block ahead.
  PlaneWord nw = plane_word_at(tplanes, tpos);
  for (uint32_t base = 0; base < n; base += 32u) {
    PlaneWord cw = nw;
    if (base + 32u < n) nw = plane_word_at(tplanes, tpos + base + 32u);
    uint32_t left = min(32u, n - base);
    for (; left >= 4u; left -= 4u) {
      uint32_t eq[4][L];
#pragma unroll
      for (int t = 0; t < 4; ++t) load(cw.b0 >> t, cw.b1 >> t, cw.v >> t, eq[t]);
      cw.b0 >>= 4;
      cw.b1 >>= 4;
      cw.v >>= 4;
#pragma unroll
      for (int t = 0; t < 4; ++t) column(eq[t]);
      if (!WHERE && best <= max_k) return true;
      // No later column can come down to k (myers.rs:194).
      if (best > max_k && err > max_k + (n - j)) return false;
    }
    for (; left; --left) {
      uint32_t eq[L];
      load(cw.b0, cw.b1, cw.v, eq);
      cw.b0 >>= 1;
      cw.b1 >>= 1;
      cw.v >>= 1;
      column(eq);
    }
  }
  if (!WHERE) return best <= max_k;
  if (best <= max_k) {
    dist = best;
    end_pos = pos;
    return true;
  }
  return false;
}

}  // namespace kira
