// wfa.cu -- the WFA batch kernel (wfa.cuh) and its CIGAR compaction.
#include <cuda_runtime.h>

#include "internal.h"
#include "wfa.cuh"

namespace kira {

namespace {

constexpr unsigned kFull = 0xFFFFFFFFu;

// router::wfa_score_budget (src/alignment/router.rs:160-165).
__device__ __forceinline__ int32_t wfa_budget(int read_len, const WfaLaunch& L) {
  const int64_t mism = (int64_t)read_len * L.budget_pct / 100 * L.budget_x;
  const int64_t indel = ((int64_t)L.budget_o + (int64_t)L.budget_e * 4) * 3;
  const int64_t b = mism > indel ? mism : indel;
  return b > INT32_MAX ? INT32_MAX : (int32_t)b;
}

__device__ __forceinline__ int wfa_low_bit(unsigned b) { return __ffs(b) - 1; }
__device__ __forceinline__ int wfa_high_bit(unsigned b) { return 31 - __clz(b); }

// Traceback in one lane (build_cigar, wfa.rs:762-952). Ops are pushed in reverse
// order into the pair's slot with push_cigar's merging (wfa.rs:954-962); returns
// the diagonal at termination (the alignment's text start). get(layer, score, k)
// returns the stored offset or kWfaNone.
template <class Get>
__device__ int wfa_traceback_t(const WfaLaunch& L, Get get, int m, int n, int s, int k,
                               uint32_t* __restrict__ slot, uint32_t& nops, bool& overflow) {
  uint32_t last = 0xFFFFFFFFu;  // op of the newest entry
  auto push = [&](uint32_t op, uint32_t len) {
    if (last == op) {
      if (nops <= L.slot_cap) slot[nops - 1] += len << 4;
      return;
    }
    if (nops < L.slot_cap) slot[nops] = (len << 4) | op;
    else overflow = true;
    ++nops;
    last = op;
  };
  const int x = L.x, oi = L.o + L.ei, od = L.o + L.ed;
  int off = m, layer = 0;
  for (uint32_t guard = 0; guard < (uint32_t)(2 * (m + n) + 8); ++guard) {
    if (s == 0 && layer == 0 && off == 0) break;
    if (layer == 0) {
      const int iv = get(1, s, k), dv = get(2, s, k);
      const int pv = s >= x ? get(0, s - x, k) : kWfaNone;
      // off is M[s][k] after its extension and the highest edge its value before, so
      // the bases between are equal: the walk (wfa.rs:807-853) down to the first landing
      // point of an edge at or below off needs no comparison.
      int low = max(0, -k);
      if (iv != kWfaNone && iv <= off) low = max(low, iv);
      if (dv != kWfaNone && dv <= off) low = max(low, dv);
      if (pv != kWfaNone && pv + 1 <= off) low = max(low, pv + 1);
      const int run = off > low ? off - low : 0;
      if (run > 0) push(0u, (uint32_t)run);
      off -= run;
      if (s == 0 && off == 0) break;
      if (pv != kWfaNone && pv + 1 == off) {
        push(0u, 1u);
        off -= 1;
        s -= x;
      } else if (iv == off) {
        layer = 1;
      } else if (dv == off) {
        layer = 2;
      } else {
        break;
      }
    } else if (layer == 1) {
      const int a = s >= oi ? get(0, s - oi, k + 1) : kWfaNone;
      if (a != kWfaNone && a + 1 == off) {
        push(1u, 1u);
        off -= 1, k += 1, s -= oi, layer = 0;
        continue;
      }
      const int b = s >= L.ei ? get(1, s - L.ei, k + 1) : kWfaNone;
      if (b != kWfaNone && b + 1 == off) {
        push(1u, 1u);
        off -= 1, k += 1, s -= L.ei;
        continue;
      }
      break;
    } else {
      const int a = s >= od ? get(0, s - od, k - 1) : kWfaNone;
      if (a != kWfaNone && a == off) {
        push(2u, 1u);
        k -= 1, s -= od, layer = 0;
        continue;
      }
      const int b = s >= L.ed ? get(2, s - L.ed, k - 1) : kWfaNone;
      if (b != kWfaNone && b == off) {
        push(2u, 1u);
        k -= 1, s -= L.ed;
        continue;
      }
      break;
    }
  }
  return k;
}

__device__ int wfa_traceback(const WfaLaunch& L, const int2* __restrict__ meta,
                             const int16_t* __restrict__ H, int m, int n, int s, int k,
                             uint32_t* __restrict__ slot, uint32_t& nops, bool& overflow) {
  auto get = [&](int layer, int sc, int kk) -> int {
    if (sc < 0) return kWfaNone;
    return wfa_get(H, wfa_unpack(meta[(uint32_t)sc * 3u + layer]), kk);
  };
  return wfa_traceback_t(L, get, m, n, s, k, slot, nops, overflow);
}

// G lanes align one pair; the 32 / G groups of a warp step in lockstep through
// an outer loop of three phases so that their warp instructions are shared:
//   fetch   -- groups without a pair take the next one and stage its bytes;
//   step    -- every group in the forward search computes its next score;
//   finish  -- groups whose search ended write the result (traceback in the
//              group's first lane).
// Sync primitives run on the full warp outside divergent code; each group reads
// its own bits of the ballots and shuffles from its own lanes.
template <int G, bool TB>
__global__ void __launch_bounds__(128) wfa_kernel(DevPairs P, WfaLaunch L) {
  constexpr int NG = 32 / G;
  constexpr unsigned kGroupBits = G == 32 ? kFull : ((1u << G) - 1u);
  extern __shared__ __align__(16) uint8_t wfa_smem[];
  const int lane = threadIdx.x & 31;
  const int g = lane / G, gl = lane % G, gbase = g * G;
  const unsigned gmask = kGroupBits << gbase;
  const uint32_t wib = threadIdx.x >> 5;
  const uint32_t grp = (blockIdx.x * (blockDim.x >> 5) + wib) * NG + (uint32_t)g;
  uint8_t* my = wfa_smem + (size_t)(wib * NG + (uint32_t)g) * L.smem_group;
  uint8_t* scr = L.scratch + (size_t)grp * L.group_bytes;
  int2* ring = L.ring_bytes ? (int2*)my : (int2*)(scr + L.ring_goff);
  uint32_t* pw = (uint32_t*)(my + L.ring_bytes + 16);
  uint32_t* tw = (uint32_t*)(my + L.ring_bytes + L.pat_region + 16);
  uint8_t* pb = (uint8_t*)pw;
  uint8_t* tb = (uint8_t*)tw;
  int2* meta = (int2*)scr;  // traceback: every score
  int16_t* H = (int16_t*)(scr + L.hist_off);
  const int x = L.x, oi = L.o + L.ei, od = L.o + L.ed;
  const uint32_t R = L.ring_len;

  int phase = 0;  // 0: needs a pair, 1: forward search, 2: no pairs left
  uint32_t p = 0, top = 0;
  int m = 0, n = 0, S_loop = 0, tbf = 0, s = 0, last_live = 0;
  for (;;) {
    // ---- fetch
    if (phase == 0) {
      uint32_t q = 0;
      if (gl == 0) q = atomicAdd(L.work, 1u);
      q = __shfl_sync(gmask, q, gbase);
      if (q >= (L.list ? min(*L.list_count, L.n) : L.n)) {
        phase = 2;
      } else {
        p = L.list ? L.list[q] : q;
        m = (int)P.read_len[p];
        n = (int)P.win_len[p];
        if (!L.valid || m == 0) {  // WfaCosts::scored refused: None; empty read: wfa.rs:555-563
          if (gl == 0) {
            kira_wfa_result res{};
            res.cost = L.valid ? 0 : -1;
            res.found = L.valid ? 1u : 0u;
            L.out[p] = res;
            if (TB) L.ncig[p] = 0;
          }
        } else {
          const uint8_t* rs = P.read_seq + P.read_off[p];
          const uint8_t* ws = P.win_seq + P.win_off[p];
          for (int i = gl; i < m; i += G) pb[i] = __ldg(rs + i);
          for (int i = gl; i < n; i += G) tb[i] = __ldg(ws + i);
          int S = L.max_score_pp ? L.max_score_pp[p] : L.max_score;
          if (!L.max_score_pp && S < 0) S = wfa_budget(m, L);
          // The all-insertion path reaches the pattern end by cost o + ei*m, so
          // the exact search ends by then; a pruned search advances its furthest
          // point by an antidiagonal at least every max(x, o + ei).
          const int64_t cap = L.drop < 0 ? (int64_t)L.o + (int64_t)L.ei * m
                                         : (int64_t)max(x, oi) * (2 * m + n + 2);
          S_loop = (int)max((int64_t)0, min((int64_t)S, cap));  // score 0 always runs
          tbf = L.tbf_pp ? L.tbf_pp[p] : L.tbf;
          tbf = min(max(tbf, 0), max(n - 1, 0));
          s = 0;
          top = 0;
          last_live = 0;
          phase = 1;
        }
      }
    }
    __syncwarp();
    if (__all_sync(kFull, phase == 2)) break;

    // ---- one score step of every searching group
    const bool fwd = phase == 1;
    int2 mv = wfa_empty();
    if (fwd && s > 0 && gl < 5) {  // M[s-x], M[s-o-ei], M[s-o-ed], I[s-ei], D[s-ed]
      const int sc = gl == 0 ? s - x : gl == 1 ? s - oi : gl == 2 ? s - od
                     : gl == 3 ? s - L.ei : s - L.ed;
      const int layer = gl < 3 ? 0 : gl - 2;
      if (sc >= 0 && sc < s) mv = ring[((uint32_t)sc % R) * 3u + layer];
    }
    WfaWave src[5];
#pragma unroll
    for (int t = 0; t < 5; ++t)
      src[t] = wfa_unpack(make_int2(__shfl_sync(kFull, mv.x, gbase + t),
                                    __shfl_sync(kFull, mv.y, gbase + t)));
    const WfaWave& mx = src[0];
    const WfaWave& moi = src[1];
    const WfaWave& mod = src[2];
    const WfaWave& ie = src[3];
    const WfaWave& de = src[4];
    int ilo = INT32_MAX, ihi = INT32_MIN, dlo = INT32_MAX, dhi = INT32_MIN;
    int mlo = INT32_MAX, mhi = INT32_MIN;
    if (fwd) {
      if (s == 0) {
        mlo = 0;
        mhi = tbf;
      } else {
        if (moi.hi >= moi.lo) ilo = min(ilo, moi.lo - 1), ihi = max(ihi, moi.hi - 1);
        if (ie.hi >= ie.lo) ilo = min(ilo, ie.lo - 1), ihi = max(ihi, ie.hi - 1);
        if (mod.hi >= mod.lo) dlo = min(dlo, mod.lo + 1), dhi = max(dhi, mod.hi + 1);
        if (de.hi >= de.lo) dlo = min(dlo, de.lo + 1), dhi = max(dhi, de.hi + 1);
        if (mx.hi >= mx.lo) mlo = min(mlo, mx.lo), mhi = max(mhi, mx.hi);
        if (ilo <= ihi) mlo = min(mlo, ilo), mhi = max(mhi, ihi);
        if (dlo <= dhi) mlo = min(mlo, dlo), mhi = max(mhi, dhi);
      }
    }
    const int iw = ilo <= ihi ? ihi - ilo + 1 : 0;
    const int dw = dlo <= dhi ? dhi - dlo + 1 : 0;
    const int mw = mlo <= mhi ? mhi - mlo + 1 : 0;
    uint32_t ib = 0, db = 0, mb = 0;
    int fin = 0;  // 1: found, 2: no alignment, 3: history bound exceeded
    if (fwd) {
      if (TB) {
        ib = top;
        db = ib + (uint32_t)iw;
        mb = db + (uint32_t)dw;
        top = mb + (uint32_t)mw;
        if (top > L.hist_cap || (uint32_t)s >= L.meta_slots) fin = 3;
      } else {
        const uint32_t sl = ((uint32_t)s % R) * 3u * L.ring_width;
        mb = sl;
        ib = sl + L.ring_width;
        db = sl + 2u * L.ring_width;
        if ((uint32_t)max(mw, max(iw, dw)) > L.ring_width) fin = 3;
      }
    }
    const int nch = fwd && !fin ? (mw + G - 1) / G : 0;
    const int maxch = __reduce_max_sync(kFull, nch);

    // Pass 1: I, D, M per diagonal; extension; trimming and done ballots.
    int ifirst = INT32_MAX, ilast = INT32_MIN, dfirst = INT32_MAX, dlast = INT32_MIN;
    int mfirst = INT32_MAX, mlast = INT32_MIN, kdone = INT32_MAX, mad = INT32_MIN;
    for (int c = 0; c < maxch; ++c) {
      const int c0 = mlo + c * G;
      const int k = c0 + gl;
      const bool act = c < nch && k <= mhi;
      int vi = kWfaNone, vd = kWfaNone, vm = kWfaNone;
      if (act) {
        if (s == 0) {
          vm = 0;
        } else {
          if (k >= ilo && k <= ihi) {
            const int a = wfa_get(H, moi, k + 1), b = wfa_get(H, ie, k + 1);
            if (a != kWfaNone && a < m) vi = max(vi, a + 1);
            if (b != kWfaNone && b < m) vi = max(vi, b + 1);
            H[ib + (uint32_t)(k - ilo)] = wfa_enc(vi);
          }
          if (k >= dlo && k <= dhi) {
            const int a = wfa_get(H, mod, k - 1), b = wfa_get(H, de, k - 1);
            if (a != kWfaNone && a + k <= n) vd = max(vd, a);
            if (b != kWfaNone && b + k <= n) vd = max(vd, b);
            H[db + (uint32_t)(k - dlo)] = wfa_enc(vd);
          }
          const int a = wfa_get(H, mx, k);
          if (a != kWfaNone && a < m && a + k < n) vm = a + 1;
          vm = max(vm, max(vi, vd));
        }
        if (vm != kWfaNone) {
          vm = wfa_extend(pw, tw, m, n, k, vm);
          mad = max(mad, 2 * vm + k);
        }
        H[mb + (uint32_t)(k - mlo)] = wfa_enc(vm);
      }
      const unsigned bi = (__ballot_sync(kFull, vi != kWfaNone) >> gbase) & kGroupBits;
      const unsigned bd = (__ballot_sync(kFull, vd != kWfaNone) >> gbase) & kGroupBits;
      const unsigned bm = (__ballot_sync(kFull, vm != kWfaNone) >> gbase) & kGroupBits;
      const unsigned bx = (__ballot_sync(kFull, act && vm >= m) >> gbase) & kGroupBits;
      if (bi) ifirst = min(ifirst, c0 + wfa_low_bit(bi)), ilast = c0 + wfa_high_bit(bi);
      if (bd) dfirst = min(dfirst, c0 + wfa_low_bit(bd)), dlast = c0 + wfa_high_bit(bd);
      if (bm) mfirst = min(mfirst, c0 + wfa_low_bit(bm)), mlast = c0 + wfa_high_bit(bm);
      if (bx && kdone == INT32_MAX) kdone = c0 + wfa_low_bit(bx);
    }
    // Pass 2 (adaptive): prune_wavefront on the extended M, then the done test.
    if (L.drop >= 0) {
#pragma unroll
      for (int o = G / 2; o > 0; o >>= 1) mad = max(mad, __shfl_xor_sync(kFull, mad, o));
      const bool prune = nch > 0 && mfirst <= mlast;
      const int th = prune ? mad - L.drop : 0;
      if (prune) mfirst = INT32_MAX, mlast = INT32_MIN, kdone = INT32_MAX;
      for (int c = 0; c < maxch; ++c) {
        const int c0 = mlo + c * G;
        const int k = c0 + gl;
        int v = kWfaNone;
        if (prune && c < nch && k <= mhi) {
          const uint32_t at = mb + (uint32_t)(k - mlo);
          v = wfa_dec(H[at]);
          if (v != kWfaNone && 2 * v + k < th) {
            v = kWfaNone;
            H[at] = wfa_enc(v);
          }
        }
        const unsigned bm = (__ballot_sync(kFull, v != kWfaNone) >> gbase) & kGroupBits;
        const unsigned bx = (__ballot_sync(kFull, v != kWfaNone && v >= m) >> gbase) & kGroupBits;
        if (prune) {
          if (bm) mfirst = min(mfirst, c0 + wfa_low_bit(bm)), mlast = c0 + wfa_high_bit(bm);
          if (bx && kdone == INT32_MAX) kdone = c0 + wfa_low_bit(bx);
        }
      }
    }
    if (fwd && !fin) {
      if (gl == 0) {
        const int2 wm = mfirst <= mlast ? wfa_pack(mfirst, mlast, mb + (uint32_t)(mfirst - mlo))
                                        : wfa_empty();
        const int2 wi = ifirst <= ilast ? wfa_pack(ifirst, ilast, ib + (uint32_t)(ifirst - ilo))
                                        : wfa_empty();
        const int2 wd = dfirst <= dlast ? wfa_pack(dfirst, dlast, db + (uint32_t)(dfirst - dlo))
                                        : wfa_empty();
        const uint32_t rs = ((uint32_t)s % R) * 3u;
        ring[rs + 0] = wm;
        ring[rs + 1] = wi;
        ring[rs + 2] = wd;
        if (TB) {
          meta[(uint32_t)s * 3u + 0] = wm;
          meta[(uint32_t)s * 3u + 1] = wi;
          meta[(uint32_t)s * 3u + 2] = wd;
        }
      }
      if (kdone != INT32_MAX) {
        fin = 1;
      } else if (s >= S_loop) {
        fin = 2;
      } else {
        // Nothing reached within the look-back window: no later score reaches anything.
        if (mfirst <= mlast || ifirst <= ilast || dfirst <= dlast) last_live = s;
        if (s - last_live > L.lookback) fin = 2;
        else ++s;
      }
    }
    __syncwarp();

    // ---- finish
    if (fwd && fin) {
      if (gl == 0) {
        kira_wfa_result res{};
        res.cost = -1;
        uint32_t nops = 0;
        if (fin == 3) {
          atomicOr(L.flags, 2u);
        } else if (fin == 1) {
          res.found = 1;
          res.cost = s;
          res.score = L.scored ? m * L.match - s : s;
          res.text_end = (uint32_t)(m + kdone);
          if (TB) {
            bool ovf = false;
            uint32_t* slot = L.slots + (size_t)p * L.slot_cap;
            const int k0 = wfa_traceback(L, meta, H, m, n, s, kdone, slot, nops, ovf);
            res.text_start = (uint32_t)max(k0, 0);
            if (ovf) atomicOr(L.flags, 1u);
          }
        }
        if (TB) L.ncig[p] = nops;
        L.out[p] = res;
      }
      phase = 0;
    }
    __syncwarp();
  }
}

// Bytes [0, len) of src to shared memory by the G lanes of a group, a word per lane
// at a time; reads only aligned words that hold one of the bytes. WIDE: word i of dst
// holds bytes i .. i + 3, so four bytes from any offset are one load.
template <int G, bool WIDE>
__device__ __forceinline__ void wfa_stage(uint32_t* dst, const uint8_t* src, int len, int gl) {
  const int a = (int)((uintptr_t)src & 3u);
  const uint32_t* w = (const uint32_t*)(src - a);
  const uint32_t sel = 0x3210u + 0x1111u * (uint32_t)a;
  for (int i = gl; 4 * i < len; i += G) {
    const uint32_t lo = __ldg(w + i);
    const uint32_t hi = 4 * (i + 1) < a + len ? __ldg(w + i + 1) : 0u;
    const uint32_t v = __byte_perm(lo, hi, sel);
    if (WIDE) {
      const uint32_t nx = __byte_perm(hi, 4 * (i + 2) < a + len ? __ldg(w + i + 2) : 0u, sel);
      ((uint4*)dst)[i] = make_uint4(v, __byte_perm(v, nx, 0x4321u), __byte_perm(v, nx, 0x5432u),
                                    __byte_perm(v, nx, 0x6543u));
    } else {
      dst[i] = v;
    }
  }
}

// wfa_extend over WIDE arrays (0 <= v <= m, 0 <= v + k <= n).
__device__ __forceinline__ int wfa_extend_wide(const uint32_t* pe, const uint32_t* te, int m,
                                               int n, int k, int v) {
  const uint32_t* a = pe + v;
  const uint32_t* b = te + v + k;
  const int lim = min(m - v, n - k - v);
  uint32_t d = a[0] ^ b[0];
  int run = 0;
  if (d == 0) {  // one diagonal of 256 off the alignment's path; 16 bytes a turn on it
    run = 4;
    while (run < lim) {
      const uint32_t d0 = a[run] ^ b[run], d1 = a[run + 4] ^ b[run + 4];
      const uint32_t d2 = a[run + 8] ^ b[run + 8], d3 = a[run + 12] ^ b[run + 12];
      if (d0 | d1 | d2 | d3) {
        if (!(d0 | d1)) run += 8;
        const uint32_t e0 = d0 | d1 ? d0 : d2, e1 = d0 | d1 ? d1 : d3;
        if (!e0) run += 4;
        d = e0 ? e0 : e1;
        break;
      }
      run += 16;
    }
  }
  if (d) run += (__ffs(d) - 1) >> 3;
  return v + min(run, lim);
}

// A reached cell of the window kernel's history: M before its extension (from bit 4),
// whether that came from I or D (else from M at a mismatch), and whether the cell's I
// and D opened there.
constexpr int kFromI = 1, kFromD = 2, kIOpen = 4, kDOpen = 8;

// Traceback over those cells in one lane: the edge order of wfa_traceback_t (mismatch,
// I, D; open before extend) was applied when the cell was computed, so a step is one
// load. hist is indexed by s * W + k.
__device__ int wfa_window_traceback(const WfaLaunch& L, const int* hist, int W, int m, int s,
                                    int k, uint32_t* __restrict__ slot, uint32_t& nops,
                                    bool& overflow) {
  uint32_t op = 0, len = 0;
  auto push = [&](uint32_t o, uint32_t l) {
    if (o != op) {
      if (len) {
        if (nops < L.slot_cap) slot[nops] = len << 4 | op;
        else overflow = true;
        ++nops;
      }
      op = o, len = 0;
    }
    len += l;
  };
  int off = m, layer = 0;
  while (s > 0) {
    const int c = hist[s * W + k];
    if (layer == 0) {
      const int pre = c >> 4;
      if (off > pre) push(0u, (uint32_t)(off - pre));
      off = pre;
      layer = c & 3;
      if (layer == 0) {
        push(0u, 1u);
        off -= 1, s -= L.x;
        continue;
      }
    }
    if (layer == kFromI) {
      push(1u, 1u);
      off -= 1, k += 1;
      layer = c & kIOpen ? 0 : kFromI;
      s -= L.ei + (layer ? 0 : L.o);
    } else {
      push(2u, 1u);
      k -= 1;
      layer = c & kDOpen ? 0 : kFromD;
      s -= L.ed + (layer ? 0 : L.o);
    }
  }
  if (off > 0) push(0u, (uint32_t)off);
  push(~0u, 0u);
  return k;
}

// Fixed-window WFA: G lanes per pair, the 32 / G pairs of a warp in lockstep over
// their rows (scores). Every cell the recurrence can reach by score smax lies in the
// window's `width` diagonals from `base` (an inserted base moves one diagonal down for
// at least ei, a deleted base one up for at least ed, the seeds sit on
// 0..text_begin_free); by score s that is lo = -(s - o) / ei to
// hi = text_begin_free + (s - o) / ed, taken G diagonals at a time from lo. Each layer
// keeps as many rows as the recurrence looks back in it, in a shared ring of int16
// with a guard column on each side; "none" is any negative value, so the reference's
// checks become plain max / select: an unreached source stays negative through the
// +1s of a search. A row's range only grows, so a slot never holds an older value
// outside it. Rows whose sources are all dead (scores 1-4 and 6 at mismatch 5, gaps 7
// and 8) are passed over: a bit per row tells which hold a value, and a dead source
// reads a row of "none". A group whose pair is done takes the next one when kWait
// groups are: a pair's cells grow with the square of its score, so a warp that waits
// for all its pairs idles most of its lanes. A pair not done by smax (and not
// exhausted) goes to fb_list.
//
// Bound by the instructions issued, 80 % of the slots: 1M pairs of 150 bases at 0-4 %
// error (265 cells a pair on average) 5.5 ms with the later passes, where a warp per
// pair over the whole window, with the offsets of every row kept for a traceback that
// compared bases again, took 8.7.
template <int G, bool TB, class Mask>
__global__ void __launch_bounds__(128) wfa_window_kernel(DevPairs P, WfaLaunch L, WfaWindow X) {
  constexpr int NG = 32 / G;
  constexpr bool kWide = G < 32;
  constexpr int kWait = (NG + 1) / 2;
  constexpr int kNone16 = -32000;
  extern __shared__ __align__(16) uint8_t wfa_smem[];
  const int lane = threadIdx.x & 31;
  const int g = lane / G, gl = lane % G, gbase = g * G;
  const unsigned gmask = (kFull >> (32 - G)) << gbase;
  const uint32_t wib = threadIdx.x >> 5;
  const int W = X.width, rowlen = W + 2, base = X.base;
  uint8_t* my = wfa_smem + (size_t)(wib * NG + (uint32_t)g) * X.group_bytes;
  uint32_t* pw = (uint32_t*)(my + X.ring_bytes + 16);
  uint32_t* tw = (uint32_t*)(my + X.ring_bytes + X.pat_bytes + 16);
  const int x = L.x, oi = L.o + L.ei, od = L.o + L.ed, ei = L.ei, ed = L.ed;
  const int rm = X.rows_m;                          // rows of M's ring
  const int ri = X.rows_i - 1, rd = X.rows_d - 1;  // of I's and D's - 1 (powers of two)
  int16_t* ringM = (int16_t*)my + 1 - base;
  int16_t* none_row = ringM + X.rows_m * rowlen;  // what a dead source reads
  int16_t* ringI = none_row + rowlen;
  int16_t* ringD = ringI + X.rows_i * rowlen;
  const uint32_t grp = (blockIdx.x * (blockDim.x >> 5) + wib) * NG + (uint32_t)g;
  int* hist = TB ? X.hist + (size_t)grp * (X.smax + 1) * W : nullptr;
  const Mask one = 1;
  const Mask bx = one << (x - 1), boi = one << (oi - 1), bod = one << (od - 1);
  const Mask bei = one << (ei - 1), bed = one << (ed - 1);
  const Mask in_ring = (one << L.lookback << 1) - one;
  const uint32_t count = X.list ? *X.list_count : L.n;

  bool alive = false, mine = false, dead = false, more = true;
  uint32_t p = 0;
  int m = 0, n = 0, S_loop = 0, s_lim = 0, tbf = 0;
  int s = 0, sm = 0, lo = 0, hi = 0, ci = 0, cd = 0;
  int done_s = -1, k_end = 0;
  Mask live_m = 0, live_g = 0;  // bit j: row s - 1 - j holds a value (in I or D)
  auto advance = [&]() {
    ++s;
    if (++sm == rm) sm = 0;
    if (++ci == ei) ci = 0, --lo;
    if (++cd == ed) cd = 0, ++hi;
  };
  for (;;) {
    const unsigned running = __ballot_sync(kFull, alive);
    const unsigned waiting = running == kFull ? 0u : __ballot_sync(kFull, !alive && (more || mine));
    if (!running && !waiting) break;
    if (!running || __popc(waiting) >= kWait * G) {
      if (mine && !alive && gl == 0) {  // finish
        if (done_s < 0 && !dead && S_loop > s_lim) {
          X.fb_list[atomicAdd(X.fb_count, 1u)] = p;  // redone from scratch
        } else {
          kira_wfa_result res{};
          res.cost = -1;
          uint32_t nops = 0;
          if (done_s >= 0) {
            res.found = 1;
            res.cost = done_s;
            res.score = L.scored ? m * L.match - done_s : done_s;
            res.text_end = (uint32_t)(m + k_end);
            if (TB) {
              bool ovf = false;
              const int k0 = wfa_window_traceback(L, hist - base, W, m, done_s, k_end,
                                                  L.slots + (size_t)p * L.slot_cap, nops, ovf);
              res.text_start = (uint32_t)max(k0, 0);
              if (ovf) atomicOr(L.flags, 1u);
            }
          }
          if (TB) L.ncig[p] = nops;
          L.out[p] = res;
        }
      }
      __syncwarp();
      uint32_t q = 0;
      if (!alive && more && gl == 0) q = atomicAdd(X.work, 1u);
      q = __shfl_sync(kFull, q, gbase);
      if (!alive) {
        mine = false;
        more = more && q < count;
        if (more) {
          p = X.list ? X.list[q] : q;
          m = (int)P.read_len[p], n = (int)P.win_len[p];
          if (!L.valid || m == 0) {  // WfaCosts::scored refused: None; empty read: wfa.rs:555-563
            if (gl == 0) {
              kira_wfa_result res{};
              res.cost = L.valid ? 0 : -1;
              res.found = L.valid ? 1u : 0u;
              L.out[p] = res;
              if (TB) L.ncig[p] = 0;
            }
          } else {
            alive = mine = true;
            for (uint32_t i = (uint32_t)gl; i < X.ring_bytes / 16u; i += G)
              ((uint4*)my)[i] = make_uint4(0x83008300u, 0x83008300u, 0x83008300u, 0x83008300u);
            wfa_stage<G, kWide>(pw, P.read_seq + P.read_off[p], m, gl);
            wfa_stage<G, kWide>(tw, P.win_seq + P.win_off[p], n, gl);
            int S = L.max_score_pp ? L.max_score_pp[p] : L.max_score;
            if (!L.max_score_pp && S < 0) S = wfa_budget(m, L);
            const int64_t cap = L.drop < 0 ? (int64_t)L.o + (int64_t)L.ei * m
                                           : (int64_t)max(x, oi) * (2 * m + n + 2);
            S_loop = (int)max((int64_t)0, min((int64_t)S, cap));
            s_lim = min(S_loop, X.smax);
            tbf = L.tbf_pp ? L.tbf_pp[p] : L.tbf;
            tbf = min(max(tbf, 0), max(n - 1, 0));
            s = sm = 0;
            lo = 0, hi = tbf, ci = cd = -L.o;
            done_s = -1;
            dead = false;
            live_m = live_g = 0;
          }
        }
      }
      __syncwarp();
      if (!__any_sync(kFull, alive)) continue;
    }

    // The next row with a live source.
    if (alive && s > 0) {
      while (!((live_m & (bx | boi | bod)) | (live_g & (bei | bed)))) {
        live_m <<= 1, live_g <<= 1;
        // Nothing reached within the look-back window: no later score reaches anything.
        dead = (live_m & in_ring) == 0;
        if (dead || s == s_lim) {
          alive = false;
          break;
        }
        advance();
      }
    }
    auto back = [&](int b) { return (sm - b + (sm < b ? rm : 0)) * rowlen; };
    const int16_t* rMx = live_m & bx ? ringM + back(x) : none_row;
    const int16_t* rMoi = (live_m & boi ? ringM + back(oi) : none_row) + 1;
    const int16_t* rMod = (live_m & bod ? ringM + back(od) : none_row) - 1;
    const int16_t* rIe = (live_g & bei ? ringI + ((s - ei) & ri) * rowlen : none_row) + 1;
    const int16_t* rDe = (live_g & bed ? ringD + ((s - ed) & rd) * rowlen : none_row) - 1;
    int16_t* wM = ringM + sm * rowlen;
    int16_t* wI = ringI + (s & ri) * rowlen;
    int16_t* wD = ringD + (s & rd) * rowlen;
    int* hs = TB ? hist + s * W - base : nullptr;
    int kd = INT32_MAX, mad = INT32_MIN;  // lowest done diagonal; prune_wavefront's maximum
    int top_m = kNone16, top_g = kNone16;
    for (int k = alive ? lo + gl : INT32_MAX; k <= hi; k += G) {
      int vi = kNone16, vd = kNone16, vm = 0, from = 0;
      if (s > 0) {
        const int i0 = rMoi[k], i1 = rIe[k], d0 = rMod[k], d1 = rDe[k], m0 = rMx[k];
        const int io = i0 < m ? i0 + 1 : kNone16, dop = d0 <= n - k ? d0 : kNone16;
        vi = max(io, i1 < m ? i1 + 1 : kNone16);
        vd = max(dop, d1 <= n - k ? d1 : kNone16);
        vm = m0 < min(m, n - k) ? m0 + 1 : kNone16;
        top_g = max(top_g, max(vi, vd));
        if (TB)
          from = (vm >= max(vi, vd) ? 0 : vi >= vd ? kFromI : kFromD) | (io == vi ? kIOpen : 0) |
                 (dop == vd ? kDOpen : 0);
        vm = max(vm, max(vi, vd));
      }
      if (vm >= 0) {
        if (TB) hs[k] = vm << 4 | from;
        vm = kWide ? wfa_extend_wide(pw, tw, m, n, k, vm) : wfa_extend(pw, tw, m, n, k, vm);
        mad = max(mad, 2 * vm + k);
        if (vm >= m) kd = min(kd, k);
      }
      top_m = max(top_m, vm);
      wM[k] = (int16_t)vm;
      wI[k] = (int16_t)vi;
      wD[k] = (int16_t)vd;
    }
    if (L.drop >= 0) {  // prune_wavefront (wfa.rs:293-346) on the extended M
      __syncwarp();
#pragma unroll
      for (int d = 1; d < G; d <<= 1) mad = max(mad, __shfl_xor_sync(kFull, mad, d));
      kd = INT32_MAX;
      for (int k = alive ? lo + gl : INT32_MAX; k <= hi; k += G) {
        const int vm = wM[k];
        if (vm < 0) continue;
        if (2 * vm + k < mad - L.drop) {
          wM[k] = (int16_t)kNone16;
        } else if (vm >= m) {
          kd = min(kd, k);
        }
      }
    }
    __syncwarp();
    const unsigned any_m = __ballot_sync(kFull, top_m >= 0) & gmask;
    const unsigned any_g = __ballot_sync(kFull, top_g >= 0) & gmask;
    if (__any_sync(kFull, kd != INT32_MAX)) {
#pragma unroll
      for (int d = 1; d < G; d <<= 1) kd = min(kd, __shfl_xor_sync(kFull, kd, d));
    }
    if (alive) {
      live_m = live_m << 1 | (Mask)(any_m != 0), live_g = live_g << 1 | (Mask)(any_g != 0);
      dead = (live_m & in_ring) == 0;
      if (kd != INT32_MAX) {
        done_s = s;
        k_end = kd;
        alive = false;
      } else if (dead || s == s_lim) {
        alive = false;
      } else {
        advance();
      }
    }
  }
}

// cigar_off / n_cigar of every result and the ops in pair order (each pair's
// slot holds its ops in reverse).
__global__ void __launch_bounds__(256) wfa_compact_kernel(WfaCompact C) {
  const uint32_t stride = gridDim.x * blockDim.x;
  for (uint32_t p = blockIdx.x * blockDim.x + threadIdx.x; p < C.n; p += stride) {
    const uint32_t off = C.off[p], n = C.ncig[p];
    C.out[p].cigar_off = off;
    C.out[p].n_cigar = n;
    if ((uint64_t)off + n > C.cap || n > C.slot_cap) continue;
    const uint32_t* src = C.slots + (size_t)p * C.slot_cap;
    for (uint32_t t = 0; t < n; ++t) C.ops[off + t] = src[n - 1u - t];
  }
}

}  // namespace

template <int G>
static cudaError_t wfa_occupancy(bool traceback, size_t smem, int threads, int* per_sm) {
  auto kern = traceback ? wfa_kernel<G, true> : wfa_kernel<G, false>;
  cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return e;
  return cudaOccupancyMaxActiveBlocksPerMultiprocessor(per_sm, kern, threads, smem);
}

cudaError_t wfa_blocks_per_sm(int group, bool traceback, size_t smem, int threads, int* per_sm) {
  switch (group) {
    case 8: return wfa_occupancy<8>(traceback, smem, threads, per_sm);
    case 16: return wfa_occupancy<16>(traceback, smem, threads, per_sm);
    case 32: return wfa_occupancy<32>(traceback, smem, threads, per_sm);
    default: return cudaErrorInvalidValue;
  }
}

template <int G>
static void wfa_launch_g(const DevPairs& P, const WfaLaunch& L, uint32_t blocks, uint32_t threads,
                         size_t smem, bool traceback, cudaStream_t st) {
  if (traceback) (wfa_kernel<G, true><<<blocks, threads, smem, st>>>(P, L), count_launch());
  else (wfa_kernel<G, false><<<blocks, threads, smem, st>>>(P, L), count_launch());
}

cudaError_t launch_wfa(const DevPairs& P, const WfaLaunch& L, uint32_t blocks,
                       uint32_t warps_per_block, bool traceback, cudaStream_t st) {
  const uint32_t groups = warps_per_block * (32u / (uint32_t)L.group);
  const size_t smem = (size_t)L.smem_group * groups;
  const uint32_t threads = 32u * warps_per_block;
  switch (L.group) {
    case 8: wfa_launch_g<8>(P, L, blocks, threads, smem, traceback, st); break;
    case 16: wfa_launch_g<16>(P, L, blocks, threads, smem, traceback, st); break;
    case 32: wfa_launch_g<32>(P, L, blocks, threads, smem, traceback, st); break;
    default: return cudaErrorInvalidValue;
  }
  return cudaGetLastError();
}

using WfaWindowKernel = void (*)(DevPairs, WfaLaunch, WfaWindow);

template <int G>
static WfaWindowKernel wfa_window_pick(bool traceback, bool small) {
  return traceback ? (small ? wfa_window_kernel<G, true, uint32_t> : wfa_window_kernel<G, true, uint64_t>)
                   : (small ? wfa_window_kernel<G, false, uint32_t> : wfa_window_kernel<G, false, uint64_t>);
}

// The row masks take 32 bits where the recurrence looks back less than 32 rows.
static WfaWindowKernel wfa_window_pick(const WfaLaunch& L, const WfaWindow& X, bool traceback) {
  const bool small = L.lookback < 32;
  switch (X.lanes) {
    case 16: return wfa_window_pick<16>(traceback, small);
    default: return wfa_window_pick<32>(traceback, small);
  }
}

cudaError_t wfa_window_blocks_per_sm(const WfaLaunch& L, const WfaWindow& X, bool traceback,
                                     int* per_sm) {
  const size_t smem = (size_t)wfa_window_pairs(X) * X.group_bytes;
  auto kern = wfa_window_pick(L, X, traceback);
  cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return e;
  return cudaOccupancyMaxActiveBlocksPerMultiprocessor(per_sm, kern, 128, smem);
}

cudaError_t launch_wfa_window(const DevPairs& P, const WfaLaunch& L, const WfaWindow& X,
                              uint32_t blocks, bool traceback, cudaStream_t st) {
  const size_t smem = (size_t)wfa_window_pairs(X) * X.group_bytes;
  (wfa_window_pick(L, X, traceback)<<<blocks, 128, smem, st>>>(P, L, X), count_launch());
  return cudaGetLastError();
}

cudaError_t launch_wfa_compact(const WfaCompact& C, int sms, cudaStream_t st) {
  uint64_t b = (C.n + 255) / 256;
  if (b < 1) b = 1;
  if (b > (uint64_t)sms * 8) b = (uint64_t)sms * 8;
  (wfa_compact_kernel<<<(int)b, 256, 0, st>>>(C), count_launch());
  return cudaGetLastError();
}

}  // namespace kira
