"""The packed banded-SW traceback from stored H bytes (warp_walk_h, csrc/bsw16.cuh),
restated cell by cell over the oracle's DP matrix (banded_sw_with, mod.rs:1370-1650):
with H itself the walk gives the oracle's start and CIGAR; with H mod 256 it does so or
reports a value left over -- also on scorings built so that wrong moves look right
(mismatch scores a multiple of 256 away from the match score)."""
import pytest

import pyoracle as O
from gpu_cases import sw_corpus
from test_scored_traceback import _matrix


def _walk(read, win, res, rs, rl, h, c, mod):
    gof, ge, go = c.gap_open + c.gap_extend, c.gap_extend, c.gap_open

    def hb(i, j):
        if i <= 0 or j <= 0 or not 0 <= j - rs[i] < rl[i]:
            return -1
        return int(h[i, j - rs[i]]) % mod

    def gap(i, j, v, di, dj):
        g = 1
        while True:
            x = hb(i - g * di, j - g * dj)
            d = (v + gof + (g - 1) * ge - x) % mod
            if x < 0 or d > go:
                return 0
            if d == 0:
                return g
            g += 1

    i, j, v, runs = res.read_end, res.ref_end, res.score, []

    def push(op, n):
        if runs and runs[-1][1] == op:
            runs[-1][0] += n
        else:
            runs.append([n, op])

    while i > 0 and j > 0 and v > 0:
        s = c.match_score if read[i - 1] == win[j - 1] else -c.mismatch
        p = hb(i - 1, j - 1)
        if (p + s - v) % mod == 0 if p >= 0 else v == s:
            push("M", 1)
            i, j, v = i - 1, j - 1, v - s
            continue
        op, n = "I", gap(i, j, v, 1, 0)
        if not n:
            op, n = "D", gap(i, j, v, 0, 1)
        if not n:
            break
        push(op, n)
        if op == "I":
            i -= n
        else:
            j -= n
        v += gof + (n - 1) * ge
    return i, j, v != 0, [(n, o) for n, o in reversed(runs)]


@pytest.mark.parametrize("scheme,mod", [
    ((1, 4, 6, 1), 1 << 30), ((2, 3, 5, 2), 1 << 30), ((1, 4, 0, 1), 1 << 30),
    ((1, 1, 2, 0), 1 << 30), ((1, 4, 6, 1), 256), ((1, 1, 0, 1), 256), ((3, 2, 4, 0), 256),
    ((26, 4, 6, 1), 256), ((26, 230, 6, 1), 256), ((13, 243, 30, 13), 256)])
def test_walk_equals_the_oracle_or_is_lost(scheme, mod):
    m, x, go, ge = scheme
    cases = sw_corpus(0x11A + go * 7 + m, 400, qmin=10, qmax=160, pad=60, max_band=40)
    for read, win, off, band, abort in cases:
        c = O.OrcCfg(m, x, go, ge, band, 100, 5)
        res, rs, rl, h, _ = _matrix(read, win, off, c, abort)
        i, j, lost, cig = _walk(read, win, res, rs, rl, h, c, mod)
        # packed_trace_wraps (csrc/internal.h)
        assert not lost or (mod == 256 and len(read) * m + max(x, go + 2 * ge) > 255)
        if not lost:
            assert (i, j) == (res.read_start, res.ref_start)
            assert cig == [(n, o) for n, o in res.cigar], (read, win, off, band)
