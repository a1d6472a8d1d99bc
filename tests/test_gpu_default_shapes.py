"""The launch shapes that only the default pick uses (kira_gpu_bsw_default_shape): one lane of
34 cells for large narrow batches, a warp per pair with 2 and 5 words a lane for the
shortest, against the oracle's banded_sw_with on reads and windows of every small length."""
import ctypes as C

import numpy as np
import pytest

import pyoracle as O

pytestmark = pytest.mark.gpu


def _workload(seed, n, qmax, band):
    rng = np.random.default_rng(seed)
    alpha = np.frombuffer(b"ACGTN", np.uint8)
    q = rng.integers(1, qmax + 1, n)
    w = q + rng.integers(0, 2 * band + 20, n)
    woff = np.cumsum(w) - w
    wins = alpha[rng.integers(0, 4, int(w.sum()))]
    wins[rng.random(len(wins)) < 0.002] = alpha[4]
    lead = rng.integers(0, w - q + 1)
    reads, roff, rlen = [], [], []
    pos = 0
    for i in range(n):
        r = wins[woff[i] + lead[i]:woff[i] + lead[i] + q[i]].copy()
        sub = rng.random(q[i]) < 0.03
        r[sub] = alpha[rng.integers(0, 4, int(sub.sum()))]
        if i % 3 == 0 and q[i] > 12:  # a gap either way
            at, ln = int(rng.integers(4, q[i] - 6)), int(rng.integers(1, 4))
            r = np.concatenate([r[:at], r[at + ln:]] if i % 2 else
                               [r[:at], alpha[rng.integers(0, 4, ln)], r[at:]])
        if i % 7 == 0:
            r = alpha[rng.integers(0, 4, len(r))]
        reads.append(r)
        roff.append(pos)
        rlen.append(len(r))
        pos += len(r)
    off = lead + rng.integers(-3, 4, n)
    off[::11] = rng.integers(-20, qmax, len(off[::11]))
    return (np.concatenate(reads + [alpha[:1]]), np.array(roff, np.uint64), np.array(rlen, np.uint32),
            np.concatenate([wins, alpha[:1]]), woff.astype(np.uint64), w.astype(np.uint32),
            off.astype(np.int32))


@pytest.mark.parametrize("band,n,qmax,shape", [(16, 20_000, 60, (1, 34)), (3, 20_011, 90, (1, 34)),
                                               (16, 40_000, 33, (1, 34)), (63, 500, 150, (32, 4)),
                                               (40, 1999, 90, (32, 4)), (5, 300, 260, (32, 4)),
                                               (159, 1000, 260, (32, 10)),
                                               (144, 4000, 60, (32, 10))])
@pytest.mark.parametrize("scoring", [(1, 4, 6, 1, True, 16), (2, 3, 5, 2, False, 16),
                                     (1, 1, 0, 1, True, 4), (3, 2, 4, 0, True, 16)])
def test_unlisted_shapes(band, n, qmax, shape, scoring):
    from kira_ls_aligner_b200 import AlignmentConfig, GpuContext, PairBatch, _abi
    m, x, go, ge, adaptive, drift = scoring
    cfg = AlignmentConfig(m, x, go, ge, band, 100, 5, adaptive, drift)
    reads, roff, rlen, wins, woff, wlen, off = _workload(band * 7 + n, n, qmax, band)
    g, k = C.c_int(), C.c_int()
    assert _abi.lib().kira_gpu_bsw_default_shape(C.byref(cfg.to_c()), band, int(rlen.max()), n,
                                                 C.byref(g), C.byref(k), None) >= 23
    assert (g.value, k.value) == shape
    with GpuContext(0) as ctx:
        res, ops, cells = ctx.bsw_batch(PairBatch(reads, roff, rlen, wins, woff, wlen, off), cfg)
    out, cig = O.banded_sw_batch(reads, roff, rlen, wins, woff, wlen, off,
                                 O.cfg(m, x, go, ge, band, 100, 5), 8, 512, adaptive=adaptive,
                                 max_drift=drift)
    for f in ("score", "ref_start", "ref_end", "read_start", "read_end", "n_cigar", "early_abort"):
        assert np.array_equal(res[f], out[f]), f
    assert cells == int(out["cells"].sum())
    c = res["n_cigar"].astype(np.int64)
    assert c.max() <= 512
    pair = np.repeat(np.arange(n), c)
    at = np.arange(len(pair)) - np.repeat(np.cumsum(c) - c, c)
    assert np.array_equal(ops[np.repeat(res["cigar_off"].astype(np.int64), c) + at], cig[pair, at])
