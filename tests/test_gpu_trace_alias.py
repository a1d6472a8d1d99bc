"""Scorings whose packed traces wrap, on the GPU: scorings that alias (int32 lanes),
mismatches above the highest score, and single walks lost at the band's edge and aligned
again, through the banded SW call and through the composed path, against the oracle."""
import numpy as np
import pytest

import pyoracle as O
from gpu_cases import oracle_sw, sw_corpus
from test_h_traceback import _walk
from test_scored_traceback import _matrix

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    from kira_ls_aligner_b200 import GpuContext
    c = GpuContext(0)
    yield c
    c.close()


def _equal(ctx, cases, scoring, plain=False):
    from kira_ls_aligner_b200 import AlignmentConfig, PairBatch, _abi, results_to_list
    cfg = AlignmentConfig(*scoring, 33, 100, 5, True, 16)
    b = PairBatch.from_pairs([c[0] for c in cases], [c[1] for c in cases],
                             band_offset=[c[2] for c in cases],
                             abort_score=[c[4] for c in cases], bandwidth=[c[3] for c in cases])
    ctx.check(_abi.lib().kira_gpu_set_plain(ctx.handle, int(plain)))
    try:
        res, ops, cells = ctx.bsw_batch(b, cfg)
    finally:
        ctx.check(_abi.lib().kira_gpu_set_plain(ctx.handle, 0))
    want = oracle_sw(cases, cfg, dp_xdrop=cfg.xdrop)
    for i, (g, w) in enumerate(zip(results_to_list(res, ops), want)):
        assert g.key() == w.key(), (i, cases[i][2:], g, w)
    assert cells == sum(w.cells for w in want)


@pytest.mark.parametrize("scoring", [(2, 255, 6, 1), (5, 508, 6, 1), (1, 255, 6, 1),
                                     (1, 270, 6, 1), (1, 1023, 6, 1), (1, 1 << 20, 6, 1),
                                     (0, 255, 6, 1), (3, 255, 0, 0)])
def test_aliasing_and_forbidden_mismatches(ctx, scoring):
    _equal(ctx, sw_corpus(0x5EA + scoring[1], 400, qmin=5, qmax=260, pad=60, max_band=33), scoring)


# (scoring, seed, longest read, pad, widest band, cases whose walk is lost)
LOST = [((26, 200, 0, 0), 1, 150, 30, 6, (42, 56, 163, 167)), ((26, 4, 6, 1), 2, 150, 30, 6, (56,)),
        ((20, 40, 3, 1), 2, 150, 30, 6, (116, 248)), ((10, 240, 0, 1), 3, 150, 60, 33, (392,))]


@pytest.mark.parametrize("scoring,seed,qmax,pad,band,lost", LOST)
@pytest.mark.parametrize("plain", [False, True])
def test_lost_walks_are_aligned_again(ctx, scoring, seed, qmax, pad, band, lost, plain):
    cases = sw_corpus(seed, 500, qmin=40, qmax=qmax, pad=pad, max_band=band)
    for k in lost:
        read, win, off, b, abort = cases[k]
        c = O.OrcCfg(*scoring, b, 100, 5)
        res, rs, rl, h, _ = _matrix(read, win, off, c, abort)
        assert _walk(read, win, res, rs, rl, h, c, 256)[2]
    _equal(ctx, cases, scoring, plain)


# The composed path: one call, a call split over two streams (2^16 pairs and more) and the
# grouped chunks of a host batch; per-pair bands and offsets are the path's own.
@pytest.mark.parametrize("pairs,chunk", [(2000, 0), (70_000, 0), (70_000, 20_000)])
def test_composed_path_on_a_wrapping_scoring(ctx, pairs, chunk):
    from kira_ls_aligner_b200 import (AlignmentConfig, PairBatch, VerifyParams, _abi, synth)
    w = synth.make_workload("wrap", pairs // 4, 200_000, cands=4, sub_lo=0.005, sub_hi=0.05,
                            seed=0x77)
    arena, woffs = w.windows_arena()
    params = VerifyParams(AlignmentConfig(26, 4, 6, 1, 6, 100, 5), 12, 8)
    batch = PairBatch(w.reads, w.read_off, w.read_len, arena, woffs, w.win_len)
    ctx.check(_abi.lib().kira_gpu_set_chunk_pairs(ctx.handle, chunk))
    try:
        res, ops, _, cells = ctx.verify_batch(batch, params)
    finally:
        ctx.check(_abi.lib().kira_gpu_set_chunk_pairs(ctx.handle, -1))
    op = O.verify_params(O.cfg(26, 4, 6, 1, 6, 100, 5), 12, 8)
    out, cig = O.verify_batch(w.reads, w.read_off, w.read_len, arena, woffs, w.win_len, op, 8, 512)
    for f in ("status", "score", "ref_start", "ref_end", "read_start", "read_end", "n_cigar"):
        assert np.array_equal(res[f], out[f]), f
    assert cells == int(out["cells"].sum())
    for p in np.nonzero(res["n_cigar"])[0]:
        a, n = int(res["cigar_off"][p]), int(res["n_cigar"][p])
        assert np.array_equal(ops[a:a + n], cig[p][:n]), p
