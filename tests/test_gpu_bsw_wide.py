"""The packed banded-SW sweep at the top of its value range (csrc/internal.h:
packed_fits): perfect and near-perfect reads whose scores reach the last packed value,
and the first lengths past it (int32 lanes), against the oracle's banded_sw_with."""
import pytest

from gpu_cases import mutate, oracle_sw, sw_corpus
from refgen import BASES, XorShift

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    from kira_ls_aligner_b200 import GpuContext
    c = GpuContext(0)
    yield c
    c.close()


# (band, read length, match score): values just below, at and above the bounds of the
# shapes that cover the band -- 16-lane and 32-lane rows of 9 words, and short reads
# with large scores on 4 lanes of 9 words.
@pytest.mark.parametrize("band,q,match", [(256, 2100, 1), (256, 3507, 1), (256, 3508, 1),
                                          (140, 3795, 1), (140, 3796, 1), (33, 150, 26),
                                          (33, 153, 26), (33, 154, 26)])
def test_top_of_the_packed_range(ctx, band, q, match):
    from kira_ls_aligner_b200 import AlignmentConfig, PairBatch, results_to_list
    rng = XorShift(0x71DE + band * 7 + q)
    cases = []
    for t in range(6):
        win = bytes(BASES[rng.next() % 4] for _ in range(q + 2 * band))
        read = win[band:band + q]
        if t:
            read = mutate(rng, read, rng.next() % (2 * t), rng.next() % 3)[:q]
        cases.append((read, win, band, band, -2**31 // 8))
    cfg = AlignmentConfig(match, 4, 6, 1, band, 100, 5, True, 16)
    b = PairBatch.from_pairs([c[0] for c in cases], [c[1] for c in cases],
                             band_offset=[c[2] for c in cases], bandwidth=[c[3] for c in cases])
    res, ops, cells = ctx.bsw_batch(b, cfg)
    want = oracle_sw(cases, cfg, dp_xdrop=cfg.xdrop)
    for i, (g, w) in enumerate(zip(results_to_list(res, ops), want)):
        assert g.key() == w.key(), (i, g, w)
    assert cells == sum(w.cells for w in want)
    assert max(w.score for w in want) == q * match


# Scorings on which walks over H mod 256 go wrong (test_h_traceback.py): those items are
# aligned again on int32 lanes.
@pytest.mark.parametrize("scoring", [(26, 230, 6, 1), (13, 243, 30, 13), (9, 247, 0, 3)])
@pytest.mark.parametrize("budget", [0, 1 << 20])
def test_wrapped_traces(ctx, scoring, budget):
    from kira_ls_aligner_b200 import AlignmentConfig, PairBatch, _abi, results_to_list
    m, x, go, ge = scoring
    cases = sw_corpus(0x3E5C + m, 500, qmin=40, qmax=150, pad=60, max_band=33)
    cfg = AlignmentConfig(m, x, go, ge, 33, 100, 5, True, 16)
    b = PairBatch.from_pairs([c[0] for c in cases], [c[1] for c in cases],
                             band_offset=[c[2] for c in cases],
                             abort_score=[c[4] for c in cases],
                             bandwidth=[c[3] for c in cases])
    ctx.check(_abi.lib().kira_gpu_set_trace_budget(ctx.handle, budget))
    try:
        res, ops, cells = ctx.bsw_batch(b, cfg)
    finally:
        ctx.check(_abi.lib().kira_gpu_set_trace_budget(ctx.handle, 0))
    want = oracle_sw(cases, cfg, dp_xdrop=cfg.xdrop)
    for i, (g, w) in enumerate(zip(results_to_list(res, ops), want)):
        assert g.key() == w.key(), (i, cases[i][2:], g, w)
    assert cells == sum(w.cells for w in want)
