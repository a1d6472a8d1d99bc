"""A captured banded-SW call is replayed only while every buffer its launches use is where
it was: another call may grow the buffers of the rescue (sized by the longest read) or of
the CIGAR scan (by the pairs), and the next identical call is captured anew."""
import numpy as np
import pytest

from gpu_cases import mutate, oracle_sw
from refgen import BASES, XorShift
from test_gpu_graphs import _counts

pytestmark = pytest.mark.gpu


def _cases(seed, n, q, band=33):
    rng = XorShift(seed)
    out = []
    for _ in range(n):
        win = bytes(BASES[rng.next() % 4] for _ in range(q + 2 * band))
        read = mutate(rng, win[band:band + q], rng.next() % 6, rng.next() % 3)[:q]
        out.append((read, win, band, band, -2**31 // 8))
    return out


def _batch(cases):
    from kira_ls_aligner_b200 import PairBatch
    return PairBatch.from_pairs([c[0] for c in cases], [c[1] for c in cases],
                                band_offset=[c[2] for c in cases],
                                bandwidth=[c[3] for c in cases])


def _equal(ctx, cases, cfg):
    from kira_ls_aligner_b200 import results_to_list
    res, ops, cells = ctx.bsw_batch(_batch(cases), cfg, 1 << 20)
    want = oracle_sw(cases, cfg, dp_xdrop=cfg.xdrop)
    assert [g.key() for g in results_to_list(res, ops)] == [w.key() for w in want]
    assert cells == sum(w.cells for w in want)


# (first batch: pairs and read length; the captured one; the call that grows)
@pytest.mark.parametrize("sizes,small,grow", [
    ((6000, 150), (60, 300), (60, 480)),      # longer reads: the rescue's trace and rows
    ((8100, 60), (8100, 60), (8200, 60))])    # one more block of the CIGAR scan
@pytest.mark.parametrize("scoring", [(1, 4, 6, 1), (5, 100, 0, 0)])
def test_a_grown_buffer_recaptures(sizes, small, grow, scoring):
    from kira_ls_aligner_b200 import AlignmentConfig, GpuContext, _abi
    cfg = AlignmentConfig(*scoring, 33, 100, 5, True, 16)
    with GpuContext(0) as ctx:
        L = _abi.lib()

        def graphs(on):
            ctx.check(L.kira_gpu_set_graphs(ctx.handle, on, None, None))
        graphs(0)
        ctx.bsw_batch(_batch(_cases(1, *sizes)), AlignmentConfig(1, 4, 6, 1, 33, 100, 5), 1 << 20)
        graphs(1)
        a = _cases(2, *small)
        _equal(ctx, a, cfg)
        c0, r0 = _counts(ctx)
        _equal(ctx, a, cfg)
        assert _counts(ctx) == (c0, r0 + 1)
        graphs(0)
        before = ctx.arena_bytes()
        _equal(ctx, _cases(3, *grow), cfg)
        assert ctx.arena_bytes() > before
        graphs(1)
        _equal(ctx, a, cfg)
        assert _counts(ctx) == (c0 + 1, r0 + 1)  # not the graph of the old buffers
        _equal(ctx, a, cfg)
        assert _counts(ctx) == (c0 + 1, r0 + 2)
