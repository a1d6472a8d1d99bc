"""The packed traceback's gap rounds (csrc/bsw16.cuh: warp_walk_h): sixteen lengths each
way in the first round, 32 a round after it. Gaps around the rounds' ends in both
directions, short reads and reads past the staged size, against the oracle."""
import pytest

from gpu_cases import oracle_sw
from refgen import BASES, XorShift

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    from kira_ls_aligner_b200 import GpuContext
    c = GpuContext(0)
    yield c
    c.close()


@pytest.mark.parametrize("q", [300, 1500])
@pytest.mark.parametrize("adaptive", [True, False])
def test_gap_lengths(ctx, q, adaptive):
    from kira_ls_aligner_b200 import AlignmentConfig, PairBatch, results_to_list
    rng = XorShift(0x6A9 + q)
    band, cases, lengths = 120, [], (1, 2, 15, 16, 17, 31, 32, 33, 47, 48, 49, 50, 64, 65, 100)
    for n in lengths:
        for deleted in (True, False):
            win = bytes(BASES[rng.next() % 4] for _ in range(q + 2 * band))
            cut = band + q // 2
            if deleted:
                read = win[band:cut] + win[cut + n:cut + n + q // 2]
            else:
                ins = bytes(BASES[rng.next() % 4] for _ in range(n))
                read = win[band:cut] + ins + win[cut:cut + q // 2]
            cases.append((read, win, band, band, -2**31 // 8))
    cfg = AlignmentConfig(2, 4, 6, 1, band, 100, 5, adaptive, 16)
    b = PairBatch.from_pairs([c[0] for c in cases], [c[1] for c in cases],
                             band_offset=[c[2] for c in cases], bandwidth=[c[3] for c in cases])
    res, ops, _ = ctx.bsw_batch(b, cfg)
    want = oracle_sw(cases, cfg, adaptive=adaptive, dp_xdrop=cfg.xdrop)
    for i, (g, w) in enumerate(zip(results_to_list(res, ops), want)):
        assert g.key() == w.key(), (i, lengths[i // 2], i % 2, g, w)
    assert any(w.cigar != want[0].cigar for w in want)
