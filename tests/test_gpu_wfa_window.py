"""The fixed-window WFA passes at their edges, against the oracle pair by pair: two
pairs a warp and a warp per pair, 64 and 128 diagonals and what is left open after
them, look-back of 31 / 32 / 63 / 64 rows (32-bit and 64-bit row masks, and past the
passes), free leading bases at the widths' limits, reads at every alignment of the
arena, odd numbers of pairs, non-ACGT bytes, and pruned fronts."""
import numpy as np
import pytest

from test_gpu_wfa import _check, ctx  # noqa: F401  (the fixture)

pytestmark = pytest.mark.gpu


def _pairs(seed, count, lo, hi, err, indel, lead=0, slack=24):
    rng = np.random.default_rng(seed)
    out = []
    for i in range(count):
        m = int(rng.integers(lo, hi + 1))
        text = rng.choice(np.frombuffer(b"ACGT", np.uint8), m + lead + slack)
        start = int(rng.integers(0, lead + 1))
        read = []
        for c in text[start:start + m]:
            r = rng.random()
            if r < err * indel / 2:
                continue
            if r < err * indel:
                read += [int(rng.choice(list(b"ACGT")))] * int(rng.integers(1, 4))
            elif r < err:
                c = rng.choice(list(b"ACGTN"))
            read.append(int(c))
        out.append((bytes(read) or b"A", bytes(text[: len(text) - i % 5])))
    return out


@pytest.mark.parametrize("traceback", [True, False])
@pytest.mark.parametrize("costs,tbf,drop,lengths,err", [
    ((4, 6, 1), 0, -1, (1, 9), 0.2),        # a few bases; texts longer than reads
    ((4, 6, 1), 0, -1, (120, 160), 0.06),   # most done within 64 diagonals
    ((4, 6, 1), 0, -1, (120, 160), 0.25),   # 128 diagonals and the general kernel
    ((4, 6, 1), 15, -1, (60, 120), 0.08),
    ((4, 6, 1), 63, -1, (60, 120), 0.08),
    ((4, 6, 1), 100, -1, (60, 120), 0.08),
    ((4, 6, 1), 0, 12, (100, 150), 0.1),    # pruned fronts
    ((4, 6, 1), 8, 6, (100, 150), 0.1),
    ((31, 6, 1), 0, -1, (60, 100), 0.04),   # look-back 31, 32, 63 and 64
    ((5, 30, 2), 0, -1, (60, 100), 0.06),
    ((63, 4, 3), 2, -1, (60, 100), 0.03),
    ((64, 4, 3), 2, -1, (60, 100), 0.03),
    ((1, 0, 1), 0, -1, (40, 90), 0.1),      # every row live
    ((4, 6, 1), 0, -1, (700, 900), 0.02),   # a warp per pair in the first pass
])
def test_window_passes(ctx, traceback, costs, tbf, drop, lengths, err):  # noqa: F811
    from kira_ls_aligner_b200 import WfaParams
    pairs = _pairs(sum(costs) * 131 + tbf + lengths[0], 41, *lengths, err, 0.4, lead=tbf)
    p = WfaParams(*costs, max_score=200, adaptive_drop=drop, text_begin_free=tbf,
                  traceback=traceback)
    got = _check(ctx, pairs, p)
    assert any(g is not None for g in got)


def test_window_passes_scored(ctx):  # noqa: F811
    from kira_ls_aligner_b200 import AlignmentConfig, WfaParams
    pairs = _pairs(5, 203, 100, 151, 0.08, 0.5) + [(b"", b"ACGT"), (b"ACGT", b"")]
    _check(ctx, pairs, WfaParams.scored_from(AlignmentConfig()))
