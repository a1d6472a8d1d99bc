"""Which WFA passes a batch takes, by its longest read (kira_gpu_wfa_batch): lengths on both
sides of the bounds past which the 64-diagonal pass, and for scores alone the 128-diagonal
one, are left out, with and without free leading text, against the oracle pair by pair."""
import pytest

from test_gpu_wfa import _check, ctx  # noqa: F401  (the fixture)
from test_gpu_wfa_window import _pairs

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("traceback", [True, False])
@pytest.mark.parametrize("tbf", [0, 15, 16])
@pytest.mark.parametrize("costs,longest", [
    ((4, 6, 1), 303), ((4, 6, 1), 304),   # 64 diagonals cover scores to 37
    ((4, 6, 1), 567), ((4, 6, 1), 568),   # 128 cover 70
    ((1, 20, 1), 900),                    # long reads that 64 serve: a warp per pair
    ((1, 0, 1), 2100),                    # 128 alone, and nothing, for single edits
])
def test_passes_by_read_length(ctx, traceback, tbf, costs, longest):  # noqa: F811
    from kira_ls_aligner_b200 import WfaParams
    for err in (0.01, 0.08):
        pairs = _pairs(longest + tbf, 10, longest // 2, longest, err, 0.4, lead=tbf)
        # One read of exactly the longest length (its text starts with it).
        head = bytes(b"ACGTTGCA"[(i * i + i // 3) % 8] for i in range(longest))
        pairs.append((head, head[:40] + head[42:] + b"ACGTACGT"))
        got = _check(ctx, pairs, WfaParams(*costs, max_score=300, text_begin_free=tbf,
                                           traceback=traceback))
        assert any(g is not None for g in got)
