"""The last WFA window pass is as wide as the batch's scores and longest read ask for: one
long gap either way, of lengths on both sides of every 32 diagonals, with and without
substitutions beside it, free leading text up to the widths' limits, and budgets that the
widest pass does and does not cover, against the oracle pair by pair."""
import numpy as np
import pytest

from test_gpu_wfa import _check, ctx  # noqa: F401  (the fixture)

pytestmark = pytest.mark.gpu

GAPS = [1, 24, 31, 32, 33, 57, 63, 64, 65, 95, 96, 97, 120, 127, 128, 129, 150, 160, 191, 193, 255]


def _pairs(seed, longest, lead):
    rng = np.random.default_rng(seed)
    bases = np.frombuffer(b"ACGT", np.uint8)
    out = []
    for k, gap in enumerate(GAPS):
        for ins in (False, True):
            if gap >= longest - 24:
                continue
            m = longest - k % 3
            text = rng.choice(bases, lead + m + 280)
            at = lead - int(rng.integers(0, lead + 1))
            cut = int(rng.integers(10, m - gap - 10)) if ins else int(rng.integers(10, m - 10))
            if ins:   # the read has `gap` bases more
                read = np.concatenate([text[at:at + cut], rng.choice(bases, gap),
                                       text[at + cut:at + m - gap]])
            else:     # and here as many fewer
                read = np.concatenate([text[at:at + cut], text[at + cut + gap:at + gap + m]])
            for p in rng.integers(0, len(read), k % 4):
                read[p] = rng.choice(bases)
            end = at + m + (0 if ins else gap) + 4 * (k % 2)
            out.append((read.tobytes(), text[:end].tobytes()))
    return out


@pytest.mark.parametrize("traceback", [True, False])
@pytest.mark.parametrize("longest,costs,tbf,budget", [
    (120, (4, 6, 1), 0, 100), (150, (4, 6, 1), 0, 134), (150, (4, 6, 1), 0, 135),
    (150, (4, 6, 1), 15, 400), (150, (4, 6, 1), 100, 400), (150, (4, 6, 1), 127, 400),
    (400, (4, 6, 1), 0, 400), (420, (9, 12, 2), 0, 300), (700, (4, 6, 1), 3, 300),
    (1500, (4, 6, 1), 0, 260), (300, (1, 0, 1), 0, 280), (300, (31, 20, 3), 0, 700)])
def test_gap_lengths(ctx, traceback, longest, costs, tbf, budget):  # noqa: F811
    from kira_ls_aligner_b200 import WfaParams
    got = _check(ctx, _pairs(longest * 7 + tbf + budget, longest, tbf),
                 WfaParams(*costs, max_score=budget, text_begin_free=tbf, traceback=traceback))
    found = [g[0] for g in got if g is not None]
    assert found and max(found) > 70


def test_scored_budget_of_the_router(ctx):  # noqa: F811
    """Scored costs (a base inserted costs one more than one deleted) and the default budget."""
    from kira_ls_aligner_b200 import AlignmentConfig, WfaParams
    for longest in (150, 213, 500):
        got = _check(ctx, _pairs(longest, longest, 0), WfaParams.scored_from(AlignmentConfig()))
        assert any(g is not None for g in got)
