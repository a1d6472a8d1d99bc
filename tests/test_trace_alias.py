"""Which scorings the packed banded SW takes when its trace of H mod 256 wraps
(packed_trace_aliases, csrc/internal.h): on those it takes, the walk of
test_h_traceback.py loses next to none of its alignments; those that lose many run on int32
lanes, as does nothing that cannot wrap."""
import pytest

import pyoracle as O
from gpu_cases import sw_corpus
from test_default_shape import _pick
from test_h_traceback import _walk
from test_scored_traceback import _matrix


def _lost(scoring, q=(100, 160)):
    m, x, go, ge = scoring
    lost = n = 0
    for read, win, off, band, abort in sw_corpus(0xA11A + x, 500, qmin=q[0], qmax=q[1], pad=40,
                                                 max_band=30):
        c = O.OrcCfg(m, x, go, ge, band, 100, 5)
        res, rs, rl, h, _ = _matrix(read, win, off, c, abort)
        n += 1
        lost += _walk(read, win, res, rs, rl, h, c, 256)[2]
    return lost / n


def _packed(scoring, q):
    return _pick(30, q, 500, scoring)[3]


# Mismatch scores next to a multiple of 256 from the match score, where the reads are long
# enough for scores that a mismatch does not end.
@pytest.mark.parametrize("scoring", [(2, 255, 6, 1), (2, 268, 6, 1), (9, 247, 0, 3),
                                     (5, 508, 6, 1), (13, 243, 30, 13), (4, 509, 6, 2)])
def test_aliasing_scorings_run_on_int32(scoring):
    assert not _packed(scoring, 160)
    # ... and only where values pass 255.
    m, x, go, ge = scoring
    for q in (1, 2, 5, 10, 30, 50, 90):
        if q * m + max(x, go + 2 * ge) <= 255:
            assert _packed(scoring, q)


@pytest.mark.parametrize("scoring", [(2, 3, 5, 2), (2, 240, 6, 1), (2, 272, 6, 1), (1, 230, 3, 1),
                                     (26, 4, 6, 1), (10, 40, 60, 10), (20, 80, 80, 20),
                                     (9, 200, 0, 3), (5, 300, 9, 1), (5, 4, 100, 27),
                                     (10, 20, 200, 1)])
def test_other_scorings_stay_packed_and_lose_next_to_none(scoring):
    assert _packed(scoring, 160)
    assert _lost(scoring) <= 0.01


# A mismatch above the highest score is one however large it is.
@pytest.mark.parametrize("mismatch", [254, 255, 256, 270, 511, 1000, 1023, 1 << 20])
def test_forbidden_mismatches_stay_packed(mismatch):
    assert _packed((1, mismatch, 6, 1), 160)
    assert _lost((1, 161, 6, 1)) == 0
