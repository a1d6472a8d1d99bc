"""The packed full-window sweep of align_batch_simd (bsw16_full_sweep) at the edges of its
row capacities, for few and many pairs, with and without abort bounds, and the score bound
past which the int32 sweep runs, against the oracle's AVX2 kernel."""
import pytest

import pyoracle as O
from refgen import XorShift
from test_gpu_align_batch_simd import _batch, _cmp

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    from kira_ls_aligner_b200 import GpuContext
    c = GpuContext(0)
    yield c
    c.close()


@pytest.mark.parametrize("n", [21, 1505])
@pytest.mark.parametrize("q,w", [(1, 1), (17, 33), (40, 80), (40, 81), (60, 128), (60, 129),
                                 (90, 144), (90, 145), (150, 272), (150, 273), (33, 320),
                                 (33, 321), (50, 544)])
def test_row_capacities(ctx, n, q, w):
    rng = XorShift(0x51D0 + w * 3 + n)
    reads, wins = _batch(rng, n, q, w)
    aborts = [int(rng.next() % (q + 20)) if rng.next() % 3 else O.ABORT_DISABLED
              for _ in range(n)] if w % 2 else None
    _cmp(ctx, reads, wins, O.cfg(1, 4, 6, 1, 33, 100, 5), O.SIMD_AVX2, O.SIMD_AVX2, aborts=aborts)


@pytest.mark.parametrize("match,mismatch,go,ge", [(1, 4, 6, 1), (1, 1, 0, 1), (1, 5, 2, 0),
                                                  (2, 1, 9, 3), (2, 5, 5, 1), (3, 4, 6, 1)])
def test_scorings_around_the_byte_range(ctx, match, mismatch, go, ge):
    # 123 bases at +2 end at 246 + the widest step: 255 / 256 is the last packed score.
    rng = XorShift(0x51D1 + match * 7 + go)
    for q in (122, 123, 124, 125):
        reads, wins = _batch(rng, 40, q, 200)
        _cmp(ctx, reads, wins, O.cfg(match, mismatch, go, ge, 33, 100, 5), O.SIMD_AVX2,
             O.SIMD_VNNI)
