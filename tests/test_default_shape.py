"""The launch shape an untuned banded-SW call takes (default_shape, csrc/api.cu), over band,
read length and item count: it covers the band, and a batch that fills the GPU never runs
more lanes a pair than it needs to."""
import ctypes as C
import itertools

import pytest


def _pick(band, q, items, scoring=(1, 4, 6, 1)):
    from kira_ls_aligner_b200 import AlignmentConfig, _abi
    cfg = AlignmentConfig(*scoring, band, 100, 5).to_c()
    g, cells, packed = C.c_int(), C.c_int(), C.c_int()
    s = _abi.lib().kira_gpu_bsw_default_shape(C.byref(cfg), band, q, items, C.byref(g),
                                              C.byref(cells), C.byref(packed))
    return s, g.value, cells.value, packed.value


BANDS = [1, 8, 16, 17, 18, 33, 35, 36, 39, 40, 48, 50, 63, 64, 67, 68, 71, 72, 100, 128, 135, 136,
         143, 144, 159, 160, 200, 256, 271]
ITEMS = [1, 50, 1199, 1200, 2999, 3000, 8000, 9999, 10000, 17999, 18000, 19999, 20000, 60000,
         400_000, 4_000_000]


@pytest.mark.parametrize("q", [50, 150, 300, 1000, 2000])
def test_covers_the_band_on_packed_lanes(q):
    for band, items in itertools.product(BANDS, ITEMS):
        s, g, cells, packed = _pick(band, q, items)
        assert 0 <= s < 26 and packed and g * cells >= 2 * band + 1, (band, items, s)


# Lanes a pair at most: 1 to band 33 (34 and 68 cells; 2 x 18 fits band 17), 2 to 67 (136)
# and 4 to 135 (272), but the shorter rows of 72, 80 and 144 cells where those fit; 288 cells
# on 16, the widest on 32.
@pytest.mark.parametrize("items", [60_000, 400_000, 4_000_000])
def test_large_batches_use_few_lanes(items):
    for band in range(1, 272):
        most = (1 if band <= 16 else 2 if band <= 17 else 1 if band <= 33 else 4 if band <= 35
                else 8 if band <= 39 else 2 if band <= 67 else 8 if band <= 71
                else 4 if band <= 135 else 16 if band <= 143 else 32)
        assert _pick(band, 150, items)[1] <= most, (band, items)


def test_more_items_never_take_more_lanes():
    for band in range(1, 272):
        lanes = [_pick(band, 150, items)[1] for items in ITEMS]
        assert lanes == sorted(lanes, reverse=True), (band, lanes)


def test_values_past_int16_run_on_int32():
    for band, items in itertools.product(BANDS, (50, 100_000)):
        s, g, cells, packed = _pick(band, 300, items, (40, 4, 6, 1))
        assert s >= 0 and not packed and g * cells >= 2 * band + 1
    assert _pick(300, 150, 10)[0] == -1 and _pick(33, 150, 10, (1, 4, -1, 1))[0] == -1
