"""The packed sweep's trace of H bytes and its moves, restated on the CPU for every packed
shape, the unlisted ones included (csrc/bsw16.cuh): a byte per cell, two words (four cells)
per 4-byte slab, rows interleaved in blocks laid out [row block][slab][row in block][lane].
Each slab is stored once and inside the item's slot, the traceback reads each cell's byte
where its lane put it, whole blocks are what one bulk copy moves, and moves by any number of
cells equal the shift of the whole row."""
import random

import pytest

# (lanes, words a lane) of kBswShapes' packed entries (csrc/kernels.cu), banded ones first.
BANDED = [(2, 9), (4, 5), (4, 9), (8, 5), (8, 9), (16, 9), (32, 9), (2, 17), (2, 18), (1, 34),
          (2, 34), (4, 34), (1, 17), (32, 2), (32, 5)]
FULL = [(8, 5), (8, 9), (8, 17), (16, 17), (32, 2), (32, 5), (32, 9)]
SHAPES = sorted(set(BANDED + FULL))


def interleave(g):
    return 8 if g <= 4 else 1 if g >= 32 else 32 // g


def strip_bytes(g, k):  # Bsw16Shape::kStripBytes: one interleave block
    return (k + 1) // 2 * interleave(g) * g * 4


def slot_bytes(g, k, max_q):  # shape_slot_bytes (csrc/internal.h)
    r, stride = interleave(g), g * 4 * ((k + 1) // 2)
    return ((max_q + 1 + r - 1) // r * r * stride + 15) // 16 * 16


def stored(g, k, i, lane, slab):
    """Address of the slab that `lane` stores for row i, within the item's slot."""
    r = interleave(g)
    return i // r * strip_bytes(g, k) + 4 * (slab * r * g + (i & (r - 1)) * g + lane)


def read(g, k, i, idx):
    """Address of band cell idx of row i (Bsw16Trace)."""
    half, r, stride = g * k, interleave(g), g * 4 * ((k + 1) // 2)
    hi = idx >= half
    lane, kk = divmod(idx - hi * half, k)
    ib = i & (r - 1)
    return (i - ib) * stride + ((kk >> 1) * r + ib) * g * 4 + lane * 4 + (kk & 1) * 2 + hi


@pytest.mark.parametrize("g,k", SHAPES)
@pytest.mark.parametrize("max_q", [1, 2, 7, 8, 31, 150, 511])
def test_rows_fill_their_slot_once(g, k, max_q):
    seen = set()
    for i in range(1, max_q + 1):
        for lane in range(g):
            for slab in range((k + 1) // 2):
                a = stored(g, k, i, lane, slab)
                assert a % 4 == 0 and a + 4 <= slot_bytes(g, k, max_q) and a not in seen
                seen.add(a)


@pytest.mark.parametrize("g,k", SHAPES)
def test_each_cell_is_read_where_it_was_stored(g, k):
    for i in (1, 2, 3, 7, 8, 9, 150):
        for idx in range(2 * g * k):
            hi = idx >= g * k
            lane, kk = divmod(idx - hi * g * k, k)
            # prmt(word 2x, word 2x + 1, 0x6420): low bytes lo 2x, hi 2x, lo 2x+1, hi 2x+1.
            assert read(g, k, i, idx) == stored(g, k, i, lane, kk // 2) + (kk & 1) * 2 + hi


@pytest.mark.parametrize("g,k", [s for s in BANDED if s[0] < 8])
def test_staged_blocks_are_whole_copies(g, k):
    # One bulk copy moves a block: 16-byte address and size; blocks tile the slot.
    n, r = strip_bytes(g, k), interleave(g)
    assert n % 16 == 0
    for i in range(1, 40):
        for lane in range(g):
            for slab in range((k + 1) // 2):
                a = stored(g, k, i, lane, slab)
                assert i // r * n <= a < (i // r + 1) * n
                assert a - i // r * n == 4 * (slab * r * g + (i & (r - 1)) * g + lane)


def move(regs, s, down, g, k, neutral):
    """bsw16_move: s cells (s < k) of the (low, high) words across lane ends."""
    out = [list(lane) for lane in regs]
    for gi in range(g):
        x = [regs[(gi - 1) % g][k - s + t] if down else regs[(gi + 1) % g][t] for t in range(s)]
        if gi == (0 if down else g - 1):
            x = [(neutral, lo) if down else (hi, neutral) for lo, hi in x]
        out[gi] = x + regs[gi][:k - s] if down else regs[gi][s:] + x
    return out


@pytest.mark.parametrize("g,k", [s for s in BANDED if s[1] >= 17])
def test_moves_equal_the_shift_of_the_row(g, k):
    cap, rng = 2 * g * k, random.Random(g * 100 + k)
    for s in [1, 2, 3, 4, 5, 15, 16, 17, 20, 37, cap - 1, cap, cap + 5]:
        for down in (False, True):
            row = [rng.randrange(1, 1 << 13) for _ in range(cap)]
            regs = [[(row[gi * k + j], row[g * k + gi * k + j]) for j in range(k)]
                    for gi in range(g)]
            left = min(s, cap)  # bsw16_realign: by 16, 4 and 1
            for step in (16, 4, 1):
                while left >= step:
                    regs, left = move(regs, step, down, g, k, 0), left - step
            want = [row[c - s if down else c + s] if 0 <= (c - s if down else c + s) < cap else 0
                    for c in range(cap)]
            got = [regs[c // k][c % k][0] for c in range(g * k)]
            got += [regs[c // k][c % k][1] for c in range(g * k)]
            assert got == want


def test_the_library_lists_the_banded_shapes():
    from kira_ls_aligner_b200 import autotune
    listed = {(g, c // 2) for (g, c), p in zip(autotune.shapes(), autotune.packed()) if p}
    assert listed == set(BANDED[:12])
