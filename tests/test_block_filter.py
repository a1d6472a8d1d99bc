"""The block filter in front of Myers (csrc/qgram.cuh), restated on the CPU: whenever it
would reject a (read, window) pair the oracle's Myers answers None, and a pair the oracle
certifies meets the bound of the certificate's mismatches. Seeded cases around the bounds
(planted reads with edits near k, random windows, non-ACGT and lower-case bytes)."""
import pytest

import pyoracle as O
from gpu_cases import mutate
from refgen import XorShift

ACGT = set(b"ACGTacgt")


def need(m, k):
    inside = m - k - 4
    return inside // 5 - k if inside > 0 else 0


def count(read, win):
    up = lambda s: bytes(s).upper()  # noqa: E731
    grams = {up(read[p:p + 5]) for p in range(len(read) - 4) if ACGT.issuperset(read[p:p + 5])}
    blocks = (win[b:b + 5] for b in range(0, len(win) - 4, 5))
    return sum(1 for b in blocks if ACGT.issuperset(b) and up(b) in grams)


def rejects(read, win, k):
    return len(read) >= 5 and need(len(read), k) > 0 and count(read, win) < need(len(read), k)


@pytest.mark.parametrize("seed", [1, 2, 3, 4])
def test_filter_rejects_only_myers_none(seed):
    rng = XorShift(0xB10C + seed)
    alpha = b"ACGT" if seed < 3 else b"ACGTNacgt"
    rejected = 0
    for _ in range(800):
        m = 5 + rng.next() % 160
        n = m + rng.next() % 120
        win = bytes(alpha[rng.next() % len(alpha)] for _ in range(n))
        k = rng.next() % 12
        start = rng.next() % (n - m + 1)
        if rng.next() % 3:
            read = mutate(rng, win[start:start + m], rng.next() % (k + 4), rng.next() % 4)
        else:
            read = bytes(alpha[rng.next() % len(alpha)] for _ in range(m))
        if read and rejects(read, win, k):
            rejected += 1
            assert O.bounded_edit_distance(read, win, k) is None, (read, win, k)
    assert rejected > 50


@pytest.mark.parametrize("d", [0, 1, 2])
def test_a_shift_with_d_mismatches_meets_the_bound(d):
    rng = XorShift(0xCE57 + d)
    for _ in range(400):
        m = 12 + rng.next() % 160
        win = bytearray(b"ACGT"[rng.next() % 4] for _ in range(m + rng.next() % 100))
        start = rng.next() % (len(win) - m + 1)
        read = bytearray(win[start:start + m])
        for _ in range(d):
            read[rng.next() % m] = b"ACGT"[rng.next() % 4]
        assert not rejects(bytes(read), bytes(win), d)
