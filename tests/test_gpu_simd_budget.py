"""align_batch_simd past the trace arena's budget: int32 lanes, whose trace is smaller, with
the same results."""
import pytest

import pyoracle as O
from refgen import XorShift
from test_gpu_align_batch_simd import _batch, _cmp

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,q,w", [(40, 60, 128), (1600, 60, 128), (1600, 150, 272)])
def test_smaller_traces_past_the_budget(n, q, w):
    from kira_ls_aligner_b200 import GpuContext, _abi
    rng = XorShift(0x51D2 + n + q)
    reads, wins = _batch(rng, n, q, w)
    held = []
    for budget in (0, 1 << 16):
        with GpuContext(0) as ctx:
            ctx.check(_abi.lib().kira_gpu_set_trace_budget(ctx.handle, budget))
            _cmp(ctx, reads, wins, O.cfg(1, 4, 6, 1, 33, 100, 5), O.SIMD_AVX2, O.SIMD_AVX2)
            held.append(ctx.arena_bytes())
    assert held[1] < held[0] - n * q * w // 4  # half a byte a cell, less the rows' ends
