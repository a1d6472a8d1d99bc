"""A chunked verification call whose last chunk holds a bad pair is refused after the earlier
chunks were enqueued; the next call on the context, larger so that its buffers move, is not
disturbed by them."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_a_refused_call_leaves_nothing_running():
    from kira_ls_aligner_b200 import GpuContext, PairBatch, VerifyParams, _abi, runtime, synth
    w = synth.make_workload("chunks", 40_000, 400_000, cands=4, sub_lo=0.005, sub_hi=0.04,
                            seed=0xC4)
    arena, woffs = w.windows_arena()
    params = VerifyParams(sieve_threshold=12, myers_k=8)

    def batch(n, bad=False):
        off = woffs[:n].copy()
        if bad:
            off[n - 1] = len(arena)
        return PairBatch(w.reads, w.read_off[:n], w.read_len[:n], arena, off, w.win_len[:n])

    with GpuContext(0) as ctx:
        want = ctx.verify_batch(batch(w.n_pairs), params)
    L = _abi.lib()
    for _ in range(3):
        with GpuContext(0) as ctx:
            ctx.check(L.kira_gpu_set_chunk_pairs(ctx.handle, 20_000))
            with pytest.raises(runtime.InvalidArgument, match="window outside"):
                ctx.verify_batch(batch(120_000, bad=True), params)
            ctx.check(L.kira_gpu_set_chunk_pairs(ctx.handle, 0))
            got = ctx.verify_batch(batch(w.n_pairs), params)
            assert np.array_equal(got[0], want[0]) and np.array_equal(got[1], want[1])
            assert got[3] == want[3]
