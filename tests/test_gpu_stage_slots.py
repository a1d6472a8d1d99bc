"""The composed path with fewer trace slots than pairs (from 2^20 pairs on): batches whose
banded-SW items fill the first round, end in it and run over into the second, in one call
and in grouped chunks, against the oracle."""
import numpy as np
import pytest

import pyoracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("pairs,chunk,sub", [(1 << 20, 0, 0.05), (1 << 20, 0, 0.02),
                                             ((1 << 20) + 35, 0, 0.05),
                                             (2_100_000, 300_000, 0.05)])
def test_more_items_than_slots(pairs, chunk, sub):
    from kira_ls_aligner_b200 import AlignmentConfig, GpuContext, PairBatch, VerifyParams, _abi, synth
    w = synth.make_workload("slots", pairs, 2_000_000, cands=1, sub_lo=sub / 2, sub_hi=sub,
                            seed=0x510)
    params = VerifyParams(AlignmentConfig(bandwidth=12), 12, 8)
    batch = PairBatch(w.reads, w.read_off, w.read_len, None, w.win_off, w.win_len)
    with GpuContext(0) as ctx:
        ctx.ref_upload(w.reference)
        ctx.check(_abi.lib().kira_gpu_set_chunk_pairs(ctx.handle, chunk))
        res, ops, _, cells = ctx.verify_batch(batch, params)
    op = O.verify_params(O.cfg(1, 4, 6, 1, 12, 100, 5), 12, 8)
    out, cig = O.verify_batch(w.reads, w.read_off, w.read_len, w.reference, w.win_off, w.win_len,
                              op, 8, 64)
    items = int((res["status"] == _abi.PAIR_SW).sum())
    assert (items > pairs // 2) == (sub > 0.03)
    for f in ("status", "score", "ref_start", "ref_end", "read_start", "read_end", "n_cigar"):
        assert np.array_equal(res[f], out[f]), f
    assert cells == int(out["cells"].sum())
    n = res["n_cigar"].astype(np.int64)
    assert n.max() < 64
    pair = np.repeat(np.arange(pairs), n)
    at = np.arange(len(pair)) - np.repeat(np.cumsum(n) - n, n)
    assert np.array_equal(ops[np.repeat(res["cigar_off"].astype(np.int64), n) + at], cig[pair, at])
