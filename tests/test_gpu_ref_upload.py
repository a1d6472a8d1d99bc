"""The resident reference's planes hold every base of the upload, its end included, from
pageable and from pinned memory: reads cut from it are at Myers distance 0."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("length", [100_003, 1_000_000, 12_345_679])
@pytest.mark.parametrize("pinned", [False, True])
def test_planes_reach_the_end_of_the_reference(length, pinned):
    import torch
    from kira_ls_aligner_b200 import GpuContext, PairBatch
    rng = np.random.default_rng(length)
    # Windows of 140 bases over the last 40,000, a read of 100 bases inside each.
    woff = np.arange(length - 40_000, length - 140, 97, dtype=np.uint64)
    n = len(woff)
    with GpuContext(0) as ctx:
        for _ in range(6):
            ref = np.frombuffer(b"ACGT", np.uint8)[rng.integers(0, 4, length)]
            src = torch.from_numpy(ref).pin_memory().numpy() if pinned else ref
            ctx.ref_upload(src)
            reads = np.concatenate([ref[int(o) + 17:int(o) + 117] for o in woff])
            batch = PairBatch(reads, np.arange(n, dtype=np.uint64) * np.uint64(100),
                              np.full(n, 100, np.uint32), None, woff, np.full(n, 140, np.uint32))
            dist, end = ctx.myers_batch(batch, 3)
            assert (dist == 0).all() and (end == 117).all()
