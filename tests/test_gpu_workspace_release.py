"""A process that makes stage calls only gets the workspace pool's memory back."""
import pytest

pytestmark = pytest.mark.gpu


def test_release(cuda):
    from ncvis_gb300 import stages
    N, k = 600_000, 30
    inds = cuda.randint(0, N, (N, k), device="cuda", dtype=cuda.int32)
    dists = cuda.rand((N, k), device="cuda")
    int(stages.symmetrize(inds, dists)[0].sum())  # set-up: both libraries' kernels are loaded
    stages.release_workspace()
    cuda.cuda.empty_cache()
    before = cuda.cuda.mem_get_info()[0]
    want = stages.symmetrize(inds, dists)[0].sum()
    cuda.cuda.empty_cache()
    cuda.cuda.synchronize()
    kept = before - cuda.cuda.mem_get_info()[0]
    assert kept > 256 << 20  # the pool holds the 630 MB of the call
    stages.release_workspace()
    assert before - cuda.cuda.mem_get_info()[0] <= 8 << 20
    assert int(stages.symmetrize(inds, dists)[0].sum()) == int(want)
    stages.release_workspace()
