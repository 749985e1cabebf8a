"""The bounded waits of the FP32 search's tensor-core form, as test_gpu_failure.py has
them for the BF16 search: with the stall diagnostic and a short limit the fit reports
NCVIS_DEVICE_TIMEOUT, whatever lists the stopped kernel left for what follows, and the
same handle fits again without it.  Sizes: the query tiles' lists of several CTAs are
merged (6,000 rows), whole tiles (38,912), and both in one sweep (39,168)."""
import pytest

from conftest import gmm

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N", [6000, 38_912, 39_168])
def test_fit(cuda, N):
    import ncvis_gb300 as ncvis
    from ncvis_gb300 import _lib
    Xd = cuda.tensor(gmm(N, 16, 6, 5.0, seed=5)[0], device="cuda")
    vis = ncvis.NCVis(random_seed=5, n_epochs=0, knn_precision="fp32")
    want = vis.fit_transform(Xd)
    vis.set_options(inject_stall=1, wait_limit_cycles=200_000)
    with pytest.raises(ncvis.NcvisError) as info:
        vis.fit_transform(Xd)
    assert info.value.code == _lib.NCVIS_DEVICE_TIMEOUT, str(info.value)
    assert "timed out" in str(info.value)
    vis.set_options(inject_stall=0, wait_limit_cycles=0)
    assert cuda.equal(vis.fit_transform(Xd), want)


def test_batched_fit(cuda):
    import ncvis_gb300 as ncvis
    from ncvis_gb300 import _lib
    Xs = [cuda.tensor(gmm(n, 16, 3, 5.0, seed=n)[0], device="cuda") for n in (700, 1300)]
    vis = ncvis.NCVis(random_seed=1, n_epochs=0, knn_precision="fp32")
    want = vis.fit_transform_batched(Xs)
    vis.set_options(inject_stall=1, wait_limit_cycles=200_000)
    with pytest.raises(ncvis.NcvisError) as info:
        vis.fit_transform_batched(Xs)
    assert info.value.code == _lib.NCVIS_DEVICE_TIMEOUT
    vis.set_options(inject_stall=0, wait_limit_cycles=0)
    assert all(cuda.equal(a, b) for a, b in zip(vis.fit_transform_batched(Xs), want))
