"""A stage call whose FP32 search runs on the CUDA cores waits for the check of its
input only: the search, tens of milliseconds here, is in flight when it returns, so
that a program goes on meanwhile."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind", ["norms too far apart", "many candidates"])
def test_search_is_left_in_flight(cuda, kind):
    from ncvis_gb300 import stages
    N, D = 40_000, 64
    X = cuda.randn((N, D), device="cuda")
    factor = 0
    if kind == "norms too far apart":
        X[0] *= 2.0 ** 30
    else:
        factor = 5
    want = stages.knn(X, 15, 0, rerank_factor=factor)
    cuda.cuda.synchronize()
    got = stages.knn(X, 15, 0, rerank_factor=factor)
    assert not cuda.cuda.current_stream().query()
    assert cuda.equal(got[0], want[0]) and cuda.equal(got[1], want[1])
