"""A fit in three dimensions, whose initial embedding pads its rows to four floats,
needs no larger arena than the rows of three dimensions take (arena_limit refuses a
fit that needs more)."""
import pytest

pytestmark = pytest.mark.gpu


def _need(fit):
    import ncvis_gb300 as ncvis
    low, high = 1, 1 << 34
    while high - low > 256:
        middle = (low + high) // 2
        try:
            fit(middle)
            high = middle
        except ncvis.NcvisError as e:
            assert "arena_limit" in str(e)
            low = middle
    return high


@pytest.mark.parametrize("batched", [False, True])
def test_three_dimensions(cuda, batched):
    import ncvis_gb300 as ncvis
    N = 50_000
    X = cuda.randn((N, 4), device="cuda")

    def fit(d):
        def run(limit):
            vis = ncvis.NCVis(d=d, n_neighbors=1, n_epochs=0, rerank_factor=1, arena_limit=limit)
            return vis.fit_transform_batched([X[:N // 2], X[N // 2:]]) if batched \
                else vis.fit_transform(X)
        return run

    # A few arrays of one float a row go with the dimensions; the padding would be six.
    assert _need(fit(3)) - _need(fit(2)) <= 3 * 4 * N
