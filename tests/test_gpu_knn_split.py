"""The FP32 search on the tensor cores (FP16 high and low parts of the rows,
src/ncvis.cpp:72-153 for what it replaces) against the search on the CUDA cores,
which a rerank factor of 5 selects for k = 15 (75 candidates per point).

Both keep more candidates than the k + 1 that are ranked, and both are ranked by
the same exact FP32 distances, so the tables agree bit for bit; only the order
of equal distances at the cut-off could differ, and (distance, index) decides
that in both.  The sizes lie at the edges of the query tile (256), the candidate
tile (128), the sweep's split of the last wave, and the column counts where the
K steps (16), the 64-column halves and the folded norm columns (3) begin."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _both(cuda, X, k, dist):
    from ncvis_gb300 import stages
    Xd = cuda.as_tensor(X, device="cuda")
    a = stages.knn(Xd, k, dist)
    b = stages.knn(Xd, k, dist, rerank_factor=5 if k >= 13 else 64 // k + 1)
    return a, b


def _points(cuda, N, D, seed):
    g = cuda.Generator(device="cuda").manual_seed(seed)
    centres = 4.0 * cuda.randn((7, D), generator=g, device="cuda")
    label = cuda.randint(0, 7, (N,), generator=g, device="cuda")
    return centres[label] + cuda.randn((N, D), generator=g, device="cuda")


@pytest.mark.parametrize("dist", [0, 1, 2, 3])
@pytest.mark.parametrize("N,D", [(64, 8), (127, 13), (129, 16), (256, 61), (257, 62), (1000, 64),
                                 (4097, 65), (3000, 125), (2049, 17), (300, 7)])
def test_same_table_as_the_cuda_cores(cuda, N, D, dist):
    a, b = _both(cuda, _points(cuda, N, D, N + D), 15, dist)
    assert cuda.equal(a[1], b[1])
    assert cuda.equal(a[0], b[0])


@pytest.mark.parametrize("N", [38656, 39168, 78000, 97280])
def test_last_wave_of_query_tiles(cuda, N):
    """151 (whole), 153 (one left), 305 and 380 query tiles: no split, a split of
    one tile, of one tile after two waves, and of half a wave."""
    a, b = _both(cuda, _points(cuda, N, 8, N), 15, 0)
    assert cuda.equal(a[1], b[1]) and cuda.equal(a[0], b[0])


@pytest.mark.parametrize("k", [1, 5, 16, 17, 30, 32, 33])
def test_neighbour_counts(cuda, k):
    """Lists of 32 and 64 candidates; 33 neighbours (66 candidates) stay on the
    CUDA cores."""
    from ncvis_gb300 import stages
    X = _points(cuda, 1500, 20, k)
    inds, dists = stages.knn(X, k, 0)
    d2 = cuda.cdist(X.double(), X.double()).square()
    ref = cuda.sort(d2, dim=1).values[:, 1:k + 1].flip(1)
    cuda.testing.assert_close(dists.double(), ref, rtol=1e-5, atol=1e-5)


@pytest.mark.parametrize("span", [12.0, 14.0, 30.0])
def test_rows_of_very_different_norms(cuda, span):
    """Norms over 2^span: within 2^13 the parts hold every row, beyond it the call
    goes to the CUDA cores; a row of zeros is held by any scale."""
    X = _points(cuda, 700, 12, 3)
    X = X / X.norm(dim=1, keepdim=True)
    X = X * cuda.exp2(cuda.linspace(0, span, 700, device="cuda"))[:, None]
    X[5] = 0
    for dist in (0, 1):
        a, b = _both(cuda, X, 15, dist)
        assert cuda.equal(a[1], b[1]) and cuda.equal(a[0], b[0])


@pytest.mark.parametrize("scale", [1e-12, 1e12])
def test_units_do_not_matter(cuda, scale):
    X = _points(cuda, 900, 24, 4)
    a, _ = _both(cuda, X, 15, 0)
    b, c = _both(cuda, X * scale, 15, 0)
    assert cuda.equal(b[0], c[0]) and cuda.equal(b[1], c[1])
    assert float((a[0] == b[0]).float().mean()) > 0.99  # up to ties of rounding


def test_exact_twins_in_index_order(cuda):
    X = _points(cuda, 400, 9, 5)
    X = cuda.cat([X, X, X])
    a, b = _both(cuda, X, 15, 0)
    assert cuda.equal(a[0], b[0])


def test_batched_problems_match_single_fits(cuda):
    """FP32 batched problems, one below and some above the tile sizes, against the
    single fits' tables through the embedding before the optimizer."""
    import ncvis_gb300 as ncvis
    Xs = [_points(cuda, n, 16, n) for n in (70, 256, 1001, 3333)]
    vis = ncvis.NCVis(n_epochs=0, random_seed=3)
    Ys = vis.fit_transform_batched(Xs)
    for X, Y in zip(Xs, Ys):
        one = ncvis.NCVis(n_epochs=0, random_seed=3).fit_transform(X)
        assert float((Y - one).abs().max()) <= 1e-5 * max(1.0, float(one.abs().max()))
        assert bool(cuda.isfinite(Y).all()) and np.isfinite(float(Y.sum()))
