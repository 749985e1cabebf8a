"""Tied distances in the FP32 search: on whole numbers (and halves) every distance is
exact in FP32, many are equal, and the table holds the k + 1 smallest (distance,
index) pairs (src/ncvis.cpp:128-153 for the rows), however the search scores its
candidates.  Coordinates above 2,048 need the FP16 parts' low halves, in rows of up to
32 columns and of more; a row of squared norm 2^23 is the largest whose sums stay below
2^24.  The reference is the stable sort of the 64-bit distances, which are exact here,
so the comparison has no tolerance."""
import pytest

pytestmark = pytest.mark.gpu


def _columns(cuda, g, N, D, kind):
    def whole(lo, hi, d=D):
        return cuda.randint(lo, hi, (N, d), generator=g, device="cuda").float()
    if kind == "binary":
        return whole(0, 2)
    if kind == "signs":
        return 2 * whole(0, 2) - 1
    if kind == "levels":
        return whole(0, 4)
    if kind == "halves":
        return 0.5 * whole(0, 5)
    if kind == "tiny units":
        return 2.0 ** -40 * whole(0, 3)
    X = whole(0, 2)
    if kind == "one column above 2,048":
        X[:, 0] = 2049 + 2 * whole(0, 3, 1)[:, 0]
    elif kind == "largest norm":
        X[:, D - 1] = 2895.0 - whole(0, 2, 1)[:, 0]
    elif kind == "pixels":
        X = whole(0, 2) * 254 + whole(0, 2)
    elif kind == "one row of other numbers":
        X[N // 2] = cuda.randn(D, generator=g, device="cuda")
    elif kind == "one long row":
        X[N // 3, 0] = 3000.0
    return X


@pytest.mark.parametrize("N,D,dist,kind", [
    (45_000, 32, 0, "binary"), (60_000, 32, 0, "binary"), (60_000, 64, 0, "binary"),
    (45_000, 32, 1, "binary"), (45_000, 24, 0, "signs"), (60_000, 16, 0, "levels"),
    (60_000, 33, 1, "levels"), (45_000, 24, 0, "halves"), (45_000, 32, 0, "tiny units"),
    (45_000, 24, 0, "one column above 2,048"), (45_000, 40, 0, "one column above 2,048"),
    (45_000, 29, 0, "largest norm"), (45_000, 40, 0, "largest norm"),
    (45_000, 40, 1, "largest norm"), (45_000, 16, 0, "pixels"), (45_000, 100, 0, "binary"),
    (45_000, 32, 0, "one row of other numbers"), (45_000, 32, 0, "one long row"),
    (1000, 16, 0, "binary"), (10_000, 24, 0, "binary")])
def test_equal_distances_go_by_index(cuda, N, D, dist, kind):
    from ncvis_gb300 import stages
    k = 15
    g = cuda.Generator(device="cuda").manual_seed(N + D)
    X = _columns(cuda, g, N, D, kind)
    inds, dists = stages.knn(X, k, dist)
    Xd = X.double()
    rows = cuda.randperm(N, generator=g, device="cuda")[:2000]
    if kind == "one row of other numbers":
        rows = rows[rows != N // 2]  # its own sums are not exact
    n2 = Xd.square().sum(1)
    ties = 0
    for q in rows.split(500):
        dot = Xd[q] @ Xd.T
        d = n2[q, None] + n2[None, :] - 2 * dot if dist == 0 else 1 - dot
        if kind == "one row of other numbers":
            d[:, N // 2] = cuda.inf  # far from every other row
        v, i = cuda.sort(d, dim=1, stable=True)
        assert cuda.equal(inds[q].long(), i[:, 1:k + 1].flip(1))
        assert cuda.equal(dists[q].double(), v[:, 1:k + 1].flip(1))
        ties += int((v[:, k] == v[:, k + 1]).sum())
    assert ties > 0


@pytest.mark.parametrize("D,kind", [(32, "binary"), (40, "one column above 2,048")])
def test_batched_problems(cuda, D, kind):
    """The batched search against the one on the CUDA cores, which a rerank factor of
    5 selects, through the embedding before the optimizer."""
    import ncvis_gb300 as ncvis
    g = cuda.Generator(device="cuda").manual_seed(D)
    Xs = [_columns(cuda, g, n, D, kind) for n in (9000, 3000)]
    got = []
    for factor in (0, 5):
        vis = ncvis.NCVis(n_epochs=0, random_seed=3, n_neighbors=15)
        vis.set_options(rerank_factor=factor)
        got.append(vis.fit_transform_batched(Xs))
    for a, b in zip(*got):
        assert cuda.equal(a, b)
