"""Inner products so small that 1 - <q, c> rounds many of them to one FP32 distance:
equal distances go by index (src/ncvis.cpp:128-153 for the rows), so the candidates
are ranked by the distance and not by the product.  The reference rounds the 64-bit
distances to FP32 and sorts them stably; a product summed in FP32 is off by less than
D 2^-24 of it, 2^-32 at most here, a 2^-8th of the distances' spacing 2^-24, and rows
with a distance that near to the middle of two FP32 numbers are left out."""
import pytest

pytestmark = pytest.mark.gpu


def _check(cuda, X, inds, k, rows):
    Xd = X.double()
    checked = 0
    for q in rows.split(500):
        d = 1 - Xd[q] @ Xd.T
        grid = d * 2.0 ** 25  # numbers below 1 are 2^-24 apart, those above 2^-23
        edge = ((grid - grid.round()).abs() < 2.0 ** -7) & (grid.round() % 2 == 1)
        v, i = cuda.sort(d.float(), dim=1, stable=True)
        cut = v[:, k:k + 1].double() + 2.0 ** -23
        clear = ~(edge & (d <= cut)).any(1)
        assert cuda.equal(inds[q][clear].long(), i[:, 1:k + 1].flip(1)[clear])
        checked += int(clear.sum())
    assert checked > 0


@pytest.mark.parametrize("exponent", [-12, -16, -18, -20, -24, -40])
@pytest.mark.parametrize("N,D", [(1000, 16), (20_000, 64)])
def test_order_of_rounded_distances(cuda, N, D, exponent):
    from ncvis_gb300 import stages
    g = cuda.Generator(device="cuda").manual_seed(N)
    X = cuda.randn((N, D), generator=g, device="cuda")
    X = X / X.norm(dim=1).max() * 2.0 ** (exponent / 2)
    inds, _ = stages.knn(X, 15, 1)
    _check(cuda, X, inds, 15, cuda.randperm(N, generator=g, device="cuda")[:1000])


def test_a_small_problem_of_a_batch(cuda):
    """Against the CUDA cores' search, which a rerank factor of 5 selects."""
    import ncvis_gb300 as ncvis
    g = cuda.Generator(device="cuda").manual_seed(2)
    Xs = [s * cuda.randn((4000, 16), generator=g, device="cuda") for s in (2.0 ** -4, 2.0 ** -14)]
    got = []
    for factor in (0, 5):
        vis = ncvis.NCVis(n_epochs=0, random_seed=3, n_neighbors=15, distance="inner_product")
        vis.set_options(rerank_factor=factor)
        got.append(vis.fit_transform_batched(Xs))
    assert cuda.equal(got[0][1], got[1][1])
