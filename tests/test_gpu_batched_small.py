"""Batched FP32 fits of many small problems: memory goes with the points, not with the
problems' number of query tiles (the tensor cores' search pads every problem to 256
rows), and the results are those of single fits on both sides of the size where the
search changes (64 points a problem on average)."""
import pytest

pytestmark = pytest.mark.gpu


def test_memory_goes_with_the_points(cuda):
    import ncvis_gb300 as ncvis
    B, n, D = 2000, 20, 64
    g = cuda.Generator(device="cuda").manual_seed(1)
    Xs = list(cuda.randn((B * n, D), generator=g, device="cuda").split(n))
    vis = ncvis.NCVis(n_epochs=0, n_neighbors=15)
    vis.fit_transform_batched(Xs[:2])  # set-up
    cuda.cuda.empty_cache()
    cuda.cuda.synchronize()
    before = cuda.cuda.mem_get_info()[0]
    out = vis.fit_transform_batched(Xs)
    del out
    cuda.cuda.empty_cache()
    cuda.cuda.synchronize()
    used = before - cuda.cuda.mem_get_info()[0]
    padded_copies = 3 * 2 * B * 256 * 72  # three FP16 copies of 64 + 3 columns, padded to 72
    assert used < padded_copies / 2


@pytest.mark.parametrize("sizes", [[20] * 8, [63] * 5, [64] * 5, [30, 40, 122], [10, 20, 30, 400]])
def test_results_of_single_fits(cuda, sizes):
    """Tolerance as for larger problems: the tables are the same, the statistics of
    the initial embedding may differ in the last FP32 bit, which the epochs carry to
    1e-5."""
    import ncvis_gb300 as ncvis
    g = cuda.Generator(device="cuda").manual_seed(len(sizes))
    Xs = [cuda.randn((n, 12), generator=g, device="cuda") for n in sizes]
    k = min(9, min(sizes) - 1)
    Ys = ncvis.NCVis(n_epochs=0, random_seed=3, n_neighbors=k).fit_transform_batched(Xs)
    for X, Y in zip(Xs, Ys):
        one = ncvis.NCVis(n_epochs=0, random_seed=3, n_neighbors=k).fit_transform(X)
        assert float((Y - one).abs().max()) <= 1e-5 * max(1.0, float(one.abs().max()))
