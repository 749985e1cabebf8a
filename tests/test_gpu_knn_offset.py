"""The FP32 search in squared L2 on rows far from the origin, where |c|^2 - 2<q, c>
cancels: its selection loses no more neighbours than the search on the CUDA cores,
which one row of a norm 2^14 times the others' selects for the same points (that row
is nobody's neighbour)."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N", [1000, 10_000, 60_000])
@pytest.mark.parametrize("D", [8, 64, 125])
@pytest.mark.parametrize("offset", [30.0, 300.0, 1000.0])
def test_recall_on_rows_with_an_offset(cuda, N, D, offset):
    from ncvis_gb300 import stages
    k = 15
    g = cuda.Generator(device="cuda").manual_seed(N + D)
    X = cuda.randn((N, D), generator=g, device="cuda") + offset
    rows = cuda.randperm(N, generator=g, device="cuda")[:1000]
    d = cuda.cdist(X[rows].double(), X.double(),
                   compute_mode="donot_use_mm_for_euclid_dist").square()
    kth = cuda.topk(d, k + 1, dim=1, largest=False).values[:, k:]
    far = cuda.cat([X, 2.0 ** 14 * X[:1]])
    lost = []
    for table in (stages.knn(X, k, 0)[0], stages.knn(far, k, 0)[0]):
        got = cuda.gather(d, 1, table[rows].long().clamp(0, N - 1))
        lost.append(int((got > kth * (1 + 1e-6)).sum()))
    assert lost[0] <= lost[1]
