"""The BF16 search with the last wave's query tiles shared out over several CTAs
(src/ncvis.cpp:72-153 for what it replaces): every row's kept candidates are the
best R by BF16 score over all rows, whichever CTA met them and whether the list was
filled by merging (below 147,456 rows, lists of 32) or by single insertions.

The reference scores the rounded rows in 64 bits, keeps the best R and ranks them
by their exact distances.  Rows are unit vectors, so a score sums D products of
magnitude 1 in all at 32 bits: at most 2 D 2^-23 < 2e-5 off for D <= 64, and rows
whose R-th and next score are closer than twice that are left out.  A distance
1 - <q, c> summed in 32 bits is within D 2^-23 < 1e-5."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("k", [15, 30])
@pytest.mark.parametrize("N,D,ordered", [
    (257, 8, True), (1000, 32, True), (4097, 17, True), (10000, 64, True), (12289, 33, True),
    (38913, 16, False), (38913, 16, True), (60013, 24, True), (60013, 24, False),
    (78000, 32, True), (131072, 20, True), (147455, 9, True), (147456, 9, True),
    (2049, 8, True)])
def test_kept_candidates_of_split_rows(cuda, N, D, ordered, k):
    from ncvis_gb300 import DISTANCES, stages
    g = cuda.Generator(device="cuda").manual_seed(N + D)
    centres = cuda.randn((9, D), generator=g, device="cuda")
    X = centres[cuda.randint(0, 9, (N,), generator=g, device="cuda")]
    X = X + 0.7 * cuda.randn((N, D), generator=g, device="cuda")
    X = X / X.norm(dim=1, keepdim=True)
    _, dists = stages.knn(X, k, DISTANCES["inner_product"], precision=1, order=ordered)
    R = 32 if k == 15 else 64
    Xd, Xb = X.double(), X.bfloat16().double()
    checked = 0
    rows = cuda.randperm(N, generator=g, device="cuda")[:3000]
    for q in rows.split(500):
        top = cuda.topk(Xb[q] @ Xb.T, R + 1, dim=1)
        clear = (top.values[:, R - 1] - top.values[:, R]) > 4e-5
        cand = top.indices[:, :R]
        d = 1 - (Xd[q][:, None, :] * Xd[cand]).sum(2)
        ref = cuda.sort(d, dim=1).values[:, 1:k + 1].flip(1)
        cuda.testing.assert_close(dists[q][clear].double(), ref[clear], rtol=0, atol=1e-5)
        checked += int(clear.sum())
    assert checked > 0
