"""init_embedding's statistics (src/ncvis.cpp:226-261) where squared deviations leave
FP32's range: their sum is infinite, and so is sigma, whatever adds it up; a finite
deviation over it is zero.  The second epoch then has a deviation of zero and divides
zero by zero, as the reference does."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("d", [1, 2, 3, 4, 5])
@pytest.mark.parametrize("N", [40, 1000, 300_003])
def test_infinite_squares(cuda, oracle, N, d):
    from ncvis_gb300 import stages
    rng = np.random.default_rng(N)
    deg = 8
    rp = np.arange(N + 1, dtype=np.int64) * deg
    cols = rng.integers(0, N, N * deg).astype(np.int32)
    alpha = np.float32(1e25)
    # One epoch by hand: sums of up to 8e25, squares of deviations beyond FP32.
    y = oracle.uniform_real(11, N * d).reshape(N, d)
    z = np.zeros((N, d), np.float32)
    for e in range(deg):
        z += alpha * y[cols[e::deg]]
    dev = z - z.astype(np.float64).sum(0).astype(np.float32) / np.float32(N)
    with np.errstate(over="ignore"):
        assert np.isinf((dev * dev).max(0)).all()
    for epochs, want in ((1, 0.0), (2, np.nan)):
        got = stages.init_embedding(cuda.tensor(rp, device="cuda"), cuda.tensor(cols, device="cuda"),
                                    d, 11, epochs, alpha).cpu().numpy()
        assert np.array_equal(got, np.full((N, d), want, np.float32), equal_nan=True)


def test_infinite_squares_in_a_hub(cuda):
    """Rows of more than 64 columns are taken by whole warps."""
    from ncvis_gb300 import stages
    N = 500
    rng = np.random.default_rng(1)
    n = np.where(np.arange(N) % 50 == 0, 200, 3)
    rp = np.concatenate([[0], np.cumsum(n)]).astype(np.int64)
    cols = rng.integers(0, N, rp[-1]).astype(np.int32)
    got = stages.init_embedding(cuda.tensor(rp, device="cuda"), cuda.tensor(cols, device="cuda"),
                                2, 11, 1, np.float32(1e25))
    assert not bool(got.any()) and bool(cuda.isfinite(got).all())
