"""init_embedding's row kernels at the row lengths where they change (one thread a
row up to 64 columns, a whole warp beyond; loads of 8 and 128 columns), in
every embedding dimension's form, against a plain statement of the recurrence
(src/ncvis.cpp:184-273) in FP32 with double statistics; and what the entry point
refuses.

Tolerance: the neighbour sums are those of one thread bit for bit, the FP64
statistics may differ in the last FP32 bit, and the epochs carry that to at most
1e-6 of the largest value."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _graph(N, seed, lengths):
    """A CSR whose rows have the given lengths in turn, columns at random."""
    rng = np.random.default_rng(seed)
    n = np.resize(np.asarray(lengths), N)
    rp = np.concatenate([[0], np.cumsum(n)]).astype(np.int64)
    return rp, rng.integers(0, N, rp[-1]).astype(np.int32)


def _stated(oracle, rp, cols, d, epochs):
    """One edge at a time in row order, FP32, multiply then add; IEEE division."""
    N = rp.size - 1
    alpha = np.float32(1 / 15)
    y = oracle.uniform_real(11, N * d).reshape(N, d)
    n = np.diff(rp)
    with np.errstate(all="ignore"):
        for _ in range(epochs):
            z = np.zeros((N, d), np.float32)
            for e in range(n.max()):
                at = np.nonzero(n > e)[0]
                z[at] += alpha * y[cols[rp[at] + e]]
            mean = z.astype(np.float64).sum(0).astype(np.float32) / np.float32(N)
            dev = z - mean
            var = (dev * dev).astype(np.float64).sum(0).astype(np.float32) / np.float32(N)
            y = dev / np.sqrt(var)
    return y


def _run(cuda, rp, cols, d, epochs, out=None):
    from ncvis_gb300 import stages
    return stages.init_embedding(cuda.tensor(rp, device="cuda"), cuda.tensor(cols, device="cuda"),
                                 d, 11, epochs, np.float32(1 / 15))


@pytest.mark.parametrize("d", [1, 2, 3, 4, 5, 8, 17, 32])
@pytest.mark.parametrize("N,lengths", [(2, [1]), (33, [7, 8, 9]), (1000, [1, 31, 32, 33, 63, 64]),
                                       (4099, [20, 64, 65, 127, 128, 129, 700, 2])])
def test_row_lengths(cuda, oracle, d, N, lengths):
    rp, cols = _graph(N, N + d, lengths)
    for epochs in (1, 2, 7):
        ref = _stated(oracle, rp, cols, d, epochs)
        got = _run(cuda, rp, cols, d, epochs).cpu().numpy()
        fine = np.isfinite(ref)
        assert np.array_equal(fine, np.isfinite(got))
        scale = max(1.0, np.abs(ref[fine]).max(initial=0.0))
        assert np.abs(got - ref)[fine].max(initial=0.0) <= 1e-6 * scale


def test_unaligned_output(cuda):
    """An embedding of 4 dimensions that starts on an 8-byte boundary."""
    import ctypes as C
    from ncvis_gb300 import _lib
    N, d = 600, 4
    rp, cols = _graph(N, 1, [24])
    t_rp, t_cols = cuda.tensor(rp, device="cuda"), cuda.tensor(cols, device="cuda")
    buf = cuda.zeros(N * d + 2, dtype=cuda.float32, device="cuda")
    out = buf[2:].view(N, d)
    _lib.check(_lib.lib().ncvis_init_embedding_device(
        N, d, t_rp.data_ptr(), t_cols.data_ptr(), 11, 3, 1 / 15, 0, C.c_void_p(out.data_ptr()),
        cuda.cuda.current_stream().cuda_stream))
    want = _run(cuda, rp, cols, d, 3)
    assert float((out - want).abs().max()) <= 1e-6 * max(1.0, float(want.abs().max()))


@pytest.mark.parametrize("d", [1, 2, 3, 4])
def test_many_rows(cuda, oracle, d):
    """Beyond 300,000 rows a row keeps its one thread whatever its length."""
    rp, cols = _graph(300_003, 5, [3, 9, 70])
    ref = _stated(oracle, rp, cols, d, 2)
    got = _run(cuda, rp, cols, d, 2).cpu().numpy()
    assert np.abs(got - ref).max() <= 1e-6 * max(1.0, np.abs(ref).max())


@pytest.mark.parametrize("d", [1, 2, 3, 4])
def test_unaligned_columns(cuda, d):
    """Columns that start off a 16-byte boundary are read one by one."""
    rp, cols = _graph(700, 3, [5, 26, 90, 64])
    want = _run(cuda, rp, cols, d, 4)
    from ncvis_gb300 import stages
    shifted = cuda.tensor(np.concatenate([[0], cols]).astype(np.int32), device="cuda")[1:]
    got = stages.init_embedding(cuda.tensor(rp, device="cuda"), shifted, d, 11, 4,
                                np.float32(1 / 15))
    assert cuda.equal(got, want)


@pytest.mark.parametrize("where,value,text", [
    ("rp", (0, 1), "row_ptr\\[0\\]"), ("rp", (300, 1), "non-decreasing"),
    ("rp", (600, 1 << 31), "too many"), ("cols", (5000, 600), "column index"),
    ("cols", (0, -1), "column index")])
def test_refuses_bad_graphs(cuda, where, value, text):
    from ncvis_gb300 import NcvisError
    rp, cols = _graph(600, 2, [24])
    {"rp": rp, "cols": cols}[where][value[0]] = value[1]
    with pytest.raises(NcvisError, match=text):
        _run(cuda, rp, cols, 2, 1)
