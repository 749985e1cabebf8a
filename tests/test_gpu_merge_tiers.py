"""Symmetrization (src/knntable.cpp:24-99) at the row lengths and table sizes where
the merge changes hands: one thread per row up to 24 and up to 48 items, one warp
per row up to 128 and up to 1,024 with the sort spread over the lanes, and tables of
up to 40,000 rows, whose rows all go to whole warps.  Bit-exact against the oracle,
with tied distances (std::sort's tie order decides the CSR)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _table(N, k, lengths, levels, seed):
    """A table whose first rows have the given lengths k + in-degree; `levels`
    distances (few: many ties)."""
    rng = np.random.default_rng(seed)
    M = len(lengths)
    inds = M + rng.integers(0, N - M - 1, size=(N, k))
    flat, owner = inds.reshape(-1), np.repeat(np.arange(N), k)
    inds += (inds >= np.arange(N)[:, None]) & (inds < N - 1)
    slots = rng.permutation(np.nonzero(owner >= M)[0])
    at = 0
    for row, length in enumerate(lengths):
        n = length - k
        flat[slots[at:at + n]] = row
        at += n
    dists = (rng.integers(0, levels, size=(N, k)) / levels).astype(np.float32)
    return inds, -np.sort(-dists, axis=1)


@pytest.mark.parametrize("levels", [3, 1 << 20])
@pytest.mark.parametrize("N", [39_000, 40_000, 40_001])
def test_row_lengths(cuda, oracle, N, levels):
    from ncvis_gb300 import stages
    k = 15
    lengths = [15, 16, 17, 23, 24, 25, 26, 31, 32, 33, 47, 48, 49, 50, 63, 64, 65, 127, 128, 129,
               130, 255, 256, 257, 1000, 1023, 1024, 1025, 1026]
    inds, dists = _table(N, k, lengths * 3, levels, N + levels)
    rp, cols, vals = oracle.symmetrize(inds, dists)
    got = stages.symmetrize(cuda.tensor(inds.astype(np.int32), device="cuda"),
                            cuda.tensor(dists, device="cuda"))
    assert np.array_equal(got[0].cpu().numpy(), rp)
    assert np.array_equal(got[1].cpu().numpy(), cols)
    assert np.array_equal(got[2].cpu().numpy().view(np.uint32), vals.view(np.uint32))
    assert np.array_equal(got[3].cpu().numpy(), np.repeat(np.arange(N), np.diff(rp)))


def test_sorted_and_reversed_hubs(cuda, oracle):
    """Hubs whose distances arrive sorted, reversed, organ-pipe and equal: the
    partitions' worst shapes, the heap sort of an exhausted budget among them."""
    from ncvis_gb300 import stages
    N, k = 5000, 8
    rng = np.random.default_rng(1)
    inds = 8 + rng.integers(0, N - 8, size=(N, k))
    dists = -np.sort(-rng.random((N, k)).astype(np.float32), axis=1)
    for h in range(8):
        src = np.arange(100 + 600 * h, 100 + 600 * h + (1000 if h % 2 else 500)) % N
        inds[src, k - 1] = h
        n = src.size
        x = np.arange(n) / n
        shape = [x, 1 - x, np.abs(x - 0.5), np.zeros(n), (np.arange(n) * 7919 % n) / n,
                 np.minimum(x, 0.3), np.where(np.arange(n) % 2, x, 1 - x), np.floor(x * 4)][h]
        dists[src, k - 1] = shape.astype(np.float32) * 0.001
    rp, cols, vals = oracle.symmetrize(inds, dists)
    got = stages.symmetrize(cuda.tensor(inds.astype(np.int32), device="cuda"),
                            cuda.tensor(dists, device="cuda"))
    assert np.array_equal(got[0].cpu().numpy(), rp)
    assert np.array_equal(got[1].cpu().numpy(), cols)
    assert np.array_equal(got[2].cpu().numpy().view(np.uint32), vals.view(np.uint32))
