"""Tables with NaN distances, which the symmetrization accepts as the reference does
(src/knntable.cpp:24-99 sorts whatever it is given): the rows come out in std::sort's
order, in every tier of the merge."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

from conftest import ROOT


def _compile(path, *flags):
    r = subprocess.run(["g++", "-std=c++17", "-O2", "-I", os.path.join(ROOT, "ncvis_gb300", "csrc"),
                        os.path.join(ROOT, "tests", "harness", "nan_rows_check.cpp"), "-o", path,
                        *flags], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    return path


def test_rows_in_order_on_the_host(tmp_path):
    """tests/harness/nan_rows_check.cpp."""
    exe = _compile(str(tmp_path / "nan_rows_check"))
    r = subprocess.run([exe, "20000"], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout + r.stderr
    ok, rows, collide = r.stdout.split()
    assert ok == "ok" and int(rows) == 20000 and int(collide) > 0


def _reference(tmp_path, inds, dists):
    lib = ctypes.CDLL(_compile(str(tmp_path / "nan_rows.so"), "-shared", "-fPIC"))
    N, k = inds.shape
    rp = np.empty(N + 1, np.int64)
    cols, vals = np.empty(2 * N * k, np.int32), np.empty(2 * N * k, np.float32)
    f = lib.nan_symmetrize
    f.restype = ctypes.c_int64
    p = [a.ctypes.data_as(ctypes.c_void_p) for a in (inds, dists, rp, cols, vals)]
    E = f(ctypes.c_int64(N), ctypes.c_int64(k), *p)
    return rp, cols[:E], vals[:E]


@pytest.mark.gpu
@pytest.mark.parametrize("share", [0.0001, 0.3, 1.0])
@pytest.mark.parametrize("N", [3000, 40_001])
def test_bit_exact(cuda, tmp_path, N, share):
    """Rows of 15 to 1,100 items, tables on both sides of the size from which short
    rows get a thread each."""
    from ncvis_gb300 import stages
    k = 15
    rng = np.random.default_rng(N)
    inds = (40 + rng.integers(0, N - 40, size=(N, k))).astype(np.int32)
    flat = inds.reshape(-1)
    slots = rng.permutation(np.arange(40 * k, N * k))
    at = 0
    for row, n in enumerate([3, 9, 10, 32, 33, 34, 60, 112, 113, 114, 300, 1000, 1009, 1010, 1085]):
        flat[slots[at:at + n]] = row
        at += n
    dists = -np.sort(-rng.integers(0, 50, size=(N, k)).astype(np.float32), axis=1)
    dists[rng.random((N, k)) < share] = np.nan
    dists[5, 3] = dists[N - 1, 0] = np.nan
    for row in (3, 6, 9, 10, 11, 14):  # rows of every tier hold one
        dists[row, 7] = np.nan
    rp, cols, vals = _reference(tmp_path, inds, dists)
    got = [t.cpu().numpy() for t in stages.symmetrize(
        cuda.tensor(inds, device="cuda"), cuda.tensor(dists, device="cuda"))]
    assert np.array_equal(got[0], rp)
    assert np.array_equal(got[1], cols)
    assert np.array_equal(got[2].view(np.uint32), vals.view(np.uint32))
    assert np.array_equal(got[3], np.repeat(np.arange(N), np.diff(rp)))
