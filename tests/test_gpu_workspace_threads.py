"""One workspace pool per device, whichever threads call: a stage call that is the
first thing a new thread does uses the pool that is there, so that what a program with
a thread per request keeps is bounded as in test_gpu_workspace.py."""
import threading

import pytest

pytestmark = pytest.mark.gpu


def test_short_lived_threads(cuda):
    from ncvis_gb300 import NCVis, _lib
    L = _lib.lib()
    N, D, k = 600_000, 4, 30
    X = cuda.randn((N, D), device="cuda")
    inds = cuda.randint(0, N, (N, k), device="cuda", dtype=cuda.int32)
    dists = cuda.rand((N, k), device="cuda")
    rp = cuda.empty(N + 1, dtype=cuda.int64, device="cuda")
    cols = cuda.empty(2 * N * k, dtype=cuda.int32, device="cuda")
    vals = cuda.empty(2 * N * k, dtype=cuda.float32, device="cuda")
    src = cuda.empty(2 * N * k, dtype=cuda.int32, device="cuda")
    import ctypes as C
    errors = []

    def call():  # about 630 MB of workspace; no CUDA call of the thread's own before it
        n = C.c_size_t(0)
        rc = L.ncvis_symmetrize_device(N, k, inds.data_ptr(), dists.data_ptr(), rp.data_ptr(),
                                       cols.data_ptr(), vals.data_ptr(), src.data_ptr(),
                                       C.byref(n), None)
        if rc != 0:
            errors.append(L.ncvis_get_last_error())

    NCVis(n_epochs=0).fit_transform(X[:50_000])  # set-up; its engine's end empties the pool
    cuda.cuda.empty_cache()
    cuda.cuda.synchronize()
    before = cuda.cuda.mem_get_info()[0]
    for _ in range(6):
        t = threading.Thread(target=call)
        t.start()
        t.join()
    assert not errors
    cuda.cuda.synchronize()
    assert before - cuda.cuda.mem_get_info()[0] <= (1 << 30) + (64 << 20)
    # And the pool that served them is the one an engine's end empties.
    vis = NCVis(n_epochs=0)
    vis.fit_transform(X[:3000])
    del vis
    cuda.cuda.empty_cache()
    cuda.cuda.synchronize()
    assert before - cuda.cuda.mem_get_info()[0] <= 64 << 20
