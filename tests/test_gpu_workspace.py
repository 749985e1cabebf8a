"""The stage calls' memory pool: what it keeps between calls is bounded, goes back
when an engine that fitted is destroyed, and serves calls from several threads on
several streams at once (src/ncvis.cpp has no counterpart: its buffers are the
host's)."""
import threading

import pytest

pytestmark = pytest.mark.gpu


def _free(cuda):
    cuda.cuda.synchronize()
    return cuda.cuda.mem_get_info()[0]


def test_kept_memory_is_bounded_and_given_back(cuda):
    from ncvis_gb300 import NCVis, stages
    X = cuda.randn((3000, 8), device="cuda")
    NCVis(n_epochs=0).fit_transform(X)  # set-up; its engine's end empties the pool
    cuda.cuda.empty_cache()
    before = _free(cuda)
    n, k = 1_500_000, 30  # a workspace above the gigabyte that may be kept
    inds = cuda.randint(0, n, (n, k), device="cuda", dtype=cuda.int32)
    dists = cuda.rand((n, k), device="cuda")
    out = stages.symmetrize(inds, dists)
    assert out[1].numel() > 0
    del out, inds, dists
    cuda.cuda.empty_cache()
    assert before - _free(cuda) <= (1 << 30) + (64 << 20)
    vis = NCVis(n_epochs=0)
    vis.fit_transform(X)
    del vis
    cuda.cuda.empty_cache()
    assert before - _free(cuda) <= 64 << 20


def test_threads_and_streams(cuda):
    from ncvis_gb300 import stages
    Xs = [cuda.randn((1500 + 137 * t, 16), device="cuda") for t in range(4)]
    want = [stages.knn(X, 10) for X in Xs]
    got, errors = [None] * 4, []

    def work(t):
        try:
            with cuda.cuda.stream(cuda.cuda.Stream()):
                for _ in range(8):
                    got[t] = stages.knn(Xs[t], 10)
                cuda.cuda.current_stream().synchronize()
        except Exception as e:  # noqa: BLE001
            errors.append(e)

    cuda.cuda.synchronize()
    threads = [threading.Thread(target=work, args=(t,)) for t in range(4)]
    [t.start() for t in threads]
    [t.join() for t in threads]
    assert not errors
    for (i, d), (wi, wd) in zip(got, want):
        assert cuda.equal(i, wi) and cuda.equal(d, wd)
