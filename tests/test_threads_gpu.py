"""Several host threads, each with indexes of its own: what a call sets on a
kernel holds for the whole process, so it must not be what another thread's
launch of the same kernel does not fit."""
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _index(song, dim, n=600, seed=0):
    rng = np.random.default_rng(seed + dim)
    data = rng.standard_normal((n, dim)).astype(np.float32)
    g = np.zeros((n, 16), dtype=np.uint64)
    g[:, 0] = 15
    g[:, 1:] = rng.integers(0, n, (n, 15))
    return song.Index(g, data, 4, 0), data[rng.integers(0, n, 8)]


@pytest.mark.parametrize("kind", ["flat", "two_level", "build"])
def test_threads_with_rows_of_different_widths(song, kind):
    """The same kernels for short and for long rows at once: every call runs
    and returns what it returns alone."""
    failures = []

    def work(call, want):
        try:
            for _ in range(100 if kind == "build" else 3000):
                if not np.array_equal(call(), want):
                    failures.append("another result")
                    return
        except Exception as e:  # noqa: BLE001
            failures.append(repr(e))

    if kind == "build":
        calls = []
        for dim in (4, 700):
            data = np.random.default_rng(dim).standard_normal((200, dim)).astype(np.float32)
            calls.append(lambda d=data: song.graph_build_gpu(d, "l2", 4, 7, 15, 40, batch_div=2, nthreads=1))
    else:
        calls = []
        for dim in (8, 4000):
            ix, q = _index(song, dim)
            if kind == "flat":
                ix.set_entries(np.arange(0, 600, 40, dtype=np.uint64), starts=2)
            else:
                ix.set_entries(np.arange(0, 600, 20, dtype=np.uint64), starts=2, coarse=8, probes=3)
                ix.debug_head_path(False)
            calls.append(lambda i=ix, x=q: i.search(x, 10, 5))
    wants = [c() for c in calls]
    threads = [threading.Thread(target=work, args=(c, w)) for c, w in zip(calls, wants)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not failures, failures
