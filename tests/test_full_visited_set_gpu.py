"""Long walks with a small queue bound: the reference's FixHash loses entries
that then stay, and one of 40 slots (pq 5) fills up with them.  The reference
itself, and the oracle, never leave such a table; the search does, and its
answers are kept here (tests/golden/full_visited_set.npz, from the kernel that
made the hash calls one after another)."""
import os

import numpy as np
import pytest

from conftest import GOLDEN

pytestmark = pytest.mark.gpu


def test_answers_with_a_full_table(song):
    from song_gb300 import datasets as D
    z = np.load(os.path.join(GOLDEN, "full_visited_set.npz"))
    x = D.mixture("unit", 20000, 2, 64, seed=2, center_seed=3)
    q = D.mixture("unit", 3825, 2, 64, seed=9, center_seed=3)
    graph = song.graph_build_gpu(x, "cos", 4, 7, 15, 100, batch_div=32)
    n = len(z["ids"])
    with song.Index(graph, x, 4, "cos") as ix:
        for m in (n, len(q)):  # a block and a warp per query
            ids, hops, evals = ix.search(q[:m], 5, 5, stats=True)
            assert np.array_equal(hops[:n], z["hops"]) and np.array_equal(evals[:n], z["evals"]), m
            assert np.array_equal(ids[:n], z["ids"].astype(np.uint64)), m
