"""The two-level entry choice at the sizes where its route or its split
changes: batches around the two-kernel limit (512 queries, or a bound on
queries x heads x dimensions) and its group of four, more or fewer tasks per warp, heads that do not fill a chunk, clusters
that do not fill a pass, and row widths at the remainders.  Starts (through
the searches they seed) equal the oracle's."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dim,metric", [(3, 0), (16, 2), (33, 1), (128, 0), (132, 2), (300, 0)])
@pytest.mark.parametrize("coarse,probes,ns", [(1, 1, 1), (65, 2, 1), (130, 3, 2), (200, 4, 4), (70, 8, 8)])
def test_two_level_choice(song, oracle, dim, metric, coarse, probes, ns):
    from song_gb300 import datasets as D
    n = 1500
    data = D.mixture("unit", n, dim, 12, seed=dim, center_seed=dim + 1)
    q = D.mixture("unit", 1100, dim, 12, seed=dim + 2, center_seed=dim + 1)
    graph = song.graph_build(data, metric, 4, 7, 15, 60, batch_div=16)
    ox = oracle.OracleIndex(data, graph, 4, metric)
    ent = np.random.default_rng(dim + coarse).choice(n, 700, replace=False).astype(np.uint64)
    starts = ox.nearest_entry_2level(q, ent, coarse, probes, ns)
    o_ids, o_hops, o_evals, _ = ox.kernel_search_from(q, starts, 12, oracle.MODE_LEX)
    with song.Index(graph, data, 4, metric) as ix:
        ix.set_entries(ent, starts=ns, coarse=coarse, probes=probes)
        for nq in (1, 3, 4, 5, 63, 257, 511, 512, 513, 1100):
            ids, hops, evals = ix.search(q[:nq], 12, 12, stats=True)
            assert np.array_equal(ids, o_ids[:nq]), nq
            assert np.array_equal(hops, o_hops[:nq]) and np.array_equal(evals, o_evals[:nq]), nq


def test_many_tasks(song, oracle):
    """More than 32768 (query, probe) pairs: two warps a task."""
    from song_gb300 import datasets as D
    data = D.mixture("byte", 2000, 64, 12, seed=1, center_seed=2)
    q = D.mixture("byte", 8200, 64, 12, seed=3, center_seed=2)
    graph = song.graph_build(data, 0, 4, 7, 15, 60, batch_div=16)
    ox = oracle.OracleIndex(data, graph, 4, 0)
    ent = np.random.default_rng(4).choice(2000, 1700, replace=False).astype(np.uint64)
    starts = ox.nearest_entry_2level(q, ent, 300, 4, 4)
    o_ids, _, _, _ = ox.kernel_search_from(q, starts, 10, oracle.MODE_LEX)
    with song.Index(graph, data, 4, 0) as ix:
        ix.set_entries(ent, starts=4, coarse=300, probes=4)
        assert np.array_equal(ix.search(q, 10, 10), o_ids)
