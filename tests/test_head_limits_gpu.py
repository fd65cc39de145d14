"""The head phase's shortlist where its bounds are not finite: norms that
overflow FP32 while the distances themselves do not (or overflow for a part of
the heads), and NaN queries.  100 heads leave four unused places in a row of
bounds; none of them may be taken.  Starts equal the oracle's.  And the route
that a batch takes: by its size, or the one it is told to take."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _case(song, metric, x_norms, q_norms, dim=64, n=1500, nq=1100):
    """Directions around a few centres, so that some distances are small
    against the norms; graph of the directions."""
    rng = np.random.default_rng(metric)
    centers = rng.standard_normal((8, dim))
    x = centers[rng.integers(0, 8, n)] + 0.3 * rng.standard_normal((n, dim))
    q = centers[rng.integers(0, 8, nq)] + 0.3 * rng.standard_normal((nq, dim))
    x /= np.linalg.norm(x, axis=1)[:, None]
    q /= np.linalg.norm(q, axis=1)[:, None]
    graph = song.graph_build(x.astype(np.float32), metric, 4, 7, 15, 60, batch_div=16)
    x *= rng.uniform(*x_norms, n)[:, None]
    q *= rng.uniform(*q_norms, nq)[:, None]
    return x.astype(np.float32), q.astype(np.float32), graph


# squared norms above 3.4e38 overflow: those of the queries, then those of about half of the rows
@pytest.mark.parametrize("metric,x_norms,q_norms", [
    (0, (3e18, 5e18), (1.9e19, 2.1e19)),
    (1, (5e17, 1e18), (1.9e19, 2.1e19)),
    (2, (0.5e-2, 1e-2), (1.9e19, 2.1e19)),
    (0, (1.7e19, 2.0e19), (1.75e19, 1.83e19)),
])
def test_norms_that_overflow(song, oracle, metric, x_norms, q_norms):
    x, q, graph = _case(song, metric, x_norms, q_norms)
    ox = oracle.OracleIndex(x, graph, 4, metric)
    ent = np.random.default_rng(5).choice(len(x), 700, replace=False).astype(np.uint64)
    with song.Index(graph, x, 4, metric) as ix:
        for probes, ns in ((1, 1), (2, 2), (4, 3)):
            starts = ox.nearest_entry_2level(q, ent, 100, probes, ns)
            o_ids, o_hops, o_evals, _ = ox.kernel_search_from(q, starts, 20, oracle.MODE_LEX)
            ix.set_entries(ent, starts=ns, coarse=100, probes=probes)
            ix.debug_head_stats(True)
            ids, hops, evals = ix.search(q, 20, 20, stats=True)
            assert ix.debug_head_stats(False)[0] == len(q)  # the tensor cores' route
            assert np.array_equal(ids, o_ids), (probes, ns)
            assert np.array_equal(hops, o_hops) and np.array_equal(evals, o_evals), (probes, ns)


@pytest.mark.parametrize("metric", [0, 1, 2])
def test_nan_queries(song, metric):
    x, q, graph = _case(song, metric, (0.5, 2.0), (0.5, 2.0))
    bad = np.arange(3, len(q), 50)
    q[bad, 7] = np.nan
    ent = np.random.default_rng(5).choice(len(x), 700, replace=False).astype(np.uint64)
    with song.Index(graph, x, 4, metric) as ix:
        ix.set_entries(ent, starts=1, coarse=100, probes=2)
        ix.debug_head_stats(True)
        ids = ix.search(q, 20, 20)
        assert ix.debug_head_stats(False)[0] == len(q)
        few = ix.search(q[:60], 20, 20)  # the two-kernel choice of small batches
        ix.set_entries(None)
        plain = ix.search(q[bad], 20, 20)
    assert np.array_equal(ids[:60], few)
    assert np.array_equal(ids[bad], plain)  # they start at vertex 0


def test_route_of_a_batch(song, oracle):
    x, q, graph = _case(song, 0, (0.5, 2.0), (0.5, 2.0))
    ox = oracle.OracleIndex(x, graph, 4, 0)
    ent = np.random.default_rng(5).choice(len(x), 700, replace=False).astype(np.uint64)
    o_ids = ox.kernel_search_from(q, ox.nearest_entry_2level(q, ent, 100, 3, 2), 20, oracle.MODE_LEX)[0]
    with song.Index(graph, x, 4, 0) as ix:
        ix.set_entries(ent, starts=2, coarse=100, probes=3)
        ix.debug_head_stats(True)
        for path, counted in ((None, 0), (True, 10), (False, 0), (None, 0)):
            assert ix.debug_head_path(path)
            assert np.array_equal(ix.search(q[:10], 20, 20), o_ids[:10])
            assert ix.debug_head_stats(True)[0] == counted, path
            assert np.array_equal(ix.search(q, 20, 20), o_ids)
            assert ix.debug_head_stats(True)[0] == (0 if path is False else len(q)), path
