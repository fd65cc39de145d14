"""The flat entry choice at the sizes where its two kernels change over and at
the edges of their tiles: few and many entries and queries, rows at the
remainders up to and past 1 KB, every list length.  Starts (through the searches
they seed) equal the oracle's."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _random_graph(n, rng):
    g = np.zeros((n, 16), dtype=np.uint64)
    g[:, 0] = 15
    g[:, 1:] = rng.integers(0, n, (n, 15))
    return g


@pytest.mark.parametrize("metric", [0, 1, 2])
@pytest.mark.parametrize("dim", [1, 4, 15, 33, 64, 130, 253, 260])
def test_starts_equal_the_oracles(song, oracle, dim, metric):
    rng = np.random.default_rng(dim + 300 * metric)
    n = 1500
    data = rng.standard_normal((n, dim)).astype(np.float32)
    data[n // 2:] = data[:n - n // 2]  # equal distances: the smaller id
    q = rng.standard_normal((4200, dim)).astype(np.float32)
    g = _random_graph(n, rng)
    ox = oracle.OracleIndex(data, g, 4, metric)
    with song.Index(g, data, 4, metric) as ix:
        for entries, ns in ((1, 1), (8, 8), (31, 2), (33, 1), (64, 4), (300, 3), (1100, 1), (1100, 8)):
            ent = np.sort(rng.permutation(n)[:entries]).astype(np.uint64)
            o_ids, o_hops, _, _ = ox.kernel_search_from(q, ox.nearest_entry(q, ent, ns=ns), 8, oracle.MODE_LEX)
            ix.set_entries(ent, starts=ns)
            for nq in (1, 4, 5, 63, 1000, 4200):
                ids, hops, _ = ix.search(q[:nq], 8, 8, stats=True)
                assert np.array_equal(ids, o_ids[:nq]) and np.array_equal(hops, o_hops[:nq]), (entries, ns, nq)


@pytest.mark.parametrize("entries", [16, 1100])
def test_nan_queries_start_at_vertex_0(song, entries):
    rng = np.random.default_rng(entries)
    data = rng.standard_normal((1500, 16)).astype(np.float32)
    q = rng.standard_normal((3000, 16)).astype(np.float32)
    q[::7, 3] = np.nan
    with song.Index(_random_graph(1500, rng), data, 4, 0) as ix:
        plain = ix.search(q[::7], 8, 8)
        ix.set_entries(np.sort(rng.permutation(1500)[:entries]).astype(np.uint64), starts=1)
        for nq in (8, 3000):
            assert np.array_equal(ix.search(q[:nq], 8, 8)[::7], plain[:(nq + 6) // 7]), nq
