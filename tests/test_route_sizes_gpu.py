"""Kernels and routes that a size or a metric selects, where the tests of each
part do not reach them: the kernels of long rows for inner product and cosine,
and the line between the two entry choices that the product of queries, heads
and dimensions draws."""
import numpy as np
import pytest

from test_search_shapes_gpu import _check, _clustered, _ring_graph

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("metric", [1, 2])
@pytest.mark.parametrize("dim,storage", [(253, "f32"), (300, "f32"), (505, "bf16"), (612, "bf16")])
def test_long_rows_of_every_metric(song, oracle, dim, storage, metric):
    """From 1 KB a row on: plain, multi-probe and learned kernels."""
    data, q = _clustered(900, dim, seed=dim)
    g = _ring_graph(song, data, metric, 4, seed=dim)
    with song.Index(g, data, 4, metric, storage=storage) as ix:
        ix.set_rerank(0)
        ox = oracle.OracleIndex(song.dequantize_rows(ix.rows(), storage, dim), g, 4, metric)
        for pq in (20, 50, 140, 270, 520):
            _check(ix, q, pq, ox.kernel_search(q, pq, oracle.MODE_LEX), pq)
        if storage == "f32":
            for pq in (20, 50):
                ix.set_multiprobe(2, 1, True)
                want = ox.kernel_search(q, pq, oracle.MODE_LEX, probes=2, finish_cnt=1, double_check=True)
                _check(ix, q, pq, want, ("multi", pq))
            ix.set_multiprobe()
        ix.set_hop_limit(1 << 30)
        for pq in (20, 50, 140):
            _check(ix, q, pq, ox.kernel_search(q, pq, oracle.MODE_LEX_EXACT), ("learned", pq))


def test_products_that_end_the_small_batches(song, oracle):
    """2^29 products: 512 queries x 2048 heads x 512 dimensions still take the
    two-kernel choice, 516 dimensions do not."""
    for dim, nq, tensor in ((512, 512, False), (516, 512, True), (516, 500, False)):
        rng = np.random.default_rng(dim)
        data = rng.standard_normal((2300, dim)).astype(np.float32)
        q = rng.standard_normal((nq, dim)).astype(np.float32)
        g = np.zeros((2300, 16), dtype=np.uint64)
        g[:, 0] = 15
        g[:, 1:] = rng.integers(0, 2300, (2300, 15))
        ent = rng.permutation(2300)[:2200].astype(np.uint64)
        ox = oracle.OracleIndex(data, g, 4, 0)
        o_ids = ox.kernel_search_from(q, ox.nearest_entry_2level(q, ent, 2048, 3, 2), 10, oracle.MODE_LEX)[0]
        with song.Index(g, data, 4, 0) as ix:
            ix.set_entries(ent, starts=2, coarse=2048, probes=3)
            ix.debug_head_stats(True)
            assert np.array_equal(ix.search(q, 10, 10), o_ids), (dim, nq)
            assert (ix.debug_head_stats(False)[0] > 0) == tensor, (dim, nq)
