"""The search kernel at the sizes where its structures change: queue bounds at
the ends of each queue segment and of the two queue kinds, row widths at the
remainders of the gather (every format), and ids laid out so that the visited
hash has long runs (consecutive ids hash to neighbouring slots) across its
end.  Bit-exact against the oracle (ids, hops, evaluations), in a small batch
(a block per query) and in one of some thousand queries (a warp per query)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _clustered(n, dim, seed, nq=24):
    """Vectors sorted along a curve, so that neighbours have neighbouring ids."""
    rng = np.random.default_rng(seed)
    t = np.sort(rng.uniform(0, 40, n))
    q = rng.uniform(0, 40, nq)
    phase, freq = rng.uniform(0, 6, dim), rng.uniform(0.2, 1.0, dim)

    def at(u):
        return np.sin(u[:, None] * freq + phase) + 0.3
    return ((at(t) + 0.05 * rng.standard_normal((n, dim))).astype(np.float32),
            (at(q) + 0.05 * rng.standard_normal((nq, dim))).astype(np.float32))


def _ring_graph(song, data, metric, shift, seed):
    """Built rows with some long-range neighbours in their last places."""
    fixed = (1 << shift) - 1
    g = song.graph_build(data, metric, shift, max(1, fixed // 2), fixed, 60, batch_div=16).reshape(len(data), -1)
    rng = np.random.default_rng(seed)
    deg = g[:, 0].astype(int)
    for v in np.nonzero(deg > 2)[0]:
        g[v, deg[v]] = rng.integers(len(data))
    return g


def _check(ix, q, pq, oracle_result, what):
    o_ids, o_hops, o_evals, _ = oracle_result
    for reps in (1, 100):
        ids, hops, evals = ix.search(np.tile(q, (reps, 1)), pq, pq, stats=True)
        assert np.array_equal(ids, np.tile(o_ids, (reps, 1))), (what, reps)
        assert np.array_equal(hops, np.tile(o_hops, reps)), (what, reps)
        assert np.array_equal(evals, np.tile(o_evals, reps)), (what, reps)


PQS = [2, 3, 30, 31, 32, 62, 63, 64, 126, 127, 128, 254, 255, 256, 510, 511, 512, 1022, 1023]


@pytest.mark.parametrize("metric", [0, 1, 2])
@pytest.mark.parametrize("shift", [1, 3, 5])
def test_queue_bounds(song, oracle, metric, shift):
    data, q = _clustered(2500, 16, seed=shift)
    g = _ring_graph(song, data, metric, shift, seed=shift)
    ox = oracle.OracleIndex(data, g, shift, metric)
    with song.Index(g, data, shift, metric) as ix:
        for pq in PQS:
            want = ox.kernel_search(q, pq, oracle.MODE_LEX)
            _check(ix, q, pq, want, pq)
            o_ids = want[0]
            for k in (1, min(pq, 32), min(pq, 33)):
                assert np.array_equal(ix.search(q, pq, k), o_ids[:, :k]), "pq %d k %d" % (pq, k)


@pytest.mark.parametrize("dim", [1, 4, 5, 31, 32, 33, 63, 124, 127, 128, 129, 200, 255, 256, 260, 500])
def test_row_widths(song, oracle, dim):
    data, q = _clustered(900, dim, seed=dim)
    for metric in (0, 1, 2):
        g = _ring_graph(song, data, metric, 5, seed=dim)
        for storage in ("f32", "bf16", "fp8"):
            with song.Index(g, data, 5, metric, storage=storage) as ix:
                ix.set_rerank(0)
                ox = oracle.OracleIndex(song.dequantize_rows(ix.rows(), storage, dim), g, 5, metric)
                _check(ix, q, 40, ox.kernel_search(q, 40, oracle.MODE_LEX), (metric, storage))


@pytest.mark.parametrize("pq", [10, 40, 100, 200, 300, 600])
def test_multi_probe_and_learned_batches(song, oracle, pq):
    """The multi-probe and the learned kernels with a block and with a warp
    per query (the latter with an exit that never fires: the exact visited
    set's search)."""
    data, q = _clustered(2500, 16, seed=7)
    g = _ring_graph(song, data, 0, 5, seed=7)
    ox = oracle.OracleIndex(data, g, 5, 0)
    with song.Index(g, data, 5, 0) as ix:
        for probes, cnt, dc in ((4, 1, False), (2, 2, True)):
            ix.set_multiprobe(probes, cnt, dc)
            want = ox.kernel_search(q, pq, oracle.MODE_LEX, probes=probes, finish_cnt=cnt, double_check=dc)
            _check(ix, q, pq, want, (probes, cnt, dc))
        ix.set_multiprobe()
        ix.set_hop_limit(1 << 30)
        _check(ix, q, pq, ox.kernel_search(q, pq, oracle.MODE_LEX_EXACT), "learned")


@pytest.mark.parametrize("dim", [252, 253, 256, 288, 508, 512, 516, 961])
def test_long_rows(song, oracle, dim):
    """Rows around 1 KB and longer, where another instance of each kernel
    reads them: FP32 from 253 dimensions, BF16 from 505."""
    data, q = _clustered(900, dim, seed=dim)
    g = _ring_graph(song, data, 0, 4, seed=dim)
    for storage in ("f32", "bf16"):
        with song.Index(g, data, 4, 0, storage=storage) as ix:
            ix.set_rerank(0)
            ox = oracle.OracleIndex(song.dequantize_rows(ix.rows(), storage, dim), g, 4, 0)
            for pq in (20, 140, 270, 520):
                _check(ix, q, pq, ox.kernel_search(q, pq, oracle.MODE_LEX), (storage, pq))
            if storage == "f32":
                ix.set_multiprobe(2, 1, True)
                want = ox.kernel_search(q, 50, oracle.MODE_LEX, probes=2, finish_cnt=1, double_check=True)
                _check(ix, q, 50, want, "multi")
                ix.set_multiprobe()
            ix.set_hop_limit(1 << 30)
            _check(ix, q, 50, ox.kernel_search(q, 50, oracle.MODE_LEX_EXACT), (storage, "learned"))
