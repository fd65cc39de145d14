"""Sizes at the limit of a block's shared memory: every one that the interface
accepts runs."""
import numpy as np
import pytest

LIMIT = 227 * 1024
PQS = [2, 3, 31, 32, 62, 63, 64, 126, 127, 254, 255, 256, 510, 511, 512, 1000, 1022, 1023]


@pytest.mark.parametrize("storage,learned,multi", [("f32", 0, 0), ("f32", 1, 0), ("f32", 0, 1), ("bf16", 0, 0),
                                                   ("bf16", 1, 0), ("fp8", 0, 0), ("bits", 0, 0)])
def test_accepted_sizes_fit_a_block(song, storage, learned, multi):
    for pq in PQS:
        def accepted(dim):
            return song.debug_shared_bytes(storage, dim, pq, learned, multi)[0] <= LIMIT
        lo, hi = 1, 65536  # the largest accepted dimension
        while lo < hi:
            mid = (lo + hi + 1) // 2
            lo, hi = (mid, hi) if accepted(mid) else (lo, mid - 1)
        assert accepted(lo)
        for dim in list(range(max(1, lo - 300), lo + 1)) + list(range(1, lo, 97)):
            by, used = song.debug_shared_bytes(storage, dim, pq, learned, multi)
            assert by <= LIMIT and used <= LIMIT, (pq, dim, by, used)


@pytest.mark.gpu
@pytest.mark.parametrize("dim,pq", [(50060, 1000), (50000, 1000), (53964, 512), (55964, 256), (57996, 2), (57921, 2),
                                    (33, 300), (16, 40)])
def test_codes_of_very_wide_vectors(song, oracle, dim, pq):
    """Bit codes leave nearly all of a warp's shared memory to the query."""
    rng = np.random.default_rng(dim + pq)
    data = rng.standard_normal((300, dim), dtype=np.float32)
    q = data[:5] + 0.5 * rng.standard_normal((5, dim), dtype=np.float32)
    g = np.zeros((300, 16), dtype=np.uint64)
    g[:, 0] = 15
    g[:, 1:] = rng.integers(0, 300, (300, 15))
    planes = song.hash_planes(dim, seed=5)
    ox = oracle.OracleIndex(oracle.hash_codes(data, planes).view(np.float32), g, 4, oracle.HAMMING)
    o_ids, o_hops, o_evals, _ = ox.kernel_search(oracle.hash_codes(q, planes).view(np.float32), pq, oracle.MODE_LEX)
    with song.Index(g, data, 4, 0, storage="bits") as ix:
        ix.set_hash_planes(planes)
        ix.set_rerank(0)
        ids, hops, evals = ix.search(q, pq, pq, stats=True)
        assert np.array_equal(ids, o_ids)
        assert np.array_equal(hops, o_hops) and np.array_equal(evals, o_evals)
        ix.set_rerank(-1)
        rr = ix.search(q, pq, min(pq, 40))
    for i, row in enumerate(o_ids):
        row = row[row != oracle.NO_ID]
        d = [oracle.kernel_distance(0, q[i], data[v]) for v in row]
        order = sorted(range(len(row)), key=lambda j: (d[j], int(row[j])))[:rr.shape[1]]
        assert list(rr[i][:len(order)]) == [row[j] for j in order], i
