"""The graph builder's one-list search where it can go wrong: rows at the
remainders of a warp's dimensions and past its registers, many equal distances
at the list's end (the step-by-step search takes over), values whose products
spread over too many binades for the integer sums, budgets at the list's
limit, and batches with a block and with a warp per vertex.  Graphs equal the
CPU builder's."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _data(kind, n, dim, rng):
    if kind == "normal":
        return rng.standard_normal((n, dim)).astype(np.float32)
    if kind == "ties":  # a few values: most distances occur many times, and rows repeat
        return rng.integers(0, 3, (n, dim)).astype(np.float32)
    if kind == "spread":  # products over ~60 binades, some of them zero
        x = rng.standard_normal((n, dim)) * 2.0 ** rng.integers(-15, 16, (n, dim))
        x[rng.random((n, dim)) < 0.1] = 0.0
        return x.astype(np.float32)
    assert kind == "tiny"  # products that are denormal
    return (rng.standard_normal((n, dim)) * 1e-21).astype(np.float32)


@pytest.mark.parametrize("metric", ["l2", "ip", "cos"])
@pytest.mark.parametrize("kind", ["normal", "ties", "spread", "tiny"])
@pytest.mark.parametrize("dim", [1, 3, 33, 128, 257, 300])
def test_equals_cpu_builder(song, metric, kind, dim):
    rng = np.random.default_rng(dim)
    data = _data(kind, 700, dim, rng)
    if metric == "cos" and ((data * data).sum(1) == 0).any():
        pytest.skip("rows of norm zero: their cosine distance is 0 / 0, which has no place in an order")
    args = (data, metric, 4, 7, 15, 60)
    assert np.array_equal(song.graph_build_gpu(*args, batch_div=16), song.graph_build(*args, batch_div=16))


@pytest.mark.parametrize("budget", [7, 31, 32, 191, 192, 193])
def test_budgets(song, budget):
    data = np.random.default_rng(budget).integers(0, 40, (1500, 8)).astype(np.float32)
    args = (data, "l2", 4, 7, 15, budget)
    assert np.array_equal(song.graph_build_gpu(*args, batch_div=32), song.graph_build(*args, batch_div=32))


@pytest.mark.parametrize("batch_div", [1, 2, 64])
def test_batch_sizes(song, batch_div):
    data = np.random.default_rng(9).standard_normal((6000, 20)).astype(np.float32)
    args = (data, "l2", 5, 15, 31, 150)
    assert np.array_equal(song.graph_build_gpu(*args, batch_div=batch_div),
                          song.graph_build(*args, batch_div=batch_div))
