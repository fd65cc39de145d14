"""The graph builder's repeated searches: only those that say so are run again,
by the kernel that can finish them.  Graphs equal the CPU builder's."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("visited_log2", [6, 9])
@pytest.mark.parametrize("batch_div", [2, 32])
def test_visited_sets_that_fill(song, visited_log2, batch_div):
    """Sets of 64 and 512 slots: a block's set is left for a warp's, which
    grows; some searches also meet too many equal distances for the one list."""
    # corners of a cube: hundreds of equal distances at the list's end
    data = np.random.default_rng(visited_log2).integers(0, 2, (2500, 16)).astype(np.float32)
    args = (data, "l2", 5, 15, 31, 150)
    want = song.graph_build(*args, batch_div=batch_div)
    song.debug_build(visited_log2)
    got = song.graph_build_gpu(*args, batch_div=batch_div)
    block, warp, steps = song.debug_build()
    assert np.array_equal(got, want)
    assert block + warp >= 2500 and warp > 0 and steps > 0


def test_step_by_step_searches_that_fill(song):
    """A budget beyond the one list's: visited sets and queues grow."""
    data = np.random.default_rng(1).integers(0, 30, (2000, 6)).astype(np.float32)
    args = (data, "l2", 5, 15, 31, 200)
    song.debug_build(6)
    got = song.graph_build_gpu(*args, batch_div=16)
    block, warp, steps = song.debug_build()
    assert np.array_equal(got, song.graph_build(*args, batch_div=16))
    assert block == warp == 0 and steps > 2000


def test_only_what_cannot_be_finished_is_repeated(song):
    """A fifth of the vertices are corners of a cube, where searches meet more
    equal distances than the one list holds; the others are far from it."""
    rng = np.random.default_rng(1)
    data = (100 + rng.standard_normal((6000, 24))).astype(np.float32)
    data[::5] = rng.integers(0, 2, (1200, 24))
    args = (data, "l2", 5, 15, 31, 150)
    want = song.graph_build(*args, batch_div=16)
    song.debug_build()
    got = song.graph_build_gpu(*args, batch_div=16)
    block, warp, steps = song.debug_build()
    assert np.array_equal(got, want)
    assert block + warp == 6000 and 0 < steps < 1200, (block, warp, steps)


def test_searches_that_all_need_steps_go_there_at_once(song):
    """Corners alone: most batches are searched step by step without the one
    list's attempt."""
    data = np.random.default_rng(3).integers(0, 2, (6000, 24)).astype(np.float32)
    args = (data, "l2", 5, 15, 31, 150)
    want = song.graph_build(*args, batch_div=16)
    song.debug_build()
    got = song.graph_build_gpu(*args, batch_div=16)
    block, warp, steps = song.debug_build()
    assert np.array_equal(got, want)
    assert steps > 3000 and block + warp < 3000, (block, warp, steps)
