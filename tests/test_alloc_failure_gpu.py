"""Every allocation of a search that fails is reported as out of memory, and the
index searches on afterwards."""
import numpy as np
import pytest

from conftest import load_golden

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind,allocations", [("plain", 2), ("flat", 4), ("two_level", 5)])
def test_first_search(song, kind, allocations):
    """Queries, ids, starts, the choice's lists (of the flat choice: when a few
    queries meet many entries) and the heads' bounds."""
    g = load_golden("l2_s5_d32")
    q = np.tile(g["queries"], (1 + 4000 // len(g["queries"]), 1))
    if kind == "flat":
        q = q[:40]
    ent = np.arange(0, len(g["data"]), 3, dtype=np.uint64)

    def index():
        ix = song.Index(g["graph"], g["data"], int(g["shift"]), int(g["metric"]))
        if kind == "flat":
            ix.set_entries(ent, starts=2)
        if kind == "two_level":
            ix.set_entries(ent, starts=2, coarse=40, probes=4)
        return ix

    with index() as ix:
        want = ix.search(q, 20, 10)
    for n in range(1, allocations + 1):
        with index() as ix:
            song.debug_fail_alloc(n)
            try:
                with pytest.raises(song.SongError) as e:
                    ix.search(q, 20, 10)
            finally:
                song.debug_fail_alloc(0)
            assert e.value.status == song.SONG_ERR_OOM, n
            assert np.array_equal(ix.search(q, 20, 10), want), n
    with index() as ix:  # and there is no further one
        song.debug_fail_alloc(allocations + 1)
        try:
            assert np.array_equal(ix.search(q, 20, 10), want)
        finally:
            song.debug_fail_alloc(0)
