"""alias_hub_grid sets the blocks that build the hubs' alias tables, with one
launch for the other rows and with a launch a class: on one block sixteen hubs
are built one after another, and the tables are the same."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("one_launch", [1, 0])
def test_hub_grid(one_launch):
    import knightking_gb300 as kk
    hubs, deg = 16, 20000
    rng = np.random.default_rng(5)
    off = np.minimum(np.arange(deg + 1, dtype=np.int64), hubs) * deg
    nbr = np.tile(np.arange(deg, dtype=np.uint32), hubs)
    w = np.exp(rng.normal(size=hubs * deg)).astype(np.float32)
    e = kk.WalkEngine(0)
    e.load_arrays(deg, off, nbr, w)
    e.set_option("alias_one_launch", one_launch)
    ms, tables = [], []
    for grid in (0, 1):
        e.set_option("alias_hub_grid", grid)
        best = 1e9
        for _ in range(8):
            e.walk_device("deepwalk", 32, paths=False, walk_length=1, weighted=True)
            best = min(best, e.last_timing()[0])
        ms.append(best)
        tables.append(e.alias_tables())
    e.close()
    assert ms[1] > 3 * ms[0], ms  # sixteen rows in turn against one
    for a, b in zip(*tables):
        np.testing.assert_array_equal(a.view(np.uint32), b.view(np.uint32))
