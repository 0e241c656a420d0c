"""Host CSRs checked and sorted on the device: the adjacency sort (by rank, in
shared memory, by segments) against a stable host sort, at the edges of its row
classes and with duplicate neighbours, for every combination of weights and
types; a graph whose rows are sorted but for one; refused graphs leave the
engine's graph as it was."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

DEGREES = [0, 1, 2, 31, 32, 33, 128, 129, 255, 256, 257, 512, 1024, 2047, 2048, 2049, 5000, 0, 3]


@pytest.fixture(scope="module")
def engine():
    import knightking_gb300 as kk
    e = kk.WalkEngine(0)
    yield e
    e.close()


def _csr(degrees, V, weighted, types, rng):
    off = np.zeros(V + 1, np.int64)
    off[1:len(degrees) + 1] = np.cumsum(degrees)
    off[len(degrees) + 1:] = off[len(degrees)]
    E = int(off[-1])
    nbr = rng.integers(0, V, E).astype(np.uint32)  # duplicates among them
    w = rng.random(E).astype(np.float32) if weighted else None
    t = rng.integers(0, 8, E).astype(np.uint8) if types else None
    return off, nbr, w, t


def _sorted(off, nbr, w, t):
    row = np.repeat(np.arange(len(off) - 1), np.diff(off))
    order = np.lexsort((np.arange(len(nbr)), nbr, row))
    return nbr[order], None if w is None else w[order], None if t is None else t[order]


def _same(engine, off, nbr, w, t):
    g = engine.download_graph()
    np.testing.assert_array_equal(g["off"], off)
    np.testing.assert_array_equal(g["nbr"], nbr)
    for a, b in ((g["w"], w), (g["type"], t)):
        assert (a is None) == (b is None)
        if b is not None:
            np.testing.assert_array_equal(a, b)


@pytest.mark.parametrize("weighted,types", [(False, False), (True, False), (False, True), (True, True)])
@pytest.mark.parametrize("degrees,V", [(DEGREES, 3000), ([4], 9), ([0, 0], 2), ([40000, 17], 41000)])
def test_sort(engine, degrees, V, weighted, types):
    off, nbr, w, t = _csr(degrees, V, weighted, types, np.random.default_rng(len(degrees)))
    engine.load_arrays(V, off, nbr, w, t)
    _same(engine, off, nbr, w, t)
    engine.sort_adjacency()
    _same(engine, off, *_sorted(off, nbr, w, t))


def test_one_row_out_of_order(engine):
    """Descents between rows are none within them: only the last row's counts."""
    off = np.array([0, 3, 3, 5, 8], np.int64)
    for last in ([1, 2, 3], [2, 1, 3]):
        nbr = np.array([1, 2, 3, 0, 2] + last, np.uint32)
        engine.load_arrays(4, off, nbr)
        engine.sort_adjacency()
        _same(engine, off, np.array([1, 2, 3, 0, 2, 1, 2, 3], np.uint32), None, None)


@pytest.mark.parametrize("what", ["neighbour", "offsets", "ends", "type"])
def test_refused_graphs(engine, what):
    import knightking_gb300 as kk
    off, nbr, w, t = _csr([5, 0, 700, 3], 900, True, True, np.random.default_rng(3))
    engine.load_arrays(900, off, nbr, w, t)
    bad = [off.copy(), nbr.copy(), w, t.copy()]
    if what == "neighbour":
        bad[1][-1] = 900
    elif what == "offsets":
        bad[0][2] = 800  # beyond the next offset and the edges
    elif what == "ends":
        bad[0][-1] -= 1
        bad[0][4:-1] = bad[0][-1]
        bad[0][0] = 1
    else:
        bad[3][0] = 8
    with pytest.raises(kk.KKError):
        engine.load_arrays(900, *bad)
    _same(engine, off, nbr, w, t)
    assert engine.walk("deepwalk", 900, walk_length=4, weighted=True).total_steps > 0
