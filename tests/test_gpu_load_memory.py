"""Device memory of graph loads: a refused graph leaves none of its own behind,
whether there was room for it or not, and the engine's graph is as it was."""

import contextlib

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

V, E = 100, 300_000_000  # 1.2 GB of neighbours


@pytest.fixture
def engine():
    import knightking_gb300 as kk
    e = kk.WalkEngine(0)
    rng = np.random.default_rng(1)
    e.load_arrays(V, np.arange(V + 1, dtype=np.int64) * 5, rng.integers(0, V, 5 * V).astype(np.uint32),
                  rng.random(5 * V, dtype=np.float32))
    e.walk("deepwalk", 1000, walk_length=5, weighted=True)
    yield e
    e.close()


def _free():
    torch = pytest.importorskip("torch")
    torch.cuda.synchronize()
    return torch.cuda.mem_get_info()[0]


@contextlib.contextmanager
def _room(left):
    """All device memory but about `left` bytes is held."""
    torch = pytest.importorskip("torch")
    held = torch.empty(_free() - left, dtype=torch.uint8, device="cuda") if left else None
    try:
        yield
    finally:
        del held
        torch.cuda.empty_cache()


@pytest.mark.parametrize("room", [None, 2_000_000_000])
def test_refused_arrays(engine, room):
    """room: for the neighbours beside the engine's graph, not for the weights."""
    import knightking_gb300 as kk
    before = engine.download_graph(), engine.walk("deepwalk", 1000, walk_length=5, weighted=True).vertices.copy()
    off = np.full(V + 1, E, np.int64)
    off[0] = 0
    nbr = np.zeros(E, np.uint32)
    nbr[-1] = V
    w = np.zeros(E, np.float32) if room else None
    with _room(room):
        free = _free()
        with pytest.raises(kk.KKError, match="neighbour id out of range"):
            engine.load_arrays(V, off, nbr, w)
        left = free - _free()
    assert left < 64 << 20, left
    after = engine.download_graph(), engine.walk("deepwalk", 1000, walk_length=5, weighted=True).vertices
    np.testing.assert_array_equal(before[0]["nbr"], after[0]["nbr"])
    np.testing.assert_array_equal(before[1], after[1])


def test_refused_file(engine, tmp_path):
    import knightking_gb300 as kk
    before = engine.walk("deepwalk", 1000, walk_length=5, weighted=True).vertices.copy()
    path = str(tmp_path / "bad.edges")
    with open(path, "wb") as f:
        f.truncate(400_000_000 - 8)  # 50 M edges 0 -> 0: 1.6 GB to sort them in
        f.seek(0, 2)
        f.write(np.array([0, V], np.uint32).tobytes())
    engine.walk("deepwalk", 1000, walk_length=5)
    free = _free()
    with pytest.raises(kk.KKError, match="edge endpoint"):
        engine.load_graph(V, path, kind="unweighted")
    assert free - _free() < 64 << 20, free - _free()
    np.testing.assert_array_equal(before, engine.walk("deepwalk", 1000, walk_length=5, weighted=True).vertices)
