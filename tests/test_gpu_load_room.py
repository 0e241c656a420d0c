"""A graph that fits the device without the one that the engine holds is loaded,
and replaces it: the arrays a typed file is sorted in, and a graph of so many
vertices that its 32-bit offsets find no room beside the graph before."""

import contextlib

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

V, OLD = 1000, 60_000_000  # 300 MB held


@pytest.fixture
def engine(tmp_path):
    import knightking_gb300 as kk
    e = kk.WalkEngine(0)
    small = str(tmp_path / "small.edges")
    np.ones((1000, 3), np.uint32).tofile(small)
    e.load_graph(V, small, kind="meta")  # the kernels are on the device from here on
    e.walk("deepwalk", 1000, walk_length=5)
    off = np.full(V + 1, OLD, np.int64)
    off[0] = 0
    e.load_arrays(V, off, np.zeros(OLD, np.uint32), None, np.zeros(OLD, np.uint8))
    yield e
    e.close()


@contextlib.contextmanager
def _room(left):
    """All device memory but about `left` bytes is held."""
    torch = pytest.importorskip("torch")
    torch.cuda.synchronize()
    held = torch.empty(torch.cuda.mem_get_info()[0] - left, dtype=torch.uint8, device="cuda")
    try:
        yield
    finally:
        del held
        torch.cuda.empty_cache()


@pytest.mark.parametrize("room", [100_000_000, 40_000_000])
def test_typed_file(engine, tmp_path, room):
    """room beside the old graph for some of the sort's arrays (260 MB, and 40 MB of graph), or for none."""
    rng = np.random.default_rng(2)
    rec = np.zeros((8_000_000, 3), np.uint32)
    rec[:, 0] = rng.integers(0, V, len(rec))
    rec[:, 1] = rng.integers(0, V, len(rec))
    rec[:, 2] = rng.integers(0, 5, len(rec))
    path = str(tmp_path / "new.edges")
    rec.tofile(path)
    with _room(room):
        engine.load_graph(V, path, kind="meta")
    g = engine.download_graph()
    order = np.argsort(rec[:, 0], kind="stable")
    np.testing.assert_array_equal(g["off"], np.concatenate([[0], np.cumsum(np.bincount(rec[:, 0], minlength=V))]))
    np.testing.assert_array_equal(g["nbr"], rec[order, 1])
    np.testing.assert_array_equal(g["type"], rec[order, 2])


@pytest.mark.parametrize("room", [190_000_000, 170_000_000])
def test_many_vertices(engine, oracle_lib, room):
    """room beside the old graph for the new one's 165 MB, not for 80 MB of 32-bit offsets."""
    v, n = 20_000_000, 1_000_000
    off = np.minimum(np.arange(v + 1, dtype=np.int64), n)
    nbr = np.random.default_rng(3).integers(0, n, n).astype(np.uint32)
    with _room(room):
        engine.load_arrays(v, off, nbr)
    got = engine.walk("deepwalk", 5000, walk_length=20, seed=4)
    prm = oracle_lib.make_params("deepwalk", walker_num=5000, weighted=False, seed=4, walk_length=20)
    lens, verts, _ = oracle_lib.walk(oracle_lib.CSR(v, off, nbr), prm, cap=21)
    np.testing.assert_array_equal(got.path_length, lens)
    np.testing.assert_array_equal(got.vertices, verts)
