"""A binary edge file's CSR out of the sorted records, four a thread (remainders
of four, sources with no edges before, between and after the others), and the
search for dead ends by a bit a vertex (vertex counts about a word of bits, one
dead vertex at either end of it): graphs and walks are the oracle's."""

import numpy as np
import pytest

from oracle import graphs as G

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def engine():
    import knightking_gb300 as kk
    e = kk.WalkEngine(0)
    yield e
    e.close()


@pytest.mark.parametrize("weighted", [True, False])
@pytest.mark.parametrize("V,n", [(1, 1), (5, 2), (7, 3), (40, 4), (3000, 5), (3000, 4097), (100, 4098), (64, 4099)])
def test_csr_from_file(engine, tmp_path, V, n, weighted):
    rng = np.random.default_rng(V + n)
    lo, hi = V // 4, max(V // 4 + 1, V - V // 4)  # no edges at either end
    g = {"V": V, "src": rng.integers(lo, hi, n).astype(np.uint32), "dst": rng.integers(0, V, n).astype(np.uint32)}
    if weighted:
        g["w"] = rng.random(n, dtype=np.float32)
    f = tmp_path / "e.bin"
    kind = "f32" if weighted else "unweighted"
    G.write_edge_file(f, g, "f32" if weighted else "none")
    engine.load_graph(V, f, kind=kind)
    got, want = engine.download_graph(), G.csr_file_order(V, g["src"], g["dst"], w=g.get("w"))
    np.testing.assert_array_equal(got["off"], want["off"])
    np.testing.assert_array_equal(got["nbr"], want["nbr"])
    if weighted:
        np.testing.assert_array_equal(got["w"], want["w"])


@pytest.mark.parametrize("V", [31, 32, 33, 64, 1000])
@pytest.mark.parametrize("dead", [None, "isolated", 0, -1])
def test_dead_ends(engine, oracle_lib, V, dead):
    """dead: none, an isolated vertex only, or the edges into the first or last vertex lead nowhere."""
    rng = np.random.default_rng(V)
    ring = np.arange(V, dtype=np.uint32)
    src = np.concatenate([ring, rng.integers(0, V, 6 * V).astype(np.uint32)])
    dst = np.concatenate([np.roll(ring, 1), rng.integers(0, V, 6 * V).astype(np.uint32)])
    if dead == "isolated":
        keep = (src != V // 2) & (dst != V // 2)
        src, dst = src[keep], dst[keep]
    elif dead is not None:
        keep = src != ring[dead]
        src, dst = src[keep], dst[keep]
    csr = G.csr_file_order(V, src, dst)
    engine.load_arrays(V, csr["off"], csr["nbr"])
    got = engine.walk("deepwalk", 4000, weighted=False, walk_length=30, seed=3)
    prm = oracle_lib.make_params("deepwalk", walker_num=4000, weighted=False, walk_length=30, seed=3)
    lens, verts, steps = oracle_lib.walk(oracle_lib.CSR(V, csr["off"], csr["nbr"], None), prm, cap=31)
    assert got.total_steps == steps
    np.testing.assert_array_equal(got.path_length, lens)
    np.testing.assert_array_equal(got.vertices, verts)
