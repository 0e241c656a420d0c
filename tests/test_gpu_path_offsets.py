"""Path offsets of fixed-length walks, computed in one launch up to 65535
walkers (blocks of 16384) and by a scan from there on, with starts that are
isolated; and kk_walk's paths on both sides of the 8 MB of vertices up to
which they follow the walk into the result's block: lengths, offsets and paths
are the oracle's."""

import numpy as np
import pytest

from oracle import graphs as G

pytestmark = pytest.mark.gpu

V = 700  # vertices 600.. are isolated


@pytest.fixture(scope="module")
def loaded():
    import knightking_gb300 as kk
    g = G.random_undirected(600, 7000, seed=8, weight="unif")
    csr = G.csr_file_order(V, g["src"], g["dst"], w=g.get("w"))
    e = kk.WalkEngine(0)
    e.load_arrays(V, csr["off"], csr["nbr"], csr.get("w"))
    yield e, csr
    e.close()


@pytest.mark.parametrize("starts", [None, 1, 37])
@pytest.mark.parametrize("app,n,length", [
    ("deepwalk", 1, 3), ("deepwalk", 1023, 5), ("deepwalk", 16383, 1), ("deepwalk", 16384, 4), ("deepwalk", 16385, 4),
    ("deepwalk", 65535, 2), ("deepwalk", 65536, 2), ("deepwalk", 70001, 0), ("deepwalk", 40000, 103),
    ("deepwalk", 2097152 // 64, 63), ("deepwalk", 2097152 // 64 + 1, 63), ("node2vec", 33000, 7),
    ("node2vec", 65537, 70)])
def test_path_offsets(loaded, oracle_lib, app, n, length, starts):
    e, csr = loaded
    kw = dict(walk_length=length, seed=n + length, walker_begin=3)
    if app == "node2vec":
        kw.update(p=0.5, q=2.0)
    if starts:
        kw["start"] = np.random.default_rng(starts).integers(0, V, starts).astype(np.uint32)
    got = e.walk(app, n, weighted=True, **kw)
    ids = 3 + np.arange(n)
    first = ids % V if not starts else kw["start"][ids % starts]
    lens = np.where(np.diff(csr["off"].astype(np.int64))[first] > 0, length + 1, 1)
    np.testing.assert_array_equal(got.path_length, lens)
    np.testing.assert_array_equal(got.offset, np.cumsum(lens) - lens)
    assert len(got.vertices) == lens.sum() and got.total_steps == lens.sum() - n
    np.testing.assert_array_equal(got.vertices[got.offset.astype(np.int64)], first)
    if starts:
        return
    ocsr = oracle_lib.CSR(V, csr["off"], csr["nbr"], csr.get("w"))
    prm = oracle_lib.make_params(app, walker_num=n, weighted=True, **kw)
    olens, verts, _ = oracle_lib.walk(ocsr.sorted_copy() if app == "node2vec" else ocsr, prm, cap=length + 1)
    np.testing.assert_array_equal(got.path_length, olens)
    np.testing.assert_array_equal(got.vertices, verts)


def test_refused_start_then_walk(loaded):
    import knightking_gb300 as kk
    e, _ = loaded
    a = e.walk("deepwalk", 3000, walk_length=9, seed=2, weighted=True)
    with pytest.raises(kk.KKError):
        e.walk("deepwalk", 3000, walk_length=9, seed=2, weighted=True, start=np.array([0, V], np.uint32))
    b = e.walk("deepwalk", 3000, walk_length=9, seed=2, weighted=True)
    np.testing.assert_array_equal(a.vertices, b.vertices)
