"""DeepWalk and PPR through the kernels of walks whose every trial is accepted,
walker for walker against the oracle: one walker, counts around a block, more
walkers than the SMs hold (lanes take several walkers in turn, paths leave in
tiles of 16), lengths around a tile, dead ends and isolated vertices, and the
32- and 64-bit offsets."""

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


def _graph(kind, weighted):
    if kind == "undirected":
        g = G.random_undirected(300, 4000, seed=3, weight="unif" if weighted else None)
        return G.csr_file_order(310, g["src"], g["dst"], w=g.get("w"))  # ten isolated vertices
    rng = np.random.default_rng(4)
    src, dst = rng.integers(0, 200, 1500), rng.integers(0, 260, 1500)  # 200.. are dead ends
    w = (1.0 + 4.0 * rng.random(1500)).astype(np.float32) if weighted else None
    return G.csr_file_order(260, src.astype(np.uint32), dst.astype(np.uint32), w=w)


@pytest.mark.parametrize("walkers,length", [(1, 1), (1, 16), (33, 0), (65, 15), (5000, 17), (300001, 16), (300001, 17),
                                            (400003, 33)])
@pytest.mark.parametrize("kind,app,weighted,offsets32,cursor",
                         [("undirected", "deepwalk", True, 1, 0), ("undirected", "deepwalk", True, 0, 0),
                          ("directed", "deepwalk", True, 1, 0), ("directed", "deepwalk", False, 1, 0),
                          ("undirected", "deepwalk", False, 1, 1), ("undirected", "ppr", False, 1, 0),
                          ("undirected", "ppr", True, 0, 0), ("directed", "ppr", False, 0, 0)])
def test_straight_walks(engine, oracle_lib, walkers, length, kind, app, weighted, offsets32, cursor):
    csr = _graph(kind, weighted)
    V = len(csr["off"]) - 1
    engine.load_arrays(V, csr["off"], csr["nbr"], csr.get("w"))
    kw = dict(terminate_prob=1.0 / (length + 1.5)) if app == "ppr" else dict(walk_length=length)
    engine.set_option("compact_offsets", offsets32)
    engine.set_option("cursor_adjacency", cursor)
    try:
        got = engine.walk(app, walkers, weighted=weighted, seed=17 + length, walker_begin=5, **kw)
    finally:
        engine.set_option("compact_offsets", 1)
        engine.set_option("cursor_adjacency", 0)
    prm = oracle_lib.make_params(app, seed=17 + length, walker_begin=5, walker_num=walkers, weighted=weighted, **kw)
    ocsr = oracle_lib.CSR(V, csr["off"], csr["nbr"], csr.get("w"))
    lens, verts, steps = oracle_lib.walk(ocsr, prm, cap=(40 * (length + 2) if app == "ppr" else length + 1))
    assert got.total_steps == steps
    np.testing.assert_array_equal(got.path_length, lens)
    np.testing.assert_array_equal(got.vertices, verts)
