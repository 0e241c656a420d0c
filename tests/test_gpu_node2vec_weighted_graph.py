"""Unweighted node2vec on a graph that has weights: the edge set holds four ids
and four weights a sector, and the weights are no ids.  Their bits here are
vertex ids (zero and denormal weights), so a sector read as eight ids answers
wrongly.  Single walks, batches and served requests against the oracle."""

import numpy as np
import pytest

from oracle import graphs as G

pytestmark = pytest.mark.gpu

V = 600


@pytest.fixture(scope="module")
def graph():
    import knightking_gb300 as kk
    rng = np.random.default_rng(11)
    g = G.random_undirected(V, 6000, seed=8, weight="unif")
    hub = rng.permutation(np.arange(1, V))[:300].astype(np.uint32)  # vertex 0's neighbours
    src = np.concatenate([g["src"], hub, np.zeros(300, np.uint32)])
    dst = np.concatenate([g["dst"], np.zeros(300, np.uint32), hub])
    bits = rng.integers(0, V, len(src)).astype(np.uint32)
    bits[rng.random(len(src)) < 0.5] = 0
    csr = G.csr_file_order(V, src, dst, w=bits.view(np.float32))
    e = kk.WalkEngine(0)
    e.load_arrays(V, csr["off"], csr["nbr"], csr["w"])
    yield e, csr
    e.close()


@pytest.mark.parametrize("p,q", [(2.0, 0.5), (0.25, 3.0), (1.0, 4.0), (0.5, 0.7)])
@pytest.mark.parametrize("call", ["walk", "batch", "hooks' kernel", "serve"])
def test_unweighted_walk(oracle_lib, graph, call, p, q):
    e, csr = graph
    n, kw = 20000, dict(seed=6, walk_length=24, p=p, q=q, weighted=False)
    job = dict(kw, walker_num=n)
    if call == "walk":
        got = e.walk("node2vec", n, **kw)
    elif call == "batch":
        got = e.batch_walk("node2vec", [dict(job, seed=7), job])[1]
    elif call == "serve":
        with e.serve("node2vec", weighted=False) as server:
            got = server.poll(server.submit(**job)).paths
    else:
        e.set_option("compact_offsets", 0)
        try:
            got = e.walk("node2vec", n, **kw)
        finally:
            e.set_option("compact_offsets", 1)
    ocsr = oracle_lib.CSR(V, csr["off"], csr["nbr"], csr["w"]).sorted_copy()
    lens, verts, steps = oracle_lib.walk(ocsr, oracle_lib.make_params("node2vec", **job), cap=25)
    assert got.total_steps == steps
    np.testing.assert_array_equal(got.path_length, lens)
    np.testing.assert_array_equal(got.vertices, verts)
