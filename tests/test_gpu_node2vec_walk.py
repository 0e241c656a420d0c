"""node2vec over the edge set, walker for walker against the oracle: rows at the
edges of the set's size classes (32, 128, 512, 1024 edges and one more) and
beyond them, duplicate edges, vertex 0 as a previous vertex, a directed graph
with missing return edges and dead ends, p and q with and without the outlier
and on both sides of q = 1, and walks of no and one step."""

import numpy as np
import pytest

from oracle import graphs as G

pytestmark = pytest.mark.gpu

DEGREES = [1, 2, 31, 32, 33, 127, 128, 129, 511, 512, 513, 1023, 1024, 1025, 3000]


@pytest.fixture(scope="module")
def engine():
    import knightking_gb300 as kk
    e = kk.WalkEngine(0)
    yield e
    e.close()


def _graph(kind, weighted):
    rng = np.random.default_rng(7)
    V = 3200
    if kind == "directed":
        src, dst = rng.integers(0, 150, 4000), rng.integers(0, 170, 4000)  # 150.. are dead ends
        V = 170
    else:
        # vertex k has DEGREES[k] neighbours at least; the others a few among themselves
        src = np.concatenate([np.full(d, k) for k, d in enumerate(DEGREES)] + [rng.integers(20, V, 3000)])
        dst = np.concatenate([rng.permutation(np.arange(100, V))[:d] for d in DEGREES] + [rng.integers(20, V, 3000)])
        if kind == "duplicates":
            src, dst = np.concatenate([src, src[::3]]), np.concatenate([dst, dst[::3]])
        src, dst = np.concatenate([src, dst]), np.concatenate([dst, src])
    keep = src != dst
    src, dst = src[keep].astype(np.uint32), dst[keep].astype(np.uint32)
    w = (1.0 + 4.0 * rng.random(len(src))).astype(np.float32) if weighted else None
    return G.csr_file_order(V, src, dst, w=w)


@pytest.mark.parametrize("p,q,length", [(0.25, 3.0, 20), (0.3, 0.4, 20), (2.0, 0.5, 33), (1.0, 1.0, 1), (4.0, 4.0, 17),
                                        (0.5, 2.0, 0)])
@pytest.mark.parametrize("kind,weighted,layout,cursor", [("rows", True, 2, 0), ("rows", True, 0, 0),
                                                         ("rows", True, 1, 0), ("rows", False, 2, 0),
                                                         ("rows", False, 2, 1), ("duplicates", True, 2, 0),
                                                         ("directed", True, 2, 0), ("directed", False, 2, 0)])
def test_node2vec_walks(engine, oracle_lib, p, q, length, kind, weighted, layout, cursor):
    csr = _graph(kind, weighted)
    V = len(csr["off"]) - 1
    kw = dict(seed=31, walker_begin=3, walk_length=length, p=p, q=q)
    engine.load_arrays(V, csr["off"], csr["nbr"], csr.get("w"))
    engine.set_option("alias_layout", layout)
    engine.set_option("cursor_adjacency", cursor)
    try:
        got = engine.walk("node2vec", 5000, weighted=weighted, **kw)
        job = engine.batch_walk("node2vec", [dict(kw, walker_num=5000, weighted=weighted)])[0]
    finally:
        engine.set_option("alias_layout", 2)
        engine.set_option("cursor_adjacency", 0)
    ocsr = oracle_lib.CSR(V, csr["off"], csr["nbr"], csr.get("w")).sorted_copy()
    prm = oracle_lib.make_params("node2vec", walker_num=5000, weighted=weighted, **kw)
    lens, verts, steps = oracle_lib.walk(ocsr, prm, cap=length + 1)
    for r in (got, job):
        assert r.total_steps == steps
        np.testing.assert_array_equal(r.path_length, lens)
        np.testing.assert_array_equal(r.vertices, verts)


@pytest.mark.parametrize("weighted", [True, False])
@pytest.mark.parametrize("offsets32", [1, 0])
def test_node2vec_batches(engine, oracle_lib, weighted, offsets32):
    """Batches on both sides of the 3072 walkers an SM up to which the kernel has
    two blocks an SM, and the kernel with the hooks (no 32-bit offsets)."""
    csr = _graph("rows", weighted)
    V = len(csr["off"]) - 1
    engine.load_arrays(V, csr["off"], csr["nbr"], csr.get("w"))
    ocsr = oracle_lib.CSR(V, csr["off"], csr["nbr"], csr.get("w")).sorted_copy()
    engine.set_option("compact_offsets", offsets32)
    try:
        for sizes in ((33, 4000, 1), (500001, 5, 120000)):
            jobs = [dict(walker_num=n, seed=9 + k, walker_begin=10 * k, walk_length=3 + 5 * k, p=(0.25, 2.0, 1.0)[k],
                         q=(3.0, 0.5, 1.0)[k], weighted=weighted) for k, n in enumerate(sizes)]
            got = engine.batch_walk("node2vec", jobs)
            one = engine.walk("node2vec", sizes[2], **{k: v for k, v in jobs[2].items() if k != "walker_num"})
            np.testing.assert_array_equal(got[2].vertices, one.vertices)
            for job, paths in zip(jobs, got):
                lens, verts, steps = oracle_lib.walk(ocsr, oracle_lib.make_params("node2vec", **job),
                                                     cap=job["walk_length"] + 1)
                assert paths.total_steps == steps
                np.testing.assert_array_equal(paths.path_length, lens)
                np.testing.assert_array_equal(paths.vertices, verts)
    finally:
        engine.set_option("compact_offsets", 1)
