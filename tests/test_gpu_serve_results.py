"""A served request's paths are the caller's: they are those of the request run
alone, packed or (walks that end early) compacted, and stay so while later
requests are served and after the server and its engine are gone."""

import numpy as np
import pytest

from oracle import graphs as G

pytestmark = pytest.mark.gpu


def _graph(dead_ends):
    rng = np.random.default_rng(6)
    if not dead_ends:
        g = G.random_undirected(400, 5000, seed=5, weight="unif")
        return 400, G.csr_file_order(400, g["src"], g["dst"], w=g["w"])
    src, dst = rng.integers(0, 300, 3000).astype(np.uint32), rng.integers(0, 400, 3000).astype(np.uint32)
    return 400, G.csr_file_order(400, src, dst, w=rng.random(3000, dtype=np.float32) + 0.5)


@pytest.mark.parametrize("dead_ends", [False, True])
def test_results_outlive_server(dead_ends):
    import knightking_gb300 as kk
    V, csr = _graph(dead_ends)
    e = kk.WalkEngine(0)
    e.load_arrays(V, csr["off"], csr["nbr"], csr["w"])
    jobs = [dict(walker_num=n, seed=50 + i, walk_length=length, p=2.0, q=0.5, walker_begin=7 * i, weighted=True)
            for i, (n, length) in enumerate([(0, 5), (1, 0), (1, 9), (33, 4), (5000, 20), (777, 61)])]
    server = e.serve("node2vec", slots=2, max_jobs=4, slot_bytes=1 << 24)
    first = [server.poll(t).paths for t in [server.submit(**j) for j in jobs]]
    kept = [(p.path_length.copy(), p.offset.copy(), p.vertices.copy()) for p in first]
    again = [server.poll(t).paths for t in [server.submit(**dict(j, seed=j["seed"] + 1)) for j in jobs]]
    assert (again[4].vertices != first[4].vertices).any() if len(again[4].vertices) == len(first[4].vertices) else True
    assert server.poll(server.submit(**jobs[4]), keep_paths=False).paths is None
    server.stop()
    alone = [e.walk("node2vec", j["walker_num"], **{k: v for k, v in j.items() if k != "walker_num"})
             if j["walker_num"] else None for j in jobs]
    e.close()
    for p, (length, offset, vertices), a in zip(first, kept, alone):
        np.testing.assert_array_equal(p.path_length, length)
        np.testing.assert_array_equal(p.offset, offset)
        np.testing.assert_array_equal(p.vertices, vertices)
        if a is not None:
            np.testing.assert_array_equal(p.path_length, a.path_length)
            np.testing.assert_array_equal(p.offset, a.offset)
            np.testing.assert_array_equal(p.vertices, a.vertices)
            assert p.total_steps == a.total_steps
