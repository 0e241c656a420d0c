"""Served node2vec batches on both sides of the 1024 walkers an SM up to which a
slot takes the kernel for small batches, and a small batch after a large one (a
slot keeps a captured graph of each): the paths are the oracle's."""

import numpy as np
import pytest

from oracle import graphs as G

pytestmark = pytest.mark.gpu

SMS = 152


@pytest.mark.parametrize("graphs", [True, False])
@pytest.mark.parametrize("weighted", [True, False])
def test_batch_sizes(oracle_lib, weighted, graphs):
    import knightking_gb300 as kk
    g = G.random_undirected(500, 6000, seed=4, weight="unif" if weighted else None)
    csr = G.csr_file_order(500, g["src"], g["dst"], w=g.get("w"))
    e = kk.WalkEngine(0)
    e.load_arrays(500, csr["off"], csr["nbr"], csr.get("w"))
    ocsr = oracle_lib.CSR(500, csr["off"], csr["nbr"], csr.get("w")).sorted_copy()
    line = 1024 * SMS
    with e.serve("node2vec", weighted=weighted, slots=1, graphs=graphs) as server:
        for k, n in enumerate((33, line, line + 1, 1, 2 * line + 77, 257 * SMS)):
            job = dict(walker_num=n, seed=k + 3, walk_length=6 + k, p=(0.25, 2.0)[k % 2], q=(3.0, 0.5)[k % 2],
                       weighted=weighted)
            got = server.poll(server.submit(**job)).paths
            lens, verts, steps = oracle_lib.walk(ocsr, oracle_lib.make_params("node2vec", **job),
                                                 cap=job["walk_length"] + 1)
            assert got.total_steps == steps
            np.testing.assert_array_equal(got.path_length, lens)
            np.testing.assert_array_equal(got.vertices, verts)
    e.close()
