"""Lengths of PPR walks, found before the walk by lanes that take a warp's
walkers in turn and finish the last of them together: at walker counts about a
warp's share, means on both sides of a warp's width, and isolated starts, the
lengths and paths are the oracle's."""

import numpy as np
import pytest

from oracle import graphs as G

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mean", [1.02, 4.0, 80.0, 900.0])
@pytest.mark.parametrize("n", [1, 33, 9728 * 2 + 1, 9728 * 34 + 5])
def test_ppr_lengths(oracle_lib, mean, n):
    import knightking_gb300 as kk
    if n * mean > 4e7:
        n = 9728 * 4 + 5
    g = G.random_undirected(500, 6000, seed=int(mean), weight=None)
    csr = G.csr_file_order(640, g["src"], g["dst"])  # vertices 500.. are isolated
    kw = dict(terminate_prob=1.0 / mean, seed=n, walker_begin=41)
    e = kk.WalkEngine(0)
    e.load_arrays(640, csr["off"], csr["nbr"])
    got = e.walk("ppr", n, weighted=False, **kw)
    e.close()
    prm = oracle_lib.make_params("ppr", walker_num=n, weighted=False, **kw)
    lens, verts, steps = oracle_lib.walk(oracle_lib.CSR(640, csr["off"], csr["nbr"], None, None), prm,
                                         cap=int(got.path_length.max()) + 1)
    assert got.total_steps == steps
    np.testing.assert_array_equal(got.path_length, lens)
    np.testing.assert_array_equal(got.vertices, verts)
