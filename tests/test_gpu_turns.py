"""Metapath walks of more walkers than the SMs hold, whose lanes take the walkers
in turn, walker for walker against the oracle: single walks and batches of
uneven jobs, weighted and not, walks of no and one step, walkers that end where
they start, and the packing of their paths."""

import numpy as np
import pytest

from oracle import graphs as G

pytestmark = pytest.mark.gpu

SCHEMES = [[1, 2, 4, 8], [2, 8, 2], [4, 1, 16, 4, 3]]


@pytest.fixture(scope="module")
def engine():
    import knightking_gb300 as kk
    e = kk.WalkEngine(0)
    yield e
    e.close()


def _load(engine, weighted):
    g = G.random_undirected(500, 7000, seed=9, weight="unif" if weighted else None, types="uniform")
    csr = G.csr_file_order(520, g["src"], g["dst"], w=g.get("w"), type=g["type"])  # twenty isolated vertices
    engine.load_arrays(520, csr["off"], csr["nbr"], csr.get("w"), csr["type"])
    return csr


def _check(oracle_lib, csr, got, weighted, walker_num, **kw):
    prm = oracle_lib.make_params("metapath", walker_num=walker_num, weighted=weighted, schemes=SCHEMES,
                                 scheme_round_robin=True, **kw)
    ocsr = oracle_lib.CSR(520, csr["off"], csr["nbr"], csr.get("w"), csr["type"])
    lens, verts, steps = oracle_lib.walk(ocsr, prm, cap=kw["walk_length"] + 1)
    assert got.total_steps == steps
    np.testing.assert_array_equal(got.path_length, lens)
    np.testing.assert_array_equal(got.vertices, verts)


@pytest.mark.parametrize("weighted", [True, False])
@pytest.mark.parametrize("walkers,length", [(400003, 0), (400003, 1), (400003, 23), (160000, 40), (5000, 40)])
def test_metapath_turns(engine, oracle_lib, weighted, walkers, length):
    csr = _load(engine, weighted)
    kw = dict(seed=5, walker_begin=11, walk_length=length)
    got = engine.walk("metapath", walkers, weighted=weighted, schemes=SCHEMES, scheme_round_robin=True, **kw)
    _check(oracle_lib, csr, got, weighted, walkers, **kw)


@pytest.mark.parametrize("weighted", [True, False])
def test_metapath_batch_turns(engine, oracle_lib, weighted):
    csr = _load(engine, weighted)
    sizes = [(200001, 12), (1, 30), (0, 5), (90000, 0), (70007, 25), (31, 1)]
    jobs = [dict(walker_num=n, seed=3 + k, walker_begin=100 * k, walk_length=length, weighted=weighted,
                 schemes=SCHEMES, scheme_round_robin=True) for k, (n, length) in enumerate(sizes)]
    for job, got in zip(jobs, engine.batch_walk("metapath", jobs)):
        _check(oracle_lib, csr, got, weighted, job["walker_num"], seed=job["seed"], walker_begin=job["walker_begin"],
               walk_length=job["walk_length"])
