"""The alias build in one launch against the oracle's tables, index for index and
bit for bit, and the classes' own launches beside it: rows at both edges of
every class, rows of one class only, and weight families whose pairings run
long, end at once or tie."""

import numpy as np
import pytest

from oracle import graphs as G

pytestmark = pytest.mark.gpu

EDGES = [1, 2, 15, 16, 17, 31, 32, 33, 127, 128, 129, 511, 512, 513, 1023, 1024, 1025, 2048, 2049, 4096, 4097, 16384,
         16385, 20011]


@pytest.fixture(scope="module")
def engine():
    import knightking_gb300 as kk
    e = kk.WalkEngine(0)
    yield e
    e.close()


@pytest.mark.parametrize("one", [1, 0])
@pytest.mark.parametrize("weights", ["lognormal", "equal", "one heavy"])
@pytest.mark.parametrize("degrees", [EDGES, [1] * 40, [16] * 33, [600] * 3, [1100, 5000], [20011]])
def test_tables(engine, oracle_lib, degrees, weights, one):
    rng = np.random.default_rng(len(degrees))
    V = max(max(degrees), len(degrees)) + 50
    src = np.concatenate([np.full(d, 7 * k % V if len(degrees) < V // 7 else k) for k, d in enumerate(degrees)])
    dst = np.concatenate([rng.permutation(V)[:d] for d in degrees])
    if weights == "lognormal":
        w = np.exp(rng.normal(size=len(src))).astype(np.float32)
    else:
        w = np.full(len(src), 1.5, np.float32)
        if weights == "one heavy":
            w[np.unique(src, return_index=True)[1]] = 1.0e6
    csr = G.csr_file_order(V, src.astype(np.uint32), dst.astype(np.uint32), w=w)
    engine.load_arrays(V, csr["off"], csr["nbr"], csr["w"])
    engine.set_option("alias_one_launch", one)
    try:
        got = engine.alias_tables()
    finally:
        engine.set_option("alias_one_launch", 1)
    want = oracle_lib.alias_build(oracle_lib.CSR(V, csr["off"], csr["nbr"], csr["w"]))
    for x, y in zip(got, want):
        np.testing.assert_array_equal(x.view(np.uint32), y.view(np.uint32))
