"""kk_walk's streamed copy-out: walks whose path lengths are known before they
run, of one epoch and 16 MB of vertices or more, leave for the result's block
segment by segment while they walk.  On both sides of that size the paths are
those of the copy after the walk (into_stream 0) and the oracle's."""

import numpy as np
import pytest

from oracle import graphs as G

pytestmark = pytest.mark.gpu

LENGTH = 19
AT = 16_000_000 // 4 // (LENGTH + 1)  # the first walker count that streams


def _same(a, b):
    assert a.total_steps == b.total_steps
    np.testing.assert_array_equal(a.path_length, b.path_length)
    np.testing.assert_array_equal(a.offset, b.offset)
    np.testing.assert_array_equal(a.vertices, b.vertices)


@pytest.mark.parametrize("n", [AT - 1, AT, AT + 4097, (1 << 20) + 1])
@pytest.mark.parametrize("app", ["deepwalk", "ppr", "node2vec"])
def test_streamed_walk(oracle_lib, app, n):
    import knightking_gb300 as kk
    g = G.random_undirected(900, 9000, seed=n % 97, weight="unif")
    csr = G.csr_file_order(1000, g["src"], g["dst"], w=g.get("w"))  # vertices 900.. are isolated
    kw = dict(seed=5, walker_begin=77)
    kw.update(dict(terminate_prob=1.0 / (LENGTH + 1)) if app == "ppr" else dict(walk_length=LENGTH))
    if app == "node2vec":
        kw.update(p=2.0, q=0.5)
    e = kk.WalkEngine(0)
    e.load_arrays(1000, csr["off"], csr["nbr"], csr.get("w"))
    walks = []
    for stream in (0, 1):
        e.set_option("into_stream", stream)
        walks.append(e.walk(app, n, weighted=True, **kw))
    _same(*walks)
    # a start vertex out of range is refused, and the next call is whole
    with pytest.raises(kk.KKError):
        e.walk(app, n, weighted=True, start=np.array([1, 1000], np.uint32), **kw)
    _same(walks[0], e.walk(app, n, weighted=True, **kw))
    e.close()
    if n != AT:
        return
    ocsr = oracle_lib.CSR(1000, csr["off"], csr["nbr"], csr.get("w"), None)
    if app == "node2vec":
        ocsr = ocsr.sorted_copy()
    prm = oracle_lib.make_params(app, walker_num=n, weighted=True, **kw)
    lens, verts, steps = oracle_lib.walk(ocsr, prm, cap=400 + 1 if app == "ppr" else LENGTH + 1)
    np.testing.assert_array_equal(walks[1].path_length, lens)
    np.testing.assert_array_equal(walks[1].vertices, verts)


def test_two_results_and_epochs():
    """Results hold blocks of their own; a walk of several epochs is copied after each."""
    import knightking_gb300 as kk
    g = G.random_undirected(900, 9000, seed=3, weight="unif")
    csr = G.csr_file_order(900, g["src"], g["dst"], w=g.get("w"))
    e = kk.WalkEngine(0)
    e.load_arrays(900, csr["off"], csr["nbr"], csr.get("w"))
    kw = dict(walk_length=LENGTH, weighted=True)
    a = e.walk("deepwalk", 2 * AT, seed=1, **kw)
    b = e.walk("deepwalk", 2 * AT, seed=2, **kw)
    assert (a.vertices != b.vertices).any()
    c = e.walk("deepwalk", 2 * AT, seed=1, rate=0.5, **kw)
    np.testing.assert_array_equal(a.vertices, c.vertices)
    _same(b, e.walk("deepwalk", 2 * AT, seed=2, **kw))
    e.close()
