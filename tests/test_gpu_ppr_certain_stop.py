"""PPR that stops at once (terminate_prob 1): every path is its start vertex, also
that of a walker whose first draw is exactly 0 (seed 12, walker 3490575), which
no extension probability above 0 would end there.  After the walk and streamed,
to the host, into buffers and on the device."""

import numpy as np
import pytest

from oracle import graphs as G

pytestmark = pytest.mark.gpu

V, SEED, WALKER = 500, 12, 3490575


def test_first_draw_is_zero():
    word = G.philox4x32_10(np.uint32([WALKER]), np.uint32(0), np.uint32(0), np.uint32(0), SEED)[0]
    assert word[0] >> 8 == 0


@pytest.mark.parametrize("begin,n", [(WALKER, 1), (WALKER - 100, 200), (0, 4_100_000)])
@pytest.mark.parametrize("call", ["walk", "into", "device"])
def test_every_path_is_its_start(begin, n, call):
    import knightking_gb300 as kk
    g = G.random_undirected(V, 6000, seed=3, weight=None)
    csr = G.csr_file_order(V, g["src"], g["dst"])
    e = kk.WalkEngine(0)
    e.load_arrays(V, csr["off"], csr["nbr"])
    kw = dict(terminate_prob=1.0, seed=SEED, walker_begin=begin, weighted=False)
    start = ((begin + np.arange(n, dtype=np.int64)) % V).astype(np.uint32)
    if call == "walk":
        p = e.walk("ppr", n, **kw)
        steps, length, offset, vertices = p.total_steps, p.path_length, p.offset, p.vertices
    elif call == "into":
        length, offset, vertices = np.zeros(n, np.uint32), np.zeros(n, np.uint64), np.zeros(n, np.uint32)
        steps = e.walk_into("ppr", n, length.ctypes.data, offset.ctypes.data, vertices.ctypes.data, n, **kw)
    else:
        torch = pytest.importorskip("torch")
        steps, *ptr = e.walk_device("ppr", n, **kw)

        class Array:
            def __init__(self, at, kind):
                self.__cuda_array_interface__ = {"shape": (n,), "typestr": kind, "data": (at, False), "version": 3}

        length, offset, vertices = (torch.as_tensor(Array(at, kind), device="cuda").cpu().numpy()
                                    for at, kind in zip(ptr, ("<i4", "<i8", "<i4")))
    assert steps == 0
    np.testing.assert_array_equal(length, 1)
    np.testing.assert_array_equal(offset, np.arange(n))
    np.testing.assert_array_equal(vertices, start)
    e.close()
