"""A node2vec walk never writes past its path's room.  A start vertex outside the
graph has room for one vertex (its walker stands on vertex 0 until the call is
refused), and a walk from hooks has the room its caller gave it: either call is
refused, leaves the graph and its tables as they were, and the next call's paths
are the oracle's."""

import ctypes
import os
import subprocess

import numpy as np
import pytest

from oracle import graphs as G

pytestmark = pytest.mark.gpu

V = 400
HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.fixture
def engine():
    import knightking_gb300 as kk
    e = kk.WalkEngine(0)  # a new one: its path buffer is as large as the call asks for
    yield e
    e.close()


@pytest.fixture(scope="module")
def hooks(tmp_path_factory):
    import knightking_gb300 as kk
    from knightking_gb300 import build
    kk.lib()
    so = str(tmp_path_factory.mktemp("hooks") / "libnode2vec_hooks.so")
    lib = os.path.dirname(kk.library_path())
    subprocess.run([build.nvcc()] + build.ARCH + build.NVCC_FLAGS +
                   ["-shared", os.path.join(HERE, "node2vec_hooks.cu"), "-o", so, "-L" + lib, "-lknightking_gb300",
                    "-Xlinker", "-rpath," + lib], check=True)
    L = ctypes.CDLL(so)
    L.kk_node2vec_hooks.restype = ctypes.c_int
    L.kk_node2vec_hooks.argtypes = [ctypes.c_void_p, ctypes.c_void_p, ctypes.c_uint32, ctypes.c_void_p]
    return L


def _csr(weighted=True):
    g = G.random_undirected(V, 5000, seed=2, weight="unif" if weighted else None)
    return G.csr_file_order(V, g["src"], g["dst"], w=g.get("w"))


def _oracle(oracle_lib, csr, n, weighted, **kw):
    ocsr = oracle_lib.CSR(V, csr["off"], csr["nbr"], csr.get("w")).sorted_copy()
    prm = oracle_lib.make_params("node2vec", walker_num=n, weighted=weighted, **kw)
    return oracle_lib.walk(ocsr, prm, cap=kw["walk_length"] + 1)


def _into(engine, n, room, **kw):
    import knightking_gb300 as kk
    length, offset, vertices = np.zeros(n, np.uint32), np.zeros(n, np.uint64), np.zeros(room, np.uint32)
    engine.walk_into("node2vec", n, length.ctypes.data, offset.ctypes.data, vertices.ctypes.data, room, **kw)
    return length, vertices


@pytest.mark.parametrize("weighted", [True, False])
@pytest.mark.parametrize("n,length,start", [
    (3, 1_000_000, [V]),                     # a buffer of three vertices
    (3, 20, [V, 0xffffffff, V + 1]),         # a buffer for the whole walks
    (300_007, 19, [5, V, 17, 3]),            # beyond 2^21 vertices, every fourth walker
    (1_000_003, 19, [V + 9]),
])
@pytest.mark.parametrize("call", ["walk", "into", "device"])
def test_starts_outside_the_graph(engine, oracle_lib, weighted, n, length, start, call):
    import knightking_gb300 as kk
    csr = _csr()
    engine.load_arrays(V, csr["off"], csr["nbr"], csr["w"])
    kw = dict(seed=4, walk_length=length, p=0.25, q=3.0, weighted=weighted)
    bad = np.array(start, np.uint32)
    with pytest.raises(kk.KKError, match="start vertex"):
        if call == "walk":
            engine.walk("node2vec", n, start=bad, **kw)
        elif call == "into":
            _into(engine, n, n * 21, start=bad, **kw)
        else:
            engine.walk_device("node2vec", n, start=bad, **kw)
    n, kw["walk_length"] = min(n, 5000), min(length, 20)
    lens, verts, _ = _oracle(oracle_lib, csr, n, **kw)
    got = engine.walk("node2vec", n, **kw)
    np.testing.assert_array_equal(got.path_length, lens)
    np.testing.assert_array_equal(got.vertices, verts)
    np.testing.assert_array_equal(_into(engine, n, len(verts), **kw)[1], verts)


@pytest.mark.parametrize("room,length,refused", [(20, 20, False), (19, 20, True), (0, 1, True), (0, 0, False),
                                                 (25, 20, False)])
def test_room_of_the_caller(engine, hooks, oracle_lib, room, length, refused):
    from knightking_gb300 import _capi
    csr = _csr(weighted=False)
    engine.load_arrays(V, csr["off"], csr["nbr"])
    opts = engine.make_opts("node2vec", 5000, seed=4, walk_length=room, p=2.0, q=0.5, weighted=False)
    out = ctypes.POINTER(_capi.KKPaths)()
    st = hooks.kk_node2vec_hooks(engine._h, ctypes.byref(opts), length, ctypes.byref(out))
    if refused:
        assert st == _capi.KK_ERR_PATH_CAPACITY
        return
    assert st == _capi.KK_OK
    _, _, lens, _, verts, _ = _capi.paths_to_numpy_owned(out)
    want = _oracle(oracle_lib, csr, 5000, False, seed=4, walk_length=length, p=2.0, q=0.5)
    np.testing.assert_array_equal(lens, want[0])
    np.testing.assert_array_equal(verts, want[1])
