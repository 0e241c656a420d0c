"""A program's own hooks among node2vec's functors, and other values in them, are
the walk's: the kernel for node2vec takes no walk but node2vec's.  Each
combination against the general kernel (the same hooks with the dynamic
component under another name), and node2vec's own against the oracle."""

import ctypes
import os
import subprocess

import numpy as np
import pytest

from oracle import graphs as G

pytestmark = pytest.mark.gpu

V, N, LENGTH = 400, 20000, 21
HERE = os.path.dirname(os.path.abspath(__file__))
HOOKS = ["none", "start", "extension", "update", "response", "lower bound", "query", "upper bound", "weights"]


@pytest.fixture(scope="module")
def hooks(tmp_path_factory):
    import knightking_gb300 as kk
    from knightking_gb300 import build
    kk.lib()
    so = str(tmp_path_factory.mktemp("hooks") / "libnode2vec_own_hooks.so")
    lib = os.path.dirname(kk.library_path())
    subprocess.run([build.nvcc()] + build.ARCH + build.NVCC_FLAGS +
                   ["--split-compile", "8", "-shared", os.path.join(HERE, "node2vec_own_hooks.cu"), "-o", so, "-L" + lib,
                    "-lknightking_gb300", "-Xlinker", "-rpath," + lib], check=True)
    L = ctypes.CDLL(so)
    L.kk_node2vec_own_hooks.restype = ctypes.c_int
    L.kk_node2vec_own_hooks.argtypes = [ctypes.c_void_p, ctypes.c_void_p, ctypes.c_int, ctypes.c_int, ctypes.c_void_p,
                                        ctypes.c_void_p]
    return L


@pytest.fixture(scope="module")
def graph():
    import knightking_gb300 as kk
    g = G.random_undirected(V, 5000, seed=2, weight="unif")
    csr = G.csr_file_order(V, g["src"], g["dst"], w=g["w"])
    e = kk.WalkEngine(0)
    e.load_arrays(V, csr["off"], csr["nbr"], csr["w"])
    yield e, csr
    e.close()


@pytest.mark.parametrize("p,q", [(0.25, 3.0), (2.0, 0.5)])
@pytest.mark.parametrize("which", range(len(HOOKS)), ids=HOOKS)
def test_own_hooks(graph, hooks, oracle_lib, which, p, q):
    from knightking_gb300 import _capi
    e, csr = graph
    w = np.ascontiguousarray(csr["w"][::-1])
    if HOOKS[which] == "weights" and p >= 1:
        return  # no outlier: nothing but the alias tables reads them
    opts = e.make_opts("node2vec", N, seed=4, walk_length=LENGTH, p=p, q=q, weighted=False)
    got = []
    for general in (0, 1):
        out = ctypes.POINTER(_capi.KKPaths)()
        st = hooks.kk_node2vec_own_hooks(e._h, ctypes.byref(opts), which, general, w.ctypes.data, ctypes.byref(out))
        assert st == _capi.KK_OK, _capi.lib().kk_last_error(e._h)
        _, _, lens, _, verts, _ = _capi.paths_to_numpy_owned(out)
        got.append((lens, verts))
    np.testing.assert_array_equal(got[0][0], got[1][0])
    np.testing.assert_array_equal(got[0][1], got[1][1])
    if HOOKS[which] == "none" and p >= 1:
        ocsr = oracle_lib.CSR(V, csr["off"], csr["nbr"], csr["w"]).sorted_copy()
        prm = oracle_lib.make_params("node2vec", walker_num=N, weighted=False, seed=4, walk_length=LENGTH, p=p, q=q)
        lens, verts, _ = oracle_lib.walk(ocsr, prm, cap=LENGTH + 1)
        np.testing.assert_array_equal(got[0][0], lens)
        np.testing.assert_array_equal(got[0][1], verts)
