"""Who holds a served request's memory: a result is views of its pinned block,
which goes back when the last of them is gone, but of small results only so many
hold blocks at a time, and a further one is copied and its block goes back at
once.  Server.poll over a library that stands in for the served one."""

import ctypes

import numpy as np
import pytest

import knightking_gb300 as kk
from knightking_gb300 import _capi


KEPT = 256  # small results that hold their blocks


LIBC = ctypes.CDLL(None)
LIBC.malloc.restype = ctypes.c_void_p
LIBC.malloc.argtypes = [ctypes.c_size_t]


def _malloc(values):
    """A copy of values that free() may have: what a test leaves behind goes to the library's own kk_paths_free."""
    size = max(values.nbytes, 8)
    a = np.frombuffer((ctypes.c_uint8 * size).from_address(LIBC.malloc(size)), values.dtype)[:len(values)]
    a[:] = values
    return a


class Library:
    """kk_serve_poll hands out the paths it is given; kk_paths_free is counted."""

    def __init__(self, lengths, cap):
        n = len(lengths)
        self.length = _malloc(np.array(lengths, np.uint32))
        self.offset = _malloc(np.arange(n, dtype=np.uint64) * np.uint64(cap))
        self.vertices = _malloc(np.arange(max(n * cap, 1), dtype=np.uint32))
        self.freed = 0
        p = self.paths = _capi.KKPaths.from_address(LIBC.malloc(ctypes.sizeof(_capi.KKPaths)))
        p.owner = None
        p.walker_num, p.walker_begin, p.epoch_walkers = n, 7, n
        p.total_steps = int(self.length.sum()) - n
        for field, array, kind in (("length", self.length, ctypes.c_uint32), ("offset", self.offset, ctypes.c_uint64),
                                   ("vertices", self.vertices, ctypes.c_uint32)):
            setattr(p, field, array.ctypes.data_as(ctypes.POINTER(kind)))

    def kk_serve_poll(self, handle, ticket, timeout_ms, result):
        result._obj.status = _capi.KK_OK
        result._obj.paths = ctypes.pointer(self.paths)
        return _capi.KK_OK

    def kk_paths_free(self, paths):
        self.freed += 1


@pytest.fixture
def server():
    s = kk.Server.__new__(kk.Server)
    s._h, s._kept = None, set()
    return s


def _poll(monkeypatch, server, lib, **kw):
    monkeypatch.setattr(_capi, "lib", lambda: lib)
    server._lib = lib
    return server.poll(1, **kw)


@pytest.mark.parametrize("n,cap", [(0, 5), (1, 1), (33, 21), (200, 81), (60000, 81)])
@pytest.mark.parametrize("dead_ends", [False, True])
@pytest.mark.parametrize("held", [0, KEPT - 1, KEPT])
def test_result(monkeypatch, server, n, cap, dead_ends, held):
    server._kept.update(range(held))  # other results that hold blocks
    lengths = [1 + (7 * i) % cap if dead_ends and cap > 1 else cap for i in range(n)]
    lib = Library(lengths, cap)
    res = _poll(monkeypatch, server, lib)
    paths = res.paths
    want = np.concatenate([lib.vertices[i * cap:i * cap + k] for i, k in enumerate(lengths)] + [np.zeros(0, np.uint32)])
    packed = np.concatenate([[0], np.cumsum(lengths)])[:n]
    gaps = not np.array_equal(packed, lib.offset)  # such paths are compacted, small or not
    small = 12 * n + 4 * len(want) < 1 << 18
    views = n and not gaps and not (small and held == KEPT)
    assert lib.freed == (0 if views else 1)
    assert len(server._kept) == held + (1 if views and small else 0)
    if views:
        assert np.shares_memory(paths.vertices, lib.vertices)
    else:
        lib.length[:], lib.offset[:], lib.vertices[:] = 0, 0, 0  # the arrays below are the caller's
    assert res.total_steps == len(want) - n
    np.testing.assert_array_equal(paths.path_length, lengths)
    np.testing.assert_array_equal(paths.offset, packed)
    np.testing.assert_array_equal(paths.vertices, want)
    last = paths.vertices
    del paths, res
    assert lib.freed == (0 if views else 1)  # a view is left
    del last
    assert lib.freed == 1 and len(server._kept) == held


def test_many_kept(monkeypatch, server):
    """Ten thousand kept results hold a bounded number of blocks, which are back
    for others as results go."""
    libs = [Library([5, 5], 5) for _ in range(10000)]
    kept = [_poll(monkeypatch, server, lib) for lib in libs]
    assert sum(not lib.freed for lib in libs) == KEPT
    last = libs[0]
    monkeypatch.setattr(_capi, "lib", lambda: last)
    del kept[:10]
    assert len(server._kept) == KEPT - 10 and last.freed == 10
    more = Library([5, 5], 5)
    res = _poll(monkeypatch, server, more)
    assert more.freed == 0 and len(server._kept) == KEPT - 9
    del res
    assert more.freed == 1
    kept.clear()
    assert not server._kept


def test_unread_results(monkeypatch, server):
    lib = Library([5, 5], 5)
    res = _poll(monkeypatch, server, lib, keep_paths=False)
    assert res.paths is None and res.total_steps == 8 and lib.freed == 1 and not server._kept
