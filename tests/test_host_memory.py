"""What the index does where device memory runs out, on the CPU (tests/host):
searches fall back to what fits, and no captured graph outlives a buffer it was
captured with."""
import ctypes

import numpy as np
import pytest

from harmony_b200 import Precision, SearchMode, _SearchParamsC
from tests import host

pytestmark = pytest.mark.skipif(not host.available(), reason="needs g++ and the CUDA headers")
MB = 1 << 20


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    L = host.build(tmp_path_factory.mktemp("host"))
    c = ctypes
    L.hb_last_error.restype = c.c_char_p
    L.hb_create.argtypes = [c.c_size_t, c.c_size_t, c.c_size_t, c.c_int, c.c_int, c.c_void_p]
    L.hb_add.argtypes = [c.c_void_p, c.c_size_t, c.c_void_p]
    L.hb_search.argtypes = [c.c_void_p, c.c_size_t, c.c_void_p, c.c_size_t, c.c_void_p, c.c_void_p, c.c_void_p]
    L.hb_destroy.argtypes = [c.c_void_p]
    L.fake_limit.argtypes = [c.c_size_t]
    L.fake_launched.argtypes = [c.c_char_p]
    for name in ("fake_used", "fake_failures", "fake_stale", "fake_captures", "fake_graph_launches"):
        getattr(L, name).restype = c.c_longlong
    return L


class HostIndex:
    def __init__(self, L, d, nlist, nprobe, n):
        L.fake_reset()
        self.L, self.d, self.h = L, d, ctypes.c_void_p()
        assert L.hb_create(d, nlist, nprobe, 1, 0, ctypes.byref(self.h)) == 0, L.hb_last_error()
        x = np.zeros((n, d), np.float32)
        assert L.hb_add(self.h, n, x.ctypes.data) == 0, L.hb_last_error()

    def search(self, nq, k, precision=Precision.FP32, graph=False):
        p = _SearchParamsC()
        self.L.hb_search_params_init(ctypes.byref(p))
        p.mode, p.precision, p.use_graph = SearchMode.ORIGINAL, precision, int(graph)
        q = np.zeros((nq, self.d), np.float32)
        D, I = np.empty((nq, k), np.float32), np.empty((nq, k), np.int64)
        rc = self.L.hb_search(self.h, nq, q.ctypes.data, k, ctypes.byref(p), D.ctypes.data, I.ctypes.data)
        assert rc == 0, self.L.hb_last_error()
        assert self.L.fake_stale() == 0  # every buffer a launch (or a replayed one) was given is there

    def room(self, bytes_left):
        self.L.fake_limit(self.L.fake_used() + bytes_left)

    def launched(self, name):
        return self.L.fake_launched(name.encode())

    def close(self):
        self.L.hb_destroy(self.h)
        assert self.L.fake_used() == 0 and self.L.fake_stale() == 0


def test_graph_is_dropped_with_its_buffers(lib):
    ix = HostIndex(lib, 64, 16, 8, 4000)
    # A screened FP32 batch that does not fit (48 KB a query) leaves the small
    # buffers at its size and gives the candidate buffers back.
    ix.room(20 * MB)
    ix.search(2000, 10)
    assert lib.fake_failures() > 0 and ix.launched("scan_exact") == 1 and ix.launched("scan_bf16") == 0
    # A graph captured with candidate buffers, then the same FP32 batch again.
    ix.room(1 << 40)
    ix.search(100, 10, Precision.BF16, graph=True)
    ix.search(100, 10, Precision.BF16, graph=True)
    assert lib.fake_captures() == 1 and lib.fake_graph_launches() == 1
    ix.room(20 * MB)
    ix.search(2000, 10)
    assert ix.launched("scan_exact") == 2
    ix.search(100, 10, Precision.BF16, graph=True)
    ix.close()
