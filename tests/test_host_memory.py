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
    for name in ("fake_used", "fake_largest", "fake_failures", "fake_stale", "fake_captures", "fake_graph_launches"):
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
        self.h = ctypes.c_void_p()
        assert self.L.fake_stale() == 0


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


def test_graph_is_dropped_where_something_else_runs_out(lib):
    """Out of memory in a call that is no allocation of the library's: the
    candidate buffers go all the same, and the graphs with them."""
    ix = HostIndex(lib, 64, 16, 8, 4000)
    ix.search(50, 300)  # (so that the second of these allocates nothing)
    for _ in range(2):
        ix.search(2000, 10, Precision.BF16, graph=True)
    assert lib.fake_captures() == 1 and lib.fake_graph_launches() == 1
    lib.fake_fail_copies(1)
    ix.search(50, 300)
    ix.search(2000, 10, Precision.BF16, graph=True)
    ix.close()


def test_exact_search_of_overflowing_queries_gets_the_candidates_memory(lib):
    """The queries that a screened batch hands to the exact scan (or all of them
    after a wait that gave up) find room where the batch alone would."""
    for overflow, err in ((2000, 0), (0, 14)):
        ix = HostIndex(lib, 64, 16, 8, 4000)
        ix.search(2000, 100)
        assert ix.launched("rerank") == 1 and ix.launched("scan_exact") == 0
        lib.fake_overflow(overflow)
        lib.fake_err(err)
        ix.room(4 * MB)  # the exact scan's slots take 13
        ix.search(2000, 100)
        assert lib.fake_failures() == 1 and ix.launched("rerank") == 2 and ix.launched("scan_exact") == 1
        # With room again, through the candidates again.
        lib.fake_overflow(0)
        lib.fake_err(0)
        ix.room(1 << 30)
        ix.search(2000, 100)
        assert ix.launched("rerank") == 3 and ix.launched("scan_exact") == 1
        ix.close()


@pytest.mark.parametrize("d", [64, 144])
@pytest.mark.parametrize("graph", [False, True])
def test_kept_candidate_memory_fails_no_later_call(lib, d, graph):
    ix = HostIndex(lib, d, 16, 8, 4000)
    before = lib.fake_used()
    ix.search(3000, 20)
    kept = lib.fake_used() - before
    assert kept > 64 * MB and ix.launched("scan_exact") == 0
    # A search beyond the candidates' k: its slots (58 MB) and results.
    ix.room(8 * MB)
    ix.search(3000, 300, graph=graph)
    assert ix.launched("scan_exact") >= 1 and lib.fake_failures() >= 1
    assert lib.fake_used() - before < kept
    ix.close()


def test_screened_search_without_room_keeps_nothing_of_the_candidates(lib):
    ix = HostIndex(lib, 144, 16, 8, 4000)
    before = lib.fake_used()
    ix.search(6000, 300)  # exact
    exact_only = lib.fake_used() - before
    ix.search(3000, 20)  # 24 MB of candidates, 49 of their rows, 9 of gathered queries
    assert lib.fake_used() - before - exact_only > 64 * MB
    ix.room(10 * MB)
    ix.search(6000, 20)
    assert lib.fake_failures() >= 1 and ix.launched("scan_exact") == 2
    # (The small buffers have grown with the batch.)
    assert lib.fake_used() - before - exact_only < 8 * MB
    ix.close()


def test_add_gets_the_candidates_memory(lib):
    ix = HostIndex(lib, 64, 16, 8, 4000)
    ix.search(4000, 20)
    ix.room(16 * MB)
    x = np.zeros((40_000, 64), np.float32)  # 10 MB, its copies and scratch
    assert lib.hb_add(ix.h, x.shape[0], x.ctypes.data) == 0, lib.hb_last_error()
    assert lib.fake_failures() >= 1
    ix.search(4000, 20)
    ix.close()


@pytest.mark.parametrize("d,n,nlist,nprobe,nq,precision", [
    (64, 300_000, 500, 17, 33, Precision.FP32), (64, 300_000, 500, 17, 33, Precision.BF16),
    (144, 300_000, 500, 17, 33, Precision.FP32), (128, 10_000, 100, 10, 100, Precision.FP32),
    (500, 20_000, 100, 16, 200, Precision.FP32)])
def test_small_first_batch_takes_no_large_block(lib, d, n, nlist, nprobe, nq, precision):
    """A block of one MiB and more is mapped on its own, which costs the first
    small batch on an index more than its search."""
    ix = HostIndex(lib, d, nlist, nprobe, n)
    assert lib.fake_largest() > MB
    ix.search(nq, 20, precision)
    assert ix.launched("scan_exact") == 0 and lib.fake_largest() < MB
    ix.search(3000, 20, precision)  # (beyond the spare memory: one block)
    assert ix.launched("scan_exact") == 0 and lib.fake_largest() > 16 * MB
    ix.close()
