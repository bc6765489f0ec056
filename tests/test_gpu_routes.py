"""GPU tests that calls of given sizes take the scan that the tests of that
scan's results mean to run: plain FP32 searches of wide vectors the candidate
matrix, narrower ones the bounded scan, the least calls and k > 256 the exact
scan, also as graphs (whose first call, which sizes the buffers, is profiled)."""
import numpy as np
import pytest

from harmony_b200 import Index, SearchMode

pytestmark = pytest.mark.gpu
SCANS = {"scan_bf16", "cand_scan", "scan_exact"}


@pytest.mark.parametrize("graph", [False, True])
@pytest.mark.parametrize("d,sizes,nq,k,scan", [
    (200, (2500, 2500, 2500, 100, 3), 301, 20, "cand_scan"), (512, (2500, 2500, 2500, 100, 3), 301, 20, "cand_scan"),
    (520, (2500, 2500, 2500, 100, 3), 301, 20, "cand_scan"), (128, (800,) * 48, 131, 256, "scan_bf16"),
    (33, (800,) * 48, 131, 1, "scan_bf16"), (64, (60, 70, 80), 3, 10, "scan_exact"), (64, (800,) * 48, 131, 257, "scan_exact"),
    (300, (60, 70, 80), 3, 10, "scan_exact")])
def test_plain_fp32_takes(d, sizes, nq, k, scan, graph):
    rng = np.random.default_rng(d + k)
    nlist, nb = len(sizes), sum(sizes)
    cent = (rng.standard_normal((nlist, d)) * 2).astype(np.float32)
    base = (np.repeat(cent, sizes, axis=0) + rng.standard_normal((nb, d)) * np.linspace(1, 0.2, d)).astype(np.float32)
    q = base[rng.integers(0, nb, nq)]
    ix = Index(d, nlist, nlist)
    ix.train(nlist, cent, lite=True)
    ix.add(nb, base)
    ix.preSearch(0, 0, 0, 0, 0, Index.Param(mode=SearchMode.ORIGINAL), "")
    ix.search_params.use_graph = graph
    D, I = np.empty((nq, k), np.float32), np.empty((nq, k), np.int64)
    ix.profile(True)
    ix.search(nq, q, k, D, I)
    assert set(ix.profile_read()) & SCANS == {scan}
    ix.profile(False)
    launches = ix.launch_count()
    D2, I2 = np.empty_like(D), np.empty_like(I)
    ix.search(nq, q, k, D2, I2)
    assert ix.launch_count() > launches and np.array_equal(D, D2) and np.array_equal(I, I2)
