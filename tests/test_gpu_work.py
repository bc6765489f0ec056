"""GPU test of the work description's multi-CTA builder (more than 32768 (query,
probe) pairs): its searches equal those of the same queries in pieces, whose
description one CTA builds."""
import numpy as np
import pytest

from harmony_b200 import Index, Precision, SearchMode

pytestmark = pytest.mark.gpu


# 9000 lists: counted straight in global memory; 700: in shared memory first,
# with a remainder of pairs in the last CTA.
@pytest.mark.parametrize("precision", [Precision.FP32, Precision.BF16])
@pytest.mark.parametrize("nlist,nprobe", [(700, 61), (9000, 60)])
def test_large_batch_equals_pieces(nlist, nprobe, precision):
    rng = np.random.default_rng(nlist)
    d, nb, nq, k = 12, 20000, 601, 5
    base = rng.standard_normal((nb, d)).astype(np.float32)
    q = rng.standard_normal((nq, d)).astype(np.float32)
    ix = Index(d, nlist, nprobe)
    ix.train(nlist, base[:nlist], lite=True)   # lists of 0 .. some dozen rows, empty ones among them
    ix.add(nb, base)
    ix.preSearch(0, 0, 0, 0, 0, Index.Param(mode=SearchMode.ORIGINAL), "")
    ix.search_params.precision = precision
    D, I = np.empty((nq, k), np.float32), np.empty((nq, k), np.int64)
    ix.search(nq, q, k, D, I)
    for a in range(0, nq, 97):
        b = min(nq, a + 97)
        Dp, Ip = np.empty((b - a, k), np.float32), np.empty((b - a, k), np.int64)
        ix.search(b - a, q[a:b], k, Dp, Ip)
        assert np.array_equal(Dp.view(np.uint32), D[a:b].view(np.uint32))
        assert np.array_equal(Ip, I[a:b])
