"""GPU tests of searches whose results overwrite their queries' memory: the same
results as into arrays of their own."""
import numpy as np
import pytest

from harmony_b200 import Index, Precision, SearchMode, datasets

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("d,precision", [(128, Precision.FP32), (128, Precision.BF16), (256, Precision.FP32),
                                         (256, Precision.FP8), (100, Precision.FP32)])
@pytest.mark.parametrize("graph", [False, True])
def test_results_over_queries(d, precision, graph):
    import torch
    nq, k = 10_000, d // 2
    base, q = datasets.config2(seed=d, nb=40_000, nq=nq, d=d, ncomp=60)
    ix = Index(d, 48, 8)
    ix.train(base.shape[0], base)
    ix.add(base.shape[0], base)
    ix.preSearch(0, 0, 0, 0, 0, Index.Param(mode=SearchMode.ORIGINAL), "")
    ix.search_params.precision = precision
    q = torch.from_numpy(q).cuda()
    D, I = torch.empty((nq, k), device="cuda"), torch.empty((nq, k), device="cuda", dtype=torch.int64)
    ix.search(nq, q, k, D, I)
    ix.search_params.use_graph = graph
    # Distances over the second half of the queries, then ids over all of them.
    buf = q.clone()
    Da, Ia = buf.view(-1)[nq * d - nq * k:].view(nq, k), torch.empty_like(I)
    ix.search(nq, buf, k, Da, Ia)
    assert torch.equal(Da, D) and torch.equal(Ia, I)
    buf = q.clone()
    Da, Ia = torch.empty_like(D), buf.view(-1).view(torch.int64).view(nq, k)
    ix.search(nq, buf, k, Da, Ia)
    assert torch.equal(Da, D) and torch.equal(Ia, I)


def test_host_results_over_queries():
    nq, d, k = 3000, 64, 64
    base, q = datasets.config2(seed=5, nb=40_000, nq=nq, d=d, ncomp=60)
    ix = Index(d, 48, 8)
    ix.train(base.shape[0], base)
    ix.add(base.shape[0], base)
    ix.preSearch(0, 0, 0, 0, 0, Index.Param(mode=SearchMode.ORIGINAL), "")
    D, I = np.empty((nq, k), np.float32), np.empty((nq, k), np.int64)
    ix.search(nq, q, k, D, I)
    Da, Ia = np.ascontiguousarray(q), np.empty_like(I)
    ix.search(nq, Da, k, Da, Ia)
    assert np.array_equal(Da, D) and np.array_equal(Ia, I)
