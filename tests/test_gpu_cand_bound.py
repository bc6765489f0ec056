"""GPU tests of the candidate-matrix scan's error bound: with every probed row
among the R candidates, the rows the bound drops before the exact re-rank may
not change the result, which is then the exact scan's (hb_search_noalloc)."""
import numpy as np
import pytest

from harmony_b200 import Index, Precision, SearchMode, lib

pytestmark = pytest.mark.gpu


# d on both sides of each width of the gathered rows (128, 256, 512, 1024).
@pytest.mark.parametrize("precision", [Precision.BF16, Precision.FP8])
@pytest.mark.parametrize("d,k", [(64, 300), (129, 1), (256, 20), (300, 100), (513, 7), (1000, 33)])
def test_dropped_rows_do_not_change_the_result(d, k, precision):
    import torch
    rng = np.random.default_rng(d + k)
    nb, nlist, P, nq = 1500, 8, 4, 37
    cent = (rng.standard_normal((nlist, d)) * 0.5).astype(np.float32)
    base = (cent[rng.integers(0, nlist, nb)] + rng.standard_normal((nb, d)) * np.linspace(1, 0.1, d)).astype(np.float32)
    base[100:140] = base[100]                       # ties
    if precision == Precision.BF16:                 # rows no distance admits (an infinite row makes its
        base[7, 3], base[8, 0] = np.nan, np.inf     # whole list's FP8 scale infinite: not exact there)
    q = (base[::41][:nq] + np.float32(0.01)).astype(np.float32)
    q[5, 0] = np.nan
    ix = Index(d, nlist, P)
    ix.train(nlist, cent, lite=True)
    ix.add(nb, base)
    ix.preSearch(0, 0, 0, 0, 0, Index.Param(mode=SearchMode.ORIGINAL), "")
    qd = torch.from_numpy(q).cuda()
    De = torch.empty((nq, k), device="cuda")
    Ie = torch.empty((nq, k), device="cuda", dtype=torch.int64)
    torch.cuda.synchronize()
    assert lib().hb_search_noalloc(ix._h, nq, qd.data_ptr(), k, De.data_ptr(), Ie.data_ptr()) == 0
    ix.search_params.precision, ix.search_params.rerank_mult = precision, -(-nb // k)
    D, I = np.empty((nq, k), np.float32), np.empty((nq, k), np.int64)
    ix.search(nq, q, k, D, I)
    assert np.array_equal(D.view(np.uint32), De.cpu().numpy().view(np.uint32))
    assert np.array_equal(I, Ie.cpu().numpy())
