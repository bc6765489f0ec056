"""GPU tests of the candidate-matrix scan over items of several row tiles and
query groups, at both sides of the width up to which the queries stay in shared
memory (512 BF16, 1024 FP8 columns), and of the one-pass selection where its
sample says nothing (the first probed list empty of near rows)."""
import numpy as np
import pytest

from harmony_b200 import Index, Precision, SearchMode, lib

pytestmark = pytest.mark.gpu


# Lists of 2500, 100 and 3 rows: eight-tile items and a remainder, 128-query
# groups and a remainder of 45.
@pytest.mark.parametrize("d,precision", [(200, Precision.FP32), (512, Precision.FP32), (520, Precision.FP32),
                                         (512, Precision.BF16), (520, Precision.BF16), (300, Precision.FP8),
                                         (1000, Precision.FP8)])
def test_tiles_equal_exact_scan(d, precision):
    import torch
    rng = np.random.default_rng(d)
    sizes, nq, k = (2500, 2500, 2500, 100, 3), 301, 20
    nlist, nb = len(sizes), sum(sizes)
    cent = (rng.standard_normal((nlist, d)) * 2).astype(np.float32)
    base = (np.repeat(cent, sizes, axis=0) + rng.standard_normal((nb, d)) * np.linspace(1, 0.2, d)).astype(np.float32)
    q = (base[rng.integers(0, nb, nq)] + np.float32(0.05) * rng.standard_normal((nq, d))).astype(np.float32)
    ix = Index(d, nlist, nlist)
    ix.train(nlist, cent, lite=True)
    ix.add(nb, base)
    ix.preSearch(0, 0, 0, 0, 0, Index.Param(mode=SearchMode.ORIGINAL), "")
    qd = torch.from_numpy(q).cuda()
    De = torch.empty((nq, k), device="cuda")
    Ie = torch.empty((nq, k), device="cuda", dtype=torch.int64)
    torch.cuda.synchronize()
    assert lib().hb_search_noalloc(ix._h, nq, qd.data_ptr(), k, De.data_ptr(), Ie.data_ptr()) == 0
    ix.search_params.precision = precision
    if precision != Precision.FP32:
        ix.search_params.rerank_mult = 50   # 1000 candidates: wider than either arithmetic's errors here
    D, I = np.empty((nq, k), np.float32), np.empty((nq, k), np.int64)
    ix.search(nq, q, k, D, I)
    assert np.array_equal(D.view(np.uint32), De.cpu().numpy().view(np.uint32))
    assert np.array_equal(I, Ie.cpu().numpy())
