"""GPU tests of the BF16 scan's admission: few and many rows of a tile under the
bound, for one and for all of a warp's queries, more at once than a warp
collects, and row counts around the edges of a tile's eighths."""
import numpy as np
import pytest

from harmony_b200 import Index, Precision, SearchMode, lib

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("k", [1, 16, 17, 100])
@pytest.mark.parametrize("kind", ["near-first", "near-last", "all-near", "ties"])
@pytest.mark.parametrize("rows", [121, 128, 129, 521])
def test_admission_equals_exact_scan(rows, kind, k):
    import torch
    rng = np.random.default_rng(rows + k)
    d, nlist, nq = 40, 6, 150
    nb = nlist * rows
    cent = (rng.standard_normal((nlist, d)) * 4).astype(np.float32)
    far = np.ones(rows, np.float32)
    if kind == "near-first":
        far[16:] = 6
    elif kind == "near-last":
        far[:-16] = 6                 # every sample row of the seed is far
    base = (np.repeat(cent, rows, axis=0)
            + np.tile(far, nlist)[:, None] * rng.standard_normal((nb, d))).astype(np.float32)
    if kind == "ties":
        base = np.repeat(base[::5], 5, axis=0)[:nb].copy()
    q = (np.repeat(cent, nq // nlist, axis=0) + 0.2 * rng.standard_normal((nq, d))).astype(np.float32)
    ix = Index(d, nlist, nlist)
    ix.train(nlist, cent, lite=True)
    ix.add(nb, base)
    ix.preSearch(0, 0, 0, 0, 0, Index.Param(mode=SearchMode.ORIGINAL), "")
    qd = torch.from_numpy(q).cuda()
    De = torch.empty((nq, k), device="cuda")
    Ie = torch.empty((nq, k), device="cuda", dtype=torch.int64)
    torch.cuda.synchronize()
    assert lib().hb_search_noalloc(ix._h, nq, qd.data_ptr(), k, De.data_ptr(), Ie.data_ptr()) == 0
    ix.search_params.precision = Precision.BF16
    D, I = np.empty((nq, k), np.float32), np.empty((nq, k), np.int64)
    ix.search(nq, q, k, D, I)
    assert np.array_equal(D.view(np.uint32), De.cpu().numpy().view(np.uint32))
    assert np.array_equal(I, Ie.cpu().numpy())
