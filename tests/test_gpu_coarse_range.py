"""GPU test of the tensor-core coarse quantizer on values whose squared norms
overflow in their sum: its probe rows are the exact quantizer's, also where every
centroid is a candidate."""
import numpy as np
import pytest

from harmony_b200 import CoarseQuantizer, Index

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nlist,P,nq", [(6, 2, 40), (37, 37, 700), (40, 30, 5), (300, 8, 700), (300, 290, 9)])
@pytest.mark.parametrize("d,scale", [(64, 2.0e18), (100, 1.6e18), (128, 1.2e17)])
def test_probe_rows_of_huge_values(nlist, P, nq, d, scale):
    rng = np.random.default_rng(nlist + d)
    cent = rng.standard_normal((nlist, d)).astype(np.float32)
    q = cent[rng.integers(0, nlist, nq)] + rng.standard_normal((nq, d)).astype(np.float32) * np.float32(0.3)
    ix = Index(d, nlist, P)
    ix.train(nlist, cent * np.float32(scale), lite=True)
    q = q * np.float32(scale)
    ix.set_coarse_quantizer(CoarseQuantizer.EXACT)
    pe, de = ix.probe_lists(q, P)
    ix.set_coarse_quantizer(CoarseQuantizer.TENSOR)
    pt, dt = ix.probe_lists(q, P)
    assert np.array_equal(pe, pt) and np.array_equal(de, dt)
    assert (pe[:, 0] >= 0).all()  # each query's own centroid is at a finite distance
