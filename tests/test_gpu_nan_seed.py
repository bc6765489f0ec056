"""GPU tests of the bounded scan's seed bound over a nearest list that holds
NaN rows, with fewer than k finite ones or just enough: a NaN row is no row the
bound may count, and without k others it has none to give.  The results are the
exact scan's bit for bit."""
import numpy as np
import pytest

from harmony_b200 import Index, Precision
from tests.test_gpu_screen import NB, NLIST, P, exact, same, screened

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("d", [128, 40])
@pytest.mark.parametrize("k,finite,nan", [(10, 12, 30), (10, 5, 30), (20, 12, 30), (33, 32, 1), (33, 5, 400),
                                          (100, 60, 100), (256, 200, 80)])
def test_nearest_list_with_few_finite_rows(d, k, finite, nan):
    rng = np.random.default_rng(d + k)
    points = (rng.standard_normal((NLIST, d)) * 2).astype(np.float32)
    ix = Index(d, NLIST, P)
    ix.train(NLIST, points, lite=True)
    cent = ix.centroid_codes  # (training shuffles the points: cent[0] is list 0's)
    # Rows of every list but the first, whose rows are `finite` near ones and
    # the NaN ones (a row without a finite distance goes to list 0, at its end).
    base = (cent[rng.integers(1, NLIST, NB)] + rng.standard_normal((NB, d)) * 0.5).astype(np.float32)
    base[:finite] = cent[0] + (rng.standard_normal((finite, d)) * 0.5).astype(np.float32)
    base[finite:finite + nan, 1] = np.nan
    base = base[rng.permutation(NB)]
    q = (cent[0] + rng.standard_normal((120, d)) * 0.5).astype(np.float32)
    ix.add(NB, base)
    assert ix.list_sizes()[0] == finite + nan
    ref = exact(ix, q, k)
    assert (ref[1] >= 0).all()  # the other lists' rows are among the k nearest
    same(screened(ix, q, k), ref)
    ix.search_params.precision = Precision.BF16
    same(screened(ix, q, k), ref)
