"""GPU tests of plain FP32 searches of vectors wider than 128 dimensions whose
squares overflow in the scan while exact distances stay finite: the results
are the exact scan's bit for bit."""
import numpy as np
import pytest

from tests.test_gpu_screen import NB, NLIST, build, exact, same, screened

pytestmark = pytest.mark.gpu


# At 1.1e18 and d = 200 a query's ||q - c||^2 + ||x - c||^2 is past FLT_MAX for
# every row of its own list, the centroid distance and the distance to its own
# row are not.  "near" keeps all lists that close (every scan value of the query
# overflows), "apart" leaves the others far away.
@pytest.mark.parametrize("d,scale", [(200, 1.1e18), (129, 1.3e18), (500, 7.5e17)])
@pytest.mark.parametrize("kind", ["near", "apart"])
def test_scan_values_that_overflow(d, scale, kind):
    rng = np.random.default_rng(d)
    cent = rng.standard_normal((NLIST, d)).astype(np.float32) * np.float32(0.05 if kind == "near" else 3.0)
    base = (cent[rng.integers(0, NLIST, NB)] + rng.standard_normal((NB, d))).astype(np.float32)
    q = base[::311][:120] + np.float32(0.01)
    s = np.float32(scale)
    base, q, cent = base * s, q * s, cent * s
    ix = build(d, base, cent)
    for k in (1, 10, 100):
        ref = exact(ix, q, k)
        assert (ref[1][:, 0] >= 0).all()  # every query has a row at a finite distance
        same(screened(ix, q, k), ref)
