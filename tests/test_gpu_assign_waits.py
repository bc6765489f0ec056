"""GPU tests of train and add on the tensor-core assignment, and of its waits
giving up: the calls then make the assignments with the exact kernel, so what
they build is the same byte for byte.  Rows up to 128 floats stay resident in
the kernel, wider ones stream."""
import numpy as np
import pytest

from harmony_b200 import Index

pytestmark = pytest.mark.gpu


def build(x, nlist, path, budget, lite):
    """(centroids, saved bytes, names of the assignment kernels that ran in train and in add)."""
    ix = Index(x.shape[1], nlist, 1)
    ix.set_wait_budget(budget)
    ix.profile(True)
    ix.train(x.shape[0], x, lite=lite)
    in_train = {n for n in ix.profile_read() if n.startswith("assign")}
    ix.add(x.shape[0], x)
    in_add = {n for n in ix.profile_read() if n.startswith("assign")}
    ix.profile(False)
    ix.save_index(path)
    return ix.centroid_codes, np.fromfile(path, np.uint8), in_train, in_add


# Sizes from which train (5e8 points x lists x padded dimensions of its sample)
# and add (5e9) take the tensor cores, off the 128-row tiles; all train on a
# sample (more than 256 points a list).
@pytest.mark.parametrize("n,nlist,d,lite", [(200_001, 385, 100, True), (60_001, 129, 700, False),
                                            (150_000, 271, 128, False)])
def test_wait_that_gives_up(n, nlist, d, lite, tmp_path):
    rng = np.random.default_rng(n + d)
    # Whole numbers: the centroid sums are exact in any order.
    x = rng.integers(0, 64, size=(nlist, d))[rng.integers(0, nlist, n)] + rng.integers(-8, 9, size=(n, d))
    x = x.astype(np.float32)
    c0, b0, t0, a0 = build(x, nlist, str(tmp_path / "tc.index"), 0, lite)
    assert t0 == {"assign_tc"} and a0 == {"assign_tc"}
    c1, b1, t1, a1 = build(x, nlist, str(tmp_path / "ex.index"), 1, lite)
    assert t1 == {"assign_tc", "assign_exact"} and a1 == {"assign_tc", "assign_exact"}
    assert np.array_equal(c0, c1) and np.array_equal(b0, b1)


@pytest.mark.parametrize("d", [100, 200])
@pytest.mark.parametrize("kind", ["nonfinite", "huge", "tiny", "ties", "far"])
def test_values_outside_the_bound(kind, d, tmp_path):
    """Points and centroids that the tensor cores may not decide: both routes
    build the same."""
    rng = np.random.default_rng(d)
    n, nlist = 120_001, 385
    x = rng.integers(0, 64, size=(nlist, d))[rng.integers(0, nlist, n)] + rng.integers(-8, 9, size=(n, d))
    x = x.astype(np.float32)
    if kind == "nonfinite":
        x[::1777, 3], x[::2991, 5], x[::3331, 7], x[::4001] = np.nan, np.inf, -np.inf, 3e38
    elif kind in ("huge", "tiny"):
        x *= np.float32(2.0 ** (56 if kind == "huge" else -70))
    elif kind == "ties":
        x = rng.integers(0, 2, size=(500, d)).astype(np.float32)[rng.integers(0, 500, n)]
    else:
        x += np.float32(2.0 ** 17)
    c0, b0, t0, a0 = build(x, nlist, str(tmp_path / "tc.index"), 0, True)
    assert t0 == {"assign_tc"} and "assign_tc" in a0
    c1, b1, t1, a1 = build(x, nlist, str(tmp_path / "ex.index"), 1, True)
    assert t1 == {"assign_tc", "assign_exact"}
    assert np.array_equal(c0, c1, equal_nan=True) and np.array_equal(b0, b1)
