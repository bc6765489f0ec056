"""GPU tests of the tensor-core nearest-centroid assignment (train, add): the
lists it builds equal the oracle's exact FP32 assignment, on sizes around its
128-row tiles and on both operand layouts (rows up to 128 floats resident,
wider rows streamed)."""
import numpy as np
import pytest

from harmony_b200 import Index

pytestmark = pytest.mark.gpu


def lists_of(ix, path):
    """{list: ids in stored order} from the saved index file."""
    ix.save_index(path)
    raw = np.fromfile(path, np.uint8)
    d, nlist = (int(v) for v in raw[:16].view(np.uint64))
    o = 8 + 8 + 4 + 4 + 8 + 8 + 8 + nlist * d * 4
    out = {}
    while o < raw.size:
        lid, n = (int(v) for v in raw[o:o + 16].view(np.uint64))
        o += 8 + 8 + 8 + 8 + 4
        out[lid] = raw[o:o + 8 * n].view(np.uint64).astype(np.int64)
        o += 8 * n + 4 * n * d + 4 * n
    return out


# add takes the tensor cores from 1.5e10 points x lists x padded dimensions
# on; n and nlist sit one off the 128-row tiles, d on both sides of the
# resident layout's limit and at an odd length.
@pytest.mark.parametrize("n,nlist,d,kind", [
    (200_001, 641, 128, "apart"), (230_000, 4097, 17, "overlap"), (180_000, 1025, 96, "far"),
    (150_000, 1000, 100, "ties"), (90_000, 383, 500, "apart"), (60_000, 513, 1000, "overlap"),
])
def test_add_equals_exact_assignment(restated, tmp_path, n, nlist, d, kind):
    rng = np.random.default_rng(n + nlist)
    spread = {"apart": 4.0, "overlap": 0.3, "far": 1.0, "ties": 1.0}[kind]
    cent = rng.standard_normal((nlist, d), dtype=np.float32) * np.float32(spread)
    if kind == "far":
        cent += np.float32(500.0)
    if kind == "ties":  # lattice points and every centroid twice: exact ties throughout
        cent = rng.integers(0, 2, size=(nlist, d)).astype(np.float32)
        cent[nlist // 2:2 * (nlist // 2)] = cent[:nlist // 2]
        x = rng.integers(0, 2, size=(n, d)).astype(np.float32)
    else:
        x = rng.standard_normal((n, d), dtype=np.float32) + cent[rng.integers(0, nlist, n)]
    ix = Index(d, nlist, 1)
    ix.train(nlist, cent, lite=True)  # nlist points: they become the centroids
    c = ix.centroid_codes
    ix.add(n, x)
    got = lists_of(ix, str(tmp_path / "a.index"))
    owner = np.full(n, -1)
    for lid, ids in got.items():
        owner[ids] = lid
    assert owner.min() >= 0 and sum(v.size for v in got.values()) == n
    # Against FP64: the assigned centroid is the nearest, to FP32 rounding of
    # the sequential sum ((d + 3) / 2^24 of the distance), for every point.
    import torch
    xt, ct = torch.from_numpy(x).cuda().double(), torch.from_numpy(c).cuda().double()
    ot = torch.from_numpy(owner).cuda()
    u = (d + 3) * 2.0 ** -24
    for s in range(0, n, 20_000):
        dist = torch.cdist(xt[s:s + 20_000], ct, compute_mode="donot_use_mm_for_euclid_dist") ** 2
        mine = dist.gather(1, ot[s:s + 20_000, None])[:, 0]
        assert bool((mine <= dist.min(1).values * (1 + 2 * u) / (1 - u) + 1e-30).all())
    # And bit for bit against the oracle's sequential FP32 loop (lowest
    # centroid on a tie) on a sample that holds every list's ends.
    pick = np.unique(np.concatenate([rng.integers(0, n, 150), [0, n - 1]] +
                                    [v[[0, -1]] for v in list(got.values())[:50]]))
    for i in pick:
        d64 = ((x[i].astype(np.float64) - c) ** 2).sum(1)
        near = np.nonzero(d64 <= d64.min() * (1 + 1e-3) + 1e-30)[0]  # every centroid the FP32 sums could put first
        dd = np.array([restated.l2(x[i], c[j]) for j in near], np.float32)
        assert owner[i] == near[dd == dd.min()].min(), i
