"""GPU tests of FP32 searches that go through the bounded scan: the results are
the exact scan's bit for bit (hb_search_noalloc always runs the exact
kernels), for every form of call the route accepts and for values outside the
error bound's range."""
import numpy as np
import pytest

from harmony_b200 import Index, SearchMode, datasets, lib

pytestmark = pytest.mark.gpu
NB, NLIST, P = 40_000, 48, 16


def build(d, base, cent=None):
    ix = Index(d, NLIST, P)
    if cent is None:
        ix.train(base.shape[0], base)
    else:
        ix.train(NLIST, cent, lite=True)
    ix.add(base.shape[0], base)
    return ix


def screened(ix, q, k, mode=SearchMode.ORIGINAL, graph=False, npq=None):
    ix.preSearch(0, 0, 0, 0, 0, Index.Param(mode=mode), "")
    sp = ix.search_params
    sp.use_graph, sp.nprobe_per_query, sp.max_nprobe = graph, npq, P if npq is not None else 0
    D, I = np.empty((q.shape[0], k), np.float32), np.empty((q.shape[0], k), np.int64)
    ix.profile(True)
    ix.profile_read()
    ix.search(q.shape[0], q, k, D, I)
    names = set(ix.profile_read())
    ix.profile(False)
    sp.use_graph, sp.nprobe_per_query, sp.max_nprobe = False, None, 0
    assert graph or names & {"scan_bf16", "cand_scan"}, names  # the route under test ran
    return D, I


def exact(ix, q, k):
    import torch
    qd = torch.from_numpy(np.ascontiguousarray(q)).cuda()
    D = torch.empty((q.shape[0], k), device="cuda")
    I = torch.empty((q.shape[0], k), device="cuda", dtype=torch.int64)
    torch.cuda.synchronize()
    assert lib().hb_search_noalloc(ix._h, q.shape[0], qd.data_ptr(), k, D.data_ptr(), I.data_ptr()) == 0, \
        lib().hb_last_error()
    return D.cpu().numpy(), I.cpu().numpy()


def same(a, b):
    assert np.array_equal(a[0].view(np.uint32), b[0].view(np.uint32)) and np.array_equal(a[1], b[1])


@pytest.mark.parametrize("d,k", [(128, 1), (128, 16), (128, 17), (96, 100), (33, 10), (65, 256)])
def test_equals_exact_scan(d, k):
    base, q = datasets.config2(seed=d + k, nb=NB, nq=131, d=d, ncomp=60)
    ix = build(d, base)
    ref = exact(ix, q, k)
    same(screened(ix, q, k), ref)
    same(screened(ix, q, k, mode=SearchMode.DIVIDE_IVF), ref)  # pruning off: the plain scan
    for _ in range(2):  # captured, then replayed
        same(screened(ix, q, k, graph=True), ref)
    npq = (np.arange(131) % (P + 1)).astype(np.int32)
    D, I = screened(ix, q, k, npq=npq)
    same((D[npq == P], I[npq == P]), (ref[0][npq == P], ref[1][npq == P]))
    assert (I[npq == 0] == -1).all()
    assert ix.bf16_stats()["queries"] == 0 and ix.bf16_fallbacks() == 0  # those report BF16 searches


@pytest.mark.parametrize("d,k", [(129, 1), (256, 20), (500, 100), (1000, 30)])
def test_wide_equals_exact_scan(d, k):
    """d > 128: the candidate matrix, every row the bound allows re-ranked."""
    nq = 40
    base, q = datasets.config3(seed=d + k, nb=NB, nq=nq, d=d, ncomp=60)
    ix = build(d, base)
    ref = exact(ix, q, k)
    same(screened(ix, q, k), ref)
    for _ in range(2):
        same(screened(ix, q, k, graph=True), ref)
    npq = (np.arange(nq) % (P + 1)).astype(np.int32)
    D, I = screened(ix, q, k, npq=npq)
    same((D[npq == P], I[npq == P]), (ref[0][npq == P], ref[1][npq == P]))
    assert (I[npq == 0] == -1).all()


@pytest.mark.parametrize("d", [64, 200])
@pytest.mark.parametrize("kind", ["nonfinite", "huge", "tiny", "ties", "far", "outlier"])
def test_values_outside_the_bound(kind, d):
    rng = np.random.default_rng(3)
    cent = (rng.standard_normal((NLIST, d)) * 3).astype(np.float32)
    base = (cent[rng.integers(0, NLIST, NB)] + rng.standard_normal((NB, d))).astype(np.float32)
    q = base[::311][:120] + np.float32(0.01)
    if kind == "nonfinite":
        base[::777, 3], base[::991, 5] = np.nan, np.inf
        q[5, 1], q[6, 2], q[7] = np.nan, np.inf, 3e38
    elif kind in ("huge", "tiny"):
        s = np.float32(1e17 if kind == "huge" else 1e-21)
        base, q, cent = base * s, q * s, cent * s
    elif kind == "ties":
        base = rng.integers(0, 2, size=(NB, d)).astype(np.float32)
        base[NB // 2:] = base[:NB // 2]
        cent, q = base[:NLIST].copy(), base[::311][:120].copy()
    elif kind == "far":
        base, q, cent = base + np.float32(3000), q + np.float32(3000), cent + np.float32(3000)
    else:
        base[17] *= np.float32(1e16)  # one list of unbounded radius
    ix = build(d, base, cent)
    for k in (10, 100):
        same(screened(ix, q, k), exact(ix, q, k))


def test_wait_budget_and_small_calls_stay_fp32():
    """The wait budget is the BF16 scan's; a call under the pair rule takes
    the exact scan."""
    base, q = datasets.config2(seed=9, nb=NB, nq=200, d=128, ncomp=60)
    ix = build(128, base)
    ref = exact(ix, q, 10)
    ix.set_wait_budget(300)
    same(screened(ix, q, 10), ref)
    ix.set_wait_budget(0)
    ix.nprobe = 1
    ref = exact(ix, q[:3], 10)
    D, I = np.empty((3, 10), np.float32), np.empty((3, 10), np.int64)
    ix.profile(True)
    ix.search(3, q[:3], 10, D, I)
    assert "scan_exact" in ix.profile_read()
    same((D, I), ref)
