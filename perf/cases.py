"""The work a user of this package has it do, as measurable cases.

Two kinds of call, both through the public ``Index``:

  search  ``Index.search`` on an index that is already filled: the three
          arithmetics (FP32, BF16, FP8), the pruned list search, fixed and
          per-query nprobe, host and device arrays, ordinary and CUDA-graph
          calls, one query up to ten thousand.
  build   ``Index.train`` + ``Index.add``.

The data are Gaussian mixtures of the shapes this repository benchmarks (see
``harmony_b200/datasets.py``), drawn on the GPU from the seed.  A search
index takes the mixture's centres as its coarse centroids: training on
exactly nlist points leaves those points as the centroids, which is how a
program brings in centroids that were trained elsewhere.  Build cases train
in earnest.
"""
import math

import numpy as np
import torch

from harmony_b200 import Index, Precision, SearchMode

# Value distributions: (kind of centres, their spread, noise, list-size skew).
#   int8bit  integers in [0, 255] (sift-like bytes)
#   apart    unit-variance components around N(0, 4^2) centres
#   overlap  unit-variance components around N(0, 0.68^2) centres
#   decay    per-dimension scale (j + 1)^-0.6
#   zipf     apart, with component weights proportional to rank^-1.1


def search_case(name, nb, d, nlist, nprobe, k, nq, precision="fp32", data="apart", mode="original", host=False,
                graph=False, ragged=False, rerank=2):
    c = dict(kind="search", nb=nb, d=d, nlist=nlist, nprobe=nprobe, k=k, nq=nq, precision=precision, data=data,
             mode=mode, host=host, graph=graph, ragged=ragged, rerank=rerank)
    if name:
        c["name"] = name
    return c


def build_case(name, nb, d, nlist, data="apart", lite=False):
    c = dict(kind="build", nb=nb, d=d, nlist=nlist, data=data, lite=lite)
    if name:
        c["name"] = name
    return c


def listed():
    return [
        # An interactive lookup: one query from host memory on the small
        # sift10k-shaped index, default arithmetic.  Launches and latency.
        search_case("one-fp32-10k", 10_000, 128, 100, 10, 10, 1, data="int8bit", host=True),
        # The same index searched the way the reference's own driver does it:
        # a batch of 100 host queries, pruning against warm-up heap tops.
        search_case("pruned-100-10k", 10_000, 128, 100, 10, 10, 100, data="int8bit", mode="divide_ivf", host=True),
        # One query against a large, skewed index: serving latency, BF16 scan,
        # the batch replayed as a CUDA graph.
        search_case("one-bf16-graph-4m", 4_000_000, 96, 4096, 64, 10, 1, "bf16", "zipf", graph=True),
        # A mid-sized arrival batch on that index, every query with its own
        # nprobe (4 .. 256).
        search_case("ragged-777-bf16-4m", 4_000_000, 96, 4096, 256, 10, 777, "bf16", "zipf", graph=True, ragged=True),
        # A small ordinary batch with odd sizes, FP32, host arrays.
        search_case("batch-33-fp32-300k", 300_001, 100, 500, 17, 20, 33, host=True),
        # Offline bulk search, default arithmetic: 10,000 queries, k = 100.
        search_case("bulk-fp32-1m", 1_000_000, 128, 1024, 32, 100, 10_000),
        # The same bulk search with the BF16 scan at a wider nprobe.
        search_case("bulk-bf16-1m", 1_000_000, 128, 1024, 64, 100, 10_000, "bf16"),
        # Wide vectors (500 dimensions), the three arithmetics.
        search_case("wide-fp32-270k", 270_000, 500, 512, 32, 100, 2_000, data="decay"),
        search_case("wide-bf16-270k", 270_000, 500, 512, 32, 100, 5_000, "bf16", "decay", rerank=4),
        search_case("wide-fp8-270k", 270_000, 500, 512, 32, 100, 5_000, "fp8", "decay", rerank=4),
        # The headline index: 10M vectors, 10,000 queries at nprobe 40.
        search_case("bulk-bf16-10m", 10_000_000, 128, 4096, 40, 10, 10_000, "bf16", "overlap"),
        # Building an index: k-means training, then adding the vectors.
        build_case("build-1m", 1_000_000, 128, 1024),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """A case of the same ranges: 10k .. 3M vectors, 16 .. 512 dimensions,
    1 .. 10,000 queries, k 1 .. 100, nprobe 1 .. 128 (or all of the lists)."""
    d = rng.choice([_log_int(rng, 16, 128), 128, 96, _log_int(rng, 129, 512)])
    nb = _log_int(rng, 10_000, min(3_000_000, 256_000_000 // d))
    nlist = max(16, min(4096, int(math.sqrt(nb) * rng.uniform(0.5, 2.0))))
    if rng.random() < 0.2:
        # 1 .. 256 training points per centroid are used, so this bounds the
        # training of the drawn builds by the listed ones.
        nb = min(nb, 1_000_000, 128_000_000 // d)
        return build_case(None, nb, d, min(nlist, 1024, nb // 8), rng.choice(["apart", "overlap"]),
                          rng.random() < 0.5)
    precision = rng.choice(["fp32", "fp32", "bf16", "bf16", "fp8"])
    mode = "divide_ivf" if precision == "fp32" and rng.random() < 0.15 else "original"
    nprobe = _log_int(rng, 1, min(nlist, 128))
    k = _log_int(rng, 1, 100)
    nq = _log_int(rng, 1, 10_000)
    # At most the pairs x dimensions of the bulk searches.
    pairs = nq * nprobe * (nb / nlist) * d
    cap = 1.5e10 if precision == "fp32" else 6e10
    if pairs > cap:
        nq = max(1, int(nq * cap / pairs))
    return search_case(None, nb, d, nlist, nprobe, k, nq, precision,
                       rng.choice(["apart", "overlap", "zipf", "decay"] + (["int8bit"] if nb <= 300_000 else [])),
                       mode, host=rng.random() < 0.3, graph=mode == "original" and rng.random() < 0.3,
                       ragged=mode == "original" and rng.random() < 0.2, rerank=rng.choice([2, 4]))


def _data(case, seed):
    """(vectors, centres, queries, per-query nprobe or None) on the GPU."""
    g = torch.Generator(device="cuda").manual_seed(seed * 7919 + 17)
    d, nb, nc, kind = case["d"], case["nb"], case["nlist"], case["data"]
    nq = case.get("nq", 0)
    scale = torch.ones(d, device="cuda")
    noise, w = 1.0, None
    if kind == "int8bit":
        centres = torch.rand((nc, d), generator=g, device="cuda") * 192.0 + 32.0
        noise = 20.0
    else:
        spread = 0.68 if kind == "overlap" else 4.0
        if kind == "decay":
            scale = (torch.arange(d, device="cuda") + 1.0) ** -0.6
        centres = torch.randn((nc, d), generator=g, device="cuda") * spread * scale
        if kind == "zipf":
            w = (torch.arange(nc, device="cuda") + 1.0) ** -1.1

    def mix(n):
        out = torch.empty((n, d), device="cuda")
        for s in range(0, n, 1 << 21):
            e = min(n, s + (1 << 21))
            if w is None:
                comp = torch.randint(0, nc, (e - s,), generator=g, device="cuda")
            else:
                comp = torch.multinomial(w, e - s, replacement=True, generator=g)
            torch.randn((e - s, d), generator=g, device="cuda", out=out[s:e])
            out[s:e].mul_(noise * scale).add_(centres[comp])
            if kind == "int8bit":
                out[s:e].round_().clamp_(0, 255)
        return out

    x, q = mix(nb), mix(nq) if nq else None
    npq = None
    if case.get("ragged"):
        npq = torch.randint(min(4, case["nprobe"]), case["nprobe"] + 1, (nq,), generator=g, device="cuda",
                            dtype=torch.int32)
    return x, centres, q, npq


def prepare(case, seed):
    x, centres, q, npq = _data(case, seed)
    if case["kind"] == "build":
        return {"case": case, "x": x}
    ix = Index(case["d"], case["nlist"], case["nprobe"])
    ix.train(case["nlist"], centres.contiguous(), lite=True)
    ix.add(case["nb"], x)
    mode = SearchMode.DIVIDE_IVF if case["mode"] == "divide_ivf" else SearchMode.ORIGINAL
    ix.preSearch(0, 0, 0, 0, 0, Index.Param(mode=mode, pruning=mode == SearchMode.DIVIDE_IVF), "")
    sp = ix.search_params
    sp.precision = {"fp32": Precision.FP32, "bf16": Precision.BF16, "fp8": Precision.FP8}[case["precision"]]
    sp.rerank_mult, sp.use_graph = case["rerank"], case["graph"]
    nq, k = case["nq"], case["k"]
    if npq is not None:
        sp.nprobe_per_query, sp.max_nprobe = npq, case["nprobe"]
    if case["host"]:
        q = q.cpu().numpy()
        sp.nprobe_per_query = None if npq is None else npq.cpu().numpy()
        D, I = np.empty((nq, k), np.float32), np.empty((nq, k), np.int64)
    else:
        D = torch.empty((nq, k), device="cuda")
        I = torch.empty((nq, k), device="cuda", dtype=torch.int64)
    return {"case": case, "ix": ix, "q": q, "D": D, "I": I}


def run(state):
    case = state["case"]
    if case["kind"] == "build":
        ix = Index(case["d"], case["nlist"], 1)
        ix.train(case["nb"], state["x"], lite=case["lite"])
        ix.add(case["nb"], state["x"])
        return {"centroids": ix.centroid_codes, "sizes": ix.list_sizes()}
    state["ix"].search(case["nq"], state["q"], case["k"], state["D"], state["I"])
    return {"D": state["D"], "I": state["I"]}


def work(case):
    nb, d, nlist = case["nb"], case["d"], case["nlist"]
    if case["kind"] == "build":
        m = min(nb, 256 * nlist)
        niter = 2 if case["lite"] else 20
        # Training reads its sample and adds up its rows once per iteration;
        # add reads every vector and writes it with its id and norm.
        return {"bytes": 4.0 * d * (niter * m + 2 * nb) + 12.0 * nb,
                "flops": 2.0 * d * nlist * (niter * m + nb)}
    nq, k = case["nq"], case["k"]
    P = (case["nprobe"] + min(4, case["nprobe"])) / 2 if case["ragged"] else case["nprobe"]
    lists = nlist * (1.0 - (1.0 - min(1.0, P / nlist)) ** nq)
    width = {"fp32": 4.0, "bf16": 2.0, "fp8": 1.0}[case["precision"]]
    return {"bytes": 4.0 * d * (nlist + nq) + lists * nb / nlist * d * width + 12.0 * nq * k,
            "flops": 2.0 * d * (nq * nlist + nq * P * nb / nlist)}


def exact(case, seed):
    """Distances of the same search in 64 bits: the nprobe nearest centres of
    each query, then the k nearest vectors assigned to them.  Ids have no
    64-bit value; trained centroids come out of an iteration whose every
    assignment feeds the next, so they have none either."""
    if case["kind"] == "build" or case["nq"] * case["nb"] > 2e10:
        return None
    x, centres, q, npq = _data(case, seed)
    nb, nq, k, P = case["nb"], case["nq"], case["k"], case["nprobe"]
    c64 = centres.double()
    cn = (c64 * c64).sum(1)
    owner = torch.empty(nb, device="cuda", dtype=torch.int64)
    step = max(1, (1 << 28) // case["nlist"])
    for s in range(0, nb, step):
        owner[s:s + step] = (cn - 2.0 * (x[s:s + step].double() @ c64.T)).argmin(1)
    D = torch.empty((nq, k), device="cuda", dtype=torch.float64)
    step = max(1, (1 << 29) // nb)
    for s in range(0, nq, step):
        qs = q[s:s + step].double()
        order = (cn - 2.0 * (qs @ c64.T)).topk(P, dim=1, largest=False).indices
        on = torch.zeros((qs.shape[0], case["nlist"]), device="cuda", dtype=torch.bool)
        keep = torch.ones_like(order, dtype=torch.bool)
        if npq is not None:
            keep = torch.arange(P, device="cuda")[None, :] < npq[s:s + step, None]
        on.scatter_(1, order, keep)
        best = torch.full((qs.shape[0], k), math.inf, device="cuda", dtype=torch.float64)
        rows = 1 << 19
        for b in range(0, nb, rows):
            xb = x[b:b + rows].double()
            v = (qs * qs).sum(1)[:, None] + (xb * xb).sum(1)[None, :] - 2.0 * (qs @ xb.T)
            v.masked_fill_(~on[:, owner[b:b + rows]], math.inf)
            top = v.topk(min(k, v.shape[1]), dim=1, largest=False).values
            best = torch.cat([best, top], 1).topk(k, dim=1, largest=False).values
        D[s:s + step] = best.clamp_min(0.0)
    none = float(np.finfo(np.float32).max)
    D = torch.where(torch.isinf(D), torch.full_like(D, none), D)
    return {"D": D.cpu().numpy() if case["host"] else D, "I": None}
