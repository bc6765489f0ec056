"""Every call that takes device arrays is ordered after torch's current stream:
on the CPU that the wait comes before the library call, on the GPU that train
and add read what torch was still producing."""
import ctypes
from types import SimpleNamespace

import numpy as np
import pytest

import harmony_b200
from harmony_b200 import Index


class Tensor:
    """What the module looks at in a CUDA tensor."""
    is_cuda, device, shape = True, "cuda:0", (2000, 16)

    def __init__(self, dtype="torch.float32"):
        self.dtype = dtype

    def data_ptr(self):
        return 256

    def is_contiguous(self):
        return True


@pytest.mark.parametrize("call", ["train", "add", "search", "train_probe_predictor"])
def test_call_waits_for_torch_first(monkeypatch, call):
    log = []

    def entry(name):
        return lambda *a: log.append(name) or 0

    ix = Index.__new__(Index)
    ix._L = SimpleNamespace(**{n: entry(n) for n in ("hb_train", "hb_add", "hb_search", "hb_train_probe_predictor",
                                                    "hb_search_params_init", "hb_get_nprobe", "hb_destroy")},
                            hb_stream=lambda h: 7)
    ix._h = ctypes.c_void_p()
    ix.param = Index.Param()
    ix.search_params = harmony_b200.SearchParams()
    ix.warmUpSearchList = ix.warmUpSearchListSize = ix.workerCount = ix.blockCount = 0
    monkeypatch.setattr(harmony_b200, "_wait_for_torch",
                        lambda stream, *arrays: log.append(("wait", stream, len([a for a in arrays if a is not None]))))
    x = Tensor()
    if call == "search":
        ix.search(2000, x, 4, Tensor(), Tensor("torch.int64"))
    else:
        getattr(ix, call)(2000, x)
    name = "hb_" + call
    waits = [e for e in log if isinstance(e, tuple)]
    assert len(waits) == 1 and waits[0][:2] == ("wait", 7) and waits[0][2] == (3 if call == "search" else 1)
    assert log.index(waits[0]) < log.index(name)


@pytest.mark.gpu
@pytest.mark.parametrize("d", [128, 100])
def test_train_and_add_read_what_torch_produces(d):
    import torch
    n, nlist = 20_000, 64
    rng = np.random.default_rng(d)
    data = torch.from_numpy(rng.integers(0, 100, size=(n, d)).astype(np.float32)).cuda()
    torch.cuda.synchronize()

    def build(late):
        x = torch.zeros((n, d), device="cuda")
        torch.cuda.synchronize()

        def produce():
            if late:
                torch.cuda._sleep(200_000_000)  # about 0.1 s
            x.copy_(data)
            if not late:
                torch.cuda.synchronize()
        ix = Index(d, nlist, 4)
        produce()
        ix.train(n, x, lite=True)
        torch.cuda.synchronize()
        x.zero_()
        torch.cuda.synchronize()
        produce()
        ix.add(n, x)
        torch.cuda.synchronize()
        return ix.centroid_codes, ix.list_sizes()

    (c0, s0), (c1, s1) = build(False), build(True)
    assert np.array_equal(c0, c1) and np.array_equal(s0, s1)
