"""The sweep's launch candidates are launches that differ: a CTA per SM, a CTA
per two SMs."""
import ctypes

import pytest

pytestmark = pytest.mark.gpu


def test_the_tuner_tries_two_sweep_launches(monkeypatch):
    import torch

    from dalia_b200 import _lib

    monkeypatch.delenv("DALIA_B200_TUNE_FORCE", raising=False)
    monkeypatch.delenv("DALIA_B200_TUNE", raising=False)
    lib, h = _lib.load(), _lib.handle()
    n, b = 3, 1237  # a shape of its own
    V = (2 * torch.eye(b, dtype=torch.float64, device="cuda")).expand(n, b, b).contiguous()
    L = torch.zeros(n - 1, b, b, dtype=torch.float64, device="cuda")
    x = torch.ones(n * b, dtype=torch.float64, device="cuda")
    one, ptr = ctypes.c_int64 * 1, ctypes.c_void_p * 1
    for _ in range(5):  # two candidates tried twice, then the decision
        _lib.check(lib.bta_pobtas_inv_batched(h.bind_stream(), 1, one(n), one(b), one(0), ptr(L.data_ptr()), None, None,
                                              ptr(V.data_ptr()), ptr(x.data_ptr()), 0), "sweep")
    torch.cuda.synchronize()
    assert bool((x == 32.0).all())
    line, = [ln for ln in _lib.tune_report() if ln.startswith("sweep|") and ":1,0,1237,1237,3 " in ln]
    assert len(line.split("ms=")[1].split(",")) == 2
