"""Calls on a GPU that is nearly full do with the workspace that one block
column needs."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

MB = 1 << 20


def _bta(n, b, a, seed):
    import torch

    g = torch.Generator(device="cuda").manual_seed(seed)
    rnd = lambda *s: torch.randn(*s, dtype=torch.float64, device="cuda", generator=g)  # noqa: E731
    D = rnd(n, b, b) / (4 * b)
    D = D + D.transpose(1, 2) + 4 * torch.eye(b, dtype=torch.float64, device="cuda")
    return [D.contiguous(), rnd(max(n - 1, 0), b, b) / (2 * b), rnd(n, a, b) / (4 * b),
            n * torch.eye(a, dtype=torch.float64, device="cuda")]


def _args(n, b, a, m):
    one, ptr = ctypes.c_int64 * 1, ctypes.c_void_p * 1
    return [1, one(n), one(b), one(a)] + [ptr(x.data_ptr() if x.numel() else None) for x in m]


def _fill(leave):
    """Takes the GPU's memory but for `leave` bytes."""
    import torch

    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    free, _ = torch.cuda.mem_get_info()
    return torch.empty(max(0, free - leave), dtype=torch.uint8, device="cuda")


def _err(got, ref):
    return max(float((x - y).norm() / y.norm()) for x, y in zip(got, ref) if y.numel())


def test_factorisation_takes_at_most_a_quarter_of_what_is_free(monkeypatch):
    import torch

    from dalia_b200 import _lib

    monkeypatch.delenv("DALIA_B200_PANEL_PERSIST", raising=False)
    lib = _lib.load()
    n, b, a = 8000, 64, 2  # tile inverses of all block columns: 250 MB
    m = _bta(n, b, a, 1)
    got, ref = [x.clone() for x in m], [x.clone() for x in m]
    info = ctypes.c_int64(-1)
    wide = _lib.Handle()
    _lib.check(lib.bta_pobtaf_batched(wide.bind_stream(), *_args(n, b, a, ref), ctypes.byref(info)), "pobtaf")
    assert wide.workspace_bytes() > 200 * MB
    del wide
    h = _lib.Handle()
    filler = _fill(600 * MB)
    _lib.check(lib.bta_pobtaf_batched(h.bind_stream(), *_args(n, b, a, got), ctypes.byref(info)), "pobtaf")
    held = h.workspace_bytes()
    del filler
    torch.cuda.empty_cache()
    assert held < 150 * MB
    # one factorisation in two launch orders: the same sums
    assert _err(got, ref) <= 1e-12


@pytest.mark.parametrize("leave", [110, 34])
def test_selected_inversion_in_parts(leave):
    """8-bit slices of blocks of 1000 with supplied inverses: the digit images of
    a group of five block columns take 160 MB, those of a step's two launches
    32, those of one product 16."""
    import torch

    from dalia_b200 import _lib

    lib = _lib.load()
    n, b, a = 6, 1000, 0
    m = _bta(n, b, a, 2)
    info = ctypes.c_int64(-1)
    h = _lib.handle()
    _lib.check(lib.bta_pobtaf_batched(h.bind_stream(), *_args(n, b, a, m), ctypes.byref(info)), "pobtaf")
    V = torch.empty_like(m[0])
    one, ptr = ctypes.c_int64 * 1, ctypes.c_void_p * 1
    _lib.check(lib.bta_block_inverses(h.bind_stream(), 1, one(n), one(b), ptr(m[0].data_ptr()), ptr(V.data_ptr())),
               "inverses")
    got, ref = [x.clone() for x in m], [x.clone() for x in m]

    def run(h, w):
        rc = lib.bta_pobtasi_batched_v(h.bind_stream(), *_args(n, b, a, w), ptr(V.data_ptr()), _lib.BTA_PREC_I8SLICE)
        return rc or lib.bta_get_status(h.bind_stream(), ctypes.byref(info))

    wide, h = _lib.Handle(), _lib.Handle()
    assert run(wide, ref) == 0
    del wide
    filler = _fill(leave * MB)
    rc = run(h, got)
    del filler, h
    torch.cuda.empty_cache()
    assert rc == 0
    # the same digits and the same integer sums, launched in other groups
    assert _err(got, ref) <= 1e-12


def test_sweeps_without_room_for_block_inverses():
    """20 blocks of 1000 go through block inverses of 160 MB, or where those
    cannot be had through the tile sweep, which needs 10 MB."""
    import torch

    from dalia_b200 import _lib

    lib = _lib.load()
    n, b, a = 20, 1000, 3
    m = _bta(n, b, a, 3)
    info = ctypes.c_int64(-1)
    _lib.check(lib.bta_pobtaf_batched(_lib.handle().bind_stream(), *_args(n, b, a, m), ctypes.byref(info)), "pobtaf")
    rhs = torch.ones(n * b + a, dtype=torch.float64, device="cuda")
    xs, held = [], []
    for leave in (None, 60):
        h = _lib.Handle()
        x = rhs.clone()
        filler = None if leave is None else _fill(leave * MB)
        rc = 0
        for trans in (0, 1):
            rc = rc or lib.bta_pobtas_batched(h.bind_stream(), *_args(n, b, a, m),
                                              (ctypes.c_void_p * 1)(x.data_ptr()), trans)
        rc = rc or lib.bta_get_status(h.bind_stream(), ctypes.byref(info))
        held.append(h.workspace_bytes())
        del filler, h
        torch.cuda.empty_cache()
        assert rc == 0
        xs.append(x)
    assert held[0] > 100 * MB > held[1]
    # well-conditioned (eigenvalues near 4): rounding of b terms
    assert _err([xs[1]], [xs[0]]) <= 1e-12
