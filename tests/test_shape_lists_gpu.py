"""A handle's task and tile lists past their limit: shapes come and go, and a
list that a captured graph reads stays."""
import ctypes

import numpy as np
import pytest

from golden_util import rel
from oracle import bta_ref

pytestmark = pytest.mark.gpu

SHAPES = [(4, 130, 3), (3, 200, 0), (6, 65, 70), (2, 257, 1)]


def _problem(n, b, a):
    import torch

    m = bta_ref.random_bta(n, b, max(a, 1), np.random.default_rng(n + b))
    if a == 0:
        m = m[:2] + (np.zeros((n, 0, b)), np.zeros((0, 0)))
    return m, [torch.from_numpy(np.ascontiguousarray(x)).cuda() for x in m]


def _run(h, n, b, a, w, prec):
    from dalia_b200 import _lib

    lib = _lib.load()
    args = [1] + [(ctypes.c_int64 * 1)(v) for v in (n, b, a)]
    args += [(ctypes.c_void_p * 1)(x.data_ptr() if x.numel() else None) for x in w]
    _lib.check(lib.bta_pobtaf_batched_ex(h.bind_stream(), *args, None, prec), "pobtaf")
    _lib.check(lib.bta_pobtasi_batched_ex(h.bind_stream(), *args, prec), "pobtasi")


def _close(n, b, a, m, w):
    dense = bta_ref.bta_to_dense(*(m if a else m[:2] + (np.zeros((n, 1, b)), np.eye(1))))
    S = bta_ref.dense_to_bta(np.linalg.inv(dense), n, b, max(a, 1))
    for got, ref in zip(w, S):
        if got.numel():  # digits of 2^-47 of the row maxima, sixteen products of b terms a step; 64-bit sums are nearer
            assert rel(got.cpu().numpy(), ref) < 16 * b * 2.0 ** -47


@pytest.mark.parametrize("prec", ["fp64", "i8slice"])
def test_shapes_past_the_limit(prec, monkeypatch):
    from dalia_b200 import _lib

    monkeypatch.setenv("DALIA_B200_LIST_BYTES", "3000")  # one or two lists
    h = _lib.Handle()
    p = {"fp64": _lib.BTA_PREC_FP64, "i8slice": _lib.BTA_PREC_I8SLICE}[prec]
    for n, b, a in SHAPES + SHAPES:
        m, w = _problem(n, b, a)
        _run(h, n, b, a, w, p)
        _close(n, b, a, m, w)


@pytest.mark.parametrize("prec", ["fp64", "i8slice"])
def test_a_captured_graph_keeps_its_lists(prec, monkeypatch):
    import torch

    from dalia_b200 import _lib

    monkeypatch.setenv("DALIA_B200_TUNE", "0")
    monkeypatch.setenv("DALIA_B200_LIST_BYTES", "3000")
    h = _lib.Handle()
    p = {"fp64": _lib.BTA_PREC_FP64, "i8slice": _lib.BTA_PREC_I8SLICE}[prec]
    n, b, a = 5, 300, 4  # needs more workspace than the others: theirs fits
    m, src = _problem(n, b, a)
    w = [x.clone() for x in src]
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        monkeypatch.setenv("DALIA_B200_LIST_BYTES", "100000000")
        _run(h, n, b, a, w, p)  # its lists and workspace are there before the capture
    side.synchronize()
    monkeypatch.setenv("DALIA_B200_LIST_BYTES", "3000")
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=side):
        for x, y in zip(w, src):
            x.copy_(y)
        _run(h, n, b, a, w, p)
    torch.cuda.synchronize()
    for s in SHAPES:  # new shapes take the place of what may go
        m2, w2 = _problem(*s)
        _run(h, *s, w2, p)
        _close(*s, m2, w2)
    for x in w:
        x.zero_()
    graph.replay()
    torch.cuda.synchronize()
    _close(n, b, a, m, w)
