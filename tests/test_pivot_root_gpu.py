"""The reciprocal square root of a pivot and the square root on the factor's
diagonal, over the range of normal numbers and at every place of a 64-wide tile:
blocks of 2 x 2 matrices [[x, 1], [1, y]], whose factor holds sqrt(x) and
1/sqrt(x)."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

HALF_ULP = 2.0 ** -53


@pytest.mark.parametrize("lo,hi", [(-1018, -700), (-700, -1), (-1, 1), (1, 700), (700, 1023)])
def test_pivot_roots(lo, hi):
    import torch

    from dalia_b200 import _lib

    lib, h = _lib.load(), _lib.handle()
    n, b = 2048, 64
    rng = np.random.default_rng(hi + 2000)
    x = np.ldexp(rng.uniform(1.0, 2.0, (n, b // 2)), rng.integers(lo, hi, (n, b // 2)))
    x[0, :4] = np.ldexp([1.0, np.nextafter(2.0, 1.0), np.nextafter(1.0, 2.0), 1.5], [lo, hi - 1, lo, hi - 1])
    i = 2 * np.arange(b // 2)
    D = np.zeros((n, b, b))
    D[:, i, i] = x
    D[:, i + 1, i] = D[:, i, i + 1] = 1.0
    D[:, i + 1, i + 1] = np.maximum(4.0, 4.0 / x)
    d = torch.from_numpy(D).cuda()
    L = torch.zeros(n - 1, b, b, dtype=torch.float64, device="cuda")
    one, ptr = ctypes.c_int64 * 1, ctypes.c_void_p * 1
    info = ctypes.c_int64(-1)
    _lib.check(lib.bta_pobtaf_batched(h.bind_stream(), 1, one(n), one(b), one(0), ptr(d.data_ptr()), ptr(L.data_ptr()),
                                      None, None, ctypes.byref(info)), "pobtaf")
    F = d.cpu().numpy()
    root = np.sqrt(x.astype(np.longdouble))
    # r = 1 - x y^2 carries the rounding of x y, half of which reaches y (1 + r / 2 + ..), which is rounded once more;
    # the series leaves out 5 r^3 / 16 with r below 4e-6
    recip = np.abs(F[:, i + 1, i] * root - 1)
    assert float(recip.max()) <= 1.5 * HALF_ULP + 2e-17
    # sqrt(x) = x / sqrt(x), rounded
    assert float(np.abs(F[:, i, i] / root - 1).max()) <= 2.5 * HALF_ULP + 4e-17
