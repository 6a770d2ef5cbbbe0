"""Task and tile lists of new launch shapes reach the device before any kernel
reads them, also on a stream that does not wait for the legacy stream."""
import ctypes
import glob
import os
import re

import numpy as np
import pytest

from oracle import bta_ref

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "dalia_b200", "csrc")


def test_no_upload_is_ordered_by_the_legacy_stream_alone():
    """cudaMemcpy to the device orders nothing on a non-blocking stream, and from
    pageable memory it may return before the bytes have arrived."""
    found = []
    for path in sorted(glob.glob(os.path.join(CSRC, "*.cu*"))):
        text = re.sub(r"//[^\n]*", "", open(path).read())
        for call in re.findall(r"cudaMemcpy\s*\(([^;]*)\)", text):
            if "HostToDevice" in call or "cudaMemcpyDefault" in call:
                found.append((os.path.basename(path), " ".join(call.split())))
    assert not found


@pytest.mark.gpu
@pytest.mark.parametrize("precision", ["fp64", "i8slice"])
def test_new_shapes_on_a_stream_of_their_own(precision):
    import torch

    from dalia_b200 import _lib

    lib = _lib.load()
    prec = {"fp64": _lib.BTA_PREC_FP64, "i8slice": _lib.BTA_PREC_I8SLICE}[precision]
    side = torch.cuda.Stream()  # non-blocking
    for n, b, a in [(5, 211, 3), (7, 130, 0), (3, 390, 70)]:
        mats = bta_ref.random_bta(n, b, max(a, 1), np.random.default_rng(b))
        if a == 0:
            mats = mats[:2] + (np.zeros((n, 0, b)), np.zeros((0, 0)))
        src = [torch.from_numpy(np.ascontiguousarray(m)).cuda() for m in mats]
        got = []
        for stream in (torch.cuda.current_stream(), side):
            stream.wait_stream(torch.cuda.current_stream())
            with torch.cuda.stream(stream):
                h = _lib.Handle()  # no list of any shape yet
                w = [x.clone() for x in src]
                args = [(ctypes.c_int64 * 1)(v) for v in (n, b, a)]
                args += [(ctypes.c_void_p * 1)(x.data_ptr() if x.numel() else None) for x in w]
                info = ctypes.c_int64(-1)
                _lib.check(lib.bta_pobtaf_batched_ex(h.bind_stream(), 1, *args, ctypes.byref(info), prec), "pobtaf")
                _lib.check(lib.bta_pobtasi_batched_ex(h.bind_stream(), 1, *args, prec), "pobtasi")
                _lib.check(lib.bta_get_status(h.bind_stream(), ctypes.byref(info)), "status")
            stream.synchronize()
            got.append(w)
        for x, y in zip(*got):
            assert x.numel() == 0 or float((x - y).norm() / x.norm()) <= 1e-12
