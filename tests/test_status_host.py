"""The error of a matrix that is not positive definite names its pivot, also when
several matrices share a launch (f factorises Q_c and Q_prior together)."""
import ctypes
import types

import numpy as np
import pytest

from dalia_b200 import _lib
from dalia_b200.model import SpatioTemporalModel


@pytest.mark.parametrize("info,text", [(7, "(pivot 7)"), ((1 << 40) + 301, "(pivot 301 of the launch's matrix 1)"),
                                       ((11 << 40) + 1, "(pivot 1 of the launch's matrix 11)")])
def test_status_names_the_pivot(info, text):
    def get_status(handle, out):
        ctypes.cast(out, ctypes.POINTER(ctypes.c_int64))[0] = info
        return _lib.BTA_ERR_NOT_SPD

    model = types.SimpleNamespace(lib=types.SimpleNamespace(bta_get_status=get_status),
                                  h=types.SimpleNamespace(bind_stream=lambda: None))
    with pytest.raises(np.linalg.LinAlgError) as e:
        SpatioTemporalModel.status(model)
    assert text in str(e.value)
