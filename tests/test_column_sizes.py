"""State columns shorter than the ensemble are refused before the library sees them, which
takes n values from, or puts them into, every column it is given."""
from __future__ import annotations

import ctypes as C

import numpy as np
import pytest

from gazpart_b200 import api


def _context(n):
    """A context's Python side without a device behind it: the library refuses its null
    handle (GPError) whatever the columns hold."""
    ctx = object.__new__(api.Context)
    ctx._h, ctx.n = C.c_void_p(), n
    return ctx


@pytest.mark.parametrize("key", ["x", "v", "qd", "oz"])
def test_short_columns_are_refused(key):
    n = 7
    ctx = _context(n)
    for values, error in ((n, api.GPError), (n + 3, api.GPError), (n - 1, ValueError), (0, ValueError)):
        st = {k: np.zeros(values if k == key else n) for k in api.STATE_KEYS}
        with pytest.raises(error):
            ctx.put_state(st)
        with pytest.raises(error):
            ctx.download_into(st)
    # an array of the right length in half the bytes
    with pytest.raises(ValueError):
        ctx.download_into({k: np.zeros(n, np.float32 if k == key else np.float64) for k in api.STATE_KEYS})
    with pytest.raises(api.GPError):
        ctx.put_state({k: np.zeros(n, np.float32 if k == key else np.float64) for k in api.STATE_KEYS})   # converted
