"""Bodies at the walls under the plain and the speculative integrate, which are kernels of
their own: both take the predictor's position with the same rounding, so they see the same
bodies meet their wall and end with the same bits."""
from __future__ import annotations

import numpy as np
import pytest

from _cases import case
from gazpart_b200 import api

pytestmark = pytest.mark.gpu
GRIDS = {"gather": 296, "integrate": 592, "bin": 592, "search": 592}


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_same_bits(precision):
    setup, fn, refs, st = case("poly")
    st = {k: np.array(v, copy=True) for k, v in st.items()}
    n = st["x"].size
    rmax = np.maximum(st["emaj"], st["emaj"] / st["apr"])
    gap = np.random.default_rng(7).uniform(0.2, 1.6, n) * rmax
    st["x"] = np.where(np.arange(n) % 2 == 0, gap, setup.lx - gap)
    st["u"] = np.where(np.arange(n) % 2 == 0, -1.0, 1.0) * rmax / setup.dtime * 0.05
    out = {}
    for spec in (False, True):
        with api.Context(setup, precision) as ctx:
            ctx.set_fields(fn)
            ctx.upload(st)
            ctx.set_launch({**GRIDS, "overlap_gather": spec, "speculative_integrate": spec})
            ctx.step(5)
            out[spec] = (ctx.status(), ctx.download())
    assert out[True][0] == out[False][0]
    assert np.count_nonzero(out[False][1]["u"] * st["u"] < 0) > n // 10      # they did rebound
    for k in api.STATE_KEYS:
        assert np.array_equal(out[True][1][k], out[False][1][k], equal_nan=True), k
