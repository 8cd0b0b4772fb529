"""INTERP_LAG3 at many points: a call large enough to sort its points gives what calls of a
few points (which do not) give, bit for bit, points outside the stencil's range included."""
from __future__ import annotations

import numpy as np
import pytest

from gazpart_b200 import api, config

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision,shape,n", [
    ("fp64", (128, 128, 128), 200_001), ("fp64", (150, 120, 110), 300_033), ("mixed", (200, 202, 204), 100_001)])
@pytest.mark.parametrize("wall", [False, True])
def test_sorted_points_change_nothing(precision, shape, n, wall):
    nx, ny, nz = shape
    setup = config.Setup(nx=nx, ny=ny, nz=nz, lx=3.0, ly=2.0, lz=1.0, wall_boundary=wall)
    rng = np.random.default_rng(1)
    f = rng.normal(size=(nz, ny, nx))
    x, y, z = (rng.uniform(0.0, length, n) for length in (3.0, 2.0, 1.0))
    x[:4], y[4:8], z[8:12] = -0.5, 2.5, np.nan              # refused points
    x[12:16], y[16:20], z[20:24] = 3.0, 2.0, 0.0            # at the edges
    with api.Context(setup, precision) as ctx:
        for c in (0, 4):
            ctx.set_field(c, f + c)
        for c in (0, 4):
            whole = ctx.interp_lag3(c, x, y, z)
            parts = np.concatenate([ctx.interp_lag3(c, x[k:k + 50_000], y[k:k + 50_000], z[k:k + 50_000])
                                    for k in range(0, n, 50_000)])
            assert np.array_equal(whole, parts, equal_nan=True)
            assert np.isnan(whole[:12]).all() and not np.isnan(whole[24:]).any()
        assert ctx.status()[0] == 6                           # GP_EOUT_OF_GRID
