"""STAT_PARTFLUID with the lanes of every warp apart: its tile of values in shared memory is
written by the lanes one way or the other (straight-line values, or the general form for the
particles without slip) before other lanes of the warp add it up.  The sums are those of
each index's own particles, and the same bits on every call."""
from __future__ import annotations

import numpy as np
import pytest

from _cases import case
from gazpart_b200 import api

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("period", [2, 3, 31])
def test_lanes_of_both_forms(period):
    setup, fn, refs, st = case("poly")
    n = 4000
    st = {k: np.ascontiguousarray(np.resize(v, n)) for k, v in st.items()}
    # fluid at rest: where period divides the index the particle is at rest too (general form)
    fn = {k: np.full_like(v, c) for (k, v), c in zip(fn.items(), (0.0, 0.0, 0.0, 1.0, -2.0, 0.5))}
    still = np.arange(n) % period == 0
    for k, c in zip("uvw", (0.1, -0.2, 0.3)):
        st[k] = np.where(still, 0.0, c)
    for i, k in enumerate(("ox", "oy", "oz")):
        st[k] = np.random.default_rng(i).normal(size=n)
    st["x"] = setup.lx * (np.arange(n) + 0.5) / n
    setup = type(setup)(**{**setup.__dict__, "dtime": 1e-300, "gravity": 0.0})   # nothing else moves
    idp = (still + 1).astype(np.int32)
    with api.Context(setup, "fp64", store_fluid=True) as ctx:
        ctx.set_fields(fn, vorticity_ghost="periodic")
        ctx.upload(st)
        ctx.set_class_groups(1, idp, 2)
        ctx.adv_particle_ellp(0)
        ctx.raise_status()
        sums = [ctx.stat_partfluid(1, sums=True) for _ in range(8)]
        at_sums = ctx.download()                       # bodies at the walls have rebounded
    for s in sums[1:]:
        assert np.array_equal(s, sums[0], equal_nan=True)
    # the spins (values 32 to 34) tell whose columns went into which sum
    for g, at in ((0, ~still), (1, still)):
        assert sums[0][g, 35] == np.count_nonzero(at)
        for i, k in enumerate(("ox", "oy", "oz")):
            of = at_sums[k][at]
            assert abs(sums[0][g, 32 + i] - of.sum()) <= 1e-12 * np.abs(of).sum(), (g, k)
