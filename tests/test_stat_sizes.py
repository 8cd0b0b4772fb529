"""STAT_PARTFLUID against the oracle at ensemble sizes around the ends of a warp's tile of 32
and of a launch's first pass, with one to eight polydisperse indices, and with particles
that the straight-line form leaves to the general one (no slip, no spin)."""
from __future__ import annotations

import numpy as np
import pytest

import pyoracle as po
from _cases import case
from gazpart_b200 import api, particles
from test_stats import _per_particle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,groups", [(1, 1), (31, 1), (33, 8), (64, 3), (65, 2), (3000, 8)])
def test_sums(n, groups):
    setup, fn, refs, st = case("poly")
    st = {k: np.ascontiguousarray(np.resize(v, n)) for k, v in st.items()}
    st["x"] = setup.lx * (np.arange(n) + 0.5) / n            # apart from one another and from the walls
    idp = (np.arange(n) % groups + 1).astype(np.int32)
    with api.Context(setup, "fp64", store_fluid=True) as ctx:
        ctx.set_fields(fn)
        ctx.upload(st)
        ctx.set_class_groups(1, idp, groups)
        ctx.adv_particle_ellp(0)
        ctx.raise_status()
        sums = ctx.stat_partfluid(1, sums=True)
        got = ctx.download(fluid=True)
    ens = po.Ensemble(setup, {k: got[k] for k in api.STATE_KEYS} | {k: st[k] for k in api.PROP_KEYS})
    for k in api.FLUID_KEYS:
        ens.a[k] = np.ascontiguousarray(got[k])
    ref = ens.stat_partfluid(idp, groups)
    per = _per_particle(ens, setup)
    for g in range(groups):
        mag = np.abs(per[idp == g + 1]).sum(axis=0)
        nan = np.isnan(ref[g])
        assert np.array_equal(np.isnan(sums[g]), nan), g
        assert np.all(np.abs(sums[g] - ref[g])[~nan] <= 1e-11 * mag[~nan] + 1e-300), g
        assert sums[g, 35] == np.count_nonzero(idp == g + 1)


def test_still_particles():
    """A particle at the fluid's velocity has Re = 0: infinite coefficients, as in the reference."""
    setup, fn, refs, st = case("poly")
    n = 40
    st = {k: np.ascontiguousarray(np.resize(v, n)) for k, v in st.items()}
    zero = {k: np.zeros_like(v) for k, v in fn.items()}
    for k in ("u", "v", "w", "ox", "oy", "oz"):
        st[k] = np.where(np.arange(n) % 2 == 0, 0.0, 0.1)
    st["x"] = setup.lx * (np.arange(n) + 0.5) / n
    idp = (np.arange(n) % 2 + 1).astype(np.int32)
    setup = type(setup)(**{**setup.__dict__, "dtime": 1e-300})   # nothing moves
    with api.Context(setup, "fp64", store_fluid=True) as ctx:
        ctx.set_fields(zero)
        ctx.upload(st)
        ctx.set_class_groups(1, idp, 2)
        ctx.adv_particle_ellp(0)
        sums = ctx.stat_partfluid(1, sums=True)
        got = ctx.download(fluid=True)
    ens = po.Ensemble(setup, {k: got[k] for k in api.STATE_KEYS} | {k: st[k] for k in api.PROP_KEYS})
    for k in api.FLUID_KEYS:
        ens.a[k] = np.ascontiguousarray(got[k])
    ref = ens.stat_partfluid(idp, 2)
    for g in range(2):
        fin = np.isfinite(ref[g])
        assert np.array_equal(np.isfinite(sums[g]), fin), g
        assert np.array_equal(np.isnan(sums[g]), np.isnan(ref[g])), g
        assert np.allclose(sums[g][fin], ref[g][fin], rtol=1e-11, atol=1e-300), g
