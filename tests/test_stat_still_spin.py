"""STAT_PARTFLUID of particles that slip but do not turn relative to the fluid: infinite
rotation coefficients, as in the reference, and no more time than for turning ones (the
straight-line values take such particles themselves)."""
from __future__ import annotations

import time

import numpy as np
import pytest

import pyoracle as po
from _cases import case
from gazpart_b200 import api, config, field, particles

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("spin", [0.0, 1e-200])   # 1e-200: its square underflows to zero
def test_values(spin):
    setup, fn, refs, st = case("poly")
    n = 70
    st = {k: np.ascontiguousarray(np.resize(v, n)) for k, v in st.items()}
    for k, v in zip(("u", "v", "w", "ox", "oy", "oz"), (0.1, -0.2, 0.3, spin, -spin, spin)):
        st[k][:] = v
    st["x"] = setup.lx * (np.arange(n) + 5.0) / (n + 10)      # off the walls
    setup = type(setup)(**{**setup.__dict__, "dtime": 1e-300, "gravity": 0.0})   # nothing moves
    with api.Context(setup, "fp64", store_fluid=True) as ctx:
        ctx.set_fields({k: np.zeros_like(v) for k, v in fn.items()})
        ctx.upload(st)
        ctx.adv_particle_ellp(0)
        ctx.raise_status()
        ctx.put_state(st)
        ctx.adv_particle_ellp(0)
        sums = ctx.stat_partfluid(1, sums=True)
        got = ctx.download(fluid=True)
    ens = po.Ensemble(setup, {k: got[k] for k in api.STATE_KEYS} | {k: st[k] for k in api.PROP_KEYS})
    for k in api.FLUID_KEYS:
        ens.a[k] = np.ascontiguousarray(got[k])
    ref = ens.stat_partfluid(np.ones(n, dtype=np.int32), 1)
    fin = np.isfinite(ref[0])
    assert not fin.all()
    assert np.array_equal(np.isfinite(sums[0]), fin) and np.array_equal(np.isnan(sums[0]), np.isnan(ref[0]))
    assert np.allclose(sums[0][fin], ref[0][fin], rtol=1e-11, atol=1e-300)


def test_time():
    n = 1_000_000
    setup = config.Setup(nx=32, ny=32, nz=32, visc=0.02, dtime=1e-300)
    zero = {k: np.zeros((32, 32, 32)) for k in field.COMPONENTS_6}
    st = particles.draw(config.ParticleSpec(n=n, ar=3.0, b=0.001, st=1.0, seed=2), setup)
    rng = np.random.default_rng(1)
    for k in ("u", "v", "w"):
        st[k] = rng.normal(size=n)
    took = []
    for spin in (0.0, 1.0):
        for k in ("ox", "oy", "oz"):
            st[k] = spin * rng.normal(size=n)
        with api.Context(setup, "fp64", store_fluid=True) as ctx:
            ctx.set_fields(zero)
            ctx.upload(st)
            ctx.adv_particle_ellp(0)
            ctx.raise_status()
            t = []
            for _ in range(12):
                t0 = time.perf_counter()
                ctx.stat_partfluid(1)
                t.append(time.perf_counter() - t0)
            took.append(np.median(t[2:]))
    assert took[0] < 1.5 * took[1], took   # twice, where the straight line is thrown away
