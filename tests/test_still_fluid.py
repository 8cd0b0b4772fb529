"""The FP64 step where components are exactly zero at every step: bodies that settle in still
fluid, along or across the fall, spinning about their axis only or about one other axis.  The
values agree with the oracle's as in any other flow, and the step takes no longer than in
one (the straight-line step takes such particles itself)."""
from __future__ import annotations

import numpy as np
import pytest

import pyoracle as po
from _cases import copy_state
from gazpart_b200 import api, config, field, particles

pytestmark = pytest.mark.gpu
TOL = 1e-12
H = 0.5 ** 0.5
# orientation (None: random), spin
CASES = {"random": (None, (0.0, 0.0, 0.0)), "across": ((1.0, 0.0, 0.0, 0.0), (0.0, 0.0, 0.0)),
         "along": ((H, 0.0, -H, 0.0), (0.0, 0.0, 0.0)), "axial spin": (None, (0.5, 0.0, 0.0)),
         "along, axial spin": ((H, 0.0, -H, 0.0), (-0.5, 0.0, 0.0)),
         "across, one spin": ((1.0, 0.0, 0.0, 0.0), (0.0, -0.5, 0.0))}


def _ensemble(name, n, setup, b):
    st = particles.draw(config.ParticleSpec(n=n, ar_range=(0.3, 4.0), b=b, st=1.0, seed=12), setup)
    quat, spin = CASES[name]
    if quat is not None:
        for k, v in zip(("qa", "qb", "qc", "qd"), quat):
            st[k][:] = v
    for k, v in zip(("u", "v", "w", "ox", "oy", "oz"), (0.0, 0.0, 0.0) + spin):
        st[k] = np.full(n, v)
    return st


@pytest.mark.parametrize("name", CASES)
@pytest.mark.parametrize("gravity", [-9.81, 0.0])
def test_values(name, gravity):
    n = 300
    setup = config.Setup(nx=12, ny=12, nz=12, visc=0.02, dtime=1e-4, gravity=gravity)
    zero = {k: np.zeros((12, 12, 12)) for k in field.COMPONENTS_6}
    import torch
    refs = [field.reference_layout(torch.from_numpy(zero[k]), "periodic").numpy().copy() for k in field.COMPONENTS_6]
    st = _ensemble(name, n, setup, 0.01)
    if gravity == 0.0:
        st["w"][:] = np.where(np.arange(n) % 2 == 0, 0.25, -0.25)
    ens = po.Ensemble(setup, copy_state(st))
    with api.Context(setup, "fp64") as ctx:
        ctx.set_fields(zero)
        ctx.upload(st)
        for s in range(4):
            ens.advance(refs)
            ctx.adv_particle_ellp(s)
        got = ctx.download()
    for group in (("x", "y", "z"), ("u", "v", "w"), ("qa", "qb", "qc", "qd"), ("ox", "oy", "oz")):
        a, b = (np.stack([s[k] for k in group]) for s in (got, ens.a))
        assert np.array_equal(np.isnan(a), np.isnan(b)), group
        err = np.linalg.norm(a - b, axis=0) / (np.linalg.norm(b, axis=0) + 1e-30)
        assert err.max() < TOL, (group, err.argmax(), err.max())


def _integrate_ms(setup, fn, st):
    with api.Context(setup, "fp64") as ctx:
        ctx.set_fields(fn)
        ctx.upload(st)
        ctx.step(2)
        return float(np.median([ctx.step_timed(1)[1]["integrate"] for _ in range(9)]))


@pytest.mark.parametrize("name", CASES)
def test_time(name):
    n = 400_000
    setup = config.Setup(nx=32, ny=32, nz=32, visc=0.02, dtime=1e-4, gravity=-9.81)
    f = {k: v.numpy().copy() for k, v in field.generate(32, seed=3, device="cpu").items()}
    zero = {k: np.zeros_like(v) for k, v in f.items()}
    st = _ensemble(name, n, setup, 0.0015)
    moving = {k: v.copy() for k, v in _ensemble("random", n, setup, 0.0015).items()}
    rng = np.random.default_rng(4)
    for k in ("u", "v", "w", "ox", "oy", "oz"):
        moving[k] = rng.normal(size=n)
    # twice the step (three times and more before) is the straight line thrown away
    assert _integrate_ms(setup, zero, st) < 1.5 * _integrate_ms(setup, f, moving)
