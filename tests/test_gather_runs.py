"""The stencil gather against the oracle at ensemble sizes around the points where its
warps take shorter runs of particles, and at the ends of a run."""
from __future__ import annotations

import numpy as np
import pytest

import pyoracle as po
from _cases import field_refs
from gazpart_b200 import api, config, field, particles

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 3, 4, 5, 33, 9472, 9473, 18945, 37889])
def test_fluid_at_particles(n):
    setup = config.Setup(nx=20, ny=22, nz=24, visc=0.02, dtime=1e-4)
    f = {k: np.random.default_rng(i).normal(size=(24, 22, 20)) for i, k in enumerate(field.COMPONENTS_6)}
    import torch
    refs = field_refs({k: torch.from_numpy(v) for k, v in f.items()})
    st = particles.draw(config.ParticleSpec(n=n, ar=2.0, b=0.002, st=1.0, seed=n), setup)
    want = [po.interp_lag3(setup, refs[c], st["x"], st["y"], st["z"]) for c in range(6)]
    for precision in ("fp64", "mixed"):
        with api.Context(setup, precision, store_fluid=True) as ctx:
            ctx.set_fields(f)
            ctx.upload(st)
            ctx.adv_particle_ellp()
            got = ctx.download(fluid=True)
            assert ctx.status()[0] == 0
        for c, k in enumerate(api.FLUID_KEYS):
            if precision == "fp64":
                assert np.array_equal(got[k], want[c]), (n, k)
            else:   # FP32 field and weights: 64 products of weights summing to at most 1.96 each axis
                assert np.max(np.abs(got[k] - want[c])) < 64 * 2 ** -24 * 7.6 * np.abs(f[field.COMPONENTS_6[c]]).max()
