"""The gather over several classes on one field, whose runs of slots are interleaved: every
particle gets its own fluid values, whatever the classes' sizes."""
from __future__ import annotations

import numpy as np
import pytest
import torch

import pyoracle as po
from _cases import field_refs
from gazpart_b200 import api, config, field, particles

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("counts", [(37889 - 32, 32), (1, 40000, 33, 5000, 15), (30000, 30001), (17,) * 40 + (40000, 16)])
@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_fluid_at_particles(counts, precision):
    setup = config.Setup(nx=20, ny=22, nz=24, visc=0.02, dtime=1e-4)
    f = {k: np.random.default_rng(i).normal(size=(24, 22, 20)) for i, k in enumerate(field.COMPONENTS_6)}
    refs = field_refs({k: torch.from_numpy(v) for k, v in f.items()})
    states = [particles.draw(config.ParticleSpec(n=n, ar=2.0, b=0.002, st=1.0, seed=i), setup)
              for i, n in enumerate(counts)]
    with api.Context(setup, precision, store_fluid=True) as ctx:
        ctx.set_fields(f)
        ctx.upload_classes(states)
        for step in range(2):                # in upload order, then in cell order
            at = ctx.download()
            want = [po.interp_lag3(setup, refs[c], at["x"], at["y"], at["z"]) for c in range(6)]
            ctx.adv_particle_ellp(step)
            got = ctx.download(fluid=True)
            assert ctx.status()[0] == 0
            for c, k in enumerate(api.FLUID_KEYS):
                if precision == "fp64":
                    assert np.array_equal(got[k], want[c]), (step, k)
                else:   # FP32 field and weights: 64 products of weights of at most 1.96 in all on each axis
                    bound = 64 * 2 ** -24 * 7.6 * np.abs(f[field.COMPONENTS_6[c]]).max()
                    assert np.max(np.abs(got[k] - want[c])) < bound, (step, k)
            ctx.collision(step, 0.0)
