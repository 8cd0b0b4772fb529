"""A field written into a slot as soon as it has been added: its zero fill is over by then,
so what the particles sample there is what the same field gives in slot 0."""
from __future__ import annotations

import numpy as np
import pytest
import torch

from gazpart_b200 import api, config, field, particles

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [24, 160])
@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_written_at_once(n, precision):
    s = config.Setup(nx=n, ny=n, nz=n, visc=0.02, dtime=1e-4)
    g = torch.Generator(device="cuda").manual_seed(n)
    f = {k: torch.randn((n, n, n), generator=g, device="cuda", dtype=torch.float64) for k in field.COMPONENTS_6}
    torch.cuda.synchronize()
    st = particles.draw(config.ParticleSpec(n=20000, ar=2.0, b=0.001, st=1.0, seed=1), s)
    got = []
    for added in (False, True):
        with api.Context(s, precision, store_fluid=True, max_particles=20000) as ctx:
            slot = ctx.add_field(n) if added else 0
            ctx.set_fields(f, slot=slot)
            ctx.add_class(st, slot)
            ctx.adv_particle_ellp()
            ctx.raise_status()
            got.append(ctx.download(fluid=True))
    for k in api.FLUID_KEYS:
        assert np.array_equal(got[0][k], got[1][k]), k
