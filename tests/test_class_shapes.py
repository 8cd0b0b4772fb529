"""A class of one shape, whose constants are formed once, against the same particles beside
one of another shape, which takes the per-particle path: equal bit for bit."""
from __future__ import annotations

import numpy as np
import pytest

from gazpart_b200 import api, config, field, particles

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 2, 33, 3000])
@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_same_as_per_particle(n, precision):
    s = config.Setup(nx=20, ny=20, nz=20, visc=0.02, dtime=1e-3)
    f = {k: np.random.default_rng(i).normal(size=(20, 20, 20)) for i, k in enumerate(field.COMPONENTS_6)}
    st = particles.draw(config.ParticleSpec(n=n, ar=2.0, b=0.002, st=1.0, seed=n), s)
    # one more particle, in its last ulp of another shape, far from the walls and the others' reach
    more = {k: np.append(v, v[0]) for k, v in st.items()}
    more["rhop"][n] = np.nextafter(more["rhop"][n], 2.0 * more["rhop"][n])
    more["x"][n] = (more["x"][n] + 0.5 * s.lx) % s.lx
    got = []
    for state in (st, more):
        with api.Context(s, precision, max_particles=n + 1) as ctx:
            ctx.set_fields(f)
            ig = ctx.add_class(state)
            for k in range(3):
                ctx.adv_particle_ellp(k)
            ctx.raise_status()
            got.append(ctx.download_class(ig))
    for k in api.STATE_KEYS:
        assert np.array_equal(got[0][k], got[1][k][:n]), k
