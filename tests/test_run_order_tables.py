"""The gather's order of runs in a class table with gaps and new classes in old places: every
particle gets its own fluid values, and each class steps as it does alone."""
from __future__ import annotations

import numpy as np
import pytest

from gazpart_b200 import api, config, field, particles

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("counts,leave,join", [((20000, 40000, 33), (1,), 0), ((30000, 15, 30001, 64), (2, 4), 0),
                                               ((20000, 40000, 33), (1, 3), 25000), ((5, 70000), (1,), 1)])
@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_classes_after_removals(counts, leave, join, precision):
    setup = config.Setup(nx=20, ny=22, nz=24, visc=0.02, dtime=1e-4)
    fn = {k: np.random.default_rng(i).normal(size=(24, 22, 20)) for i, k in enumerate(field.COMPONENTS_6)}
    states = [particles.draw(config.ParticleSpec(n=n, ar=2.0, b=0.002, st=1.0, seed=i), setup)
              for i, n in enumerate(counts + ((join,) if join else ()))]
    with api.Context(setup, precision, max_particles=sum(counts) + join) as ctx:
        ctx.set_fields(fn)
        ctx.upload_classes(states[:len(counts)])
        for ig in leave:
            ctx.remove_class(ig)
        stay = {i + 1: i for i in range(len(counts)) if i + 1 not in leave}
        if join:
            stay[ctx.add_class(states[-1])] = len(counts)
        ctx.step(3)
        ctx.raise_status()
        got = {i: ctx.download_class(ig) for ig, i in stay.items()}
    for i, end in got.items():
        with api.Context(setup, precision) as alone:
            alone.set_fields(fn)
            alone.upload(states[i])
            alone.step(3)
            want = alone.download()
        for k in api.STATE_KEYS:
            assert np.array_equal(end[k], want[k]), (i, k)
