"""Tracking alone (advances without a collision phase between them) after a class has left:
the first advance closes the gaps its particles left in the pool, and the next ones must take
the particles from where that put them.  The classes that stay end bit for bit where each
ends alone in a context of its own."""
from __future__ import annotations

import numpy as np
import pytest

from _cases import field_refs, init_state
from gazpart_b200 import api, config, field

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("counts,leave,join", [((900, 500), 1, 0), ((40, 3000, 700), 2, 0), ((900, 500), 1, 77),
                                               ((1, 1), 1, 0)])
@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_advances_in_a_row(counts, leave, join, precision):
    setup = config.Setup(nx=24, ny=24, nz=24, visc=0.05, dtime=1e-3)
    f = field.generate(24, seed=6, device="cpu")
    fn, refs = {k: v.numpy().copy() for k, v in f.items()}, field_refs(f)
    states = [init_state(setup, config.ParticleSpec(n=n, ar=2.0, b=0.01, st=1.0, seed=60 + i), f, refs)
              for i, n in enumerate(counts + ((join,) if join else ()))]
    want = {}
    for i, st in enumerate(states):
        with api.Context(setup, precision) as alone:
            alone.set_fields(fn)
            alone.upload(st)
            for s in range(3):
                alone.adv_particle_ellp(s)
            alone.step(2)
            want[i] = alone.download()
    with api.Context(setup, precision, max_particles=sum(counts) + join) as ctx:
        ctx.set_fields(fn)
        ctx.upload_classes(states[:len(counts)])
        ctx.remove_class(leave)
        stay = {i + 1: i for i in range(len(counts)) if i + 1 != leave}
        if join:
            stay[ctx.add_class(states[-1])] = len(counts)
        for s in range(3):
            ctx.adv_particle_ellp(s)
        ctx.step(2)
        ctx.raise_status()
        for ig, i in stay.items():
            got = ctx.download_class(ig)
            for k in api.STATE_KEYS:
                assert np.array_equal(got[k], want[i][k]), (ig, k)
