"""The accepted pairs of a packed ensemble against the oracle's serial walk, with fewer and
with more colliding pairs than one block of the matching takes alone (2,048)."""
from __future__ import annotations

import numpy as np
import pytest

import pyoracle as po
from _cases import copy_state
from gazpart_b200 import api, config, particles

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,least", [(6_000, 1), (70_000, 2_049)])
def test_accepted_pairs(n, least):
    setup = config.Setup(nx=16, ny=16, nz=16, visc=0.05, dtime=1e-3)
    b = 0.03 * (20_000 / n) ** (1.0 / 3.0)
    st = particles.draw(config.ParticleSpec(n=n, ar_range=(0.4, 3.0), b=b, st=1.0, seed=11), setup)
    rng = np.random.default_rng(2)
    for k in ("u", "v", "w", "ox", "oy", "oz"):
        st[k] = rng.normal(size=n)
    res = po.Ensemble(setup, copy_state(st)).collide(prefilter=True, nthreads=8)
    assert res["rc"] == 0
    with api.Context(setup, "fp64") as ctx:
        ctx.upload(st)
        cnt = ctx.collision(1, 0.0)
        home, near = ctx.collision_pairs()
        assert cnt["n_coll"] >= least
        assert np.array_equal(home, res["home"]) and np.array_equal(near, res["near"])
        ctx.collision(1, 0.0)                      # the matching left its arrays clean
        assert ctx.status()[0] == 0
