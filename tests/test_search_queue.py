"""The sweep's queue of candidates for the exact tests: ensembles in which a warp has none,
fewer than 32, and many times 32 of them, against the oracle's accepted pairs."""
from __future__ import annotations

import numpy as np
import pytest

import pyoracle as po
from _cases import copy_state
from gazpart_b200 import api, config, particles

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,b,clump", [(2, 0.005, 0.01), (9, 0.02, 0.05), (33, 0.02, 0.08), (300, 0.02, 0.2),
                                       (1500, 0.02, 0.3), (3000, 0.012, 1.0), (5000, 0.001, 1.0)])
def test_accepted_pairs(n, b, clump):
    setup = config.Setup(nx=16, ny=16, nz=16, lx=1.0, ly=1.0, lz=1.0, visc=0.05)
    st = particles.draw(config.ParticleSpec(n=n, ar_range=(0.5, 2.0), b=b, st=1.0, seed=n), setup)
    rng = np.random.default_rng(n)
    for k in "xyz":
        st[k] = 0.5 - 0.5 * clump + clump * rng.random(n)
    for k in ("u", "v", "w", "ox", "oy", "oz"):
        st[k] = rng.normal(size=n)
    res = po.Ensemble(setup, copy_state(st)).collide(prefilter=True, nthreads=8)
    with api.Context(setup, "fp64") as ctx:
        ctx.upload(st)
        cnt = ctx.collision(1, 0.0)
        home, near = ctx.collision_pairs()
    assert cnt["n_contact"] == res["n_contacts"]
    assert np.array_equal(home, res["home"]) and np.array_equal(near, res["near"])
