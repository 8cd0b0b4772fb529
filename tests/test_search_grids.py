"""Candidate pairs on search grids at the ends of their range, against the oracle: three
cells a side (every neighbour wraps), long and flat boxes, boxes far from unit length (the
float tests' slack follows it), walls in x, particles above the one-cell cut and many in
one cell."""
from __future__ import annotations

import numpy as np
import pytest

import pyoracle as po
from _cases import copy_state
from gazpart_b200 import api, config, particles

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,lengths,b,periodic,clump", [
    (40, (1.0, 1.0, 1.0), 0.04, True, False),            # three or four cells a side
    (3000, (1.0, 1.0, 1.0), 0.02, True, False),
    (3000, (1.0, 1.0, 1.0), 0.02, False, False),         # no wrap in x
    (4000, (4.0, 1.5, 1.0), 0.02, True, False),
    (3000, (2000.0, 2000.0, 2000.0), 40.0, True, False),
    (3000, (1e-3, 1e-3, 1e-3), 2e-5, True, False),
    (2000, (1.0, 1.0, 1.0), 0.004, True, True),          # most particles in a few cells
])
def test_accepted_pairs_on_search_grids(n, lengths, b, periodic, clump):
    setup = config.Setup(nx=16, ny=16, nz=16, lx=lengths[0], ly=lengths[1], lz=lengths[2], visc=0.05,
                         periodicity=periodic)
    st = particles.draw(config.ParticleSpec(n=n, ar_range=(0.5, 2.0), b=b, st=1.0, seed=5), setup)
    if n > 1000:                                          # a few above the search grid's cut
        st["emaj"][:2] *= 2.0
    rng = np.random.default_rng(6)
    if clump:
        for k in "xyz":
            st[k] = 0.45 + 0.1 * rng.random(n)
    for k in ("u", "v", "w", "ox", "oy", "oz"):
        st[k] = rng.normal(size=n)
    res = po.Ensemble(setup, copy_state(st)).collide(prefilter=True, nthreads=8)
    with api.Context(setup, "fp64") as ctx:
        ctx.upload(st)
        cnt = ctx.collision(1, 0.0)
        home, near = ctx.collision_pairs()
    assert cnt["n_contact"] == res["n_contacts"] and cnt["n_contact"] > 0
    assert np.array_equal(home, res["home"]) and np.array_equal(near, res["near"])
