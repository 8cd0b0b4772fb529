"""The one-pass scan of the search grid's counts (tiles of 2,048) through what rests on it:
accepted pairs against the oracle with grids of one tile, of a tile and its neighbours, and
of more tiles than one look-back takes at a time."""
from __future__ import annotations

import numpy as np
import pytest

import pyoracle as po
from _cases import copy_state
from gazpart_b200 import api, config, particles

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [500, 3_440, 4_394, 150_000])   # 7^3, 12^3, 13^3 and 42^3 cells
def test_pairs_over_scan_sizes(n):
    setup = config.Setup(nx=16, ny=16, nz=16, visc=0.05)
    b = 0.012 * (20_000 / n) ** (1.0 / 3.0)
    st = particles.draw(config.ParticleSpec(n=n, ar_range=(0.5, 2.0), b=b, st=1.0, seed=3), setup)
    rng = np.random.default_rng(4)
    for k in ("u", "v", "w", "ox", "oy", "oz"):
        st[k] = rng.normal(size=n)
    res = po.Ensemble(setup, copy_state(st)).collide(prefilter=True, nthreads=8)
    with api.Context(setup, "fp64") as ctx:
        ctx.upload(st)
        for phase in range(2):                   # the counters are clear for the second phase
            cnt = ctx.collision(1, 0.0)
            if phase == 0:
                home, near = ctx.collision_pairs()
                assert cnt["n_contact"] == res["n_contacts"]
                assert np.array_equal(home, res["home"]) and np.array_equal(near, res["near"])
        assert ctx.status()[0] == 0
