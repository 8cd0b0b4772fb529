"""One advance against the oracle at the ends of its number ranges.

The FP64 device step runs as straight-line code where every operand lies in a safe range
and falls back to the general step otherwise; the particles here make it do both: slips
from zero to far beyond the correlations' range, spins equal to half the vorticity, slips
along the symmetry axis (no transverse part) and bodies at the x planes.  The powers, sines
and cosines of the two sides may differ by an ulp, as in the other state comparisons."""
from __future__ import annotations

import numpy as np
import pytest

import pyoracle as po
from _cases import copy_state
from gazpart_b200 import api, config, field, particles

pytestmark = pytest.mark.gpu
TOL = 1e-12


@pytest.mark.parametrize("slip", [0.0, 1e-70, 1e-40, 1e-16, 1e-6, 1.0, 1e3])
@pytest.mark.parametrize("spin", ["fluid", "zero", "random"])
def test_advance_over_its_number_range(slip, spin):
    import torch
    n = 400
    setup = config.Setup(nx=12, ny=12, nz=12, visc=0.02, dtime=1e-4)
    uf, vort = (0.4, -0.3, 0.2), (2.0, -1.0, 0.5)
    f = {k: torch.full((12, 12, 12), v, dtype=torch.float64)
         for k, v in zip(field.COMPONENTS_6, uf + vort)}
    refs = [field.reference_layout(f[k], "periodic").numpy().copy() for k in field.COMPONENTS_6]
    rng = np.random.default_rng(5)
    st = particles.draw(config.ParticleSpec(n=n, ar_range=(0.2, 5.0), b=0.01, st=1.0, seed=8), setup)
    st["x"][:60] = rng.uniform(0.0, 0.02, 60)              # at the walls, some intersecting them
    st["x"][60:80] = setup.lx - rng.uniform(0.0, 0.02, 20)
    d = rng.normal(size=(3, n))
    for k in (80, 81, 82, 83):                              # slip along the symmetry axis
        st["qa"][k], st["qb"][k], st["qc"][k], st["qd"][k] = 1.0, 0.0, 0.0, 0.0
        d[:, k] = (1.0 if k % 2 else -1.0, 0.0, 0.0)
    got_f = [po.interp_lag3(setup, refs[c], st["x"], st["y"], st["z"]) for c in range(6)]
    for k, c in zip("uvw", range(3)):
        st[k] = got_f[c] + slip * d[c]
    if spin == "fluid":
        particles.body_half_vorticity(st, *got_f[3:])
    elif spin == "random":
        for k in ("ox", "oy", "oz"):
            st[k] = rng.normal(size=n)
    ens = po.Ensemble(setup, copy_state(st))
    ens.advance(refs)
    with api.Context(setup, "fp64") as ctx:
        ctx.set_fields({k: v.numpy() for k, v in f.items()}, vorticity_ghost="periodic")
        ctx.upload(st)
        ctx.adv_particle_ellp(1)
        got = ctx.download()
    for group in (("x", "y", "z"), ("u", "v", "w"), ("qa", "qb", "qc", "qd"), ("ox", "oy", "oz")):
        a, b = (np.stack([s[k] for k in group]) for s in (got, ens.a))
        assert np.array_equal(np.isnan(a), np.isnan(b)), group
        ok = ~np.isnan(b).any(axis=0)
        err = np.linalg.norm((a - b)[:, ok], axis=0) / (np.linalg.norm(b[:, ok], axis=0) + 1e-30)
        assert err.max() < TOL, (group, np.flatnonzero(ok)[err.argmax()], err.max())
