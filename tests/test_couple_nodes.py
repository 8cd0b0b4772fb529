"""The live fluid's field nodes: coupling leaves the same field as uploading the same
velocity and vorticity component by component, on meshes whose rows end inside, at and
after a warp's 32 nodes."""
from __future__ import annotations

import numpy as np
import pytest

from gazpart_b200 import api, config, dns, field, particles

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dims", [(4, 6, 8), (28, 6, 4), (30, 8, 6), (62, 4, 10)])
@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("vorticity", [False, True])
def test_same_as_upload(dims, precision, vorticity):
    nx, ny, nz = dims
    s = config.Setup(nx=nx, ny=ny, nz=nz, visc=0.02, dtime=1e-4)
    rng = np.random.default_rng(nx)
    f = {k: rng.normal(size=(nz, ny, nx)) for k in field.COMPONENTS_6}
    pts = [rng.uniform(0.0, edge * (1 - 1e-9), 4000) for edge in (s.lx, s.ly, s.lz)]
    with api.Context(s, precision) as one, api.Context(s, precision) as two, dns.Fluid(s) as fl:
        fl.set_velocity(f["u"], f["v"], f["w"])
        for ctx in (one, two):
            ctx.set_fields(f)                       # what a coupling without vorticity leaves
        if vorticity:
            vort = fl.vorticity()
            two.set_fields({**f, **dict(zip(field.COMPONENTS_6[3:], vort))})
            for c in range(3):
                one.set_field(c, np.zeros((nz, ny, nx)))
        else:
            for c in range(3):
                one.set_field(c, np.zeros((nz, ny, nx)))
        fl.couple(one, with_vorticity=vorticity)
        for c in range(6):
            a, b = one.interp_lag3(c, *pts), two.interp_lag3(c, *pts)
            assert np.array_equal(a, b), (c, np.abs(a - b).max())
