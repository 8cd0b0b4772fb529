"""The contact solve at the ends of its number range, against the oracle, bit for bit.

The device runs a Levenberg-Marquardt step as straight-line code where every operand lies
in a safe exponent range, and falls back to the general step otherwise.  The pairs here
make it do both: body sizes whose residuals and norms leave the range, touching and nearly
coincident bodies (gaps that shrink towards zero), needles and plates."""
from __future__ import annotations

import numpy as np
import pytest

import pyoracle as po
from gazpart_b200 import api, config

pytestmark = pytest.mark.gpu


def _pairs(rng, n, size, ar, near):
    """n pairs of minor semi-axis about `size`, aspect ratio ar or 1 / ar, centres at
    near[0]..near[1] of the sum of the largest semi-axes."""
    a = np.where(rng.random((n, 2)) < 0.5, ar, 1.0 / ar) * rng.uniform(0.9, 1.1, (n, 2))
    e = size * np.maximum(a, 1.0) * rng.uniform(0.8, 1.2, (n, 2))
    q = rng.normal(size=(n, 2, 4))
    q /= np.linalg.norm(q, axis=2, keepdims=True)
    d = rng.normal(size=(n, 3))
    d /= np.linalg.norm(d, axis=1, keepdims=True)
    reach = np.maximum(e, e / a).sum(axis=1)
    b1 = rng.uniform(0.0, 3.0, (n, 3)) * size
    b2 = b1 + d * (reach * rng.uniform(near[0], near[1], n))[:, None]
    return np.stack([e[:, 0], a[:, 0], e[:, 1], a[:, 1]], axis=1), np.hstack([b1, b2]), q.reshape(n, 8)


@pytest.mark.parametrize("size,ar,near", [
    (1e-3, 3.0, (0.1, 1.0)),       # ordinary bodies
    (1e-3, 1.02, (0.98, 1.0)),     # touching, nearly spheres
    (1e-3, 40.0, (0.02, 0.6)),     # needles and plates
    (1e-3, 2.0, (1e-9, 1e-6)),     # nearly coincident centres
    (1e-7, 2.0, (0.2, 1.0)),       # norms around MINPACK's rdwarf
    (1e-60, 2.0, (0.2, 1.0)),      # residuals below the safe range
    (1e4, 2.0, (0.2, 1.0)),
    (1e8, 2.0, (0.2, 1.0)),        # norms around MINPACK's rgiant
    (1e80, 2.0, (0.2, 1.0)),       # residuals above the safe range
])
def test_contact_solve_over_its_number_range(size, ar, near):
    n = 200
    shapes, centres, quats = _pairs(np.random.default_rng(17), n, size, ar, near)
    with api.Context(config.Setup(nx=8, ny=8, nz=8), "fp64") as ctx:
        flag, e1, e2, cn = ctx.ellipsoid_contact_detection(shapes, centres, quats)
    for i in range(n):
        s, c, q = shapes[i], centres[i], quats[i]
        r = po.contact_detection(s[0], s[1], s[2], s[3], c[:3], q[:4], c[3:], q[4:])
        assert flag[i] == r["flag"], i
        for got, want in ((e1[i], r["ept1"]), (e2[i], r["ept2"]), (cn[i], r["cnormal"])):
            assert np.array_equal(got, want, equal_nan=True), (i, got, want)
