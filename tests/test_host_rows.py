"""gp_step_host at the sizes where some or all of its column sets go through rows (from
800,000 particles on the way out, 1,600,000 on the way in), and with two classes one of which
came after another had left: the state of put, step and download in turn, bit for bit."""
from __future__ import annotations

import numpy as np
import pytest

from gazpart_b200 import api, config, field, particles

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("counts", [(799_999,), (800_001,), (1_600_003,), (900_000, 257, 800_100)])
@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_step_host_equals_put_step_download(counts, precision):
    setup = config.Setup(nx=16, ny=16, nz=16, visc=0.02, dtime=1e-4)
    fn = {k: v.numpy().copy() for k, v in field.generate(16, seed=2, device="cpu").items()}
    states = [particles.draw(config.ParticleSpec(n=n, ar=2.0, b=0.002, st=1.0, seed=i), setup)
              for i, n in enumerate(counts)]
    ends = []
    for call in ("three", "one"):
        with api.Context(setup, precision, max_particles=sum(counts)) as ctx:
            ctx.set_fields(fn)
            if len(counts) == 1:
                ctx.upload(states[0])
                st = states[0]
            else:
                ctx.upload_classes(states[:2])
                ctx.remove_class(1)
                ctx.step(1)
                ctx.add_class(states[2])
                st = ctx.download()
            st = {k: np.array(st[k], copy=True) for k in api.STATE_KEYS}
            for _ in range(2):
                if call == "one":
                    ctx.step_host(st)
                else:
                    ctx.put_state(st)
                    ctx.step(1)
                    ctx.download_into(st)
            ctx.raise_status()
            ends.append(st)
    for k in api.STATE_KEYS:
        assert np.array_equal(ends[0][k], ends[1][k]), k
