"""The state columns between the caller's order and the pool's: a state put on the device
and read back, after a step has moved the pool out of the caller's order, is the same
values, on device and host arrays, whole and class by class, below and above the size from
which the copies go through rows, with remainders of their tile of 256."""
from __future__ import annotations

import ctypes as C

import numpy as np
import pytest

from gazpart_b200 import _lib, api, config, particles

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("counts", [(1,), (257, 3), (500_001, 300_255), (1_600_001, 259)])
def test_put_and_read_back(counts):
    import torch
    setup = config.Setup(nx=16, ny=16, nz=16, visc=0.02, dtime=1e-4)
    rng = np.random.default_rng(3)
    states = [particles.draw(config.ParticleSpec(n=n, ar=2.0, b=0.002, st=1.0, seed=i), setup)
              for i, n in enumerate(counts)]
    n = sum(counts)
    new = {k: rng.random(n) for k in api.STATE_KEYS}
    with api.Context(setup, "mixed") as ctx:
        ctx.upload_classes(states)
        ctx.step(2)                              # the pool is in cell order now
        dev = {k: torch.from_numpy(v).cuda() for k, v in new.items()}
        ctx.put_state(dev)
        out = {k: torch.full((n,), -1.0, dtype=torch.float64, device="cuda") for k in api.STATE_KEYS}
        cols = (C.c_void_p * 13)(*[C.c_void_p(out[k].data_ptr()) for k in api.STATE_KEYS])
        assert _lib.lib().gp_download_state(ctx._h, n, cols, None, 1) == 0
        host = ctx.download()
        for k in api.STATE_KEYS:
            assert np.array_equal(out[k].cpu().numpy(), new[k]) and np.array_equal(host[k], new[k]), k
        last = ctx.download_class(len(counts))
        ctx.put_state({k: v[::-1].copy() for k, v in new.items()})     # host arrays in
        again = ctx.download()
        for k in api.STATE_KEYS:
            assert np.array_equal(last[k], new[k][n - counts[-1]:]), k
            assert np.array_equal(again[k], new[k][::-1]), k
        # a missing column is refused, as the copies it replaces refused it
        cols[4] = None
        assert _lib.lib().gp_download_state(ctx._h, n, cols, None, 1) != 0
