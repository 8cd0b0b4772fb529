"""Device columns that end before the ensemble does are refused by the host, before any
kernel touches them; columns that just hold it, at an offset in their allocation too, are
taken."""
from __future__ import annotations

import ctypes as C

import numpy as np
import pytest

from gazpart_b200 import _lib, api, config, particles

pytestmark = pytest.mark.gpu
EBADARG = 9


def _columns(t):
    return (C.c_void_p * 13)(*[C.c_void_p(t[k].data_ptr()) for k in api.STATE_KEYS])


def _must_be_short(at, need):
    """Nothing may be asked of the library here that the driver itself does not call short."""
    cuda = C.CDLL("libcuda.so.1")
    base, size, handle = C.c_uint64(), C.c_size_t(), C.c_uint64()
    assert cuda.cuMemGetAddressRange_v2(C.byref(base), C.byref(size), C.c_uint64(at)) == 0
    assert at + need > base.value + size.value
    assert cuda.cuMemRetainAllocationHandle(C.byref(handle), C.c_void_p(at)) != 0   # not mapped in pieces


@pytest.mark.parametrize("n,offset", [(400_000, 0), (400_000, 1), (900_001, 3)])
@pytest.mark.parametrize("short", ["x", "qc", "oz"])
def test_short_columns(n, offset, short):
    import torch
    setup = config.Setup(nx=16, ny=16, nz=16, visc=0.02, dtime=1e-4)
    st = particles.draw(config.ParticleSpec(n=n, ar=2.0, b=0.002, st=1.0, seed=1), setup)
    rng = np.random.default_rng(2)
    torch.cuda.empty_cache()
    # one allocation for all columns, which ends with the last of them
    flat = torch.empty(13 * n + offset, dtype=torch.float64, device="cuda")
    cols = {k: flat[offset + i * n:offset + (i + 1) * n] for i, k in enumerate(api.STATE_KEYS)}
    new = {k: rng.random(n) for k in api.STATE_KEYS}
    for k in api.STATE_KEYS:
        cols[k].copy_(torch.from_numpy(new[k]))
    torch.cuda.synchronize()
    with api.Context(setup, "mixed") as ctx:
        ctx.upload(st)
        L = _lib.lib()
        assert L.gp_put_state(ctx._h, n, _columns(cols), 1) == 0
        got = ctx.download()
        # a column that begins with the allocation's last values
        at = flat.data_ptr() + flat.numel() * 8 - 8
        _must_be_short(at, 8 * n)
        bad = _columns(cols)
        bad[api.STATE_KEYS.index(short)] = C.c_void_p(at)
        assert L.gp_put_state(ctx._h, n, bad, 1) == EBADARG
        assert L.gp_download_state(ctx._h, n, bad, None, 1) == EBADARG
        assert L.gp_download_class(ctx._h, 1, bad, 1) == EBADARG
        after = ctx.download()
    for k in api.STATE_KEYS:
        assert np.array_equal(got[k], new[k]) and np.array_equal(after[k], new[k]), k
