"""Admission counts at least the device memory that a job's particles take: pool, search,
pair and contact buffers, and the staging they come and go through."""
from __future__ import annotations

import numpy as np
import pytest

from gazpart_b200 import api, config, particles, serving

pytestmark = pytest.mark.gpu


def test_bytes_per_particle_cover_the_memory_taken():
    import torch
    setup = config.Setup(nx=8, ny=8, nz=8, visc=0.02, dtime=1e-4)

    def used(n):
        """Bytes taken by a context with n particles, after a step and their way out."""
        st = particles.draw(config.ParticleSpec(n=n, ar=2.0, b=0.0004, st=1.0, seed=1), setup)
        before = torch.cuda.mem_get_info()[0]
        with api.Context(setup, "mixed", max_particles=n) as ctx:
            ig = ctx.add_class(st)
            ctx.step(1)
            ctx.raise_status()
            ctx.remove_class(ig)
            return before - torch.cuda.mem_get_info()[0]

    used(1 << 20)                                  # the library's own first allocations
    # every array's bytes are a multiple of the allocator's 2 MiB at these sizes, but the cells'
    a, b = 1 << 21, 1 << 22
    taken = (used(b) - used(a)) / (b - a)
    assert taken <= serving.BYTES_PER_PARTICLE + 4 * (1 << 21) / (b - a), taken
    assert taken >= 0.9 * serving.BYTES_PER_PARTICLE, taken      # and little more
