"""ecs_step_host with a tile of more ions than a staging chunk holds: its
download goes out in pieces, and the call stays on the pipelined path instead
of uploading and sorting the ions again.

The pipelined path makes the identities the host indices and, without a sort,
returns the ions in the order they came in, so the identities are 0, 1, 2, ...;
an upload sorts.  Moments, potential and ions (as a set) equal the
device-resident step's bit for bit, as in the other host-step tests.
"""
import numpy as np
import pytest

import ecsprt_gb300 as E
from test_gpu_host_step import as_set

pytestmark = pytest.mark.gpu


# capacity, ions, those of one tile: chunks of 65536 ions (four pieces, a last
# one of 3 ions) and of 524288 (two)
@pytest.mark.parametrize("cap, n, dense", [(300_000, 300_000, 196_611), (1 << 24, 900_000, 600_003)])
@pytest.mark.parametrize("sort_every", [2, 1000])
@pytest.mark.parametrize("shift", [(0, 0), (3, 30)])
def test_tile_larger_than_a_chunk(built, cap, n, dense, sort_every, shift):
    p = E.params_from_options("-Nx 8 -Ny 8 -Nz 8 -dx 1 -dy 1 -dz 1 -qi 1 -mi 1 -B0 0.1 -viT 0.1 -vi0x 0.1 "
                              "-nue 8.79e9 -Te 11604.5 -E0 0 -mn 0")
    rng = np.random.default_rng(n)
    pos = rng.uniform(0, 8, (n, 3))
    pos[:dense] = [4, 0, 2] + rng.uniform(0.01, 0.99, (dense, 3)) * [4, 4, 2]  # one tile
    order = rng.permutation(n)
    pos, vel = pos[order], 0.1 * rng.standard_normal((n, 3))
    phi = 1e-3 * rng.standard_normal((8, 8, 8))
    steps = 3
    ref = []
    with E.Context(p, E.ECS_PREC_MIXED, np_capacity=cap) as ctx:
        ctx.set_sort_every(sort_every)
        ctx.upload_particles(pos, vel)
        ctx.phi = phi
        for _ in range(steps):
            ctx.step(0.01, 1e-8, 400)
            ref.append((ctx.moments, ctx.phi, as_set(*ctx.download_particles())))
    with E.Context(p, E.ECS_PREC_MIXED, np_capacity=cap) as ctx:
        ctx.set_sort_every(sort_every)
        ctx.upload_particles(pos, vel)
        ctx.phi = phi
        hp, hv = (E.pinned_empty((3 * n + 64,))[s:s + 3 * n].reshape(n, 3) for s in shift)
        hp[:], hv[:] = pos, vel
        hm, hphi = E.pinned_empty(ctx.shape + (4,)), E.pinned_empty(ctx.shape)
        for s in range(steps):
            ctx.step_host(hp, hv, 0.01, 1e-8, 400, hm, hphi)
            m, ph, ions = ref[s]
            assert np.array_equal(hm, m), s
            assert np.array_equal(hphi, ph), s
            assert np.array_equal(as_set(hp, hv), ions), s
            if sort_every > steps and s > 0:
                assert np.array_equal(ctx.particle_ids(), np.arange(n)), s
