"""The moments that ecs_step_host hands back leave in pieces of a staging buffer,
which for few ions is much smaller than the moments: one, two and five pieces,
a last one of a few cells.  Against the moments of the same context (read
whole) and of the device-resident step, bit for bit; -lhs identity, so that a
density with empty cells is stepped too.
"""
import numpy as np
import pytest

import ecsprt_gb300 as E

pytestmark = pytest.mark.gpu


# a piece holds 1.5 cells an ion and 32 more: 13 * 11 * 10 = 1430 cells
@pytest.mark.parametrize("n, pieces", [(932, 1), (931, 2), (300, 3), (170, 5)])
def test_moments_in_pieces(built, n, pieces):
    assert -(-1430 // ((2 * (3 * n + 64)) // 4)) == pieces
    p = E.params_from_options("-Nx 13 -Ny 11 -Nz 10 -dx 1 -dy 1 -dz 1 -qi 1 -mi 1 -B0 0.1 -viT 1 -vi0x 0.7 -nue 8.79e9 "
                              "-Te 11604.5 -E0 0 -mn 0 -lhs identity")
    rng = np.random.default_rng(n)
    pos, vel = rng.uniform(0, 1, (n, 3)) * [13, 11, 10], rng.standard_normal((n, 3))
    steps = 4
    ref = []
    with E.Context(p, E.ECS_PREC_MIXED, np_capacity=n) as ctx:
        ctx.upload_particles(pos, vel)
        for _ in range(steps):
            ctx.step(1e-3, 1e-8, 10)
            ref.append(ctx.moments)
    with E.Context(p, E.ECS_PREC_MIXED, np_capacity=n) as ctx:
        ctx.upload_particles(pos, vel)
        hp, hv = E.pinned_empty((n, 3)), E.pinned_empty((n, 3))
        hp[:], hv[:] = pos, vel
        hm, hphi = E.pinned_empty(ctx.shape + (4,)), E.pinned_empty(ctx.shape)
        for s in range(steps):
            hm[:] = np.nan
            ctx.step_host(hp, hv, 1e-3, 1e-8, 10, hm, hphi)
            assert np.array_equal(hm, ctx.moments), s
            assert np.array_equal(hm, ref[s]), s
