"""The FP64 pass sets colliding ions aside in a queue of their warp and finishes
them 32 at a time: no ion may be lost, taken twice or given another's numbers.

Every ion's random numbers come from its own state, so its position and velocity
after a step do not depend on the ions beside it in the arrays, which decide when
a queue drains and what is left in it at the end.  Ions in their order, reversed
and shuffled, and the separate slots (push, collide, move, collect) all give the
same ions, moments and collision count bit for bit.  Counts: less than a warp, a
warp and one, and several sets of 32 for each warp with a ragged last one, at
rates that fill the queue every set and every few sets.
"""
import numpy as np
import pytest

import ecsprt_gb300 as E

pytestmark = pytest.mark.gpu


def run(p, pos, vel, phi, fused):
    with E.Context(p, E.ECS_PREC_FP64, np_capacity=len(pos)) as ctx:
        ctx.upload_particles(pos, vel)
        ctx.phi = phi
        collisions = None
        if fused:
            collisions = ctx.step(0.1, 1e-8, 10).collisions  # -lhs identity: any density is solved
        else:
            ctx.push(0.1)
            ctx.collide(0.1)
            ctx.update_positions(0.1)
            ctx.collect()
        return (*ctx.download_particles(), ctx.moments, collisions)


@pytest.mark.parametrize("n", [5, 33, 300_007])
@pytest.mark.parametrize("nui", [0.5, 8.0])
@pytest.mark.parametrize("zbc", ["periodic", "inject-reflect"])
def test_queue_does_not_depend_on_the_order(built, n, nui, zbc):
    p = E.params_from_options("-Nx 12 -Ny 10 -Nz 8 -dx 1 -dy 1 -dz 1 -qi 1 -mi 1 -B0 0.1 -viT 1 -vi0x 1.0 "
                              f"-nui {nui} -nue 8.79e9 -Te 11604.5 -E0 0 -lhs identity -zBC {zbc}")
    rng = np.random.default_rng(n)
    pos, vel = rng.random((n, 3)) * [12, 10, 8], rng.standard_normal((n, 3))
    phi = 0.1 * rng.standard_normal((8, 10, 12))
    p0, v0, m0, c0 = run(p, pos, vel, phi, True)
    pushed = run(E.params_from_options(f"-Nx 12 -Ny 10 -Nz 8 -dx 1 -dy 1 -dz 1 -qi 1 -mi 1 -B0 0.1 -viT 1 -vi0x 1.0 "
                                       f"-nue 8.79e9 -Te 11604.5 -E0 0 -mn 0 -lhs identity -zBC {zbc}"),
                 pos, vel, phi, True)[1]
    hit = int((v0 != pushed).any(axis=1).sum())
    if n > 1000:
        assert hit > (0.3 if nui > 1 else 0.02) * n
        assert c0 >= hit  # an ion may collide more than once
    for order in (np.arange(n)[::-1], rng.permutation(n)):
        p1, v1, m1, c1 = run(p, pos[order], vel[order], phi, True)
        assert np.array_equal(p1, p0[order])
        assert np.array_equal(v1, v0[order])
        assert np.array_equal(m1, m0)
        assert c1 == c0
    p2, v2, m2, _ = run(p, pos, vel, phi, False)
    assert np.array_equal(p2, p0)
    assert np.array_equal(v2, v0)
    assert np.array_equal(m2, m0)
