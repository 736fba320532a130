"""The tile kernel's split of a tile's ions into lane pairs, at the counts where
it can go wrong: one ion, odd counts, around a warp's and a block's worth, and
around the ions of one window (4000), in one tile, in several and in an empty
neighbourhood.

Sums are exact integers and each ion's random numbers are keyed by its identity,
so the order-free kernel (sorting off) gives the same moments bit for bit: after
a deposit, after the pass that counts for a sort and after the one that follows.
"""
import numpy as np
import pytest

import ecsprt_gb300 as E

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 2, 3, 31, 32, 33, 255, 256, 257, 511, 513, 2047, 2049, 3999, 4000, 4001, 8003])
@pytest.mark.parametrize("spread", ["cell", "tile", "grid"])
def test_tile_pass_equals_order_free_pass(built, n, spread):
    nx, ny, nz = 13, 10, 7
    p = E.params_from_options(f"-Nx {nx} -Ny {ny} -Nz {nz} -dx 1 -dy 1 -dz 1 -qi 1 -mi 1 -B0 0.1 -viT 1 -vi0x 1.0 "
                              "-nui 0.02 -nue 8.79e9 -Te 11604.5 -E0 0")
    rng = np.random.default_rng(n)
    size = {"cell": [1, 1, 1], "tile": [4, 4, 2], "grid": [nx, ny, nz]}[spread]
    origin = {"cell": [5, 6, 3], "tile": [4, 4, 2], "grid": [0, 0, 0]}[spread]
    pos = np.array(origin) + rng.random((n, 3)) * size
    vel = rng.standard_normal((n, 3))
    phi = rng.standard_normal((nz, ny, nx))
    out = []
    for every in (2, 0):
        with E.Context(p, E.ECS_PREC_MIXED, np_capacity=n) as ctx:
            ctx.set_sort_every(every)
            ctx.upload_particles(pos, vel)
            ctx.collect()
            m = [ctx.moments]
            for _ in range(3):
                ctx.phi = phi  # the field of every step is given: no solve of a near-empty grid
                ctx.push(0.1)
                ctx.update_positions(0.1)
                ctx.collect()
                m.append(ctx.moments)
            out.append(m)
    for a, b in zip(*out):
        assert np.array_equal(a, b)
