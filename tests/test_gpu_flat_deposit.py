"""The 2-D deposit of the mixed path (k_particles32<true>) adds ions one by one
or by cells, as the cells of a warp's ions fall.

The deposit's sums are integers, so the moments of the same ions are equal bit
for bit in any ion order; against FP64 sums of the weights (numpy) the
density's tolerance is that of the 2-D parity tests, 1e-6 relative.
"""
import numpy as np
import pytest

import ecsprt_gb300 as E

pytestmark = pytest.mark.gpu


def _density(pos, nx, ny):
    c = np.floor(pos).astype(int)
    o = pos - c
    out = np.zeros((ny, nx))
    for b in range(4):
        xb, yb = b & 1, b >> 1
        w = np.where(xb, o[:, 0], 1 - o[:, 0]) * np.where(yb, o[:, 1], 1 - o[:, 1])
        np.add.at(out, ((c[:, 1] + yb) % ny, (c[:, 0] + xb) % nx), w)
    return out


# one ion, a warp less one, a warp and one (last warp nearly empty), warps of
# exactly 8 and 9 cells (either side of the rule), one cell a warp, many
@pytest.mark.parametrize("n, cells", [(1, 1), (31, 1), (33, 33), (256, 8), (288, 9), (512, 16), (4096, 5), (5000, 323)])
def test_moments_do_not_depend_on_the_order(built, n, cells):
    nx, ny = 19, 17
    p = E.params_from_options(f"-ndim 2 -Nx {nx} -Ny {ny} -dx 1 -dy 1 -qi 1 -mi 1 -B0 0.1 -viT 1 -vi0x 1.0 "
                              "-nue 8.79e9 -Te 11604.5 -E0 0 -mn 0")
    rng = np.random.default_rng(n + cells)
    cell = rng.permutation(nx * ny)[np.arange(n) % cells]
    pos = np.stack([cell % nx + rng.random(n), cell // nx + rng.random(n)], -1)
    vel = rng.standard_normal((n, 2))
    moments = []
    for order in (np.arange(n), np.argsort(cell, kind="stable"), rng.permutation(n)):
        with E.Context(p, E.ECS_PREC_MIXED, np_capacity=n) as ctx:
            ctx.set_sort_every(0)
            ctx.upload_particles(pos[order], vel[order])
            ctx.collect()
            moments.append(ctx.moments)
    ref = _density(pos, nx, ny)
    assert np.abs(moments[0][0, ..., 0] - ref).max() <= 1e-6 * ref.max()
    assert np.array_equal(moments[0], moments[1])
    assert np.array_equal(moments[0], moments[2])
