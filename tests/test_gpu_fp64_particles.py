"""The FP64 particle pass at the edges of its integer arithmetic, bit for bit
against the oracle: cell widths that are powers of two (an exponent shift) and
others (a corrected reciprocal), positions at zero, on cell faces, one step
below the upper bound and at tiny values, exact-zero and tiny weights, and ion
counts around a warp.
"""
import ctypes

import numpy as np
import pytest

import ecsprt_gb300 as E
from ecsprt_gb300 import _lib
from oracle import oracle as orc

pytestmark = pytest.mark.gpu


def ions(rng, n, L, widths):
    pos = rng.uniform(0, 1, (n, 3)) * L
    k = min(n, 64)
    for d in range(3):
        cell = rng.integers(0, int(round(L[d] / widths[d])), k)
        pos[:k:4, d] = (cell * widths[d])[::4] % L[d]     # on a face
        pos[1:k:4, d] = np.nextafter(L[d], 0.0)           # below the upper bound
        pos[2:k:4, d] = 0.0
        pos[3:k:4, d] = 10.0 ** -rng.uniform(5, 200, pos[3:k:4, d].shape)
    pos = np.where(pos >= L, np.nextafter(L, 0.0), pos)
    vel = rng.standard_normal((n, 3))
    vel[:k:5] = 0.0
    return pos, vel


@pytest.mark.parametrize("widths", [(1.0, 1.0, 1.0), (0.25, 2.0, 0.5), (0.7, 1.0 / 3.0, 3.0), (1e-3, 5.1, 1.0)],
                         ids=lambda w: "x".join(f"{x:.3g}" for x in w))
@pytest.mark.parametrize("n", [1, 33, 5000])
@pytest.mark.parametrize("zbc", ["periodic", "inject-reflect"])
def test_fp64_pass_bit_exact(built, widths, n, zbc):
    nx, ny, nz = 7, 6, 9
    p = E.params_from_options(f"-Nx {nx} -Ny {ny} -Nz {nz} -dx {widths[0]!r} -dy {widths[1]!r} -dz {widths[2]!r} -qi 1 "
                              f"-mi 1 -B0 0.1 -viT 1 -vi0x 0.5 -nue 8.79e9 -Te 11604.5 -E0 0 -mn 0 -zBC {zbc}")
    rng = np.random.default_rng(11)
    L = np.array([p.Lx, p.Ly, p.Lz])
    pos, vel = ions(rng, n, L, widths)
    vel *= np.array(widths) / 0.1 * 0.4  # up to about a cell a step
    vel = np.clip(vel, -15.0, 15.0)
    phi = rng.standard_normal((nz, ny, nx)) * 10.0 ** rng.integers(-12, 1, (nz, ny, nx))
    phi[::2, ::3] = 0.0
    O = orc.Oracle(p)
    sn, sf = ctypes.c_int32(), ctypes.c_int32()
    assert _lib.gpu().ecs_fix_shifts(ctypes.byref(p), E.ECS_PREC_FP64, ctypes.byref(sn), ctypes.byref(sf)) == 0
    with E.Context(p, E.ECS_PREC_FP64, np_capacity=n) as ctx:
        ctx.upload_particles(pos, vel)
        ctx.phi = phi
        ctx.collect()
        m0 = ctx.moments
        ctx.push(0.1)
        _, v1 = ctx.download_particles()
        ctx.update_positions(0.1)
        p2, v2 = ctx.download_particles()
    want0, _ = O.collect_fixed(pos, vel, sn.value, sf.value)
    assert np.array_equal(m0, want0)
    w1 = O.push(pos, vel, phi, 0.1)
    assert np.array_equal(v1, w1)
    wp, wv = O.move(pos, w1, 0.1)
    assert np.array_equal(p2, wp)
    assert np.array_equal(v2, wv)
