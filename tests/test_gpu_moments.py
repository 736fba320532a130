"""Moments from the fixed-point accumulators (k_moments), bit for bit against
the oracle's fixed-point deposit: sums above 2^53 quanta, which the conversion
to FP64 rounds to nearest even (thousands of ions in a cell), small ones and
zeros, both signs of the flux, in both layouts of the accumulators (FP64 and
2-D interleaved; the mixed 3-D path's against its interleaved 2-D twin is
covered by the parity tests).
"""
import ctypes

import numpy as np
import pytest

import ecsprt_gb300 as E
from ecsprt_gb300 import _lib
from oracle import oracle as orc

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ndim", [2, 3])
@pytest.mark.parametrize("n, cells", [(1, 1), (20000, 3), (5000, 200)])
def test_fp64_moments_bit_exact(built, ndim, n, cells):
    nx, ny, nz = 9, 7, (5 if ndim == 3 else 1)
    p = E.params_from_options(f"-ndim {ndim} -Nx {nx} -Ny {ny} -dx 1 -dy 1 -qi 1 -mi 1 -B0 0.1 -viT 1 -vi0x 1.0 "
                              f"-nue 8.79e9 -Te 11604.5 -E0 0 -mn 0" + (f" -Nz {nz} -dz 1" if ndim == 3 else ""))
    rng = np.random.default_rng(n + ndim)
    cell = rng.integers(0, cells, n) % (nx * ny * nz)
    pos = np.stack([cell % nx, cell // nx % ny, cell // (nx * ny)], -1)[:, :ndim] + rng.random((n, ndim))
    vel = rng.standard_normal((n, ndim))
    sn, sf = ctypes.c_int32(), ctypes.c_int32()
    assert _lib.gpu().ecs_fix_shifts(ctypes.byref(p), E.ECS_PREC_FP64, ctypes.byref(sn), ctypes.byref(sf)) == 0
    with E.Context(p, E.ECS_PREC_FP64, np_capacity=n) as ctx:
        ctx.upload_particles(pos, vel)
        ctx.collect()
        m = ctx.moments
    ref, _ = orc.Oracle(p).collect_fixed(pos, vel, sn.value, sf.value)
    assert np.array_equal(m, ref)


def test_mixed_3d_moments_are_whole_quanta(built):
    """Mixed sums stay below 2^53 quanta here, so every moment times 2^S is a
    whole number and the totals are the ions' own: 0 tolerance for the first,
    the deposit's half quantum an entry for the second."""
    p = E.params_from_options("-Nx 8 -Ny 6 -Nz 5 -dx 1 -dy 1 -dz 1 -qi 1 -mi 1 -B0 0.1 -viT 1 -vi0x 1.0 -nue 8.79e9 "
                              "-Te 11604.5 -E0 0 -mn 0")
    rng = np.random.default_rng(3)
    n = 4000
    pos, vel = rng.random((n, 3)) * [8, 6, 5], rng.standard_normal((n, 3)).astype(np.float32).astype(float)
    sn, sf = ctypes.c_int32(), ctypes.c_int32()
    assert _lib.gpu().ecs_fix_shifts(ctypes.byref(p), E.ECS_PREC_MIXED, ctypes.byref(sn), ctypes.byref(sf)) == 0
    with E.Context(p, E.ECS_PREC_MIXED, np_capacity=n) as ctx:
        ctx.upload_particles(pos, vel)
        ctx.collect()
        m = ctx.moments
    q = m * 2.0 ** np.array([sn.value] + 3 * [sf.value])
    assert np.array_equal(q, np.rint(q))
    assert (m[..., 1:] < 0).any() and (m[..., 1:] > 0).any()
    # weights are FP32 products: 3 roundings of 2^-24 a weight, 8 weights an ion
    assert np.abs(m[..., 0].sum() - n) <= n * 8 * (3 * 2.0 ** -24 + 2.0 ** -(sn.value + 1))
    for d in range(3):
        tol = np.abs(vel[:, d]).sum() * 8 * 3 * 2.0 ** -24 + n * 8 * 2.0 ** -(sf.value + 1)
        assert abs(m[..., 1 + d].sum() - vel[:, d].sum()) <= tol
