"""ecs_ctx_device_bytes, by which the server admits requests against its memory
budget, against a sum over the arrays that a context and its solver hold, level
by level of the multigrid hierarchy: periodic grids (every axis halved),
reflecting z (all planes kept on every level) and 2-D (two axes halved), in
both precisions.  Arrays of more than 1 MiB take whole 2 MiB pages.  The
estimate adds the staging of the host transfers, and 16 MiB for what is small
and for the pages of the ion arrays (9 at most, a MiB each on average)."""
import ctypes

import pytest

import ecsprt_gb300 as E
from ecsprt_gb300 import _lib

M = 30  # FGMRES restart length


def _levels(nx, ny, nz, reflect):
    out = [(nx, ny, nz)]
    while len(out) < 12:
        halved = [nx, ny] + ([] if nz == 1 or reflect else [nz])
        if any(a % 2 for a in halved) or (not reflect and min(halved) < 8):
            break
        nx, ny = nx // 2, ny // 2
        nz = nz if nz == 1 or reflect else nz // 2
        out.append((nx, ny, nz))
    return out


def _arrays(nx, ny, nz, reflect, fp64, identity, cap):
    """Bytes of every array, one entry each."""
    n, ne = nx * ny * nz, (nx + 1) * (ny + 1) * (nz + 1)
    tiles = -(-nx // 4) * -(-ny // 4) * -(-nz // 2)
    t = 8 if fp64 else 4
    a = [8 * n, 32 * n, 32 * n, 8 * n, 8 * n]  # potential, moments, accumulators, right-hand side, residual
    a += [(32 if fp64 else 16) * ne, (M + 2) * 4096 * 8, t * n * (M + 1), t * n * (M if fp64 else M + 1)]
    a += 6 * [8 * cap] if fp64 else [32 * cap, 32 * cap, 4 * cap, 4 * cap, 128 * tiles, 128 * tiles, 8 * tiles + 4]
    if identity:
        return a
    a.append(88 * n)
    for l, (x, y, z) in enumerate(_levels(nx, ny, nz, reflect)):
        cells = x * y * z
        a += (11 if fp64 or z > 128 else 7) * [t * cells] + 2 * [t * x * y] + ([88 * cells] if fp64 and l > 0 else [])
    return a + ([t * cells * cells] if cells <= 128 else [])


@pytest.mark.parametrize("fp64", [False, True], ids=["mixed", "fp64"])
@pytest.mark.parametrize("grid", [(4, 4, 4, False), (128, 128, 128, False), (256, 256, 128, False), (100, 72, 50, False),
                                  (64, 64, 256, False), (256, 256, 128, True), (512, 512, 64, True), (37, 50, 61, True),
                                  (64, 64, 200, True), (1024, 1024, 1, False), (258, 130, 1, False)], ids=str)
@pytest.mark.parametrize("identity,ppc", [(False, 0), (False, 16), (True, 0)])
def test_estimate_covers_every_array(built, grid, fp64, identity, ppc):
    nx, ny, nz, reflect = grid
    o = f"-Nx {nx} -Ny {ny} -dx 1 -dy 1 " + ("-ndim 2 -mn 0" if nz == 1 else f"-Nz {nz} -dz 1")
    p = E.params_from_options(o + (" -zBC inject-reflect" if reflect else "") + (" -lhs identity" if identity else ""))
    cap = nx * ny * nz * ppc
    est = _lib.gpu().ecs_ctx_device_bytes(ctypes.byref(p), E.ECS_PREC_FP64 if fp64 else E.ECS_PREC_MIXED, cap)
    arrays = _arrays(nx, ny, nz, reflect, fp64, identity, cap)
    pages = sum(-(-b // (2 << 20)) * (2 << 20) if b > 1 << 20 else b for b in arrays)
    staging = 0 if cap == 0 else 5 * 48 * min(cap, 1 << 22) + (5 << 21)  # five buffers of at most 2^22 ions
    assert pages <= est <= pages + staging + (17 << 20)
