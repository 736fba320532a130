"""The right-hand side's integer products and its reductions at the edges of
their ranges: power-of-two spacings (exponent additions) and others, with and
without a background field, exact zeros and tiny differences, grids of less
than a block, a ragged last block, and more cells than 256 a block.  Against
the oracle (1e-14 relative, the tolerance of the other RHS tests)."""
import numpy as np
import pytest

import ecsprt_gb300 as E
from oracle import oracle as orc
from test_zz_no_alloc import _cudart, _rel_inf, _rhs_noalloc, _rhs_with_context

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("spacing", [(1.0, 1.0, 1.0), (0.5, 4.0, 2.0), (0.7, 1.0, 1.0 / 3.0)], ids=str)
@pytest.mark.parametrize("grid,zbc", [((5, 4, 6), "periodic"), ((33, 31, 29), "periodic"), ((12, 10, 9), "inject-reflect"),
                                      ((128, 128, 65), "periodic")], ids=str)
@pytest.mark.parametrize("E0", [0.0, 0.3])
def test_rhs_at_range_edges(built, spacing, grid, zbc, E0):
    nx, ny, nz = grid
    p = E.params_from_options(f"-Nx {nx} -Ny {ny} -Nz {nz} -dx {spacing[0]!r} -dy {spacing[1]!r} -dz {spacing[2]!r} "
                              f"-qi 1 -mi 1 -B0 0.1 -viT 1 -nue 8.79e9 -Te 11604.5 -E0 {E0} -zBC {zbc}")
    rng = np.random.default_rng(3)
    m = rng.standard_normal((nz, ny, nx, 4))
    m[..., 0] += 16.0
    m[::2, ::3, :, :] = np.round(m[::2, ::3, :, :], 1)  # equal neighbours: differences of exactly zero
    m[1, 1, :, 1:] *= 1e-250
    want = orc.Oracle(p).rhs(m)
    assert _rel_inf(_rhs_with_context(p, m), want) <= 1e-14
    assert _rel_inf(_rhs_noalloc(_cudart(), p, m), want) <= 1e-14
