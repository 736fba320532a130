"""The multigrid smoother's kernels at the edges of their ranges.

A wrong z-line factor, halo row or transfer still lets FGMRES converge, only
more slowly, so each grid's iteration count is pinned to that of the plain
launches (one right-hand side and one z-line solve a sweep, factors read from
memory): columns of one, two and sixteen segments with a partial last one, of
more than 128 cells (segments of 16), coarsest levels solved by the inverse,
by the single block and by clusters of 1 to 16 CTAs with uneven rows, levels
coarsened in x and y only, and -ndim 2.
"""
import numpy as np
import pytest

import ecsprt_gb300 as E
from ecsprt_gb300 import workloads as W

pytestmark = pytest.mark.gpu

# (nx, ny, nz[, "reflect"]): FGMRES iterations to 1e-8, mixed precision
ITERATIONS = {
    (12, 10, 9): 6, (17, 13, 11): 8, (21, 19, 25): 11, (33, 31, 29): 17, (50, 36, 28): 11, (66, 54, 42): 15,
    (9, 25, 100): 15, (64, 64, 9): 24, (16, 16, 160): 10, (30, 30, 30): 9, (48, 48, 48): 9,
    (33, 21, 32, "reflect"): 14, (64, 64, 32, "reflect"): 9, (130, 66, 1): 29, (128, 128, 1): 10,
    # rows four cells a thread: the smallest level that takes them, rows of one and of 128 packs, ghosts, one plane
    (128, 128, 4): 43, (132, 100, 68): 14, (4, 256, 128): 81, (512, 128, 4, "reflect"): 8, (256, 256, 1): 10,
}


def params(grid):
    nx, ny, nz, *zbc = grid
    return E.params_from_options(
        f"-Nx {nx} -Ny {ny} -dx 1 -dy 1 -qi 1 -mi 1 -B0 0.1 -viT 1 -nue 8.79e9 -Te 11604.5 -E0 0 " +
        ("-ndim 2 -mn 0" if nz == 1 else f"-Nz {nz} -dz 1") + (" -zBC inject-reflect" if zbc else ""))


@pytest.mark.parametrize("grid", list(ITERATIONS), ids=lambda g: "x".join(map(str, g)))
def test_iterations_at_segment_and_cluster_edges(built, grid):
    nx, ny, nz = grid[:3]
    rng = np.random.default_rng(5)
    d = rng.lognormal(0, 0.1, (nz, ny, nx)) * (1 + W.fourier_modes((nz, ny, nx), 12, 0.05, rng))
    d = np.maximum(d, 0.05)
    with E.Context(params(grid), E.ECS_PREC_MIXED) as ctx:
        phi, st = ctx.solve_density(d)
        phi = phi.copy()
        again, _ = ctx.solve_density(d)
    assert st.relres <= 1e-8
    assert st.iterations <= ITERATIONS[grid]
    assert np.array_equal(phi, again)  # fixed orders throughout: bit-identical on repetition


@pytest.mark.parametrize("prec", [E.ECS_PREC_FP64, E.ECS_PREC_MIXED])
@pytest.mark.parametrize("grid", [(4, 4, 4), (4, 4, 8), (5, 5, 5), (4, 8, 4), (5, 5, 4, "reflect"), (5, 5, 5, "reflect")],
                         ids=lambda g: "x".join(map(str, g)))
def test_coarsest_inverse_is_the_inverse(built, grid, prec):
    """Grids of one level (64 to 128 cells: each kernel, and its last row) are solved
    by the coarsest inverse alone: one or two preconditioned steps, for each
    of the two refinement sweeps in mixed precision."""
    nx, ny, nz = grid[:3]
    rng = np.random.default_rng(7)
    d = 1.0 + 0.3 * rng.standard_normal((nz, ny, nx)).clip(-2, 2)
    with E.Context(params(grid), prec) as ctx:
        _, st = ctx.solve_density(d)
    assert st.relres <= 1e-8
    assert st.iterations <= (2 if prec == E.ECS_PREC_FP64 else 4)
