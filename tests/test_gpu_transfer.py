"""The multigrid's fused transfer kernels at the edges of their tiles.

A wrong residual or transfer still lets FGMRES converge, only more slowly, so
each grid's iteration count is pinned to that of the separate kernels: tiles
that end inside the grid along every axis, levels of a few cells more than the
single-block cycle takes, an odd number of planes that are not coarsened, and
-ndim 2, in both precisions.
"""
import numpy as np
import pytest

import ecsprt_gb300 as E

pytestmark = pytest.mark.gpu

# (nx, ny, nz[, "reflect"]): FGMRES iterations to 1e-8, FP64 and mixed
ITERATIONS = {
    (10, 12, 8): (8, 9), (14, 22, 6): (9, 9), (18, 34, 10): (9, 10), (40, 24, 20): (9, 9),
    (10, 12, 7, "reflect"): (8, 8), (34, 18, 5, "reflect"): (8, 8), (36, 20, 33, "reflect"): (8, 9),
    (34, 18, 1): (10, 11), (68, 100, 1): (12, 13), (258, 130, 1): (35, 42),
}


@pytest.mark.parametrize("prec", [E.ECS_PREC_FP64, E.ECS_PREC_MIXED])
@pytest.mark.parametrize("grid", list(ITERATIONS), ids=lambda g: "x".join(map(str, g)))
def test_iterations_at_tile_edges(built, grid, prec):
    nx, ny, nz, *zbc = grid
    p = E.params_from_options(
        f"-Nx {nx} -Ny {ny} -dx 1 -dy 1 -qi 1 -mi 1 -B0 0.1 -viT 1 -nue 8.79e9 -Te 11604.5 -E0 0 " +
        ("-ndim 2 -mn 0" if nz == 1 else f"-Nz {nz} -dz 1") + (" -zBC inject-reflect" if zbc else ""))
    d = np.random.default_rng(5).lognormal(0, 0.1, (nz, ny, nx))
    with E.Context(p, prec) as ctx:
        _, st = ctx.solve_density(d)
    assert st.relres <= 1e-8
    assert st.iterations <= ITERATIONS[grid][prec == E.ECS_PREC_MIXED]
