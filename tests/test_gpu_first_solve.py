"""A context's solver state is zeroed when its first solve allocates it, on the
context's own stream: the default stream is not ordered with it, and its memset
waits behind the transfers of a host step, so that it could run during the solve
and end it with a potential of 0.

The sources are read for any other work on the default stream; on the GPU, fresh
contexts take a host step first, whose transfers are long beside the solve, and
give the potential of the device-resident step bit for bit.
"""
import re

import numpy as np
import pytest

import ecsprt_gb300 as E
from ecsprt_gb300 import build as b


@pytest.mark.parametrize("src", sorted(b.CSRC.glob("*.cu")), ids=lambda s: s.name)
def test_no_work_on_the_default_stream(src):
    text = re.sub(r"//[^\n]*", "", src.read_text())
    assert not re.findall(r"\bcudaMem(?:set|cpy)(?:2D|3D)?\(", text)
    for config in re.findall(r"<<<(.*?)>>>", text, re.S):
        assert config.count(",") >= 3, config


@pytest.mark.gpu
@pytest.mark.parametrize("prec", [E.ECS_PREC_MIXED, E.ECS_PREC_FP64])
def test_first_solve_behind_transfers(built, prec):
    p = E.params_from_options("-Nx 8 -Ny 8 -Nz 8 -dx 1 -dy 1 -dz 1 -qi 1 -mi 1 -B0 0.1 -viT 0.1 -vi0x 0.1 "
                              "-nue 8.79e9 -Te 11604.5 -E0 0 -mn 0")
    n = 300_000
    rng = np.random.default_rng(17)
    pos, vel = rng.uniform(0, 8, (n, 3)), 0.1 * rng.standard_normal((n, 3))
    hp, hv = E.pinned_empty((n, 3)), E.pinned_empty((n, 3))
    with E.Context(p, prec, np_capacity=n) as ctx:
        ctx.upload_particles(pos, vel)
        ctx.step(0.01, 1e-8, 400)
        want = ctx.phi
    assert np.abs(want).max() > 0.0
    for _ in range(12):
        with E.Context(p, prec, np_capacity=n) as ctx:
            hp[:], hv[:] = pos, vel
            ctx.step_host(hp, hv, 0.01, 1e-8, 400)
            assert np.array_equal(ctx.phi, want)
