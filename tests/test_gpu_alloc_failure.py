"""A call that runs out of memory leaves the context usable: whichever of its
allocations fails, it returns ECS_ERR_NOMEM, and the same call made again gives
the bits of a context that never failed.  (A multigrid hierarchy, a set of staging
buffers or a pair of Krylov bases that stays half-made is taken for a whole one
by the next call; the server hands such a context to the next request.)

No memory is filled up: a library loaded before the CUDA runtime answers one
cudaMalloc or cudaMallocHost, chosen by its number, with an error.
"""
import os
import subprocess
import sys

import pytest

from conftest import ROOT

pytestmark = pytest.mark.gpu

SHIM = r"""
#define _GNU_SOURCE
#include <dlfcn.h>
#include <stddef.h>
static long left = -1, failed = 0;
void shim_arm(long n) { left = n; failed = 0; }
long shim_failed(void) { return failed; }
static int fails(void) { if (left < 0 || left-- > 0) return 0; failed = 1; return 1; }
static int real(const char *name, void **p, size_t n) {
  void *rt = dlopen("libcudart.so.13", RTLD_LAZY | RTLD_NOLOAD);
  int (*f)(void **, size_t) = rt ? (int (*)(void **, size_t))dlsym(rt, name) : NULL;
  return f ? f(p, n) : 999;
}
int cudaMalloc(void **p, size_t n) { return fails() ? 2 : real("cudaMalloc", p, n); }
int cudaMallocHost(void **p, size_t n) { return fails() ? 2 : real("cudaMallocHost", p, n); }
"""

PROGRAM = r"""
import ctypes, sys
import numpy as np
import ecsprt_gb300 as E

what, prec = sys.argv[1], {"mixed": E.ECS_PREC_MIXED, "fp64": E.ECS_PREC_FP64}[sys.argv[2]]
shim = ctypes.CDLL(None)
shim.shim_arm.argtypes = [ctypes.c_long]
shim.shim_failed.restype = ctypes.c_long
p = E.params_from_options("-Nx 20 -Ny 12 -Nz 16 -dx 1 -dy 1 -dz 1 -qi 1 -mi 1 -B0 0.1 -viT 1 -nue 8.79e9 -Te 11604.5 -E0 0 -mn 0")
n = 20 * 12 * 16 * 8
rng = np.random.default_rng(1)
pos, vel = rng.random((n, 3)) * [20, 12, 16], 0.1 * rng.standard_normal((n, 3))
density = 1.0 + 0.3 * rng.random((16, 12, 20))

def call(ctx, first):
    if what == "request":
        return ctx.solve_density(density)[0].copy()
    if what == "slots":
        ctx.moments = np.stack([density, density, density, density], -1)
        ctx.compute_potential(1e-8, 200)
        return ctx.phi
    if what == "step":  # the ions anew: a step that failed behind its particle pass has moved them
        ctx.upload_particles(pos, vel)
        ctx.phi = np.zeros_like(density)
        ctx.step(0.01, 1e-8, 200)
        return ctx.phi
    ctx.phi = np.zeros_like(density)  # two host steps: the second is pipelined
    hp, hv = pos.copy(), vel.copy()
    hm = np.empty(density.shape + (4,))
    for _ in range(2):
        ctx.step_host(hp, hv, 0.01, 1e-8, 200, hm)
    return np.concatenate([ctx.phi.ravel(), hm.ravel()])

def fresh():
    return E.Context(p, prec, np_capacity=n)

with fresh() as ctx:
    want = call(ctx, True)
at = 0
while True:
    shim.shim_arm(at)
    ctx = None
    try:
        ctx = fresh()
        got = call(ctx, True)
    except E.EcsError as e:
        assert e.code == E._lib.ECS_ERR_NOMEM, e
        assert shim.shim_failed() == 1, e
    failed = shim.shim_failed()
    shim.shim_arm(-1)
    if failed:
        if ctx is None:
            ctx = fresh()
        got = call(ctx, False)
    assert np.array_equal(got, want), at
    ctx.close()
    if not failed:
        break
    at += 1
print("allocations", at)
assert at >= 20
"""


@pytest.mark.parametrize("prec", ["mixed", "fp64"])
@pytest.mark.parametrize("what", ["request", "slots", "step", "host"])
def test_every_allocation_may_fail(built, tmp_path, what, prec):
    (tmp_path / "shim.c").write_text(SHIM)
    (tmp_path / "program.py").write_text(PROGRAM)
    subprocess.run(["gcc", "-shared", "-fPIC", "-O1", "-o", str(tmp_path / "shim.so"), str(tmp_path / "shim.c"), "-ldl"],
                   check=True)
    env = dict(os.environ, LD_PRELOAD=str(tmp_path / "shim.so"), PYTHONPATH=str(ROOT))
    r = subprocess.run([sys.executable, str(tmp_path / "program.py"), what, prec], env=env, capture_output=True, text=True,
                       timeout=300, cwd=ROOT)
    assert r.returncode == 0, r.stdout + r.stderr
