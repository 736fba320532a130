"""The work that a user of ecsprt_gb300 has it do, as cases that can be timed.

Each case goes through the entry points that a program calls (the Python
``Context`` and the C ABI of include/ecsgpu.h), at sizes of this repository's
benchmark, serving workloads and tests:

* ``rhs``    the right-hand side on device buffers that the caller owns
             (``ecs_rhs_noalloc``), for a framework with its own memory pool;
* ``solve``  one stand-alone potential solve (``solve_density``): a density in
             page-locked host memory in, the potential out;
* ``step``   the time loop of the ``pic`` program over one output interval:
             ``steps`` whole time steps, then the moments and the potential
             read into page-locked host arrays (FP64: the ions too; the mixed
             path's cell sort leaves ions of one cell in any order, so there
             the moments, which do not depend on it, stand for them);
* ``slots``  the same loop through the reference's operator slots (push,
             collide, move, collect, potential), without collisions;
* ``host``   time steps through host buffers (``step_host``): ions in and out
             of page-locked host memory every step.

``exact`` restates the right-hand side, the operator and the particle update
in torch FP64, with the potential solved by FFT-preconditioned BiCGStab.
"""
from __future__ import annotations

import ctypes
import math

import numpy as np
import torch

import ecsprt_gb300 as E
from ecsprt_gb300 import _lib

DT = 0.1
RTOL = 1e-8
MAX_IT = 300
PREC = {"mixed": E.ECS_PREC_MIXED, "fp64": E.ECS_PREC_FP64}


def listed():
    return [
        # a caller with its own memory pool asks for the right-hand side alone: the smallest call
        {"name": "rhs_32", "kind": "rhs", "nx": 32, "ny": 32, "nz": 32},
        # stand-alone solves of the serving workload: its smallest grid ...
        {"name": "solve_32", "kind": "solve", "prec": "mixed", "nx": 32, "ny": 32, "nz": 32},
        # ... and a large one whose multigrid ends at 6^3
        {"name": "solve_96", "kind": "solve", "prec": "mixed", "nx": 96, "ny": 96, "nz": 96},
        # a grid that the user's domain dictates: it coarsens once, then an axis is odd
        {"name": "solve_ragged", "kind": "solve", "prec": "mixed", "nx": 100, "ny": 72, "nz": 50},
        # the plain FP64 solver, for users who do not want mixed precision
        {"name": "solve_fp64_64", "kind": "solve", "prec": "fp64", "nx": 64, "ny": 64, "nz": 64},
        # a small simulation (an ensemble member, 16 ions a cell): latency of the whole step
        {"name": "step_32", "kind": "step", "prec": "mixed", "nx": 32, "ny": 32, "nz": 32, "ppc": 16, "bcz": "periodic",
         "steps": 10},
        # the benchmark's time step: 128^3, 64 ions a cell
        {"name": "step_128", "kind": "step", "prec": "mixed", "nx": 128, "ny": 128, "nz": 128, "ppc": 64,
         "bcz": "periodic", "steps": 4},
        # the largest: 256 x 256 x 128 with a reflecting z, 32 ions a cell
        {"name": "step_reflect_256", "kind": "step", "prec": "mixed", "nx": 256, "ny": 256, "nz": 128, "ppc": 32,
         "bcz": "reflect", "steps": 2},
        # the plain FP64 path, which follows the reference operand for operand
        {"name": "step_fp64_64", "kind": "step", "prec": "fp64", "nx": 64, "ny": 64, "nz": 64, "ppc": 64,
         "bcz": "periodic", "steps": 2},
        # -ndim 2
        {"name": "step_2d_256", "kind": "step", "prec": "mixed", "nx": 256, "ny": 256, "nz": 1, "ppc": 64,
         "bcz": "periodic", "steps": 4},
        # the reference's loop order through its operator slots
        {"name": "slots_64", "kind": "slots", "prec": "mixed", "nx": 64, "ny": 64, "nz": 64, "ppc": 16},
        # ions that live in the caller's host arrays
        {"name": "host_64", "kind": "host", "prec": "mixed", "nx": 64, "ny": 64, "nz": 64, "ppc": 64, "steps": 2},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _axis(rng, lo, hi):
    """A grid axis: odd, even, or a multiple of 8 or 16, as domains come."""
    n = _log_int(rng, lo, hi)
    m = rng.choice((1, 2, 4, 8, 16))
    return max(lo, n // m * m)


def draw(rng):
    kind = rng.choice(("rhs", "solve", "solve", "solve", "step", "step", "step", "step", "slots", "host"))
    if kind == "rhs":
        return {"kind": kind, "nx": _axis(rng, 8, 128), "ny": _axis(rng, 8, 128), "nz": _axis(rng, 8, 128)}
    if kind == "solve":
        prec = rng.choice(("mixed", "mixed", "fp64"))
        hi = 128 if prec == "mixed" else 80
        return {"kind": kind, "prec": prec, "nx": _axis(rng, 16, hi), "ny": _axis(rng, 16, hi), "nz": _axis(rng, 16, hi)}
    prec = rng.choice(("mixed", "mixed", "mixed", "fp64"))
    case = {"kind": kind, "prec": prec}
    hi = 96 if prec == "mixed" else 48
    if kind == "step" and rng.random() < 0.3:  # -ndim 2
        case |= {"nx": _axis(rng, 32, 320), "ny": _axis(rng, 32, 320), "nz": 1, "bcz": "periodic"}
    else:
        case |= {"nx": _axis(rng, 16, hi), "ny": _axis(rng, 16, hi), "nz": _axis(rng, 16, hi)}
        if kind == "step":
            case["bcz"] = rng.choice(("periodic", "periodic", "reflect"))
    case["ppc"] = _log_int(rng, 8, 96)
    if kind != "slots":
        case["steps"] = rng.choice((2, 3, 4))
    return case


# ---- what a program has in hand ------------------------------------------------
def _params(case):
    """The benchmark's plasma: kappa_e about 2, ions of thermal speed 1 drifting along x."""
    flat = case["nz"] == 1
    o = f"-Nx {case['nx']} -Ny {case['ny']} -dx 1 -dy 1 " + ("-ndim 2 " if flat else f"-Nz {case['nz']} -dz 1 ")
    o += "-qi 1 -mi 1 -B0 0.1 -viT 1 -vi0x 1.0 -nui 0.02 -nue 8.79e9 -Te 11604.5 -E0 0"
    if flat or case["kind"] in ("slots", "host"):
        o += " -mn 0"  # no neutrals (collisions are not defined in 2-D)
    if case.get("bcz") == "reflect":
        o += " -zBC inject-reflect"
    return E.params_from_options(o)


def _density(case, seed):
    """The serving workload's density, lognormal(0, 0.1) x (1 + 12 Fourier modes of amplitude 0.05), FP64."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    nz, ny, nx = case["nz"], case["ny"], case["nx"]
    n = torch.exp(0.1 * torch.randn((nz, ny, nx), generator=g, device="cuda", dtype=torch.float64))
    z, y, x = (2.0 * math.pi * torch.arange(m, device="cuda", dtype=torch.float64) / m for m in (nz, ny, nx))
    r = np.random.default_rng(seed)
    s = torch.zeros_like(n)
    for _ in range(12):
        k, ph = r.integers(-4, 5, size=3), r.uniform(0.0, 2.0 * math.pi)
        s += 0.05 * torch.cos(int(k[2]) * z[:, None, None] + int(k[1]) * y[None, :, None] + int(k[0]) * x + ph)
    return n * (1.0 + s)


def _ions(case, seed):
    """Ions (x by inversion of 1 + 0.05 sin(2 pi x/L) to first order, y and z uniform), Maxwellian plus the drift."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    N = case["nx"] * case["ny"] * case["nz"] * case["ppc"]
    u = torch.rand((N, 3), generator=g, device="cuda", dtype=torch.float64)
    u[:, 0] = (u[:, 0] + 0.05 / (2.0 * math.pi) * (torch.cos(2.0 * math.pi * u[:, 0]) - 1.0)) % 1.0
    pos = u * torch.tensor([case["nx"], case["ny"], case["nz"]], device="cuda", dtype=torch.float64)
    vel = torch.randn((N, 3), generator=g, device="cuda", dtype=torch.float64)
    vel[:, 0] += 1.0
    return pos, vel


def _pinned(t):
    a = E.pinned_empty(tuple(t.shape))
    torch.from_numpy(a).copy_(t)
    return a


def _phi(case):
    """A smooth potential, the one that the ions start with."""
    nz, ny, nx = case["nz"], case["ny"], case["nx"]
    z, y, x = (2.0 * np.pi * np.arange(m) / m for m in (nz, ny, nx))
    return 0.1 * np.sin(x)[None, None, :] + 0.05 * np.cos(y)[None, :, None] + 0.05 * np.sin(2 * z)[:, None, None]


def prepare(case, seed):
    p = _params(case)
    shape = (p.Nz, p.Ny, p.Nx)
    s = {"case": case, "p": p}
    if case["kind"] == "rhs":
        g = torch.Generator(device="cuda").manual_seed(seed)
        m = torch.randn(shape + (4,), generator=g, device="cuda", dtype=torch.float64)
        m[..., 0] = 16.0 * _density(case, seed)
        m[..., 1:] *= 4.0
        s |= {"moments": m, "rhs": torch.empty(shape, device="cuda", dtype=torch.float64)}
        return s
    if case["kind"] == "solve":
        s["ctx"] = E.Context(p, PREC[case["prec"]])
        s["density"] = _pinned(_density(case, seed))
        s["phi"] = E.pinned_empty(shape)
        return s
    N = p.Nx * p.Ny * p.Nz * case["ppc"]
    s["ctx"] = ctx = E.Context(p, PREC[case["prec"]], np_capacity=N)
    s["phi"], s["mom"] = E.pinned_empty(shape), E.pinned_empty(shape + (4,))
    ctx.phi = _phi(case)
    if case["kind"] == "step":
        ctx.init_particles(E.ECS_INIT_MODES, N, seed, modes=[(1, 0, 0, 0.05, -0.5 * math.pi)])
        if case["prec"] == "fp64":
            s["pos"], s["vel"] = E.pinned_empty((N, ctx.nd)), E.pinned_empty((N, ctx.nd))
        return s
    pos, vel = _ions(case, seed)
    s["pos"], s["vel"] = _pinned(pos), _pinned(vel)
    if case["kind"] == "slots":
        ctx.upload_particles(s["pos"], s["vel"])
    return s


def _read(ctx, s):
    """The moments and the potential of this output time, into the program's page-locked arrays."""
    ctx._check(_lib.gpu().ecs_moments_download(ctx.handle, ctypes.c_void_p(s["mom"].ctypes.data)))
    ctx._check(_lib.gpu().ecs_phi_download(ctx.handle, ctypes.c_void_p(s["phi"].ctypes.data)))


def run(s):
    kind = s["case"]["kind"]
    if kind == "rhs":
        rc = _lib.gpu().ecs_rhs_noalloc(ctypes.byref(s["p"]), ctypes.c_void_p(s["moments"].data_ptr()),
                                        ctypes.c_void_p(s["rhs"].data_ptr()),
                                        ctypes.c_void_p(torch.cuda.current_stream().cuda_stream))
        if rc:
            raise E.EcsError(rc, _lib.gpu().ecs_last_error(None).decode())
        return s["rhs"]
    ctx = s["ctx"]
    if kind == "solve":
        phi, _ = ctx.solve_density(s["density"], (1.0, 0.5, 0.25), RTOL, MAX_IT, phi_out=s["phi"])
        return phi
    if kind == "slots":
        ctx.update_velocities(DT)
        ctx.update_positions(DT)
        ctx.collect()
        ctx.compute_potential(RTOL, MAX_IT)
        _read(ctx, s)
        return {"moments": s["mom"], "phi": s["phi"]}
    collisions = 0
    for _ in range(s["case"]["steps"]):
        if kind == "host":
            st = ctx.step_host(s["pos"], s["vel"], DT, RTOL, MAX_IT, moments_out=s["mom"], phi_out=s["phi"])
        else:
            st = ctx.step(DT, RTOL, MAX_IT)
        collisions += st.collisions
    out = {"moments": s["mom"], "phi": s["phi"], "collisions": int(collisions)}
    if kind == "step":
        _read(ctx, s)
        if s["case"]["prec"] == "fp64":  # the program's particle output
            ctx._check(_lib.gpu().ecs_particles_download(ctx.handle, ctypes.c_void_p(s["pos"].ctypes.data),
                                                         ctypes.c_void_p(s["vel"].ctypes.data)))
            out |= {"pos": s["pos"], "vel": s["vel"]}
    return out


def work(case):
    """The ions' state read and written each step (28 bytes mixed, 48 in FP64 and on the host), the
    grid fields in and out of each field phase (moments, potential), FP64."""
    cells = case["nx"] * case["ny"] * case["nz"]
    if case["kind"] == "rhs":
        return {"bytes": 40.0 * cells, "flops": 40.0 * cells}
    if case["kind"] == "solve":
        return {"bytes": 16.0 * cells, "flops": 40.0 * cells}
    steps = case.get("steps", 1)
    ion = 96.0 if case["prec"] == "fp64" or case["kind"] == "host" else 56.0
    n = cells * case["ppc"]
    return {"bytes": steps * (ion * n + 40.0 * cells), "flops": steps * (250.0 * n + 40.0 * cells)}


# ---- the same in plain torch, FP64 ------------------------------------------------
def _sh(f, dx=0, dy=0, dz=0):
    """f at (i + dx, j + dy, k + dz) on a periodic grid."""
    return torch.roll(f, (-dz, -dy, -dx), (0, 1, 2))


def _exact_rhs(p, n, gx, gy, gz):
    kap = p.kappa_e
    dndx = (_sh(n, dx=1) - _sh(n, dx=-1)) / (2 * p.dx)
    dndy = (_sh(n, dy=1) - _sh(n, dy=-1)) / (2 * p.dy)
    d2 = ((_sh(n, dx=1) - 2 * n + _sh(n, dx=-1)) / p.dx ** 2 + (_sh(n, dy=1) - 2 * n + _sh(n, dy=-1)) / p.dy ** 2 +
          (1 + kap * kap) * (_sh(n, dz=1) - 2 * n + _sh(n, dz=-1)) / p.dz ** 2)
    div = ((_sh(gx, dx=1) - _sh(gx, dx=-1)) / (2 * p.dx) + (_sh(gy, dy=1) - _sh(gy, dy=-1)) / (2 * p.dy) +
           (_sh(gz, dz=1) - _sh(gz, dz=-1)) / (2 * p.dz))
    b = p.scale * ((dndy - kap * dndx) * p.E0 + p.cth * d2 + p.cG * div)
    return b - b.mean()


def _exact_solve(p, n, b):
    """phi with A(n) phi = b and zero mean, by BiCGStab preconditioned with the mean density's operator."""
    kap, sc = p.kappa_e, p.scale
    sx, sy, sz = sc / (2 * p.dx ** 2), sc / (2 * p.dy ** 2), sc * (1 + kap * kap) / (2 * p.dz ** 2)
    so = sc * kap / (8 * p.dx * p.dy)
    xp, xm, yp, ym, zp, zm = _sh(n, dx=1), _sh(n, dx=-1), _sh(n, dy=1), _sh(n, dy=-1), _sh(n, dz=1), _sh(n, dz=-1)
    rows = [((1, 0, 0), sx * (xp + n) + so * (yp - ym)), ((-1, 0, 0), sx * (n + xm) - so * (yp - ym)),
            ((0, 1, 0), sy * (yp + n) - so * (xp - xm)), ((0, -1, 0), sy * (n + ym) + so * (xp - xm)),
            ((0, 0, 1), sz * (zp + n)), ((0, 0, -1), sz * (n + zm)),
            ((1, 1, 0), so * (yp - xp)), ((1, -1, 0), so * (xp - ym)),
            ((-1, 1, 0), so * (xm - yp)), ((-1, -1, 0), so * (ym - xm))]
    diag = -(sx * (xp + 2 * n + xm) + sy * (yp + 2 * n + ym) + sz * (zp + 2 * n + zm))

    def A(x):
        y = diag * x
        for (i, j, k), c in rows:
            y = y + c * _sh(x, i, j, k)
        return y

    ang = [2 * math.pi * torch.fft.fftfreq(m, device=n.device, dtype=torch.float64) for m in n.shape]
    ez, ey, ex = (2 * (torch.cos(a) - 1) for a in ang)
    lam = 2 * n.mean() * (sz * ez[:, None, None] + sy * ey[None, :, None] + sx * ex)
    lam[0, 0, 0] = 1.0

    def M(r):
        f = torch.fft.fftn(r) / lam
        f[0, 0, 0] = 0.0
        return torch.fft.ifftn(f).real

    x = torch.zeros_like(b)
    r = b.clone()
    r0, rho, alpha, om, v, q = r.clone(), 1.0, 1.0, 1.0, torch.zeros_like(b), torch.zeros_like(b)
    for _ in range(200):
        rho1 = float((r0 * r).sum())
        q = r + (rho1 / rho) * (alpha / om) * (q - om * v)
        y = M(q)
        v = A(y)
        alpha = rho1 / float((r0 * v).sum())
        h = r - alpha * v
        z = M(h)
        t = A(z)
        om = float((t * h).sum() / (t * t).sum())
        x = x + alpha * y + om * z
        r = h - om * t
        rho = rho1
        if float(r.norm()) <= 1e-13 * float(b.norm()):
            break
    x = x + M(b - A(x))
    return x - x.mean()


def _exact_slots(case, seed):
    """One pass of the operator slots from the state that prepare() makes."""
    p = _params(case)
    pos, vel = _ions(case, seed)
    phi = torch.from_numpy(_phi(case)).cuda()
    N = (p.Nx, p.Ny, p.Nz)
    # differences at the nodes 0..N along each axis: central, and the backward formula at node N
    ext = torch.nn.functional.pad(phi[None, None], (0, 1, 0, 1, 0, 1), mode="circular")[0, 0]
    D = []
    for axis in range(3):
        dim = 2 - axis
        d = torch.roll(phi, -1, dim) - torch.roll(phi, 1, dim)
        d = torch.nn.functional.pad(d[None, None], (0, 1, 0, 1, 0, 1), mode="circular")[0, 0].clone()
        last = ext.narrow(dim, 0, 1) * 3 - 4 * ext.narrow(dim, N[axis] - 1, 1) + ext.narrow(dim, N[axis] - 2, 1)
        d.narrow(dim, N[axis], 1).copy_(last)
        D.append(d)
    cell = pos.floor().long()
    w = pos - cell
    i, j, k = cell.unbind(1)
    wx, wy, wz = w.unbind(1)
    f = []
    for d in D:
        # the reference's order: y with wy, then the z pair with wx, then the x pair with wz
        a = [[d[k + c, j, i + e] + wy * (d[k + c, j + 1, i + e] - d[k + c, j, i + e]) for e in (0, 1)] for c in (0, 1)]
        c0, c1 = (a[0][e] + wx * (a[1][e] - a[0][e]) for e in (0, 1))
        f.append(c0 + wz * (c1 - c0))
    t0 = 0.5 * (p.qi / p.mi) * DT
    t = t0 * p.B0
    sB = 2 * t / (1 + t * t)
    vm = [vel[:, a] - 0.5 / h * t0 * f[a] for a, h in enumerate((p.dx, p.dy, p.dz))]
    vt = vm[0] + vm[1] * t
    vy = vm[1] - vt * sB
    vel = torch.stack((vt + vy * t, vy, vm[2]), 1)
    L = torch.tensor(N, device=pos.device, dtype=torch.float64)
    pos = (pos + vel * DT) % L
    cell = pos.floor().long() % L.long()
    w = pos - pos.floor()
    mom = torch.zeros((4, p.Nx * p.Ny * p.Nz), device=pos.device, dtype=torch.float64)
    for c in range(8):
        b = (c & 1, c >> 1 & 1, c >> 2)
        wt = torch.ones_like(w[:, 0])
        node = [(cell[:, a] + b[a]) % N[a] for a in range(3)]
        for a in range(3):
            wt = wt * (w[:, a] if b[a] else 1 - w[:, a])
        at = (node[2] * p.Ny + node[1]) * p.Nx + node[0]
        for q in range(4):
            mom[q].index_add_(0, at, wt if q == 0 else wt * vel[:, q - 1])
    mom = mom.reshape((4, p.Nz, p.Ny, p.Nx))
    phi = _exact_solve(p, mom[0], _exact_rhs(p, *mom))
    return {"moments": mom.permute(1, 2, 3, 0).contiguous().cpu().numpy(), "phi": phi.cpu().numpy()}


def exact(case, seed):
    p = _params(case)
    if case["kind"] == "rhs":
        m = prepare(case, seed)["moments"]
        return _exact_rhs(p, *m.unbind(3))
    if case["kind"] == "solve":
        n = _density(case, seed)
        return _exact_solve(p, n, _exact_rhs(p, n, n, 0.5 * n, 0.25 * n)).cpu().numpy()
    if case["kind"] == "slots":
        return _exact_slots(case, seed)
    return None  # collisions and several steps: no values but the ions' own random streams give
