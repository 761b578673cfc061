"""Performance cases of the framework: what its users have it do, through its public entry points.

A pass is one leg of a run as the drop-in drivers make it: the state of the host program goes to the device
handle (`upload`), the main loop runs for a number of steps (`advance`), and the snapshot comes back (`download`).
The handle is kept from pass to pass, as a program that runs more than one leg keeps it, and so are the page-locked
host arrays.  Snapshots of single-precision runs are kept in single precision.  The drop-in functions, the batched
ensemble and the recorded run with its vector-Jacobian product are cases of their own.

    listed()            the cases
    draw(rng)           one more case of the same ranges
    prepare(case, seed) the inputs, the handle and the host arrays
    run(state)          one pass, and its outputs
    exact(case, seed)   the same outputs from plain torch in 64 bits (None where that would take too long)
    work(case)          bytes and operations that a pass cannot do without
"""
from __future__ import annotations

import math

import numpy as np
import torch
from torch.utils.checkpoint import checkpoint

from core_collapse_b200 import adjoint, batch, euler2d, mhd2d, mhd3d, ns2d

DEVICE = "cuda" if torch.cuda.is_available() else "cpu"
F64 = torch.float64


def _case(name, kind, nx, ny, precision, steps, **more):
    return {"name": name, "kind": kind, "nx": nx, "ny": ny, "precision": precision, "steps": steps, **more}


def listed():
    return [
        # the framework's benchmark: the larger grid of the precision ladder, single precision
        _case("mhd2d fft 4096 fp32", "mhd2d", 4096, 4096, "fp32", 60, poisson="fft", boundary="periodic", ic="orszag"),
        # the smaller grid of the precision ladder, double precision
        _case("mhd2d fft 1024 fp64", "mhd2d", 1024, 1024, "fp64", 60, poisson="fft", boundary="periodic", ic="orszag"),
        # an odd, ragged grid with outflow boundaries, no gravity, single precision
        _case("mhd2d ragged 1003x777 fp32", "mhd2d", 1003, 777, "fp32", 60, poisson="none", boundary="outflow",
              ic="collapse"),
        # the collapse workload: outflow, the reference's fixed 600 SOR sweeps a solve
        _case("mhd2d sor 256 fp64", "mhd2d", 256, 256, "fp64", 3, poisson="sor", boundary="outflow", ic="collapse",
              sweeps=600, omega=1.9),
        # the reference's three calls at its default parameters, host arrays in and out of each
        _case("mhd2d drop-in 192 fp64", "dropin", 192, 192, "fp64", 1, poisson="sor", boundary="periodic", ic="core",
              sweeps=600, omega=1.8),
        # the 3D benchmark: random-phase turbulence, ideal gas, single precision
        _case("mhd3d 256 fp32", "mhd3d", 256, 256, "fp32", 20, nz=256, boundary="periodic", ic="turbulence"),
        # a ragged 3D core collapse with the hybrid equation of state and outflow boundaries, double precision
        _case("mhd3d core 90x70x52 fp64", "mhd3d", 90, 70, "fp64", 20, nz=52, boundary="outflow", ic="core"),
        # the Euler solver at the reference's default grid and SOR tolerance: the smallest grid of a real run
        _case("euler2d sor 50 fp64", "euler2d", 50, 50, "fp64", 2, poisson="sor", boundary="periodic", tol=1e-10),
        # the Euler solver with enclosed-mass gravity at a production size, single precision
        _case("euler2d enclosed 2048 fp32", "euler2d", 2048, 2048, "fp32", 40, poisson="enclosed", boundary="periodic"),
        # the Navier-Stokes solver at the reference's default configuration: every launch counts
        _case("ns2d 128 fp64", "ns2d", 128, 128, "fp64", 150, gravity=True, viscosity=True),
        # a batched ensemble of collapse runs of uneven grid sizes
        _case("ensemble 128 fp32", "ensemble", 0, 0, "fp32", 150, instances=128),
        # forward run with checkpoints and its vector-Jacobian product
        _case("adjoint 512 fp64", "adjoint", 512, 512, "fp64", 30, poisson="direct", boundary="outflow", ic="collapse",
              every=10),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """One more case: another size, boundary, precision, solver or option of the same ranges."""
    kind = rng.choice(["mhd2d fft", "mhd2d none", "mhd2d none", "mhd2d sor", "dropin", "mhd3d", "mhd3d", "euler2d sor",
                       "euler2d radial", "ns2d", "ensemble", "adjoint"])
    precision = rng.choice(["fp32", "fp64"])
    boundary = rng.choice(["periodic", "outflow", "mixed"])
    steps = rng.randint(12, 40)
    if kind == "mhd2d fft":
        nx, ny = 1 << rng.randint(6, 11), 1 << rng.randint(6, 11)
        return _case("", "mhd2d", nx, ny, precision, steps, poisson="fft", boundary="periodic", ic="orszag",
                     compensated=precision == "fp32" and rng.random() < 0.25)
    if kind == "mhd2d none":
        nx, ny = _log(rng, 40, 1800), _log(rng, 40, 1800)
        return _case("", "mhd2d", nx, ny, precision, steps, poisson="none", boundary=boundary, ic="collapse")
    if kind == "mhd2d sor":
        nx, ny = 2 * _log(rng, 16, 200), 2 * _log(rng, 16, 200)
        return _case("", "mhd2d", nx, ny, precision, 2, poisson="sor", boundary=boundary, ic="collapse",
                     sweeps=rng.randint(100, 600), omega=round(rng.uniform(1.6, 1.9), 2))
    if kind == "dropin":
        n = 2 * _log(rng, 24, 128)
        return _case("", "dropin", n, n, "fp64", 1, poisson="sor", boundary="periodic", ic="core",
                     sweeps=rng.randint(200, 600), omega=1.8)
    if kind == "mhd3d":
        n = [_log(rng, 20, 120) for _ in range(3)]
        return _case("", "mhd3d", n[0], n[1], precision, rng.randint(6, 20), nz=n[2], boundary=boundary,
                     ic=rng.choice(["turbulence", "core"]))
    if kind == "euler2d sor":
        return _case("", "euler2d", 2 * _log(rng, 16, 64), 2 * _log(rng, 16, 64), precision, 1, poisson="sor",
                     boundary="periodic", tol=1e-8)
    if kind == "euler2d radial":
        nx, ny = _log(rng, 48, 1500), _log(rng, 48, 1500)
        return _case("", "euler2d", nx, ny, precision, steps, poisson=rng.choice(["enclosed", "shells"]),
                     boundary=boundary)
    if kind == "ns2d":
        gravity = rng.random() < 0.7
        nx, ny = (1 << rng.randint(6, 10), 1 << rng.randint(6, 10)) if gravity else (_log(rng, 48, 1200),
                                                                                       _log(rng, 48, 1200))
        return _case("", "ns2d", nx, ny, precision, steps, gravity=gravity, viscosity=rng.random() < 0.8)
    if kind == "ensemble":
        return _case("", "ensemble", 0, 0, precision, rng.randint(10, 30), instances=_log(rng, 6, 60))
    return _case("", "adjoint", _log(rng, 48, 400), _log(rng, 48, 400), precision, rng.randint(8, 20),
                 poisson="direct", boundary="outflow", ic="collapse", every=rng.choice([4, 5, 10]))


# ------------------------------------------------------------------ parameters

def _periodic(boundary, axis):
    return boundary == "periodic" or (boundary == "mixed" and axis == 0)


def _params2(c):
    """The collapse / Orszag-Tang physics of the benchmark workloads; the drop-in case keeps the reference's defaults."""
    if c["kind"] == "dropin":
        return mhd2d.Params(Nx=c["nx"], Ny=c["ny"], sor_iters=c["sweeps"], sor_omega=c["omega"])
    return mhd2d.Params(Nx=c["nx"], Ny=c["ny"], x0=-1.0, x1=1.0, y0=-1.0, y1=1.0,
                        periodic_x=_periodic(c["boundary"], 0), periodic_y=_periodic(c["boundary"], 1),
                        gamma=5.0 / 3.0, G=1.0, eta=1e-3, cfl=0.4, gravity_on=c["poisson"] != "none",
                        poisson="fft" if c["poisson"] == "none" else c["poisson"], sor_iters=c.get("sweeps", 600),
                        sor_omega=c.get("omega", 1.9), precision=c["precision"],
                        compensated=bool(c.get("compensated", False)), t_end=1e30)


def _params3(c):
    more = dict(Nx=c["nx"], Ny=c["ny"], Nz=c["nz"], eta=5e-4, cfl=0.4, precision=c["precision"], t_end=1e30,
                periodic_x=_periodic(c["boundary"], 0), periodic_y=_periodic(c["boundary"], 1),
                periodic_z=_periodic(c["boundary"], 2))
    return mhd3d.Params3.ideal_gas(**more) if c["ic"] == "turbulence" else mhd3d.Params3(**more)


def _params_eh(c):
    return euler2d.ParamsEH(Nx=c["nx"], Ny=c["ny"], poisson=c["poisson"], precision=c["precision"], t_end=1e30,
                            sor_tol=c.get("tol", 1e-10), periodic_x=_periodic(c["boundary"], 0),
                            periodic_y=_periodic(c["boundary"], 1))


def _params_ns(c):
    return ns2d.ParamsNS(Nx=c["nx"], Ny=c["ny"], precision=c["precision"], gravity_on=c["gravity"],
                         viscosity_on=c["viscosity"], t_end=1e30)


def _ensemble(c, seed):
    """Parameters and initial-condition settings of the instances: the benchmark's collapse ensemble."""
    rng = np.random.default_rng(1000 + seed)
    sides = np.random.default_rng(c["instances"]).choice((64, 96, 128, 192, 256), c["instances"])
    out = []
    for i, side in enumerate(int(n) for n in sides):
        one = dict(kind="mhd2d", nx=side, ny=side, precision=c["precision"], poisson="direct", boundary="outflow")
        p = _params2(one)
        p.eta = float(10.0 ** rng.uniform(-4.0, -2.0))
        out.append((p, dict(amp=float(rng.uniform(2.0, 20.0)), width=float(rng.uniform(0.05, 0.2)),
                            bx0=float(rng.uniform(0.0, 0.2)), seed=seed * 100003 + i)))
    return out


# ------------------------------------------------------------------ initial states (FP64, on DEVICE)

def _axis(a, b, n):
    h = (b - a) / n
    faces = a + h * torch.arange(n + 1, dtype=F64, device=DEVICE)
    return faces, faces[:-1] + 0.5 * h


def _noise(n, seed, normal=False):
    g = torch.Generator().manual_seed(seed)
    v = torch.randn(n, generator=g, dtype=F64) if normal else 2.0 * torch.rand(n, generator=g, dtype=F64) - 1.0
    return v.to(DEVICE)


def _conserve2(p, rho, u, v, P, bx, by):
    """[rho, mx, my, mz, E, Bz, Bx_f, By_f] of a planar flow."""
    bxc, byc = 0.5 * (bx[:, 1:] + bx[:, :-1]), 0.5 * (by[1:] + by[:-1])
    E = P / (p.gamma - 1.0) + 0.5 * rho * (u * u + v * v) + 0.5 * (bxc * bxc + byc * byc)
    z = torch.zeros_like(rho)
    return [rho, rho * u, rho * v, z, E, z.clone(), bx, by]


def _state2(p, ic, seed):
    """Orszag-Tang vortex with a dense core; Gaussian collapse core with 1% noise; the reference's rotating core."""
    r = np.random.default_rng(seed)
    xf, xc = _axis(p.x0, p.x1, p.Nx)
    yf, yc = _axis(p.y0, p.y1, p.Ny)
    rx, ry = xc[None, :] - 0.5 * (p.x0 + p.x1), yc[:, None] - 0.5 * (p.y0 + p.y1)
    r2 = rx * rx + ry * ry
    shape = (p.Ny, p.Nx)
    if ic == "orszag":
        amp, width, ax, ay = r.uniform(3.0, 5.0), r.uniform(0.08, 0.14), r.uniform(0, 1), r.uniform(0, 1)
        tau = 2.0 * math.pi
        A = (torch.cos(tau * (yf + ay))[:, None] / tau + torch.cos(2 * tau * (xf + ax))[None, :] / (2 * tau))
        A = A / math.sqrt(4.0 * math.pi)
        rho = 25.0 / (36.0 * math.pi) + amp * torch.exp(-r2 / (2.0 * width * width))
        u = (-torch.sin(tau * (yc + ay)))[:, None].expand(shape)
        v = torch.sin(tau * (xc + ax))[None, :].expand(shape)
        P = torch.full(shape, 5.0 / (12.0 * math.pi), dtype=F64, device=DEVICE)
    elif ic == "core":
        core, edge, vin, rot = r.uniform(0.10, 0.14), 0.02, r.uniform(1.0, 1.5), r.uniform(0.8, 1.2)
        d = torch.sqrt(r2) + 1e-14
        cut = 0.5 * (1.0 - torch.tanh((d - core) / edge))
        corner = torch.sqrt((xf[None, :] - 0.5 * (p.x0 + p.x1)) ** 2 + (yf[:, None] - 0.5 * (p.y0 + p.y1)) ** 2)
        cutA = 0.5 * (1.0 - torch.tanh((corner - core) / edge))
        A = 0.15 * (yf[:, None] - p.y0) + 0.05 * core * cutA * torch.sin(2 * math.pi * (xf[None, :] - p.x0) / (p.x1 - p.x0))
        rho = 1.0 + 19.0 * cut
        P = 0.15 * rho ** 1.05
        vr, vp = -vin * torch.clamp(d / core, max=1.0) * cut, rot * d * cut
        u, v = (vr * rx - vp * ry) / d, (vr * ry + vp * rx) / d
    else:
        s = ic if isinstance(ic, dict) else dict(amp=r.uniform(6.0, 12.0), width=r.uniform(0.08, 0.14), bx0=0.05, seed=seed)
        noise = _noise(p.Nx * p.Ny, s["seed"]).reshape(shape)
        rho = (1.0 + s["amp"] * torch.exp(-r2 / (2.0 * s["width"] ** 2))) * (1.0 + 0.01 * noise)
        A = s["bx0"] * (yf[:, None] - p.y0).expand(p.Ny + 1, p.Nx + 1)
        u = v = torch.zeros(shape, dtype=F64, device=DEVICE)
        P = 0.1 * rho ** (5.0 / 3.0)
    bx = (A[1:] - A[:-1]) / p.dy if ic in ("orszag", "core") else torch.full((p.Ny, p.Nx + 1), s["bx0"], dtype=F64,
                                                                              device=DEVICE)
    return _conserve2(p, rho, u, v, P, bx, -(A[:, 1:] - A[:, :-1]) / p.dx)


def _phases(shape, offset, modes, ph):
    """Re sum_n exp(i ph_n + 2 pi i n.(j + offset) / N) on a grid of `shape` = (nz, ny, nx)."""
    nz, ny, nx = shape
    out = torch.zeros(shape, dtype=torch.complex128, device=DEVICE)
    shift = 2.0 * np.pi * (modes[:, 0] * offset[0] / nx + modes[:, 1] * offset[1] / ny + modes[:, 2] * offset[2] / nz)
    idx = tuple(torch.from_numpy(np.ascontiguousarray(modes[:, 2 - a] % shape[a])).to(DEVICE) for a in range(3))
    out.index_put_(idx, torch.from_numpy(np.exp(1j * (ph + shift))).to(DEVICE), accumulate=True)
    return torch.fft.ifftn(out, norm="forward").real


def _state3(p, ic, seed):
    """Random-phase velocity and vector potential, |k| in [1, 4]; or the reference's infalling, rotating core."""
    shape = (p.Nz, p.Ny, p.Nx)
    r = np.random.default_rng(seed)
    if ic == "turbulence":
        g = np.stack(np.meshgrid(*[np.arange(-4, 5)] * 3, indexing="ij"), -1).reshape(-1, 3)
        k = np.sqrt((g ** 2).sum(1))
        modes = g[(k >= 1.0) & (k <= 4.0)]
        ph = r.uniform(0.0, 2.0 * np.pi, size=(6, len(modes)))
        v = [_phases(shape, (0.5, 0.5, 0.5), modes, ph[a]) for a in range(3)]
        vs = 0.5 / torch.sqrt(sum(a * a for a in v).mean())
        u, v, w = (a * vs for a in v)
        A = [_phases(shape, o, modes, ph[3 + a]) for a, o in enumerate(((.5, 0, 0), (0, .5, 0), (0, 0, .5)))]
        nxt = lambda a, d: torch.roll(a, -1, d)  # noqa: E731
        b = [(nxt(A[2], 1) - A[2]) / p.dy - (nxt(A[1], 0) - A[1]) / p.dz,
             (nxt(A[0], 0) - A[0]) / p.dz - (nxt(A[2], 2) - A[2]) / p.dx,
             (nxt(A[1], 2) - A[1]) / p.dx - (nxt(A[0], 1) - A[0]) / p.dy]
        cc = [0.5 * (b[a] + nxt(b[a], 2 - a)) for a in range(3)]
        scale = 0.3 / torch.sqrt(sum(a * a for a in cc).mean())
        faces = [torch.cat([b[a], b[a].narrow(2 - a, 0, 1)], 2 - a) * scale for a in range(3)]
        rho = torch.ones(shape, dtype=F64, device=DEVICE)
        P = torch.full(shape, 0.6, dtype=F64, device=DEVICE)
    else:
        core, edge, vin, rot = r.uniform(0.12, 0.18), 0.03, r.uniform(0.4, 0.7), r.uniform(0.8, 1.2)
        (xf, xc), (yf, yc), (_, zc) = _axis(p.x0, p.x1, p.Nx), _axis(p.y0, p.y1, p.Ny), _axis(p.z0, p.z1, p.Nz)
        mid = [0.5 * (p.x0 + p.x1), 0.5 * (p.y0 + p.y1), 0.5 * (p.z0 + p.z1)]
        rx, ry, rz = xc[None, None, :] - mid[0], yc[None, :, None] - mid[1], zc[:, None, None] - mid[2]
        d = torch.sqrt(rx * rx + ry * ry + rz * rz) + 1e-14
        cut = 0.5 * (1.0 - torch.tanh((d - core) / edge))
        rho = (1.0 + 99.0 * cut) * (1.0 + 0.01 * _noise(d.numel(), seed).reshape(shape))
        P = 0.3 * rho ** (5.0 / 3.0)
        vr = -vin * torch.clamp(d / core, max=1.0) * cut
        u, v, w = vr * rx / d - rot * ry * cut, vr * ry / d + rot * rx * cut, vr * rz / d
        ec = torch.sqrt((xf[None, :] - mid[0]) ** 2 + (yf[:, None] - mid[1]) ** 2)
        Az = 0.05 * 0.5 * (1.0 - torch.tanh((ec - core) / edge)) * torch.sin(2 * math.pi * xf)[None, :] * torch.sin(2 * math.pi * yf)[:, None]
        bx, by = (Az[1:] - Az[:-1]) / p.dy + 0.15, -(Az[:, 1:] - Az[:, :-1]) / p.dx
        faces = [bx[None].expand(p.Nz, -1, -1), by[None].expand(p.Nz, -1, -1),
                 torch.full((p.Nz + 1, p.Ny, p.Nx), 0.1, dtype=F64, device=DEVICE)]
    cc = [0.5 * (faces[a].narrow(2 - a, 1, shape[2 - a]) + faces[a].narrow(2 - a, 0, shape[2 - a])) for a in range(3)]
    E = _Eos3(p).energy([rho, u, v, w, P, *cc])
    return [rho, rho * u, rho * v, rho * w, E, *faces]


def _state_eh(p, seed):
    """The reference's random blob: 10% noise in density and pressure, a Gaussian bump, 5% velocity noise."""
    _, xc = _axis(p.x0, p.x1, p.Nx)
    _, yc = _axis(p.y0, p.y1, p.Ny)
    n = [_noise(p.Nx * p.Ny, seed * 4 + k).reshape(p.Ny, p.Nx) for k in range(4)]
    r2 = (xc[None, :] - 0.5) ** 2 + (yc[:, None] - 0.5) ** 2
    rho, P = 1.0 + 0.1 * n[0] + 0.5 * torch.exp(-r2 / (2.0 * 0.08 ** 2)), 1.0 + 0.1 * n[1]
    u, v = 0.05 * n[2], 0.05 * n[3]
    return [rho, rho * u, rho * v, P / (p.gamma - 1.0) + 0.5 * rho * (u * u + v * v)]


def _state_ns(p, seed):
    """The reference's collapse state: Gaussian overdensity, 1% density noise, Mach 0.05 velocity noise."""
    _, xc = _axis(p.x0, p.x1, p.Nx)
    _, yc = _axis(p.y0, p.y1, p.Ny)
    n = [_noise(p.Nx * p.Ny, seed * 3 + k, normal=True).reshape(p.Ny, p.Nx) for k in range(3)]
    r2 = (xc[None, :] - 0.5) ** 2 + (yc[:, None] - 0.5) ** 2
    rho = 1.0 + torch.exp(-0.5 * r2 / 0.01) + 0.01 * n[0]
    vamp = 0.05 * math.sqrt(p.gamma * 0.05)
    u, v = vamp * n[1], vamp * n[2]
    return [rho, rho * u, rho * v, 0.05 / (p.gamma - 1.0) + 0.5 * rho * (u * u + v * v)]


def _inputs(c, seed):
    """The parameters and the initial state of a single-grid case."""
    if c["kind"] in ("mhd2d", "dropin", "adjoint"):
        p = _params2(c)
        return p, _state2(p, c["ic"], seed)
    if c["kind"] == "mhd3d":
        p = _params3(c)
        return p, _state3(p, c["ic"], seed)
    if c["kind"] == "euler2d":
        p = _params_eh(c)
        return p, _state_eh(p, seed)
    p = _params_ns(c)
    return p, _state_ns(p, seed)


FIELDS = {"mhd2d": ("rho", "mx", "my", "mz", "E", "Bz", "Bx_f", "By_f"),
          "mhd3d": ("rho", "mx", "my", "mz", "E", "Bx_f", "By_f", "Bz_f"),
          "euler2d": ("rho", "mx", "my", "E"), "ns2d": ("rho", "mx", "my", "E")}
FIELDS["dropin"] = FIELDS["adjoint"] = FIELDS["ensemble"] = FIELDS["mhd2d"]


# ------------------------------------------------------------------ a pass

def _host(n, dtype=F64):
    return torch.empty(n, dtype=dtype, pin_memory=DEVICE == "cuda")


def _to_host(state):
    out = []
    for a in state:
        out.append(_host(a.numel()))
        out[-1].copy_(a.reshape(-1))
    return out


def _wrap(kind, tensors):
    """The framework's state containers over host tensors."""
    a = [t.numpy() for t in tensors]
    if kind == "mhd3d":
        return (mhd3d.State3(*a),)
    if kind == "euler2d":
        return (euler2d.StateEH(*a),)
    if kind == "ns2d":
        return (ns2d.StateNS(*a),)
    return mhd2d.Ucc(*a[:6]), mhd2d.Bfaces(*a[6:])


def prepare(case, seed):
    c, kind = case, case["kind"]
    st = {"case": c}
    if kind == "ensemble":
        made = _ensemble(c, seed)
        st["solver"] = batch.BatchSolver([p for p, _ in made])
        st["states"] = [_wrap(kind, _to_host(_state2(p, ic, 0))) for p, ic in made]
        st["out"], offset = {}, [0] * 8
        dtype = torch.float32 if c["precision"] == "fp32" else F64
        for k, f in enumerate(FIELDS[kind]):
            sizes = [(U.arrays() + [B.Bx_f, B.By_f])[k].size for U, B in st["states"]]
            st["out"][f] = torch.empty(sum(sizes), dtype=dtype)
        st["parts"] = [torch.split(st["out"][f], [(U.arrays() + [B.Bx_f, B.By_f])[k].size for U, B in st["states"]])
                       for k, f in enumerate(FIELDS[kind])]
        return st
    p, state = _inputs(c, seed)
    host = _to_host(state)
    st["p"], st["input"] = p, _wrap(kind, host)
    if kind == "dropin":
        return st
    if kind == "adjoint":
        st["solver"] = adjoint.AdjointSolver(p, c["every"], c["steps"])
        st["target"] = np.ascontiguousarray(np.roll(st["input"][0].rho, 3) * 1.02)
        return st
    st["solver"] = {"mhd2d": mhd2d.Mhd2dSolver, "mhd3d": mhd3d.Mhd3dSolver, "euler2d": euler2d.Euler2dSolver,
                    "ns2d": ns2d.Ns2dSolver}[kind](p)
    st["down"] = [_host(t.numel()) for t in host]
    st["output"] = _wrap(kind, st["down"])
    st["kept"] = [_host(t.numel(), torch.float32) for t in host] if c["precision"] == "fp32" else st["down"]
    return st


def run(state):
    c, kind = state["case"], state["case"]["kind"]
    if kind == "dropin":
        return _run_dropin(state)
    if kind == "ensemble":
        return _run_ensemble(state)
    if kind == "adjoint":
        return _run_adjoint(state)
    s = state["solver"]
    s.upload(*state["input"])
    t = s.advance(c["steps"], 0.0)
    s.download(*state["output"])
    if c["precision"] == "fp32":
        for kept, down in zip(state["kept"], state["down"]):
            kept.copy_(down)
    return {"t": t, **dict(zip(FIELDS[kind], state["kept"]))}


def _run_dropin(state):
    p = state["p"]
    U, B = (a.copy() for a in state["input"])
    g = mhd2d.compute_poisson_gravity_periodic(p, U.rho, p.dx, p.dy)
    dt = mhd2d.compute_dt(p, U, B, p.dx, p.dy)
    mhd2d.rk2_step(p, U, B, g, p.dx, p.dy, dt)
    return {"t": dt, "gx": g.gx, "gy": g.gy, **dict(zip(FIELDS["dropin"], U.arrays() + [B.Bx_f, B.By_f]))}


def _run_ensemble(state):
    s = state["solver"]
    for i, (U, B) in enumerate(state["states"]):
        s.upload(i, U, B)
    t = s.advance(state["case"]["steps"], np.zeros(s.n))
    for i in range(s.n):
        U, B = s.download(i)
        for part, a in zip(state["parts"], U.arrays() + [B.Bx_f, B.By_f]):
            part[i].copy_(torch.from_numpy(a))
    return {"t": t.astype(np.float32) if state["case"]["precision"] == "fp32" else t, **state["out"]}


def _run_adjoint(state):
    s, c = state["solver"], state["case"]
    s.upload(*state["input"])
    t = s.forward(c["steps"])
    U, B = s.download()
    loss, lamU, lamB = adjoint.density_loss_adjoint(state["p"], U.rho, state["target"])
    gU, gB, geta = s.vjp(lamU, lamB)
    out = {"t": t, "loss": loss, "grad_eta": geta}
    dtype = np.float32 if c["precision"] == "fp32" else np.float64
    for name, f, g in zip(FIELDS["adjoint"], U.arrays() + [B.Bx_f, B.By_f], gU.arrays() + [gB.Bx_f, gB.By_f]):
        out[name], out["grad_" + name] = f.astype(dtype, copy=False), g.astype(dtype, copy=False)
    return out


# ------------------------------------------------------------------ work

# words of state that one step has to read and write (two stages of a second-order scheme, gravity read in each)
# and operations of the scheme per cell and step, by solver
_WORDS = {"mhd2d": 42, "dropin": 42, "ensemble": 42, "mhd3d": 40, "euler2d": 22, "ns2d": 22, "adjoint": 42}
_FLOPS = {"mhd2d": 1600, "dropin": 1600, "ensemble": 1600, "mhd3d": 2400, "euler2d": 500, "ns2d": 450, "adjoint": 1600}


def _cells(c):
    if c["kind"] == "ensemble":
        return c["instances"] * 26726       # mean cells of an instance
    return c["nx"] * c["ny"] * c.get("nz", 1)


def work(case):
    c, n = case, _cells(case)
    word = 4 if c["precision"] == "fp32" else 8
    b, f = n * _WORDS[c["kind"]] * word, n * _FLOPS[c["kind"]]
    solves = 2
    if c.get("poisson") == "sor":           # one read of the density and one write of the potential; 12 operations a sweep
        sweeps = c.get("sweeps") or 20 * max(c["nx"], c["ny"])
        b, f = b + solves * 16 * n, f + solves * 12 * n * sweeps
    elif c.get("poisson") == "fft" or c.get("gravity"):
        b, f = b + solves * 2 * word * n, f + solves * 5 * n * math.log2(max(2, n))
    elif c.get("poisson") == "direct" or c["kind"] == "ensemble":
        b, f = b + solves * 2 * word * n, f + solves * 4 * n * math.sqrt(n / c.get("instances", 1))
    if c["kind"] == "adjoint":              # the forward run, its recomputation from the checkpoints, the reverse
        b, f = 4 * b, 4 * f
    return {"bytes": float(b * c["steps"]), "flops": float(f * c["steps"])}


# ------------------------------------------------------------------ the same in plain torch, 64 bits

def _cell(n, per, lo, hi):
    i = torch.arange(lo, hi, device=DEVICE)
    return i % n if per else i.clamp(0, n - 1)


def _face(n, per, lo, hi):
    i = torch.arange(lo, hi, device=DEVICE)
    return i % (n + 1) if per else i.clamp(0, n)


def _take(a, dim, idx):
    return a.index_select(dim, idx)


def _vmax(a, b):
    b = b if isinstance(b, torch.Tensor) else torch.full_like(a, b)
    return torch.where(a < b, b, a)


def _vmin(a, b):
    return torch.where(b < a, b, a)


def _over(ok, a, b):
    """a / b where ok, else 0, with no division by what is not ok."""
    return torch.where(ok, a / torch.where(ok, b, torch.ones_like(b)), torch.zeros_like(a))


def _root(a):
    """sqrt of max(a, 0) with a zero derivative at 0."""
    ok = a > 0.0
    return torch.where(ok, torch.sqrt(torch.where(ok, a, torch.ones_like(a))), torch.zeros_like(a))


def _minmod(a, b):
    return torch.where(a * b <= 0.0, torch.zeros_like(a), torch.where(a.abs() < b.abs(), a, b))


def _slope(wm, w, wp):
    dm, dp = w - wm, wp - w
    return _minmod(0.5 * (dm + dp), _minmod(2.0 * dm, 2.0 * dp))


class _Ideal:
    def __init__(self, p):
        self.p = p

    def energy(self, W):
        r, u, v, w, P, bx, by, bz = W
        return P / (self.p.gamma - 1.0) + 0.5 * r * (u * u + v * v + w * w) + 0.5 * (bx * bx + by * by + bz * bz)

    def a2(self, W):
        return self.p.gamma * W[4] / _vmax(W[0], self.p.floor_rho)

    def prim(self, rho, mx, my, mz, E, bx, by, bz):
        rho = _vmax(rho, self.p.floor_rho)
        u, v, w = mx / rho, my / rho, mz / rho
        P = (self.p.gamma - 1.0) * (E - 0.5 * rho * (u * u + v * v + w * w) - 0.5 * (bx * bx + by * by + bz * bz))
        return [rho, u, v, w, _vmax(P, self.p.floor_P), bx, by, bz]

    def floors(self, U, bx, by, bz):
        """U = [rho, mx, my, mz, E, ...] with the density and the pressure floored."""
        rho = _vmax(U[0], self.p.floor_rho)
        u, v, w = U[1] / rho, U[2] / rho, U[3] / rho
        km = 0.5 * rho * (u * u + v * v + w * w) + 0.5 * (bx * bx + by * by + bz * bz)
        g1 = self.p.gamma - 1.0
        E = torch.where(g1 * (U[4] - km) < self.p.floor_P, km + self.p.floor_P / g1, U[4])
        return [rho, U[1], U[2], U[3], E, *U[5:]]


class _Eos3:
    """Cold polytropes joined at nuclear density, stiffened above the bounce density, plus a thermal ideal gas."""

    def __init__(self, p):
        self.p = p

    def cold(self, rho):
        p = self.p
        rho = _vmax(rho, p.floor_rho)
        if p.K1 == 0.0 and p.Kbounce == 0.0:
            z = torch.zeros_like(rho)
            return z, z, z
        K2 = p.K1 * p.rho_nuc ** (p.gamma1 - p.gamma2)
        P1, e1 = p.K1 * rho ** p.gamma1, p.K1 * rho ** (p.gamma1 - 1.0) / (p.gamma1 - 1.0)
        en1 = p.K1 * p.rho_nuc ** (p.gamma1 - 1.0) / (p.gamma1 - 1.0)
        en2 = K2 * p.rho_nuc ** (p.gamma2 - 1.0) / (p.gamma2 - 1.0)
        P2, e2 = K2 * rho ** p.gamma2, en1 + (K2 * rho ** (p.gamma2 - 1.0) / (p.gamma2 - 1.0) - en2)
        gb = p.gamma_bounce
        pb = p.Kbounce * (rho ** gb - p.rho_bounce ** gb)
        eb = p.Kbounce * (rho ** (gb - 1.0) - p.rho_bounce ** (gb - 1.0)) / (gb - 1.0)
        g3 = (p.gamma2 * P2 + gb * pb) / _vmax(P2 + pb, p.floor_P)
        low, high = rho < p.rho_nuc, rho >= p.rho_bounce
        P = torch.where(low, P1, torch.where(high, P2 + pb, P2))
        e = torch.where(low, e1, torch.where(high, e2 + eb, e2))
        g = torch.where(low, torch.full_like(rho, p.gamma1), torch.where(high, g3, torch.full_like(rho, p.gamma2)))
        return P, e, g

    def internal(self, rho, P):
        Pc, ec, _ = self.cold(rho)
        return rho * (ec + _vmax(P - Pc, 0.0) / ((self.p.gamma_th - 1.0) * rho))

    def energy(self, W):
        r, u, v, w, P, bx, by, bz = W
        rho = _vmax(r, self.p.floor_rho)
        return 0.5 * rho * (u * u + v * v + w * w) + 0.5 * (bx * bx + by * by + bz * bz) + self.internal(rho, P)

    def a2(self, W):
        rho = _vmax(W[0], self.p.floor_rho)
        Pc, _, g = self.cold(rho)
        return _vmax((g * Pc + self.p.gamma_th * _vmax(W[4] - Pc, 0.0)) / rho, 0.0)

    def prim(self, rho, mx, my, mz, E, bx, by, bz):
        rho = _vmax(rho, self.p.floor_rho)
        u, v, w = mx / rho, my / rho, mz / rho
        e = _vmax(E - 0.5 * rho * (u * u + v * v + w * w) - 0.5 * (bx * bx + by * by + bz * bz), 0.0) / rho
        Pc, ec, _ = self.cold(rho)
        P = _vmax(Pc + (self.p.gamma_th - 1.0) * rho * _vmax(e - ec, 0.0), self.p.floor_P)
        return [rho, u, v, w, P, bx, by, bz]

    def floors(self, U, bx, by, bz):
        W = self.prim(*U[:5], bx, by, bz)
        return [W[0], U[1], U[2], U[3], self.energy(W), *U[5:]]


def _fast(eos, W, bn):
    rho = _vmax(W[0], 1e-300)
    a2, va, vn = eos.a2(W), (W[5] * W[5] + W[6] * W[6] + W[7] * W[7]) / rho, bn * bn / rho
    return _root(0.5 * (a2 + va + _root((a2 + va) * (a2 + va) - 4.0 * a2 * vn)))


def _hlld(eos, L, R, Bn):
    """HLLD flux [rho, m1, m2, m3, E, Bt1, Bt2] along the first component; star states jumped from the outer ones,
    HLL where the normal field vanishes."""
    side = []
    L, R = [*L[:5], Bn, *L[6:]], [*R[:5], Bn, *R[6:]]
    cf = [_fast(eos, W, Bn) for W in (L, R)]
    SL, SR = _vmin(L[1] - cf[0], R[1] - cf[1]), _vmax(L[1] + cf[0], R[1] + cf[1])
    for W, S in ((L, SL), (R, SR)):
        r, u, v, w, P, bx, by, bz = W
        pt, E, vB = P + 0.5 * (bx * bx + by * by + bz * bz), eos.energy(W), u * bx + v * by + w * bz
        F = [r * u, r * u * u + pt - bx * bx, r * u * v - bx * by, r * u * w - bx * bz, (E + pt) * u - bx * vB,
             u * by - v * bx, u * bz - w * bx]
        side.append(dict(U=[r, r * u, r * v, r * w, E, by, bz], F=F, pt=pt, vB=vB, S=S, s=S - u))
    l, r = side
    den = L[0] * l["s"] - R[0] * r["s"]
    SM = _over(den.abs() > 1e-14, r["pt"] - l["pt"] + L[0] * L[1] * l["s"] - R[0] * R[1] * r["s"], den)
    pts = l["pt"] + L[0] * l["s"] * (SM - L[1])
    for W, d in ((L, l), (R, r)):
        q = d["S"] - SM
        d["q"] = q
        inside = (SL < 0.0) & (SR > 0.0) & (q != 0.0)
        d["rs"] = _over(inside, W[0] * d["s"], q)
        dd = W[0] * d["s"] * q - Bn * Bn
        ok = (dd.abs() > 1e-14) & inside
        num = W[0] * d["s"] * d["s"] - Bn * Bn
        d["by"] = torch.where(ok, _over(ok, W[6] * num, dd), W[6])
        d["bz"] = torch.where(ok, _over(ok, W[7] * num, dd), W[7])
        d["v"] = W[2] - _over(ok, Bn * (d["by"] - W[6]), W[0] * d["s"] * q)
        d["w"] = W[3] - _over(ok, Bn * (d["bz"] - W[7]), W[0] * d["s"] * q)
        d["sq"] = _root(_vmax(d["rs"], 1e-300))
    sgn = torch.where(Bn >= 0.0, 1.0, -1.0).to(F64)
    a, b = l["sq"], r["sq"]
    d2, mhd = a + b, Bn.abs() >= 1e-12
    vss = _over(mhd, a * l["v"] + b * r["v"] + (r["by"] - l["by"]) * sgn, d2)
    wss = _over(mhd, a * l["w"] + b * r["w"] + (r["bz"] - l["bz"]) * sgn, d2)
    bys = _over(mhd, a * r["by"] + b * l["by"] + a * b * (r["v"] - l["v"]) * sgn, d2)
    bzs = _over(mhd, a * r["bz"] + b * l["bz"] + a * b * (r["w"] - l["w"]) * sgn, d2)
    left = SM > 0.0
    outer = torch.where(left, SM - _over(mhd, Bn.abs(), a) > 0.0, ~(SM + _over(mhd, Bn.abs(), b) > 0.0))
    pick = lambda x, y: torch.where(left, x, y)  # noqa: E731
    vs, ws = torch.where(outer, pick(l["v"], r["v"]), vss), torch.where(outer, pick(l["w"], r["w"]), wss)
    by, bz = torch.where(outer, pick(l["by"], r["by"]), bys), torch.where(outer, pick(l["bz"], r["bz"]), bzs)
    rs, S, q = pick(l["rs"], r["rs"]), pick(SL, SR), pick(l["q"], r["q"])
    u0, E0, pt0 = pick(L[1], R[1]), pick(l["U"][4], r["U"][4]), pick(l["pt"], r["pt"])
    Es = _over(q != 0.0, (S - u0) * E0 - (pt0 * u0 - Bn * pick(l["vB"], r["vB"])) + pts * SM
               - Bn * (SM * Bn + vs * by + ws * bz), q)
    Us = [rs, rs * SM, rs * vs, rs * ws, Es, by, bz]
    span = _over(SR - SL > 0.0, torch.ones_like(SL), SR - SL)
    out = []
    for k in range(7):
        FL, FR, UL, UR = l["F"][k], r["F"][k], l["U"][k], r["U"][k]
        star = pick(FL, FR) + S * (Us[k] - pick(UL, UR))
        hll = (SR * FL - SL * FR + SL * SR * (UR - UL)) * span
        out.append(torch.where(SL >= 0.0, FL, torch.where(SR <= 0.0, FR, torch.where(mhd, star, hll))))
    return out


def _faces(p, W, dim, n, per, skip, limit):
    """Left and right states of the n + 1 faces along `dim`: piecewise linear, the monotonised central limiter."""
    lo, hi = _cell(n, per, -1, n - 1), _cell(n, per, 1, n + 1)
    plus, minus = [], []
    for k, a in enumerate(W):
        s = 0.0 if k == skip else 0.5 * _slope(_take(a, dim, lo), a, _take(a, dim, hi))
        plus.append(a + s)
        minus.append(a - s)
    for k, f in limit:
        plus[k], minus[k] = _vmax(plus[k], f), _vmax(minus[k], f)
    li, ri = _cell(n, per, -1, n), _cell(n, per, 0, n + 1)
    return [_take(a, dim, li) for a in plus], [_take(a, dim, ri) for a in minus]


def _diff(a, dim):
    n = a.shape[dim] - 1
    return a.narrow(dim, 1, n) - a.narrow(dim, 0, n)


def _mean(a, dim):
    n = a.shape[dim] - 1
    return 0.5 * (a.narrow(dim, 1, n) + a.narrow(dim, 0, n))


def _grad_phi(phi, p, px, py):
    nx, ny = p.Nx, p.Ny
    gx = -(_take(phi, 1, _cell(nx, px, 1, nx + 1)) - _take(phi, 1, _cell(nx, px, -1, nx - 1))) / (2.0 * p.dx)
    gy = -(_take(phi, 0, _cell(ny, py, 1, ny + 1)) - _take(phi, 0, _cell(ny, py, -1, ny - 1))) / (2.0 * p.dy)
    return gx, gy


def _spectral(p, rho):
    """phi_k = -4 pi G rho_k / k^2 on a periodic box."""
    k = [2.0 * math.pi * torch.fft.fftfreq(n, 1.0 / n, dtype=F64, device=DEVICE) / w
         for n, w in ((p.Ny, p.y1 - p.y0), (p.Nx, p.x1 - p.x0))]
    k2 = k[0][:, None] ** 2 + k[1][None, :] ** 2
    f = torch.where(k2 > 0.0, -4.0 * math.pi * p.G / torch.where(k2 > 0.0, k2, 1.0), 0.0)
    return torch.fft.ifft2(torch.fft.fft2(rho - rho.mean()) * f).real


def _direct(p, rho):
    """The zero-mean solution of the 5-point problem, by the eigenvectors of its second differences."""
    mats = []
    for n, per, h in ((p.Nx, p.periodic_x, p.dx), (p.Ny, p.periodic_y, p.dy)):
        i = torch.arange(n, dtype=F64, device=DEVICE)
        if per:
            a = 2.0 * math.pi * i[:, None] * i[None, :] / n
            Q, s = (torch.cos(a) + torch.sin(a)) / math.sqrt(n), torch.sin(math.pi * i / n)
        else:
            Q = torch.cos(math.pi * i[:, None] * (2 * i[None, :] + 1) / (2 * n)) * math.sqrt(2.0 / n)
            Q[0] /= math.sqrt(2.0)
            s = torch.sin(math.pi * i / (2 * n))
        mats.append((Q, -4.0 * s * s / (h * h)))
    (Qx, lx), (Qy, ly) = mats
    lam = ly[:, None] + lx[None, :]
    f = torch.where(lam < 0.0, 1.0 / torch.where(lam < 0.0, lam, 1.0), 0.0)
    hat = Qy @ (4.0 * math.pi * p.G * (rho - rho.mean())) @ Qx.T
    return Qy.T @ (hat * f) @ Qx


def _sor(p, rho, px, py, sweeps, omega, tol):
    """Red-black successive over-relaxation from zero, the mean removed after each sweep."""
    nx, ny = p.Nx, p.Ny
    ix, iy = 1.0 / p.dx ** 2, 1.0 / p.dy ** 2
    rhs = 4.0 * math.pi * p.G * (rho - rho.mean())
    red = ((torch.arange(ny, device=DEVICE)[:, None] + torch.arange(nx, device=DEVICE)[None, :]) % 2) == 0
    e, w = _cell(nx, px, 1, nx + 1), _cell(nx, px, -1, nx - 1)
    u, d = _cell(ny, py, 1, ny + 1), _cell(ny, py, -1, ny - 1)
    phi = torch.zeros_like(rho)
    for _ in range(sweeps):
        for colour in (red, ~red):
            pn = ((_take(phi, 1, e) + _take(phi, 1, w)) * ix + (_take(phi, 0, u) + _take(phi, 0, d)) * iy - rhs)
            phi = torch.where(colour, phi + omega * (pn / (2.0 * (ix + iy)) - phi), phi)
        phi = phi - phi.mean()
        if tol > 0.0:
            lap = (_take(phi, 1, e) - 2.0 * phi + _take(phi, 1, w)) * ix + (_take(phi, 0, u) - 2.0 * phi + _take(phi, 0, d)) * iy
            if float((lap - rhs).abs().max()) < tol:
                break
    return phi


class _Exact2:
    """The 2D resistive MHD step: U = [rho, mx, my, mz, E, Bz], bx on x faces, by on y faces."""

    def __init__(self, p, gravity):
        self.p, self.eos, self.gravity = p, _Ideal(p), gravity

    def potential(self, rho):
        p = self.p
        if self.gravity == "fft":
            return _spectral(p, rho)
        if self.gravity == "direct":
            return _direct(p, rho)
        return _sor(p, rho, p.periodic_x, p.periodic_y, p.sor_iters, p.sor_omega, p.sor_tol)

    def accel(self, rho):
        return None if self.gravity == "none" else _grad_phi(self.potential(rho), self.p, self.p.periodic_x, self.p.periodic_y)

    def prim(self, s):
        return self.eos.prim(*s[:5], _mean(s[6], 1), _mean(s[7], 0), s[5])

    def dt(self, s):
        p = self.p
        W = self.prim(s)
        m = max(1e-14, float((W[1].abs() + _fast(self.eos, W, W[5])).max()), float((W[2].abs() + _fast(self.eos, W, W[6])).max()))
        h = min(p.dx, p.dy)
        return min(p.cfl * h / m, 0.25 * h * h / float(p.eta) if float(p.eta) > 0.0 else 1e100)

    def stage(self, s, g, dt, eta):
        p, eos = self.p, self.eos
        nx, ny, px, py = p.Nx, p.Ny, p.periodic_x, p.periodic_y
        bx, by = s[6], s[7]
        W = self.prim(s)
        limit = ((0, p.floor_rho), (4, p.floor_P))
        L, R = _faces(p, W, 1, nx, px, 5, limit)
        F = _hlld(eos, L, R, bx)
        L, R = _faces(p, W, 0, ny, py, 6, limit)
        swap = lambda a: [a[0], a[2], a[1], a[3], a[4], a[6], a[5], a[7]]  # noqa: E731
        G = _hlld(eos, swap(L), swap(R), by)
        G = [G[0], G[2], G[1], *G[3:]]
        U = [s[k] + dt * (-_diff(F[m], 1) / p.dx - _diff(G[m], 0) / p.dy) for k, m in enumerate((0, 1, 2, 3, 4, 6))]
        bxc, byc = W[5], W[6]
        U = eos.floors(U, bxc, byc, U[5])
        # edge EMF, then the faces
        cx0, cx1, cy0, cy1 = _cell(nx, px, -1, nx), _cell(nx, px, 0, nx + 1), _cell(ny, py, -1, ny), _cell(ny, py, 0, ny + 1)
        ez = 0.25 * (-_take(F[5], 0, cy0) - _take(F[5], 0, cy1) + _take(G[5], 1, cx0) + _take(G[5], 1, cx1))
        if float(p.eta) > 0.0:
            ez = ez + eta * ((_take(by, 1, cx1) - _take(by, 1, cx0)) / p.dx - (_take(bx, 0, cy1) - _take(bx, 0, cy0)) / p.dy)
        bx, by = bx - dt * _diff(ez, 0) / p.dy, by + dt * _diff(ez, 1) / p.dx
        bxc, byc = _mean(bx, 1), _mean(by, 0)
        if g is not None:
            rho, u, v = U[0], U[1] / U[0], U[2] / U[0]
            U = [rho, U[1] + dt * rho * g[0], U[2] + dt * rho * g[1], U[3], U[4] + dt * rho * (u * g[0] + v * g[1]), U[5]]
            U = eos.floors(U, bxc, byc, U[5])
        if float(p.eta) > 0.0:              # Joule heating and the diffusion of Bz
            bz = U[5]
            e, w = _take(bz, 1, _cell(nx, px, 1, nx + 1)), _take(bz, 1, _cell(nx, px, -1, nx - 1))
            n, d = _take(bz, 0, _cell(ny, py, 1, ny + 1)), _take(bz, 0, _cell(ny, py, -1, ny - 1))
            byp, bxp = _take(by[:-1], 1, _cell(nx, px, 1, nx + 1)), _take(bx[:, :-1], 0, _cell(ny, py, 1, ny + 1))
            jz = (byp - by[:-1]) / p.dx - (bxp - bx[:, :-1]) / p.dy
            j2 = ((n - d) / (2.0 * p.dy)) ** 2 + ((e - w) / (2.0 * p.dx)) ** 2 + jz * jz
            E = U[4] + dt * eta * j2
            bz = bz + dt * eta * ((e - 2.0 * bz + w) / p.dx ** 2 + (n - 2.0 * bz + d) / p.dy ** 2)
            U = eos.floors([*U[:4], E, bz], bxc, byc, bz)
        return [*U, bx, by]

    def step(self, dt, eta, g, *s):
        s1 = self.stage(s, self.accel(s[0]) if g is None else g, dt, eta)
        s2 = self.stage(s1, self.accel(s1[0]), dt, eta)
        s = [0.5 * (a + b) for a, b in zip(s, s2)]
        return [*self.eos.floors(s[:6], _mean(s[6], 1), _mean(s[7], 0), s[5]), s[6], s[7]]


class _Exact3:
    """The 3D resistive MHD step: U = [rho, mx, my, mz, E], the three face fields; axes (z, y, x)."""

    def __init__(self, p):
        self.p, self.eos = p, _Eos3(p)
        self.n, self.h = (p.Nx, p.Ny, p.Nz), (p.dx, p.dy, p.dz)
        self.per = (p.periodic_x, p.periodic_y, p.periodic_z)

    def centred(self, B):
        return [_mean(B[a], 2 - a) for a in range(3)]

    def padded(self, B):
        """Cell-centred B on -1 .. n along every axis, from the faces' own wrap."""
        out = []
        for a in range(3):
            f = B[a]
            for d in range(3):
                n, per = self.n[d], self.per[d]
                if d == a:
                    f = 0.5 * (_take(f, 2 - d, _face(n, per, -1, n + 1)) + _take(f, 2 - d, _face(n, per, 0, n + 2)))
                else:
                    f = _take(f, 2 - d, _cell(n, per, -1, n + 1))
            out.append(f)
        return out

    def prim(self, s):
        return self.eos.prim(*s[:5], *self.centred(s[5:]))

    def dt(self, s):
        W = self.prim(s)
        m = max([1e-14] + [float((W[1 + a].abs() + _fast(self.eos, W, W[5 + a])).max()) for a in range(3)])
        h = min(self.h)
        return min(self.p.cfl * h / m, 0.25 * h * h / self.p.eta if self.p.eta > 0.0 else 1e100)

    def stage(self, s, dt):
        p, eos, n, h, per = self.p, self.eos, self.n, self.h, self.per
        B, W = s[5:], self.prim(s)
        rate, emf = [0.0] * 5, {}
        for a in range(3):                  # a: the normal; b, c: the other two, in cyclic order (y: z before x swapped)
            b, c = ((1, 2), (0, 2), (0, 1))[a]
            order = [0, 1 + a, 1 + b, 1 + c, 4, 5 + a, 5 + b, 5 + c]
            L, R = _faces(p, W, 2 - a, n[a], per[a], 5 + a, ((0, p.floor_rho), (4, p.floor_P)))
            F = _hlld(eos, [L[k] for k in order], [R[k] for k in order], B[a])
            for k, m in ((0, 0), (1 + a, 1), (1 + b, 2), (1 + c, 3), (4, 4)):
                rate[k] = rate[k] - _diff(F[m], 2 - a) / h[a]
            # F[5] is the flux of B_b, F[6] of B_c; E_k = -eps_kab F(B_b)
            eps = {(0, 1): 1.0, (1, 2): 1.0, (2, 0): 1.0, (1, 0): -1.0, (2, 1): -1.0, (0, 2): -1.0}
            emf[(a, c)] = -eps[(a, b)] * F[5]
            emf[(a, b)] = -eps[(a, c)] * F[6]
        U = eos.floors([s[k] + dt * rate[k] for k in range(5)], *W[5:])
        pad = self.padded(B)
        E = []
        for k in range(3):                  # edge EMF along axis k, from the faces normal to the other two
            a, b = ((1, 2), (2, 0), (0, 1))[k]
            fa, fb = emf[(a, k)], emf[(b, k)]
            lo = lambda f, d: _take(f, 2 - d, _cell(n[d], per[d], -1, n[d]))  # noqa: E731
            hi = lambda f, d: _take(f, 2 - d, _cell(n[d], per[d], 0, n[d] + 1))  # noqa: E731
            e = 0.25 * (lo(fa, b) + hi(fa, b) + lo(fb, a) + hi(fb, a))
            if p.eta > 0.0:
                def cut(f, d):              # on edges: cells 0 .. n - 1 along k, -1 .. n along d differenced, 0 .. n along the third
                    o = a if d == b else b
                    f = f.narrow(2 - k, 1, n[k]).narrow(2 - o, 1, n[o] + 1)
                    return _diff(f, 2 - d) / h[d]
                e = e + p.eta * (cut(pad[b], a) - cut(pad[a], b))
            E.append(e)
        new = []
        for a in range(3):                  # dB_a/dt = -(dE_c/db - dE_b/dc)
            b, c = (a + 1) % 3, (a + 2) % 3
            new.append(B[a] - dt / h[b] * _diff(E[c], 2 - b) + dt / h[c] * _diff(E[b], 2 - c))
        if p.eta > 0.0:
            pad = self.padded(new)

            def central(f, d):
                for o in range(3):
                    if o != d:
                        f = f.narrow(2 - o, 1, n[o])
                return (f.narrow(2 - d, 2, n[d]) - f.narrow(2 - d, 0, n[d])) / (2.0 * h[d])
            j = [central(pad[2], 1) - central(pad[1], 2), central(pad[0], 2) - central(pad[2], 0),
                 central(pad[1], 0) - central(pad[0], 1)]
            U[4] = U[4] + dt * p.eta * (j[0] ** 2 + j[1] ** 2 + j[2] ** 2)
        return [*eos.floors(U, *self.centred(new)), *new]

    def step(self, dt, s):
        s2 = self.stage(self.stage(s, dt), dt)
        s = [0.5 * (a + b) for a, b in zip(s, s2)]
        return [*self.eos.floors(s[:5], *self.centred(s[5:])), *s[5:]]


def _hllc(p, L, R, tiny, with_star_pressure):
    """HLLC flux [rho, normal, tangential, E]; states [rho, normal, tangential, P]."""
    g1 = p.gamma - 1.0
    a = [torch.sqrt(p.gamma * W[3] / _vmax(W[0], p.floor_rho)) for W in (L, R)]
    SL, SR = _vmin(L[1] - a[0], R[1] - a[1]), _vmax(L[1] + a[0], R[1] + a[1])
    den = L[0] * (SL - L[1]) - R[0] * (SR - R[1])
    num = R[3] - L[3] + L[0] * L[1] * (SL - L[1]) - R[0] * R[1] * (SR - R[1])
    SM = _over(den.abs() > tiny, num, den)
    sides = []
    for W, S in ((L, SL), (R, SR)):
        r, n, t, P = W
        E = P / g1 + 0.5 * r * (n * n + t * t)
        F, U = [r * n, r * n * n + P, r * n * t, (E + P) * n], [r, r * n, r * t, E]
        q = S - SM
        rs = _over(q != 0.0, r * (S - n), q)
        ps = P + r * (S - n) * (SM - n) if with_star_pressure else P
        Us = [rs, rs * SM, rs * t, _over(q != 0.0, (S - n) * E - P * n + ps * SM, q)]
        sides.append((F, [F[k] + S * (Us[k] - U[k]) for k in range(4)]))
    return [torch.where(SL >= 0.0, sides[0][0][k], torch.where(SR <= 0.0, sides[1][0][k],
            torch.where(SM > 0.0, sides[0][1][k], sides[1][1][k]))) for k in range(4)]


class _ExactEh:
    """The Euler step with gravity in the right-hand side."""

    def __init__(self, p):
        self.p = p
        _, xc = _axis(p.x0, p.x1, p.Nx)
        _, yc = _axis(p.y0, p.y1, p.Ny)
        centre = (p.xc, p.yc) if p.poisson == "shells" else (0.5 * (p.x0 + p.x1), 0.5 * (p.y0 + p.y1))
        self.rx, self.ry = (xc[None, :] - centre[0]).expand(p.Ny, -1), (yc[:, None] - centre[1]).expand(-1, p.Nx)
        self.r = torch.sqrt(self.rx ** 2 + self.ry ** 2)

    def accel(self, rho):
        p = self.p
        rho = _vmax(rho, p.floor_rho)
        if p.poisson == "sor":
            return _grad_phi(_sor(p, rho, True, True, p.sor_max_iter, p.sor_omega, p.sor_tol), p, True, True)
        m = (rho * p.dx * p.dy).reshape(-1)
        if p.poisson == "shells":
            nr = max(8, p.Nr_bins)
            dr = max(float(self.r.max()), 1e-12) / nr
            shell = torch.floor(self.r / dr).long().clamp(0, nr - 1).reshape(-1)
            total = torch.cumsum(torch.zeros(nr, dtype=F64, device=DEVICE).index_add_(0, shell, m), 0)
            f = -p.G * total[shell].reshape(rho.shape) / (self.r ** 2 + p.softening ** 2) ** 1.5
            return f * self.rx, f * self.ry
        r, order = torch.sort(self.r.reshape(-1))
        total = torch.cumsum(m[order], 0)
        end = torch.searchsorted(r, r + 1e-12, right=True) - 1
        enclosed = torch.empty_like(m)
        enclosed[order] = total[end]
        r2 = self.r ** 2 + p.softening ** 2
        f = -p.G * enclosed.reshape(rho.shape) / r2 / torch.sqrt(r2)
        return f * self.rx, f * self.ry

    def prim(self, U):
        p = self.p
        r = _vmax(U[0], p.floor_rho)
        u, v = U[1] / r, U[2] / r
        return [r, u, v, _vmax((p.gamma - 1.0) * (U[3] - 0.5 * r * (u * u + v * v)), p.floor_P)]

    def floors(self, U):
        W, g1 = self.prim(U), self.p.gamma - 1.0
        kin = 0.5 * W[0] * (W[1] ** 2 + W[2] ** 2)
        return [W[0], U[1], U[2], torch.where(g1 * (U[3] - kin) < self.p.floor_P, kin + self.p.floor_P / g1, U[3])]

    def dt(self, U):
        p, W = self.p, self.prim(U)
        a = torch.sqrt(p.gamma * W[3] / W[0])
        return p.cfl * min(p.dx, p.dy) / max(float((W[1].abs() + a).max()), float((W[2].abs() + a).max()))

    def rhs(self, U):
        p, W = self.p, self.prim(self.floors(U))
        limit = ((0, p.floor_rho), (3, p.floor_P))
        F = _hllc(p, *_faces(p, W, 1, p.Nx, p.periodic_x, -1, limit), 1e-14, False)
        L, R = _faces(p, W, 0, p.Ny, p.periodic_y, -1, limit)
        G = _hllc(p, [L[0], L[2], L[1], L[3]], [R[0], R[2], R[1], R[3]], 1e-14, False)
        G = [G[0], G[2], G[1], G[3]]
        d = [-_diff(F[k], 1) / p.dx - _diff(G[k], 0) / p.dy for k in range(4)]
        g, rho = self.accel(U[0]), _vmax(U[0], p.floor_rho)
        return [d[0], d[1] + rho * g[0], d[2] + rho * g[1], d[3] + U[1] * g[0] + U[2] * g[1]]

    def step(self, dt, U):
        V = self.floors([a + dt * k for a, k in zip(U, self.rhs(U))])
        return self.floors([0.5 * a + 0.5 * (b + dt * k) for a, b, k in zip(U, V, self.rhs(V))])


class _BoxNs:
    """The parameters with their cell sizes."""

    def __init__(self, p):
        self.__dict__.update(vars(p), dx=(p.x1 - p.x0) / p.Nx, dy=(p.y1 - p.y0) / p.Ny)


class _ExactNs:
    """The Navier-Stokes step: first-order HLLC, viscous stress from face-averaged gradients, spectral gravity."""

    def __init__(self, p):
        self.p = _BoxNs(p)

    prim = _ExactEh.prim

    def dt(self, U):
        p, W = self.p, self.prim(U)
        a = torch.sqrt(p.gamma * W[3] / W[0])
        h = min(p.dx, p.dy)
        dt = p.cfl * h / max(float((W[1].abs() + a).max()), float((W[2].abs() + a).max()))
        return min(dt, p.cfl_visc * h * h * float(W[0].min()) / p.mu) if p.viscosity_on and p.mu > 0.0 else dt

    def rhs(self, U):
        p, W = self.p, self.prim(U)
        nxt = lambda a, d: torch.roll(a, -1, d)  # noqa: E731
        prv = lambda a, d: torch.roll(a, 1, d)  # noqa: E731
        flux = []
        grad = {(c, d): (nxt(W[c], d) - prv(W[c], d)) / (2.0 * (p.dx if d == 1 else p.dy)) for c in (1, 2) for d in (0, 1)}
        for d in (1, 0):
            o = [0, 1, 2, 3] if d == 1 else [0, 2, 1, 3]
            F = _hllc(p, [W[k] for k in o], [nxt(W[k], d) for k in o], 0.0, True)
            F = [F[k] for k in o]
            if p.viscosity_on and p.mu > 0.0:
                m = {k: 0.5 * (a + nxt(a, d)) for k, a in grad.items()}
                div = m[(1, 1)] + m[(2, 0)]
                xy = p.mu * (m[(1, 0)] + m[(2, 1)])
                nn = p.mu * (2.0 * (m[(1, 1)] if d == 1 else m[(2, 0)]) - 2.0 / 3.0 * div)
                tx, ty = (nn, xy) if d == 1 else (xy, nn)
                u, v = 0.5 * (W[1] + nxt(W[1], d)), 0.5 * (W[2] + nxt(W[2], d))
                F = [F[0], F[1] - tx, F[2] - ty, F[3] - (u * tx + v * ty)]
            flux.append(F)
        r = [-(flux[0][k] - prv(flux[0][k], 1)) / p.dx - (flux[1][k] - prv(flux[1][k], 0)) / p.dy for k in range(4)]
        if p.gravity_on:
            gx, gy = _grad_phi(_spectral(p, W[0]), p, True, True)
            r = [r[0], r[1] + W[0] * gx, r[2] + W[0] * gy, r[3] + W[0] * (W[1] * gx + W[2] * gy)]
        return r

    def step(self, dt, U):
        k1 = self.rhs(U)
        V = [a + dt * k for a, k in zip(U, k1)]
        V[0] = _vmax(V[0], self.p.floor_rho)
        out = [a + 0.5 * dt * (k + m) for a, k, m in zip(U, k1, self.rhs(V))]
        return [_vmax(out[0], self.p.floor_rho), *out[1:]]


def _seconds(c):
    """About how long exact() takes on a GPU: launches of small operations, or their memory traffic."""
    n = _cells(c) / c.get("instances", 1)
    ops = {"mhd2d": 1500, "dropin": 1500, "ensemble": 1500, "mhd3d": 2600, "euler2d": 900, "ns2d": 700, "adjoint": 9000}
    ops = ops[c["kind"]] * (2.5 if c["kind"] == "mhd3d" and c["ic"] == "core" else 1.0)
    if c.get("poisson") == "sor":
        ops += 2 * (c.get("sweeps") or 60 * max(c["nx"], c["ny"])) * (40 if c["kind"] == "euler2d" else 22)
    return c["steps"] * c.get("instances", 1) * ops * max(7e-6, n * 24 / 4e12)


def _flat(names, state):
    return {k: a.reshape(-1) for k, a in zip(names, state)}


def exact(case, seed):
    c = case
    if _seconds(c) > 20.0 or DEVICE == "cpu" and _cells(c) > 70000:
        return None
    names = FIELDS[c["kind"]]
    if c["kind"] == "ensemble":
        ends, times = [], []
        for p, ic in _ensemble(c, seed):
            s, t = _march2(_Exact2(p, "direct"), _state2(p, ic, 0), c["steps"])
            ends.append([a.reshape(-1) for a in s])
            times.append(t)
        return {"t": torch.tensor(times, dtype=F64), **{k: torch.cat([e[j] for e in ends]) for j, k in enumerate(names)}}
    p, s = _inputs(c, seed)
    if c["kind"] == "dropin":
        solver = _Exact2(p, "sor")
        g, dt = solver.accel(s[0]), solver.dt(s)
        return {"t": dt, "gx": g[0].reshape(-1), "gy": g[1].reshape(-1), **_flat(names, solver.step(dt, p.eta, g, *s))}
    if c["kind"] == "mhd2d":
        s, t = _march2(_Exact2(p, c["poisson"]), s, c["steps"])
        return {"t": t, **_flat(names, s)}
    if c["kind"] == "adjoint":
        return _exact_adjoint(c, p, s)
    solver = {"mhd3d": _Exact3, "euler2d": _ExactEh, "ns2d": _ExactNs}[c["kind"]](p)
    t = 0.0
    for _ in range(c["steps"]):
        dt = solver.dt(s)
        s = solver.step(dt, s)
        t += dt
    return {"t": t, **_flat(names, s)}


def _march2(solver, s, steps):
    t = 0.0
    for _ in range(steps):
        dt = solver.dt(s)
        s = solver.step(dt, solver.p.eta, None, *s)
        t += dt
    return s, t


def _exact_adjoint(c, p, s):
    """The gradient by reverse mode through the plain step, the recorded dt held fixed."""
    solver = _Exact2(p, c["poisson"])
    target = torch.roll(s[0].reshape(-1), 3) * 1.02
    first = [a.detach().clone().contiguous().requires_grad_(True) for a in s]
    eta = torch.tensor(p.eta, dtype=F64, device=DEVICE, requires_grad=True)
    state, t = first, 0.0
    for _ in range(c["steps"]):
        with torch.no_grad():
            dt = solver.dt(state)
        state = checkpoint(solver.step, dt, eta, None, *state, use_reentrant=False)
        t += dt
    loss = 0.5 * ((state[0].reshape(-1) - target) ** 2).sum()
    grads = torch.autograd.grad(loss, [*first, eta], allow_unused=True)
    out = {"t": t, "loss": float(loss.detach()), "grad_eta": float(grads[-1])}
    for k, a, g in zip(FIELDS["adjoint"], state, grads):
        out[k], out["grad_" + k] = a.detach().reshape(-1), g.reshape(-1)
    return out
