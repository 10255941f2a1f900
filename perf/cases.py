"""The workloads this engine is timed on, through its Python API.

A case is one call of a user's loop: advance the state (`step`, a batch step, a
Born `Compute`) and read the wave function back, as a program that watches an
evolution does.  The handle (an Evolver, an Instance, a Batch, a scattering
solver) and the page-locked buffers a program reads into are made once, in
`prepare`.  complex64 ("mixed") states are kept in single precision after the
read.  Inputs are Gaussian packets and seeded potentials of the shapes that the
benchmark configurations and the tests use.
"""
import math
import random

import numpy as np
import torch

import qusim_gb300 as q

DEV = "cuda" if torch.cuda.is_available() else "cpu"


def listed():
    return [
        # the smallest call: one step of the smallest resident line, as an
        # interactive program steps and plots it (Evolver1D.step, GetPsi)
        dict(name="line_64_c128_o2", kind="line", n=64, precision="fp64", order=2, steps=1, wall=False, fnes=False,
             imag=False),
        # the plain 1D configuration: N = 4096, O2, read every 200 steps
        dict(name="line_4096_c64_o2", kind="line", n=4096, precision="mixed", order=2, steps=200, wall=False,
             fnes=False, imag=False),
        # a box of any length (not a power of two) between infinite walls
        dict(name="wall_1000_c128_o4", kind="line", n=1000, precision="fp64", order=4, steps=20, wall=True,
             fnes=False, imag=False),
        # a long line in double precision, renormalised after each call (four-step passes)
        dict(name="line_131072_c128_o2", kind="line", n=131072, precision="fp64", order=2, steps=20, wall=False,
             fnes=True, imag=False),
        # a small 2D grid, double precision: launches and latency
        dict(name="grid_256x128_c128_o4", kind="grid", nx=256, ny=128, precision="fp64", order=4, steps=20,
             fnes=False, imag=False),
        # the 1024^2 configuration: random Gaussian bumps, O4, both precisions
        dict(name="grid_1024_c64_o4", kind="grid", nx=1024, ny=1024, precision="mixed", order=4, steps=50,
             fnes=False, imag=False),
        dict(name="grid_1024_c128_o4", kind="grid", nx=1024, ny=1024, precision="fp64", order=4, steps=10,
             fnes=False, imag=False),
        # sides that are not powers of two (Bluestein row and column passes)
        dict(name="grid_450x700_c128_o2", kind="grid", nx=450, ny=700, precision="fp64", order=2, steps=10,
             fnes=False, imag=False),
        # the largest: the 4096^2 double-slit configuration, complex64
        dict(name="grid_4096_c64_o4", kind="grid", nx=4096, ny=4096, precision="mixed", order=4, steps=40,
             fnes=False, imag=False),
        # the 256^3 configuration
        dict(name="volume_256_c64_o4", kind="volume", nx=256, ny=256, nz=256, precision="mixed", order=4, steps=20),
        # the batched 1D configuration: independent lines of 2^10 .. 2^16 sites
        dict(name="batch_256_c64_o2", kind="batch", count=256, emin=10, emax=16, precision="mixed", order=2,
             steps=400),
        # 2D scattering by the preconditioned Born series
        dict(name="born_1024_c64", kind="born", nx=1024, ny=1024, precision="mixed", updates=200),
    ]


def _loguniform(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["line", "line", "line", "grid", "grid", "grid", "volume", "batch", "born"])
    precision = rng.choice(["fp64", "mixed"])
    order = rng.choice([2, 4])
    mixed = precision == "mixed"
    budget = rng.uniform(0.002, 0.01)  # rough seconds of stepping

    def steps(sites, rate):
        return max(1, min(200, int(budget * rate / (sites * (2.5 if order == 4 else 1.0)))))

    if kind == "line":
        n = _loguniform(rng, 64, 1 << 20) | 1 if rng.random() < 0.5 else 1 << rng.randint(6, 20)
        wall = rng.random() < 0.25
        imag = rng.random() < 0.2
        if imag:
            order = 2
        rate = (8e8 if n <= 8192 else 2e10) if mixed else (8e7 if n <= 4096 else 1.2e9)
        if n & (n - 1):
            rate /= 16 if n <= 4096 else 4
        if wall:
            rate /= 2
        return dict(kind="line", n=n, precision=precision, order=order, steps=steps(n, rate), wall=wall,
                    fnes=imag or rng.random() < 0.25, imag=imag)
    if kind == "grid":
        if rng.random() < 0.6:
            nx, ny = 1 << rng.randint(7, 12), 1 << rng.randint(7, 12)
        else:
            nx, ny = _loguniform(rng, 20, 1500), _loguniform(rng, 20, 1500)
        if not mixed:
            while nx * ny > 1 << 22:
                nx, ny = (nx // 2, ny) if nx >= ny else (nx, ny // 2)
        rate = 2.5e10 if mixed else 1.5e9
        if nx & (nx - 1) or ny & (ny - 1):
            rate /= 8
        imag = rng.random() < 0.2
        if imag:
            order = 2
        return dict(kind="grid", nx=nx, ny=ny, precision=precision, order=order, steps=steps(nx * ny, rate),
                    fnes=imag or rng.random() < 0.25, imag=imag)
    if kind == "volume":
        e = [rng.randint(5, 8) for _ in range(3)]
        if not mixed:
            while sum(e) > 20:
                e[e.index(max(e))] -= 1
        nx, ny, nz = (1 << v for v in e)
        return dict(kind="volume", nx=nx, ny=ny, nz=nz, precision=precision, order=order,
                    steps=steps(nx * ny * nz, 2e10 if mixed else 1.5e9))
    if kind == "batch":
        emin = rng.randint(8, 12)
        emax = rng.randint(emin, 15)
        count = rng.randint(16, 200)
        return dict(kind="batch", count=count, emin=emin, emax=emax, precision=precision, order=order,
                    steps=steps(count * (1 << emax) / 2, 5e10 if mixed else 3e9))
    nx, ny = 1 << rng.randint(8, 11), 1 << rng.randint(8, 10)
    return dict(kind="born", nx=nx, ny=ny, precision=precision, updates=rng.randint(10, 100) if mixed else
                rng.randint(4, 10))


# --- inputs --------------------------------------------------------------------


def _axis(n, dx):
    return (torch.arange(n, dtype=torch.float64, device=DEV) - n // 2) * dx


def _packet(x, k, c, s):
    return torch.exp(1j * k * x) * torch.exp(-((x - c) ** 2) / (4 * s * s))


def _line_inputs(n, wall, rng):
    """A packet and eight bumps on n sites of spacing 0.1 (a few sites wide on the shortest lines)."""
    dx = 0.1
    x = _axis(n, dx)
    box = n * dx
    s = min(rng.uniform(2.0, 20.0), box / 20)
    k = rng.uniform(0.5, 3.0)
    psi = _packet(x, k, -box * rng.uniform(0.15, 0.25), s)
    V = torch.zeros(n, dtype=torch.float64, device=DEV)
    for _ in range(8):
        c, h, w = rng.uniform(-box / 2, box / 2), rng.uniform(-1, 1), min(rng.uniform(1, 5), box / 10)
        V += h * torch.exp(-((x - c) ** 2) / (2 * w * w))
    if wall:
        psi[0] = 0
    psi /= torch.sqrt((psi.abs() ** 2).sum() * dx)
    return psi, V, dx


def _grid_inputs(nx, ny, rng):
    """1024^2 configuration: packet k = (1.5, 0) and sixteen Gaussian bumps; from 4096 rows on the double slit with noise."""
    slit = nx >= 4096 and ny >= 4096
    dx = dy = 400.0 / 4096 if slit else 200.0 / 1024
    x, y = _axis(nx, dx), _axis(ny, dy)
    bx, by = nx * dx, ny * dy
    sx, sy = min(8.0, bx / 12), min(8.0, by / 12)
    k = rng.uniform(1.2, 2.0)
    px, py = _packet(x, k, -bx * rng.uniform(0.12, 0.2), sx), _packet(y, rng.uniform(-0.3, 0.3), 0.0, sy)
    psi = px[:, None] * py[None, :]
    psi /= torch.sqrt((px.abs() ** 2).sum() * (py.abs() ** 2).sum() * dx * dy)
    if slit:
        g = torch.Generator(device=DEV)
        g.manual_seed(rng.randrange(1 << 31))
        wall = (x.abs() < 1.0)[:, None] & ~(((y - 6.0).abs() < 1.0) | ((y + 6.0).abs() < 1.0))[None, :]
        V = wall.to(torch.float64) * 10.0
        V += torch.rand((nx, ny), dtype=torch.float64, device=DEV, generator=g) * 0.02 - 0.01
    else:
        ax, ay = [], []
        for _ in range(16):
            cx, cy = rng.uniform(-0.15, 0.15) * bx, rng.uniform(-0.15, 0.15) * by
            h, w = rng.uniform(-1, 1), min(rng.uniform(1, 5), bx / 10, by / 10)
            ax.append(h * torch.exp(-((x - cx) ** 2) / (2 * w * w)))
            ay.append(torch.exp(-((y - cy) ** 2) / (2 * w * w)))
        V = torch.stack(ax, 1) @ torch.stack(ay, 0)
    return psi, V, dx, dy


def _volume_inputs(shape, rng):
    d = 0.2
    ax = [_axis(n, d) for n in shape]
    p = [_packet(a, k, 0.0, min(2.0, len(a) * d / 12)) for a, k in zip(ax, (1.5, -0.5, 0.8))]
    psi = p[0][:, None, None] * p[1][None, :, None] * p[2][None, None, :]
    psi /= torch.sqrt((psi.abs() ** 2).sum() * d ** 3)
    c = [rng.uniform(-2, 2) for _ in range(3)]
    g = [torch.exp(-((a - b) ** 2) / 2) for a, b in zip(ax, c)]
    V = 0.8 * g[0][:, None, None] * g[1][None, :, None] * g[2][None, None, :]
    return psi, V, d


def _batch_inputs(case, rng):
    pick = random.Random(case["count"])  # the sizes belong to the case, the packets and potentials to the seed
    sizes = [1 << pick.randint(case["emin"], case["emax"]) for _ in range(case["count"])]
    got = [_line_inputs(n, False, rng) for n in sizes]
    return [g[0] for g in got], [g[1] for g in got]


BORN_EN = 2.0


def _born_inputs(nx, ny, rng):
    """A Gaussian well with a weak absorbing spot, 21 points per wavelength (10 on the smaller grids)."""
    d = 300.0 / 2048 if min(nx, ny) >= 1024 else 0.32  # the box holds 24 wavelengths
    x, y = _axis(nx, d), _axis(ny, d)
    cx, cy = rng.uniform(-5, 5), rng.uniform(-5, 5)
    V = 0.3 * torch.exp(-(x[:, None] ** 2 + y[None, :] ** 2) / 4) + 0j
    V = V - 0.02j * torch.exp(-((x[:, None] - cx) ** 2 + (y[None, :] - cy) ** 2) / 8)
    return V, d


def _dt(case):
    dt = 0.02 if case["kind"] == "grid" else 0.01
    return -1j * dt if case.get("imag") else dt


def _inputs(case, seed):
    rng = random.Random(int(seed) * 1000003 + 17)
    kind = case["kind"]
    if kind == "line":
        return _line_inputs(case["n"], case["wall"], rng)
    if kind == "grid":
        return _grid_inputs(case["nx"], case["ny"], rng)
    if kind == "volume":
        return _volume_inputs((case["nx"], case["ny"], case["nz"]), rng)
    if kind == "batch":
        return _batch_inputs(case, rng)
    return _born_inputs(case["nx"], case["ny"], rng)


# --- handles and passes -----------------------------------------------------------


def _host(t):
    return t.cpu().numpy()


def _buffers(shape, mixed):
    """The page-locked array a program reads into, and its single-precision copy for complex64 states."""
    out = torch.empty(shape, dtype=torch.complex128, pin_memory=DEV == "cuda")
    return out, (torch.empty(shape, dtype=torch.complex64) if mixed else None)


def prepare(case, seed):
    kind, mixed = case["kind"], case["precision"] == "mixed"
    ctx = q.default_context()
    got = _inputs(case, seed)
    if kind == "line" and case["n"] == 64 and not mixed:
        # the Evolver API, as the reference's programs use it
        psi, V, dx = got
        n = case["n"]
        e = q.Evolver1D()
        e.init(_host(psi), True, _dt(case), case["fnes"], _host(V), -n // 2 * dx, n // 2 * dx, n,
               q.BoundaryCondition.InfiniteWall if case["wall"] else q.BoundaryCondition.Period,
               q.SolverMethod.SplittingMethodO2 if case["order"] == 2 else q.SolverMethod.SplittingMethodO4, 1.0, 1.0,
               q.Options().Gb300().Batch(case["steps"]))
        return dict(kind="evolver", e=e)
    if kind == "batch":
        psis, Vs = got
        b = q.Batch(ctx, [_host(p) for p in psis], [_host(v) for v in Vs], [0.1] * len(psis), [_dt(case)] * len(psis),
                    case["order"], case["precision"])
        out, keep = _buffers((sum(b.sizes),), mixed)
        views, at = [], 0
        flat = out.numpy()
        for i, n in enumerate(b.sizes):
            views.append((b.instance(i), flat[at:at + n]))
            at += n
        return dict(kind="batch", b=b, views=views, steps=case["steps"], out=out, keep=keep)
    if kind == "born":
        V, d = got
        nx, ny = case["nx"], case["ny"]
        s = q.QuPerturbation2D()
        s.init(_host(V), -nx // 2 * d, nx // 2 * d, nx, -ny // 2 * d, ny // 2 * d, ny, BORN_EN, 0.0, 1.0, 0.0,
               q.SolverMethod.BornSerise, 1.0, 1.0,
               q.Options().Gb300().Precision(case["precision"]).Order(case["updates"]).Preconditional(True)
               .VellekoopPreconditioner())
        return dict(kind="born", s=s, keep=torch.empty((nx, ny), dtype=torch.complex64) if mixed else None)
    psi, V = _host(got[0]), _host(got[1])
    if kind == "line":
        inst = q.Instance.create_1d(ctx, psi, V, got[2], _dt(case), case["order"], case["precision"],
                                    boundary=q.BoundaryCondition.InfiniteWall if case["wall"]
                                    else q.BoundaryCondition.Period)
    elif kind == "grid":
        inst = q.Instance.create_2d(ctx, psi, V, got[2], got[3], _dt(case), case["order"], case["precision"])
    else:
        inst = q.Instance.create_3d(ctx, psi, V, got[2], got[2], got[2], _dt(case), case["order"], case["precision"])
    out, keep = _buffers(psi.shape, mixed)
    return dict(kind="instance", inst=inst, steps=case["steps"], fnes=bool(case.get("fnes")), out=out, view=out.numpy(),
                keep=keep)


def run(state):
    kind = state["kind"]
    if kind == "evolver":
        state["e"].step()
        return state["e"].GetPsi()
    if kind == "born":
        s = state["s"]
        s.Compute()
        psi = s.GetPsi()
        if state["keep"] is not None:
            psi = state["keep"].copy_(torch.from_numpy(psi))
        return psi
    if kind == "batch":
        state["b"].step(state["steps"])
        for view, out in state["views"]:
            view.get_psi(out)
    else:
        state["inst"].step(state["steps"], state["fnes"])
        state["inst"].get_psi(state["view"])
    return state["out"] if state["keep"] is None else state["keep"].copy_(state["out"])


def _sites(case):
    kind = case["kind"]
    if kind == "line":
        return case["n"], 2 * case["n"] if case["wall"] else case["n"]
    if kind == "grid" or kind == "born":
        return (case["nx"] * case["ny"],) * 2
    if kind == "volume":
        return (case["nx"] * case["ny"] * case["nz"],) * 2
    mean = sum(1 << e for e in range(case["emin"], case["emax"] + 1)) / (case["emax"] - case["emin"] + 1)
    return (case["count"] * mean,) * 2


def work(case):
    """psi and V in, psi out; the two transforms of each kinetic factor at 5 N log2 N, six operations per phase product."""
    n, ext = _sites(case)
    c = 8 if case["precision"] == "mixed" else 16
    log = math.log2(max(2, ext if case["kind"] != "batch" else ext / case["count"]))
    if case["kind"] == "born":
        return {"bytes": n * (2 * c + 16), "flops": case["updates"] * n * (10 * log + 40)}
    nsub = 1 if case["order"] == 2 else 3
    flops = case["steps"] * (nsub * (10 * ext * log + 6 * ext) + (nsub + 1) * 6 * n)
    return {"bytes": n * (2 * c + 8), "flops": flops}


# --- the same in 64 bits -----------------------------------------------------------


def _fold2(n):
    i = torch.arange(n, dtype=torch.float64, device=DEV)
    return torch.where(i > n // 2, n - i, i) ** 2


def _evolve(psi, V, spacing, dt, order, steps, wall=False, fnes=False):
    """Split steps of psi (its last len(spacing) axes) with torch's FFT; hbar = m = 1."""
    t = 2.0 ** (1.0 / 3.0)
    if order == 2:
        vc, tc = [0.5, 0.5], [1.0]
    else:
        c1, c2, d1, d2 = 1 / (2 * (2 - t)), (1 - t) / (2 * (2 - t)), 1 / (2 - t), -t / (2 - t)
        vc, tc = [c1, c2, c2, c1], [d1, d2, d1]
    axes = tuple(range(-len(spacing), 0))
    n0 = psi.shape[-1]
    if wall:
        psi[..., 0] = 0

        def ext(p):
            z = torch.zeros(p.shape[:-1] + (1,), dtype=p.dtype, device=p.device)
            return torch.cat([p, z, -p[..., 1:].flip(-1)], -1)
    dims = [2 * n0] if wall else list(psi.shape[-len(spacing):])
    k2 = torch.zeros(dims, dtype=torch.float64, device=DEV)
    for a, (n, d) in enumerate(zip(dims, spacing)):
        shape = [1] * len(dims)
        shape[a] = n
        k2 = k2 + (_fold2(n) * (2 * math.pi / (d * n)) ** 2 / 2).reshape(shape)
    ev = {c: torch.exp(-1j * dt * c * V) for c in set(vc)}
    et = {c: torch.exp(-1j * dt * c * k2) for c in set(tc)}
    for _ in range(steps):
        for j, c in enumerate(tc):
            psi = psi * ev[vc[j]]
            f = torch.fft.fftn(ext(psi) if wall else psi, dim=axes)
            f *= et[c]
            psi = torch.fft.ifftn(f, dim=axes)
            if wall:
                psi = psi[..., :n0].clone()
                psi[..., 0] = 0
        psi = psi * ev[vc[-1]]
    if fnes:
        psi = psi / torch.sqrt((psi.abs() ** 2).sum() * math.prod(spacing))
    return psi


def _born_exact(case, V, d):
    nx, ny = case["nx"], case["ny"]
    k0 = math.sqrt(2 * BORN_EN)
    x = (torch.arange(nx, dtype=torch.float64, device=DEV) - nx // 2) * d
    psi0 = torch.exp(1j * k0 * x)[:, None].expand(nx, ny)

    def layer(n):
        i = torch.arange(n, dtype=torch.float64, device=DEV)
        z = torch.where(i < n // 2, i, n - i) * d * k0
        u = 1 - z * z / 225.0
        return -0.8 * BORN_EN * torch.where(u > 0, torch.exp(-0.015 * z * z / torch.sqrt(u.clamp(min=1e-300))), 0.0)

    V = V + 1j * (layer(nx)[:, None] + layer(ny)[None, :])
    eps = float(V.abs().max())
    kin = (_fold2(nx) * (2 * math.pi / (d * nx)) ** 2 / 2)[:, None] + (_fold2(ny) * (2 * math.pi / (d * ny)) ** 2 / 2)
    green = 1.0 / (BORN_EN - kin + 1j * eps)
    g = 1.0 - 1j * V / eps
    psi = torch.zeros_like(V)
    for _ in range(case["updates"]):
        a = (V + 1j * eps) * psi + V.real * psi0
        a = torch.fft.ifft2(torch.fft.fft2(a) * green)
        psi = (1.0 - g) * psi + g * a
    return psi.cpu()


def exact(case, seed):
    kind = case["kind"]
    got = _inputs(case, seed)
    dt = _dt(case)
    if kind == "born":
        return _born_exact(case, *got)
    if kind == "line":
        return _evolve(got[0], got[1], (got[2],), dt, case["order"], case["steps"], case["wall"], case["fnes"]).cpu()
    if kind == "grid":
        return _evolve(got[0], got[1], got[2:4], dt, case["order"], case["steps"], False, case["fnes"]).cpu()
    if kind == "volume":
        return _evolve(got[0], got[1], (got[2],) * 3, dt, case["order"], case["steps"]).cpu()
    psis, Vs = got
    res = [None] * len(psis)
    for n in sorted({len(p) for p in psis}):
        at = [i for i, p in enumerate(psis) if len(p) == n]
        r = _evolve(torch.stack([psis[i] for i in at]), torch.stack([Vs[i] for i in at]), (0.1,), dt, case["order"],
                    case["steps"])
        for i, v in zip(at, r):
            res[i] = v
    return torch.cat(res).cpu()
