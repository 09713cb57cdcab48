"""The work a simulation code has this framework do, as measurable cases.

Each case is one call (or the calls of one step) through the public entry points of gamer_b200: the
fluid solver of a refinement level (MHM, MHM_RP, CTU; hydro and MHD; FP32, mixed, FP64), a whole
multi-level sub-step from its captured graph, the drop-in call on host arrays, the ghost-zone fill
before a solve, the close of a step after it, and K differentiable steps with their backward pass.
The configurations and sizes are those of bench.py, its workloads and the tests.

``listed`` names the cases, ``draw`` gives more of the same ranges, ``prepare`` makes what the caller
has in hand, ``run`` is one pass, ``work`` the bytes and operations it cannot do without, and
``exact`` the same outputs from a 64-bit evaluation of the scheme in plain torch.
"""
from __future__ import annotations

import math

import torch
import torch.nn.functional as nnf

from gamer_b200 import fluid
from gamer_b200.adjoint import mhm_steps
from gamer_b200.fluid import FluidSolver, SolverParams

GAMMA = 5.0 / 3.0
GM1 = GAMMA - 1.0
PS = 16                        # width of a patch group in cells
CELLS = PS ** 3
LEVELS = (512, 1536, 3072, 1024)
DEV = "cuda:0"
CHUNK = 64                     # patch groups per chunk of the 64-bit evaluation


# ---------------------------------------------------------------------------------------------------
# the cases
# ---------------------------------------------------------------------------------------------------
def listed():
    return [
        # one 32^3 root level: the smallest level GAMER hands to the solver, where a step waits for it
        dict(name="mhm_fp32_8", kind="solve", scheme="mhm", lr="plm", rs="hllc", prec="fp32", dual=False, flow="lognormal", npg=8),
        # the headline: a 256^3 level of the Kelvin-Helmholtz layer, device-resident arrays
        dict(name="mhm_fp32_4096", kind="solve", scheme="mhm", lr="plm", rs="hllc", prec="fp32", dual=False, flow="kh", npg=4096),
        # third-order reconstruction with Roe's solver in the mixed policy on a 160^3 level
        dict(name="mhm_ppm_roe_mixed_1000", kind="solve", scheme="mhm", lr="ppm", rs="roe", prec="mixed", dual=False, flow="kh", npg=1000),
        # a double-precision build (GAMER's FLOAT8) on a 128^3 level
        dict(name="mhm_fp64_512", kind="solve", scheme="mhm", lr="plm", rs="hllc", prec="fp64", dual=False, flow="lognormal", npg=512),
        # the MHM_RP scheme (mixed policy) on a level of an odd 9 x 9 x 9 patch groups
        dict(name="mhm_rp_mixed_729", kind="solve", scheme="mhm_rp", lr="plm", rs="hllc", prec="mixed", dual=False, flow="kh", npg=729),
        # the CTU scheme on the headline's level
        dict(name="ctu_fp32_4096", kind="solve", scheme="ctu", lr="plm", rs="hllc", prec="fp32", dual=False, flow="kh", npg=4096),
        # magnetised CTU (HLLD, constrained transport) with the coarse-fine flux and EMF planes
        dict(name="ctu_mhd_fp32_2048", kind="mhd", lr="plm", prec="fp32", npg=2048),
        # every level of a sub-step (uneven counts) with dual energy on a blast wave, graph replay
        dict(name="levels_dual_fp32", kind="levels", prec="fp32", n0=512, n1=1536, n2=3072, n3=1024),
        # GAMER's own call on (pinned) host arrays, one batch of 64 patch groups, FLU_NXT 22
        dict(name="host_fp32_64", kind="host", prec="fp32", nxt=22, flow="lognormal", npg=64),
        # the ghost-zone fill of a level of 512 patch groups: interpolation from the parents, assembly
        dict(name="ghost_fill_512", kind="ghost", prec="fp32", px=8, py=8, pz=8),
        # the close of a step: unphysical cells, coarse-fine flux fix-up, the next time step
        dict(name="close_fp32_2048", kind="close", prec="fp32", npg=2048),
        # a gradient: eight differentiable steps of a 128 x 128 x 256 box and their backward pass
        dict(name="adjoint_k8_1024", kind="adjoint", prec="fp32", px=8, py=8, pz=16, K=8),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """One more case of the ranges of the listed ones: any number of patch groups, the options that
    are used together with each scheme, every precision policy."""
    kind = rng.choice(["solve", "solve", "solve", "mhd", "levels", "host", "ghost", "close", "adjoint"])
    if kind == "solve":
        scheme = rng.choice(["mhm", "mhm", "mhm_rp", "ctu"])
        lr = "plm" if scheme == "mhm_rp" else rng.choice(["plm", "ppm"])
        rs = rng.choice(["hllc", "roe"]) if scheme == "mhm" else "hllc"
        prec = rng.choice(["fp32", "mixed", "fp64"])
        return dict(kind=kind, scheme=scheme, lr=lr, rs=rs, prec=prec,
                    dual=scheme == "mhm" and rng.random() < 0.3, flow=rng.choice(["kh", "lognormal"]),
                    npg=_log(rng, 1, 1024 if prec == "fp64" or lr == "ppm" else 3000))
    if kind == "mhd":
        prec = rng.choice(["fp32", "fp32", "mixed", "fp64"])
        return dict(kind=kind, lr=rng.choice(["plm", "ppm"]), prec=prec,
                    npg=_log(rng, 8, 300 if prec == "fp64" else 900))
    if kind == "levels":
        return dict(kind=kind, prec=rng.choice(["fp32", "mixed"]), n0=_log(rng, 1, 64), n1=_log(rng, 8, 512),
                    n2=_log(rng, 8, 1500), n3=_log(rng, 8, 1500))
    if kind == "host":
        prec = rng.choice(["fp32", "mixed", "fp64"])
        return dict(kind=kind, prec=prec, nxt=rng.choice([20, 22]), flow=rng.choice(["kh", "lognormal"]),
                    npg=_log(rng, 8, 600))
    if kind == "ghost":
        return dict(kind=kind, prec=rng.choice(["fp32", "fp64"]), px=rng.randint(2, 8), py=rng.randint(2, 8),
                    pz=rng.randint(2, 8))
    if kind == "close":
        return dict(kind=kind, prec=rng.choice(["fp32", "mixed", "fp64"]), npg=_log(rng, 8, 2048))
    return dict(kind=kind, prec=rng.choice(["fp32", "fp32", "fp64"]), px=rng.randint(1, 4), py=rng.randint(1, 4),
                pz=rng.randint(1, 6), K=rng.randint(1, 4))


# ---------------------------------------------------------------------------------------------------
# initial states: periodic boxes [v][z][y][x] in double on the GPU, cut into windows
# ---------------------------------------------------------------------------------------------------
def _gen(seed):
    g = torch.Generator(device=DEV)
    g.manual_seed(seed)
    return g


def _normal(g, shape, std=1.0):
    return std * torch.randn(shape, generator=g, device=DEV, dtype=torch.float64)


def _smooth(g, shape, std, kmax=3):
    """Gaussian noise of the Fourier modes |k_i| <= kmax with the given standard deviation."""
    f = torch.fft.fftn(_normal(g, shape))
    for axis, n in enumerate(shape):
        keep = (torch.fft.fftfreq(n, 1.0 / n, device=DEV).abs() <= kmax).to(torch.float64)
        f = f * keep.reshape([-1 if a == axis else 1 for a in range(3)])
    x = torch.fft.ifftn(f).real
    x = x - x.mean()
    return x * (std / x.std())


def _conserved(rho, v, p, dual=False):
    u = [rho, rho * v[0], rho * v[1], rho * v[2], p / GM1 + 0.5 * rho * (v[0] ** 2 + v[1] ** 2 + v[2] ** 2)]
    if dual:
        u.append(p * rho ** (1.0 - GAMMA))
    return torch.stack(u)


def _axes(shape):
    return [((torch.arange(n, device=DEV, dtype=torch.float64) + 0.5) / n).reshape([-1 if a == i else 1 for a in range(3)])
            for i, n in enumerate(shape)]


def _flow(g, shape, flow, dual=False):
    """kh: a shear layer; lognormal: smoothed lognormal density, cell-by-cell lognormal pressure and
    velocities up to the sound speed; smooth: a few long waves; blast: a Mach-10 blast on a lognormal
    background."""
    z, y, x = _axes(shape)
    if flow == "kh":
        inner = ((y - 0.5).abs() < 0.25) & (x > -1) & (z > -1)
        rho = torch.where(inner, 2.0, 1.0).to(torch.float64)
        vx = torch.where(inner, 0.5, -0.5).to(torch.float64)
        vy = 0.01 * torch.sin(4.0 * math.pi * x) + _normal(g, shape, 1e-4)
        return _conserved(rho, (vx, vy, torch.zeros_like(vx)), torch.full_like(rho, 2.5), dual)
    if flow == "smooth":
        v = [0.3 * _smooth(g, shape, 1.0, 4) for _ in range(3)]
        return _conserved(1.0 + 0.1 * _smooth(g, shape, 1.0, 4), v, 1.0 + 0.1 * _smooth(g, shape, 1.0, 4), dual)
    rho = torch.exp(_smooth(g, shape, 0.3))
    p = torch.exp(_normal(g, shape, 0.2))
    rand = 2.0 * torch.rand((3,) + tuple(shape), generator=g, device=DEV, dtype=torch.float64) - 1.0
    if flow == "lognormal":
        return _conserved(rho, rand * torch.sqrt(GAMMA * p / rho), p, dual)
    p = p * 1e-2
    inside = ((x - 0.5) ** 2 + (y - 0.5) ** 2 + (z - 0.5) ** 2) < 0.01
    v = torch.where(inside, 0.0, rand * 10.0 * math.sqrt(GAMMA * 1e-2))
    return _conserved(torch.where(inside, rho * 1e3, rho), v, torch.where(inside, p * 1e5, p), dual)


def _cfl(box, dh, cfl):
    rho, v = box[0], box[1:4] / box[0]
    p = GM1 * (box[4] - 0.5 * rho * (v ** 2).sum(0))
    return cfl * dh / float((v.abs() + torch.sqrt(GAMMA * p / rho)).max())


def _windows(box, nxt, extra=(0, 0, 0)):
    """[v][Z][Y][X] periodic -> [npg][v][nxt(+extra)^3] windows, patch groups x fastest; ``extra``
    faces more along (x, y, z)."""
    g = (nxt - PS) // 2
    for axis, e in ((1, extra[2]), (2, extra[1]), (3, extra[0])):
        n = box.shape[axis]
        idx = torch.arange(-g, n + g + e, device=DEV) % n
        box = box.index_select(axis, idx).unfold(axis, nxt + e, PS)
    # box: [v][pz][py][px][z][y][x]
    return box.permute(1, 2, 3, 0, 4, 5, 6).reshape((-1, box.shape[0]) + tuple(box.shape[4:])).contiguous()


def _dims(npg):
    """(pz, py, px) of a box with at least npg patch groups."""
    p = max(1, math.ceil(round(npg ** (1.0 / 3.0), 9)))
    while p ** 3 < npg:
        p += 1
    q = max(1, math.ceil(npg / (p * p)))
    return q, p, p


def _dtype(prec):
    return torch.float64 if prec == "fp64" else torch.float32


def _nxt(scheme, lr):
    return {"mhm": 20, "ctu": 20, "mhm_rp": 22}[scheme] + (2 if lr == "ppm" else 0)


def _hydro(case, seed, nxt, cfl=0.4):
    """Windows of the case's flow in its storage type, dt and dh."""
    pz, py, px = _dims(case["npg"])
    shape = (pz * PS, py * PS, px * PS)
    box = _flow(_gen(seed), shape, case["flow"], case.get("dual", False))
    dh = 1.0 / max(shape)
    return _windows(box, nxt)[:case["npg"]].to(_dtype(case["prec"])).contiguous(), _cfl(box, dh, cfl), dh


def _magnetised(case, seed, nxt):
    """Windows of a beta ~ 1 lognormal state with a divergence-free face-centred field: the discrete
    curl of a smooth edge-centred vector potential plus a mean field."""
    g = _gen(seed)
    pz, py, px = _dims(case["npg"])
    shape = (pz * PS, py * PS, px * PS)
    rho = torch.exp(_smooth(g, shape, 0.3))
    p = torch.exp(_smooth(g, shape, 0.2))
    v = [0.5 * torch.sqrt(GAMMA * p / rho) * _smooth(g, shape, 1.0) for _ in range(3)]
    a = [0.6 * max(shape) / (8.0 * math.pi) * _smooth(g, shape, 1.0, 4) for _ in range(3)]
    d = lambda f, axis: torch.roll(f, -1, 2 - axis) - f  # noqa: E731  (axis 0 is x, the last)
    b = [0.8 + d(a[2], 1) - d(a[1], 2), 0.6 + d(a[0], 2) - d(a[2], 0), 0.5 + d(a[1], 0) - d(a[0], 1)]
    bcc = [0.5 * (b[i] + torch.roll(b[i], -1, 2 - i)) for i in range(3)]
    u = _conserved(rho, v, p)
    u[4] += 0.5 * (bcc[0] ** 2 + bcc[1] ** 2 + bcc[2] ** 2)
    dh = 1.0 / max(shape)
    a2 = (GAMMA * p + bcc[0] ** 2 + bcc[1] ** 2 + bcc[2] ** 2) / rho
    dt = 0.3 * dh / float((torch.stack(v).abs() + torch.sqrt(a2)).max())
    n, dtype = case["npg"], _dtype(case["prec"])
    mag = torch.stack([_windows(b[i][None], nxt, [int(i == k) for k in range(3)])[:n].reshape(n, -1) for i in range(3)], 1)
    return _windows(u, nxt)[:n].to(dtype).contiguous(), mag.to(dtype).contiguous(), dt, dh


def _levels(case, seed):
    """The windows of four levels one after the other (each level half the cell size of the one
    above), from a blast on a lognormal background."""
    npg = [case["n%d" % i] for i in range(4)]
    win, dts, dhs = [], [], []
    for lv, n in enumerate(npg):
        pz, py, px = _dims(n)
        shape = (pz * PS, py * PS, px * PS)
        box = _flow(_gen(seed * 4 + lv), shape, "blast", True)
        dh = 1.0 / (64 << lv)
        win.append(_windows(box, 20)[:n])
        dts.append(_cfl(box, dh, 0.3))
        dhs.append(dh)
    return torch.cat(win).to(_dtype(case["prec"])).contiguous(), npg, dts, dhs


# the ghost-zone fill: a coarse level, the fine patch groups over a part of it
def _ghost(case, seed):
    g = _gen(seed)
    px, py, pz = case["px"], case["py"], case["pz"]
    dtype = _dtype(case["prec"])
    coarse = _flow(g, (pz * 8, py * 8, px * 8), "lognormal")
    # 12^3 coarse cells around each window of 20^3 fine cells: its 10^3 parents and one cell more
    idx = [torch.arange(-2, n + 2, device=DEV) % n for n in coarse.shape[1:]]
    c = coarse
    for axis in range(3):
        c = c.index_select(axis + 1, idx[axis]).unfold(axis + 1, 12, 8)
    c = c.permute(1, 2, 3, 0, 4, 5, 6).reshape(-1, 5, 12, 12, 12)
    fine = _windows(_flow(g, (pz * PS, py * PS, px * PS), "lognormal"), PS)
    # two thirds of the coarse level is refined; the windows of the refined part are filled
    total = px * py * pz
    have = torch.zeros(total, dtype=torch.bool, device=DEV)
    have[torch.randperm(total, generator=g, device=DEV)[:(2 * total + 2) // 3]] = True
    number = torch.where(have, torch.cumsum(have, 0) - 1, -1).view(pz, py, px)
    have = have.view(pz, py, px)
    nbr = torch.stack([torch.roll(number, (-dz, -dy, -dx), (0, 1, 2))
                       for dz in (-1, 0, 1) for dy in (-1, 0, 1) for dx in (-1, 0, 1)], -1)[have].to(torch.int32)
    keep = have.view(-1)
    return c[keep].to(dtype).contiguous(), fine[keep].to(dtype).contiguous(), nbr.contiguous()


# the close: a solver output with a few cells that went unphysical, and patches with flux differences
def _close(case, seed):
    n, dtype = case["npg"], _dtype(case["prec"])
    g = _gen(seed)
    pz, py, px = _dims(n)
    shape = (pz * PS, py * PS, px * PS)
    box = _flow(g, shape, "lognormal")
    dh = 1.0 / max(shape)
    win = _windows(box, 20)[:n].to(dtype).contiguous()
    out = win[:, :, 2:-2, 2:-2, 2:-2].clone()
    bad = torch.rand(out[:, 0].shape, generator=g, device=DEV) < 1.0e-5
    out[:, 0] = torch.where(bad, -out[:, 0], out[:, 0])
    flux = _normal(g, (n, 9, 5, PS, PS), 0.1).to(dtype)
    patch = _windows(box, PS)[:n].reshape(n, 5, 2, 8, 2, 8, 2, 8).permute(0, 2, 4, 6, 1, 3, 5, 7)
    patch = patch.reshape(8 * n, 5, 8, 8, 8).to(dtype).contiguous()
    diff = (_normal(g, (8 * n, 6, 5, 8, 8), 1e-2) * dh).to(dtype)
    has = (torch.rand((8 * n, 6), generator=g, device=DEV) < 0.4).to(torch.uint8)
    return win, out, bad, flux, patch, diff, has, _cfl(box, dh, 0.2), dh


def _adjoint_box(case, seed):
    shape = (case["pz"] * PS, case["py"] * PS, case["px"] * PS)
    g = _gen(seed)
    box = _flow(g, shape, "smooth")
    w = _normal(g, shape)
    dh = 1.0 / max(shape)
    return box.to(_dtype(case["prec"])), w, _cfl(box, dh, 0.4), dh


# ---------------------------------------------------------------------------------------------------
# what the caller has in hand, and one pass
# ---------------------------------------------------------------------------------------------------
def prepare(case, seed):
    kind, prec = case["kind"], case["prec"]
    if kind == "solve":
        nc = 6 if case["dual"] else 5
        s = FluidSolver(scheme=case["scheme"], lr=case["lr"], rsolver=case["rs"], precision=prec, dual_energy=case["dual"],
                        gamma=GAMMA)
        x, dt, dh = _hydro(case, seed, s.flu_nxt)
        n = case["npg"]
        out = torch.zeros((n, nc, PS, PS, PS), dtype=x.dtype, device=DEV)
        flux = torch.zeros((n, 9, nc, PS, PS), dtype=x.dtype, device=DEV)
        de = torch.full((n, PS, PS, PS), 48, dtype=torch.int8, device=DEV) if case["dual"] else None
        return dict(case=case, s=s, x=x, out=out, flux=flux, de=de, prm=SolverParams(dt=dt, dh=dh, StoreFlux=True))
    if kind == "mhd":
        s = FluidSolver(scheme="ctu", lr=case["lr"], rsolver="hlld", precision=prec, gamma=GAMMA)
        x, mag, dt, dh = _magnetised(case, seed, s.flu_nxt)
        n = case["npg"]
        return dict(case=case, s=s, x=x, mag=mag, out=torch.zeros((n, 5, PS, PS, PS), dtype=x.dtype, device=DEV),
                    flux=torch.zeros((n, 9, 5, PS, PS), dtype=x.dtype, device=DEV),
                    mag_out=torch.zeros((n, 3, 17 * PS * PS), dtype=x.dtype, device=DEV),
                    ele=torch.zeros((n, 9, 2, 17 * PS), dtype=x.dtype, device=DEV),
                    prm=SolverParams(dt=dt, dh=dh, StoreFlux=True, StoreElectric=True))
    if kind == "levels":
        s = FluidSolver(precision=prec, dual_energy=True, gamma=GAMMA)
        x, npg, dts, dhs = _levels(case, seed)
        n = x.shape[0]
        out = torch.zeros((n, 6, PS, PS, PS), dtype=x.dtype, device=DEV)
        flux = torch.zeros((n, 9, 6, PS, PS), dtype=x.dtype, device=DEV)
        de = torch.full((n, PS, PS, PS), 48, dtype=torch.int8, device=DEV)
        graph = s.capture_levels(x, out, npg, dts, dhs, SolverParams(dt=dts[0], dh=dhs[0], StoreFlux=True), flux=flux, de_out=de)
        return dict(case=case, s=s, graph=graph, out=out, flux=flux, de=de)
    if kind == "host":
        s = FluidSolver(precision=prec, flu_nxt=case["nxt"], gamma=GAMMA)
        x, dt, dh = _hydro(case, seed, case["nxt"])
        n = case["npg"]
        out = torch.zeros((n, 5, PS, PS, PS), dtype=x.dtype).pin_memory().numpy()
        flux = torch.zeros((n, 9, 5, PS, PS), dtype=x.dtype).pin_memory().numpy()
        return dict(case=case, s=s, x=x.cpu().pin_memory().numpy(), out=out, flux=flux,
                    prm=SolverParams(dt=dt, dh=dh, StoreFlux=True))
    if kind == "ghost":
        c, fine, nbr = _ghost(case, seed)
        n = c.shape[0]
        return dict(case=case, c=c, fine=fine, nbr=nbr, status=torch.zeros(1, dtype=torch.int32, device=DEV),
                    cint=torch.zeros((n, 5, 20, 20, 20), dtype=c.dtype, device=DEV),
                    win=torch.zeros((n, 5, 20, 20, 20), dtype=c.dtype, device=DEV))
    if kind == "close":
        win, out, _, flux, patch, diff, has, dt, dh = _close(case, seed)
        s = FluidSolver(precision=prec, gamma=GAMMA)
        return dict(case=case, s=s, win=win, out=out, flux=flux, patch=patch, diffs=[diff, -diff], has=has,
                    counts=torch.zeros(2, dtype=torch.int32, device=DEV),
                    dts=torch.zeros(8 * case["npg"], dtype=out.dtype, device=DEV), prm=SolverParams(dt=dt, dh=dh))
    box, w, dt, dh = _adjoint_box(case, seed)
    s = FluidSolver(precision=prec, gamma=GAMMA)
    return dict(case=case, s=s, box=box, w=w, prm=SolverParams(dt=dt, dh=dh))


def run(state):
    st, kind = state, state["case"]["kind"]
    if kind == "solve":
        st["s"].solve_device(st["x"], st["out"], st["prm"], flux=st["flux"], de_out=st["de"])
        return dict(out=st["out"], flux=st["flux"], de=st["de"])
    if kind == "mhd":
        st["s"].solve_device(st["x"], st["out"], st["prm"], flux=st["flux"], mag_in=st["mag"], mag_out=st["mag_out"],
                             ele=st["ele"])
        return dict(out=st["out"], flux=st["flux"], mag=st["mag_out"], ele=st["ele"])
    if kind == "levels":
        st["graph"].launch()
        return dict(out=st["out"], flux=st["flux"], de=st["de"])
    if kind == "host":
        st["s"].solve_host(st["x"], st["prm"], flu_out=st["out"], flux=st["flux"])
        return dict(out=st["out"], flux=st["flux"])
    if kind == "ghost":
        fluid.interpolate_device(st["c"], st["cint"], "cquad", (1, 1, 1), (10, 10, 10), iterate=True, status=st["status"])
        fluid.assemble_windows_device(st["fine"], st["nbr"], st["cint"], st["win"])
        return dict(cint=st["cint"], win=st["win"], status=st["status"])
    if kind == "close":
        st["s"].correct_unphysical_device(st["win"], st["out"], st["prm"], flux=st["flux"], counts=st["counts"])
        # a new set of flux differences each step (here: the last one's, reversed)
        st["s"].flux_fixup_device(st["patch"], st["diffs"][0], st["has"], st["prm"])
        st["diffs"].reverse()
        st["s"].dt_cfl(st["out"], st["prm"].dh, safety=0.5, from_output=True, dt_out=st["dts"])
        return dict(out=st["out"], flux=st["flux"], patch=st["patch"], dt=st["dts"], counts=st["counts"])
    x = st["box"].clone().requires_grad_(True)
    y = mhm_steps(x, st["case"]["K"], st["s"], st["prm"])
    (y[0].double() * st["w"]).sum().backward()
    return dict(box=y.detach(), grad=x.grad)


# ---------------------------------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------------------------------
# floating-point operations of one updated cell and step, counted from the scheme's formulae with
# every face and face state formed once: per direction the limited slopes and face values (PLM 9 a
# variable, PPM 3 x 9 + 25), primitive -> conserved and the fluxes of two face states (60), and the
# Riemann problem (HLLC 110, Roe 200, HLLD 350); Hancock (60 a direction) or the tracing, transverse
# correction and second Riemann problem of CTU; the conversion (20) and the update (40)
def _flops_cell(scheme, lr, rs, nc):
    face = (52 if lr == "ppm" else 9) * nc
    riem = {"hllc": 110, "roe": 200, "hlld": 350}[rs]
    if scheme == "mhm":
        return 20 + 3 * (face + 60 + 60 + riem) + 40
    if scheme == "mhm_rp":
        return 20 + 3 * riem + 60 + 3 * (face + 30 + riem) + 40
    trace = 60 if rs == "hlld" else 30
    emf = 2 * 3 * 60 if rs == "hlld" else 0
    return 20 + 3 * (face + trace + 30 + 2 * riem + 40) + emf + 40


def work(case):
    kind, b = case["kind"], 8 if case["prec"] == "fp64" else 4
    if kind == "solve":
        nc, n = 6 if case["dual"] else 5, case["npg"]
        per = (_nxt(case["scheme"], case["lr"]) ** 3 + CELLS + 9 * PS * PS) * nc * b + (CELLS if case["dual"] else 0)
        return dict(bytes=n * per, flops=n * CELLS * _flops_cell(case["scheme"], case["lr"], case["rs"], nc))
    if kind == "mhd":
        nx = 24 if case["lr"] == "ppm" else 22
        per = (5 * nx ** 3 + 3 * (nx + 1) * nx * nx + 5 * CELLS + 3 * 17 * PS * PS + 45 * PS * PS + 18 * 17 * PS) * b
        return dict(bytes=case["npg"] * per, flops=case["npg"] * CELLS * _flops_cell("ctu", case["lr"], "hlld", 8))
    if kind == "levels":
        n = sum(case["n%d" % i] for i in range(4))
        return dict(bytes=n * ((20 ** 3 + CELLS + 9 * PS * PS) * 6 * b + CELLS), flops=n * CELLS * _flops_cell("mhm", "plm", "hllc", 6))
    if kind == "host":
        return dict(bytes=case["npg"] * (case["nxt"] ** 3 + CELLS + 9 * PS * PS) * 5 * b,
                    flops=case["npg"] * CELLS * _flops_cell("mhm", "plm", "hllc", 5))
    if kind == "ghost":
        # two thirds of the positions hold a patch group: coarse cells and interiors in, both
        # windows out, the interpolated one in again; 7 one-dimensional stencils of 10 a parent's child
        n = (2 * case["px"] * case["py"] * case["pz"] + 2) // 3
        return dict(bytes=n * 5 * (12 ** 3 + 3 * 20 ** 3) * b, flops=n * 5 * 1000 * 8 * 30)
    if kind == "close":
        # every output cell read by the scan and by the time step, and written nowhere; the layers of
        # the patches' flux faces (0.4 of them) read and written, their fluxes read
        n = case["npg"]
        return dict(bytes=n * b * (2 * 5 * CELLS + 8 * 0.4 * 6 * 64 * 5 * 3), flops=n * CELLS * 40)
    cells = case["px"] * case["py"] * case["pz"] * CELLS
    f = _flops_cell("mhm", "plm", "hllc", 5)
    # a step reads and writes the box; its adjoint reads the box and the gradient and writes one (double)
    return dict(bytes=case["K"] * cells * 5 * (3 * b + 16), flops=case["K"] * cells * f * 5)


# four times the largest error against ``exact`` seen over the listed cases and 80 drawn ones: rel,
# and max, which a few cells reach that take another branch of a limiter, of the upwinding of an EMF
# or of the dual-energy switch in another rounding
_TOL = {
    "hydro": {"fp32": (6e-7, 1e-5), "fp64": (2e-15, 1e-13)},
    "mhd": {"fp32": (2.5e-4, 0.05), "fp64": (5e-13, 1e-10)},
    "levels": {"fp32": (4e-6, 0.01)},
    "ghost": {"fp32": (2e-7, 2e-6), "fp64": (1e-15, 1e-14)},
    "close": {"fp32": (3e-7, 1e-5), "fp64": (1e-15, 1e-14)},
    "adjoint": {"fp32": (6e-3, 0.9), "fp64": (1e-11, 1e-6)},
}


def tolerance(case):
    kind = {"solve": "hydro", "host": "hydro"}.get(case["kind"], case["kind"])
    rel, most = _TOL[kind]["fp64" if case["prec"] == "fp64" else "fp32"]
    return {"rel": rel, "max": most, "differ": 1e-4 if kind == "levels" or case.get("dual") else 0.0}


# ---------------------------------------------------------------------------------------------------
# the scheme in 64 bits: arrays [n][v][z][y][x], axis 0 / 1 / 2 = x / y / z
# ---------------------------------------------------------------------------------------------------
def _dim(d):
    return -1 - d


def _cut(a, d, lo, n):
    return a.narrow(_dim(d), lo, n)


def _box(a, lo, n):
    """n cells from cell lo along each axis (numbers, or one per axis)."""
    lo = (lo,) * 3 if isinstance(lo, int) else lo
    n = (n,) * 3 if isinstance(n, int) else n
    for d in range(3):
        a = _cut(a, d, lo[d], n[d])
    return a


def _e(d, k=1):
    return tuple(k if i == d else 0 for i in range(3))


def _plus(a, b):
    return tuple(x + y for x, y in zip(a, b))


def _prim(u, emag=0.0):
    rho = u[:, 0:1]
    v = u[:, 1:4] / rho
    p = (GM1 * (u[:, 4:5] - 0.5 * rho * (v * v).sum(1, keepdim=True) - emag)).clamp(min=0.0)
    return torch.cat([rho, v, p, u[:, 5:]], 1)


def _cons(w, emag=0.0):
    rho, v = w[:, 0:1], w[:, 1:4]
    e = 0.5 * rho * (v * v).sum(1, keepdim=True) + w[:, 4:5] / GM1 + emag
    return torch.cat([rho, rho * v, e, w[:, 5:]], 1)


def _limit(l, c, r):
    a, b = c - l, r - c
    s = torch.minimum(torch.minimum(1.5 * a.abs(), 1.5 * b.abs()), 0.5 * (a + b).abs())
    return torch.where(a * b > 0, s * torch.sign(a + b), torch.zeros_like(s))


def _faces(w, d, lo, n, lr):
    """Left and right face values along d of the n^3 cells from cell lo."""
    at = lambda k: _box(w, _plus((lo,) * 3, _e(d, k)), n)  # noqa: E731
    l, c, r = at(-1), at(0), at(1)
    if lr == "plm":
        h = 0.5 * _limit(l, c, r)
        return c - h, c + h
    dl, dc, dr = _limit(at(-2), l, c), _limit(l, c, r), _limit(c, r, at(2))
    fl = 0.5 * (c + l) - (dc - dl) / 6.0
    fr = 0.5 * (c + r) - (dr - dc) / 6.0
    df, d6 = fr - fl, 6.0 * (c - 0.5 * (fl + fr))
    flat = (fr - c) * (c - fl) <= 0
    new_l = torch.where(flat, c, torch.where(df * d6 > df * df, 3.0 * c - 2.0 * fr, fl))
    new_r = torch.where(flat, c, torch.where(~(df * d6 > df * df) & (df * d6 < -df * df), 3.0 * c - 2.0 * fl, fr))
    return (torch.maximum(torch.minimum(new_l, torch.maximum(c, l)), torch.minimum(c, l)),
            torch.maximum(torch.minimum(new_r, torch.maximum(c, r)), torch.minimum(c, r)))


def _flux(u, p, d, b=None):
    """Physical flux along d; ``b``: the cell's magnetic field (u[:, 5:8]) enters."""
    vn = u[:, 1 + d:2 + d] / u[:, 0:1]
    f = vn * u
    f = torch.cat([f[:, :4], vn * (u[:, 4:5] + p), f[:, 5:]], 1)
    add = torch.zeros_like(f)
    add[:, 1 + d] = p[:, 0]
    if b is not None:
        em, v = 0.5 * (b * b).sum(1), u[:, 1:4] / u[:, 0:1]
        bn = b[:, d]
        add[:, 1 + d] += em
        add[:, 1:4] -= bn[:, None] * b
        add[:, 4] += vn[:, 0] * em - bn * (b * v).sum(1)
        add[:, 5:8] -= bn[:, None] * v
    return f + add


def _upwind_passive(f, L, R, nc):
    if nc == 5:
        return f
    m = f[:, 0:1]
    return torch.cat([f, torch.where(m >= 0, m * L[:, 5:] / L[:, 0:1], m * R[:, 5:] / R[:, 0:1])], 1)


def _hlle(L, R, d):
    nc, wl, wr = L.shape[1], _prim(L), _prim(R)
    cl, cr = (torch.sqrt(GAMMA * w[:, 4:5] / w[:, 0:1]) for w in (wl, wr))
    ul, ur = wl[:, 1 + d:2 + d], wr[:, 1 + d:2 + d]
    sl = torch.minimum(ul - cl, ur - cr).clamp(max=0.0)
    sr = torch.maximum(ul + cl, ur + cr).clamp(min=0.0)
    fl, fr = (_flux(u, w[:, 4:5], d)[:, :5] for u, w in ((L, wl), (R, wr)))
    f = (sr * (fl - sl * L[:, :5]) - sl * (fr - sr * R[:, :5])) / (sr - sl)
    return _upwind_passive(f, L, R, nc)


def _hllc(L, R, d):
    nc, wl, wr = L.shape[1], _prim(L), _prim(R)
    pl, pr, ul, ur = wl[:, 4:5], wr[:, 4:5], wl[:, 1 + d:2 + d], wr[:, 1 + d:2 + d]
    cl, cr = torch.sqrt(GAMMA * pl / wl[:, 0:1]), torch.sqrt(GAMMA * pr / wr[:, 0:1])
    sl, sr = torch.minimum(ul - cl, ur - cr), torch.maximum(ul + cl, ur + cr)
    al, ar = L[:, 0:1] * (ul - sl), R[:, 0:1] * (ur - sr)
    vs = (pl - pr + al * ul - ar * ur) / (al - ar)
    ps = ((al * (pr + ar * ur) - ar * (pl + al * ul)) / (al - ar)).clamp(min=0.0)
    left = vs >= 0
    u, p = torch.where(left, L, R), torch.where(left, pl, pr)
    s = torch.where(left, sl.clamp(max=0.0), sr.clamp(min=0.0))
    f = _flux(u, p, d)[:, :5] - s * u[:, :5]
    gap = vs - s
    still = gap == 0
    gap = torch.where(still, torch.ones_like(gap), gap)
    star = -s * ps / gap
    add = torch.zeros_like(f)
    add[:, 1 + d] = 1.0
    f = torch.where(still, f, f * vs / gap + star * torch.cat([add[:, :4], vs], 1))
    return _upwind_passive(f, L, R, nc)


def _roe(L, R, d):
    """Roe with the check of the intermediate states (HLLE where one is unphysical)."""
    nc, wl, wr = L.shape[1], _prim(L), _prim(R)
    perm = [0, 1 + d, 1 + (d + 1) % 3, 1 + (d + 2) % 3, 4]
    back = [perm.index(i) for i in range(5)]
    fl, fr = (_flux(u, w[:, 4:5], d) for u, w in ((L, wl), (R, wr)))
    l, r = L[:, perm], R[:, perm]
    sl, sr = torch.sqrt(L[:, 0]), torch.sqrt(R[:, 0])
    mean = lambda a, b: (sl * a + sr * b) / (sl + sr)  # noqa: E731
    u, v, w = (mean(wl[:, perm[i]], wr[:, perm[i]]) for i in (1, 2, 3))
    H = mean((L[:, 4] + wl[:, 4]) / L[:, 0], (R[:, 4] + wr[:, 4]) / R[:, 0])
    q = u * u + v * v + w * w
    a2 = GM1 * (H - 0.5 * q)
    a = torch.sqrt(a2)
    J = (r - l).unbind(1)
    A2, A3 = J[2] - v * J[0], J[3] - w * J[0]
    A1 = GM1 / a2 * (J[0] * (H - u * u) + u * J[1] - J[4] + v * A2 + w * A3)
    A0 = 0.5 / a * (J[0] * (u + a) - J[1] - a * A1)
    A4 = J[0] - A0 - A1
    one, zero = torch.ones_like(u), torch.zeros_like(u)
    E = [[one, u - a, v, w, H - u * a], [one, u, v, w, 0.5 * q], [zero, zero, one, zero, v], [zero, zero, zero, one, w],
         [one, u + a, v, w, H + u * a]]
    E = [torch.stack(e, 1) for e in E]
    state, bad = l, torch.zeros_like(u, dtype=torch.bool)
    for A, e, test in ((A0, E[0], True), (A1, E[1], False), (A2, E[2], False), (A3, E[3], True)):
        state = state + A[:, None] * e
        if test:
            ip = state[:, 4] - 0.5 * (state[:, 1:4] ** 2).sum(1) / state[:, 0]
            bad |= (state[:, 0] <= 0) | (ip <= 0)
    speeds = [(u - a).abs(), u.abs(), u.abs(), u.abs(), (u + a).abs()]
    diss = sum((A * s)[:, None] * e for A, s, e in zip((A0, A1, A2, A3, A4), speeds, E))
    f = 0.5 * (fl[:, :5] + fr[:, :5] - diss[:, back])
    f = _upwind_passive(f, L, R, nc)
    right, left = (u - a >= 0)[:, None], (u + a <= 0)[:, None]
    f = torch.where(bad[:, None], _hlle(L, R, d), f)
    return torch.where(right, fl, torch.where(left, fr, f))


_SOLVER = {"hllc": _hllc, "roe": _roe}


def _riemann(rs, L, R, d):
    f = _SOLVER[rs](L, R, d)
    if rs != "roe" and not f.requires_grad:
        f = torch.where(torch.isnan(f).any(1, keepdim=True), _hlle(L, R, d), f)
    return f


def _floor(u, emag=0.0):
    """Density and internal energy at or above zero, passive fields above it."""
    rho = u[:, 0:1].clamp(min=0.0)
    eint = u[:, 4:5] - 0.5 * (u[:, 1:4] ** 2).sum(1, keepdim=True) / rho - emag
    e = torch.where(eint < 0, u[:, 4:5] - eint, u[:, 4:5])
    return torch.cat([rho, u[:, 1:4], e, u[:, 5:]], 1)


def _planes(F):
    """The nine coarse-fine flux planes [n][9][v][16][16] of the fluxes of the 16^3 cells' faces."""
    return torch.stack([F[d].select(_dim(d), i) for d in range(3) for i in (0, 8, 16)], 1)


def _update(u, F, k):
    for d in range(3):
        u = u - k * (_cut(F[d], d, 1, PS) - _cut(F[d], d, 0, PS))
    return u


def _dual_fix(u):
    """Energy from the dual-energy field where the internal energy is a small part, else the reverse."""
    rho, kin = u[:, 0:1], 0.5 * (u[:, 1:4] ** 2).sum(1, keepdim=True) / u[:, 0:1]
    dual = u[:, 5:6].clamp(min=1.1754944e-38)
    eint = u[:, 4:5] - kin
    use = eint / kin < 2e-2
    fixed = torch.cat([u[:, :4], torch.where(use, kin + dual * rho ** GM1 / GM1, u[:, 4:5]),
                       torch.where(use, dual, (eint * GM1 * rho ** -GM1).clamp(min=1.1754944e-38))], 1)
    return torch.where((rho > 0) & (2.0 * u[:, 4:5] > kin), fixed, torch.cat([u[:, :5], dual], 1))


def _face_fluxes(rs, fc):
    """Fluxes of the faces of the inner 16^3 of 18^3 cells from their face states fc[2d], fc[2d+1]."""
    F = []
    for d in range(3):
        n, lo = [PS] * 3, [1] * 3
        n[d], lo[d] = PS + 1, 0
        F.append(_riemann(rs, _box(fc[2 * d + 1], lo, n), _box(fc[2 * d], _plus(lo, _e(d)), n), d))
    return F


def _mhm(u, k, lr, rs):
    """One MHM step of windows u; k = dt/dh per patch group.  Returns the 16^3 output and the fluxes."""
    ng = 2 if lr == "ppm" else 1
    trim = (u.shape[-1] - (PS + 2 + 2 * ng)) // 2
    u = _box(u, trim, PS + 2 + 2 * ng)
    w, fc, acc, bad = _prim(u), [], 0.0, False
    for d in range(3):
        for f in _faces(w, d, ng, PS + 2, lr):
            fc.append((_cons(f), f[:, 4:5]))
        acc = acc + _flux(*fc[-1], d) - _flux(*fc[-2], d)
    pres = [p for _, p in fc]
    fc = [c - 0.5 * k * acc for c, _ in fc]
    for c, p in zip(fc, pres):
        bad = bad | (c[:, 0:1] < 1.2e-38) | (c[:, 4:5] < 1.2e-38) | (p < 0)
    here = _box(u, ng, PS + 2)
    F = _face_fluxes(rs, [torch.where(bad, here, _floor(c)) for c in fc])
    out = _update(_box(u, ng + 1, PS), F, k)
    return (_dual_fix(out) if u.shape[1] == 6 else out), F


def _mhm_rp(u, k, lr, rs):
    F = []
    for d in range(3):
        n = [20] * 3
        n[d] = 21
        lo = _plus((1, 1, 1), _e(d, -1))
        F.append(_riemann(rs, _box(u, lo, n), _box(u, _plus(lo, _e(d)), n), d))
    half = _box(u, 1, 20)
    for d in range(3):
        half = half - 0.5 * k * (_cut(F[d], d, 1, 20) - _cut(F[d], d, 0, 20))
    w = _prim(_floor(half))
    F = _face_fluxes(rs, [_cons(f) for d in range(3) for f in _faces(w, d, 1, PS + 2, lr)])
    return _update(_box(u, 3, PS), F, k), F


def _jacobian(w, d, x):
    """A(w) x: the primitive-variable Jacobian along d (hydro, or MHD with 8 variables and the
    normal field fixed) applied to the variables x."""
    n, t1, t2 = 1 + d, 1 + (d + 1) % 3, 1 + (d + 2) % 3
    rho, vn = w[:, 0], w[:, n]
    y = vn[:, None] * x
    add = torch.zeros_like(y)
    add[:, 0] = rho * x[:, n]
    add[:, n] = x[:, 4] / rho
    add[:, 4] = GAMMA * w[:, 4] * x[:, n]
    if w.shape[1] == 8:
        bn, b1, b2 = 5 + d, 5 + (d + 1) % 3, 5 + (d + 2) % 3
        add[:, n] += (w[:, b1] * x[:, b1] + w[:, b2] * x[:, b2]) / rho
        add[:, t1] = -w[:, bn] * x[:, b1] / rho
        add[:, t2] = -w[:, bn] * x[:, b2] / rho
        add[:, b1] = w[:, b1] * x[:, n] - w[:, bn] * x[:, t1]
        add[:, b2] = w[:, b2] * x[:, n] - w[:, bn] * x[:, t2]
    return y + add


def _trace(c, fl, fr, d, k, lr):
    """Characteristic tracing over dt/2 with all waves: the sum over the waves of a linear (PLM) or
    quadratic (PPM) function of the eigenvalue is that function of the Jacobian."""
    h, df = 0.5 * k, fr - fl
    if c.shape[1] == 8:
        df = torch.cat([df[:, :5 + d], torch.zeros_like(df[:, :1]), df[:, 6 + d:]], 1)
    if lr == "plm":
        cor = -h * _jacobian(c, d, df)
        return fl + cor, fr + cor
    d6 = 6.0 * (c - 0.5 * (fl + fr))
    if c.shape[1] == 8:
        d6 = torch.cat([d6[:, :5 + d], torch.zeros_like(df[:, :1]), d6[:, 6 + d:]], 1)
    quad = -4.0 / 3.0 * h * h * _jacobian(c, d, _jacobian(c, d, d6))
    return fl - h * _jacobian(c, d, df + d6) + quad, fr - h * _jacobian(c, d, df - d6) + quad


def _ctu(u, k, lr, rs):
    ng, n = (2 if lr == "ppm" else 1), PS + 2
    w, fc, F = _prim(u), [], []
    c = _box(w, ng, n)
    for d in range(3):
        for f in _trace(c, *_faces(w, d, ng, n, lr), d, k, lr):
            fc.append(_cons(torch.cat([f[:, :4], f[:, 4:5].clamp(min=0.0)], 1)))
    for d in range(3):
        F.append(_riemann(rs, _cut(fc[2 * d + 1], d, 0, n - 1), _cut(fc[2 * d], d, 1, n - 1), d))
    for d in range(3):
        tg = 0.0
        for t in ((d + 1) % 3, (d + 2) % 3):
            # along t the 16 inner cells, along the other transverse axis the 16 inner ones, along d all
            o = 3 - d - t
            g = _cut(F[t], o, 1, PS)
            tg = tg + _cut(g, t, 1, PS) - _cut(g, t, 0, PS)
        for q in (2 * d, 2 * d + 1):
            lo, m = [1] * 3, [PS] * 3
            lo[d], m[d] = 0, n
            fc[q] = _floor(_box(fc[q], lo, m) - 0.5 * k * tg)
    F = [_riemann(rs, _cut(fc[2 * d + 1], d, 0, PS + 1), _cut(fc[2 * d], d, 1, PS + 1), d) for d in range(3)]
    return _update(_box(u, ng + 1, PS), F, k), F


# ---- MHD ------------------------------------------------------------------------------------------
def _minmod(a, b):
    return torch.where(a * b > 0, torch.sign(a) * torch.minimum(a.abs(), b.abs()), torch.zeros_like(a))


def _emag(b):
    return 0.5 * (b * b).sum(1, keepdim=True)


def _fast(a2, bn2, bt2):
    s = a2 + bn2 + bt2
    return torch.sqrt(0.5 * (s + torch.sqrt((bn2 + bt2 - a2) ** 2 + 4.0 * a2 * bt2)))


def _hlld(L, R, d):
    perm = [0, 1 + d, 1 + (d + 1) % 3, 1 + (d + 2) % 3, 4, 5 + d, 5 + (d + 1) % 3, 5 + (d + 2) % 3]
    back = [perm.index(i) for i in range(8)]
    side = []
    Bx = L[:, 5 + d]
    for U in (L, R):
        w = _prim(U[:, :5], _emag(U[:, 5:]))
        F = _flux(U, w[:, 4:5], d, U[:, 5:])[:, perm].unbind(1)
        u = U[:, perm].unbind(1)
        v = [w[:, perm[i]] for i in (1, 2, 3)]
        bt2 = u[6] ** 2 + u[7] ** 2
        side.append(dict(u=u, F=F, v=v, pt=w[:, 4] + 0.5 * (Bx * Bx + bt2),
                         c=_fast(GAMMA * w[:, 4] / u[0], Bx * Bx / u[0], bt2 / u[0])))
    l, r = side
    S0 = torch.minimum(l["v"][0] - l["c"], r["v"][0] - r["c"])
    S4 = torch.maximum(l["v"][0] + l["c"], r["v"][0] + r["c"])
    ml, mr = (S0 - l["v"][0]) * l["u"][0], (S4 - r["v"][0]) * r["u"][0]
    S2 = (mr * r["v"][0] - ml * l["v"][0] - r["pt"] + l["pt"]) / (mr - ml)
    pts = l["pt"] + ml * (S2 - l["v"][0])
    for q, S in ((l, S0), (r, S4)):
        u, v = q["u"], q["v"]
        sd, sm = S - v[0], S - S2
        rho = u[0] * sd / sm
        den = u[0] * sd * sm - Bx * Bx
        y, z = (v[i] - Bx * u[5 + i] * (sd - sm) / den for i in (1, 2))
        by, bz = (u[i] * (u[0] * sd * sd - Bx * Bx) / den for i in (6, 7))
        vb = S2 * Bx + y * by + z * bz
        e = (sd * u[4] - q["pt"] * v[0] + pts * S2 + Bx * (v[0] * Bx + v[1] * u[6] + v[2] * u[7] - vb)) / sm
        q.update(s=[rho, rho * S2, rho * y, rho * z, e, Bx, by, bz], y=y, z=z, vb=vb, sq=torch.sqrt(rho))
    S1, S3 = S2 - Bx.abs() / l["sq"], S2 + Bx.abs() / r["sq"]
    sg = torch.where(Bx < 0, -1.0, 1.0).to(Bx.dtype)
    a, b = l["sq"], r["sq"]
    y = (a * l["y"] + b * r["y"] + sg * (r["s"][6] - l["s"][6])) / (a + b)
    z = (a * l["z"] + b * r["z"] + sg * (r["s"][7] - l["s"][7])) / (a + b)
    by = (a * r["s"][6] + b * l["s"][6] + sg * a * b * (r["y"] - l["y"])) / (a + b)
    bz = (a * r["s"][7] + b * l["s"][7] + sg * a * b * (r["z"] - l["z"])) / (a + b)
    vb = S2 * Bx + y * by + z * bz
    for q, s in ((l, -1.0), (r, 1.0)):
        rho = q["s"][0]
        q["d"] = [rho, q["s"][1], rho * y, rho * z, q["s"][4] + s * q["sq"] * sg * (q["vb"] - vb), Bx, by, bz]
    f = []
    for i in range(8):
        fl = l["F"][i] + S0 * (l["s"][i] - l["u"][i])
        fr = r["F"][i] + S4 * (r["s"][i] - r["u"][i])
        g = torch.where(S2 >= 0, torch.where(S1 >= 0, fl, fl + S1 * (l["d"][i] - l["s"][i])),
                        torch.where(S3 > 0, fr + S3 * (r["d"][i] - r["s"][i]), fr))
        f.append(torch.where(S0 >= 0, l["F"][i], torch.where(S4 <= 0, r["F"][i], g)))
    f[5] = torch.zeros_like(f[5])
    return torch.stack(f, 1)[:, back]


def _pad(F, d):
    """One unused layer at the upper end of axis d, so that the fluxes of all directions have one shape."""
    pad = [0] * 6
    pad[2 * d + 1] = 1
    return nnf.pad(F, pad)


def _emf(F, w, d, off):
    """E_d on the edges of the cells of the padded fluxes F (face above cell i at i): the mean of the
    four face values and of the four upwinded derivatives; w: cell primitives, cell (0,0,0) at off."""
    T1, T2 = (d + 1) % 3, (d + 2) % 3
    m = F[0].shape[-1]
    n = [m - 1] * 3
    n[d] = m - 2
    at = lambda a, *s: _box(a, [int(i == d) + sum(int(i == t) for t in s) for i in range(3)], n)  # noqa: E731
    wc = [_box(w, [off + int(i == d) + (a if i == T1 else b if i == T2 else 0) for i in range(3)], n)
          for a, b in ((0, 0), (1, 0), (0, 1), (1, 1))]
    cell = [c[:, 5 + T1] * c[:, 1 + T2] - c[:, 5 + T2] * c[:, 1 + T1] for c in wc]   # 00, 10, 01, 11
    e1 = [-at(F[T1], *s)[:, 5 + T2] for s in ((), (T2,))]
    e2 = [at(F[T2], *s)[:, 5 + T1] for s in ((), (T1,))]
    m1 = [at(F[T1], *s)[:, 0] for s in ((), (T2,))]
    m2 = [at(F[T2], *s)[:, 0] for s in ((), (T1,))]

    def up(mass, lo, hi, cl, ch):
        return torch.where(mass > 0, lo - cl, torch.where(mass < 0, hi - ch, 0.5 * (lo - cl + hi - ch)))

    e = e1[0] + e1[1] + e2[0] + e2[1]
    e = e + up(m2[0], e1[0], e1[1], cell[0], cell[2]) + up(m2[1], e1[0], e1[1], cell[1], cell[3])
    e = e + up(m1[0], e2[0], e2[1], cell[0], cell[1]) + up(m1[1], e2[0], e2[1], cell[2], cell[3])
    return 0.25 * e


def _curl(E, b, k, d):
    """b_d advanced over k by the edge EMFs around each face."""
    T1, T2 = (d + 1) % 3, (d + 2) % 3
    diff = lambda a, t: _cut(a, t, 1, a.shape[_dim(t)] - 1) - _cut(a, t, 0, a.shape[_dim(t)] - 1)  # noqa: E731
    return b + k * (diff(E[T1], T2) - diff(E[T2], T1))


def _ctu_mhd(u, b, k, lr):
    """One CTU+MHD step: u [n][5][N^3], b the three face fields [n][..]; k = dt/dh per patch group."""
    N = u.shape[-1]
    g = (N - 20) // 2                            # input cells left of face-state cell 0 of 20
    bcc = torch.stack([0.5 * (_cut(b[d], d, 0, N) + _cut(b[d], d, 1, N)) for d in range(3)], 1)
    w = torch.cat([_prim(u, _emag(bcc)), bcc], 1)
    c = _box(w, g, 20)
    bl = [_box(b[d], g, 20) for d in range(3)]
    br = [_box(b[d], _plus((g,) * 3, _e(d)), 20) for d in range(3)]
    db = [(y - x)[:, None] for x, y in zip(bl, br)]
    k4 = k[:, 0]
    fc = []
    for d in range(3):
        T1, T2 = (d + 1) % 3, (d + 2) % 3
        for f, bn in zip(_trace(c, *_faces(w, d, g, 20, lr), d, k, lr), (bl[d], br[d])):
            f = f.clone()
            f[:, 5 + T1] += (0.5 * k * c[:, 1 + T1:2 + T1] * _minmod(db[d], -db[T1]))[:, 0]
            f[:, 5 + T2] += (0.5 * k * c[:, 1 + T2:2 + T2] * _minmod(db[d], -db[T2]))[:, 0]
            f[:, 5 + d] = bn
            f[:, 4].clamp_(min=0.0)
            fc.append(_cons(f, _emag(f[:, 5:])))
    F = [_pad(_hlld(_cut(fc[2 * d + 1], d, 0, 19), _cut(fc[2 * d], d, 1, 19), d), d) for d in range(3)]
    E = [_emf(F, w, d, g) for d in range(3)]      # 19 edges across, 18 along
    bh = []
    for d in range(3):
        n = [18] * 3
        n[d] = 19
        bh.append(_curl(E, _box(b[d], g + 1, n), 0.5 * k4, d))
    dif = [_box(F[d], 1, 18) - _box(F[d], _plus((1, 1, 1), _e(d, -1)), 18) for d in range(3)]
    ci = _box(c, 1, 18)
    dbi = [_box(x, 1, 18) for x in db]
    full = []
    for d in range(3):
        T1, T2 = (d + 1) % 3, (d + 2) % 3
        m1 = ci[:, 1 + T1:2 + T1] * _minmod(-dbi[T2], dbi[d])
        m2 = ci[:, 1 + T2:2 + T2] * _minmod(-dbi[T1], dbi[d])
        for q, face in ((2 * d, 0), (2 * d + 1, 1)):
            x = _box(fc[q], 1, 18).clone()
            x[:, :5] -= 0.5 * k * (dif[T1] + dif[T2])[:, :5]
            Ed = E[d]
            dz = _cut(Ed, T2, 1, 18) - _cut(Ed, T2, 0, 18)       # along T2, on the 19 edges along T1
            dy = _cut(Ed, T1, 1, 18) - _cut(Ed, T1, 0, 18)
            x[:, 5 + T1] -= 0.25 * k4 * (_cut(dz, T1, 0, 18) + _cut(dz, T1, 1, 18))
            x[:, 5 + T2] += 0.25 * k4 * (_cut(dy, T2, 0, 18) + _cut(dy, T2, 1, 18))
            h = 0.5 * k * dbi[d]
            x[:, 1:4] += h * torch.stack([ci[:, 5 + i] for i in range(3)], 1)
            x[:, 4] += (0.5 * k * (ci[:, 5 + T1:6 + T1] * m1 + ci[:, 5 + T2:6 + T2] * m2))[:, 0]
            x[:, 5 + T1] += (0.5 * k * m1)[:, 0]
            x[:, 5 + T2] += (0.5 * k * m2)[:, 0]
            x[:, 5 + d] = _cut(bh[d], d, face, 18)
            full.append(torch.cat([_floor(x[:, :5], _emag(x[:, 5:])), x[:, 5:]], 1))
    half = _box(u, g + 1, 18)[:, :4] - 0.5 * k * (dif[0] + dif[1] + dif[2])[:, :4]
    bhc = torch.stack([0.5 * (_cut(bh[d], d, 0, 18) + _cut(bh[d], d, 1, 18)) for d in range(3)], 1)
    wh = torch.cat([half[:, :1], half[:, 1:] / half[:, :1], half[:, :1], bhc], 1)
    G = [_pad(_hlld(_cut(full[2 * d + 1], d, 0, 17), _cut(full[2 * d], d, 1, 17), d), d) for d in range(3)]
    E = [_emf(G, wh, d, 0) for d in range(3)]     # 17 edges across, 16 along
    bo = []
    for d in range(3):
        n = [PS] * 3
        n[d] = PS + 1
        bo.append(_curl(E, _box(b[d], g + 2, n), k4, d))
    inner = []
    for d in range(3):
        n = [PS] * 3
        n[d] = PS + 1
        inner.append(_box(G[d], [0 if i == d else 1 for i in range(3)], n)[:, :5])
    out = _update(_box(u, g + 2, PS), inner, k)
    # the EMFs on the nine planes: [plane][first / second transverse component][17 x 16]
    ele = [None] * 18
    for p in range(3):
        ele[2 * (3 + p) + 1] = E[0].select(-2, 8 * p).transpose(-1, -2)          # [x][z]
        ele[2 * (6 + p) + 0] = E[0].select(-3, 8 * p)                            # [y][x]
        ele[2 * (6 + p) + 1] = E[1].select(-3, 8 * p)                            # [y][x]
        ele[2 * p + 0] = E[1].select(-1, 8 * p)                                  # [z][y]
        ele[2 * p + 1] = E[2].select(-1, 8 * p)                                  # [z][y]
        ele[2 * (3 + p) + 0] = E[2].select(-2, 8 * p).transpose(-1, -2)          # [x][z]
    n = u.shape[0]
    return (out, _planes(inner), torch.stack([x.reshape(n, -1) for x in bo], 1),
            torch.stack([e.reshape(n, -1) for e in ele], 1).reshape(n, 9, 2, -1))


# ---- the ghost-zone fill ----------------------------------------------------------------------------
def _cquad(c, d):
    """Conservative quadratic interpolation along d (monotonicity coefficient 2): the cells between
    the first and the last, in pairs."""
    n = c.shape[_dim(d)] - 2
    l, m, r = (_cut(c, d, i, n) for i in range(3))
    s, a, b = 0.125 * (r - l), 0.25 * (m - l), 0.25 * (r - m)
    lim = torch.where(a.abs() < b.abs(), torch.minimum(2.0 * a.abs(), b.abs()), torch.minimum(a.abs(), 2.0 * b.abs()))
    s = torch.where(a * b > 0, torch.sign(a) * torch.minimum(s * torch.sign(a), lim), torch.zeros_like(s))
    both = torch.stack([m - s, m + s], _dim(d))
    return both.flatten(both.dim() + _dim(d) - 1, both.dim() + _dim(d))


def _physical(u):
    return ((u[:, 0] > 0) & (u[:, 4] - 0.5 * (u[:, 1:4] ** 2).sum(1) / u[:, 0] > -1e-12))[:, None]


def _interpolate(c):
    """Conserved first; the parents with an unphysical child again in primitive variables."""
    f = _cquad(_cquad(_cquad(c, 0), 1), 2)
    w = _cons(_cquad(_cquad(_cquad(_prim(c), 0), 1), 2))
    ok = _physical(f).to(f.dtype)
    ok = -nnf.max_pool3d(-ok, 2)
    return torch.where(nnf.interpolate(ok, scale_factor=2) > 0.5, f, w)


def _assemble(fine, nbr, cint):
    n, nxt = fine.shape[0], cint.shape[-1]
    g = (nxt - PS) // 2
    win = cint.clone()
    for s in range(27):
        off = (s % 3 - 1, s // 3 % 3 - 1, s // 9 - 1)
        lo = [0 if o < 0 else g if o == 0 else g + PS for o in off]
        m = [PS if o == 0 else g for o in off]
        src = [lo[i] - g - PS * off[i] for i in range(3)]
        from_p = torch.arange(n, device=DEV) if s == 13 else nbr[:, s].long()
        has = from_p >= 0
        part = _box(fine[from_p.clamp(min=0)], src, m)
        dst = _box(win, lo, m)
        dst.copy_(torch.where(has[:, None, None, None, None], part, dst))
    return win


# ---- the close ----------------------------------------------------------------------------------------
def _first_order(win, k):
    """Every cell of the windows' interiors advanced with first-order HLLE fluxes, and the fluxes."""
    F = []
    for d in range(3):
        n = [PS] * 3
        n[d] = PS + 1
        lo = [2] * 3
        lo[d] = 1
        F.append(_hlle(_box(win, lo, n), _box(win, _plus(lo, _e(d)), n), d))
    return _floor(_update(_box(win, 2, PS), F, k)), _planes(F)


def _fixup(u, flux, has, dh):
    u = u.clone()
    for s in range(6):
        d, up = s // 2, s % 2
        f = flux[:, s] * ((1.0 if up else -1.0) / dh)
        old = u.select(_dim(d), 7 if up else 0)
        new = old + f
        eint = new[:, 4] - 0.5 * (new[:, 1:4] ** 2).sum(1) / new[:, 0]
        ok = (new[:, 0] > 0) & (eint > 0) & (has[:, s, None, None] != 0)
        old.copy_(torch.where(ok[:, None], new, old))
    return u


_LOCAL = ((0, 0, 0), (1, 0, 0), (0, 1, 0), (0, 0, 1), (1, 1, 0), (0, 1, 1), (1, 0, 1), (1, 1, 1))


def _dt(out, dh):
    w = _prim(out)
    s = (w[:, 1:4].abs() + torch.sqrt(GAMMA * w[:, 4:5] / w[:, 0:1])).amax(1)
    s = torch.stack([s[:, 8 * z:8 * z + 8, 8 * y:8 * y + 8, 8 * x:8 * x + 8].amax((1, 2, 3)) for x, y, z in _LOCAL], 1)
    return (0.5 * dh / s).reshape(-1)


def _chunks(n):
    return ((a, min(n, a + CHUNK)) for a in range(0, n, CHUNK))


def _gather(parts):
    return [torch.cat(p) for p in zip(*parts)]


def exact(case, seed):
    kind = case["kind"]
    if kind in ("solve", "host"):
        x, dt, dh = _hydro(case, seed, case["nxt"] if kind == "host" else _nxt(case["scheme"], case["lr"]))
        step = {"mhm": _mhm, "mhm_rp": _mhm_rp, "ctu": _ctu}[case.get("scheme", "mhm")]
        parts = []
        for a, b in _chunks(x.shape[0]):
            out, F = step(x[a:b].double(), dt / dh, case.get("lr", "plm"), case.get("rs", "hllc"))
            parts.append((out, _planes(F)))
        out, flux = _gather(parts)
        return dict(out=out, flux=flux, de=None) if kind == "solve" else dict(out=out, flux=flux)
    if kind == "levels":
        x, npg, dts, dhs = _levels(case, seed)
        k = torch.cat([torch.full((n,), dt / dh, dtype=torch.float64, device=DEV) for n, dt, dh in zip(npg, dts, dhs)])
        parts = []
        for a, b in _chunks(x.shape[0]):
            out, F = _mhm(x[a:b].double(), k[a:b, None, None, None, None], "plm", "hllc")
            parts.append((out, _planes(F)))
        out, flux = _gather(parts)
        return dict(out=out, flux=flux, de=None)
    if kind == "mhd":
        nxt = 24 if case["lr"] == "ppm" else 22
        x, mag, dt, dh = _magnetised(case, seed, nxt)
        parts = []
        for a, b in _chunks(x.shape[0]):
            m, n = mag[a:b].double(), b - a
            faces = [m[:, d].reshape([n] + [nxt + int(i == d) for i in (2, 1, 0)]) for d in range(3)]
            k = torch.full((n, 1, 1, 1, 1), dt / dh, dtype=torch.float64, device=DEV)
            parts.append(_ctu_mhd(x[a:b].double(), faces, k, case["lr"]))
        out, flux, bo, ele = _gather(parts)
        return dict(out=out, flux=flux, mag=bo, ele=ele)
    if kind == "ghost":
        c, fine, nbr = _ghost(case, seed)
        cint = torch.cat([_interpolate(c[a:b].double()) for a, b in _chunks(c.shape[0])])
        return dict(cint=cint, win=_assemble(fine.double(), nbr, cint), status=None)
    if kind == "close":
        win, out, bad, flux, patch, diff, has, dt, dh = _close(case, seed)
        parts = []
        for a, b in _chunks(win.shape[0]):
            new, planes = _first_order(win[a:b].double(), dt / dh)
            o = torch.where(bad[a:b, None], new, out[a:b].double())
            near = []
            for d in range(3):
                q = [bad[a:b].select(_dim(d), i) for i in (0, 7, 8, 15)]
                near += [q[0], q[1] | q[2], q[3]]
            f = torch.where(torch.stack(near, 1)[:, :, None], planes, flux[a:b].double())
            parts.append((o, f, _dt(o, dh)))
        o, f, dts = _gather(parts)
        return dict(out=o, flux=f, patch=_fixup(patch.double(), diff.double(), has, dh), dt=dts, counts=None)
    return _exact_adjoint(case, seed)


def _exact_adjoint(case, seed):
    box, w, dt, dh = _adjoint_box(case, seed)
    boxes = [box.double()]
    pz, py, px = case["pz"], case["py"], case["px"]
    npg = pz * py * px

    def back(out):
        out = out.reshape(pz, py, px, 5, PS, PS, PS).permute(3, 0, 4, 1, 5, 2, 6)
        return out.reshape(5, pz * PS, py * PS, px * PS)

    for _ in range(case["K"]):
        win = _windows(boxes[-1], 20)
        boxes.append(back(torch.cat([_mhm(win[a:b], dt / dh, "plm", "hllc")[0] for a, b in _chunks(npg)])))
    grad = torch.zeros_like(boxes[0])
    grad[0] = w
    for k in reversed(range(case["K"])):
        box_k = boxes[k].detach().requires_grad_(True)
        win = _windows(box_k, 20)
        gout = _windows(grad, PS)
        leaf = win.detach()
        gwin = torch.empty_like(leaf)
        for a, b in _chunks(npg):
            x = leaf[a:b].clone().requires_grad_(True)
            out, _ = _mhm(x, dt / dh, "plm", "hllc")
            gwin[a:b] = torch.autograd.grad(out, x, gout[a:b])[0]
        grad = torch.autograd.grad(win, box_k, gwin)[0]
    return dict(box=boxes[-1], grad=grad)
