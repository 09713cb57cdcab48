"""The plane-streaming hydro CTU kernel against the separate kernels (ctu_hydro.cu), which take the
same patch groups in calls too small for it; both against each other in every policy, reconstruction
and solver that the streaming kernel is built for."""
import numpy as np
import pytest

from gamer_b200 import ic
from gamer_b200.fluid import FluidSolver, SolverParams

pytestmark = pytest.mark.gpu
GAMMA = 5.0 / 3.0


def _solve(s, x, prm, part):
    """Solve in calls of at most ``part`` patch groups."""
    import torch
    n = x.shape[0]
    out = torch.full((n, 5, 16, 16, 16), float("nan"), dtype=x.dtype, device="cuda")
    flux = torch.full((n, 9, 5, 16, 16), float("nan"), dtype=x.dtype, device="cuda")
    for a in range(0, n, part):
        b = min(n, a + part)
        s.solve_device(x[a:b], out[a:b], prm, flux=flux[a:b] if prm.StoreFlux else None)
    torch.cuda.synchronize()
    assert s.status() == 0
    return out, flux


# sizes that take the streaming kernel: the line, a CTA with one, two and (one CTA per SM) up to five
# patch groups, a partly filled last wave
@pytest.mark.parametrize("prec,lr,rs,kw,npg", [(p, l, r, k, n) for p, l, r, k, sizes in [
    ("fp32", "plm", "hllc", {}, (100, 301, 600)), ("fp32", "plm", "hllc", dict(LR_Limiter="vanleer"), (155, 590)),
    ("fp32", "plm", "hllc", dict(MinDens=1.0, MinPres=0.9, MinEint=1.4), (301, 600)), ("fp32", "plm", "hlle", {}, (100, 301, 600)),
    ("fp32", "plm", "hlle", dict(LR_Limiter="albada"), (310,)),
    ("mixed", "plm", "hllc", {}, (245, 580)), ("mixed", "plm", "hlle", dict(MinDens=1.0, MinPres=0.9, MinEint=1.4), (580, 888)),
    ("fp32", "ppm", "hllc", {}, (105, 240, 600)), ("fp32", "ppm", "hllc", dict(LR_Limiter="central"), (290, 580)),
    ("fp32", "ppm", "hlle", {}, (120, 240, 600)),
    ("fp64", "plm", "hllc", {}, (100, 240, 301, 600)), ("fp64", "plm", "hlle", {}, (240,)), ("fp64", "plm", "hlle", dict(LR_Limiter="albada"), (290, 580)),
    ("fp64", "plm", "hllc", dict(LR_Limiter="vl_gminmod"), (148,)),
] for n in sizes])
def test_streaming_kernel_equals_separate_kernels(cuda_device, npg, prec, lr, rs, kw):
    import torch
    p = 7 if npg > 343 else 5
    box = ic.lognormal_box(p, seed=npg, gamma=GAMMA)
    dh = 1.0 / (16 * p)
    dt = ic.cfl_dt(box, GAMMA, dh, cfl=0.4)
    s = FluidSolver(scheme="ctu", lr=lr, rsolver=rs, precision=prec, gamma=GAMMA)
    x = ic.cut_patch_groups(box, s.flu_nxt).astype(s.np_dtype)
    x = torch.from_numpy(np.concatenate([x] * (-(-npg // x.shape[0])))[:npg]).cuda()
    prm = SolverParams(dt=dt, dh=dh, **kw)
    assert s.ctu_one_kernel(npg, prm) and not s.ctu_one_kernel(16, prm)
    out, flux = _solve(s, x, prm, npg)
    ref, rflux = _solve(s, x, prm, 16)
    # both are the same scheme with sums in another order: a few rounding errors of the largest term,
    # scaled by the variable's rms, and a bounded share of cells that take another limiter or
    # upwind branch
    eps = 2.0 ** -52 if prec == "fp64" else 2.0 ** -23
    for g, r in ((out, ref), (flux, rflux)):
        g, r = g.double(), r.double()
        assert bool(torch.isfinite(g).all()) and bool(torch.isfinite(r).all())
        v = 1 if g.dim() == 5 and g.shape[1] == 5 else 2
        rms = (r * r).mean(dim=[d for d in range(g.dim()) if d != v], keepdim=True).sqrt()
        err = (g - r).abs() / (r.abs() + rms)
        assert float((err > 64 * eps).double().mean()) < 1e-3
        assert float(err.max()) < 4e4 * eps


def test_streaming_kernel_without_flux_planes(cuda_device):
    """StoreFlux off: the same outputs, nothing written to the flux array."""
    import torch
    box = ic.lognormal_box(5, seed=3, gamma=GAMMA)
    dh = 1.0 / 80
    dt = ic.cfl_dt(box, GAMMA, dh, cfl=0.4)
    s = FluidSolver(scheme="ctu", precision="fp32", gamma=GAMMA)
    x = torch.from_numpy(ic.cut_patch_groups(box, 20).astype(np.float32)).cuda()
    assert s.ctu_one_kernel(125, SolverParams(dt=dt, dh=dh))
    a, _ = _solve(s, x, SolverParams(dt=dt, dh=dh), 125)
    b, f = _solve(s, x, SolverParams(dt=dt, dh=dh, StoreFlux=False), 125)
    assert torch.equal(a, b) and bool(torch.isnan(f).all())


@pytest.mark.parametrize("prec,lr,rs", [("fp32", "plm", "hllc"), ("mixed", "plm", "hllc"), ("fp32", "ppm", "hllc"), ("fp64", "plm", "hllc"),
                                        ("fp32", "plm", "hlle")])
def test_streaming_kernel_rescues_faces_without_pressure(cuda_device, prec, lr, rs):
    """Streams without pressure along x, y and z in some patch groups: the HLLC flux of their
    faces is 0/0 and the HLLE flux stands in, in half and full step, for the x and the y lane of the packed
    solver each on its own.  Same as the separate kernels, whose solver is scalar."""
    import torch
    npg = 580
    box = ic.lognormal_box(5, seed=7, gamma=GAMMA)
    dh = 1.0 / 80
    s = FluidSolver(scheme="ctu", lr=lr, rsolver=rs, precision=prec, gamma=GAMMA)
    x = ic.cut_patch_groups(box, s.flu_nxt).astype(s.np_dtype)
    x = np.concatenate([x] * (-(-npg // x.shape[0])))[:npg]
    cold = range(0, npg, 5)
    for p in cold:
        d = (p // 5) % 3                                    # the streams' direction: x, y, z
        u = np.zeros((5, 10, 10, 10))
        u[0] = 1.0
        half = [slice(None)] * 3
        u[1 + d] = 1.0
        half[2 - d] = slice(5, 10)
        u[(1 + d,) + tuple(half)] = 2.0
        u[4] = 0.5 * u[1 + d] ** 2
        x[p, :, 6:16, 6:16, 6:16] = u
    prm = SolverParams(dt=ic.cfl_dt(box, GAMMA, dh, cfl=0.2), dh=dh)
    assert s.ctu_one_kernel(npg, prm)
    t = torch.from_numpy(x).cuda()
    out, flux = _solve(s, t, prm, npg)
    ref, rflux = _solve(s, t, prm, 16)
    eps = 2.0 ** -52 if prec == "fp64" else 2.0 ** -23
    for g, r in ((out, ref), (flux, rflux)):
        g, r = g.double(), r.double()
        fin = torch.isfinite(r)
        assert torch.equal(fin, torch.isfinite(g))
        assert bool(fin[list(cold)].any())
        v = 1 if g.dim() == 5 and g.shape[1] == 5 else 2
        g, r = torch.where(fin, g, 0.0), torch.where(fin, r, 0.0)
        rms = (r * r).mean(dim=[d for d in range(g.dim()) if d != v], keepdim=True).sqrt()
        err = (g - r).abs() / (r.abs() + rms)
        # as above; the edges of the streams are jumps, where more cells switch branches
        assert float((err > 64 * eps).double().mean()) < 2e-3
        assert float(err.max()) < 4e4 * eps


@pytest.mark.parametrize("prec,npg,chunk", [("fp32", 560, 0), ("fp32", 560, 100), ("fp32", 60, 7), ("mixed", 600, 0), ("fp64", 520, 0)])
def test_host_calls_equal_device_calls_whatever_the_chunks(cuda_device, prec, npg, chunk):
    """The kernel is chosen once for a call: neither the chunks of the host-array entry point (512, or
    fewer) nor a last, small chunk give other bits than the same call on device arrays."""
    import torch
    box = ic.lognormal_box(4, seed=npg, gamma=GAMMA)
    dh = 1.0 / 64
    s = FluidSolver(scheme="ctu", precision=prec, gamma=GAMMA)
    x = ic.cut_patch_groups(box, 20).astype(s.np_dtype)
    x = np.concatenate([x] * (-(-npg // x.shape[0])))[:npg]
    prm = SolverParams(dt=ic.cfl_dt(box, GAMMA, dh, cfl=0.4), dh=dh)
    assert s.ctu_one_kernel(npg, prm) == (npg == 560 or prec == "fp64")
    out, flux = _solve(s, torch.from_numpy(x).cuda(), prm, npg)
    if chunk:
        s.set_mhd_chunk(chunk)
    hout, hflux, _ = s.solve_host(x, prm)
    assert np.array_equal(hout, out.cpu().numpy()) and np.array_equal(hflux, flux.cpu().numpy())
