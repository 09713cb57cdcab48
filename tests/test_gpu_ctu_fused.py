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


@pytest.mark.parametrize("npg", [240, 301, 600])
@pytest.mark.parametrize("prec,lr,rs,kw", [
    ("fp32", "plm", "hllc", {}), ("fp32", "plm", "hllc", dict(LR_Limiter="vanleer")),
    ("fp32", "plm", "hllc", dict(MinDens=1.0, MinPres=0.9, MinEint=1.4)), ("mixed", "plm", "hllc", {}),
    ("fp32", "ppm", "hllc", {}), ("fp32", "ppm", "hllc", dict(LR_Limiter="central")), ("mixed", "ppm", "hllc", {}),
    ("fp32", "plm", "roe", {}), ("fp32", "plm", "hlle", {}), ("fp32", "ppm", "hlle", {}),
    ("fp64", "plm", "hllc", {}), ("fp64", "plm", "roe", {}), ("fp64", "plm", "hlle", dict(LR_Limiter="albada")),
])
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
    a, _ = _solve(s, x, SolverParams(dt=dt, dh=dh), 125)
    b, f = _solve(s, x, SolverParams(dt=dt, dh=dh, StoreFlux=False), 125)
    assert torch.equal(a, b) and bool(torch.isnan(f).all())


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
    out, flux = _solve(s, torch.from_numpy(x).cuda(), prm, npg)
    if chunk:
        s.set_mhd_chunk(chunk)
    hout, hflux, _ = s.solve_host(x, prm)
    assert np.array_equal(hout, out.cpu().numpy()) and np.array_equal(hflux, flux.cpu().numpy())
