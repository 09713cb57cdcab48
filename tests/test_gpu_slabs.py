"""Patch groups solved in slabs along z (the last, partly filled wave of a call) equal the same patch
groups solved whole, bit for bit: a call that reports failed patch groups keeps them whole."""
import numpy as np
import pytest

from gamer_b200 import ic
from gamer_b200.fluid import FluidSolver, SolverParams

pytestmark = pytest.mark.gpu
GAMMA = 5.0 / 3.0


def _windows(npg, nxt, dtype, dual=False):
    box = ic.lognormal_box(4, seed=npg + nxt, gamma=GAMMA, dual=dual)
    x = ic.cut_patch_groups(box, nxt).astype(dtype)
    dh = 1.0 / 64
    return np.concatenate([x] * (-(-npg // x.shape[0])))[:npg], ic.cfl_dt(box, GAMMA, dh, cfl=0.4), dh


@pytest.mark.parametrize("npg", [1, 3, 8, 37, 64, 148, 297, 350])
@pytest.mark.parametrize("kw,nxt", [
    (dict(precision="fp32"), 20), (dict(precision="fp32", rsolver="roe"), 22), (dict(precision="mixed", lr="ppm", rsolver="roe"), 22),
    (dict(precision="fp64"), 20), (dict(precision="fp64", lr="ppm"), 24), (dict(precision="fp32", dual_energy=True), 20),
    (dict(scheme="mhm_rp", precision="mixed"), 22), (dict(scheme="mhm_rp", precision="fp64"), 22)])
def test_slabs_equal_whole_patch_groups(cuda_device, npg, kw, nxt):
    import torch
    s = FluidSolver(gamma=GAMMA, flu_nxt=nxt, **kw)
    x, dt, dh = _windows(npg, nxt, s.np_dtype, s.dual)
    t = torch.from_numpy(x).cuda()
    prm = SolverParams(dt=dt, dh=dh)
    got = []
    for report in (True, False):
        out = torch.full((npg, s.ncomp, 16, 16, 16), float("nan"), dtype=t.dtype, device="cuda")
        flux = torch.full((npg, 9, s.ncomp, 16, 16), float("nan"), dtype=t.dtype, device="cuda")
        de = torch.full((npg, 16, 16, 16), 48, dtype=torch.int8, device="cuda") if s.dual else None
        fail = torch.full((npg,), 7, dtype=torch.int32, device="cuda") if report else None
        s.solve_device(t, out, prm, flux=flux, de_out=de, pg_fail=fail)
        torch.cuda.synchronize()
        assert s.status() == 0
        assert fail is None or not bool(fail.any())
        got.append((out, flux, de))
    for a, b in zip(*got):
        assert a is None or torch.equal(a, b)
    assert bool(torch.isfinite(got[0][0]).all()) and bool(torch.isfinite(got[0][1]).all())


@pytest.mark.parametrize("npg", [5, 300])
def test_unphysical_cells_are_reported_from_slabs(cuda_device, npg):
    """A patch group with a cell that ends up unphysical sets the status bit, whole or in slabs."""
    import torch
    s = FluidSolver(gamma=GAMMA, precision="fp32")
    x, dt, dh = _windows(npg, 20, np.float32)
    x[npg - 1, 4, 15, 9, 9] = 1.0e-3 * x[npg - 1, 4, 15, 9, 9]          # total energy below the kinetic one
    t = torch.from_numpy(x).cuda()
    out = torch.empty((npg, 5, 16, 16, 16), dtype=t.dtype, device="cuda")
    fail = torch.zeros(npg, dtype=torch.int32, device="cuda")
    s.solve_device(t, out, SolverParams(dt=dt, dh=dh, StoreFlux=False), pg_fail=fail)
    torch.cuda.synchronize()
    whole = s.status()
    s.solve_device(t, out, SolverParams(dt=dt, dh=dh, StoreFlux=False))
    torch.cuda.synchronize()
    assert s.status() == whole and (whole != 0) == bool(fail.any())


@pytest.mark.parametrize("lr,nxt", [("plm", 22), ("ppm", 24)])
@pytest.mark.parametrize("prec", ["fp32", "mixed"])
@pytest.mark.parametrize("npg", [1, 9, 148, 333])
def test_mhm_rp_float_half_step_against_fp64(cuda_device, lr, nxt, prec, npg):
    """The float half step with per-cell pressures and sound speeds against the FP64 solver (another
    kernel) on the same float-rounded input."""
    import torch
    x, dt, dh = _windows(npg, nxt, np.float32)
    got = []
    for p in (prec, "fp64"):
        s = FluidSolver(scheme="mhm_rp", lr=lr, precision=p, gamma=GAMMA)
        t = torch.from_numpy(x.astype(s.np_dtype)).cuda()
        out = torch.full((npg, 5, 16, 16, 16), float("nan"), dtype=t.dtype, device="cuda")
        flux = torch.full((npg, 9, 5, 16, 16), float("nan"), dtype=t.dtype, device="cuda")
        s.solve_device(t, out, SolverParams(dt=dt, dh=dh), flux=flux)
        torch.cuda.synchronize()
        assert s.status() == 0
        got.append((out.double(), flux.double()))
    for g, r in zip(*got):
        v = 1 if g.dim() == 5 and g.shape[1] == 5 else 2
        rms = (r * r).mean(dim=[d for d in range(g.dim()) if d != v], keepdim=True).sqrt()
        # float rounding of a two-step scheme (a few dozen operations on each path), and the share of
        # cells that take another limiter branch
        err = (g - r).abs() / (r.abs() + rms)
        assert float((err > 64 * 2.0 ** -23).double().mean()) < 1e-3
        assert float(err.max()) < 5e-3


@pytest.mark.parametrize("prec,npg,offset", [("fp32", 1, 0), ("fp32", 19, 0), ("fp32", 296, 0), ("fp32", 301, 0), ("fp32", 369, 0), ("fp32", 370, 0), ("fp32", 391, 0), ("fp32", 400, 1),
                                             ("mixed", 297, 0), ("mixed", 888, 0), ("mixed", 901, 0), ("fp64", 296, 0), ("fp64", 299, 1)])
def test_dt_of_solver_outputs_equals_dt_of_patches(cuda_device, prec, npg, offset):
    """One CTA per patch group (outputs, 16-byte aligned) against one per patch (patch arrays)."""
    import torch
    s = FluidSolver(precision=prec, gamma=GAMMA)
    x, _, dh = _windows(npg, 16, s.np_dtype)
    flat = torch.zeros(x.size + offset, dtype=s.torch_dtype, device="cuda")
    flat[offset:] = torch.from_numpy(x.reshape(-1)).cuda()
    got = s.dt_cfl(flat[offset:].view(x.shape), dh, from_output=True)
    flu, _ = ic.patches_from_output(x)
    ref = s.dt_cfl(torch.from_numpy(np.ascontiguousarray(flu)).cuda(), dh)
    torch.cuda.synchronize()
    assert torch.equal(got, ref)


@pytest.mark.parametrize("prec,npg", [("fp32", 300), ("fp32", 420), ("mixed", 300), ("mixed", 600), ("mixed", 900)])
def test_dt_of_an_aligned_array_is_not_slower(cuda_device, prec, npg):
    """The kernel with 16-byte loads is used where it gains: an array that allows them takes no longer
    than one off the boundary, which is read patch by patch."""
    import torch
    s = FluidSolver(precision=prec, gamma=GAMMA)
    x, _, dh = _windows(npg, 16, s.np_dtype)
    us = []
    for offset in (0, 1):
        flat = torch.zeros(x.size + offset, dtype=s.torch_dtype, device="cuda")
        flat[offset:] = torch.from_numpy(x.reshape(-1)).cuda()
        u, dt = flat[offset:].view(x.shape), torch.empty(8 * npg, dtype=s.torch_dtype, device="cuda")
        s.dt_cfl(u, dh, from_output=True, dt_out=dt)
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            for _ in range(50):
                s.dt_cfl(u, dh, from_output=True, dt_out=dt)
        best = float("inf")
        for _ in range(8):
            a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            a.record()
            graph.replay()
            b.record()
            torch.cuda.synchronize()
            best = min(best, a.elapsed_time(b) * 20)
        us.append(best)
    # 10 % for the spread of such short kernels; with the line at 296 patch groups in every policy mixed
    # took 1.27 and 1.14 times as long at 300 and 600
    assert us[0] < 1.1 * us[1], us


@pytest.mark.parametrize("npgs", [(3, 5), (40, 0, 200, 61), (290, 37), (1, 296, 300)])
@pytest.mark.parametrize("kw", [dict(precision="fp32"), dict(precision="mixed", dual_energy=True), dict(precision="fp64")])
def test_slabs_of_a_multi_level_call(cuda_device, npgs, kw):
    """Levels with time steps and cell sizes of their own, the slabs of the last wave across their
    borders: the bits of the call that keeps its patch groups whole, and of one call per level."""
    import torch
    s = FluidSolver(gamma=GAMMA, **kw)
    n = sum(npgs)
    x, dt, dh = _windows(n, 20, s.np_dtype, s.dual)
    t = torch.from_numpy(x).cuda()
    dts, dhs = [dt / 2 ** l for l in range(len(npgs))], [dh / 2 ** l for l in range(len(npgs))]
    got = []
    for way in ("whole", "slabs", "levels"):
        out = torch.full((n, s.ncomp, 16, 16, 16), float("nan"), dtype=t.dtype, device="cuda")
        flux = torch.full((n, 9, s.ncomp, 16, 16), float("nan"), dtype=t.dtype, device="cuda")
        de = torch.full((n, 16, 16, 16), 48, dtype=torch.int8, device="cuda") if s.dual else None
        if way == "levels":
            a = 0
            for m, d, h in zip(npgs, dts, dhs):
                if m:
                    s.solve_device(t[a:a + m], out[a:a + m], SolverParams(dt=d, dh=h), flux=flux[a:a + m],
                                   de_out=None if de is None else de[a:a + m])
                a += m
        else:
            s.solve_levels_device(t, out, npgs, dts, dhs, SolverParams(dt=dt, dh=dh), flux=flux, de_out=de,
                                  pg_fail=torch.zeros(n, dtype=torch.int32, device="cuda") if way == "whole" else None)
        torch.cuda.synchronize()
        got.append((out, flux, de))
    for other in got[1:]:
        for a, b in zip(got[0], other):
            assert a is None or torch.equal(a, b)
    assert bool(torch.isfinite(got[0][0]).all())
