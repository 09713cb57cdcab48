"""The float CTU+MHD fluxes formed slice by slice from face states in shared memory, against the FP64
solver, whose kernels store the face states, on the same float-rounded input (sizes, reconstructions,
limiters and floors)."""
import numpy as np
import pytest

from gamer_b200 import ic
from gamer_b200.fluid import FluidSolver, SolverParams

pytestmark = pytest.mark.gpu
GAMMA = 5.0 / 3.0


@pytest.mark.parametrize("npg", [1, 8, 27])
@pytest.mark.parametrize("lr,prec,kw", [("plm", "fp32", {}), ("plm", "mixed", {}), ("ppm", "fp32", {}), ("ppm", "mixed", {}),
                                        ("plm", "fp32", dict(LR_Limiter="vanleer")), ("plm", "fp32", dict(LR_Limiter="central")),
                                        ("ppm", "fp32", dict(LR_Limiter="albada")), ("plm", "fp32", dict(MinMod_Coeff=2.0)),
                                        ("plm", "fp32", dict(MinDens=0.9, MinPres=0.8, MinEint=1.2))])
def test_slices_against_fp64(cuda_device, npg, lr, prec, kw):
    import torch
    p = 3 if npg > 8 else 2
    u, b = ic.mhd_box(p, seed=npg, gamma=GAMMA)
    dh = 1.0 / (16 * p)
    a2 = GAMMA * (u[4] / u[0]) + sum(f ** 2 for f in b) / u[0]
    dt = 0.2 * dh / float(np.max(np.abs(u[1:4] / u[0]) + np.sqrt(a2)))
    nxt = 24 if lr == "ppm" else 22
    x = ic.cut_patch_groups(u, nxt)[:npg].astype(np.float32)
    m = ic.cut_mag_windows(b, nxt)[:npg].astype(np.float32)
    got = []
    for pr in (prec, "fp64"):
        s = FluidSolver(scheme="ctu", lr=lr, rsolver="hlld", precision=pr, gamma=GAMMA)
        t, tm = (torch.from_numpy(v.astype(s.np_dtype)).cuda() for v in (x, m))
        f = lambda *shape: torch.full(shape, float("nan"), dtype=t.dtype, device="cuda")  # noqa: E731
        out, flux, mag, ele = f(npg, 5, 16, 16, 16), f(npg, 9, 5, 16, 16), f(npg, 3, 17 * 256), f(npg, 9, 2, 272)
        s.solve_device(t, out, SolverParams(dt=dt, dh=dh, StoreElectric=True, **kw), flux=flux, mag_in=tm, mag_out=mag, ele=ele)
        torch.cuda.synchronize()
        assert s.status() == 0
        got.append([v.double() for v in (out, flux, mag, ele)])
    # 2-norms relative to the FP64 solver.  A value is some 50 roundings of terms up to ten times its
    # size (the EMFs are differences of products v x B ten times theirs): 50^1/2 x 10 x 2^-23 = 8e-6.  Edges and faces
    # whose upwind side or limiter branch differs, up to 1e-3 of them, move by up to 3e-2 of the
    # field: (1e-3)^1/2 x 3e-2 = 1e-3 in the EMFs, and dt/dh ~ 0.05 of that in the updated field
    for g, r, tol in zip(*got, (8e-6, 2e-5, 5e-5, 1e-3)):
        assert bool(torch.isfinite(g).all())
        assert float((g - r).norm() / r.norm()) < tol
    assert float(np.abs(ic.div_b(got[0][2].cpu().numpy())).max()) < 4e-6 * float(got[0][2].abs().max())
