"""The packed float2 paths of the MHM and MHM_RP kernels where they differ in kind from the scalar ones: faces
whose HLLC flux is 0/0 (each lane rescued on its own), PPM with user passive scalars or
characteristic limiting.  Compared with configurations that take other code for the same numbers, and
with the FP64 solver, which is scalar throughout."""
import numpy as np
import pytest

from gamer_b200 import ic
from gamer_b200.fluid import FluidSolver, SolverParams

pytestmark = pytest.mark.gpu
GAMMA = 5.0 / 3.0
DH = 1.0 / 32


def _solve(x, prm, **kw):
    import torch
    s = FluidSolver(gamma=GAMMA, **kw)
    t = torch.from_numpy(np.ascontiguousarray(ic.cut_patch_groups(x, s.flu_nxt).astype(s.np_dtype))).cuda()
    n = t.shape[0]
    out = torch.full((n, s.ncomp, 16, 16, 16), float("nan"), dtype=t.dtype, device="cuda")
    flux = torch.full((n, 9, s.ncomp, 16, 16), float("nan"), dtype=t.dtype, device="cuda")
    de = torch.full((n, 16, 16, 16), 48, dtype=torch.int8, device="cuda") if s.dual else None
    s.solve_device(t, out, prm, flux=flux, de_out=de)
    torch.cuda.synchronize()
    return out.double(), flux.double(), de


def _cold(dual):
    """Streams without pressure along x, y and z on a lognormal background, in float."""
    box = ic.lognormal_box(2, seed=12, gamma=GAMMA, dual=dual)
    for d, (z, y, x) in enumerate([(3, 18, 4), (20, 3, 19), (19, 20, 5)]):
        u = np.zeros((box.shape[0], 9, 9, 9))
        u[0], u[1 + d] = 1.0, 1.0
        half = [slice(None)] * 3
        half[2 - d] = slice(4, 9)
        u[(1 + d,) + tuple(half)] = 2.0
        u[4] = 0.5 * u[1 + d] ** 2
        if dual:
            u[5] = 1e-3
        box[:, z:z + 9, y:y + 9, x:x + 9] = u
    return box.astype(np.float32).astype(np.float64)


def _with_scalars(box, frac):
    return np.concatenate([box[:5], box[:1] * frac, box[5:]])


def _close(a, b, share, largest):
    """Scaled by the variable's rms: all but ``share`` of the values within 64 rounding errors, all within
    ``largest``; not-a-numbers in the same places."""
    import torch
    fin = torch.isfinite(b)
    assert torch.equal(fin, torch.isfinite(a))
    a, b = torch.where(fin, a, 0.0), torch.where(fin, b, 0.0)
    v = 1 if a.dim() == 5 and a.shape[1] != 9 else 2
    rms = (b * b).mean(dim=[d for d in range(a.dim()) if d != v], keepdim=True).sqrt() + 1e-30
    err = (a - b).abs() / (b.abs() + rms)
    assert float((err > 64 * 2.0 ** -23).double().mean()) < share and float(err.max()) < largest


@pytest.mark.parametrize("scheme", ["mhm", "mhm_rp"])
@pytest.mark.parametrize("lr", ["plm", "ppm"])
@pytest.mark.parametrize("prec", ["fp32", "mixed"])
@pytest.mark.parametrize("dual", [False, True])
def test_rescue_of_packed_faces(cuda_device, scheme, lr, prec, dual):
    """With two user scalars (here zero) the faces are solved one by one, in MHM and in both steps of
    MHM_RP; the fluid must not notice.  The streams' faces do reach the rescue: their HLLC flux is 0/0."""
    box = _cold(dual)
    prm = SolverParams(dt=0.1 * DH, dh=DH)
    got = _solve(box, prm, scheme=scheme, lr=lr, precision=prec, dual_energy=dual)
    ref = _solve(_with_scalars(box, np.zeros((2, 1, 1, 1))), prm, scheme=scheme, lr=lr, precision=prec, dual_energy=dual, npassive_user=2)
    keep = list(range(5)) + ([7] if dual else [])
    # the same scheme in the same precision with other contractions; the streams' edges are jumps,
    # where a limiter or an upwind side may switch
    _close(got[0], ref[0][:, keep], 2e-3, 5e-3)
    _close(got[1], ref[1][:, :, keep], 2e-3, 5e-3)
    if dual:
        assert int((got[2] != ref[2]).sum()) <= 4


@pytest.mark.parametrize("prec", ["fp32", "mixed"])
@pytest.mark.parametrize("kw,params", [
    (dict(lr="ppm", npassive_user=2), {}), (dict(lr="ppm", npassive_user=2), dict(FracIdx=(0, 1))),
    (dict(lr="ppm", npassive_user=2), dict(FracIdx=(0,), NormIdx=(0, 1))),
    (dict(lr="ppm", char_reconstruction=True), {}), (dict(lr="ppm", char_reconstruction=True, npassive_user=2, rsolver="roe"), {}),
    (dict(lr="ppm", dual_energy=True, rsolver="hlle"), {}), (dict(lr="ppm", scheme="mhm_rp", npassive_user=2), {})])
def test_packed_ppm_options_against_fp64(cuda_device, prec, kw, params):
    dual = kw.get("dual_energy", False)
    box = ic.lognormal_box(2, seed=21, gamma=GAMMA, dual=dual)
    if kw.get("npassive_user"):
        f = np.random.default_rng(5).random((2,) + box.shape[1:])
        box = _with_scalars(box, f / f.sum(0) if params.get("NormIdx") else f)
    box = box.astype(np.float32).astype(np.float64)
    prm = SolverParams(dt=ic.cfl_dt(box[:5], GAMMA, DH, cfl=0.4), dh=DH, **params)
    got = _solve(box, prm, precision=prec, **kw)
    ref = _solve(box, prm, precision="fp64", **kw)
    # float rounding of some hundred operations, and the share of cells that take another limiter branch
    _close(got[0], ref[0], 2e-3, 2e-2)
    _close(got[1], ref[1], 5e-3, 2e-2)
