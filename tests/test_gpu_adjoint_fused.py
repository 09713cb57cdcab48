"""The plane-streaming adjoint kernel (calls that fill the GPU) against the separate kernels (smaller
calls on the same patch groups), through the C ABI."""
import ctypes

import numpy as np
import pytest

from gamer_b200 import ic
from gamer_b200.fluid import FluidSolver, SolverParams, _check, _dptr

pytestmark = pytest.mark.gpu
GAMMA = 5.0 / 3.0


def _adjoint(s, x, gout, prm, ws_pg):
    import torch
    n = x.shape[0]
    nbytes = ctypes.c_ulonglong()
    _check(s.lib.gb_fluid_adjoint_workspace_bytes(s.h, ws_pg, ctypes.byref(nbytes)), "workspace")
    ws = torch.zeros(nbytes.value, dtype=torch.uint8, device="cuda")
    gin = torch.full((n, 5, 20, 20, 20), float("nan"), dtype=torch.float64, device="cuda")
    p = prm.c()
    _check(s.lib.gb_fluid_adjoint_step_device(s.h, _dptr(x), _dptr(gout), _dptr(gin), n, ctypes.byref(p), _dptr(ws),
                                              nbytes.value, ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)),
           "gb_fluid_adjoint_step_device")
    torch.cuda.synchronize()
    assert s.status() == 0
    return gin, ws[:4 * n].view(torch.int32)


def _case(npg, cold):
    import torch
    box = ic.lognormal_box(5, seed=npg, gamma=GAMMA)
    x = np.concatenate([ic.cut_patch_groups(box, 20)] * 3)[:npg].astype(np.float32)
    if cold:
        # streams without pressure: the HLLC flux of their faces is 0/0, the HLLE rescue's is not
        for p in range(0, npg, 7):
            x[p, :, 6:11, 6:11, 6:11] = np.array([1.0, 1.0, 1.0, 1.0, 1.5])[:, None, None, None]
            x[p, 1, 6:11, 6:11, 8:11] = 2.0
            x[p, 4, 6:11, 6:11, 8:11] = 3.0
    g = np.random.default_rng(npg).standard_normal((npg, 5, 16, 16, 16))
    dh = 1.0 / 80
    prm = SolverParams(dt=ic.cfl_dt(box, GAMMA, dh, cfl=0.4), dh=dh)
    return torch.from_numpy(x).cuda(), torch.from_numpy(g).cuda(), prm


@pytest.mark.parametrize("npg,cold", [(99, False), (100, False), (148, True), (149, False), (300, False), (301, True)])
def test_fused_adjoint_equals_the_separate_kernels(cuda_device, npg, cold):
    import torch
    s = FluidSolver(precision="fp32", gamma=GAMMA)
    x, gout, prm = _case(npg, cold)
    got, flags = _adjoint(s, x, gout, prm, npg)
    want = torch.cat([_adjoint(s, x[i:i + 50].contiguous(), gout[i:i + 50].contiguous(), prm, 50)[0]
                      for i in range(0, npg, 50)])
    if cold:
        assert int((flags != 0).sum()) == len(range(0, npg, 7))      # done again with the rescue
    ok = torch.isfinite(want)
    assert torch.equal(ok, torch.isfinite(got))
    # both sum in double; a face state may differ in its last bit (2^-24), which the derivatives of
    # the wave speeds enlarge about tenfold
    err = torch.where(ok, got - want, 0.0).norm() / torch.where(ok, want, 0.0).norm()
    assert float(err) < 1e-6


def test_unaligned_and_small_workspace_calls_still_run(cuda_device):
    """d loss / d U_out off a 16-byte boundary, and a workspace of one patch group."""
    import torch
    s = FluidSolver(precision="fp32", gamma=GAMMA)
    x, gout, prm = _case(148, False)
    want, _ = _adjoint(s, x, gout, prm, 148)
    off = torch.empty(gout.numel() + 1, dtype=torch.float64, device="cuda")[1:].view(gout.shape)
    off.copy_(gout)
    for g, ws_pg in ((off, 148), (gout, 1)):
        got, _ = _adjoint(s, x, g, prm, ws_pg)
        assert float((got - want).norm() / want.norm()) < 1e-6       # bound as above


@pytest.mark.parametrize("dims,nxt,prec", [((1, 2, 3), 20, "fp32"), ((2, 1, 1), 24, "fp64"), ((3, 2, 1), 24, "fp32"), ((2, 2, 2), 22, "fp32")])
def test_box_gather_of_wide_and_unaligned_boxes(cuda_device, dims, nxt, prec):
    """Windows cut in quadruples (widths 20, 24), by columns (others), and from a box off a 16-byte
    boundary equal the periodic indexing; and the transpose adds every image once."""
    import torch
    from gamer_b200.fluid import load_library
    lib = load_library()
    npx, npy, npz = dims
    dt = torch.float64 if prec == "fp64" else torch.float32
    n = (5, 16 * npz, 16 * npy, 16 * npx)
    box = torch.randn(n, dtype=dt, device="cuda")
    g = (nxt - 16) // 2
    ix = [torch.stack([(torch.arange(nxt) - g + 16 * p) % (16 * q) for p in range(q)]) for q in (npz, npy, npx)]
    want = torch.stack([box[:, ix[0][p // (npy * npx)].cuda()][:, :, ix[1][p // npx % npy].cuda()][:, :, :, ix[2][p % npx].cuda()]
                        for p in range(npx * npy * npz)])
    st = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
    for shift in (0, 1):
        b = torch.empty(box.numel() + shift, dtype=dt, device="cuda")[shift:].view(n)
        b.copy_(box)
        win = torch.empty(want.shape, dtype=dt, device="cuda")
        assert lib.gb_box_gather_device(_dptr(b), _dptr(win), npx, npy, npz, nxt, 5, 2 if prec == "fp64" else 0, st) == 0
        assert torch.equal(win, want)
    w = torch.randn(want.shape, dtype=torch.float64, device="cuda")
    wt = torch.empty(n, dtype=torch.float64, device="cuda")
    assert lib.gb_box_gather_adjoint_device(_dptr(w), _dptr(wt), npx, npy, npz, nxt, 5, st) == 0
    ref = torch.zeros(n, dtype=torch.float64, device="cuda")
    for p in range(npx * npy * npz):
        z, y, xx = (ix[0][p // (npy * npx)].cuda(), ix[1][p // npx % npy].cuda(), ix[2][p % npx].cuda())
        for k in range(nxt):                    # one plane at a time; the indices of y and x repeat at most
            for j in range(nxt):
                ref[:, z[k], y[j]].index_add_(1, xx, w[p, :, k, j])
    # sums of at most 2^3 (24 wide, one patch group per axis: 2^3) doubles of order one
    assert float((wt - ref).abs().max()) < 1e-13
