"""Interpolate_Iterate over slabs of parents staged in shared memory, and the window assembly, at the
sizes where their tiles, slabs and alignment change.  The interpolation is compared with the plain
kernel (one thread per parent and variable, the same operations) and with one-parent regions; the
assembly with numpy.  Both bit for bit."""
import numpy as np
import pytest

from gamer_b200 import fluid

pytestmark = pytest.mark.gpu


def _coarse(rng, nb, cz, cy, cx, dtype, bad=0.0):
    """Conserved states of nb regions; a share of them with a kinetic energy close to the total one,
    so that interpolated children come out unphysical."""
    rho = np.exp(rng.normal(0, 0.4, (nb, cz, cy, cx)))
    p = np.exp(rng.normal(0, 0.4, rho.shape))
    v = rng.normal(0, 1.0, (3,) + rho.shape)
    p = np.where(rng.random(rho.shape) < bad, 1e-3 * p, p)
    e = p / (5.0 / 3.0 - 1.0) + 0.5 * rho * (v ** 2).sum(0)
    return np.stack([rho, rho * v[0], rho * v[1], rho * v[2], e], 1).astype(dtype)


@pytest.mark.parametrize("dtype", ["float32", "float64"])
@pytest.mark.parametrize("scheme,shape,nb", [
    ("cquad", (12, 12, 12), 3), ("cquad", (11, 7, 5), 4), ("cquad", (3, 3, 3), 5), ("cquad", (4, 70, 71), 1),
    ("cquad", (5, 150, 150), 1), ("minmod3d", (9, 6, 13), 2), ("vanleer", (8, 8, 8), 2), ("quad", (6, 12, 10), 2),
    ("cquar", (14, 14, 14), 2), ("quar", (7, 6, 9), 2), ("minmod1d", (10, 5, 8), 2)])
@pytest.mark.parametrize("offset", [0, 1])
def test_iterate_equals_plain_where_every_child_is_physical(cuda_device, dtype, scheme, shape, nb, offset):
    import torch
    g = 2 if scheme in ("cquar", "quar") else 1
    rng = np.random.default_rng(sum(shape) + offset)
    c = _coarse(rng, nb, *shape, dtype)
    c[:, 4] *= 50.0                               # pressure-dominated: no child can fail
    flat = torch.zeros(c.size + offset, dtype=getattr(torch, dtype), device="cuda")
    flat[offset:] = torch.from_numpy(c.reshape(-1)).cuda()
    t = flat[offset:].view(c.shape)               # offset 1: not 16-byte aligned
    rng3 = tuple(n - 2 * g for n in reversed(shape))
    fshape = (nb, 5) + tuple(2 * n for n in reversed(rng3))
    a, b = (torch.full(fshape, float("nan"), dtype=t.dtype, device="cuda") for _ in range(2))
    status = torch.zeros(1, dtype=torch.int32, device="cuda")
    reduce_ok = scheme not in ("minmod3d", "minmod1d", "vanleer")
    fluid.interpolate_device(t, a, scheme, (g, g, g), rng3, iterate=True, status=status, mono_max_iter=10 if reduce_ok else 0)
    fluid.interpolate_device(t, b, scheme, (g, g, g), rng3)
    torch.cuda.synchronize()
    assert int(status) == 0 and torch.equal(a, b)


@pytest.mark.parametrize("dtype", ["float32", "float64"])
@pytest.mark.parametrize("shape", [(12, 12, 12), (5, 9, 7)])
def test_iterating_parents_equal_one_parent_regions(cuda_device, dtype, shape):
    """Unphysical children (the primitive and the reduced-coefficient attempts) anywhere in a region."""
    import torch
    rng = np.random.default_rng(8)
    nb, (cz, cy, cx) = 2, shape
    c = torch.from_numpy(_coarse(rng, nb, cz, cy, cx, dtype, bad=0.5)).cuda()
    whole = torch.full((nb, 5, 2 * cz - 4, 2 * cy - 4, 2 * cx - 4), float("nan"), dtype=c.dtype, device="cuda")
    plain = torch.empty_like(whole)
    status = torch.zeros(1, dtype=torch.int32, device="cuda")
    fluid.interpolate_device(c, whole, "cquad", (1, 1, 1), (cx - 2, cy - 2, cz - 2), iterate=True, status=status)
    fluid.interpolate_device(c, plain, "cquad", (1, 1, 1), (cx - 2, cy - 2, cz - 2))
    cubes = c.unfold(2, 3, 1).unfold(3, 3, 1).unfold(4, 3, 1)            # [nb][5][z][y][x][3][3][3]
    n = (cz - 2, cy - 2, cx - 2)
    cubes = cubes.permute(0, 2, 3, 4, 1, 5, 6, 7).reshape(-1, 5, 3, 3, 3).contiguous()
    one = torch.empty((cubes.shape[0], 5, 2, 2, 2), dtype=c.dtype, device="cuda")
    st1 = torch.zeros(1, dtype=torch.int32, device="cuda")
    fluid.interpolate_device(cubes, one, "cquad", (1, 1, 1), (1, 1, 1), iterate=True, status=st1)
    one = one.view((nb,) + n + (5, 2, 2, 2)).permute(0, 4, 1, 5, 2, 6, 3, 7).reshape(whole.shape)
    torch.cuda.synchronize()
    assert torch.equal(whole, one) and int(status) == int(st1)
    assert not torch.equal(whole, plain)          # the case does reach the later attempts


@pytest.mark.parametrize("dtype", ["float32", "float64"])
@pytest.mark.parametrize("scheme,shape,nb", [("cquad", (3, 3, 3), 301), ("cquad", (4, 3, 5), 1000), ("cquad", (10, 3, 10), 37),
                                             ("quar", (5, 6, 7), 45), ("cquad", (3, 3, 2500), 2), ("quar", (5, 6, 900), 1)])
def test_packed_and_cut_regions_equal_the_cells_on_their_own(cuda_device, dtype, scheme, shape, nb):
    """Several small regions in one CTA and rows cut along x, with parents that iterate: each region
    alone gives the same bits, and so does the same range inside a larger coarse array (whose planes are
    not contiguous in the staged box)."""
    import torch
    g = 2 if scheme == "quar" else 1
    rng = np.random.default_rng(nb)
    c = torch.from_numpy(_coarse(rng, nb, *shape, dtype, bad=0.3)).cuda()
    n = tuple(s - 2 * g for s in shape)
    args = (scheme, (g, g, g), tuple(reversed(n)))

    def fill(cdata, args):
        out = torch.full((cdata.shape[0], 5) + tuple(2 * k for k in n), float("nan"), dtype=c.dtype, device="cuda")
        status = torch.zeros(1, dtype=torch.int32, device="cuda")
        fluid.interpolate_device(cdata, out, *args, iterate=True, status=status)
        torch.cuda.synchronize()
        return out, int(status)
    got, st = fill(c, args)
    assert not bool(torch.isnan(got[:, 0]).any())
    wide = torch.full((nb, 5) + tuple(s + 3 for s in shape), float("nan"), dtype=c.dtype, device="cuda")
    wide[:, :, 1:-2, 2:-1, 3:] = c
    sub, st2 = fill(wide, (scheme, (3 + g, 2 + g, 1 + g), args[2]))
    assert torch.equal(sub, got) and st2 == st
    for b in sorted({0, nb // 2, nb - 1}):
        assert torch.equal(fill(c[b:b + 1].contiguous(), args)[0], got[b:b + 1])
    if scheme == "cquad":
        # and the parents one by one, the last ones of the region and of the batch
        i = [k - 1 for k in n]
        one = c[-1:, :, i[0]:i[0] + 3, i[1]:i[1] + 3, i[2]:i[2] + 3].contiguous()
        out = torch.empty((1, 5, 2, 2, 2), dtype=c.dtype, device="cuda")
        fluid.interpolate_device(one, out, "cquad", (1, 1, 1), (1, 1, 1), iterate=True,
                                 status=torch.zeros(1, dtype=torch.int32, device="cuda"))
        assert torch.equal(out, got[-1:, :, -2:, -2:, -2:])


@pytest.mark.parametrize("nb,shape,bad", [(8000, (4, 4, 4), 0.0), (4000, (3, 3, 10), 0.0), (1, (70, 70, 70), 0.0), (342, (12, 12, 12), 1.0)])
def test_iterating_regions_keep_the_gpu_busy(cuda_device, nb, shape, bad):
    """Many small regions, one large one, and regions where every parent iterates, against the plain
    kernel (one thread per parent and variable of the whole call) on the same regions: about as long
    where no parent iterates, and not many times as long where they do."""
    import torch
    c = torch.from_numpy(_coarse(np.random.default_rng(1), min(nb, 64), *shape, "float32", bad=bad)).cuda()
    if not bad:
        c[:, 4] *= 50.0
    c = c[torch.arange(nb, device="cuda") % c.shape[0]].contiguous()
    n = tuple(s - 2 for s in reversed(shape))
    out = torch.empty((nb, 5) + tuple(2 * k for k in reversed(n)), dtype=c.dtype, device="cuda")
    status = torch.zeros(1, dtype=torch.int32, device="cuda")

    def ms(**kw):
        best = float("inf")
        for _ in range(6):
            a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            a.record()
            for _ in range(20):
                fluid.interpolate_device(c, out, "cquad", (1, 1, 1), n, **kw)
            b.record()
            torch.cuda.synchronize()
            best = min(best, a.elapsed_time(b))
        return best
    # measured 1.1 to 1.7 and, iterating, 2.3; with one CTA per region or plane and each parent iterating
    # on its own 3.0 to 15 and 5.0
    assert ms(iterate=True, status=status) < (3.5 if bad else 2.4) * ms()


def _assembled(fine, nbr, cint, nxt):
    npg, nc = fine.shape[:2]
    g = (nxt - 16) // 2
    win = np.full((npg, nc, nxt, nxt, nxt), np.nan, fine.dtype)
    edge = [slice(0, g), slice(g, g + 16), slice(g + 16, nxt)]
    for p in range(npg):
        for s in range(27):
            d = (s // 9 - 1, s // 3 % 3 - 1, s % 3 - 1)
            to = tuple(edge[x + 1] for x in d)
            at = tuple(slice(16 - g, 16) if x < 0 else slice(0, g) if x > 0 else slice(0, 16) for x in d)
            src = p if s == 13 else nbr[p, s]
            if 0 <= src < npg:
                win[(p, slice(None)) + to] = fine[(src, slice(None)) + at]
            elif src < 0 and cint is not None:
                win[(p, slice(None)) + to] = cint[(p, slice(None)) + to]
    return win


@pytest.mark.parametrize("dtype", ["float32", "float64"])
@pytest.mark.parametrize("nxt,npg,nc,offset,with_cint", [(18, 3, 5, 0, True), (20, 5, 5, 0, True), (20, 1, 1, 0, False),
                                                         (22, 4, 6, 0, True), (24, 2, 8, 0, True), (26, 2, 2, 0, True),
                                                         (20, 3, 5, 1, True), (48, 1, 1, 0, True)])
def test_assembly_against_numpy(cuda_device, dtype, nxt, npg, nc, offset, with_cint):
    import torch
    rng = np.random.default_rng(nxt + npg)
    fine = rng.standard_normal((npg, nc, 16, 16, 16)).astype(dtype)
    cint = rng.standard_normal((npg, nc, nxt, nxt, nxt)).astype(dtype) if with_cint else None
    nbr = rng.integers(-1, npg + 1, (npg, 27)).astype(np.int32)         # npg: not a patch group of the batch
    n = npg * nc * nxt ** 3
    flat = torch.zeros(n + offset, dtype=getattr(torch, dtype), device="cuda")
    win = flat[offset:].view(npg, nc, nxt, nxt, nxt)
    fluid.assemble_windows_device(torch.from_numpy(fine).cuda(), torch.from_numpy(nbr).cuda(),
                                  None if cint is None else torch.from_numpy(cint).cuda(), win)
    torch.cuda.synchronize()
    np.testing.assert_array_equal(win.cpu().numpy(), _assembled(fine, nbr, cint, nxt))
