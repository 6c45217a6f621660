"""tcgen05 implicit-GEMM convolutions against a plain PyTorch FP32 reference
(torch.nn.functional.conv3d on the same BF16-rounded inputs).  Input
channel counts that are multiples of 16 take the TMA-staged kernel, 2 -> 16
and 16 -> 1 the direct CUDA-core kernel, the others the gathering one; all
are covered.  Products of
BF16 values are exact in FP32, so the only differences are FP32 summation
order: 1e-3 relative of each output's magnitude."""
import numpy as np
import pytest
import torch
import torch.nn.functional as Fn

from gpu_util import ptr, require_cuda

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def lib():
    return require_cuda()


def _close(got, exp, tol=1e-3):
    got = got.double()
    exp = exp.double()
    scale = exp.abs().max().item() + 1e-30
    err = (got - exp).abs().max().item() / scale
    assert err <= tol, err


def _tensors(nb, C, nz, ny, nx, Cout, seed):
    g = torch.Generator().manual_seed(seed)
    x = torch.randn(nb, C, nz, ny, nx, generator=g).bfloat16().float()
    w = (torch.randn(Cout, C, 3, 3, 3, generator=g) / np.sqrt(27 * C)).bfloat16().float()
    b = torch.randn(Cout, generator=g) * 0.1
    return x.cuda(), w.cuda(), b.cuda()


def _cl(x):
    """(nb, C, z, y, x) -> the library's BF16 activation layout: C / 8 planes
    of [voxel][8 channels] when C is a multiple of 8, else [voxel][C]."""
    nb, C = x.shape[:2]
    if C % 8:
        return x.permute(0, 2, 3, 4, 1).contiguous().bfloat16()
    return x.reshape(nb, C // 8, 8, *x.shape[2:]).permute(1, 0, 3, 4, 5, 2).contiguous().bfloat16()


def _wk(w):   # (Cout, C, 3, 3, 3) -> [Cout][27][C] bf16
    return w.permute(0, 2, 3, 4, 1).reshape(w.shape[0], 27, w.shape[1]).contiguous().bfloat16()


@pytest.mark.parametrize("C,Cout,dims,nb", [(16, 32, (8, 10, 12), 2), (2, 16, (9, 7, 11), 1),
                                            (96, 32, (6, 8, 8), 1), (16, 1, (8, 8, 8), 2),
                                            (32, 64, (8, 16, 8), 1), (48, 16, (4, 8, 8), 1),
                                            (32, 16, (5, 9, 13), 2), (16, 96, (6, 6, 40), 1),
                                            (64, 128, (4, 8, 8), 1),
                                            # many tiles per CTA: every stage and both
                                            # accumulators of the persistent kernel cycle
                                            (48, 16, (40, 64, 64), 1), (16, 16, (24, 40, 48), 2),
                                            (32, 64, (16, 32, 32), 1), (2, 16, (33, 35, 37), 1),
                                            (16, 1, (33, 35, 37), 1)])
def test_forward(lib, C, Cout, dims, nb):
    nz, ny, nx = dims
    x, w, b = _tensors(nb, C, nz, ny, nx, Cout, 1)
    ref = torch.relu(Fn.conv3d(x, w, b, padding=1))
    y = torch.empty(nb, nz, ny, nx, Cout, dtype=torch.float32, device="cuda")
    xc, wk = _cl(x), _wk(w)      # held until the call returns
    rc = lib.pyro_conv3_forward(ptr(xc), C, nx, ny, nz, nb, ptr(wk), Cout, ptr(b), 1,
                                ptr(y), 1, None)
    assert rc == 0, lib.pyro_last_error()
    _close(y.permute(0, 4, 1, 2, 3), ref)


@pytest.mark.parametrize("Cin,Cout,dims", [(16, 32, (8, 10, 12)), (48, 16, (6, 8, 8)),
                                           (96, 32, (4, 8, 8)), (32, 64, (8, 8, 8)),
                                           (16, 8, (5, 7, 9)), (64, 16, (3, 17, 20)),
                                           (48, 16, (20, 32, 32))])
def test_backward_data_and_weight(lib, Cin, Cout, dims):
    nz, ny, nx = dims
    nb = 1
    x, w, _ = _tensors(nb, Cin, nz, ny, nx, Cout, 2)
    g = torch.Generator().manual_seed(3)
    dy = torch.randn(nb, Cout, nz, ny, nx, generator=g).bfloat16().float().cuda()
    xr = x.clone().requires_grad_(True)
    wr = w.clone().requires_grad_(True)
    out = Fn.conv3d(xr, wr, None, padding=1)
    out.backward(dy)
    dx = torch.empty(nb, nz, ny, nx, Cin, dtype=torch.float32, device="cuda")
    dyc, wk, xc = _cl(dy), _wk(w), _cl(x)
    rc = lib.pyro_conv3_backward_data(ptr(dyc), Cout, nx, ny, nz, nb, ptr(wk), Cin, None,
                                      ptr(dx), 1, None)
    assert rc == 0, lib.pyro_last_error()
    _close(dx.permute(0, 4, 1, 2, 3), xr.grad)
    # masked by the input activation (ReLU derivative)
    rc = lib.pyro_conv3_backward_data(ptr(dyc), Cout, nx, ny, nz, nb, ptr(wk), Cin,
                                      ptr(xc), ptr(dx), 1, None)
    assert rc == 0
    _close(dx.permute(0, 4, 1, 2, 3), xr.grad * (x > 0))
    dw = torch.zeros(Cout, 27, Cin, dtype=torch.float32, device="cuda")
    rc = lib.pyro_conv3_backward_weight(ptr(xc), Cin, ptr(dyc), Cout, nx, ny, nz, nb,
                                        ptr(dw), None)
    assert rc == 0, lib.pyro_last_error()
    _close(dw, wr.grad.permute(0, 2, 3, 4, 1).reshape(Cout, 27, Cin))


@pytest.mark.parametrize("Cin,Cout,dims,nb", [
    (8, 16, (3, 5, 7), 1),       # one plane, a row shorter than a tile
    (16, 16, (4, 9, 33), 2),     # a ragged tile in x and y, two volumes
    (24, 48, (5, 8, 16), 1),     # three groups of output channels
    (96, 32, (3, 6, 40), 2),     # two groups of input channels
    (104, 16, (2, 3, 17), 1),    # a prime count of planes
    (128, 128, (2, 4, 32), 1),   # the most channels
    (64, 64, (1, 1, 1), 1),      # a single voxel
    (16, 16, (40, 61, 70), 1),   # many tiles per CTA
])
def test_backward_weight_tma(lib, Cin, Cout, dims, nb):
    """The TMA-staged weight gradient accumulates into dw; FP32 sums of exact
    products in another order, as above."""
    nz, ny, nx = dims
    x, w, _ = _tensors(nb, Cin, nz, ny, nx, Cout, 4)
    g = torch.Generator().manual_seed(5)
    dy = torch.randn(nb, Cout, nz, ny, nx, generator=g).bfloat16().float().cuda()
    wr = w.clone().requires_grad_(True)
    Fn.conv3d(x, wr, None, padding=1).backward(dy)
    ref = wr.grad.permute(0, 2, 3, 4, 1).reshape(Cout, 27, Cin)
    dw = torch.full((Cout, 27, Cin), 0.5, dtype=torch.float32, device="cuda")
    xc, dyc = _cl(x), _cl(dy)
    rc = lib.pyro_conv3_backward_weight(ptr(xc), Cin, ptr(dyc), Cout, nx, ny, nz, nb,
                                        ptr(dw), None)
    assert rc == 0, lib.pyro_last_error()
    _close(dw - 0.5, ref)


@pytest.mark.parametrize("off", [(1, 0), (0, 1), (2, 4)])
def test_backward_weight_unaligned(lib, off):
    """Tensors that start off a 16-byte boundary are gathered: the same sums."""
    nb, Cin, Cout, (nz, ny, nx) = 1, 16, 32, (5, 6, 7)
    x, w, _ = _tensors(nb, Cin, nz, ny, nx, Cout, 14)
    g = torch.Generator().manual_seed(15)
    dy = torch.randn(nb, Cout, nz, ny, nx, generator=g).bfloat16().float().cuda()
    wr = w.clone().requires_grad_(True)
    Fn.conv3d(x, wr, None, padding=1).backward(dy)
    ref = wr.grad.permute(0, 2, 3, 4, 1).reshape(Cout, 27, Cin)
    moved = []
    for t, o in zip((_cl(x), _cl(dy)), off):
        m = torch.zeros(t.numel() + 8, dtype=t.dtype, device="cuda")
        m[o:o + t.numel()] = t.reshape(-1)
        moved.append(m[o:])
    dw = torch.zeros((Cout, 27, Cin), dtype=torch.float32, device="cuda")
    rc = lib.pyro_conv3_backward_weight(ptr(moved[0]), Cin, ptr(moved[1]), Cout, nx, ny, nz, nb,
                                        ptr(dw), None)
    assert rc == 0, lib.pyro_last_error()
    _close(dw, ref)


@pytest.mark.parametrize("C,Cout,dims,nb", [
    (16, 16, (1, 1, 1), 1),      # a single voxel
    (16, 16, (5, 17, 9), 2),     # ragged in every direction, two volumes
    (16, 16, (64, 160, 80), 1),  # four planes per tile, many tiles per CTA
    (48, 16, (33, 70, 41), 1),   # the same with three channel groups
    (16, 1, (70, 90, 60), 1),    # eight planes per tile, one column each
    (16, 48, (21, 33, 40), 1),   # two planes per tile, wide columns
    (64, 64, (3, 20, 30), 1),    # output channels split over CTAs
    (128, 128, (2, 5, 11), 1),   # the most channels
    (32, 24, (4, 18, 10), 1),    # 8-channel planes, not a multiple of 16
    (16, 100, (2, 9, 8), 1),     # channels that fill no plane
])
def test_forward_tiles(lib, C, Cout, dims, nb):
    """FP32 output against the reference as above; BF16 output, bit for bit the
    same sums rounded."""
    nz, ny, nx = dims
    x, w, b = _tensors(nb, C, nz, ny, nx, Cout, 6)
    ref = torch.relu(Fn.conv3d(x, w, b, padding=1))
    xc, wk = _cl(x), _wk(w)
    y32 = torch.full((nb, nz, ny, nx, Cout), 7.0, device="cuda")
    y16 = torch.full((nb * nz * ny * nx * Cout,), 7.0, dtype=torch.bfloat16, device="cuda")
    for y, f32 in ((y32, 1), (y16, 0)):
        rc = lib.pyro_conv3_forward(ptr(xc), C, nx, ny, nz, nb, ptr(wk), Cout, ptr(b), 1, ptr(y),
                                    f32, None)
        assert rc == 0, lib.pyro_last_error()
    got = y32.permute(0, 4, 1, 2, 3)
    _close(got, ref)
    if Cout % 8 == 0:
        bf = y16.view(Cout // 8, nb, nz, ny, nx, 8).permute(1, 0, 5, 2, 3, 4).reshape(ref.shape)
    else:
        bf = y16.view(nb, nz, ny, nx, Cout).permute(0, 4, 1, 2, 3)
    assert torch.equal(bf, got.bfloat16())


@pytest.mark.parametrize("C,Cout,dims", [(2, 16, (5, 7, 11)), (16, 1, (5, 7, 11)),
                                         (16, 1, (1, 3, 2))])
def test_narrow_layers_sum_in_fp32_order(lib, C, Cout, dims):
    """2 -> 16 and 16 -> 1 channels: one FP32 fused multiply-add per product in
    the order (dz, dy, 8 channels, dx, channel), bit for bit.  Operands kept
    away from 0 leave every product plus partial sum exact in FP64, so the
    rounding to FP32 is the fused one."""
    nz, ny, nx = dims
    x, w, b = _tensors(1, C, nz, ny, nx, Cout, 21)
    x = torch.where(x.abs() < 2.0 ** -8, torch.zeros_like(x), x)
    w = torch.where(w.abs() < 2.0 ** -10, torch.zeros_like(w), w)
    xp = Fn.pad(x, (1,) * 6).double()
    acc = b.view(1, -1, 1, 1, 1).expand(1, Cout, nz, ny, nx).clone()
    for dz in range(3):
        for dy in range(3):
            for c0 in range(0, C, 8):
                for dx in range(3):
                    for c in range(c0, min(c0 + 8, C)):
                        s = xp[:, c:c + 1, dz:dz + nz, dy:dy + ny, dx:dx + nx]
                        p = s * w[:, c, dz, dy, dx].double().view(1, -1, 1, 1, 1)
                        acc = (p + acc.double()).float()
    y = torch.empty(1, nz, ny, nx, Cout, dtype=torch.float32, device="cuda")
    xc, wk = _cl(x), _wk(w)
    rc = lib.pyro_conv3_forward(ptr(xc), C, nx, ny, nz, 1, ptr(wk), Cout, ptr(b), 0, ptr(y), 1,
                                None)
    assert rc == 0, lib.pyro_last_error()
    assert torch.equal(y.permute(0, 4, 1, 2, 3), acc)


def _bad_voxels(x, at, channel):
    """x with NaN, Inf and -Inf at three voxels, and the mask of the voxels
    within one cell of them."""
    bad, near = x.clone(), torch.zeros(x.shape[2:], dtype=torch.bool, device=x.device)
    for (z, y, xx), v in zip(at, (float("nan"), float("inf"), -float("inf"))):
        bad[0, channel, z, y, xx] = v
        near[max(z - 1, 0):z + 2, max(y - 1, 0):y + 2, max(xx - 1, 0):xx + 2] = True
    return bad, near


@pytest.mark.parametrize("C,Cout,dims", [(16, 16, (40, 100, 90)),  # four planes per tile
                                         (48, 16, (40, 100, 90)),
                                         (16, 48, (40, 100, 90)),  # two
                                         (32, 4, (41, 65, 40)),    # columns padded to 16
                                         (16, 16, (3, 17, 9))])    # a plane per tile
@pytest.mark.parametrize("relu", [0, 1])
def test_forward_not_finite_stays_local(lib, C, Cout, dims, relu):
    """A voxel that is not finite reaches the outputs of its 27 neighbours, and
    every other output keeps its bits."""
    nz, ny, nx = dims
    x, w, b = _tensors(1, C, nz, ny, nx, Cout, 31)
    at = [(nz // 2, ny // 3, nx // 2), (nz - 1, ny - 1, 0), (0, ny // 2, nx - 1)]
    bad, near = _bad_voxels(x, at, C - 3)
    wk = _wk(w)
    for f32 in (1, 0):
        out = []
        for t in (x, bad):
            y = torch.full((nz * ny * nx * Cout,), 7.0,
                           dtype=torch.float32 if f32 else torch.bfloat16, device="cuda")
            tc = _cl(t)
            rc = lib.pyro_conv3_forward(ptr(tc), C, nx, ny, nz, 1, ptr(wk), Cout, ptr(b), relu,
                                        ptr(y), f32, None)
            assert rc == 0, lib.pyro_last_error()
            if f32 or Cout % 8:
                out.append(y.view(nz, ny, nx, Cout))
            else:
                out.append(y.view(Cout // 8, nz, ny, nx, 8).permute(1, 2, 3, 0, 4)
                           .reshape(nz, ny, nx, Cout))
        assert torch.equal(out[1][~near], out[0][~near])
        assert relu or not torch.isfinite(out[1][near]).any()


@pytest.mark.parametrize("Cin,Cout,dims", [(16, 16, (40, 100, 90)), (48, 16, (40, 100, 90)),
                                           (16, 32, (21, 65, 40))])
def test_backward_data_not_finite_stays_local(lib, Cin, Cout, dims):
    """The same of the data gradient, masked, into a tensor of its own and over
    the mask."""
    nz, ny, nx = dims
    dy, _, _ = _tensors(1, Cout, nz, ny, nx, 1, 32)
    act, w, _ = _tensors(1, Cin, nz, ny, nx, Cout, 33)
    at = [(nz // 2, ny // 3, nx // 2), (nz - 1, ny - 1, 0), (0, ny // 2, nx - 1)]
    bad, near = _bad_voxels(dy, at, 5)
    wk, actc = _wk(w), _cl(act)
    out = []
    for t, inplace in ((dy, False), (bad, False), (bad, True)):
        tc, ac = _cl(t), actc.clone()
        dx = ac if inplace else torch.full_like(ac, 7.0)
        rc = lib.pyro_conv3_backward_data(ptr(tc), Cout, nx, ny, nz, 1, ptr(wk), Cin, ptr(ac),
                                          ptr(dx), 0, None)
        assert rc == 0, lib.pyro_last_error()
        out.append(dx.view(Cin // 8, nz, ny, nx, 8).permute(1, 2, 3, 0, 4)
                   .reshape(nz, ny, nx, Cin))
    on = act[0].permute(1, 2, 3, 0) > 0
    far = ~near
    assert torch.equal(out[1][far], out[0][far])
    assert torch.equal(out[2][far], out[0][far])
    for o in out[1:]:
        assert not torch.isfinite(o[near][on[near]]).any()
        assert (o[near][~on[near]] == 0).all()


@pytest.mark.parametrize("Cin,Cout,dims", [(16, 16, (5, 9, 33)),    # ragged tiles in x and y
                                           (8, 32, (4, 18, 20)),
                                           (16, 80, (4, 6, 20)),    # a width that the gather pads
                                           (48, 16, (24, 30, 64))])  # several tiles per CTA
@pytest.mark.parametrize("which", ["x", "dy"])
def test_backward_weight_not_finite_stays_local(lib, Cin, Cout, dims, which):
    """Voxels on the volume's edges that are not finite: an x reaches the entries
    that a pair of voxels inside the volume has it in, and no other; a dy the
    entries of its channel (with the zeros around x in all taps).  The others
    are the sums of the finite tensors (FP32 sums in another order, as above)."""
    nz, ny, nx = dims
    t = {"x": _tensors(1, Cin, nz, ny, nx, 1, 41)[0], "dy": _tensors(1, Cout, nz, ny, nx, 1, 42)[0]}
    at = [(nz - 1, ny - 1, nx - 1), (0, ny // 2, 0), (nz // 2, 0, nx - 1)]
    w = torch.zeros(Cout, Cin, 3, 3, 3, device="cuda", requires_grad=True)
    Fn.conv3d(t["x"], w, None, padding=1).backward(t["dy"])
    ref = w.grad.permute(0, 2, 3, 4, 1).reshape(Cout, 27, Cin)
    hit = torch.zeros(Cout, 27, Cin, dtype=torch.bool, device="cuda")
    bad = t[which].clone()
    for k, ((z, y, x), v) in enumerate(zip(at, (float("nan"), float("inf"), -float("inf")))):
        c = 3 + 2 * k
        bad[0, c, z, y, x] = v
        for tap in range(27):  # x at v meets dy at v - tap
            d = (tap // 9 - 1, tap // 3 % 3 - 1, tap % 3 - 1)
            if which == "dy":
                hit[c, tap] = True
            elif all(0 <= p - s < n for p, s, n in zip((z, y, x), d, dims)):
                hit[:, tap, c] = True
    t[which] = bad
    xc, dc = _cl(t["x"]), _cl(t["dy"])
    dw = torch.zeros(Cout, 27, Cin, device="cuda")
    rc = lib.pyro_conv3_backward_weight(ptr(xc), Cin, ptr(dc), Cout, nx, ny, nz, 1, ptr(dw), None)
    assert rc == 0, lib.pyro_last_error()
    assert not torch.isfinite(dw[hit]).any()
    assert torch.isfinite(dw[~hit]).all()
    _close(dw[~hit], ref[~hit])


@pytest.mark.parametrize("Cin,Cout,dims", [(16, 16, (64, 64, 128)), (48, 16, (40, 64, 64)),
                                           (16, 32, (30, 37, 130))])
def test_backward_weight_error_bounded_by_the_gather(lib, Cin, Cout, dims):
    """Sums over many voxels: the TMA-staged gradient is no further from 64 bits
    than the gather GEMM's, which the same values off a 16-byte boundary take."""
    nz, ny, nx = dims
    g = torch.Generator(device="cuda").manual_seed(51)
    x = torch.randn(1, Cin, nz, ny, nx, device="cuda", generator=g).abs().bfloat16().float()
    dy = torch.randn(1, Cout, nz, ny, nx, device="cuda", generator=g).bfloat16().float()
    ref = torch.empty(Cout, 27, Cin, dtype=torch.float64, device="cuda")
    xp, d = Fn.pad(x, (1,) * 6).double()[0], dy.double().reshape(Cout, -1)
    for t in range(27):
        z0, y0, x0 = t // 9, t // 3 % 3, t % 3
        ref[:, t] = d @ xp[:, z0:z0 + nz, y0:y0 + ny, x0:x0 + nx].reshape(Cin, -1).t()
    xc, dc = _cl(x).reshape(-1), _cl(dy)
    off = torch.zeros(xc.numel() + 8, dtype=xc.dtype, device="cuda")[1:]
    off[:xc.numel()] = xc
    errs = []
    for xv in (xc, off):
        dw = torch.zeros(Cout, 27, Cin, device="cuda")
        rc = lib.pyro_conv3_backward_weight(ptr(xv), Cin, ptr(dc), Cout, nx, ny, nz, 1, ptr(dw),
                                            None)
        assert rc == 0, lib.pyro_last_error()
        errs.append(((dw - ref).norm() / ref.norm()).item())
    assert errs[0] <= errs[1], errs


@pytest.mark.parametrize("Cin,Cout", [(8, 16), (3, 32)])
def test_gather_unaligned(lib, Cin, Cout):
    """The gather GEMM's outputs, mask and bias at 2- or 4-byte alignment: the
    bits of the aligned call."""
    nz, ny, nx = 5, 6, 7
    x, w, b = _tensors(1, Cin, nz, ny, nx, Cout, 61)
    dy, _, _ = _tensors(1, Cin, nz, ny, nx, 1, 62)
    act, w2, _ = _tensors(1, Cout, nz, ny, nx, Cin, 63)
    n = nz * ny * nx * Cout
    xc, wk, dc, wk2, ac = _cl(x), _wk(w), _cl(dy), _wk(w2), _cl(act).reshape(-1)
    outs = []
    for o in (0, 1, 3):
        y = torch.zeros(n + 8, dtype=torch.bfloat16, device="cuda")
        dx, m = torch.zeros_like(y), torch.zeros_like(y)
        bb = torch.zeros(Cout + 4, device="cuda")
        bb[o:o + Cout] = b
        m[o:o + n] = ac
        assert lib.pyro_conv3_forward(ptr(xc), Cin, nx, ny, nz, 1, ptr(wk), Cout, ptr(bb[o:]), 1,
                                      ptr(y[o:]), 0, None) == 0, lib.pyro_last_error()
        # channels swapped: Cin gradients into Cout masked ones
        assert lib.pyro_conv3_backward_data(ptr(dc), Cin, nx, ny, nz, 1, ptr(wk2), Cout,
                                            ptr(m[o:]), ptr(dx[o:]), 0, None) == 0
        outs.append((y[o:o + n].clone(), dx[o:o + n].clone()))
    for y, dx in outs[1:]:
        assert torch.equal(y, outs[0][0]) and torch.equal(dx, outs[0][1])


def test_direct_unaligned_is_refused(lib):
    """Tensors off the boundary of the direct kernel's accesses."""
    x = torch.zeros(4 * 5 * 6 * 16 + 8, dtype=torch.bfloat16, device="cuda")
    w, y = torch.zeros_like(x), torch.zeros(4096, device="cuda")
    for C, Cout, xo, yo in ((16, 1, 1, 0), (16, 1, 4, 0), (2, 16, 1, 0), (2, 16, 0, 1)):
        rc = lib.pyro_conv3_forward(ptr(x[xo:]), C, 6, 5, 4, 1, ptr(w), Cout, None, 0,
                                    ptr(y.bfloat16()[yo:]) if yo else ptr(y), 0, None)
        assert rc < 0
