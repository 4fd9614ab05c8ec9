"""Multi-plane SATs, box filters and their autograd backward on the GPU.

Plane stacks are integer-exact against the oracle plane by plane.  Box means
and gradients are floating point (f32 through an f32 SAT) and are compared
with float64 torch references with the tolerances written below:

  box means        |m - m64| <= 4 * eps32 * max|S64| / area + 1e-7
  gradients        |g - g64| <= 1e-4 * max(1, max|g64|)
  central FD       |g - fd|  <= 1e-4 * max(1, max|fd|)   (FP64 loss, h = 1e-3)
"""
import numpy as np
import pytest
import torch

import sat_gb300
from sat_gb300 import autograd as AG
from sat_gb300 import api
from tests.util import bits, to_dev, to_np

pytestmark = pytest.mark.gpu

EPS32 = float(np.finfo(np.float32).eps)


def sat64(x: torch.Tensor) -> torch.Tensor:
    return x.double().cumsum(-1).cumsum(-2)


def box_means64(x: torch.Tensor, radii) -> torch.Tensor:
    """Clipped box means in float64 by the four-corner rule on a zero-padded
    SAT (differentiable, for reference gradients)."""
    H, W = x.shape[-2:]
    S = torch.nn.functional.pad(sat64(x), (1, 0, 1, 0))  # S[y+1, x+1] = SAT(y, x)
    ys = torch.arange(H, device=x.device)
    xs = torch.arange(W, device=x.device)
    outs = []
    for r in radii:
        ya, yb = (ys - r).clamp(min=0), (ys + r).clamp(max=H - 1)
        xa, xb = (xs - r).clamp(min=0), (xs + r).clamp(max=W - 1)
        s = (S[..., yb + 1, :][..., xb + 1] - S[..., ya, :][..., xb + 1]
             - S[..., yb + 1, :][..., xa] + S[..., ya, :][..., xa])
        area = ((yb - ya + 1).double()[:, None] * (xb - xa + 1).double()[None, :])
        outs.append(s / area)
    return torch.stack(outs, dim=-3)


def test_planes_integer_exact(cuda, oracle):
    n, c, h, w = 2, 3, 131, 277
    a = oracle.gen("u8", 11, (n * c * h, w)).reshape(n, c, h, w)
    x = to_dev(a)
    out = to_np(sat_gb300.sat(x, torch.uint32))
    for i in range(n):
        for j in range(c):
            ref = oracle.sat_serial(a[i, j], np.uint32)
            assert np.array_equal(bits(out[i, j]), bits(ref)), (i, j)


def test_planes_pitched_and_reverse(cuda, oracle):
    """Planes whose rows are a slice of wider rows (pitch > width), forward
    and reverse, f32 -> f32 and u8 -> u32."""
    p, h, w, pitch = 5, 97, 200, 256
    a = oracle.gen("u8", 12, (p * h, w)).reshape(p, h, w)
    base = torch.zeros((p, h, pitch), dtype=torch.uint8, device=cuda)
    base[..., :w] = to_dev(a)
    x = base[..., :w]
    for rev in (False, True):
        out = to_np(sat_gb300.sat(x, torch.uint32, reverse=rev))
        for i in range(p):
            ref = oracle.sat_reverse(a[i], np.uint32) if rev else oracle.sat_serial(a[i], np.uint32)
            assert np.array_equal(bits(out[i]), bits(ref)), (i, rev)
    af = oracle.gen("f32n", 13, (p * h, w)).astype(np.float32).reshape(p, h, w)
    outf = to_np(sat_gb300.sat(to_dev(af), torch.float32))
    for i in range(p):
        ref = oracle.sat_fp64(af[i])
        den = oracle.sat_fp64(af[i], absval=True)
        assert np.max(np.abs(outf[i] - ref) / np.maximum(den, 1e-30)) <= 1e-5


@pytest.mark.parametrize("mode", ["plain", "compensated"])
def test_planes_float_modes(cuda, oracle, mode):
    """Stacks through the default kernels of each accumulator: f64 outputs
    (warp-specialized tiles) and compensated f32 (register tiles)."""
    p, h, w = 6, 77, 301
    a = oracle.gen("f32n", 15, (p * h, w)).astype(np.float32).reshape(p, h, w)
    if mode == "plain":
        out = to_np(sat_gb300.sat(to_dev(a), torch.float64))
        tol = 1e-13
    else:
        out = to_np(sat_gb300.sat(to_dev(a), torch.float32, mode="compensated"))
        tol = 2e-7
    for i in range(p):
        ref = oracle.sat_fp64(a[i])
        den = oracle.sat_fp64(a[i], absval=True)
        assert np.max(np.abs(out[i].astype(np.float64) - ref) / np.maximum(den, 1e-30)) <= tol, i


def test_planes_many_small(cuda, oracle):
    """More planes than tiles per plane: 300 planes of 40 x 70."""
    a = oracle.gen("u8", 14, (300 * 40, 70)).reshape(300, 40, 70)
    out = to_np(sat_gb300.sat(to_dev(a), torch.uint32))
    for i in (0, 1, 150, 299):
        assert np.array_equal(bits(out[i]), bits(oracle.sat_serial(a[i], np.uint32))), i


@pytest.mark.parametrize("shape", [(1, 1, 37, 53), (2, 3, 64, 64), (1, 2, 5, 300)])
def test_box_means_forward(cuda, shape):
    g = torch.Generator(device="cpu").manual_seed(21)
    x = torch.randn(shape, generator=g, dtype=torch.float32).to(cuda)
    radii = (0, 1, 3, 40)  # 40 exceeds every side: the whole image
    m = AG.box_filter_means(x, radii)
    ref = box_means64(x, radii)
    H, W = shape[-2:]
    smax = float(sat64(x.abs()).max())
    for k, r in enumerate(radii):
        area_min = (min(r, H - 1) + 1) * (min(r, W - 1) + 1)
        tol = 4 * EPS32 * smax / area_min + 1e-7
        err = float((m[..., k, :, :].double() - ref[..., k, :, :]).abs().max())
        assert err <= tol, (r, err, tol)


def _four_corner64(S: torch.Tensor, radii):
    """Box means in float64 from the given SAT S (..., H, W) by the four-corner
    rule, and per element the magnitudes |A| + |B| of its two row-segment
    differences A = S(yb,xb) - S(yb,xa-1), B = S(ya-1,xb) - S(ya-1,xa-1)."""
    H, W = S.shape[-2:]
    P = torch.nn.functional.pad(S.double(), (1, 0, 1, 0))
    ys = torch.arange(H, device=S.device)
    xs = torch.arange(W, device=S.device)
    means, mags = [], []
    for r in radii:
        ya, yb = (ys - r).clamp(min=0), (ys + r).clamp(max=H - 1)
        xa, xb = (xs - r).clamp(min=0), (xs + r).clamp(max=W - 1)
        A = P[..., yb + 1, :][..., xb + 1] - P[..., yb + 1, :][..., xa]
        B = P[..., ya, :][..., xb + 1] - P[..., ya, :][..., xa]
        area = ((yb - ya + 1).double()[:, None] * (xb - xa + 1).double()[None, :])
        means.append((A - B) / area)
        mags.append((A.abs() + B.abs()) / area)
    return torch.stack(means, dim=-3), torch.stack(mags, dim=-3)


@pytest.mark.parametrize("shape", [(2, 3, 256, 256), (1, 1, 1024, 1024)])
def test_box_means_forward_interior_blocks(cuda, shape):
    """Sizes where most blocks of the forward kernel are interior (every
    output of the 32 x 64 block has the whole window of the largest radius and
    the row and column before it), so the branch-free path is what is checked.
    Each mean is compared with the four-corner rule evaluated in float64 on the
    kernel's own f32 SAT: the kernel does two f32 subtractions of corner
    values, one of the differences and a multiply by the f32 1/area^2, so
    |m - m64| <= 2 eps32 (|A| + |B|) / area + 4 eps32 |m64| per element.  The
    means are also checked end to end against float64 from x with the file's
    tolerance."""
    g = torch.Generator(device="cpu").manual_seed(31)
    x = torch.randn(shape, generator=g, dtype=torch.float32).to(cuda)
    radii = (3, 7, 15)
    S = sat_gb300.sat(x, torch.float32)
    m = api.box_means_from_sat(S, radii)
    m64, mag = _four_corner64(S, radii)
    err = (m.double() - m64).abs()
    bound = 2 * EPS32 * mag + 4 * EPS32 * m64.abs() + 1e-30
    assert bool((err <= bound).all()), float((err / bound).max())
    # the interior fraction really is the bulk: blocks of 32 columns x 64 rows
    H, W = shape[-2:]
    rmax = max(radii)
    bx = [x0 for x0 in range(0, W, 32) if x0 - rmax - 1 >= 0 and x0 + 31 + rmax <= W - 1]
    by = [y0 for y0 in range(0, H, 64) if y0 - rmax - 1 >= 0 and y0 + 63 + rmax <= H - 1]
    frac = len(bx) * len(by) / ((-(-W // 32)) * (-(-H // 64)))
    assert frac >= (0.8 if H >= 1024 else 0.35), frac  # 420 of 512 blocks at 1024^2, 12 of 32 at 256^2
    ref = box_means64(x, radii)
    smax = float(sat64(x.abs()).max())
    for k, r in enumerate(radii):
        tol = 4 * EPS32 * smax / (r + 1) ** 2 + 1e-7
        assert float((m[..., k, :, :].double() - ref[..., k, :, :]).abs().max()) <= tol, r


def test_box_means_huge_radius_is_the_whole_image(cuda):
    """A radius far beyond the image (up to INT_MAX) filters like radius
    max(H, W) - 1, whose window already covers the whole image."""
    x = torch.rand((2, 33, 70), device=cuda)
    S = sat_gb300.sat(x, torch.float32)
    m = api.box_means_from_sat(S, (69, 1 << 20, 2**31 - 1))
    full = x.double().mean(dim=(-2, -1))[:, None, None, None].expand(2, 3, 33, 70)
    assert torch.allclose(m.double(), full, atol=1e-5)
    assert torch.equal(m[:, 0], m[:, 1]) and torch.equal(m[:, 0], m[:, 2])


def test_box_means_single_radius_matches_full_sum(cuda):
    x = torch.rand((3, 17, 29), device=cuda)
    m = AG.box_filter_means(x, (100,))
    full = x.double().mean(dim=(-2, -1))
    assert torch.allclose(m[:, 0].double(), full[:, None, None].expand(3, 17, 29), atol=1e-6)


def _grads(x, radii, wts):
    xg = x.clone().requires_grad_(True)
    loss = (AG.box_filter_means(xg, radii) * wts).sum()
    loss.backward()
    x64 = x.double().clone().requires_grad_(True)
    loss64 = (box_means64(x64, radii) * wts.double()).sum()
    loss64.backward()
    return xg.grad, x64.grad


@pytest.mark.parametrize("shape", [(2, 3, 64, 64), (1, 1, 33, 150), (1, 1, 1, 9)])
def test_box_grad_vs_float64_cumsum(cuda, shape):
    g = torch.Generator(device="cpu").manual_seed(22)
    x = torch.randn(shape, generator=g).to(cuda)
    radii = (3, 7, 15)
    wts = torch.randn(shape[:-2] + (3,) + shape[-2:], generator=g).to(cuda)
    gx, g64 = _grads(x, radii, wts)
    tol = 1e-4 * max(1.0, float(g64.abs().max()))
    assert float((gx.double() - g64).abs().max()) <= tol


@pytest.mark.parametrize("shape,radii", [
    ((1, 2, 200, 333), (2, 9, 32)),   # interior blocks next to border blocks, ragged block edges
    ((1, 1, 130, 170), (33,)),        # a radius whose window spans most of the image: no interior block
    ((1, 1, 97, 131), (0, 1, 32, 70)),  # radius 0, and a radius wider than the image on one side
])
def test_box_grad_tiles_and_large_radii(cuda, shape, radii):
    g = torch.Generator(device="cpu").manual_seed(25)
    x = torch.randn(shape, generator=g).to(cuda)
    wts = torch.randn(shape[:-2] + (len(radii),) + shape[-2:], generator=g).to(cuda)
    gx, g64 = _grads(x, radii, wts)
    tol = 1e-4 * max(1.0, float(g64.abs().max()))
    assert float((gx.double() - g64).abs().max()) <= tol


def test_box_grad_central_fd(cuda):
    """64 x 64 crops: the kernel gradient against FP64 central differences
    (h = 1e-3) of the FP64 loss at 24 random pixels."""
    g = torch.Generator(device="cpu").manual_seed(23)
    x = torch.randn((1, 3, 64, 64), generator=g).to(cuda)
    radii = (3, 7, 15)
    wts = torch.randn((1, 3, 3, 64, 64), generator=g).to(cuda)
    xg = x.clone().requires_grad_(True)
    (AG.box_filter_means(xg, radii) * wts).sum().backward()
    grad = xg.grad.double()
    x64 = x.double()
    h = 1e-3
    rng = np.random.default_rng(23)
    pts = [(int(rng.integers(3)), int(rng.integers(64)), int(rng.integers(64))) for _ in range(20)]
    pts += [(0, 0, 0), (1, 63, 63), (2, 0, 63), (0, 63, 0)]
    fds, ours = [], []
    for c, i, j in pts:
        e = torch.zeros_like(x64)
        e[0, c, i, j] = h
        lp = float((box_means64(x64 + e, radii) * wts.double()).sum())
        lm = float((box_means64(x64 - e, radii) * wts.double()).sum())
        fds.append((lp - lm) / (2 * h))
        ours.append(float(grad[0, c, i, j]))
    fds, ours = np.array(fds), np.array(ours)
    assert np.max(np.abs(fds - ours)) <= 1e-4 * max(1.0, np.max(np.abs(fds)))


def test_sat_function_grad(cuda):
    g = torch.Generator(device="cpu").manual_seed(24)
    x = torch.randn((2, 45, 71), generator=g).to(cuda)
    w = torch.randn((2, 45, 71), generator=g).to(cuda)
    xg = x.clone().requires_grad_(True)
    (AG.sat(xg) * w).sum().backward()
    x64 = x.double().clone().requires_grad_(True)
    (sat64(x64) * w.double()).sum().backward()
    assert float((xg.grad.double() - x64.grad).abs().max()) <= 1e-4 * float(x64.grad.abs().max())


def test_box_layer_module(cuda):
    layer = AG.BoxFilter((1, 2))
    x = torch.randn((2, 8, 8), device=cuda, requires_grad=True)
    y = layer(x)
    assert y.shape == (2, 2, 8, 8)
    y.sum().backward()
    assert x.grad is not None and x.grad.shape == x.shape


def test_box_filter_rejects_bad_args(cuda):
    x = torch.randn((4, 4), device=cuda)
    s = api.sat(x)
    with pytest.raises(sat_gb300.SatError):
        api.box_means_from_sat(s, ())
    with pytest.raises(sat_gb300.SatError):
        api.box_means_from_sat(s, (1, 2, 3, 4, 5))
    with pytest.raises(sat_gb300.SatError):
        api.box_means_from_sat(s, (-1,))
    with pytest.raises(sat_gb300.SatError):
        api.box_means_from_sat(s.double(), (1,))


@pytest.mark.parametrize("shape,radii", [((2, 3, 256, 256), (3, 7, 15)), ((1, 2, 200, 333), (2, 9, 32)),
                                         ((1, 1, 97, 131), (0, 1, 32, 70)), ((3, 1, 1, 9), (1,)),
                                         ((2, 1, 1, 1), (0, 3)), ((1, 2, 300, 1), (4,)),
                                         ((1, 1, 129, 257), (1, 128))])
def test_grad_x_matches_separate_calls(cuda, shape, radii):
    """satgb_box_filter_bwd_x (adjoint gather into the output, reverse SAT in
    place) against the separate calls (adjoint into a dL/dSAT tensor, then the
    reverse SAT into a new tensor): to 1e-5 of the largest gradient, and both
    to the float64 autograd gradient."""
    g = torch.Generator(device="cpu").manual_seed(27)
    wts = torch.randn(shape[:-2] + (len(radii),) + shape[-2:], generator=g).to(cuda)
    gx = api.box_means_grad_x(wts, radii)
    two = sat_gb300.sat(api.box_means_adjoint(wts, radii), torch.float32, reverse=True)
    scale = max(1.0, float(two.abs().max()))
    assert float((gx - two).abs().max()) <= 1e-5 * scale
    x = torch.randn(shape, generator=g).to(cuda)
    x64 = x.double().clone().requires_grad_(True)
    (box_means64(x64, radii) * wts.double()).sum().backward()
    assert float((gx.double() - x64.grad).abs().max()) <= 1e-4 * max(1.0, float(x64.grad.abs().max()))


def test_grad_x_pitched_planes(cuda):
    """Gradient planes and the output as strided views (row pitch > width)."""
    g = torch.Generator(device="cpu").manual_seed(28)
    base = torch.randn((2, 2, 70, 96), generator=g).to(cuda)
    wts = base[..., :90]
    out_base = torch.full((2, 70, 100), float("nan"), device=cuda)
    out = out_base[..., :90]
    api.box_means_grad_x(wts, (2, 5), out=out)
    ref = sat_gb300.sat(api.box_means_adjoint(wts.contiguous(), (2, 5)), torch.float32, reverse=True)
    assert float((out - ref).abs().max()) <= 1e-5 * max(1.0, float(ref.abs().max()))
    assert bool(torch.isnan(out_base[..., 90:]).all())  # the row padding is never written


def window_error(r, area=True):
    """Bound of a window sum's rounding error over N(0, 1) inputs in the one-launch
    kernels, over the smallest clipped area: a column's running sum is updated twice a
    row for at most 256 rows (|V| <= 6 sqrt(2r + 1)) and enters 2r + 1 times; a prefix
    over 256 columns of them (|p| <= 96 sqrt(2r + 1)) carries at most 40 roundings."""
    eps, n = 2.0 ** -24, 2 * r + 1
    return eps * n ** 0.5 * (256 * 6 * n + 40 * 96) / (r + 1) ** 2


@pytest.mark.parametrize("shape,radii", [
    ((1, 2, 33, 224), (15,)),          # one whole block of 7 column groups
    ((2, 1, 129, 225), (3, 7, 15)),    # one column past it, one row past a strip, rows unaligned
    ((1, 1, 70, 448), (3, 7, 15)),     # two whole blocks
    ((1, 3, 40, 31), (0, 1, 2, 30)),   # narrower than a column group, windows wider than the plane
    ((1, 1, 300, 260), (11, 31)),      # aligned rows, last group not whole
    ((1, 1, 1, 500), (5,)), ((1, 1, 500, 1), (5,)), ((1, 1, 1, 1), (2,)),
    ((1, 2, 150, 300), (0, 15)), ((2, 1, 90, 100), (3, 3, 7)),  # radius 0; a radius twice
    ((1, 1, 140, 200), (64,)),         # too large for the one-launch kernels
])
def test_box_layer_windows(cuda, shape, radii):
    """Box means straight from the image and their gradient, at the edges of the
    kernels' blocks, strips and column groups, against float64."""
    g = torch.Generator(device="cpu").manual_seed(29)
    x = torch.randn(shape, generator=g).to(cuda).requires_grad_(True)
    w = torch.randn(shape[:-2] + (len(radii),) + shape[-2:], generator=g).to(cuda)
    m = AG.box_filter_means(x, radii)
    m.backward(w)
    x64 = x.detach().double().requires_grad_(True)
    m64 = box_means64(x64, radii)
    m64.backward(w.double())
    for k, r in enumerate(radii):
        err = float((m[..., k, :, :].double() - m64[..., k, :, :]).abs().max())
        assert err <= window_error(r), (r, err)
    err = float((x.grad.double() - x64.grad).abs().max())
    assert err <= sum(window_error(r) for r in radii), err


def test_box_layer_views_and_offsets(cuda):
    """Pitched planes and a base that is not 16-byte aligned, and outputs whose row
    padding stays untouched."""
    g = torch.Generator(device="cpu").manual_seed(30)
    base = torch.randn((3, 50, 260), generator=g).to(cuda)
    for x in (base[..., :256], base[..., 1:250], base[..., 4:260]):
        h, w = x.shape[-2:]
        out = torch.full((3, 2, h, w + 4), float("nan"), device=cuda)
        m = api.box_means(x, (3, 9), out=out[..., :w])
        ref = box_means64(x, (3, 9))
        for k, r in enumerate((3, 9)):
            assert float((m[:, k].double() - ref[:, k]).abs().max()) <= window_error(r)
        assert bool(torch.isnan(out[..., w:]).all())


def test_box_means_scratch_belongs_to_the_stream(cuda):
    """The scratch SAT of radii too large for one launch, on a stream that is not the current one: a block that
    the current stream still writes is not taken for it, and none of it is handed to the current
    stream while the call's launches are to come."""
    g = torch.Generator(device="cpu").manual_seed(41)
    x = torch.randn((6, 500, 600), generator=g).to(cuda)
    want = api.box_means(x, (80,))
    side = torch.cuda.Stream()
    torch.cuda.synchronize()
    for _ in range(3):
        old = torch.empty_like(x)
        torch.cuda._sleep(20_000_000)
        old.fill_(float("nan"))  # after the sleep
        del old
        with torch.cuda.stream(side):
            out = torch.zeros_like(want)
            torch.cuda._sleep(5_000_000)
        api.box_means(x, (80,), out=out, stream=side)
        late = [torch.full_like(x, float("nan")) for _ in range(4)]
        torch.cuda.synchronize()
        # (the SAT's sums may differ in their last bits: 2^-24 of |S| < 1e4 over windows of 41 x 41 at least)
        assert float((out - want).abs().max()) <= 1e-5
        assert all(bool(torch.isnan(t).all()) for t in late)


@pytest.mark.parametrize("radii", [(34,), (35,), (40,), (64,), (33, 34), (3, 7, 52), (50, 51, 52, 64), (64, 64, 64, 64)])
def test_box_means_without_a_scratch_sat(cuda, radii):
    """The C call takes every set of radii up to 64 without a scratch SAT; above, where the image is
    large enough for them, it says that it needs one."""
    import ctypes
    L = sat_gb300._lib.load()
    g = torch.Generator(device="cpu").manual_seed(43)
    x = torch.randn((2, 150, 170), generator=g).to(cuda)
    out = torch.empty((2, len(radii), 150, 170), device=cuda)

    def call(radii, width):
        d = api._box_desc(x[..., :width], out[..., :width], radii)
        dx, pitch, plane = d.d_sat, d.sat_pitch, d.sat_plane_stride
        d.d_sat = None
        return L.satgb_box_filter_fwd_x(ctypes.byref(d), dx, pitch, plane, torch.cuda.current_stream().cuda_stream)

    assert call(radii, 170) == sat_gb300._lib.OK
    ref = box_means64(x, radii)
    for k, r in enumerate(radii):
        assert float((out[:, k].double() - ref[:, k]).abs().max()) <= window_error(r)
    assert call(radii[:-1] + (65,), 170) == sat_gb300._lib.ERR_NOT_FOUND
    x = x[:, :65].contiguous()  # radius 65 and above are the whole image here: 64
    out = torch.empty((2, len(radii), 65, 170), device=cuda)
    assert call(radii[:-1] + (1000,), 60) == sat_gb300._lib.OK
    ref = box_means64(x[..., :60], radii[:-1] + (1000,))
    for k, r in enumerate(radii[:-1] + (64,)):
        assert float((out[:, k, :, :60].double() - ref[:, k]).abs().max()) <= window_error(min(r, 29))


@pytest.mark.parametrize("value", [float("inf"), float("-inf"), float("nan")])
@pytest.mark.parametrize("shape,radii", [((1, 300, 700), (3, 7, 15)), ((2, 150, 333), (5,)), ((1, 70, 64), (1, 9, 20, 31))])
def test_box_layer_infinities_spoil_no_more_than_the_sat_path(cuda, shape, radii, value):
    """An infinity or NaN in x spoils means whose window's last row and column are not before it only (those
    the SAT's four corners take it into), one in the means' gradient the pixels up to its window's last
    row and column only (the reverse SAT's); every other element is what it is without it, and every
    mean whose window holds it is not finite."""
    g = torch.Generator(device="cpu").manual_seed(47)
    x = torch.randn(shape, generator=g).to(cuda)
    w = torch.randn(shape[:-2] + (len(radii),) + shape[-2:], generator=g).to(cuda)
    H, W = shape[-2:]
    ys = torch.arange(H, device=cuda)[:, None]
    xs = torch.arange(W, device=cuda)[None, :]
    m64 = box_means64(x, radii)
    x64 = x.double().requires_grad_(True)
    (dx64,) = torch.autograd.grad(box_means64(x64, radii), x64, w.double())
    for r0, c0 in [(H // 2, W // 3), (0, 0), (H - 1, W - 1), (H // 3, W - 2), (H - 2, 5)]:
        x2 = x.clone()
        x2[0, r0, c0] = value
        m = api.box_means(x2, radii)
        for k, r in enumerate(radii):
            sound = ((ys + r).clamp(max=H - 1) < r0) | ((xs + r).clamp(max=W - 1) < c0)
            err = (m[0, k].double() - m64[0, k]).abs()
            assert bool((err[sound] <= window_error(r)).all()), (r0, c0, r)
            holds = ((ys - r0).abs() <= r) & ((xs - c0).abs() <= r)
            assert not bool(m[0, k][holds].isfinite().any()), (r0, c0, r)
        for k, r in enumerate(radii):
            w2 = w.clone()
            w2[0, k, r0, c0] = value
            dx = api.box_means_grad_x(w2, radii)
            sound = (ys > r0 + r) | (xs > c0 + r)
            err = (dx[0].double() - dx64[0]).abs()
            assert bool((err[sound] <= sum(window_error(q) for q in radii)).all()), (r0, c0, r)
            holds = ((ys - r0).abs() <= r) & ((xs - c0).abs() <= r)
            assert not bool(dx[0][holds].isfinite().any()), (r0, c0, r)
        for i in range(1, shape[0]):
            assert bool(m[i].isfinite().all()) and bool(dx[i].isfinite().all())


@pytest.mark.parametrize("shape,radii,scratch", [
    ((4, 64, 16), (15,), 0), ((4, 64, 33), (24,), 0), ((4, 64, 64), (31,), 0), ((4, 64, 128), (23, 60), 1),  # narrow planes
    ((2, 300, 300), (27,), 0), ((2, 300, 300), (3, 31), 0), ((2, 300, 300), (34,), 0), ((2, 300, 300), (35,), 1),  # few blocks
    ((600, 256, 256), (31,), 0), ((300, 256, 256), (3, 33), 0), ((300, 256, 256), (3, 34), 1), ((300, 256, 258), (35,), 1),
    ((300, 100, 256), (3, 5, 51), 0), ((300, 100, 256), (3, 5, 52), 1), ((60, 100, 1000), (3, 5, 17, 50), 0),
    ((60, 100, 1000), (3, 5, 17, 51), 1), ((600, 64, 36), (17, 31), 0),
])
def test_box_layer_both_ways(cuda, shape, radii, scratch):
    """Means and gradient on both sides of the choice between one launch and the way through the SAT: plane widths,
    radii, numbers of blocks.  Bounds: window_error, and through the SAT 4 roundings of its largest value over the smallest
    window, for the gradient 8 of the sum of all 4 |g| / area."""
    g = torch.Generator(device=cuda).manual_seed(67)
    x = torch.randn(shape, generator=g, device=cuda)
    w = torch.randn(shape[:1] + (len(radii),) + shape[1:], generator=g, device=cuda)
    out = torch.empty_like(w)
    import ctypes
    d = api._box_desc(x, out, radii)
    for d_sat, pitch in ((d.d_sat, d.sat_pitch), (None, 0), (1, 0)):  # neither is looked at
        d.d_sat, d.sat_pitch, d.sat_plane_stride = d_sat, pitch, 0
        assert sat_gb300._lib.load().satgb_box_filter_fwd_x_scratch(ctypes.byref(d)) == scratch
    api.box_means(x, radii, out=out)
    dx = api.box_means_grad_x(w, radii)
    H, W = shape[-2:]
    dtol = 0.0
    for n in (0, shape[0] // 2, shape[0] - 1):
        x64 = x[n].double().requires_grad_(True)
        m64 = box_means64(x64, radii)
        (dx64,) = torch.autograd.grad(m64, x64, w[n].double())
        smax = float(sat64(x[n]).abs().max())
        dtol = 0.0
        for k, r in enumerate(radii):
            area = (min(r, H - 1) + 1) * (min(r, W - 1) + 1)
            tol = window_error(min(r, max(H, W) - 1)) + 4 * EPS32 * smax / area + 1e-7
            err = float((out[n, k].double() - m64[k]).abs().max())
            assert err <= tol, (n, r, err, tol)
            dtol += window_error(min(r, max(H, W) - 1)) + 8 * EPS32 * 4 * float(w[n, k].abs().sum()) / area
        err = float((dx[n].double() - dx64).abs().max())
        assert err <= dtol, (n, err, dtol)


def test_box_layer_error_is_that_of_windows(cuda):
    """Rounding errors of the one-launch kernels stay those of window sums: over N(0, 1) planes of 1024^2 a column's running sum
    (|V| about sqrt(2r + 1)) takes 256 roundings, which add as a random walk, and a prefix of 256 of them a few more, 3e-7
    of a mean's unit in all (standard deviation, radius 3); bound: 17 of those, for the three radii's gradient sqrt(3)
    times as many.  Through the SAT, whose values reach thousands, the largest error is several times the bound."""
    g = torch.Generator(device="cpu").manual_seed(71)
    x = torch.randn((3, 1024, 1024), generator=g).to(cuda)
    w = torch.randn((3, 3, 1024, 1024), generator=g).to(cuda)
    radii = (3, 7, 15)
    x64 = x.double().requires_grad_(True)
    m64 = box_means64(x64, radii)
    (dx64,) = torch.autograd.grad(m64, x64, w.double())
    assert float((api.box_means(x, radii).double() - m64).abs().max()) <= 5e-6
    assert float((api.box_means_grad_x(w, radii).double() - dx64).abs().max()) <= 9e-6


def test_capture_without_a_workspace(cuda):
    """Calls that have a way without a look-back workspace are captured on a stream that has none, also at sizes where the
    other way is faster; on a stream that has one they take either."""
    g = torch.Generator(device=cuda).manual_seed(73)
    x = torch.randn((40, 300, 900), generator=g, device=cuda)
    w = torch.randn((40, 3, 300, 900), generator=g, device=cuda)
    c = torch.randint(0, 5, (8192, 640), generator=g, device=cuda).float()

    def calls():
        return (api.box_means(x, (4, 40, 50)), api.box_means_grad_x(w, (4, 30, 50)), api.box_means_grad_x(w[:, :1].contiguous(), (31,)),
                sat_gb300.scan_cols(c, torch.float32))

    want = calls()
    torch.cuda.synchronize()
    sat_gb300.release()  # (streams come from a pool)
    for warm in (False, True):
        side = torch.cuda.Stream()
        if warm:
            with torch.cuda.stream(side):
                calls()
            torch.cuda.synchronize()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=side):
            got = calls()
        for t in got:
            t.zero_()
        graph.replay()
        torch.cuda.synchronize()
        for a, b in zip(got, want):  # (the two ways round differently: 2^-24 of a SAT of thousands over windows of 16 at least)
            assert float((a - b).abs().max()) <= 2e-4
