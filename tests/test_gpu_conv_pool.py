"""Convolution / pooling kernels against plain fp32 torch references (forward and every gradient)."""
import pytest
import torch
import torch.nn.functional as tF

from momijo_b200.ops import conv as cv

pytestmark = pytest.mark.gpu


def _close(a, b, tol, fro):
    a, b = a.float(), b.float()
    err = ((a - b).abs().max() / b.abs().max().clamp_min(1e-6)).item()
    ferr = ((a - b).norm() / b.norm().clamp_min(1e-6)).item()
    assert err < tol and ferr < fro, (err, ferr)


def _ref(fn, tensors, dy):
    """fp32 CPU reference values and gradients."""
    ts = [t.detach().float().cpu().requires_grad_(True) for t in tensors]
    y = fn(*ts)
    y.backward(dy.float().cpu())
    return y, [t.grad for t in ts]


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("N,C,H,W,OC,k,s,p,d,g", [
    (2, 3, 17, 19, 8, 3, 1, 1, 1, 1), (2, 8, 16, 16, 16, 3, 2, 1, 1, 1), (1, 4, 12, 12, 6, 5, 1, 2, 2, 2),
    (2, 6, 9, 9, 6, 3, 1, 1, 1, 6), (2, 16, 14, 14, 32, 3, 1, 1, 1, 1)])
def test_conv2d_forward_and_gradients(dtype, N, C, H, W, OC, k, s, p, d, g):
    torch.manual_seed(0)
    x = torch.randn(N, C, H, W, device="cuda").to(dtype).requires_grad_(True)
    w = (torch.randn(OC, C // g, k, k, device="cuda") * 0.2).to(dtype).requires_grad_(True)
    b = torch.randn(OC, device="cuda").to(dtype).requires_grad_(True)
    y = cv.conv2d(x, w, b, s, p, d, g)
    dy = torch.randn_like(y)
    y.backward(dy)
    yr, (gx, gw, gb) = _ref(lambda a, c, e: tF.conv2d(a, c, e, s, p, d, g), (x, w, b), dy)
    tol, fro = (1e-4, 1e-5) if dtype == torch.float32 else (3e-2, 1e-2)
    _close(y, yr.cuda(), tol, fro)
    _close(x.grad, gx.cuda(), tol, fro)
    _close(w.grad, gw.cuda(), tol, fro)
    _close(b.grad, gb.cuda(), tol, fro)


def test_im2col_col2im_match_unfold_fold():
    torch.manual_seed(1)
    x = torch.randn(2, 5, 11, 13, device="cuda")
    cols = cv.im2col(x, (3, 2), (2, 1), (1, 0))
    ref = tF.unfold(x, (3, 2), padding=(1, 0), stride=(2, 1)).transpose(1, 2).reshape(-1, 5 * 6)
    assert torch.equal(cols, ref)
    back = cv.col2im(cols, x.shape, (3, 2), (2, 1), (1, 0))
    c = ref.reshape(2, -1, 30).transpose(1, 2)
    _close(back, tF.fold(c, (11, 13), (3, 2), padding=(1, 0), stride=(2, 1)), 1e-5, 1e-6)


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("k,s,p", [(2, 2, 0), (3, 1, 1), (3, 2, 1)])
def test_pooling_and_deterministic_backward(dtype, k, s, p):
    torch.manual_seed(2)
    x = torch.randn(2, 4, 15, 14, device="cuda").to(dtype).requires_grad_(True)
    for fn, ref in ((lambda t: cv.max_pool2d(t, k, s, p), lambda t: tF.max_pool2d(t, k, s, p)),
                    (lambda t: cv.avg_pool2d(t, k, s, p), lambda t: tF.avg_pool2d(t, k, s, p, count_include_pad=False))):
        x.grad = None
        y = fn(x)
        dy = torch.randn_like(y)
        y.backward(dy)
        g1 = x.grad.clone()
        yr, (gx,) = _ref(ref, (x,), dy)
        tol, fro = (1e-5, 1e-6) if dtype == torch.float32 else (2e-2, 1e-2)
        _close(y, yr.cuda(), tol, fro)
        _close(g1, gx.cuda(), tol, fro)
        x.grad = None
        fn(x).backward(dy)
        assert torch.equal(g1, x.grad)     # overlapping windows, no atomics: bitwise reproducible
    y, idx = cv.max_pool2d(x, k, s, p, return_indices=True)
    yr, ir = tF.max_pool2d(x.detach().float(), k, s, p, return_indices=True)
    assert torch.equal(idx, ir)


def test_conv_transpose2d():
    torch.manual_seed(3)
    x = torch.randn(2, 6, 7, 9, device="cuda", requires_grad=True)
    w = (torch.randn(6, 4, 3, 3, device="cuda") * 0.2).requires_grad_(True)
    b = torch.randn(4, device="cuda", requires_grad=True)
    y = cv.conv_transpose2d(x, w, b, 2, 1)
    dy = torch.randn_like(y)
    y.backward(dy)
    yr, (gx, gw, gb) = _ref(lambda a, c, e: tF.conv_transpose2d(a, c, e, 2, 1), (x, w, b), dy)
    _close(y, yr.cuda(), 1e-4, 1e-5)
    _close(x.grad, gx.cuda(), 1e-4, 1e-5)
    _close(w.grad, gw.cuda(), 1e-4, 1e-5)
    _close(b.grad, gb.cuda(), 1e-4, 1e-5)


def test_layers_use_native_kernels():
    from momijo_b200 import _C
    from momijo_b200.learn.nn.conv import Conv2d, MaxPool2d

    conv = Conv2d(3, 8, 3, pad=(1, 1)).cuda()
    pool = MaxPool2d(2, stride=(2, 2))
    before = _C.launches
    y = pool(conv(torch.randn(2, 3, 16, 16, device="cuda")))
    y.sum().backward()
    assert _C.launches - before >= 5
    assert conv.weight.grad is not None and y.shape == (2, 8, 8, 8)


@pytest.mark.parametrize("N,C,H,W,OC,k,s,p,d,g", [
    (1, 1, 5, 7, 1, 3, 1, 1, 1, 1),          # one filter, fewer positions than a tile
    (2, 3, 13, 11, 17, 5, 2, 2, 1, 1),       # a row past a 16-channel tile; strided classes of unequal size
    (1, 33, 9, 9, 65, 3, 1, 1, 1, 1),        # a channel past a 32- and a 64-channel tile
    (3, 16, 12, 10, 48, 1, 3, 0, 1, 1),      # stride larger than the kernel: classes that meet no tap
    (2, 8, 15, 14, 12, 3, 2, 2, 2, 2),       # dilation and stride share a factor; groups
    (1, 4, 20, 20, 4, 3, 1, 1, 1, 4),        # depthwise stays with the direct kernels
    (2, 5, 6, 6, 7, (1, 5), (4, 1), (0, 2), (1, 1), 1),
    (16, 64, 60, 60, 64, 3, 1, 1, 1, 1),     # several slices and full tiles
])
def test_conv2d_tile_edges_against_64_bits(N, C, H, W, OC, k, s, p, d, g):
    kh, kw = (k, k) if isinstance(k, int) else k
    gen = torch.Generator(device="cuda").manual_seed(5)
    r = lambda *shape: torch.randn(*shape, generator=gen, device="cuda").requires_grad_()
    x, w, b = r(N, C, H, W), r(OC, C // g, kh, kw), r(OC)
    y = cv.conv2d(x, w, b, s, p, d, g)
    dy = torch.randn_like(y)
    got = [y, *torch.autograd.grad(y, [x, w, b], dy)]
    x64, w64, b64 = (v.detach().double().requires_grad_() for v in (x, w, b))
    y64 = tF.conv2d(x64, w64, b64, s, p, d, g)
    want = [y64, *torch.autograd.grad(y64, [x64, w64, b64], dy.double())]
    # rounding of a sum of n products grows like sqrt(n) * 2^-24 of its norm; 4x for the spread of one draw
    terms = [C // g * kh * kw, OC // g * kh * kw, N * y.shape[2] * y.shape[3], N * y.shape[2] * y.shape[3]]
    for a, e, n in zip(got, want, terms):
        assert float((a.double() - e).norm()) <= 4 * 2.0 ** -24 * (n + 1) ** 0.5 * float(e.norm()) + 1e-12


@pytest.mark.parametrize("N,C,H,W,OC,k,s,p,d", [(2, 7, 9, 11, 16, 3, 1, 1, 1), (1, 16, 13, 8, 56, 3, 2, 1, 1),
                                                (2, 24, 10, 10, 72, (3, 1), 1, 1, 2), (1, 64, 33, 5, 48, 1, 1, 0, 1),
                                                (1, 16, 13, 8, 49, 3, 2, 1, 1), (2, 9, 7, 10, 17, 3, 1, 1, 1),
                                                (4, 24, 55, 57, 16, 3, 1, 1, 1)])     # patches of 64 columns to a warp
@pytest.mark.parametrize("direct_dx", [False, True])
def test_bf16_lowered_convolution(monkeypatch, direct_dx, N, C, H, W, OC, k, s, p, d):
    """The patch matrix (exact: it only moves values) and both ways of the input gradient; results rounded to bf16. The product takes filters in eights only: 49 and 17 stay direct."""
    monkeypatch.setattr(cv, "_direct_dx", lambda *shape: direct_dx)
    kh, kw = (k, k) if isinstance(k, int) else k
    gen = torch.Generator(device="cuda").manual_seed(4)
    r = lambda *shape: torch.randn(*shape, generator=gen, device="cuda").bfloat16()
    x, w = r(N, C, H, W), r(OC, C, kh, kw)
    for dtype in (torch.bfloat16, torch.float32):
        K = C * kh * kw
        for ldc in (K, (K + 7) // 8 * 8, K + 3):
            cols = cv.im2col(x.to(dtype), (kh, kw), s, p, d, ldc=ldc)
            want = tF.unfold(x.float(), (kh, kw), d, p, s).transpose(1, 2).reshape(-1, K)
            assert torch.equal(cols[:, :K].float(), want) and not cols[:, K:].any()
    x.requires_grad_(), w.requires_grad_()
    y = cv.conv2d(x, w, None, s, p, d)
    dy = r(*y.shape)
    got = [y, *torch.autograd.grad(y, [x, w], dy)]
    x64, w64 = (v.detach().double().requires_grad_() for v in (x, w))
    y64 = tF.conv2d(x64, w64, None, s, p, d)
    for a, e in zip(got, [y64, *torch.autograd.grad(y64, [x64, w64], dy.double())]):
        # 2^-9 for the result's rounding; the product route rounds k * k terms of each gradient as well
        assert float((a.double() - e).norm()) <= 2.0 ** -7.5 * float(e.norm())


def _taps_by_slices(x, w, dy, s, p, d):
    """y, dx and dw of a convolution as sums over the taps that lie inside the image, in 64 bits: nothing is multiplied
    by a padding zero."""
    x, w, dy = x.double().cpu(), w.double().cpu(), dy.double().cpu()
    y, dx, dw = torch.zeros_like(dy), torch.zeros_like(x), torch.zeros_like(w)
    (OH, OW), (H, W) = dy.shape[2:], x.shape[2:]
    for kh in range(w.shape[2]):
        for kw in range(w.shape[3]):
            rows = [(o, o * s - p + kh * d) for o in range(OH) if 0 <= o * s - p + kh * d < H]
            cols = [(o, o * s - p + kw * d) for o in range(OW) if 0 <= o * s - p + kw * d < W]
            if not rows or not cols:
                continue
            o = (..., slice(rows[0][0], rows[-1][0] + 1), slice(cols[0][0], cols[-1][0] + 1))
            i = (..., slice(rows[0][1], rows[-1][1] + 1, s), slice(cols[0][1], cols[-1][1] + 1, s))
            y[o] += (x[i][:, None] * w[None, :, :, kh, kw, None, None]).sum(2)
            dx[i] += (dy[o][:, :, None] * w[None, :, :, kh, kw, None, None]).sum(1)
            dw[:, :, kh, kw] += (dy[o][:, :, None] * x[i][:, None]).sum((0, 3, 4))
    return y, dx, dw


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("H,s,p,d", [(14, 1, 1, 1), (37, 2, 1, 1), (37, 1, 2, 2), (60, 3, 2, 1), (40, 1, 1, 1)])
def test_infinite_values_meet_only_taps_inside_the_image(dtype, H, s, p, d):
    gen = torch.Generator(device="cuda").manual_seed(6)
    N, C, OC, k = 3, 4, 5, 3
    OH = (H + 2 * p - d * (k - 1) - 1) // s + 1
    r = lambda *shape: torch.randn(*shape, generator=gen, device="cuda").to(dtype)
    x, w, dy = r(N, C, H, H), r(OC, C, k, k), r(N, OC, OH, OH)
    inf_w = w.clone()
    inf_w[2, 1, 0, 2] = float("inf")           # a corner tap: outside the image for a row and a column of pixels
    inf_dy = dy.clone()
    inf_dy[1, 3, 0, OH - 1] = float("-inf")    # a corner pixel: some of its taps are outside
    for wt, grad in ((inf_w, dy), (w, inf_dy)):
        xg, wg = x.clone().requires_grad_(), wt.clone().requires_grad_()
        y = cv.conv2d(xg, wg, None, s, p, d)
        got = [y, *torch.autograd.grad(y, [xg, wg], grad)]
        for a, e in zip(got, _taps_by_slices(x, wt, grad, s, p, d)):
            a, fin = a.detach().double().cpu(), torch.isfinite(e)
            assert torch.equal(torch.isnan(a), torch.isnan(e)) and torch.equal(a[~fin], e[~fin])
            # sums of up to n products: 4 * 2^-24 * sqrt(n) of the norm, and 2^-8 for a bf16 result
            tol = 4 * 2.0 ** -24 * (N * OH * OH) ** 0.5 + (2.0 ** -8 if dtype == torch.bfloat16 else 0.0)
            assert float((a - e)[fin].norm()) <= tol * float(e[fin].norm())


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("N,C,spatial", [(1, 1, 1), (257, 8, 1), (300, 3, 7), (5, 300, 33), (3, 5, 257), (9, 2, 2049),
                                         (40, 2, 1024), (2, 64, 9000)])
def test_channel_sums(dtype, N, C, spatial):
    """Fewer positions than threads and more, one block to a channel and several, against 64 bits."""
    gen = torch.Generator(device="cuda").manual_seed(7)
    dy = torch.randn(N, C, spatial, generator=gen, device="cuda").to(dtype)
    got, want = cv._channel_sum(dy, N, C, spatial).double(), dy.double().sum((0, 2))
    # chains of at most a few hundred additions, of sums no larger than the values' own sum
    tol = 2.0 ** -24 * 32 * dy.double().abs().sum((0, 2)) + (2.0 ** -8 * want.abs() if dtype == torch.bfloat16 else 0)
    assert ((got - want).abs() <= tol).all()
