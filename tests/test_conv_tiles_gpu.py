"""3x3 layers at the edges of how their work is cut: pairs of CTAs with an odd box left over, resident and streamed filters, one to
three taps a CTA in the weight gradient; and residual panels that are asked for ahead.  Against fp64 PyTorch."""
import pytest
import torch
import torch.nn.functional as F

pytestmark = pytest.mark.gpu


def _cl(t):
    return t.contiguous(memory_format=torch.channels_last)


def _close(got, ref, magnitude):
    """bf16 rounding of the result (2^-9), and fp32 sums: an error of 2^-24 of the magnitudes for each of up to 2^5 roundings in a
    row of the accumulation, with a margin of four."""
    assert ((got.double() - ref).abs() <= ref.abs() * 2 ** -8 + magnitude * 2 ** -17).all()


# n, h, w, channels: pairs with 175, 91 and 76 boxes, a width that fills no tile, two blocks of input channels; tiles of one CTA with all
# filters there; too few boxes for 128 columns; weight gradients with 1, 2 and 3 taps,
# and with all nine (odd rows, 40 output channels, small images)
@pytest.mark.parametrize("n,h,w,cin,cout", [(25, 28, 28, 128, 128), (13, 28, 28, 128, 128), (19, 28, 28, 64, 128), (31, 20, 22, 192, 128),
                                            (5, 56, 56, 64, 64), (9, 28, 28, 64, 96), (1, 28, 28, 128, 128), (40, 8, 8, 64, 64),
                                            (64, 56, 56, 64, 64), (24, 56, 56, 64, 40), (1024, 8, 8, 64, 64), (40, 34, 40, 64, 64), (24, 14, 14, 256, 256), (8, 7, 7, 512, 512)])
def test_3x3(n, h, w, cin, cout):
    from eagersgd_b200.ops import functional as ops
    from eagersgd_b200.ops.gemm import check_error
    g = torch.Generator().manual_seed(n + h + w)
    rnd = lambda *s: _cl(torch.randn(*s, generator=g)).bfloat16().cuda()
    x, wt, dy = rnd(n, cin, h, w), (rnd(cout, cin, 3, 3) / 8).requires_grad_(), rnd(n, cout, h, w)
    xg = x.clone(memory_format=torch.preserve_format).requires_grad_()
    y, stats = ops.conv2d(xg, wt, 1, 1, want_stats=True)
    y.backward(dy)
    check_error(y.device)
    xd, wd, dd = x.double(), wt.detach().double(), dy.double()
    _close(y, F.conv2d(xd, wd, None, 1, 1), F.conv2d(xd.abs(), wd.abs(), None, 1, 1))
    yd = y.double()
    for got, terms in ((stats[0], yd), (stats[1], yd * yd)):
        assert ((got.double() - terms.sum((0, 2, 3))).abs() <= terms.abs().sum((0, 2, 3)) * 2 ** -16).all()
    dx = lambda a, b: torch.nn.grad.conv2d_input(x.shape, a, b, 1, 1)
    dw = lambda a, b: torch.nn.grad.conv2d_weight(a, wt.shape, b, 1, 1)
    _close(xg.grad, dx(wd, dd), dx(wd.abs(), dd.abs()))
    _close(wt.grad, dw(xd, dd), dw(xd.abs(), dd.abs()))


# one tile, several tiles of a CTA with rows left over, columns that fill no panel, pairs; reductions split over clusters of 8, 4 and 2
# CTAs, with shares that are empty and columns that fill no tile
@pytest.mark.parametrize("n,h,cin,cout,k", [(1, 7, 64, 256, 1), (33, 31, 64, 256, 1), (130, 14, 128, 200, 1), (50, 14, 512, 1024, 1), (70, 14, 64, 136, 3),
                                            (25, 28, 128, 128, 3), (1, 7, 512, 512, 3), (1, 9, 128, 200, 3),
                                            (1, 14, 1024, 256, 1), (2, 14, 256, 256, 3), (8, 14, 256, 256, 3), (3, 13, 1096, 72, 1), (1, 130, 192, 64, 3)])
def test_residual(n, h, cin, cout, k):
    from eagersgd_b200.ops import functional as ops
    g = torch.Generator().manual_seed(n + h + k)
    rnd = lambda *s: _cl(torch.randn(*s, generator=g)).bfloat16().cuda()
    x, wt, res = rnd(n, cin, h, h), rnd(cout, cin, k, k) / 8, rnd(n, cout, h, h)
    coef = torch.rand(2, cout, generator=g).cuda() + 0.5
    y = ops.conv_bn_eval(x, wt, 1, k // 2, coef, True, res)
    conv = lambda a, b: F.conv2d(a, b, None, 1, k // 2)
    scale, shift = coef.double().view(2, 1, cout, 1, 1)
    xd, wd = x.double(), wt.double()
    _close(y, F.relu(conv(xd, wd) * scale + shift + res.double()), conv(xd.abs(), wd.abs()) * scale + shift + res.double().abs())


# odd sizes, rows in two boxes, one image and many, channels that fill no block
@pytest.mark.parametrize("n,h,w,cin,cout", [(1, 7, 9, 64, 256), (5, 15, 31, 72, 40), (2, 5, 300, 64, 128), (130, 8, 8, 256, 512), (1, 1, 1, 8, 8), (1, 13, 15, 1024, 512)])
def test_strided_1x1_inference(n, h, w, cin, cout):
    from eagersgd_b200.ops import functional as ops
    g = torch.Generator().manual_seed(n + h + w)
    rnd = lambda *s: _cl(torch.randn(*s, generator=g)).bfloat16().cuda()
    x, wt = rnd(n, cin, h, w), rnd(cout, cin, 1, 1) / 8
    coef = torch.rand(2, cout, generator=g).cuda() + 0.5
    y = ops.conv_bn_eval(x, wt, 2, 0, coef, True, None)
    conv = lambda a, b: F.conv2d(a, b, None, 2)
    scale, shift = coef.double().view(2, 1, cout, 1, 1)
    xd, wd = x.double(), wt.double()
    _close(y, F.relu(conv(xd, wd) * scale + shift), conv(xd.abs(), wd.abs()) * scale + shift)
