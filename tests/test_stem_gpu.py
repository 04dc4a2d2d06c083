"""The 7x7 / 2 stem of RGB images straight from the images, forward and filter gradient, against fp64 PyTorch."""
import pytest
import torch
import torch.nn.functional as F

pytestmark = pytest.mark.gpu

# n, h, w: one band of an image, the narrowest rows, rows of 1.25 tiles, the widest; bands of two rows (few images) and of eight
# (from six bands an SM on), the last with tiles that the band does not fill; then sizes that keep the matrix of windows
SHAPES = [(1, 16, 8), (2, 32, 40), (1, 16, 320), (3, 224, 224), (1, 48, 16), (900, 16, 8), (450, 32, 24), (230, 64, 72), (2, 16, 328), (2, 24, 24), (2, 32, 20), (2, 33, 40)]


def _cl(t):
    return t.contiguous(memory_format=torch.channels_last)


def _case(n, h, w):
    g = torch.Generator().manual_seed(n + h + w)
    x, wt = _cl(torch.randn(n, 3, h, w, generator=g)).bfloat16().cuda(), _cl(torch.randn(64, 3, 7, 7, generator=g) * 0.1).bfloat16().cuda()
    return x, wt, F.conv2d(x.double(), wt.double(), None, 2, 3)


def _close(got, ref, magnitude):
    """bf16 rounding of the result (2^-9), and fp32 sums: an error of 2^-24 of the magnitudes for each of up to 2^5 roundings in a
    row of the accumulation, with a margin of four."""
    assert ((got.double() - ref).abs() <= ref.abs() * 2 ** -8 + magnitude * 2 ** -17).all()


@pytest.mark.parametrize("n,h,w", SHAPES)
def test_training(n, h, w):
    from eagersgd_b200.ops import functional as ops
    from eagersgd_b200.ops.gemm import check_error
    x, wt, ref = _case(n, h, w)
    images, param = x.clone(memory_format=torch.preserve_format), wt.clone(memory_format=torch.preserve_format).requires_grad_()
    y, stats = ops.conv2d(images, param, 2, 3, want_stats=True)
    images.fill_(float("nan"))                       # the next batch arrives before the backward pass
    _close(y, ref, F.conv2d(x.double().abs(), wt.double().abs(), None, 2, 3))
    yd = y.double()
    # fp32 sums in some order: the random walk of their roundings stays far below 2^-16 of the sum of magnitudes
    for got, terms in ((stats[0], yd), (stats[1], yd * yd)):
        assert ((got.double() - terms.sum((0, 2, 3))).abs() <= terms.abs().sum((0, 2, 3)) * 2 ** -16).all()
    dy = torch.randn(ref.shape, generator=torch.Generator().manual_seed(1)).cuda().bfloat16()
    y.backward(_cl(dy))
    check_error(y.device)
    grad = lambda a, b: torch.nn.grad.conv2d_weight(a, wt.shape, b, 2, 3)
    _close(param.grad, grad(x.double(), dy.double()), grad(x.double().abs(), dy.double().abs()))


@pytest.mark.parametrize("n,h,w", SHAPES[:6])
def test_inference(n, h, w):
    from eagersgd_b200.ops import functional as ops
    x, wt, ref = _case(n, h, w)
    x[0, 1, 5, 3] = float("inf")
    g = torch.Generator().manual_seed(7)
    gamma, beta, mean, var = (torch.rand(64, generator=g).cuda() + 0.5 for _ in range(4))
    coef = ops.bn_coefficients([(gamma, beta, mean, var)], {})[0]
    y = ops.conv_bn_eval(x, wt, 2, 3, coef, True)
    scale, shift = coef.double().view(2, 1, 64, 1, 1)
    seen = F.conv2d(torch.isinf(x).double(), torch.ones_like(wt).double(), None, 2, 3) > 0        # windows with the infinity
    want = F.relu(ref * scale + shift)
    big = F.conv2d(torch.nan_to_num(x.double(), posinf=1.0).abs(), wt.double().abs(), None, 2, 3) * scale.abs() + shift.abs()
    _close(torch.where(seen, 0.0, y.double()), torch.where(seen, 0.0, want), big)
    assert not torch.isfinite(y[seen]).any() or (y[seen & torch.isfinite(y)] == 0).all()          # +inf, or -inf behind the ReLU
