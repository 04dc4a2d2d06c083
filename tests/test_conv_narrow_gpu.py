"""Convolutions of 16, 32 and 64 channels (rows in shared memory, ldmatrix) against fp32 PyTorch: image sizes that fill no
tile, several images per tile, one image, stride 2, and the shortcut's gradient in the data gradient."""
import pytest
import torch
import torch.nn.functional as F

pytestmark = pytest.mark.gpu


def _cl(t):
    return t.contiguous(memory_format=torch.channels_last)


@pytest.mark.parametrize("n,ci,h,w,co,stride", [(128, 16, 32, 32, 16, 1), (1, 16, 32, 32, 16, 1), (3, 16, 5, 7, 16, 1), (37, 16, 32, 32, 32, 2),
                                                (5, 16, 9, 11, 32, 2), (100, 32, 16, 16, 32, 1), (2, 32, 3, 3, 32, 1), (100, 32, 16, 16, 64, 2),
                                                (7, 32, 1, 1, 32, 1), (100, 64, 8, 8, 64, 1), (1, 64, 8, 8, 64, 1), (9, 64, 13, 6, 64, 1),
                                                (2, 16, 224, 224, 16, 1), (600, 64, 8, 8, 64, 1), (64, 64, 8, 8, 64, 1), (65, 64, 8, 8, 64, 1)])
def test_conv_narrow(n, ci, h, w, co, stride):
    from eagersgd_b200.ops import functional as ops
    from eagersgd_b200.ops.gemm import check_error
    g = torch.Generator().manual_seed(n + ci + h + co)
    rnd = lambda *s: torch.randn(*s, generator=g).cuda()
    x = _cl(rnd(n, ci, h, w)).bfloat16().requires_grad_()
    wt = _cl(rnd(co, ci, 3, 3) / (9 * ci) ** 0.5).bfloat16().requires_grad_()
    y, st, tap = ops.conv2d(x, wt, stride, 1, want_stats=True, tap_input=True)
    xr, wr = x.detach().float().requires_grad_(), wt.detach().float().requires_grad_()
    yr = F.conv2d(xr, wr, None, stride, 1)
    assert (y.float() - yr).norm() < 4e-3 * yr.norm()
    yf = y.detach().float()
    assert torch.allclose(st[0], yf.sum((0, 2, 3)), rtol=1e-3, atol=1e-2 * yf.numel() ** 0.5 / co)
    assert torch.allclose(st[1], (yf * yf).sum((0, 2, 3)), rtol=1e-3)
    dy, d2 = _cl(rnd(*yr.shape)).bfloat16(), _cl(rnd(n, ci, h, w)).bfloat16()
    ((y * dy).sum() + (tap * d2).sum()).backward()
    ((yr * dy.float()).sum() + (xr * d2.float()).sum()).backward()
    check_error(y.device)
    assert (x.grad.float() - xr.grad).norm() < 6e-3 * xr.grad.norm()
    assert (wt.grad.float() - wr.grad).norm() < 6e-3 * wr.grad.norm()


@pytest.mark.parametrize("n,ci,h,w,co,stride", [(700, 16, 32, 32, 16, 1), (1500, 32, 16, 16, 32, 1), (400, 16, 33, 31, 32, 2), (300, 16, 5, 3, 32, 2),
                                                (149, 32, 1, 17, 32, 1), (147, 16, 1, 1, 16, 1), (90, 32, 3, 50, 64, 2), (37, 64, 2, 29, 64, 1)])
def test_runs_of_rows(n, ci, h, w, co, stride):
    """Runs of output rows that are longer than shared memory (several passes), that span many images, and that are one row."""
    test_conv_narrow(n, ci, h, w, co, stride)
