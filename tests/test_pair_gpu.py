"""GEMMs and convolutions on pairs of CTAs at their edges: a second half past the last row, column and reduction remainders,
every operand order, every epilogue; convolutions with an odd number of pixel boxes."""
import pytest
import torch
import torch.nn.functional as F

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m,n,k", [(129, 136, 264), (256, 256, 320), (257, 264, 328), (385, 520, 1000), (3000, 200, 4096), (640, 19000, 272)])
@pytest.mark.parametrize("a_kmajor,b_kmajor", [(True, True), (True, False), (False, False)])
def test_pair_gemm(m, n, k, a_kmajor, b_kmajor):
    from eagersgd_b200.ops.gemm import check_error, gemm
    g = torch.Generator().manual_seed(m + n + k)
    pad = lambda v: (v + 7) // 8 * 8
    rnd = lambda r, c: torch.randn(r, pad(c), generator=g).cuda().to(torch.bfloat16)[:, :c]
    a, b = (rnd(m, k) if a_kmajor else rnd(k, m)), (rnd(n, k) if b_kmajor else rnd(k, n))
    af, bf = (a if a_kmajor else a.t()).float(), (b if b_kmajor else b.t()).float()
    ref = af @ bf.t()
    close = lambda x, y: (x.float() - y).norm() < 4e-3 * y.norm()
    out = torch.empty(m, pad(n), device="cuda")[:, :n]
    assert close(gemm(a, b, a_kmajor=a_kmajor, b_kmajor=b_kmajor, out=out), ref)
    if n <= 600:
        acc = torch.ones(m, pad(n), device="cuda")[:, :n]
        gemm(a, b, a_kmajor=a_kmajor, b_kmajor=b_kmajor, out=acc, splits=3, accumulate=True)
        assert close(acc - 1.0, ref)
        res, s, q = rnd(m, n), torch.zeros(n, device="cuda"), torch.zeros(n, device="cuda")
        y = gemm(a, b, a_kmajor=a_kmajor, b_kmajor=b_kmajor, out=torch.empty(m, pad(n), device="cuda", dtype=torch.bfloat16)[:, :n],
                 residual=res, col_sum=s, col_sqsum=q)
        assert close(y, ref + res.float())
        assert torch.allclose(s, y.float().sum(0), rtol=1e-3, atol=0.2) and torch.allclose(q, (y.float() ** 2).sum(0), rtol=1e-3)
    check_error(a.device)


@pytest.mark.parametrize("n,ci,h,co,k,stride", [(3, 128, 7, 256, 3, 1), (200, 64, 14, 256, 3, 1), (310, 256, 7, 512, 3, 1), (37, 320, 28, 264, 3, 2),
                                                (75, 256, 14, 256, 3, 2), (2, 64, 150, 256, 3, 1)])
def test_pair_convolution(n, ci, h, co, k, stride):
    from eagersgd_b200.ops import functional as ops
    from eagersgd_b200.ops.gemm import check_error
    g = torch.Generator().manual_seed(n + ci + h)
    rnd = lambda *s: torch.randn(*s, generator=g).cuda().to(torch.bfloat16).contiguous(memory_format=torch.channels_last)
    x, w = rnd(n, ci, h, h).requires_grad_(), (rnd(co, ci, k, k) * 0.05).requires_grad_()
    y, st = ops.conv2d(x, w, stride, k // 2, want_stats=True)
    xr, wr = x.detach().float().requires_grad_(), w.detach().float().requires_grad_()
    yr = F.conv2d(xr, wr, None, stride, k // 2)
    dy = rnd(*yr.shape)
    y.backward(dy)
    yr.backward(dy.float())
    check_error(y.device)
    for a, b in ((y, yr), (x.grad, xr.grad), (w.grad, wr.grad)):
        assert (a.float() - b).norm() < 6e-3 * b.norm()
    yf = y.detach().float()
    assert torch.allclose(st[1], (yf * yf).sum((0, 2, 3)), rtol=1e-3)
