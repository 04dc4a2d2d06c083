"""The batch-norm backward whose reduction and ReLU mask sit in the epilogue of the next convolution's data gradient, against
fp32 autograd: tile remainders, every kernel family that has the epilogue, shortcuts on both sides, and somebody listening."""
import pytest
import torch
import torch.nn.functional as F

pytestmark = pytest.mark.gpu


# channels, outputs of the convolution, filter, image, batch
@pytest.mark.parametrize("c,k,r,h,n", [(64, 72, 1, 5, 3), (128, 64, 1, 16, 2), (256, 64, 1, 28, 3), (1024, 256, 1, 7, 5), (64, 64, 3, 30, 65),
                                       (128, 128, 3, 28, 2), (256, 256, 3, 14, 3), (512, 512, 3, 7, 3), (16, 16, 3, 13, 3),
                                       (32, 32, 3, 16, 9), (64, 64, 3, 8, 2), (24, 40, 3, 9, 2), (64, 64, 3, 140, 1)])
@pytest.mark.parametrize("residual,relu,hook", [(False, True, False), (True, True, False), (True, False, False), (True, True, True)])
def test_fused_batch_norm_backward(c, k, r, h, n, residual, relu, hook):
    from eagersgd_b200 import _build
    from eagersgd_b200.ops import functional as ops
    from eagersgd_b200.ops.gemm import check_error
    ext = _build.load_torch()
    gen = torch.Generator().manual_seed(c * 100 + h)
    rnd = lambda *s: torch.randn(*s, generator=gen).cuda().to(torch.bfloat16).contiguous(memory_format=torch.channels_last)
    y, res, g_out, g_tap = rnd(n, c, h, h), rnd(n, c, h, h), rnd(n, k, h, h), rnd(n, c, h, h)
    w = (rnd(k, c, r, r) * 0.1).requires_grad_()
    gamma = (torch.rand(c, generator=gen) + 0.5).cuda().requires_grad_()
    beta = (torch.randn(c, generator=gen) * 0.3).cuda().requires_grad_()
    y.requires_grad_()
    res.requires_grad_()
    params = [gamma, beta, w]
    acc = [torch.zeros_like(p, dtype=torch.float32, memory_format=torch.preserve_format) for p in params]
    sinks = ext.GradSinks([3], lambda bucket: None)
    for p, a in zip(params, acc):
        sinks.add(p, a, 0)
    seen = []

    def run():
        z = ops.bn_act(y, gamma, beta, None, None, 0.1, relu, res if residual else None)
        if hook:
            z.register_hook(lambda g: seen.append(g.clone()))
        out, _, tap = ops.conv2d(z, w, 1, r // 2, tap_input=True)
        ((out.float() * g_out.float()).sum() + (tap.float() * g_tap.float()).sum()).backward()

    sinks.begin_step()
    sinks.set_active(True)
    run()
    sinks.set_active(False)
    check_error(y.device)

    yr, rr, wr, gr, br = [t.detach().float().requires_grad_() for t in (y, res, w, gamma, beta)]
    z = F.batch_norm(yr, None, None, gr, br, True, 0.1, 1e-5) + (rr if residual else 0.0)
    z = F.relu(z) if relu else z
    z.retain_grad()
    ((F.conv2d(z, wr, None, 1, r // 2) * g_out.float()).sum() + (z * g_tap.float()).sum()).backward()
    pairs = [(y.grad, yr.grad), (acc[0], gr.grad), (acc[1], br.grad), (acc[2], wr.grad)]
    if residual:
        pairs.append((res.grad, rr.grad))
    if hook:
        pairs.append((seen[0], z.grad))        # whoever listens gets the gradient of z itself, not behind the ReLU
    for i, (a, b) in enumerate(pairs):
        assert (a.float() - b).norm() < 2e-2 * b.norm(), (i, float((a.float() - b).norm() / b.norm()))
    sinks.close()
