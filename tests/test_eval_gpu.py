"""Inference convolutions with batch norm, shortcut and ReLU in the epilogue: every kernel kind against fp32 PyTorch, and whole
networks against the unfused path."""
import pytest
import torch
import torch.nn.functional as F

pytestmark = pytest.mark.gpu


def _cl(t):
    return t.contiguous(memory_format=torch.channels_last)


# n, cin, h, w, cout, k, stride: 1x1 plain and strided, shared boxes with and without resident filters, per-tap, strided,
# widths that fill no tile, narrow layers, the stem
@pytest.mark.parametrize("shape", [(3, 64, 9, 7, 256, 1, 1), (2, 256, 8, 8, 64, 1, 2), (5, 64, 14, 14, 64, 3, 1), (3, 128, 28, 28, 128, 3, 1),
                                   (1, 512, 7, 7, 512, 3, 1), (3, 64, 8, 8, 192, 3, 2), (7, 16, 32, 32, 16, 3, 1), (2, 40, 9, 11, 24, 3, 1),
                                   (130, 8, 5, 5, 8, 3, 1), (2, 3, 33, 33, 64, 7, 2)])
@pytest.mark.parametrize("residual,relu", [(True, True), (False, True), (False, False)])
def test_conv_bn_eval(shape, residual, relu):
    from eagersgd_b200.ops import functional as ops
    from eagersgd_b200.ops.gemm import check_error
    n, ci, h, w, co, k, s = shape
    g = torch.Generator().manual_seed(sum(shape))
    rnd = lambda *d: torch.randn(*d, generator=g).cuda()
    x, wt = _cl(rnd(n, ci, h, w)).bfloat16(), _cl(rnd(co, ci, k, k) / (ci * k * k) ** 0.5).bfloat16()
    gamma, beta, mean, var = rnd(co).abs() + 0.5, rnd(co), rnd(co) * 0.3, rnd(co).abs() + 0.5
    pad = (k - 1) // 2
    ref = F.batch_norm(F.conv2d(x.float(), wt.float(), None, s, pad), mean, var, gamma, beta, False, 0.1, ops.BN_EPS)
    res = _cl(rnd(*ref.shape)).bfloat16() if residual else None
    ref = ref + res.float() if residual else ref
    ref = F.relu(ref) if relu else ref
    coef = ops.bn_coefficients([(gamma, beta, mean, var)], {})[0]
    y = ops.conv_bn_eval(x, wt, s, pad, coef, relu, res)
    check_error(y.device)
    assert y.shape == ref.shape and (y.float() - ref).norm() < 4e-3 * ref.norm()
    assert float((y.float() - ref).abs().max()) < 0.05 * float(ref.abs().max())


@pytest.mark.parametrize("make", [lambda R: R.imagenet_resnet(50, 1, 101), lambda R: R.imagenet_resnet(18, 2, 11), lambda R: R.cifar_resnet(20, 1, 10)])
def test_networks_match_the_unfused_path_and_follow_their_parameters(make):
    from eagersgd_b200.models import resnet as R
    from eagersgd_b200.ops import functional as ops
    from eagersgd_b200.train.step import prepare_model
    torch.manual_seed(0)
    net = prepare_model(make(R), torch.device("cuda")).eval()
    for m in net.modules():
        if isinstance(m, torch.nn.BatchNorm2d):
            m.weight.data.uniform_(0.3, 0.8)
            m.running_mean.normal_(0, 0.1)
            m.running_var.uniform_(0.5, 1.5)
    for n in (1, 5):
        x = _cl(torch.randn(n, 3, 64, 64, device="cuda")).bfloat16()
        with torch.no_grad():
            y = net(x)
            with ops.reference_ops():
                ref = net(x).float()
        assert (y.float() - ref).norm() < 2e-2 * ref.norm()
        assert torch.allclose(y, net(x.requires_grad_()).detach().float(), rtol=0.1, atol=0.05 * float(ref.abs().max()))
    with torch.no_grad():                        # the coefficients are those of the call, not of the first one
        for m in net.modules():
            if isinstance(m, torch.nn.BatchNorm2d):
                m.running_mean.add_(0.2)
        y2 = net(x.detach())
        with ops.reference_ops():
            ref2 = net(x.detach()).float()
    assert (y2.float() - ref2).norm() < 2e-2 * ref2.norm() and not torch.equal(y, y2)
    seen = []
    net.blocks[0].register_forward_hook(lambda *a: seen.append(1))
    with torch.no_grad():
        net(x.detach())
    assert seen == [1]                           # a listener gets the layer-by-layer path


def test_a_captured_pass_outlives_a_change_beside_it():
    """A network that gets another child looks at its layers anew; what a captured pass reads stays where it is."""
    from eagersgd_b200.models import resnet as R
    from eagersgd_b200.train.step import prepare_model
    torch.manual_seed(1)
    net = prepare_model(R.cifar_resnet(20, 1, 10), torch.device("cuda")).eval()
    x = _cl(torch.randn(2, 3, 32, 32, device="cuda")).bfloat16()
    with torch.no_grad():
        want = net(x).clone()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            y = net(x)
        net.extra = torch.nn.Linear(2, 2)
        assert torch.equal(net(x), want)
        junk = [torch.full((n,), 7.0, device="cuda") for n in (256, 1024, 1376, 4096)]      # whatever has been freed is used again
        graph.replay()
        torch.cuda.synchronize()
    assert torch.equal(y, want) and len(junk) == 4
