"""The fused inference and training paths of a ResNet step aside for a layer that somebody has changed since the network was
built.  The kernels are stood in for by PyTorch, so that the choice of the path is what is tested."""
import pytest
import torch
import torch.nn.functional as F
from torch import nn

from eagersgd_b200.models import resnet as R
from eagersgd_b200.ops import functional as ops


def exchanged_norm(net, seen):
    net.blocks[0].bns[0] = R._bn(net.blocks[0].bns[0].num_features)


def exchanged_kind_of_norm(net, seen):
    class Shift(nn.Module):
        def forward(self, y, relu=True, residual=None, stats=None):
            seen.append(1)
            y = y + 1 + (0 if residual is None else residual)
            return y.relu() if relu else y
    net.blocks[0].bns[1] = Shift()


def parametrized_convolution(net, seen):
    class Twice(nn.Module):
        def forward(self, w):
            seen.append(1)
            return 2 * w
    torch.nn.utils.parametrize.register_parametrization(net.blocks[1].convs[0], "weight", Twice())


def plain_tensor_for_a_parameter(net, seen):
    conv = net.blocks[0].convs[1]
    w = conv.weight.detach() * 3
    del conv.weight
    conv.weight = w


def subclass_of_a_convolution(net, seen):
    class Doubled(R._Conv):
        def forward(self, x, tap_input=False):
            seen.append(1)
            return super().forward(2 * x, tap_input)
    net.blocks[0].convs[0].__class__ = Doubled


def subclass_of_a_block(net, seen):
    class Skipped(R._Block):
        def forward(self, x):
            seen.append(1)
            return x
    net.blocks[0].__class__ = Skipped


def forward_of_an_instance(net, seen):
    conv = net.blocks[0].convs[0]
    inner = conv.forward
    conv.forward = lambda *a, **k: (seen.append(1), inner(*a, **k))[1]


def hook_on_a_layer(net, seen):
    net.blocks[0].convs[0].register_forward_hook(lambda *a: seen.append(1))


def global_hook(net, seen):
    return torch.nn.modules.module.register_module_forward_hook(lambda m, *a: seen.append(1) if m is net.blocks[0].convs[0] else None)


CHANGES = [exchanged_norm, exchanged_kind_of_norm, parametrized_convolution, plain_tensor_for_a_parameter, subclass_of_a_convolution,
           subclass_of_a_block, forward_of_an_instance, hook_on_a_layer, global_hook]
UNSEEN = (exchanged_norm, plain_tensor_for_a_parameter)       # changes of data alone: no call to see


def settle(net):
    torch.manual_seed(3)
    for m in net.modules():
        if isinstance(m, nn.BatchNorm2d):
            m.weight.data.uniform_(0.3, 0.8)
            m.running_mean.normal_(0, 0.1)
            m.running_var.uniform_(0.5, 1.5)


@pytest.fixture
def stubs(monkeypatch):
    """The library's calls in PyTorch; the list counts those of the fused path."""
    fused = []

    def coefficients(layers, store):
        if not layers.unchanged():
            return None
        out = []
        for m in layers.norms:
            s = m.weight * torch.rsqrt(m.running_var + ops.BN_EPS)
            out.append(torch.stack([s, m.bias - m.running_mean * s]))
        return out

    def conv(x, w, stride, pad, coef, relu, residual=None):
        fused.append(1)
        y = F.conv2d(x, w, None, stride, pad)
        if coef is not None:
            y = y * coef[0].view(1, -1, 1, 1) + coef[1].view(1, -1, 1, 1)
        y = y if residual is None else y + residual
        return y.relu() if relu else y

    def block(x, layers, proj=None):
        s = x if proj is None else conv(x, proj[0], proj[1], proj[2], proj[3], False)
        for i, (w, stride, pad, c) in enumerate(layers):
            x = conv(x, w, stride, pad, c, True, s if i == len(layers) - 1 else None)
        return x

    def train_block(x, layers, proj=None):
        fused.append(1)

        def layer(x, l, relu, residual=None):
            y = F.batch_norm(F.conv2d(x, l[0], None, l[1], l[2]), l[5], l[6], l[3], l[4], True, l[7], ops.BN_EPS)
            y = y if residual is None else y + residual
            return y.relu() if relu else y
        s = x if proj is None else layer(x, proj, False)
        for i, l in enumerate(layers):
            x = layer(x, l, True, s if i == len(layers) - 1 else None)
        return x

    monkeypatch.setattr(ops, "native", lambda x: not ops._reference_only)
    monkeypatch.setattr(ops, "eval_coefficients", coefficients)
    monkeypatch.setattr(ops, "conv_bn_eval", conv)
    monkeypatch.setattr(ops, "residual_block_eval", block)
    monkeypatch.setattr(ops, "residual_block", train_block)
    for name in ("conv2d", "bn_act", "max_pool_3x3_s2", "global_avg_pool", "linear"):
        def plain(*a, _f=getattr(ops, name), **k):
            with ops.reference_ops():
                return _f(*a, **k)
        monkeypatch.setattr(ops, name, plain)
    return fused


# a block of version 2 has no norm behind its last convolution
@pytest.mark.parametrize("change,version", [(c, v) for c in CHANGES for v in (1, 2) if (c, v) != (exchanged_kind_of_norm, 2)])
def test_inference_sees_a_changed_layer(stubs, change, version):
    net = R.cifar_resnet(14, version).eval()
    settle(net)
    x = torch.randn(2, 3, 16, 16)
    with torch.no_grad():
        before = net(x)
        assert stubs                                 # the fused path, as long as nothing has changed
        with ops.reference_ops():
            assert torch.allclose(before, net(x), atol=1e-4)
        seen = []
        handle = change(net, seen)
        net.eval()
        try:
            after = net(x)
            assert bool(seen) != (change in UNSEEN)
            with ops.reference_ops():
                assert torch.allclose(after, net(x), atol=1e-4)
        finally:
            if handle is not None:
                handle.remove()


@pytest.mark.parametrize("change", CHANGES)
def test_training_sees_a_changed_layer(stubs, change):
    net = R.cifar_resnet(14).train()
    settle(net)
    x = torch.randn(4, 3, 16, 16)
    net(x)
    assert stubs
    seen = []
    handle = change(net, seen)
    net.train()
    try:
        state = {k: v.clone() for k, v in net.state_dict().items()}
        after = net(x)
        assert bool(seen) != (change in UNSEEN)
        net.load_state_dict(state)
        with ops.reference_ops():
            assert torch.allclose(after, net(x), atol=1e-4)
    finally:
        if handle is not None:
            handle.remove()
