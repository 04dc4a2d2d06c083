"""A residual block through one library call against the same block called layer by layer (which a hook on a layer asks for)."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind,cin,filters,stride,project,training", [
    ("building", 16, 16, 1, False, True), ("building", 16, 32, 2, True, True), ("building", 24, 24, 1, False, True),
    ("bottleneck", 64, 64, 1, True, True), ("bottleneck", 256, 64, 1, False, True), ("bottleneck", 256, 128, 2, True, True),
    ("building", 16, 32, 2, True, False), ("bottleneck", 256, 64, 1, False, False), ("bottleneck", 256, 128, 2, True, False)])
def test_block_in_one_call(kind, cin, filters, stride, project, training):
    from eagersgd_b200.models.resnet import ResNet, _Block
    from eagersgd_b200.train import prepare_model
    torch.manual_seed(cin + filters)
    net = ResNet(kind, [1], 8, cin, 3, 1, False, [stride])
    net.blocks[0] = _Block(cin, filters, stride, kind, 1, project, [])
    net = prepare_model(net, torch.device("cuda")).train(training)
    for m in net.modules():
        if isinstance(m, torch.nn.BatchNorm2d):
            torch.nn.init.uniform_(m.weight, 0.5, 1.5)
            torch.nn.init.uniform_(m.running_mean, -0.2, 0.2)
    block = net.blocks[0]
    x = torch.randn(3, cin, 10, 10).cuda().to(torch.bfloat16).contiguous(memory_format=torch.channels_last)
    results = []
    for layerwise in (False, True):
        state = {k: v.clone() for k, v in net.state_dict().items()}
        hook = block.convs[0].register_forward_hook(lambda *a: None) if layerwise else None
        net.zero_grad()
        if training:
            xi = x.clone().requires_grad_()
            y = block(xi)
            y.float().square().sum().backward()
            out = [y.detach(), xi.grad] + [p.grad for p in block.parameters()] + [b.clone() for b in block.buffers()]
        else:
            with torch.no_grad():
                img = torch.linspace(-1, 1, 3 * 3 * 10 * 10).view(3, 3, 10, 10).cuda().to(torch.bfloat16)
                out = [net.features(img.contiguous(memory_format=torch.channels_last))]
        results.append([o.float().clone() for o in out])
        net.load_state_dict(state)
        if hook is not None:
            hook.remove()
    for a, b in zip(*results):
        assert (a - b).norm() <= 1e-2 * b.norm() + 1e-6, tuple(a.shape)
