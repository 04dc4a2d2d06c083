"""Narrow residual blocks in training, where a batch norm between two convolutions is made by the second one's kernel and a
layer's backward pass is one launch, against the same blocks called layer by layer: rows of odd widths, images that share a block
of the kernel, and everybody who could notice that a gradient or an activation is not there yet."""
import contextlib
import ctypes as C

import pytest
import torch
import torch.nn.functional as F

pytestmark = pytest.mark.gpu


def _blocks(channels, depth):
    from eagersgd_b200.models.resnet import ResNet, _Block
    from eagersgd_b200.train import prepare_model
    torch.manual_seed(channels)
    net = ResNet("building", [1], 8, channels, 3, 1, False, [1])
    net.blocks = torch.nn.ModuleList(_Block(channels, channels, 1, "building", 1, False, []) for _ in range(depth))
    net = prepare_model(net, torch.device("cuda")).train()
    g = torch.Generator(device="cuda").manual_seed(channels)
    for m in net.modules():
        if isinstance(m, torch.nn.BatchNorm2d):
            m.weight.data.copy_(torch.rand(m.num_features, device="cuda", generator=g) + 0.5)
            m.bias.data.copy_(torch.randn(m.num_features, device="cuda", generator=g) * 0.2)
    return net.blocks


def _run(blocks, x, dy, layerwise, context=contextlib.nullcontext, node_hook=None, backwards=1):
    """Output, input gradient, parameter gradients (through sinks) and running statistics of one pass; launches of this package."""
    from eagersgd_b200 import _build
    from eagersgd_b200.ops.gemm import check_error
    from eagersgd_b200.parallel import _native as N
    ext = _build.load_torch()
    params = [p for p in blocks.parameters()]
    acc = [torch.zeros_like(p, dtype=torch.float32, memory_format=torch.preserve_format) for p in params]
    sinks = ext.GradSinks([len(params)], lambda bucket: None)
    for p, a in zip(params, acc):
        sinks.add(p, a, 0)
    state = {k: v.clone() for k, v in blocks.state_dict().items()}
    hooks = [b.convs[0].register_forward_hook(lambda *a: None) for b in blocks] if layerwise else []
    xi = x.clone().requires_grad_()
    sinks.begin_step()
    sinks.set_active(True)
    n0 = N.launch_count()
    with context():
        y = xi
        for b in blocks:
            y = b(y)
        if node_hook is not None:
            node_hook(y)
        for i in range(backwards):
            y.backward(dy, retain_graph=i + 1 < backwards)
    launches = N.launch_count() - n0
    sinks.set_active(False)
    sinks.close()
    for h in hooks:
        h.remove()
    check_error(x.device)
    out = [y.detach(), xi.grad] + acc + [b.clone() for b in blocks.buffers()]
    blocks.load_state_dict(state)
    return [o.float() for o in out], launches


# For what a route forgets, counts twice or reads too early; the kernels' arithmetic is tested below.  Two runs of the SAME route
# differ by up to 5 % on these random networks (sums meet in atomics, and a bf16 rounding or a ReLU that falls the other way
# moves everything behind it), and both are 2 to 12 % from the same network in 64 bits.
def _compare(a, b):
    for i, (p, q) in enumerate(zip(a, b)):
        assert (p - q).norm() <= 0.15 * q.norm() + 1e-6, (i, tuple(p.shape), float((p - q).norm() / q.norm()))


def _data(c, n, h, w):
    g = torch.Generator(device="cuda").manual_seed(n + h)
    rnd = lambda: torch.randn(n, c, h, w, device="cuda", generator=g).to(torch.bfloat16).contiguous(memory_format=torch.channels_last)
    return rnd(), rnd()


# the last two: more rows a block of the kernel than its backward pass takes at a time, and than the forward pass does
@pytest.mark.parametrize("c,n,h,w", [(16, 3, 13, 9), (16, 1, 1, 1), (16, 200, 5, 7), (32, 2, 16, 16), (32, 149, 1, 17), (32, 37, 8, 3), (64, 5, 8, 8),
                                     (64, 40, 8, 8), (16, 300, 32, 32), (16, 620, 32, 32)])
def test_blocks_against_layers(c, n, h, w):
    blocks, (x, dy) = _blocks(c, 2), _data(c, n, h, w)
    one, launches = _run(blocks, x, dy, False)
    ref, more = _run(blocks, x, dy, True)
    _compare(one, ref)
    assert launches < more


@pytest.mark.parametrize("c", [16, 32])
@pytest.mark.parametrize("who", ["node hooks", "saved tensors", "anomaly", "two backward passes", "captured gradient"])
def test_somebody_is_looking(c, who):
    blocks, (x, dy) = _blocks(c, 2), _data(c, 4, 12, 10)
    ref, _ = _run(blocks, x, dy, True)
    if who == "node hooks":
        def attach(seen):
            def to(y):
                todo, done = [y.grad_fn], set()
                while todo:
                    node = todo.pop()
                    if node is None or node in done:
                        continue
                    done.add(node)
                    if "ConvFn" in node.name():
                        node.register_prehook(lambda grads: seen.append(grads[0].float().clone()))
                    todo += [f for f, _ in node.next_functions]
            return to
        a, b = [], []
        one, _ = _run(blocks, x, dy, False, node_hook=attach(a))
        _run(blocks, x, dy, True, node_hook=attach(b))
        assert len(a) == len(b) == 4
        _compare(a, b)               # what a convolution's backward gets is its output's gradient
    elif who == "saved tensors":
        class Elsewhere(torch.autograd.graph.saved_tensors_hooks):
            def __init__(self):
                super().__init__(lambda t: t.detach().clone(memory_format=torch.preserve_format), lambda t: t)
        one, _ = _run(blocks, x, dy, False, Elsewhere)
    elif who == "anomaly":
        one, _ = _run(blocks, x, dy, False, lambda: torch.autograd.set_detect_anomaly(True))
    elif who == "two backward passes":
        one, _ = _run(blocks, x, dy, False, backwards=2)
        n = 1 + 1 + len(list(blocks.parameters()))
        one = one[:1] + [o / 2 for o in one[1:n]] + one[n:]
    else:
        xi = x.clone().requires_grad_()
        from eagersgd_b200 import _build
        params = [p for p in blocks.parameters()]
        sinks = _build.load_torch().GradSinks([len(params)], lambda bucket: None)
        acc = [torch.zeros_like(p, dtype=torch.float32, memory_format=torch.preserve_format) for p in params]
        for p, t in zip(params, acc):
            sinks.add(p, t, 0)
        sinks.begin_step()
        sinks.set_active(True)
        y = xi
        for b in blocks:
            y = b(y)
        (gx,) = torch.autograd.grad(y, [xi], dy)
        sinks.set_active(False)
        sinks.close()
        one, ref = [gx.float()], [ref[1]]
    _compare(one, ref)


@pytest.mark.parametrize("c", [16, 32])
def test_backward_pass_after_one_that_broke_off(c):
    """An error between a batch norm's backward and its convolution's (here the convolution's input has changed) leaves nothing
    behind that a second pass over the kept graph would trip over."""
    from eagersgd_b200 import _build
    blocks, (x, dy) = _blocks(c, 1), _data(c, 4, 12, 10)
    params = [p for p in blocks.parameters()]
    sinks = _build.load_torch().GradSinks([len(params)], lambda bucket: None)
    for p in params:
        sinks.add(p, torch.zeros_like(p, dtype=torch.float32, memory_format=torch.preserve_format), 0)
    sinks.begin_step()
    sinks.set_active(True)
    xi = x.clone().requires_grad_()
    y = blocks[0](xi)
    version = xi._version
    with torch.no_grad():
        xi.add_(0)
    with pytest.raises(RuntimeError, match="inplace"):
        y.backward(dy, retain_graph=True)
    torch._C._autograd._unsafe_set_version_counter((xi,), (version,))
    assert xi.grad is None
    y.backward(dy)
    sinks.set_active(False)
    sinks.close()
    ref, _ = _run(blocks, x, dy, True)
    _compare([xi.grad.float()], [ref[1]])


# ---------------------------------------------------------------------------------------------------- the kernels
class _BnGrad(C.Structure):
    _fields_ = [("y", C.c_void_p), ("mask", C.c_void_p), ("aux", C.c_void_p), ("sums", C.c_void_p)]


def _p(t, elements=0):
    return None if t is None else C.c_void_p(t.data_ptr() + elements * t.element_size())


def _problem(c, n, h, w):
    g = torch.Generator(device="cuda").manual_seed(c * 1000 + n + h)
    rnd = lambda *s: torch.randn(*s, device="cuda", generator=g)
    act = lambda: rnd(n, h, w, c).to(torch.bfloat16)
    weight = (rnd(c, 3, 3, c) / (9 * c) ** 0.5).to(torch.bfloat16)            # stored [out][3][3][in]
    return rnd, act, weight


def _nchw(t):
    return t.double().permute(0, 3, 1, 2)


def _close(a, b, rel):
    assert (a.double() - b).norm() <= rel * b.norm() + 1e-9, float((a.double() - b).norm() / b.norm())


SHAPES = [(16, 1, 1, 1), (16, 3, 13, 9), (16, 150, 2, 33), (16, 37, 32, 32), (32, 2, 16, 16), (32, 149, 1, 17), (32, 100, 7, 5)]


@pytest.mark.parametrize("c,n,h,w", SHAPES + [(64, 1, 8, 8), (64, 128, 8, 8), (64, 3, 5, 70), (16, 900, 32, 32)])
@pytest.mark.parametrize("relu,mask", [(True, True), (True, False), (False, False)])
def test_batch_norm_on_the_way_into_a_convolution(c, n, h, w, relu, mask):
    from eagersgd_b200.parallel import _native as N
    lib = N.cuda()
    rnd, act, weight = _problem(c, n, h, w)
    by, m = act() * 2, n * h * w
    z, y = torch.full_like(by, 9.0), torch.full_like(by, 9.0)
    bits = torch.zeros(m, c // 8, dtype=torch.uint8, device="cuda") if mask else None
    bsums = torch.stack([by.float().sum((0, 1, 2)), by.float().square().sum((0, 1, 2))])
    gamma, beta, aux, sums = rnd(c).abs() + 0.5, rnd(c), torch.zeros(4, c, device="cuda"), torch.zeros(2, c, device="cuda")
    rm, rv = rnd(c), rnd(c).abs()
    rm0, rv0 = rm.clone(), rv.clone()
    rc = lib.esgd_conv_narrow_bn_fwd(_p(by), _p(z), _p(bits), _p(bsums), _p(bsums, c), _p(gamma), _p(beta), _p(rm), _p(rv), _p(aux), int(relu),
                                     C.c_float(0.1), C.c_float(1e-5), _p(weight), _p(y), n, h, w, c, _p(sums), _p(sums, c),
                                     C.c_void_p(torch.cuda.current_stream().cuda_stream))
    assert rc == 0
    mean = by.double().mean((0, 1, 2))
    var = (by.double().square().mean((0, 1, 2)) - mean * mean).clamp_min(0)
    invstd = (var + 1e-5).rsqrt()
    zr = (by.double() - mean) * invstd * gamma.double() + beta.double()
    zr = zr.relu() if relu else zr
    if m > 1:                       # of one pixel the variance is a difference of equal numbers
        _close(z, zr, 4e-3)         # a bf16 rounding: 2^-9
    if mask:
        want = (z.view(m, c // 8, 8) > 0).to(torch.int32) << torch.arange(8, device="cuda", dtype=torch.int32)
        assert torch.equal(bits.to(torch.int32), want.sum(-1).to(torch.int32))
    if m > 1:
        assert torch.allclose(aux[0].double(), mean, rtol=1e-4, atol=1e-5) and torch.allclose(aux[1].double(), invstd, rtol=1e-3)
        assert torch.allclose(rm.double(), 0.9 * rm0.double() + 0.1 * mean, rtol=1e-4, atol=1e-5)
        assert torch.allclose(rv.double(), 0.9 * rv0.double() + 0.1 * var * m / (m - 1), rtol=1e-3)
    yr = F.conv2d(_nchw(z), _nchw(weight), None, 1, 1).permute(0, 2, 3, 1)       # of the z that was stored
    _close(y, yr, 4e-3)
    _close(sums[0], y.double().sum((0, 1, 2)), 1e-3)
    _close(sums[1], y.double().square().sum((0, 1, 2)), 1e-3)


@pytest.mark.parametrize("c,n,h,w", SHAPES)
@pytest.mark.parametrize("residual,behind", [(False, None), (True, "mask"), (True, "no mask")])
def test_backward_pass_of_a_layer(c, n, h, w, residual, behind):
    from eagersgd_b200.parallel import _native as N
    lib = N.cuda()
    rnd, act, weight = _problem(c, n, h, w)
    x, dz, y, py, m = act(), act(), act(), act(), n * h * w
    res = act() if residual else None
    aux, paux = torch.stack([rnd(c) * 0.1, rnd(c).abs() + 0.5, rnd(c), rnd(c)]), torch.stack([rnd(c) * 0.1, rnd(c).abs() + 0.5])
    gamma, sums = rnd(c).abs() + 0.5, torch.stack([rnd(c), rnd(c)]) * m ** 0.5                # dbeta, dgamma
    accs, dw = [torch.ones(c, device="cuda"), torch.ones(c, device="cuda") * 2], torch.ones(c, 3, 3, c, device="cuda")
    dx, psums = torch.full_like(x, 9.0), torch.zeros(2, c, device="cuda")
    bits = torch.randint(0, 256, (m, c // 8), dtype=torch.uint8, device="cuda") if behind == "mask" else None
    bn = _BnGrad(py.data_ptr(), bits.data_ptr() if bits is not None else 0, paux.data_ptr(), psums.data_ptr())
    rc = lib.esgd_conv_narrow_bwd(_p(x), _p(weight), _p(dz), _p(y), _p(aux), _p(gamma), _p(sums), _p(sums, c), _p(accs[0]), _p(accs[1]), _p(dx),
                                  _p(dw), n, h, w, c, _p(res), C.byref(bn) if behind else None,
                                  C.c_void_p(torch.cuda.current_stream().cuda_stream))
    assert rc == 0
    a, g, s = aux.double(), gamma.double(), sums.double() / m
    dy = g * a[1] * (dz.double() - s[0] - (y.double() - a[0]) * a[1] * s[1])
    xr, wr = _nchw(x).requires_grad_(), _nchw(weight).requires_grad_()
    F.conv2d(xr, wr, None, 1, 1).backward(dy.permute(0, 3, 1, 2))
    dxr = xr.grad.permute(0, 2, 3, 1) + (res.double() if residual else 0.0)
    if bits is not None:
        on = (bits.to(torch.int32).unsqueeze(-1) >> torch.arange(8, device="cuda", dtype=torch.int32)) & 1
        dxr = dxr * on.view(n, h, w, c)
        assert bool((dx[on.view(n, h, w, c) == 0] == 0).all())
    _close(dx, dxr, 6e-3)           # dy and dx are rounded to bf16
    _close(dw - 1.0, wr.grad.permute(0, 2, 3, 1), 6e-3)
    assert torch.allclose(accs[0], 1.0 + sums[1]) and torch.allclose(accs[1], 2.0 + sums[0])
    if behind:
        d = dx.double()
        hat = (py.double() - paux[0].double()) * paux[1].double()
        scale = 1e-3 * d.abs().sum((0, 1, 2)).max()
        assert torch.allclose(psums[0].double(), d.sum((0, 1, 2)), rtol=1e-3, atol=float(scale))
        assert torch.allclose(psums[1].double(), (d * hat).sum((0, 1, 2)), rtol=1e-3, atol=float(3 * scale))


def test_backward_pass_of_a_layer_refuses_what_does_not_fit():
    from eagersgd_b200.parallel import _native as N
    lib = N.cuda()
    t = torch.zeros(64, device="cuda")
    args = lambda n, h, w, c, off=0: [_p(t, off)] + [_p(t)] * 11 + [n, h, w, c, None, None, None]
    assert lib.esgd_conv_narrow_bwd(*args(620, 32, 32, 16)) == -100 and lib.esgd_conv_narrow_bwd(*args(2, 4, 3000, 32)) == -100
    assert lib.esgd_conv_narrow_bwd(*args(2, 4, 4, 64)) == -100 and lib.esgd_conv_narrow_bwd(*args(2, 4, 4, 16, 1)) == -100
    assert lib.esgd_conv_narrow_bwd(*args(0, 4, 4, 16)) == -1
