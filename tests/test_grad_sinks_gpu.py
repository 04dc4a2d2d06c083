"""Gradients that operators add straight to the optimizer's buckets, against the same steps with every gradient through autograd."""
import pytest
import torch
from torch.utils.checkpoint import checkpoint

pytestmark = pytest.mark.gpu
LR, MOMENTUM = 0.1, 0.9


def _layers(seed, n=3, width=64):
    g = torch.Generator().manual_seed(seed)
    return [torch.nn.Parameter((torch.randn(width, width, generator=g) / width ** 0.5).cuda().bfloat16()) for _ in range(n)]


def _optimizer(params, **kw):
    import eagersgd_b200 as es
    from eagersgd_b200.optim.eager import SoloAllreduceOptimizer
    return SoloAllreduceOptimizer(torch.optim.SGD(params, lr=LR, momentum=MOMENTUM), es.Group(), **kw)


def _train(loss_of_step, steps, sinks, params=None, seed=0):
    """``steps`` optimizer steps; returns the momentum buffers after each (the gradients, in fp32) and how the buckets went."""
    params = _layers(seed) if params is None else params
    opt = _optimizer(params, overlap=sinks)        # without sinks: every gradient through autograd, then every bucket in step()
    if not sinks:
        opt._sinks_conflict = True
    launches = []
    inner = opt._launch
    opt._launch = lambda b, *a: (launches.append("early" if a else "step") if not b.launched else None, inner(b, *a))[1]
    x = torch.randn(32, 64, generator=torch.Generator().manual_seed(9)).cuda().bfloat16()
    out = []
    for k in range(steps):
        opt.zero_grad()
        with opt.grad_sinks():
            loss_of_step(k, x, params).backward()
        opt.step()
        torch.cuda.synchronize()
        out.append([m.float().clone() for _, m in opt.momentum_buffers()])
    opt.check()
    opt.close()
    return out, launches


def _mlp(x, params):
    from eagersgd_b200.ops import functional as ops
    for w in params:
        x = ops.linear(x, w).bfloat16()
    return x.float().square().mean()


def _same(a, b, tol):
    for sa, sb in zip(a, b):
        for u, v in zip(sa, sb):
            assert v.norm() > 0 and (u - v).norm() <= tol * v.norm(), (u.norm(), v.norm())


# bf16 gradients of the autograd route are rounded once (2^-9), the sinks' are not
TOL = 1e-2


def test_plain_steps_go_early():
    loss = lambda k, x, ps: _mlp(x, ps)
    (a, launches), (b, _) = _train(loss, 3, True), _train(loss, 3, False)
    _same(a, b, TOL)
    assert launches == ["early"] * 3


@pytest.mark.parametrize("first", [0, 1, 3])
@pytest.mark.parametrize("which", [0, 1, 2])
def test_a_parameter_with_a_second_route_from_some_step_on(which, first):
    def loss(k, x, ps):
        y = _mlp(x, ps)
        return y + 0.01 * ps[which].float().square().sum() if k >= first else y
    (a, _), (b, _) = _train(loss, 5, True), _train(loss, 5, False)
    _same(a, b, TOL)


def test_a_second_route_in_one_step_alone():
    def loss(k, x, ps):
        y = _mlp(x, ps)
        return y + 0.01 * ps[1].float().square().sum() if k == 2 else y
    (a, _), (b, _) = _train(loss, 5, True), _train(loss, 5, False)
    _same(a, b, TOL)


@pytest.mark.parametrize("reentrant", [True, False])
def test_a_weight_shared_by_two_checkpointed_segments(reentrant):
    from eagersgd_b200.ops import functional as ops

    def loss(k, x, ps):
        h = ops.linear(x, ps[0]).bfloat16()
        for _ in range(2):
            h = checkpoint(lambda t: ops.linear(t, ps[1]).bfloat16(), h, use_reentrant=reentrant)
        return ops.linear(h, ps[2]).float().square().mean()
    (a, _), (b, _) = _train(loss, 3, True), _train(loss, 3, False)
    _same(a, b, TOL)


def test_a_parameter_with_a_hook_keeps_its_gradient():
    params = _layers(1)
    opt = _optimizer(params, overlap=False)        # a bucket that goes early is cleared behind the copy
    opt.prepare_grad_sinks()
    seen = []
    handle = params[1].register_hook(lambda g: seen.append(g.float().norm().item()))
    x = torch.ones(32, 64, device="cuda", dtype=torch.bfloat16)
    for hooked in (True, False):
        opt.zero_grad()
        with opt.grad_sinks():
            _mlp(x, params).backward()
        assert (len(seen) == 1) and bool(params[1].grad.any()) == hooked
        opt.step()
        if hooked:
            handle.remove()
    opt.check()
    opt.close()


def test_a_second_optimizer_over_the_parameters_of_a_closed_one():
    loss = lambda k, x, ps: _mlp(x, ps)
    params = _layers(0)
    _train(loss, 2, True, params=params)
    copies = [torch.nn.Parameter(p.detach().clone()) for p in params]
    (a, launches), (b, _) = _train(loss, 2, True, params=params), _train(loss, 2, False, params=copies)
    _same(a, b, TOL)
    assert launches == ["early"] * 2


def test_closing_one_of_two_owners_leaves_the_parameter_to_the_other():
    from eagersgd_b200 import _build
    (w,) = _layers(3, 1)
    owners = [_build.load_torch().GradSinks([1], lambda i: None) for _ in range(2)]
    accs = [torch.zeros(w.numel(), device="cuda") for _ in owners]
    for o, acc in zip(owners, accs):
        o.add(w, acc, 0)
    owners[0].close()
    owners[1].begin_step()
    owners[1].set_active(True)
    _mlp(torch.ones(32, 64, device="cuda", dtype=torch.bfloat16), [w]).backward()
    owners[1].set_active(False)
    assert w.grad is None and bool(accs[1].any()) and not bool(accs[0].any()) and owners[1].used(w)
    owners[1].close()


def test_saved_tensor_hooks_can_let_go_of_activations():
    """Offloading what backward needs to the host: the operators keep no activation on the GPU beside it, and the gradients are
    those of a pass without hooks."""
    from eagersgd_b200 import _build
    from eagersgd_b200.ops import functional as ops
    g = torch.Generator().manual_seed(6)
    cl = lambda *s: torch.randn(*s, generator=g).cuda().bfloat16().contiguous(memory_format=torch.channels_last)
    x, w1, w2 = cl(4, 64, 64, 64), (cl(64, 64, 3, 3) * 0.1).requires_grad_(), (cl(64, 64, 3, 3) * 0.1).requires_grad_()
    gamma, beta = torch.rand(64, generator=g).cuda().requires_grad_(), torch.zeros(64, device="cuda").requires_grad_()
    params = [w1, gamma, beta, w2]
    accs = [torch.zeros_like(p, dtype=torch.float32, memory_format=torch.preserve_format) for p in params]
    sinks = _build.load_torch().GradSinks([4], lambda i: None)
    for p, a in zip(params, accs):
        sinks.add(p, a, 0)

    def run():
        y, st = ops.conv2d(x, w1, 1, 1, want_stats=True)
        z = ops.bn_act(y, gamma, beta, None, None, stats=st)
        return ops.conv2d(z, w2, 1, 1)[0].float().square().mean()

    results, held = [], []
    for offload in (False, True, False, True):             # the second time round nothing is allocated once and for all
        for a in accs:
            a.zero_()
        sinks.begin_step()
        sinks.set_active(True)
        torch.cuda.synchronize()
        m0 = torch.cuda.memory_allocated()
        if offload:
            with torch.autograd.graph.saved_tensors_hooks(lambda t: t.cpu(), lambda t: t.cuda()):
                loss = run()
        else:
            loss = run()
        held.append(torch.cuda.memory_allocated() - m0)
        loss.backward()
        sinks.set_active(False)
        results.append([a.clone() for a in accs])
        del loss
    sinks.close()
    assert held[3] < x.numel() * 2 <= held[2] and max(held[3], 0) < 1 << 20, held
    for a, b in zip(results[2], results[3]):
        assert (a - b).norm() <= 1e-2 * b.norm()            # the masked gradient's sums in one kernel, or in another


def test_steps_with_the_weight_gradients_on_a_stream_of_their_own():
    """The same network captured (the weight gradients of all its convolutions go to the side stream) and not (none does)."""
    import eagersgd_b200 as es
    from eagersgd_b200.models.resnet import cifar_resnet
    from eagersgd_b200.train.step import TrainStep
    g = torch.Generator().manual_seed(2)
    x = torch.randn(16, 3, 32, 32, generator=g).cuda().bfloat16().contiguous(memory_format=torch.channels_last)
    y = torch.randint(0, 10, (16,), generator=g).cuda()
    results = []
    for graph in (False, True):
        torch.manual_seed(4)
        step = TrainStep(cifar_resnet(8), es.Group(), lr=1e-3)
        if graph:
            step.capture(x, y, warmup=2)
        for _ in range(2 if graph else 4):
            loss = step.run_device(x, y)
        torch.cuda.synchronize()
        results.append((float(loss), [b.mom.clone() for b in step.opt.buckets]))
        step.opt.check()
        step.close()
    assert abs(results[0][0] - results[1][0]) <= 1e-3 * abs(results[1][0])
    for a, b in zip(results[0][1], results[1][1]):
        assert (a - b).norm() <= 2e-2 * b.norm()        # bf16 activations, sums that meet in atomics
