"""The operators refuse operands that do not fit one another before a kernel is given their pointers."""
import pytest
import torch

from eagersgd_b200 import _build

BF16, F32 = torch.bfloat16, torch.float32


def _t(*shape, dtype=BF16, device="cpu"):
    t = torch.zeros(*shape, dtype=dtype, device=device)
    return t.contiguous(memory_format=torch.channels_last) if t.dim() == 4 else t


# operator -> (arguments that fit, made for a device; name of an argument -> what does not fit in its place)
def _linear(d):
    return dict(x=_t(16, 32, device=d), w=_t(24, 32, device=d), b=_t(24, device=d))


def _conv1x1(d):
    return dict(x=_t(2, 16, 8, 8, device=d), w=_t(24, 16, 1, 1, device=d))


def _conv3x3(d):
    return dict(x=_t(2, 16, 8, 8, device=d), w=_t(16, 16, 3, 3, device=d))


def _stem(d):
    return dict(x=_t(2, 3, 8, 8, device=d), w=_t(16, 3, 3, 3, device=d))


def _eval(d):
    return dict(x=_t(2, 16, 8, 8, device=d), w=_t(16, 16, 3, 3, device=d), coef=_t(32, dtype=F32, device=d),
                residual=_t(2, 16, 8, 8, device=d))


def _bn(d):
    return dict(y=_t(2, 16, 4, 4, device=d), gamma=_t(16, dtype=F32, device=d), beta=_t(16, dtype=F32, device=d),
                res=_t(2, 16, 4, 4, device=d), rm=_t(16, dtype=F32, device=d), rv=_t(16, dtype=F32, device=d),
                stats=_t(2, 16, dtype=F32, device=d))


def _ce(d):
    return dict(logits=_t(8, 10, dtype=F32, device=d), labels=torch.zeros(8, dtype=torch.int64, device=d))


def _lstm(d):
    return dict(x=_t(3, 8, 16, device=d), w_ih=_t(32, 16, device=d), w_hh=_t(32, 8, device=d), bias=_t(32, dtype=F32, device=d))


def _call(op, a):
    e = _build.load_torch()
    if op is _linear:
        return e.linear(a["x"], a["w"], a["b"])
    if op is _eval:
        return e.conv_bn_eval(a["x"], a["w"], 1, 1, a["coef"], a["residual"], True, True)
    if op is _bn:
        return e.bn_act(a["y"], a["gamma"], a["beta"], a["res"], a["rm"], a["rv"], 0.1, True, a["stats"])
    if op is _ce:
        return e.softmax_ce(a["logits"], a["labels"])
    if op is _lstm:
        return e.lstm_layer(a["x"], a["w_ih"], a["w_hh"], a["bias"])
    return e.conv2d(a["x"], a["w"], 1, a["w"].shape[2] // 2, True, False, True)


MISFITS = [
    (_linear, "w", lambda d: _t(24, 16, device=d)), (_linear, "w", lambda d: _t(24, 40, device=d)),
    (_linear, "x", lambda d: _t(16, 32, 8, device=d)), (_linear, "x", lambda d: _t(16, 32, dtype=F32, device=d)),
    (_linear, "b", lambda d: _t(16, device=d)),
    (_conv1x1, "w", lambda d: _t(24, 8, 1, 1, device=d)), (_conv1x1, "w", lambda d: _t(24, 24, 1, 1, device=d)),
    (_conv1x1, "w", lambda d: _t(24, 16, 1, 1, dtype=F32, device=d)),
    (_conv3x3, "w", lambda d: _t(16, 8, 3, 3, device=d)), (_conv3x3, "w", lambda d: _t(16, 16, 3, 3, dtype=F32, device=d)),
    (_stem, "w", lambda d: _t(16, 1, 3, 3, device=d)), (_stem, "w", lambda d: _t(16, 3, 3, 3, dtype=torch.int32, device=d)),
    (_eval, "w", lambda d: _t(16, 32, 3, 3, device=d)), (_eval, "coef", lambda d: _t(16, dtype=F32, device=d)),
    (_eval, "residual", lambda d: _t(2, 16, 4, 4, device=d)), (_eval, "residual", lambda d: _t(2, 16, 8, 8, dtype=F32, device=d)),
    (_bn, "gamma", lambda d: _t(8, dtype=F32, device=d)), (_bn, "beta", lambda d: _t(16, device=d)),
    (_bn, "res", lambda d: _t(1, 16, 4, 4, device=d)), (_bn, "rm", lambda d: _t(8, dtype=F32, device=d)),
    (_bn, "rv", lambda d: _t(16, device=d)), (_bn, "stats", lambda d: _t(16, dtype=F32, device=d)),
    (_ce, "labels", lambda d: torch.zeros(7, dtype=torch.int64, device=d)), (_ce, "logits", lambda d: _t(8, 10, 2, dtype=F32, device=d)),
    (_lstm, "w_ih", lambda d: _t(32, 8, device=d)), (_lstm, "w_hh", lambda d: _t(64, 8, device=d)),
    (_lstm, "w_hh", lambda d: _t(32, 16, device=d)), (_lstm, "bias", lambda d: _t(8, dtype=F32, device=d)),
    (_lstm, "x", lambda d: _t(24, 16, device=d)),
]
NAMES = {_linear: "linear", _ce: "softmax_ce", _lstm: "lstm_layer", _bn: "bn_act"}


def _refuses(op, name, misfit, device):
    a = dict(op(device))
    a[name] = misfit(device)
    with pytest.raises(RuntimeError, match="^%s: " % NAMES.get(op, "conv2d")):      # the operator's own words
        _call(op, a)


@pytest.mark.parametrize("op,name,misfit", MISFITS)
def test_operands_that_do_not_fit_are_refused(op, name, misfit):
    _refuses(op, name, misfit, "cpu")


@pytest.mark.parametrize("stride,pad", [(0, 1), (-1, 1), (1, -1)])
def test_no_kernel_for_a_stride_or_padding_that_is_none(stride, pad):
    a = _conv3x3("cpu")
    assert _build.load_torch().conv2d(a["x"], a["w"], stride, pad, False, False, True) is None


def test_a_filter_larger_than_the_padded_image_is_refused():
    with pytest.raises(RuntimeError, match="conv2d: the filter"):
        _build.load_torch().conv2d(_t(2, 16, 2, 8), _t(16, 16, 3, 3), 1, 0, False, False, True)


@pytest.mark.gpu
@pytest.mark.parametrize("op", sorted({m[0] for m in MISFITS}, key=lambda f: f.__name__))
def test_the_same_on_the_gpu(op):
    d = "cuda:0"
    assert _call(op, op(d)) is not None
    for o, name, misfit in MISFITS:
        if o is op:
            _refuses(op, name, misfit, d)
            a = dict(op(d))
            a[name] = op("cpu")[name]              # an operand on another device than the input
            with pytest.raises(RuntimeError):
                _call(op, a)
    torch.cuda.synchronize()
    assert _call(op, op(d)) is not None


def _shifted(t, by=1):
    """The same values in memory that starts ``by`` elements past an aligned address."""
    flat = torch.empty(t.numel() + 16, dtype=t.dtype, device=t.device)[by:by + t.numel()]
    v = flat.as_strided(t.size(), t.stride())
    v.copy_(t)
    assert v.data_ptr() % 16
    return v


@pytest.mark.gpu
@pytest.mark.parametrize("what", ["input", "weight", "gradient"])
@pytest.mark.parametrize("cin,cout,k,stride", [(16, 16, 3, 1), (32, 32, 3, 1), (64, 64, 3, 1), (16, 32, 3, 2), (128, 64, 3, 1), (64, 128, 1, 1),
                                               (64, 64, 1, 2), (3, 16, 3, 1)])
def test_convolutions_take_tensors_that_start_anywhere(cin, cout, k, stride, what):
    from eagersgd_b200.ops import functional as ops
    g = torch.Generator().manual_seed(cin + cout + k)
    x, w = torch.randn(3, cin, 8, 8, generator=g), torch.randn(cout, cin, k, k, generator=g)
    cl = lambda t: t.cuda().bfloat16().contiguous(memory_format=torch.channels_last)
    x, w = cl(x), cl(w)
    dy = cl(torch.randn(3, cout, (8 - 1) // stride + 1, (8 - 1) // stride + 1, generator=g))

    def run(x, w, dy):
        x, w = x.detach().requires_grad_(cin > 3), w.detach().requires_grad_()
        y, st = ops.conv2d(x, w, stride, k // 2, want_stats=True)
        y.backward(dy)
        return [t.float() for t in (y.detach(), st, w.grad, x.grad) if t is not None]

    ref = run(x, w, dy)
    got = run(_shifted(x) if what == "input" else x, _shifted(w) if what == "weight" else w, _shifted(dy) if what == "gradient" else dy)
    for a, b in zip(got, ref):
        assert (a - b).norm() <= 1e-3 * b.norm()         # sums meet in atomics; the operands are the same


@pytest.mark.gpu
def test_the_other_operators_take_tensors_that_start_anywhere():
    from eagersgd_b200.ops import functional as ops
    from eagersgd_b200.ops.lstm import lstm_layer
    g = torch.Generator().manual_seed(1)
    rnd = lambda *s: torch.randn(*s, generator=g).cuda()
    cl = lambda t: t.bfloat16().contiguous(memory_format=torch.channels_last)
    x4, r4, gamma, beta = cl(rnd(2, 16, 6, 6)), cl(rnd(2, 16, 6, 6)), rnd(16), rnd(16)
    x2, w2, b2 = rnd(16, 32).bfloat16(), rnd(24, 32).bfloat16(), rnd(24).bfloat16()
    x3, w_ih, w_hh, b3 = rnd(3, 8, 16).bfloat16(), (0.1 * rnd(512, 16)).bfloat16(), (0.1 * rnd(512, 128)).bfloat16(), rnd(512)
    calls = [(lambda x, r, a, b: ops.bn_act(x, a, b, None, None, residual=r), (x4, r4, gamma, beta)),
             (ops.linear, (x2, w2, b2)), (ops.max_pool_3x3_s2, (x4,)), (ops.global_avg_pool, (x4,)), (lstm_layer, (x3, w_ih, w_hh, b3))]
    for f, args in calls:
        def run(args, shift_dy):
            args = [a.detach().requires_grad_() for a in args]
            y = f(*args)
            dy = torch.ones_like(y)
            y.backward(_shifted(dy) if shift_dy else dy)
            return [y.detach().float()] + [a.grad.float() for a in args]
        ref = run(args, False)
        for got in (run([_shifted(a) for a in args], False), run(args, True)):
            for a, b in zip(got, ref):
                assert (a - b).norm() <= 1e-3 * b.norm() + 1e-6


@pytest.mark.gpu
@pytest.mark.parametrize("rows", [65535 * 16, 65535 * 16 + 1, 2 * 65535 * 16 + 17])
def test_linear_over_more_rows_than_a_grid_has_blocks(rows):
    """The gradient of a dense layer over a million rows and more; its bias gradient is the column sum."""
    from eagersgd_b200.ops import functional as ops
    g = torch.Generator(device="cuda").manual_seed(rows)
    x = torch.randn(rows, 8, device="cuda", generator=g).bfloat16().requires_grad_()
    w, b = torch.randn(10, 8, device="cuda", generator=g).bfloat16().requires_grad_(), torch.zeros(10, device="cuda").requires_grad_()
    dy = torch.randn(rows, 10, device="cuda", generator=g)
    ops.linear(x, w, b).backward(dy)
    dy16 = dy.bfloat16().double()
    for got, ref, tol in ((x.grad, dy16 @ w.detach().double(), 4e-3), (w.grad, dy16.t() @ x.detach().double(), 4e-3),
                          (b.grad, dy.double().sum(0), 1e-4)):
        assert (got.double() - ref).norm() <= tol * ref.norm()      # one bf16 rounding; fp32 sums of a million terms


@pytest.mark.gpu
def test_stem_filters_in_fp32():
    """The stem packs its filters, from any floating type; the gradient comes back in that type."""
    from eagersgd_b200.ops import functional as ops
    g = torch.Generator().manual_seed(5)
    x = torch.randn(2, 3, 16, 16, generator=g).cuda().bfloat16().contiguous(memory_format=torch.channels_last)
    w = torch.randn(16, 3, 7, 7, generator=g).cuda().bfloat16().float()
    outs = []
    for dtype in (torch.bfloat16, torch.float32):
        wt = w.to(dtype).requires_grad_()
        y, _ = ops.conv2d(x, wt, 2, 3)
        y.square().sum().backward()
        assert wt.grad.dtype == dtype
        outs.append((y.detach().float(), wt.grad.float()))
    assert torch.equal(outs[0][0], outs[1][0]) and (outs[0][1] - outs[1][1]).norm() <= 1e-3 * outs[0][1].norm()


@pytest.mark.gpu
def test_conv1x1_takes_a_matrix_and_no_larger_filter():
    from eagersgd_b200.ops import functional as ops
    g = torch.Generator().manual_seed(6)
    x = torch.randn(2, 16, 8, 8, generator=g).cuda().bfloat16().contiguous(memory_format=torch.channels_last)
    w = torch.randn(24, 16, generator=g).cuda().bfloat16().requires_grad_()
    y = ops.conv1x1(x, w)
    assert torch.equal(y, ops.conv1x1(x, w.view(24, 16, 1, 1)))
    y.sum().backward()
    assert w.grad.shape == w.shape
    with pytest.raises(RuntimeError):
        ops.conv1x1(x, torch.zeros(24, 16, 3, 3, device="cuda", dtype=torch.bfloat16))


@pytest.mark.gpu
@pytest.mark.parametrize("width", [10, 16, 1 << 16])
def test_softmax_of_a_column_slice(width):
    """The gradient of a slice is no larger than the slice, whatever it was cut from."""
    from eagersgd_b200.ops import functional as ops
    g = torch.Generator().manual_seed(width)
    labels = torch.randint(0, 10, (64,), generator=g).cuda()
    logits = torch.randn(64, width, generator=g).cuda()[:, :10].requires_grad_()
    torch.cuda.synchronize()
    before = torch.cuda.memory_allocated()
    loss = ops.softmax_cross_entropy(logits, labels)
    assert torch.cuda.memory_allocated() - before < 1 << 16
    loss.backward()
    ref = logits.detach().clone().requires_grad_()
    want = torch.nn.functional.cross_entropy(ref, labels)
    want.backward()
    assert abs(loss.item() - want.item()) < 1e-5 and torch.allclose(logits.grad, ref.grad, atol=1e-6)


@pytest.mark.gpu
def test_conv2d_with_a_stride_per_dimension():
    from eagersgd_b200.ops import functional as ops
    g = torch.Generator().manual_seed(8)
    cl = lambda *s: torch.randn(*s, generator=g).cuda().bfloat16().contiguous(memory_format=torch.channels_last)
    x, w = cl(2, 64, 9, 9), cl(64, 64, 3, 3)
    for stride, padding in (((2, 1), (1, 1)), ((1, 2), 0), (1, (0, 1))):
        y, stats, tap = ops.conv2d(x, w, stride, padding, want_stats=True, tap_input=True)
        ref = torch.nn.functional.conv2d(x.float(), w.float(), None, stride, padding)
        assert stats is None and tap is x and (y.float() - ref).norm() < 5e-3 * ref.norm()
