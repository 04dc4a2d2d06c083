"""The persistent LSTM recurrence (weights resident on chip) against the fp32 restatement, at the edges of its range:
one step, two steps, every way the weights divide between shared and tensor memory, both batch paddings."""
import ctypes as C

import pytest
import torch
import torch.nn.functional as F

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("T,B,H", [(1, 8, 128), (2, 8, 128), (3, 16, 128), (7, 16, 384), (6, 24, 640), (5, 8, 1024), (9, 24, 1152),
                                   (4, 32, 1536), (33, 16, 2048), (4, 32, 1920), (5, 24, 2048), (4, 32, 2048)])
def test_persistent_recurrence(T, B, H):
    from eagersgd_b200.ops.gemm import check_error
    from eagersgd_b200.ops.lstm import lstm_layer, lstm_layer_reference
    from eagersgd_b200.parallel import _native as N
    lib = N.cuda()
    lib.esgd_lstm_persistent_ok.argtypes = [C.c_int] * 3
    # 2048 units backward with more than 16 sequences: the clusters are not all resident, the loop of launches takes it
    assert lib.esgd_lstm_persistent_ok(B, H, 0) == 1 and lib.esgd_lstm_persistent_ok(B, H, 1) == (H < 2048 or B <= 16)
    g = torch.Generator().manual_seed(T * 1000 + H)
    rnd = lambda *s: torch.randn(*s, generator=g).cuda()
    x = (rnd(T, B, 64) * 0.5).to(torch.bfloat16).requires_grad_()
    w_ih = (rnd(4 * H, 64) * 0.1).to(torch.bfloat16).requires_grad_()
    w_hh = (rnd(4 * H, H) / H ** 0.5).to(torch.bfloat16).requires_grad_()
    bias = (rnd(4 * H) * 0.1).requires_grad_()
    y = lstm_layer(x, w_ih, w_hh, bias)
    dy = rnd(T, B, H).to(torch.bfloat16)
    y.backward(dy)
    check_error(y.device)
    ref = [t.detach().float().requires_grad_() for t in (x, w_ih, w_hh, bias)]
    yr = lstm_layer_reference(*ref)
    yr.backward(dy.float())
    assert (y.float() - yr).norm() < 1e-2 * yr.norm()
    for a, b in zip((x, w_ih, w_hh, bias), ref):
        if float(b.grad.norm()) > 0:       # a single step has no recurrent gradient
            assert (a.grad.float() - b.grad).norm() < 2e-2 * b.grad.norm(), tuple(a.shape)
            assert F.cosine_similarity(a.grad.float().flatten(), b.grad.flatten(), dim=0) > 0.999
        else:
            assert float(a.grad.float().abs().max()) == 0.0


@pytest.mark.parametrize("T,B,H", [(5, 32, 128), (12, 32, 256), (3, 24, 384), (40, 8, 2048), (65, 16, 1024)])
def test_issuers_blocks_and_padding(T, B, H):
    """Fewer blocks of the state than warps that fetch or multiply them, batches that fill half of a product, and sequences over
    which every barrier goes round more than once."""
    test_persistent_recurrence(T, B, H)


@pytest.mark.parametrize("T,B,H", [(700, 8, 128), (700, 32, 128), (501, 16, 256), (400, 24, 512), (300, 8, 896)])
def test_long_sequences_with_fewer_blocks_than_fetching_warps(T, B, H):
    """1 to 7 blocks of the state a CTA and eight warps that fetch them, over hundreds of steps: no wait runs out (a warp that has
    no block must not follow the steps, which do not wait for it), and every pass over the same inputs gives the same states."""
    from eagersgd_b200.ops.gemm import check_error
    from eagersgd_b200.ops.lstm import lstm_layer
    g = torch.Generator().manual_seed(T + B + H)
    rnd = lambda *s: torch.randn(*s, generator=g).cuda()
    x = (rnd(T, B, 64) * 0.5).to(torch.bfloat16).requires_grad_()
    w_ih, w_hh = (rnd(4 * H, 64) * 0.1).to(torch.bfloat16), (rnd(4 * H, H) / H ** 0.5).to(torch.bfloat16)
    bias, dy = rnd(4 * H) * 0.1, rnd(T, B, H).to(torch.bfloat16)
    seen = []
    for _ in range(5):
        x.grad = None
        y = lstm_layer(x, w_ih, w_hh, bias)
        y.backward(dy)
        check_error(y.device)
        seen.append((y.detach().clone(), x.grad))
    # the order of every sum is fixed, in the recurrence and in the product behind it
    assert all(torch.equal(a, b) for other in seen[1:] for a, b in zip(seen[0], other))


def test_shapes_outside_the_persistent_range_take_the_loop():
    from eagersgd_b200.parallel import _native as N
    lib = N.cuda()
    lib.esgd_lstm_persistent_ok.argtypes = [C.c_int] * 3
    for B, H in ((40, 128), (12, 128), (16, 192), (16, 2176), (16, 64)):
        assert lib.esgd_lstm_persistent_ok(B, H, 0) == 0
