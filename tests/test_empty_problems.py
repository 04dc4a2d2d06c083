"""A launcher that is given an empty problem, or an operand that its loads cannot start at, answers with an error code.  Each
call runs in a process of its own: an integer division by zero ends it."""
import subprocess
import sys

import pytest

from eagersgd_b200 import _build

# launcher, arguments of a small problem (pointers as text), position of the size that is set to zero
_P = "C.c_void_p(0)"
EMPTY = [("esgd_conv_narrow_fwd", [_P] * 3 + [2, 8, 8, 64, 64, 1] + [_P] * 3 + [0] + [_P] * 3, (3, 4, 5, 8)),
         ("esgd_conv_narrow_fwd", [_P] * 3 + [2, 32, 32, 16, 16, 1] + [_P] * 3 + [0] + [_P] * 3, (3, 4, 5, 8)),
         ("esgd_conv_narrow_dgrad", [_P] * 3 + [2, 8, 8, 32, 32] + [_P] * 3, (3, 4, 5)),
         ("esgd_conv_narrow_wgrad", [_P] * 3 + [2, 8, 8, 32, 64, 1, _P], (3, 4, 5, 8)),
         ("esgd_bn_stats", [_P, "C.c_int64(64)", 8] + [_P] * 3, (2,)),
         ("esgd_bn_fwd", [_P] * 11 + ["C.c_int64(64)", 8, 1, "C.c_float(0.1)", "C.c_float(1e-5)", _P], (12,))]


@pytest.mark.parametrize("fn,args,zero", [(f, a, z) for f, a, zs in EMPTY for z in zs])
def test_an_empty_problem_is_an_error_code_and_not_the_end_of_the_process(fn, args, zero):
    args = [str(0 if i == zero else a) for i, a in enumerate(args)]
    code = "import ctypes as C\nprint(C.CDLL(%r).%s(%s))" % (_build.build_cuda(), fn, ", ".join(args))
    r = subprocess.run([sys.executable, "-c", code], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0 and int(r.stdout) < 0, (r.returncode, r.stdout, r.stderr[-300:])


@pytest.mark.parametrize("fn,args", [(f, a) for f, a, _ in EMPTY if "narrow" in f])
def test_an_operand_that_is_not_aligned_is_left_to_another_kernel(fn, args):
    args = [str(a) for a in args]
    args[0] = "C.c_void_p(4098)"                   # 16-byte loads would start there
    code = "import ctypes as C\nprint(C.CDLL(%r).%s(%s))" % (_build.build_cuda(), fn, ", ".join(args))
    r = subprocess.run([sys.executable, "-c", code], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0 and int(r.stdout) == -100, (r.returncode, r.stdout, r.stderr[-300:])


@pytest.mark.parametrize("fn,args", [("esgd_maxpool3x3s2_fwd", [_P] * 3 + [0, 8, 8, 64, _P]), ("esgd_maxpool3x3s2_bwd", [_P] * 3 + [0, 8, 8, 64, _P]),
                                     ("esgd_avgpool_fwd", [_P] * 2 + [0, 49, 64, _P])])
def test_pooling_no_images_is_nothing_to_do(fn, args):
    code = "import ctypes as C\nprint(C.CDLL(%r).%s(%s))" % (_build.build_cuda(), fn, ", ".join(str(a) for a in args))
    r = subprocess.run([sys.executable, "-c", code], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0 and int(r.stdout) == 0, (r.returncode, r.stdout, r.stderr[-300:])


@pytest.mark.gpu
def test_pooling_no_images():
    import torch
    from eagersgd_b200.ops import functional as ops
    for f, shape in ((ops.max_pool_3x3_s2, (0, 64, 4, 4)), (ops.global_avg_pool, (0, 64))):
        x = torch.empty(0, 64, 8, 8, device="cuda", dtype=torch.bfloat16).contiguous(memory_format=torch.channels_last).requires_grad_()
        y = f(x)
        assert y.shape == shape
        y.sum().backward()
        assert x.grad.shape == x.shape
