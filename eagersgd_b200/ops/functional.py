"""Operators over the hand-written sm_100a kernels (NHWC bf16 activations).

Activations are 4-D ``channels_last`` tensors, i.e. ``[N, H, W, C]`` in memory,
which makes a 1x1 convolution a plain ``[N*H*W, Cin] x [Cout, Cin]^T`` GEMM on
the tcgen05 tensor cores, with the batch-norm statistics accumulated in the GEMM
epilogue.  The autograd functions around the kernels are C++ (csrc/torch/ops.cpp);
this module chooses between them and the same mathematics in PyTorch, which is
what CPU tensors, other data types and the oracles in the tests use.
"""
from __future__ import annotations

import contextlib
import os
from typing import Optional

import torch
import torch.nn.functional as F

from .. import _build

BN_EPS = 1e-5

_ext_module = None


def _ext():
    global _ext_module
    if _ext_module is None:
        _ext_module = _build.load_torch()
    return _ext_module


_reference_only = False
_default_arena = None


@contextlib.contextmanager
def zero_arena(device, numel: int, arena=None):
    """Serve the operators' zeroed fp32 scratch from one buffer of ``numel`` floats for the duration of a step: a single
    memset instead of a fill kernel per operator.  ``arena`` (``new_zero_arena()``): the buffer of the caller's own, which
    a captured CUDA graph needs for as long as it is replayed; default: one shared by the process."""
    global _default_arena
    if arena is None:
        if _default_arena is None:
            _default_arena = new_zero_arena()
        arena = _default_arena
    arena.begin(torch.device(device), numel)
    try:
        yield
    finally:
        arena.end()


def new_zero_arena():
    return _ext().ZeroArena()


def zeros_f32(shape, device):
    return _ext().zeros_f32(list(shape), torch.device(device))


class reference_ops:
    """Context manager: run every op through its PyTorch restatement (the test oracle)."""

    def __enter__(self):
        global _reference_only
        self._prev, _reference_only = _reference_only, True

    def __exit__(self, *a):
        global _reference_only
        _reference_only = self._prev


def native(x: torch.Tensor) -> bool:
    return x.is_cuda and x.dtype == torch.bfloat16 and not _reference_only


# Narrow convolutions (16- and 32-channel layers) on the tensor-core path; ESGD_SMALL_CHANNELS=library keeps them on
# PyTorch's convolution instead.
_SMALL_CHANNELS_NATIVE = os.environ.get("ESGD_SMALL_CHANNELS", "native") != "library"


# --------------------------------------------------------------------------- convolution / dense
def wgrad_splits(pixels: int, cout: int, cin: int, sms: int = 148) -> int:
    """Split-K factor of a weight-gradient GEMM (K = pixels)."""
    return _ext().wgrad_splits(pixels, cout, cin, sms)


def _conv1x1_reference(x, w, want_stats, tap_input):
    y = F.conv2d(x, w)
    outs = (y,)
    if want_stats:
        yf = y.float()
        outs += (torch.stack([yf.sum((0, 2, 3)), (yf * yf).sum((0, 2, 3))]).detach(),)
    if tap_input:
        outs += (x,)
    return outs if len(outs) > 1 else y


def conv1x1(x: torch.Tensor, w: torch.Tensor, want_stats: bool = False, tap_input: bool = False):
    """1x1 convolution.  ``tap_input=True`` appends ``x`` itself to the outputs (use it for the shortcut of a
    residual block: the two gradients of ``x`` are then added inside the data-gradient GEMM)."""
    if native(x):
        if tuple(w.shape[2:]) != (1, 1):        # [outputs, inputs] does as well; anything larger is no 1x1 filter
            w = w.reshape(w.shape[0], x.shape[1], 1, 1)
        r = _ext().conv2d(x, w, 1, 0, want_stats, tap_input, _SMALL_CHANNELS_NATIVE)
        if r is not None:
            outs = tuple(t for t in r if t is not None)
            return outs if len(outs) > 1 else outs[0]
    return _conv1x1_reference(x, w, want_stats, tap_input)


def conv2d(x: torch.Tensor, w: torch.Tensor, stride: int = 1, padding: int = 0, want_stats: bool = False,
           tap_input: bool = False):
    """NHWC convolution; returns ``(y, stats)`` (``stats`` is None unless produced by the kernel epilogue).

    1x1 kernels run as tcgen05 GEMMs (a strided 1x1 first gathers the kept pixels).  With ``tap_input`` a
    third value is returned: the tensor a residual block should feed its shortcut from (the input itself, or
    for the fused 1x1 path an alias whose gradient is added inside the data-gradient GEMM).
    """
    if native(x) and not isinstance(stride, (tuple, list)) and not isinstance(padding, (tuple, list, str)):
        r = _ext().conv2d(x, w, stride, padding, want_stats, tap_input, _SMALL_CHANNELS_NATIVE)
        if r is None and w.shape[2] == 1 and w.shape[3] == 1 and padding == 0 and stride > 2:
            xs = x[:, :, ::stride, ::stride].contiguous(memory_format=torch.channels_last)
            r = _ext().conv2d(xs, w, 1, 0, want_stats, False, _SMALL_CHANNELS_NATIVE)
            r = r and (r[0], r[1], x)
        if r is not None:
            return r if tap_input else r[:2]
    y = F.conv2d(x, w, None, stride, padding)
    return (y, None, x) if tap_input else (y, None)


def linear(x: torch.Tensor, w: torch.Tensor, b: Optional[torch.Tensor] = None) -> torch.Tensor:
    """Dense layer; fp32 logits out of bf16 operands on the native path, for any number of outputs."""
    if native(x) and (w.shape[0] % 8 == 0 or _SMALL_CHANNELS_NATIVE):
        r = _ext().linear(x, w, b)
        if r is not None:
            return r
    return F.linear(x, w, b)


# --------------------------------------------------------------------------- batch norm (+ residual) (+ ReLU)
def bn_act(y: torch.Tensor, gamma: torch.Tensor, beta: torch.Tensor, running_mean: Optional[torch.Tensor],
           running_var: Optional[torch.Tensor], momentum: float = 0.003, relu: bool = True,
           residual: Optional[torch.Tensor] = None, stats: Optional[torch.Tensor] = None,
           training: bool = True) -> torch.Tensor:
    """z = act(batch_norm(y) [+ residual]) with batch statistics (training) in fused kernels."""
    if native(y) and training and y.shape[1] % 8 == 0 and gamma.dtype == torch.float32:
        return _ext().bn_act(y, gamma, beta, residual, running_mean, running_var, momentum, relu, stats)
    z = F.batch_norm(y, running_mean, running_var, gamma, beta, training, momentum, BN_EPS)
    if residual is not None:
        z = z + residual
    return F.relu(z) if relu else z


def residual_block(x: torch.Tensor, layers, proj=None) -> Optional[torch.Tensor]:
    """A residual block in training: ``conv2d`` and ``bn_act`` of every layer -- (filter, stride, padding, gamma, beta, running
    mean, running variance, momentum) -- in one call, the shortcut through ``proj`` (a layer without ReLU) or straight; None for
    shapes the kernels do not take."""
    return _ext().residual_block(x, layers, proj, _SMALL_CHANNELS_NATIVE) if native(x) else None


# --------------------------------------------------------------------------- inference: convolution + batch norm in one kernel
def bn_coefficients(layers, store):
    """Scale and shift (``[2 * C]`` fp32, one after the other) of each inference batch norm in ``layers`` -- tuples of gamma,
    beta, running mean, running variance -- from one launch; empty unless all of them are fp32 and on the GPU.  ``store``: a
    dict of the caller's that keeps the device table."""
    if "bn" not in store:
        store["bn"] = _ext().BnCoefficients()
    return store["bn"].compute(layers)


def eval_layers(children, modules, convs, norms):
    """The layers of a network for which ``conv_bn_eval`` and ``residual_block_eval`` stand in: pairs of a module and the type it
    was built as (None: a container), its convolutions and its batch norms, and the network's ``_modules``."""
    return _ext().EvalLayers(children, modules, convs, norms)


def eval_coefficients(layers, store) -> Optional[list]:
    """Like ``bn_coefficients`` for the batch norms of ``eval_layers``, one after the other; None when one of the layers is no
    longer what it was, is in training mode or has a hook, or when a tensor is not fp32 on the GPU."""
    if "bn" not in store:
        store["bn"] = _ext().BnCoefficients()
    return layers.coefficients(store["bn"])


def conv_bn_eval(x: torch.Tensor, w: torch.Tensor, stride: int, padding: int, coef: Optional[torch.Tensor], relu: bool,
                 residual: Optional[torch.Tensor] = None) -> Optional[torch.Tensor]:
    """act(scale * conv(x) + shift [+ residual]) rounded once, without autograd; None for shapes the kernels do not take."""
    return _ext().conv_bn_eval(x, w, stride, padding, coef, residual, relu, _SMALL_CHANNELS_NATIVE)


def residual_block_eval(x: torch.Tensor, layers, proj=None) -> Optional[torch.Tensor]:
    """A residual block in inference, like ``residual_block``: layers of (filter, stride, padding, coefficients)."""
    return _ext().residual_block_eval(x, layers, proj, _SMALL_CHANNELS_NATIVE)


# --------------------------------------------------------------------------- softmax cross-entropy
def softmax_cross_entropy(logits: torch.Tensor, labels: torch.Tensor) -> torch.Tensor:
    """Mean sparse softmax cross-entropy; forward and gradient come out of one kernel."""
    if logits.is_cuda and logits.dtype in (torch.float32, torch.bfloat16) and labels.dtype == torch.int64 \
            and not _reference_only:
        return _ext().softmax_ce(logits, labels)
    return F.cross_entropy(logits.float(), labels)


# --------------------------------------------------------------------------- pooling
def max_pool_3x3_s2(x: torch.Tensor) -> torch.Tensor:
    if native(x) and x.shape[1] % 8 == 0:
        return _ext().max_pool(x)
    return F.max_pool2d(x, 3, 2, 1)


def global_avg_pool(x: torch.Tensor) -> torch.Tensor:
    """[N, C, H, W] -> [N, C] mean over H, W."""
    if native(x) and x.shape[1] % 8 == 0:
        return _ext().avg_pool(x)
    return torch.flatten(F.adaptive_avg_pool2d(x, 1), 1)
