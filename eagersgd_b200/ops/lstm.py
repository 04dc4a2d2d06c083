"""LSTM layer on the hand-written kernels: tensor-core projections + a persistent recurrence.

* ``x . W_ih^T`` for every time step is ONE tcgen05 GEMM ([T*B, I] x [4H, I]^T).
* The recurrence is one kernel per direction that keeps the recurrent weights on chip for the whole sequence
  (csrc/cuda/lstm_persistent.cu), for H a multiple of 128 up to 2048 and batches up to 32 (backward at H = 2048: up to 16);
  other shapes take a native loop of split-K GEMMs and cell kernels (csrc/cuda/lstm_cell.cu).
* The three weight / input gradients are single large GEMMs over all time steps.
* The autograd function around them is C++ (csrc/torch/ops.cpp).

Stands where the reference calls ``torch.nn.LSTM`` (cuDNN) in its video classifier
(deep500 samples/ucf101_resnetlstm.py:41-59).  Gate order i, f, g, o; weights are
``[4H, in]`` as in ``torch.nn.LSTM``.
"""
from __future__ import annotations

import torch

from .. import _build


def lstm_layer(x: torch.Tensor, w_ih: torch.Tensor, w_hh: torch.Tensor, bias: torch.Tensor) -> torch.Tensor:
    """x: [T, B, I] -> h: [T, B, H], zero initial state.  ``bias`` is b_ih + b_hh (fp32 [4H])."""
    T, B, I = x.shape
    H = w_hh.shape[1]
    if x.is_cuda and x.dtype == torch.bfloat16 and B % 8 == 0 and I % 8 == 0 and H % 8 == 0:
        return _build.load_torch().lstm_layer(x.contiguous(), w_ih, w_hh, bias.float())
    return lstm_layer_reference(x, w_ih, w_hh, bias)


def lstm_layer_reference(x, w_ih, w_hh, bias):
    """Plain PyTorch restatement (oracle and CPU path)."""
    T, B, _ = x.shape
    H = w_hh.shape[1]
    h = x.new_zeros(B, H)
    c = x.new_zeros(B, H, dtype=torch.float32)
    out = []
    for t in range(T):
        pre = (x[t] @ w_ih.t() + h @ w_hh.t()).float() + bias.float()
        i, f, g, o = pre.chunk(4, dim=-1)
        c = torch.sigmoid(f) * c + torch.sigmoid(i) * torch.tanh(g)
        h = (torch.sigmoid(o) * torch.tanh(c)).to(x.dtype)
        out.append(h)
    return torch.stack(out)
