"""ResNet v1 / v1.5 / v2 for CIFAR (6n+2) and ImageNet (18 … 200).

Architecture, initialisation and *variable creation order* follow the reference
model so that checkpoints can be exported in its layout
(test-models/.../official/resnet/resnet_model.py:51-554, cifar10_main.py:179-219,
imagenet_main_eagersgd.py:290-330; PyTorch variants in
deep500/networks/pytorch_resnet.py): fixed padding for strided convolutions,
batch-norm momentum 0.997 / eps 1e-5, zero-initialised gamma on the last
batch-norm of every residual block, projection shortcuts created before the
main path, the stride on the 3x3 convolution of a bottleneck ("v1.5").
Activations are NHWC (channels_last) bf16 on GPUs.
"""
from __future__ import annotations

import weakref
from typing import List, Tuple

import torch
import torch.nn as nn

from ..ops import functional as ops

BN_MOMENTUM_TF = 0.997  # tf decay; torch momentum = 1 - decay
BN_EPS = 1e-5

# what the fused inference path keeps per network (its layers, the device table of its batch norms); not an attribute of the
# module, which has to stay copyable and picklable
_eval_state = weakref.WeakKeyDictionary()

IMAGENET_BLOCKS = {
    18: ("building", [2, 2, 2, 2]), 34: ("building", [3, 4, 6, 3]), 50: ("bottleneck", [3, 4, 6, 3]),
    101: ("bottleneck", [3, 4, 23, 3]), 152: ("bottleneck", [3, 8, 36, 3]), 200: ("bottleneck", [3, 24, 36, 3]),
}


class BatchNormAct(nn.BatchNorm2d):
    """Batch norm fused with an optional residual add and ReLU (one kernel pass each way)."""

    # Ghost batch norm: statistics over consecutive groups of this many samples instead of the whole batch
    # (the reference's --virtual_batch_size, official/resnet/resnet_model.py:45-60); None: the whole batch.
    virtual_batch_size = None

    def forward(self, y, relu: bool = True, residual=None, stats=None):  # noqa: D102
        v = self.virtual_batch_size
        if v and self.training and y.shape[0] > v:
            outs = [ops.bn_act(y[i:i + v], self.weight, self.bias, self.running_mean, self.running_var, self.momentum,
                               relu, None if residual is None else residual[i:i + v], None, True)
                    for i in range(0, y.shape[0], v)]
            return torch.cat(outs)
        return ops.bn_act(y, self.weight, self.bias, self.running_mean, self.running_var, self.momentum, relu,
                          residual, stats, self.training)


def _bn(ch: int, zero_gamma: bool = False) -> BatchNormAct:
    bn = BatchNormAct(ch, eps=BN_EPS, momentum=1.0 - BN_MOMENTUM_TF)
    if zero_gamma:
        nn.init.zeros_(bn.weight)
    return bn


class _Conv(nn.Conv2d):
    """conv2d_fixed_padding: explicit symmetric padding when strided (resnet_model.py:63-101).

    ``forward`` returns ``(y, stats)`` where ``stats`` holds the per-channel sum and sum of
    squares of ``y`` when the kernel produced them in its epilogue (else ``None``).
    """

    def __init__(self, cin, cout, k, stride):
        super().__init__(cin, cout, k, stride=stride, padding=(k - 1) // 2, bias=False)
        # variance_scaling_initializer() of the reference: fan-in scaling
        nn.init.kaiming_normal_(self.weight, mode="fan_in", nonlinearity="linear")

    def forward(self, x, tap_input: bool = False):  # noqa: D102
        return ops.conv2d(x, self.weight, self.stride[0], self.padding[0], want_stats=self.training,
                          tap_input=tap_input)


def _bare(m: nn.Module, cls) -> bool:
    """Calling ``m`` does what ``cls.forward`` does in training, and nothing else."""
    return type(m) is cls and m.training and not (m._forward_hooks or m._forward_pre_hooks or m._backward_hooks or
                                                  m._backward_pre_hooks or "forward" in m.__dict__)


def _train_layer(conv, bn):
    """A convolution and its batch norm for ``ops.residual_block``; None when somebody could see the two being skipped."""
    if not _bare(conv, _Conv) or not _bare(bn, BatchNormAct) or bn.virtual_batch_size or bn.momentum is None or not bn.affine:
        return None
    w, p, b = conv._parameters.get("weight"), bn._parameters, bn._buffers
    if w is None or "running_mean" not in b or "running_var" not in b or p.get("weight") is None or p.get("bias") is None:
        return None
    return (w, conv.stride[0], conv.padding[0], p["weight"], p["bias"], b["running_mean"], b["running_var"], bn.momentum)


class _Block(nn.Module):
    def __init__(self, cin, filters, stride, kind, version, project, registry):
        super().__init__()
        self.kind, self.version = kind, version
        cout = filters * 4 if kind == "bottleneck" else filters
        self.proj = self.proj_bn = None
        if version == 2:
            self.pre_bn = _bn(cin)
            registry.append(("bn", self.pre_bn))
        if project:
            self.proj = _Conv(cin, cout, 1, stride)
            registry.append(("conv", self.proj))
            if version == 1:
                self.proj_bn = _bn(cout)
                registry.append(("bn", self.proj_bn))
        convs, bns = [], []
        if kind == "bottleneck":
            spec = [(cin, filters, 1, 1), (filters, filters, 3, stride), (filters, cout, 1, 1)]
        else:
            spec = [(cin, filters, 3, stride), (filters, filters, 3, 1)]
        for idx, (ci, co, k, s) in enumerate(spec):
            conv = _Conv(ci, co, k, s)
            convs.append(conv)
            registry.append(("conv", conv))
            last = idx == len(spec) - 1
            if version == 1 or not last:
                bn = _bn(co, zero_gamma=(last and version == 1))
                bns.append(bn)
                registry.append(("bn", bn))
        self.convs = nn.ModuleList(convs)
        self.bns = nn.ModuleList(bns)
        self.cout = cout

    def _fused_train(self, x):
        """The block in one call of the operators' library, or None where its layers have to be called one by one."""
        if not self.training or not ops.native(x) or nn.modules.module._has_any_global_hook():
            return None
        m = self._modules
        if len(m["convs"]) != len(m["bns"]):
            return None
        layers = [_train_layer(c, b) for c, b in zip(m["convs"]._modules.values(), m["bns"]._modules.values())]
        proj = _train_layer(self.proj, self.proj_bn) if self.proj is not None else None
        if any(e is None for e in layers) or (proj is None) != (self.proj is None):
            return None
        return ops.residual_block(x, layers, proj)

    def forward(self, x):
        n = len(self.convs)
        if self.version == 1:
            y = self._fused_train(x)
            if y is not None:
                return y
            # The shortcut branches off the first convolution's tapped input: both gradients of x then meet
            # inside that convolution's data-gradient kernel instead of in a separate addition.
            yc, st, shortcut = self.convs[0](x, tap_input=True)
            if self.proj is not None:
                ys, sts = self.proj(shortcut)
                shortcut = self.proj_bn(ys, relu=False, stats=sts)
            y = x
            for i in range(n):
                if i > 0:
                    yc, st = self.convs[i](y)
                # the last batch norm also adds the shortcut and applies the block's final ReLU
                y = self.bns[i](yc, relu=True, residual=shortcut if i == n - 1 else None, stats=st)
            return y
        pre = self.pre_bn(x, relu=True)
        shortcut = self.proj(pre)[0] if self.proj is not None else x
        y = pre
        for i in range(n):
            yc, st = self.convs[i](y)
            y = self.bns[i](yc, relu=True, stats=st) if i < n - 1 else yc
        return y + shortcut


class ResNet(nn.Module):
    def __init__(self, kind: str, blocks: List[int], num_classes: int, num_filters: int, first_kernel: int,
                 first_stride: int, first_pool: bool, block_strides: List[int], version: int = 1):
        super().__init__()
        assert version in (1, 2)
        self.version = version
        self.registry: List[Tuple[str, nn.Module]] = []  # creation order, for the tf-models variable names
        self.stem = _Conv(3, num_filters, first_kernel, first_stride)
        self.registry.append(("conv", self.stem))
        self.stem_bn = None
        if version == 1:
            self.stem_bn = _bn(num_filters)
            self.registry.append(("bn", self.stem_bn))
        self.first_pool = first_pool
        layers = []
        cin = num_filters
        for i, nb in enumerate(blocks):
            filters = num_filters * (2 ** i)
            for j in range(nb):
                blk = _Block(cin, filters, block_strides[i] if j == 0 else 1, kind, version, j == 0, self.registry)
                layers.append(blk)
                cin = blk.cout
        self.blocks = nn.ModuleList(layers)
        self.final_bn = None
        if version == 2:
            self.final_bn = _bn(cin)
            self.registry.append(("bn", self.final_bn))
        self.fc = nn.Linear(cin, num_classes)
        self.registry.append(("dense", self.fc))
        self.feature_dim = cin

    # ---- inference: every convolution with its batch norm, shortcut and ReLU as one kernel
    def _eval_layers(self):
        """What the fused pass stands in for, or None when the network has another structure."""
        m = self._modules
        stem, blocks = m["stem"], m["blocks"]
        convs, norms, modules = [stem], [b for b in (m.get("stem_bn"), m.get("final_bn")) if b is not None], [(blocks, None)]
        for blk in blocks._modules.values():
            if type(blk) is not _Block or blk.version != self.version:
                return None
            m = blk._modules
            proj, proj_bn, pre_bn = m.get("proj"), m.get("proj_bn"), m.get("pre_bn")
            if len(m["convs"]) != len(m["bns"]) + (blk.version == 2) or (blk.version == 1 and (proj is None) != (proj_bn is None)):
                return None
            modules += [(blk, _Block), (m["convs"], None), (m["bns"], None)]
            convs += [c for c in (*m["convs"]._modules.values(), proj) if c is not None]
            norms += [b for b in (*m["bns"]._modules.values(), proj_bn, pre_bn) if b is not None]
        modules += [(c, _Conv) for c in convs] + [(b, BatchNormAct) for b in norms]
        return ops.eval_layers(self._modules, modules, convs, norms)

    def _fused_eval(self, x):
        """The coefficients of the network's batch norms by module, when the fused inference path applies: no gradients,
        every layer in evaluation mode and what it was built as, and nobody listening to a layer's output; else None.  Asked
        in every pass: a layer may have been exchanged, parametrized or hooked since the last one."""
        if self.training or torch.is_grad_enabled() or not ops.native(x) or nn.modules.module._has_any_global_hook():
            return None
        st = _eval_state.setdefault(self, {})
        for renewed in (False, True):
            layers = self._eval_layers() if renewed else st.get("layers")
            coef = ops.eval_coefficients(layers, st) if layers is not None else None
            if coef is not None:
                st["layers"] = layers
                return dict(zip(layers.norms, coef))
        return None

    @staticmethod
    def _conv_eval(conv, bn, x, coef, relu, residual=None):
        y = ops.conv_bn_eval(x, conv.weight, conv.stride[0], conv.padding[0], coef[bn] if bn is not None else None, relu, residual)
        if y is None:
            y = conv(x)[0]
            if bn is not None:
                return bn(y, relu=relu, residual=residual)
            y = y + residual if residual is not None else y
        return y

    def _features_eval(self, x, coef):
        conv = self._conv_eval
        x = conv(self.stem, self.stem_bn, x, coef, self.stem_bn is not None)
        if self.first_pool:
            x = ops.max_pool_3x3_s2(x)
        for blk in self.blocks:
            if self.version == 1:
                m = blk._modules
                layers = [(c._parameters["weight"], c.stride[0], c.padding[0], coef[b])
                          for c, b in zip(m["convs"]._modules.values(), m["bns"]._modules.values())]
                proj = blk.proj
                y = ops.residual_block_eval(x, layers, None if proj is None else
                                            (proj._parameters["weight"], proj.stride[0], proj.padding[0], coef[blk.proj_bn]))
                if y is not None:
                    x = y
                    continue
            n, y, shortcut = len(blk.convs), x, x
            if self.version == 1:
                if blk.proj is not None:
                    shortcut = conv(blk.proj, blk.proj_bn, x, coef, False)
                for i in range(n):
                    y = conv(blk.convs[i], blk.bns[i], y, coef, True, shortcut if i == n - 1 else None)
            else:
                y = blk.pre_bn(x, relu=True)
                if blk.proj is not None:
                    shortcut = conv(blk.proj, None, y, coef, False)
                for i in range(n):
                    last = i == n - 1
                    y = conv(blk.convs[i], None if last else blk.bns[i], y, coef, not last, shortcut if last else None)
            x = y
        if self.final_bn is not None:
            x = self.final_bn(x, relu=True)
        return ops.global_avg_pool(x)

    def features(self, x):
        coef = self._fused_eval(x)
        if coef is not None:
            return self._features_eval(x, coef)
        x, st = self.stem(x)
        if self.stem_bn is not None:
            x = self.stem_bn(x, relu=True, stats=st)
        if self.first_pool:
            x = ops.max_pool_3x3_s2(x)
        for blk in self.blocks:
            x = blk(x)
        if self.final_bn is not None:
            x = self.final_bn(x, relu=True)
        return ops.global_avg_pool(x)

    def forward(self, x):
        """Logits (fp32 on the native path)."""
        return ops.linear(self.features(x), self.fc.weight, self.fc.bias)


def imagenet_resnet(size: int = 50, version: int = 1, num_classes: int = 1001) -> ResNet:
    """ImagenetModel (imagenet_main_eagersgd.py:290-330).  ``version=1`` is the
    reference's v1 with the stride on the 3x3 convolution, i.e. "ResNet v1.5"."""
    kind, blocks = IMAGENET_BLOCKS[size]
    return ResNet(kind, blocks, num_classes, 64, 7, 2, True, [1, 2, 2, 2], version)


def cifar_resnet(size: int = 32, version: int = 1, num_classes: int = 10) -> ResNet:
    """Cifar10Model: 6n+2 layers, 16/32/64 filters, building blocks (cifar10_main.py:179-219)."""
    if size % 6 != 2:
        raise ValueError("resnet_size must be 6n + 2")
    n = (size - 2) // 6
    return ResNet("building", [n] * 3, num_classes, 16, 3, 1, False, [1, 2, 2], version)


def count_parameters(model: nn.Module) -> Tuple[int, int]:
    ps = [p for p in model.parameters() if p.requires_grad]
    return len(ps), sum(p.numel() for p in ps)
