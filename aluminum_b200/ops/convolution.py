"""Convolutions in training under 16-bit autocast.

A network's first convolution - 7 x 7, every two pixels, border 3, three channels - on a layout that tensor cores take
(``kernels/stem.cu``); autograd in ``src/torch/activations_autograd.cpp``.

:func:`stem_conv` takes the module that a network holds and runs it that way in training under 16-bit autocast; everything else -
other shapes, images that want a gradient, evaluation, hooks, tracing, functorch transforms - calls the module.  :func:`cast_weights`
casts the weights of several convolutions at once.
"""
from __future__ import annotations

import torch
from torch import nn

from .. import _lib
from .activations import _PLAIN, _TYPES, _bare, _modes_off


def _plain(conv: nn.Module) -> bool:
    """A convolution that is nothing but its weight: no bias, hooks, padding by copies or forward of its own."""
    return type(conv) is nn.Conv2d and _bare(conv) and conv._parameters.get("bias", conv) is None and conv.padding_mode == "zeros"


def _weight_ok(weight, device: int) -> bool:
    return (type(weight) in _PLAIN and weight.dtype == torch.float32 and weight.requires_grad and not weight.is_inference()
            and weight.get_device() == device)


def cast_weights(convs, x: torch.Tensor):
    """The weights of the convolutions in autocast's type, cast with one launch (and their gradients with one), for
    :func:`convolve`; None where autocast is left to cast each in its turn."""
    if not (_modes_off() and torch.is_grad_enabled() and torch.is_autocast_enabled("cuda") and type(x) is torch.Tensor):
        return None
    dtype, device = torch.get_autocast_dtype("cuda"), x.get_device()
    if dtype not in _TYPES or x.dtype != dtype or device != torch.cuda.current_device():
        return None
    weights = []
    for c in convs:
        weight = c._parameters.get("weight") if _plain(c) else None
        if not _weight_ok(weight, device):
            return None
        weights.append(weight)
    return _lib.torch_ops().cast_all.default(weights, dtype)


def convolve(conv: nn.Module, x: torch.Tensor, weight) -> torch.Tensor:
    """``conv(x)`` with its weight in another type; None: the module."""
    if weight is None:
        return conv(x)
    return torch.conv2d(x, weight, None, conv.stride, conv.padding, conv.dilation, conv.groups)


def stem_applies(conv: nn.Module, x: torch.Tensor) -> bool:
    """Whether :func:`stem_conv` runs its own layout of x, and not the module."""
    # (_modes_off() first: a compiler that traces this function sees a constant there and nothing of what follows)
    if not (_modes_off() and torch.is_grad_enabled() and torch.is_autocast_enabled("cuda") and _plain(conv) and conv.training
            and conv.in_channels == 3 and conv.kernel_size == (7, 7) and conv.stride == (2, 2) and conv.padding == (3, 3)
            and conv.dilation == (1, 1) and conv.groups == 1):
        return False
    weight, dtype = conv.weight, torch.get_autocast_dtype("cuda")
    return (dtype in _TYPES and type(x) is torch.Tensor and x.dim() == 4 and x.is_cuda and x.dtype in (torch.float32, dtype) and not x.requires_grad
            and not x.is_inference() and x.shape[1] == 3 and 0 < x.shape[0] * (x.shape[2] + 8) < 1 << 30 and 0 < x.shape[2]
            and 0 < x.shape[3] <= 700 and x.get_device() == torch.cuda.current_device()
            and _weight_ok(weight, x.get_device()) and weight.shape[1:] == (3, 7, 7) and weight.shape[0] % 8 == 0 and 0 < weight.shape[0] <= 4096)


def stem_conv(conv: nn.Module, x: torch.Tensor) -> torch.Tensor:
    """``conv(x)``."""
    if stem_applies(conv, x):
        return _lib.torch_ops().stem_conv.default(x, conv.weight, torch.get_autocast_dtype("cuda"))
    return conv(x)
