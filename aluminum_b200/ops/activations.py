"""Training batch norm of channels-last activations with the residual addition and the ReLU behind it fused in
(``kernels/batchnorm.cu``), and max pooling (``kernels/maxpool.cu``); autograd in ``src/torch/activations_autograd.cpp``.

The functions take the modules that a network holds (``nn.BatchNorm2d``, ``nn.ReLU``, ``nn.MaxPool2d``) and run the kernels
where they do exactly what the modules would: 16-bit channels-last CUDA activations in training, plain modules without
hooks, ordinary reverse-mode autograd.  Everything else - evaluation, other types and layouts, hooks, tracing,
functorch transforms, forward-mode AD - calls the modules.
"""
from __future__ import annotations

import torch
from torch import nn
from torch.autograd import forward_ad

from .. import _lib

_PLAIN = (torch.Tensor, nn.Parameter)
_TYPES = (torch.bfloat16, torch.float16)


def _bare(m: nn.Module) -> bool:
    """Neither a hook nor a forward of the instance's own would be missed by not calling the module."""
    return not ("forward" in m.__dict__ or m._forward_hooks or m._forward_pre_hooks or m._backward_hooks or m._backward_pre_hooks)


def _activation_ok(x) -> bool:
    return (type(x) is torch.Tensor and not x.is_inference() and x.dim() == 4 and x.dtype in _TYPES and x.is_cuda
            and x.is_contiguous(memory_format=torch.channels_last) and x.shape[1] % 8 == 0 and x.data_ptr() % 16 == 0
            and x.numel() >= 2 * x.shape[1] > 0)


def _parameter_ok(t, channels: int, device: int) -> bool:
    """A plain tensor with one fp32 value per channel (of another length the module raises; a subclass may have no memory of its own)."""
    return (type(t) in _PLAIN and t.dtype == torch.float32 and t.numel() == channels and t.get_device() == device and t.is_contiguous()
            and not t.is_inference() and t.data_ptr() % 16 == 0)


def _count_ok(t, device: int) -> bool:
    return t is None or (type(t) in _PLAIN and t.dtype == torch.int64 and t.numel() == 1 and t.get_device() == device and not t.is_inference())


def _modes_off() -> bool:
    g = nn.modules.module
    return not (torch.compiler.is_compiling() or torch.jit.is_tracing() or torch.is_inference_mode_enabled() or forward_ad._current_level >= 0
                or torch._C._functorch.peek_interpreter_stack() is not None or torch._C._len_torch_dispatch_stack()
                or torch._C._len_torch_function_stack()
                or g._global_forward_hooks or g._global_forward_pre_hooks or g._global_backward_hooks or g._global_backward_pre_hooks)


def _tensors(bn: nn.Module, x):
    """Weight, bias, running statistics and count of a batch norm that the kernels may run on x, else None."""
    # (_modes_off() first: a compiler that traces this function sees a constant there and nothing of what follows)
    if not (_modes_off() and type(bn) is nn.BatchNorm2d and bn.training and bn.track_running_stats and bn.momentum is not None
            and _activation_ok(x) and _bare(bn)):
        return None
    c, device = bn.num_features, x.get_device()
    found = weight, bias, mean, var, count = bn.weight, bn.bias, bn.running_mean, bn.running_var, bn.num_batches_tracked
    if (x.shape[1] == c and device == torch.cuda.current_device() and _parameter_ok(weight, c, device) and _parameter_ok(bias, c, device)
            and _parameter_ok(mean, c, device) and _parameter_ok(var, c, device) and _count_ok(count, device)):
        return found
    return None


def _fused(bn: nn.Module, x, relu, residual):
    """The arguments of the fused operators, or None where the modules are called."""
    found = _tensors(bn, x)
    if (found is not None and (relu is None or (type(relu) is nn.ReLU and _bare(relu)))
            and (residual is None or (_activation_ok(residual) and residual.shape == x.shape and residual.dtype == x.dtype
                                      and residual.get_device() == x.get_device()))):
        weight, bias, mean, var, count = found
        return x, weight, bias, residual, mean, var, count, bn.momentum, bn.eps, relu is not None
    return None


def batch_norm_act(bn: nn.Module, x: torch.Tensor, relu: nn.Module | None = None, residual: torch.Tensor | None = None) -> torch.Tensor:
    """``relu(bn(x) + residual)``; without ``relu`` or ``residual`` the same without that part."""
    args = _fused(bn, x, relu, residual)
    if args is not None:
        return _lib.torch_ops().batch_norm_act.default(*args)
    y = bn(x)
    if residual is not None:
        y = y + residual
    return y if relu is None else relu(y)


def batch_norm_act_twice(bn: nn.Module, x: torch.Tensor, relu: nn.Module | None = None, residual: torch.Tensor | None = None):
    """:func:`batch_norm_act` for a result that is used in two places, as two tensors (on the same memory where the kernels run): the
    backward then adds their two gradients where it reads them."""
    args = _fused(bn, x, relu, residual)
    if args is not None:
        return _lib.torch_ops().batch_norm_act_twice.default(*args)
    y = batch_norm_act(bn, x, relu, residual)
    return y, y


def _one(v) -> int:
    """The value of an int or of a pair of equal ints, else 0."""
    if isinstance(v, (tuple, list)):
        return v[0] if len(v) == 2 and v[0] == v[1] and type(v[0]) is int else 0
    return v if type(v) is int else 0


def max_pool(pool: nn.Module, x: torch.Tensor) -> torch.Tensor:
    """``pool(x)``."""
    if _modes_off() and type(pool) is nn.MaxPool2d and _activation_ok(x) and x.get_device() == torch.cuda.current_device() and _bare(pool):
        k, stride, pad = _one(pool.kernel_size), _one(pool.stride), pool.padding if pool.padding == 0 else _one(pool.padding)
        if (0 < k <= 15 and stride > 0 and _one(pool.dilation) == 1 and not pool.ceil_mode and not pool.return_indices
                and (pad > 0 or pool.padding == 0) and 2 * pad <= k and min(x.shape[2:]) + 2 * pad >= k
                and x.numel() * (1 + pad) ** 2 < 1 << 34):   # (the kernels count threads of 8 elements in 32 bits)
            return _lib.torch_ops().max_pool.default(x, k, stride, pad)
    return pool(x)
