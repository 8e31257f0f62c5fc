"""Element-wise and halo kernels exposed as functions on PyTorch tensors."""
from .activations import batch_norm_act, batch_norm_act_twice, max_pool
from .convolution import stem_conv
from .elementwise import fill_u32, scale_cast, sgd_momentum_step
from .halo import HaloExchange, halo_pack, halo_unpack

__all__ = ["batch_norm_act", "batch_norm_act_twice", "max_pool", "stem_conv", "scale_cast", "sgd_momentum_step", "fill_u32", "HaloExchange", "halo_pack", "halo_unpack"]
