"""Element-wise and halo kernels exposed as functions on PyTorch tensors."""
from .activations import batch_norm_act, max_pool
from .elementwise import fill_u32, scale_cast, sgd_momentum_step
from .halo import HaloExchange, halo_pack, halo_unpack

__all__ = ["batch_norm_act", "max_pool", "scale_cast", "sgd_momentum_step", "fill_u32", "HaloExchange", "halo_pack", "halo_unpack"]
