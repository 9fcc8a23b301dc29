"""Latent attention caches one row [latent | rotated key part] per position, shared by all heads.  A step attends over it in one of two
forms, whose choice is here for every model that has such layers:

  * ABSORBED: W_uk^T q against the cached rows themselves (one key head that is also the value), then W_uv per head;
  * EXPANDED: one tensor-core product turns the rows of the sequence into keys | values per head, then ordinary multi-head attention.
"""
from .. import abi

EXPAND_MIN_TOKENS = 128    # steps from this size on expand a latent layer's keys and values per head (bfloat16 sessions)


def expands(T: int, rank: int, rot_dim: int, dim: int, vdim: int, wdt: int, force_float32: bool = False) -> bool:
    """Whether a step of T tokens runs expanded.  Expanding costs 2 R (rank + rot_dim) H (dim + rot_dim + vdim) FLOPs on the tensor cores per step over
    R cached rows; the absorbed form costs (2 rank - dim - vdim) more multiply-adds per (query, key, head) in f32.  Worth it for long steps of
    bfloat16 sessions whose rows fit the tensor-core product (a multiple of 8 values, at least 64); short steps stay absorbed.

    float32 sessions stay absorbed unless asked (`force_float32`): one form for every step length, and no keys | values of the whole ring in
    memory.  Their products run on the tensor cores too, so what is better depends on the layer.  Two layers, a step after 0 / 4096 positions: 16 heads of
    128 over latents of 512, which only the SIMT attention takes absorbed: 128 tokens 755 / 3726 us absorbed and 1110 / 1189 expanded, 1024 tokens
    2523 / 15443 and 1500 / 1779; 8 heads of 64 over latents of 256: 128 tokens 331 / 398 and 382 / 398, 1024 tokens 584 / 1044 and 595 / 683."""
    row = rank + rot_dim
    return (wdt == abi.W_BF16 or force_float32) and T >= EXPAND_MIN_TOKENS and row % 8 == 0 and row >= 64 and 2 * rank > dim + vdim
