"""The FlashAttention forward / grad primitives, backed by ``libacct_b200.so``.

Mirrors the reference's op registration module
(train/acctransformer/flash_attention/ops/flash_attention/flash_attention_impl.py:96-154):

* ``get_flash_attention(prev_block_num, next_block_num, tiling_stgy_name)`` returns the forward
  primitive ``fa(query, key, value, attn_mask=None, dropout_mask=None, alibi_mask=None)
  -> (output, rowsum)``; ``output`` has q's dtype and shape, ``rowsum`` is the fp32
  log-sum-exp ``[B, N, S_q]`` (:132-140).  No scaling happens inside the primitive.
* ``get_flash_attention_grad(...)`` returns the grad primitive
  ``fa_grad(query, key, value, output, do, rowsum, attn_mask, dropout_mask, alibi_mask)
  -> (dq, dk, dv)`` in fp32 (:99-105).
* The forward primitive is differentiable: its backward calls the grad primitive and casts
  dq/dk/dv to the input dtype, like the reference's ``bprop`` (:117-124).

The tensors are torch CUDA tensors in ``[B, N, S, D]`` layout.  An ``attn_mask`` whose shape is
``(128, 128)`` or ``(1, 128, 128)`` is the causal-tile form and is applied to diagonal 128x128
tiles only (ops/flash_attention/attention.py:279-285); any other mask is ``[1 or B, S_q, S_k]``.
``dropout_mask`` is either the reference's 16-bit ``{0, 1/keep_prob}`` tensor or a uint8 ``{0,1}``
tensor together with ``keep_prob``.  ``tiling_stgy_name`` is accepted for compatibility; tile
sizes are fixed inside the CUDA kernels.
"""
from __future__ import annotations

import torch

from .... import ops as _ops
from ...._lib import host as _host

__all__ = ["get_flash_attention", "get_flash_attention_grad"]


def _mask_tiles(attn_mask):
    """Per-tile summary of a full attn_mask (made once per mask tensor, see ops.mask_tile_classes), with which the
    kernels read only the 128x128 tiles of the mask that are neither all 0 nor all 1; None for no mask / the tile form."""
    if attn_mask is None or _is_tile_mask(attn_mask) or not attn_mask.is_cuda:
        return None
    return _ops.mask_tile_classes(attn_mask)


_TILE_SHAPES = ((128, 128), (1, 128, 128))


def _is_tile_mask(attn_mask):
    if attn_mask is None:
        return False
    return attn_mask.shape in _TILE_SHAPES


def get_flash_attention_grad(prev_block_num=65536, next_block_num=65536, tiling_stgy_name='sparse',
                             scale=1.0, causal=False, deterministic=False):
    """Returns the grad primitive (fp32 dq, dk, dv).  ``deterministic`` makes dq bit-reproducible from run to
    run (the reference's tests require that of its gradients, tests/train/flash_attention/st/test_sharding.py:91-115)
    at some cost in speed; dk and dv always are."""

    def fa_grad(query, key, value, output, do, rowsum, attn_mask=None, dropout_mask=None, alibi_mask=None,
                keep_prob=1.0, grads_fp32=True, dropout_seed=None, dropout_offset=0):
        return _ops.fa_backward(query, key, value, output, rowsum, do, attn_mask,
                                mask_tile128=_is_tile_mask(attn_mask), causal=causal,
                                dropout_mask=dropout_mask, keep_prob=keep_prob, alibi=alibi_mask,
                                prev_block_num=prev_block_num, next_block_num=next_block_num, scale=scale,
                                grads_fp32=grads_fp32, deterministic=deterministic,
                                dropout_seed=dropout_seed, dropout_offset=dropout_offset,
                                mask_tiles=_mask_tiles(attn_mask))

    fa_grad.prev_block_num = prev_block_num
    fa_grad.next_block_num = next_block_num
    fa_grad.tiling_stgy_name = tiling_stgy_name
    return fa_grad


class _Traced(torch.autograd.Function):
    """The operator as torch.jit.trace can record it: a Python function that runs again on the new inputs.  (The tracer
    does not see the native path and would put its result into the graph as a constant.)"""

    @staticmethod
    def forward(ctx, query, key, value, attn_mask, dropout_mask, alibi_mask, options):
        output, rowsum = _native(query, key, value, attn_mask, dropout_mask, alibi_mask, **options)
        ctx.options = options
        ctx.save_for_backward(query, key, value, output, rowsum, attn_mask, dropout_mask, alibi_mask)
        ctx.mark_non_differentiable(rowsum)
        return output, rowsum

    @staticmethod
    def backward(ctx, d_output, _d_rowsum):
        query, key, value, output, rowsum, attn_mask, dropout_mask, alibi_mask = ctx.saved_tensors
        grads = _ops.fa_backward(query, key, value, output, rowsum, d_output.contiguous(), attn_mask,
                                 mask_tile128=_is_tile_mask(attn_mask), dropout_mask=dropout_mask, alibi=alibi_mask,
                                 mask_tiles=_mask_tiles(attn_mask), **ctx.options)
        return (*grads, None, None, None, None)


def _apply(query, key, value, attn_mask, dropout_mask, alibi_mask, causal, keep_prob, prev_block_num, next_block_num,
           scale, tri_block=0, deterministic=False, dropout_seed=None, dropout_offset=0):
    """The differentiable operator: (output, rowsum), by the native host path (its custom function calls the grad
    kernels and hands back dq, dk, dv in the input type)."""
    if torch.jit.is_tracing():
        return _Traced.apply(query, key, value, attn_mask, dropout_mask, alibi_mask,
                             dict(causal=causal, keep_prob=keep_prob, prev_block_num=prev_block_num,
                                  next_block_num=next_block_num, scale=scale, tri_block=tri_block,
                                  deterministic=deterministic, dropout_seed=dropout_seed, dropout_offset=dropout_offset))
    return _native(query, key, value, attn_mask, dropout_mask, alibi_mask, causal, keep_prob, prev_block_num,
                   next_block_num, scale, tri_block, deterministic, dropout_seed, dropout_offset)


def _native(query, key, value, attn_mask, dropout_mask, alibi_mask, causal, keep_prob, prev_block_num, next_block_num,
            scale, tri_block, deterministic, dropout_seed, dropout_offset):
    tiles, tile_form = None, False
    if attn_mask is not None:
        tile_form = _is_tile_mask(attn_mask)
        tiles = _mask_tiles(attn_mask)
    return _host().fa_apply(query, key, value, attn_mask, dropout_mask, alibi_mask, tiles, tile_form, causal, keep_prob,
                            prev_block_num, next_block_num, scale, tri_block, deterministic, dropout_seed, dropout_offset)


def get_flash_attention(prev_block_num=65536, next_block_num=65536, tiling_stgy_name='sparse',
                        scale=1.0, causal=False, deterministic=False):
    """Returns the forward primitive.  ``scale`` (default 1: the raw primitive) and ``causal``
    (an in-kernel triangle that needs no mask tensor) are this library's additions."""

    def fa_forward(query, key, value, attn_mask=None, dropout_mask=None, alibi_mask=None, keep_prob=1.0,
                   dropout_seed=None, dropout_offset=0, implicit_causal=False):
        # dropout_seed / dropout_offset: dropout decided inside the kernels (no mask tensor); the backward that
        # autograd runs later reuses the same two values
        # implicit_causal: the caller has established that attn_mask is exactly the causal mask; the kernels then
        # generate the triangle and the tensor is not read
        if implicit_causal:
            attn_mask = None
        return _apply(query, key, value, attn_mask, dropout_mask, alibi_mask, causal or implicit_causal, keep_prob,
                      prev_block_num, next_block_num, scale, 0, deterministic, dropout_seed, dropout_offset)

    fa_forward.prev_block_num = prev_block_num
    fa_forward.next_block_num = next_block_num
    fa_forward.tiling_stgy_name = tiling_stgy_name
    fa_forward.prim_attrs = {}

    def add_prim_attr(name, value):
        fa_forward.prim_attrs[name] = value

    fa_forward.add_prim_attr = add_prim_attr
    fa_forward.shard = lambda strategy: fa_forward.prim_attrs.__setitem__("in_strategy", strategy)
    return fa_forward
