"""``store_kvcache`` of the reference (layers/attention.py:33-40) on the CUDA
library: the K / V rows of the prompt tokens of a prefill go to their slots of
the shared paged cache.  Same signature and the same checks; the work is done
by ``dfb_store_kvcache`` (no Triton, no CPU fallback)."""

from __future__ import annotations

import struct

# Looked up at the first call (the package imports without torch and without the built library) and kept: one call of
# store_kvcache on a short prompt takes a few microseconds, of which the imports and attribute chains of a call were two.
_torch = _store = _prefill = _check = _stream = _bf16 = _i32 = _device = _empty = None
# the arguments of the two native calls as one block of 64-bit words (a bytes object of its own per call): ctypes takes
# 1.5 us to convert twelve arguments one by one, 0.5 for the block
_store_words, _prefill_words = struct.Struct("12q").pack, struct.Struct("15qd8q").pack


def _load():
    global _torch, _store, _prefill, _check, _stream, _bf16, _i32, _device, _empty
    import torch

    from . import native

    lib = native.lib()
    _store, _prefill, _check = lib.dfb_store_kvcache_words, lib.dfb_prefill_attention_words, native.check
    _bf16, _i32, _empty = torch.bfloat16, torch.int32, torch.empty
    # the raw handle of the current stream; the public call builds a Stream object (1 us) around it, and the public call for the
    # device asks first whether CUDA is up, as it is once a tensor lies there (0.2 us against 0.1)
    _stream = getattr(torch._C, "_cuda_getCurrentRawStream", None) or (lambda device: torch.cuda.current_stream().cuda_stream)
    _device = getattr(torch._C, "_cuda_getDevice", None) or torch.cuda.current_device
    _torch = torch


def store_kvcache(key, value, k_cache, v_cache, slot_mapping, status=None) -> None:
    """``key`` / ``value``: ``[N, kv_heads, head_dim]`` bf16 CUDA tensors (any row
    stride); ``k_cache`` / ``v_cache``: one layer's ``[num_blocks, block_size,
    kv_heads, head_dim]`` views, bf16 and dense; ``slot_mapping``: int32 ``[N]``, -1 = skip.
    ``status``: optional int32 CUDA tensor ``[4]`` that receives a bad slot."""
    if _torch is None:
        _load()
    rows = key.shape
    n, num_heads, head_dim = rows
    d = num_heads * head_dim
    k_stride, k_head, k_one = key.stride()
    v_stride, v_head, v_one = value.stride()
    assert k_one == 1 and v_one == 1
    assert k_head == head_dim and v_head == head_dim
    v_rows = value.shape
    assert v_rows == rows or (v_rows[0] >= n and v_rows[1] * v_rows[2] >= d)
    # slot s is row s of both caches: their blocks lie one behind the other, and V has as many as K
    shape = k_cache.shape
    slots = shape[0] * shape[1]
    if not (k_cache.is_contiguous() and v_cache.is_contiguous() and k_cache.numel() == slots * d and v_cache.shape == shape):
        v_shape, k_strides, v_strides = v_cache.shape, k_cache.stride(), v_cache.stride()
        assert k_strides[1] == d and v_strides[1] == d and v_shape[0] * v_shape[1] >= slots
        assert k_strides[0] == shape[1] * d or shape[0] == 1
        assert v_strides[0] == v_shape[1] * d or v_shape[0] == 1
    assert slot_mapping.numel() == n
    if not (key.dtype is value.dtype is k_cache.dtype is v_cache.dtype is _bf16):
        raise TypeError("store_kvcache moves bf16 rows")
    if slot_mapping.dtype != _i32 or not slot_mapping.is_cuda:
        raise TypeError("slot_mapping must be an int32 CUDA tensor")
    if n == 0:
        return
    code = _store(_store_words(key.data_ptr(), value.data_ptr(), k_stride, v_stride, k_cache.data_ptr(), v_cache.data_ptr(),
                               slot_mapping.data_ptr(), n, d, slots,
                               status.data_ptr() if status is not None else 0, _stream(_device())))
    if code:
        _check(code, "dfb_store_kvcache")


def prefill_attention(q, k, v, cu_seqlens_q, max_seqlen_q: int, softmax_scale: float, cu_seqlens_k=None,
                      block_table=None, status=None):
    """The reference's ``flash_attn_varlen_func(q, k, v, cu_seqlens_q=…, cu_seqlens_k=…, max_seqlen_q=…,
    softmax_scale=s, causal=True, block_table=…)`` of ``layers/attention.py:64-70``.  ``q`` ``[N, q_heads, 128]``
    bf16 (any row stride), ``cu_seqlens_*`` int32 CUDA ``[batch + 1]``.  Without ``block_table``: ``k`` / ``v``
    ``[N, kv_heads, 128]``, the projections of the same tokens.  With it (prefix cache): ``k`` / ``v`` are one
    layer's cache ``[num_blocks, block_size, kv_heads, 128]`` and ``block_table`` the int32 CUDA
    ``[batch, columns]`` table.  Returns ``[N, q_heads, 128]`` bf16."""
    if _torch is None:
        _load()
    n, q_heads, head_dim = q.shape
    q_stride, q_head, q_one = q.stride()
    k_strides, v_strides = k.stride(), v.stride()
    assert q_one == 1 and k_strides[-1] == 1 and v_strides[-1] == 1 and q_head == head_dim
    if q.dtype != _bf16 or k.dtype != _bf16 or v.dtype != _bf16:
        raise TypeError("prefill_attention takes bf16 tensors")
    if cu_seqlens_q.dtype != _i32 or not cu_seqlens_q.is_cuda:
        raise TypeError("cu_seqlens_q must be an int32 CUDA tensor")
    batch = cu_seqlens_q.numel() - 1
    if cu_seqlens_k is not None:
        if cu_seqlens_k.dtype != _i32 or not cu_seqlens_k.is_cuda:
            raise TypeError("cu_seqlens_k must be an int32 CUDA tensor")
        assert cu_seqlens_k.numel() > batch
    # K and V are read at the same places: V has what K has
    if block_table is not None:
        num_blocks, block_size, kv_heads = k.shape[:3]
        v_blocks, v_block_size, v_heads = v.shape[:3]
        k_rows, v_rows = num_blocks * block_size, v_blocks * v_block_size
        k_stride, v_stride, kv_rows = k_strides[1], v_strides[1], 0
        assert k_strides[2] == head_dim and v_strides[2] == head_dim and k_strides[0] == block_size * k_stride
        assert v_blocks >= num_blocks and v_block_size == block_size and (v_strides[0] == block_size * v_stride or v_blocks == 1)
        if block_table.dtype != _i32 or not block_table.is_cuda or block_table.stride(-1) != 1 or cu_seqlens_k is None:
            raise TypeError("the prefix-cache case needs an int32 CUDA block table and cu_seqlens_k")
        assert block_table.shape[0] >= batch
        bt_ptr, bt_stride = block_table.data_ptr(), block_table.stride(0)
    else:
        k_rows, kv_heads = k.shape[:2]
        v_rows, v_heads = v.shape[:2]
        kv_rows = min(k_rows, v_rows)
        assert k_strides[1] == head_dim and v_strides[1] == head_dim
        num_blocks = block_size = 0
        k_stride, v_stride = k_strides[0], v_strides[0]
        bt_ptr, bt_stride = 0, 0
    assert v_heads >= kv_heads and k.numel() == k_rows * kv_heads * head_dim and v.numel() == v_rows * v_heads * head_dim
    out = _empty((n, q_heads, head_dim), dtype=_bf16, device=q.device)
    if n == 0:
        return out
    code = _prefill(_prefill_words(
        q.data_ptr(), k.data_ptr(), v.data_ptr(), out.data_ptr(), cu_seqlens_q.data_ptr(),
        cu_seqlens_k.data_ptr() if cu_seqlens_k is not None else 0, batch, int(max_seqlen_q),
        q_stride, k_stride, v_stride, q_heads * head_dim, q_heads, kv_heads, head_dim, float(softmax_scale), bt_ptr,
        bt_stride, block_size, num_blocks, status.data_ptr() if status is not None else 0, n, kv_rows, _stream(_device())))
    if code:
        _check(code, "dfb_prefill_attention")
    return out
