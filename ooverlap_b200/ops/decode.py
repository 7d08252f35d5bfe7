"""Decode-path kernels of the model runner: RoPE fused with the KV-cache write, SwiGLU, grouped-query decode
attention over a static cache.

Capability parity: the reference leaves the model's own ops to vLLM
(patches/vllm/v0.25.0/vllm/model_executor/models/qwen2.py); this library's serving path needs them so that one
decode step is a fixed sequence of kernels (seven per transformer layer, five on one GPU) that a CUDA graph replays.
"""
from __future__ import annotations

import ctypes
import math
from typing import Optional

import torch

from .. import _lib
from . import solutions
from .gemm import RowSums, _check_operands, _plain_args, _scaled_rows, _scope, _set_row_sums, gemm, gemm_plan_splits
from ..utils.dtypes import dtype_code
from ..utils.stream import current_stream_ptr as _stream


def rope_tables(max_len: int, head_dim: int, theta: float, device) -> tuple[torch.Tensor, torch.Tensor]:
    """fp32 ``cos`` / ``sin`` tables of shape [max_len, head_dim / 2] for rotation pairs (2i, 2i + 1)."""
    inv = 1.0 / (theta ** (torch.arange(0, head_dim, 2, device=device, dtype=torch.float32) / head_dim))
    ang = torch.arange(max_len, device=device, dtype=torch.float32).unsqueeze(-1) * inv
    return ang.cos().contiguous(), ang.sin().contiguous()


def _rope_args(dtype, B: int, T: int, heads: int, kv_heads: int, hd: int, k_cache: torch.Tensor, v_cache: torch.Tensor,
               cos: torch.Tensor, sin: torch.Tensor, pos, batch0: int, q_out: torch.Tensor) -> "_lib.RopeArgs":
    if k_cache.shape[-1] != hd or k_cache.shape != v_cache.shape:
        raise ValueError("head geometry does not match the cache")
    if k_cache.dim() != 4 or k_cache.shape[1] != kv_heads or k_cache.stride(3) != 1 or k_cache.stride(2) != hd \
            or k_cache.stride(1) != k_cache.shape[2] * hd or v_cache.stride() != k_cache.stride():
        raise ValueError("cache must be [batch, kv_heads, max_len, hd] with contiguous (kv_heads, max_len, hd)")
    if batch0 + B > k_cache.shape[0]:
        raise ValueError("sequences outside the cache")
    max_len = k_cache.shape[2]
    if cos.dtype != torch.float32 or cos.shape != (max_len, hd // 2) or not cos.is_contiguous() or sin.shape != cos.shape:
        raise ValueError("cos / sin must be contiguous fp32 [max_len, hd/2] tables")
    if isinstance(pos, torch.Tensor):
        if pos.dtype != torch.int64 or pos.numel() != 1 or not pos.is_cuda:
            raise ValueError("pos must be a one-element int64 CUDA tensor")
        pos_dev, pos0 = pos.data_ptr(), 0
    else:
        pos_dev, pos0 = 0, int(pos)
    # Fields in the order of the structure, qkv left null.
    return _lib.RopeArgs.from_buffer_copy(_lib.ROPE_ARGS.pack(
        dtype_code(dtype), B, T, heads, kv_heads, hd, 0, q_out.data_ptr(), k_cache.data_ptr(), v_cache.data_ptr(), k_cache.stride(0), max_len,
        batch0, cos.data_ptr(), sin.data_ptr(), pos_dev, pos0))


def rope_kv_write(qkv: torch.Tensor, B: int, T: int, heads: int, kv_heads: int, k_cache: torch.Tensor,
                  v_cache: torch.Tensor, cos: torch.Tensor, sin: torch.Tensor, pos, *, batch0: int = 0,
                  q_out: Optional[torch.Tensor] = None) -> torch.Tensor:
    """Rotates the query and key heads of ``qkv`` ([B*T, (heads + 2*kv_heads) * hd]) and writes keys and values
    into one layer's cache ([batch, kv_heads, max_len, hd]) at positions ``pos .. pos + T - 1`` of sequences
    ``batch0 .. batch0 + B - 1``.  ``pos`` is an int, or a device ``int64`` tensor with one element (read by the
    kernel, so a captured launch follows it).  Returns the rotated queries, [B*T, heads * hd]."""
    if qkv.dim() != 2 or not qkv.is_contiguous() or qkv.shape[0] != B * T:
        raise ValueError("qkv must be a contiguous [B*T, (heads + 2*kv_heads) * hd] tensor")
    hd = qkv.shape[1] // (heads + 2 * kv_heads)
    if hd * (heads + 2 * kv_heads) != qkv.shape[1]:
        raise ValueError("head geometry does not match qkv")
    if q_out is None:
        q_out = torch.empty((B * T, heads * hd), dtype=qkv.dtype, device=qkv.device)
    a = _rope_args(qkv.dtype, B, T, heads, kv_heads, hd, k_cache, v_cache, cos, sin, pos, batch0, q_out)
    a.qkv = qkv.data_ptr()
    _lib.check(_lib.lib().oob_rope_kv_write(ctypes.byref(a), _stream()))
    return q_out


def gemm_rope_kv_write(x: torch.Tensor, wqkv: torch.Tensor, B: int, T: int, heads: int, kv_heads: int,
                       k_cache: torch.Tensor, v_cache: torch.Tensor, cos: torch.Tensor, sin: torch.Tensor, pos, *,
                       batch0: int = 0, q_out: Optional[torch.Tensor] = None, fused: Optional[bool] = None) -> torch.Tensor:
    """``rope_kv_write(x @ wqkv.T, ...)``: the QKV projection followed by the rotation and the cache write.

    When the GEMM is one that the tiled kernels would split over K (every decode-step shape), rotation and cache write are
    done from the fp32 sums by the kernel that has them (the weight-streaming kernel, or the one that sums the splits);
    otherwise (or with ``fused=False``) the GEMM is followed by :func:`rope_kv_write`.  ``x`` may be a ``RowSums`` (see
    ``gemm_add_norm``).  Returns the rotated queries, [B*T, heads * hd]."""
    if q_out is None and fused is None and solutions.no_gemm_table():
        done = _lib.fast().gemm_rope_kv_write(x, wqkv, B, T, heads, kv_heads, k_cache, v_cache, cos, sin, pos, batch0, _scope.static_b)
        if done is not None:
            return done
    sums = x
    if isinstance(x, RowSums):
        if fused is False:
            raise ValueError("row sums need the kernel that this call rules out")
        x = _scaled_rows(x)
    _check_operands(x, wqkv)
    M, N, K = x.shape[0], wqkv.shape[0], x.shape[1]
    if M != B * T:
        raise ValueError("x must have B*T rows")
    hd = N // (heads + 2 * kv_heads)
    if hd * (heads + 2 * kv_heads) != N or hd % 8 != 0:
        raise ValueError("head geometry does not match the QKV weight")
    can_fuse = sums is not x or gemm_plan_splits(M, N, K) > 1
    if fused is None:
        fused = can_fuse
    if fused and not can_fuse:
        raise ValueError("this problem is not split over K, so the epilogue has no kernel to run in")
    if not fused:
        return rope_kv_write(gemm(x, wqkv), B, T, heads, kv_heads, k_cache, v_cache, cos, sin, pos, batch0=batch0,
                             q_out=q_out)
    if q_out is None:
        q_out = torch.empty((M, heads * hd), dtype=x.dtype, device=x.device)
    r = _rope_args(x.dtype, B, T, heads, kv_heads, hd, k_cache, v_cache, cos, sin, pos, batch0, q_out)
    args = _plain_args(x, wqkv, q_out)
    args.ldc = N  # C itself is not written; a valid aligned pointer keeps the checks uniform
    _set_row_sums(args, sums)
    args.epilogue = _lib.EPILOGUE_ROPE_KV
    args.epilogue_args = ctypes.addressof(r)
    _lib.check(_lib.lib().oob_gemm(None, args, _stream()))
    return q_out


def silu_mul(gu: torch.Tensor, out: Optional[torch.Tensor] = None) -> torch.Tensor:
    """``silu(gu[:, :F]) * gu[:, F:]`` for a [rows, 2F] tensor with unit column stride."""
    if gu.dim() != 2 or gu.stride(1) != 1 or gu.shape[1] % 16 != 0:
        raise ValueError("gu must be [rows, 2F] with F a multiple of 8 and unit column stride")
    rows, F = gu.shape[0], gu.shape[1] // 2
    if out is None:
        out = torch.empty((rows, F), dtype=gu.dtype, device=gu.device)
    elif out.shape != (rows, F) or not out.is_contiguous() or out.dtype != gu.dtype:
        raise ValueError("bad output tensor")
    _lib.check(_lib.lib().oob_silu_mul(dtype_code(gu.dtype), ctypes.c_void_p(gu.data_ptr()), gu.stride(0),
                                       ctypes.c_void_p(out.data_ptr()), rows, F, _stream()))
    return out


def attn_decode(q: torch.Tensor, k_cache: torch.Tensor, v_cache: torch.Tensor, pos, *, batch0: int = 0,
                scale: Optional[float] = None, out: Optional[torch.Tensor] = None, splits: int = 0,
                len_bound: int = 0, cache_ready: bool = False) -> torch.Tensor:
    """One decode step of grouped-query attention: ``q`` is [B, heads, 128], the cache is
    [batch, kv_heads, max_len, 128] and keys ``0 .. pos`` of sequences ``batch0 .. batch0 + B - 1`` are attended
    (``pos``: int or one-element device ``int64`` tensor, the index of the newest key).  Returns [B, heads * 128].

    The CTAs of a cluster share the keys of one (sequence, KV head) by the length found on the device; ``splits`` > 1 adds
    that many clusters, whose results a second kernel merges.  0 picks both from ``B * kv_heads`` and ``len_bound`` (an
    upper bound of the context length of this and any replayed launch; default ``max_len``).

    ``cache_ready`` promises that neither the call before this one on the stream nor, in a chain of this library's kernels, one of
    those before it writes a position on the device or a key or value other than the newest of each sequence: they are then
    loaded while the kernel before still runs.  Not so behind a call that appends several tokens."""
    if scale is None and out is None:
        done = _lib.fast().attn_decode(q, k_cache, v_cache, pos, batch0, splits, len_bound, cache_ready)
        if done is not None:
            return done
    if q.dim() != 3 or q.shape[2] != 128 or not q.is_contiguous():
        raise ValueError("q must be a contiguous [B, heads, 128] tensor")
    B, H, hd = q.shape
    if k_cache.dim() != 4 or k_cache.shape[3] != hd or k_cache.shape != v_cache.shape or k_cache.dtype != q.dtype:
        raise ValueError("cache must be [batch, kv_heads, max_len, 128] of the query's dtype")
    KV, max_len = k_cache.shape[1], k_cache.shape[2]
    if k_cache.stride(3) != 1 or k_cache.stride(2) != hd or k_cache.stride(1) != max_len * hd \
            or v_cache.stride() != k_cache.stride():
        raise ValueError("cache must have contiguous (kv_heads, max_len, hd)")
    if H % KV or H // KV > 16 or batch0 + B > k_cache.shape[0]:
        raise ValueError("bad head counts or sequences outside the cache")
    if out is None:
        out = torch.empty((B, H * hd), dtype=q.dtype, device=q.device)
    lib = _lib.lib()
    bound = len_bound or max_len
    if splits == 0:
        splits = lib.oob_attn_decode_auto_splits(B, KV, bound)
    if isinstance(pos, torch.Tensor):
        if pos.dtype != torch.int64 or pos.numel() != 1 or not pos.is_cuda:
            raise ValueError("pos must be a one-element int64 CUDA tensor")
        pos_dev, length = pos.data_ptr(), 0
    else:
        pos_dev, length = 0, int(pos) + 1
    ws = None
    if splits > 1:
        # Of this call alone, in stream order (and in the graph's pool under capture): a workspace shared by calls would be
        # written by two streams at once, and one that a later call outgrows would be freed under a captured graph.
        ws = torch.empty(lib.oob_attn_decode_workspace_bytes(B, H, splits), dtype=torch.uint8, device=q.device)
    # Fields in the order of the structure.
    a = _lib.AttnDecodeArgs.from_buffer_copy(_lib.ATTN_ARGS.pack(
        dtype_code(q.dtype), B, H, KV, q.data_ptr(), k_cache.data_ptr(), v_cache.data_ptr(), k_cache.stride(0), max_len, batch0,
        out.data_ptr(), pos_dev, length, scale if scale is not None else 1.0 / math.sqrt(hd), splits, bound,
        ws.data_ptr() if ws is not None else 0, cache_ready))
    _lib.check(lib.oob_attn_decode(ctypes.byref(a), _stream()))
    return out


def attn_decode_reference(q, k_cache, v_cache, pos: int, *, batch0: int = 0, scale: Optional[float] = None):
    """fp32 PyTorch oracle of :func:`attn_decode`."""
    B, H, hd = q.shape
    KV = k_cache.shape[1]
    G = H // KV
    scale = scale if scale is not None else 1.0 / math.sqrt(hd)
    k = k_cache[batch0:batch0 + B, :, :pos + 1].float().repeat_interleave(G, dim=1)  # [B, H, L, hd]
    v = v_cache[batch0:batch0 + B, :, :pos + 1].float().repeat_interleave(G, dim=1)
    s = torch.einsum("bhd,bhld->bhl", q.float(), k) * scale
    p = torch.softmax(s, dim=-1)
    return torch.einsum("bhl,bhld->bhd", p, v).reshape(B, H * hd)
