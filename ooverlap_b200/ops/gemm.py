"""Plain tcgen05 GEMM: ``C[M, N] = A[M, K] @ B[N, K]^T`` (B in torch ``Linear.weight`` layout).

Capability parity: ``gemm_plain_sm90_dispatch`` / the cuBLAS column GEMM of the
reference's legacy binding (src/gemm/gemm_plain_sm90_dispatch.h:19-46,
src/pybind.cpp:266-324).  One hand-written sm_100a kernel replaces the 122
generated CUTLASS instances.
"""
from __future__ import annotations

import contextlib
import ctypes
import threading
from typing import NamedTuple, Optional

import torch

from .. import _lib
from . import solutions
from ..utils.dtypes import dtype_code
from ..utils.stream import current_stream_ptr


class _Scope(threading.local):
    static_b = 0  # GemmArgs.b_static


_scope = _Scope()


@contextlib.contextmanager
def static_weights(*, beyond_l2: bool = False):
    """GEMMs that this thread launches in this block take their ``b`` to be a weight: neither the kernel before the call on the
    stream nor, in a chain of this library's kernels, one of those before it writes ``b``.  The weight-streaming kernel then
    loads its first weights while the kernel before it still runs.  Elsewhere ``b`` may be any tensor, also the result of
    the call just before.  The promise is about weights alone: see ``attn_decode`` for its cache.

    ``beyond_l2``: the weights of the block, used again and again, are more together than L2 holds (from some 100 MB on).  Those of 8 MB and
    more then leave it first, which keeps activations and keys in it; without, only weights that are too large by themselves do."""
    before = _scope.static_b
    _scope.static_b = 2 if beyond_l2 else 1
    try:
        yield
    finally:
        _scope.static_b = before


def _check_operands(a: torch.Tensor, b: torch.Tensor) -> None:
    if a.dtype not in (torch.float16, torch.bfloat16) or a.dtype != b.dtype:
        raise TypeError("GEMM operands must both be fp16 or both bf16")
    if a.dim() != 2 or b.dim() != 2 or a.shape[1] != b.shape[1]:
        raise ValueError(f"shape mismatch: A {tuple(a.shape)} x B^T {tuple(b.shape)}")
    if a.stride(1) != 1 or b.stride(1) != 1:
        raise ValueError("A and B must be row-major (unit stride along K)")
    if not a.is_cuda or not b.is_cuda:
        raise ValueError("GEMM operands must be CUDA tensors")


def fill_gemm_args(args: _lib.GemmArgs, a: torch.Tensor, b: torch.Tensor) -> None:
    args.dtype = dtype_code(a.dtype)
    args.M, args.K = a.shape
    args.N = b.shape[0]
    args.A, args.lda = a.data_ptr(), a.stride(0)
    args.B, args.ldb = b.data_ptr(), b.stride(0)


_TAILS = (_lib.GEMM_TAIL, _lib.GEMM_TAIL_STATIC, _lib.GEMM_TAIL_CHAIN)


def _packed_plain_args(a: torch.Tensor, b: torch.Tensor, out: torch.Tensor) -> bytes:
    """The arguments of a call that asks for nothing, packed in one step: a third of the time of assigning them one by one (0.17 and
    0.75 us)."""
    return _lib.GEMM_HEAD.pack(_lib.GEMM_PLAIN, dtype_code(a.dtype), a.shape[0], b.shape[0], a.shape[1], a.data_ptr(), a.stride(0),
                               b.data_ptr(), b.stride(0), out.data_ptr(), out.stride(0)
                               ) + _TAILS[_scope.static_b]


def _plain_args(a: torch.Tensor, b: torch.Tensor, out: torch.Tensor) -> _lib.GemmArgs:
    return _lib.GemmArgs.from_buffer_copy(_packed_plain_args(a, b, out))


def gemm(a: torch.Tensor, b: torch.Tensor, out: Optional[torch.Tensor] = None, *, max_ctas: int = 0,
         splits: int = 0, pair: int = 0, skinny: int = 0, splitk_reduce: int = 0,
         gemv: int = 0, stream_k: int = 0, order: Optional[torch.Tensor] = None) -> torch.Tensor:
    """``out = a @ b.T`` with fp32 accumulation in TMEM.

    ``order`` (two-SM kernel): an int64 CUDA tensor ``[2 * tiles, 2]`` (``tiles`` = 256x256 tiles of the output) that
    the kernel fills with the tile-order record: per 128-row half of every tile the globaltimer nanoseconds at which
    it was stored and ``pair << 32 | index in the pair's sequence``; see :func:`tile_order`.  The record is of 256-column tiles:
    a call with one runs on these whatever width it would take without.

    ``splits`` > 1 splits K over that many CTAs per output tile (fp32 partials in the library's workspace,
    summed in split order), 1 turns it off; 0 leaves it to the kernel that the shape takes (few rows or few tiles: the
    weight-streaming kernel, else the two-SM kernel; the tiled kernels split by shape where both are ruled out).

    ``pair`` selects the two-SM kernel (tiles of 256 rows and 128 to 512 columns computed by CTA pairs with
    ``tcgen05.mma.cta_group::2``; each CTA stages half of the B block): 0 uses it for problems with more than 128 rows that
    the weight-streaming kernel is not expected to compute faster, 1 whenever the problem is unsplit, -1 never.

    ``stream_k`` (two-SM kernel): when the tile count is not a multiple of the pair count, the last wave and the
    remainder are cut along K into equal ranges, one per pair, so that no pair idles; pairs that compute part of a tile
    park fp32 accumulators in a library-owned workspace and the pair with the first part sums them in pair order
    (bit-reproducible).  0 uses it when the idle share would exceed 3 % of the run and neither whole tiles nor narrower
    ones are expected to be faster, 1 whenever there is a remainder, -1 never.

    ``skinny`` selects the weight-streaming kernel for few rows (the weight rows fill the tensor-core instruction's
    128-row dimension, the tokens are its other one; K is split over the CTAs of a cluster that sum their parts through
    distributed shared memory, deterministic): 0 uses it up to 128 rows (up to 48, or 8 where K is long, of a weight with
    over 296 tiles of 128), and above where it is expected to be faster than the two-SM kernel, 1 whenever it can
    (``splits`` then asks for that many CTAs per tile, at most 8), -1 never.

    ``splitk_reduce`` says where a split-K sum is taken: -1 inside the GEMM kernel (the warp that delivers the last
    partial of a 32-row quadrant), 0 or 1 in a second kernel launched right after it (faster at every ``M``).
    The order of summation, and so the result, is the same.

    ``gemv`` = 1 uses the CUDA-core streaming kernel for ``M <= 4`` (a warp per weight row, no tensor cores, no
    split-K hand-off); 0 uses it where it measured faster (one row of a small or a very large weight,
    two rows of a tiny one), -1 never."""
    if out is None and order is None and not (max_ctas or splits or pair or skinny or splitk_reduce or gemv or stream_k) \
            and solutions.no_gemm_table():
        done = _lib.fast().gemm(a, b, _scope.static_b)
        if done is not None:
            return done
    _check_operands(a, b)
    M, N = a.shape[0], b.shape[0]
    if out is None:
        out = torch.empty((M, N), dtype=a.dtype, device=a.device)
    elif out.shape != (M, N) or out.dtype != a.dtype or out.stride(1) != 1:
        raise ValueError("bad output tensor")
    if not (splits or pair or skinny or gemv or stream_k or max_ctas):
        # Nothing asked for: a profiled configuration for exactly this shape (bench.gemm_profile) beats the rule.
        sol = solutions.lookup_gemm(M, N, a.shape[1], "bf16" if a.dtype == torch.bfloat16 else "fp16")
        if sol is not None:
            splits, pair, skinny = int(sol.get("splits", 0)), int(sol.get("pair", 0)), int(sol.get("skinny", 0))
            gemv, stream_k = int(sol.get("gemv", 0)), int(sol.get("stream_k", 0))
    if order is None and not (splits or pair or skinny or splitk_reduce or gemv or stream_k or max_ctas):
        rc = _lib.lib().packed_gemm(None, _packed_plain_args(a, b, out), current_stream_ptr())
        if rc:
            _lib.check(rc)
        return out
    args = _plain_args(a, b, out)
    args.max_ctas = max_ctas
    args.splits = splits
    args.pair = pair
    args.skinny = skinny
    args.splitk_reduce = splitk_reduce
    args.gemv = gemv
    args.stream_k = stream_k
    if order is not None:
        check_order_buffer(order, M, N)
        args.order = order.data_ptr()
    rc = _lib.lib().oob_gemm(None, args, current_stream_ptr())
    if rc:
        _lib.check(rc)
    return out


def order_buffer(M: int, N: int, device="cuda") -> torch.Tensor:
    """A zeroed tile-order record for an [M, N] output of the two-SM kernel (``order=`` of :func:`gemm`,
    ``order_buffer`` of the overlap ops)."""
    tiles = ((M + 255) // 256) * ((N + 255) // 256)
    return torch.zeros((2 * tiles, 2), dtype=torch.int64, device=device)


def check_order_buffer(order: torch.Tensor, M: int, N: int) -> None:
    tiles = ((M + 255) // 256) * ((N + 255) // 256)
    if order.dtype != torch.int64 or not order.is_cuda or not order.is_contiguous() or order.numel() < 4 * tiles:
        raise ValueError(f"order must be a contiguous int64 CUDA tensor of at least {2 * tiles} x 2 words")


def tile_order(order: torch.Tensor, in_sequence: bool = True) -> list:
    """Decodes a tile-order record into a list of dicts sorted by completion time: ``unit`` (2 * tile's number in the
    schedule + CTA of the pair), ``t_us`` (microseconds after the first completion), ``pair`` and ``index`` (the
    tile's position in that pair's own sequence).  Halves the kernel never wrote (rows past M) are left out.

    The CTAs of a pair store their halves on their own, and one may be a tile ahead of the other.  ``in_sequence``: such a half counts as
    complete when the tiles before it in its pair's sequence are, so that the list follows every pair's sequence; False
    gives the times as they were stamped.

    Capability parity: the reference records in which order its GEMM finishes tiles to derive reorder hints
    (tool/search.py, the tile-order capture of src/gemm/gemm_with_signal_sm90.h); here the schedule is fixed by the
    kernel (PairSched) and the record shows how the hardware actually ran it."""
    done = [(t, u, int(w >> 32), int(w & 0xFFFFFFFF)) for u, (t, w) in enumerate(order.detach().cpu().tolist()) if t > 0]
    if not done:
        return []
    if in_sequence:
        seen = {}  # pair -> (index, latest time of the tiles up to it, the same of those before it)
        done.sort(key=lambda d: (d[2], d[3]))
        for i, (t, u, pair, index) in enumerate(done):
            last, upto, before = seen.get(pair, (index, 0, 0))
            if index != last:
                before = upto
            done[i] = (max(t, before), u, pair, index)
            seen[pair] = (index, max(upto, t), before)
    t0 = min(d[0] for d in done)
    return [dict(unit=u, t_us=(t - t0) / 1e3, pair=pair, index=index)
            for t, u, pair, index in sorted(done, key=lambda d: (d[0], d[3], d[1]))]


def stable_tile_waves(records, wave: int) -> dict:
    """Compares the tile-order records of several launches of one shape (each the output of :func:`tile_order`, or a
    plain list of unit numbers in completion order) and reports what is reproducible about the order.

    ``wave`` is the number of units that complete together (CTAs of the GEMM grid; for the two-SM kernel
    2 x pairs, since every CTA of a pair records its half).  A unit's wave in a launch is its position in the
    completion order divided by ``wave``.  Returns ``waves`` (per unit: its wave when that is the same in every
    launch, else -1), ``stable_fraction``, ``hint`` (all units ordered by their median wave, then by number: an order
    that a consumer may rely on at wave granularity) and ``min_group_waves`` (the smallest g such that every unit stays
    inside the same group of g consecutive waves in every launch: the finest chunking of the output by completion
    time that holds from launch to launch).

    Capability parity: the monitor rounds of the reference's search (tool/search.py:639-754) keep the tiles that land
    in the same wave window every time and derive a stable order and a minimum group size from them.  The fused
    kernels of this library signal every tile on its own and need no such hint; the analysis is for diagnosis and for
    choosing slab boundaries of the ``chunked`` strategy."""
    if wave < 1:
        raise ValueError("wave must be at least 1")
    orders = [[(r["unit"] if isinstance(r, dict) else int(r)) for r in rec] for rec in records]
    if not orders or not orders[0]:
        return dict(waves=[], stable_fraction=0.0, hint=[], min_group_waves=0)
    units = sorted(orders[0])
    if any(sorted(o) != units for o in orders):
        raise ValueError("the records do not cover the same units")
    pos = [{u: i // wave for i, u in enumerate(o)} for o in orders]
    per_unit = {u: [p[u] for p in pos] for u in units}
    waves = [per_unit[u][0] if len(set(per_unit[u])) == 1 else -1 for u in units]
    n_waves = (len(units) + wave - 1) // wave
    g = 1
    while g < n_waves and any(len({w // g for w in ws}) > 1 for ws in per_unit.values()):
        g += 1
    median = {u: sorted(ws)[len(ws) // 2] for u, ws in per_unit.items()}
    return dict(waves=waves, stable_fraction=sum(1 for w in waves if w >= 0) / len(units),
                hint=sorted(units, key=lambda u: (median[u], u)), min_group_waves=g)


def reserve_workspace(splitk_bytes: int = 0) -> None:
    """Allocates the library's GEMM scratch on the current device now: the stream-K workspace of the two-SM kernel and,
    when ``splitk_bytes`` > 0, a split-K workspace of that size (see :func:`splitk_workspace_bytes`).  Call it before
    capturing a CUDA graph: nothing can be allocated during capture, and a GEMM that would need to grow its workspace
    then fails instead."""
    _lib.check(_lib.lib().oob_gemm_reserve_workspace(int(splitk_bytes)))


def splitk_workspace_bytes(M: int, N: int, K: int, *, max_ctas: int = 0, splits: int = 0) -> int:
    """Split-K workspace bytes :func:`gemm` needs for this shape (0 when the problem is not split)."""
    return int(_lib.lib().oob_gemm_splitk_bytes(M, N, K, max_ctas, splits))


def gemm_plan_splits(M: int, N: int, K: int, *, max_ctas: int = 0, splits: int = 0) -> int:
    """Number of K splits the tiled kernels use for this shape (1 = the problem is not split)."""
    return int(_lib.lib().oob_gemm_plan_splits(M, N, K, max_ctas, splits))


class RowSums(NamedTuple):
    """Sums of squares of the rows of a residual stream, one per 128 columns: the norm that is still to be applied to
    ``scaled`` (the stream times the norm's weight) by the GEMM that reads it."""
    scaled: torch.Tensor  # [M, hidden]
    ssq: torch.Tensor     # [ceil(hidden / 128), M] fp32
    eps: float


def _scaled_rows(x: RowSums) -> torch.Tensor:
    """``x.scaled``, once ``x.ssq`` is seen to belong to it.  The kernel reads ``ssq`` as dense ``[ceil(K / 128), M]`` fp32: for some of
    the rows, slices of both tensors are only that when the sums have been copied (``ssq[:, rows].contiguous()``)."""
    want = ((x.scaled.shape[1] + 127) // 128, x.scaled.shape[0]) if x.scaled.dim() == 2 else ()
    if x.ssq.dtype != torch.float32 or x.ssq.shape != want or x.ssq.device != x.scaled.device or not x.ssq.is_contiguous():
        raise ValueError(f"row sums must be a contiguous fp32 tensor {list(want)} beside the [M, K] rows that they belong to")
    return x.scaled


def _set_row_sums(args: _lib.GemmArgs, x) -> None:
    if isinstance(x, RowSums):
        args.row_ssq, args.row_parts, args.row_eps = x.ssq.data_ptr(), x.ssq.shape[0], x.eps


DEFERRED_NORM_MAX_ROWS = 128


def gemm_add_norm(a: torch.Tensor, b: torch.Tensor, residual: torch.Tensor, weight: torch.Tensor, eps: float) -> tuple:
    """The row-parallel projection in front of an RMSNorm on one GPU, for up to 128 rows: ``h = residual + a @ b.T`` and the norm of ``h``
    as a :class:`RowSums`, which :func:`gemm_swiglu` and ``gemm_rope_kv_write`` take in place of the normalised rows.  They
    divide by the rms after the product, where the sums are still fp32: no norm kernel runs.  Returns ``(RowSums, h)``."""
    _check_operands(a, b)
    M, N = a.shape[0], b.shape[0]
    if M > DEFERRED_NORM_MAX_ROWS or N % 8 != 0:
        raise ValueError(f"at most {DEFERRED_NORM_MAX_ROWS} rows, and columns in multiples of 8")
    if residual.shape != (M, N) or residual.dtype != a.dtype or residual.stride(1) != 1 or residual.stride(0) % 4 != 0 \
            or weight.shape != (N,) or weight.dtype != a.dtype or not weight.is_contiguous() or residual.device != a.device \
            or weight.device != a.device:
        raise ValueError("residual must be [M, N] with unit column stride and weight [N], both of the operands' dtype and device")
    h = torch.empty((M, N), dtype=a.dtype, device=a.device)
    scaled = torch.empty_like(h)
    ssq = torch.empty(((N + 127) // 128, M), dtype=torch.float32, device=a.device)
    epi = _lib.AddEpilogue(residual.data_ptr(), residual.stride(0), weight.data_ptr(), scaled.data_ptr(), ssq.data_ptr())
    args = _plain_args(a, b, h)
    args.epilogue = _lib.EPILOGUE_ADD
    args.epilogue_args = ctypes.addressof(epi)
    _lib.check(_lib.lib().oob_gemm(None, args, current_stream_ptr()))
    return RowSums(scaled, ssq, eps), h


def gemm_swiglu(a: torch.Tensor, b: torch.Tensor, out: Optional[torch.Tensor] = None, *, max_ctas: int = 0,
                fused: Optional[bool] = None) -> torch.Tensor:
    """``silu(a @ b[:F].T) * (a @ b[F:].T)`` for a gate/up weight ``b`` of shape [2F, K]; returns [M, F].

    The activation is applied to the fp32 sums by the kernel that has them (the weight-streaming kernel, the two-SM kernel's
    epilogue or the split-K sum): no separate launch and no 16-bit round trip of the [M, 2F] intermediate.  Where none of
    them may run (``OOB_GEMM_PAIR=0``, one CTA), for one row of a large weight, and with ``fused=False`` the GEMM is followed
    by the stand-alone SwiGLU kernel.  ``fused=True`` insists on a problem that the tiled kernels would split over K (every
    decode-step shape) and raises otherwise.  ``a`` may be a :class:`RowSums` (see
    :func:`gemm_add_norm`)."""
    if out is None and fused is None and max_ctas == 0:
        done = _lib.fast().gemm_swiglu(a, b, _scope.static_b)
        if done is not None:
            return done
    from .decode import silu_mul
    sums = a
    if isinstance(a, RowSums):
        if max_ctas or fused is False:
            raise ValueError("row sums need the kernel that this call rules out")
        a = _scaled_rows(a)
    _check_operands(a, b)
    M, N = a.shape[0], b.shape[0]
    if N % 16 != 0:
        raise ValueError("the gate/up weight must have 2F rows with F a multiple of 8")
    F = N // 2
    if out is None:
        out = torch.empty((M, F), dtype=a.dtype, device=a.device)
    elif out.shape != (M, F) or out.dtype != a.dtype or out.stride(1) != 1 or out.stride(0) % 8 != 0:
        raise ValueError("bad output tensor")
    can_fuse = gemm_plan_splits(M, N, a.shape[1], max_ctas=max_ctas) > 1
    if fused and not can_fuse:
        raise ValueError("this problem is not split over K, so the epilogue has no kernel to run in")
    if fused is False:
        return silu_mul(gemm(a, b, max_ctas=max_ctas), out)
    epi = _lib.SwigluEpilogue(F)
    args = _plain_args(a, b, out)
    _set_row_sums(args, sums)
    args.max_ctas = max_ctas
    args.epilogue = _lib.EPILOGUE_SWIGLU if can_fuse else _lib.EPILOGUE_SWIGLU_TILE
    args.epilogue_args = ctypes.addressof(epi)
    rc = _lib.lib().oob_gemm(None, args, current_stream_ptr())
    if rc == _lib.ERR_UNSUPPORTED and not can_fuse and sums is a:  # no kernel that has the sums may or can apply it: two kernels
        dense = silu_mul(gemm(a, b, max_ctas=max_ctas), out if out.is_contiguous() else None)
        return out if dense is out else out.copy_(dense)
    if rc:
        _lib.check(rc)
    return out
