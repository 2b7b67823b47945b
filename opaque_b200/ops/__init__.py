"""Python front-ends of the sm_100a kernels, each with a plain-PyTorch reference.

Every ``*_ref`` function is the fp32 PyTorch statement of the same operation; it is the
numerics oracle in the tests and the implementation used on CPU.  The CUDA entry points fail
loudly when the kernel library cannot be loaded on a GPU machine — there is no silent
fallback on device tensors.

Kernel inventory (reference counterparts: packages/opaque-patches/src/opaque/api/patches/kernels/*,
packages/opaque-engine/src/opaque/api/engine/clipping/_pytree.py:475-564,
packages/opaque-dpsgd/src/opaque/api/dpsgd/noise/_gaussian.py:235-278,
packages/opaque-optimizers/src/opaque/api/optimizers/_adam.py:120-270):
  wgrad_clip            clip-weighted weight-gradient GEMM with (peer) reduce epilogue   [tcgen05]
  ghost_norm            per-example gradient norms of linear / embedding layers          [tcgen05]
  rms_norm / fused add  forward, dX, per-example dW
  glu                   SwiGLU / GeGLU forward and backward
  rope_qk               joint rotary embedding of Q and K (GQA, position ids)
  cross_entropy         online-softmax NLL with in-place dlogits (softcap, scale, smoothing)
  philox_normal_add_    counter-based Gaussian noise
  rows_sumsq / clip_weighted_sum / embedding_wgrad   direct-norm path for small parameters
  shard_step            noise (iid | BLT | banded) + AdamW-BC + bf16 write-back to every rank
"""
from __future__ import annotations

import functools
import math
import struct
from typing import Sequence

import torch

from . import lib
from .lib import DeviceWaitTimeout, KernelLibraryError, StatusWord

DEFAULT_WAIT_BUDGET_S = 2.0


def _c(t: torch.Tensor) -> torch.Tensor:
    return t if t.is_contiguous() else t.contiguous()


def _need_bf16(*ts: torch.Tensor) -> None:
    for t in ts:
        if t.dtype != torch.bfloat16:
            raise TypeError(f"expected bf16 tensors, got {t.dtype}")


# =============================================================================== wgrad / ghost

def pick_block_n(n: int) -> int:
    """Output tile width of the clip-weighted GEMM for ``n`` columns."""
    if n > 128:
        return 256
    return 128 if n > 64 else 64


def pick_splits(work_tiles: int, rows: int, sms: int, *, max_splits: int | None = None) -> int:
    """K-splits that balance the persistent grid: maximise ``items / (waves · sms)`` for ``items = tiles · splits``.

    Every split keeps at least 8 k-blocks of 64 rows; ties go to the smaller split count (less reduction traffic).
    """
    cap = max(1, rows // (64 * 8))
    if max_splits is not None:
        cap = min(cap, max_splits)
    cap = min(cap, max(1, 2 * sms // max(work_tiles, 1)) if work_tiles < sms else 4)
    best, best_eff = 1, 0.0
    for s in range(1, cap + 1):
        items = work_tiles * s
        eff = items / (math.ceil(items / sms) * sms)
        if eff > best_eff + 0.02:
            best, best_eff = s, eff
    return best


def _check_wgrad(a, b, out, num_groups, splits, out_offset, ldm, ldn, n_valid, accumulate, group_stride, group_out_offset, peer_table,
                 shard_elems) -> tuple[int, int, int, int]:
    """Argument checks of :func:`wgrad_clip`; returns ``(T, M, N, ldm)``."""
    _need_bf16(a, b)
    T, M = a.shape
    N = b.shape[1]
    if b.shape[0] != T:
        raise ValueError("a and b must have the same number of rows")
    if a.stride(1) != 1 or b.stride(1) != 1:
        raise ValueError("operands must be row-major")
    if ldm is None:
        ldm = N
    if not accumulate and splits != 1:
        raise ValueError("store mode cannot split K")
    n_lim = min(N, n_valid) if n_valid else N
    if out is not None:
        if out.dtype != torch.float32:
            raise TypeError("the destination must be fp32")
        last_group = int(group_out_offset.max()) if group_out_offset is not None else (num_groups - 1) * group_stride
        hi = out_offset + last_group + (M - 1) * ldm + (n_lim - 1) * ldn
        room = out.untyped_storage().nbytes() // 4 - out.storage_offset()
        if min(out_offset, ldm, ldn) < 0 or hi >= room:
            raise ValueError(f"wgrad_clip would write element {hi} of a destination holding {room}")
    elif peer_table is None or shard_elems <= 0:
        raise ValueError("give either a destination tensor or a peer table with shard_elems")
    return T, M, N, ldm


_WGRAD_DESC, _WGRAD_PE_DESC, _GHOST_DESC = struct.Struct("5Q6q7i4x"), struct.Struct("4Q4q6i"), struct.Struct("6Q3q4i")


def _batch_splits(tiles: int, rows: int, max_splits: int | None = None, peer: bool = False) -> int:
    """K-splits of a launch that holds ``tiles`` output tiles over all of its problems: none once they make four waves
    (the last, partly filled wave then costs little, and every split adds a pass of reductions over the outputs)."""
    sms = lib.sm_count()
    if tiles >= 4 * sms or (peer and tiles * 2 >= sms):
        return 1
    return pick_splits(max(tiles, 1), rows, sms, max_splits=max_splits)


@functools.lru_cache(maxsize=4096)
def _packed_splits(tiles: int, rows: int, most: int, peer: int) -> int:
    return _batch_splits(tiles, rows, most if most > 0 else None, bool(peer))


def _native(name: str, wait_budget_s: float = DEFAULT_WAIT_BUDGET_S):
    """The compiled packer of a batch entry point, or ``None``; it returns False for problems that Python should look at."""
    steps = block_steps() if wait_budget_s == DEFAULT_WAIT_BUDGET_S else None
    return None if steps is None else getattr(steps, name)


def wgrad_clip_batch(problems: Sequence[dict], out: torch.Tensor | None, *, accumulate: bool = True, peer_table: torch.Tensor | None = None,
                     shard_elems: int = 0, block_n: int = 256, status: StatusWord | None = None,
                     wait_budget_s: float = DEFAULT_WAIT_BUDGET_S) -> None:
    """Several :func:`wgrad_clip` problems with one destination in one launch (per 56): dictionaries with that function's
    ``a``, ``b`` and optional ``row_scale``, ``seg_offsets``, ``num_groups``, ``out_offset``, ``ldm``, ``ldn``, ``n_valid``,
    ``group_stride``.  ``block_n`` is 256 or 64.  K is split (``accumulate`` only, ungrouped problems) when the whole list
    would leave SMs idle."""
    native = _native("wgrad_batch", wait_budget_s) if accumulate and block_n == 256 else None
    if native is not None and native(problems, out, peer_table, shard_elems, status.ptr() if status else 0):
        return
    tiles = sum(pr.get("num_groups", 1) * math.ceil(pr["a"].shape[1] / 128) * math.ceil(pr["b"].shape[1] / block_n) for pr in problems)
    jobs = []
    for pr in problems:
        a, b, groups = pr["a"], pr["b"], pr.get("num_groups", 1)
        splits = _batch_splits(tiles, a.shape[0], peer=peer_table is not None) if accumulate and groups == 1 else 1
        off, gstride, nv, ldn = pr.get("out_offset", 0), pr.get("group_stride", 0), pr.get("n_valid", 0), pr.get("ldn", 1)
        T, M, N, ldm = _check_wgrad(a, b, out, groups, splits, off, pr.get("ldm"), ldn, nv, accumulate, gstride, None, peer_table, shard_elems)
        jobs.append((T / (groups * splits), _WGRAD_DESC.pack(
            a.data_ptr(), b.data_ptr(), lib.ptr(pr.get("row_scale")) or 0, lib.ptr(pr.get("seg_offsets")) or 0, 0, a.stride(0), b.stride(0),
            gstride, off, ldm, ldn, T, M, N, groups, splits, nv, int(accumulate))))
    jobs.sort(key=lambda j: -j[0])                       # longest items first: the tail of the launch is made of short ones
    rc = lib.load().ob_wgrad_clip_batch(b"".join(j[1] for j in jobs), len(jobs), lib.ptr(out), lib.ptr(peer_table), shard_elems, block_n,
                                        status.ptr() if status else None, wait_budget_s, lib.sm_count(), lib.stream())
    lib.check(rc, "wgrad_clip_batch")


def wgrad_clip(a: torch.Tensor, b: torch.Tensor, out: torch.Tensor | None, *, row_scale: torch.Tensor | None = None,
               seg_offsets: torch.Tensor | None = None, num_groups: int = 1, splits: int | None = None,
               out_offset: int = 0, ldm: int | None = None, ldn: int = 1, n_valid: int = 0, accumulate: bool = True,
               group_stride: int = 0, group_out_offset: torch.Tensor | None = None,
               peer_table: torch.Tensor | None = None, shard_elems: int = 0, block_n: int | None = None,
               status: StatusWord | None = None, wait_budget_s: float = DEFAULT_WAIT_BUDGET_S) -> None:
    """``flat[out_offset + g_off + m*ldm + n*ldn] (+)= Σ_t s[t]·a[t, m]·b[t, n]`` over each segment.

    ``a`` is ``[T, M]`` (scaled operand, e.g. output gradients), ``b`` is ``[T, N]`` (layer inputs),
    both bf16 with 16-byte aligned rows.  ``out`` is the flat fp32 destination, or ``None`` with a
    ``peer_table`` (int64 device tensor of per-rank shard base pointers) and ``shard_elems``.
    """
    bn = block_n or pick_block_n(min(b.shape[1], n_valid) if n_valid else b.shape[1])
    sms = lib.sm_count()
    if splits is None:
        tiles = num_groups * math.ceil(a.shape[1] / 128) * math.ceil(b.shape[1] / bn)
        splits = pick_splits(tiles, a.shape[0] // max(num_groups, 1), sms) if accumulate else 1
    T, M, N, ldm = _check_wgrad(a, b, out, num_groups, splits, out_offset, ldm, ldn, n_valid, accumulate, group_stride, group_out_offset,
                                peer_table, shard_elems)
    rc = lib.load().ob_wgrad_clip(
        a.data_ptr(), b.data_ptr(), T, M, N, a.stride(0), b.stride(0), lib.ptr(row_scale), lib.ptr(seg_offsets),
        num_groups, splits, lib.ptr(out), lib.ptr(peer_table), shard_elems, lib.ptr(group_out_offset), group_stride,
        out_offset, ldm, ldn, n_valid, int(accumulate), bn, status.ptr() if status else None, wait_budget_s, sms,
        lib.stream())
    lib.check(rc, "wgrad_clip")


def direct_norm2(a: torch.Tensor, g: torch.Tensor, norm2: torch.Tensor, rows_per_example: int, *, splits: int | None = None,
                 status: StatusWord | None = None, wait_budget_s: float = DEFAULT_WAIT_BUDGET_S) -> torch.Tensor:
    """``norm2[e] += ‖a_eᵀ g_e‖²_F`` for example e = rows ``[e·R, (e+1)·R)`` of ``a [T, d_in]`` and ``g [T, d_out]``.

    The direct form of a per-example gradient norm: the per-example products pass through tensor memory tile by tile
    (the clip-weighted weight-gradient kernel with a different epilogue) and only their squares are summed.
    ``2·R·d_in·d_out`` FLOPs per example against ``R²·(d_in + d_out)`` for :func:`ghost_norm`; see
    :func:`pick_norm_path`.  ``R % 64 == 0``.
    """
    _need_bf16(a, g)
    T, M = a.shape
    N = g.shape[1]
    if g.shape[0] != T or a.stride(1) != 1 or g.stride(1) != 1:
        raise ValueError("a [T, d_in] and g [T, d_out] must be row-major with the same number of rows")
    if rows_per_example <= 0 or rows_per_example % 64 or T % rows_per_example:
        raise ValueError("rows_per_example must be a multiple of 64 that divides the number of rows")
    B = T // rows_per_example
    if norm2.dtype != torch.float32 or norm2.numel() < B or not norm2.is_contiguous():
        raise ValueError("norm2 must hold one contiguous fp32 value per example")
    sms = lib.sm_count()
    if splits is None:
        tiles = math.ceil(M / 128) * math.ceil(N / 256)
        splits = pick_splits(tiles, T, sms, max_splits=B)
    desc = _WGRAD_PE_DESC.pack(a.data_ptr(), g.data_ptr(), 0, norm2.data_ptr(), a.stride(0), g.stride(0), 0, N, B, rows_per_example, M, N,
                               splits, 0)
    rc = lib.load().ob_wgrad_clip_pe_batch(desc, 1, None, None, 0, status.ptr() if status else None, wait_budget_s, sms, lib.stream())
    lib.check(rc, "direct_norm2")
    return norm2


def pick_norm_path(rows_per_example: int, d_in: int, d_out: int, examples: int | None = None, sms: int = 148) -> str:
    """``"ghost"`` (Gram matrices, ``R²·(d_in + d_out)`` FLOPs on the upper triangle) or ``"direct"`` (the per-example
    product itself, ``2·R·d_in·d_out``) for one layer.  The Gram kernel runs at about 0.7 of the product kernel's rate, so
    the direct form wins once ``R > 1.4·d_in·d_out / (d_in + d_out)``; it needs ``R % 64 == 0``.

    With few ``examples`` an output head is the exception, at any length: a Gram item runs all ``(d_in + d_out) / 64`` k-blocks
    (about 280 clocks each, 530 off the diagonal) on one SM, and with fewer items than SMs the launch waits for it: with 3 x 199
    rows and 2048 + 151936 columns 670 of the 735 us that the norms of a whole model took.  The direct form spreads over the
    output tiles."""
    if examples is not None and d_in + d_out > 16384:
        blocks = -(-rows_per_example // 128)
        tiles = -(-examples * -(-d_in // 128) * -(-d_out // 256) // sms) * (-(-rows_per_example // 64) * 512 + 1500)
        if examples * blocks * (blocks + 1) <= sms and 1.5 * tiles < (d_in + d_out) / 64 * (280 if blocks == 1 else 530):
            return "direct"
    if rows_per_example % 64:
        return "ghost"
    return "direct" if rows_per_example * (d_in + d_out) > 1.4 * d_in * d_out else "ghost"


def wgrad_clip_per_example(a: torch.Tensor, b: torch.Tensor, out: torch.Tensor | None, *, ex_scale: torch.Tensor | None,
                           rows_per_example: int, out_offset: int = 0, ldm: int | None = None, accumulate: bool = True,
                           splits: int | None = None, peer_table: torch.Tensor | None = None, shard_elems: int = 0,
                           status: StatusWord | None = None, wait_budget_s: float = DEFAULT_WAIT_BUDGET_S) -> None:
    """``flat[out_offset + m*ldm + n] (+)= Σ_e c[e] · a_eᵀ b_e`` with example e = rows ``[e·R, (e+1)·R)``, ``R % 64 == 0``.

    The clip factor multiplies each example's fp32 partial product in the epilogue (TMEM → registers), so the operand
    tiles go from TMA straight to the tensor core and ``c`` is applied unrounded.
    """
    _need_bf16(a, b)
    T, M = a.shape
    N = b.shape[1]
    if b.shape[0] != T or a.stride(1) != 1 or b.stride(1) != 1:
        raise ValueError("a [T, M] and b [T, N] must be row-major with the same number of rows")
    if rows_per_example <= 0 or rows_per_example % 64 or T % rows_per_example:
        raise ValueError("rows_per_example must be a multiple of 64 that divides the number of rows")
    B = T // rows_per_example
    if ex_scale is not None and (ex_scale.dtype != torch.float32 or ex_scale.numel() < B or not ex_scale.is_contiguous()):
        raise ValueError("ex_scale must hold one contiguous fp32 factor per example")
    if ldm is None:
        ldm = N
    sms = lib.sm_count()
    if splits is None:
        tiles = math.ceil(M / 128) * math.ceil(N / 256)
        splits = pick_splits(tiles, T, sms, max_splits=B) if accumulate else 1
        if peer_table is not None and tiles * 2 >= sms:
            splits = 1                      # every extra split sends the whole tile over NVLink once more
    if out is not None:
        if out.dtype != torch.float32:
            raise TypeError("the destination must be fp32")
        hi = out_offset + (M - 1) * ldm + N - 1
        room = out.untyped_storage().nbytes() // 4 - out.storage_offset()
        if min(out_offset, ldm) < 0 or hi >= room:
            raise ValueError(f"wgrad_clip_per_example would write element {hi} of a destination holding {room}")
    elif peer_table is None or shard_elems <= 0:
        raise ValueError("give either a destination tensor or a peer table with shard_elems")
    desc = _WGRAD_PE_DESC.pack(a.data_ptr(), b.data_ptr(), lib.ptr(ex_scale) or 0, 0, a.stride(0), b.stride(0), out_offset, ldm, B,
                               rows_per_example, M, N, splits, int(accumulate))
    rc = lib.load().ob_wgrad_clip_pe_batch(desc, 1, lib.ptr(out), lib.ptr(peer_table), shard_elems, status.ptr() if status else None,
                                           wait_budget_s, sms, lib.stream())
    lib.check(rc, "wgrad_clip_per_example")


def _check_pe(a, b, rows_per_example) -> tuple[int, int, int, int]:
    _need_bf16(a, b)
    T, M = a.shape
    if b.shape[0] != T or a.stride(1) != 1 or b.stride(1) != 1:
        raise ValueError("a [T, M] and b [T, N] must be row-major with the same number of rows")
    if rows_per_example <= 0 or T % rows_per_example:
        raise ValueError("rows_per_example must divide the number of rows")
    return T, M, b.shape[1], T // rows_per_example


def wgrad_clip_per_example_batch(problems: Sequence[tuple], out: torch.Tensor | None, rows_per_example: int, *,
                                 peer_table: torch.Tensor | None = None, shard_elems: int = 0, status: StatusWord | None = None,
                                 wait_budget_s: float = DEFAULT_WAIT_BUDGET_S) -> None:
    """Several accumulating :func:`wgrad_clip_per_example` problems ``(a, b, ex_scale, out_offset, ldm)`` in one launch (per 56).
    ``rows_per_example`` may have any length here: an example's last 64-row block is filled up with zeros."""
    native = _native("wgrad_pe_batch", wait_budget_s)
    if native is not None and native(problems, out, rows_per_example, peer_table, shard_elems, status.ptr() if status else 0):
        return
    tiles = sum(math.ceil(pr[0].shape[1] / 128) * math.ceil(pr[1].shape[1] / 256) for pr in problems)
    descs = []
    for a, b, ex_scale, off, ldm in problems:
        T, M, N, B = _check_pe(a, b, rows_per_example)
        if ex_scale is not None and (ex_scale.dtype != torch.float32 or ex_scale.numel() < B or not ex_scale.is_contiguous()):
            raise ValueError("ex_scale must hold one contiguous fp32 factor per example")
        if out is not None:
            if out.dtype != torch.float32:
                raise TypeError("the destination must be fp32")
            hi = off + (M - 1) * ldm + N - 1
            room = out.untyped_storage().nbytes() // 4 - out.storage_offset()
            if min(off, ldm) < 0 or hi >= room:
                raise ValueError(f"wgrad_clip_per_example would write element {hi} of a destination holding {room}")
        elif peer_table is None or shard_elems <= 0:
            raise ValueError("give either a destination tensor or a peer table with shard_elems")
        splits = _batch_splits(tiles, T, B, peer_table is not None)
        descs.append(_WGRAD_PE_DESC.pack(a.data_ptr(), b.data_ptr(), lib.ptr(ex_scale) or 0, 0, a.stride(0), b.stride(0), off, ldm, B,
                                         rows_per_example, M, N, splits, 1))
    rc = lib.load().ob_wgrad_clip_pe_batch(b"".join(descs), len(descs), lib.ptr(out), lib.ptr(peer_table), shard_elems,
                                           status.ptr() if status else None, wait_budget_s, lib.sm_count(), lib.stream())
    lib.check(rc, "wgrad_clip_per_example_batch")


def direct_norm2_batch(problems: Sequence[tuple], rows_per_example: int, *, status: StatusWord | None = None,
                       wait_budget_s: float = DEFAULT_WAIT_BUDGET_S) -> None:
    """Several :func:`direct_norm2` problems ``(a, g, norm2)`` in one launch (per 56), for any ``rows_per_example``."""
    tiles = sum(math.ceil(pr[0].shape[1] / 128) * math.ceil(pr[1].shape[1] / 256) for pr in problems)
    descs = []
    for a, g, norm2 in problems:
        T, M, N, B = _check_pe(a, g, rows_per_example)
        if norm2.dtype != torch.float32 or norm2.numel() < B or not norm2.is_contiguous():
            raise ValueError("norm2 must hold one contiguous fp32 value per example")
        descs.append(_WGRAD_PE_DESC.pack(a.data_ptr(), g.data_ptr(), 0, norm2.data_ptr(), a.stride(0), g.stride(0), 0, N, B, rows_per_example,
                                         M, N, _batch_splits(tiles, T, B), 0))
    rc = lib.load().ob_wgrad_clip_pe_batch(b"".join(descs), len(descs), None, None, 0, status.ptr() if status else None, wait_budget_s,
                                           lib.sm_count(), lib.stream())
    lib.check(rc, "direct_norm2_batch")


def wgrad_clip_ref(a, b, *, row_scale=None, seg_offsets=None, num_groups=1):
    """fp32 oracle: returns ``[num_groups, M, N]``."""
    af, bf = a.float(), b.float()
    if row_scale is not None:
        af = af * row_scale.float()[:, None]
    if seg_offsets is None:
        return (af.t() @ bf)[None]
    offs = seg_offsets.tolist()
    return torch.stack([af[offs[g]:offs[g + 1]].t() @ bf[offs[g]:offs[g + 1]] for g in range(num_groups)])


def _check_ghost(a, g, norm2, tokens_per_example, ids, seg_offsets, seg_out):
    """Argument checks of :func:`ghost_norm`; returns ``(rows, segments, d_in, d_out, input pitch, input pointer)``."""
    _need_bf16(g)
    rows, dg = g.shape
    if seg_offsets is None:
        B = rows // tokens_per_example
        if B * tokens_per_example != rows:
            raise ValueError("rows must be a multiple of tokens_per_example")
        if norm2.numel() < B:
            raise ValueError("one accumulator per example is required")
    else:
        if seg_offsets.dtype != torch.int32 or (seg_out is not None and seg_out.dtype != torch.int32):
            raise TypeError("segment tables must be int32")
        B = seg_offsets.numel() - 1
        if seg_out is not None and seg_out.numel() != B:
            raise ValueError("seg_out needs one entry per segment")
    if ids is None:
        _need_bf16(a)
        if a.shape[0] != rows:
            raise ValueError("a and g must have the same number of rows")
        da, lda, ap = a.shape[1], a.stride(0), a.data_ptr()
    else:
        if ids.dtype != torch.int32 or ids.numel() != rows:
            raise TypeError("ids must be int32 with one entry per row")
        da, lda, ap = 0, 0, None
    return rows, B, da, dg, lda, ap


def ghost_norm_batch(problems: Sequence[tuple], *, status: StatusWord | None = None, wait_budget_s: float = DEFAULT_WAIT_BUDGET_S) -> None:
    """Several :func:`ghost_norm` problems ``(a, g, norm2, tokens_per_example, ids, seg_offsets, seg_out)`` in one launch per
    Gram block shape (and per 56 problems): their items share one work list, longest first."""
    native = _native("ghost_batch", wait_budget_s)
    if native is not None and native(problems, status.ptr() if status else 0):
        return
    jobs = []
    for a, g, norm2, tokens, ids, seg_offsets, seg_out in problems:
        rows, B, da, dg, lda, ap = _check_ghost(a, g, norm2, tokens, ids, seg_offsets, seg_out)
        jobs.append((da + dg, _GHOST_DESC.pack(ap or 0, g.data_ptr(), lib.ptr(ids) or 0, norm2.data_ptr(), lib.ptr(seg_offsets) or 0,
                                               lib.ptr(seg_out) or 0, lda, g.stride(0), rows, B, tokens, da, dg)))
    jobs.sort(key=lambda j: -j[0])
    rc = lib.load().ob_ghost_norm_batch(b"".join(j[1] for j in jobs), len(jobs), status.ptr() if status else None, wait_budget_s,
                                        lib.sm_count(), lib.stream())
    lib.check(rc, "ghost_norm_batch")


def ghost_norm(a: torch.Tensor | None, g: torch.Tensor, norm2: torch.Tensor, tokens_per_example: int, *,
               ids: torch.Tensor | None = None, seg_offsets: torch.Tensor | None = None,
               seg_out: torch.Tensor | None = None, status: StatusWord | None = None,
               wait_budget_s: float = DEFAULT_WAIT_BUDGET_S) -> None:
    """``norm2[i] += ‖A_iᵀ G_i‖_F²`` for every segment i of rows.

    Uniform layout: segment i is rows ``[i·T, (i+1)·T)``.  Ragged layout: ``seg_offsets`` (int32 ``[S+1]``) gives the
    row range of each segment (none longer than ``tokens_per_example``) and ``seg_out`` (int32 ``[S]``) the
    accumulator each segment adds to (e.g. the example an (expert, example) group belongs to).
    With ``ids`` (int32, one per row) the inputs are one-hot rows (embedding layer) and ``a`` is unused.
    """
    ghost_norm_batch([(a, g, norm2, tokens_per_example, ids, seg_offsets, seg_out)], status=status, wait_budget_s=wait_budget_s)


PAIR_GEMM = True          # dense (ungrouped) products run on CTA pairs (256 x 256 tiles, tcgen05 cta_group::2)


def _check_b(b: torch.Tensor, layout: str, K: int, what: str) -> int:
    if b.ndim != 2 or b.stride(1) != 1:
        raise ValueError(f"{what} must be a row-major 2-D matrix")
    kn = layout == "kn"
    if (b.shape[0] if kn else b.shape[1]) != K:
        raise ValueError(f"{what}: inner dimensions differ")
    return b.shape[1] if kn else b.shape[0]


_PAIR_TILES = {"auto": -1, "512x256": 0, "256x256": 1}


def _pair_tile(tile: str) -> int:
    if tile not in _PAIR_TILES:
        raise ValueError("tile must be '512x256', '256x256' or 'auto'")
    return _PAIR_TILES[tile]


def gemm_pair(a: torch.Tensor, b: torch.Tensor, *, b_layout: str = "nk", a2: torch.Tensor | None = None,
              b2: torch.Tensor | None = None, b2_layout: str = "nk", bias: torch.Tensor | None = None,
              out: torch.Tensor | None = None, status: StatusWord | None = None,
              wait_budget_s: float = DEFAULT_WAIT_BUDGET_S, tile: str = "auto") -> torch.Tensor:
    """``a @ op(b) + a2 @ op(b2) + bias`` on CTA pairs (``tcgen05 … cta_group::2``; bf16 in/out, fp32 accumulation).

    Layouts as in :func:`gemm`; the second segment has its own layout, so ``dX = dG·Wg + dU·Wu`` (both weights
    stored ``[K, N]`` from the product's point of view) and the LoRA data gradient ``dY·W + q·A`` are one launch each.
    ``tile``: ``"512x256"`` (one tile fills tensor memory; fewest operand bytes per FLOP), ``"256x256"`` (two accumulators
    alternate, so a tile drains during the whole main loop of the next) or ``"auto"`` (by size); the same bits either way.
    """
    _need_bf16(a, b)
    if a.ndim != 2 or a.stride(1) != 1:
        raise ValueError("a must be a row-major 2-D matrix")
    M, K = a.shape
    N = _check_b(b, b_layout, K, "b")
    K2 = 0
    if a2 is not None:
        _need_bf16(a2, b2)
        if a2.ndim != 2 or a2.shape[0] != M or a2.stride(1) != 1:
            raise ValueError("second segment: a2 must be [M, K2] row-major")
        K2 = a2.shape[1]
        if _check_b(b2, b2_layout, K2, "b2") != N:
            raise ValueError("second segment: b2 must cover the same N")
    if bias is not None:
        _need_bf16(bias)
        if bias.numel() != N or not bias.is_contiguous():
            raise ValueError("bias must hold N contiguous values")
    if out is None:
        out = torch.empty(M, N, dtype=torch.bfloat16, device=a.device)
    elif out.shape != (M, N) or out.dtype != torch.bfloat16 or out.stride(1) != 1:
        raise ValueError("out must be a row-major bf16 [M, N] matrix")
    rc = lib.load().ob_gemm_pair(
        a.data_ptr(), b.data_ptr(), None, lib.ptr(a2), lib.ptr(b2), None, lib.ptr(bias), out.data_ptr(), None, None,
        M, N, K, K2, a.stride(0), b.stride(0), a2.stride(0) if a2 is not None else 0,
        b2.stride(0) if b2 is not None else 0, out.stride(0), int(b_layout == "kn"), int(b2_layout == "kn"), 0, 0, _pair_tile(tile),
        status.ptr() if status else None, wait_budget_s, lib.sm_count(), lib.stream())
    lib.check(rc, "gemm_pair")
    return out


def lora_pack(factors: Sequence[tuple[torch.Tensor, torch.Tensor]]) -> tuple[torch.Tensor, torch.Tensor]:
    """``(a_cat [3r, in], b_block [Σout, 3r])`` of three LoRA pairs ``(A [r, in], B [out, r])``: the A factors stacked, the B
    factors on the diagonal of a zero matrix (contiguous bf16, ``r % 8 == 0``)."""
    (aq, bq), (ak, bk), (av, bv) = factors
    r, d_in = aq.shape
    outs = (bq.shape[0], bk.shape[0], bv.shape[0])
    if any(a.shape != (r, d_in) or b.shape[1] != r or a.dtype != torch.bfloat16 or b.dtype != torch.bfloat16 or not a.is_contiguous()
           or not b.is_contiguous() for a, b in factors):
        raise ValueError("lora_pack: contiguous bf16 factors A [r, in], B [out, r] of one rank")
    a_cat = torch.empty(3 * r, d_in, dtype=aq.dtype, device=aq.device)
    b_block = torch.empty(sum(outs), 3 * r, dtype=aq.dtype, device=aq.device)
    rc = lib.load().ob_lora_pack(aq.data_ptr(), ak.data_ptr(), av.data_ptr(), bq.data_ptr(), bk.data_ptr(), bv.data_ptr(), a_cat.data_ptr(),
                                 b_block.data_ptr(), r, d_in, *outs, lib.sm_count(), lib.stream())
    lib.check(rc, "lora_pack")
    return a_cat, b_block


def die_map() -> list[int] | None:
    """Die (0 / 1) of every SM of the current device by ``%smid``, or ``None`` when no two-die split was measured.

    Probed once per device and process by timing atomics from every SM (a line's home L2 slice answers faster to SMs of
    its own die); the CTA-pair GEMMs use it to keep tiles that share operands on one die.  Synchronises the device on
    the first call, so call it outside CUDA-graph captures (the GEMM entry points skip the probe while capturing).
    """
    import ctypes
    buf = (ctypes.c_ubyte * 256)()
    n = lib.load().ob_die_map(buf, 256)
    return [int(buf[i]) for i in range(n)] if n > 0 else None


def set_die_aware_tiles(on: bool) -> bool:
    """Switch the die-aware tile assignment of the CTA-pair GEMMs on or off for later launches; returns the old setting.

    On: the clusters of each die (see :func:`die_map`) claim tiles from one contiguous range of the raster, so operands
    shared by neighbouring tiles cross the die-to-die link once.  Off (default): cluster ``c`` takes tiles ``c, c + n, …``.
    Measured: fewer sectors over the link, no change in kernel time.
    """
    return bool(lib.load().ob_pair_set_die_aware(1 if on else 0))


_GLU_ACT = {"silu": 0, "gelu": 1, "gelu_pytorch_tanh": 2, "gelu_tanh": 2}


def gemm_glu(a: torch.Tensor, w_gate: torch.Tensor, w_up: torch.Tensor, *, act: str = "silu", save_preact: bool = True,
             status: StatusWord | None = None, wait_budget_s: float = DEFAULT_WAIT_BUDGET_S):
    """Gated-MLP up-projection in ONE launch: ``act(a W_gᵀ) * (a W_uᵀ)`` with both products in one accumulator tile.

    ``w_gate`` and ``w_up`` are ``[I, K]`` as stored.  Returns ``(h, gate, up)``; ``gate`` / ``up`` (the bf16
    pre-activations the backward pass needs) are ``None`` with ``save_preact=False``.
    """
    _need_bf16(a, w_gate, w_up)
    if a.ndim != 2 or a.stride(1) != 1 or w_gate.ndim != 2 or w_gate.shape != w_up.shape or w_gate.stride(1) != 1 \
            or w_up.stride(1) != 1 or w_gate.stride(0) != w_up.stride(0) or w_gate.shape[1] != a.shape[1]:
        raise ValueError("gemm_glu: a [M, K] and w_gate, w_up [I, K] row-major with equal pitch")
    M, K = a.shape
    inter = w_gate.shape[0]
    h = torch.empty(M, inter, dtype=torch.bfloat16, device=a.device)
    g = torch.empty_like(h) if save_preact else None
    u = torch.empty_like(h) if save_preact else None
    rc = lib.load().ob_gemm_pair(
        a.data_ptr(), w_gate.data_ptr(), w_up.data_ptr(), None, None, None, None, h.data_ptr(), lib.ptr(g), lib.ptr(u),
        M, 2 * inter, K, 0, a.stride(0), w_gate.stride(0), 0, 0, h.stride(0), 0, 0, 1, _GLU_ACT[act], -1,
        status.ptr() if status else None, wait_budget_s, lib.sm_count(), lib.stream())
    lib.check(rc, "gemm_glu")
    return h, g, u


def gemm_glu_bwd(dy: torch.Tensor, w_down: torch.Tensor, gate: torch.Tensor, up: torch.Tensor, *, act: str = "silu",
                 status: StatusWord | None = None, wait_budget_s: float = DEFAULT_WAIT_BUDGET_S):
    """Backward of ``y = (act(gate) * up) @ w_downᵀ`` up to the pre-activations, in ONE launch: ``(dgate, dup)``.

    ``dy [M, d]``, ``w_down [d, I]`` as stored, ``gate`` / ``up [M, I]`` (the bf16 pre-activations :func:`gemm_glu` kept).
    The product ``dH = dy @ w_down`` lives only in tensor memory: the epilogue rounds it to bf16 (what a stored ``dH``
    would hold), multiplies with ``up * act'(gate)`` and ``act(gate)`` and stores the two gradients.  ``I % 64 == 0``.
    """
    _need_bf16(dy, w_down, gate, up)
    if dy.ndim != 2 or dy.stride(1) != 1 or w_down.ndim != 2 or w_down.stride(1) != 1 or w_down.shape[0] != dy.shape[1]:
        raise ValueError("gemm_glu_bwd: dy [M, d] and w_down [d, I] must be row-major")
    M, K = dy.shape
    inter = w_down.shape[1]
    if gate.shape != (M, inter) or up.shape != (M, inter) or gate.stride(1) != 1 or up.stride(1) != 1 \
            or gate.stride(0) != up.stride(0) or inter % 64:
        raise ValueError("gemm_glu_bwd: gate / up must be [M, I] with equal pitch and I % 64 == 0")
    dg = torch.empty(M, inter, dtype=torch.bfloat16, device=dy.device)
    du = torch.empty_like(dg)
    rc = lib.load().ob_gemm_pair_glu_bwd(dy.data_ptr(), w_down.data_ptr(), gate.data_ptr(), up.data_ptr(), dg.data_ptr(),
                                         du.data_ptr(), M, inter, K, dy.stride(0), w_down.stride(0), gate.stride(0),
                                         dg.stride(0), 1, _GLU_ACT[act], status.ptr() if status else None, wait_budget_s,
                                         lib.sm_count(), lib.stream())
    lib.check(rc, "gemm_glu_bwd")
    return dg, du


def _act_single(M: int, N: int, K: int, kernel: str) -> bool:
    """Which kernel :func:`gemm_act` and :func:`gemm_act_bwd` run: the single-CTA one (64-column tiles) or the pair kernel."""
    if kernel == "auto":
        return N % 64 == 0 and _plan_code(M, N, K, 0, 2) != 0
    return {"single": True, "pair": False}[kernel]


def gemm_act(a: torch.Tensor, b: torch.Tensor, bias: torch.Tensor | None = None, *, act: str = "gelu_tanh", save_preact: bool = True,
             kernel: str = "auto", status: StatusWord | None = None, wait_budget_s: float = DEFAULT_WAIT_BUDGET_S):
    """``x = a bᵀ + bias`` and ``h = act(x)`` of the rounded ``x`` in one launch; returns ``(h, x)``, ``x`` ``None`` without
    ``save_preact``.  ``kernel``: ``"pair"``, ``"single"`` (``N % 64 == 0``) or ``"auto"``; the same bits."""
    _need_bf16(a, b)
    if a.ndim != 2 or a.stride(1) != 1 or b.ndim != 2 or b.stride(1) != 1 or b.shape[1] != a.shape[1]:
        raise ValueError("gemm_act: a [M, K] and b [N, K] row-major")
    M, K = a.shape
    N = b.shape[0]
    if bias is not None:
        _need_bf16(bias)
        if bias.numel() != N or not bias.is_contiguous():
            raise ValueError("bias must hold N contiguous values")
    h = torch.empty(M, N, dtype=torch.bfloat16, device=a.device)
    x = torch.empty_like(h) if save_preact else None
    st = status.ptr() if status else None
    if _act_single(M, N, K, kernel):
        rc = lib.load().ob_gemm_tn_act(a.data_ptr(), b.data_ptr(), lib.ptr(bias), h.data_ptr(), lib.ptr(x), M, N, K, a.stride(0), b.stride(0), 0,
                                       _GLU_ACT[act], 0, st, wait_budget_s, lib.sm_count(), lib.stream())
    else:
        rc = lib.load().ob_gemm_pair(a.data_ptr(), b.data_ptr(), None, None, None, None, lib.ptr(bias), h.data_ptr(), lib.ptr(x), None, M, N, K, 0,
                                     a.stride(0), b.stride(0), 0, 0, N, 0, 0, 2, _GLU_ACT[act], -1, st, wait_budget_s, lib.sm_count(), lib.stream())
    lib.check(rc, "gemm_act")
    return h, x


def gemm_act_bwd(dy: torch.Tensor, w: torch.Tensor, x: torch.Tensor, *, act: str = "gelu_tanh", kernel: str = "auto",
                 status: StatusWord | None = None, wait_budget_s: float = DEFAULT_WAIT_BUDGET_S) -> torch.Tensor:
    """``(dy @ w) * act'(x)`` in one launch, the product rounded to bf16 first: ``dy [M, K]``, ``w [K, N]`` as stored (the second
    projection of an MLP), ``x [M, N]`` the contiguous pre-activations.  ``N % 64 == 0``; ``kernel`` as in :func:`gemm_act`."""
    _need_bf16(dy, w, x)
    if dy.ndim != 2 or dy.stride(1) != 1 or w.ndim != 2 or w.stride(1) != 1 or w.shape[0] != dy.shape[1]:
        raise ValueError("gemm_act_bwd: dy [M, K] and w [K, N] must be row-major")
    M, K = dy.shape
    N = w.shape[1]
    if x.shape != (M, N) or not x.is_contiguous() or N % 64:
        raise ValueError("gemm_act_bwd: x must be a contiguous [M, N] with N % 64 == 0")
    dx = torch.empty(M, N, dtype=torch.bfloat16, device=dy.device)
    st = status.ptr() if status else None
    if _act_single(M, N, K, kernel):
        rc = lib.load().ob_gemm_tn_act(dy.data_ptr(), w.data_ptr(), None, dx.data_ptr(), x.data_ptr(), M, N, K, dy.stride(0), w.stride(0), 1,
                                       _GLU_ACT[act], 1, st, wait_budget_s, lib.sm_count(), lib.stream())
    else:
        rc = lib.load().ob_gemm_pair_glu_bwd(dy.data_ptr(), w.data_ptr(), x.data_ptr(), None, dx.data_ptr(), None, M, N, K, dy.stride(0),
                                             w.stride(0), N, N, 1, _GLU_ACT[act], st, wait_budget_s, lib.sm_count(), lib.stream())
    lib.check(rc, "gemm_act_bwd")
    return dx


def pick_glu_bwd(M: int, inter: int, sms: int = 148) -> bool:
    """Whether :func:`gemm_glu_bwd` beats a plain data gradient and the element-wise GLU backward (the same bits): once its 256 x 256
    tiles are more than one wave.  A lone tile's epilogue has no main loop to hide behind (us, separate / fused: 128 x 8192 12.5 / 20.1,
    597 x 5632 21.1 / 21.6, both K = 2048; 1024 x 14336 x 4096, three waves, 129 / 122; 5439 x 8192 x 2048 218 / 183)."""
    return -(-M // 256) * -(-inter // 256) > sms // 2


def gemm_glu_ref(a, w_gate, w_up, *, act="silu"):
    """fp32 oracle of :func:`gemm_glu` (returns ``h`` only)."""
    g, u = a.float() @ w_gate.float().t(), a.float() @ w_up.float().t()
    if act == "silu":
        return torch.nn.functional.silu(g) * u
    return torch.nn.functional.gelu(g, approximate="tanh" if "tanh" in act else "none") * u


def linear_ce_forward(hidden: torch.Tensor, weight: torch.Tensor, labels: torch.Tensor, *, ignore_index: int = -100,
                      softcap: float = 0.0, label_smoothing: float = 0.0, store_logits: bool = False,
                      status: StatusWord | None = None, wait_budget_s: float = DEFAULT_WAIT_BUDGET_S):
    """Output head and token cross-entropy in one tcgen05 kernel: ``(nll, lse, logits | None)``.

    ``hidden [R, d]``, ``weight [V, d]`` (bf16), ``labels [R]`` (int64).  Every 256-column logits tile is reduced to
    per-row statistics in the GEMM epilogue, straight out of tensor memory; a small second kernel combines the tiles of
    a row in a fixed order (bit-reproducible).  The logits reach memory only with ``store_logits=True`` (bf16, after
    the soft cap), which is what :func:`linear_ce_dlogits_` turns into gradients in place.
    Reference counterpart: packages/opaque-patches/src/opaque/api/patches/kernels/linear_cross_entropy.py:98-208.
    """
    _need_bf16(hidden, weight)
    if hidden.ndim != 2 or weight.ndim != 2 or hidden.stride(1) != 1 or weight.stride(1) != 1 or hidden.shape[1] != weight.shape[1]:
        raise ValueError("linear_ce_forward: hidden [R, d] and weight [V, d] must be row-major")
    R, K = hidden.shape
    V = weight.shape[0]
    lab = labels.reshape(-1).to(torch.int64).contiguous()
    if lab.numel() != R:
        raise ValueError("one label per row is required")
    tiles = 2 * ((V + 255) // 256)                  # two column groups per 256-wide tile
    partials = torch.empty(max(R, 1) * tiles * 4, dtype=torch.float32, device=hidden.device)     # scratch of the epilogue
    nll = torch.empty(R, dtype=torch.float32, device=hidden.device)
    lse = torch.empty(R, dtype=torch.float32, device=hidden.device)
    logits = None
    ldo = 0
    if store_logits:
        ldo = (V + 7) // 8 * 8                       # 16-byte aligned rows for the vector stores
        logits = torch.empty(R, ldo, dtype=torch.bfloat16, device=hidden.device)[:, :V]
    rc = lib.load().ob_linear_ce_fwd(hidden.data_ptr(), weight.data_ptr(), lab.data_ptr(), lib.ptr(logits), partials.data_ptr(),
                                     nll.data_ptr(), lse.data_ptr(), R, V, K, hidden.stride(0), weight.stride(0), ldo,
                                     float(softcap), float(label_smoothing), ignore_index,
                                     status.ptr() if status else None, wait_budget_s, lib.sm_count(), lib.stream())
    lib.check(rc, "linear_ce_forward")
    return nll, lse, logits


def linear_ce_dlogits_(logits: torch.Tensor, labels: torch.Tensor, lse: torch.Tensor, row_weight: torch.Tensor | None = None, *,
                       ignore_index: int = -100, softcap: float = 0.0, label_smoothing: float = 0.0) -> torch.Tensor:
    """In place: the logits stored by :func:`linear_ce_forward` become ``row_weight · ∂nll/∂(raw logits)`` (one read, one write)."""
    _need_bf16(logits)
    if logits.ndim != 2 or logits.stride(1) != 1:
        raise ValueError("logits must be a row-major matrix")
    lab = labels.reshape(-1).to(torch.int64).contiguous()
    rc = lib.load().ob_linear_ce_dlogits(logits.data_ptr(), lab.data_ptr(), lse.data_ptr(), lib.ptr(row_weight), logits.shape[0],
                                         logits.shape[1], logits.stride(0), float(softcap), float(label_smoothing), ignore_index,
                                         lib.stream())
    lib.check(rc, "linear_ce_dlogits")
    return logits


def _waves_us(tiles: int, slots: int, nk: int, start: float, per_kb: float, per_busy: float, per_tile: float) -> float:
    """``start`` plus, for every wave of ``tiles`` over ``slots``, ``nk`` k-blocks (dearer the more slots are busy) and a tile's own cost."""
    full, rest = divmod(tiles, slots)
    us = start + full * (nk * (per_kb + per_busy * slots) + per_tile)
    return us + (nk * (per_kb + per_busy * rest) + per_tile if rest else 0.0)


def _single_us(M: int, N: int, nk: int, width: int, sms: int) -> float:
    """Estimated microseconds of the single-CTA kernel along ``nk`` k-blocks, tiles ``width`` columns wide.

    This and :func:`_pair_us` are fitted to launches back to back in a CUDA graph with weights from HBM: over 238 shapes of 1 to 16384
    rows the kernel and width with the smallest estimate took 0.25 % longer than the best one on average (4.6 % at most from 64 rows on)."""
    tiles = -(-M // 128) * -(-N // width)
    return _waves_us(tiles, sms, nk, *((3.95, 0.3506, 0.00026, 0.96) if width == 256 else (4.07, 0.1804, 0.00012, 0.12)))


def _pair_us(M: int, N: int, nk: int, sms: int) -> float:
    """The same for CTA pairs on 256 x 256 tiles."""
    return _waves_us(-(-M // 256) * -(-N // 256), max(sms // 2, 1), nk, 5.80, 0.2715, 0.00103, 0.64)


@functools.lru_cache(maxsize=4096)
def pick_tile_width(M: int, N: int, nk: int, sms: int = 148) -> int:
    """Columns per tile of the single-CTA kernel: 64 where one such tile covers ``N`` (16384 x 48 x 4096: 27.6 us, 32.9 with 256),
    or where all narrow tiles run at once and are faster by :func:`_single_us` (128 x 768 x 768: 6.1 and 8.6; 128 x 2048 x 8192: 28.5
    and 51.7); beyond one wave they lose (3663 x 768 x 768: 11.3 and 9.3)."""
    if N <= 64:
        return 64
    fits = -(-M // 128) * -(-N // 64) <= sms
    return 64 if fits and _single_us(M, N, nk, 64, sms) < _single_us(M, N, nk, 256, sms) else 256


@functools.lru_cache(maxsize=4096)
def pick_gemm_plan(M: int, N: int, K: int, K2: int = 0, sms: int = 148) -> str:
    """``"pair"`` or ``"single"`` for an ungrouped ``[M, K] x [K, N]`` product (plus a ``K2`` segment): the same bits either way.

    The one with the smaller estimate of :func:`_pair_us` and :func:`_single_us` at the better tile width (256 x 2048 x 8192: 42.1 and
    27.3 us measured; 3663 x 3072 x 768: 18.7 and 20.5; 3663 x 768 x 768: 10.3 and 9.3; 8192 x 4096 x 4096: 167 and 182).
    """
    nk = -(-K // 64) + -(-K2 // 64)
    return "pair" if _pair_us(M, N, nk, sms) <= _single_us(M, N, nk, pick_tile_width(M, N, nk, sms), sms) else "single"


def gemm(a: torch.Tensor, b: torch.Tensor, *, b_layout: str = "nk", a2: torch.Tensor | None = None,
         b2: torch.Tensor | None = None, bias: torch.Tensor | None = None, group_offs: torch.Tensor | None = None,
         out: torch.Tensor | None = None, status: StatusWord | None = None,
         wait_budget_s: float = DEFAULT_WAIT_BUDGET_S, kernel: str = "auto", b2_layout: str = "nk", alpha: float = 1.0,
         block_n: int | None = None) -> torch.Tensor:
    """``a @ op(b) + a2 @ b2ᵀ + bias`` on the tcgen05 path (bf16 in/out, fp32 accumulation).

    ``b_layout="nk"``: ``b`` is ``[N, K]`` (a weight matrix as stored; ``op(b) = bᵀ``);  ``"kn"``: ``b`` is ``[K, N]``
    (``op(b) = b`` — data gradients ``dY @ W`` without a transposed copy).  ``a2 [M, r]``, ``b2 [N, r]`` add a
    low-rank segment accumulated in the same tile (LoRA-fused linear).  With ``group_offs`` (int32 ``[E + 1]`` row
    offsets, rows sorted by group) ``b`` is ``[E, N, K]`` / ``[E, K, N]`` and rows of group e use slab e (MoE experts).
    ``kernel``: ``"pair"`` (two CTAs per tile, :func:`gemm_pair`), ``"single"`` (one CTA per 128 x ``block_n`` tile, 256 or 64
    columns, by default :func:`pick_tile_width`'s choice) or ``"auto"`` (:func:`pick_gemm_plan` for ungrouped products while
    :data:`PAIR_GEMM` is on; grouped products always run on single CTAs).  ``b2_layout="kn"``: ``b2`` is stored ``[r, N]``.  ``alpha`` scales the fp32 products (not the bias;
    single-CTA kernel only, so ``"auto"`` takes it when ``alpha`` is given).
    """
    if group_offs is None and kernel == "auto" and PAIR_GEMM:
        kernel = pick_gemm_plan(a.shape[0], b.shape[1] if b_layout == "kn" else b.shape[0], a.shape[1], 0 if a2 is None else a2.shape[1],
                                lib.sm_count())
        if alpha != 1.0:
            kernel = "single"
    if group_offs is None and kernel == "pair":
        if alpha != 1.0:
            raise ValueError("alpha runs on the single-CTA kernel")
        return gemm_pair(a, b, b_layout=b_layout, a2=a2, b2=b2, b2_layout=b2_layout, bias=bias, out=out, status=status,
                         wait_budget_s=wait_budget_s)
    _need_bf16(a, b)
    if a.ndim != 2 or a.stride(1) != 1:
        raise ValueError("a must be a row-major 2-D matrix")
    M, K = a.shape
    kn = {"nk": 0, "kn": 1}[b_layout]
    grouped = group_offs is not None
    if grouped:
        if group_offs.dtype != torch.int32 or b.ndim != 3 or not b.is_contiguous():
            raise TypeError("grouped mode needs int32 offsets and a contiguous [E, ., .] weight stack")
        E = group_offs.numel() - 1
        if b.shape[0] != E:
            raise ValueError("one weight slab per group is required")
        b2d = b.view(-1, b.shape[-1])
        N = b.shape[2] if kn else b.shape[1]
        if (b.shape[1] if kn else b.shape[2]) != K:
            raise ValueError("inner dimensions differ")
        if kn and K % 64:
            raise ValueError("grouped [K, N] slabs need K to be a multiple of 64")
    else:
        if b.ndim != 2 or b.stride(1) != 1:
            raise ValueError("b must be a row-major 2-D matrix")
        E, b2d = 0, b
        N = b.shape[1] if kn else b.shape[0]
        if (b.shape[0] if kn else b.shape[1]) != K:
            raise ValueError("inner dimensions differ")
    K2 = 0
    if a2 is not None:
        _need_bf16(a2, b2)
        K2 = a2.shape[1]
        if a2.shape[0] != M or a2.stride(1) != 1 or _check_b(b2, b2_layout, K2, "b2") != N:
            raise ValueError("low-rank segment: a2 [M, r], b2 [N, r] (or [r, N])")
    if bias is not None:
        _need_bf16(bias)
        if bias.numel() != N or not bias.is_contiguous():
            raise ValueError("bias must hold N contiguous values")
    if out is None:
        out = torch.empty(M, N, dtype=torch.bfloat16, device=a.device)
    elif out.shape != (M, N) or out.dtype != torch.bfloat16 or out.stride(1) != 1:
        raise ValueError("out must be a row-major bf16 [M, N] matrix")
    if block_n is None:
        block_n = 256 if grouped else pick_tile_width(M, N, -(-K // 64) + -(-K2 // 64), lib.sm_count())
    rc = lib.load().ob_gemm_tn(a.data_ptr(), b2d.data_ptr(), lib.ptr(a2), lib.ptr(b2), lib.ptr(bias), out.data_ptr(), M, N,
                               K, K2, a.stride(0), b2d.stride(0), a2.stride(0) if a2 is not None else 0,
                               b2.stride(0) if b2 is not None else 0, out.stride(0), kn, int(b2_layout == "kn"), alpha,
                               lib.ptr(group_offs), E, block_n, status.ptr() if status else None, wait_budget_s, lib.sm_count(), lib.stream())
    lib.check(rc, "gemm")
    return out


def _plan_code(M: int, N: int, K: int, K2: int, mode: int) -> int:
    """:func:`gemm`'s choice as a number: 0 for the pair kernel, else the single-CTA kernel's tile width.  ``mode`` 1: single-CTA only.
    2: a product with an activation in its epilogue, which wide single-CTA tiles do not have (us, element-wise launch apart / pair /
    64-column tiles, N = 3072, K = 768, forward: 128 rows 8.4 / 13.1 / 8.0, 512 12.5 / 13.3 / 10.6, 1024 13.9 / 13.7 / 13.7, 1285 14.8 /
    14.2 / 19.0, 3663 27.7 / 26.4, 16384 117 / 98)."""
    sms = lib.sm_count()
    nk = -(-K // 64) + -(-K2 // 64)
    if mode == 2:
        return 0 if _pair_us(M, N, nk, sms) <= _single_us(M, N, nk, 64, sms) else 64
    return 0 if mode == 0 and pick_gemm_plan(M, N, K, K2, sms) == "pair" else pick_tile_width(M, N, nk, sms)


@functools.lru_cache(maxsize=None)
def block_steps():
    """The compiled launch sequences (``csrc/block_steps.cpp``), or ``None`` without a GPU or where they cannot be built or loaded."""
    if not torch.cuda.is_available():
        return None
    return lib.load_block_steps(_plan_code, _packed_splits, DEFAULT_WAIT_BUDGET_S)


def gemm_ref(a, b, *, b_layout="nk", a2=None, b2=None, bias=None, group_offs=None):
    """fp32 oracle of :func:`gemm`."""
    af = a.float()
    if group_offs is None:
        y = af @ (b.float() if b_layout == "kn" else b.float().t())
    else:
        offs = group_offs.tolist()
        N = b.shape[2] if b_layout == "kn" else b.shape[1]
        y = af.new_zeros(a.shape[0], N)
        for e in range(len(offs) - 1):
            be = b[e].float() if b_layout == "kn" else b[e].float().t()
            y[offs[e]:offs[e + 1]] = af[offs[e]:offs[e + 1]] @ be
    if a2 is not None:
        y = y + a2.float() @ b2.float().t()
    if bias is not None:
        y = y + bias.float()
    return y


def ghost_set_wide(mode: int | bool) -> int:
    """Gram block shape of :func:`ghost_norm`: 1 = 128x256 blocks for examples of >= 1024 rows (default), 2 = 128x256
    whenever an example spans two row blocks, 0 = always 128x128.  Returns the previous setting."""
    return int(lib.load().ob_ghost_set_wide(int(mode)))


def ghost_norm_ref(a, g, tokens_per_example, *, ids=None):
    """PyTorch reference of ``ghost_norm``: per-example squared gradient norms from Gram matrices."""
    B = g.shape[0] // tokens_per_example
    gg = g.float().view(B, tokens_per_example, -1)
    sg = gg @ gg.transpose(1, 2)
    if ids is None:
        aa = a.float().view(B, tokens_per_example, -1)
        sa = aa @ aa.transpose(1, 2)
    else:
        i = ids.view(B, tokens_per_example)
        sa = (i[:, :, None] == i[:, None, :]).float()
    return (sa * sg).sum(dim=(1, 2))


# =============================================================================== small DP kernels

def philox_normal_add_(x: torch.Tensor, *, seed: int, offset: int = 0, std: float = 1.0, stream_id: int = 0) -> torch.Tensor:
    """In place ``x[i] += std·z(seed, offset + i)`` with ``z`` standard normal, counter-based."""
    if not x.is_contiguous():
        raise ValueError("philox_normal_add_ needs a contiguous tensor")
    code = {torch.float32: 0, torch.bfloat16: 1}[x.dtype]
    rc = lib.load().ob_philox_normal_add(x.data_ptr(), code, x.numel(), seed & (2**64 - 1), offset, float(std),
                                         stream_id, lib.sm_count(), lib.stream())
    lib.check(rc, "philox_normal_add")
    return x


def rows_sumsq(g: torch.Tensor, norm2: torch.Tensor) -> None:
    """``norm2[e] += Σ_p g[e, p]²`` for fp32 ``g [E, P]``."""
    if g.dtype != torch.float32 or g.stride(1) != 1 or norm2.numel() < g.shape[0]:
        raise ValueError("rows_sumsq needs a row-major fp32 matrix and one accumulator per row")
    rc = lib.load().ob_rows_sumsq(g.data_ptr(), g.shape[0], g.shape[1], g.stride(0), norm2.data_ptr(), lib.sm_count(),
                                  lib.stream())
    lib.check(rc, "rows_sumsq")


def clip_weighted_sum(g: torch.Tensor, c: torch.Tensor, out: torch.Tensor | None, *, flat_offset: int = 0,
                      peer_table: torch.Tensor | None = None, shard_elems: int = 0) -> None:
    """``flat[flat_offset + p] += Σ_e c[e]·g[e, p]`` (to the owning rank when a peer table is given)."""
    if out is not None and flat_offset + g.shape[1] > out.numel():
        raise ValueError("clip_weighted_sum would write past the end of the destination")
    if c.numel() < g.shape[0]:
        raise ValueError("one clip factor per example is required")
    rc = lib.load().ob_clip_weighted_sum(g.data_ptr(), c.data_ptr(), g.shape[0], g.shape[1], g.stride(0),
                                         lib.ptr(out), lib.ptr(peer_table), shard_elems, flat_offset, lib.sm_count(),
                                         lib.stream())
    lib.check(rc, "clip_weighted_sum")


CLIP_TREE_MAX_LEAVES = 64


def clip_tree(leaves: Sequence[torch.Tensor], bound: float, *, shrink: float, ulp: float, auto: bool = False, gamma: float = 0.0,
              factor: float = 1.0) -> tuple[list[torch.Tensor], torch.Tensor, torch.Tensor]:
    """Clip every example of a materialised fp32 gradient tree and sum: ``(sums, norms [E], clipped_norms [E])``.

    ``leaves`` are contiguous ``[E, ...]`` fp32 CUDA tensors.  ``norm_e`` runs over all of them (fp32 squares, fp64 sums);
    the factor of example e is ``bound / (norm + gamma)`` (``auto``) or ``min(1, bound / norm)``, shrunk to ``· shrink − ulp``
    first and 0 where it is not finite; ``sums[i] = factor · Σ_e c_e · leaves[i][e]``.  Non-finite values count as 0.
    """
    import ctypes
    E, n = leaves[0].shape[0], len(leaves)
    if n > CLIP_TREE_MAX_LEAVES or any(x.dtype != torch.float32 or not x.is_contiguous() or x.shape[0] != E for x in leaves):
        raise ValueError(f"clip_tree takes up to {CLIP_TREE_MAX_LEAVES} contiguous fp32 leaves with one leading example axis")
    dev = leaves[0].device
    sums = [torch.empty(x.shape[1:], dtype=torch.float32, device=dev) for x in leaves]
    numel = (ctypes.c_longlong * n)(*[s.numel() for s in sums])
    partial = torch.empty(max(E * lib.load().ob_clip_tree_chunks(numel, n), 1), dtype=torch.float64, device=dev)
    rows = torch.empty(3, E, dtype=torch.float32, device=dev)
    rc = lib.load().ob_clip_tree((ctypes.c_void_p * n)(*[x.data_ptr() for x in leaves]), (ctypes.c_void_p * n)(*[s.data_ptr() for s in sums]),
                                 numel, n, E, bound, gamma, shrink, ulp, int(auto), factor, partial.data_ptr(), rows[0].data_ptr(),
                                 rows[1].data_ptr(), rows[2].data_ptr(), lib.stream())
    lib.check(rc, "clip_tree")
    return sums, rows[0], rows[2]


def embedding_wgrad(g: torch.Tensor, ids: torch.Tensor, out: torch.Tensor | None, *, row_scale=None, flat_offset=0,
                    peer_table=None, shard_elems=0) -> None:
    """``flat[flat_offset + ids[t]·D + d] += s[t]·g[t, d]``."""
    _need_bf16(g)
    if ids.dtype != torch.int64:
        raise TypeError("ids must be int64")
    if ids.numel() != g.shape[0]:
        raise ValueError("one id per gradient row is required")
    rc = lib.load().ob_embedding_wgrad(g.data_ptr(), ids.data_ptr(), lib.ptr(row_scale), g.shape[0], g.shape[1],
                                       g.stride(0), lib.ptr(out), lib.ptr(peer_table), shard_elems, flat_offset,
                                       lib.sm_count(), lib.stream())
    lib.check(rc, "embedding_wgrad")


def push_grad_(local: torch.Tensor, peer_table: torch.Tensor, shard_elems: int, *, status: StatusWord | None = None) -> None:
    """Add a full-length local fp32 gradient into the owners' shards (peer reductions) and clear it.

    With a ``status`` word that is already set (a bounded wait expired earlier) the kernel does nothing."""
    if local.dtype != torch.float32 or not local.is_contiguous() or local.numel() % 4 or shard_elems % 4:
        raise ValueError("push_grad_: contiguous fp32 buffer with a length and shard size that are multiples of 4")
    rc = lib.load().ob_push_grad(local.data_ptr(), local.numel(), peer_table.data_ptr(), shard_elems,
                                 status.ptr() if status else None, lib.sm_count(), lib.stream())
    lib.check(rc, "push_grad")


def shard_step(*, grad=None, peer_grad=None, master, m, v, params_local=None, peer_params=None, world=1, global_offset=0, seed=0,
               noise_std=0.0, inv_normalize=1.0, lr=1e-3, betas=(0.9, 0.999), eps=1e-8, weight_decay=0.0, step=1,
               phi_hat=0.0, decoupled_wd=True, ftrl_state=None, ftrl_mode=0, ftrl_coef: Sequence[float] = (),
               nbuf=0, ring_head=0, noisy_out=None, skip_update=False, status: StatusWord | None = None,
               optimizer: str = "adam", nesterov: bool = False) -> None:
    """One fused pass over a shard: noise, optimizer update on fp32 masters, bf16 write-back to all ranks.

    ``optimizer``: ``"adam"`` (Adam / AdamW / AdamW-BC by ``decoupled_wd`` and ``phi_hat``), ``"sgd"`` (momentum
    ``betas[0]``, PyTorch semantics, optional Nesterov; ``v`` unused) or ``"lion"`` (``betas``; ``v`` unused).

    ``peer_grad`` (int64 device table of ``world`` full-length fp32 accumulation buffers, one per rank) selects the
    pull form: the shard's gradient is the sum over ranks, in rank order, of ``buffer_r[global_offset + i]``, read through
    peer pointers inside this kernel — the reduce-scatter is fused in, uses no atomics and gives the same bits on every
    run.  ``grad`` is then unused and nothing is cleared (each rank clears its own buffer after the closing barrier).

    ``step`` is 1-based; ``phi_hat`` is the bias-corrected noise-variance EMA (0 disables the correction).  With a
    ``status`` word that is already set (the gradient barrier before this call gave up) the kernel touches nothing:
    a partially reduced shard is neither noised, applied nor cleared.
    """
    if (grad is None) == (peer_grad is None):
        raise ValueError("shard_step takes either grad (this shard's reduced gradient) or peer_grad (the pull form)")
    if grad is not None and grad.numel() != master.numel():
        raise ValueError("grad and master must have the shard's length")
    coef = torch.tensor(list(ftrl_coef) or [0.0], dtype=torch.float32)
    import ctypes
    arr = (ctypes.c_float * len(coef))(*coef.tolist())
    rc = lib.load().ob_shard_step(
        lib.ptr(grad), lib.ptr(peer_grad), lib.ptr(master), lib.ptr(m), lib.ptr(v), lib.ptr(ftrl_state), lib.ptr(peer_params),
        lib.ptr(params_local), lib.ptr(noisy_out), master.numel(), global_offset, world, seed & (2**64 - 1),
        float(noise_std), float(inv_normalize), ftrl_mode, nbuf, ring_head, ctypes.cast(arr, ctypes.c_void_p),
        len(coef), float(lr), float(betas[0]), float(betas[1]), float(eps), float(weight_decay),
        1.0 - betas[0] ** step, 1.0 - betas[1] ** step, float(phi_hat), int(decoupled_wd), int(skip_update),
        {"adam": 0, "sgd": 1, "lion": 2}[optimizer], int(nesterov),
        status.ptr() if status else None, lib.sm_count(), lib.stream())
    lib.check(rc, "shard_step")


from . import functional  # noqa: E402
from .functional import (activation, add_layer_norm, cross_entropy, cross_entropy_ref, fused_add_rms_norm, geglu, glu_ref,  # noqa: E402
                         layer_norm, merge_heads3, plain_torch_ops, rms_norm, rms_norm_ref, rope_qk, rope_qk_ref, rope_tables, rows_group_sum_, swiglu)

__all__ = [
    "gemm", "gemm_pair", "block_steps", "lora_pack", "pick_gemm_plan", "gemm_glu", "gemm_glu_bwd", "pick_glu_bwd", "gemm_act", "gemm_act_bwd", "direct_norm2", "pick_norm_path", "die_map", "set_die_aware_tiles", "linear_ce_forward", "linear_ce_dlogits_", "gemm_glu_ref", "gemm_ref", "ghost_set_wide", "push_grad_", "wgrad_clip_per_example", "wgrad_clip_batch", "wgrad_clip_per_example_batch", "direct_norm2_batch", "ghost_norm_batch", "plain_torch_ops", "layer_norm", "add_layer_norm", "activation", "rows_group_sum_", "merge_heads3",
    "DeviceWaitTimeout", "KernelLibraryError", "StatusWord", "clip_tree", "clip_weighted_sum", "cross_entropy",
    "cross_entropy_ref", "embedding_wgrad", "fused_add_rms_norm", "geglu", "ghost_norm", "ghost_norm_ref", "glu_ref",
    "philox_normal_add_", "pick_block_n", "pick_splits", "rms_norm", "rms_norm_ref", "rope_qk", "rope_qk_ref",
    "rope_tables", "rows_sumsq", "shard_step", "swiglu", "wgrad_clip", "wgrad_clip_ref",
]
