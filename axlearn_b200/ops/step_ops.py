"""The ends of a decoding step (``csrc/step_frame.cu``): token embeddings in front, greedy pick and bookkeeping behind."""

from __future__ import annotations

import ctypes
from typing import Optional, Sequence

import torch

from axlearn_b200.ops import cuda_ops

c_void_p, c_int, c_int64 = ctypes.c_void_p, ctypes.c_int, ctypes.c_int64
_MAX_KEPT = 4
_configured = False


class _StepEndArgs(ctypes.Structure):
    _fields_ = [("logits", c_void_p), ("logits_out", c_void_p), ("tokens", c_void_p), ("lengths", c_void_p),
                ("active", c_void_p), ("kept_dst", c_void_p * _MAX_KEPT), ("kept_src", c_void_p * _MAX_KEPT),
                ("ld", c_int64), ("B", c_int), ("V", c_int), ("kept", c_int)]


def _lib():
    global _configured
    h = cuda_ops.lib()
    if not _configured:
        h.axb_step_end.argtypes = [ctypes.POINTER(_StepEndArgs), c_void_p]
        h.axb_embed_rows.argtypes = [c_void_p, c_void_p, c_void_p, c_void_p, c_int, c_int64, c_int, c_int, c_int64, c_int,
                                     c_void_p, c_void_p]
        h.axb_take_tokens.argtypes = [c_void_p, c_void_p, c_int, c_int64, c_int64, c_void_p, c_void_p]
        h.axb_add_counts.argtypes = [c_void_p, c_void_p, c_void_p, c_int, c_void_p]
        h.axb_add_counts.restype = c_int
        h.axb_step_end.restype = h.axb_embed_rows.restype = h.axb_take_tokens.restype = c_int
        _configured = True
    return h


def _row_vector(t: torch.Tensor, batch: int) -> bool:
    return t.is_cuda and t.dtype == torch.int32 and t.shape == (batch,) and t.is_contiguous()


def step_end(logits: torch.Tensor, tokens: torch.Tensor, *, logits_out: Optional[torch.Tensor] = None,
             lengths: Optional[torch.Tensor] = None, active: Optional[torch.Tensor] = None,
             kept: Sequence[tuple] = ()) -> None:
    """``tokens[b] = argmax(logits[b])`` (torch's order), ``logits_out = logits``, ``lengths += active`` and
    ``dst.copy_(src)`` for the pairs of ``kept``, in one launch where the tensors are what the kernel takes (fp32 logits
    on the GPU, int32 vectors)."""
    b, v = logits.shape
    if not (logits.is_cuda and logits.dtype == torch.float32 and logits.stride(1) == 1 and logits.stride(0) >= v
            and len(kept) <= _MAX_KEPT and tokens.dtype == torch.int64 and tokens.is_contiguous()
            and (logits_out is None or (logits_out.dtype == torch.float32 and logits_out.is_contiguous()))
            and (lengths is None or (_row_vector(lengths, b) and _row_vector(active, b)))
            and all(_row_vector(x, b) and _row_vector(y, b) for x, y in kept)):
        for dst, src in kept:
            dst.copy_(src)
        if lengths is not None:
            lengths.add_(active)
        if logits_out is not None:
            logits_out.copy_(logits)
        tokens.copy_(logits.argmax(dim=-1))
        return
    p = cuda_ops._p  # pylint: disable=protected-access
    args = _StepEndArgs(logits.data_ptr(), p(logits_out), tokens.data_ptr(), p(lengths), p(active))
    for i, (dst, src) in enumerate(kept):
        args.kept_dst[i], args.kept_src[i] = dst.data_ptr(), src.data_ptr()
    args.ld, args.B, args.V, args.kept = logits.stride(0), b, v, len(kept)
    rc = _lib().axb_step_end(ctypes.byref(args), cuda_ops._stream())  # pylint: disable=protected-access
    cuda_ops._check(rc, "axb_step_end")  # pylint: disable=protected-access


def advance(counts: torch.Tensor, by) -> torch.Tensor:
    """``counts + by``: tokens seen, per sequence.  In a captured step a link of its chain of kernels (the operator behind
    the last layer and the order it forces cost 4 us of a step, and the output product its head start)."""
    if (cuda_ops.launches_chained() and isinstance(by, torch.Tensor) and counts.dim() == 1
            and _row_vector(counts, counts.shape[0]) and _row_vector(by, counts.shape[0])):
        out = torch.empty_like(counts)
        rc = _lib().axb_add_counts(counts.data_ptr(), by.data_ptr(), out.data_ptr(), counts.numel(),
                                   cuda_ops._stream())  # pylint: disable=protected-access
        cuda_ops._check(rc, "axb_add_counts")  # pylint: disable=protected-access
        return out
    return counts + by


def assert_ids(ok: torch.Tensor) -> None:
    """An assertion on the device, as in torch's embedding: the next synchronisation reports it."""
    torch._assert_async(ok, "token id outside the embedding table")  # pylint: disable=protected-access


def take_tokens(ids: torch.Tensor, tokens: torch.Tensor, low: int, high: int, ok: torch.Tensor) -> None:
    """``tokens.copy_(ids)`` (``tokens``: int64 on the GPU) for ids that have to lie in ``[low, high)``.

    Ids in host memory raise ``IndexError`` before anything is launched.  Of ids on the GPU ``ok`` (a bool) tells whether
    all do; the others become 0."""
    if not ids.is_cuda:
        if ids.numel() and not (low <= int(ids.min()) and int(ids.max()) < high):
            raise IndexError(f"token id outside the embedding table: ids go from {low} to {high - 1}")
        tokens.copy_(ids)
        ok.fill_(True)
        return
    if not (ids.dtype == torch.int64 and ids.shape == tokens.shape and ids.is_contiguous() and ids.device == tokens.device):
        tokens.copy_(ids)
        ids = tokens
    rc = _lib().axb_take_tokens(ids.data_ptr(), tokens.data_ptr(), tokens.numel(), low, high, ok.data_ptr(),
                                cuda_ops._stream())  # pylint: disable=protected-access
    cuda_ops._check(rc, "axb_take_tokens")  # pylint: disable=protected-access


def embed_rows_supported(table: torch.Tensor, ids: torch.Tensor) -> bool:
    return (table.is_cuda and table.dtype == torch.bfloat16 and table.dim() == 2 and table.stride(1) == 1
            and table.shape[1] % 8 == 0 and table.stride(0) % 8 == 0 and table.stride(0) >= table.shape[1]
            and table.data_ptr() % 16 == 0 and ids.is_cuda and ids.dtype == torch.int64 and ids.is_contiguous())


def embed_rows(table: torch.Tensor, ids: torch.Tensor, *, wrap: bool = False, lengths: Optional[torch.Tensor] = None,
               max_len: int = 0) -> torch.Tensor:
    """``table[ids]`` (bf16 rows) ``[..., width]``; ``wrap``: negative ids count from the end.  Ids outside the table give
    NaN rows and a status that ``cuda_ops.check_status`` raises.  ``lengths`` (one per id): ``min(lengths + 1, max_len)``
    in the same launch."""
    out = torch.empty((*ids.shape, table.shape[1]), dtype=table.dtype, device=table.device)
    rc = _lib().axb_embed_rows(table.data_ptr(), ids.data_ptr(), out.data_ptr(),
                               cuda_ops._p(lengths), max_len, ids.numel(), table.shape[0],  # pylint: disable=protected-access
                               table.shape[1], table.stride(0), 1 if wrap else 0,
                               cuda_ops.status_word(table.device).data_ptr(), cuda_ops._stream())  # pylint: disable=protected-access
    cuda_ops._check(rc, "axb_embed_rows")  # pylint: disable=protected-access
    return out
