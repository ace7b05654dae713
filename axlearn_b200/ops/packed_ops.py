"""Ragged prompts without their padding: the live tokens of all sequences, one after the other.

A batch of right-padded prompts ``[B, T]`` of which a third is padding pays a third of its products, norms and activations
for rows that nobody reads.  Between the embedding and the output norm everything but the sequence mixers works row by row,
so there the rows are the live tokens alone, ``[1, rows, D]``; the mixers' kernels take the row at which each sequence
begins and let nothing of a neighbour into a sequence, be it NaN.  Served batches of prompts and 16 steps, one B200, twenty
sets of lengths in turn, median and largest us, padded / packed: Sagisun, 1B widths, 8 prompts of up to 1500 tokens, 6841 6868
/ 5885 6185; Zukitar, 16 of up to 1000, 11325 11670 / 9794 10027.
"""

from __future__ import annotations

import contextlib
import threading
from typing import Optional

import torch

from axlearn_b200.ops import cuda_ops

Tensor = torch.Tensor

# Rows padded / packed of a batch decide: where the lengths are known on the GPU alone, the host has to wait for them,
# which ends what it had launched ahead (up to 0.6 ms; full prompts in four chunks of 16 x 400 with lengths from the host,
# waited for or not, 9.05 / 8.81 ms).  Batches with three eighths of padding and 16 steps, padded / packed us (Sagisun,
# Zukitar): 8 x 400 4197 / 4321, 6353 / 6538; 32 x 128 4933 / 4882, 8590 / 8566; 16 x 400 5187 / 5048, 8169 / 7950;
# 8 x 1000 5700 / 5259, 7979 / 7516.
MIN_TOKENS = 5000
MIN_PADDING = 0.1  # as a share of the rows


_known = threading.local()


@contextlib.contextmanager
def lengths_known(live: Tensor, lengths: Optional[Tensor]):
    """Where the calling thread packs prompts of ``live [B]`` (int32, on the GPU) inside, they have these ``lengths [B]`` (the
    same in host memory; None: nobody knows them there), so that it does not wait for the GPU to tell them.  Lengths that a
    model has made of them are others, and are waited for."""
    before = getattr(_known, "live", None), getattr(_known, "lengths", None)
    _known.live, _known.lengths = live, lengths
    try:
        yield
    finally:
        _known.live, _known.lengths = before


def _known_lengths(live: Tensor) -> Optional[Tensor]:
    lengths = getattr(_known, "lengths", None)
    if lengths is None:
        return None
    given = _known.live
    same = (live.data_ptr(), live.shape, live.stride(), live.dtype) == (
        given.data_ptr(), given.shape, given.stride(), given.dtype)
    return lengths if same else None


class PackedRows:
    """Where the live tokens of a padded batch lie.  ``first``, ``live``: int32 ``[B]``, the first row of a sequence and how
    many it has; ``rows`` of all; ``max_len``: T of the padded batch; ``some_empty``: a sequence has no token, so no row that
    could stand for it.  Waits for ``live`` (int32, on the GPU) unless ``known``, the same in host memory, is given."""

    def __init__(self, live: Tensor, max_len: int, known: Optional[Tensor] = None):
        b = live.shape[0]
        self.max_len = max_len
        made = torch.empty(2 * b + 2 + 2 * b * max_len, dtype=torch.int32, device=live.device)
        self.first, self.live, total, self._rows_of, self._row_of = made.split([b, b, 2, b * max_len, b * max_len])
        cuda_ops._check(cuda_ops.lib().axb_pack_rows(  # pylint: disable=protected-access
            live.data_ptr(), b, max_len, self.first.data_ptr(), self.live.data_ptr(), total.data_ptr(),
            self._rows_of.data_ptr(), self._row_of.data_ptr(), cuda_ops._stream()), "axb_pack_rows")  # pylint: disable=protected-access
        if known is None:
            self.rows, some_empty = total.tolist()
            self.some_empty = bool(some_empty)
        else:
            self.rows, self.some_empty = _live_rows(known, max_len), int(known.min()) <= 0

    def pack(self, x: Tensor) -> Tensor:
        """``[B, T, D] -> [1, rows, D]``."""
        return x.reshape(-1, x.shape[-1]).index_select(0, self._rows_of[:self.rows])[None]

    def unpack(self, x: Tensor) -> Tensor:
        """``[1, rows, D] -> [B, T, D]``, zeros for padding."""
        x = x.contiguous()
        out = torch.empty((self.live.shape[0], self.max_len, x.shape[-1]), dtype=x.dtype, device=x.device)
        cuda_ops._check(cuda_ops.lib().axb_unpack_rows(  # pylint: disable=protected-access
            x.data_ptr(), out.data_ptr(), self._row_of.data_ptr(), self._row_of.numel(), x.shape[-1] * x.element_size(),
            cuda_ops._stream()), "axb_unpack_rows")  # pylint: disable=protected-access
        return out


def _live_rows(lengths: Tensor, max_len: int) -> int:
    return int(lengths.clamp(0, max_len).sum())


def pack_prompts(live: Tensor, max_len: int) -> Optional[PackedRows]:
    """The packing of right-padded prompts of ``live [B]`` tokens, None where it does not pay.  Waits for ``live`` unless its
    values are known (``lengths_known``)."""
    b = live.shape[0]
    if not 2 <= b <= 65535 or b * max_len < MIN_TOKENS or b * max_len >= 1 << 31:
        return None

    def pays(rows):
        return 128 <= rows <= (1 - MIN_PADDING) * b * max_len

    known = _known_lengths(live)
    if known is not None and not pays(_live_rows(known, max_len)):
        return None
    packed = PackedRows(live.to(torch.int32).contiguous(), max_len, known)
    return packed if pays(packed.rows) else None
