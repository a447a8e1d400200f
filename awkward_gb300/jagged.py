"""Jagged getitem on (offsets, content) pairs, following awkward's own call sequence.

Host-side mirror of the parts of awkward's getitem path on this library's
kernels, for CUDA tensors:

* ``getitem_jagged_mask``  -- ``array[mask]`` with a jagged boolean mask of the
  same offsets: the mask becomes a jagged local index
  (src/awkward/_slicing.py:476-530), which is applied with
  ``awkward_ListArray_getitem_jagged_apply`` (src/awkward/contents/listarray.py:573-616)
  and the content carried (``NumpyArray._carry``);
* ``getitem_jagged_index`` -- ``array[idx]`` with a jagged int64 index
  (same apply + carry); ``index_select`` does it in one kernel (the apply
  with the content gathered at each carry), ``mask_select`` does
  ``array[mask]`` without the local index;
* ``getitem_inner_range``  -- ``array[..., start:stop:step]`` on the innermost
  list level of a two-level ListOffsetArray, in one kernel (``range_select``);
  ``inner_range`` and ``take`` are awkward's own steps:
  ``awkward_ListArray_getitem_next_range_carrylength``, the carry allocation,
  ``awkward_ListArray_getitem_next_range`` and the carry
  (src/awkward/contents/listarray.py:795-862).

awkward's own steps read sizes that depend on data back from the device where
awkward reads them (the carry length, the total of true mask entries); the
one-call functions write into a buffer that is large enough and read size and
error back with one wait at their end (see _WHOLE_SOURCE, _WHOLE_CONTENT).
Errors follow awkward's protocol and surface as ``ValueError``.
"""

from __future__ import annotations

import os
import threading

import numpy as np
import torch

from . import _abi
from ._messages import TIMEOUT_MESSAGE, messages
from .kernel_table import FAULT_ENV, backend, raw_stream

SLICE_NONE = np.iinfo(np.int64).max  # awkward's kSliceNone


# Up to this many bytes a result whose size depends on the data is written into
# a buffer as long as its source, so that no size is read first -- if the source
# has no more than _PER_LIST entries a list: a few lists of a large array take a
# buffer of their own span, after one read of it (about 10 us).
_WHOLE_SOURCE = 64 << 20
_PER_LIST = 64

_LOCAL = threading.local()


class _Call:
    """The stream of one call and the thread's error word there.  A call takes the
    word and, when it has read it back and left it clear, puts it by for the next
    call of the thread on that stream; the word of a call that fails before that
    (a launch that is refused, a read during a capture) is not used again."""

    def __init__(self, device):
        self.key = (device.index, raw_stream(device.index))
        self.stream = self.key[1]
        try:
            self.words = _LOCAL.words
        except AttributeError:
            self.words = _LOCAL.words = {}
        self.err = self.words.pop(self.key, None)
        if self.err is None:
            self.err = torch.full((1,), -1, dtype=torch.int64, device=device)
        self.address = self.err.data_ptr()

    def finish(self, what, family, *addresses):
        """The device words at `addresses`; the call's error as ValueError."""
        *got, word = _abi.read_words(self.stream, *addresses, self.address)
        if word != -1:
            self.err.fill_(-1)
        if len(self.words) >= 64:
            self.words.clear()
        self.words[self.key] = self.err
        if word != -1:
            code = word & 255
            msg = messages(family)[code] if family else (TIMEOUT_MESSAGE if code else "index out of range")
            raise ValueError(f"{msg} in compiled CUDA code ({what})")
        return got

    def span(self, offsets, n, source, itemsize):
        """Entries to allocate for elements of the lists' span: their number, or
        `source` (no fewer) when that is small enough."""
        if n <= 0:
            return 0
        if source * itemsize <= _WHOLE_SOURCE and source <= _PER_LIST * n:
            return source
        first, last = _abi.read_words(self.stream, offsets.data_ptr(), offsets.data_ptr() + 8 * n)
        return last - first


def _array(name, t, dtype=None):
    """`t` as the library reads it: a contiguous CUDA tensor, of `dtype` if that is given."""
    if type(t) is torch.Tensor and t.is_cuda and t.dtype is (dtype or t.dtype) and t.is_contiguous():
        return t
    if not isinstance(t, torch.Tensor) or not t.is_cuda:
        raise TypeError(f"{name} must be a CUDA tensor")
    if dtype is not None and t.dtype is not dtype:
        raise TypeError(f"{name} must have dtype {dtype}, not {t.dtype}")
    return t.contiguous()


def _mask(mask):
    """`mask` (bool, or any type of one byte) as contiguous bytes."""
    m = _array("mask", mask)
    if m.element_size() != 1:
        raise TypeError(f"mask must have entries of one byte, not {m.dtype}")
    return m if m.dtype is torch.uint8 else m.view(torch.uint8)


def take(content, carry, check=True):
    """content[carry] (a gather); raises ValueError for a carry outside the content."""
    out = torch.empty(carry.numel(), dtype=content.dtype, device=content.device)
    if check:
        call = _Call(content.device)
        stream, address = call.stream, call.address
    else:
        unread = torch.full((1,), -1, dtype=torch.int64, device=content.device)
        stream, address = raw_stream(content.device.index), unread.data_ptr()
    rc = _abi.ext_cfunc("awkward_gb300_take")(
        out.data_ptr(), content.data_ptr(), content.element_size(), carry.data_ptr(),
        carry.numel(), content.numel(), 0, address, stream)
    if rc != 0:
        raise RuntimeError(f"awkward_gb300_take: cudaError {rc}")
    if check:
        call.finish("take", None)
    return out


def jagged_mask_to_index(offsets, mask):
    """(index offsets, local index) of the true entries of a jagged boolean mask;
    raises ValueError for lists that reach past the mask."""
    offsets, m = _array("offsets", offsets, torch.int64), _mask(mask)
    n = offsets.numel() - 1
    call = _Call(offsets.device)
    tooffsets = torch.empty(n + 1, dtype=torch.int64, device=offsets.device)
    toindex = torch.empty(max(call.span(offsets, n, m.numel(), 8), 1), dtype=torch.int64,
                          device=offsets.device)
    rc = _abi.ext_cfunc("awkward_gb300_jagged_mask_to_index_within")(
        tooffsets.data_ptr(), toindex.data_ptr(), m.data_ptr(), m.numel(), offsets.data_ptr(), n,
        call.address, call.stream)
    if rc != 0:
        raise RuntimeError(f"awkward_gb300_jagged_mask_to_index: cudaError {rc}")
    (k,) = call.finish("awkward_gb300_jagged_mask_to_index", None, tooffsets.data_ptr() + 8 * n)
    return tooffsets, toindex[:k]


def mask_select(offsets, content, mask, with_carry=False):
    """array[mask] at once (awkward_gb300_jagged_mask_select_within): the new
    offsets, the selected content and, with `with_carry`, the carry (each
    selected element's position in the content) -- the same outputs as
    getitem_jagged_mask without its intermediate local index.  Raises
    ValueError for lists that reach past the mask."""
    offsets, m = _array("offsets", offsets, torch.int64), _mask(mask)
    content = _array("content", content)
    n = offsets.numel() - 1
    call = _Call(offsets.device)
    itemsize = content.element_size()
    span = max(call.span(offsets, n, m.numel(), itemsize + (8 if with_carry else 0)), 1)
    tooffsets = torch.empty(n + 1, dtype=torch.int64, device=offsets.device)
    out = torch.empty(span, dtype=content.dtype, device=content.device)
    carry = torch.empty(span, dtype=torch.int64, device=offsets.device) if with_carry else None
    rc = _abi.ext_cfunc("awkward_gb300_jagged_mask_select_within")(
        tooffsets.data_ptr(), out.data_ptr(), carry.data_ptr() if with_carry else None,
        m.data_ptr(), m.numel(), offsets.data_ptr(), content.data_ptr(), itemsize, n, span,
        call.address, call.stream)
    if rc != 0:
        raise RuntimeError(f"awkward_gb300_jagged_mask_select_within: cudaError {rc}")
    (k,) = call.finish("awkward_gb300_jagged_mask_select", None, tooffsets.data_ptr() + 8 * n)
    if with_carry:
        return tooffsets, out[:k], carry[:k]
    return tooffsets, out[:k]


def index_select(offsets, content, index_offsets, index, with_carry=False):
    """array[idx] with a jagged int64 index in one pass
    (awkward_gb300_jagged_index_select): the new offsets, the gathered
    content and, with `with_carry`, the carry -- the same outputs as
    getitem_jagged_index without writing and re-reading the carry.  Errors
    are jagged_apply's, raised as ValueError."""
    offsets = _array("offsets", offsets, torch.int64)
    index_offsets = _array("index_offsets", index_offsets, torch.int64)
    index, content = _array("index", index, torch.int64), _array("content", content)
    n = offsets.numel() - 1
    k = index.numel()
    call = _Call(offsets.device)
    tooffsets = torch.empty(n + 1, dtype=torch.int64, device=offsets.device)
    out = torch.empty(max(k, 1), dtype=content.dtype, device=content.device)
    carry = torch.empty(max(k, 1), dtype=torch.int64, device=offsets.device) if with_carry else None
    # a one-element stand-in keeps the pointers valid when the content is empty
    src = content if content.numel() > 0 else torch.zeros(1, dtype=content.dtype,
                                                          device=content.device)
    rc = _abi.ext_cfunc("awkward_gb300_jagged_index_select")(
        tooffsets.data_ptr(), out.data_ptr(), carry.data_ptr() if with_carry else None,
        index_offsets.data_ptr(), index.data_ptr(), k, offsets.data_ptr(), src.data_ptr(),
        content.element_size(), content.numel(), n, call.address, call.stream)
    if rc != 0:
        raise RuntimeError(f"awkward_gb300_jagged_index_select: cudaError {rc}")
    (m,) = call.finish("awkward_gb300_jagged_index_select", "awkward_ListArray_getitem_jagged_apply",
                       tooffsets.data_ptr() + 8 * max(n, 0))
    if with_carry:
        return tooffsets, out[:m], carry[:m]
    return tooffsets, out[:m]


def jagged_apply(offsets, index_offsets, index, contentlen):
    """(tooffsets, tocarry) of a jagged int index applied to lists with these offsets."""
    be = backend()
    n = offsets.numel() - 1
    tooffsets = torch.empty(n + 1, dtype=torch.int64, device=offsets.device)
    tocarry = torch.empty(max(index.numel(), 1), dtype=torch.int64, device=offsets.device)
    be["awkward_ListArray_getitem_jagged_apply", np.int64, np.int64, np.int64, np.int64,
       np.int64, np.int64, np.int64](
        tooffsets, tocarry, index_offsets[:-1].contiguous(), index_offsets[1:].contiguous(), n,
        index, index.numel(), offsets[:-1].contiguous(), offsets[1:].contiguous(), contentlen)
    be.synchronize()
    return tooffsets, tocarry[: index.numel()]


def getitem_jagged_index(offsets, content, index_offsets, index):
    tooffsets, tocarry = jagged_apply(offsets, index_offsets, index, content.numel())
    return tooffsets, take(content, tocarry)


def getitem_jagged_mask(offsets, content, mask):
    index_offsets, index = jagged_mask_to_index(offsets, mask)
    return getitem_jagged_index(offsets, content, index_offsets, index)


def inner_range(inner_offsets, start=None, stop=None, step=None):
    """(nextoffsets, nextcarry) of [start:stop:step] on every list of one level."""
    be = backend()
    n = inner_offsets.numel() - 1
    st, sp = inner_offsets[:-1].contiguous(), inner_offsets[1:].contiguous()
    a = SLICE_NONE if start is None else start
    b = SLICE_NONE if stop is None else stop
    c = 1 if step is None else step
    carrylength = torch.empty(1, dtype=torch.int64, device=inner_offsets.device)
    be["awkward_ListArray_getitem_next_range_carrylength", np.int64, np.int64, np.int64](
        carrylength, st, sp, n, a, b, c)
    be.synchronize()
    length = int(carrylength.item())
    nextcarry = torch.empty(max(length, 1), dtype=torch.int64, device=inner_offsets.device)
    nextoffsets = torch.empty(n + 1, dtype=torch.int64, device=inner_offsets.device)
    be["awkward_ListArray_getitem_next_range", np.int64, np.int64, np.int64, np.int64](
        nextoffsets, nextcarry, st, sp, n, a, b, c)
    be.synchronize()
    return nextoffsets, nextcarry[:length]


# Up to this many bytes a range selection is written into a buffer as long as the
# content (or the lists' span, when the content has more than _PER_LIST elements a
# list), so that its size need not be counted first.
_WHOLE_CONTENT = 1 << 30


def range_select(inner_offsets, content, start=None, stop=None, step=None):
    """(nextoffsets, selected content) of [start:stop:step] on every list of one
    level in one pass (awkward_gb300_jagged_range_select): inner_range and take
    without writing and re-reading the carry.  Offsets are checked as the kernel
    table checks them (TypeError unless CUDA int64), strided ones made contiguous."""
    inner_offsets = _array("inner_offsets", inner_offsets, torch.int64)
    content = _array("content", content)
    n = inner_offsets.numel() - 1
    bounds = (SLICE_NONE if start is None else start, SLICE_NONE if stop is None else stop,
              1 if step is None else step)
    nextoffsets = torch.empty(n + 1, dtype=torch.int64, device=inner_offsets.device)
    size = content.numel()
    call = _Call(content.device)
    if size > _PER_LIST * n:
        size = min(size, max(call.span(inner_offsets, n, size, content.element_size()), 0))
    out = None
    if size * content.element_size() <= _WHOLE_CONTENT:
        try:
            out = torch.empty(max(size, 1), dtype=content.dtype, device=content.device)
        except torch.cuda.OutOfMemoryError:
            pass
    counted = out is None
    if counted:
        be = backend()
        total = torch.empty(1, dtype=torch.int64, device=inner_offsets.device)
        be["awkward_ListArray_getitem_next_range_carrylength", np.int64, np.int64, np.int64](
            total, inner_offsets[:-1], inner_offsets[1:], n, *bounds)
        be.synchronize()
        size = int(total.item())
    while True:
        if out is None:
            out = torch.empty(max(size, 1), dtype=content.dtype, device=content.device)
        rc = _abi.ext_cfunc("awkward_gb300_jagged_range_select")(
            nextoffsets.data_ptr(), out.data_ptr(), size, inner_offsets.data_ptr(),
            content.data_ptr(), content.element_size(), content.numel(), n, *bounds,
            call.address, call.stream)
        if rc != 0:
            raise RuntimeError(f"awkward_gb300_jagged_range_select: cudaError {rc}")
        (k,) = call.finish("take", None, nextoffsets.data_ptr() + 8 * n)
        if k <= size:
            break
        # overlapping lists: more selected than the content holds
        size, out, call = k, None, _Call(content.device)
    # (a small part of the content does not keep a buffer of all of it)
    return nextoffsets, out[:k] if counted or 2 * k >= size else out[:k].clone()


def getitem_inner_range(outer_offsets, inner_offsets, content, start=None, stop=None, step=None):
    """array[..., start:stop:step] of a two-level ListOffsetArray: the outer offsets
    are unchanged; returns (outer_offsets, new inner offsets, new content).  By
    awkward's own steps where faults are injected into them, and for wider items
    than the library gathers (an empty selection of them needs no gather)."""
    if FAULT_ENV in os.environ or content.element_size() > 8:
        nextoffsets, nextcarry = inner_range(inner_offsets, start, stop, step)
        return outer_offsets, nextoffsets, take(content, nextcarry)
    return (outer_offsets, *range_select(inner_offsets, content, start, stop, step))
