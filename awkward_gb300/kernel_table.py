"""Kernel table over libawkward_gb300 with awkward's key scheme and error protocol.

This mirrors the part of awkward's CUDA backend that sits on the accelerated
path, for callers holding torch CUDA tensors (the cupy adapter in
``cupy_adapter.py`` installs the same entry points into awkward itself):

* ``backend[(family, *dtypes)]`` returns a kernel, keyed exactly like
  ``CupyBackend.__getitem__`` (src/awkward/_backends/cupy.py:30-57): the
  family name followed by the numpy dtype of every pointer argument in spec
  order (dev/generate-kernel-signatures.py:225-236, 419-422);
* calling the kernel with the spec's arguments launches it asynchronously on
  the current torch stream, appending ``(invocation_index, err_code)`` like
  ``CupyKernel.__call__`` (src/awkward/_kernels.py:185-232);
* ``backend.synchronize()`` waits for the stream and raises
  ``ValueError("<message> in compiled CUDA code (<family>)")`` for the first
  failing invocation, like ``synchronize_cuda``
  (src/awkward/_connect/cuda/__init__.py:257-294).

Arguments: List[T] -> a contiguous CUDA tensor of dtype T (bool as
torch.bool); List[List[T]] -> a sequence of such tensors; scalars -> Python
numbers.

Fault injection (host side, for testing callers' error handling): with
``AWKWARD_GB300_FAULT="<specialization or family>:<code>"`` every call of a
matching kernel still launches, and then the stream's error word records
``invocation_index * 256 + code`` exactly as a failing kernel would, so the
next ``synchronize()`` raises that code's message (code 32: the library's
"bounded wait gave up").  No kernel is made to fail on the GPU.
"""

from __future__ import annotations

import collections
import os
import threading

import numpy as np
import torch

from . import _abi
from ._messages import TIMEOUT_MESSAGE, messages
from ._signatures import SIGNATURES

ERROR_BITS = 8
NO_ERROR = (1 << 64) - 1
MAX_PENDING_INVOCATIONS = 8192

NP_OF_C = {
    "bool": np.bool_, "int8_t": np.int8, "uint8_t": np.uint8, "int16_t": np.int16,
    "uint16_t": np.uint16, "int32_t": np.int32, "uint32_t": np.uint32,
    "int64_t": np.int64, "uint64_t": np.uint64, "float": np.float32, "double": np.float64,
}
TORCH_OF_C = {
    "bool": torch.bool, "int8_t": torch.int8, "uint8_t": torch.uint8, "int16_t": torch.int16,
    "uint16_t": torch.uint16, "int32_t": torch.int32, "uint32_t": torch.uint32,
    "int64_t": torch.int64, "uint64_t": torch.uint64, "float": torch.float32,
    "double": torch.float64,
}


def kernel_key(name):
    """(family, *numpy dtype types of the pointer arguments) of a specialization."""
    rec = SIGNATURES[name]
    return (rec["family"],) + tuple(NP_OF_C[a[1]] for a in rec["args"] if a[3] > 0)


FAULT_ENV = "AWKWARD_GB300_FAULT"


def injected_fault(name, family, env=None):
    """The error code AWKWARD_GB300_FAULT forces on kernel ``name``, or None.

    The variable holds ``<specialization or family>:<code>`` with code in
    0..255; anything else is ignored.
    """
    spec = (os.environ if env is None else env).get(FAULT_ENV, "")
    target, sep, code = spec.rpartition(":")
    if not sep or target not in (name, family):
        return None
    try:
        c = int(code)
    except ValueError:
        return None
    return c if 0 <= c < (1 << ERROR_BITS) else None


class _Invocation:
    __slots__ = ("name", "keepalive")

    def __init__(self, name, keepalive):
        self.name = name
        self.keepalive = keepalive


class _StreamContext:
    """Error word and pending invocations of one stream, for all threads that use it.

    Invocations are numbered on through every synchronisation: calls[i] is number
    first + i.  A number is given out and its kernel launched under the lock, and a
    call stays in the list until the word has been read behind it.  So an error of
    any thread's call finds its name, whoever reads the word."""

    def __init__(self, device):
        self.err = torch.full((1,), -1, dtype=torch.int64, device=device)  # NO_ERROR
        self.address = self.err.data_ptr()
        self.lock = threading.Lock()
        self.first = 0
        self.calls = []
        # (the word of a context made during a capture is filled by the graph's replays)
        self.captured = torch.cuda.is_current_stream_capturing()

    def record_error(self, invocation, code, stream):
        """Lower the error word to invocation*256 + code on `stream` (as atomicMin does)."""
        word = invocation * (1 << ERROR_BITS) + code
        with torch.cuda.stream(stream):
            w = torch.full_like(self.err, word)
            self.err.copy_(torch.where((self.err < 0) | (self.err > w), w, self.err))


# The current stream of a device as a raw cudaStream_t (torch.cuda.current_stream
# builds a Stream object, which costs more than a launch).
raw_stream = torch._C._cuda_getCurrentRawStream


# Device arrays of row pointers (the int64_t** arguments), by device and
# addresses: uploading one is a blocking host-to-device copy, so a repeated
# call with the same rows reuses the array (it holds nothing but those
# addresses, so a cached array is right whatever tensors now live there).
_PTR_ARRAYS: collections.OrderedDict = collections.OrderedDict()
_PTR_ARRAYS_MAX = 256


def _pointer_array(dev, addresses):
    key = (dev.index, addresses)
    arr = _PTR_ARRAYS.get(key)
    if arr is None:
        arr = torch.tensor(list(addresses) or [0], dtype=torch.int64, device=dev)
        _PTR_ARRAYS[key] = arr
        if len(_PTR_ARRAYS) > _PTR_ARRAYS_MAX:
            _PTR_ARRAYS.popitem(last=False)
    else:
        _PTR_ARRAYS.move_to_end(key)
    return arr


class GB300Kernel:
    """One specialization, callable with the spec's arguments."""

    def __init__(self, backend, name):
        self.backend = backend
        self.name = name
        self.family = SIGNATURES[name]["family"]
        self.args = SIGNATURES[name]["args"]
        self.dir = [a[2] for a in self.args]
        self.is_ptr = [a[3] > 0 for a in self.args]
        # what a call checks, worked out once: pointer depth, dtype, name
        self._plan = [(a[3], TORCH_OF_C[a[1]], a[0]) for a in self.args]
        self._f = _abi.cfunc(name)

    def __repr__(self):
        return f"<GB300Kernel {self.name}>"

    def _rows(self, an, dtype, v, index):
        """(pointer array, rows, device index) of a list-of-lists argument."""
        rows = list(v)
        for t in rows:
            if not isinstance(t, torch.Tensor) or not t.is_cuda or t.dtype != dtype:
                raise TypeError(f"{self.name}: rows of {an} must be CUDA {dtype} tensors")
            index = t.get_device()
        dev = torch.device("cuda", torch.cuda.current_device() if index < 0 else index)
        return _pointer_array(dev, tuple(t.data_ptr() for t in rows)), rows, index

    def __call__(self, *args):
        if len(args) != len(self._plan):
            raise ValueError(f"{self.name}: takes {len(self._plan)} arguments, not {len(args)}")
        cargs = []
        keep = []
        index = -1
        for (depth, dtype, an), v in zip(self._plan, args):
            if depth == 0:
                cargs.append(v.item() if hasattr(v, "item") else v)
            elif depth == 1:
                if not isinstance(v, torch.Tensor) or not v.is_cuda:
                    raise TypeError(f"{self.name}: argument {an} must be a CUDA tensor")
                if v.dtype is not dtype:
                    raise TypeError(f"{self.name}: argument {an} must have dtype "
                                    f"{dtype}, not {v.dtype}")
                if not v.is_contiguous():
                    raise ValueError(f"{self.name}: argument {an} must be contiguous")
                index = v.get_device()
                cargs.append(v.data_ptr())
                keep.append(v)
            else:
                ptrs, rows, index = self._rows(an, dtype, v, index)
                keep.extend(rows)
                keep.append(ptrs)
                cargs.append(ptrs.data_ptr())
        if index < 0:
            index = torch.cuda.current_device()
        stream = raw_stream(index)
        ctx = self.backend._context(index, stream)
        if len(ctx.calls) >= MAX_PENDING_INVOCATIONS:
            self.backend.synchronize(torch.cuda.current_stream(index))
            ctx = self.backend._context(index, stream)
        fault = injected_fault(self.name, self.family) if FAULT_ENV in os.environ else None
        call = _Invocation(self.family, keep)
        with ctx.lock:
            calls = ctx.calls
            number = ctx.first + len(calls)
            calls.append(call)
            rc = self._f(*cargs, number, ctx.address, stream)
            if fault is not None and rc == 0:
                ctx.record_error(number, fault, torch.cuda.current_stream(index))
        if rc != 0:
            raise RuntimeError(f"{self.name}: CUDA launch failed with cudaError {rc}")


class GB300Backend:
    """Kernel table ``backend[(family, *dtypes)]`` over libawkward_gb300."""

    def __init__(self):
        self._by_key = {kernel_key(n): n for n in SIGNATURES}
        self._kernels = {}
        self._contexts = {}

    def keys(self):
        return list(self._by_key)

    def __contains__(self, key):
        return self._norm(key) in self._by_key

    @staticmethod
    def _norm(key):
        return (key[0],) + tuple(np.dtype(k).type for k in key[1:])

    def __getitem__(self, key):
        k = self._norm(key)
        name = self._by_key.get(k)
        if name is None:
            raise KeyError(f"no GB300 kernel for {key}")
        kern = self._kernels.get(name)
        if kern is None:
            kern = self._kernels[name] = GB300Kernel(self, name)
        return kern

    def by_name(self, name):
        return self[kernel_key(name)]

    def _context(self, index, stream):
        """The context of raw stream `stream` of device `index`."""
        ctx = self._contexts.get((index, stream))
        if ctx is None:
            ctx = self._contexts.setdefault((index, stream),
                                            _StreamContext(torch.device("cuda", index)))
        return ctx

    def selftest_lookback_timeout(self, spin_limit=1000):
        """Launch the look-back self-test (awkward_gb300_selftest_lookback_timeout)
        on the current stream as one more invocation: its wait on a tile that
        never publishes runs out after `spin_limit` polls, so the next
        synchronize() raises the "bounded wait gave up" ValueError."""
        index = torch.cuda.current_device()
        stream = raw_stream(index)
        name = "awkward_gb300_selftest_lookback_timeout"
        ctx = self._context(index, stream)
        with ctx.lock:
            number = ctx.first + len(ctx.calls)
            ctx.calls.append(_Invocation(name, []))
            rc = _abi.ext_cfunc(name)(int(spin_limit), number, ctx.address, stream)
        if rc != 0:
            raise RuntimeError(f"look-back self-test: CUDA launch failed with cudaError {rc}")

    def synchronize(self, stream=None):
        """Wait for the stream; raise ValueError for the first failed invocation."""
        if stream is None:
            index = torch.cuda.current_device()
            raw, current = raw_stream(index), True
        else:
            index, raw = stream.device.index, stream.cuda_stream
            current = stream == torch.cuda.current_stream()
        ctx = self._contexts.get((index, raw))
        if ctx is None:
            (stream or torch.cuda.current_stream()).synchronize()
            return
        with ctx.lock:  # (all calls before this number are on the stream)
            launched = ctx.first + len(ctx.calls)
        # reading the word waits for the current stream; without an error the
        # word is as good as new and the context stays
        if not current:
            stream.synchronize()
        word = int(ctx.err.item()) & NO_ERROR
        inv = None
        with ctx.lock:
            if word != NO_ERROR:  # no launch until the word is clear again
                stream = stream or torch.cuda.current_stream()
                stream.synchronize()
                word = int(ctx.err.item()) & NO_ERROR
                if word != NO_ERROR:  # (else another thread has raised it meanwhile)
                    at = (word >> ERROR_BITS) - ctx.first
                    inv = ctx.calls[at] if 0 <= at < len(ctx.calls) else None
                    with torch.cuda.stream(stream):
                        ctx.err.fill_(-1)
            over = launched - ctx.first
            if over > 0:
                del ctx.calls[:over]
                ctx.first = launched
        if ctx.captured:
            self._contexts.pop((index, raw), None)
        if word == NO_ERROR:
            return
        code = word & ((1 << ERROR_BITS) - 1)
        if inv is None:  # a call that a graph has launched again
            what = TIMEOUT_MESSAGE if code == TIMEOUT_CODE else f"error {code}"
            raise ValueError(f"{what} in compiled CUDA code (a replayed call)")
        raise ValueError(f"{messages(inv.name)[code]} in compiled CUDA code ({inv.name})")


_BACKEND = None


def backend():
    """The process-wide kernel table."""
    global _BACKEND
    if _BACKEND is None:
        _BACKEND = GB300Backend()
    return _BACKEND
