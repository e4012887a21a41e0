"""Device plumbing: the CUDA device, the current stream, table uploads and scratch.

PyTorch only provides memory, streams and host<->device copies here; every
computation on symmetric-tensor data goes through the C ABI in ``_native``.
"""

import os

# Sector buffers range from tens of KB to ~11 GB (chi = 256 SU(2) CTMRG) and are
# allocated and freed every move; with the caching allocator's fixed segments
# that pattern fragments until a large request fails with most of the reserved
# memory unused.  Growable segments are the default here unless the process
# configured the allocator itself; the setting only takes effect when this
# module is imported before torch's first CUDA allocation.
os.environ.setdefault("PYTORCH_CUDA_ALLOC_CONF", "expandable_segments:True")

import numpy as np  # noqa: E402
import torch  # noqa: E402

from . import _native  # noqa: E402

_available = []
_devices = {}


def device():
    """The CUDA device tensors live on.  Raises when CUDA is unavailable: there is
    no CPU fallback for any symmetric-tensor operation."""
    if not _available:
        if not torch.cuda.is_available():
            msg = "frostspin_b200 needs a CUDA device (B200, sm_100a); none is available"
            raise RuntimeError(msg)
        _available.append(True)
    index = torch.cuda.current_device()
    d = _devices.get(index)
    if d is None:
        d = _devices[index] = torch.device("cuda", index)
    return d


def stream():
    """cudaStream_t of torch's current stream, as an integer handle."""
    return torch._C._cuda_getCurrentRawStream(torch.cuda.current_device())


def ptr(t):
    return t.data_ptr() if t is not None and t.numel() > 0 else None


def upload(arr):
    """Copy a numpy array (any dtype, structured included) into a new uint8 device
    buffer.  The bytes go through pinned host memory (torch's caching host
    allocator keeps that block alive until the copy has run), so the copy is
    asynchronous and the host does not wait for the stream."""
    a = np.ascontiguousarray(arr)
    raw = torch.from_numpy(a.view(np.uint8).reshape(-1))
    if raw.numel() == 0:
        return torch.empty(0, dtype=torch.uint8, device=device())
    return raw.pin_memory().to(device(), non_blocking=True)


def upload_f64(arr):
    a = np.ascontiguousarray(arr, dtype=np.float64)
    return torch.from_numpy(a).pin_memory().to(device(), non_blocking=True)


class KeptTables:
    """Device tables uploaded once and used by later calls, whatever their stream.
    The first call on a stream other than the upload's waits for the upload and
    marks the tables as used there, so that an evicted plan's memory is not
    handed on while that stream still reads it.  Inside a graph capture new
    tables are not kept (their upload runs with the graph) and kept ones are
    not waited for (an event from outside the capture cannot be)."""

    __slots__ = ("_kept",)

    def __init__(self):
        self._kept = None

    def get(self, make, s):
        """The tables of make() (nested tuples of tensors and None), for launches on
        the current stream s."""
        if self._kept is None:
            tables = make()
            if not torch.cuda.is_current_stream_capturing():
                ready = torch.cuda.Event()
                ready.record()
                self._kept = (tables, ready, {s})
            return tables
        tables, ready, joined = self._kept
        if s not in joined and not torch.cuda.is_current_stream_capturing():
            current = torch.cuda.current_stream()
            current.wait_event(ready)
            _mark_used(tables, current)
            joined.add(s)
        return tables


def _mark_used(tables, on):
    if isinstance(tables, tuple):
        for t in tables:
            _mark_used(t, on)
    elif tables is not None:
        tables.record_stream(on)


def reduction_buffer(device):
    """Memory of one two-pass reduction: its result, then fs_reduce_partials()
    doubles.  Allocated per call, so that reductions on several streams or
    threads never share partial sums (torch's allocator orders reuse by stream)."""
    return torch.empty(1 + _native.reduce_partials(), dtype=torch.float64, device=device)


def empty_f64(n):
    return torch.empty(int(n), dtype=torch.float64, device=device())


def zeros_f64(n):
    return torch.zeros(int(n), dtype=torch.float64, device=device())
