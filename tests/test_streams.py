"""Calls of several streams in flight at once: nothing a launch still reads or
writes is shared with, or unready for, a launch on another stream."""

import numpy as np
import pytest
import torch

from frostspin_b200 import _native, linalg
from frostspin_b200 import device as dev


@pytest.fixture
def launches(monkeypatch):
    """The C ABI calls of host-memory tensors, recorded instead of made."""
    calls = []
    monkeypatch.setattr(dev, "device", lambda: torch.device("cpu"))
    monkeypatch.setattr(dev, "stream", lambda: 0)
    monkeypatch.setattr(dev, "upload", lambda a: torch.from_numpy(
        np.ascontiguousarray(a).view(np.uint8).reshape(-1).copy()))
    monkeypatch.setattr(_native, "call", lambda name, *args, entry=None: calls.append((name, args)))
    return calls


@pytest.mark.parametrize("n", [1, 200])   # tables by value and in device memory
def test_reductions_in_flight_share_no_partial_sums(n, launches):
    x = torch.zeros(n, dtype=torch.float64)
    off = np.arange(n)
    one = np.ones(n, dtype=np.int64)
    pairs = [(i, i, 1, 1, False, False, 1.0) for i in range(n)]
    results = [linalg.weighted_reduce(x, off, one, one, squares=True),
               linalg.weighted_reduce(x, off, one, one, squares=False),
               linalg.pair_contract(x, x, pairs), linalg.pair_contract(x, x, pairs)]
    spans = []
    for (_, args), r in zip(launches, results, strict=True):
        *_, part, n_part, out, _ = args
        assert n_part >= _native.reduce_partials()
        assert out == r.data_ptr() and r.dim() == 0
        spans += [(part, part + 8 * n_part), (out, out + 8)]
    spans.sort()
    assert all(a[1] <= b[0] for a, b in zip(spans, spans[1:], strict=False))


@pytest.mark.gpu
def test_reductions_on_two_streams():
    """Sums over different data, launched in turn on two streams."""
    rng = np.random.default_rng(1)
    lengths = np.array([900_001, 33, 250_000])
    off = np.concatenate([[0], np.cumsum(lengths)[:-1]])
    data = [torch.from_numpy(rng.standard_normal(int(lengths.sum()))).cuda() for _ in range(2)]
    pairs = [(int(off[0]), int(off[0]), 900_001, 1, False, False, 1.0)]

    def sums(x):
        return [linalg.weighted_reduce(x, off, lengths, [1.0, 3.0, 5.0], squares=True),
                linalg.pair_contract(x, x, pairs)]

    want = [[float(v) for v in sums(x)] for x in data]
    streams = [torch.cuda.Stream() for _ in range(2)]
    torch.cuda.synchronize()
    got = [[], []]
    for _ in range(100):
        for i, s in enumerate(streams):
            with torch.cuda.stream(s):
                got[i].append(sums(data[i]))
    torch.cuda.synchronize()
    for i in range(2):
        assert all([float(v) for v in r] == want[i] for r in got[i])
