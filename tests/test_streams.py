"""Calls of several streams in flight at once: nothing a launch still reads or
writes is shared with, or unready for, a launch on another stream."""

import numpy as np
import pytest
import torch

from frostspin_b200 import _native, linalg
from frostspin_b200 import device as dev
from frostspin_b200.symmetric_tensor import abelian_symmetric_tensor as ab
from frostspin_b200.symmetric_tensor import lie_group_symmetric_tensor as lie
from frostspin_b200.symmetric_tensor import o2_symmetric_tensor as o2


def _clear_plans():
    for cache in (ab._PLAN_CACHE, lie._MAP_CACHE, o2._PLAN_CACHE):
        cache.clear()


@pytest.fixture
def launches(monkeypatch):
    """The C ABI calls of host-memory tensors, recorded instead of made.  The kernel's
    limits are asked for before, and no plan with host tables outlives the test."""
    calls = []
    lie._fused_limits()
    _clear_plans()
    monkeypatch.setattr(dev, "device", lambda: torch.device("cpu"))
    monkeypatch.setattr(dev, "stream", lambda: 0)
    monkeypatch.setattr(dev, "upload", lambda a: torch.from_numpy(
        np.ascontiguousarray(a).view(np.uint8).reshape(-1).copy()))
    monkeypatch.setattr(_native, "call", lambda name, *args, entry=None: calls.append((name, args)))
    yield calls
    _clear_plans()


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


class _FakeEvent:
    def record(self):
        self.upload_stream = dev.stream()


class _FakeStream:
    def __init__(self, log):
        self.log = log

    def wait_event(self, event):
        self.log.append(("wait", dev.stream(), event.upload_stream))


def _tensor(cls, leg):
    rng = np.random.default_rng(3)
    sig = np.array([False, False, True, True])
    irreps, shapes = cls.get_block_sizes((leg, leg), (leg, leg), sig)
    flat = torch.from_numpy(rng.standard_normal(int((shapes[:, 0] * shapes[:, 1]).sum())))
    return cls.from_flat((leg, leg), (leg, leg), flat, irreps, sig)


LEGS = {"U1": np.array([-1, -1, 0, 0, 0, 1, 2], dtype=np.int8), "SU2": np.array([[3, 2], [1, 3]]),
        "O2": np.array([[1, 3, 2], [-1, 0, 1]])}


def _class(sym):
    import frostspin_b200 as fb

    return {"U1": fb.U1SymmetricTensor, "SU2": fb.SU2SymmetricTensor, "O2": fb.O2SymmetricTensor}[sym]


@pytest.mark.parametrize("sym", list(LEGS))
def test_kept_tables_are_awaited_on_other_streams(sym, launches, monkeypatch):
    """A plan's tables, uploaded on stream 1: the first launch on stream 2 comes
    after a wait for the upload and with every table marked as used there."""
    current, marks = [1], []
    monkeypatch.setattr(dev, "stream", lambda: current[0])
    monkeypatch.setattr(torch.cuda, "Event", _FakeEvent)
    monkeypatch.setattr(torch.cuda, "current_stream", lambda: _FakeStream(launches))
    monkeypatch.setattr(torch.cuda, "is_current_stream_capturing", lambda: False)
    monkeypatch.setattr(torch.Tensor, "record_stream", lambda t, s: marks.append(t.data_ptr()))
    monkeypatch.setattr(dev, "upload_f64", lambda a: torch.from_numpy(
        np.array(a, dtype=np.float64)))
    t = _tensor(_class(sym), LEGS[sym])

    def permute(stream):
        current[0] = stream
        launches.clear()
        marks.clear()
        t.permute((3, 0), (2, 1))
        return list(launches)

    first = permute(1)
    assert not any(c[0] == "wait" for c in first) and not marks
    again = permute(2)
    assert [c for c in again if c[0] != "wait"] and again[0][0] == "wait"
    assert all(c[1:] == (2, 1) for c in again if c[0] == "wait")
    assert len(marks) >= 2
    # joined once: later calls on either stream wait no more
    for s in (1, 2):
        assert not any(c[0] == "wait" for c in permute(s)) and not marks


@pytest.mark.gpu
def test_plan_uploaded_behind_a_busy_stream():
    """A plan first used on a stream with work queued before its upload, then at
    once on another stream."""
    for sym, leg in LEGS.items():
        t = _tensor(_class(sym), leg)
        want = t.permute((3, 0), (2, 1)).data.clone()
        _clear_plans()
        busy, other = torch.cuda.Stream(), torch.cuda.Stream()
        torch.cuda.synchronize()
        with torch.cuda.stream(busy):
            torch.cuda._sleep(20_000_000)    # about 10 ms, ends by itself
            a = t.permute((3, 0), (2, 1)).data
        with torch.cuda.stream(other):
            b = t.permute((3, 0), (2, 1)).data
        torch.cuda.synchronize()
        assert torch.equal(a, want) and torch.equal(b, want)


@pytest.mark.gpu
def test_kept_tables_under_capture():
    """A warmed-up permute captured on a side stream and replayed."""
    for sym, leg in LEGS.items():
        t = _tensor(_class(sym), leg)
        want = t.permute((3, 0), (2, 1)).data.clone()
        torch.cuda.synchronize()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            out = t.permute((3, 0), (2, 1)).data
        out.zero_()
        graph.replay()
        torch.cuda.synchronize()
        assert torch.equal(out, want)


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
