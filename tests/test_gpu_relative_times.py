"""Forms of one call that may differ in speed by a small factor only, timed in turn
on the device behind a buffer write that clears the L2 cache: the best of several
launches each, with margins far above the spread of the timings."""

import numpy as np
import pytest
import torch

from frostspin_b200 import _native, linalg

pytestmark = pytest.mark.gpu


def _best_us(*calls, reps=7):
    """Best device time of each call, in microseconds."""
    flush = torch.empty(1 << 26, dtype=torch.float64, device="cuda")
    best = [float("inf")] * len(calls)
    for r in range(reps + 1):
        for i, f in enumerate(calls):
            for _ in range(8):      # long enough to hide the host's work of the call
                flush.zero_()
            s, e = (torch.cuda.Event(enable_timing=True) for _ in range(2))
            s.record()
            f()
            e.record()
            torch.cuda.synchronize()
            if r:
                best[i] = min(best[i], s.elapsed_time(e) * 1e3)
    return best


@pytest.mark.parametrize("shape", [(1, 4_000_000), (4_000_000, 1), (3, 1_000_001), (900_001, 7)])
def test_thin_crossed_contraction(shape):
    """A thin block against one of the other storage order: within twice the time
    of the same block against one of its own (6 times with 64 x 64 tiles)."""
    m, n = shape
    x, y = (torch.randn(m * n, dtype=torch.float64, device="cuda") for _ in range(2))
    same, crossed = _best_us(
        lambda: linalg.pair_contract(x, y, [(0, 0, m, n, False, True, 1.0)]),
        lambda: linalg.pair_contract(x, y, [(0, 0, m, n, False, False, 1.0)]))
    assert crossed <= 2 * same, (crossed, same)


@pytest.mark.parametrize("left", [False, True])
@pytest.mark.parametrize("shape", [(1, 4_000_000), (4_000_000, 1), (3, 1_000_001), (900_001, 4)])
def test_thin_transposed_diagonal_product(shape, left):
    """The same for the product of a transposed block with a diagonal (up to 15
    times with 64 x 64 tiles)."""
    m, n = shape
    x = torch.randn(m * n, dtype=torch.float64, device="cuda")
    d = torch.randn(max(m, n), dtype=torch.float64, device="cuda")
    same, turned = _best_us(
        lambda: linalg.diag_mul(x, d, [(0, 0, 0, m, n, False, left)], m * n),
        lambda: linalg.diag_mul(x, d, [(0, 0, 0, m, n, True, left)], m * n))
    assert turned <= 2 * same, (turned, same)


def _sectors(shapes):
    arr = np.zeros(len(shapes), dtype=_native.GEMM_PROBLEM_DTYPE)
    keep = []
    for i, (M, N, K) in enumerate(shapes):
        a, b, c = (torch.randn(n, dtype=torch.float64, device="cuda") for n in (M * K, K * N, M * N))
        keep += [a, b, c]
        arr[i] = (a.data_ptr(), b.data_ptr(), c.data_ptr(), K, N, N, M, N, K, 0, 0, 0, 1.0, 0.0)
    return arr, keep


@pytest.mark.parametrize("shapes", [
    [(4, 60000, 3), (1, 10000, 1), (2, 30000, 1), (3, 50000, 2)] * 2,
    [(8, 10000, 8)] * 30,
    [(1 + i % 7, 10000, 1 + i % 5) for i in range(40)],
])
def test_wide_gemm_shares(shapes, monkeypatch):
    """Many sectors and very uneven ones: the wide kernel is faster than the
    streaming one (0.45 to 0.54 of its time; 1.0 to 1.4 with uneven shares)."""
    arr, keep = _sectors(shapes)
    assert int(arr["N"].sum()) >= 3e5

    def launch(unit):
        def f():
            monkeypatch.setattr(linalg, "_WIDE_COLUMNS", unit)
            linalg._launch_dgemm(arr)
        return f

    streaming, wide = _best_us(launch(1 << 60), launch(0))
    assert wide <= 0.8 * streaming, (wide, streaming)
    del keep


@pytest.mark.parametrize("n", [96, 256])
def test_many_blocks(n):
    """A diagonal product and a contraction of many small blocks: within 4 times
    the same over one block of their total size (walking up to a share took 6 to 9
    times)."""
    m = k = 40
    x, y = (torch.randn(n * m * k, dtype=torch.float64, device="cuda") for _ in range(2))
    d = torch.randn(n * m * k, dtype=torch.float64, device="cuda")
    size = m * k
    one, many = _best_us(
        lambda: linalg.diag_mul(x, d, [(0, 0, 0, n * m, k, False, False)], x.numel()),
        lambda: linalg.diag_mul(x, d, [(i * size, i * size, i * k, m, k, False, False)
                                       for i in range(n)], x.numel()))
    assert many <= 4 * one, (many, one)
    one, many = _best_us(
        lambda: linalg.pair_contract(x, y, [(0, 0, n * m, k, False, True, 1.0)]),
        lambda: linalg.pair_contract(x, y, [(i * size, i * size, m, k, False, True, 1.0)
                                            for i in range(n)]))
    assert many <= 4 * one, (many, one)


def test_sum_of_tiny_blocks():
    """60 blocks of 2 elements: within twice the time of one block of 120 (3.5 times
    while one CTA walked them all)."""
    x = torch.randn(120, dtype=torch.float64, device="cuda")
    one, many = _best_us(
        lambda: [linalg.weighted_reduce(x, [0], [120], [1.0], squares=True) for _ in range(10)],
        lambda: [linalg.weighted_reduce(x, 2 * np.arange(60), [2] * 60, [1.0] * 60, squares=True)
                 for _ in range(10)])
    assert many <= 2 * one, (many, one)
