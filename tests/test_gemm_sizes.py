"""Sizes beyond the 32 bits of a GEMM problem are refused, not wrapped."""

import numpy as np
import pytest
import torch

from frostspin_b200 import linalg

INT32 = 2**31 - 1


def _block_gemm(M, N, K):
    """block_gemm on blocks of one element repeated without memory."""
    one = torch.zeros(1, dtype=torch.float64)
    buf = [one.expand(max(m * n for m, n in zip(x, y, strict=True)))
           for x, y in ((M, K), (K, N), (M, N))]
    off = np.zeros(len(M), dtype=np.int64)
    a, b, c = buf
    linalg.block_gemm(a, off, False, b, off, False, c, off, *(np.array(x) for x in (M, N, K)))


@pytest.mark.parametrize("big", [2**31, 2**32, 2**32 + 5])
@pytest.mark.parametrize("side", [0, 1, 2])
def test_block_sides_beyond_32_bits_are_refused(big, side, monkeypatch):
    ran = []
    monkeypatch.setattr(linalg, "run_gemm_table", lambda arr, keep: ran.append(arr))
    sizes = [[3, 1], [2, 1], [4, 1]]
    sizes[side][1] = big
    with pytest.raises(OverflowError):
        _block_gemm(*sizes)
    assert not ran


def test_largest_sides_run(monkeypatch):
    ran = []
    monkeypatch.setattr(linalg, "run_gemm_table", lambda arr, keep: ran.append(arr))
    for sizes in ([[1], [INT32], [1]], [[INT32], [2], [1]], [[1], [1], [INT32]], [[3], [0], [4]]):
        _block_gemm(*sizes)
        assert [int(ran[-1][k][0]) for k in "MNK"] == [s[0] for s in sizes]
