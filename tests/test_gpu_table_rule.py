"""Large launches of the per-tile GEMM kernel go through tables in device memory:
both sides of the line run the same kernel, with equal results."""

import numpy as np
import pytest

from frostspin_b200 import _native, linalg

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mixed", [False, True])
def test_both_sides_of_the_line(mixed, monkeypatch):
    import torch

    rng = np.random.default_rng(3)
    shapes = [(70, 300, 260), (1, 65, 700), (129, 64, 257), (64, 1, 300)]
    arr = np.zeros(len(shapes), dtype=_native.GEMM_PROBLEM_DTYPE)
    keep, outs = [], []
    for i, (M, N, K) in enumerate(shapes):
        ta, tb = (i % 2, i // 2) if mixed else (0, 0)
        a, b = (torch.from_numpy(rng.standard_normal(n)).cuda() for n in (M * K, K * N))
        outs.append(torch.zeros(M * N, dtype=torch.float64, device="cuda"))
        keep += [a, b]
        arr[i] = (a.data_ptr(), b.data_ptr(), outs[-1].data_ptr(), M if ta else K, K if tb else N,
                  N, M, N, K, ta, tb, 0, 1.0, 0.0)
    flops = linalg._flops(arr)
    got = []
    for limit, tables in ((flops * 1.01, 0), (flops, 1)):
        monkeypatch.setattr(linalg, "_TABLE_FLOPS", limit)
        before = _native.CALL_COUNTS.get("fs_expand_tiles", 0)
        linalg._launch_dgemm(arr)
        assert _native.CALL_COUNTS.get("fs_expand_tiles", 0) == before + tables
        got.append([c.clone() for c in outs])
        for c in outs:
            c.zero_()
    for x, y in zip(*got, strict=True):
        assert float(x.abs().sum()) > 0 and torch.equal(x, y)
    del keep
