"""The wide grouped GEMM (small op(A) in shared memory, columns streamed by
independent warps) at its edges: K around its k steps and limits, M around the
8- and 16-row blocks, ragged and tiny N beside wide ones, every transpose, beta.
FP64 sums of K products: |error| <= (K + 2) eps sum |a| |b| + 2 eps |beta c|."""

import numpy as np
import pytest

from frostspin_b200 import _native

pytestmark = pytest.mark.gpu

EPS = np.finfo(float).eps
SHORT = [(1, 70001, 1), (7, 30000, 3), (8, 65, 4), (9, 20011, 5), (16, 7, 31), (17, 999, 32),
         (33, 15, 8), (51, 16, 0), (0, 100, 4), (4, 0, 4)]
MID = [(64, 40000, 64), (65, 20003, 33), (23, 17, 63), (120, 5001, 48), (5, 1, 60)]
LONG = [(150, 50001, 128), (13, 9, 127), (24, 30000, 65), (180, 4100, 120)]


@pytest.mark.parametrize("beta", [0.0, -0.5])
@pytest.mark.parametrize("trans", [(0, 0), (0, 1), (1, 0), (1, 1)])
@pytest.mark.parametrize("shapes", [SHORT, MID, LONG])
def test_wide_gemm(shapes, trans, beta, monkeypatch):
    import torch

    from frostspin_b200 import linalg

    monkeypatch.setattr(linalg, "_WIDE_COLUMNS", 0)
    rng = np.random.default_rng(7)
    ta, tb = trans
    arr = np.zeros(len(shapes), dtype=_native.GEMM_PROBLEM_DTYPE)
    keep, refs = [], []
    for i, (M, N, K) in enumerate(shapes):
        A, B, C = rng.standard_normal((M, K)), rng.standard_normal((K, N)), rng.standard_normal((M, N))
        if beta == 0.0:
            C[:] = np.nan
        dA, dB, dC = (torch.from_numpy(np.ascontiguousarray(x)).cuda()
                      for x in (A.T if ta else A, B.T if tb else B, C))
        arr[i] = (dA.data_ptr(), dB.data_ptr(), dC.data_ptr(), M if ta else K, K if tb else N, N,
                  M, N, K, ta, tb, 0, 1.5, beta)
        ref = 1.5 * (A @ B) + (beta * C if beta else 0.0)
        bound = 1.5 * (K + 2) * EPS * (np.abs(A) @ np.abs(B)) + (2 * EPS * np.abs(ref) if K else 0)
        bound = bound + (2 * EPS * np.abs(beta * C) if beta else 0.0)
        keep += [dA, dB]
        refs.append((dC, ref, bound))
    assert linalg._wide(arr)
    before = _native.CALL_COUNTS.get("fs_grouped_dgemm_wide", 0)
    linalg._dgemm(arr)
    assert _native.CALL_COUNTS.get("fs_grouped_dgemm_wide", 0) == before + 1
    for dC, ref, bound in refs:
        assert np.all(np.abs(dC.cpu().numpy() - ref) <= bound)


def test_limits_are_checked_on_the_host():
    lib = _native.lib()
    arr = np.zeros(41, dtype=_native.GEMM_PROBLEM_DTYPE)
    assert lib.fs_grouped_dgemm_wide(arr.ctypes.data, 41, None) == -7
    assert lib.fs_grouped_dgemm_wide(None, 1, None) == -1
    arr["K"][0] = 129
    assert lib.fs_grouped_dgemm_wide(arr.ctypes.data, 1, None) == -7
    arr["K"][0], arr["M"][0] = 128, 190
    assert lib.fs_grouped_dgemm_wide(arr.ctypes.data, 1, None) == -7
    arr["M"][0] = -1
    assert lib.fs_grouped_dgemm_wide(arr.ctypes.data, 1, None) == -1
