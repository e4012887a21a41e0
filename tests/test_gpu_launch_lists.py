"""Tables passed by value with a launch against the same tables in device memory:
every list length where the form changes (40 and 360 GEMM problems, 48 split-K
items, 96 reduction blocks), mixed, uniform and thin launches, empty problems.
Both forms run the same kernels, so results are equal bit for bit."""

import numpy as np
import pytest

from frostspin_b200 import _native

pytestmark = pytest.mark.gpu


def _problems(rng, n, thin, mixed):
    import torch

    arr = np.zeros(n, dtype=_native.GEMM_PROBLEM_DTYPE)
    keep, outs = [], []
    for i in range(n):
        M, N, K = (int(x) for x in rng.integers(0 if i % 7 == 3 else 1, 33 if thin else 140, 3))
        if thin:
            N = int(rng.integers(1, 1500))
        ta, tb = (i % 2, i % 3 == 0) if mixed else (0, 0)
        a = torch.from_numpy(rng.standard_normal(M * K + 1)).cuda()
        b = torch.from_numpy(rng.standard_normal(K * N + 1)).cuda()
        c = torch.zeros(M * N + 1, dtype=torch.float64, device="cuda")
        keep += [a, b]
        outs.append(c)
        arr[i] = (a.data_ptr(), b.data_ptr(), c.data_ptr(), M if ta else K, K if tb else N, N,
                  M, N, K, ta, tb, 0, 1.0, 0.0)
    return arr, keep, outs


@pytest.mark.parametrize("n", [1, 40, 41, 360, 361])
@pytest.mark.parametrize("kind", ["mixed", "uniform", "thin"])
def test_gemm_lists_equal_tables(n, kind, monkeypatch):
    import torch

    from frostspin_b200 import linalg

    arr, keep, outs = _problems(np.random.default_rng(n), n, kind == "thin", kind == "mixed")
    linalg.grouped_dgemm_table(arr.copy())
    got = [c.clone() for c in outs]
    for c in outs:
        c.zero_()
    monkeypatch.setattr(_native, "FS_DGEMM_LIST_MAX", 0)
    linalg.grouped_dgemm_table(arr.copy())
    torch.cuda.synchronize()
    assert any(float(c.abs().sum()) > 0 for c in got)
    for x, y in zip(got, outs, strict=True):
        assert torch.equal(x, y)
    del keep


def test_list_entry_points_refuse_what_tables_cannot_hold():
    """Lengths, shapes and flags are checked on the host, before any launch."""
    lib = _native.lib()
    arr = np.zeros(361, dtype=_native.GEMM_PROBLEM_DTYPE)
    assert lib.fs_grouped_dgemm_list(arr.ctypes.data, 361, 0, None) == -7
    assert lib.fs_grouped_dgemm_list(arr.ctypes.data, 2, 3, None) == -1
    assert lib.fs_grouped_dgemm_list(None, 2, 0, None) == -1
    assert lib.fs_grouped_dgemm_list(arr.ctypes.data, 0, 0, None) == 0
    arr["M"][:2] = 33
    assert lib.fs_grouped_dgemm_list(arr.ctypes.data, 2, 2, None) == -1
    arr["transA"][1] = 1
    assert lib.fs_grouped_dgemm_list(arr.ctypes.data, 2, 1, None) == -1
    assert lib.fs_splitk_reduce_list(arr.ctypes.data, 49, 1, None) == -7


@pytest.mark.parametrize("n", [1, 96, 97])
def test_block_lists_equal_tables(n, monkeypatch):
    import torch

    from frostspin_b200 import linalg

    rng = np.random.default_rng(n)
    m, k = rng.integers(1, 70, n), rng.integers(1, 70, n)
    size = m * k
    off = np.concatenate([[0], np.cumsum(size)[:-1]])
    x, y = (torch.from_numpy(rng.standard_normal(int(size.sum()))).cuda() for _ in range(2))
    d = torch.from_numpy(rng.standard_normal(int(k.sum()))).cuda()
    doff = np.concatenate([[0], np.cumsum(k)[:-1]])

    def all_of():
        return [
            linalg.weighted_reduce(x, off, size, m, squares=True),
            linalg.weighted_reduce(x, off, size, m, squares=False),
            linalg.pair_contract(x, y, [(o, o, a, b, False, False, 2.0)
                                        for o, a, b in zip(off, m, k, strict=True)]),
            linalg.diag_mul(x, d, [(o, o, e, a, b, False, False)
                                   for o, e, a, b in zip(off, doff, m, k, strict=True)],
                            x.numel()),
        ]

    got = all_of()
    monkeypatch.setattr(_native, "FS_LIST_MAX", 0)
    for a, b in zip(got, all_of(), strict=True):
        assert torch.equal(a, b)


def test_split_k_lists_equal_tables(monkeypatch):
    import torch

    from frostspin_b200 import linalg

    g = torch.Generator(device="cuda")
    g.manual_seed(1)
    ab = [(torch.randn(40, 5000, dtype=torch.float64, device="cuda", generator=g),
           torch.randn(5000, 30, dtype=torch.float64, device="cuda", generator=g))
          for _ in range(3)]
    lefts, rights = [a for a, _ in ab], [b for _, b in ab]
    got = linalg.matmul_blocks(lefts, rights)[0]
    monkeypatch.setattr(_native, "FS_SPLIT_LIST_MAX", 0)
    monkeypatch.setattr(_native, "FS_DGEMM_LIST_MAX", 0)
    assert torch.equal(got, linalg.matmul_blocks(lefts, rights)[0])
