"""The offset table of the fused SU(2) kernel and the tasks made for it: the limit
binds for every number of pieces, a task beyond it is refused on the host, and the
kernel runs tasks that reach it exactly."""

import os
import re

import numpy as np
import pytest

from frostspin_b200 import _native
from frostspin_b200.symmetric_tensor import su2_fused_plan as sp
from frostspin_b200.symmetric_tensor.abelian_plan import magic_divisor

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def _group(dims, n_in, n_out, K=1):
    g = np.zeros(1, dtype=_native.SU2_GROUP_DTYPE)
    nd = len(dims)
    g["ndim"], g["ncols"], g["M"], g["K"] = nd, int(np.prod(dims)), K, K
    g["dims"] = 1
    g["dims"][0, :nd] = dims
    m, s = magic_divisor(np.maximum(g["dims"].astype(np.int64), 1))
    g["divm"], g["divs"] = m, s
    g["in_count"], g["out_count"], g["out_first"] = n_in, n_out, n_in
    return g


def _entries(g, tasks):
    """(piece, plane) entries of each task."""
    nd = int(g["ndim"][0])
    plane = int(np.prod(g["dims"][0, max(nd - 2, 0):nd])) if nd else 1
    start, count = tasks["start"].astype(np.int64), tasks["count"].astype(np.int64)
    return ((start + count - 1) // plane - start // plane + 1) * int(
        g["in_count"][0] + g["out_count"][0])


def test_limits_match_the_header():
    text = open(os.path.join(ROOT, "include", "frostspin_b200.h")).read()
    for name in ("FS_SU2_TASK_ROWS", "FS_SU2_TASK_TABLE"):
        assert int(re.search(rf"#define {name} (\d+)", text).group(1)) == getattr(_native, name)
    assert sp.TASK_TABLE == _native.FS_SU2_TASK_TABLE


@pytest.mark.parametrize(("n_in", "n_out"), [(1, 1), (1, 2), (8, 8), (16, 16)])
@pytest.mark.parametrize("L", [1, 2, 3])
def test_the_limit_binds_and_is_checked(n_in, n_out, L, monkeypatch):
    g = _group((1_000_000, 1, L), n_in, n_out)   # enough that TASK_COEFFS does not bind
    tasks = sp.make_tasks(g)
    sp.check_tasks(g, tasks)
    most = int(_entries(g, tasks).max())
    # full: one more plane would not fit
    assert most <= _native.FS_SU2_TASK_TABLE < most + n_in + n_out
    # without the limit the tasks are larger, and refused
    monkeypatch.setattr(sp, "TASK_TABLE", 10**9)
    monkeypatch.setattr(sp, "TASK_ROWS", 10**9)
    wrong = sp.make_tasks(g)
    assert int(_entries(g, wrong).max()) > _native.FS_SU2_TASK_TABLE
    with pytest.raises(AssertionError, match="offset table"):
        sp.check_tasks(g, wrong)


@pytest.mark.parametrize("dims", [(), (7,), (3, 5), (2, 9000), (4, 1, 6, 2), (300, 40)])
def test_columns_are_covered_once(dims):
    g = _group(dims, 3, 2)
    tasks = sp.make_tasks(g)
    sp.check_tasks(g, tasks)
    for bad in (tasks[1:], np.concatenate([tasks, tasks[:1]])):
        with pytest.raises(AssertionError):
            sp.check_tasks(g, bad)
    short = tasks.copy()
    short["count"][-1] -= 1
    with pytest.raises(AssertionError):
        sp.check_tasks(g, short)


@pytest.mark.gpu
@pytest.mark.parametrize(("n", "K"), [(1, 1), (16, 16), (3, 12), (16, 32)])
def test_device_tasks_at_the_limit(n, K):
    """Tasks as long as the table allows, n pieces a side of K / n rows; the result against the numpy application
    ((K + 2) eps sum |u| |x| for sums of K products)."""
    import torch

    from frostspin_b200 import device as dev

    rng = np.random.default_rng(K)
    dims = (20000, 1, 2) if n == 1 else (700, 1, 2)
    g = _group(dims, n, n, K)
    cols, rows = int(np.prod(dims)), K // n
    pieces = np.zeros(2 * n, dtype=_native.SU2_PIECE_DTYPE)
    for i in range(2 * n):
        p = pieces[i]
        p["base"], p["sr"], p["sc"], p["row0"] = (i % n) * rows * cols, rows, 1, (i % n) * rows
        p["sr_stride"], p["sc_stride"] = cols, 1
        p["ext"][:3] = (2, 2, 1) if i >= n else (1, 1, dims[0])     # innermost legs apart
    step = dims[2] * (_native.FS_SU2_TASK_TABLE // (2 * n))      # full tables
    start = np.arange(0, cols, step)
    tasks = np.zeros(start.size, dtype=_native.PERM_TASK_DTYPE)
    tasks["start"], tasks["count"] = start, np.minimum(step, cols - start)
    sp.check(g, pieces, K * cols, K * cols, K * K)
    sp.check_tasks(g, tasks)
    assert _native.FS_SU2_TASK_TABLE - 2 * n < int(_entries(g, tasks).max())
    U, src = rng.standard_normal(K * K), rng.standard_normal(K * cols)
    want = sp.emulate(g, pieces, tasks, U, src, np.full(K * cols, np.nan))
    scale = sp.emulate(g, pieces, tasks, np.abs(U), np.abs(src), np.full(K * cols, np.nan))
    d_g, d_p, d_t = (dev.upload(a) for a in (g, pieces, tasks))
    d_u, d_src = dev.upload_f64(U), dev.upload_f64(src)
    out = torch.full((K * cols,), float("nan"), dtype=torch.float64, device="cuda")
    flag = torch.zeros(1, dtype=torch.int32, device="cuda")
    _native.call("fs_su2_permute_fused", d_src.data_ptr(), src.size, out.data_ptr(), out.numel(),
                 d_g.data_ptr(), 1, d_p.data_ptr(), 2 * n, d_u.data_ptr(), U.size,
                 d_t.data_ptr(), tasks.size, flag.data_ptr(), dev.stream())
    assert int(flag.item()) == 0
    assert np.all(np.abs(out.cpu().numpy() - want) <= (K + 2) * np.finfo(float).eps * scale)
