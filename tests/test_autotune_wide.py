"""The autotuner and the wide FP64 kernel: classes that occur in its launches are
timed on it too, with the launch's columns, and a problem's FP64 time is that of
the kernel its launch would take."""

import numpy as np
import pytest

from frostspin_b200 import _native, autotune, linalg

MODE = "ozaki2_11"


@pytest.fixture(autouse=True)
def _empty_table():
    autotune.clear()
    yield
    autotune.set_enabled(False)
    autotune.clear()


def _launch(*shapes):
    arr = np.zeros(len(shapes), dtype=_native.GEMM_PROBLEM_DTYPE)
    for i, s in enumerate(shapes):
        arr["M"][i], arr["N"][i], arr["K"][i] = s
    return arr


WIDE = _launch(*[(300, 40000, 70)] * 9)            # 0.36 M columns
NARROW = _launch((300, 40000, 70), (20, 20, 20))   # the same class, few columns
LONG = _launch((300, 40000, 127), (900, 900, 900)) # the same class, not for the wide kernel


def test_classes_of_wide_launches_are_timed_on_the_wide_kernel(monkeypatch):
    timed = []

    def time_launch(M, N, K, ta, tb, copies, modes, reps):
        timed.append((M, N, K, copies, modes))
        return {m: {"fp64": 3.0, "fp64_wide": 1.0}.get(m, 2.0) * 1e-14 * 2 * M * N * K * copies
                for m in modes}

    monkeypatch.setattr(autotune, "_time_launch", time_launch)
    assert linalg._wide(WIDE) and not linalg._wide(NARROW) and not linalg._wide(LONG)
    autotune.tune([NARROW, LONG], MODE)
    assert all(modes == ("fp64", MODE) for *_, modes in timed)
    timed.clear()
    autotune.tune([NARROW, WIDE, LONG], MODE)
    # only the new kernel is timed, on a problem and the columns of its own launch
    assert timed == [(300, 8192, 70, 40, ("fp64_wide",))]
    # mixed beats the tile kernels, the wide kernel beats mixed
    assert autotune.decide(WIDE, MODE) == [False] * 9
    assert autotune.decide(NARROW, MODE)[0] is True
    assert autotune.decide(LONG, MODE)[0] is True
    per = 2.0 * 300 * 40000 * 70 * 1e-14
    got = autotune.predict([WIDE], MODE)
    assert abs(got["fp64"] - 9 * per) < 1e-9 and abs(got["chosen"] - 9 * per) < 1e-9
    got = autotune.predict([NARROW], MODE)
    assert abs(got["fp64"] - 3 * per) < 1e-9 and abs(got["chosen"] - 2 * per) < 1e-9


@pytest.mark.gpu
def test_timed_kernels_are_the_ones_of_the_launches():
    """tune() on a wide launch counts launches of both FP64 kernels; the tuned
    dispatch then runs the launch in one arithmetic with results within bounds."""
    import torch

    g = torch.Generator(device="cuda")
    g.manual_seed(1)
    shapes = [(300, 40000, 70)] * 9
    lefts, rights = ([torch.randn(*s, dtype=torch.float64, device="cuda", generator=g) for s in x]
                     for x in ([(m, k) for m, _, k in shapes], [(k, n) for _, n, k in shapes]))
    with linalg.record_gemm_calls() as records:
        want = linalg.matmul_blocks(lefts, rights)[0]
    count = _native.CALL_COUNTS
    before = dict(count)
    autotune.tune(records, MODE)
    for name in ("fs_grouped_dgemm_wide", "fs_grouped_dgemm_uniform", "fs_ozaki2_gemm_pair"):
        assert count.get(name, 0) > before.get(name, 0), name
    row = autotune.table()[MODE, autotune.shape_class(300, 40000, 70)]
    assert 0 < row["fp64_wide"] < row["fp64"]
    autotune.set_enabled(True)
    with linalg.gemm_precision_mode(MODE):
        got = linalg.matmul_blocks(lefts, rights)[0]
    assert float((got - want).abs().max()) <= 1e-9 * float(want.abs().max())
