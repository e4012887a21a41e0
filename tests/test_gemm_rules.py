"""Which FP64 kernel a launch goes to, by sizes alone (linalg._wide)."""

import numpy as np
import pytest

from frostspin_b200 import _native, linalg


def _launch(columns, n, M, K):
    arr = np.zeros(n, dtype=_native.GEMM_PROBLEM_DTYPE)
    arr["M"], arr["K"] = M, K
    arr["N"] = columns // n
    arr["N"][0] += columns - int(arr["N"].sum())
    return arr


# a strip of 16 columns for each of 16 warps of 148 SMs is 37 888 columns
@pytest.mark.parametrize(("n", "M", "K", "least"), [
    (1, 20, 20, 75_776),      # up to 3 sectors
    (3, 20, 40, 75_776),
    (3, 20, 41, 101_035),     # long K
    (4, 20, 20, 113_664),     # more sectors
    (40, 20, 40, 113_664),
    (9, 100, 120, 151_552),
    (9, 56, 16, 113_664),     # rows that fill 64 x 64 tiles, short K
    (9, 56, 17, 265_216),     # ... and K from 17 on
    (2, 120, 64, 176_811),
    (9, 55, 64, 265_216),
    (9, 48, 40, 113_664),
])
def test_columns_of_the_wide_kernel(n, M, K, least):
    assert linalg._wide(_launch(least, n, M, K))
    assert not linalg._wide(_launch(least - 1, n, M, K))


def test_limits_of_the_wide_kernel():
    assert not linalg._wide(_launch(10**6, 41, 20, 20))
    assert not linalg._wide(_launch(10**6, 9, 20, 129))
    assert linalg._wide(_launch(10**6, 9, 180, 128))
    assert not linalg._wide(_launch(10**6, 9, 190, 128))
