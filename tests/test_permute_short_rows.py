"""Row tasks of the abelian permute around the sizes where the number of loads per
thread changes (512 entries): one EB per task size, present and absent sources,
rows of 1 to many entries, bit for bit against the numpy application of the plan."""

import numpy as np
import pytest

from frostspin_b200.symmetric_tensor import abelian_plan as ap


@pytest.mark.gpu
@pytest.mark.parametrize("shift", [0, 1])
def test_row_tasks_bit_exact(shift):
    import torch

    from frostspin_b200 import linalg

    legs = [(1, 1), (1, 511), (511, 1), (2, 256), (512, 1), (1, 513), (27, 19), (171, 3), (73, 7),
            (1, 2049), (300, 7), (1024, 2), (1025, 2), (5, 4096), (3, 2731), (1, 9000)]
    absent = [i % 5 == 3 for i in range(len(legs))]
    dims, ostr, nstr, ob, nb = [], [], [], [], []
    so, sn = shift, shift
    for (a, b), gone in zip(legs, absent, strict=True):
        dims.append([a, b])
        ostr.append([1, a])
        nstr.append([b, 1])
        ob.append(-1 if gone else so)
        nb.append(sn)
        so += 0 if gone else a * b
        sn += a * b
    ebs, _ = ap._pack_ebs(*(np.array(x, dtype=np.int64) for x in (dims, ostr, nstr, ob, nb)),
                          ~np.array(absent))
    tables = (ebs, ap._make_tasks(ebs), ap._make_tile_tasks(ebs))
    assert tables[2].size == 0      # all by rows
    src = np.random.default_rng(1).standard_normal(so)

    class Plan:
        size = sn

    Plan.ebs = ebs
    want = ap.emulate_permute(Plan, src)
    out = torch.full((sn,), float("nan"), dtype=torch.float64, device="cuda")
    linalg.run_copies(tables, linalg.upload_copies(tables), torch.from_numpy(src).cuda(), out)
    got = out.cpu().numpy()
    assert np.array_equal(got[shift:], want[shift:])
