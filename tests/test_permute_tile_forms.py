"""Transposed blocks in every form their tiles accept: the tile leg first, in the
middle and next to the last, one to six outer legs around it, legs of one entry, negative
and padded strides, remainders of the 32 x 32 tiles.  Both parts on the CPU with a
numpy reading of the tasks, and on the device, bit for bit against a transpose."""

import numpy as np
import pytest

from frostspin_b200.symmetric_tensor import abelian_plan as ap

# (output dimensions, position of the tile leg); the last leg is the other tile leg
FORMS = [
    ((40, 33), 0),
    ((3, 40, 33), 1),
    ((40, 3, 33), 0),
    ((2, 3, 35, 31), 2),
    ((2, 35, 3, 31), 1),
    ((35, 2, 3, 31), 0),
    ((2, 1, 3, 6, 65), 3),
    ((2, 3, 65, 1, 2, 7), 2),
    ((33, 2, 1, 3, 2, 32), 0),
    ((2, 1, 2, 3, 2, 64, 9), 5),
    ((2, 2, 1, 2, 3, 2, 8, 40), 6),
]


@pytest.fixture(autouse=True)
def _tiles_at_any_size(monkeypatch):
    monkeypatch.setattr(ap, "TILE_TOTAL", 0)


def _case(rng, dims, leg, gap, flip):
    """One EB: the input has `leg` innermost, the others in random order with `gap`
    unused elements after each row; flip: an outer leg backwards."""
    r = len(dims)
    rest = [int(k) for k in rng.permutation([k for k in range(r) if k != leg])]
    ostr = [0] * r
    step = 1
    for k in [leg, *reversed(rest)]:
        ostr[k] = step
        step = step * dims[k] + (gap if k == leg else 0)
    base = 0
    outer = [k for k in range(r - 1) if k != leg and dims[k] > 1]
    if flip and outer:
        k = outer[-1]
        base = ostr[k] * (dims[k] - 1)
        ostr[k] = -ostr[k]
    nstr = [int(x) for x in np.cumprod([1, *dims[:0:-1]])[::-1]]
    return ostr, nstr, base, step


def _tables(forms, gap, flip, seed=0):
    """FORMS of one rank in one table (a table's EBs share their number of legs)."""
    rng = np.random.default_rng(seed)
    dims, ostr, nstr, ob, nb = [], [], [], [], []
    so, sn = 3, 1
    for d, leg in forms:
        o, n, base, size = _case(rng, d, leg, gap, flip)
        dims.append(d)
        ostr.append(o)
        nstr.append(n)
        ob.append(so + base)
        nb.append(sn)
        so += size
        sn += int(np.prod(d))
    ebs, _ = ap._pack_ebs(*(np.array(x, dtype=np.int64) for x in (dims, ostr, nstr, ob, nb)),
                          np.ones(len(forms), dtype=bool))
    return ebs, ap._make_tasks(ebs), ap._make_tile_tasks(ebs), so, sn


def _by_rank():
    ranks = sorted({len(d) for d, _ in FORMS})
    return [[f for f in FORMS if len(f[0]) == r] for r in ranks]


def _apply(ebs, tasks, tiles, src, n_out):
    """The tasks read one by one: rows of every EB without a tile leg, tiles of the
    others in the order the header states."""
    out = np.full(n_out, np.nan)
    for table, tiled in ((tasks, False), (tiles, True)):
        for t in table:
            e = ebs[int(t["eb"])]
            r, a = int(e["ndim"]), int(e["tile_leg"])
            assert (a >= 0) == tiled
            d = [int(x) for x in e["dims"][:r]]
            o, n = ([int(x) for x in e[k][:r]] for k in ("ostride", "nstride"))
            legs = [k for k in range(r - 1) if not tiled or k != a]
            for u in range(int(t["start"]), int(t["start"]) + int(t["count"])):
                a0 = b0 = 0
                q, na, nb = u, 1, d[-1]
                if tiled:
                    ta, tb = -(-d[a] // 32), -(-d[-1] // 32)
                    q, rem = divmod(u, ta * tb)
                    b0, a0 = 32 * (rem // ta), 32 * (rem % ta)
                    na, nb = min(32, d[a] - a0), min(32, d[-1] - b0)
                so, dof = int(e["obase"]), int(e["nbase"])
                for k in reversed(legs):
                    q, i = divmod(q, d[k])
                    so += i * o[k]
                    dof += i * n[k]
                assert q == 0
                for i in range(na):
                    for j in range(nb):
                        s, w = so + (b0 + j) * o[-1], dof + (b0 + j) * n[-1]
                        if tiled:
                            s, w = s + (a0 + i) * o[a], w + (a0 + i) * n[a]
                        assert np.isnan(out[w])
                        out[w] = src[s]
    return out


@pytest.mark.parametrize("flip", [False, True])
@pytest.mark.parametrize("gap", [0, 3])
def test_tasks_move_every_entry_once(gap, flip):
    for forms in _by_rank():
        ebs, tasks, tiles, n_in, n_out = _tables(forms, gap, flip)
        assert (ebs["tile_leg"] >= 0).any()
        src = np.arange(n_in, dtype=float)

        class Plan:
            size = n_out

        Plan.ebs = ebs
        assert np.array_equal(_apply(ebs, tasks, tiles, src, n_out), ap.emulate_permute(Plan, src),
                              equal_nan=True)


@pytest.mark.gpu
@pytest.mark.parametrize("seed", [0, 1, 2])
@pytest.mark.parametrize("flip", [False, True])
@pytest.mark.parametrize("gap", [0, 3])
def test_device_moves_every_entry(gap, flip, seed):
    import torch

    from frostspin_b200 import linalg

    for forms in _by_rank():
        ebs, tasks, tiles, n_in, n_out = _tables(forms, gap, flip, seed)
        src = np.random.default_rng(seed).standard_normal(n_in)

        class Plan:
            size = n_out

        Plan.ebs = ebs
        want = ap.emulate_permute(Plan, src)
        out = torch.full((n_out,), float("nan"), dtype=torch.float64, device="cuda")
        tables = (ebs, tasks, tiles)
        linalg.run_copies(tables, linalg.upload_copies(tables), torch.from_numpy(src).cuda(), out)
        assert np.array_equal(out.cpu().numpy(), want, equal_nan=True)
