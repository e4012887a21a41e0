"""Tile tasks of the transposed elementary blocks: which blocks take them, that
rows and tiles together cover every entry once, and the device permute bit for
bit against the numpy application of the same plan."""

import numpy as np
import pytest

from frostspin_b200.symmetric_tensor import abelian_plan as ap

# (tile leg, middle leg, last leg): edges of the 32 x 32 tiles and of the rule
LEGS = [(6, 3, 22), (5, 3, 40), (8, 2, 16), (8, 2, 15), (31, 4, 33), (32, 1, 32), (33, 2, 65),
        (64, 3, 7), (6, 2, 129), (100, 5, 31)]


@pytest.fixture(autouse=True)
def _tiles_at_any_size(monkeypatch):
    monkeypatch.setattr(ap, "TILE_TOTAL", 0)


def _tables(legs, in_shift=0, out_shift=0, gap=0):
    """One EB per entry of `legs`: input order (last, middle, tile leg), output
    order (tile leg, middle, last); `gap` unused elements between input rows."""
    dims, ostr, nstr, ob, nb = [], [], [], [], []
    so, sn = in_shift, out_shift
    for a, m, b in legs:
        dims.append([a, m, b])
        ostr.append([1, a + gap, (a + gap) * m])
        nstr.append([m * b, b, 1])
        ob.append(so)
        nb.append(sn)
        so += (a + gap) * m * b
        sn += a * m * b
    ebs, _ = ap._pack_ebs(*(np.array(x, dtype=np.int64) for x in (dims, ostr, nstr, ob, nb)),
                          np.ones(len(legs), dtype=bool))
    return ebs, ap._make_tasks(ebs), ap._make_tile_tasks(ebs), so, sn


def test_rows_and_tiles_cover_every_entry_once():
    ebs, tasks, tiles, _, _ = _tables(LEGS)
    tiled = ebs["tile_leg"] >= 0
    assert list(tiled) == [min(a, b) >= 6 and a * b >= 128 for a, _, b in LEGS]
    assert not np.isin(tasks["eb"], np.flatnonzero(tiled)).any()
    assert np.isin(tiles["eb"], np.flatnonzero(tiled)).all()
    assert tiles["count"].max() <= ap.MAX_TASK_TILES
    for e, (a, m, b) in enumerate(LEGS):
        table = tiles if tiled[e] else tasks
        mine = table[table["eb"] == e]
        units = m * -(-a // 32) * -(-b // 32) if tiled[e] else a * m
        assert np.array_equal(mine["start"], np.cumsum(mine["count"]) - mine["count"])
        assert mine["count"].sum() == units


def test_absent_sources_and_kept_legs_stay_on_rows():
    d = np.array([[40, 40]] * 3)
    o = np.array([[1, 40], [40, 1], [1, 40]])
    n = np.array([[40, 1]] * 3)
    ebs, _ = ap._pack_ebs(d, o, n, np.array([0, 0, -1]), np.zeros(3, int),
                          np.array([True, True, False]))
    assert list(ebs["tile_leg"]) == [0, -1, -1]


def test_small_permutes_stay_on_rows(monkeypatch):
    total = sum(a * m * b for a, m, b in LEGS if min(a, b) >= 6 and a * b >= 128)
    for limit, any_tiled in ((total, True), (total + 1, False)):
        monkeypatch.setattr(ap, "TILE_TOTAL", limit)
        ebs, tasks, tiles, _, _ = _tables(LEGS)
        assert (ebs["tile_leg"] >= 0).any() == any_tiled == (tiles.size > 0)


@pytest.mark.gpu
@pytest.mark.parametrize("shifts", [(0, 0, 0), (1, 0, 0), (3, 5, 1)])
@pytest.mark.parametrize("legs", [LEGS, [x for x in LEGS if min(x) >= 2], [(300, 40, 70)],
                                  [(33, 1, 40)] * 40])
def test_device_tiles_bit_exact(legs, shifts):
    import torch

    from frostspin_b200 import linalg

    ebs, tasks, tiles, n_in, n_out = _tables(legs, *shifts)
    src = np.random.default_rng(1).standard_normal(n_in)

    class Plan:
        size = n_out

    Plan.ebs = ebs
    want = ap.emulate_permute(Plan, src)
    d_src = torch.from_numpy(src).cuda()
    out = torch.full((n_out,), float("nan"), dtype=torch.float64, device="cuda")
    tables = (ebs, tasks, tiles)
    linalg.run_copies(tables, linalg.upload_copies(tables), d_src, out)
    assert np.array_equal(out.cpu().numpy(), want, equal_nan=True)


@pytest.mark.gpu
def test_tiles_of_many_buffers():
    """Transposed permutes collected by shared_launches: one multi-buffer launch."""
    from frostspin_b200 import U1SymmetricTensor, _native, linalg
    from frostspin_b200.symmetric_tensor.abelian_symmetric_tensor import plan_cache_clear

    plan_cache_clear()
    rng = np.random.default_rng(2)
    ts = []
    for n in (40, 23, 70):
        r = np.sort(rng.integers(-1, 2, n)).astype(np.int8)
        d = np.array([-1, 0, 0, 1], dtype=np.int8)
        ts.append(U1SymmetricTensor.random((r,), (d, r), np.array([0, 1, 1], bool), rng=rng))
    want = [t.permute((2, 1), (0,)) for t in ts]
    before = _native.CALL_COUNTS.get("fs_permute_tiles_multi", 0)
    with linalg.shared_launches():
        got = [t.permute((2, 1), (0,)) for t in ts]
    assert _native.CALL_COUNTS.get("fs_permute_tiles_multi", 0) == before + 1
    for g, w, t in zip(got, want, ts, strict=True):
        dense = t.toarray().transpose(2, 1, 0)
        assert np.array_equal(g.toarray(), w.toarray())
        assert np.array_equal(g.toarray(), dense)
    plan_cache_clear()   # later tests plan with the shipped limit
