"""Infinities and NaN in sums, contractions and products of blocks: they come out as
numpy gives them when they lie in a block, and never from the elements around it
(padding of 64 x 64 tiles, runs of 4096 elements, aligned 16-byte loads)."""

import numpy as np
import pytest
import torch

from frostspin_b200 import linalg

pytestmark = pytest.mark.gpu

SHAPES = [(1, 1), (63, 65), (64, 64), (1, 4097), (4097, 1), (3, 5000), (130, 70), (5, 7)]
SPECIAL = [np.inf, -np.inf, np.nan]


def _blocks(rng, gap=3):
    """Finite blocks of non-zero values with NaN between them."""
    off, parts, at = [], [np.full(gap, np.nan)], gap
    for m, n in SHAPES:
        parts += [rng.uniform(0.5, 2.0, m * n), np.full(gap, np.nan)]
        off.append(at)
        at += m * n + gap
    return np.concatenate(parts), off


def _same(got, want):
    return (np.isnan(got) and np.isnan(want)) or got == want or abs(got - want) <= 1e-9 * abs(want)


@pytest.mark.parametrize("trans", [(False, False), (False, True), (True, False), (True, True)])
def test_contractions(trans):
    rng = np.random.default_rng(1)
    ha, off = _blocks(rng)
    hb, _ = _blocks(rng)
    db = torch.from_numpy(hb).cuda()
    for bad in (None, *SPECIAL):
        for i, (o, (m, n)) in enumerate(zip(off, SHAPES, strict=True)):
            h = ha.copy()
            if bad is not None:
                h[o + (m * n) // 2] = bad
            a, b = h[o:o + m * n], hb[o:o + m * n]
            a = a.reshape(n, m).T if trans[0] else a.reshape(m, n)
            b = b.reshape(m, n).T if trans[1] else b.reshape(n, m)
            got = float(linalg.pair_contract(torch.from_numpy(h).cuda(), db,
                                             [(o, o, m, n, *trans, 2.0)]))
            assert _same(got, 2.0 * (a * b.T).sum()), (bad, i)


@pytest.mark.parametrize("squares", [False, True])
def test_sums(squares):
    rng = np.random.default_rng(2)
    h0, off = _blocks(rng)
    size = [m * n for m, n in SHAPES]
    for bad in (None, *SPECIAL):
        for i in range(len(SHAPES)):
            h = h0.copy()
            if bad is not None:
                h[off[i] + size[i] - 1] = bad
            x = np.concatenate([h[o:o + n] for o, n in zip(off, size, strict=True)])
            got = float(linalg.weighted_reduce(torch.from_numpy(h).cuda(), off, size,
                                               [1.0] * len(size), squares=squares))
            assert _same(got, (x * x).sum() if squares else x.sum()), (bad, i)


@pytest.mark.parametrize("x_trans", [False, True])
@pytest.mark.parametrize("left", [False, True])
def test_diagonal_products(x_trans, left):
    rng = np.random.default_rng(3)
    h, off = _blocks(rng)
    entries, diag, at = [], [], 0
    want = np.full(h.size, 7.0)
    for i, (o, (m, n)) in enumerate(zip(off, SHAPES, strict=True)):
        d = rng.uniform(0.5, 2.0, m if left else n)
        d[d.size // 2] = SPECIAL[i % 3]
        h[o] = SPECIAL[(i + 1) % 3]
        x = h[o:o + m * n].reshape(n, m).T if x_trans else h[o:o + m * n].reshape(m, n)
        want[o:o + m * n] = (d[:, None] * x if left else x * d).ravel()
        entries.append((o, o, at, m, n, x_trans, left))
        diag.append(d)
        at += d.size
    got = linalg.diag_mul(torch.from_numpy(h).cuda(), torch.from_numpy(np.concatenate(diag)).cuda(),
                          entries, h.size).cpu().numpy()
    for o, (m, n) in zip(off, SHAPES, strict=True):
        assert np.array_equal(got[o:o + m * n], want[o:o + m * n], equal_nan=True)
