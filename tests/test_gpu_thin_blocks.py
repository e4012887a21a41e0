"""Thin blocks whose two sides run in different storage orders, at the edges of
the element-wise forms: short sides around their limits of 16 (contractions) and 10
(diagonal products), long ones around 4096, runs of 4096 elements that
end inside a row, odd offsets, infinities beside the block.  A product is one
rounding; a sum of n terms differs from numpy's by at most n eps sum |terms|."""

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

SHAPES = [(1, 1), (1, 4096), (1, 4097), (4097, 1), (2, 4096), (2, 4097), (3, 4100), (4101, 3),
          (5, 9000), (7, 12293), (12293, 7), (9, 5000), (4999, 9), (10, 4500), (4500, 10),
          (15, 5001), (5000, 15), (16, 4097), (4097, 16), (15, 15), (2, 1), (3, 1365)]
EPS = np.finfo(np.float64).eps


def _buffer(rng, gap):
    """Blocks with `gap` infinities before and after each."""
    parts, off, at = [], [], 0
    for m, n in SHAPES:
        parts += [np.full(gap, np.inf), rng.standard_normal(m * n)]
        off.append(at + gap)
        at += gap + m * n
    host = np.concatenate([*parts, np.full(gap, np.inf)])
    return host, torch.from_numpy(host).cuda(), off


@pytest.mark.parametrize("trans", [False, True])
@pytest.mark.parametrize("gap", [1, 2])
def test_crossed_contraction(trans, gap):
    from frostspin_b200 import linalg

    rng = np.random.default_rng(gap)
    ha, da, off = _buffer(rng, gap)
    hb, db, _ = _buffer(rng, gap)
    terms, pairs = [], []
    for i, (o, (m, n)) in enumerate(zip(off, SHAPES, strict=True)):
        a = ha[o:o + m * n].reshape(n, m).T if trans else ha[o:o + m * n].reshape(m, n)
        b = hb[o:o + m * n].reshape(m, n).T if trans else hb[o:o + m * n].reshape(n, m)
        terms.append(((1 + i) * a * b.T).ravel())
        pairs.append((o, o, m, n, trans, trans, 1.0 + i))
        one = float(linalg.pair_contract(da, db, pairs[-1:]))
        assert abs(one - terms[-1].sum()) <= m * n * EPS * np.abs(terms[-1]).sum()
    terms = np.concatenate(terms)
    got = float(linalg.pair_contract(da, db, pairs))
    assert abs(got - terms.sum()) <= terms.size * EPS * np.abs(terms).sum()


@pytest.mark.parametrize("left", [False, True])
@pytest.mark.parametrize("gap", [1, 2])
def test_diagonal_product_of_transposed_blocks(left, gap):
    from frostspin_b200 import linalg

    rng = np.random.default_rng(gap)
    host, dx, off = _buffer(rng, gap)
    want = np.full(host.size, np.nan)
    entries, diag, at = [], [], 0
    for o, (m, n) in zip(off, SHAPES, strict=True):
        d = rng.standard_normal(m if left else n)
        x = host[o:o + m * n].reshape(n, m).T
        want[o:o + m * n] = (d[:, None] * x if left else x * d).ravel()
        entries.append((o, o, at, m, n, True, left))
        diag.append(d)
        at += d.size
    dd = torch.from_numpy(np.concatenate(diag)).cuda()
    got = linalg.diag_mul(dx, dd, entries, host.size).cpu().numpy()
    inside = ~np.isnan(want)
    assert np.array_equal(got[inside], want[inside])
