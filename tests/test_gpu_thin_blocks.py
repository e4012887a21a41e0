"""Thin blocks whose two sides run in different storage orders, at the edges of
the element-wise form: sides around its limit of 16, runs of 4096 elements that
end inside a row, odd offsets, infinities beside the block.  A product is one
rounding; a sum of n terms differs from numpy's by at most n eps sum |terms|."""

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

SHAPES = [(1, 1), (1, 4096), (4097, 1), (2, 2048), (2, 2049), (3, 1365), (1366, 3), (5, 9000),
          (7, 12293), (12293, 7), (15, 3000), (3001, 15), (16, 300), (300, 16), (15, 15), (2, 1)]
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
