"""Block-list reductions and diagonal products at the edges of their units: shares
of odd length at odd element offsets, 64 x 64 tiles with remainders, 4096-element
runs, every storage order.  Products are single roundings (exact equality); sums
of n terms differ from numpy's by at most n eps sum |terms|."""

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

SHAPES = [(1, 1), (1, 4097), (63, 65), (64, 64), (65, 129), (4095, 1), (3, 2731), (130, 257)]
EPS = np.finfo(np.float64).eps


def _buffer(rng, sizes):
    """Blocks back to back after one leading element, so that most start at odd offsets."""
    offsets = 1 + np.concatenate([[0], np.cumsum(sizes)[:-1]]).astype(np.int64)
    host = rng.standard_normal(int(sum(sizes)) + 1)
    return host, torch.from_numpy(host).cuda(), offsets


@pytest.mark.parametrize("squares", [True, False])
@pytest.mark.parametrize("lengths", [[1], [2, 1, 3], [511, 512, 513], [7] * 300,
                                     [296 * 512 - 1], [1_200_007, 5, 0, 33]])
def test_weighted_reduce(lengths, squares):
    from frostspin_b200 import linalg

    rng = np.random.default_rng(len(lengths))
    host, dev_buf, off = _buffer(rng, lengths)
    w = rng.integers(1, 8, len(lengths)).astype(np.float64)
    got = float(linalg.weighted_reduce(dev_buf, off, lengths, w, squares=squares))
    terms = [wi * (host[o:o + n] ** 2 if squares else host[o:o + n])
             for o, n, wi in zip(off, lengths, w, strict=True)]
    terms = np.concatenate(terms)
    assert abs(got - terms.sum()) <= terms.size * EPS * np.abs(terms).sum()


@pytest.mark.parametrize("a_trans", [False, True])
@pytest.mark.parametrize("b_trans", [False, True])
def test_pair_contract(a_trans, b_trans):
    from frostspin_b200 import linalg

    rng = np.random.default_rng(3)
    sizes = [m * n for m, n in SHAPES]
    ha, da, off = _buffer(rng, sizes)
    hb, db, _ = _buffer(rng, sizes)
    w = rng.integers(1, 8, len(SHAPES)).astype(np.float64)

    def block(h, o, m, n, trans):
        x = h[o:o + m * n]
        return x.reshape(n, m).T if trans else x.reshape(m, n)

    terms, trace = [], []
    for o, (m, n), wi in zip(off, SHAPES, w, strict=True):
        a, b = block(ha, o, m, n, a_trans), block(hb, o, n, m, b_trans)
        terms.append((wi * a * b.T).ravel())
        trace.append(wi * np.diagonal(a))
    terms, trace = np.concatenate(terms), np.concatenate(trace)
    pairs = [(o, o, m, n, a_trans, b_trans, wi) for o, (m, n), wi in zip(off, SHAPES, w, strict=True)]
    got = float(linalg.pair_contract(da, db, pairs))
    assert abs(got - terms.sum()) <= terms.size * EPS * np.abs(terms).sum()
    pairs = [(o, -1, m, n, a_trans, False, wi) for o, (m, n), wi in zip(off, SHAPES, w, strict=True)]
    got = float(linalg.pair_contract(da, None, pairs))
    assert abs(got - trace.sum()) <= trace.size * EPS * np.abs(trace).sum()


@pytest.mark.parametrize("trans", [False, True])
@pytest.mark.parametrize("left", [False, True])
def test_diag_mul(trans, left):
    from frostspin_b200 import linalg

    rng = np.random.default_rng(5)
    sizes = [m * n for m, n in SHAPES]
    hx, dx, off = _buffer(rng, sizes)
    hd, dd, doff = _buffer(rng, [m if left else n for m, n in SHAPES])
    entries, expect, out_off = [], [], 0
    for o, do, (m, n) in zip(off, doff, SHAPES, strict=True):
        x = hx[o:o + m * n]
        x = x.reshape(n, m).T if trans else x.reshape(m, n)
        d = hd[do:do + (m if left else n)]
        expect.append((x * (d[:, None] if left else d[None, :])).ravel())
        entries.append((o, out_off, do, m, n, trans, left))
        out_off += m * n
    got = linalg.diag_mul(dx, dd, entries, out_off).cpu().numpy()
    assert np.array_equal(got, np.concatenate(expect))
