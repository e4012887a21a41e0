"""Block lists longer than a CTA has threads (256 and 512), with empty blocks at
the edges of its scan: sums and products of every block.  Small integers, so that
sums are exact in any order."""

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 255, 256, 257, 511, 512, 513, 1100])
def test_every_block_counts_once(n):
    from frostspin_b200 import linalg

    rng = np.random.default_rng(n)
    m, k = rng.integers(1, 90, n), rng.integers(1, 20, n)
    for i in {0, 255, 256, 511, n - 1} & set(range(n)):
        m[i] = 0                                  # empty blocks
    size = m * k
    off = 3 + np.concatenate([[0], np.cumsum(size)[:-1]])
    total = int(size.sum()) + 3
    x, y = (torch.from_numpy(rng.integers(-9, 10, total).astype(float)).cuda() for _ in range(2))
    hx, hy = x.cpu().numpy(), y.cpu().numpy()
    w = rng.integers(1, 5, n).astype(float)
    d = torch.from_numpy(rng.integers(-9, 10, int(k.sum())).astype(float)).cuda()
    hd, doff = d.cpu().numpy(), np.concatenate([[0], np.cumsum(k)[:-1]])
    square = crossed = trace = 0.0
    want = np.zeros(total)
    for i in range(n):
        a, b = (h[off[i]:off[i] + size[i]] for h in (hx, hy))
        square += w[i] * (a * a).sum()
        crossed += w[i] * (a.reshape(m[i], k[i]) * b.reshape(k[i], m[i]).T).sum()
        trace += w[i] * np.diagonal(a.reshape(m[i], k[i])).sum()
        want[off[i]:off[i] + size[i]] = (a.reshape(m[i], k[i]) * hd[doff[i]:doff[i] + k[i]]).ravel()
    assert float(linalg.weighted_reduce(x, off, size, w, squares=True)) == square
    pairs = [(o, o, a, b, False, False, c) for o, a, b, c in zip(off, m, k, w, strict=True)]
    assert float(linalg.pair_contract(x, y, pairs)) == crossed
    pairs = [(o, -1, a, b, False, False, c) for o, a, b, c in zip(off, m, k, w, strict=True)]
    assert float(linalg.pair_contract(x, None, pairs)) == trace
    out = linalg.diag_mul(x, d, [(o, o, e, a, b, False, False) for o, e, a, b in
                                 zip(off, doff, m, k, strict=True)], total).cpu().numpy()
    assert np.array_equal(out[3:], want[3:])
