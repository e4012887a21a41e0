"""Ozaki II residue slices at the edges of the split kernel's units (32 rows x
128 k, 8 k per thread and row): row counts and K around them, both storage
orders, odd element offsets.  Every slice byte is compared with numpy's."""

import numpy as np
import pytest

from frostspin_b200 import _native

pytestmark = pytest.mark.gpu

SHAPES = [(1, 1), (31, 7), (32, 8), (33, 9), (64, 127), (65, 128), (130, 129), (97, 257), (257, 40)]


@pytest.mark.parametrize("rows_contiguous", [False, True])
@pytest.mark.parametrize("n", [8, 11, 14])
def test_slices(n, rows_contiguous):
    import torch

    from frostspin_b200 import linalg
    from frostspin_b200 import device as dev

    rng = np.random.default_rng(n)
    ops = np.zeros(len(SHAPES), dtype=_native.OZ2_OPERAND_DTYPE)
    keep, hosts, bufs = [], [], []
    for i, (rows, K) in enumerate(SHAPES):
        X = rng.standard_normal((rows, K)) * np.exp(rng.normal(0, 3, (rows, 1)))
        X[rows // 2] *= i % 2
        flat = np.concatenate([[0.0], (X.T if rows_contiguous else X).ravel()])
        d = torch.from_numpy(flat).cuda()
        art, kt = 2 * -(-rows // 256), -(-K // 128)
        sl = torch.full((n * kt * art * 16384,), 99, dtype=torch.int8, device="cuda")
        ex = torch.zeros(rows, dtype=torch.int32, device="cuda")
        bits = linalg.ozaki2_bits(n, K)[0]
        ops[i] = (d.data_ptr() + 8, 1 if rows_contiguous else K, rows if rows_contiguous else 1,
                  sl.data_ptr(), ex.data_ptr(), rows, K, art, kt, bits, 0)
        keep += [d, ex]
        bufs.append(sl)
        hosts.append((X, art, kt, bits))
    d_ops = dev.upload(ops)
    max_units = int((ops["rowtiles"].astype(np.int64) * 4 * ops["ktiles"]).max())
    _native.call("fs_ozaki2_split", d_ops.data_ptr(), ops.size, 257, max_units, n, dev.stream())
    for (X, art, kt, bits), sl in zip(hosts, bufs, strict=True):
        rows, K = X.shape
        e = np.frexp(np.abs(X).max(axis=1))[1]
        A = np.zeros((art * 128, kt * 128), dtype=object)
        scaled = np.rint(np.ldexp(X, (bits - e)[:, None]))
        A[:rows, :K] = np.vectorize(int, otypes=[object])(scaled)
        got = sl.cpu().numpy().reshape(n, kt, art, 128, 8, 16)
        for m, p in enumerate(linalg.OZ2_MODULI[:n]):
            r = np.array(A % p, dtype=np.int64)
            r = np.where(r > (p - 1) // 2, r - p, r).astype(np.int64)
            r = ((r + 128) % 256 - 128).astype(np.int8)   # 128 mod 256 is the byte -128
            tile = r.reshape(art, 128, kt, 8, 16).transpose(2, 0, 1, 3, 4)
            want = np.empty_like(tile)
            for row in range(8):                           # 16-byte chunk c at c ^ (row mod 8)
                for c in range(8):
                    want[:, :, row::8, c ^ row] = tile[:, :, row::8, c]
            assert np.array_equal(got[m], want), (X.shape, p)
