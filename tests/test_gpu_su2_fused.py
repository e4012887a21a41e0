"""The fused SU(2) kernel on synthetic groups at the edges of its forms: every
width of the FP64-pipe and tensor-core products, several pieces with absent
ones, planes and rows with remainders, whole (64-bit) offsets.  Expected values:
the numpy application of the same tables.  A product of K terms differs by at
most (K + 2) eps sum |u| |x| whatever the order of its sum."""

import numpy as np
import pytest

from frostspin_b200._native import SU2_GROUP_DTYPE, SU2_PIECE_DTYPE
from frostspin_b200.symmetric_tensor import su2_fused_plan as sp
from frostspin_b200.symmetric_tensor.abelian_plan import magic_divisor

pytestmark = pytest.mark.gpu

WIDTHS = [1, 2, 3, 4, 5, 6, 7, 8, 9, 12, 13, 16, 17, 20, 21, 24, 25, 31, 32]
DIMS = [(), (1000,), (33, 3), (3, 5, 7), (2, 9, 1, 31), (4, 3, 2, 5, 6), (2, 5000)]


def _strides(shape):
    return np.cumprod([1, *shape[::-1]])[::-1][1:].astype(np.int64)


def _split(rng, total):
    """total = sum of sr * sc over a few pieces."""
    out = []
    while total:
        n = int(rng.integers(1, total + 1)) if len(out) < 6 else total
        sr = int(rng.choice([d for d in range(1, n + 1) if n % d == 0]))
        out.append((sr, n // sr))
        total -= n
    return out


def _tables(rng, widths, dims_of, reverse):
    groups, pieces, src_size, out_size, u_size = [], [[], []], 0, 0, 0
    sizes = [0, 0]
    for K in widths:
        dims = dims_of(K)
        nd = len(dims)
        g = np.zeros((), dtype=SU2_GROUP_DTYPE)
        g["u_off"], g["ncols"], g["ndim"], g["M"], g["K"] = u_size, int(np.prod(dims)), nd, K, K
        g["dims"] = 1
        g["dims"][:nd] = dims
        m, s = magic_divisor(np.maximum(g["dims"].astype(np.int64), 1))
        g["divm"], g["divs"] = m, s
        u_size += K * K
        for side in (0, 1):
            row = 0
            first = len(pieces[side])
            for i, (sr, sc) in enumerate(_split(rng, K)):
                order = rng.permutation(nd)            # order of the legs in the buffer
                shape = [sr, *[dims[j] for j in order], sc] if sc % 2 else [
                    sr, sc, *[dims[j] for j in order]]
                st = _strides(shape)
                p = np.zeros((), dtype=SU2_PIECE_DTYPE)
                p["sr"], p["sc"], p["row0"] = sr, sc, row
                p["sr_stride"] = st[0]
                p["sc_stride"] = st[-1] if sc % 2 else st[1]
                legs = st[1:-1] if sc % 2 else st[2:]
                base = sizes[side]
                for j, x in zip(order, legs, strict=True):
                    p["ext"][j] = x
                if reverse and nd:
                    j = nd - 1                         # innermost output leg backwards
                    base += (dims[j] - 1) * int(p["ext"][j])
                    p["ext"][j] *= -1
                p["base"] = -1 if side == 0 and i == 1 and K % 3 == 0 else base
                sizes[side] += int(np.prod(shape))
                row += sr * sc
                pieces[side].append(p)
            g["in_first" if side == 0 else "out_first"] = first
            g["in_count" if side == 0 else "out_count"] = len(pieces[side]) - first
        groups.append(g)
    gtab = np.array(groups, dtype=SU2_GROUP_DTYPE)
    gtab["out_first"] += len(pieces[0])
    ptab = np.array(pieces[0] + pieces[1], dtype=SU2_PIECE_DTYPE)
    return gtab, ptab, u_size, sizes[0], sizes[1]


@pytest.mark.parametrize("reverse", [False, True])
@pytest.mark.parametrize("case", range(len(DIMS)))
def test_every_width(case, reverse):
    import torch

    from frostspin_b200 import _native
    from frostspin_b200 import device as dev

    rng = np.random.default_rng(10 * case + reverse)
    gtab, ptab, n_u, n_src, n_out = _tables(rng, WIDTHS, lambda K: DIMS[(case + K) % len(DIMS)],
                                            reverse)
    tasks = sp.make_tasks(gtab)
    if not reverse:
        sp.check(gtab, ptab, n_src, n_out, n_u)
    U, src = rng.standard_normal(n_u), rng.standard_normal(n_src)
    want = sp.emulate(gtab, ptab, tasks, U, src, np.full(n_out, np.nan))
    scale = sp.emulate(gtab, ptab, tasks, np.abs(U), np.abs(src), np.full(n_out, np.nan))
    assert not np.isnan(want).any()
    d = [dev.upload(a) for a in (gtab, ptab, tasks)]
    d_u, d_src = dev.upload_f64(U), dev.upload_f64(src)
    out = torch.full((n_out,), float("nan"), dtype=torch.float64, device="cuda")
    flag = torch.zeros(1, dtype=torch.int32, device="cuda")
    _native.call("fs_su2_permute_fused", d_src.data_ptr(), n_src, out.data_ptr(), n_out,
                 d[0].data_ptr(), gtab.size, d[1].data_ptr(), ptab.size, d_u.data_ptr(), n_u,
                 d[2].data_ptr(), tasks.size, flag.data_ptr(), dev.stream())
    got = out.cpu().numpy()
    assert int(flag.item()) == 0
    assert np.all(np.abs(got - want) <= (max(WIDTHS) + 2) * np.finfo(float).eps * scale)
