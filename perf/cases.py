"""Performance cases of the symmetric-tensor operations and of one CTMRG iteration.

A case is a dict of plain values.  `op` names the operation of the public API it
runs, `sym` the symmetry, the other entries its sizes:

  permute   SymmetricTensor.permute (abelian, SU(2) and O(2))
  matmul    A @ B over shared sectors, at a GEMM precision of
            linalg.set_gemm_precision
  contract  norm, full contraction and trace of enlarged corners (observables)
  absorb    bond weights on a leg, then normalisation (simple update, CTMRG)
  corner    ctm_contract.contract_ul: one enlarged corner of the double layer
  ctmrg     SequentialCTMRG.iterate and the reduced density matrices

Legs: a U(1) leg of n states carries charges around 0 with Gaussian
degeneracies, an SU(2) or O(2) leg the lowest irreps.  Site tensors have the
leg order (physical, ancilla | up, right, down, left), edges (chi | D, D, chi)
and corners (chi | chi).
"""

import math

import numpy as np
import torch

from frostspin_b200 import O2SymmetricTensor, SU2SymmetricTensor, U1SymmetricTensor, linalg
from frostspin_b200.ctmrg import SequentialCTMRG
from frostspin_b200.ctmrg.ctm_contract import contract_ul
from frostspin_b200.symmetric_tensor import DiagonalTensor

CLASSES = {"U1": U1SymmetricTensor, "SU2": SU2SymmetricTensor, "O2": O2SymmetricTensor}

# leg permutations of the CTMRG moves: name -> (row axes, column axes)
AXES = {
    "pair": ((0, 2), (1, 3)),            # two-site matrix of a rank-4 tensor
    "turn": ((3, 1, 2), (0,)),           # edge seen from its other end: the last leg moves first
    "fuse": ((1, 2, 0), (3,)),           # edge as (D, D, chi | chi)
    "bond": ((0, 1, 4, 5), (2, 3)),      # site tensor with two bonds as columns
    "corner": ((2, 0, 4), (3, 1, 5)),    # enlarged corner to (chi, D, D | chi, D, D)
}


# ------------------------------------------------------------------------ legs
def split(total, weights):
    """`total` states over the weights, by largest remainder."""
    raw = np.asarray(weights, dtype=float) / np.sum(weights) * total
    deg = np.floor(raw).astype(int)
    order = np.argsort(deg - raw, kind="stable")
    deg[order[: total - deg.sum()]] += 1
    return deg


def u1_leg(n, step=1):
    """n states with charges that are multiples of `step`, Gaussian degeneracies."""
    qmax = 4 if n >= 48 else 2 if n >= 6 else 1
    q = np.arange(-qmax, qmax + 1)
    return np.repeat(step * q, split(n, np.exp(-(q**2) / 8.0))).astype(np.int8)


def su2_leg(n):
    """Integer spins with about n states in all (a multiplet of irrep d counts d)."""
    d = np.array([1, 3, 5] if n < 32 else [1, 3, 5, 7])
    deg = np.maximum(1, np.rint(n * np.array([0.11, 0.53, 0.36, 0.25])[: d.size] / d / 1.1)).astype(int)
    return np.array([deg, d])


def o2_leg(n):
    """0odd, 0even and the two-dimensional irreps 1 and 2, about n states."""
    deg = np.maximum(1, np.rint(n * np.array([0.15, 0.25, 0.2, 0.1])).astype(int))
    return np.array([deg, [-1, 0, 1, 2]])


def leg(sym, n, step=1):
    return u1_leg(n, step) if sym == "U1" else su2_leg(n) if sym == "SU2" else o2_leg(n)


def physical(sym):
    return np.array([1, -1], dtype=np.int8) if sym == "U1" else np.array([[1], [2]])


def structure(case):
    """The legs of the case's tensors: a list of (row legs, column legs, signature)."""
    op, sym, chi, D = case["op"], case["sym"], case["chi"], case["D"]
    c, b = leg(sym, chi, 2), leg(sym, D, 2)
    F, T = False, True
    if op == "permute" and case["kind"] == "pair":
        c = leg(sym, chi)
        return [((c, c), (c, c), [F, F, T, T])]
    if op == "permute" and case["kind"] == "corner":
        return [((b, b), (b, b, c, c), [F, F, T, T, F, T])]
    if op == "permute" and case["kind"] == "bond" or op == "ctmrg":
        p = physical(sym)
        return [((p, p), (b, b, b, b), [T, F, T, T, T, T])]
    if op == "permute":
        return [((c,), (b, b, c), [F, F, T, T])]
    if op == "matmul" and case["kind"] == "pair":
        c = leg(sym, chi)
        return [((c, c), (c, c), [F, F, T, T]), ((c, c), (c, c), [F, F, T, T])]
    if op == "matmul":  # a chi x chi corner on a wide half network
        return [((c,), (c,), [F, T]), ((c,), (b, b, c, b, b), [F, F, T, T, F, T])]
    if op == "contract":
        return [((c, b, b), (c, b, b), [F, F, T, T, T, F])] * 2
    if op == "absorb":
        return [((b, b, c), (c,), [F, T, F, T])]
    p = physical(sym)
    return [((c,), (c,), [F, T]), ((c,), (b, b, c), [F, F, T, T]), ((c,), (b, b, c), [F, F, T, T]),
            ((p, p), (b, b, b, b), [T, F, T, T, T, T])]


# ----------------------------------------------------------------------- cases
def listed():
    return [
        # a site tensor's legs regrouped, as in every step of every move at small
        # bond dimension: what one call costs
        {"name": "u1_permute_site", "op": "permute", "kind": "bond", "sym": "U1", "chi": 0, "D": 5},
        # an edge tensor turned round, at odd sizes: the innermost leg changes place
        {"name": "u1_permute_turn", "op": "permute", "kind": "turn", "sym": "U1", "chi": 601, "D": 15},
        # the kernel benchmark of the U(1) path: 256 states a leg, 455 M coefficients
        {"name": "u1_permute_pair", "op": "permute", "kind": "pair", "sym": "U1", "chi": 256, "D": 0},
        # an SU(2) enlarged corner brought to matrix form
        {"name": "su2_permute_corner", "op": "permute", "kind": "corner", "sym": "SU2", "chi": 96, "D": 22},
        # O(2): cast, abelian permute, cast back
        {"name": "o2_permute_pair", "op": "permute", "kind": "pair", "sym": "O2", "chi": 89, "D": 0},
        # the sector products of a two-site matrix, ragged, in double precision
        {"name": "u1_matmul_pair", "op": "matmul", "kind": "pair", "sym": "U1", "chi": 77, "D": 0, "precision": "fp64"},
        # a corner applied to a wide half network: short inner sizes, many columns
        {"name": "u1_matmul_wide", "op": "matmul", "kind": "wide", "sym": "U1", "chi": 250, "D": 9, "precision": "fp64"},
        # large sectors on the int8 tensor cores, the default arithmetic of the benchmark
        {"name": "u1_matmul_mixed", "op": "matmul", "kind": "pair", "sym": "U1", "chi": 181, "D": 0, "precision": "ozaki2_11"},
        # observables of an SU(2) environment: norm, contraction and trace of enlarged corners
        {"name": "su2_contract", "op": "contract", "sym": "SU2", "chi": 128, "D": 16},
        # bond weights absorbed and the result normalised, as in each simple-update step
        {"name": "u1_absorb", "op": "absorb", "sym": "U1", "chi": 401, "D": 25},
        # one enlarged corner of the SU(2) double layer, moderate sizes
        {"name": "su2_corner", "op": "corner", "sym": "SU2", "chi": 96, "D": 16, "precision": "fp64"},
        # a whole iteration (four moves) of a small U(1) network and its density matrices
        {"name": "u1_ctmrg", "op": "ctmrg", "sym": "U1", "chi": 24, "D": 3, "precision": "fp64"},
    ]


def draw(rng):
    def size(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    op = rng.choice(["permute", "permute", "permute", "matmul", "matmul", "contract", "absorb", "corner"])
    sym = rng.choice(["U1", "SU2"])
    if op == "permute":
        kind = rng.choice(["bond", "turn", "fuse", "pair", "corner"])
        if kind == "bond":
            return {"op": op, "kind": kind, "sym": sym, "chi": 0, "D": size(3, 28)}
        if kind == "pair":
            sym = rng.choice(["U1", "O2"])
            return {"op": op, "kind": kind, "sym": sym, "chi": size(20, 89 if sym == "O2" else 220), "D": 0}
        if kind == "corner":
            return {"op": op, "kind": kind, "sym": sym, "chi": size(24, 128), "D": size(4, 24 if sym == "SU2" else 9)}
        return {"op": op, "kind": kind, "sym": sym, "chi": size(40, 700), "D": size(4, 28)}
    if op == "matmul":
        if rng.random() < 0.5:
            return {"op": op, "kind": "wide", "sym": sym, "chi": size(30, 256), "D": size(3, 10), "precision": "fp64"}
        chi = size(24, 140)
        return {"op": op, "kind": "pair", "sym": "U1", "chi": chi, "D": 0,
                "precision": rng.choice(["fp64", "ozaki2_11", "ozaki2_13", "ozaki7"])}
    if op == "contract":
        return {"op": op, "sym": sym, "chi": size(24, 160), "D": size(4, 18 if sym == "SU2" else 9)}
    if op == "absorb":
        return {"op": op, "sym": sym, "chi": size(40, 600), "D": size(4, 28)}
    return {"op": op, "sym": sym, "chi": size(16, 96), "D": size(3, 16 if sym == "SU2" else 8), "precision": "fp64"}


# ---------------------------------------------------------------------- inputs
def flats(case, seed):
    """Per tensor of the case: (rows, columns, signature, irreps, shapes, flat device buffer)."""
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed) & 0x7FFFFFFF)
    out = []
    for rows, cols, sig in structure(case):
        sig = np.array(sig)
        irreps, shapes = CLASSES[case["sym"]].get_block_sizes(rows, cols, sig)
        n = int((shapes[:, 0] * shapes[:, 1]).sum())
        x = torch.randn(n, dtype=torch.float64, device="cuda", generator=g)
        if "precision" in case and case["op"] == "matmul":
            # environment tensors: magnitudes fall over a few decades
            x *= torch.pow(10.0, -3 * torch.rand(n, dtype=torch.float64, device="cuda", generator=g))
        out.append((rows, cols, sig, irreps, shapes, x))
    return out


def weights_of(tensor, seed):
    """Positive, decreasing bond weights, one per row of the column leg's blocks."""
    _, cols, _, irreps, shapes, _ = tensor
    g = torch.Generator(device="cuda")
    g.manual_seed((int(seed) & 0x7FFFFFFF) + 1)
    w = []
    for n in shapes[:, 1]:
        u = torch.rand(int(n), dtype=torch.float64, device="cuda", generator=g)
        w.append(torch.exp(-6 * torch.sort(u).values))
    return cols[0], irreps, w


def prepare(case, seed):
    cls = CLASSES[case["sym"]]
    if case["op"] == "ctmrg":
        # the site tensors of the AB/BA cell and an environment under way
        linalg.set_gemm_precision(case["precision"])
        A = site_pair(case, seed)
        ctm = SequentialCTMRG.from_elementary_tensors("AB\nBA", A, case["chi"], cutoff=1e-10, degen_ratio=0.9999)
        ctm.iterate()
        return {"case": case, "ctm": ctm}
    made = flats(case, seed)
    state = {"case": case, "tensors": [cls.from_flat(r, c, x, q, s) for r, c, s, q, _, x in made]}
    if case["op"] == "absorb":
        rep, irreps, w = weights_of(made[0], seed)
        dims = [cls.irrep_dimension(q) for q in irreps]
        state["weights"] = DiagonalTensor(w, rep, irreps, dims, case["sym"])
    return state


def site_pair(case, seed):
    """The two random site tensors of a checkerboard cell."""
    ((rows, cols, sig),) = structure(case)
    rng = np.random.default_rng(int(seed))
    cls = CLASSES[case["sym"]]
    out = []
    for s in (sig, [True, False, False, False, False, False]):
        out.append(cls.random(rows, cols, s, rng=rng))
    return out


def run(state):
    case = state["case"]
    op = case["op"]
    if "precision" in case and linalg.gemm_precision() != case["precision"]:
        linalg.set_gemm_precision(case["precision"])
    if op == "ctmrg":
        ctm = state["ctm"].copy()
        ctm.iterate()
        return [r.data for x, y in ctm.site_coords for r in (ctm.compute_rdm1x2(x, y), ctm.compute_rdm2x1(x, y))]
    ts = state["tensors"]
    if op == "permute":
        return ts[0].permute(*AXES[case["kind"]]).data
    if op == "matmul":
        return (ts[0] @ ts[1]).data
    if op == "contract":
        a, b = ts
        return [a.norm_device(), np.float64(a.full_contract(b)), np.float64(b.trace())]
    if op == "absorb":
        t = ts[0] * state["weights"]
        t /= t.norm_device()
        return t.data
    return contract_ul(*ts).data


# ------------------------------------------------------------------------ work
def products(case):
    """Block sizes (M, N, K) of the case's matrix products."""
    cls = CLASSES[case["sym"]]

    def one(rows, mid, cols, srow, smid, scol):
        qa, sa = cls.get_block_sizes(rows, mid, np.array(srow + smid))
        qb, sb = cls.get_block_sizes(mid, cols, np.array([not s for s in smid] + scol))
        _, i, j = np.intersect1d(qa, qb, return_indices=True)
        return sum(2.0 * int(m) * int(k) * int(n) for (m, k), n in zip(sa[i], sb[j][:, 1], strict=True))

    F, T = False, True
    if case["op"] == "matmul":
        (r, m, s), (_, c, s2) = structure(case)
        return one(r, m, c, s[: len(r)], s[len(r):], s2[len(m):])
    b, c, p = leg(case["sym"], case["D"], 2), leg(case["sym"], case["chi"], 2), physical(case["sym"])
    flops = one((b, b, c), (c,), (c,), [F, T, F], [T], [T])
    flops += one((b, b, c), (c,), (b, b, c), [F, T, F], [T], [F, T, T])
    # the site tensor and its dagger on the rank-6 half
    flops += one((p, p, b, b), (b, b), (b, b, c, c), [T, F, T, T], [T, T], [T, T, F, T])
    flops += one((b, b), (p, p, b, b), (b, b, c, c), [F, F], [F, T, F, F], [T, T, F, T])
    return flops


def work(case):
    cls = CLASSES[case["sym"]]
    n = []
    for rows, cols, sig in structure(case):
        _, s = cls.get_block_sizes(rows, cols, np.array(sig))
        n.append(float((s[:, 0] * s[:, 1]).sum()))
    op = case["op"]
    if op == "permute":
        return {"bytes": 16 * n[0], "flops": 0}
    if op == "contract":
        return {"bytes": 8 * (n[0] + n[1]), "flops": 4 * n[0]}
    if op == "absorb":
        return {"bytes": 16 * n[0], "flops": 4 * n[0]}
    if op == "matmul":
        (r, _, s), (m, c, s2) = structure(case)
        _, sh = cls.get_block_sizes(r, c, np.array(list(s[: len(r)]) + list(s2[len(m):])))
        return {"bytes": 8 * (n[0] + n[1] + float((sh[:, 0] * sh[:, 1]).sum())), "flops": products(case)}
    rows, cols, sig = corner_legs(case)
    _, sh = cls.get_block_sizes(rows, cols, np.array(sig))
    corner = float((sh[:, 0] * sh[:, 1]).sum())
    if op == "corner":
        return {"bytes": 8 * (sum(n) + corner), "flops": products(case)}
    # four moves over two sites: an enlarged corner and three products of
    # corner size for each projector pair, every site and direction
    sec = float((sh[:, 0].astype(float) ** 3).sum())
    return {"bytes": 8 * 8 * (n[0] + 2 * corner), "flops": 8 * (products(case) + 6 * sec)}


# ----------------------------------------------------------------------- exact
def charges(reps, signature):
    """Fused U(1) charges of the legs, C order."""
    q = np.zeros(1, dtype=np.int64)
    for r, s in zip(reps, signature, strict=True):
        q = (q[:, None] + (-1 if s else 1) * r.astype(np.int64)[None, :]).ravel()
    return q


def sectors(rows, cols, sig):
    """Row and column indices of every charge both sides hold, in charge order."""
    sig = np.asarray(sig)
    a, b = charges(rows, sig[: len(rows)]), charges(cols, ~sig[len(rows):])
    return [(np.flatnonzero(a == q), np.flatnonzero(b == q)) for q in np.intersect1d(a, b)]


def to_dense(rows, cols, sig, x):
    m, n = (int(np.prod([r.size for r in rs])) for rs in (rows, cols))
    out = torch.zeros(m, n, dtype=torch.float64, device=x.device)
    at = 0
    for i, j in sectors(rows, cols, sig):
        k = i.size * j.size
        ti, tj = (torch.from_numpy(v).to(x.device) for v in (i, j))
        out[ti[:, None], tj[None, :]] = x[at : at + k].view(i.size, j.size)
        at += k
    return out.view([r.size for r in rows + cols])


def from_dense(rows, cols, sig, t):
    t = t.reshape(int(np.prod([r.size for r in rows])), -1)
    return torch.cat([t[torch.from_numpy(i).to(t.device)][:, torch.from_numpy(j).to(t.device)].reshape(-1)
                      for i, j in sectors(rows, cols, sig)])


def blocks_of(shapes, x):
    at = 0
    for m, n in shapes:
        yield x[at : at + m * n].view(int(m), int(n))
        at += int(m * n)


def exact(case, seed):
    op, sym = case["op"], case["sym"]
    if op == "ctmrg":
        return None
    made = flats(case, seed)
    if op == "contract":
        dims = [abs(int(q)) if sym == "SU2" else 1 for q in made[0][3]]
        a, b = (list(blocks_of(t[4], t[5])) for t in made)
        sums = [math.sqrt(math.fsum(d * float((x * x).sum()) for d, x in zip(dims, a, strict=True))),
                math.fsum(d * float((x * y.T).sum()) for d, x, y in zip(dims, a, b, strict=True)),
                math.fsum(d * float(y.diagonal().sum()) for d, y in zip(dims, b, strict=True))]
        return [np.float64(v) for v in sums]
    if op == "absorb":
        _, irreps, w = weights_of(made[0], seed)
        dims = [abs(int(q)) if sym == "SU2" else 1 for q in irreps]
        out = [x * v for x, v in zip(blocks_of(made[0][4], made[0][5]), w, strict=True)]
        norm = math.sqrt(math.fsum(d * float((x * x).sum()) for d, x in zip(dims, out, strict=True)))
        return torch.cat([x.reshape(-1) / norm for x in out])
    if op == "matmul":
        a, b = made
        out = []
        qb = [int(q) for q in b[3]]
        right = list(blocks_of(b[4], b[5]))
        for q, x in zip(a[3], blocks_of(a[4], a[5]), strict=True):
            if int(q) in qb:
                out.append((x @ right[qb.index(int(q))]).reshape(-1))
        return torch.cat(out)
    if sym != "U1":
        return None  # needs Clebsch-Gordan coefficients
    dense = 1.0
    for r in (made[0][0] + made[0][1] if op == "permute" else (made[1][0] + made[2][0] + made[3][1])):
        dense *= r.size
    if dense > 3e8:
        return None  # the dense tensor would be too large
    full = [to_dense(r, c, s, x) for r, c, s, _, _, x in made]
    if op == "permute":
        rows, cols, sig, _, _, _ = made[0]
        ra, ca = AXES[case["kind"]]
        legs = rows + cols
        return from_dense(tuple(legs[i] for i in ra), tuple(legs[i] for i in ca), sig[list(ra + ca)],
                          full[0].permute(ra + ca))
    C, T1, T4, A = full
    half = torch.einsum("xuvb,bc,clmy->xuvlmy", T1, C, T4)
    one = torch.einsum("paurdl,xuvlmy->pardxvmy", A, half)
    both = torch.einsum("pavRSm,pardxvmy->rRxdSy", A, one)
    return from_dense(*corner_legs(case), both)


def corner_legs(case):
    c, b = leg(case["sym"], case["chi"], 2), leg(case["sym"], case["D"], 2)
    return (b, b, c), (b, b, c), [True, False, False, True, False, True]
