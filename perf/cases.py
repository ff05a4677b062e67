"""The work a user of the package has it do, as timed cases.

Each case is a dict of plain values; its "kind" names the path:

  solve      HBSMAT.solve of a factored HBS operator (float64, mode N or T)
  apply      HBSMAT.matmat and rmatmat
  refined    HBSMAT.solve_refined(inner='tensor'): a served wide batch
  construct  an interface block compressed from its sketches with the ULV
             interleaved (construct_drawn), then used once: solve and apply
  thomas     BlockTridiagonalSolver: factorize and solve
  rb         RedBlackSolver: factorize and solve
  rb_solve   RedBlackSolver: solve with the factors kept
  rbhbs      RedBlackSolverHBS: factorize (every Schur complement compressed)
             and solve
  grouped    solve_grouped_device over HBS operators of uneven sizes

Operators and right-hand sides are made on the device from the seed: exact
random HBS operators in the layout of sslablu_gb300.synthetic (leaf diagonal
shifted by 16, the I + S form of the interface systems), and Gaussian-kernel
couplings of neighbouring interfaces (as synthetic.slab_couplings, with the
quadrature weight that keeps their norm below 1/2 at every interface size, as
a slab map's is) with the kernel width and offsets drawn.
"""
import math

import numpy as np
import torch

from sslablu_gb300.direct_solve.omsdirectsolve import BlockTridiagonalSolver, RedBlackSolver
from sslablu_gb300.direct_solve.omsdirectsolveHBS import RedBlackSolverHBS, dense_to_linop
from sslablu_gb300.grouped import solve_grouped_device
from sslablu_gb300.matAssembly.HBS.HBSnew import HBSMAT, samples_for
from sslablu_gb300.matAssembly.HBS.slabTree import slabTree

F64 = torch.float64


def listed():
    return [
        # one right-hand side through a short interface: the latency of a call
        {"name": "solve_one", "kind": "solve", "leaf": 64, "levels": 4, "rank": 32, "fac": 2,
         "nrhs": 1, "mode": "N"},
        # the benchmark's operator and batch: N = 4096, leaf 64, rank 32, 16 columns
        {"name": "solve_16", "kind": "solve", "leaf": 64, "levels": 7, "rank": 32, "fac": 2,
         "nrhs": 16, "mode": "N"},
        # a transposed solve as the sampling of a Schur complement does it:
        # the largest interface, one column per sketch sample
        {"name": "solve_sketch_T", "kind": "solve", "leaf": 64, "levels": 8, "rank": 32, "fac": 2,
         "nrhs": 261, "mode": "T"},
        # operator products of both orientations (GMRES, sampling, residuals)
        {"name": "apply_64", "kind": "apply", "leaf": 64, "levels": 7, "rank": 32, "fac": 2,
         "nrhs": 64},
        # a wide served batch solved to 1e-10 on the tensor cores
        {"name": "refined_1024", "kind": "refined", "leaf": 64, "levels": 7, "rank": 32, "fac": 2,
         "nrhs": 1024},
        # compression + ULV of a dense 4096-point interface block (rank 32, leaf 64)
        {"name": "construct_4096", "kind": "construct", "leaf": 64, "levels": 7, "rank": 32,
         "fac": 2, "nrhs": 16},
        # an interface plane (quad tree) with a leaf that is no power of two
        {"name": "construct_quad", "kind": "construct", "leaf": 36, "levels": 4, "rank": 20,
         "fac": 4, "nrhs": 5},
        # eight vertical slabs: 7 interfaces of 256 points, one right-hand side
        {"name": "thomas_256", "kind": "thomas", "m": 256, "nblk": 7, "nrhs": 1},
        # the dense direct solver at 1024-point interfaces: one system factored and solved
        {"name": "rb_1024", "kind": "rb", "m": 1024, "nblk": 8, "nrhs": 64},
        # further right-hand sides through kept factors, a ragged interface
        {"name": "rb_solve_700", "kind": "rb_solve", "m": 700, "nblk": 8, "nrhs": 64},
        # the HBS direct solver: four slabs, 512-point interfaces
        {"name": "rbhbs_512", "kind": "rbhbs", "m": 512, "nblk": 4, "leaf": 64, "rank": 24,
         "nrhs": 16},
        # a batch of uneven interface operators, 8 columns each, in one call
        {"name": "grouped_48", "kind": "grouped", "count": 48, "nrhs": 8, "rank_lo": 16,
         "rank_hi": 48, "sizes_lo": 128, "sizes_hi": 2048},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["solve", "solve", "apply", "refined", "construct", "construct", "thomas",
                       "rb", "rb_solve", "rbhbs", "grouped"])
    if kind in ("solve", "apply"):
        c = {"kind": kind, "leaf": rng.randint(24, 80), "rank": rng.randint(8, 40), "fac": 2,
             "levels": rng.randint(2, 7), "nrhs": _log(rng, 1, 261)}
        if kind == "solve":
            c["mode"] = rng.choice(["N", "T"])
        return c
    if kind == "refined":
        return {"kind": kind, "leaf": rng.randint(40, 80), "rank": rng.randint(8, 40), "fac": 2,
                "levels": rng.randint(4, 7), "nrhs": _log(rng, 256, 1024)}
    if kind == "construct":
        if rng.random() < 0.35:
            return {"kind": kind, "leaf": rng.randint(24, 40), "rank": rng.randint(8, 20),
                    "fac": 4, "levels": rng.randint(2, 4), "nrhs": _log(rng, 1, 32)}
        return {"kind": kind, "leaf": rng.randint(32, 64), "rank": rng.randint(8, 32), "fac": 2,
                "levels": rng.randint(3, 7), "nrhs": _log(rng, 1, 32)}
    if kind == "thomas":
        return {"kind": kind, "m": _log(rng, 24, 512), "nblk": rng.randint(2, 9),
                "nrhs": _log(rng, 1, 64)}
    if kind in ("rb", "rb_solve"):
        return {"kind": kind, "m": _log(rng, 48, 1000), "nblk": rng.choice([2, 4, 8]),
                "nrhs": _log(rng, 1, 100)}
    if kind == "rbhbs":
        leaf = rng.choice([32, 48, 64])
        return {"kind": kind, "m": leaf * rng.choice([2, 4, 8]), "nblk": rng.choice([2, 4]),
                "leaf": leaf, "rank": rng.randint(14, 26), "nrhs": _log(rng, 1, 64)}
    return {"kind": "grouped", "count": _log(rng, 4, 48), "nrhs": rng.randint(1, 16),
            "rank_lo": 16, "rank_hi": rng.randint(20, 48), "sizes_lo": 128,
            "sizes_hi": rng.choice([512, 1024, 2048])}


# ---------------------------------------------------------------- inputs
def _gen(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(1000003 * int(seed) + 17)
    return g


def _randn(g, *shape):
    return torch.randn(shape, generator=g, dtype=F64, device="cuda")


def _orth(g, nb, n, k):
    return torch.linalg.qr(_randn(g, nb, n, k))[0]


def _hbs_factors(case, g):
    """(U, D, V, Nbvec) of an exact random HBS operator, blocks as (Nb, n, .)
    tensors: orthonormal U and V, Gaussian D projected off them below the
    root, singular values of the leaf couplings 1 -> 1e-12, D + 16 I."""
    nl, L, k, fac = case["leaf"], case["levels"], case["rank"], case["fac"]
    U, D, V, Nbvec = [], [], [], []
    nb, n = fac ** (L - 1), nl
    for t in range(L):
        kk = min(k, nl) if t == 0 else k
        d = _randn(g, nb, n, n)
        if t < L - 1:
            u, v = _orth(g, nb, n, kk), _orth(g, nb, n, kk)
            d = d - u @ (u.mT @ d @ v) @ v.mT
            if t == 0:
                u = u * (10.0 ** (-12.0 * torch.arange(kk, device="cuda", dtype=F64)
                                  / max(kk - 1, 1)))
            U.append(u)
            V.append(v)
        if t == 0:
            d = d + 16.0 * torch.eye(n, dtype=F64, device="cuda")
        D.append(d)
        Nbvec.append(nb)
        nb, n = nb // fac, fac * kk
    return U, D, V, Nbvec


def _flat(m):
    return m.reshape(-1, m.shape[-1])


def _hbs_op(case, g):
    U, D, V, Nbvec = _hbs_factors(case, g)
    H = HBSMAT().set_mats([_flat(u) for u in U], [_flat(d) for d in D], [_flat(v) for v in V],
                          Nbvec, fac=case["fac"])
    H.compute_ULV()
    return H


def _hbs_size(case):
    return case["leaf"] * case["fac"] ** (case["levels"] - 1)


def _hbs_dense(U, D, V):
    """The dense matrix of an HBS operator (tree order)."""
    A = D[-1][0]
    for t in range(len(D) - 2, -1, -1):
        nb, n, k = U[t].shape
        A = A.reshape(nb, k, nb, k)
        A = torch.einsum("aik,akbl->aibl", U[t], A)
        A = torch.einsum("aibl,bjl->aibj", A, V[t]).contiguous()
        i = torch.arange(nb, device="cuda")
        A[i, :, i, :] += D[t]
        A = A.reshape(nb * n, nb * n)
    return A


def _tree(case):
    """A tree over the points of an interface: a line (binary) or a square
    plane (quad), with the case's leaf size and depth."""
    nl, L = case["leaf"], case["levels"]
    if case["fac"] == 2:
        N = nl * 2 ** (L - 1)
        XX = np.stack([np.zeros(N), (np.arange(N) + 0.5) / N], 1)
        return slabTree(XX, False, nl)
    side = 2 ** (L - 1)
    c = (np.arange(side) + 0.5) / side
    # nl points in every cell of a side x side grid
    r = np.random.default_rng(7).uniform(-0.4 / side, 0.4 / side, (nl, 2))
    cells = np.stack(np.meshgrid(c, c, indexing="ij"), -1).reshape(-1, 1, 2)
    XX = (cells + r[None]).reshape(-1, 2)
    return slabTree(np.concatenate([np.full((XX.shape[0], 1), 0.5), XX], 1), True, nl)


class _FixedTree:
    """The tree of an operator whose points are already in leaf order."""

    def __init__(self, N, leaves, levels):
        self.perm_leaf = np.arange(N)
        self.nleaves = leaves
        self.nlevels = levels


def _construct_tree(case):
    N = _hbs_size(case)
    if case["fac"] == 2:
        t = _tree(case)
        if t.nleaves == 2 ** (case["levels"] - 1) and t.nlevels == case["levels"]:
            return t
    return _FixedTree(N, case["fac"] ** (case["levels"] - 1), case["levels"])


def _construct_inputs(case, seed):
    g = _gen(seed)
    U, D, V, _ = _hbs_factors(case, g)
    tree = _construct_tree(case)
    A = torch.empty((_hbs_size(case),) * 2, dtype=F64, device="cuda")
    p = torch.as_tensor(np.asarray(tree.perm_leaf), device="cuda")
    A[p[:, None], p[None, :]] = _hbs_dense(U, D, V)
    N, s = A.shape[0], samples_for(case["rank"], case["leaf"], case["fac"])
    return A, tree, _randn(g, N, s), _randn(g, N, s), _randn(g, N, case["nrhs"])


def _couplings(case, seed):
    """[(S_{i,i-1}, S_{i,i+1})] of an interface system I + S and its
    right-hand sides: 1.2 / m exp(-c (x - y -+ d_i)^2), zero outer blocks."""
    g, m, n = _gen(seed), case["m"], case["nblk"]
    x = torch.linspace(0, 1, m, dtype=F64, device="cuda")
    r = torch.rand((n, 4), generator=g, dtype=F64, device="cuda")

    def blk(c, d):
        return 1.2 / m * torch.exp(-(15.0 + 10.0 * c) * (x[:, None] - x[None, :] - d) ** 2)
    zero = torch.zeros((m, m), dtype=F64, device="cuda")
    S = []
    for i in range(n):
        S.append((blk(r[i, 0], 0.15 + 0.1 * r[i, 1]) if i > 0 else zero,
                  blk(r[i, 2], -0.15 - 0.1 * r[i, 3]) if i < n - 1 else zero))
    return S, _randn(g, m * n, case["nrhs"])


def _group_members(case, seed):
    """Sizes and ranks of a batch come from its shape alone; the values of
    the operators from the seed."""
    rng = np.random.default_rng([case["count"], case["rank_hi"], case["sizes_hi"]])
    sizes = [n for n in (128, 256, 512, 1024, 2048) if case["sizes_lo"] <= n <= case["sizes_hi"]]
    return [{"leaf": 64, "levels": int(math.log2(int(rng.choice(sizes)) // 64)) + 1, "fac": 2,
             "rank": int(rng.integers(case["rank_lo"], case["rank_hi"] + 1)),
             "nrhs": case["nrhs"]} for _ in range(case["count"])]


# ---------------------------------------------------------------- the passes
def prepare(case, seed):
    kind = case["kind"]
    if kind in ("solve", "apply", "refined"):
        g = _gen(seed)
        H = _hbs_op(case, g)
        return {"case": case, "H": H, "b": _randn(g, _hbs_size(case), case["nrhs"])}
    if kind == "construct":
        A, tree, Om, Psi, b = _construct_inputs(case, seed)
        return {"case": case, "A": A, "tree": tree, "Om": Om, "Psi": Psi, "b": b}
    if kind in ("thomas", "rb", "rb_solve"):
        S, b = _couplings(case, seed)
        st = {"case": case, "S": S, "b": b}
        if kind == "rb_solve":
            st["solver"] = RedBlackSolver(case["m"])
            st["solver"].factorize(S, None)
        return st
    if kind == "rbhbs":
        S, b = _couplings(case, seed)
        levels = int(math.log2(case["m"] // case["leaf"])) + 1
        tree = _construct_tree({"leaf": case["leaf"], "levels": levels, "fac": 2})
        ops = []
        for row in S:
            pair = [dense_to_linop(B) for B in row]
            for o in pair:
                o.tree, o.quad = tree, False
            ops.append(pair)
        return {"case": case, "ops": ops, "tree": tree, "b": b}
    g = _gen(seed)
    members = _group_members(case, seed)
    Hs = [_hbs_op(m, g) for m in members]
    return {"case": case, "Hs": Hs, "bs": [_randn(g, _hbs_size(m), m["nrhs"]) for m in members]}


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "solve":
        return state["H"].solve(state["b"], mode=case["mode"])
    if kind == "apply":
        return {"Ax": state["H"].matmat(state["b"]), "ATx": state["H"].rmatmat(state["b"])}
    if kind == "refined":
        return state["H"].solve_refined(state["b"], tol=1e-10, inner="tensor")[0]
    if kind == "construct":
        H = HBSMAT(state["A"], state["tree"], case["fac"] == 4)
        H.construct_drawn(case["rank"], state["Om"], state["Psi"])
        return {"x": H.solve(state["b"]), "Ax": H.matmat(state["b"])}
    if kind == "thomas":
        s = BlockTridiagonalSolver(case["m"])
        s.factorize(state["S"], None)
        return s.solve(state["b"])
    if kind == "rb":
        s = RedBlackSolver(case["m"])
        s.factorize(state["S"], None)
        return s.solve(state["b"])
    if kind == "rb_solve":
        return state["solver"].solve(state["b"])
    if kind == "rbhbs":
        s = RedBlackSolverHBS(case["m"], case["rank"], state["tree"], False, sketch_seed=5)
        s.factorize(state["ops"])
        return s.solve(state["b"])
    return solve_grouped_device(state["Hs"], [b.clone() for b in state["bs"]])


# ---------------------------------------------------------------- what a pass needs
def _hbs_work(case, both):
    """Bytes of the operator's U, V, D and of the vectors; flops of one pass
    over the tree: an apply multiplies by D, U and V, a solve (Q^T, then
    [W R^-1; its D product]) by about twice as many entries."""
    nb, n, byt, fl = case["fac"] ** (case["levels"] - 1), case["leaf"], 0, 0
    for t in range(case["levels"]):
        k = min(case["rank"], case["leaf"]) if t == 0 else case["rank"]
        if t == case["levels"] - 1:
            byt, fl = byt + 8 * n * n, fl + (4 if both else 2) * n * n
        else:
            byt += 8 * nb * (n * n + 2 * n * k)
            fl += 2 * nb * (n * n + (2 if t and both else 1) * n * (n + k) if both
                            else n * n + 2 * n * k)
        nb, n = nb // case["fac"], case["fac"] * k
    c, N = case["nrhs"], _hbs_size(case)
    return byt + 16 * N * c, fl * c


def work(case):
    kind = case["kind"]
    if kind == "solve":
        b, f = _hbs_work(case, True)
        return {"bytes": b, "flops": f}
    if kind == "apply":
        b, f = _hbs_work(case, False)
        return {"bytes": b + 8 * _hbs_size(case) * case["nrhs"], "flops": 2 * f}
    if kind == "refined":
        (b, f), (_, r) = _hbs_work(case, True), _hbs_work(case, False)
        return {"bytes": b, "flops": f + r}
    if kind == "construct":
        N, s = _hbs_size(case), samples_for(case["rank"], case["leaf"], case["fac"])
        (b, f), (_, r) = _hbs_work(case, True), _hbs_work(case, False)
        # sampling with the dense block both ways; per level two QRs of the
        # s x n sketch blocks with the samples carried, two SVDs, the ULV
        fl, nb, n = 4.0 * N * N * s, case["fac"] ** (case["levels"] - 1), case["leaf"]
        for t in range(case["levels"]):
            fl += nb * (2 * (2.0 * s * n * n + 4.0 * s * n * n + 12.0 * n ** 3) + 10.0 * n ** 3)
            nb, n = nb // case["fac"], case["fac"] * min(case["rank"], case["leaf"])
        return {"bytes": 8.0 * N * N + 16.0 * N * s + b, "flops": fl + f + r}
    if kind == "grouped":
        parts = [_hbs_work(m, True) for m in _group_members(case, 0)]
        return {"bytes": sum(p[0] for p in parts), "flops": sum(p[1] for p in parts)}
    m, n, c = float(case["m"]), case["nblk"], case["nrhs"]
    vec = 16.0 * m * n * c
    sol = (6.0 * n - 4.0) * m * m * c
    if kind == "thomas":
        return {"bytes": 16.0 * (n - 1) * m * m + vec,
                "flops": n * 2.0 / 3.0 * m ** 3 + (n - 1) * 4.0 * m ** 3 + sol}
    if kind == "rb":
        return {"bytes": 16.0 * (n - 1) * m * m + vec,
                "flops": (2 * n - 1) * 2.0 / 3.0 * m ** 3 + (n - 1) * 12.0 * m ** 3 + 2 * sol}
    if kind == "rb_solve":
        return {"bytes": 24.0 * (2 * n - 1) * m * m + vec, "flops": 2 * sol}
    # rbhbs: the sampling products with the dense couplings at the first
    # level, and three compressions per eliminated block
    N, s = m, samples_for(case["rank"], case["leaf"], 2)
    one, nb, w = 0.0, case["m"] // case["leaf"], float(case["leaf"])
    while nb:
        one += nb * (12.0 * s * w * w + 34.0 * w ** 3)
        nb, w = nb // 2, 2.0 * min(case["rank"], case["leaf"])
    return {"bytes": 16.0 * (n - 1) * m * m + vec,
            "flops": (n - 1) * 3 * one + 12.0 * n * N * N * s + sol}


# ---------------------------------------------------------------- in 64 bits
def _dense_of(case, g):
    U, D, V, _ = _hbs_factors(case, g)
    return _hbs_dense(U, D, V)


def exact(case, seed):
    kind = case["kind"]
    if kind in ("solve", "apply", "refined"):
        g = _gen(seed)
        A = _dense_of(case, g)
        b = _randn(g, _hbs_size(case), case["nrhs"])
        if kind == "apply":
            return {"Ax": A @ b, "ATx": A.mT @ b}
        return torch.linalg.solve(A.mT if case.get("mode") == "T" else A, b)
    if kind == "construct":
        A, _, _, _, b = _construct_inputs(case, seed)
        return {"x": torch.linalg.solve(A, b), "Ax": A @ b}
    if kind == "grouped":
        g = _gen(seed)
        members = _group_members(case, seed)
        As = [_dense_of(m, g) for m in members]
        return [torch.linalg.solve(A, _randn(g, _hbs_size(m), m["nrhs"]))
                for A, m in zip(As, members)]
    S, b = _couplings(case, seed)
    m, n = case["m"], case["nblk"]
    A = torch.eye(m * n, dtype=F64, device="cuda")
    for i, (lo, up) in enumerate(S):
        if i > 0:
            A[i * m:(i + 1) * m, (i - 1) * m:i * m] = lo
        if i < n - 1:
            A[i * m:(i + 1) * m, (i + 1) * m:(i + 2) * m] = up
    return torch.linalg.solve(A, b)
