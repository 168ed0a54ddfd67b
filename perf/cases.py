"""The calls whose speed this framework stands for, each through its public Python API.

A two-site DMRG program spends its time in a handful of calls: the contraction of two site
tensors, the effective-Hamiltonian matvec, the environment update, the sector SVD with
truncation (and the plain one of ``bMPS.move_oc``), now and then an ``eigh``, and the
``dmrg`` driver that strings them together.  The cases below are those calls over the sizes
the models of ``networks`` and ``bench.py`` are run at (bond dimensions from a few dozen to
4096, U(1) and U(1) x U(1) charges) and in the three block-GEMM precisions.

``listed`` names a dozen of them, ``draw`` draws others from the same ranges.  Results stay
on the device as btensor handles, as in a user's program; ``Read`` downloads one when its
numbers are asked for.  Singular and eigenvectors are determined only up to signs, so a
decomposition is read as its values, the product of its factors and the factors' Gram
matrices.
"""
import functools
import itertools
import math

import numpy as np
import torch

import quantit_gb300 as q
from quantit_gb300 import algorithms, linalg, networks
from quantit_gb300.conserved import Z, ZZ

CUTOFF = 1e-10          # the truncation cutoff of bench.py's sweeps
CYL_LX, CYL_LY = 4, 6   # the 6-leg cylinder of bench.py, cut to the length its middle bond needs


# --------------------------------------------------------------------------- results
class Read(list):
    """The numbers of a result that lives on the device: an iterable of arrays, downloaded
    when it is iterated."""

    def __init__(self, get):
        super().__init__()
        self._get = get

    def __iter__(self):
        return iter(self._get())


def flat(t):
    """All blocks of a btensor in block-list order, as one array."""
    b = t.blocks()
    return np.concatenate([v.ravel() for _, v in b]) if b else np.zeros(0)


def read_tensor(t):
    return Read(lambda: [flat(t)])


def sector_sizes(theta, split):
    """{left charge: (rows, columns)} of the sector matrices of a tensor split after ``split`` legs."""
    sbd, ssz, cv, _ = theta.structure()
    first = np.concatenate([[0], np.cumsum(sbd)]).astype(int)
    out = {}
    for k in theta.block_indices():
        at = [int(first[d]) + i for d, i in enumerate(k)]
        charge = sum(cv[a].values[0] for a in at[:split])
        rows, cols = out.setdefault(charge, ({}, {}))
        rows[k[:split]] = math.prod(ssz[a] for a in at[:split])
        cols[k[split:]] = math.prod(ssz[a] for a in at[split:])
    return {c: (sum(r.values()), sum(n.values())) for c, (r, n) in sorted(out.items())}


def padded(x, n):
    """x in the leading corner of zeros of size n along every axis: a truncated result in the
    room of the whole one."""
    out = np.zeros([n] * x.ndim)
    out[tuple(slice(0, m) for m in x.shape)] = x
    return out


def read_svd(theta, U, d, V, split):
    """Values in descending order, U diag(d) V^T on theta's blocks, U^T U and V^T V."""
    def get():
        full = [min(mn) for mn in sector_sizes(theta, split).values()]
        dv = {k[0]: torch.from_numpy(v).cuda() for k, v in d.blocks()}
        rows, cols = {}, {}
        for side, out in ((U, rows), (V, cols)):
            for k, v in side.blocks():
                out.setdefault(k[-1], []).append((k[:-1], torch.from_numpy(v).cuda().reshape(-1, v.shape[-1])))
        prod = {}
        for s, val in dv.items():
            for (ku, u), (kv, v) in itertools.product(rows[s], cols[s]):
                p = (u * val) @ v.T
                prod[ku + kv] = prod[ku + kv] + p if ku + kv in prod else p
        sizes = theta._sizes()
        parts = []
        for k in theta.block_indices():
            n = math.prod(theta._shape_of(sizes, k))
            parts.append(prod[k].reshape(-1).cpu().numpy() if k in prod else np.zeros(n))
        grams = []
        for side in (rows, cols):
            g = [padded(sum(b.T @ b for _, b in side[s]).cpu().numpy() if s in dv else np.zeros((0, 0)), n).ravel()
                 for s, n in enumerate(full)]
            grams.append(np.concatenate(g))
        values = np.sort(np.concatenate([v.cpu().numpy() for v in dv.values()]))[::-1]
        return [padded(values, sum(full)), np.concatenate(parts)] + grams
    return Read(get)


def read_eigh(rho, d, U):
    """Eigenvalues in ascending order, U diag(d) U^T on rho's blocks, U^T U."""
    def get():
        dv = {k[0]: torch.from_numpy(v).cuda() for k, v in d.blocks()}
        vec = {k[-1]: (k[0], torch.from_numpy(v).cuda()) for k, v in U.blocks()}
        prod = {}
        for s, val in dv.items():
            row, u = vec[s]
            prod[row] = (u * val) @ u.T
        parts = [prod[k[0]].reshape(-1).cpu().numpy() for k in rho.block_indices()]
        gram = np.concatenate([(vec[s][1].T @ vec[s][1]).reshape(-1).cpu().numpy() for s in sorted(dv)])
        values = np.sort(np.concatenate([v.cpu().numpy() for v in dv.values()]))
        return [values, np.concatenate(parts), gram]
    return Read(get)


def dense(t):
    sizes = t._sizes()
    sbd, ssz = sizes
    offs, a = [], 0
    for n in sbd:
        offs.append(np.concatenate([[0], np.cumsum(ssz[a:a + n])]).astype(int))
        a += n
    out = np.zeros([int(o[-1]) for o in offs])
    for k, v in t.blocks():
        out[tuple(slice(offs[d][i], offs[d][i + 1]) for d, i in enumerate(k))] = v
    return out


def read_state(mps):
    """The state vector of a short chain (its MPS is determined only up to a gauge)."""
    def get():
        psi = np.ones((1, 1))
        for t in mps:
            a = dense(t)
            psi = (psi @ a.reshape(a.shape[0], -1)).reshape(-1, a.shape[2])
        return [psi.ravel()]
    return Read(get)


# --------------------------------------------------------------------------- inputs
def bond(D, parity=0, width=3.4):
    """A bond leg of a spin-1/2 chain: total dimension D over the charges 2Sz of one parity,
    Gaussian section sizes of the width seen on the 6 x 12 cylinder at D = 2048."""
    qs = [c for c in range(-12, 13) if (c - parity) % 2 == 0]
    w = np.exp(-np.array(qs, dtype=float) ** 2 / (2 * width * width))
    raw = D * w / w.sum()
    n = np.floor(raw).astype(int)
    for i in np.argsort(-(raw - n), kind="stable")[:D - int(n.sum())]:
        n[i] += 1
    return [(int(m), c) for m, c in zip(n, qs) if m > 0]


PHYS = [(1, 1), (1, -1)]


def inverse(leg):
    return [(n, -c) for n, c in leg]


def tensor(legs, blocks):
    return q.from_blocks([[(n, Z(c)) for n, c in leg] for leg in legs], Z(0), blocks)


def blocks_of(legs):
    """(index, shape) of every block the charges allow."""
    for idx in itertools.product(*[range(len(leg)) for leg in legs]):
        if sum(leg[i][1] for leg, i in zip(legs, idx)) == 0:
            yield idx, tuple(leg[i][0] for leg, i in zip(legs, idx))


def site_legs(D):
    """Two neighbouring site tensors A(a, s, b), B(b, t, c) in the bulk of a chain."""
    a, b = bond(D, 0), bond(D, 1)
    return [a, PHYS, inverse(b)], [b, PHYS, inverse(a)]


def site_pair(D, seed):
    rng = np.random.default_rng(seed)
    out = []
    for legs in site_legs(D):
        out.append(tensor(legs, [(k, rng.standard_normal(s)) for k, s in blocks_of(legs)]))
    return out


def schmidt(leg, decay):
    """Falling weights of a bond leg's states, section by section: ``decay`` decades, steep
    first and flatter later, the outer sections smaller."""
    return [10.0 ** (-decay * (np.arange(n) / n) ** 0.6 - 0.1 * abs(c)) for n, c in leg]


def graded_theta(D, decay, seed):
    """A two-site tensor theta(a, s, t, c) = lambda_a G lambda_c, G Gaussian: its outer legs
    carry the Schmidt weights of the neighbouring bonds, as in a DMRG state, and its singular
    values fall over about ``decay`` decades (8 on the 6-leg cylinder; 14, into FP64's
    resolution, on the chain)."""
    rng = np.random.default_rng(seed)
    left, right = bond(D, 0), inverse(bond(D, 0))
    lw, rw = schmidt(left, decay / 2), schmidt(right, decay / 2)
    out = []
    for k, shp in blocks_of([left, PHYS, PHYS, right]):
        out.append((k, lw[k[0]][:, None, None, None] * rng.standard_normal(shp) * rw[k[3]]))
    norm = math.sqrt(sum(float(np.sum(x * x)) for _, x in out))
    return tensor([left, PHYS, PHYS, right], [(k, x / norm) for k, x in out])


def symmetric(D, seed):
    """A symmetric rank-2 tensor, charge sector by charge sector (an operator on a bond)."""
    rng = np.random.default_rng(seed)
    leg = bond(D, 0)
    blocks = []
    for i, (n, _) in enumerate(leg):
        x = rng.standard_normal((n, n))
        blocks.append(((i, i), (x + x.T) / math.sqrt(8.0 * n)))
    return tensor([leg, inverse(leg)], blocks)


@functools.lru_cache(maxsize=None)
def model(name, D):
    """(MPO, total charge) of a chain long enough for its middle bond to reach D."""
    if name == "cylinder":
        return networks.cylinder_heisenberg(CYL_LX, CYL_LY, 1.0, "snake", compress=True), Z(0)
    if name == "hubbard":
        L = 2 * math.ceil(math.log(max(D, 4), 4)) + 4
        return networks.hubbard(L, 4.0), ZZ(L, 0)
    L = 2 * math.ceil(math.log2(max(D, 4))) + 4
    return networks.heisenberg(L), Z(0)


def chain_state(case, seed):
    """The pieces of a bond update in the middle of a model's chain, on a random MPS."""
    mpo, total = model(case["model"], case["D"])
    mps = networks.random_bMPS(case["D"], mpo, total, seed=int(seed))
    b = len(mpo) // 2 - 1
    q.set_gemm_mode("f64")
    left, right = algorithms.environments(mpo, mps, [b])[b]
    if case["kind"] == "env":
        return {"W": mpo[b], "A": mps[b], "L": left}
    return {"theta": mps[b].tensordot(mps[b + 1], ([2], [0])),
            "H": algorithms.compute_2sites_hamil(mpo[b], mpo[b + 1]), "L": left, "R": right}


# --------------------------------------------------------------------------- the cases
def listed():
    return [
        # theta = A(b) B(b+1) of a short or low-entangled chain: the smallest call, all latency
        {"name": "dot_f64_site_24", "kind": "site", "mode": "f64", "D": 24},
        # the benchmark's two-leg contraction in plain FP64 (the default precision)
        {"name": "dot_f64_pair_2048", "kind": "pair", "mode": "f64", "D": 2048},
        # its largest size in the mixed precision that the headline sweeps use
        {"name": "dot_tf32x3_pair_4096", "kind": "pair", "mode": "tf32x3", "D": 4096},
        # the same call at a ragged bond dimension in the other mixed precision
        {"name": "dot_bf16x3_pair_1531", "kind": "pair", "mode": "bf16x3", "D": 1531},
        # the matvec of a fermion chain: two charges, many small blocks
        {"name": "matvec_f64_hubbard_512", "kind": "matvec", "model": "hubbard", "mode": "f64", "D": 512},
        # the headline's matvec: 6-leg cylinder (wide MPO), D = 2048, mixed precision
        {"name": "matvec_tf32x3_cylinder_2048", "kind": "matvec", "model": "cylinder", "mode": "tf32x3", "D": 2048},
        # the environment update of a spin chain at an odd bond dimension, FP64
        {"name": "env_f64_chain_777", "kind": "env", "model": "heisenberg", "mode": "f64", "D": 777},
        # the untruncated site SVD of bMPS.move_oc on a small chain
        {"name": "svd_f64_site_48", "kind": "site_svd", "mode": "f64", "D": 48},
        # the truncating SVD of a bond update, FP64, chain-like spectrum
        {"name": "svd_f64_theta_600", "kind": "svd", "mode": "f64", "D": 600, "decay": 14.0},
        # the headline's truncating SVD: mixed precision, cylinder-like spectrum
        {"name": "svd_tf32x3_theta_2048", "kind": "svd", "mode": "tf32x3", "D": 2048, "decay": 8.0},
        # eigh of a bond operator
        {"name": "eigh_f64_300", "kind": "eigh", "mode": "f64", "D": 300},
        # a whole solve's sweeps on a small anisotropic chain, FP64: the driver end to end
        {"name": "dmrg_f64_L16_D32", "kind": "dmrg", "mode": "f64", "D": 32, "L": 16, "delta": 0.7, "sweeps": 2},
    ]


def draw(rng):
    def size(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(["site", "pair", "pair", "matvec", "matvec", "env", "site_svd", "svd", "svd", "eigh", "dmrg"])
    mode = rng.choice(["f64", "f64", "tf32x3", "bf16x3"])
    if kind in ("site", "pair"):
        return {"kind": kind, "mode": mode, "D": size(16, 4096)}
    if kind in ("matvec", "env"):
        name = rng.choice(["heisenberg", "hubbard", "cylinder"])
        top = {"heisenberg": 1024, "hubbard": 1024, "cylinder": 1024 if mode == "f64" else 2048}[name]
        return {"kind": kind, "model": name, "mode": mode, "D": size(32, top)}
    if kind == "site_svd":
        return {"kind": kind, "mode": mode, "D": size(12, 400)}
    if kind == "svd":
        mode = rng.choice(["f64", "tf32x3"])
        return {"kind": kind, "mode": mode, "D": size(24, 700 if mode == "f64" else 2048),
                "decay": rng.choice([8.0, 14.0])}
    if kind == "eigh":
        return {"kind": kind, "mode": "f64", "D": size(16, 500)}
    return {"kind": "dmrg", "mode": "f64", "D": size(8, 32), "L": rng.randrange(8, 17),
            "delta": round(rng.uniform(0.2, 0.9), 3), "sweeps": 2}


def prepare(case, seed):
    q.ensure_init(0)
    kind, D = case["kind"], case["D"]
    state = {"case": case}
    if kind == "site":
        state["A"], state["B"] = site_pair(D, seed)
    elif kind == "pair":
        state["A"], state["B"] = networks.theta_pair(D, seed=int(seed))
    elif kind in ("matvec", "env"):
        state.update(chain_state(case, seed))
    elif kind == "site_svd":
        state["A"] = site_pair(D, seed)[0]
    elif kind == "svd":
        state["theta"] = graded_theta(D, case["decay"], seed)
    elif kind == "eigh":
        state["rho"] = symmetric(D, seed)
    else:
        q.set_gemm_mode("f64")
        state["mpo"] = networks.xxz(case["L"], case["delta"])
        mps = networks.random_bmps(case["L"], D, target=case["L"] % 2, seed=int(seed))
        state["mps"] = mps.move_oc(0).normalize_center()
    return state


def run(state):
    case = state["case"]
    kind = case["kind"]
    q.set_gemm_mode(case["mode"])
    if kind == "site":
        return read_tensor(state["A"].tensordot(state["B"], ([2], [0])))
    if kind == "pair":
        return read_tensor(state["A"].tensordot(state["B"], ([2, 3], [1, 0])))
    if kind == "matvec":
        return read_tensor(algorithms.hamil2site_times_state(state["theta"], state["H"], state["L"], state["R"]))
    if kind == "env":
        return read_tensor(algorithms.compute_left_env(state["W"], state["A"], state["L"]))
    if kind == "site_svd":
        return read_svd(state["A"], *linalg.svd(state["A"], 2), 2)
    if kind == "svd":
        return read_svd(state["theta"], *linalg.svd(state["theta"], 2, CUTOFF, min_size=4, max_size=case["D"]), 2)
    if kind == "eigh":
        return read_eigh(state["rho"], *linalg.eigh(state["rho"]))
    opts = algorithms.dmrg_options(cutoff=CUTOFF, convergence_criterion=0.0, max_bond=case["D"], min_bond=4,
                                   maximum_iterations=case["sweeps"], gemm=case["mode"])
    mps = networks.bMPS(list(state["mps"]), state["mps"].orthogonality_center)
    energy = algorithms.dmrg(state["mpo"], mps, opts)
    return {"energy": energy, "state": read_state(mps)}


# --------------------------------------------------------------------------- what a pass cannot do without
def product(A, B, da, db):
    """The block structure of a contraction of {index: shape} tensors, and its flops."""
    fa = [i for i in range(len(next(iter(A)))) if i not in da]
    fb = [i for i in range(len(next(iter(B)))) if i not in db]
    by = {}
    for k, s in B.items():
        by.setdefault(tuple(k[i] for i in db), []).append((tuple(k[i] for i in fb), tuple(s[i] for i in fb)))
    out, flops = {}, 0.0
    for k, s in A.items():
        head, shp = tuple(k[i] for i in fa), tuple(s[i] for i in fa)
        K = math.prod(s[i] for i in da)
        for tail, st in by.get(tuple(k[i] for i in da), ()):
            out[head + tail] = shp + st
            flops += 2.0 * math.prod(shp) * math.prod(st) * K
    return out, flops


def shape(t):
    sizes = t._sizes()
    return {k: t._shape_of(sizes, k) for k in t.block_indices()}


def numel(*shapes):
    return float(sum(math.prod(s) for x in shapes for s in x.values()))


MATVEC = (("L", ([0], [0])), ("H", ([0, 2, 3], [0, 4, 5])), ("R", ([1, 4], [0, 1])))
LEFT_ENV = (("A", ([0], [0])), ("W", ([0, 2], [0, 3])), ("conj", ([0, 2], [0, 1])))


def sector_flops(p, n):
    """LAPACK's count for a thin SVD of a p x n matrix."""
    p, n = max(p, n), min(p, n)
    return 4.0 * p * p * n + 8.0 * p * n * n + 9.0 * n ** 3


def svd_work(legs, split, keep):
    sec = {}
    for side, part in ((0, legs[:split]), (1, legs[split:])):
        for combo in itertools.product(*part):
            c = sum(x[1] for x in combo)
            key = c if side == 0 else -c
            sec.setdefault(key, [0, 0])[side] += math.prod(x[0] for x in combo)
    flops = sum(sector_flops(m, n) for m, n in sec.values() if m and n)
    nnz = sum(m * n for m, n in sec.values())
    total = sum(min(m, n) for m, n in sec.values())
    frac = min(1.0, keep / max(total, 1))
    factors = sum(frac * min(m, n) * (m + n + 1) for m, n in sec.values())
    return {"bytes": 8.0 * (nnz + factors), "flops": flops}


def work(case):
    kind, D = case["kind"], case["D"]
    if kind == "site":
        A, B = ({k: s for k, s in blocks_of(legs)} for legs in site_legs(D))
        C, f = product(A, B, [2], [0])
        return {"bytes": 8.0 * numel(A, B, C), "flops": f}
    if kind == "pair":
        b = networks.gaussian_sections(D)
        A = dict(blocks_of([b, PHYS, PHYS, inverse(b)]))
        B = dict(blocks_of([b, inverse(PHYS), PHYS, inverse(b)]))
        C, f = product(A, B, [2, 3], [1, 0])
        return {"bytes": 8.0 * numel(A, B, C), "flops": f}
    if kind in ("matvec", "env"):
        state = prepare(case, 0)
        s = {k: shape(t) for k, t in state.items() if k != "case"}
        if kind == "matvec":
            cur, rest, steps = s["L"], s["theta"], MATVEC
            cur, f = product(cur, rest, [0], [0])
            for name, (da, db) in steps[1:]:
                cur, g = product(cur, s[name], da, db)
                f += g
            return {"bytes": 8.0 * numel(s["L"], s["R"], s["H"], s["theta"], cur), "flops": f}
        cur, f = product(s["L"], s["A"], [0], [0])
        for name, (da, db) in LEFT_ENV[1:]:
            cur, g = product(cur, s["A" if name == "conj" else name], da, db)
            f += g
        return {"bytes": 8.0 * numel(s["L"], s["A"], s["W"], cur), "flops": f}
    if kind == "site_svd":
        return svd_work(site_legs(D)[0], 2, D)
    if kind == "svd":
        return svd_work([bond(D, 0), PHYS, PHYS, inverse(bond(D, 0))], 2, D)
    if kind == "eigh":
        leg = bond(D, 0)
        return {"bytes": 8.0 * sum(2 * n * n + n for n, _ in leg), "flops": sum(9.0 * n ** 3 for n, _ in leg)}
    # a sweep visits every inner bond twice: two matvecs, one environment update and one SVD each
    L, w = case["L"], 5
    bonds = [{0: 1}] + networks.bond_sectors(L, D, [1, -1], L % 2) + [{L % 2: 1}]
    flops, elems = 0.0, 0.0
    for i in range(L - 1):
        left, right = bonds[i], bonds[i + 2]
        rows, cols = {}, {}
        for c, n in left.items():
            for s in (1, -1):
                rows[c + s] = rows.get(c + s, 0) + n
        for c, n in right.items():
            for s in (1, -1):
                cols[c - s] = cols.get(c - s, 0) + n
        nnz = sum(n * cols.get(c, 0) for c, n in rows.items())
        big = (max(left.values()) + max(right.values())) / 2.0
        flops += 2 * (4.0 * w * nnz * big) + 2.0 * w * nnz * big
        flops += sum(sector_flops(n, cols[c]) for c, n in rows.items() if c in cols)
        elems += 6.0 * nnz
    return {"bytes": 16.0 * elems * case["sweeps"], "flops": 2.0 * flops * case["sweeps"]}


# --------------------------------------------------------------------------- the same in plain 64-bit torch
def blocks(t):
    return {k: torch.from_numpy(v).cuda() for k, v in t.blocks()}


def tdot(A, B, da, db):
    """Block contraction of {index: array} tensors."""
    ra, rb = len(next(iter(A))), len(next(iter(B)))
    fa = [i for i in range(ra) if i not in da]
    fb = [i for i in range(rb) if i not in db]
    by = {}
    for k, x in B.items():
        by.setdefault(tuple(k[i] for i in db), []).append((tuple(k[i] for i in fb), x))
    out = {}
    for k, x in A.items():
        head = tuple(k[i] for i in fa)
        for tail, y in by.get(tuple(k[i] for i in da), ()):
            z = torch.tensordot(x, y, (list(da), list(db)))
            out[head + tail] = out[head + tail] + z if head + tail in out else z
    return out


def in_order(x):
    return np.concatenate([x[k].reshape(-1).cpu().numpy() for k in sorted(x)])


def kept(sig, tol, min_size, max_size):
    """The threshold of the reference's truncation (sources/btensor_linalg.cpp:658-682,
    sources/LinearAlgebra.cpp:57-75) on values sorted in descending order."""
    last = len(sig) - 1
    acc = sig[last] ** 2
    while last >= min_size:
        if acc > tol * tol and last < max_size:
            break
        last -= 1
        acc += sig[last] ** 2
    return sig[last] * (1.0 - 2.0 * np.finfo(float).eps)


def exact_svd(t, rows_of, split, truncated, D):
    """Sector SVDs in LAPACK, truncated by the reference's rule: read_svd's arrays."""
    x = blocks(t)
    sec = {}
    for k, v in x.items():
        sec.setdefault(rows_of(k), []).append(k)
    done = {}
    for Q, keys in sorted(sec.items()):
        rk = sorted({k[:split] for k in keys})
        ck = sorted({k[split:] for k in keys})
        rn = {r: math.prod(next(x[k].shape for k in keys if k[:split] == r)[:split]) for r in rk}
        cn = {c: math.prod(next(x[k].shape for k in keys if k[split:] == c)[split:]) for c in ck}
        M = torch.zeros(sum(rn.values()), sum(cn.values()), dtype=torch.float64, device="cuda")
        at = {}
        r0 = 0
        for r in rk:
            c0 = 0
            for c in ck:
                if r + c in x:
                    M[r0:r0 + rn[r], c0:c0 + cn[c]] = x[r + c].reshape(rn[r], cn[c])
                    at[r + c] = (r0, rn[r], c0, cn[c])
                c0 += cn[c]
            r0 += rn[r]
        u, s, vh = np.linalg.svd(M.cpu().numpy(), full_matrices=False)
        done[Q] = (u, s, vh, at)
    sig = np.sort(np.concatenate([v[1] for v in done.values()]))[::-1]
    low = kept(sig, CUTOFF, 4, D) if truncated else -1.0
    prod, gram = {}, []
    for Q, (u, s, vh, at) in sorted(done.items()):
        n = int((s > low).sum())
        gram.append(padded(np.eye(n), len(s)).ravel())
        p = (u[:, :n] * s[:n]) @ vh[:n]
        for k, (r0, rn, c0, cn) in at.items():
            prod[k] = p[r0:r0 + rn, c0:c0 + cn].ravel()
    gram = np.concatenate(gram)
    return [padded(sig[sig > low], len(sig)), np.concatenate([prod[k] for k in sorted(prod)]), gram, gram]


def exact(case, seed):
    kind, D = case["kind"], case["D"]
    if kind == "dmrg":
        return None
    state = prepare(case, seed)
    if kind == "site":
        return [in_order(tdot(blocks(state["A"]), blocks(state["B"]), [2], [0]))]
    if kind == "pair":
        return [in_order(tdot(blocks(state["A"]), blocks(state["B"]), [2, 3], [1, 0]))]
    if kind == "matvec":
        x = tdot(blocks(state["L"]), blocks(state["theta"]), [0], [0])
        x = tdot(x, blocks(state["H"]), [0, 2, 3], [0, 4, 5])
        return [in_order(tdot(x, blocks(state["R"]), [1, 4], [0, 1]))]
    if kind == "env":
        x = tdot(blocks(state["L"]), blocks(state["A"]), [0], [0])
        x = tdot(x, blocks(state["W"]), [0, 2], [0, 3])
        return [in_order(tdot(x, blocks(state["A"]), [0, 2], [0, 1]))]
    if kind == "site_svd":
        legs = site_legs(D)[0]
        return exact_svd(state["A"], lambda k: legs[0][k[0]][1] + PHYS[k[1]][1], 2, False, D)
    if kind == "svd":
        left = bond(D, 0)
        return exact_svd(state["theta"], lambda k: left[k[0]][1] + PHYS[k[1]][1], 2, True, D)
    x = blocks(state["rho"])
    vals, parts, gram = [], [], []
    for k in sorted(x):
        a = x[k].cpu().numpy()
        vals.append(np.linalg.eigvalsh(a))
        parts.append(a.ravel())
        gram.append(np.eye(len(a)).ravel())
    return [np.sort(np.concatenate(vals)), np.concatenate(parts), np.concatenate(gram)]
