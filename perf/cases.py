"""Timing cases of the framework: the calls a DMRG or tSDRG program makes, over the sizes it makes them at.

Seven kinds of call, all through the package's public entry points:

* ``matvec``, ``env``, ``gauge``: the steps of one site update of ``FiniteDMRG`` in the default
  'fp64' form (bonds of tens to a few hundred) and in the 'mixed' form (up to chi = 1024);
* ``eigshmv``: the local eigensolve through ``linalg.eigshmv`` at its default tolerance;
* ``chains``: the site-update steps of many lockstep chains (``BatchedFiniteDMRG``);
* ``eigh``: the dense block spectra of tSDRG (``kernels.eigh_batched``);
* ``spectrum``: the Schmidt values on the middle bond of an MPS;
* ``tsdrg``, ``sweep``: whole calls (``BatchedTSDRG.run``, two sweeps of ``FiniteDMRG`` on a random-field chain).

Environments are built with the channel structure of the XXZ MPO (identity, S+, S-, Sz, H) so that
the effective Hamiltonians are symmetric with a spectrum like a block's; site tensors have
Schmidt values that decay over three decades.
"""
from __future__ import annotations

import math

import numpy as np
import torch

import tnpy_gb300 as tnpy
from tnpy_gb300 import kernels as K
from tnpy_gb300 import linalg
from tnpy_gb300.finite_dmrg import Direction
from tnpy_gb300.matrix_product_state import MatrixProductState, MatrixProductStateMeasurements, OneSiteOperator
from tnpy_gb300.model.random_heisenberg import RandomCouplingHeisenberg, RandomHeisenberg
from tnpy_gb300.model.xxz import XXZ

D, PHYS = 5, 2  # MPO bond of the XXZ / Heisenberg chains, spin 1/2
DELTA = -0.5


def listed():
    return [
        # bulk site of the benchmark chain (XXZ, n = 100, chi = 1024, mixed): the perturbation's product
        {"name": "matvec_mixed_1024", "kind": "matvec", "precision": "mixed", "chi_l": 1024, "chi_r": 1024},
        # default precision at an ordinary bond, odd sizes as enlarged or truncated bonds give them
        {"name": "matvec_fp64_201x168", "kind": "matvec", "precision": "fp64", "chi_l": 201, "chi_r": 168},
        # bulk environment update of the benchmark chain
        {"name": "env_mixed_1024", "kind": "env", "precision": "mixed", "direction": 1, "chi_l": 1024, "chi_r": 1024},
        # leftward environment update of a default-precision run
        {"name": "env_fp64_112x99", "kind": "env", "precision": "fp64", "direction": -1, "chi_l": 112, "chi_r": 99},
        # bulk gauge move of the benchmark chain
        {"name": "gauge_mixed_1024", "kind": "gauge", "precision": "mixed", "direction": 1, "chi_l": 1024,
         "chi_r": 1024, "chi_other": 1024},
        # leftward gauge move of a default-precision run
        {"name": "gauge_fp64_130x190", "kind": "gauge", "precision": "fp64", "direction": -1, "chi_l": 130,
         "chi_r": 190, "chi_other": 150},
        # local eigensolve of a small chain (n = 32, chi = 32): many short launches
        {"name": "eigshmv_32", "kind": "eigshmv", "chi_l": 32, "chi_r": 32},
        # site update of lockstep chains (n = 64, chi = 64) without the eigensolve
        {"name": "chains_64x64", "kind": "chains", "precision": "mixed", "batch": 64, "chi": 64},
        # dense tSDRG blocks: a block of up to 32 states merged with one spin, many realisations
        {"name": "eigh_128x64", "kind": "eigh", "count": 128, "node": 32, "keep": 32},
        # middle-bond entanglement spectrum of a mid-sized state
        {"name": "spectrum_n16_128", "kind": "spectrum", "n": 16, "chi": 128},
        # a small disorder ensemble, start to finish
        {"name": "tsdrg_8xn16_16", "kind": "tsdrg", "chains": 8, "n": 16, "chi": 16},
        # a rightward and a leftward sweep of a small default-precision run
        {"name": "sweep_n16_32", "kind": "sweep", "precision": "fp64", "n": 16, "chi": 32},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["matvec", "matvec", "env", "env", "gauge", "gauge", "eigshmv", "chains", "eigh", "spectrum",
                       "tsdrg", "sweep"])
    c = {"kind": kind}
    if kind in ("matvec", "env", "gauge"):
        c["precision"] = rng.choice(["fp64", "mixed"])
        lo, hi = (16, 320) if c["precision"] == "fp64" else (64, 1000)
        c["chi_l"] = _log(rng, lo, hi)
        c["chi_r"] = min(hi, max(lo, int(c["chi_l"] * rng.uniform(0.6, 1.6))))
        if kind != "matvec":
            c["direction"] = rng.choice([1, -1])
        if kind == "gauge":
            c["chi_other"] = min(hi, max(lo, int(c["chi_l"] * rng.uniform(0.6, 1.6))))
    elif kind == "eigshmv":
        c["chi_l"] = _log(rng, 12, 48)
        c["chi_r"] = min(48, max(12, int(c["chi_l"] * rng.uniform(0.6, 1.6))))
    elif kind == "chains":
        c.update(precision=rng.choice(["fp64", "mixed"]), batch=_log(rng, 4, 64), chi=_log(rng, 12, 64))
    elif kind == "eigh":
        node = rng.randint(4, 32)
        c.update(count=_log(rng, 1, 256), node=node, keep=rng.randint(1, node))
    elif kind == "spectrum":
        c.update(n=rng.randint(8, 16), chi=_log(rng, 20, 128))
    elif kind == "tsdrg":
        c.update(chains=rng.randint(1, 8), n=rng.randint(6, 16), chi=_log(rng, 4, 16))
    else:
        c.update(precision=rng.choice(["fp64", "mixed"]), n=rng.randint(10, 16), chi=_log(rng, 12, 32))
    return c


# ---- inputs -----------------------------------------------------------------------------------
def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed))


def _randn(g, *shape):
    return torch.randn(*shape, generator=g, dtype=torch.float64, device="cuda")


def _block(g, chi, left, batch=()):
    """Environment [*batch, chi, D, chi] of a block with H = diag(energies) + weak mixing and
    boundary spin operators, in the channel order of the XXZ MPO."""
    sp = 0.5 * _randn(g, *batch, chi, chi) / math.sqrt(chi)
    sz = _randn(g, *batch, chi, chi) / math.sqrt(chi)
    sz = 0.25 * (sz + sz.mT)
    h = _randn(g, *batch, chi, chi) / math.sqrt(chi)
    e = torch.rand(*batch, chi, generator=g, dtype=torch.float64, device="cuda").sort(-1).values
    h = 0.05 * (h + h.mT) + torch.diag_embed(-8.0 + 6.0 * e)
    eye = torch.eye(chi, dtype=torch.float64, device="cuda").expand(*batch, chi, chi)
    if left:
        ops = [eye, -0.5 * sp, -0.5 * sp.mT, -DELTA * sz, h]
    else:
        ops = [h, sp.mT, sp, sz, eye]
    return torch.stack(ops, -2).contiguous()


def _mpo_tensor():
    return torch.from_numpy(np.ascontiguousarray(XXZ(4, DELTA).mpo[1])).to("cuda", torch.float64)


def _site(g, chi_l, chi_r, batch=()):
    """Site tensor with Schmidt-like weights over three decades on both bonds, unit norm."""
    a = _randn(g, *batch, chi_l, PHYS, chi_r)
    wl = torch.logspace(0, -3, chi_l, dtype=torch.float64, device="cuda").sqrt()
    wr = torch.logspace(0, -3, chi_r, dtype=torch.float64, device="cuda").sqrt()
    a = a * wl[:, None, None] * wr
    return (a / torch.linalg.vector_norm(a, dim=(-3, -2, -1), keepdim=True)).contiguous()


def _mps_tensors(seed, n, chi):
    g = _gen(seed)
    dims = [min(chi, PHYS ** min(i, n - i)) for i in range(n + 1)]
    return [_site(g, dims[i], dims[i + 1]) for i in range(n)]


def _gauge_dims(case):
    """Site dimensions with the split bond within the fused one, as every MPS bond is."""
    cl, cr = case["chi_l"], case["chi_r"]
    return (cl, min(cr, PHYS * cl)) if case["direction"] == 1 else (min(cl, PHYS * cr), cr)


def _blocks(seed, count, node):
    """tSDRG two-block Hamiltonians: a `node`-state block with a conserved Sz merged with a spin."""
    rng = np.random.RandomState(seed % 2**32)
    szs, sps = np.diag([0.5, -0.5]), np.array([[0.0, 1.0], [0.0, 0.0]])
    out = []
    for _ in range(count):
        q = np.round(rng.normal(scale=1.2, size=node))
        sp = 0.4 * rng.normal(size=(node, node)) * (q[:, None] == q[None, :] + 1)
        sz = 0.2 * rng.normal(size=(node, node)) * (q[:, None] == q[None, :])
        sz = 0.5 * (sz + sz.T) + np.diag(0.2 * q)
        h = np.kron(np.diag(np.sort(rng.uniform(-4, 0, node))), np.eye(2)) + np.kron(np.eye(node), rng.uniform(-1, 1) * szs)
        j = rng.uniform(0.1, 1.0)
        out.append(h + j * (np.kron(sz, szs) + 0.5 * (np.kron(sp, sps.T) + np.kron(sp.T, sps))))
    return out


def _chain_models(case, seed):
    return [RandomCouplingHeisenberg(case["n"], h=0.5, seed=(7 * seed + 101 * c) % 2**31) for c in range(case["chains"])]


def prepare(case, seed):
    kind = case["kind"]
    g = _gen(seed)
    s = {"case": case, "w": _mpo_tensor()}
    if kind == "matvec":
        s.update(L=_block(g, case["chi_l"], True), R=_block(g, case["chi_r"], False),
                 x=_site(g, case["chi_l"], case["chi_r"]))
    elif kind == "env":
        left = case["direction"] == 1
        s.update(E=_block(g, case["chi_l"] if left else case["chi_r"], left), a=_site(g, case["chi_l"], case["chi_r"]))
    elif kind == "gauge":
        cl, cr = _gauge_dims(case)
        nb = _site(g, cr, case["chi_other"]) if case["direction"] == 1 else _site(g, case["chi_other"], cl)
        s.update(site=_site(g, cl, cr), nb=nb)
    elif kind == "eigshmv":
        cl, cr = case["chi_l"], case["chi_r"]
        op = OneSiteOperator(_block(g, cl, True), s["w"], _block(g, cr, False), (cl, PHYS, cr))
        s.update(op=op, v0=_site(g, cl, cr).reshape(-1, 1))
    elif kind == "chains":
        b, chi = case["batch"], case["chi"]
        s.update(L=_block(g, chi, True, (b,)), R=_block(g, chi, False, (b,)), x=_site(g, chi, chi, (b,)),
                 nb=_site(g, chi, chi, (b,)), wb=s["w"].expand(b, D, D, PHYS, PHYS).contiguous())
    elif kind == "eigh":
        s["mats"] = [torch.from_numpy(h).to("cuda") for h in _blocks(seed, case["count"], case["node"])]
    elif kind == "spectrum":
        s["mps"] = MatrixProductState(_mps_tensors(seed, case["n"], case["chi"]))
    elif kind == "tsdrg":
        s["mpos"] = [m.mpo for m in _chain_models(case, seed)]
    else:
        mpo = RandomHeisenberg(case["n"], h=0.5, seed=seed % 2**32).mpo
        f = tnpy.FiniteDMRG(mpo, case["chi"], precision=case["precision"], seed=seed, compute_variance=False)
        f.sweep(Direction.RIGHTWARD, tol=1e-10)
        f.sweep(Direction.LEFTWARD, tol=1e-10)
        s["dmrg"] = f
    return s


# ---- one pass ---------------------------------------------------------------------------------
def run(s):
    case = s["case"]
    kind = case["kind"]
    if kind == "matvec":
        return K.matvec1(s["L"], s["w"], s["R"], s["x"], precision=case["precision"])
    if kind == "env":
        return K.env_update(case["direction"], s["E"], s["a"], s["w"], precision=case["precision"])
    if kind == "gauge":
        a, nb = s["site"].clone(), s["nb"].clone()  # the move rewrites both in place
        K.gauge_move(case["direction"], a, nb, precision=case["precision"])
        return a, nb
    if kind == "eigshmv":
        e, v = linalg.eigshmv(s["op"], s["v0"])
        return e, v
    if kind == "chains":
        p = case["precision"]
        psi, nb = s["x"].clone(), s["nb"].clone()
        psi.add_(K.batched_matvec1(s["L"], s["wb"], s["R"], psi, precision=p), alpha=1e-5)
        K.batched_gauge_move(1, psi, nb, precision=p)
        return psi, nb, K.batched_env_update(1, s["L"], psi, s["wb"], precision=p)
    if kind == "eigh":
        return K.eigh_batched(s["mats"], keep=case["keep"])
    if kind == "spectrum":
        mps = s["mps"]
        return MatrixProductStateMeasurements(mps).entanglement_spectrum(mps.n_sites // 2 - 1)
    if kind == "tsdrg":
        t = tnpy.BatchedTSDRG(s["mpos"], case["chi"]).run()
        return t.evals, np.array(t.merges)
    f = s["dmrg"]
    return f.sweep(Direction.RIGHTWARD, tol=1e-10), f.sweep(Direction.LEFTWARD, tol=1e-10)


# ---- what a pass cannot do without ------------------------------------------------------------
def work(case):
    kind = case["kind"]
    if kind in ("matvec", "env"):
        cl, cr = case["chi_l"], case["chi_r"]
        if kind == "matvec":
            f = 2 * D * PHYS * (cl * cl * cr + cl * cr * cr) + 2 * cl * cr * (D * PHYS) ** 2
            return {"bytes": 8 * (D * (cl * cl + cr * cr) + 2 * PHYS * cl * cr), "flops": f}
        f = 2 * D * PHYS * (cl * cl * cr + cl * cr * cr) + 2 * cl * cr * (D * PHYS) ** 2
        return {"bytes": 8 * (D * (cl * cl + cr * cr) + PHYS * cl * cr), "flops": f}
    if kind == "gauge":
        cl, cr = _gauge_dims(case)
        m, n = (cl * PHYS, cr) if case["direction"] == 1 else (cr * PHYS, cl)
        far = PHYS * case["chi_other"]
        return {"bytes": 16 * (m * n + n * far), "flops": 4 * m * n * n - 4 * n**3 / 3 + n * n * far}
    if kind == "eigshmv":  # a dozen products and orthogonalisations at least
        w = work({**case, "kind": "matvec"})
        return {"bytes": 8 * D * (case["chi_l"] ** 2 + case["chi_r"] ** 2), "flops": 12 * w["flops"]}
    if kind == "chains":
        b, chi = case["batch"], case["chi"]
        one = [work({"kind": k, "chi_l": chi, "chi_r": chi, "chi_other": chi, "direction": 1})
               for k in ("matvec", "gauge", "env")]
        return {"bytes": b * 8 * (3 * D + 4 * PHYS) * chi * chi, "flops": b * sum(w["flops"] for w in one)}
    if kind == "eigh":
        n = 2 * case["node"]
        return {"bytes": case["count"] * 8 * n * (n + case["keep"]), "flops": case["count"] * 9.0 * n**3}
    if kind == "spectrum":
        n, chi = case["n"], case["chi"]
        dims = [min(chi, PHYS ** min(i, n - i)) for i in range(n + 1)]
        f = sum(work({"kind": "gauge", "direction": 1, "chi_l": dims[i], "chi_r": dims[i + 1],
                      "chi_other": dims[i + 1]})["flops"] for i in range(n // 2))
        return {"bytes": 8 * PHYS * sum(a * b for a, b in zip(dims, dims[1:])), "flops": 2 * f + 8.0 / 3 * max(dims) ** 3}
    if kind == "tsdrg":  # two block spectra per merge, `chi` pairs of each
        m = case["chi"] ** 2
        return {"bytes": case["chains"] * case["n"] * 8 * D * D * case["chi"] ** 2,
                "flops": case["chains"] * 2 * case["n"] * (4.0 / 3 * m**2 * min(m, 8 * case["chi"]))}
    n, chi = case["n"], case["chi"]
    w = work({"kind": "matvec", "chi_l": chi, "chi_r": chi})
    return {"bytes": 2 * n * w["bytes"], "flops": 2 * n * 6 * w["flops"]}


# ---- 64-bit values, plain torch and numpy -----------------------------------------------------
def _matvec(L, w, R, x):
    t = torch.einsum("...awb,...asc->...wbsc", L, x)
    t = torch.einsum("...wbsc,...wvst->...btcv", t, w)
    return torch.einsum("...btcv,...cvd->...btd", t, R)


def _env(direction, E, a, w):
    if direction == 1:
        t = torch.einsum("...awb,...asc->...wbsc", E, a)
        t = torch.einsum("...wbsc,...wvst->...btcv", t, w)
        return torch.einsum("...btcv,...btd->...cvd", t, a)
    t = torch.einsum("...asc,...cvd->...asvd", a, E)
    t = torch.einsum("...asvd,...wvst->...awtd", t, w)
    return torch.einsum("...awtd,...btd->...awb", t, a)


def _gauge(direction, a, nb):
    cl, d, cr = a.shape[-3:]
    a, nb = a.cpu(), nb.cpu()
    if direction == 1:
        q, r = torch.linalg.qr(a.reshape(*a.shape[:-3], cl * d, cr))
        return q.reshape(a.shape), torch.einsum("...ij,...jsk->...isk", r, nb)
    q, r = torch.linalg.qr(a.reshape(*a.shape[:-3], cl, d * cr).mT)
    return q.mT.reshape(a.shape), torch.einsum("...asj,...ij->...asi", nb, r)


def _spectrum(tensors):
    t = [a.cpu().numpy() for a in tensors]
    n = len(t)
    left = np.ones((1, 1))
    for a in t[: n // 2]:
        m = np.tensordot(left, a, 1)
        left = np.linalg.qr(m.reshape(-1, m.shape[2]))[1]
    right = np.ones((1, 1))
    for a in t[: n // 2 - 1 : -1]:
        m = np.tensordot(a, right, 1)
        right = np.linalg.qr(m.reshape(m.shape[0], -1).T)[1].T
    lam = np.linalg.svd(left @ right, compute_uv=False)
    return lam / np.linalg.norm(lam)


def _tsdrg(model, chi):
    """Greedy merging of the pair with the largest gap (numpy), lowest spectrum of the last block."""
    j, f = model.couplings, model.fields
    sz, sp = np.diag([0.5, -0.5]), np.array([[0.0, 1.0], [0.0, 0.0]])
    # a block: Hamiltonian, first and last spin's (S+, Sz)
    blocks = [(f[i] * sz, (sp, sz), (sp, sz)) for i in range(len(f))]
    bonds = list(j)
    ids, merges, nxt = list(range(len(f))), [], len(f)

    def join(a, b, jj):
        na, nb = len(a[0]), len(b[0])
        h = np.kron(a[0], np.eye(nb)) + np.kron(np.eye(na), b[0])
        (p1, z1), (p2, z2) = a[2], b[1]
        return h + jj * (np.kron(z1, z2) + 0.5 * (np.kron(p1, p2.T) + np.kron(p1.T, p2)))

    def solve(i):
        e, v = np.linalg.eigh(join(blocks[i], blocks[i + 1], bonds[i]))
        e, v = e[:chi], v[:, :chi]
        gaps = np.diff(e)
        return (gaps[chi - 1] if gaps.size > chi else gaps[-1]), e, v

    found = [solve(i) for i in range(len(bonds))]
    while True:
        b = int(np.argmax([s[0] for s in found]))
        _, e, v = found[b]
        x, y = blocks[b], blocks[b + 1]
        nx, ny = len(x[0]), len(y[0])
        up = lambda o, first: v.T @ (np.kron(o, np.eye(ny)) if first else np.kron(np.eye(nx), o)) @ v
        merges.append((ids[b], ids[b + 1], nxt))
        blocks[b : b + 2] = [(np.diag(e), tuple(up(o, True) for o in x[1]), tuple(up(o, False) for o in y[2]))]
        ids[b : b + 2] = [nxt]
        nxt += 1
        bonds.pop(b)
        found.pop(b)
        if not bonds:
            return e, merges
        for i in ([b - 1] if b > 0 else []) + ([b] if b < len(bonds) else []):
            found[i] = solve(i)


def exact(case, seed):
    kind = case["kind"]
    if kind == "sweep":  # no closed value: the truncated variational energy
        return None
    if kind == "tsdrg":
        done = [_tsdrg(m, case["chi"]) for m in _chain_models(case, seed)]
        return [e for e, _ in done], np.array([m for _, m in done])
    if kind == "eigh":
        hs = _blocks(seed, case["count"], case["node"])
        return np.stack([np.linalg.eigvalsh(h)[: case["keep"]] for h in hs]), None
    if kind == "spectrum":
        return _spectrum(_mps_tensors(seed, case["n"], case["chi"]))
    s = prepare(case, seed)
    if kind == "matvec":
        return _matvec(s["L"], s["w"], s["R"], s["x"])
    if kind == "env":
        return _env(case["direction"], s["E"], s["a"], s["w"])
    if kind == "gauge":
        return _gauge(case["direction"], s["site"], s["nb"])
    if kind == "eigshmv":
        op, cl, cr = s["op"], case["chi_l"], case["chi_r"]
        n = cl * PHYS * cr
        h = torch.einsum("awb,wvst,cvd->ascbtd", op.left, op.w, op.right).reshape(n, n)
        e = torch.linalg.eigvalsh(0.5 * (h + h.T).cpu())
        return float(e[0]), None
    psi = s["x"] + 1e-5 * _matvec(s["L"], s["wb"], s["R"], s["x"])
    q, nb = _gauge(1, psi, s["nb"])
    return q, nb, _env(1, s["L"].cpu(), q, s["wb"].cpu())
