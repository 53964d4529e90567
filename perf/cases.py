"""
Timing cases of the Hartree-Fock path: the calls an MD program or an SCF host
makes, from one water in 6-31G* (19 AOs) to (H2O)32 in cc-pVDZ (800 AOs).

  jk      integral-direct J and K of one density (RHF) or two (UHF), in FP64
          or with the small quartets in FP32 (the ``fp32_cutoff`` option)
  delta   J and K of a density change, as every SCF iteration after the first
          builds them (density-weighted screening)
  grad    the two-electron nuclear gradient at given densities
  frame   what a new geometry costs before the first Fock build: primitive
          pairs, Schwarz bounds, S, T, V, dipole, and the one-electron gradient
  force   SCF to convergence and the analytic gradient at the frames of a
          trajectory, from the density that the frame before left
  batch   SCF and gradient of several molecules of uneven size at once

Geometries are molecules this package generates (aimd_b200.geometry) as a
running trajectory meets them: thermally displaced and freely rotated.
Densities are sums over localised occupied orbitals, which decay with distance
as those of a closed-shell insulator do.
"""

from __future__ import annotations

import functools
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.getcwd(), "ab-initio-md_b200"))

from aimd_b200 import geometry  # noqa: E402
from aimd_b200 import integrals as I  # noqa: E402
from aimd_b200.basis import build_basis  # noqa: E402
from aimd_b200.batch import BatchSolver  # noqa: E402
from aimd_b200.engine import engine_for  # noqa: E402
from aimd_b200.gradients import scf_gradient_device  # noqa: E402
from aimd_b200.scf import SCFOptions, SCFSolver, run_device  # noqa: E402

THR, THR_GRAD, THR_DELTA = 1e-12, 1e-14, 1e-13      # the SCF's and the gradient's defaults


def listed():
    return [
        # single points and short MD of a small molecule: latency and launches
        {"name": "jk_water", "kind": "jk", "mol": "water", "n": 1, "basis": "6-31g*", "spins": 1, "cutoff": 0.0},
        # an open-shell run of a drawn organic molecule: two densities, odd sizes
        {"name": "jk_uhf_molecule", "kind": "jk", "mol": "tree", "n": 9, "basis": "6-31g*", "spins": 2, "cutoff": 0.0},
        # the benchmark's cluster, one full Fock build, in FP64 and as the
        # benchmark's mixed-precision path builds it (FP32 quartets below 1e-3)
        {"name": "jk_water32_mixed", "kind": "jk", "mol": "water", "n": 32, "basis": "cc-pvdz", "spins": 1, "cutoff": 1e-3},
        {"name": "jk_water32", "kind": "jk", "mol": "water", "n": 32, "basis": "cc-pvdz", "spins": 1, "cutoff": 0.0},
        # an SCF iteration after the first, on the medium cluster and on a large one
        {"name": "delta_water8", "kind": "delta", "mol": "water", "n": 8, "basis": "cc-pvdz", "spins": 1, "cutoff": 0.0},
        {"name": "delta_water27", "kind": "delta", "mol": "water", "n": 27, "basis": "cc-pvdz", "spins": 1, "cutoff": 0.0},
        # forces: a small molecule, the medium cluster, the benchmark's cluster
        {"name": "grad_methanol", "kind": "grad", "mol": "methanol", "n": 1, "basis": "6-31g**", "spins": 1, "cutoff": 0.0},
        {"name": "grad_water8", "kind": "grad", "mol": "water", "n": 8, "basis": "cc-pvdz", "spins": 1, "cutoff": 0.0},
        {"name": "grad_water32", "kind": "grad", "mol": "water", "n": 32, "basis": "cc-pvdz", "spins": 1, "cutoff": 0.0},
        # the set-up of every MD step of the benchmark's cluster
        {"name": "frame_water32", "kind": "frame", "mol": "water", "n": 32, "basis": "cc-pvdz", "spins": 1, "cutoff": 0.0},
        # whole MD steps of a small molecule
        {"name": "force_methanol", "kind": "force", "mol": "methanol", "n": 1, "basis": "6-31g**", "spins": 1, "cutoff": 0.0},
        # a screening run over conformers
        {"name": "batch_molecules", "kind": "batch", "mol": "tree", "n": 6, "basis": "6-31g*", "spins": 1, "cutoff": 0.0},
    ]


def draw(rng):
    kind = rng.choice(["jk", "jk", "delta", "grad", "grad", "frame", "force"])
    mol = rng.choice(["water", "water", "tree"])
    # waters of the cluster, or heavy-atom trees by their number in the family
    top = {"jk": 32, "delta": 32, "grad": 24, "frame": 32, "force": 3}[kind]
    n = round(math.exp(rng.uniform(0.0, math.log(top)))) if mol == "water" else rng.randrange(100)
    basis = rng.choice(["sto-3g", "6-31g", "6-31g*", "6-31g**", "cc-pvdz", "cc-pvdz"])
    spins = 2 if kind in ("jk", "delta", "grad") and n <= 16 and rng.random() < 0.3 else 1
    cutoff = rng.choice({"jk": [0.0, 0.0, 1e-7, 1e-3], "delta": [0.0, 0.0, 1e-7], "grad": [0.0, 0.0, 1e-7]}.get(kind, [0.0]))
    return {"kind": kind, "mol": mol, "n": n, "basis": basis, "spins": spins, "cutoff": cutoff}


# ------------------------------------------------------------------ inputs

@functools.lru_cache(maxsize=None)
def _resting(mol, n):
    """Symbols and positions (bohr) before the thermal displacement."""
    if mol == "methanol":
        return geometry.methanol()
    if mol == "tree":
        return geometry.random_molecule(n)
    if n == 1:
        return geometry.water()
    # n waters of the 32-water cube nearest to its middle
    sym, x = geometry.water_cluster(32, seed=1)
    mid = x.reshape(32, 3, 3)[:, 0]
    keep = np.sort(np.argsort(np.linalg.norm(mid - mid.mean(axis=0), axis=1))[:n])
    return sym[:3] * n, x.reshape(32, 9)[keep].reshape(-1, 3)


def _geometry(case, seed, frame=0):
    """Thermal displacements (0.03 bohr) of the resting geometry, freely rotated; frames are 0.01 bohr apart."""
    sym, x = _resting(case["mol"], case["n"])
    rng = np.random.default_rng([seed, 1])
    q, _ = np.linalg.qr(rng.normal(size=(3, 3)))
    x = (x + rng.normal(scale=0.03, size=x.shape)) @ q
    for _ in range(frame):
        x = x + rng.normal(scale=0.01, size=x.shape)
    return sym, x


def _density(basis, seed, scale=1.0):
    """A symmetric density of localised orbitals: one per electron pair, centred near an atom, decaying by 1.1 per bohr."""
    rng = np.random.default_rng([seed, 2])
    z = np.asarray(basis.atomic_numbers)
    home = np.repeat(np.arange(len(z)), np.maximum(1, z // 2))
    at = basis.positions[home] + rng.normal(scale=0.3, size=(len(home), 3))
    r = np.linalg.norm(basis.positions[np.asarray(basis.ao_atom)][:, None] - at[None], axis=2)
    C = rng.normal(scale=0.4, size=r.shape) * np.exp(-1.1 * r)
    return scale * 2.0 * C @ C.T


def _gpu(x):
    return torch.as_tensor(np.ascontiguousarray(x), device="cuda", dtype=torch.float64)


def prepare(case, seed):
    sym, x = _geometry(case, seed)
    kind = case["kind"]
    if kind == "batch":
        mols = [geometry.random_molecule(100 * case["n"] + i) for i in range(case["n"])]
        rng = np.random.default_rng([seed, 3])
        frames = [[p + rng.normal(scale=0.03, size=p.shape) for _, p in mols] for _ in range(2)]
        opts = SCFOptions(warn_unconverged=False)
        return {"kind": kind, "solver": BatchSolver(mols, case["basis"], opts), "frames": frames}
    if kind == "force":
        solver = SCFSolver(sym, case["basis"])
        frames = [_geometry(case, seed, k)[1] for k in range(3)]
        start = run_device(solver, frames[0])
        return {"kind": kind, "solver": solver, "frames": frames[1:], "guess": start.spin[0] + start.spin[1]}
    basis = build_basis(sym, x, case["basis"])
    state = {"kind": kind, "basis": basis, "cutoff": case["cutoff"]}
    D = [_density(basis, seed + 1000 * s) for s in range(case["spins"])]
    if kind == "delta":
        # the change of an SCF's middle iterations: 1e-3 of the density
        state["D"] = _gpu(np.stack([1e-3 * (d - _density(basis, seed + 77 + s)) for s, d in enumerate(D)]))
    else:
        state["D"] = _gpu(np.stack(D))
    if kind == "grad":
        state["P"] = state["D"].sum(dim=0)
    if kind == "frame":
        state["frames"] = [basis, basis.with_positions(_geometry(case, seed, 1)[1])]
        state["P"] = state["D"][0]
        state["W"] = _gpu(_density(basis, seed + 5, -0.5))
    engine_for(basis)
    return state


# --------------------------------------------------------------------- run

def run(state):
    kind = state["kind"]
    if kind == "jk":
        return I.jk_device(state["basis"], state["D"], THR, True, state["cutoff"])
    if kind == "delta":
        J, K = engine_for(state["basis"]).jk_delta_acc(state["D"], THR, THR_DELTA, state["cutoff"])
        return J + J.transpose(1, 2), K + K.transpose(1, 2)
    if kind == "grad":
        k = 0.5 if state["D"].shape[0] == 1 else 1.0
        return I.two_electron_gradient_device(state["basis"], state["P"], state["D"], k, THR_GRAD, state["cutoff"])
    if kind == "frame":
        out = []
        for b in state["frames"]:
            Q = engine_for(b).schwarz()
            S, T, M, V = I.one_electron_device(b)
            out.append({"Q": Q, "S": S, "T": T, "M": M, "V": V,
                        "g": I.one_electron_gradient_device(b, state["P"], state["W"])})
        return out
    if kind == "force":
        out, guess = [], state["guess"]
        for x in state["frames"]:
            st = run_device(state["solver"], x, guess)
            guess = st.spin[0] + st.spin[1]
            out.append({"energy": st.energy, "gradient": scf_gradient_device(st), "fock": st.fock, "density": guess})
        return out
    res = [r for x in state["frames"] for r in state["solver"].run(x)]
    return {"energy": np.array([r.energy for r in res]), "gradient": np.concatenate([r.gradient for r in res]),
            "dipole": np.stack([r.dipole for r in res])}


# -------------------------------------------------------------------- work

def _quartets(basis):
    """
    (unique shell quartets that a Schwarz bound of 1e-12 leaves, by the s-type
    estimate of each shell pair's bound; FP64 operations of their integrals):
    per primitive quartet the recursion to R_tuv (a multiplication and an
    addition an entry and level), then both Hermite-to-Cartesian steps of the
    contracted quartet over the non-zero boxes (a quarter of the dense ones).
    """
    sh = basis.nshell
    x = basis.shell_centers
    p0 = np.asarray(basis.shell_prim)
    l = np.asarray(basis.shell_l)
    amin = np.array([basis.prim_exp[p0[s]:p0[s + 1]].min() for s in range(sh)])
    npr = np.diff(p0)
    i, j = np.tril_indices(sh)
    r2 = ((x[i] - x[j]) ** 2).sum(axis=1)
    a, b = amin[i], amin[j]
    p = a + b
    q = (4 * a * b / p ** 2) ** 0.75 * np.exp(-a * b / p * r2) * (2.0 * p / math.pi) ** 0.25
    npp = npr[i] * npr[j]
    lp = l[i] + l[j]
    nc = ((l + 1) * (l + 2) // 2)
    ncd = nc[i] * nc[j]
    nh = lambda L: (L + 1) * (L + 2) * (L + 3) // 6  # noqa: E731
    flops = total = 0.0
    cls = [np.flatnonzero(lp == L) for L in range(5)]
    for L1 in range(5):
        for L2 in range(L1 + 1):
            A, B = cls[L1], cls[L2]
            if not len(A) or not len(B):
                continue
            order = B[np.argsort(-q[B])]
            kept = np.searchsorted(-q[order], -1e-12 / q[A], side="right")
            cp, cn = np.concatenate([[0.0], np.cumsum(npp[order])]), np.concatenate([[0.0], np.cumsum(ncd[order])])
            half = 0.5 if L1 == L2 else 1.0
            per = 2.0 * sum(nh(L1 + L2 - n) for n in range(L1 + L2 + 1))
            total += half * kept.sum()
            flops += half * per * (npp[A] * cp[kept]).sum()
            flops += half * 0.25 * 2.0 * (nh(L1) * nh(L2) * cn[kept] + nh(L1) * ncd[A] * cn[kept]).sum()
    return total, flops


@functools.lru_cache(maxsize=None)
def _counted(mol, n, name):
    sym, x = _resting(mol, n)
    b = build_basis(sym, x, name)
    kept, flops = _quartets(b)
    return b.nao, b.natm, float(kept), float(flops), b.nshell * (b.nshell + 1) // 2


def work(case):
    kind = case["kind"]
    if kind == "batch":
        parts = [_counted("tree", 100 * case["n"] + i, case["basis"]) for i in range(case["n"])]
        # about ten Fock builds and a gradient of each molecule, at two frames
        return {"bytes": sum(2 * 11 * 24 * p[0] ** 2 for p in parts), "flops": sum(2 * 13 * p[3] for p in parts)}
    nao, natm, _, flops, pairs = _counted(case["mol"], case["n"], case["basis"])
    s = case["spins"]
    nn = 8.0 * nao * nao
    if kind in ("jk", "delta"):
        return {"bytes": 3 * s * nn, "flops": flops * (1.0 if kind == "jk" else 0.5)}
    if kind == "grad":
        return {"bytes": (s + 1) * nn + 24 * natm, "flops": 3.0 * flops}
    if kind == "frame":
        return {"bytes": 2 * (8 * nn + 8 * pairs), "flops": 2 * 2.0e2 * pairs * natm}
    return {"bytes": 2 * 11 * 3 * nn, "flops": 2 * 13 * flops}


# ------------------------------------------------------------------- exact

def exact(case, seed):
    """Plain 64-bit Hermite (McMurchie-Davidson) integrals without screening, for the small molecules."""
    if case["kind"] not in ("jk", "delta", "grad"):
        return None
    sym, x = _geometry(case, seed)
    basis = build_basis(sym, x, case["basis"])
    if basis.nao > (100 if case["kind"] != "grad" else 30):
        return None
    D = [_density(basis, seed + 1000 * s) for s in range(case["spins"])]
    if case["kind"] == "delta":
        D = [1e-3 * (d - _density(basis, seed + 77 + s)) for s, d in enumerate(D)]
    D = _gpu(np.stack(D))
    if case["kind"] == "grad":
        pos = _gpu(x).requires_grad_(True)
        eri = _eri(basis, pos)
        P = D.sum(dim=0)
        k = 0.5 if len(D) == 1 else 1.0
        e = 0.5 * torch.einsum("mnls,mn,ls->", eri, P, P) - 0.5 * k * torch.einsum("mnls,xml,xns->", eri, D, D)
        return torch.autograd.grad(e, pos)[0]
    with torch.no_grad():
        eri = _eri(basis, _gpu(x))
        return torch.einsum("mnls,xls->xmn", eri, D), torch.einsum("mlns,xls->xmn", eri, D)


class _Boys(torch.autograd.Function):
    """F_0 .. F_N (stacked) of T: the ascending series below 40, the asymptotic form above; dF_n/dT = -F_{n+1}."""

    @staticmethod
    def forward(ctx, T, N):
        M = N + 1
        low = torch.clamp(T, max=40.0)
        term = torch.full_like(T, 1.0 / (2 * M + 1))
        top = term.clone()
        for k in range(1, 170):
            term = term * (2.0 * low / (2 * M + 2 * k + 1))
            top = top + term
        ex = torch.exp(-T)
        F = [None] * (M + 1)
        F[M] = torch.exp(-low) * top
        for n in range(M - 1, -1, -1):
            F[n] = (2.0 * low * F[n + 1] + torch.exp(-low)) / (2 * n + 1)
        big = T > 40.0
        up = torch.sqrt(math.pi / torch.clamp(T, min=1.0)) * 0.5
        for n in range(M + 1):
            F[n] = torch.where(big, up, F[n])
            up = ((2 * n + 1) * up - ex) / (2.0 * torch.clamp(T, min=1.0))
        F = torch.stack(F)
        ctx.save_for_backward(F)
        return F[:M]

    @staticmethod
    def backward(ctx, g):
        (F,) = ctx.saved_tensors
        return -(g * F[1:]).sum(dim=0), None


def _pairs(basis, pos):
    """Per angular class (la, lb): exponents, centres and Hermite rows of all primitive pairs, and their AO pairs."""
    p0, l, atom = np.asarray(basis.shell_prim), np.asarray(basis.shell_l), np.asarray(basis.shell_atom)
    got = {}
    for i in range(basis.nshell):
        for j in range(basis.nshell):
            if (l[i], i) < (l[j], j):
                continue
            ka, kb = (v.reshape(-1) for v in np.meshgrid(np.arange(p0[i], p0[i + 1]), np.arange(p0[j], p0[j + 1]), indexing="ij"))
            w = got.setdefault((int(l[i]), int(l[j])), [[], [], [], []])
            w[0].append(ka), w[1].append(kb), w[2].append(np.full(len(ka), i)), w[3].append(np.full(len(ka), j))
    out = []
    for (la, lb), w in sorted(got.items()):
        ka, kb, si, sj = (np.concatenate(v) for v in w)
        a, b = _gpu(basis.prim_exp[ka]), _gpu(basis.prim_exp[kb])
        c = _gpu(basis.prim_coef[ka] * basis.prim_coef[kb])
        A, B = pos[torch.as_tensor(atom[si], device="cuda")], pos[torch.as_tensor(atom[sj], device="cuda")]
        p = a + b
        P = (a[:, None] * A + b[:, None] * B) / p[:, None]
        E = []
        for d in range(3):
            ab = A[:, d] - B[:, d]
            e = {(0, 0): [torch.exp(-a * b / p * ab * ab)]}
            for n in range(1, la + lb + 1):
                for i in range(max(0, n - lb), min(la, n) + 1):
                    j = n - i
                    old, s = (e[i - 1, j], P[:, d] - A[:, d]) if i else (e[i, j - 1], P[:, d] - B[:, d])
                    z = torch.zeros_like(p)
                    g = lambda t: old[t] if 0 <= t < len(old) else z  # noqa: B023,E731
                    e[i, j] = [s * g(t) + (t + 1) * g(t + 1) + g(t - 1) / (2 * p) for t in range(n + 1)]
            E.append(e)
        cart = lambda L: [(u, v, L - u - v) for u in range(L, -1, -1) for v in range(L - u, -1, -1)]  # noqa: E731
        odd = lambda n: math.prod(range(n, 0, -2)) if n > 0 else 1  # noqa: E731
        norm = lambda u: math.sqrt(odd(2 * sum(u) - 1) / math.prod(odd(2 * k - 1) for k in u))  # noqa: E731
        L = la + lb
        herm = [(t, u, v) for t in range(L + 1) for u in range(L + 1 - t) for v in range(L + 1 - t - u)]
        ao = torch.as_tensor(np.asarray(basis.shell_ao)[:-1], device="cuda")
        I_, J_ = torch.as_tensor(si, device="cuda"), torch.as_tensor(sj, device="cuda")
        rows = []
        for x, u in enumerate(cart(la)):
            for y, v in enumerate(cart(lb)):
                f = norm(u) * norm(v) * c
                pick = lambda d, t: E[d][u[d], v[d]][t] if t <= u[d] + v[d] else None  # noqa: B023,E731
                r = []
                for h in herm:
                    k = [pick(d, h[d]) for d in range(3)]
                    r.append(torch.zeros_like(p) if any(q is None for q in k) else f * k[0] * k[1] * k[2])
                rows.append((ao[I_] + x, ao[J_] + y, I_ != J_, torch.stack(r)))
        out.append((L, herm, p, P, rows))
    return out


def _hermite(p, P, q, Q, L):
    """{(t, u, v): R} of all primitive pairs of p against q, to total degree L."""
    X = [P[:, None, d] - Q[None, :, d] for d in range(3)]
    s = p[:, None] + q[None, :]
    al = p[:, None] * q[None, :] / s
    F = _Boys.apply(al * (X[0] ** 2 + X[1] ** 2 + X[2] ** 2), L)
    pref = 2.0 * math.pi ** 2.5 / (p[:, None] * q[None, :] * torch.sqrt(s))
    R = {}
    for n in range(L, -1, -1):
        new = {(0, 0, 0): pref * (-2.0 * al) ** n * F[n]}
        for t in range(L - n + 1):
            for u in range(L - n - t + 1):
                for v in range(L - n - t - u + 1):
                    if t + u + v == 0:
                        continue
                    d = 0 if t else (1 if u else 2)
                    h = [t, u, v]
                    h[d] -= 1
                    r = X[d] * R[tuple(h)]
                    if h[d]:
                        k = h[d]
                        h[d] -= 1
                        r = r + k * R[tuple(h)]
                    new[t, u, v] = r
        R = new
    return R


def _eri(basis, pos):
    """(mn|ls), all of it: Hermite integrals of the classes, contracted into AO pairs by dense products."""
    n = basis.nao
    prs = _pairs(basis, pos)
    full = torch.zeros((n * n, n * n), dtype=torch.float64, device="cuda")

    def spread(rows, k, lo, hi):
        """[n n, primitive pairs lo..hi]: Hermite entry k of every AO pair."""
        out = torch.zeros((n * n, hi - lo), dtype=torch.float64, device="cuda")
        col = torch.arange(hi - lo, device="cuda")
        for m, l_, two, r in rows:
            v = r[k, lo:hi]
            out = out.index_put((m[lo:hi] * n + l_[lo:hi], col), v, accumulate=True)
            off = two[lo:hi]                # pairs of two shells stand for both orders
            out = out.index_put(((l_ * n + m)[lo:hi][off], col[off]), v[off], accumulate=True)
        return out

    for L1, h1, p, P, r1 in prs:
        for lo in range(0, len(p), 1024):
            hi = min(len(p), lo + 1024)
            acc = [torch.zeros((hi - lo, n * n), dtype=torch.float64, device="cuda") for _ in h1]
            for L2, h2, q, Q, r2 in prs:
                R = _hermite(p[lo:hi], P[lo:hi], q, Q, L1 + L2)
                for kk, g in enumerate(h2):
                    ket = spread(r2, kk, 0, len(q)).T * (-1.0) ** sum(g)
                    for k, h in enumerate(h1):
                        acc[k] = acc[k] + R[h[0] + g[0], h[1] + g[1], h[2] + g[2]] @ ket
            for k in range(len(h1)):
                full = full + spread(r1, k, lo, hi) @ acc[k]
    return full.reshape(n, n, n, n)
