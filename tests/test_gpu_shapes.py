"""
The integral kernels at the edges of their work split, against the oracle:
molecules of 1 to 33 atoms (fewer and more nuclei than the lanes of a warp),
every basis set's classes and contraction counts, ket lists shorter than a
warp and longer than one queue.

Tolerances: 1e-10 per unit of the result's largest element (at least 1) for
FP64 sums of up to 1e5 terms whose own rounding is 1e-16 and whose
fixed-point step is 6e-14.
"""

from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

MOLECULES = [("atom", "cc-pvdz"), ("water", "sto-3g"), ("water", "cc-pvdz"), ("tree7", "6-31g"), ("tree2", "6-31g*"),
             ("cluster11", "6-31g**")]


def _case(name, basis_name):
    from aimd_b200 import geometry as G
    from aimd_b200.basis import build_basis
    if name == "atom":
        sym, x = ["O"], np.array([[0.1, -0.2, 0.3]])
    elif name == "water":
        sym, x = G.water()
    elif name.startswith("tree"):
        sym, x = G.random_molecule(int(name[4:]))
    else:
        sym, x = G.water_cluster(int(name[7:]), seed=2)
    basis = build_basis(sym, x, basis_name)
    rng = np.random.default_rng(7)
    r = np.linalg.norm(x[:, None] - x[None], axis=2)[np.ix_(basis.ao_atom, basis.ao_atom)]
    D = rng.normal(size=(2, basis.nao, basis.nao)) * np.exp(-0.3 * r)
    return basis, 0.5 * (D + D.transpose(0, 2, 1))


def _close(got, ref, what):
    tol = 1e-10 * max(1.0, float(np.abs(ref).max()))
    assert np.abs(np.asarray(got) - ref).max() <= tol, what


@pytest.mark.parametrize("name,basis_name", MOLECULES)
def test_two_electron_gradient(name, basis_name):
    from aimd_b200 import integrals as I
    from oracle import hf_oracle as O
    b, D = _case(name, basis_name)
    _close(I.two_electron_gradient(b, D[0], [D[0]], 0.5), O.two_electron_gradient(b, D[0], [D[0]], 0.5), "RHF")
    _close(I.two_electron_gradient(b, D[0] + D[1], list(D), 1.0),
           O.two_electron_gradient(b, D[0] + D[1], list(D), 1.0), "UHF")
    _close(I.two_electron_gradient(b, D[0], [], 0.0), O.two_electron_gradient(b, D[0], [], 0.0), "no exchange")


@pytest.mark.parametrize("name,basis_name", MOLECULES)
def test_jk_and_difference_build(name, basis_name):
    """Full builds, and difference builds (queued ket pairs) whose threshold drops at most 1e-15 a quartet."""
    import torch
    from aimd_b200 import integrals as I
    from aimd_b200.engine import engine_for
    from oracle import hf_oracle as O
    b, D = _case(name, basis_name)
    J, K = I.jk(b, D)
    Jr, Kr = O.jk_direct(b, D)
    _close(J, Jr, "J")
    _close(K, Kr, "K")
    Dt = torch.as_tensor(D, device="cuda")
    for scale in (1.0, 1e-4):
        Ja, Ka = engine_for(b).jk_delta_acc(scale * Dt, 1e-12, 1e-15 * scale)
        _close((Ja + Ja.transpose(1, 2)).cpu().numpy() / scale, Jr, "difference J")
        _close((Ka + Ka.transpose(1, 2)).cpu().numpy() / scale, Kr, "difference K")


@pytest.mark.parametrize("name,basis_name", MOLECULES)
def test_schwarz_bounds(name, basis_name):
    from aimd_b200 import integrals as I
    from oracle import hf_oracle as O
    b, _ = _case(name, basis_name)
    Q = O.schwarz_bounds(b)
    # Q^2 = max (ab|ab) is what is computed: rounding is relative to the largest integral
    assert np.abs(I.schwarz_bounds(b) ** 2 - Q ** 2).max() <= 1e-12 * max(1.0, Q.max() ** 2)


@pytest.mark.parametrize("name,basis_name", MOLECULES)
def test_one_electron(name, basis_name):
    from aimd_b200 import integrals as I
    from oracle import hf_oracle as O
    b, D = _case(name, basis_name)
    S, T, V = I.one_electron_matrices(b)
    for got, ref, what in zip((S, T, V), O.one_electron_matrices(b), "STV"):
        _close(got, ref, what)
    _close(I.dipole_integrals(b), O.dipole_integrals(b), "dipole")
    _close(I.one_electron_gradient(b, D[0], D[1]), O.one_electron_gradient(b, D[0], D[1]), "gradient")


@pytest.mark.parametrize("distance", [0.3, 1.4, 2.9, 4.4, 5.1, 6.3, 9.0, 17.0])
def test_boys_arguments(distance):
    """An O-H pair from overlapping to far apart: Boys arguments 0 to some thousands, both sides of the table's end."""
    from aimd_b200 import integrals as I
    from aimd_b200.basis import build_basis
    from oracle import hf_oracle as O
    x = np.array([[0.0, 0.0, 0.0], distance * np.array([0.48, 0.60, 0.64])])
    b = build_basis(["O", "H"], x, "cc-pvdz")
    rng = np.random.default_rng(3)
    D = rng.normal(size=(b.nao, b.nao))
    D = D + D.T
    for got, ref, what in zip(I.jk(b, D), O.jk_direct(b, D), "JK"):
        _close(got, ref, what)
    _close(I.two_electron_gradient(b, D, [D], 0.5), O.two_electron_gradient(b, D, [D], 0.5), "gradient")


def _cluster(n):
    from aimd_b200 import geometry as G
    from aimd_b200.basis import build_basis
    # n waters on a grid of 3.1 A: any n, no random placement
    _, mono = G.water()
    k = int(np.ceil(n ** (1.0 / 3.0)))
    cells = [(i, j, m) for i in range(k) for j in range(k) for m in range(k)][:n]
    x = np.concatenate([mono - mono[0] + 5.86 * np.array(c, dtype=float) for c in cells])
    b = build_basis(["O", "H", "H"] * n, x, "cc-pvdz")
    rng = np.random.default_rng(1)
    r = np.linalg.norm(x[:, None] - x[None], axis=2)[np.ix_(b.ao_atom, b.ao_atom)]
    D = rng.normal(size=r.shape) * np.exp(-0.5 * r)
    return b, 0.5 * (D + D.T)


@pytest.mark.parametrize("n", [1, 9, 44])
def test_jk_row_layouts_agree(n, monkeypatch):
    """
    K rows in shared and in global memory, D rows staged or not: at 44 waters
    (1100 AOs) the dp kernels no longer hold both sets of rows.
    """
    import torch
    from aimd_b200.engine import Engine
    b, D = _cluster(n)
    Dt = torch.as_tensor(D[None], device="cuda")
    out = []
    for rows in ("0", "1"):
        monkeypatch.setenv("AIMD_JK_GLOBAL_K_ROWS", rows)
        eng = Engine(b)
        eng.set_geometry(b.positions)
        out.append([t.cpu().numpy() for t in eng.jk_acc(Dt, 1e-12)])
    for x, y in zip(*out):
        _close(x, y, "row layouts")


@pytest.mark.parametrize("n", [1, 8, 27])
def test_gradient_exchange_layouts_agree(n):
    """One exchange density, and the same with a second one of zeros (twice the D rows, which at 27 waters do not fit)."""
    import torch
    from aimd_b200 import integrals as I
    b, D = _cluster(n)
    Dt = torch.as_tensor(D, device="cuda")
    one = I.two_electron_gradient_device(b, Dt, Dt[None].contiguous(), 0.5).cpu().numpy()
    two = I.two_electron_gradient_device(b, Dt, torch.stack([Dt, torch.zeros_like(Dt)]), 0.5).cpu().numpy()
    none = I.two_electron_gradient_device(b, Dt, torch.empty((0, b.nao, b.nao), dtype=torch.float64, device="cuda"), 0.5)
    _close(two, one, "exchange densities")
    assert np.isfinite(none.cpu().numpy()).all()


@pytest.mark.parametrize("n", [1, 2, 9])
def test_split_lengths_agree(n):
    """Items split by the launch's work (1, 2 waters: the shortest, 9: the shape's own length) under several launch shapes."""
    import torch
    from aimd_b200.engine import Engine
    b, D = _cluster(n)
    Dt = torch.as_tensor(D[None], device="cuda")
    out = []
    for shape in ((8, 32), (8, 4), (64, 4096), (1, 5)):
        eng = Engine(b)
        eng.set_geometry(b.positions)
        eng.set_launch_shape(*shape)
        out.append([t.cpu().numpy() for t in (*eng.jk_acc(Dt, 1e-12), *eng.jk_delta_acc(Dt, 1e-12, 1e-15))])
    for other in out[1:]:
        for x, y in zip(out[0], other):
            _close(y, x, "launch shape")
