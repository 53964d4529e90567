"""
The FP32 instantiations of the integral kernels at the edges of their work
split: the molecules and basis sets of the FP64 tests, two densities, K rows in
global memory, difference builds, launch shapes; against the same call in FP64.

Tolerance. A quartet in FP32 is off by at most some 1e-5 of its Schwarz product
Q1 Q2, which is below the cutoff: 6e-8 for each of the operations of up to 4096
primitive quartets that enter with either sign. An element of J or K sums at most
n^2 of them times elements of D, with either sign: n max|D| 1e-5 min(cutoff,
max Q^2). The gradient carries two densities, and a derivative of up to ten times
the integral.
"""

from __future__ import annotations

import numpy as np
import pytest

from test_gpu_shapes import MOLECULES, _case, _cluster

pytestmark = pytest.mark.gpu
CUTOFFS = [1e-7, 1e-3, 1e3]         # a tail of the quartets, most, all


def _engine(b):
    from aimd_b200.engine import Engine
    eng = Engine(b)
    eng.set_geometry(b.positions)
    return eng


def _tol(eng, D, cutoff):
    q2 = float(eng.schwarz().max()) ** 2
    return 1e-5 * eng.nao * float(D.abs().max()) * min(cutoff, q2) + 1e-10


def _builds(eng, D, cutoff):
    return (*eng.jk_acc(D, 1e-12, cutoff), *eng.jk_delta_acc(D, 1e-12, 1e-15, cutoff))


@pytest.mark.parametrize("rows", ["0", "1"])
@pytest.mark.parametrize("cutoff", CUTOFFS)
@pytest.mark.parametrize("name,basis_name", MOLECULES)
def test_jk_two_densities(name, basis_name, cutoff, rows, monkeypatch):
    import torch
    monkeypatch.setenv("AIMD_JK_GLOBAL_K_ROWS", rows)
    b, D = _case(name, basis_name)
    eng = _engine(b)
    D = torch.as_tensor(D, device="cuda")
    ref, got = _builds(eng, D, 0.0), _builds(eng, D, cutoff)
    # a difference build applies the cutoff to Q1 Q2 max|D|, which is the same bound divided by max|D|
    m = max(1.0, 1.0 / float(D.abs().max()))
    for x, y in zip(got, ref):
        assert float((x - y).abs().max()) <= m * _tol(eng, D, cutoff)
    for x, y in zip(_builds(eng, D, cutoff), got):          # and the same bits again
        assert torch.equal(x, y)


@pytest.mark.parametrize("cutoff", CUTOFFS)
@pytest.mark.parametrize("name,basis_name", MOLECULES)
def test_gradient(name, basis_name, cutoff):
    import torch
    from aimd_b200 import integrals as I
    b, D = _case(name, basis_name)
    D = torch.as_tensor(D, device="cuda")
    none = torch.empty((0, b.nao, b.nao), dtype=torch.float64, device="cuda")
    for Dc, Dx, k in ((D[0], D[:1].contiguous(), 0.5), (D[0] + D[1], D, 1.0), (D[0], none, 0.0)):
        Dc = Dc.contiguous()
        ref = I.two_electron_gradient_device(b, Dc, Dx, k)
        got = I.two_electron_gradient_device(b, Dc, Dx, k, fp32_cutoff=cutoff)
        top = torch.cat([Dc[None], Dx]).abs().max()
        from aimd_b200.engine import engine_for
        assert float((got - ref).abs().max()) <= 10 * (1 + len(Dx)) * float(top) * _tol(engine_for(b), top, cutoff)


@pytest.mark.parametrize("n", [1, 9, 44])
def test_launch_shapes(n):
    """Items split and chunks cut in other ways, up to 1100 AOs: the same FP32 values summed in another order."""
    import torch
    b, D = _cluster(n)
    D = torch.as_tensor(D[None], device="cuda")
    eng = _engine(b)
    ref = _builds(eng, D, 1e-3)
    for shape in ((8, 32), (4, 4096), (1, 5)) if n < 44 else ((8, 32), (4, 4096)):
        eng.set_launch_shape(*shape)
        for x, y in zip(_builds(eng, D, 1e-3), ref):
            assert float((x - y).abs().max()) <= max(1.0, 1.0 / float(D.abs().max())) * _tol(eng, D, 1e-3)
