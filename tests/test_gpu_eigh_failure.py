"""
What aimd_eigh says of matrices it cannot solve (NaN in every output), that the
SCF raises for it, and matrices whose squares leave the range of FP64.
"""

from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _run(A, V=None):
    import torch
    from aimd_b200 import _lib
    n = A.shape[0]
    out = torch.full_like(A, 7.0) if V is None else V.contiguous().clone()
    w = torch.full((n,), 7.0, dtype=A.dtype, device=A.device)
    _lib.check(_lib.load().aimd_eigh(n, A.data_ptr(), out.data_ptr(), w.data_ptr(), int(V is not None),
                                     torch.cuda.current_stream().cuda_stream), "aimd_eigh")
    return w, out


def _matrix(n):
    import torch
    g = torch.Generator().manual_seed(n)
    A = torch.randn(n, n, generator=g, dtype=torch.float64)
    return (A + A.T).cuda()


@pytest.mark.parametrize("bad", [float("nan"), float("inf"), -float("inf")])
@pytest.mark.parametrize("n", [1, 2, 33, 64])
def test_not_finite(n, bad):
    import torch
    for at in {(0, 0), (n - 1, 0), (n - 1, n - 1)}:
        A = _matrix(n)
        A[at] = bad
        w, V = _run(A)
        assert bool(torch.isnan(w).all()) and bool(torch.isnan(V).all())
    # starting vectors
    U = torch.eye(n, dtype=torch.float64, device="cuda")
    U[0, n - 1] = bad
    w, V = _run(_matrix(n), U)
    assert bool(torch.isnan(w).all()) and bool(torch.isnan(V).all())


def test_upper_triangle_is_not_read():
    import torch
    A = _matrix(9)
    w, V = _run(A)
    B = torch.tril(A) + torch.triu(torch.full_like(A, float("nan")), 1)
    w2, V2 = _run(B)
    assert torch.equal(w, w2) and torch.equal(V, V2)


@pytest.mark.parametrize("exponent", [-1060, -1000, -600, 0, 600, 1000])
@pytest.mark.parametrize("n", [2, 7, 64])
def test_scaled_by_a_power_of_two(n, exponent):
    """Scaling is exact, so the vectors are the same bits; the eigenvalues too, where they are normal numbers."""
    import torch
    A = torch.round(_matrix(n) * 2.0 ** 10)             # whole numbers: nothing is lost at 2^-1060
    w, V = _run(A)
    s = torch.as_tensor(np.ldexp(A.cpu().numpy(), exponent)).cuda()
    assert bool(torch.isfinite(s).all())
    w2, V2 = _run(s)
    assert torch.equal(V, V2)
    back = np.ldexp(w2.cpu().numpy(), -exponent)
    step = np.ldexp(1.0, -1074 - exponent) if exponent < -1000 else 0.0
    assert np.abs(back - w.cpu().numpy()).max() <= step


def test_scf_raises_for_nan_vectors(monkeypatch):
    """A Fock matrix that turns NaN after the commutator was found finite: the failure the host cannot see in the call."""
    import torch
    from aimd_b200 import _lib, geometry
    from aimd_b200.scf import run_scf
    lib = _lib.load()
    real = lib.aimd_eigh
    calls = []

    class Lib:
        def __getattr__(self, name):
            return getattr(lib, name)

        def aimd_eigh(self, n, A, V, w, warm, stream):
            calls.append(n)
            if len(calls) == 2:
                bad = torch.full((n, n), float("nan"), dtype=torch.float64, device="cuda")
                return real(n, bad.data_ptr(), V, w, warm, stream)
            return real(n, A, V, w, warm, stream)

    monkeypatch.setattr(_lib, "load", lambda: Lib())
    sym, x = geometry.water()
    with pytest.raises(torch.linalg.LinAlgError):
        run_scf(sym, x, "sto-3g")
    assert len(calls) == 2
