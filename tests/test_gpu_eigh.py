"""
The one-CTA symmetric eigensolver (aimd_eigh) against its definition: sizes 1
to the limit, odd and even, degenerate and graded spectra, started from scratch
and from the vectors of a nearby matrix. Residual and orthogonality bounds are
those of a backward-stable solver, a modest multiple of n eps |A|.
"""

from __future__ import annotations

import pytest

pytestmark = pytest.mark.gpu


def _run(A, V=None):
    import torch
    from aimd_b200 import _lib
    n = A.shape[0]
    warm = V is not None
    V = V.clone() if warm else torch.full_like(A, float("nan"))
    w = torch.empty(n, dtype=A.dtype, device=A.device)
    _lib.check(_lib.load().aimd_eigh(n, A.data_ptr(), V.data_ptr(), w.data_ptr(), int(warm),
                                     torch.cuda.current_stream().cuda_stream), "aimd_eigh")
    return w, V


def _check(A, w, V):
    import torch
    n = A.shape[0]
    bound = 50 * n * 2.3e-16
    scale = float(torch.linalg.matrix_norm(A)) + 1e-300
    assert float((A @ V - V * w).abs().max()) <= bound * scale
    assert float((V.T @ V - torch.eye(n, dtype=A.dtype, device=A.device)).abs().max()) <= bound
    assert bool((w[1:] >= w[:-1]).all())


@pytest.mark.parametrize("kind", ["random", "degenerate", "graded", "diagonal", "zero"])
@pytest.mark.parametrize("n", [1, 2, 3, 7, 19, 32, 33, 50, 63, 64])
def test_eigh(n, kind):
    import torch
    g = torch.Generator().manual_seed(n)
    A = torch.randn(n, n, generator=g, dtype=torch.float64)
    A = A + A.T
    if kind != "random":
        Q, _ = torch.linalg.qr(A)
        d = {"degenerate": torch.tensor([-1.0, 2.0]).repeat(n)[:n], "graded": 10.0 ** -torch.linspace(0, 14, n),
             "diagonal": torch.arange(n), "zero": torch.zeros(n)}[kind].double()
        A = torch.diag(d) if kind == "diagonal" else Q @ torch.diag(d) @ Q.T
        A = 0.5 * (A + A.T)
    A = A.cuda()
    w, V = _run(A)
    _check(A, w, V)
    assert float((w - torch.linalg.eigvalsh(A)).abs().max()) <= 1e-13 * n * (1.0 + float(A.abs().max()))
    # a nearby matrix from these vectors
    E = torch.randn(n, n, generator=g, dtype=torch.float64).cuda()
    B = A + 1e-4 * (E + E.T)
    w, V = _run(B, V)
    _check(B, w, V)


def test_size_limit_is_refused():
    import torch
    from aimd_b200 import _lib
    A = torch.eye(_lib.EIGH_MAX + 1, dtype=torch.float64, device="cuda")
    with pytest.raises(_lib.NativeError, match="aimd_eigh"):
        _run(A)
