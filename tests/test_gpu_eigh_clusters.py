"""
Spectra of aimd_eigh whose eigenvalues lie as close as the off-diagonal
elements that a sweep leaves: I + spread R, close pairs, and both from the
vectors of a nearby matrix.

Bounds: a sweep is n - 1 rounds of rotations, each of which rounds A and the
vectors by some 2.5 eps of the norm (Frobenius), independently; ten sweeps give
2.5 sqrt(10 n) eps = 8 sqrt(n) eps, taken as 12 sqrt(n) eps. A start from given vectors adds
the product V^T A V and their own departure from orthogonality: twice that.
"""

from __future__ import annotations

import pytest

pytestmark = pytest.mark.gpu
EPS = 2.3e-16


def _residuals(A, V=None):
    import torch
    from aimd_b200 import _lib
    n = A.shape[0]
    out = torch.full_like(A, float("nan")) if V is None else V.contiguous().clone()
    w = torch.empty(n, dtype=A.dtype, device=A.device)
    _lib.check(_lib.load().aimd_eigh(n, A.data_ptr(), out.data_ptr(), w.data_ptr(), int(V is not None),
                                     torch.cuda.current_stream().cuda_stream), "aimd_eigh")
    assert bool((w[1:] >= w[:-1]).all())
    eye = torch.eye(n, dtype=A.dtype, device=A.device)
    norm = float(torch.linalg.matrix_norm(A))
    return (float(torch.linalg.matrix_norm(A @ out - out * w)) / norm,
            float(torch.linalg.matrix_norm(out.T @ out - eye)) / n ** 0.5)


@pytest.mark.parametrize("spread", [0.0, 1e-15, 1e-14, 1e-13, 1e-12, 1e-10, 1e-6])
@pytest.mark.parametrize("kind", ["identity", "pairs"])
@pytest.mark.parametrize("n", [2, 3, 7, 32, 33, 50, 63, 64])
def test_close_eigenvalues(n, kind, spread):
    import torch
    g = torch.Generator().manual_seed(1000 + n)
    R = torch.randn(n, n, generator=g, dtype=torch.float64)
    R = R + R.T
    Q, _ = torch.linalg.qr(torch.randn(n, n, generator=g, dtype=torch.float64))
    if kind == "identity":
        A = torch.eye(n, dtype=torch.float64) + spread * n ** 0.5 * R / torch.linalg.matrix_norm(R)
    else:
        d = 1 + torch.arange(n // 2 + 1).repeat_interleave(2)[:n].double() + spread * torch.arange(n).double()
        A = Q @ torch.diag(d) @ Q.T
    A = (0.5 * (A + A.T)).cuda()
    bound = 12 * n ** 0.5 * EPS
    assert max(_residuals(A)) <= bound
    near = torch.linalg.eigh(A + 1e-4 * (R + R.T).cuda() / n)[1]
    assert max(_residuals(A, near)) <= 2 * bound
