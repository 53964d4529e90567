"""
s shells of 40 to 45 primitives (up to 2025 primitive pairs a block pair):
Schwarz bounds, one-electron integrals and J/K against the oracle. Tolerance:
1e-10 per unit of the result's largest element, as for the other shapes: sums of
up to 4e6 terms whose own rounding is 1e-16.
"""

from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _basis(n):
    """Oxygen with an s shell of n primitives and a p shell of three, hydrogen with an s shell of five."""
    from aimd_b200.basis import BasisSet
    ls, num = [0, 1, 0], [n, 3, 5]
    exps = [np.geomspace(0.2, 4000.0, n), np.geomspace(0.3, 8.0, 3), np.geomspace(0.15, 20.0, 5)]
    coefs = [0.7 * e ** 0.6 / k for e, k in zip(exps, num)]
    return BasisSet("long", ["O", "H"], np.array([[0.0, 0.0, 0.0], [0.3, 1.1, -1.4]]), [0, 0, 1], ls,
                    np.concatenate([[0], np.cumsum(num)]), np.concatenate(exps), np.concatenate(coefs))


def _close(got, ref):
    assert np.abs(np.asarray(got) - ref).max() <= 1e-10 * max(1.0, float(np.abs(ref).max()))


@pytest.mark.parametrize("n", [40, 41, 43, 45])
def test_long_s_contraction(n):
    from aimd_b200 import integrals as I
    from oracle import hf_oracle as O
    b = _basis(n)
    Q = O.schwarz_bounds(b)
    _close(I.schwarz_bounds(b) ** 2, Q ** 2)
    for got, ref in zip(I.one_electron_matrices(b), O.one_electron_matrices(b)):
        _close(got, ref)
    rng = np.random.default_rng(n)
    D = rng.normal(size=(b.nao, b.nao))
    for got, ref in zip(I.jk(b, D + D.T), O.jk_direct(b, D + D.T)):
        _close(got, ref)
