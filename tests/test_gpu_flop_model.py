"""
The benchmark's flop models against plain loops over the kept block quartets of
water: J/K also against the oracle's model, the gradient as its kernels
evaluate it (whole numbers below 2^53, so equal).
"""

from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _nh(L):
    return (L + 1) * (L + 2) * (L + 3) // 6


def _nc(l):
    return (l + 1) * (l + 2) // 2


@pytest.mark.parametrize("basis_name", ["sto-3g", "6-31g*"])
def test_models(basis_name):
    import bench
    from aimd_b200 import geometry
    from aimd_b200.basis import build_basis
    from aimd_b200.engine import engine_for
    from oracle import hf_oracle as O
    sym, x = geometry.water()
    b = build_basis(sym, x, basis_name)
    eng = engine_for(b)
    Q, npp = eng.schwarz().cpu().numpy(), eng.pair_data()[0]
    l, n = eng.blocks["l"], eng.blocks["ncon"]
    pairs = [(int(l[i]), int(l[j]), int(n[i]) * int(n[j])) for i in range(eng.nblock) for j in range(i + 1)]
    jk = grad = 0
    for p1, (a, b1, _) in enumerate(pairs):
        for p2 in range(p1 + 1):
            if Q[p1] * Q[p2] < 1e-12:
                continue
            c, d, k = pairs[p2]
            La, Lc, nab, cols = a + b1, c + d, _nc(a) * _nc(b1), _nc(c) * _nc(d) * k
            quartets = int(npp[p1]) * int(npp[p2])
            jk += quartets * (2 * sum(_nh(La + Lc - m) for m in range(La + Lc + 1))
                              + cols * (2 * _nh(La) * _nh(Lc) + 2 * _nh(La) * nab))
            grad += quartets * (2 * sum(_nh(La + Lc + 1 - m) for m in range(La + Lc + 2))
                                + cols * (2 * (_nh(La + 1) + _nh(La)) * _nh(Lc) + 6 * _nh(La)))
            grad += int(npp[p1]) * cols * 8 * _nh(La) * nab
    assert bench.flop_model_device(eng, b)[0] == jk
    assert np.isclose(jk, O.flop_model(b)["flop"], rtol=1e-12)
    assert bench.flop_model_device(eng, b, grad=True)[0] == grad
