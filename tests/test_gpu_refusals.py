"""
Basis sets whose primitive pairs do not fit a CTA's shared memory are refused
before any launch, with the entry point and the pair class named.
"""

from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _contracted(shells):
    """One oxygen with the given (l, number of primitives) shells."""
    from aimd_b200.basis import BasisSet
    exps, coefs, start, ls = [], [], [0], []
    for l, n in shells:
        exps += list(np.geomspace(0.15, 40.0, n))
        coefs += list(0.3 / n + 0.1 * np.cos(np.arange(n)) / n)
        start.append(start[-1] + n)
        ls.append(l)
    return BasisSet("contracted", ["O"], np.zeros((1, 3)), [0] * len(ls), ls, start, exps, coefs)


@pytest.mark.parametrize("shells,cls", [([(0, 50)], 0), ([(1, 40)], 2), ([(0, 3), (2, 20)], 5)])
def test_refusal_names_the_pair_class(shells, cls):
    from aimd_b200._lib import NativeError
    from aimd_b200.engine import Engine
    b = _contracted(shells)
    with pytest.raises(NativeError, match=rf"schwarz \(pair class {cls}\).*shared memory"):
        Engine(b).set_geometry(b.positions)
