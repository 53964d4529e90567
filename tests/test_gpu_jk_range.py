"""
The fixed-point range of the J/K accumulators (sums up to 2^17 max|D|): the
largest sums for a given max|D| are those of a density whose elements are all
alike, against the oracle, at several magnitudes of it.
"""

from __future__ import annotations

import numpy as np
import pytest

from test_gpu_shapes import _cluster

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 8])
def test_equal_density_elements(n):
    from aimd_b200 import integrals as I
    from oracle import hf_oracle as O
    b, _ = _cluster(n)
    one = np.ones((b.nao, b.nao))
    ref = O.jk_direct(b, one)
    assert max(np.abs(r).max() for r in ref) < 2.0 ** 17 / 100     # far from the end at 200 AOs
    for m in (1.0, -0.9999, 3e-7, 2.0 ** 25):
        # 1e-10 per unit of the largest element, as for the other shapes: sums of 4e4 terms rounded to 2^-45 of max|D|
        for got, r in zip(I.jk(b, m * one), ref):
            assert np.abs(np.asarray(got) / m - r).max() <= 1e-10 * np.abs(r).max()
