"""Sums weighted by a negative power of k^2: the weight of one mode is the
nearest double to 1 / k^(2 e), as one division gives it (not a power of a
rounded 1 / k^2, which is off by up to e units and, over the few low modes that
carry such a sum, leaves its mark).

Tolerance: exact powers of two around the weight, k^(2 e) below 2^53 and so
exact, and one reciprocal of at most 0.5 + 2^-13 units.
"""
from fractions import Fraction

import numpy as np
import pytest

from tests._helpers import params

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("e", [1, 2, 3, 4])
def test_weight_of_one_mode(gpu, e):
    n = 64
    c = gpu.Context(params(n, iflow=0)[1], 0)
    for kx, ky in ((1, 1), (1, 2), (2, 3), (3, 7), (7, 11), (9, 17), (21, 1), (13, 15), (1, 20)):
        a = np.zeros((n // 2 + 1, n), np.complex128)
        a[kx, ky] = 1.0
        got = Fraction(c.energy(a, -e)) * Fraction(n) ** 4 / 2
        exact = Fraction(1, (kx * kx + ky * ky) ** e)
        unit = Fraction(float(np.spacing(float(exact))))
        assert abs(got - exact) <= unit * (Fraction(1, 2) + Fraction(1, 2 ** 13)), (kx, ky, e)
