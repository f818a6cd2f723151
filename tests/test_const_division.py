"""The corrected product that replaces a division by 3 or 6 in the weights epilogue: exact rational
arithmetic with each fused operation rounded once, against the correctly rounded quotient."""
from fractions import Fraction

import numpy as np
import pytest


@pytest.mark.parametrize("D", [3, 6])
def test_corrected_product_is_the_rounded_quotient(D):
    rng = np.random.default_rng(D)
    R = 1.0 / D
    xs = np.concatenate([rng.standard_normal(4000) * 10.0 ** rng.integers(-40, 40, 4000),          # products of doubles
                         rng.standard_normal(2000).astype(np.float32).astype(np.float64),            # fp32 sums
                         np.nextafter(np.arange(1.0, 500.0), 0), np.nextafter(np.arange(1.0, 500.0), 1e9), [0.0, -0.0]])
    for x in xs:
        q = x * R
        e = float(Fraction(x) - D * Fraction(q))        # fma(-D, q, x)
        got = float(Fraction(e) * Fraction(R) + Fraction(q))   # fma(e, R, q)
        assert got == x / D
