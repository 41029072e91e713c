"""The fit's reciprocal, quotient and root (trax_fit_math.cuh) against CUDA's correctly rounded division and root.

The scale of an operand only moves exponents, so every mantissa of one binade (a reciprocal) or of two (a root: even
and odd exponents) covers all operands; other binades guard the range.  With a correctly rounded reciprocal the
quotient is correctly rounded by Markstein's theorem, of which random operands are a check.  Equality, no tolerance."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _mantissas(exponent, binades):
    bits = np.arange(binades << 23, dtype=np.uint32) + np.uint32((127 + exponent) << 23)
    return bits.view(np.float32)


@pytest.mark.parametrize("exponent", [0, 1, -100, 99])
def test_reciprocal_of_every_mantissa(trax_lib, exponent):
    b = _mantissas(exponent, 1)
    want = trax_lib.math_eval("div", np.ones_like(b), b)
    for s in (1, -1):
        assert np.array_equal(trax_lib.math_eval("fit_reciprocal", s * b), s * want)


@pytest.mark.parametrize("exponent", [0, -100, 98])
def test_root_of_every_mantissa(trax_lib, exponent):
    x = _mantissas(exponent, 2)
    assert np.array_equal(trax_lib.math_eval("fit_root", x), trax_lib.math_eval("sqrt", x))
    assert np.array_equal(trax_lib.math_eval("fit_root", np.float32([0.0, 1.0, 4.0])), np.float32([0, 1, 2]))


@pytest.mark.parametrize("spread", [0, 50])
def test_quotients(trax_lib, spread):
    rng = np.random.default_rng(spread)
    n = 1 << 23
    a, b = ((1 + rng.random(n, dtype=np.float32)) * np.float32(2.0) ** rng.integers(-spread, spread + 1, n)
            * rng.choice(np.float32([-1, 1]), n) for _ in range(2))
    a, b = a.astype(np.float32), b.astype(np.float32)
    a[: n // 4] = b[: n // 4] * (1 + rng.random(n // 4, dtype=np.float32)).astype(np.float32)  # close to a tie more often
    a[:8], b[8:16] = 0.0, 1.0
    want = trax_lib.math_eval("div", a, b)
    assert np.array_equal(trax_lib.math_eval("fit_quotient", a, b), want)


def test_divisors_that_make_a_row_unusable(trax_lib):
    """Where a division gives an infinity or NaN, or its divisor is not finite, the quotient is NaN."""
    b = np.float32([0.0, -0.0, np.inf, -np.inf, np.nan, 0.0])
    a = np.float32([1.0, 1.0, 1.0, 0.0, 1.0, 0.0])
    assert np.isnan(trax_lib.math_eval("fit_quotient", a, b)).all()
