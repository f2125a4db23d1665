"""Pivots over the whole range that FP64 division covers: near the ends of the normal numbers, where the fast reciprocal's
approximation would flush to zero, and below them."""

from __future__ import annotations

import numpy as np
import pytest

from tests.test_gpu_parity import _sym_inverse

pytestmark = pytest.mark.gpu


def test_one_channel_from_the_subnormals_to_the_top():
    """1 x 1 matrices against IEEE division.  The call averages A with its transpose and the result with its own, so a and
    1/a stay below half of the largest number: 2^-1023 < |a| < 2^1023."""
    rng = np.random.default_rng(2)
    exponents = np.concatenate([np.repeat([-1023, -1022, -1021, -1020, 1018, 1019, 1020, 1021, 1022], 256), rng.integers(-1023, 1023, 2048)])
    a = np.ldexp(rng.uniform(1.0, 2.0, exponents.size), exponents) * np.sign(rng.normal(size=exponents.size))
    assert np.abs(a).min() > 2.0**-1023 and np.abs(a).max() < 2.0**1023 and (np.abs(a) < 2.0**-1022).any()
    X = _sym_inverse(a.reshape(-1, 1, 1), False).reshape(-1)
    want = 1.0 / a
    # one unit in the last place, which is 2^-1074 where 1/a is subnormal
    assert (np.abs(X - want) <= np.maximum(2.0**-52 * np.abs(want), 2.0**-1074)).all()


# 150 x 128 and 330: the 64-tile sweep with two CTAs an SM, and with more steps than slots
@pytest.mark.parametrize("exponent", [-1023, -1021, 1019, 1020, 1021])
@pytest.mark.parametrize("n,batch", [(9, 1), (40, 1), (100, 1), (150, 1), (150, 128), (330, 2)])
def test_scaled_matrices(n, batch, exponent):
    """A = 2^exponent (D + small): diagonal 1.5 to 1.9 and weak couplings, both exact at every scale.  The inverse is that of
    the unscaled matrix times 2^-exponent; its elements carry at most the rounding of 51-bit (subnormal) numbers per
    elimination step, and an absolute unit 2^-1074 where the inverse itself is subnormal."""
    rng = np.random.default_rng(n)
    noise = np.round(rng.uniform(-1.0, 1.0, (n, n)) * 0.02 / np.sqrt(n) * 2.0**20) * 2.0**-20
    A = np.tril(noise, -1)
    A = A + A.T + np.diag(np.round(rng.uniform(1.5, 1.9, n) * 2.0**20) * 2.0**-20)
    X = _sym_inverse(np.repeat(np.ldexp(A, exponent)[None], batch, axis=0), False)
    np.testing.assert_array_equal(X, np.repeat(X[:1], batch, axis=0))
    X = X[0]
    # compared at the scale of the unscaled inverse, in two exact steps
    X = np.ldexp(np.ldexp(X, exponent // 2), exponent - exponent // 2)
    np.testing.assert_allclose(X, np.linalg.inv(A), rtol=0, atol=4 * n * (2.0**-51 + 2.0 ** (exponent - 1074)))
    np.testing.assert_array_equal(X, X.T)


def test_a_zero_pivot_is_still_reported():
    A = np.diag([1.0, 2.0, 0.0, 3.0])[None]
    with pytest.raises(RuntimeError, match="singular or non-finite"):
        _sym_inverse(A, False)
