"""The 64-wide Gauss-Jordan exchange inside the sweep: sizes around its 8-column panels and 64-row blocks, and
matrices whose diagonal is zero, so that every pivot has to come from another row of the block.

The matrices are orthogonal up to a factor (products of reflections of a symmetric exchange pattern), so the inverse is known
to be as large as the matrix and a backward-stable elimination errs by a modest multiple of n * 2^-53.
"""

from __future__ import annotations

import numpy as np
import pytest

from tests.test_gpu_parity import _sym_inverse

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [2, 7, 8, 9, 16, 31, 33, 57, 63, 64])
def test_zero_diagonal_needs_row_exchanges(n):
    """Pairs (i, n-1-i) coupled by 1, nothing on the diagonal (a middle channel by itself), small symmetric noise."""
    rng = np.random.default_rng(n)
    A = np.zeros((3, n, n))
    for i in range(n):
        A[:, i, n - 1 - i] = 1.0 + i % 3 if i <= n - 1 - i else 1.0 + (n - 1 - i) % 3
    noise = rng.normal(size=(3, n, n)) * 0.02 / np.sqrt(n)
    noise = noise + noise.transpose(0, 2, 1)
    noise[:, np.arange(n), np.arange(n)] = 0.0
    A = A + noise
    X = _sym_inverse(A, False)
    np.testing.assert_allclose(X, np.linalg.inv(A), rtol=0, atol=64 * n * 2.0**-53 * np.abs(X).max())
    np.testing.assert_array_equal(X, X.transpose(0, 2, 1))


@pytest.mark.parametrize("n", [5, 64])
def test_a_nan_is_reported(n):
    A = np.eye(n)[None].copy()
    A[0, n // 2, n // 2] = np.nan
    with pytest.raises(RuntimeError, match="singular or non-finite"):
        _sym_inverse(A, False)
