"""The BF -> SF transform skips the 32-row chunks of B that hold only zeros: block-diagonal B with blocks across chunk and tile edges,
empty columns, dense B, real and complex Y, against the plain product in 64 bits; an infinity or NaN in Y spreads
exactly as the full product spreads it."""

from __future__ import annotations

import numpy as np
import pytest
import torch

from pyticc_b200.match.asymptotic import transform_device

pytestmark = pytest.mark.gpu


def _block_diagonal(n, size, seed):
    rng = np.random.default_rng(seed)
    B = np.zeros((n, n))
    for a in range(0, n, size):
        b = min(n, a + size)
        B[a:b, a:b] = np.linalg.qr(rng.normal(size=(b - a, b - a)))[0]
    return B


def _run(Y, B):
    return transform_device(torch.as_tensor(Y, device="cuda"), torch.as_tensor(B, device="cuda")).cpu().numpy()


@pytest.mark.parametrize("n,size", [(5, 2), (130, 31), (257, 33), (400, 1), (400, 400), (520, 130)])
@pytest.mark.parametrize("is_complex", [False, True])
def test_matches_the_full_product(n, size, is_complex):
    rng = np.random.default_rng(n + size)
    Y = rng.normal(size=(2, n, n))
    if is_complex:
        Y = Y + 1j * rng.normal(size=Y.shape)
    B = _block_diagonal(n, size, n)
    if size == 31:
        B[:, 40:90] = 0.0  # columns without an entry
    np.testing.assert_allclose(_run(Y, B), B.T @ Y @ B, rtol=0, atol=8 * n * 2.0**-53 * np.abs(Y).max())


@pytest.mark.parametrize("value", [np.inf, np.nan])
def test_a_non_finite_value_spreads_as_in_the_full_product(value):
    n = 300
    rng = np.random.default_rng(7)
    Y = rng.normal(size=(2, n, n))
    Y[1, 17, 250] = value
    got = _run(Y, _block_diagonal(n, 20, 3))
    with np.errstate(invalid="ignore"):
        want = _block_diagonal(n, 20, 3).T @ Y @ _block_diagonal(n, 20, 3)
    assert np.array_equal(np.isnan(got[1]), np.isnan(want[1]))
    assert np.isfinite(got[0]).all()
