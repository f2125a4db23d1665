"""What makes the transform multiply all chunks of B: a non-finite value in the plane in hand (real and imaginary planes apart),
or one that the first product brought about."""

from __future__ import annotations

import numpy as np
import pytest
import torch

from pyticc_b200.match.asymptotic import transform_device

pytestmark = pytest.mark.gpu


def _run(Y, B):
    return transform_device(torch.as_tensor(Y, device="cuda"), torch.as_tensor(B, device="cuda")).cpu().numpy()


def _pairs(n):
    """Block diagonal, 2 x 2 blocks of ones (a last channel by itself)."""
    return np.kron(np.eye((n + 1) // 2), np.ones((2, 2)))[:n, :n]


@pytest.mark.parametrize("n", [100, 261, 400])
@pytest.mark.parametrize("imaginary", [False, True])
def test_planes_are_independent(n, imaginary):
    rng = np.random.default_rng(n)
    planes = rng.normal(size=(2, 2, n, n))  # real, imaginary; two matrices
    planes[int(imaginary), 1, n // 3, n - 2] = np.nan
    got = _run(np.ascontiguousarray(np.moveaxis(planes, 0, -1)).view(np.complex128)[..., 0], _pairs(n))
    B = _pairs(n)
    for plane, part in zip(planes, (got.real, got.imag), strict=True):
        want = B.T @ plane @ B
        np.testing.assert_array_equal(np.isnan(part), np.isnan(want))
        # sums of four normal numbers
        np.testing.assert_allclose(part[~np.isnan(want)], want[~np.isnan(want)], rtol=0, atol=8 * 2.0**-53 * np.abs(plane[np.isfinite(plane)]).max() * 4)


@pytest.mark.parametrize("n", [100, 400])
def test_an_overflow_between_the_products(n):
    Y = np.random.default_rng(n).normal(size=(1, n, n))
    Y[0, 6:8, n - 1] = 1.0e308  # summed by the first product
    B = _pairs(n)
    with np.errstate(over="ignore", invalid="ignore"):
        want = (B.T @ Y[0]) @ B
    got = _run(Y, B)[0]
    assert not np.isfinite(want).all()
    np.testing.assert_array_equal(np.isnan(got), np.isnan(want))
    np.testing.assert_array_equal(np.isposinf(got), np.isposinf(want))
