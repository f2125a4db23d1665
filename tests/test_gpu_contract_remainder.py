"""Four radial points a CTA with a remainder of two (9 tiles x 514 points), the one that the other sizes leave out."""

from __future__ import annotations

import numpy as np
import pytest

from pyticc_b200.matrix.interaction import VBasisBF, contract_device

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("is_complex", [False, True])
def test_two_points_left_over(is_complex):
    n_R, n_grid, n = 514, 37, 103
    rng = np.random.default_rng(n_R)
    groups = {0: tuple(range(33)), 1: tuple(range(33, n))}
    parts = [{K: rng.normal(size=(len(m), n_grid)) for K, m in groups.items()} for _ in range(2 if is_complex else 1)]
    w = rng.normal(size=(n_R, n_grid))
    V = contract_device(VBasisBF(n, (n_grid,), groups, parts[0], parts[1] if is_complex else None, 0.7), None, w).cpu().numpy()
    want = np.zeros((n_R, n, n))
    for K, m in groups.items():
        for part in parts:
            want[np.ix_(range(n_R), m, m)] += 0.7 * np.matmul(part[K][None] * w[:, None, :], part[K].T)
    # sums of at most 2 n_grid products of three standard normal numbers (each below 60), one rounding a step
    np.testing.assert_allclose(V, want, rtol=0, atol=4 * n_grid * 2.0**-53 * 60.0)
    np.testing.assert_array_equal(V, V.transpose(0, 2, 1))
