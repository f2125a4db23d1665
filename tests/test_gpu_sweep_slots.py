"""The 64-tile sweep writes its panel slots again every second step and its pivot slots every third: with more steps than
slots, and few or many CTAs in flight, the same matrices give the same bits on every run, and their inverse."""

from __future__ import annotations

import numpy as np
import pytest

from tests.test_gpu_parity import _sym_inverse

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,batch", [(300, 24), (577, 1), (577, 9), (641, 30), (1100, 3)])
def test_slots_are_free_before_they_are_written_again(n, batch):
    rng = np.random.default_rng(n + batch)
    A = rng.normal(size=(batch, n, n))
    A = A + A.transpose(0, 2, 1) + np.diag(rng.uniform(3.0, 6.0, n) * np.sqrt(n) * np.sign(rng.normal(size=n)))
    inv = np.linalg.inv(A)
    first = _sym_inverse(A, False)
    # a backward-stable elimination of a diagonally dominant matrix errs by a modest multiple of n * 2^-53
    np.testing.assert_allclose(first, inv, rtol=0, atol=4 * n * 2.0**-53 * np.abs(inv).max())
    for _ in range(6):
        np.testing.assert_array_equal(_sym_inverse(A, False), first)
