"""The 64-tile sweep (few or small matrices): every count of block rows from 2 on, ragged last blocks, odd and even
tile counts (the transpose it writes for the upper half of a diagonal 128-tile), batches below and above one wave of
CTAs, and several sweeps in one call (the flags run on from sweep to sweep).  The inverse of a diagonally dominant
symmetric matrix errs by a modest multiple of n * 2^-53 of its largest element."""

from __future__ import annotations

import numpy as np
import pytest

from oracle import ldmd as o_ldmd
from pyticc_b200.propagation.logd import propagate_logD
from tests.test_gpu_parity import _sym_inverse

pytestmark = pytest.mark.gpu


def _matrices(seed, n, batch):
    rng = np.random.default_rng(seed)
    A = rng.normal(size=(batch, n, n))
    return A + A.transpose(0, 2, 1) + np.diag(rng.uniform(3.0, 6.0, n) * np.sqrt(n) * np.sign(rng.normal(size=n)))


@pytest.mark.parametrize("n,batch", [(129, 1), (192, 70), (193, 3), (256, 40), (257, 2), (320, 9), (385, 5), (449, 30), (641, 6), (1025, 2)])
def test_inverse_and_exact_symmetry(n, batch):
    A = _matrices(n, n, batch)
    X = _sym_inverse(A, False)
    inv = np.linalg.inv(A)
    np.testing.assert_allclose(X, inv, rtol=0, atol=4 * n * 2.0**-53 * np.abs(inv).max())
    np.testing.assert_array_equal(X, X.transpose(0, 2, 1))


@pytest.mark.parametrize("n,is_complex", [(141, False), (300, False), (97, True), (160, True)])
def test_many_sectors_in_one_call(n, is_complex):
    """24 sweeps of the work matrices and two batches of Q_mid sweeps share the flags of one call."""
    rng = np.random.default_rng(n)
    n_sector, n_energy, mu = 12, 3, 3.0
    base = rng.normal(size=(n, n)) * 0.1
    base = base + base.T + np.diag(np.linspace(60.0, 10.0, n))
    W = np.asarray([base + 0.01 * k * np.eye(n) for k in range(2 * n_sector + 1)])
    hs = np.full(n_sector, 0.04)
    E = np.linspace(0.2, 1.1, n_energy)
    Y0 = o_ldmd.initialize_inelastic(W[0][None] - 2 * mu * E[:, None, None] * np.eye(n))
    if is_complex:
        Y0 = Y0 * (1.0 + 0.1j)
    got = propagate_logD(Y0, E, mu, hs, W[0:-1:2], W[1::2], W[2::2]).cpu().numpy()
    want = o_ldmd.propagate_logD(Y0, E, mu, hs, W[0:-1:2], W[1::2], W[2::2])
    np.testing.assert_allclose(got, want, rtol=0, atol=1e-12 * np.abs(want).max())


def test_reciprocal_of_one_channel():
    """1 x 1 matrices: the pivot's reciprocal against IEEE division, within one unit in the last place."""
    rng = np.random.default_rng(1)
    a = rng.uniform(1.0, 2.0, 4096) * 2.0 ** rng.integers(-300, 300, 4096) * np.sign(rng.normal(size=4096))
    X = _sym_inverse(a.reshape(-1, 1, 1), False).reshape(-1)
    assert np.abs((X - 1.0 / a) * a).max() <= 2.0**-52
