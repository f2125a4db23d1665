"""Propagation of matrices of at most 128 rows in one launch: the edges of its three tile sizes (32, 64, 128 rows; a
complex matrix has two rows a channel), ragged 8-column panels, several blocks and energies, one and many sectors,
against the oracle on the same inputs.  The channels are closed or weakly open over a short range, where the
recurrence does not amplify rounding: 1e-12 of the largest element."""

from __future__ import annotations

import numpy as np
import pytest
import torch

from oracle import ldmd as o_ldmd
from pyticc_b200 import _native as nat
from pyticc_b200.propagation.logd import propagate_blocks_device, propagate_logD

pytestmark = pytest.mark.gpu


def _inputs(seed, n, n_sector, n_energy, is_complex, n_block=1):
    rng = np.random.default_rng(seed)
    base = rng.normal(size=(n_block, n, n)) * 0.15
    base = base + base.transpose(0, 2, 1)
    base[:, np.arange(n), np.arange(n)] += np.linspace(50.0, 4.0, n)
    W = np.stack([base * (1.0 - 0.01 * k) for k in range(2 * n_sector + 1)], axis=1)  # (block, point, n, n)
    hs = rng.uniform(0.02, 0.05, n_sector)
    E = np.linspace(0.2, 1.1, n_energy)
    mu = 3.0
    Y0 = np.stack([o_ldmd.initialize_inelastic(W[g, 0][None] - 2 * mu * E[:, None, None] * np.eye(n)) for g in range(n_block)])
    if is_complex:
        Z = rng.normal(size=Y0.shape) * 0.05
        Y0 = Y0 + 1j * (Z + Z.transpose(0, 1, 3, 2))
    return W, hs, E, mu, Y0


@pytest.mark.parametrize("n", [1, 8, 21, 31, 32, 33, 57, 64, 65, 72, 100, 127, 128])
@pytest.mark.parametrize("n_sector", [1, 5])
def test_real(n, n_sector):
    W, hs, E, mu, Y0 = _inputs(n, n, n_sector, 3, False)
    W, Y0 = W[0], Y0[0]
    got = propagate_logD(Y0, E, mu, hs, W[0:-1:2], W[1::2], W[2::2]).cpu().numpy()
    want = o_ldmd.propagate_logD(Y0, E, mu, hs, W[0:-1:2], W[1::2], W[2::2])
    np.testing.assert_allclose(got, want, rtol=0, atol=1e-12 * np.abs(want).max())


@pytest.mark.parametrize("n", [1, 5, 16, 17, 32, 33, 50, 64])
def test_complex(n):
    W, hs, E, mu, Y0 = _inputs(100 + n, n, 4, 2, True)
    W, Y0 = W[0], Y0[0]
    got = propagate_logD(Y0, E, mu, hs, W[0:-1:2], W[1::2], W[2::2]).cpu().numpy()
    want = o_ldmd.propagate_logD(Y0, E, mu, hs, W[0:-1:2], W[1::2], W[2::2])
    np.testing.assert_allclose(got, want, rtol=0, atol=1e-12 * np.abs(want).max())


@pytest.mark.parametrize("n,n_block,n_energy", [(20, 7, 90), (40, 5, 3), (90, 2, 80)])
def test_blocks(n, n_block, n_energy):
    """More matrices than the chip holds at once, and W of each block at its own stride."""
    n_sector = 3
    W, hs, E, mu, Y0 = _inputs(n, n, n_sector, n_energy, False, n_block)
    dev = nat.require_cuda()
    Wd, Yd = torch.as_tensor(W, device=dev).contiguous(), torch.as_tensor(Y0, device=dev).contiguous()
    stride = 2 * n * n
    got = propagate_blocks_device(Yd, torch.as_tensor(E, device=dev), mu, torch.as_tensor(hs, device=dev), Wd[0, 0], Wd[0, 1], Wd[0, 2], stride=(stride,) * 3, block_stride=(2 * n_sector + 1) * n * n)
    got = got.cpu().numpy()
    for g in range(n_block):
        want = o_ldmd.propagate_logD(Y0[g], E, mu, hs, W[g, 0:-1:2], W[g, 1::2], W[g, 2::2])
        np.testing.assert_allclose(got[g], want, rtol=0, atol=1e-12 * np.abs(want).max())


def test_a_singular_matrix_is_reported():
    n, dev = 10, nat.require_cuda()
    W = np.zeros((1, n, n))
    W[0, 2, 2] = np.nan
    with pytest.raises(RuntimeError, match="singular or non-finite"):
        propagate_logD(np.eye(n)[None], np.array([0.1]), 1.0, np.array([0.1]), W, W, W, device=dev)
