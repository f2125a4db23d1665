"""A caller of the C entry may hand over Y at any multiple of 8 bytes: same bits as at an aligned address."""

from __future__ import annotations

import numpy as np
import pytest
import torch

from pyticc_b200 import _native as nat

pytestmark = pytest.mark.gpu


def _propagate(n: int, is_complex: bool, shift: int) -> np.ndarray:
    lib, dev = nat.load_library(), nat.require_cuda()
    rng = np.random.default_rng(n)
    n_sector, n_energy, mu, parts = 2, 3, 3.0, 2 if is_complex else 1
    base = rng.normal(size=(n, n)) * 0.1
    base = base + base.T + np.diag(np.linspace(60.0, 10.0, n))
    W = torch.as_tensor(np.asarray([base + 0.01 * k * np.eye(n) for k in range(2 * n_sector + 1)]), device=dev)
    E = torch.as_tensor(np.linspace(0.2, 1.1, n_energy), device=dev)
    h = torch.full((n_sector,), 0.04, dtype=torch.float64, device=dev)
    count = n_energy * n * n * parts
    buffer = torch.zeros(count + 2, dtype=torch.float64, device=dev)
    Y = np.asarray([np.diag(np.linspace(3.0, 7.0, n)) + 0.01 * e * (base + base.T) for e in range(n_energy)])
    Y = np.stack([Y, 0.1 * Y], axis=-1) if is_complex else Y
    buffer[shift : shift + count] = torch.as_tensor(Y.reshape(-1), device=dev)
    nbytes = nat.size_query(lib.ticc_ldmd_workspace_size, n, n_energy, n_sector, int(is_complex), nat.PRECISION_FP64)
    work = torch.empty(nbytes, dtype=torch.uint8, device=dev)
    status = nat.DeviceStatus(dev)
    stride, one = 2 * n * n, n * n * 8
    at = W.data_ptr()
    nat.check(
        lib.ticc_ldmd_propagate(buffer.data_ptr() + 8 * shift, int(is_complex), nat.ptr(E), n_energy, mu, nat.ptr(h), at, stride, at + one, stride, at + 2 * one, stride,
                                n_sector, n, nat.PRECISION_FP64, nat.ptr(work), nbytes, status.pointer, nat.stream_handle(dev)),
        "ticc_ldmd_propagate",
    )
    status.raise_if_failed("ticc_ldmd_propagate")
    assert buffer[:shift].abs().sum() == 0 and buffer[shift + count :].abs().sum() == 0
    return buffer[shift : shift + count].cpu().numpy()


# n: the whole-call kernel, and the passes over one and over several 128-tiles (odd sizes)
@pytest.mark.parametrize("n", [21, 141, 201])
@pytest.mark.parametrize("is_complex", [False, True])
def test_log_derivative_at_eight_byte_addresses(n, is_complex):
    np.testing.assert_array_equal(_propagate(n, is_complex, 1), _propagate(n, is_complex, 0))
