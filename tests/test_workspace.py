"""A workspace sized for the largest of several calls serves the smaller ones: what a call cannot do without grows with every
size (CPU: from the refusal of a null workspace), and a call given only that much stays inside it (GPU)."""

from __future__ import annotations

import ctypes
import re

import numpy as np
import pytest
import torch

from pyticc_b200 import _native as nat

FAKE = ctypes.c_void_p(256)  # never read: a call without workspace is refused on the host


def _needed(call, *args) -> int:
    assert call(*args) == nat.ERR_WORKSPACE
    return int(re.search(r"(\d+) needed", nat.last_error()).group(1))


def _inverse(n, batch, is_complex=0):
    lib = nat.load_library()
    return _needed(lib.ticc_sym_inverse, FAKE, n, batch, is_complex, None, 0, None, None), nat.size_query(lib.ticc_sym_inverse_workspace_size, n, batch, is_complex)


def _propagation(n, n_energy, n_block, n_sector, is_complex=0, precision=nat.PRECISION_FP64):
    lib = nat.load_library()
    need = _needed(lib.ticc_ldmd_propagate_blocks, FAKE, is_complex, FAKE, n_energy, 1.0, FAKE, FAKE, 0, FAKE, 0, FAKE, 0, 0, n_sector, n, n_block, precision, None, 0, None, None)
    return need, nat.size_query(lib.ticc_ldmd_blocks_workspace_size, n, n_energy, n_block, n_sector, is_complex, precision)


def _matching(n, n_energy, is_complex=0):
    lib = nat.load_library()
    need = _needed(lib.ticc_match_smatrix, FAKE, is_complex, 10.0, FAKE, n_energy, 1.0, FAKE, FAKE, n, n, FAKE, FAKE, None, 0, None, None)
    return need, nat.size_query(lib.ticc_match_workspace_size, n, n_energy, is_complex, n)


def _check(sizes):
    largest = 0
    for need, asked in sizes:
        assert need <= asked
        assert need >= largest  # so that the query for an earlier, smaller call never exceeds what a later one was sized for
        largest = need


@pytest.mark.parametrize("is_complex", [0, 1])
def test_needs_grow_with_every_size(is_complex):
    batches = [1, 2, 3, 4, 16, 24, 25, 64, 128, 167, 168, 169, 400, 1000]
    channels = [1, 64, 65, 128, 129, 192, 193, 231, 256, 257, 320, 577, 640, 641, 660, 1984, 4096, 4097]
    for n in channels:
        _check(_inverse(n, b, is_complex) for b in batches)
        _check(_matching(n, b, is_complex) for b in batches)
        _check(_propagation(n, b, 1, 8, is_complex) for b in batches)
        _check(_propagation(n, 4, b, 3, is_complex) for b in batches)
        _check(_propagation(n, 4, 1, s, is_complex) for s in (1, 2, 8, 63, 64, 65, 100))
    for b in batches:
        _check(_inverse(n, b, is_complex) for n in channels)
        _check(_propagation(n, b, 1, 8, is_complex) for n in channels)
        _check(_matching(n, b, is_complex) for n in channels)


# GPU: exactly the bytes that the refusal names, inside a larger buffer whose rest stays as it was
def _bounded(nbytes):
    buffer = torch.full((nbytes + 4096,), 77, dtype=torch.uint8, device=nat.require_cuda())
    return buffer, lambda: bool((buffer[nbytes:] == 77).all())


@pytest.mark.gpu
@pytest.mark.parametrize("n,batch", [(192, 5), (231, 9), (660, 2)])
def test_inverse_in_the_least_workspace(n, batch):
    lib, dev = nat.load_library(), nat.require_cuda()
    rng = np.random.default_rng(n)
    A = rng.normal(size=(batch, n, n))
    A = A + A.transpose(0, 2, 1) + np.diag(rng.uniform(3.0, 6.0, n) * np.sqrt(n))
    need, asked = _inverse(n, batch)
    assert need < asked
    work, untouched = _bounded(need)
    t, status = torch.as_tensor(A, device=dev), nat.DeviceStatus(dev)
    nat.check(lib.ticc_sym_inverse(nat.ptr(t), n, batch, 0, nat.ptr(work), need, status.pointer, nat.stream_handle(dev)), "inverse")
    status.raise_if_failed("inverse")
    assert untouched()
    inv = np.linalg.inv(A)
    np.testing.assert_allclose(t.cpu().numpy(), inv, rtol=0, atol=4 * n * 2.0**-53 * np.abs(inv).max())


@pytest.mark.gpu
@pytest.mark.parametrize("n,n_block,n_sector", [(141, 1, 4), (300, 2, 5)])
def test_propagation_in_the_least_workspace(n, n_block, n_sector):
    lib, dev = nat.load_library(), nat.require_cuda()
    rng = np.random.default_rng(n)
    n_energy = 3
    base = rng.normal(size=(n, n)) * 0.1
    base = base + base.T + np.diag(np.linspace(60.0, 10.0, n))
    W = torch.as_tensor(np.asarray([[base + (0.01 * k + g) * np.eye(n) for k in range(2 * n_sector + 1)] for g in range(n_block)]), device=dev)
    E = torch.linspace(0.2, 1.1, n_energy, dtype=torch.float64, device=dev)
    h = torch.full((n_sector,), 0.04, dtype=torch.float64, device=dev)
    start = torch.diag_embed(torch.sqrt(torch.diagonal(W[:, 0], dim1=-2, dim2=-1)))[:, None].repeat(1, n_energy, 1, 1).contiguous()
    need, asked = _propagation(n, n_energy, n_block, n_sector)
    assert need < asked
    got = []
    for nbytes in (need, asked):
        Y, status = start.clone(), nat.DeviceStatus(dev)
        work, untouched = _bounded(nbytes)
        at, one, stride = W.data_ptr(), 8 * n * n, 2 * n * n
        nat.check(
            lib.ticc_ldmd_propagate_blocks(nat.ptr(Y), 0, nat.ptr(E), n_energy, 3.0, nat.ptr(h), at, stride, at + one, stride, at + 2 * one, stride, (2 * n_sector + 1) * n * n,
                                           n_sector, n, n_block, nat.PRECISION_FP64, nat.ptr(work), nbytes, status.pointer, nat.stream_handle(dev)),
            "propagate",
        )
        status.raise_if_failed("propagate")
        assert untouched()
        got.append(Y.cpu().numpy())
    np.testing.assert_allclose(got[0], got[1], rtol=0, atol=1e-12 * np.abs(got[1]).max())
