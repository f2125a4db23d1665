"""What the device status says about a singular pivot does not depend on the path that found it: the batch item among its
own kind (matrix of the call, or sector of a Q_mid) and the 128-wide block."""

from __future__ import annotations

import numpy as np
import pytest
import torch

from pyticc_b200 import _native as nat

pytestmark = pytest.mark.gpu


def _status(call) -> list[int]:
    dev = nat.require_cuda()
    status = nat.DeviceStatus(dev)
    call(nat.load_library(), dev, status)
    return status.tensor.cpu().tolist()


@pytest.mark.parametrize("channel", [5, 70, 130, 200, 299])
@pytest.mark.parametrize("noalloc", [False, True])  # the 64-tile sweep, and 128-wide steps
def test_singular_matrix_of_a_batch(channel, noalloc):
    A = np.repeat(np.eye(300)[None], 3, axis=0)
    A[1, channel, channel] = 0.0

    def call(lib, dev, status):
        t = torch.as_tensor(A, device=dev)
        if noalloc:
            nat.check(lib.ticc_sym_inverse_noalloc(nat.ptr(t), 300, 3, 0, status.pointer, nat.stream_handle(dev)), "noalloc")
        else:
            nbytes = nat.size_query(lib.ticc_sym_inverse_workspace_size, 300, 3, 0)
            work = torch.empty(nbytes, dtype=torch.uint8, device=dev)
            nat.check(lib.ticc_sym_inverse(nat.ptr(t), 300, 3, 0, nat.ptr(work), nbytes, status.pointer, nat.stream_handle(dev)), "inverse")
        torch.cuda.synchronize(dev)

    assert _status(call)[:3] == [1, 1, channel // 128]


@pytest.mark.parametrize("n,channel", [(20, 12), (141, 130), (141, 60)])
def test_singular_correction_of_a_sector(n, channel):
    """I - h^2 (W_mid - diag)/6 with two channels coupled by 6/h^2 is exactly singular in that sector."""
    n_sector, n_energy = 4, 3
    W = np.repeat(np.diag(np.linspace(60.0, 10.0, n))[None], 2 * n_sector + 1, axis=0)
    W[5, channel, channel + 1] = W[5, channel + 1, channel] = 6.0  # the midpoint of sector 2

    def call(lib, dev, status):
        Wd = torch.as_tensor(W, device=dev)
        E = torch.linspace(0.2, 1.0, n_energy, dtype=torch.float64, device=dev)
        h = torch.ones(n_sector, dtype=torch.float64, device=dev)
        Y = torch.eye(n, dtype=torch.float64, device=dev).repeat(n_energy, 1, 1).contiguous()
        nbytes = nat.size_query(lib.ticc_ldmd_workspace_size, n, n_energy, n_sector, 0, nat.PRECISION_FP64)
        work = torch.empty(nbytes, dtype=torch.uint8, device=dev)
        at, one, stride = Wd.data_ptr(), 8 * n * n, 2 * n * n
        nat.check(
            lib.ticc_ldmd_propagate(nat.ptr(Y), 0, nat.ptr(E), n_energy, 1.0, nat.ptr(h), at, stride, at + one, stride, at + 2 * one, stride, n_sector, n,
                                    nat.PRECISION_FP64, nat.ptr(work), nbytes, status.pointer, nat.stream_handle(dev)),
            "propagate",
        )
        torch.cuda.synchronize(dev)

    assert _status(call)[:3] == [1, 2, channel // 128]
