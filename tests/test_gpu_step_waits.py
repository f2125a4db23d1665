"""Both sweeps' bounded waits, and the 128-wide steps on shapes that the 64-tile sweep leaves to them."""

from __future__ import annotations

import numpy as np
import pytest

from pyticc_b200 import _native as nat
from tests.test_gpu_parity import _sym_inverse
from tests.test_zz_no_alloc import _no_alloc

pytestmark = pytest.mark.gpu


def _matrices(n, batch):
    rng = np.random.default_rng(n + batch)
    A = rng.normal(size=(batch, n, n))
    return A + A.transpose(0, 2, 1) + np.diag(rng.uniform(3.0, 6.0, n) * np.sqrt(n) * np.sign(rng.normal(size=n)))


# the 64-tile sweep takes a 300 x 3 batch from a workspace; without one, and for 64 matrices of 512 rows, 128-wide steps run
PATHS = [(_no_alloc, 300, 3), (lambda A, c: _sym_inverse(A, c), 512, 64), (lambda A, c: _sym_inverse(A, c), 300, 3)]


@pytest.mark.parametrize("inverse,n,batch", PATHS, ids=["steps-noalloc", "steps-workspace", "64-tiles"])
def test_a_wait_that_runs_out_is_reported_and_the_next_call_is_right(inverse, n, batch):
    """With the poll limit at 0 every wait gives up at once: status 6, and the next call (default limit) is right."""
    lib = nat.load_library()
    A = _matrices(n, batch)
    nat.check(lib.ticc_debug_set_step_poll_limit(0), "ticc_debug_set_step_poll_limit")
    try:
        with pytest.raises(RuntimeError, match="gave up waiting"):
            inverse(A, False)
    finally:
        nat.check(lib.ticc_debug_set_step_poll_limit(1 << 22), "ticc_debug_set_step_poll_limit")
    inv = np.linalg.inv(A)
    np.testing.assert_allclose(inverse(A, False), inv, rtol=0, atol=4 * n * 2.0**-53 * np.abs(inv).max())


@pytest.mark.parametrize("n", [129, 300, 520])
def test_steps_on_small_batches(n):
    """The sizes of the small-batch inverse tests, through the 128-wide steps that those no longer reach."""
    A = _matrices(n, 3)
    X = _no_alloc(A, False)
    inv = np.linalg.inv(A)
    np.testing.assert_allclose(X, inv, rtol=0, atol=4 * n * 2.0**-53 * np.abs(inv).max())
    np.testing.assert_array_equal(X, X.transpose(0, 2, 1))


def test_the_shapes_take_the_paths_they_are_meant_for():
    lib = nat.load_library()
    for n, batch, steps in ((512, 64, True), (300, 3, False)):
        padded = -(-n // 128) * 128
        least = 8 * batch * (padded * padded + 128 * padded + 32784)  # matrices and 128-wide scratch alone
        assert (nat.size_query(lib.ticc_sym_inverse_workspace_size, n, batch, 0) < least + 4096) == steps
