"""The contraction's 32-row tiles: groups of every size around a tile and a warp's 16-row part, odd quadrature sizes and real and complex
rows, against the plain weighted product in 64 bits; cross-group elements stay zero and V is exactly symmetric."""

from __future__ import annotations

import numpy as np
import pytest

from pyticc_b200.matrix.interaction import VBasisBF, contract_device

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("sizes", [(1,), (15, 16, 17), (31, 32, 33), (48, 1, 65), (130,)])
@pytest.mark.parametrize("n_grid,is_complex", [(5, False), (33, True), (96, False)])
def test_groups_around_the_tile(sizes, n_grid, is_complex):
    rng = np.random.default_rng(sum(sizes) + n_grid)
    n = sum(sizes)
    order = rng.permutation(n)
    groups, at = {}, 0
    for K, size in enumerate(sizes):
        groups[K] = tuple(int(c) for c in order[at : at + size])
        at += size
    real = {K: rng.normal(size=(len(m), n_grid)) for K, m in groups.items()}
    imag = {K: rng.normal(size=(len(m), n_grid)) for K, m in groups.items()} if is_complex else None
    w = rng.normal(size=(3, n_grid))
    V = contract_device(VBasisBF(n, (n_grid,), groups, real, imag, 0.7), None, w).cpu().numpy()
    want = np.zeros((3, n, n))
    for K, m in groups.items():
        for part in (real,) if imag is None else (real, imag):
            want[np.ix_(range(3), m, m)] += 0.7 * np.einsum("ag,rg,bg->rab", part[K], w, part[K])
    np.testing.assert_allclose(V, want, rtol=0, atol=4 * n_grid * 2.0**-53 * 60.0)
    np.testing.assert_array_equal(V, V.transpose(0, 2, 1))
    np.testing.assert_array_equal(V[want == 0.0], 0.0)


@pytest.mark.parametrize("n_R", [245, 246, 511, 512, 513, 515])
@pytest.mark.parametrize("is_complex", [False, True])
def test_radial_points_sharing_a_tile(n_R, is_complex):
    """9 tiles: 2205 to 4635 (tile, radial point) units take two and four radial points a CTA, with remainders of one to three."""
    rng = np.random.default_rng(n_R)
    sizes, n_grid = (33, 70), 37
    n = sum(sizes)
    groups = {0: tuple(range(0, 33)), 1: tuple(range(33, n))}
    real = {K: rng.normal(size=(len(m), n_grid)) for K, m in groups.items()}
    imag = {K: rng.normal(size=(len(m), n_grid)) for K, m in groups.items()} if is_complex else None
    w = rng.normal(size=(n_R, n_grid))
    V = contract_device(VBasisBF(n, (n_grid,), groups, real, imag, 0.7), None, w).cpu().numpy()
    want = np.zeros((n_R, n, n))
    for m in groups.values():
        for part in (real,) if imag is None else (real, imag):
            rows = part[0] if m[0] == 0 else part[1]
            want[np.ix_(range(n_R), m, m)] += 0.7 * np.matmul(rows[None] * w[:, None, :], rows.T)
    np.testing.assert_allclose(V, want, rtol=0, atol=4 * n_grid * 2.0**-53 * 60.0)
    np.testing.assert_array_equal(V, V.transpose(0, 2, 1))
