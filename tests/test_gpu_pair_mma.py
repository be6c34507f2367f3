"""Pair densities on the FP64 tensor cores (pair_mma.cuh): every count of 8-state blocks (padded states),
orbital counts below, at and off the 4 of a step and either side of the diagonal folding, atom counts
below, at and off a batch, dense and sparse products, both precisions.

Reference: the densities' Gram through the FP64 form's oracle would mix in the transforms, so the check is
the on-site interaction alone: a kernel that is zero off the origin turns V into a multiple of rho, and an
integral into that multiple of sum_a rho_l(a) rho_r(a), which numpy gives in FP64.

Tolerance: FP64 1e-12 of the largest integral (sums of at most 500 atoms x 40 orbitals); FP32 forms round
densities once (2^-24) and transform in FP32: the documented 1e-6 of the largest.
"""
import numpy as np
import pytest

import coulombo_lattice_b200 as cl

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mode", [cl.MODE_FP64_PLAIN, cl.MODE_FP32_ROUNDS])
@pytest.mark.parametrize("n_states,n_orb,atoms,every",
                         [(1, 1, 1, 1), (1, 20, 7, 1), (2, 3, 8, 1), (4, 10, 33, 1), (7, 5, 100, 1), (8, 20, 500, 1),
                          (8, 17, 65, 3), (9, 16, 64, 1), (12, 20, 129, 1), (16, 15, 40, 5), (17, 20, 31, 7),
                          (24, 1, 300, 11), (25, 20, 9, 13), (32, 13, 50, 97), (33, 4, 77, 101), (40, 20, 41, 499),
                          (40, 1, 250, 997), (40, 40, 12, 997), (41, 6, 20, 1999)])
def test_shapes(mode, n_states, n_orb, atoms, every):
    rng = np.random.default_rng(100 * n_states + n_orb)
    dims = (16, 8, 9)
    cells = np.sort(rng.choice(16 * 8 * 9, size=atoms, replace=False)).astype(np.int64)
    st = rng.standard_normal((n_states, atoms, n_orb)) + 1j * rng.standard_normal((n_states, atoms, n_orb))
    st /= np.sqrt(np.sum(np.abs(st) ** 2, axis=(1, 2), keepdims=True))
    G = np.zeros((10, 9, 17))
    G[0, 0, 0] = 2.5
    specs = cl.enumerate_integrals("****", n_states, 0)[::every]
    with cl.CoulombCalculator(dims, (1.0, 1.0, 1.0), mode) as cc:
        cc.initialize_grid(G)
        cc.set_states(st, cells, 0)
        got = cc.compute(specs)
    i1, i2, i3, i4 = (specs.astype(int) - 1).T
    want = np.empty(len(specs), dtype=complex)
    for k in range(len(specs)):
        left = np.sum(st[i1[k]].conj() * st[i4[k]], axis=1)
        right = np.sum(st[i2[k]].conj() * st[i3[k]], axis=1)
        want[k] = 2.5 * np.sum(left * right)
    tol = 1e-12 if cl.mode_is_fp64(mode) else 1e-6
    assert np.abs(got - want).max() <= tol * np.abs(want).max()
