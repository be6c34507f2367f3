"""Pair densities on the FP64 tensor cores at the ends of their range: up to 4 states, whose atoms share a tile, and orbital
counts that come in slices; states below, at and off a tile, orbitals below, at and off a slice, atoms below, at and
off a batch, one and several batches a block, both precisions.

Reference and tolerances as in test_gpu_pair_mma.py: a Coulomb kernel that is zero off the origin makes an integral a
multiple of sum_a rho_l(a) rho_r(a), which numpy gives in FP64; 1e-12 of the largest in FP64, the documented 1e-6 in
the FP32 forms.
"""
import numpy as np
import pytest

import coulombo_lattice_b200 as cl

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mode", [cl.MODE_FP64_PLAIN, cl.MODE_FP32_ROUNDS])
@pytest.mark.parametrize("n_states,n_orb,atoms,every",
                         [(1, 1, 1, 1), (1, 5, 63, 1), (1, 20, 64, 1), (1, 20, 65, 1), (1, 500, 70, 1), (2, 1, 31, 1),
                          (2, 10, 32, 1), (2, 20, 500, 1), (2, 16, 33, 1), (2, 17, 1, 1), (3, 1, 15, 1), (3, 20, 17, 1),
                          (3, 300, 40, 1), (4, 5, 16, 1), (4, 20, 1000, 1), (4, 250, 33, 1), (5, 20, 9, 1),
                          (8, 109, 20, 1), (8, 128, 8, 1), (8, 300, 11, 1), (11, 81, 17, 3), (12, 73, 1100, 7),
                          (12, 160, 9, 7), (17, 64, 30, 11), (24, 97, 12, 31), (30, 50, 10, 97), (40, 41, 9, 499),
                          (40, 96, 5, 499)])
def test_shapes(mode, n_states, n_orb, atoms, every):
    rng = np.random.default_rng(1000 * n_states + n_orb)
    cells = np.sort(rng.choice(16 * 8 * 9, size=atoms, replace=False)).astype(np.int64)
    st = rng.standard_normal((n_states, atoms, n_orb)) + 1j * rng.standard_normal((n_states, atoms, n_orb))
    st /= np.sqrt(np.sum(np.abs(st) ** 2, axis=(1, 2), keepdims=True))
    G = np.zeros((10, 9, 17))
    G[0, 0, 0] = 2.5
    specs = cl.enumerate_integrals("****", n_states, 0)[::every]
    with cl.CoulombCalculator((16, 8, 9), (1.0, 1.0, 1.0), mode) as cc:
        cc.initialize_grid(G)
        cc.set_states(st, cells, 0)
        got = cc.compute(specs)
    rho = np.einsum("iao,jao->ija", st.conj(), st)
    i1, i2, i3, i4 = (specs.astype(int) - 1).T
    want = 2.5 * np.sum(rho[i1, i4] * rho[i2, i3], axis=1)
    tol = 1e-12 if cl.mode_is_fp64(mode) else 1e-6
    assert np.abs(got - want).max() <= tol * np.abs(want).max()
