"""Pair densities in tiles of 4 x 4 states where the tensor-core kernel would take them (CL_NO_PAIR_REG12=1): more than
12 states, counts that are and are not multiples of 4, dense and sparse products, both precisions.

Reference and tolerances as for the tensor-core kernel: a Coulomb kernel that is zero off the origin makes an
integral a multiple of sum_a rho_l(a) rho_r(a), which numpy gives in FP64; 1e-12 of the largest in FP64, the documented
1e-6 in the FP32 forms.
"""
import numpy as np
import pytest

import coulombo_lattice_b200 as cl

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mode", [cl.MODE_FP64_PLAIN, cl.MODE_FP32_ROUNDS])
@pytest.mark.parametrize("n_states,n_orb,atoms,pattern,every",
                         [(13, 20, 61, "****", 7), (16, 3, 200, "****", 7), (22, 4, 90, "eheh", 1),
                          (24, 20, 33, "eeee,hhhh", 5), (39, 5, 17, "****", 997), (40, 20, 41, "****", 499),
                          (40, 20, 9, "eheh", 101)])
def test_tiles(mode, n_states, n_orb, atoms, pattern, every, monkeypatch):
    monkeypatch.setenv("CL_NO_PAIR_REG12", "1")
    rng = np.random.default_rng(100 * n_states + n_orb)
    cells = np.sort(rng.choice(16 * 8 * 9, size=atoms, replace=False)).astype(np.int64)
    st = rng.standard_normal((n_states, atoms, n_orb)) + 1j * rng.standard_normal((n_states, atoms, n_orb))
    st /= np.sqrt(np.sum(np.abs(st) ** 2, axis=(1, 2), keepdims=True))
    G = np.zeros((10, 9, 17))
    G[0, 0, 0] = 2.5
    specs = cl.enumerate_integrals(pattern, n_states, n_states // 2)[::every]
    with cl.CoulombCalculator((16, 8, 9), (1.0, 1.0, 1.0), mode) as cc:
        cc.initialize_grid(G)
        cc.set_states(st, cells, n_states // 2)
        got = cc.compute(specs)
    i1, i2, i3, i4 = (specs.astype(int) - 1).T
    left = np.einsum("kao,kao->ka", st[i1].conj(), st[i4])
    right = np.einsum("kao,kao->ka", st[i2].conj(), st[i3])
    want = 2.5 * np.sum(left * right, axis=1)
    tol = 1e-12 if cl.mode_is_fp64(mode) else 1e-6
    assert np.abs(got - want).max() <= tol * np.abs(want).max()
