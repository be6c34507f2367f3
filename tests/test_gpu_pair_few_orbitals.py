"""Pair densities of few orbitals and many states on both sides of the choice between the tensor-core and the tile
kernel (CL_NO_PAIR_TILE=1: the tensor cores whatever the products): the diagonal products alone, one tile, one row of
tiles, a few anywhere, all; blocks that are full and ragged, orbitals below, at and off a step, both precisions.

Reference and tolerances as in test_gpu_pair_mma.py: a Coulomb kernel that is zero off the origin makes an integral a
multiple of sum_a rho_l(a) rho_r(a), which numpy gives in FP64; 1e-12 of the largest in FP64, the documented 1e-6 in
the FP32 forms.
"""
import numpy as np
import pytest

import coulombo_lattice_b200 as cl

pytestmark = pytest.mark.gpu

PRODUCTS = {
    "all": lambda n: [(i, j) for i in range(n) for j in range(i + 1)],
    "diagonal": lambda n: [(i, i) for i in range(n)],
    "corner": lambda n: [(i, i % 8) for i in range(n - 1, n - 9, -1)] + [(n - 1, n - 1)],
    "row": lambda n: [(n - 1, j) for j in range(n)],
    "few": lambda n: [(i, (7 * i + 3) % (i + 1)) for i in range(n) if i % 3 != 1] + [(n - 1, n - 2)],
    # states of two kinds, products of one of each
    "across": lambda n: [(i, j) for i in range(n // 2 + 4, n) for j in range(0, n // 2 - 4, 3)],
}


@pytest.mark.parametrize("mode", [cl.MODE_FP64_PLAIN, cl.MODE_FP32_ROUNDS])
@pytest.mark.parametrize("tensor_cores", [False, True])
@pytest.mark.parametrize("products", sorted(PRODUCTS))
@pytest.mark.parametrize("n_states,n_orb,atoms",
                         [(17, 2, 300), (17, 10, 25), (20, 5, 33), (24, 3, 65), (25, 4, 31), (32, 8, 40), (36, 3, 1),
                          (40, 5, 1000), (40, 10, 9)])
def test_products(mode, tensor_cores, products, n_states, n_orb, atoms, monkeypatch):
    if tensor_cores:
        monkeypatch.setenv("CL_NO_PAIR_TILE", "1")
    rng = np.random.default_rng(100 * n_states + n_orb)
    cells = np.sort(rng.choice(16 * 8 * 9, size=atoms, replace=False)).astype(np.int64)
    st = rng.standard_normal((n_states, atoms, n_orb)) + 1j * rng.standard_normal((n_states, atoms, n_orb))
    st /= np.sqrt(np.sum(np.abs(st) ** 2, axis=(1, 2), keepdims=True))
    G = np.zeros((10, 9, 17))
    G[0, 0, 0] = 2.5
    named = list(dict.fromkeys(PRODUCTS[products](n_states)))
    # each product with the first one and with itself, either factor conjugated
    specs = np.array([(named[0][0], p[0], p[1], named[0][1]) for p in named] + [(p[1], p[0], p[1], p[0]) for p in named],
                     dtype=np.int16) + 1
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
