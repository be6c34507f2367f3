"""Potentials in the caller's atom order (unsorted atoms, several atoms of one cell) and eager calls of
different requests in turn on one context, whose device lists and buffers are kept between calls.

Tolerance: repeated calls differ only in the order of FP64 atomic sums (1e-12 of the largest value); the
forms against the oracle's potentials by their documented errors (1e-10, 1e-6 of the largest).
"""
import numpy as np
import pytest

import coulombo_lattice_b200 as cl
from oracle import coulomb as C

pytestmark = pytest.mark.gpu


def _system(n_states=10):
    rng = np.random.default_rng(5)
    dims = (16, 12, 8)
    cells = rng.permutation(np.concatenate([rng.choice(16 * 12 * 8, size=300, replace=False)] * 1))
    cells = np.concatenate([cells, cells[:20]]).astype(np.int64)  # 20 cells named twice: the later atom counts
    st = rng.standard_normal((n_states, len(cells), 3)) + 1j * rng.standard_normal((n_states, len(cells), 3))
    st /= np.sqrt(np.sum(np.abs(st) ** 2, axis=(1, 2), keepdims=True))
    return dims, cells, st


@pytest.mark.parametrize("mode", cl.ALL_MODES)
def test_order(mode):
    dims, cells, st = _system(3)
    g = C.kernel_spectrum(C.kernel_octant(dims, (1.0, 1.0, 1.0), 2.0, 1.5), dims)
    want = []
    for s in range(3):
        rho = C.pair_density_atoms(st[s], st[s])
        want.append(C.prepare(C.scatter_density(rho, cells, dims), g).reshape(-1)[cells].real)
    want = np.array(want)
    with cl.CoulombCalculator(dims, (1.0, 1.0, 1.0), mode) as cc:
        cc.initialize(dielectric=2.0, onsite=1.5)
        cc.set_states(st, cells, 0)
        got = cc.potentials()
        again = cc.potentials()
    tol = 1e-10 if cl.mode_is_fp64(mode) else 1e-6
    assert np.abs(got - want).max() <= tol * np.abs(want).max()
    assert np.array_equal(got, again)


@pytest.mark.parametrize("mode", cl.ALL_MODES)
def test_eager_calls_in_turn(mode):
    dims, cells, st = _system()
    lists = [cl.enumerate_integrals(p, 10, 5) for p in ("eeee", "1234", "eeee,hhhh,ehhe,eheh")]
    with cl.CoulombCalculator(dims, (1.0, 1.0, 1.0), mode) as cc:
        cc.initialize(dielectric=2.0, onsite=1.5)
        cc.set_states(st, cells, 5)
        first = [cc.compute(s) for s in lists]
        pot = cc.potentials()
        for k in (2, 0, 1, 0, 2):
            got = cc.compute(lists[k])
            assert np.abs(got - first[k]).max() <= 1e-12 * np.abs(first[k]).max()
            assert np.array_equal(cc.potentials(), pot)
