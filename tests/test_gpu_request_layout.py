"""Prepared requests and captured batches after their context has changed: larger eager calls that move its
buffers, other orbitals, atoms, states or class sets, another kernel; and states that are no longer loaded.

Reference: the eager integrals of a fresh context with the same contents.  Both run the same kernels on the
same numbers, and only the order of the FP64 sums over atoms differs: 1e-12 of the largest integral.
"""
import numpy as np
import pytest

import coulombo_lattice_b200 as cl
from coulombo_lattice_b200 import synth

pytestmark = pytest.mark.gpu

DIMS = (24, 24, 24)
STEP = (synth.A_ZB / 4,) * 3
SPECS = np.array([[1, 2, 2, 1], [1, 1, 1, 1], [2, 1, 3, 3]], dtype=np.int16)


def _zincblende(cells):
    lat = synth.zincblende_lattice(cells)
    return synth.cell_indices(lat, DIMS)


def _scattered(n, seed):
    return np.sort(np.random.default_rng(seed).choice(24 ** 3, size=n, replace=False)).astype(np.int64)


def _states(n, atoms, orbitals, seed):
    rng = np.random.default_rng(seed)
    s = rng.standard_normal((n, atoms, orbitals)) + 1j * rng.standard_normal((n, atoms, orbitals))
    return s / np.sqrt((np.abs(s) ** 2).sum(axis=(1, 2), keepdims=True))


def _contents(kind):
    """(states, cells): 4 states of 10 orbitals on a 4 x 4 x 4 box, changed as `kind` says."""
    cells = _zincblende({"more atoms": (6, 6, 6), "fewer atoms": (2, 3, 2)}.get(kind, (4, 4, 4)))
    if kind == "other classes":
        cells = _scattered(300, 7)
    orbitals = {"fewer orbitals": 3, "more orbitals": 25}.get(kind, 10)
    n = {"more states": 9}.get(kind, 4)
    return _states(n, cells.size, orbitals, len(kind)), cells


def _fresh(mode, contents, specs, dielectric=10.0):
    with cl.CoulombCalculator(DIMS, STEP, mode) as cc:
        cc.initialize(dielectric=dielectric)
        cc.set_states(contents[0], contents[1], 0)
        return cc.compute(specs)


def _close(got, want):
    assert np.abs(got - want).max() <= 1e-12 * np.abs(want).max()


@pytest.mark.parametrize("mode", cl.ALL_MODES)
def test_batch_after_larger_calls(mode):
    first = _contents("first")
    want = _fresh(mode, first, SPECS)
    with cl.CoulombCalculator(DIMS, STEP, mode) as cc, cl.CoulombCalculator(DIMS, STEP, mode) as other:
        for c in (cc, other):
            c.initialize(dielectric=10.0)
            c.set_states(*first, 0)
        reqs = [cc.request(SPECS), other.request(SPECS)]
        batch = cl.Batch(reqs)
        for larger in (lambda: None, lambda: cc.compute(cl.enumerate_integrals("****", 4, 0)), cc.potentials,
                       lambda: other.compute(cl.enumerate_integrals("****", 4, 0))):
            larger()
            for got in batch.run():
                _close(got, want)
        batch.close()
        for r in reqs:
            r.close()


@pytest.mark.parametrize("mode", cl.ALL_MODES)
@pytest.mark.parametrize("kind", ["fewer orbitals", "more orbitals", "more atoms", "fewer atoms", "more states",
                                  "other classes"])
def test_requests_follow_other_contents(mode, kind):
    first, then = _contents("first"), _contents(kind)
    with cl.CoulombCalculator(DIMS, STEP, mode) as cc:
        cc.initialize(dielectric=10.0)
        cc.set_states(*first, 0)
        req = cc.request(SPECS)
        batch = cl.Batch([req])
        _close(batch.run()[0], _fresh(mode, first, SPECS))
        cc.set_states(*then, 0)
        _close(batch.run()[0], _fresh(mode, then, SPECS))
        cc.compute_states(*first, 0, SPECS)
        _close(req.run(), _fresh(mode, first, SPECS))
        cc.set_states(*then, 0)
        _close(req.run(), _fresh(mode, then, SPECS))
        _close(batch.run()[0], _fresh(mode, then, SPECS))
        batch.close()
        req.close()


@pytest.mark.parametrize("mode", cl.ALL_MODES)
def test_batch_after_another_kernel(mode):
    first = _contents("first")
    with cl.CoulombCalculator(DIMS, STEP, mode) as cc:
        cc.initialize(dielectric=10.0)
        cc.set_states(*first, 0)
        req = cc.request(SPECS)
        req.run()
        batch = cl.Batch([req])
        for dielectric in (10.0, 4.0, 10.0):
            cc.initialize(dielectric=dielectric)
            _close(batch.run()[0], _fresh(mode, first, SPECS, dielectric))
        batch.close()
        req.close()


@pytest.mark.parametrize("mode", [cl.MODE_FP64_PLAIN, cl.MODE_FP32_SUBLATTICE])
def test_states_no_longer_loaded(mode):
    first = _contents("first")
    with cl.CoulombCalculator(DIMS, STEP, mode) as cc:
        cc.initialize(dielectric=10.0)
        cc.set_states(*first, 0)
        req = cc.request(SPECS)
        batch = cl.Batch([req])
        want = batch.run()[0]
        cc.set_states(first[0][:2], first[1], 0)
        for call in (req.run, batch.run):
            with pytest.raises(cl.CoulomboError) as e:
                call()
            assert e.value.code == 2  # CL_ERR_STATE
        cc.set_states(*first, 0)
        _close(req.run(), want)
        _close(batch.run()[0], want)
        batch.close()
        req.close()


def test_destroyed_after_their_context():
    first = _contents("first")
    for _ in range(4):
        cc = cl.CoulombCalculator(DIMS, STEP, cl.MODE_FP32_SUBLATTICE)
        cc.initialize(dielectric=10.0)
        cc.set_states(*first, 0)
        req = cc.request(SPECS)
        batch = cl.Batch([req])
        want = batch.run()[0]
        cc.close()
        req.close()
        batch.close()
        _close(_fresh(cl.MODE_FP32_SUBLATTICE, first, SPECS), want)
