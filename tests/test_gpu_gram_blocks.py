"""The blocks of the Gram (gram_blocks.hpp): only the pairs of densities that a request's steps name, and
below the diagonal only where both sides hold the same densities.

Integral lists with one, two and many blocks (symmetric or not), against the oracle, in every form and
through every Gram (FP64 tensor cores, fused and split TF32x3), and the paths with their own layouts:
compute_states, shards, round splits.

Tolerance: FP64 forms 1e-10 of the largest integral (sums of a few hundred terms of like size), FP32
forms their documented 1e-6 of it.
"""
import numpy as np
import pytest

import coulombo_lattice_b200 as cl
from coulombo_lattice_b200 import synth
from oracle import host as H

pytestmark = pytest.mark.gpu

STEP = (synth.A_ZB / 4,) * 3
N, HOLES = 12, 6
# two symmetric blocks; one symmetric; left and right differ; every product with itself (78 blocks);
# exchange pairs only; every 29th of all integrals (one block, not all pairs named); one integral
LISTS = ["eeee,hhhh,ehhe,eheh", "eeee", "ehhe", "abab", "eheh,1111", "****/29", "1234"]


def _system(cells=(2, 3, 2)):
    dims = synth.grid_of(cells)
    lat = synth.zincblende_lattice(cells)
    rng = np.random.default_rng(7)
    st = rng.standard_normal((N, len(lat), 3)) + 1j * rng.standard_normal((N, len(lat), 3))
    st /= np.sqrt(np.sum(np.abs(st) ** 2, axis=(1, 2), keepdims=True))
    return dims, st, synth.cell_indices(lat, dims)


def _specs(text):
    pattern, _, every = text.partition("/")
    return cl.enumerate_integrals(pattern, N, HOLES)[::int(every or 1)]


_want = {}


def _oracle(text, dims, st, cells, specs):
    if text not in _want:
        _want[text] = np.array(H.compute_integrals(list(st), cells, dims, STEP, [tuple(int(v) for v in s) for s in specs],
                                                   dielectric=10.89, onsite=2.0))
    return _want[text]


def _close(got, want, mode):
    tol = 1e-10 if cl.mode_is_fp64(mode) else 1e-6
    assert np.abs(got - want).max() <= tol * np.abs(want).max()


@pytest.mark.parametrize("text", LISTS)
@pytest.mark.parametrize("mode,env", [(m, {}) for m in cl.ALL_MODES] +
                         [(cl.MODE_FP32_SUBLATTICE, {"CL_TC_FUSED": "1"}), (cl.MODE_FP32_SUBLATTICE, {"CL_TC_SPLIT": "1"}),
                          (cl.MODE_FP32_SUBLATTICE, {"CL_TC_MIN_ATOMS": "0"}), (cl.MODE_FP32_ROUNDS, {"CL_TC_SPLIT": "1"}),
                          (cl.MODE_FP32_SUBLATTICE, {"CL_TC_FUSED": "1", "CL_TC_NO_WS": "1"})])
def test_lists(text, mode, env, monkeypatch):
    for k, v in env.items():
        monkeypatch.setenv(k, v)
    dims, st, cells = _system()
    specs = _specs(text)
    want = _oracle(text, dims, st, cells, specs)
    with cl.CoulombCalculator(dims, STEP, mode) as cc:
        cc.initialize(dielectric=10.89, onsite=2.0)
        cc.set_states(st, cells, HOLES)
        _close(cc.compute(specs), want, mode)
        req = cc.request(specs)
        _close(req.run(), want, mode)
        req.close()
        _close(sum(cc.compute_shard(specs, k, 3) for k in range(3)), want, mode)
        if not cc.form_info()["sublattice"]:
            _close(cc.compute_rounds(specs, 0x35) + cc.compute_rounds(specs, 0xCA), want, mode)
        _close(cc.compute_states(st, cells, HOLES, specs), want, mode)


@pytest.mark.parametrize("n_states", [1, 3, 4, 8, 9, 15])
@pytest.mark.parametrize("cells", [(1, 1, 1), (2, 2, 5), (4, 5, 4)])
def test_fp64_gram_shapes(n_states, cells):
    """1 to 120 densities a side (register tiles of 1, 3 x 3, 5 x 5 and 8 x 4, k slices from 8 to 1, two
    tiles a side) over 8, 160 and 640 atoms, against the same sums of the oracle's potentials."""
    dims = synth.grid_of(cells)
    lat = synth.zincblende_lattice(cells)
    rng = np.random.default_rng(n_states)
    st = rng.standard_normal((n_states, len(lat), 2)) + 1j * rng.standard_normal((n_states, len(lat), 2))
    st /= np.sqrt(np.sum(np.abs(st) ** 2, axis=(1, 2), keepdims=True))
    specs = cl.enumerate_integrals("****", n_states, 0)[::1 if n_states < 9 else 31]
    idx = synth.cell_indices(lat, dims)
    want = np.array(H.compute_integrals(list(st), idx, dims, STEP, [tuple(int(v) for v in s) for s in specs],
                                        dielectric=10.89, onsite=2.0))
    for mode in (cl.MODE_FP64_SUBLATTICE, cl.MODE_FP32_SUBLATTICE, cl.MODE_FP32_ROUNDS):
        with cl.CoulombCalculator(dims, STEP, mode) as cc:
            cc.initialize(dielectric=10.89, onsite=2.0)
            cc.set_states(st, idx, 0)
            _close(cc.compute(specs), want, mode)


def test_odd_atom_count_rows_off_16_bytes():
    """An odd number of atoms puts every other FP32 row off a 16-byte boundary (8-byte copies)."""
    dims, st, cells = _system()
    st, cells = st[:, :-1], cells[:-1]
    specs = _specs("eheh")
    want = np.array(H.compute_integrals(list(st), cells, dims, STEP, [tuple(int(v) for v in s) for s in specs],
                                        dielectric=10.89, onsite=2.0))
    for mode in (cl.MODE_FP64_PLAIN, cl.MODE_FP32_SUBLATTICE):
        with cl.CoulombCalculator(dims, STEP, mode) as cc:
            cc.initialize(dielectric=10.89, onsite=2.0)
            cc.set_states(st, cells, HOLES)
            _close(cc.compute(specs), want, mode)


@pytest.mark.parametrize("text", ["eeee,hhhh,ehhe,eheh", "eheh,1111", "****/29"])
@pytest.mark.parametrize("mode", cl.ALL_MODES)
def test_overlapped_upload_sums_alike(text, mode, monkeypatch):
    """compute_states transforms its densities in other groups than a request but reduces them in the same
    tiles: only the order of the FP64 additions of the atom splits differs (1e-12 of the largest value)."""
    monkeypatch.setenv("CL_TC_MIN_ATOMS", "0")
    dims, st, cells = _system((4, 5, 4))
    specs = _specs(text)
    with cl.CoulombCalculator(dims, STEP, mode) as cc:
        cc.initialize(dielectric=10.89, onsite=2.0)
        cc.set_states(st, cells, HOLES)
        want = cc.compute(specs)
        req = cc.request(specs)
        got = req.run().copy()
        req.close()
        over = cc.compute_states(st, cells, HOLES, specs)
    tol = 1e-12 * np.abs(want).max()
    assert np.abs(got - want).max() <= tol
    assert np.abs(over - want).max() <= tol
