"""The quadrant plane passes (plane_w.cuh): square class planes of every compiled length, all atoms of the
quadrant present (pairwise copies) and a quarter of them missing (rows of masks, odd atom counts, cleared
slots between densities), over one and several densities a block and ragged last row batches.

Tolerance: the FP32 transforms' documented error, 1e-6 of the largest integral; FP64, 1e-12 of it.
"""
import numpy as np
import pytest

import coulombo_lattice_b200 as cl
from coulombo_lattice_b200 import synth
from oracle import host as H

pytestmark = pytest.mark.gpu

LENGTHS = [12, 16, 18, 20, 24, 30, 32, 36, 40, 48, 50, 54, 60, 64, 72, 80, 90, 96, 100, 108, 120, 128]


SL_MODES = [cl.MODE_FP32_SUBLATTICE, cl.MODE_FP64_SUBLATTICE]


@pytest.mark.parametrize("mode", SL_MODES)
@pytest.mark.parametrize("drop", [0.0, 0.25])
@pytest.mark.parametrize("n", LENGTHS)
def test_lengths(n, drop, mode, monkeypatch):
    dims = (2 * n, 2 * n, 24 if n <= 32 else 12 * 2)
    lat = synth.zincblende_lattice((n // 2, n // 2, 6))
    lat = lat[lat[:, 2] < (24 if n <= 32 else 4)]
    rng = np.random.default_rng(n)
    if drop:
        lat = lat[rng.random(len(lat)) >= drop]
    n_states = 4 if n <= 32 else 2
    st = rng.standard_normal((n_states, len(lat), 2)) + 1j * rng.standard_normal((n_states, len(lat), 2))
    st /= np.sqrt(np.sum(np.abs(st) ** 2, axis=(1, 2), keepdims=True))
    cells = synth.cell_indices(lat, dims)
    specs = [tuple(int(v) for v in s) for s in cl.enumerate_integrals("****", n_states, 1)]
    step = (synth.A_ZB / 4,) * 3
    want = np.array(H.compute_integrals(list(st), cells, dims, step, specs, dielectric=10.89, onsite=3.0))

    tol = 1e-12 if cl.mode_is_fp64(mode) else 1e-6

    def run():
        with cl.CoulombCalculator(dims, step, mode) as cc:
            cc.initialize(dielectric=10.89, onsite=3.0)
            cc.set_states(st, cells, 1)
            assert cc.form_info()["lengths"][:2] == (n, n)
            cc.set_profiling(True)
            v = cc.compute(specs)
            assert "y_pass" not in cc.kernel_profile()  # x and y in one launch
            return v, cc.potentials()

    got, pot = run()
    assert np.abs(got - want).max() <= tol * np.abs(want).max()
    monkeypatch.setenv("CL_NO_QPLANE", "1")
    with cl.CoulombCalculator(dims, step, cl.MODE_FP64_SUBLATTICE) as cc:
        cc.initialize(dielectric=10.89, onsite=3.0)
        cc.set_states(st, cells, 1)
        ref = cc.potentials()
    assert np.abs(pot - ref).max() <= tol * np.abs(ref).max()


@pytest.mark.parametrize("mode", SL_MODES)
@pytest.mark.parametrize("drop", [0.0, 0.25])
@pytest.mark.parametrize("k", range(len(LENGTHS)))
def test_two_lengths(k, drop, mode):
    """Planes of two lengths: every length once as x and once as y (against one 7 places on, shorter and
    longer), two grids of two classes among them when neither length divides by 4."""
    nx, ny = LENGTHS[k], LENGTHS[(k + 7) % len(LENGTHS)]
    dims = (2 * nx, 2 * ny, 24)
    lat = synth.zincblende_lattice((nx // 2, ny // 2, 6))
    lat = lat[lat[:, 2] < (24 if nx * ny <= 1024 else 4)]
    rng = np.random.default_rng(k)
    if drop:
        lat = lat[rng.random(len(lat)) >= drop]
    n_states = 4 if nx * ny <= 1024 else 2
    st = rng.standard_normal((n_states, len(lat), 2)) + 1j * rng.standard_normal((n_states, len(lat), 2))
    st /= np.sqrt(np.sum(np.abs(st) ** 2, axis=(1, 2), keepdims=True))
    cells = synth.cell_indices(lat, dims)
    specs = [tuple(int(v) for v in s) for s in cl.enumerate_integrals("****", n_states, 1)]
    step = (synth.A_ZB / 4,) * 3
    want = np.array(H.compute_integrals(list(st), cells, dims, step, specs, dielectric=10.89, onsite=3.0))
    with cl.CoulombCalculator(dims, step, mode) as cc:
        cc.initialize(dielectric=10.89, onsite=3.0)
        cc.set_states(st, cells, 1)
        assert cc.form_info()["lengths"][:2] == (nx, ny)
        cc.set_profiling(True)
        got = cc.compute(specs)
        assert "y_pass" not in cc.kernel_profile()
    tol = 1e-12 if cl.mode_is_fp64(mode) else 1e-6
    assert np.abs(got - want).max() <= tol * np.abs(want).max()
