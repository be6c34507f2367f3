"""The z pass that mixes the classes of a frequency in registers (zmix_wht.cuh), every compiled length.

Zinc-blende boxes (8 classes) and grids with two classes modulo 2, in both precisions, with z axes of every
compiled transform length: splits with one and two phase-A rounds, tails of a column block (x y planes
of 36 and 144 columns against blocks of 8 and 16), one and several densities a warp group, and
structures whose grid origin falls on any of the classes (all signs of the axis phases).

Tolerance: the FP32 transforms' documented error, 1e-6 of the largest integral; FP64, 1e-12 of it (2^-52
times a few tens over transforms of at most 2^18 points).
"""
import numpy as np
import pytest

import coulombo_lattice_b200 as cl
from coulombo_lattice_b200 import synth
from oracle import host as H

pytestmark = pytest.mark.gpu

ZB = [12, 16, 18, 20, 24, 30, 32, 36, 40, 48, 50, 54, 60, 64, 72, 80, 90, 96, 100, 108, 120, 128]
PAIR = [18, 20, 24, 30, 32, 36, 40, 48, 50, 54, 60, 64, 72, 80, 90, 96, 100, 108, 120, 128, 144, 150, 160, 180, 192,
        240, 256]


SL_MODES = [cl.MODE_FP32_SUBLATTICE, cl.MODE_FP64_SUBLATTICE]


def _check(lat, dims, m, classes, n_states, seed, mode):
    rng = np.random.default_rng(seed)
    st = rng.standard_normal((n_states, len(lat), 2)) + 1j * rng.standard_normal((n_states, len(lat), 2))
    st /= np.sqrt(np.sum(np.abs(st) ** 2, axis=(1, 2), keepdims=True))
    cells = (lat[:, 2] * dims[1] + lat[:, 1]) * dims[0] + lat[:, 0]
    specs = [tuple(int(v) for v in s) for s in cl.enumerate_integrals("****", n_states, 1)]
    step = (synth.A_ZB / 4,) * 3
    want = np.array(H.compute_integrals(list(st), cells, dims, step, specs, dielectric=10.89, onsite=3.0))
    with cl.CoulombCalculator(dims, step, mode) as cc:
        cc.initialize(dielectric=10.89, onsite=3.0)
        cc.set_states(st, cells, 1)
        info = cc.form_info()
        got = cc.compute(specs)
    assert info["sublattice"] and info["m"] == m and info["classes"] == classes
    tol = 1e-12 if cl.mode_is_fp64(mode) else 1e-6
    assert np.abs(got - want).max() <= tol * np.abs(want).max()


def _crop(cells, origin, dims):
    """Sites of a zinc-blende box inside [origin, origin + dims), moved to the origin."""
    lat = synth.zincblende_lattice(cells) - np.array(origin)
    return lat[np.all((lat >= 0) & (lat < np.array(dims)), axis=1)]


@pytest.mark.parametrize("mode", SL_MODES)
@pytest.mark.parametrize("n", ZB)
def test_zincblende_lengths(n, mode):
    dims = (12, 12, 2 * n)
    _check(_crop((3, 3, n // 2), (0, 0, 0), dims), dims, 4, 8, 2 if n > 64 else 4, n, mode)


@pytest.mark.parametrize("mode", SL_MODES)
@pytest.mark.parametrize("origin", [(1, 0, 0), (0, 2, 0), (0, 0, 3), (3, 1, 2), (2, 3, 1), (3, 3, 3), (2, 2, 2)])
@pytest.mark.parametrize("nz", [24, 32])  # coefficients of every kz (R2 = 2: half of them), R2 = 2
def test_zincblende_origins(origin, nz, mode):
    dims = (12, 20, nz)
    _check(_crop((4, 6, nz // 4 + 1), origin, dims), dims, 4, 8, 2, sum(origin), mode)


@pytest.mark.parametrize("mode", SL_MODES)
@pytest.mark.parametrize("n", PAIR)
def test_two_class_lengths(n, mode):
    dims = (6, 6, n)
    _check(_crop((2, 2, n // 4 + 1), (0, 0, 0), dims), dims, 2, 2, 2 if n > 64 else 4, n, mode)


@pytest.mark.parametrize("mode", SL_MODES)
@pytest.mark.parametrize("origin", [(1, 0, 0), (0, 1, 0), (0, 0, 1), (1, 1, 1)])
def test_two_class_origins(origin, mode):
    dims = (10, 6, 18)
    _check(_crop((4, 3, 6), origin, dims), dims, 2, 2, 3, sum(origin), mode)
