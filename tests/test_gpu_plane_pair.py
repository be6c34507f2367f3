"""The quadrant plane passes on class planes modulo 2, with the z pass of two classes: square planes and planes of
two lengths, the box's atoms all there and a quarter of them missing.

Tolerance: the FP32 transforms' documented error, 1e-6 of the largest integral; FP64, 1e-12 of it.
"""
import numpy as np
import pytest

import coulombo_lattice_b200 as cl
from coulombo_lattice_b200 import synth
from oracle import host as H

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mode", [cl.MODE_FP32_SUBLATTICE, cl.MODE_FP64_SUBLATTICE])
@pytest.mark.parametrize("drop", [0.0, 0.25])
@pytest.mark.parametrize("dims", [(18, 18, 18), (30, 30, 20), (54, 54, 18), (90, 90, 18), (18, 24, 20), (24, 18, 32),
                                  (54, 72, 18), (128, 50, 20), (12, 54, 24)])
def test_two_classes(dims, drop, mode):
    lat = synth.zincblende_lattice(tuple(-(-d // 4) for d in dims))
    lat = lat[np.all(lat < np.array(dims), axis=1)]
    rng = np.random.default_rng(sum(dims))
    lat = lat[rng.random(len(lat)) >= drop]
    st = rng.standard_normal((2, len(lat), 2)) + 1j * rng.standard_normal((2, len(lat), 2))
    st /= np.sqrt(np.sum(np.abs(st) ** 2, axis=(1, 2), keepdims=True))
    cells = synth.cell_indices(lat, dims)
    specs = [tuple(int(v) for v in s) for s in cl.enumerate_integrals("****", 2, 1)]
    step = (synth.A_ZB / 4,) * 3
    want = np.array(H.compute_integrals(list(st), cells, dims, step, specs, dielectric=10.89, onsite=3.0))
    with cl.CoulombCalculator(dims, step, mode) as cc:
        cc.initialize(dielectric=10.89, onsite=3.0)
        cc.set_states(st, cells, 1)
        info = cc.form_info()
        assert (info["m"], info["classes"], info["lengths"]) == (2, 2, dims)
        cc.set_profiling(True)
        got = cc.compute(specs)
        assert "y_pass" not in cc.kernel_profile()  # x and y in one launch
    tol = 1e-12 if cl.mode_is_fp64(mode) else 1e-6
    assert np.abs(got - want).max() <= tol * np.abs(want).max()
