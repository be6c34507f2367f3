"""Error of the FP32 sub-lattice transforms (z pass that mixes in registers, quadrant plane passes) on smooth
densities, where the rounding of their constants adds up: it is the same in every line.

Reference: the FP64 sub-lattice form, whose own error is below 1e-14, on the same states; both sum the products
in FP64 (at most 65,536 atoms, or CL_TC_MIN_ATOMS).  Tolerance: one rounding of a float, 2^-24 = 6.0e-8, in the
root-mean-square sense over the integrals.  Counted for these lengths, the constants of six transforms (three axes,
both ways) shift an integral by at most 4e-8, and the tables and the data's own rounding add about 2e-8.
"""
import numpy as np
import pytest

import coulombo_lattice_b200 as cl
from coulombo_lattice_b200 import synth

pytestmark = pytest.mark.gpu


def _gaussians(cells_idx, dims, n):
    x = np.stack([cells_idx % dims[0], cells_idx // dims[0] % dims[1], cells_idx // (dims[0] * dims[1])]).astype(float)
    half = 0.5 * (x.max(axis=1) - x.min(axis=1))
    r2 = (((x - x.mean(axis=1)[:, None]) / half[:, None]) ** 2).sum(axis=0)
    states = np.stack([np.exp(-r2 / (2 * (0.3 + 0.05 * s) ** 2)) for s in range(n)]).astype(complex)
    return states[:, :, None] / np.sqrt((np.abs(states) ** 2).sum(axis=1))[:, None, None]


@pytest.mark.parametrize("cells,dims", [((6,) * 3, (24,) * 3), ((9,) * 3, (36,) * 3), ((10,) * 3, (40,) * 3),
                                        ((12,) * 3, (48,) * 3), ((15,) * 3, (60,) * 3), ((18,) * 3, (72,) * 3),
                                        ((20,) * 3, (80,) * 3), ((27,) * 3, (108,) * 3), ((13,) * 3, (54,) * 3),
                                        ((13, 18, 20), (54, 72, 80)), ((9, 10, 15), (36, 40, 60))])
def test_smooth_densities(cells, dims, monkeypatch):
    monkeypatch.setenv("CL_TC_MIN_ATOMS", str(1 << 40))
    idx = synth.cell_indices(synth.zincblende_lattice(cells), dims)
    states = _gaussians(idx, dims, 4)
    specs = cl.enumerate_integrals("eeee", 4, 0)
    got = {}
    for mode in (cl.MODE_FP32_SUBLATTICE, cl.MODE_FP64_SUBLATTICE):
        with cl.CoulombCalculator(dims, (synth.A_ZB / 4,) * 3, mode) as cc:
            cc.initialize(dielectric=10.89)
            cc.set_states(states, idx, 0)
            assert cc.form_info()["sublattice"]
            got[mode] = cc.compute(specs)
    want = got[cl.MODE_FP64_SUBLATTICE]
    error = np.sqrt((np.abs(got[cl.MODE_FP32_SUBLATTICE] - want) ** 2).sum() / (np.abs(want) ** 2).sum())
    assert error <= 2.0 ** -24, error
