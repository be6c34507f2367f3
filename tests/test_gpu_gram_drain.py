"""The fused TF32x3 Gram adds every k-tile of 32 atoms to FP64 by itself where a request takes more than one tile of 64
left and 40 right densities, as the Gram after the split pass does.

Reference: the split pass's Gram on the same potentials and densities (CL_TC_SPLIT=1).  Both split to the same
TF32 parts and issue the same MMAs over one range of atoms (640 atoms are 20 k-tiles, one split), so only the order
of FP64 additions differs: 1e-12 of the largest integral.
"""
import numpy as np
import pytest

import coulombo_lattice_b200 as cl
from coulombo_lattice_b200 import synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n_states,pattern", [(9, "****"), (11, "****"), (12, "****"), (12, "eeee,hhhh,ehhe,eheh"),
                                              (16, "eeee,hhhh")])
def test_every_k_tile_goes_to_fp64(n_states, pattern, monkeypatch):
    monkeypatch.setenv("CL_TC_MIN_ATOMS", "0")
    d = synth.build("c2", cells=(4, 5, 4))
    d["states"] = synth.make_states(d["pos"], 4, n_states, 40 * n_states, "gauss")
    specs = cl.enumerate_integrals(pattern, n_states, n_states // 2)[::3]
    got = {}
    for split in (False, True):
        if split:
            monkeypatch.setenv("CL_TC_SPLIT", "1")
        with cl.CoulombCalculator(d["dims"], (synth.A_ZB / 4,) * 3, cl.MODE_FP32_SUBLATTICE) as cc:
            cc.initialize(dielectric=10.89)
            cc.set_states(d["states"], d["cells_idx"], n_states // 2)
            cc.set_profiling(True)
            got[split] = cc.compute(specs)
            assert ("gram_split" in cc.kernel_profile()) == split
    assert np.abs(got[False] - got[True]).max() <= 1e-12 * np.abs(got[True]).max()
