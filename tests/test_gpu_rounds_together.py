"""The rounds of a small grid in one launch of each pass: any subset of the rounds against the same rounds
one call each, on register passes, generic passes (lengths below 16), fused plane passes and mixes.

Tolerance: the same kernels on the same values, summed over the rounds in FP64 in another order: 1e-12 of
the largest integral in FP64; in FP32 the passes' values are the same too.
"""
import numpy as np
import pytest

import coulombo_lattice_b200 as cl

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mode", [cl.MODE_FP64_PLAIN, cl.MODE_FP32_ROUNDS])
@pytest.mark.parametrize("dims", [(16, 16, 16), (6, 10, 5), (45, 18, 8), (64, 64, 3), (15, 64, 20)])
@pytest.mark.parametrize("mask", [0xFF, 0x81, 0x36, 0x01])
def test_subsets(mode, dims, mask):
    rng = np.random.default_rng(mask)
    m = int(np.prod(dims))
    cells = np.sort(rng.choice(m, size=m // 2, replace=False)).astype(np.int64)
    st = rng.standard_normal((3, len(cells), 2)) + 1j * rng.standard_normal((3, len(cells), 2))
    st /= np.sqrt(np.sum(np.abs(st) ** 2, axis=(1, 2), keepdims=True))
    specs = cl.enumerate_integrals("****", 3, 1)
    with cl.CoulombCalculator(dims, (1.0, 1.1, 0.9), mode) as cc:
        cc.initialize(dielectric=3.0, onsite=2.0)
        cc.set_states(st, cells, 1)
        got = cc.compute_rounds(specs, mask)
        want = sum(cc.compute_rounds(specs, 1 << r) for r in range(8) if (mask >> r) & 1)
    assert np.abs(got - want).max() <= 1e-12 * np.abs(want).max()
