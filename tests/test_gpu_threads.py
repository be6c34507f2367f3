"""Contexts on threads of their own whose launches of one kernel need different amounts of shared memory: every call
succeeds and repeats what a single thread gets.

FP64: the same launches on the same data, so only the order of FP64 sums may differ: 1e-12 of the largest value.
"""
import threading

import numpy as np
import pytest

import coulombo_lattice_b200 as cl

pytestmark = pytest.mark.gpu


# the passes for any length, and the segment kernel of the pair densities
@pytest.mark.parametrize("env", [{"CL_NO_REGISTER_FFT": "1"}, {"CL_NO_PAIR_REG12": "1", "CL_NO_PAIR_TILE": "1"},
                                 {"CL_NO_PAIR_REG12": "1"}])
def test_two_shapes(env, monkeypatch):
    for k, v in env.items():
        monkeypatch.setenv(k, v)

    def make(dims, n_states, n_orb):
        rng = np.random.default_rng(n_states)
        cells = np.sort(rng.choice(int(np.prod(dims)), size=60, replace=False)).astype(np.int64)
        st = rng.standard_normal((n_states, 60, n_orb)) + 1j * rng.standard_normal((n_states, 60, n_orb))
        specs = cl.enumerate_integrals("eeee", n_states, 0)[:40]
        cc = cl.CoulombCalculator(dims, (1.0, 1.0, 1.0), cl.MODE_FP64_PLAIN)
        cc.initialize(dielectric=10.0)
        cc.set_states(st, cells, 0)
        return cc, specs

    made = [make((16, 8, 9), 2, 3), make((60, 30, 45), 5, 20)]
    want = [cc.compute(s) for cc, s in made]
    failures = []

    def work(cc, specs, w):
        for _ in range(300):
            try:
                got = cc.compute(specs)
            except cl.CoulomboError as e:
                failures.append(str(e))
                return
            if np.abs(got - w).max() > 1e-12 * np.abs(w).max():
                failures.append("values differ")
                return

    threads = [threading.Thread(target=work, args=(cc, s, w)) for (cc, s), w in zip(made, want)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    for cc, _ in made:
        cc.close()
    assert not failures, failures
