"""Performance cases of the Coulomb-integral path, through its public entry points.

A case is a zinc-blende structure on the a/4 grid (conventional cells per axis; the whole box, or
the atoms of the inscribed ellipsoid, as in a dot), seeded LCAO states (Gaussian envelopes of s,
p and d shape times a complex normal value per orbital), an integral list, a form (`mode`: all
FP64 or FP32 transforms, 8 rounds or sub-lattice) and the entry point that a program calls:

  request     a prepared request (`CoulombCalculator.request`), run again and again
  batch       prepared requests of several structures as one graph (`Batch`)
  compute     `CoulombCalculator.compute` on loaded states
  states      `CoulombCalculator.compute_states`: host coefficients in, integrals out
  potentials  `CoulombCalculator.potentials` of the loaded states
  grid        `prepare` / `calculate` on dense grids, the reference's own seam

Grids are padded to products of 2, 3 and 5 as the command line does it, so box sizes also decide
which decomposition runs: grids divisible by 4 have 8 atom classes, those only divisible by 2
have 2, and the rest take the 8 rounds.

The FP32 forms compute with 24-bit transforms (documented error: 1e-6 of an integral), so a
program that asks for them keeps single precision results; the FP64 forms' stay in double.
"""
import math

import numpy as np
import torch

import coulombo_lattice_b200 as cl

A_ZB = 5.65           # lattice constant, Angstrom
DIELECTRIC = 10.89
E2_4PE0 = 14.39963737103201  # e^2/(4 pi eps0), eV Angstrom
MODES = {"fp64": cl.MODE_FP64_PLAIN, "fp32": cl.MODE_FP32_ROUNDS, "fp64sub": cl.MODE_FP64_SUBLATTICE,
         "fp32sub": cl.MODE_FP32_SUBLATTICE}
CLASSES = "eeee,hhhh,ehhe,eheh"
BASIS = ((0, 0, 0), (0, 2, 2), (2, 0, 2), (2, 2, 0), (1, 1, 1), (1, 3, 3), (3, 1, 3), (3, 3, 1))


def _case(name, entry, mode, cells, orbitals, electrons, holes, integrals=CLASSES, shape="box", onsite=0.0, boxes=1):
    return {"name": name, "entry": entry, "mode": mode, "lx": cells[0], "ly": cells[1], "lz": cells[2],
            "orbitals": orbitals, "electrons": electrons, "holes": holes, "integrals": integrals, "shape": shape,
            "onsite": onsite, "boxes": boxes}


def listed():
    return [
        # a quantum dot of 4,096 atoms, no spin: the smallest request, bound by launches and latency
        _case("box8_fp32sub", "request", "fp32sub", (8, 8, 8), 10, 2, 2),
        # the same in the reference's own all-FP64 method, called once a request
        _case("box8_fp64", "compute", "fp64", (8, 8, 8), 10, 2, 2),
        # a medium lens-dot box (110,592 atoms, with spin), 12 states: 5,184 integrals
        _case("box24_fp32sub", "request", "fp32sub", (24, 24, 24), 20, 6, 6),
        # the same box where FP64 results are asked for
        _case("box24_fp64sub", "request", "fp64sub", (24, 24, 24), 20, 6, 6),
        # the multi-million-atom box: 2,097,152 atoms, 4 e + 4 h states, 1,024 integrals
        _case("box64_fp32sub", "request", "fp32sub", (64, 64, 64), 20, 4, 4),
        # every integral of 40 states (configuration interaction): 2,560,000 over 262,144 atoms
        _case("box32_allpairs", "request", "fp32sub", (32, 32, 32), 20, 20, 20, "ijkl"),
        # uneven structures of a size study, one graph launch a step
        _case("batch_uneven", "batch", "fp32sub", (12, 12, 12), 20, 4, 4, CLASSES, "box", 0.0, 6),
        # a donor in an 11-cell ball: its 44-point axes pad to 45, which has no sub-lattice
        _case("ball11_rounds", "request", "fp32sub", (11, 11, 11), 10, 4, 0, "eeee", "ball", 5.0),
        # a flat, ragged dot: axes of 54, 72 and 80 points, two atom classes
        _case("ball13x18x20", "request", "fp32sub", (13, 18, 20), 20, 4, 4, CLASSES, "ball"),
        # potentials of 8 states on a 100-point grid (the `potentials` tool)
        _case("potentials25", "potentials", "fp32sub", (25, 25, 25), 20, 4, 4, ""),
        # the `coulombo` tool's call: host coefficients in, integrals out
        _case("states16_host", "states", "fp32sub", (16, 16, 16), 20, 4, 4),
        # dense grids through the reference's calculator interface, FP64
        _case("grid16_fp64", "grid", "fp64", (16, 16, 16), 1, 1, 0, ""),
    ]


def draw(rng):
    entry = rng.choice(["request"] * 6 + ["batch", "compute", "states", "potentials", "grid"])
    mode = rng.choice(["fp32sub"] * 5 + ["fp64sub", "fp64sub", "fp64", "fp32"])
    orbitals = rng.choice([1, 5, 10, 10, 20, 20, 20])
    shape = rng.choice(["box", "box", "ball"])
    boxes = rng.randint(2, 6) if entry == "batch" else 1
    allpairs = entry in ("request", "compute") and rng.random() < 0.2
    while True:
        top = 64 if entry in ("request", "compute") else 26
        side = math.exp(rng.uniform(math.log(6), math.log(top)))
        cells = tuple(max(4, min(64, round(side * math.exp(rng.uniform(-0.25, 0.25))))) for _ in range(3))
        if rng.random() < 0.3:
            cells = (cells[0],) * 3
        if allpairs:
            n = rng.randint(6, 40 if entry == "request" else 12)
            electrons, holes, integrals = n, 0, "ijkl"
        elif rng.random() < 0.25:
            electrons, holes, integrals = rng.randint(1, 8), 0, "eeee"
        else:
            electrons, holes, integrals = rng.randint(1, 6), rng.randint(1, 6), CLASSES
        n = electrons + holes
        atoms = 8 * cells[0] * cells[1] * cells[2] * (1 if boxes == 1 else 2 * boxes)
        dims = _dims(cells)
        work = n * (n + 1) // 2 * atoms
        slow = mode in ("fp64", "fp32") or any(d % 4 for d in dims)
        if work <= (4e6 if mode == "fp64" else 8e6 if slow else 16e6 if mode == "fp64sub" else 60e6) and n * atoms * orbitals * 16 <= (
                3e8 if entry == "states" else 3e9):
            break
    integrals = "" if entry in ("potentials", "grid") else integrals
    c = _case("", entry, mode, cells, orbitals, electrons, holes, integrals, shape, rng.choice([0.0, 0.0, 5.0]), boxes)
    del c["name"]
    return c


# ---------------------------------------------------------------------------------------------
# structures and states
# ---------------------------------------------------------------------------------------------
def _dims(cells):
    return tuple(cl.round_up_235(4 * c) for c in cells)


def _boxes(case):
    """(cells, index) of each structure: later boxes of a batch grow by two cells along z, then y, then x."""
    out = []
    for b in range(case["boxes"]):
        grow = [case["lx"], case["ly"], case["lz"]]
        for k in range(2 * b):
            grow[2 - k % 3] += 2
        out.append((tuple(grow), b))
    return out


def _sites(cells, shape):
    """Grid cells of the atoms (ascending) on the padded grid, and their integer positions."""
    dims = _dims(cells)
    occ = np.zeros(dims[::-1], dtype=bool)
    for x, y, z in BASIS:
        occ[z:4 * cells[2]:4, y:4 * cells[1]:4, x:4 * cells[0]:4] = True
    if shape == "ball":
        r = [((np.arange(dims[d]) - 2 * cells[d] + 1.5) / (2.0 * cells[d])) ** 2 for d in range(3)]
        occ &= (r[2][:, None, None] + r[1][None, :, None] + r[0][None, None, :]) <= 1.0
    idx = np.flatnonzero(occ).astype(np.int64)
    return idx, dims


def _states(case, cells, idx, dims, seed):
    """[states][atoms][orbitals] complex128 on the GPU, holes first, each normalised."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    i = torch.from_numpy(idx).cuda()
    pos = torch.stack([i % dims[0], (i // dims[0]) % dims[1], i // (dims[0] * dims[1])]).double()
    d = (pos - pos.mean(dim=1, keepdim=True)) / torch.tensor([[2.0 * c] for c in cells], dtype=torch.float64, device="cuda")
    n, orb = case["electrons"] + case["holes"], case["orbitals"]
    r2 = (d * d).sum(0)
    shapes = [torch.ones_like(r2), d[0], d[1], d[2], d[0] * d[1], d[0] ** 2 - d[1] ** 2]
    out = torch.empty((n, idx.size, orb), dtype=torch.complex128, device="cuda")
    for s in range(n):
        sigma = 0.3 + 0.04 * (s % 5)
        env = torch.exp(-r2 / (2 * sigma * sigma)) * shapes[s % len(shapes)]
        re_im = torch.view_as_real(out[s])
        re_im.normal_(generator=g)
        re_im *= env[:, None, None]
        out[s] /= torch.linalg.vector_norm(out[s])
    return out


def _specs(case):
    n, holes = case["electrons"] + case["holes"], case["holes"]
    return np.ascontiguousarray(cl.enumerate_integrals(case["integrals"], n, holes))


def _calculator(case, dims):
    calc = cl.CoulombCalculator(dims, (A_ZB / 4,) * 3, MODES[case["mode"]])
    calc.initialize(dielectric=DIELECTRIC, onsite=case["onsite"])
    return calc


def _density(case, cells, idx, dims, seed):
    """A pair density on the dense grid [z, y, x] (the calculator interface's input)."""
    s = _states({**case, "electrons": 2, "holes": 0}, cells, idx, dims, seed)
    rho = torch.zeros(dims[2] * dims[1] * dims[0], dtype=torch.complex128, device="cuda")
    rho[torch.from_numpy(idx).cuda()] = (s[0].conj() * s[1]).sum(1)
    return rho.view(dims[2], dims[1], dims[0])


def prepare(case, seed):
    state = {"entry": case["entry"], "single": case["mode"] in ("fp32", "fp32sub"), "runs": []}
    for cells, b in _boxes(case):
        idx, dims = _sites(cells, case["shape"])
        calc = _calculator(case, dims)
        if case["entry"] == "grid":
            state["left"] = _density(case, cells, idx, dims, 2 * seed).cpu().numpy()
            state["right"] = _density(case, cells, idx, dims, 2 * seed + 1).cpu().numpy()
            state["runs"].append(calc)
            continue
        states = _states(case, cells, idx, dims, 16 * seed + b).cpu().numpy()
        if case["entry"] == "states":
            state["call"] = (states, idx, case["holes"], _specs(case))
            state["runs"].append(calc)
            continue
        calc.set_states(states, idx, case["holes"])
        if case["entry"] in ("request", "batch"):
            state["runs"].append(calc.request(_specs(case)))
        else:
            state["specs"] = _specs(case) if case["integrals"] else None
            state["runs"].append(calc)
    if case["entry"] == "batch":
        state["batch"] = cl.Batch(state["runs"])
    return state


def run(state):
    entry, first = state["entry"], state["runs"][0]
    if entry == "request":
        out = [first.run()]
    elif entry == "batch":
        out = state["batch"].run()
    elif entry == "compute":
        out = [first.compute(state["specs"])]
    elif entry == "states":
        out = [first.compute_states(*state["call"])]
    elif entry == "potentials":
        v = first.potentials()
        return v.astype(np.float32) if state["single"] else v
    else:
        first.prepare(state["left"])
        value = np.array([first.calculate(state["right"])])
        out = [value, first.potential()]
    return [v.astype(np.complex64) for v in out] if state["single"] else out


# ---------------------------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------------------------
def work(case):
    n = case["electrons"] + case["holes"]
    if case["entry"] == "grid":
        dims = _dims((case["lx"], case["ly"], case["lz"]))
        points = float(dims[0] * dims[1] * dims[2])
        return {"bytes": 3 * 16.0 * points, "flops": 2 * 5 * 8 * points * math.log2(8 * points) + 8 * points}
    moved = flops = 0.0
    for cells, _ in _boxes(case):
        atoms = float(_sites(cells, case["shape"])[0].size)
        dims = _dims(cells)
        moved += 16.0 * n * atoms * case["orbitals"]
        if case["entry"] == "potentials":
            pairs, grams, results = n, 0, 8.0 * n * atoms
        else:
            specs = _specs(case).astype(np.int64)
            hi = np.maximum(specs[:, [0, 1]], specs[:, [3, 2]])
            lo = np.minimum(specs[:, [0, 1]], specs[:, [3, 2]])
            prod = hi * (hi - 1) // 2 + lo
            pairs = np.unique(prod).size
            grams = np.unique(np.sort(prod, axis=1), axis=0).shape[0]
            results = 16.0 * len(specs)
        moved += results
        # a zero-padded transform each way (as many points as the grid has) of every pair density
        points = float(dims[0] * dims[1] * dims[2])
        flops += pairs * (8.0 * atoms * case["orbitals"] + 2 * 5 * points * math.log2(points)) + 8.0 * grams * atoms
    return {"bytes": moved, "flops": flops}


# ---------------------------------------------------------------------------------------------
# the same in plain 64-bit torch: zero-padded FFT convolution with the Coulomb kernel
# ---------------------------------------------------------------------------------------------
def _kernel(dims, onsite):
    """Spectrum of G(|r|) on the doubled grid (even extension, [z, y, x])."""
    ax = []
    for d in (2, 1, 0):
        k = torch.arange(2 * dims[d], device="cuda", dtype=torch.float64)
        ax.append((torch.minimum(k, 2 * dims[d] - k) * (A_ZB / 4)) ** 2)
    g = (ax[0][:, None, None] + ax[1][None, :, None] + ax[2][None, None, :]).sqrt_()
    g[0, 0, 0] = 1.0
    g = (E2_4PE0 / DIELECTRIC) / g
    g[0, 0, 0] = onsite
    return torch.fft.fftn(g.to(torch.complex128)).real.contiguous()


def _convolve(rho, spectrum, dims):
    pad = torch.fft.fftn(rho, s=(2 * dims[2], 2 * dims[1], 2 * dims[0]))
    pad *= spectrum
    return torch.fft.ifftn(pad)[:dims[2], :dims[1], :dims[0]]


def exact(case, seed):
    out = []
    for cells, b in _boxes(case):
        idx, dims = _sites(cells, case["shape"])
        spectrum = _kernel(dims, case["onsite"])
        if case["entry"] == "grid":
            v = _convolve(_density(case, cells, idx, dims, 2 * seed), spectrum, dims)
            value = (v * _density(case, cells, idx, dims, 2 * seed + 1)).sum().reshape(1)
            return [value.cpu(), v.contiguous().cpu()]
        c = _states(case, cells, idx, dims, 16 * seed + b)
        n, at = c.shape[0], torch.from_numpy(idx).cuda()
        only_diagonal = case["entry"] == "potentials"
        pairs = [(i, i) for i in range(n)] if only_diagonal else [(i, j) for i in range(n) for j in range(i + 1)]
        rho = torch.empty((len(pairs), idx.size), dtype=torch.complex128, device="cuda")
        v = torch.empty_like(rho)
        grid = torch.zeros(dims[0] * dims[1] * dims[2], dtype=torch.complex128, device="cuda")
        for p, (i, j) in enumerate(pairs):
            rho[p] = (c[i].conj() * c[j]).sum(1)
            grid[at] = rho[p]
            v[p] = _convolve(grid.view(dims[2], dims[1], dims[0]), spectrum, dims).reshape(-1)[at]
        del c, grid, spectrum
        if only_diagonal:
            return v.real.contiguous().cpu()
        # (l|r) = sum V_l rho_r; products named the other way round are conjugated
        plain, mixed = v @ rho.T, v @ rho.conj().T
        s = torch.from_numpy(_specs(case).astype(np.int64)).cuda() - 1

        def product(a, b2):
            hi, lo = torch.maximum(a, b2), torch.minimum(a, b2)
            return hi * (hi + 1) // 2 + lo, a < b2

        l, lc = product(s[:, 0], s[:, 3])
        r, rc = product(s[:, 1], s[:, 2])
        val = torch.where(lc == rc, plain[l, r], mixed[l, r])
        out.append(torch.where(lc, val.conj(), val).cpu())
    return out
