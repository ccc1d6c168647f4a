"""Performance cases of the H.psi / eigensolver path, through the mirror API.

Every case is one call (or the few calls that belong together) a user of
``qimpy_gb300.electrons`` / ``davidson`` makes on data resident on the GPU:

* ``hamiltonian``  ``Electrons.hamiltonian(C)``, the call the eigensolvers
  repeat; complex or real (Gamma-point) wavefunctions, FP64 (complex128) or the
  mixed form (complex64); returns H C and the projections <beta|C>;
* ``overlap``      ``Wavefunction.dot``, the subspace overlaps;
* ``rotate``       ``Wavefunction.matmul``, the band rotations;
* ``rayleigh``     both on the same bands, as one Rayleigh-Ritz update does;
* ``scf``          a few Davidson iterations from given bands and the density of
  the result, what one cycle of a self-consistent field loop asks for; returns
  the eigenvalues and the density (the bands' phases are arbitrary).

Cells are orthorhombic or face-centred cubic, with Gaussian-well potentials,
Gaussian-shell projectors and damped random start vectors of the workloads in
``qimpy_gb300.workloads``, generated on the device from the seed alone.
"""
from __future__ import annotations

import math

import torch

from qimpy_gb300 import davidson, electrons, workloads
from qimpy_gb300.sphere import factor_axis

DEV = "cuda"

#: Projector shells (l, sigma) per atom by name: 4, 9 and 18 projectors.
SHELLS = {
    "sp": [(0, 1.0), (1, 0.9)],
    "spd": [(0, 0.9), (1, 0.9), (2, 1.1)],
    "2spd": [(0, 0.9), (1, 0.9), (2, 0.9), (0, 1.4), (1, 1.4), (2, 1.4)],
}


def _case(name, kind, dtype, cell, sides, ecut, grid, nk, nb, atoms, shells, real=False, nb2=0, steps=0):
    c = {"kind": kind, "dtype": dtype, "real": real, "cell": cell, "a": sides[0], "b": sides[1], "c": sides[2],
         "ecut": ecut, "n0": grid[0], "n1": grid[1], "n2": grid[2], "nk": nk, "nb": nb, "nb2": nb2,
         "atoms": atoms, "shells": shells, "steps": steps}
    return dict(c, name=name) if name else c


def listed():
    si2 = ("fcc", (10.26,) * 3, 20.0, (36,) * 3)
    si64 = ("ortho", (20.52,) * 3, 20.0, (96,) * 3)
    cu32 = ("ortho", (13.64,) * 3, 30.0, (72,) * 3)
    return [
        # The smallest call: a molecule-sized cell on an odd, non-cubic grid.
        _case("h_fp64_tiny", "hamiltonian", "c128", "ortho", (5.0, 6.5, 8.0), 5.0, (15, 20, 25), 2, 6, 3, "sp"),
        # A primitive cell with a k-mesh: the smallest cell of ordinary use, in
        # the plain form and in the mixed form.
        _case("h_fp64_si2", "hamiltonian", "c128", *si2, 8, 18, 2, "sp"),
        _case("h_mixed_si2", "hamiltonian", "c64", *si2, 8, 18, 2, "sp"),
        # A 64-atom supercell at Gamma: one 32-band block in the plain form, all
        # bands in the mixed form.
        _case("h_fp64_si64", "hamiltonian", "c128", *si64, 1, 32, 64, "sp"),
        _case("h_mixed_si64", "hamiltonian", "c64", *si64, 1, 160, 64, "sp"),
        # A transition metal: many projectors per atom, several k-points.
        _case("h_mixed_cu32", "hamiltonian", "c64", *cu32, 4, 200, 32, "2spd"),
        # Real wavefunctions at Gamma: an odd band count in a mid-size cell
        # (FP64), and the 64-atom cell with its extra bands (mixed).
        _case("h_real_fp64", "hamiltonian", "c128", "ortho", (12.0, 14.0, 15.5), 20.0, (56, 60, 64), 1, 45, 20, "sp",
              real=True),
        _case("h_real_mixed_si64", "hamiltonian", "c64", *si64, 1, 176, 64, "sp", real=True),
        # Subspace products of a Davidson iteration: the overlap of the expanded
        # bands with the expansion and the rotation back, FP64 and mixed.
        _case("overlap_fp64_si64", "overlap", "c128", *si64, 1, 352, 0, "sp", nb2=176),
        _case("rotate_fp64_si64", "rotate", "c128", *si64, 1, 352, 0, "sp", nb2=176),
        _case("rayleigh_mixed_cu32", "rayleigh", "c64", *cu32, 4, 400, 0, "sp", nb2=200),
        # One cycle of a self-consistent field loop on the primitive cell.
        _case("scf_fp64_si2", "scf", "c128", *si2, 8, 18, 2, "sp", steps=5),
    ]


def _n_estimate(case) -> float:
    vol = case["a"] * case["b"] * case["c"] / (4.0 if case["cell"] == "fcc" else 1.0)
    n = vol * (2.0 * case["ecut"]) ** 1.5 / (6.0 * math.pi**2)
    return n / 2.0 if case["real"] else n


def work(case):
    """Compulsory bytes and operations of one pass."""
    z = 16 if case["dtype"] == "c128" else 8
    n, nk, nb, nb2 = _n_estimate(case), case["nk"], case["nb"], case["nb2"]
    P = case["atoms"] * sum(2 * l + 1 for l, _ in SHELLS[case["shells"]])
    N = case["n0"] * case["n1"] * case["n2"]
    fft = 10.0 * N * math.log2(N) * (0.5 if case["real"] else 1.0)
    if case["kind"] == "hamiltonian":
        cplx = 8.0 if not case["real"] else 4.0
        return {"bytes": nk * n * z * (2 * nb + P) + N * z / 2 + nk * nb * P * z,
                "flops": nk * nb * (fft + 2 * cplx * P * n)}
    if case["kind"] == "overlap":
        return {"bytes": nk * (n * (nb + nb2) * z + nb * nb2 * 16), "flops": 8.0 * nk * nb * nb2 * n}
    if case["kind"] == "rotate":
        return {"bytes": nk * (n * (nb + nb2) * z + nb * nb2 * 16), "flops": 8.0 * nk * nb * nb2 * n}
    if case["kind"] == "rayleigh":
        return {"bytes": nk * (n * (nb + 2 * nb2) * z + 2 * nb * nb2 * 16), "flops": 16.0 * nk * nb * nb2 * n}
    # scf: per iteration H of the expansion, two overlaps and three rotations.
    per = nb * (fft + 16.0 * P * n) + 8.0 * n * nb * (2 * 2 * nb + 4 * nb)
    return {"bytes": case["steps"] * nk * n * z * 10 * nb + 8.0 * N,
            "flops": case["steps"] * nk * per + nk * nb * fft / 2}


# ---------------------------------------------------------------------------
# Drawn cases
# ---------------------------------------------------------------------------


def _grid_size(side: float, ecut: float, cubic_rule: bool) -> int:
    """Smallest FFT size that holds the density's sphere (twice the
    wavefunctions') along an axis; multiples of 4 where `cubic_rule`."""
    n = side * 2.0 * math.sqrt(2.0 * ecut) / math.pi
    n = int(4 * math.ceil(n / 4.0)) if cubic_rule else int(math.ceil(n))
    while True:
        try:
            factor_axis(n)
            return n
        except ValueError:
            n += 4 if cubic_rule else 1


def _log_int(rng, lo, hi) -> int:
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _seconds(c) -> float:
    """Rough cost of a case, to keep drawn ones within the largest listed."""
    w = work(c)
    return w["flops"] / (0.9e12 if c["dtype"] == "c128" else 2e13)


def draw(rng):
    while True:
        kind = rng.choice(["hamiltonian"] * 6 + ["overlap", "rotate", "rayleigh", "scf"])
        dtype = "c64" if kind == "rayleigh" else "c128" if kind in ("overlap", "rotate", "scf") \
            else rng.choice(["c128", "c64"])
        real = kind == "hamiltonian" and rng.random() < 0.3
        ecut = round(rng.uniform(6.0, 30.0), 3)
        cell = rng.choice(["fcc", "ortho"])
        if cell == "fcc":
            a = math.exp(rng.uniform(math.log(7.0), math.log(14.0)))
            sides = (round(a, 3),) * 3
            grid = (_grid_size(a / math.sqrt(2.0), ecut, False),) * 3
        else:
            a = math.exp(rng.uniform(math.log(5.0), math.log(20.0)))
            sides = tuple(round(a * rng.uniform(0.8, 1.2), 3) for _ in range(3))
            even = rng.random() < 0.5
            grid = tuple(_grid_size(s, ecut, even) for s in sides)
        if not 12 <= min(grid) <= max(grid) <= 108:
            continue
        nk = 1 if real else _log_int(rng, 1, 8)
        atoms = _log_int(rng, 1, 64) if kind in ("hamiltonian", "scf") else 0
        shells = rng.choice(["sp", "spd", "2spd"])
        if kind == "scf":
            atoms, steps, nb = min(atoms, 8), 5, _log_int(rng, 6, 40)
            nb2 = 0
        elif kind == "hamiltonian":
            nb, nb2, steps = _log_int(rng, 3, 200), 0, 0
        else:
            nb2, steps = _log_int(rng, 5, 200), 0
            nb = rng.choice([nb2, 2 * nb2, nb2 + rng.randint(1, nb2)])
        c = _case(None, kind, dtype, cell, sides, ecut, grid, nk, nb, atoms, shells, real, nb2, steps)
        n = _n_estimate(c) / (2.0 if real else 1.0)
        if n < 60 or 2.5 * max(nb, nb2) >= n or (kind == "scf" and (n > 4000 or 5 * nb >= n)):
            continue
        if _seconds(c) > 0.015 or nk * nb * _n_estimate(c) > 2e7:
            continue
        return c


# ---------------------------------------------------------------------------
# Inputs
# ---------------------------------------------------------------------------


def _cell(case):
    a, b, c = case["a"], case["b"], case["c"]
    if case["cell"] == "fcc":
        R = torch.tensor([[0, a / 2, a / 2], [a / 2, 0, a / 2], [a / 2, a / 2, 0]], dtype=torch.float64).T
    else:
        R = torch.diag(torch.tensor([a, b, c], dtype=torch.float64))
    G = 2.0 * math.pi * torch.linalg.inv(R.T)
    nk = case["nk"]
    if nk == 1:
        k = torch.zeros((1, 3), dtype=torch.float64)
    else:  # a fixed low-discrepancy set of general k-points
        i = torch.arange(1, nk + 1, dtype=torch.float64)[:, None]
        k = i * torch.tensor([0.8191725133961645, 0.6710436067037893, 0.5497004779019703], dtype=torch.float64)
        k = k - torch.floor(k) - 0.5
    return R, G, k


def _basis(case):
    """The plane waves below the cutoff per k, ascending in the grid's linear
    index, padded to a common length: (linear index, iG, inside, KE)."""
    R, G, k = _cell(case)
    shape = (case["n0"], case["n1"], case["n2"])
    ax = [torch.arange(s, device=DEV) for s in shape]
    ax = [torch.where(x <= s // 2, x, x - s) for x, s in zip(ax, shape)]
    if case["real"]:
        ax[2] = ax[2][: shape[2] // 2 + 1]
    iG = torch.stack(torch.meshgrid(*ax, indexing="ij"), dim=-1).reshape(-1, 3)
    Gd, kd = G.to(DEV), k.to(DEV)
    inside = [0.5 * ((iG.to(torch.float64) + q) @ Gd.T).square().sum(dim=1) < case["ecut"] for q in kd]
    n_tot = max(int(w.sum()) for w in inside)
    index = torch.zeros((len(inside), n_tot), dtype=torch.int64, device=DEV)
    mask = torch.zeros((len(inside), n_tot), dtype=torch.bool, device=DEV)
    for i, w in enumerate(inside):
        j = torch.nonzero(w).flatten()
        index[i, : j.numel()], mask[i, : j.numel()] = j, True
    kiG = iG[index].to(torch.float64) + kd[:, None, :]
    q = kiG @ Gd.T
    return {"shape": shape, "index": index, "iG": iG[index], "mask": mask, "kiG": kiG, "q": q,
            "ke": 0.5 * q.square().sum(dim=-1), "volume": abs(float(torch.linalg.det(R)))}


def _solid(l, q):
    x, y, z = q.unbind(-1)
    if l == 0:
        return [torch.full_like(x, 0.5 / math.sqrt(math.pi))]
    if l == 1:
        return [math.sqrt(0.75 / math.pi) * t for t in (y, z, x)]
    s, r2 = math.sqrt(15.0 / (4.0 * math.pi)), x * x + y * y + z * z
    return [s * x * y, s * y * z, math.sqrt(5.0 / (16.0 * math.pi)) * (3.0 * z * z - r2), s * x * z,
            0.5 * s * (x * x - y * y)]


def _symmetrize(case, b, X):
    """c(-G) = conj(c(G)) on the Gz = 0 plane of half-basis bands."""
    z0 = torch.nonzero((b["iG"][0, :, 2] == 0) & b["mask"][0]).flatten()
    N0, N1, _ = b["shape"]
    g = b["iG"][0, z0]
    key = (g[:, 0] % N0) * N1 + g[:, 1] % N1
    neg = (-g[:, 0] % N0) * N1 + (-g[:, 1]) % N1
    order = torch.argsort(key)
    partner = z0[order[torch.searchsorted(key[order], neg)]]
    X[..., z0] = 0.5 * (X[..., z0] + X[..., partner].conj())
    return X


def _inputs(case, seed, b):
    """V(r), beta, D and the bands of a case: a function of case and seed."""
    g = torch.Generator(device=DEV).manual_seed(int(seed) * 7919 + 13)
    dt = torch.complex128 if case["dtype"] == "c128" else torch.complex64
    f64 = torch.float64

    def normal(*shape):
        return torch.complex(torch.randn(shape, generator=g, device=DEV, dtype=f64),
                             torch.randn(shape, generator=g, device=DEV, dtype=f64))

    def bands(count):
        X = torch.empty((b["index"].shape[0], count, b["index"].shape[1]), dtype=dt, device=DEV)
        scale = b["mask"] / (1.0 + b["ke"])
        for lo in range(0, count, 64):
            X[:, lo:lo + 64] = normal(X.shape[0], min(64, count - lo), X.shape[2]) * scale[:, None]
        return _symmetrize(case, b, X) if case["real"] else X

    out = {"C": bands(case["nb"])}
    if case["kind"] in ("overlap", "rayleigh"):
        out["X"] = bands(case["nb2"])
    if case["kind"] in ("rotate", "rayleigh"):
        out["M"] = normal(b["index"].shape[0], case["nb"], case["nb2"]) / math.sqrt(2.0 * case["nb"])
    if case["kind"] not in ("hamiltonian", "scf"):
        return out
    # Gaussian wells (depth 2 Ha, width 1.2 bohr) at random atoms, plus smooth
    # modes of rms 0.3 Ha.
    R, Gb, _ = _cell(case)
    R, shape = R.to(DEV), b["shape"]
    pos = torch.rand((case["atoms"], 3), generator=g, device=DEV, dtype=f64)
    frac = torch.stack(torch.meshgrid(*[torch.arange(s, device=DEV, dtype=f64) / s for s in shape], indexing="ij"), -1)
    V = torch.zeros(shape, dtype=f64, device=DEV)
    for tau in pos:
        d = frac - tau
        r = (d - torch.round(d)) @ R.T
        V -= 2.0 * torch.exp(-r.square().sum(-1) / 2.88)
    G1 = [torch.fft.fftfreq(s, d=1.0 / s, device=DEV, dtype=f64) for s in shape]
    G2 = (torch.stack(torch.meshgrid(*G1, indexing="ij"), -1) @ Gb.to(DEV).T).square().sum(-1)
    modes = torch.fft.ifftn(normal(*shape) * torch.exp(-G2 / 8.0), norm="forward").real
    V += modes * (0.3 / modes.square().mean().sqrt())
    out["V"] = V if dt == torch.complex128 else V.to(torch.float32).to(f64)
    # Projectors of Gaussian shells on every atom; symmetric D blocks.
    shells = SHELLS[case["shells"]]
    pa = sum(2 * l + 1 for l, _ in shells)
    rows = []
    for l, sigma in shells:
        rad = (2.0 * math.pi) ** 1.5 * sigma ** (2 * l + 3) * torch.exp(-0.5 * sigma**2 * b["q"].square().sum(-1))
        rows += [(-1j) ** l * (rad * s) for s in _solid(l, b["q"])]
    ang = torch.stack([r.to(torch.complex128) for r in rows], dim=1)
    beta = torch.empty((ang.shape[0], case["atoms"] * pa, ang.shape[2]), dtype=dt, device=DEV)
    for i, tau in enumerate(pos):
        phase = torch.exp(-2j * math.pi * (b["kiG"] @ tau)) * (b["mask"] / math.sqrt(b["volume"]))
        beta[:, i * pa:(i + 1) * pa] = ang * phase[:, None]
    out["beta"] = beta
    D = torch.randn((case["atoms"], pa, pa), generator=g, device=DEV, dtype=f64)
    D = 0.5 * (D + D.transpose(1, 2))
    out["D"] = D.to(dt)
    return out


def prepare(case, seed):
    real = bool(case["real"])
    dt = torch.complex128 if case["dtype"] == "c128" else torch.complex64
    R, G, k = _cell(case)
    shape = (case["n0"], case["n1"], case["n2"])
    nk = case["nk"]
    layout = None if real else workloads.make_basis_device(G.numpy(), k.numpy(), case["ecut"], shape, DEV)
    basis = electrons.Basis(R.numpy(), k.numpy(), [1.0 / nk] * nk, case["ecut"], shape, DEV, dt, layout=layout,
                            real=real)
    d = _inputs(case, seed, _basis(case))
    state = {"kind": case["kind"], "basis": basis, "C": d["C"], "M": d.get("M"), "X": d.get("X")}
    if case["kind"] in ("hamiltonian", "scf"):
        extra = max(1, case["nb"] // 9)
        state["el"] = electrons.Electrons(basis, electrons.Ions(basis, d["beta"], d["D"]), d["V"],
                                          case["nb"] - extra, extra)
    if case["kind"] == "scf":
        state["steps"] = case["steps"]
        state["C"] = electrons.Wavefunction(basis, coeff=d["C"]).orthonormalize().coeff
        state["f"] = torch.ones((nk, case["nb"]), dtype=torch.float64, device=DEV)
    return state


def run(state):
    basis, kind = state["basis"], state["kind"]
    C = electrons.Wavefunction(basis, coeff=state["C"])
    if kind == "hamiltonian":
        el = state["el"]
        HC = el.hamiltonian(C)
        return [HC.coeff, C.projT(el.ions)]
    if kind == "overlap":
        return C.dot(electrons.Wavefunction(basis, coeff=state["X"])).wait()
    if kind == "rotate":
        return C.matmul(state["M"]).coeff
    if kind == "rayleigh":
        return [C.dot(electrons.Wavefunction(basis, coeff=state["X"])).wait(), C.matmul(state["M"]).coeff]
    el = state["el"]
    el.C = C
    davidson.Davidson(el, n_iterations=state["steps"], eig_threshold=1e-10)()
    return [el.eig, basis.collect_density(el.C, state["f"])]


# ---------------------------------------------------------------------------
# The same in 64 bits, by plain torch
# ---------------------------------------------------------------------------


def exact(case, seed):
    if case["kind"] == "scf":
        return None  # an unfinished iteration has no value of its own
    b = _basis(case)
    d = _inputs(case, seed, b)
    z = torch.complex128
    C = d["C"].to(z)
    if case["kind"] == "overlap":
        return C.conj() @ d["X"].to(z).transpose(1, 2)
    if case["kind"] == "rotate":
        return d["M"].transpose(1, 2) @ C
    if case["kind"] == "rayleigh":
        M = d["M"].to(torch.complex64).to(z)
        return [C.conj() @ d["X"].to(z).transpose(1, 2), M.transpose(1, 2) @ C]
    shape, V, beta, D = b["shape"], d["V"], d["beta"].to(z), d["D"].to(z)
    HC = b["ke"][:, None] * C
    half = (shape[0], shape[1], shape[2] // 2 + 1) if case["real"] else shape
    for ik in range(C.shape[0]):
        idx = b["index"][ik][b["mask"][ik]]
        for lo in range(0, C.shape[1], 16):
            x = C[ik, lo:lo + 16, : idx.numel()]
            grid = torch.zeros((x.shape[0], math.prod(half)), dtype=z, device=DEV)
            grid[:, idx] = x
            grid = grid.reshape(-1, *half)
            if case["real"]:
                psi = torch.fft.irfftn(grid, s=shape, dim=(1, 2, 3), norm="forward") * V
                grid = torch.fft.rfftn(psi, dim=(1, 2, 3), norm="forward")
            else:
                psi = torch.fft.ifftn(grid, dim=(1, 2, 3), norm="forward") * V
                grid = torch.fft.fftn(psi, dim=(1, 2, 3), norm="forward")
            HC[ik, lo:lo + 16, : idx.numel()] += grid.reshape(x.shape[0], -1)[:, idx]
    HC *= b["mask"][:, None]
    if case["real"]:
        w = torch.where(b["iG"][0, :, 2] == 0, 1.0, 2.0).to(torch.float64)
        proj = ((C * w) @ beta.conj().transpose(1, 2)).real.to(z)
    else:
        proj = C @ beta.conj().transpose(1, 2)
    Dp = torch.einsum("arc,kbac->kbar", D, proj.reshape(*proj.shape[:2], *D.shape[:2])).reshape(proj.shape)
    HC += Dp @ beta
    return [HC, proj]
