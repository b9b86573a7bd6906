"""Timed workloads of the library, from single operator applications to whole solves.

Every case goes through the Python binding's public calls, with device tensors
where the caller's data lives on the device and host arrays where the call
takes host arrays. Inputs are seeded; the cells are diamond / zincblende
supercells or random sites at silicon's volume per atom.
"""
import math
import pathlib
import sys

import numpy as np
import torch

sys.path.insert(0, str(pathlib.Path(__file__).resolve().parents[1] / "sparse-dft_b200"))

from sdft_b200 import density as dens  # noqa: E402
from sdft_b200 import synthetic  # noqa: E402
from sdft_b200.operator import Context, PlaneWaveOperator, rayleigh_ritz  # noqa: E402
from sdft_b200.serving import SolveServer  # noqa: E402

THIRD = 1.0 / 3.0
SI = 10.26    # bohr, cubic cell of diamond silicon
GAAS = 10.68  # bohr, cubic cell of zincblende GaAs
SMEARING_HA = 0.01
EXACT_NPW = 3600  # plane waves up to which the dense pencil is diagonalised for exact()


# --- The cases ---------------------------------------------------------------

def listed():
    return [
        # H~x and S~x of a handful of bands of a tiny cell: launch latency.
        _cell("pair_tiny_mixed", "pair", reps=1, a=7.0, ecut=4.0, columns=6, precision="mixed"),
        # The same call on the 64-atom silicon supercell's full block in the search precision:
        # what a Davidson iteration and a correction step spend most of their time in.
        _cell("pair_si64_mixed", "pair", reps=2, a=SI, ecut=15.0, columns=160, precision="mixed"),
        # An off-Gamma k-point of the 64-atom GaAs supercell in FP64 with a ragged block:
        # re-application and certification of a block, and the plain FP64 form.
        _cell("pair_gaas64_fp64", "pair", reps=2, a=GAAS, ecut=18.0, k=THIRD, columns=97, precision="fp64"),
        # A whole cold FP64 solve of a small cell at a k-point, and its density.
        _cell("solve_gaas8_fp64", "solve", reps=1, a=GAAS, ecut=6.0, k=THIRD, bands=20, precision="fp64"),
        # The headline solve: Si64, 160 bands, mixed search with the FP64 certificate, and its density.
        _cell("solve_si64_mixed", "solve", reps=2, a=SI, ecut=15.0, bands=160, precision="mixed"),
        # One SCF iteration: new V(G) and D on the resident operator, a warm-started solve,
        # one-centre occupations and the band density.
        _cell("scf_12atoms_mixed", "scf", atoms=12, ecut=12.0, bands=30, precision="mixed"),
        # Four k-points of a small cell submitted together to the solve server.
        _cell("serve_gaas8_4k", "serve", reps=1, a=GAAS, ecut=8.0, bands=20, kpoints=4, precision="mixed"),
        # Band density of the occupied bands of Si64 on the wavefunction support's double (f = 4).
        _cell("density_si64_f4", "density", reps=2, a=SI, ecut=15.0, factor=4.0, bands=128),
        # Hartree + PBE with a frozen core on Si64's density support.
        _cell("functional_si64_core", "functional", reps=2, a=SI, ecut=15.0, factor=4.0, core=True),
        # Collinear spin functional of the 8-atom cell.
        _cell("collinear_si8_core", "collinear", reps=1, a=SI, ecut=15.0, factor=4.0, core=True),
        # Compensation charge and its adjoint on Si64 with a fine support.
        _cell("compensation_si64_f8", "compensation", reps=2, a=SI, ecut=15.0, factor=8.0),
        # Rayleigh-Ritz of a Davidson pencil half way to its restart.
        {"name": "ritz_640", "kind": "ritz", "n": 640, "requested": 160},
    ]


def _cell(name, kind, *, reps=0, a=0.0, atoms=0, k=0.0, **more):
    case = {"name": name, "kind": kind, "reps": reps, "a": a, "atoms": atoms, "k": k}
    case.update(more)
    return case


def _log(rng, low, high):
    return math.exp(rng.uniform(math.log(low), math.log(high)))


def draw(rng):
    kind = rng.choice(("pair", "pair", "pair", "solve", "scf", "serve", "density", "functional", "collinear",
                       "compensation", "ritz"))
    if kind == "ritz":
        n = int(_log(rng, 24, 1280))
        return {"kind": kind, "n": n, "requested": max(1, int(n * rng.uniform(0.1, 0.5)))}
    most = {"pair": 64, "solve": 14, "scf": 14, "serve": 8, "density": 64, "functional": 48, "collinear": 16,
            "compensation": 64}[kind]
    atoms = int(round(_log(rng, 2, most)))
    k = rng.choice((0.0, round(rng.uniform(-0.5, 0.5), 3)))
    case = _cell("", kind, atoms=atoms, k=k, ecut=round(rng.uniform(8.0, 16.0), 2))
    del case["name"]
    if kind == "pair":
        case.update(columns=int(round(_log(rng, 1, 160))), precision=rng.choice(("mixed", "fp64")))
    elif kind in ("solve", "scf", "serve"):
        case.update(bands=max(8, round(2.5 * atoms)), precision=rng.choice(("mixed", "fp64")))
        if kind == "serve":
            case.update(kpoints=rng.randint(2, 6), k=0.0)
    elif kind == "density":
        case.update(factor=rng.choice((4.0, 4.0, 8.0)), bands=int(round(_log(rng, 2, 2 * atoms + 2))))
    else:
        case.update(factor=rng.choice((2.0, 4.0)), k=0.0)
        if kind != "compensation":
            case["core"] = rng.random() < 0.5
    return case


# --- Inputs ------------------------------------------------------------------

_context = None


def _ctx():
    """The program's context, on torch's stream."""
    global _context
    if _context is None:
        _context = Context(0, stream=torch.cuda.current_stream().cuda_stream)
    return _context


def _rng(seed, salt=0):
    return np.random.Generator(np.random.PCG64([seed, salt]))


def _geometry(case, seed):
    """Cubic lattice constant, fractional positions and species of the case's cell."""
    if case["reps"]:
        positions, species = synthetic.zincblende_sites(case["reps"])
        return case["a"] * case["reps"], positions, species
    rng = _rng(seed, 1)
    count = case["atoms"]
    a = (count * synthetic.SI_VOLUME_PER_ATOM) ** (1.0 / 3.0)
    return a, rng.uniform(0.0, 1.0, size=(count, 3)), rng.integers(0, 2, size=count)


def _operator_inputs(case, seed, kpoint=None, potential=None):
    a, positions, species = _geometry(case, seed)
    k = case["k"]
    return synthetic.build_operator("case", a, 1, case["ecut"], case.get("bands", 1), depths=(-2.2, -1.8),
                                    kpoint=(k, k / 2, -k) if kpoint is None else kpoint, seed=seed,
                                    sites=(positions, species), potential=potential, q_scaling="linear")


def _kpoints(case, seed):
    rng = _rng(seed, 2)
    return [(0.0, 0.0, 0.0)] + [tuple(float(v) for v in rng.uniform(-0.5, 0.5, size=3))
                                for _ in range(case["kpoints"] - 1)]


def _serve_inputs(case, seed):
    out = []
    for k in _kpoints(case, seed):
        out.append(_operator_inputs(case, seed, k, (out[0].v_hkl, out[0].v_values) if out else None))
    return out


def _block(npw, columns, seed):
    """A column-major block of unit Gaussian coefficients, the layout of a Davidson basis block."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    x = torch.randn((columns, npw, 2), dtype=torch.float64, device="cuda", generator=g)
    return torch.view_as_complex(x).T


def _support(a, ecut):
    hkl, _, _ = synthetic.enumerate_g_vectors(np.eye(3) * (2 * math.pi / a), ecut * synthetic.HARTREE_TO_EV)
    return np.ascontiguousarray(hkl, dtype=np.int32)


def _gaussians(a, positions, keys, charge, width):
    """n_G of one normalised Gaussian charge per site."""
    q = torch.tensor(keys, dtype=torch.float64, device="cuda") * (2 * math.pi / a)
    tau = torch.tensor(positions * a, dtype=torch.float64, device="cuda")
    total = torch.zeros(q.shape[0], dtype=torch.complex128, device="cuda")
    scale = torch.tensor(charge, dtype=torch.float64, device="cuda")
    for site in range(tau.shape[0]):
        total += scale[site] * torch.polar(torch.ones_like(q[:, 0]), -(q @ tau[site]))
    return (total * torch.exp(-0.25 * width * width * (q * q).sum(dim=1)) / a ** 3).cpu().numpy()


def _functional_inputs(case, seed):
    """Lattice, one or two channels of (keys, values) and the frozen core of a valence-like density:
    smooth Gaussians on every site over a uniform background, positive everywhere."""
    a, positions, _ = _geometry(case, seed)
    rng = _rng(seed, 3)
    cut = case["ecut"] * case["factor"]
    keys = _support(a, cut)
    sites = positions.shape[0]
    zero = np.nonzero(~keys.any(axis=1))[0]
    channels = []
    for charge, width in (((4.0, 1.9),) if case["kind"] == "functional" else ((2.4, 1.9), (1.7, 2.1))):
        values = _gaussians(a, positions, keys, charge * rng.uniform(0.8, 1.2, size=sites), width)
        values[zero] += 0.004
        channels.append((keys, values))
    core = (None, None)
    if case["core"]:
        core_keys = _support(a, 0.5 * cut)
        core = (core_keys, _gaussians(a, positions, core_keys, rng.uniform(0.8, 1.2, size=sites), 1.1))
    return np.eye(3) * a, channels, core


def _compensation_inputs(case, seed):
    a, positions, _ = _geometry(case, seed)
    aug = synthetic.augmentation()
    transform = synthetic.lm_transform(aug)
    keys = _support(a, case["ecut"] * case["factor"])
    g = torch.Generator(device="cuda").manual_seed(seed)
    dim = int(round(math.sqrt(transform.shape[1])))
    rho = torch.view_as_complex(torch.randn((positions.shape[0], dim, dim, 2), dtype=torch.float64, device="cuda",
                                            generator=g))
    rho = 0.5 * (rho + rho.conj().transpose(1, 2))
    v = torch.view_as_complex(torch.randn((keys.shape[0], 2), dtype=torch.float64, device="cuda", generator=g))
    q2 = torch.tensor((keys.astype(np.float64) ** 2).sum(axis=1) * (2 * math.pi / a) ** 2, device="cuda")
    return np.eye(3) * a, positions, keys, aug, transform, rho.resolve_conj().contiguous(), v / (1.0 + q2)


def _ritz_inputs(case, seed):
    """Projected pencil of a Davidson basis: a spectrum up to the kinetic cutoff, S the identity up to
    the basis's orthonormality."""
    n = case["n"]
    g = torch.Generator(device="cuda").manual_seed(seed)

    def square():
        return torch.view_as_complex(torch.randn((n, n, 2), dtype=torch.float64, device="cuda", generator=g))

    q, _ = torch.linalg.qr(square())
    spectrum = torch.rand(n, dtype=torch.float64, device="cuda", generator=g) ** 1.5 * 20.0 - 0.6
    h = (q * spectrum) @ q.mH
    e = square() * 1e-10
    s = torch.eye(n, dtype=torch.complex128, device="cuda") + e + e.mH
    return [np.asfortranarray((0.5 * (m + m.mH)).cpu().numpy()) for m in (h, s)]


def _scf_step(inputs, seed):
    """V(G) and D of the next SCF iteration."""
    rng = _rng(seed, 4)
    e = rng.standard_normal(inputs.d.shape) + 1j * rng.standard_normal(inputs.d.shape)
    return inputs.v_values * 1.01, inputs.d + 0.002 * (e + np.conj(np.transpose(e, (0, 2, 1))))


def _density_case(case, seed):
    a, _, _ = _geometry(case, seed)
    k = case["k"]
    shift = np.array([k, k / 2, -k])
    hkl, _, kinetic = synthetic.enumerate_g_vectors(np.eye(3) * (2 * math.pi / a),
                                                    case["ecut"] * synthetic.HARTREE_TO_EV, shift)
    decay = torch.tensor(np.exp(-0.5 * kinetic / synthetic.HARTREE_TO_EV), device="cuda")
    psi = _block(hkl.shape[0], case["bands"], seed).T * decay
    psi = psi / torch.linalg.vector_norm(psi, dim=1, keepdim=True)
    occupations = np.sort(_rng(seed, 5).uniform(1.0, 2.0, size=case["bands"]))[::-1].copy()
    return hkl, psi.contiguous(), occupations, a ** 3, _support(a, case["factor"] * case["ecut"])


# --- One pass ----------------------------------------------------------------

def prepare(case, seed):
    kind = case["kind"]
    state = {"kind": kind, "case": case, "context": _ctx()}
    if kind in ("pair", "solve", "scf"):
        inputs = _operator_inputs(case, seed)
        state["op"] = PlaneWaveOperator(_ctx(), inputs)
        if kind == "pair":
            state["x"] = _block(inputs.npw, case["columns"], seed)
            return state
        state["inputs"] = inputs
        state["support"] = _support(float(inputs.lattice[0, 0]), 4.0 * case["ecut"])
        if kind == "scf":
            state["warm"] = state["op"].davidson(case["bands"], 256, 1e-10, precision=case["precision"])["eigenvectors"]
            state["v"], state["d"] = _scf_step(inputs, seed)
    elif kind == "serve":
        state["inputs"] = _serve_inputs(case, seed)
        state["server"] = SolveServer(0, 40e9, 4)
    elif kind == "density":
        state["args"] = _density_case(case, seed)
    elif kind in ("functional", "collinear"):
        state["args"] = _functional_inputs(case, seed)
    elif kind == "compensation":
        lattice, positions, keys, aug, transform, rho, v = _compensation_inputs(case, seed)
        state["charge"] = dens.CompensationCharge(_ctx(), lattice, positions, keys, aug, transform)
        state["rho"], state["v"] = rho, v
    else:
        state["h"], state["s"] = _ritz_inputs(case, seed)
    return state


def _occupations(eigenvalues, electrons):
    """Fermi-Dirac occupations in [0, 2] that hold the electron count."""
    low, high = eigenvalues[0] - 1.0, eigenvalues[-1] + 1.0
    for _ in range(80):
        mu = 0.5 * (low + high)
        f = 2.0 / (1.0 + np.exp(np.clip((eigenvalues - mu) / SMEARING_HA, -700.0, 700.0)))
        low, high = (mu, high) if f.sum() < electrons else (low, mu)
    return f


def _electrons(bands):
    return 2.0 * (bands - max(1, bands // 5))


def run(state):
    kind, case, ctx = state["kind"], state["case"], state["context"]
    if kind == "pair":
        h, s = state["op"].apply_pair(state["x"], precision=case["precision"])
        return {"h": h, "s": s}
    if kind in ("solve", "scf"):
        op, inputs = state["op"], state["inputs"]
        if kind == "scf":
            op.update(inputs.v_hkl, state["v"], state["d"], inputs.q)
        solved = op.davidson(case["bands"], 256, 1e-10 if kind == "scf" else 1e-12, precision=case["precision"],
                             initial=state.get("warm"))
        vectors = solved["eigenvectors"]
        f = _occupations(solved["eigenvalues"], _electrons(case["bands"]))
        out = {"eigenvalues": solved["eigenvalues"],
               "density": dens.band_density(ctx, inputs.hkl, vectors, f, inputs.volume, state["support"])}
        if kind == "scf":
            out["onsite"] = dens.onsite_density(ctx, op.project(vectors.T), 8, f)
        return out
    if kind == "serve":
        tickets = [state["server"].submit(x, precision=case["precision"]) for x in state["inputs"]]
        return [state["server"].wait(t)["eigenvalues"] for t in tickets]
    if kind == "density":
        return dens.band_density(ctx, *state["args"])
    if kind == "functional":
        lattice, channels, core = state["args"]
        return _fields(dens.density_functionals(ctx, lattice, *channels[0], *core))
    if kind == "collinear":
        lattice, channels, core = state["args"]
        got = dens.collinear_functionals(ctx, lattice, *channels[0], *channels[1], *core)
        return {name: _fields(got[name]) for name in ("up", "down")}
    if kind == "compensation":
        return {"density": state["charge"].density(state["rho"]), "projection": state["charge"].project(state["v"])}
    values, vectors = rayleigh_ritz(ctx, state["h"], state["s"], case["requested"])
    # A Ritz vector's phase is free: the caller's basis weights stand for it.
    return {"values": values, "weights": vectors.real ** 2 + vectors.imag ** 2}


def _fields(got):
    return {"potential": got["potential"], "xc_potential": got["xc_potential"], "hkl": got["hkl"],
            "energies": np.array([got["hartree_energy"], got["xc_energy"], got["vxc_density"],
                                  got["sampled_electrons"]]),
            "hartree_stress": got["hartree_stress"], "xc_stress": got["xc_stress"]}


# --- What a pass cannot do without -------------------------------------------

def _sizes(case):
    """Volume, atoms and plane waves (from the sphere's volume)."""
    atoms = 8 * case["reps"] ** 3 if case["reps"] else case["atoms"]
    volume = (case["a"] * case["reps"]) ** 3 if case["reps"] else atoms * synthetic.SI_VOLUME_PER_ATOM
    return volume, atoms, volume * (2.0 * case["ecut"]) ** 1.5 / (6.0 * math.pi ** 2)


def _pair_work(volume, atoms, npw, columns, ecut):
    """One joint application: x in, H~x and S~x out, B and V(r) once; the transforms of the sphere's
    doubled box, one projection and two back-projections."""
    grid = volume * (4.0 * math.sqrt(2.0 * ecut) / (2.0 * math.pi)) ** 3
    return (16.0 * npw * (3 * columns + 8 * atoms) + 8.0 * grid,
            columns * (10.0 * grid * math.log2(grid) + 24.0 * 8 * atoms * npw))


def work(case):
    kind = case["kind"]
    if kind == "ritz":
        n, m = case["n"], case["requested"]
        return {"bytes": 16.0 * (2 * n * n + n * m), "flops": 16.0 / 3.0 * n ** 3 + 8.0 * n * n * m}
    volume, atoms, npw = _sizes(case)
    if kind == "pair":
        b, f = _pair_work(volume, atoms, npw, case["columns"], case["ecut"])
        return {"bytes": b, "flops": f}
    if kind in ("solve", "scf", "serve"):
        # At least one application of the block for each decade of the residual, cold (12) or warm (6).
        times = 6 if kind == "scf" else 12
        b, f = _pair_work(volume, atoms, npw, case["bands"], case["ecut"])
        solves = case.get("kpoints", 1)
        return {"bytes": solves * times * b, "flops": solves * times * f}
    factor = case["factor"]
    keys = npw * factor ** 1.5
    box = volume * (2.0 * math.sqrt(2.0 * factor * case["ecut"]) / (2.0 * math.pi)) ** 3
    if kind == "density":
        return {"bytes": 16.0 * (npw * case["bands"] + keys) + 12.0 * (npw + keys),
                "flops": case["bands"] * (5.0 * box * math.log2(box) + 4.0 * box)}
    if kind in ("functional", "collinear"):
        channels = 1 if kind == "functional" else 2
        return {"bytes": keys * (12.0 + 16.0) * (1 + 2 * channels + (0.35 if case["core"] else 0.0)),
                "flops": channels * 8 * 8 * 2.5 * box * math.log2(8 * box) + 8 * box * 200.0}
    # Compensation: form factors and keys once for each direction; per key and atom a phase and nine terms.
    return {"bytes": 2 * keys * (9 * 8 + 12 + 16.0), "flops": 2 * keys * atoms * 60.0}


def tolerance(case):
    kind = case["kind"]
    if kind == "pair":
        # Mixed: FP32 transforms and BF16 split products, 1e-7 to 9e-7 off FP64; FP64: 1e-16 to 5e-16 off.
        return {"rel": 4e-6, "max": 2e-4} if case["precision"] == "mixed" else {"rel": 4e-15, "max": 1e-12}
    if kind == "scf":
        # Residuals of 1e-10 Ha over the gaps between bands: densities 2e-13 to 1e-12 off.
        return {"rel": 1e-9, "max": 1e-7}
    if kind in ("solve", "serve"):
        # Residuals of 1e-12 Ha over the gaps: densities up to 7e-15 off, and more where bands nearly meet.
        return {"rel": 1e-11, "max": 1e-9}
    if kind == "ritz":
        # Vector weights: FP64 rounding over the gaps of a random spectrum, 3e-13 at n = 640.
        return {"rel": 1e-10, "max": 1e-7}
    if kind in ("functional", "collinear"):
        return {"rel": 1e-13, "max": 1e-10}  # 6e-17 to 1.2e-15 off
    return {"rel": 1e-14, "max": 1e-12}  # densities and projections: 4e-16 to 2e-15 off


# --- The same results in plain FP64 torch ------------------------------------

def _gpu(v, dtype=None):
    t = torch.as_tensor(np.ascontiguousarray(v))
    return (t if dtype is None else t.to(dtype)).cuda()


def _wrapped(keys, shape):
    k = [np.mod(keys[:, i], shape[i]).astype(np.int64) for i in range(3)]
    return _gpu((k[0] * shape[1] + k[1]) * shape[2] + k[2])


class _Pencil:
    """H~ and S~ by direct FP64 transforms on an alias-free box."""

    def __init__(self, inputs, v=None, d=None):
        hkl = inputs.hkl
        width = hkl.max(axis=0) - hkl.min(axis=0)
        self.shape = tuple(int(2 * w + 1) for w in width)
        self.count = int(np.prod(self.shape))
        self.index = _wrapped(hkl, self.shape)
        keep = np.all(np.abs(inputs.v_hkl) <= width[None, :], axis=1)
        grid = torch.zeros(self.count, dtype=torch.complex128, device="cuda")
        grid[_wrapped(inputs.v_hkl[keep], self.shape)] = _gpu((inputs.v_values if v is None else v)[keep])
        self.v = torch.fft.ifftn(grid.view(self.shape)).real * self.count
        self.t = _gpu(inputs.kinetic_ev / inputs.hartree_to_ev)[:, None]
        self.b = _gpu(inputs.amplitudes)
        self.d, self.q = _gpu(inputs.d if d is None else d), _gpu(inputs.q)
        self.one = 1.0 + inputs.regularization

    def _blocks(self, blocks, p):
        atoms, n = blocks.shape[0], blocks.shape[1]
        return torch.bmm(blocks, p.view(atoms, n, -1)).reshape(p.shape)

    def apply(self, x):
        h = self.t * x
        for c in range(x.shape[1]):
            grid = torch.zeros(self.count, dtype=torch.complex128, device="cuda")
            grid[self.index] = x[:, c]
            grid = torch.fft.fftn(torch.fft.ifftn(grid.view(self.shape)) * self.v)
            h[:, c] += grid.view(-1)[self.index]
        p = (self.b @ x).contiguous()
        return h + self.b.mH @ self._blocks(self.d, p), self.one * x + self.b.mH @ self._blocks(self.q, p)

    def lowest(self, count):
        n = self.t.shape[0]
        h, s = self.apply(torch.eye(n, dtype=torch.complex128, device="cuda"))
        h, s = _solve_pencil(h, s)
        return h[:count], s[:, :count]


def _solve_pencil(h, s):
    """All solutions of h y = e s y (s positive definite)."""
    low = torch.linalg.cholesky(0.5 * (s + s.mH))
    w = torch.linalg.solve_triangular(low, 0.5 * (h + h.mH), upper=False)
    w = torch.linalg.solve_triangular(low, w.mH, upper=False)
    e, y = torch.linalg.eigh(0.5 * (w + w.mH))
    return e, torch.linalg.solve_triangular(low.mH, y, upper=True)


def _density_exact(hkl, psi, occupations, volume, support):
    span = np.maximum(hkl.max(axis=0), 0) - np.minimum(hkl.min(axis=0), 0)
    shape = tuple(int(max(3, 2 * max(a, b) + 1)) for a, b in zip(np.abs(support).max(axis=0), span))
    count = int(np.prod(shape))
    index, total = _wrapped(hkl, shape), torch.zeros(shape, dtype=torch.float64, device="cuda")
    for band in range(psi.shape[0]):
        grid = torch.zeros(count, dtype=torch.complex128, device="cuda")
        grid[index] = psi[band]
        grid = torch.fft.ifftn(grid.view(shape)) * count
        total += float(occupations[band]) / volume * (grid.real ** 2 + grid.imag ** 2)
    return (torch.fft.fftn(total.to(torch.complex128)) / count).reshape(-1)[_wrapped(support, shape)]


def _radial_weights(r):
    """Simpson panels from the outer end of a logarithmic mesh."""
    h, w, k = math.log(r[1] / r[0]), np.zeros(r.size), r.size
    while k >= 3:
        w[k - 1] += r[k - 1] * h / 3.0
        w[k - 2], w[k - 3] = 4.0 * r[k - 2] * h / 3.0, r[k - 3] * h / 3.0
        if k == 3:
            break
        k -= 2
    return w


def _spherical_bessel(x):
    """j_0, j_1, j_2: closed forms, the power series below 0.5."""
    small = x < 0.5
    y = torch.where(small, torch.ones_like(x), x)
    closed = [torch.sin(y) / y, torch.sin(y) / y ** 2 - torch.cos(y) / y,
              (3.0 / y ** 3 - 1.0 / y) * torch.sin(y) - 3.0 / y ** 2 * torch.cos(y)]
    out = []
    for l in range(3):
        term = torch.ones_like(x)
        for k in range(1, l + 1):
            term = term * x / (2.0 * k + 1.0)
        value = term
        for k in range(1, 16):
            term = -term * x * x / (2.0 * k * (2.0 * l + 2.0 * k + 1.0))
            value = value + term
        out.append(torch.where(small, value, closed[l]))
    return out


def _harmonics(q):
    """Real spherical harmonics up to l = 2 in (l, m) order; 0 for l > 0 at the origin."""
    r = torch.linalg.vector_norm(q, dim=1)
    n = q / torch.where(r < 1e-14, torch.ones_like(r), r)[:, None]
    x, y, z = n[:, 0], n[:, 1], n[:, 2]
    c0, c1, c2 = 0.5 / math.sqrt(math.pi), math.sqrt(0.75 / math.pi), 0.5 * math.sqrt(15.0 / math.pi)
    s5 = 0.25 * math.sqrt(5.0 / math.pi)
    out = [c0 * torch.ones_like(x), c1 * y, c1 * z, c1 * x, c2 * x * y, c2 * y * z,
           s5 * (3.0 * z * z - 1.0), c2 * x * z, 0.5 * c2 * (x * x - y * y)]
    return [v if i == 0 else torch.where(r < 1e-14, torch.zeros_like(v), v) for i, v in enumerate(out)]


def _compensation_exact(lattice, positions, keys, aug, transform, rho, v):
    a = float(lattice[0, 0])
    q = _gpu(keys, torch.float64) * (2.0 * math.pi / a)
    shell, inverse = np.unique((keys.astype(np.int64) ** 2).sum(axis=1), return_inverse=True)
    radius = _gpu(np.sqrt(shell.astype(np.float64)) * (2.0 * math.pi / a) * 1.8897261254578281)
    bessel = _spherical_bessel(radius[:, None] * _gpu(aug["radial_grid"])[None, :])
    weights = _gpu(_radial_weights(aug["radial_grid"]))
    integrals = [bessel[l] @ (weights * _gpu(aug["compensation_r2"][l])) for l in range(3)]
    integrals[0] = torch.where(radius < 1e-14, torch.ones_like(radius), integrals[0])
    where, harmonics, form = _gpu(inverse.reshape(-1)), _harmonics(q), []
    for l, turn in ((0, 1.0), (1, -1j), (2, -1.0)):
        for m in range(2 * l + 1):
            form.append(turn * 4.0 * math.pi * harmonics[l * l + m] * integrals[l][where])
    form = torch.stack([f.to(torch.complex128) for f in form])
    t = _gpu(transform)
    moments = rho.reshape(rho.shape[0], -1) @ t.T
    m = np.abs(keys).max(axis=0)
    opposite = np.full(tuple(2 * m + 1), -1, dtype=np.int64)
    opposite[tuple((keys + m).T)] = np.arange(keys.shape[0])
    partner = _gpu(opposite[tuple((m - keys).T)])
    mirrored = torch.where(partner < 0, torch.zeros_like(v), v[partner.clamp(min=0)])
    total, projected = torch.zeros_like(v), []
    frac, k = _gpu(positions), _gpu(keys, torch.float64)
    for atom in range(frac.shape[0]):
        turns = k @ frac[atom]
        phase = torch.polar(torch.ones_like(turns), -2.0 * math.pi * (turns - torch.round(turns)))
        total += phase * (moments[atom] @ form) / a ** 3
        projected.append(((form @ (mirrored * phase)) @ t).view(rho.shape[1:]))
    return {"density": total, "projection": torch.stack(projected)}


def _pw92(rs, a, alpha, b1, b2, b3, b4):
    root = torch.sqrt(rs)
    return -2 * a * (1 + alpha * rs) * torch.log1p(1 / (2 * a * (b1 * root + b2 * rs + b3 * rs * root + b4 * rs * rs)))


def _pbe(up, down, uu, ud, dd):
    """PBE energy density of two spin densities and their gradient products."""
    kappa, beta, gamma = 0.804, 0.06672455060314922, 0.031090690869654895
    mu = beta * math.pi ** 2 / 3.0

    def exchange(n, sigma):
        n = 2 * n
        kf = (3 * math.pi ** 2 * n) ** (1 / 3)
        s2 = 4 * sigma / (4 * kf * kf * n * n)
        return 0.5 * n * (-0.75 / math.pi * kf) * (1 + kappa - kappa / (1 + mu / kappa * s2))

    n = up + down
    z = (up - down) / n
    rs = (3 / (4 * math.pi * n)) ** (1 / 3)
    f = ((1 + z) ** (4 / 3) + (1 - z) ** (4 / 3) - 2) / 0.5198420997897463295
    fzz = 8 / (9 * 0.5198420997897463295)
    eu = _pw92(rs, 0.0310907, 0.21370, 7.5957, 3.5876, 1.6382, 0.49294)
    ep = _pw92(rs, 0.01554535, 0.20548, 14.1189, 6.1977, 3.3662, 0.62517)
    ac = -_pw92(rs, 0.0168869, 0.11125, 10.357, 3.6231, 0.88026, 0.49671)
    ec = eu + ac * f / fzz * (1 - z ** 4) + (ep - eu) * f * z ** 4
    phi = 0.5 * ((1 + z) ** (2 / 3) + (1 - z) ** (2 / 3))
    ks2 = 4 * (3 * math.pi ** 2 * n) ** (1 / 3) / math.pi
    t2 = (uu + 2 * ud + dd) / (4 * phi ** 2 * ks2 * n * n)
    at = beta / gamma / torch.expm1(-ec / (gamma * phi ** 3)) * t2
    h = gamma * phi ** 3 * torch.log1p(beta / gamma * t2 * (1 + at) / (1 + at + at * at))
    return exchange(up, uu) + exchange(down, dd) + n * (ec + h)


def _functional_exact(case, lattice, channels, core):
    a = float(lattice[0, 0])
    volume, polarised = a ** 3, len(channels) == 2
    union = {tuple(k) for k in channels[0][0].tolist()}
    if core[0] is not None:
        union |= {tuple(k) for k in core[0].tolist()}
    support = np.array(sorted(union), dtype=np.int32)
    q = _gpu(support, torch.float64) * (2.0 * math.pi / a)
    q2 = (q * q).sum(dim=1)
    m = np.abs(support).max(axis=0)
    shape = tuple(int(2 * max(3, 2 * v + 1)) for v in m)
    count = int(np.prod(shape))
    place = np.full(tuple(2 * m + 1), -1, dtype=np.int64)
    place[tuple((support + m).T)] = np.arange(support.shape[0])

    def on_support(keys, values):
        out = torch.zeros(support.shape[0], dtype=torch.complex128, device="cuda")
        if keys is not None:
            out[_gpu(place[tuple((keys + m).T)])] = _gpu(values)
        return out

    index = _wrapped(support, shape)

    def field(c):
        grid = torch.zeros(count, dtype=torch.complex128, device="cuda")
        grid[index] = c
        return (torch.fft.ifftn(grid.view(shape)).real * count).reshape(-1)

    def modes(f):
        return torch.fft.fftn(f.view(shape).to(torch.complex128)).reshape(-1)[index] / count

    rho = [on_support(*c) for c in channels]
    frozen = on_support(*core)
    total = sum(rho)
    coulomb = q2 > 1e-12
    safe = torch.where(coulomb, q2, torch.ones_like(q2))
    hartree = torch.where(coulomb, 4 * math.pi * total / safe, torch.zeros_like(total))
    norm = torch.where(coulomb, (total.real ** 2 + total.imag ** 2) / safe, torch.zeros_like(q2))
    e_h = float(2 * math.pi * volume * norm.sum())
    stress_h = 4 * math.pi * torch.einsum("g,gi,gj->ij", norm / safe, q, q).cpu().numpy() - np.eye(3) * e_h / volume
    share = 0.5 if polarised else 1.0
    densities = [field(r + share * frozen) for r in rho]
    gradients = [[field(1j * q[:, i] * (r + share * frozen)) for i in range(3)] for r in rho]
    if polarised:
        n, g = densities, gradients
    else:
        n, g = [0.5 * densities[0]] * 2, [[0.5 * v for v in gradients[0]]] * 2
    variables = [v.clone().requires_grad_(True) for v in
                 (n[0], n[1], sum(x * x for x in g[0]), sum(x * y for x, y in zip(g[0], g[1])), sum(x * x for x in g[1]))]
    energy = _pbe(*variables)
    d = torch.autograd.grad(energy.sum(), variables)
    energy = energy.detach()
    if polarised:
        potentials = [d[0], d[1]]
        responses = [[2 * d[2] * g[0][i] + d[3] * g[1][i] for i in range(3)],
                     [2 * d[4] * g[1][i] + d[3] * g[0][i] for i in range(3)]]
    else:
        # d/dn at zero polarisation; both channels carry half the gradient.
        potentials = [0.5 * (d[0] + d[1])]
        responses = [[(2 * d[2] + d[3]) * g[0][i] for i in range(3)]]
    pressure = energy.clone()
    for s in range(len(channels)):
        pressure -= potentials[s] * densities[s] + sum(r * x for r, x in zip(responses[s], gradients[s]))
    stress = np.zeros((3, 3))
    for i in range(3):
        for j in range(3):
            term = -sum(responses[s][i] * gradients[s][j] for s in range(len(channels)))
            stress[i, j] = float((term + (pressure if i == j else 0.0)).mean())
    e_xc = float(energy.mean()) * volume
    partner = _gpu(place[tuple((m - support).T)])
    zero = place[tuple(m)]
    out = []
    for s in range(len(channels)):
        vxc = modes(potentials[s]) - 1j * sum(q[:, i] * modes(responses[s][i]) for i in range(3))
        pairing = float(volume * (rho[s] * vxc[partner]).real.sum())
        half = 0.5 if polarised else 1.0
        out.append({"potential": hartree + vxc, "xc_potential": vxc, "hkl": support,
                    "energies": np.array([half * e_h, half * e_xc, pairing, volume * float(rho[s][zero].real)]),
                    "hartree_stress": half * stress_h, "xc_stress": half * stress})
    return {"up": out[0], "down": out[1]} if polarised else out[0]


def exact(case, seed):
    kind = case["kind"]
    if kind == "pair":
        inputs = _operator_inputs(case, seed)
        h, s = _Pencil(inputs).apply(_block(inputs.npw, case["columns"], seed))
        return {"h": h, "s": s}
    if kind in ("solve", "scf"):
        if _sizes(case)[2] > EXACT_NPW:
            return None
        inputs = _operator_inputs(case, seed)
        pencil = _Pencil(inputs, *(_scf_step(inputs, seed) if kind == "scf" else ()))
        values, vectors = pencil.lowest(case["bands"])
        f = _occupations(values.cpu().numpy(), _electrons(case["bands"]))
        support = _support(float(inputs.lattice[0, 0]), 4.0 * case["ecut"])
        out = {"eigenvalues": values,
               "density": _density_exact(inputs.hkl, vectors.T, f, inputs.volume, support)}
        if kind == "scf":
            p = (pencil.b @ vectors).view(-1, 8, case["bands"])
            out["onsite"] = torch.einsum("n,ain,ajn->aij", _gpu(f).to(torch.complex128), p, p.conj())
        return out
    if kind == "serve":
        if _sizes(case)[2] * case["kpoints"] ** (1 / 3) > EXACT_NPW:
            return None
        return [_Pencil(x).lowest(case["bands"])[0] for x in _serve_inputs(case, seed)]
    if kind == "density":
        return _density_exact(*_density_case(case, seed))
    if kind in ("functional", "collinear"):
        return _functional_exact(case, *_functional_inputs(case, seed))
    if kind == "compensation":
        return _compensation_exact(*_compensation_inputs(case, seed))
    values, vectors = _solve_pencil(*(_gpu(m) for m in _ritz_inputs(case, seed)))
    kept = vectors[:, :case["requested"]]
    return {"values": values[:case["requested"]], "weights": kept.real ** 2 + kept.imag ** 2}
