"""Device Rayleigh-Ritz eigensolver (the reference's rayleigh_ritz,
src/pw_core.cpp:56-136) against the dense FP64 oracle: eigenvalues, residuals
||H y - e S y|| and S-orthonormality, on the paths the Davidson solve takes
(S = I exactly, S within 1e-6 of I, S far from I), with degenerate spectra and
at the largest Davidson subspace (160 roots: 1280)."""
import pathlib

import numpy as np
import pytest

from oracle import sdft_oracle

pytestmark = pytest.mark.gpu

GOLDEN = pathlib.Path(__file__).resolve().parent / "golden"


def random_unitary(n, rng):
    q, r = np.linalg.qr(rng.standard_normal((n, n)) + 1j * rng.standard_normal((n, n)))
    return q * (np.diag(r) / np.abs(np.diag(r)))


def pencil(n, rng, spectrum=None, overlap=0.0):
    u = random_unitary(n, rng)
    lam = np.sort(rng.uniform(-2.0, 30.0, n)) if spectrum is None else spectrum
    h = (u * lam) @ u.conj().T
    h = 0.5 * (h + h.conj().T)
    e = rng.standard_normal((n, n)) + 1j * rng.standard_normal((n, n))
    s = np.eye(n) + overlap * 0.5 * (e + e.conj().T) / np.sqrt(n)
    return h, s


def check(context, h, s, requested, eig_tol=1e-11, res_tol=1e-11):
    from sdft_b200.operator import rayleigh_ritz
    values, vectors = rayleigh_ritz(context, np.tril(h), np.tril(s), requested)
    count = requested or h.shape[0]
    expected = sdft_oracle.generalized_eigenvalues(h, s, count)
    scale = max(1.0, np.max(np.abs(expected)))
    assert np.max(np.abs(values - expected)) < eig_tol * scale
    residual = h @ vectors - (s @ vectors) * values[None, :]
    assert np.max(np.linalg.norm(residual, axis=0)) < res_tol * scale
    gram = vectors.conj().T @ s @ vectors
    assert np.max(np.abs(gram - np.eye(count))) < 1e-11


@pytest.mark.parametrize("n,requested", [(2, 0), (37, 10), (320, 0), (800, 320), (7, 3), (9, 0), (31, 15), (65, 0),
                                         (129, 0)])
def test_identity_overlap(context, n, requested):
    """Odd orders with an odd number of wanted pairs included: the workspace
    keeps its complex arrays 16-byte aligned whatever m * wanted is."""
    rng = np.random.Generator(np.random.PCG64(n))
    h, s = pencil(n, rng)
    check(context, h, s, requested)


@pytest.mark.parametrize("overlap", [1e-9, 5e-7, 3e-6])
def test_near_identity_overlap_uses_loewdin(context, overlap):
    rng = np.random.Generator(np.random.PCG64(11))
    h, s = pencil(500, rng, overlap=overlap)
    check(context, h, s, 160)


def test_far_from_identity_overlap_falls_back(context):
    rng = np.random.Generator(np.random.PCG64(12))
    h, s = pencil(300, rng, overlap=0.2)
    check(context, h, s, 100)


def test_degenerate_and_clustered_spectrum(context):
    rng = np.random.Generator(np.random.PCG64(13))
    n = 640
    lam = np.sort(np.concatenate([np.repeat([-1.0, 0.5, 2.0], [3, 6, 2]), [3.0, 3.0 + 1e-13, 3.0 + 4e-12],
                                  rng.uniform(4.0, 40.0, n - 14)]))
    h, s = pencil(n, rng, spectrum=lam)
    check(context, h, s, 320)


def test_largest_davidson_subspace(context):
    rng = np.random.Generator(np.random.PCG64(14))
    h, s = pencil(1280, rng, overlap=1e-10)
    check(context, h, s, 320)


def test_davidson_shaped_pencil(context):
    """Thick-restart shape: a diagonal block of Ritz values coupled to a new block."""
    rng = np.random.Generator(np.random.PCG64(15))
    k0, n = 320, 480
    h = np.zeros((n, n), dtype=complex)
    h[:k0, :k0] = np.diag(np.sort(rng.uniform(-0.5, 2.0, k0)))
    c = 1e-3 * (rng.standard_normal((k0, n - k0)) + 1j * rng.standard_normal((k0, n - k0)))
    h[:k0, k0:] = c
    h[k0:, :k0] = c.conj().T
    d = rng.standard_normal((n - k0, n - k0)) + 1j * rng.standard_normal((n - k0, n - k0))
    h[k0:, k0:] = 0.5 * (d + d.conj().T) + 5.0 * np.eye(n - k0)
    check(context, h, np.eye(n), 320)


def spaced(n, rng):
    """n ascending eigenvalues on [-2, 30] at least half a mean spacing (16 / n) apart: inverse iteration finds
    the vectors one by one, orthogonal to eps ||T|| / gap (2.2e-16 x 30 x 400 / 16 = 2e-13 at n = 400), so a
    random spectrum's smallest gap would set the orthogonality measured here, not the reduction."""
    return -2.0 + 32.0 * (np.arange(n) + rng.uniform(0.25, 0.75, n)) / n


@pytest.mark.parametrize("n", [2, 3, 16, 17, 64, 65, 127, 128, 129, 255, 256, 257, 258, 400])
def test_tridiagonalisation_orders(context, n):
    """The call's reduction at the orders where the solves' one changes kernels
    (test_reduction_inside_solves)."""
    rng = np.random.Generator(np.random.PCG64(100 + n))
    h, s = pencil(n, rng, spectrum=spaced(n, rng))
    check(context, h, s, 0)


@pytest.mark.parametrize("n", [511, 512, 513, 769, 1025])
def test_grid_reduction_orders(context, n):
    """Orders around the kernels' 256 rows per thread slot, and odd column counts per CTA."""
    rng = np.random.Generator(np.random.PCG64(300 + n))
    h, s = pencil(n, rng, spectrum=spaced(n, rng))
    check(context, h, s, n // 3)


@pytest.mark.parametrize("n", [5, 130, 300])
def test_tridiagonalisation_of_decoupled_blocks(context, n):
    """Columns that are already reduced (trivial reflectors) and exact zeros among coupled blocks."""
    rng = np.random.Generator(np.random.PCG64(200 + n))
    half = n // 2
    lam = rng.permutation(spaced(n, rng))
    h = np.diag(lam).astype(complex)
    h[half:, half:], _ = pencil(n - half, rng, spectrum=np.sort(lam[half:]))
    check(context, h, np.eye(n), 0)


def paired_pencil(n):
    """Hermitian matrix whose eigenvalues come in pairs about 1e-6 apart: a random matrix of order n / 2 times the
    2 x 2 identity, plus 2^-20 of another. Every entry is an integer over a power of two, so the matrix is the same
    on any machine."""
    rng = np.random.Generator(np.random.PCG64(400 + n))

    def hermitian(m):
        a = rng.integers(-2**9, 2**9, (m, m)) + 1j * rng.integers(-2**9, 2**9, (m, m))
        return (np.tril(a) + np.tril(a, -1).conj().T - 1j * np.diag(np.diag(a).imag)) / 2.0**8

    return np.kron(hermitian(n // 2), np.eye(2)) + hermitian(n) / 2.0**20


@pytest.mark.parametrize("n", [96, 300, 700])
def test_vectors_of_near_pairs_are_the_recorded_ones(context, n):
    """The weights |y|^2 of pairs 1e-6 apart turn the reduction's rounding into eps ||T|| / gap (1e-9 to 1e-8 here), so the
    call is held to the results that it gave before solves got a reduction of their own, as recorded on a B200
    (148 SMs) at commit 2fc5f5b. With the same tridiagonal matrix and eigenvalues only the back-transformation's
    rounding is left, sqrt(n) eps per vector (6e-15)."""
    from sdft_b200.operator import rayleigh_ritz
    recorded = np.load(GOLDEN / "ritz_pairs.npz")
    values, vectors = rayleigh_ritz(context, paired_pencil(n), np.eye(n), 12)
    weights = vectors.real ** 2 + vectors.imag ** 2
    assert np.array_equal(values, recorded[f"values_{n}"])
    assert np.linalg.norm(weights - recorded[f"weights_{n}"]) < 1e-13 * np.linalg.norm(recorded[f"weights_{n}"])


@pytest.fixture(scope="module")
def free_electrons(context):
    """An operator without potential or projectors, H = T and S = 1 exactly, its levels in Ha, and plane waves whose
    levels are at least 0.01 Ha apart."""
    import dataclasses

    from sdft_b200 import synthetic
    from sdft_b200.operator import PlaneWaveOperator
    x = synthetic.tiny(ecut_ha=30.0, kpoint=(0.1371, 0.2719, 0.4133), roots=4)
    x = dataclasses.replace(x, v_values=x.v_values * 0.0, d=x.d * 0.0, q=x.q * 0.0, regularization=0.0)
    levels = x.kinetic_ev / x.hartree_to_ev
    apart = []
    for g in np.argsort(levels):
        if not apart or levels[g] >= levels[apart[-1]] + 0.01:
            apart.append(g)
    op = PlaneWaveOperator(context, x)
    yield op, levels, np.array(apart)
    op.close()


@pytest.mark.parametrize("n,coupled", [(2, 2), (3, 3), (16, 16), (17, 17), (64, 64), (65, 65), (127, 127), (128, 128),
                                       (129, 129), (255, 255), (256, 256), (257, 257), (258, 258), (400, 400),
                                       (511, 511), (512, 512), (513, 513), (769, 769), (1025, 1025), (5, 3), (130, 65),
                                       (300, 150)])
def test_reduction_inside_solves(free_electrons, n, coupled):
    """The reduction that solves use, at chosen orders through the RMM trial's first rotation: a block that spans n
    plane waves, the last `coupled` of them mixed by a random unitary matrix (the others are decoupled: trivial
    reflectors and exact zeros), has their levels as Ritz values. Orders around the cluster kernel's tiles (128, 256),
    its hand-over from the grid kernel (257 and up) and the grid kernel's 256 rows per thread slot. Bars as in check():
    vectors eps ||T|| / gap = 7e-13 apart at 30 and 0.01 Ha."""
    op, levels, apart = free_electrons
    rng = np.random.Generator(np.random.PCG64(500 + n + coupled))
    rows = rng.permutation(apart)[:n]
    mix = np.eye(n, dtype=complex)
    mix[n - coupled:, n - coupled:] = random_unitary(coupled, rng)
    block = np.zeros((n, op.npw), dtype=complex)
    block[:, rows] = mix.T
    got = op.rmm_trial(n, block, 2, 2e-9)
    assert got["trial_manifold"] and got["iterations"] == 1
    values, vectors = got["eigenvalues"], got["eigenvectors"].T
    scale = levels[rows].max()
    assert np.max(np.abs(values - np.sort(levels[rows]))) < 1e-11 * scale
    assert np.max(np.linalg.norm((levels[:, None] - values) * vectors, axis=0)) < 1e-11 * scale
    assert np.max(np.abs(vectors.conj().T @ vectors - np.eye(n))) < 1e-11
