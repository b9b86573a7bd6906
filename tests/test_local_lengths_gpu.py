"""The fused local H~psi at every grid length its register-resident kernels
are compiled for (FP32: the half-line pencils of even lengths up to 72 points,
the one-thread pencils of odd ones, the pair-split pencils above, and the
pair-split plane passes of even lengths) and lengths that take the four-step
planes and pencils (all of them in FP64), on small cubic cells whose alias-free
grid rule (src/plane_wave_operator.cpp:445-457) lands on that length; a k-point
of (k, k, k) makes the span odd where needed. Lengths without a split (125) and
plane waves outside the grid rule follow on callers' grids.

Bars: the FP32 local apply (mixed form) within 2e-5 relative of the FP64
one (the mixed bar of tests/native/plane_wave_operator_smoke.cpp), per column
and for the block; the FP64 apply within 1e-12 of the numpy oracle's local
term; the mixed full H~x / S~x pair bit-identical to separate applies.
"""
import ctypes

import numpy as np
import pytest

from conftest import probe_block, relative_error
from oracle import sdft_oracle
from sdft_b200 import _capi as C
from sdft_b200 import synthetic
from sdft_b200.operator import PlaneWaveOperator

pytestmark = pytest.mark.gpu

# grid length -> (Ecut in Ha, k) for synthetic.tiny (a = 7 bohr, diamond Si8-like sites).
CELLS = {35: (26.0, 0.0), 40: (33.0, 0.0), 42: (40.5, 0.0), 45: (45.0, 0.5), 48: (53.5, 0.5), 49: (58.5, 0.0),
         54: (63.5, 0.5), 56: (74.0, 0.5), 60: (79.0, 0.0), 63: (91.0, 0.0), 70: (103.5, 0.0), 72: (124.0, 0.5),
         75: (131.0, 0.0), 80: (145.5, 0.0), 81: (161.5, 0.0), 84: (169.5, 0.5), 90: (178.0, 0.0),
         96: (204.5, 0.5), 98: (232.5, 0.0), 100: (242.5, 0.5), 112: (294.0, 0.0), 120: (316.0, 0.0),
         128: (400.0, 0.5)}
# Lengths checked against the numpy oracle as well: small ones, and the four-step
# transforms of 7 x 14, 8 x 14, 10 x 12 and 8 x 16 points (radices above 10).
ORACLE_LENGTHS = {35, 40, 45, 49, 98, 112, 120, 128}
COLUMNS = 6


@pytest.mark.parametrize("n", sorted(CELLS))
def test_local_apply_mixed_matches_fp64_at_grid_length(context, n):
    import torch
    ecut, k = CELLS[n]
    inputs = synthetic.tiny(ecut_ha=ecut, kpoint=(k, k, k), roots=4)
    op = PlaneWaveOperator(context, inputs)
    try:
        assert op.shape == (n, n, n)
        x = probe_block(op.npw, COLUMNS, 100 + n)
        xd = torch.from_numpy(np.ascontiguousarray(x.T)).cuda().T
        y64 = op.local_apply(xd, precision="fp64")
        y32 = op.local_apply(xd, precision="mixed")
        context.synchronize()
        a64 = y64.T.cpu().numpy().T
        a32 = y32.T.cpu().numpy().T
        assert relative_error(a32, a64) < 2e-5
        for c in range(COLUMNS):
            assert relative_error(a32[:, c], a64[:, c]) < 2e-5
        if n in ORACLE_LENGTHS:  # the numpy oracle's local term (FFTs of the full grid)
            oracle = sdft_oracle.Operator(inputs)
            assert relative_error(a64, oracle.local(x)) < 1e-12
        hy, sy = op.apply_pair(xd, precision="mixed")
        h = op.apply(xd, overlap=False, precision="mixed")
        s = op.apply(xd, overlap=True, precision="mixed")
        context.synchronize()
        assert torch.equal(hy, h) and torch.equal(sy, s)
    finally:
        op.close()


def test_operator_above_65535_plane_waves(context):
    """An operator whose plane-wave count exceeds the CUDA grid's y limit
    (65 535): the tensor-core packing of B^H (one packed row per plane wave)
    and the mixed applies stride past it."""
    import torch
    inputs = synthetic.build_operator("large", 10.26, 1, 122.0, 8)
    assert inputs.hkl.shape[0] > 65535
    op = PlaneWaveOperator(context, inputs)
    try:
        x = probe_block(op.npw, 4, 65536)
        xd = torch.from_numpy(np.ascontiguousarray(x.T)).cuda().T
        for overlap in (False, True):
            y64 = op.apply(xd, overlap=overlap, precision="fp64")
            y32 = op.apply(xd, overlap=overlap, precision="mixed")
            context.synchronize()
            assert relative_error(y32.T.cpu().numpy(), y64.T.cpu().numpy()) < 2e-5
    finally:
        op.close()


# (Ecut, k) -> grid: axes of different lengths and splits (12 = 3 x 4, 14 = 2 x 7, 20 = 4 x 5, 18 = 3 x 6,
# 30 = 5 x 6, 27 = 3 x 9, 49 = 7 x 7, 48 = 6 x 8), and 125 = 5 x 25, which has none.
MIXED_AXES = {(4.0, (0.5, 0.0, 0.0)): (12, 14, 14), (9.0, (0.5, 0.25, 0.0)): (20, 18, 18),
              (20.0, (0.0, 0.5, 0.5)): (30, 27, 27), (60.0, (0.0, 0.5, 0.0)): (49, 48, 49),
              (390.0, (0.0, 0.0, 0.0)): (125, 125, 125)}


@pytest.mark.parametrize("cell", list(MIXED_AXES), ids=lambda c: "x".join(str(n) for n in MIXED_AXES[c]))
def test_local_apply_on_unequal_axes(context, cell):
    """FP64 against the numpy oracle: both sum about 3 x 2 x log2(n^3) < 130 rounded terms of 1.1e-16 in
    another order, so 130 x 1.1e-16 = 1.5e-14 bounds their relative difference; the mixed form at its bar."""
    ecut, k = cell
    inputs = synthetic.tiny(ecut_ha=ecut, kpoint=k, roots=4)
    op = PlaneWaveOperator(context, inputs)
    try:
        assert op.shape == MIXED_AXES[cell]
        x = probe_block(op.npw, 3, 7)
        expected = sdft_oracle.Operator(inputs).local(x)
        assert relative_error(op.local_apply(x, precision="fp64"), expected) < 1.5e-14
        assert relative_error(op.local_apply(x, precision="mixed"), expected) < 2e-5
    finally:
        op.close()


@pytest.mark.parametrize("n", [40, 42, 54, 70, 72])
@pytest.mark.parametrize("columns", [1, 2, 5])
def test_half_line_pencils_at_column_counts(context, n, columns):
    """Even lengths whose pencils are worked off in two half-length spectra, two columns to a CTA: one column, one
    pair, and an odd count whose last pair has one. Bar as above (FP32 against FP64, per column)."""
    import torch
    ecut, k = CELLS[n]
    op = PlaneWaveOperator(context, synthetic.tiny(ecut_ha=ecut, kpoint=(k, k, k), roots=4))
    try:
        assert op.shape == (n, n, n) and 2 * op.active_rows <= n
        # strides given outright: torch does not keep them for a single column
        xd = torch.empty_strided((op.npw, columns), (1, op.npw), dtype=torch.complex128, device="cuda")
        xd.copy_(torch.from_numpy(probe_block(op.npw, columns, 300 + n)))
        y64 = op.local_apply(xd, precision="fp64")
        y32 = op.local_apply(xd, precision="mixed")
        context.synchronize()
        for c in range(columns):
            assert relative_error(y32.T[c].cpu().numpy(), y64.T[c].cpu().numpy()) < 2e-5
    finally:
        op.close()


def accelerated_local(context, shape, indices, potential, kinetic, x, precision):
    """T x + V(r) x through the accelerator's entry, which takes any grid and plane waves. x: (npw, columns)."""
    n, columns = x.shape
    xin, out = np.ascontiguousarray(x.T), np.zeros((columns, n), dtype=np.complex128)
    dims = np.array(shape, dtype=np.int32)
    C.check(C.library().sdft_b200_local_hamiltonian(
        context.handle, dims.ctypes.data_as(C.I32), indices.ctypes.data_as(C.U64), n, kinetic.ctypes.data_as(C.D),
        potential.ctypes.data_as(C.D), ctypes.c_void_p(xin.ctypes.data), columns, ctypes.c_void_p(out.ctypes.data),
        C.FP64 if precision == "fp64" else C.MIXED, 0))
    return out.T


# Grid and the rows that plane waves take along each axis (None: all).
GRIDS = {
    # an axis of 125 points (no split): the two-buffer plane kernels, the radix-stage pencils, planes through the slab
    "n1=125": ((12, 125, 20), (6, 60, 10)), "n2=125": ((14, 20, 125), (7, 9, 63)), "n0=125": ((125, 10, 12), (62, 5, 6)),
    "planes=125": ((8, 125, 125), (4, 50, 61)), "planes=125x45": ((10, 125, 45), (5, 60, 20)),
    # even FP32 lengths whose rows do not differ mod n0 / 2: four-step pencils instead of two half-length spectra
    "all rows of 40": ((40, 8, 9), (None, 4, 5)), "all rows of 70": ((70, 15, 14), (None, 7, 7)),
    "36 rows of 70": ((70, 15, 14), (36, 7, 7)), "all rows of 72": ((72, 72, 72), (None, None, None)),
    # and rows that do, on planes smaller than a block of 128 lines and a little larger
    "35 rows of 70": ((70, 6, 5), (35, 3, 3)), "21 rows of 42": ((42, 10, 14), (21, 5, 7)),
}


@pytest.mark.parametrize("grid", list(GRIDS))
def test_local_apply_on_callers_grids(context, grid):
    """FP64 within 130 rounded terms of 1.1e-16 of numpy's transforms, as above; the mixed form at its bar."""
    shape, rows = GRIDS[grid]
    rng = np.random.Generator(np.random.PCG64(sum(shape)))
    axes = [np.arange(n) if r is None else np.arange(-((r - 1) // 2), r // 2 + 1) % n for n, r in zip(shape, rows)]
    box = (axes[0][:, None, None] * shape[1] + axes[1][None, :, None]) * shape[2] + axes[2][None, None, :]
    # one plane wave at least on every row of the first axis
    indices = np.unique(np.concatenate([rng.permutation(box.ravel())[:2000], box[:, 0, 0]])).astype(np.uint64)
    indices = np.ascontiguousarray(rng.permutation(indices))
    assert len(np.unique(indices // np.uint64(shape[1] * shape[2]))) == (rows[0] or shape[0])
    potential = rng.standard_normal(shape)
    kinetic = rng.uniform(0.0, 10.0, len(indices))
    x = probe_block(len(indices), 3, 11)
    field = np.zeros((3, int(np.prod(shape))), dtype=np.complex128)
    field[:, indices.astype(np.int64)] = x.T
    field = np.fft.ifftn(field.reshape(3, *shape), axes=(1, 2, 3)) * potential
    field = np.fft.fftn(field, axes=(1, 2, 3)).reshape(3, -1)
    expected = field[:, indices.astype(np.int64)].T + kinetic[:, None] * x
    assert relative_error(accelerated_local(context, shape, indices, potential, kinetic, x, "fp64"), expected) < 1.5e-14
    assert relative_error(accelerated_local(context, shape, indices, potential, kinetic, x, "mixed"), expected) < 2e-5
