"""Collinear spin functional on the device (sdft_b200_collinear_functionals).

Against the reference's evaluate_collinear_density_functionals
(tests/golden/collinear_*.npz, up and down Gaussian densities with different
supports, with and without a frozen core split between the channels): the
bars of test_oracle_pins.check_collinear (energies, electrons and
<n_s, v_xc,s> 1e-12 relative, stresses 1e-11, minimum 1e-10, counts of
negative samples exact, potentials 1e-11, or 1e-6 where floored samples make
the reference's own response ill-conditioned). At the Si64 scale (142^3 = 2 x
71 per axis) the nonmagnetic limit n_up = n_down = n/2 reproduces the
spin-unpolarised functional: total XC energy within 1e-10 relative, each
channel's v_xc and potential within 1e-6 of the unpolarised ones, Hartree
split equally.
"""
import numpy as np
import pytest

from conftest import relative_error
from sdft_b200 import _capi as C
from sdft_b200 import density, synthetic
from test_oracle_pins import COLLINEAR_POTENTIAL_TOL, check_collinear, collinear_inputs

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("name", ["si8", "triclinic"])
@pytest.mark.parametrize("label", ["plain", "core"])
def test_collinear_matches_reference(context, golden, name, label):
    case, core = collinear_inputs(name, label)
    result = density.collinear_functionals(context, case["lattice"], case["up_keys"], case["up"], case["down_keys"],
                                           case["down"], core.get("core_hkl"), core.get("core"))
    check_collinear(result, golden(f"collinear_{name}"), label, COLLINEAR_POTENTIAL_TOL[name])


def test_nonmagnetic_limit_is_the_unpolarised_functional(context):
    c = synthetic.functional_case("si64")
    half = 0.5 * c["values"]
    spin = density.collinear_functionals(context, c["lattice"], c["keys"], half, c["keys"], half)
    plain = density.density_functionals(context, c["lattice"], c["keys"], c["values"])
    assert spin["up"]["grid"] == plain["grid"] == (142, 142, 142)
    assert np.array_equal(spin["hkl"], plain["hkl"])
    total_xc = spin["up"]["xc_energy"] + spin["down"]["xc_energy"]
    assert abs(total_xc - plain["xc_energy"]) <= 1e-10 * abs(plain["xc_energy"])
    assert abs(2 * spin["up"]["hartree_energy"] - plain["hartree_energy"]) <= 1e-12 * plain["hartree_energy"]
    for channel in ("up", "down"):
        assert relative_error(spin[channel]["xc_potential"], plain["xc_potential"]) < 1e-6
        assert relative_error(spin[channel]["potential"], plain["potential"]) < 1e-6
    assert relative_error(spin["up"]["xc_potential"], spin["down"]["xc_potential"]) < 1e-12


def test_collinear_host_checks(context):
    c = synthetic.collinear_case("triclinic")
    with pytest.raises(ValueError, match="invalid collinear density/lattice"):
        density.collinear_functionals(context, np.zeros((3, 3)), c["up_keys"], c["up"], c["down_keys"], c["down"])
    with pytest.raises(ValueError, match="invalid collinear XC padding"):
        density.collinear_functionals(context, c["lattice"], c["up_keys"], c["up"], c["down_keys"], c["down"],
                                      padding=9)
    bad = c["up"].copy()
    bad[0] = np.nan
    with pytest.raises(ValueError, match="nonfinite spin density"):
        density.collinear_functionals(context, c["lattice"], c["up_keys"], bad, c["down_keys"], c["down"])


@pytest.mark.parametrize("pinned", [False, True])
def test_outputs_may_be_the_input_arrays(context, pinned):
    """Both forms through the C entry with the support, the potentials and the densities in the same (pageable or
    page-locked) arrays, the keys in random order: the same results, bit for bit, as with arrays of their own."""
    import ctypes

    import torch
    rng = np.random.Generator(np.random.PCG64(31))
    every = np.stack(np.meshgrid(*[np.arange(-9, 10)] * 3, indexing="ij"), axis=-1).reshape(-1, 3)
    hkl = np.ascontiguousarray(every[rng.permutation(len(every))], dtype=np.int32)
    decay = np.exp(-0.5 * (hkl.astype(float) ** 2).sum(axis=1))
    values = [f * decay * np.exp(-2j * np.pi * (hkl @ rng.uniform(size=3))) for f in (0.02, 0.013)]
    lattice = np.ascontiguousarray(np.diag([9.0, 10.0, 11.0]).reshape(9))
    lib, n, count = C.library(), len(hkl), ctypes.c_size_t()

    def array(source):
        t = torch.from_numpy(np.ascontiguousarray(source).copy())
        return t.pin_memory().numpy() if pinned else t.numpy()

    def fields(a):
        return a.ctypes.data_as(C.D)

    def collinear(inplace):
        keys, up, down = array(hkl), array(values[0]), array(values[1])
        support, pu, pd = (keys, up, down) if inplace else (array(hkl * 0), array(up * 0), array(down * 0))
        xu, xd = array(up * 0), array(down * 0)
        result = (C.Functionals * 2)()
        C.check(lib.sdft_b200_collinear_functionals(
            context.handle, fields(lattice), n, keys.ctypes.data_as(C.I32), fields(up), n, keys.ctypes.data_as(C.I32),
            fields(down), 0, None, None, 0, support.ctypes.data_as(C.I32), fields(pu), fields(pd), fields(xu),
            fields(xd), n, ctypes.byref(count), result))
        return [support, pu, pd, xu, xd], [r.as_dict() for r in result]

    def unpolarised(inplace):
        keys, density = array(hkl), array(values[0])
        support, potential = (keys, density) if inplace else (array(hkl * 0), array(density * 0))
        xc, result = array(density * 0), C.Functionals()
        C.check(lib.sdft_b200_density_functionals(
            context.handle, fields(lattice), n, keys.ctypes.data_as(C.I32), fields(density), 0, None, None, 0,
            support.ctypes.data_as(C.I32), fields(potential), fields(xc), n, ctypes.byref(count), ctypes.byref(result)))
        return [support, potential, xc], [result.as_dict()]

    for form in (collinear, unpolarised):
        (own, own_scalars), (same, same_scalars) = form(False), form(True)
        assert count.value == n
        for a, b in zip(own, same):
            assert np.array_equal(a, b)
        for a, b in zip(own_scalars, same_scalars):
            assert all(np.array_equal(a[key], b[key]) for key in a)
