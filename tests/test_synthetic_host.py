"""The seeded input generators' shortcuts against their direct forms (CPU).

- V(G) noise pairing: on a key set closed under G -> -G in lexicographic
  order, -G sits at the mirrored index; the generated V(G) is bit-identical
  to the dictionary lookup and Hermitian.
- The serving stream's closed-form Q scale equals the bisection's to 1e-12
  (lambda_min((1+reg) I + s R Q R) is linear in s), and its requests reuse
  one V(G) per cell across their k-points with the same draws as a fresh
  build.
"""
import numpy as np

from sdft_b200 import synthetic


def _dictionary_potential(x, noise=0.05, noise_cut=4.0, width=1.0, seed=2026):
    """local_potential with the -G partner found by dictionary lookup."""
    import math
    rng = np.random.Generator(np.random.PCG64(seed))
    depths = np.array([(-2.0, -2.0)[s] for s in x.species], dtype=np.float64)
    volume = abs(float(np.linalg.det(x.lattice)))
    hkl, cart = synthetic._potential_keys(x.reciprocal, noise_cut * x.ecut_ha)
    tau = x.positions @ x.lattice
    g2 = np.einsum("ij,ij->i", cart, cart)
    shape = (2.0 * math.pi * width * width) ** 1.5 / volume * np.exp(-0.5 * g2 * width * width)
    values = shape * (np.exp(-1j * (cart @ tau.T)) @ depths)
    positive = (hkl[:, 0] > 0) | ((hkl[:, 0] == 0) & ((hkl[:, 1] > 0) | ((hkl[:, 1] == 0) & (hkl[:, 2] > 0))))
    zero = np.all(hkl == 0, axis=1)
    draws = rng.standard_normal((hkl.shape[0], 2))
    noise_values = noise * (draws[:, 0] + 1j * draws[:, 1]) / math.sqrt(2.0)
    noise_values[zero] = noise * draws[zero, 0]
    values = values + np.where(positive | zero, noise_values, 0.0)
    index = {tuple(key): i for i, key in enumerate(hkl.tolist())}
    negative = np.nonzero(~(positive | zero))[0]
    partner = np.array([index[(-hkl[i, 0], -hkl[i, 1], -hkl[i, 2])] for i in negative], dtype=np.int64)
    values[negative] = np.conj(values[partner])
    values[zero] = values[zero].real
    return values


def test_potential_pairing_matches_dictionary_lookup():
    x = synthetic.tiny()
    assert np.array_equal(x.v_values, _dictionary_potential(x, seed=7))
    position = {tuple(k): i for i, k in enumerate(x.v_hkl.tolist())}
    mirror = np.array([position[(-h, -k, -l)] for h, k, l in x.v_hkl.tolist()])
    assert np.array_equal(x.v_values[mirror], np.conj(x.v_values))


def test_linear_q_scale_matches_bisection():
    for x in (synthetic.tiny(), synthetic.tiny(seed=3), synthetic.si8()):
        q_raw = x.q / x.q_scale
        exact = synthetic._scale_q_linear(x.amplitudes, q_raw, x.regularization)
        assert abs(exact - x.q_scale) <= 1e-12 * x.q_scale
        floor = synthetic.overlap_minimum(x.amplitudes, exact * q_raw, x.regularization)
        assert abs(floor - 0.3) < 1e-10


def test_serving_request_reuses_the_cell_potential():
    request = synthetic.serving_request(3)
    assert len(request) > 1
    first = request[0]
    for op in request[1:]:
        assert np.array_equal(op.v_hkl, first.v_hkl) and np.array_equal(op.v_values, first.v_values)
        assert np.array_equal(op.d, first.d)  # the same draws follow V(G)
    fresh = synthetic.build_operator("fresh", (first.positions.shape[0] * synthetic.SI_VOLUME_PER_ATOM) ** (1 / 3),
                                     1, first.ecut_ha, first.roots, depths=(-2.2, -1.8),
                                     kpoint=tuple(request[1].kpoint), seed=4242 * 1000 + 3,
                                     sites=(first.positions, first.species), q_scaling="linear")
    assert np.array_equal(fresh.v_values, request[1].v_values) and np.array_equal(fresh.q, request[1].q)


def test_bench_reference_arm_without_the_reference(monkeypatch, capsys):
    """Where the reference's library is not built the arm says so in one line instead of failing."""
    import argparse
    import json

    import bench
    from oracle import ref_oracle
    monkeypatch.setattr(ref_oracle, "available", lambda: False)
    bench.run_reference(argparse.Namespace(gpus=1, steps=1, warmup=0))
    line = json.loads(capsys.readouterr().out)
    assert line["impl"] == "reference" and line["unavailable"]
