"""Runs of layers taken in one launch (small sums inside ``ps_propagate``), against the oracle.

A run holds the sum in the blocks' shared memory from layer to layer; it must give every layer's
count and the final terms bit for bit, at the sizes where its split can go wrong: fewer terms than
blocks, shares of unequal length, a sum that outgrows the blocks on the way (the run ends and the
per-layer kernels go on), TopN boundaries with and without ties and NaN, folded and unfolded noise,
layers without partners and layers it does not take (more than four generator bits, general tables).
"""

from __future__ import annotations

import numpy as np
import pytest

import paulistrings_b200 as ps
from paulistrings_b200 import truncation, workloads

from _util import assert_same_terms, oracle_arrays, oracle_channels, oracle_policy, oracle_sum

pytestmark = pytest.mark.gpu


def _run(nq, x, z, c, circ, pol, dtype="f64", direction="heisenberg"):
    g = ps.GpuPauliSum(nq, dtype)
    g.upload(x, z, c)
    st = g.propagate(circ, pol, direction, with_stats=True)
    o = oracle_sum(nq, x, z, c, dtype)
    after = o.propagate(oracle_channels(circ), oracle_policy(pol), direction)
    assert st.terms_after == [int(v) for v in after]
    assert_same_terms(g.download(), oracle_arrays(o), what=f"{nq} {dtype} {len(x)}")
    return g, st


@pytest.mark.parametrize("dtype", ["f64", "f32"])
@pytest.mark.parametrize("nq", [20, 64, 100, 128, 200])
@pytest.mark.parametrize("count", [1, 2, 147, 148, 149, 2961])
def test_threshold_runs(nq, count, dtype):
    x, z, c = workloads.random_observable(nq, count, seed=count)
    g, st = _run(nq, x, z, c, workloads.random_pair_layers(nq, 1, seed=nq + count), truncation.coeff(3e-3), dtype)
    prof = g.read_profile()
    assert prof["k_layer_run"]["launches"] >= 1
    assert prof["k_merge"]["launches"] == 0  # every layer ran inside


@pytest.mark.parametrize("dtype", ["f64", "f32"])
@pytest.mark.parametrize("nq,cap", [(20, 1), (20, 149), (24, 5000), (100, 3001), (200, 2999)])
@pytest.mark.parametrize("values", ["normal", "few", "equal", "wide"])
def test_topn_runs(nq, cap, dtype, values):
    """TopN after every layer: distinct magnitudes, whole blocks tied at the boundary (the quota
    cuts them in key order), all equal, and magnitudes over hundreds of octaves (the boundary
    leaves the window of the last one)."""
    count = max(1, min(cap, 2000))
    x, z, c = workloads.random_observable(nq, count, seed=cap)
    rng = np.random.default_rng(cap)
    if values == "few":
        c = rng.choice([0.25, -0.25, 0.5, 0.125], size=count)
    elif values == "equal":
        c = np.ones(count)
    elif values == "wide":
        c = c * 2.0 ** rng.integers(-60, 60, count)
    _run(nq, x, z, c, workloads.random_pair_layers(nq, 2, seed=cap + 1), truncation.topn(cap), dtype)


def test_topn_run_with_nan():
    x, z, c = workloads.random_observable(16, 300, seed=5)
    c[::7] = np.nan
    _run(16, x, z, c, workloads.random_pair_layers(16, 1, seed=8), truncation.topn(400))


@pytest.mark.parametrize("dtype", ["f64", "f32"])
def test_a_sum_that_outgrows_the_blocks(dtype):
    """Four-word keys: the run ends at the layer that no longer fits, the per-layer kernels take
    over."""
    nq = 200
    x, z, c = workloads.random_observable(nq, 90000, seed=3)
    circ = ps.Circuit(nq)
    for ch in list(workloads.random_pair_layers(nq, 3, seed=4))[:130]:
        circ.append(ch)
    g, _ = _run(nq, x, z, c, circ, truncation.coeff(1e-12), dtype)
    assert g.read_profile()["k_merge"]["launches"] > 0


@pytest.mark.parametrize("dtype", ["f64", "f32"])
@pytest.mark.parametrize("policy", [truncation.coeff(1e-4), truncation.coeff(1e-9) & truncation.topn(700),
                                    truncation.weight(3) | truncation.coeff(0.02)])
def test_mixed_channels(policy, dtype):
    """Noise in front of rotations and at the end, quarter turns, wide rotations of few and many
    generator bits, Hadamard and damping (partner path) and CNOT (sort path) in one circuit."""
    rng = np.random.default_rng(11)
    for nq in (12, 70):
        circ = ps.Circuit(nq)
        circ.depolarize(0.05, range(nq))
        for k in range(40):
            a, b, d = (int(q) for q in rng.choice(nq, size=3, replace=False))
            t = float(rng.uniform(-3, 3))
            kind = k % 10
            if kind == 0:
                circ.pauli_rotation("XYZ", [a, b, d], t)          # four bits
            elif kind == 1:
                circ.pauli_rotation("YYX", [a, b, d], t)          # five bits
            elif kind == 2:
                circ.h(a)
                circ.amplitude_damping(0.1, [b])
            elif kind == 3:
                circ.cnot(a, b)
            elif kind == 4:
                circ.dephase(0.02, [a, b, d])
                circ.pauli_channel(0.01, 0.02, 0.03, [a])
            elif kind == 5:
                circ.s(a)
                circ.pauli_rotation("ZZ", [a, b], np.pi / 2)
                circ.pauli_rotation("X", [d], np.pi)
            else:
                circ.pauli_rotation("".join(rng.choice(list("XYZ"), 2)), [a, b], t)
        circ.depolarize(0.01, range(nq))
        x, z, c = workloads.random_observable(nq, 60, seed=nq)
        _run(nq, x, z, c, circ, policy, dtype, "forward")
