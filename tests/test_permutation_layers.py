"""CNOT, CZ, SWAP and unitaries equal to them as steps on the partner path, against the oracle: through
the run kernel, and (per-kernel profiling on) through the per-layer kernels, bit for bit, with
coefficients that are not finite, thresholds and weights that the steps in between must not see, a
TopN budget, and a failure between steps."""

from __future__ import annotations

import numpy as np
import pytest

import paulistrings_b200 as ps
from paulistrings_b200 import _lib, truncation, workloads
from paulistrings_b200.circuit import Circuit, gates

from _util import assert_same_terms, oracle_arrays, oracle_channels, oracle_policy, oracle_sum

pytestmark = pytest.mark.gpu

SWAP = np.array([[1, 0, 0, 0], [0, 0, 1, 0], [0, 1, 0, 0], [0, 0, 0, 1]], dtype=complex)
ISWAP = np.array([[1, 0, 0, 0], [0, 0, 1j, 0], [0, 1j, 0, 0], [0, 0, 0, 1]], dtype=complex)


def _circuit(nq):
    rng = np.random.default_rng(nq)
    c = Circuit(nq)
    for k in range(18):
        a, b = (int(q) for q in rng.choice(nq, size=2, replace=False))
        c.append([gates.cnot(a, b), gates.cz(a, b), gates.swap(a, b), gates.unitary_2q(a, b, SWAP),
                  gates.unitary_2q(a, b, ISWAP), gates.pauli_rotation("XY", [a, b], 0.3)][k % 6])
    return c


@pytest.mark.parametrize("dtype", ["f64", "f32"])
@pytest.mark.parametrize("nq,count", [(6, 40), (64, 3001), (70, 1290), (200, 900)])
@pytest.mark.parametrize("policy", [None, truncation.coeff(0.01) & truncation.weight(5), truncation.topn(1000)])
@pytest.mark.parametrize("per_layer", [False, True])
def test_permutations(nq, count, dtype, policy, per_layer):
    x, z, c = workloads.random_observable(nq, count, seed=nq)
    if policy is None:
        c[::17] = np.nan
        c[5::19] = np.inf
    circ = _circuit(nq)
    g = ps.GpuPauliSum(nq, dtype)
    g.set_profiling(per_layer)
    g.upload(x, z, c)
    st = g.propagate(circ, policy, "heisenberg", with_stats=True)
    o = oracle_sum(nq, x, z, c, dtype)
    after = o.propagate(oracle_channels(circ), oracle_policy(policy), "heisenberg")
    assert st.terms_after == [int(v) for v in after]
    assert_same_terms(g.download(), oracle_arrays(o), what=f"{nq} {dtype}")


def test_a_failed_permutation_leaves_the_store():
    nq = 32
    x, z, c = workloads.random_observable(nq, 5000, seed=2)
    circ = Circuit(nq)
    circ.cnot(3, 9)
    for k in range(12):
        g = ps.GpuPauliSum(nq)
        g.set_profiling(True)
        g.upload(x, z, c)
        before = g.download()
        _lib.check(_lib.lib().ps_inject_fault(g._h, _lib.PS_FAULT_OOM, k), g._h, "inject")
        try:
            g.propagate(circ)
            done = True
        except MemoryError:
            done = False
        _lib.check(_lib.lib().ps_inject_fault(g._h, _lib.PS_FAULT_NONE, 0), g._h, "disarm")
        if not done:
            assert_same_terms(g.download(), before, what=f"failed after {k}")
            g.propagate(circ)
        o = oracle_sum(nq, *before)
        o.propagate(oracle_channels(circ), None)
        assert_same_terms(g.download(), oracle_arrays(o), what=f"after {k}")
