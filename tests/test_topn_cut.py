"""TopN cut in place between rotation layers, against the oracle.

When the last boundary is known and a pass drops little, the rows a TopN pass drops stay in the
merge's slots and the next layer reads around them.  Per-kernel profiling keeps small sums on the
per-layer kernels, so these sizes reach the cut: budgets around a tile's rows, layers with few and
many partners, ties that the budget cuts (the pass compacts instead), magnitudes far apart (the
boundary leaves the window), a budget no layer reaches, and a failure between two such layers.
"""

from __future__ import annotations

import numpy as np
import pytest

import paulistrings_b200 as ps
from paulistrings_b200 import _lib, truncation, workloads

from _util import assert_same_terms, oracle_arrays, oracle_channels, oracle_policy, oracle_sum

pytestmark = pytest.mark.gpu


def _inputs(nq, count, seed, values="normal"):
    x, z, c = workloads.random_observable(nq, count, seed=seed)
    rng = np.random.default_rng(seed)
    if values == "few":
        c = rng.choice([0.25, -0.25, 0.5, 0.125], size=count)
    elif values == "wide":
        c = c * 2.0 ** rng.integers(-40, 40, count)
    return x, z, c


def _compare(nq, dtype, arrays, circ, pol, direction="heisenberg"):
    g = ps.GpuPauliSum(nq, dtype)
    g.set_profiling(True)
    g.upload(*arrays)
    st = g.propagate(circ, pol, direction, with_stats=True)
    o = oracle_sum(nq, *arrays, dtype)
    after = o.propagate(oracle_channels(circ), oracle_policy(pol), direction)
    assert st.terms_after == [int(v) for v in after]
    assert_same_terms(g.download(), oracle_arrays(o), what=f"cut {nq} {dtype}")
    return g.read_profile(), len(circ)


@pytest.mark.parametrize("dtype", ["f64", "f32"])
@pytest.mark.parametrize("nq,cap", [(20, 1279), (20, 1281), (24, 30000), (64, 20011), (100, 1291), (100, 30011),
                                    (200, 769), (200, 9001)])
@pytest.mark.parametrize("values", ["normal", "few", "wide"])
def test_cut_layers(nq, cap, dtype, values):
    arrays = _inputs(nq, min(cap, 4000), cap, values)
    circ = workloads.random_pair_layers(nq, 3 if nq < 100 else 2, seed=cap)
    prof, layers = _compare(nq, dtype, arrays, circ, truncation.topn(cap))
    if values == "normal" and nq <= 24:
        assert prof["k_topn_compact"]["launches"] < layers  # some passes compacted nothing


@pytest.mark.parametrize("dtype", ["f64", "f32"])
def test_cut_with_threshold_and_dense_partners(dtype):
    """A quench: every generator splits a large share of the terms, many equal pairs, rows dropped by
    the threshold beside the cut."""
    nq = 16
    circ = workloads.tfim_2d(4, 4, J=1.0, h=1.0, dt=0.3)
    labels = workloads.tfim_magnetization(4, "X")
    x = np.array([ps.parse_label(k, 1)[0] for k in labels], np.uint64)
    z = np.array([ps.parse_label(k, 1)[1] for k in labels], np.uint64)
    c = np.array(list(labels.values()))
    prof, layers = _compare(nq, dtype, (x, z, c), circ, truncation.topn(20000) & truncation.coeff(1e-9))
    assert prof["k_topn_compact"]["launches"] < layers


def test_a_failure_between_cut_layers_keeps_the_last_completed_layer():
    """Allocations that fail after k successes stop the run at different layers, before a layer or
    before its pass; the store, cut, slotted or compacted, is that of the last one that completed."""
    nq, cap = 20, 6000
    arrays = _inputs(nq, 3000, 77)
    circ = workloads.random_pair_layers(nq, 2, seed=7)
    pol = truncation.topn(cap)
    order = list(circ)[::-1]
    states, applied = [], []
    o = oracle_sum(nq, *arrays)
    states.append(oracle_arrays(o))
    for ch in order:
        one = ps.Circuit(nq)
        one.append(ch)
        layer = oracle_sum(nq, *states[-1])
        layer.propagate(oracle_channels(one), None, "heisenberg")
        applied.append(oracle_arrays(layer))
        o.propagate(oracle_channels(one), oracle_policy(pol), "heisenberg")
        states.append(oracle_arrays(o))
    stopped = 0
    for k in range(0, 60, 3):
        g = ps.GpuPauliSum(nq)
        g.set_profiling(True)
        g.upload(*arrays)
        _lib.check(_lib.lib().ps_inject_fault(g._h, _lib.PS_FAULT_OOM, k), g._h, "inject")
        try:
            g.propagate(circ, pol, "heisenberg")
        except MemoryError:
            stopped += 1
        _lib.check(_lib.lib().ps_inject_fault(g._h, _lib.PS_FAULT_NONE, 0), g._h, "disarm")
        n = len(g)
        got = g.download()
        assert n == len(got[2])
        assert any(len(s[2]) == n and all(np.array_equal(p, q) for p, q in zip(got, s)) for s in states + applied), k
    assert stopped > 3
