"""The measured cases: what programs that use this package have it do, through its public calls.

A case is one whole user call or loop: a sum goes in from host arrays (or stays on the device, for
a readout), a circuit is propagated layer by layer under a truncation policy, and the readout and
the terms come back.  The circuits are the package's own workloads (``paulistrings_b200.workloads``:
transverse-field Ising quenches, the open XXZ chain, layers of random two-qubit rotations) and
Clifford-plus-rotation bricks; the seed sets fields, angles and observables, so that another seed
is another run of a parameter sweep.
"""

import math
import sys
from pathlib import Path

import numpy as np
import torch

sys.path.insert(0, str(Path.cwd() / "paulistrings-rs_b200"))

import paulistrings_b200 as ps  # noqa: E402
from paulistrings_b200 import learned, truncation, workloads  # noqa: E402


def listed():
    return [
        # a first script: a 16-site lattice, a dictionary of labels in, a number out (latency of a call)
        {"name": "quench16_host_f64", "kind": "host", "family": "tfim", "L": 4, "steps": 2, "weight": 4},
        # the 36-site lattice under a coefficient threshold, one point of a field sweep
        {"name": "quench36_coeff_f64", "kind": "run", "family": "tfim", "L": 6, "steps": 5, "eps": 1e-5, "dtype": "f64",
         "rows": 400000},
        # the same with depolarizing noise after each step, in single precision
        {"name": "quench36_noisy_f32", "kind": "run", "family": "tfim", "L": 6, "steps": 5, "eps": 1e-5, "dtype": "f32",
         "noise": 1e-3, "rows": 400000},
        # a 64-site quench under a term budget, read out after every step
        {"name": "quench64_topn1M_f64", "kind": "series", "family": "tfim", "L": 8, "steps": 6, "cap": 1000003,
         "dtype": "f64"},
        # the same under a learned budget: a scorer ranks the terms, its predictions carried between rescorings
        {"name": "quench64_scored200k_f32", "kind": "series", "family": "tfim", "L": 8, "steps": 6, "cap": 200003,
         "dtype": "f32", "scored": True},
        # a wide register (four words per key half): the spread of one spin in a 256-site chain
        {"name": "xxz256_topn50k_f64", "kind": "series", "family": "xxz", "L": 256, "steps": 8, "cap": 50000,
         "dtype": "f64"},
        # the widest budget: dense random two-qubit layers, 2^26 terms, the whole sum brought back
        {"name": "pairs64_topn64M_f64", "kind": "run", "family": "pairs", "L": 64, "steps": 3, "terms": 65536,
         "cap": 1 << 26, "eps": 1e-10, "dtype": "f64"},
        # a middle budget on two words, forward in time, single precision, an odd register and budget
        {"name": "pairs101_topn3M_f32", "kind": "run", "family": "pairs", "L": 101, "steps": 3, "terms": 30011,
         "cap": 3000017, "dtype": "f32", "direction": "forward"},
        # Clifford gates, unitaries and rotations in one circuit (the tables that are not rotations)
        {"name": "clifford40_weight_f64", "kind": "run", "family": "clifford", "L": 40, "steps": 2, "terms": 20000,
         "eps": 1e-4, "weight": 12, "dtype": "f64", "rows": 1000000},
        # terms collected elsewhere, unsorted and with repeats, made into a sum
        {"name": "ingest_1500k_w2", "kind": "ingest", "L": 127, "terms": 1500007, "dtype": "f64"},
        # one readout of a resident sum in a product state
        {"name": "readout_5M_w1", "kind": "readout", "L": 60, "terms": 5000011, "dtype": "f64"},
        # one training batch of the scorer: forward and backward, loss and gradients back
        {"name": "scorer_gradients_16k", "kind": "gradients", "L": 64, "terms": 16384},
    ]


def draw(rng):
    def spread(lo, hi):
        return int(math.exp(rng.uniform(math.log(lo), math.log(hi))))

    dtype = rng.choice(["f64", "f64", "f32"])
    what = rng.choice(["host", "coeff", "noisy", "topn", "topn", "scored", "xxz", "pairs", "pairs", "clifford",
                       "ingest", "readout", "gradients"])
    if what == "host":
        return {"kind": "host", "family": "tfim", "L": rng.randint(3, 5), "steps": rng.randint(1, 2),
                "weight": rng.randint(2, 7)}
    if what in ("coeff", "noisy"):
        c = {"kind": "run", "family": "tfim", "L": rng.randint(4, 7), "steps": rng.randint(2, 5),
             "eps": 10 ** rng.uniform(-5, -3), "dtype": dtype, "rows": 4000000}
        if what == "noisy":
            c["noise"] = 10 ** rng.uniform(-4, -2)
        return c
    if what in ("topn", "scored"):
        c = {"kind": "series", "family": "tfim", "L": rng.randint(5, 8), "steps": rng.randint(2, 6),
             "cap": spread(1000, 2000000), "dtype": dtype}
        if what == "scored":
            c.update({"scored": True, "dtype": "f32"})
        return c
    if what == "xxz":
        return {"kind": "series", "family": "xxz", "L": rng.randint(20, 256), "steps": rng.randint(3, 8),
                "cap": spread(1000, 200000), "dtype": dtype}
    if what == "pairs":
        return {"kind": "run", "family": "pairs", "L": rng.randint(24, 200), "steps": rng.randint(1, 3),
                "terms": spread(1000, 60000), "cap": spread(20000, 20000000), "dtype": dtype,
                "direction": rng.choice(["forward", "heisenberg"]), "approx": rng.random() < 0.25}
    if what == "clifford":
        return {"kind": "run", "family": "clifford", "L": rng.randint(6, 100), "steps": rng.randint(1, 2),
                "terms": spread(500, 20000), "eps": 10 ** rng.uniform(-4, -2), "weight": rng.randint(6, 14),
                "dtype": dtype, "rows": 4000000}
    if what == "ingest":
        return {"kind": "ingest", "L": rng.randint(40, 250), "terms": spread(1000, 1500000), "dtype": dtype}
    if what == "readout":
        return {"kind": "readout", "L": rng.randint(10, 250), "terms": spread(1000, 5000000), "dtype": dtype}
    return {"kind": "gradients", "L": rng.randint(10, 64), "terms": spread(256, 16384)}


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------

def _random_terms(rng, qubits, count):
    """Distinct random strings of weight 1-4 (as the package's random observable) and normal
    coefficients; as many as there are when the register has fewer than ``count``."""
    W = ps.width_for(qubits)
    extra = 2 * count + 64
    x = np.zeros((extra, W), np.uint64)
    z = np.zeros((extra, W), np.uint64)
    weight = rng.integers(1, 5, extra)
    rows = np.arange(extra)
    for k in range(4):
        on = weight > k
        q = rng.integers(0, qubits, extra)
        p = rng.integers(1, 4, extra)
        bit = np.uint64(1) << (q % 64).astype(np.uint64)
        for arr, has in ((x, (p & 1) != 0), (z, (p & 2) != 0)):
            m = on & has
            arr[rows[m], q[m] // 64] |= bit[m]
    keys = np.concatenate([x, z], axis=1)
    order = np.lexsort(keys.T[::-1])
    s = keys[order]
    first = np.ones(extra, bool)
    first[1:] = (s[1:] != s[:-1]).any(axis=1)
    keep = np.zeros(extra, bool)
    keep[order] = first
    pick = np.nonzero(keep)[0][:count]
    x, z = x[pick], z[pick]
    c = rng.normal(size=len(x))
    return np.ascontiguousarray(x), np.ascontiguousarray(z), c / np.linalg.norm(c)


def _collected_terms(rng, qubits, count):
    """``count`` rows in no order, a fifth of them repeats of the others."""
    x, z, _ = _dense_terms(rng, qubits, count - count // 5)
    x[:, 0] ^= np.uint64(1) << np.uint64(min(qubits, 64) - 1)  # and some X there
    pick = rng.permutation(np.concatenate([np.arange(len(x)), rng.integers(0, len(x), count - len(x))]))
    return np.ascontiguousarray(x[pick]), np.ascontiguousarray(z[pick]), rng.normal(size=count)


def _dense_terms(rng, qubits, count):
    """Strings that are mostly Z and identity, as a sum read out in a product state is."""
    W = ps.width_for(qubits)
    live = np.array([(1 << max(0, min(64, qubits - 64 * w))) - 1 for w in range(W)], np.uint64)
    z = rng.integers(0, 1 << 63, (count, W), dtype=np.uint64) * np.uint64(2) + rng.integers(0, 2, (count, W), dtype=np.uint64)
    x = np.zeros((count, W), np.uint64)
    hit = rng.random(count) < 0.5
    q = rng.integers(0, qubits, count)
    x[np.nonzero(hit)[0], q[hit] // 64] = np.uint64(1) << (q[hit] % 64).astype(np.uint64)
    return x, np.ascontiguousarray(z & live), rng.normal(size=count)


def _clifford_bricks(rng, n, steps):
    c = ps.Circuit(n)
    for s in range(steps):
        perm = rng.permutation(n)
        for k in range(n // 2):
            a, b = int(perm[2 * k]), int(perm[2 * k + 1])
            kind = rng.integers(0, 4)
            if kind == 0:
                c.cnot(a, b)
            elif kind == 1:
                c.cz(a, b)
            elif kind == 2:
                c.swap(a, b)
            else:
                c.h(a)
                c.cnot(a, b)
                c.s(b)
        for q in rng.choice(n, size=max(1, n // 4), replace=False):
            c.rz(math.pi / 4, int(q))
        a, b = (int(v) for v in rng.choice(n, size=2, replace=False))
        g = rng.normal(size=(4, 4)) + 1j * rng.normal(size=(4, 4))
        u, r = np.linalg.qr(g)
        c.unitary_2q(a, b, u * (np.diag(r) / np.abs(np.diag(r))))
    return c


def _circuit(case, rng):
    """(circuit of one propagate call, number of calls, qubits)."""
    if case["family"] == "tfim":
        L, h = case["L"], float(rng.uniform(0.95, 1.05))
        steps = 1 if case["kind"] == "series" else case["steps"]
        return workloads.tfim_2d(L, steps, J=1.0, h=h, dt=0.1, noise_p=case.get("noise")), L * L
    if case["family"] == "xxz":
        return workloads.xxz_chain(case["L"], 1, Jz=float(rng.uniform(0.45, 0.55)), dt=0.1), case["L"]
    if case["family"] == "pairs":
        return workloads.random_pair_layers(case["L"], case["steps"], seed=int(rng.integers(1 << 60))), case["L"]
    return _clifford_bricks(rng, case["L"], case["steps"]), case["L"]


def _observable(case, rng, qubits):
    W = ps.width_for(qubits)
    if case["family"] == "tfim":
        labels = workloads.tfim_magnetization(case["L"], "X")
        xz = [ps.parse_label(k, W) for k in labels]
        return np.stack([v[0] for v in xz]), np.stack([v[1] for v in xz]), np.array(list(labels.values()))
    if case["family"] == "xxz":
        x, z = np.zeros((1, W), np.uint64), np.zeros((1, W), np.uint64)
        q = qubits // 2
        z[0, q // 64] = np.uint64(1) << np.uint64(q % 64)
        return x, z, np.ones(1)
    return _random_terms(rng, qubits, case["terms"])


def _policy(case, scorer):
    pol = None
    for kind, make in (("cap", truncation.approx_topn if case.get("approx") else truncation.topn),
                       ("eps", truncation.coeff), ("weight", truncation.weight)):
        if kind not in case:
            continue
        if kind == "cap" and scorer is not None:
            p = truncation.scored_topn(case["cap"], scorer, rescore_every=scorer.layers_per_unit)
        else:
            p = make(case[kind])
        pol = p if pol is None else pol & p
    return pol


def _readout_state(case, qubits):
    if case["family"] == "xxz":
        return workloads.neel_state(qubits)
    return "x+" if case["family"] == "tfim" else "z+"


def _pinned(rows, W):
    x = torch.zeros((rows, W), dtype=torch.int64, pin_memory=True).numpy().view(np.uint64)
    z = torch.zeros((rows, W), dtype=torch.int64, pin_memory=True).numpy().view(np.uint64)
    return x, z, torch.zeros(rows, dtype=torch.float64, pin_memory=True).numpy()


def _scorer_rows(case, rng):
    W = ps.width_for(case["L"])
    n = case["terms"]
    live = np.uint64((1 << case["L"]) - 1)
    x = rng.integers(0, 1 << 63, (n, W), dtype=np.uint64) & rng.integers(0, 1 << 63, (n, W), dtype=np.uint64) & live
    z = rng.integers(0, 1 << 63, (n, W), dtype=np.uint64) & rng.integers(0, 1 << 63, (n, W), dtype=np.uint64) & live
    logc = rng.uniform(-12, -2, n).astype(np.float32)
    rem = rng.integers(1, 20, n).astype(np.float32)
    return learned.pack_keys(x, z), logc, rem, (logc - rng.exponential(2.0, n)).astype(np.float32)


def _scorer_params(case, rng):
    """Weights of a scorer part way through its training (trained weights are of this size)."""
    lay = learned.layout(case["L"])
    p = np.zeros(lay["total"], np.float32)
    for name, scale in (("embed", 0.1), ("u", 0.1), ("b1", 0.1), ("w2", 1 / math.sqrt(128)), ("b2", 0.1), ("w3", 0.1)):
        p[lay[name]] = rng.normal(scale=scale, size=lay[name].stop - lay[name].start)
    return p


def prepare(case, seed):
    rng = np.random.default_rng(seed)
    kind = case["kind"]
    if kind == "gradients":
        sc = learned.Scorer(case["L"], layers_per_unit=96.0, seed=1)
        sc.set_params(_scorer_params(case, rng))
        return {"case": case, "scorer": sc, "rows": _scorer_rows(case, rng)}
    if kind == "ingest":
        x, z, c = _collected_terms(rng, case["L"], case["terms"])
        return {"case": case, "x": x, "z": z, "c": c}
    if kind == "readout":
        g = ps.GpuPauliSum(case["L"], case["dtype"])
        g.upload(*_dense_terms(rng, case["L"], case["terms"]))
        state = "".join("01"[b] for b in rng.integers(0, 2, case["L"]))
        return {"case": case, "g": g, "state": state}
    circuit, qubits = _circuit(case, rng)
    x, z, c = _observable(case, rng, qubits)
    st = {"case": case, "circuit": circuit, "state": _readout_state(case, qubits),
          "direction": case.get("direction", "heisenberg")}
    if kind == "host":
        st["obs"] = ps.PauliSum.from_arrays(x, z, c, qubits)
        st["policy"] = _policy(case, None)
        return st
    scorer = None
    if case.get("scored"):
        scorer = learned.Scorer(qubits, layers_per_unit=len(circuit), seed=int(rng.integers(1 << 30)), residual=True)
    st.update({"g": ps.GpuPauliSum(qubits, case["dtype"]), "x": x, "z": z, "c": c, "policy": _policy(case, scorer)})
    # a program that knows its budget keeps pinned buffers for the result (rows past it stay zero)
    st["out"] = _pinned(case.get("cap") or case["rows"], ps.width_for(qubits))
    return st


# ---------------------------------------------------------------------------
# one pass
# ---------------------------------------------------------------------------

def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "gradients":
        keys, logc, rem, target = state["rows"]
        grads, loss = state["scorer"].gradients(keys, logc, rem, target)
        return {"grads": grads, "loss": loss}
    if kind == "ingest":
        s = ps.PauliSum.from_arrays(state["x"], state["z"], state["c"], case["L"], dtype=case["dtype"])
        return _terms(s.x_array(), s.z_array(), s.coefficients_array())
    if kind == "readout":
        return state["g"].expectation(state["state"])
    if kind == "host":
        s = ps.propagated(state["obs"], state["circuit"], state["policy"], state["direction"])
        value = s.expectation(state["state"])
        return {"value": value, **_terms(s.x_array(), s.z_array(), s.coefficients_array())}
    g = state["g"]
    g.upload(state["x"], state["z"], state["c"])
    steps = case["steps"] if kind == "series" else 1
    values = []
    for k in range(steps):
        g.propagate(state["circuit"], state["policy"], state["direction"],
                    remaining_layers=len(state["circuit"]) * (steps - k))
        values.append(g.expectation(state["state"]))
    g.download(out=state["out"])
    return {"values": np.array(values), "terms": len(g), **_terms(*state["out"])}


def _terms(x, z, c):
    return {"x": x.view(np.int64), "z": z.view(np.int64), "c": c}


# ---------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------

# mean terms entering a layer of the threshold runs, as a power of the run's inverse threshold and
# size (fitted to the lattices above; the budgets' runs count the budget over the layers they fill)
def _mean_terms(case):
    if "cap" in case:
        return case["cap"] * (0.35 if case["family"] == "xxz" else 0.5)
    if case["family"] == "clifford":
        return case["terms"] * 4
    if "eps" not in case:
        return 2000
    return case["L"] ** 2 * 20 * case["steps"] * (1e-3 / case["eps"]) ** 0.3


def work(case):
    kind = case["kind"]
    if kind == "gradients":
        n, H = case["terms"], 128
        return {"bytes": n * 28 + 4 * learned.layout(case["L"])["total"], "flops": n * (6 * H * H + 4 * case["L"] * H)}
    row = 16 * ps.width_for(case["L"] ** 2 if case.get("family") == "tfim" else case["L"])
    coef = 4 if case.get("dtype") == "f32" else 8
    if kind == "ingest":
        return {"bytes": case["terms"] * 2 * (row + 8), "flops": 0}
    if kind == "readout":
        return {"bytes": case["terms"] * (row + coef), "flops": 0}
    per_step = {"tfim": 3 * case["L"] ** 2 * (4 / 3 if case.get("noise") else 1), "xxz": 3 * (case["L"] - 1) * 0.2,
                "pairs": 1.5 * case["L"], "clifford": 0.9 * case["L"]}[case["family"]]
    return {"bytes": per_step * case["steps"] * _mean_terms(case) * 2 * (row + coef), "flops": 0}


def tolerance(case):
    if case["kind"] == "gradients":
        return {"rel": 1e-2, "max": 0.3}  # bf16 operands, f32 sums
    if case["kind"] == "readout":
        # a sum of coefficients of both signs in another order: 64-bit rounding over the largest partial sums
        return {"rel": 1e-10 if case["dtype"] == "f64" else 1e-9}
    # Every product and two-term sum rounds once, in the same order in every correct version, so the
    # strings are the same and the coefficients equal up to the readout's summation order.
    return {"rel": 1e-11 if case.get("dtype", "f64") == "f64" else 1e-6, "max": 1e-9 if case.get("dtype", "f64") == "f64" else 1e-5,
            "differ": 0.0}


# ---------------------------------------------------------------------------
# the same in plain numpy, 64 bits
# ---------------------------------------------------------------------------

def _merged(keys, c):
    """Equal rows summed, exact zeros dropped, sorted by key."""
    order = np.lexsort(keys.T[::-1])
    k, v = keys[order], c[order]
    first = np.ones(len(k), bool)
    first[1:] = (k[1:] != k[:-1]).any(axis=1)
    at = np.nonzero(first)[0]
    s = np.add.reduceat(v, at) if len(at) else v
    keep = s != 0
    return k[at][keep], s[keep]


def _value(keys, c, state, qubits):
    W = ps.width_for(qubits)
    ax, az, neg = ps.product_basis(state, qubits, W)
    x, z = keys[:, :W], keys[:, W:]
    sup = x | z
    ok = ~(((x ^ (sup & ax)) | (z ^ (sup & az))).any(axis=1))
    odd = np.bitwise_count(sup & neg).sum(axis=1) & 1
    return float(np.sum(np.where(odd[ok] == 1, -c[ok], c[ok])))


def _rotated(keys, c, paulis, qubits, theta, W):
    """A rotation layer read backwards: k -> cos c k + sin c (i G k), for the terms that anticommute with G."""
    g = np.zeros(2 * W, np.uint64)
    for p, q in zip(paulis, qubits):
        bit = np.uint64(1) << np.uint64(q % 64)
        if p in "XY":
            g[q // 64] |= bit
        if p in "ZY":
            g[W + q // 64] |= bit
    gx, gz = g[:W], g[W:]
    x, z = keys[:, :W], keys[:, W:]
    count = lambda a: np.bitwise_count(a).sum(axis=-1).astype(np.int64)  # noqa: E731
    anti = (count((x & gz) ^ (z & gx)) & 1).astype(bool)
    xa, za = x[anti], z[anti]
    # the power of i in (term)(G), each written as i^(#Y) X^x Z^z
    phase = (2 * count(za & gx) + count(xa & za) + int(count(gx & gz)) - count((xa ^ gx) & (za ^ gz)) + 1) & 3
    sign = np.where(phase & 2, -1.0, 1.0)
    s, co = math.sin(-theta), math.cos(theta)
    own = np.where(anti, c * co, c)
    return _merged(np.concatenate([keys, keys[anti] ^ g]), np.concatenate([own, sign * c[anti] * s]))


def _gradients64(case, params, keys, logc, rem, target):
    """The scorer's loss and gradients with its stored (bfloat16) weights, in 64 bits."""
    H, nq = 128, case["L"]
    lay = learned.layout(nq)
    p = torch.from_numpy(params).to(torch.bfloat16).to(torch.float64)
    part = {k: p[v].clone().requires_grad_(True) for k, v in lay.items() if k != "total"}
    W = ps.width_for(nq)
    q = np.arange(nq)
    bit = lambda a: (a[:, q // 64] >> (q % 64).astype(np.uint64)) & np.uint64(1)  # noqa: E731
    pauli = torch.from_numpy((bit(keys[:, :W]) | (bit(keys[:, W:]) << np.uint64(1))).astype(np.int64))
    hot = torch.stack([pauli == k for k in (1, 2, 3)], dim=2).reshape(len(keys), -1).to(torch.float64)
    f = torch.stack([(pauli != 0).sum(1).to(torch.float64), torch.from_numpy(logc).double(),
                     torch.from_numpy(rem).double()], dim=1) * torch.tensor([0.1, 0.1, 0.1], dtype=torch.float32).double()
    gelu = lambda v: 0.5 * v * (1 + torch.tanh(0.7978845608028654 * (v + 0.044715 * v ** 3)))  # noqa: E731
    z1 = hot @ part["embed"].reshape(-1, H) + f @ part["u"].reshape(3, H) + part["b1"]
    y = part["b3"] + gelu(gelu(z1) @ part["w2"].reshape(H, H) + part["b2"]) @ part["w3"]
    loss = ((y - torch.from_numpy(target).double()) ** 2).mean()
    loss.backward()
    return {"grads": torch.cat([part[k].grad.reshape(-1) for k in lay if k != "total"]).numpy(), "loss": loss.item()}


def exact(case, seed):
    rng = np.random.default_rng(seed)
    kind = case["kind"]
    if kind == "gradients":
        params = _scorer_params(case, rng)
        return _gradients64(case, params, *_scorer_rows(case, rng))
    if kind == "ingest":
        x, z, c = _collected_terms(rng, case["L"], case["terms"])
        c = c.astype(np.float32).astype(np.float64) if case["dtype"] == "f32" else c
        return {"x": None, "z": None, "c": _merged(np.concatenate([x, z], axis=1), c)[1]}
    if kind == "readout":
        x, z, c = _dense_terms(rng, case["L"], case["terms"])
        c = c.astype(np.float32).astype(np.float64) if case["dtype"] == "f32" else c
        state = "".join("01"[b] for b in rng.integers(0, 2, case["L"]))
        return _value(np.concatenate([x, z], axis=1), c, state, case["L"])
    if kind != "host":
        return None  # thousands of sorted layers: more than 20 seconds in numpy
    circuit, qubits = _circuit(case, rng)
    x, z, c = _observable(case, rng, qubits)
    W = ps.width_for(qubits)
    keys, c = _merged(np.concatenate([x, z], axis=1), c)
    for ch in reversed(list(circuit)):
        keys, c = _rotated(keys, c, ch.paulis, ch.qubits, ch.theta, W)
        keep = np.bitwise_count(keys[:, :W] | keys[:, W:]).sum(axis=1) <= case["weight"]
        keys, c = keys[keep], c[keep]
    return {"value": _value(keys, c, _readout_state(case, qubits), qubits), "x": None, "z": None, "c": c}
