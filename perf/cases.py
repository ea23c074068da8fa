"""Performance cases: the work a program has the engine do, through its public entry points.

Each case is a dict of plain values.  ``listed()`` gives one case per kind of work, ``draw``
another one of the same kinds with its sizes spread over the range the listed one stands for.
``prepare`` makes what a program holds before the call (packed gate lists, terms, networks),
``run`` is one pass and returns everything it computes: terms (bit planes as 64-bit words and
FP64 coefficients), live counts, expectation values, gradients, parameters.  ``exact`` gives
the values of a pass in 64 bits from plain numpy, where they can be had in seconds.

The kinds:

chain          a small open transverse-field Ising chain from one Z, start to end on one sum
calls          the same physics through one method call per gate, as an interactive program
kicked         2D kicked Ising with a weight cap, start to end on one sum (the headline)
clifford_t     random Clifford+T brickwork on up to 64 qubits, where terms hardly merge
noise          a noisy 2D circuit: rotations, depolarising and Pauli errors, amplitude damping
lossy          a circuit with atom loss on lossy words: rotations, CZ, the three loss channels
batch          hundreds of uneven chains advanced together, built from host circuits each time
kicked_layer   one kicked-Ising layer on a sum of millions of terms
trotter_layer  one generic-angle 2D Trotter layer (gate-by-gate rotations) on a large sum
budget         term-budget truncation of a large sum by a network's score
readout        overlap, trace, expectation, weights and equality of two large sums
train          the priority network: training epochs, a gradient, predictions
"""

import math
import random

import numpy as np
import torch

from ppvm_b200 import gates as G
from ppvm_b200.batch import Instance, PauliSumBatch
from ppvm_b200.circuits import lattice_bonds
from ppvm_b200.learned import N_PARAMS, TermPriorityNet
from ppvm_b200.paulisum import OP_DTYPE, GateList, LossyPauliSum, PauliSum
from ppvm_b200.sharded import DeviceShare

HALF_PI = math.pi / 2
OP_BYTES = OP_DTYPE.itemsize


def listed():
    return [
        # the configuration the repository names for a CPU-sized chain; at most some 800 terms
        {"name": "chain_20", "kind": "chain", "qubits": 20, "steps": 10, "threshold": 1e-4},
        # a loop of single-gate calls on a few dozen terms: launches and latency only
        {"name": "gate_calls_12", "kind": "calls", "qubits": 12, "steps": 2, "threshold": 1e-5},
        # the headline: 12 x 12 lattice, 20 layers, weight cap 10
        {"name": "kicked_12x12", "kind": "kicked", "side": 12, "layers": 20, "threshold": 1e-5, "cap": 10},
        # Clifford+T in its spread-out regime, three T gates a layer
        {"name": "clifford_t_64", "kind": "clifford_t", "qubits": 64, "layers": 10, "threshold": 1e-6},
        # a noisy lattice of odd side (one plane word, 49 qubits)
        {"name": "noise_7x7", "kind": "noise", "side": 7, "layers": 5, "threshold": 2e-5, "cap": 8},
        # atom loss on a register of 40 sites
        {"name": "lossy_40", "kind": "lossy", "qubits": 40, "layers": 4, "threshold": 1e-5, "cap": 7},
        # the 256-instance serving batch
        {"name": "batch_256", "kind": "batch", "count": 256, "threshold": 1e-5},
        # the largest sums: millions of terms on 144 qubits (three plane words)
        {"name": "kicked_layer_4m", "kind": "kicked_layer", "side": 12, "terms": 4000000, "threshold": 1e-7, "cap": 12},
        # gate-by-gate rotations, 81 qubits (two plane words)
        {"name": "trotter_layer_500k", "kind": "trotter_layer", "side": 9, "terms": 500000, "threshold": 1e-6, "cap": 10},
        # 2 million terms cut to the budget of one million
        {"name": "budget_2m", "kind": "budget", "side": 10, "terms": 2000000, "budget": 1000000, "digit_bits": 8},
        # two sums of a million terms that share half of their words
        {"name": "readout_1m", "kind": "readout", "qubits": 100, "terms": 1000000},
        # the network's training set and minibatch as the learned-truncation study uses them
        {"name": "train_16k", "kind": "train", "samples": 16384, "batch": 512, "epochs": 4},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["chain", "calls", "kicked", "clifford_t", "noise", "lossy", "batch", "kicked_layer",
                       "trotter_layer", "budget", "readout", "train"])
    if kind == "chain":
        return {"kind": kind, "qubits": rng.randint(8, 40), "steps": rng.randint(4, 10),
                "threshold": round(math.exp(rng.uniform(math.log(1e-4), math.log(1e-3))), 6)}
    if kind == "calls":
        return {"kind": kind, "qubits": rng.randint(5, 12), "steps": rng.randint(1, 2),
                "threshold": round(math.exp(rng.uniform(math.log(1e-5), math.log(1e-3))), 7)}
    if kind == "kicked":
        return {"kind": kind, "side": rng.randint(6, 12), "layers": rng.randint(8, 20),
                "threshold": round(math.exp(rng.uniform(math.log(1e-5), math.log(1e-4))), 7), "cap": rng.randint(7, 10)}
    if kind == "clifford_t":
        return {"kind": kind, "qubits": rng.randint(33, 64), "layers": rng.randint(5, 9), "threshold": 1e-6}
    if kind == "noise":
        return {"kind": kind, "side": rng.randint(4, 7), "layers": rng.randint(3, 5),
                "threshold": round(math.exp(rng.uniform(math.log(2e-5), math.log(2e-4))), 7), "cap": rng.randint(6, 8)}
    if kind == "lossy":
        return {"kind": kind, "qubits": rng.randint(17, 40), "layers": rng.randint(2, 4),
                "threshold": round(math.exp(rng.uniform(math.log(1e-5), math.log(1e-4))), 7), "cap": rng.randint(5, 7)}
    if kind == "batch":
        return {"kind": kind, "count": _log_int(rng, 16, 250), "threshold": 1e-5}
    if kind == "kicked_layer":
        return {"kind": kind, "side": rng.randint(11, 12), "terms": _log_int(rng, 50000, 3900000), "threshold": 1e-7,
                "cap": 12}
    if kind == "trotter_layer":
        return {"kind": kind, "side": rng.randint(8, 9), "terms": _log_int(rng, 20000, 490000), "threshold": 1e-6,
                "cap": 10}
    if kind == "budget":
        terms = _log_int(rng, 30000, 1900000)
        return {"kind": kind, "side": rng.randint(9, 12), "terms": terms, "budget": int(terms * rng.uniform(0.1, 0.9)),
                "digit_bits": rng.choice([8, 11])}
    if kind == "readout":
        return {"kind": kind, "qubits": rng.randint(30, 190), "terms": _log_int(rng, 1000, 900000)}
    return {"kind": kind, "samples": _log_int(rng, 1000, 16000), "batch": rng.choice([256, 512, 777]),
            "epochs": rng.randint(1, 4)}


# ---- gate lists ---------------------------------------------------------------------------


def _pack(rows):
    """``(code, q0, q1, value, (p0, p1, p2))`` rows as the packed records of the C ABI."""
    arr = np.zeros(len(rows), dtype=OP_DTYPE)
    code, q0, q1, val, p = zip(*rows)
    arr["code"], arr["q0"], arr["q1"], arr["theta"], arr["p"] = code, q0, q1, val, p
    return GateList(arr)


def _z_word(n, q):
    return "I" * q + "Z" + "I" * (n - 1 - q)


def _chain_ops(n, steps, tzz, tx):
    """Heisenberg list of an open chain: RX everywhere, TRUNCATE, RZZ on every bond, TRUNCATE."""
    step = [G.r1(G.RX, i, tx) for i in reversed(range(n))] + [G.truncate()]
    step += [G.r2(G.RZZ, i, i + 1, tzz) for i in reversed(range(n - 1))] + [G.truncate()]
    return step * steps


def _chain_list(n, steps, tzz, tx):
    """``_chain_ops`` packed, one step written and repeated."""
    return GateList(np.tile(_pack(_chain_ops(n, 1, tzz, tx)).arr, steps))


def _angles(case, seed):
    """Seeded angles near the nominal ones (within two percent)."""
    r = random.Random(1000003 * seed + 17)
    return lambda nominal: nominal * r.uniform(0.98, 1.02)


def _kicked_layers(side, angles):
    n, bonds = side * side, lattice_bonds(side)
    zz = [G.r2(G.RZZ, a, b, -HALF_PI) for a, b in reversed(bonds)] + [G.truncate()]
    return [zz + [G.r1(G.RX, q, t) for q in reversed(range(n))] + [G.truncate()] for t in angles]


def _trotter_layer(side, tzz, tx):
    n, bonds = side * side, lattice_bonds(side)
    ops = [G.r1(G.RX, q, tx) for q in reversed(range(n))] + [G.truncate()]
    for i, (a, b) in enumerate(reversed(bonds)):  # a TRUNCATE per row of bonds keeps the peak near the end's size
        ops += [G.r2(G.RZZ, a, b, tzz)] + ([G.truncate()] if i % side == side - 1 else [])
    return ops + [G.truncate()]


def _clifford_t_ops(n, layers, seed):
    """Random one-qubit Cliffords, a CNOT brick and three T gates a layer, Heisenberg order, and
    an observable of 16 dense words (each T splits half of the terms: some 16 * 1.5^T at the end)."""
    r = random.Random(7919 * seed + 5)
    ops = []
    for layer in range(layers):
        ops += [G.r1(G.RZ, q, math.pi / 4) for q in r.sample(range(n), 3)] + [G.truncate()]
        ops += [G.g2(G.CNOT, a, a + 1) for a in range(layer % 2, n - 1, 2)]
        ops += [G.g1(r.choice((G.H, G.S, G.S_DAG)), q) for q in range(n)]
    return ops, ["".join(r.choice("IXYZ") for _ in range(n)) for _ in range(16)]


def _noise_ops(side, layers, t):
    n, bonds = side * side, lattice_bonds(side)
    tzz, tx = t(0.35), t(0.3)
    ops = []
    for _ in range(layers):
        ops += [G.amplitude_damping(q, 0.01) for q in range(0, n, 3)]
        ops += [G.depolarize1(q, 2e-3) for q in range(n)]
        ops += [G.r1(G.RX, q, tx) for q in range(n)] + [G.truncate()]
        for i, (a, b) in enumerate(bonds):
            ops += [G.depolarize2(a, b, 5e-3), G.r2(G.RZZ, a, b, tzz)]
            ops += [G.truncate()] if i % side == side - 1 else []
        ops += [G.truncate()] + [G.pauli_error(q, (1e-3, 5e-4, 2e-3)) for q in range(n)]
    return ops


def _lossy_ops(n, layers, t):
    ops = []
    for layer in range(layers):
        ops += [G.reset_loss_channel(q) for q in range((layer * 5) % n, n, max(1, n // 3))] + [G.truncate()]
        ops += [G.loss_channel(q, 0.02) for q in range(n)]
        ops += [G.r1(G.RX, q, t(0.4)) for q in range(n)] + [G.truncate()]
        ops += [G.g2(G.CZ, a, a + 1) for a in range(layer % 2, n - 1, 2)]
        ops += [G.correlated_loss_channel(a, a + 1, (0.01, 0.02, 0.05)) for a in range(layer % 2, n - 1, 6)]
        ops += [G.r2(G.RZZ, a, a + 1, t(0.5)) for a in range(1 - layer % 2, n - 1, 2)] + [G.truncate()]
    return ops


# ---- terms on the device ------------------------------------------------------------------


def _device_terms(s, room):
    """The sum's terms in order, as the first rows of device arrays for ``room`` terms (planes,
    coefficients; zeros after the last term), and their number; the sum is left empty."""
    n, m = len(s), np.zeros(s.W, dtype=np.uint64)
    if n > room:
        raise ValueError("%d terms, room for %d" % (n, room))
    rows, _ = DeviceShare(s).export(m, m, 1)
    out = torch.nn.functional.pad(rows.view(-1, 2 * s.W + 1), (0, 0, 0, room - n))
    return {"count": n, "planes": out[:, : 2 * s.W], "coefficients": out[:, 2 * s.W].view(torch.float64)}


def _host_terms(s, room):
    """The same from the host export, as numpy arrays."""
    x, z, c = s.export()
    n = len(c)
    if n > room:
        raise ValueError("%d terms, room for %d" % (n, room))
    pad = ((0, room - n), (0, 0))
    return {"count": n, "x": np.pad(x.view(np.int64), pad), "z": np.pad(z.view(np.int64), pad),
            "c": np.pad(c, (0, room - n))}


def _room(case):
    """Terms that a pass of the case can end with, rounded up generously."""
    kind = case["kind"]
    if kind in ("chain", "calls"):
        return 4096
    if kind == "kicked":
        return int(1e6 * max(0.1, 1e-5 / case["threshold"]))
    if kind == "clifford_t":
        return 1 << (case["layers"] + 13)
    if kind == "noise":
        return int(6e5 * max(0.1, 2e-5 / case["threshold"]))
    if kind == "lossy":
        return 200000
    if kind == "kicked_layer":
        return 5 * case["terms"] + 2500000
    return 24 * case["terms"] + 3000000  # trotter_layer


def _sum_of_rows(rows, n, capacity, **kw):
    """A sum that holds the given device rows (2W + 1 words a term)."""
    s = PauliSum(["I" * n], n, capacity=capacity, **kw)
    m = np.zeros(s.W, dtype=np.uint64)
    share = DeviceShare(s)
    share.export(m, m, 1)  # drops the placeholder term
    share.append(rows)
    return s


def _grown_rows(s, layers, terms):
    """The first ``terms`` rows of ``s`` once the layers, applied in turn, have made that many."""
    for layer in layers:
        s.run(layer)
        if len(s) >= terms:
            break
    if len(s) < terms:
        raise ValueError("the layers make only %d terms of %d" % (len(s), terms))
    m = np.zeros(s.W, dtype=np.uint64)
    rows, _ = DeviceShare(s).export(m, m, 1)
    return rows.view(-1, 2 * s.W + 1)[:terms].contiguous()


# ---- prepare ------------------------------------------------------------------------------


def prepare(case, seed):
    kind, st = case["kind"], {"case": case}
    t = _angles(case, seed)
    if kind == "chain":
        n = case["qubits"]
        st["ops"] = _chain_list(n, case["steps"], t(0.2), t(0.2))
        st["word"] = _z_word(n, n // 2)
    elif kind == "calls":
        st["tzz"], st["tx"] = t(0.2), t(0.2)
        st["word"] = _z_word(case["qubits"], case["qubits"] // 2)
    elif kind == "kicked":
        side = case["side"]
        st["ops"] = _pack(sum(_kicked_layers(side, [t(0.6)] * case["layers"]), []))
        st["word"] = _z_word(side * side, (side // 2) * side + side // 2)
    elif kind == "clifford_t":
        ops, st["words"] = _clifford_t_ops(case["qubits"], case["layers"], seed)
        st["ops"] = _pack(ops)
    elif kind == "noise":
        side = case["side"]
        st["ops"] = _pack(_noise_ops(side, case["layers"], t))
        st["word"] = _z_word(side * side, (side // 2) * side + side // 2)
    elif kind == "lossy":
        st["ops"] = _pack(_lossy_ops(case["qubits"], case["layers"], t))
        st["word"] = _z_word(case["qubits"], case["qubits"] // 2)
    elif kind == "batch":
        r = random.Random(31 * seed + 3)
        st["instances"] = []
        for _ in range(case["count"]):
            n, steps, h = r.randint(16, 128), r.randint(5, 30), r.uniform(0.5, 1.5)
            st["instances"].append(Instance(n, [(_z_word(n, n // 2), 1.0)], _chain_list(n, steps, 0.1, 0.1 * h),
                                            case["threshold"]))
    elif kind == "kicked_layer":
        side, terms = case["side"], case["terms"]
        n, q = side * side, (side // 2) * side + side // 2
        layers = [_pack(x) for x in _kicked_layers(side, [t(0.6)] * 40)]
        s = PauliSum([_z_word(n, q)], n, min_abs_coeff=case["threshold"], max_pauli_weight=case["cap"],
                     clifford_angles=True)
        rows = _grown_rows(s, layers, terms)
        st["base"] = _sum_of_rows(rows, n, _room(case), min_abs_coeff=case["threshold"], max_pauli_weight=case["cap"],
                                  clifford_angles=True)
        st["ops"] = layers[0]
    elif kind == "trotter_layer":
        side, terms = case["side"], case["terms"]
        n, q = side * side, (side // 2) * side + side // 2
        layer = _pack(_trotter_layer(side, t(0.3), t(0.3)))
        s = PauliSum([_z_word(n, q)], n, min_abs_coeff=case["threshold"], max_pauli_weight=case["cap"])
        rows = _grown_rows(s, [layer] * 40, terms)
        st["base"] = _sum_of_rows(rows, n, _room(case), min_abs_coeff=case["threshold"], max_pauli_weight=case["cap"])
        st["ops"] = layer
    elif kind == "budget":
        side, terms = case["side"], case["terms"]
        st["base"] = _sum_of_rows(_random_rows(side * side, terms, seed), side * side, terms + 64, min_abs_coeff=1e-9)
        st["net"] = TermPriorityNet(seed=seed)
    elif kind == "readout":
        n, terms = case["qubits"], case["terms"]
        rows = _random_rows(n, terms + terms // 2, seed)
        st["a"] = _sum_of_rows(rows[:terms].contiguous(), n, terms + 64)
        other = rows[terms // 2:].clone()
        st["b"] = _sum_of_rows(other[torch.randperm(len(other), generator=_gen(seed + 1), device="cuda")], n,
                               len(other) + 64)
        st["patterns"] = ["Z?*", "[XZ]?*", "_%d[XYZ]?*" % (n // 2)]
    else:
        r = np.random.default_rng(seed)
        m = case["samples"]
        st["features"], st["targets"] = _training_pairs(r, m)
        st["net"] = TermPriorityNet(seed=seed)
        st["params"] = _net_params(r)
        st["seed"] = seed
    return st


def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(seed)


def _random_rows(n, terms, seed):
    """Distinct words of low weight (mean 6) with coefficients spread over six decades, as rows."""
    g, W, dev = _gen(seed), (n + 63) // 64, "cuda"
    p = min(0.5, 6.0 / n)
    bit = torch.ones((), dtype=torch.int64, device=dev) << torch.arange(64, device=dev)
    planes = torch.zeros(0, 2 * W, dtype=torch.int64, device=dev)
    while len(planes) < terms:
        m = terms - len(planes) + 64 + terms // 8
        new = torch.zeros(m, 2 * W, dtype=torch.int64, device=dev)
        for w in range(W):
            k = min(64, n - 64 * w)
            pauli = torch.randint(1, 4, (m, k), generator=g, device=dev, dtype=torch.uint8)
            pauli *= (torch.rand(m, k, generator=g, device=dev) < p)
            new[:, w] = ((pauli & 1).to(torch.int64) * bit[:k]).sum(1)
            new[:, W + w] = ((pauli >> 1).to(torch.int64) * bit[:k]).sum(1)
            del pauli
        planes = torch.unique(torch.cat([planes, new]), dim=0)
    planes = planes[torch.randperm(len(planes), generator=g, device=dev)[:terms]]
    size = 10.0 ** (-6.0 * torch.rand(terms, generator=g, device=dev, dtype=torch.float64))
    sign = torch.where(torch.rand(terms, generator=g, device=dev) < 0.5, -1.0, 1.0).to(torch.float64)
    return torch.cat([planes, (size * sign).view(torch.int64).unsqueeze(1)], dim=1)


def _training_pairs(r, m):
    """Features as the engine's terms have them, and labels that fall with weight and depth."""
    weight = r.integers(1, 17, m)
    nx = r.binomial(weight, 0.4)
    ny = r.binomial(weight - nx, 0.4)
    left = r.integers(0, 5, m)
    lg = -7.0 * r.random(m)
    bonds = r.binomial(2 * weight, 0.3)
    f = np.stack([weight / 16, (lg + 6) / 6, left / 8, nx / 8, ny / 8, (weight - nx - ny) / 8, bonds / 8,
                  weight * left / 64], axis=1).astype(np.float32)
    y = np.maximum(lg - 0.25 * weight - 0.3 * left + 0.2 * r.standard_normal(m), -12.0).astype(np.float32)
    return np.ascontiguousarray(f), y


def _net_params(r):
    p = np.zeros(N_PARAMS, dtype=np.float32)
    p[0:512] = r.uniform(-1, 1, 512) / math.sqrt(8)
    p[576:4672] = r.uniform(-1, 1, 4096) / 8
    p[4736:4800] = r.uniform(-1, 1, 64) / 8
    return p


# ---- run ----------------------------------------------------------------------------------


def run(st):
    case = st["case"]
    kind = case["kind"]
    if kind == "chain":
        n = case["qubits"]
        s = PauliSum([st["word"]], n, min_abs_coeff=case["threshold"])
        s.run(st["ops"])
        return {"expectation": s.overlap_with_zero(), "live": _i64(s.live_counts()), **_host_terms(s, _room(case))}
    if kind == "calls":
        n = case["qubits"]
        s = PauliSum([st["word"]], n, min_abs_coeff=case["threshold"], exact_order=True)
        for _ in range(case["steps"]):
            for q in reversed(range(n)):
                s.rx(q, st["tx"])
            for q in reversed(range(n - 1)):
                s.rzz(q, q + 1, st["tzz"])
        return {"expectation": s.overlap_with_zero(), **_host_terms(s, _room(case))}
    if kind == "kicked":
        s = PauliSum([st["word"]], case["side"] ** 2, min_abs_coeff=case["threshold"], max_pauli_weight=case["cap"],
                     clifford_angles=True)
        s.run(st["ops"])
        return {"expectation": s.overlap_with_zero(), "live": _i64(s.live_counts()), **_device_terms(s, _room(case))}
    if kind == "clifford_t":
        s = PauliSum(st["words"], case["qubits"], min_abs_coeff=case["threshold"])
        s.run(st["ops"])
        return {"expectation": s.overlap_with_zero(), "live": _i64(s.live_counts()), **_device_terms(s, _room(case))}
    if kind == "noise":
        s = PauliSum([st["word"]], case["side"] ** 2, min_abs_coeff=case["threshold"], max_pauli_weight=case["cap"])
        s.run(st["ops"])
        return {"expectation": s.overlap_with_zero(), "live": _i64(s.live_counts()), **_device_terms(s, _room(case))}
    if kind == "lossy":
        s = LossyPauliSum([st["word"]], case["qubits"], min_abs_coeff=case["threshold"], max_pauli_weight=case["cap"],
                          max_loss_weight=2)
        s.run(st["ops"])
        return {"expectation": s.overlap_with_zero(), "live": _i64(s.live_counts()), **_device_terms(s, _room(case))}
    if kind == "batch":
        b = PauliSumBatch(st["instances"])
        b.run()
        per, total = b.term_gate_updates()
        return {"expectations": b.overlap_with_zero(), "updates": _i64(per), "total": int(total)}
    if kind in ("kicked_layer", "trotter_layer"):
        s = st["base"].copy()
        s.run(st["ops"])
        return {"expectation": s.overlap_with_zero(), "live": _i64(s.live_counts()), **_device_terms(s, _room(case))}
    if kind == "budget":
        s = st["base"].copy()
        s.truncate_budget(case["budget"], st["net"], case["side"], 2, case["digit_bits"])
        return _device_terms(s, case["budget"])
    if kind == "readout":
        a, b = st["a"], st["b"]
        return {"overlap": a.overlap(b), "expectation": a.overlap_with_zero(),
                "traces": [a.trace(p) for p in st["patterns"]], "heaviest": a.current_max_weight(),
                "equal": bool(a == b)}
    net = st["net"]
    net.params = st["params"]
    grad, loss = net.grad(st["features"], st["targets"])
    scores = net.predict(st["features"])
    last = net.train(st["features"], st["targets"], epochs=case["epochs"], batch=case["batch"], lr=2e-3,
                     seed=st["seed"])
    return {"grad": grad, "loss": loss, "scores": scores, "params": net.params, "last": last}


def _i64(a):
    return np.ascontiguousarray(a).view(np.int64)


# ---- work ---------------------------------------------------------------------------------


def work(case):
    """Bytes each pass reads and writes at least once (its inputs and outputs); term counts that
    a circuit decides are rough figures for its nominal angles."""
    kind = case["kind"]
    if kind in ("chain", "calls"):
        n, steps = case["qubits"], case["steps"]
        final = min(40.0 * steps, 800.0)
        return {"bytes": OP_BYTES * steps * 2.0 * n + 24.0 * final, "flops": 6.0 * steps * n * final / 3}
    if kind == "kicked":
        side, grow = case["side"], (1e-5 / case["threshold"]) * 2.0 ** (case["cap"] - 10)
        final = 2e5 * grow  # the sum peaks near layer 12 and then dies out
        term = 16.0 * ((side * side + 63) // 64) + 8
        return {"bytes": OP_BYTES * case["layers"] * 3.0 * side * side + term * final, "flops": 6.0 * final}
    if kind == "clifford_t":
        final = 16 * 1.5 ** (3 * case["layers"])
        return {"bytes": OP_BYTES * case["layers"] * 1.5 * case["qubits"] + 24.0 * final, "flops": 6.0 * final}
    if kind == "noise":
        side = case["side"]
        final = 2e5 * (2e-5 / case["threshold"]) * (case["layers"] / 5.0) ** 4
        return {"bytes": OP_BYTES * case["layers"] * 7.0 * side * side + 24.0 * final, "flops": 10.0 * final}
    if kind == "lossy":
        final = 1e5 * (case["layers"] / 4.0) ** 4
        return {"bytes": OP_BYTES * case["layers"] * 3.0 * case["qubits"] + 40.0 * final, "flops": 10.0 * final}
    if kind == "batch":
        gates = case["count"] * 17.5 * 2 * 72
        return {"bytes": OP_BYTES * gates + case["count"] * 16.0, "flops": 3.0 * gates * 500}
    if kind in ("kicked_layer", "trotter_layer"):
        side, out = case["side"], (3.9, 1e6) if kind == "kicked_layer" else (12.0, 9e5)
        term = 16.0 * ((side * side + 63) // 64) + 8
        terms = case["terms"] * (1 + out[0]) + out[1]
        return {"bytes": OP_BYTES * 3.0 * side * side + term * terms, "flops": 6.0 * terms}
    if kind == "budget":
        term = 16.0 * ((case["side"] ** 2 + 63) // 64) + 8
        return {"bytes": term * (case["terms"] + case["budget"]), "flops": 9344.0 * case["terms"]}
    if kind == "readout":
        term = 16.0 * ((case["qubits"] + 63) // 64) + 8
        return {"bytes": 2.0 * term * case["terms"], "flops": 6.0 * case["terms"]}
    m = case["samples"]
    return {"bytes": 40.0 * m + 16.0 * N_PARAMS, "flops": 9344.0 * m * (4 + 3 * case["epochs"])}


# ---- exact --------------------------------------------------------------------------------


def _chain_exact(n, word, ops, thr):
    """The terms after the list, in insertion order, from a plain dictionary."""
    q0 = word.index("Z")
    terms = {(0, 1 << q0): 1.0}
    for code, a, b, theta, _ in ops:
        if code == G.TRUNCATE:
            terms = {k: v for k, v in terms.items() if not abs(v) < thr}
            continue
        sn, cs = math.sin(theta), math.cos(theta)
        gx, gz = ((1 << a), 0) if code == G.RX else (0, (1 << a) | (1 << b))
        new = {}
        for (x, z), v in terms.items():
            if not (bin(x & gz).count("1") + bin(z & gx).count("1")) & 1:
                continue
            if code == G.RX:
                sign = -1.0 if (x >> a) & 1 else 1.0
            else:  # the anticommuting qubit decides: Y gives +, X gives -
                q = a if (x >> a) & 1 else b
                sign = 1.0 if (z >> q) & 1 else -1.0
            new[(x ^ gx, z ^ gz)] = v * (sign * sn)
            terms[(x, z)] = v * cs
        for k, v in new.items():
            terms[k] = terms[k] + v if k in terms else v
    return terms


def _expect(terms):
    return math.fsum(v for (x, _), v in terms.items() if x == 0)


def exact(case, seed):
    kind = case["kind"]
    t = _angles(case, seed)
    if kind == "chain":
        n, tzz, tx = case["qubits"], t(0.2), t(0.2)
        terms = _chain_exact(n, _z_word(n, n // 2), _chain_ops(n, case["steps"], tzz, tx), case["threshold"])
        return {"expectation": _expect(terms), "live": None, "count": None, "x": None, "z": None, "c": None}
    if kind == "calls":
        n, tzz, tx = case["qubits"], t(0.2), t(0.2)
        ops = [o for op in _chain_ops(n, case["steps"], tzz, tx) if op[0] != G.TRUNCATE for o in (op, G.truncate())]
        terms = _chain_exact(n, _z_word(n, n // 2), ops, case["threshold"])
        c = np.zeros(_room(case))
        c[: len(terms)] = list(terms.values())
        return {"expectation": _expect(terms), "count": None, "x": None, "z": None, "c": c}
    if kind == "readout":
        return _readout_exact(case, seed)
    if kind == "train":
        r = np.random.default_rng(seed)
        f, y = _training_pairs(r, case["samples"])
        grad, loss, scores = _net_exact(_net_params(r), f, y)
        return {"grad": grad, "loss": loss, "scores": scores, "params": None, "last": None}
    return None


def _readout_exact(case, seed):
    n, m = case["qubits"], case["terms"]
    W = (n + 63) // 64
    rows = _random_rows(n, m + m // 2, seed).cpu().numpy()
    x, z = rows[:, :W].view(np.uint64), rows[:, W:2 * W].view(np.uint64)
    c = np.ascontiguousarray(rows[:, 2 * W]).view(np.float64)
    no_x = ~x[:m].any(1)
    no_y = ~(x[:m] & z[:m]).any(1)
    q = n // 2
    code = ((x[:m, q // 64] >> np.uint64(q % 64)) & np.uint64(1)) + 2 * ((z[:m, q // 64] >> np.uint64(q % 64)) & np.uint64(1))
    before = np.zeros(m, dtype=bool)  # a Pauli other than I below qubit q
    for w in range(q // 64 + 1):
        mask = np.uint64((1 << (min(q - 64 * w, 64))) - 1)
        before |= ((x[:m, w] | z[:m, w]) & mask) != 0
    # pattern "_q[XYZ]?*": only I up to and at qubit q, anything after it
    third = (code == 0) & ~before
    return {"overlap": math.fsum(c[m // 2:m] ** 2), "expectation": math.fsum(c[:m][no_x]),
            "traces": [math.fsum(c[:m][no_x]), math.fsum(c[:m][no_y]), math.fsum(c[:m][third])],
            "heaviest": None, "equal": None}


def _erf(v):
    return torch.erf(torch.from_numpy(v)).numpy()


def _net_exact(p, f, y):
    p, f, y = p.astype(np.float64), f.astype(np.float64), y.astype(np.float64)
    w1, b1, w2, b2, w3, b3 = (p[:512].reshape(64, 8), p[512:576], p[576:4672].reshape(64, 64), p[4672:4736],
                              p[4736:4800], p[4800])
    gelu = lambda v: 0.5 * v * (1 + _erf(v / math.sqrt(2)))  # noqa: E731
    slope = lambda v: 0.5 * (1 + _erf(v / math.sqrt(2))) + v * np.exp(-v * v / 2) / math.sqrt(2 * math.pi)  # noqa: E731
    z1 = f @ w1.T + b1
    h1 = gelu(z1)
    z2 = h1 @ w2.T + b2
    h2 = gelu(z2)
    s = h2 @ w3 + b3
    d = 2 * (s - y) / len(y)
    d2 = np.outer(d, w3) * slope(z2)
    d1 = (d2 @ w2) * slope(z1)
    grad = np.concatenate([(d1.T @ f).ravel(), d1.sum(0), (d2.T @ h1).ravel(), d2.sum(0), h2.T @ d, [d.sum()]])
    return grad, float(np.mean((s - y) ** 2)), s
