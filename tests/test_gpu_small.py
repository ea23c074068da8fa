"""Small sums: the one-CTA list interpreter against the oracle and against the pipelines.

Sums of at most 512 terms start in the interpreter; PPVM_SMALL=never (read once per process)
sends them through the pipelines from the first op, so the parity cases run again that way in a
child process.  The cases here are the interpreter's edges: the start limit (512 terms), the
region's size (2048 terms, 1024 above 192 qubits), more ops than one launch takes, local
stretches at the composed pass's limit, wide runs, and fused runs that outgrow the region in the
middle.  Term order (the fused runs' too) and every coefficient are compared with the pipelines'
bit for bit, the term set with the oracle's."""

import json
import os
import subprocess
import sys

import numpy as np
import pytest

from ppvm_b200 import gates as G
from ppvm_b200.paulisum import PauliSum

from tests.helpers import oracle_from
from tests.test_gpu_parity import same, same_set

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def random_terms(rng, n, m):
    terms = {}
    while len(terms) < m:
        w = "".join("IXYZ"[int(rng.choice(4, p=[0.7, 0.1, 0.1, 0.1]))] for _ in range(n))
        terms[w] = float(rng.uniform(-1, 1))
    return list(terms.items())


def mixed_ops(rng, n, layers, locals_per_layer=6):
    ops = []
    for _ in range(layers):
        ops += [G.r1(G.RX, int(q), float(rng.uniform(-2, 2))) for q in rng.permutation(n)[: min(n, 6)]] + [G.truncate()]
        ops += [G.amplitude_damping(int(rng.integers(n)), 0.05)]
        ops += [G.r1(G.RZ, int(q), float(rng.uniform(-2, 2))) for q in rng.permutation(n)[: min(n, 4)]]
        for _ in range(locals_per_layer):
            q = int(rng.integers(n))
            ops.append([G.g1(G.H, q), G.g1(G.S, q), G.depolarize1(q, 0.01), G.pauli_error(q, (0.01, 0.02, 0.03)),
                        G.g1(G.SQRT_Y_DAG, q)][int(rng.integers(5))])
        if n > 1:
            a, b = (int(v) for v in rng.choice(n, 2, replace=False))
            ops += [G.g2(G.CNOT, a, b), G.depolarize2(a, b, 0.02), G.r2(G.RZZ, a, b, 0.4), G.r2(G.RYY, a, b, -0.3),
                    G.r2(G.RXX, a, b, np.pi / 2)]
        ops += [G.r1(G.RY, int(rng.integers(n)), 0.7), G.truncate()]
    return ops


def cases():
    rng = np.random.default_rng(0)
    out = []
    for n in (1, 2, 5, 20, 63, 64, 65, 130, 200, 300):
        out.append((n, random_terms(rng, n, min(20, 2 ** n)), mixed_ops(rng, n, 6), 1e-3, None))
    for m in (511, 512, 513):  # the start limit
        out.append((40, random_terms(rng, 40, m), mixed_ops(rng, 40, 2), 1e-3, 20))
    for n in (30, 200):
        for k in (9, 10, 11):  # 2^k terms from one word: up to, at and past the region
            w = "Z" * k + "I" * (n - k)
            rx = [G.r1(G.RX, q, 0.3 + 0.01 * q) for q in range(k)]
            out.append((n, [(w, 1.0)], rx + [G.truncate()] + rx[:2] + [G.truncate()], 1e-9, None))
            out.append((n, [(w, 1.0), ("X" * n, 0.5)], [op for r in rx for op in (r, G.truncate())], 1e-9, None))
    # a run of 13 coordinates (too wide for a group), and one that doubles past the region midway
    out.append((20, [("Z" * 13 + "I" * 7, 1.0)], [G.r1(G.RX, q, 0.2) for q in range(20)] + [G.truncate()], 1e-4, None))
    out.append((14, random_terms(rng, 14, 400), [G.r1(G.RX, q, 0.2) for q in range(14)] + [G.truncate()], 1e-3, None))
    for k in (63, 64, 65, 300):  # local stretches around the composed pass's limit
        ops = [G.g1((G.H, G.S, G.SQRT_X)[i % 3], i % 12) for i in range(k)]
        out.append((12, random_terms(rng, 12, 50), ops + [G.r1(G.RX, 3, 0.4), G.truncate()] + ops[:5], 1e-6, None))
    # more ops than one launch takes, the sum small all along
    out.append((10, random_terms(rng, 10, 8), mixed_ops(rng, 10, 150, 2), 0.02, 4))
    return out


def results(exact):
    out = []
    for n, terms, ops, thr, maxw in cases():
        s = PauliSum([w for w, _ in terms], n, [c for _, c in terms], min_abs_coeff=thr, max_pauli_weight=maxw,
                     exact_order=exact, clifford_angles=True)
        s.run(ops)
        x, z, c = s.export()
        out.append([x.tobytes().hex(), z.tobytes().hex(), c.tobytes().hex(), s.live_counts().tobytes().hex()])
    return out


@pytest.mark.parametrize("exact", [True, False])
def test_interpreter_equals_the_pipelines_bit_for_bit(exact):
    script = f"import json; from tests.test_gpu_small import results; print(json.dumps(results({exact})))"
    r = subprocess.run([sys.executable, "-c", script], cwd=ROOT, env=dict(os.environ, PPVM_SMALL="never"),
                       capture_output=True, text=True, timeout=600)
    assert r.returncode == 0, r.stdout[-2000:] + r.stderr[-2000:]
    want = json.loads(r.stdout.strip().splitlines()[-1])
    for i, (a, b) in enumerate(zip(results(exact), want)):
        assert a == b, cases()[i][0]


@pytest.mark.parametrize("exact", [True, False])
def test_interpreter_matches_the_oracle(exact):
    for n, terms, ops, thr, maxw in cases():
        s = PauliSum([w for w, _ in terms], n, [c for _, c in terms], min_abs_coeff=thr, max_pauli_weight=maxw,
                     exact_order=exact, clifford_angles=True)
        o = oracle_from(terms, n, thr, maxw, clifford_angles=True)
        s.run(ops)
        want = o.run_ops(ops, counts=True)
        assert np.array_equal(s.live_counts(), want), n
        same_set(s, o)
        for op in ops[:12]:  # one call per op
            s.run([op])
            o.run_ops([op])
        (same if exact else same_set)(s, o)


def test_parity_cases_through_the_pipelines():
    r = subprocess.run([sys.executable, "-m", "pytest", "tests/test_gpu_parity.py", "tests/test_gpu_noise.py",
                        "tests/test_gpu_tableau.py", "-m", "gpu", "-x", "-q"],
                       cwd=ROOT, env=dict(os.environ, PPVM_SMALL="never"), capture_output=True, text=True, timeout=900)
    assert r.returncode == 0, r.stdout[-3000:] + r.stderr[-2000:]
    assert " passed" in r.stdout
