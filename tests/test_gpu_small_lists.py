"""Lists of two to four ops on small sums, with a fused run that does not start the list.

So few ops reach the one-CTA interpreter as a kernel argument; the run's terms must come in the
order in which the fused run writes them, whichever op of the list it starts at.  Order, bits and live
counts are compared with the pipelines' (PPVM_SMALL=never, in a child process), terms with
the oracle's."""

import json
import os
import subprocess
import sys

import numpy as np
import pytest

from ppvm_b200 import gates as G
from ppvm_b200.paulisum import PauliSum

from tests.helpers import oracle_from
from tests.test_gpu_parity import same_set
from tests.test_gpu_small import random_terms

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def cases():
    rng = np.random.default_rng(5)
    out = []
    for n in (3, 20, 65, 200):
        q = [int(v) for v in rng.choice(n, 3, replace=False)]
        for code in (G.RX, G.RZ):
            run = [G.r1(code, v, 0.3 + 0.1 * i) for i, v in enumerate(q)]
            other = G.r1(G.RZ if code == G.RX else G.RX, q[0], 0.2)
            for ops in ([G.r2(G.RZZ, q[0], q[1], 0.4)] + run[:2], [other] + run, [G.g1(G.H, q[2]), other] + run[:2],
                        [G.truncate(), G.amplitude_damping(q[1], 0.1)] + run[1:], [G.g1(G.H, q[0])] + run[:2] + [other],
                        run[:2] + [run[0], run[2]], [G.r1(G.RY, q[0], 0.7)] + run[:2] + [G.truncate()]):
                out.append((n, random_terms(rng, n, min(30, 4 ** n // 2)), ops))
    return out


def results():
    out = []
    for n, terms, ops in cases():
        s = PauliSum([w for w, _ in terms], n, [c for _, c in terms], min_abs_coeff=1e-6)
        row = []
        for _ in range(3):
            s.run(ops)
            x, z, c = s.export()
            row.append([x.tobytes().hex(), z.tobytes().hex(), c.tobytes().hex(), s.live_counts().tobytes().hex()])
        out.append(row)
    return out


def test_short_lists_equal_the_pipelines_in_order():
    script = "import json; from tests.test_gpu_small_lists import results; print(json.dumps(results()))"
    r = subprocess.run([sys.executable, "-c", script], cwd=ROOT, env=dict(os.environ, PPVM_SMALL="never"),
                       capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout[-2000:] + r.stderr[-2000:]
    want = json.loads(r.stdout.strip().splitlines()[-1])
    for case, a, b in zip(cases(), results(), want):
        assert a == b, (case[0], [int(op[0]) for op in case[2]])


def test_short_lists_match_the_oracle():
    for n, terms, ops in cases():
        s = PauliSum([w for w, _ in terms], n, [c for _, c in terms], min_abs_coeff=1e-6)
        o = oracle_from(terms, n, thr=1e-6)
        for _ in range(3):
            s.run(ops)
            o.run_ops(ops)
            same_set(s, o)
