"""Sums of several host threads, from their first calls on in a fresh process: the one-CTA interpreter,
the fused runs and the composed Clifford pass set up their kernels on first use, one plane width
after another, while other threads do the same."""

import os
import subprocess
import sys
import threading

import numpy as np
import pytest

from ppvm_b200 import gates as G
from ppvm_b200.paulisum import PauliSum

from tests.helpers import oracle_from
from tests.test_gpu_parity import same_set
from tests.test_gpu_small import mixed_ops, random_terms

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def cases():
    rng = np.random.default_rng(9)
    out = []
    for i in range(24):
        n = (20, 65, 130, 200, 300, 400)[i % 6]
        m = 40 if i % 2 else 700  # the interpreter, the pipelines
        clifford = [G.g1((G.H, G.S)[j % 2], j % n) for j in range(100)]
        out.append((n, random_terms(rng, n, m), clifford + mixed_ops(rng, n, 2)))
    return out


def check():
    got, want = {}, {}

    def work(part, gate):
        gate.wait()
        for i, (n, terms, ops) in part:
            s = PauliSum([w for w, _ in terms], n, [c for _, c in terms], min_abs_coeff=1e-3, clifford_angles=True)
            s.run(ops)
            got[i] = s

    all_cases = list(enumerate(cases()))
    gate = threading.Barrier(8)
    threads = [threading.Thread(target=work, args=(all_cases[t::8], gate)) for t in range(8)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    for i, (n, terms, ops) in all_cases:
        want[i] = oracle_from(terms, n, 1e-3, clifford_angles=True)
        want[i].run_ops(ops)
        same_set(got[i], want[i])
    print("checked", len(got))


def test_first_calls_of_eight_threads():
    for _ in range(3):
        r = subprocess.run([sys.executable, "-c", "from tests.test_gpu_threads import check; check()"], cwd=ROOT,
                           capture_output=True, text=True, timeout=300)
        assert r.returncode == 0, r.stdout[-2000:] + r.stderr[-2000:]
        assert "checked 24" in r.stdout
