"""Live counts of long fused runs on a few groups.

A run of more than 32 gates on at most 8 groups is one block of the group kernels (one warp's worth in
lane mode), whose warps all add the children they made per gate before one warp publishes the
counts and clears them.  Counts that are read too early are missing from this run and left over
for the next, so every list runs several times on the same sum and on fresh ones.  The small sums'
interpreter is off, and one group per lane is forced in a second child process."""

import os
import subprocess
import sys

import numpy as np
import pytest

from ppvm_b200 import gates as G
from ppvm_b200.paulisum import PauliSum

from tests.helpers import oracle_from
from tests.test_gpu_parity import same_set

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def words(rng, n, groups):
    out = {}
    while len(out) < groups:  # 1 to 6 coordinates each, one of them among the last gates
        w = ["I"] * n
        for q in rng.choice(n, int(rng.integers(0, 6)), replace=False):
            w[int(q)] = "Z"
        w[n - 1 - int(rng.integers(n // 4))] = "Z"
        out["".join(w)] = float(rng.uniform(0.5, 1))
    return list(out.items())


def check(n, gates, groups, repeats=12):
    rng = np.random.default_rng(1000 * gates + groups)
    terms = words(rng, n, groups)
    perm = [int(q) for q in rng.permutation(n)[:gates]]
    ops = [G.r1(G.RX, q, 0.3 + 0.001 * q) for q in perm] + [G.truncate()]
    o = oracle_from(terms, n, thr=1e-12)
    want = [o.run_ops(ops, counts=True) for _ in range(3)]
    for _ in range(repeats):
        s = PauliSum([w for w, _ in terms], n, [c for _, c in terms], min_abs_coeff=1e-12)
        for w in want:
            s.run(ops)
            assert np.array_equal(s.live_counts(), w)
        same_set(s, o)


CASES = [(n, gates, groups) for n, gates in [(64, 33), (64, 64), (128, 100), (256, 256)] for groups in (1, 2, 7, 8, 9)]


@pytest.mark.parametrize("mode", ["tiled", "lanes"])
def test_counts_of_long_runs_on_few_groups(mode):
    script = "from tests.test_gpu_run_counts import CASES, check\nfor c in CASES: check(*c)\nprint('checked', len(CASES))"
    r = subprocess.run([sys.executable, "-c", script], cwd=ROOT, capture_output=True, text=True, timeout=600,
                       env=dict(os.environ, PPVM_SMALL="never", PPVM_RUN_GROUP_MODE=mode))
    assert r.returncode == 0, r.stdout[-2000:] + r.stderr[-2000:]
    assert f"checked {len(CASES)}" in r.stdout
