"""Growth of batched instances, inside the launches and through the host.

An instance that runs out of room takes its next region from the pool's spare words inside the
kernel; PPVM_BATCH_GROW=host (read once per process) leaves no spare words, so that every
growth stops at the failing op and goes through the host's re-layout.  Both against the
oracle: lists that double the sum from 1 term past the initial 256, over several growths,
with the growth inside the first and inside a later layer."""

import os
import subprocess
import sys

import pytest

from ppvm_b200 import gates as G
from ppvm_b200.batch import Instance, PauliSumBatch

from tests.test_gpu_batch import check_batch

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.mark.parametrize("n", [8, 9, 13, 64, 65, 130])
def test_instances_that_double_past_their_region(n):
    # a word of m Zs under RX on each of them makes 2^m terms: m = 8 fills 256 exactly, 9 and more grow
    insts = []
    for m in (1, 7, 8, 9, 10, 13):
        if m > n:
            continue
        w = "Z" * m + "I" * (n - m)
        rx = [G.r1(G.RX, q, 0.3 + 0.01 * q) for q in range(m)]
        zz = [G.r2(G.RZZ, q, q + 1, 0.2) for q in range(m - 1)]
        insts.append(Instance(n, [(w, 1.0)], rx + [G.truncate()] + zz + [G.truncate()], 1e-9, None))
        insts.append(Instance(n, [(w, 1.0)], rx[: m // 2] + [G.truncate(), G.truncate()] + rx[m // 2:] + zz, 0.0, None))
    b = PauliSumBatch(insts)
    for _ in range(2):  # again on the grown regions
        b.run()
        check_batch(b)
    assert int(b.capacities().max()) >= (1 << min(n, 13))


def test_growth_through_the_host_matches_the_oracle():
    env = dict(os.environ, PPVM_BATCH_GROW="host")
    r = subprocess.run([sys.executable, "-m", "pytest", "tests/test_gpu_batch.py", "tests/test_gpu_batch_growth.py",
                        "-m", "gpu", "-x", "-q", "-k", "not through_the_host and not from_the_pool"],
                       cwd=ROOT, env=env, capture_output=True, text=True, timeout=900)
    assert r.returncode == 0, r.stdout[-3000:] + r.stderr[-2000:]
    assert " passed" in r.stdout
