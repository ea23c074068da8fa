"""A batch whose pool could not grow: the run fails, and the next one starts from a pool laid out anew.

PPVM_TEST_FAIL_ALLOC=batch-pool (read once per process) makes every growth of a batch's pool fail as
if the device had no memory left.  After the failed run the instance table must not describe the
pool that was never allocated: the next run, whose regions start at the grown capacity, lays out
afresh and matches the oracle."""

import json
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

SCRIPT = r"""
import json
from ppvm_b200 import gates as G
from ppvm_b200._lib import PPVMError
from ppvm_b200.batch import Instance, PauliSumBatch
from tests.test_gpu_batch import check_batch
insts = []
for i in range(40):  # every fourth instance makes 512 terms, in regions that start with 256
    m = 9 if i % 4 == 0 else 4
    rx = [G.r1(G.RX, q, 0.3 + 0.01 * q) for q in range(m)]
    insts.append(Instance(20, [("Z" * m + "I" * (20 - m), 1.0)], rx + [G.truncate(), G.truncate()], 1e-12, None))
out = []
for run in ("run", "run_persistent"):
    b = PauliSumBatch(insts)
    try:
        getattr(b, run)()
        out.append(0)
    except PPVMError as e:
        out.append(e.status)
    for _ in range(3):  # the second launches the layers, the third as graphs
        getattr(b, run)()
        check_batch(b)
    out.append(int(b.capacities().max()))
print(json.dumps(out))
"""


def test_run_after_a_failed_growth():
    env = dict(os.environ, PPVM_BATCH_GROW="host", PPVM_TEST_FAIL_ALLOC="batch-pool")
    r = subprocess.run([sys.executable, "-c", SCRIPT], cwd=ROOT, env=env, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout[-2000:] + r.stderr[-2000:]
    first, cap, first_p, cap_p = json.loads(r.stdout.strip().splitlines()[-1])
    assert first == first_p == 2  # PPVM_ECAPACITY
    assert cap >= 512 and cap_p >= 512
