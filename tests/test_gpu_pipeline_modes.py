"""The fused runs' modes on small sums, through the pipelines.

Sums of up to 512 terms go to the one-CTA interpreter unless PPVM_SMALL=never is set, and then no group
kernel runs at all.  Here it is set, together with a group mode, with scratch placement from the
first group on, or with scratch memory that cannot be had, so that the small parity cases test the
kernels that the setting names.  (All settings are read once per process.)"""

import json
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

SETTINGS = {
    "tiles": {"PPVM_RUN_GROUP_MODE": "tiled"},
    "lanes": {"PPVM_RUN_GROUP_MODE": "lanes"},
    "scratch": {"PPVM_RUN_SCRATCH_MIN_GROUPS": "1"},
    "no scratch memory": {"PPVM_RUN_SCRATCH_MIN_GROUPS": "1", "PPVM_TEST_FAIL_ALLOC": "run-scratch"},
}

FAMILIES = r"""
import json
from ppvm_b200 import gates as G
from ppvm_b200.paulisum import PauliSum
s = PauliSum(["ZZIZ", "XZYI"], 4, [1.0, 0.5], min_abs_coeff=0.0)
s.profile(True)
s.run([G.r1(G.RX, q, 0.3) for q in range(4)] + [G.truncate()])
s.profile(False)
print(json.dumps(sorted(k for k, v in s.profile_read().items() if v["launches"])))
"""


@pytest.mark.parametrize("name", list(SETTINGS))
def test_small_parity_cases_in_each_mode(name):
    env = dict(os.environ, PPVM_SMALL="never", **SETTINGS[name])
    r = subprocess.run([sys.executable, "-c", FAMILIES], cwd=ROOT, env=env, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout[-2000:] + r.stderr[-2000:]
    ran = json.loads(r.stdout.strip().splitlines()[-1])
    assert "run_groups" in ran and "small" not in ran
    assert ("run_place" in ran) == (name == "scratch")
    r = subprocess.run([sys.executable, "-m", "pytest", "tests/test_gpu_parity.py", "-m", "gpu", "-x", "-q",
                        "-k", "fused or random or kicked or wide or growth or cached or reused or clifford_t"],
                       cwd=ROOT, env=env, capture_output=True, text=True, timeout=900)
    assert r.returncode == 0, r.stdout[-3000:] + r.stderr[-2000:]
    assert " passed" in r.stdout
