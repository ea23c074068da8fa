"""Training an epoch in one cluster launch gives the parameters of the step-by-step launches.

Minibatches of at most 16 blocks (1024 samples) train a whole epoch per launch;
PPVM_MLP_EPOCH=never (read once per process, so in a child process) takes two launches per step
instead.  Bit-identical parameters and losses at the edges of the 16-sample tiles, the 64-sample
blocks and the cluster size, with a short last minibatch, over several epochs and calls."""

import json
import os
import subprocess
import sys

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CASES = [(1, 1, 1), (40, 16, 2), (65, 17, 3), (130, 64, 2), (200, 65, 3), (1500, 512, 3), (2000, 777, 2),
         (2048, 1024, 4), (2100, 1025, 2), (300, 4096, 2)]


def trained():
    from ppvm_b200.learned import TermPriorityNet

    out = []
    for n, batch, epochs in CASES:
        rng = np.random.default_rng(n)
        f = rng.standard_normal((n, 8)).astype(np.float32)
        y = (f.sum(1) * 0.3 - 2).astype(np.float32)
        net = TermPriorityNet(seed=n)
        losses = [net.train(f, y, epochs=epochs, batch=batch, lr=2e-3, seed=5), net.train(f, y, epochs=1, batch=batch)]
        out.append([net.params.tobytes().hex(), [float(v).hex() for v in losses], net.predict(f[:20]).tobytes().hex()])
    return out


def test_epoch_launches_equal_step_launches():
    script = "import json; from tests.test_gpu_learned_epochs import trained; print(json.dumps(trained()))"
    r = subprocess.run([sys.executable, "-c", script], cwd=ROOT, env=dict(os.environ, PPVM_MLP_EPOCH="never"),
                       capture_output=True, text=True, timeout=600)
    assert r.returncode == 0, r.stdout[-2000:] + r.stderr[-2000:]
    want = json.loads(r.stdout.strip().splitlines()[-1])
    for case, a, b in zip(CASES, trained(), want):
        assert a == b, case
