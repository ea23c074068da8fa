"""The choice between the two group kernels of a fused run.

It goes by the number of groups, by their members and by how many of them are too large for one lane
(more than three coordinates).  Both sides of each line, and lists whose runs alternate between the sides, must
give the list that the tile kernel alone gives, bit for bit and in order (in a child process with
PPVM_RUN_GROUP_MODE=tiled); the smaller ones also match the oracle."""

import hashlib
import json
import os
import subprocess
import sys

import numpy as np
import pytest
import torch

from ppvm_b200 import gates as G
from ppvm_b200.paulisum import PauliSum
from ppvm_b200.sharded import DeviceShare

from tests.helpers import oracle_from, planes
from tests.test_gpu_parity import same_set

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def terms_of(n, m, large, big):
    """m words over n qubits, each its own group of an RX run on the first 10: `large` of them hold Z
    on `big` of these, the others on one to three."""
    rng = np.random.default_rng(n + m + large)
    tail = rng.permutation(4 ** 10)[:m]  # distinct X/I patterns on the last 20 qubits
    out = []
    for i in range(m):
        k = big if i < large else int(rng.integers(1, 4))
        head = ["I"] * 10
        for q in rng.choice(10, k, replace=False):
            head[int(q)] = "Z"
        last = "".join("IX"[int(tail[i]) >> b & 1] for b in range(20))
        out.append(("".join(head) + "I" * (n - 30) + last, float(rng.uniform(-1, 1))))
    return [out[int(i)] for i in rng.permutation(m)]


RX = [G.r1(G.RX, q, 0.3 + 0.01 * q) for q in range(10)]
RZ = [G.r1(G.RZ, q, 0.2 + 0.01 * q) for q in (1, 4, 7, 25, 28)]
SHORT = [G.r1(G.RX, q, 0.3) for q in (2, 5, 8)]
T = [G.truncate()]


def cases():
    out = []
    for m in (8191, 8192, 9000):  # the number of groups from which lanes are taken
        out.append((40, m, m // 16, 5, RX + T, 1e-3))
    for large in (0, 1, 1125, 9000):
        for n in (40, 144, 300):
            out.append((n, 9000, large, 6, RX + T, 1e-2))
    out.append((100, 20000, 1000, 10, RX, 0.05))  # groups of 2^10 slots on warps of the lane kernel
    for large in (16400, 16300, 20000):  # around one in 16 of 262,250 groups, twice: single, then full members
        out.append((40, 262250, large, 4, RX, 0.0))
    for n in (40, 144):  # runs that alternate: full small groups, large groups, RZ runs, a few terms left
        out.append((n, 9000, 600, 7, RX + T + RZ + T + RX + SHORT + T + RZ + RX + T, 0.02))
        out.append((n, 9000, 9000, 4, SHORT + T + RX + T + SHORT + RZ + T + [G.r2(G.RXX, 0, 1, 0.3)] + RX + T, 0.02))
    return out


def large_sum(n, terms, ops):
    """As run(), the terms brought in as rows (word by word takes a minute)."""
    s = PauliSum(["I" * n], n, min_abs_coeff=0.0, capacity=1 << 21)
    share, zero = DeviceShare(s), np.zeros(s.W, dtype=np.uint64)
    share.export(zero, zero, 1)
    x, z = planes([w for w, _ in terms], n)
    c = np.array([c for _, c in terms])
    share.append(torch.from_numpy(np.concatenate([x, z, c.view(np.uint64)[:, None]], axis=1).view(np.int64)).reshape(-1))
    for _ in range(2):
        s.run(ops)
    return s


def run(case):
    n, m, large, big, ops, thr = case
    terms = terms_of(n, m, large, big)
    if m > 100000:
        return terms, large_sum(n, terms, ops)
    s = PauliSum([w for w, _ in terms], n, [c for _, c in terms], min_abs_coeff=thr)
    for _ in range(2):
        s.run(ops)  # storage grows, and runs are replayed, in some of these
    return terms, s


def digests():
    out = []
    for case in cases():
        _, s = run(case)
        x, z, c = s.export()
        out.append([len(s), hashlib.sha256(x.tobytes() + z.tobytes() + c.tobytes()).hexdigest(),
                    hashlib.sha256(s.live_counts().tobytes()).hexdigest()])
    return out


def test_either_group_kernel_gives_the_same_list():
    script = "import json; from tests.test_gpu_run_rule import digests; print(json.dumps(digests()))"
    r = subprocess.run([sys.executable, "-c", script], cwd=ROOT, capture_output=True, text=True, timeout=600,
                       env=dict(os.environ, PPVM_RUN_GROUP_MODE="tiled"))
    assert r.returncode == 0, r.stdout[-2000:] + r.stderr[-2000:]
    want = json.loads(r.stdout.strip().splitlines()[-1])
    for case, a, b in zip(cases(), digests(), want):
        assert a == b, case[:4]


@pytest.mark.parametrize("case", [0, 1, 4, 7, 16, 19, 20])
def test_the_rule_matches_the_oracle(case):
    c = cases()[case]
    terms, s = run(c)
    o = oracle_from(terms, c[0], c[5])
    for _ in range(2):
        o.run_ops(c[4])
    same_set(s, o)
