"""Fused runs on many groups of 2^7 to 2^10 slots.

From 2^15 groups on a warp of the tile kernel takes up to four groups, as many as fit its slots on
average; those that do not fit are run again to be written.  The fused result must equal the same gates
one by one (exact order), every coefficient bit for bit, with and without a truncation, in order and
with scratch placement (forced, in a child process)."""

import os
import subprocess
import sys

import numpy as np
import pytest
import torch

from ppvm_b200 import gates as G
from ppvm_b200._lib import lib
from ppvm_b200.paulisum import PauliSum
from ppvm_b200.sharded import DeviceShare

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def base_rows(n, m, k):
    """m words, each its own group of an RX run on the first 10 qubits: Z on k of them (k = 0: 3 to 10, by
    word), and X or I on the last 24 as the word's number says."""
    rng = np.random.default_rng(100 * k + n)
    W = (n + 63) // 64
    rows = np.zeros((m, 2 * W + 1), dtype=np.uint64)
    ks = np.full(m, k) if k else rng.integers(3, 11, m)
    order = rng.random((m, 10)).argsort(1)
    for j in range(10):
        rows[:, W] |= np.where(j < ks, np.uint64(1) << order[:, j].astype(np.uint64), np.uint64(0))
    number = rng.permutation(1 << 20)[:m].astype(np.uint64)
    at = n - 24
    for b in range(20):
        q = at + b
        rows[:, q // 64] |= ((number >> np.uint64(b)) & np.uint64(1)) << np.uint64(q % 64)
    rows[:, 2 * W] = rng.uniform(-1, 1, m).view(np.uint64)
    return torch.from_numpy(rows.view(np.int64)).reshape(-1), int((2.0 ** ks).sum())


def sum_of(n, rows, room, thr, exact):
    s = PauliSum(["I" * n], n, min_abs_coeff=thr, capacity=room, exact_order=exact)
    zero = np.zeros(s.W, dtype=np.uint64)
    share = DeviceShare(s)
    share.export(zero, zero, 1)
    share.append(rows)
    return s


def check(n, m, k, thr):
    rows, room = base_rows(n, m, k)
    room += 4096
    ops = [G.r1(G.RX, q, 0.3 + 0.02 * q) for q in range(10)] + ([G.truncate()] if thr else [])
    one = sum_of(n, rows, room, thr, True)
    one.run(ops)
    fused = sum_of(n, rows, room, thr, False)
    fused.run(ops)
    assert len(fused) == len(one) and (len(one) == room - 4096) == (thr == 0.0)
    assert fused == one
    fused.run(ops)  # full groups now
    one.run(ops)
    assert fused == one
    del fused, one
    assert lib().ppvm_release_cached_memory() == 0


CASES = [(40, 33000, 8, 1e-3), (40, 33000, 9, 0.0), (40, 33000, 10, 1e-5), (130, 40000, 7, 1e-3), (130, 33000, 0, 1e-4),
         (300, 33000, 9, 1e-4), (40, 3000, 10, 0.0), (300, 9000, 0, 0.0),
         (40, 262200, 6, 1e-3), (40, 262200, 5, 0.0)]  # 64 slots: in order, 32: placed from the scratch


@pytest.mark.parametrize("case", range(len(CASES)))
def test_fused_equals_gate_by_gate(case):
    check(*CASES[case])


def test_scratch_placement_of_large_groups():
    script = "from tests.test_gpu_run_large_groups import check\n" \
             "for c in [(40, 3000, 10, 0.0), (130, 9000, 9, 1e-4), (300, 9000, 0, 1e-4), (40, 33000, 7, 0.0)]: check(*c)\n" \
             "print('checked')"
    r = subprocess.run([sys.executable, "-c", script], cwd=ROOT, capture_output=True, text=True, timeout=300,
                       env=dict(os.environ, PPVM_RUN_SCRATCH_MIN_GROUPS="1"))
    assert r.returncode == 0, r.stdout[-2000:] + r.stderr[-2000:]
    assert "checked" in r.stdout
