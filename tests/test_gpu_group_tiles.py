"""Group, export, copy and one-child channel kernels at their edges.

Fused runs: groups of 0 to 11 coordinates (2^10 slots is the largest a group fills; 11 falls back),
group counts around 2^15 (four groups per warp from there on, the last tile partly filled), against
the oracle bit for bit; scratch placement (forced on every run, in a child process) gives the same
list in the same order as ordered placement.  Copies, one-part exports and the one-child channels
(amplitude damping, loss) run at sizes around a block and a tile; order and bits are exact."""

import hashlib
import json
import os
import subprocess
import sys

import numpy as np
import pytest

from ppvm_b200 import gates as G
from ppvm_b200.paulisum import LossyPauliSum, PauliSum
from ppvm_b200.sharded import DeviceShare

from tests.helpers import lossy_oracle_from, oracle_from
from tests.test_gpu_parity import same, same_set

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def distinct_words(rng, n, m, letters="IXYZ", p=None):
    words = {}
    while len(words) < m:
        for row in rng.choice(len(letters), size=(m, n), p=p):
            words["".join(letters[int(v)] for v in row)] = None
    return list(words)[:m]


def coordinate_case(k):
    """600 invariants (X patterns over 20 qubits), each with one word of Z on all k run qubits and
    up to two of Z or I."""
    rng = np.random.default_rng(40 + k)
    n = 20 + max(k, 2)
    rest = "I" * (n - 20 - k)
    words = {}
    for inv in distinct_words(rng, 20, 600, "IX"):
        for bits in [[1] * k, rng.integers(0, 2, k), rng.integers(0, 2, k)]:
            words["".join("IZ"[int(b)] for b in bits) + rest + inv] = None
    terms = [(w, float(c)) for w, c in zip(words, rng.uniform(-1, 1, len(words)))]
    ops = [G.r1(G.RX, q, 0.3 + 0.05 * q) for q in range(max(k, 2))] + [G.truncate()]
    return n, terms, ops, 1e-2


def count_case(m):
    rng = np.random.default_rng(m)
    n = 40
    words = ["I" * 6 + w for w in distinct_words(rng, n - 6, m, "IX")]
    hot = rng.integers(0, 4, size=(m, 6))
    words = ["".join("IZIZ"[int(v)] for v in h) + w[6:] for h, w in zip(hot, words)]
    terms = [(w, float(c)) for w, c in zip(words, rng.uniform(-1, 1, m))]
    ops = [G.r1(G.RX, q, 0.4) for q in range(6)] + [G.truncate()]
    return n, terms, ops, 1e-2


def gpu_run(n, terms, ops, thr):
    s = PauliSum([w for w, _ in terms], n, [c for _, c in terms], min_abs_coeff=thr, exact_order=False)
    s.run(ops)
    return s


def digests():
    out = []
    for case in [coordinate_case(k) for k in (1, 5, 6, 10)] + [count_case(m) for m in (1500, 33001)]:
        x, z, c = gpu_run(*case).export()
        out.append(hashlib.sha256(x.tobytes() + z.tobytes() + c.tobytes()).hexdigest())
    return out


@pytest.mark.parametrize("k", range(0, 12))
def test_groups_of_k_coordinates(k):
    n, terms, ops, thr = coordinate_case(k)
    o = oracle_from(terms, n, thr)
    o.run_ops(ops)
    same_set(gpu_run(n, terms, ops, thr), o)


@pytest.mark.parametrize("m", [32767, 32768, 32769, 40003])
def test_group_counts_around_four_per_warp(m):
    n, terms, ops, thr = count_case(m)
    o = oracle_from(terms, n, thr)
    o.run_ops(ops)
    same_set(gpu_run(n, terms, ops, thr), o)


def test_scratch_placement_keeps_the_order():
    script = "import json; from tests.test_gpu_group_tiles import digests; print(json.dumps(digests()))"
    r = subprocess.run([sys.executable, "-c", script], cwd=ROOT, capture_output=True, text=True, timeout=600,
                       env=dict(os.environ, PPVM_RUN_SCRATCH_MIN_GROUPS="1"))
    assert r.returncode == 0, r.stdout[-2000:] + r.stderr[-2000:]
    assert json.loads(r.stdout.strip().splitlines()[-1]) == digests()


@pytest.mark.parametrize("n", [20, 100, 300])
@pytest.mark.parametrize("m", [1, 255, 256, 257, 3000])
def test_copies_and_one_part_exports(n, m):
    rng = np.random.default_rng(n + m)
    terms = list(zip(distinct_words(rng, n, m), rng.uniform(-1, 1, m)))
    s = PauliSum([w for w, _ in terms], n, [float(c) for _, c in terms], min_abs_coeff=0.0)
    x, z, c = s.export()
    for got, want in zip(s.copy().export(), (x, z, c)):
        assert got.tobytes() == want.tobytes()
    share = DeviceShare(s)
    zero = np.zeros(s.W, dtype=np.uint64)
    rows, counts = share.export(zero, zero, 1)
    assert counts.tolist() == [m] and len(s) == 0
    want = np.concatenate([x, z, c.view(np.uint64)[:, None]], axis=1)
    assert np.array_equal(rows.cpu().numpy().view(np.uint64).reshape(m, -1), want)
    share.append(rows)
    for got, ref in zip(s.export(), (x, z, c)):
        assert got.tobytes() == ref.tobytes()


@pytest.mark.parametrize("m", [1, 513, 1023, 1024, 1025, 2049, 5000])
@pytest.mark.parametrize("lossy", [False, True])
def test_one_child_channels(lossy, m):
    rng = np.random.default_rng(m)
    n = 70
    letters, p = ("IXYZL", [0.6, 0.08, 0.08, 0.12, 0.12]) if lossy else ("IXYZ", [0.6, 0.1, 0.1, 0.2])
    # the first four qubits carry the channels; many terms differ there alone
    base = distinct_words(rng, n - 4, max(1, m // 20), letters, p)
    words = {}
    while len(words) < m:
        words["".join(letters[int(v)] for v in rng.integers(0, len(letters), 4)) + base[int(rng.integers(len(base)))]] = None
    terms = [(w, float(c)) for w, c in zip(words, rng.uniform(-1, 1, m))]
    ops = [G.amplitude_damping(0, 0.2), G.amplitude_damping(1, 1.0), G.amplitude_damping(0, 0.0)]
    if lossy:
        ops += [G.loss_channel(0, 0.2), G.loss_channel(3, 0.0), G.loss_channel(2, 1.0), G.amplitude_damping(2, 0.1),
                G.loss_channel(69, 0.3)]
    cls, orc = (LossyPauliSum, lossy_oracle_from) if lossy else (PauliSum, oracle_from)
    s = cls([w for w, _ in terms], n, [c for _, c in terms], min_abs_coeff=0.0, exact_order=True, capacity=m)
    o = orc(terms, n, thr=0.0)
    for op in ops:  # capacity m: the first op that appends also grows and replays
        s.run([op])
        o.run_ops([op])
        same(s, o)
