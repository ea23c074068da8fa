"""Amplitude damping and the loss channel on sums whose grid is larger than what is resident at once.

The apply kernel of these channels commits the new live count in its last block, and blocks of the
same grid that have no tile may start after that.  From some 0.7 to 1.3 million terms such blocks
exist for sure (8 blocks an SM are launched, 5 fit), and the appended children cross tile borders, so
that the new count has more tiles than the old one.  Every repeat on a fresh copy must give the
oracle's list, bit for bit and in order.  Also: an op that outgrows the capacity writes nothing,
and is applied once when it is replayed on the grown storage."""

import numpy as np
import pytest

from ppvm_b200 import gates as G
from ppvm_b200._lib import lib
from ppvm_b200.paulisum import LossyPauliSum, PauliSum

from tests.helpers import lossy_oracle_from, oracle_from
from tests.test_gpu_parity import same

pytestmark = pytest.mark.gpu


def spread(k):
    """2^k terms (Z or Y on each of the first k qubits) from one."""
    return [G.r1(G.RX, q, 0.4 + 0.01 * q) for q in range(k)]


def digest(s):
    return [a.tobytes() for a in s.export()]


@pytest.mark.parametrize("n", [40, 80])
def test_damping_at_a_million_terms(n):
    w = "Z" * 19 + "I" * (n - 19)
    base = PauliSum([w], n, min_abs_coeff=0.0, exact_order=True, capacity=1 << 21)
    o = oracle_from([(w, 1.0)], n, thr=0.0)
    base.run(spread(19))  # 524288 terms, then 786432 and 1179648
    o.run_ops(spread(19))
    ops = [G.amplitude_damping(0, 0.2), G.amplitude_damping(7, 0.1)]
    o.run_ops(ops)
    want = digest(o)
    for _ in range(20):
        s = base.copy()
        s.run(ops[:1])
        s.run(ops[1:])
        assert digest(s) == want
        s = base.copy()
        s.run(ops)  # in one list the bound on the live count, and with it the grid, doubles per op
        assert digest(s) == want


def test_loss_at_a_million_terms():
    n, w = 40, "Z" * 17 + "I" * 23
    base = LossyPauliSum([w], n, min_abs_coeff=0.0, exact_order=True, capacity=1 << 21)
    o = lossy_oracle_from([(w, 1.0)], n, thr=0.0)
    head = spread(17) + [G.reset_loss_channel(q) for q in (0, 5, 9, 16)]  # 663552 terms, a third of them L on each
    base.run(head)
    o.run_ops(head)
    ops = [G.loss_channel(5, 0.2), G.loss_channel(16, 0.3)]  # 884736 and 1179648
    o.run_ops(ops)
    want = digest(o)
    for _ in range(20):
        s = base.copy()
        s.run(ops)
        assert digest(s) == want


@pytest.mark.parametrize("lossy", [False, True])
@pytest.mark.parametrize("m", [4096, 4097, 6000])
def test_replay_after_growth(lossy, m):
    # no cached handle with more room: the storage holds 4096 terms at least, and m exactly from there on
    assert lib().ppvm_release_cached_memory() == 0
    rng = np.random.default_rng(m)
    n = 70
    letter = "L" if lossy else "Z"
    words = {}
    while len(words) < m:  # a third with the parent letter on qubit 0, half of these with their counterpart
        body = "".join("IXYZ"[int(v)] for v in rng.integers(0, 4, n - 1))
        for c in ([letter], [letter, "I"], ["X"], ["Y"])[int(rng.integers(4))]:
            words[c + body] = None
    terms = [(w, float(c)) for w, c in zip(list(words)[:m], rng.uniform(-1, 1, m))]
    cls, orc = (LossyPauliSum, lossy_oracle_from) if lossy else (PauliSum, oracle_from)
    op = G.loss_channel(0, 0.3) if lossy else G.amplitude_damping(0, 0.3)
    s = cls([w for w, _ in terms], n, [c for _, c in terms], min_abs_coeff=0.0, exact_order=True, capacity=m)
    o = orc(terms, n, thr=0.0)
    launches = s.launch_count()
    s.run([op])
    o.run_ops([op])
    assert s.launch_count() - launches == 4  # both kernels twice: the first apply found no room
    same(s, o)
    s.run([op])  # no child is new now
    o.run_ops([op])
    same(s, o)
