"""Stretches of local ops on small sums around the lengths from which they go to the composed Clifford
pass (64 ops up to 256 qubits, 48 above), between rotations and with heads of fewer and more than 64
ops before them, against the oracle."""

import numpy as np
import pytest

from ppvm_b200 import gates as G
from ppvm_b200.paulisum import PauliSum

from tests.helpers import oracle_from
from tests.test_gpu_parity import same
from tests.test_gpu_small import random_terms

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [5, 256, 257, 400])
@pytest.mark.parametrize("k", [47, 48, 49, 63, 64, 65])
def test_local_stretches(n, k):
    rng = np.random.default_rng(n + k)
    terms = random_terms(rng, n, 60)
    local = [G.g1((G.H, G.S, G.SQRT_X, G.Y)[int(rng.integers(4))], int(rng.integers(n))) for _ in range(k)]
    rot = [G.r1((G.RX, G.RY, G.RZ)[i % 3], int(rng.integers(n)), 0.3) for i in range(3)]
    head = [G.r1(G.RY, 1, 0.1 + 0.01 * i) for i in range(70)]
    s = PauliSum([w for w, _ in terms], n, [c for _, c in terms], min_abs_coeff=1e-3, exact_order=True)
    o = oracle_from(terms, n, 1e-3)
    for ops in (rot + local, local + rot + [G.truncate()], head + local + rot + local, local):
        s.run(ops)
        want = o.run_ops(ops, counts=True)
        assert np.array_equal(s.live_counts(), want)
        same(s, o)
