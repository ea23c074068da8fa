"""The profile's algorithmic bytes: an op's or run's bytes once, however many launches it takes.

A fused run whose groups could go one per lane launches both group kernels, one of which returns at
once; the loss channel launches two kernels."""

import numpy as np
import pytest

from ppvm_b200 import gates as G
from ppvm_b200.paulisum import LossyPauliSum, PauliSum

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m", [3000, 20000])  # below and above the size from which both kernels are launched
def test_group_bytes_of_a_run(m):
    rng = np.random.default_rng(m)
    n = 64
    words = list(dict.fromkeys("".join("IXYZ"[int(v)] for v in row)
                               for row in rng.choice(4, p=[0.9, 0.04, 0.03, 0.03], size=(2 * m, n))))[:m]
    s = PauliSum(words, n, rng.uniform(-1, 1, m).tolist(), min_abs_coeff=0.0, capacity=1 << 17)
    untouched = sum(not set(w[:8]) & set("YZ") for w in words)
    s.profile(True)
    s.run([G.r1(G.RX, q, 0.3) for q in range(8)])
    s.profile(False)
    groups = s.profile_read()["run_groups"]
    assert groups["launches"] == 1
    assert groups["bytes"] == (m - untouched + len(s) - untouched) * (16 + 8)


def test_bytes_of_a_loss_channel():
    rng = np.random.default_rng(3)
    n, m = 70, 2000
    words = list(dict.fromkeys("".join("IXYZL"[int(v)] for v in rng.integers(0, 5, n)) for _ in range(m)))
    s = LossyPauliSum(words, n, rng.uniform(-1, 1, len(words)).tolist(), min_abs_coeff=0.0)
    s.profile(True)
    s.run([G.loss_channel(4, 0.2)])
    s.profile(False)
    loss = s.profile_read()["loss"]
    assert loss["launches"] == 1 and len(s) > len(words)
    assert loss["bytes"] == (len(words) + len(s)) * (16 * 4 + 8)
