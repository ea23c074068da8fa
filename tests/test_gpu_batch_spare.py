"""Spare words of live batches: bounded together, given back, and nothing depends on them.

Every batch reserves room for its instances to grow into inside a launch, up to 1 GB; all live
batches of a device together reserve at most 4 GB, and the others grow through the host."""

import pytest
import torch

from ppvm_b200 import gates as G
from ppvm_b200._lib import lib
from ppvm_b200.batch import Instance, PauliSumBatch

from tests.test_gpu_batch import check_batch

pytestmark = pytest.mark.gpu

REGION = 64 << 20  # a region of 2^20 terms is 54 MB


def used():
    return torch.cuda.mem_get_info()[1] - torch.cuda.mem_get_info()[0]


def batch():
    rx = [G.r1(G.RX, q, 0.3 + 0.01 * q) for q in range(9)]
    w = "Z" * 9 + "I" * 11
    insts = [Instance(20, [(w, 1.0)], rx + [G.truncate(), G.truncate()], 1e-12, None) for _ in range(2)]
    b = PauliSumBatch(insts, capacity=[1 << 20, 256])  # the second instance outgrows its region
    b.run()
    return b


def test_spare_words_of_many_batches():
    torch.zeros(1, device="cuda")
    for _ in range(2):  # again: what the first batches held has been given back
        assert lib().ppvm_release_cached_memory() == 0
        before = used()
        batches = [batch() for _ in range(10)]
        assert lib().ppvm_release_cached_memory() == 0  # pools that a growth through the host replaced
        for b in batches:
            check_batch(b)
            assert int(b.capacities()[1]) >= 512
        held = used() - before
        assert 3 << 30 < held < (4 << 30) + 10 * REGION + (256 << 20), held
        del batches, b
