"""Instances that grew inside a launch run from shared memory again in the next run, when they fit.

Shared memory of the batch kernel's launches, from the profiler's trace: after the growth it must hold
the grown regions (32 bytes and more a term), not only the initial ones."""

import json

import pytest
import torch

from ppvm_b200 import gates as G
from ppvm_b200.batch import Instance, PauliSumBatch

from tests.test_gpu_batch import check_batch

pytestmark = pytest.mark.gpu


def shared_bytes(path, run):
    with torch.profiler.profile(activities=[torch.profiler.ProfilerActivity.CUDA]) as prof:
        run()
        torch.cuda.synchronize()
    prof.export_chrome_trace(str(path))
    events = [e for e in json.loads(path.read_text())["traceEvents"] if "k_batch<" in e.get("name", "")]
    if not events:
        pytest.skip("the profiler recorded no kernels on this machine")
    return max(int(e["args"]["shared memory"]) for e in events)


def test_grown_instances_become_resident(tmp_path):
    torch.zeros(1, device="cuda")
    insts = []
    for m in (3, 9):  # 2^m terms; the initial regions hold 256
        rx = [G.r1(G.RX, q, 0.3 + 0.01 * q) for q in range(m)]
        insts.append(Instance(20, [("Z" * m + "I" * (20 - m), 1.0)], rx + [G.truncate(), G.truncate()], 1e-12, None))
    b = PauliSumBatch(insts)
    first = shared_bytes(tmp_path / "a.json", b.run_persistent)
    check_batch(b)
    cap = int(b.capacities().max())
    assert cap >= 512
    second = shared_bytes(tmp_path / "b.json", b.run_persistent)
    check_batch(b)
    assert first < 32 * cap <= second  # planes, coefficients and links alone take 32 bytes a term
    third = shared_bytes(tmp_path / "c.json", b.run_persistent)  # nothing grows any more
    check_batch(b)
    assert third == second
