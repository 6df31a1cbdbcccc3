"""Device memory of batches (B200): ordinary ones reuse the library's pool, so that neither making nor
releasing one waits for the device, and large ones give their memory back.
"""
import numpy as np
import pytest
import torch

import gx

pytestmark = pytest.mark.gpu

PARAMS = gx.PhysicsParams(1.0, 0.05)


def free_bytes():
    torch.cuda.synchronize()
    return torch.cuda.mem_get_info()[0]


def evaluate(sizes):
    n = int(np.sum(sizes))
    x = np.random.default_rng(5).normal(size=(6, n))
    b = gx.Batch(np.concatenate([[0], np.cumsum(sizes)]), PARAMS)
    b.set_state(*x, np.full(n, 1.0 / n))
    b.compute_accelerations(gx.PRECISION_MIXED)
    acc = b.get_state()["ax"]
    return b, acc


def test_the_next_batch_reuses_the_memory():
    sizes = [1024 + 512 * (k % 20) for k in range(100)]
    first, acc = evaluate(sizes)
    first.diagnostics()
    first.close()
    left = free_bytes()
    for _ in range(3):
        b, again = evaluate(sizes)
        assert free_bytes() == left
        b.diagnostics()
        b.close()
        assert free_bytes() == left and np.array_equal(acc, again)


def test_a_large_batch_gives_its_memory_back():
    sizes = [16] * 300_000  # 384 MB of state
    before = free_bytes()
    b, _ = evaluate(sizes)
    assert before - free_bytes() >= 80 * 16 * 300_000
    b.close()
    assert before - free_bytes() <= 64 << 20  # the lists of items stay in the pool
