"""Kept plans of the batched solver beside one another: a tall batch's plan, then a short batch's (which
needs a tenth of the shared memory), then the tall plan again, in both precisions and forms."""
from __future__ import annotations

import numpy as np
import pytest
import torch

from remora_b200 import ops

pytestmark = pytest.mark.gpu


def _systems(n: int, count: int, dtype):
    rs = np.random.default_rng(n)
    mats = []
    for _ in range(count):
        G = rs.standard_normal((n, n))
        mats.append(G @ G.T / n + np.eye(n))
    return ops.BatchedSystems(mats, [rs.standard_normal(n) for _ in range(count)], dtype=dtype)


@pytest.mark.parametrize("autotune", [False, True])
@pytest.mark.parametrize("dtype", [torch.float64, torch.float32])
def test_tall_plan_after_a_short_one(cuda, dtype, autotune):
    tall, short = _systems(512, 3, dtype), _systems(16, 5, dtype)
    A0, b0 = tall.A.clone(), tall.b.clone()
    tall.solve(autotune=autotune)
    want = (tall.A.clone(), tall.b.clone())
    short.solve(autotune=autotune)
    tall.A.copy_(A0)
    tall.b.copy_(b0)
    tall.solve(autotune=autotune)
    torch.cuda.synchronize()
    assert not tall.info.any() and not short.info.any()
    assert torch.equal(tall.A, want[0]) and torch.equal(tall.b, want[1])
