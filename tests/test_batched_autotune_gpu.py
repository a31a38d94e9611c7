"""The batched solver's autotuner in a fresh process: every candidate runs once before it is timed (a
first launch loads its kernel), and the caller's systems come out as without it."""
from __future__ import annotations

import subprocess
import sys
from pathlib import Path

import pytest

pytestmark = pytest.mark.gpu

PROGRAM = """
import numpy as np
import torch
from remora_b200 import _lib, ops
rs = np.random.default_rng(1)
mats = [(lambda G: G @ G.T / 40 + np.eye(40))(rs.standard_normal((40, 40))) for _ in range(20)]
rhs = [rs.standard_normal(40) for _ in range(20)]
count = _lib.lib().rc_launch_count
def solve(autotune):
    s = ops.BatchedSystems(mats, rhs)
    torch.cuda.synchronize()
    before = count()
    s.solve(autotune=autotune)
    torch.cuda.synchronize()
    assert not s.info.any()
    return count() - before, s
plain, a = solve(False)
tuned, b = solve(True)
again, c = solve(True)
assert torch.equal(a.A, b.A) and torch.equal(a.b, b.b) and torch.equal(a.A, c.A)
print(plain, tuned - plain, again - plain)
"""


def test_candidates_are_warm_when_timed(cuda):
    root = Path(__file__).resolve().parents[1]
    res = subprocess.run([sys.executable, "-c", PROGRAM], cwd=root, capture_output=True, text=True, timeout=300)
    assert res.returncode == 0, res.stderr
    _, tuning, kept = map(int, res.stdout.split())
    assert tuning == 2 * 2  # two candidates, each once cold and once timed
    assert kept == 0
