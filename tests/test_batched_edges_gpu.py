"""The batched solver at the edges of its 32-row panels and warp tiles: every size's factor
against Higham's componentwise bound |A - L L^T| <= g |L||L^T|, g = (n + 1) 2^-53 (float
matrices: plus the two roundings of a stored factor and of the updates that reach it, one per
panel), the solution's residual against the same factor (|L L^T x - b| <= 3 n u |L||L^T||x|, u
the element type's unit), the untouched upper triangles, and failing pivots."""
from __future__ import annotations

import numpy as np
import pytest
import torch

from remora_b200 import ops

pytestmark = pytest.mark.gpu

SIZES = [1, 2, 15, 16, 17, 31, 32, 33, 48, 63, 64, 65, 95, 96, 97, 127, 129, 160, 255, 256, 257, 289, 480, 511, 512]


def _spd(n: int) -> np.ndarray:
    G = np.random.default_rng(n).standard_normal((n, n))
    return G @ G.T / n + 0.1 * np.eye(n)


@pytest.mark.parametrize("dtype", [torch.float64, torch.float32])
def test_batched_every_edge(cuda, dtype):
    np_t = np.float64 if dtype == torch.float64 else np.float32
    mats = [np.triu(_spd(n), 1) * 7.0 + np.tril(_spd(n)) for n in SIZES]  # the upper part is not read
    mats = [m.astype(np_t).astype(np.float64) for m in mats]
    rhs = [np.random.default_rng(n).standard_normal(n).astype(np_t).astype(np.float64) for n in SIZES]
    s = ops.BatchedSystems(mats, rhs, dtype=dtype)
    s.solve(autotune=False)
    assert not s.info.any()
    u = 2.0 ** -53 if dtype == torch.float64 else 2.0 ** -24
    for i, n in enumerate(SIZES):
        F = s.factor(i).double().cpu().numpy()
        assert np.array_equal(np.triu(F, 1), np.triu(mats[i], 1)), n
        L = np.tril(F).astype(np.longdouble)
        S = np.tril(mats[i]) + np.tril(mats[i], -1).T
        aL = np.abs(L) @ np.abs(L).T
        g = (n + 1) * 2.0 ** -53 + ((2 + (n + 31) // 32) * u if dtype == torch.float32 else 0.0)
        assert (np.abs(S - L @ L.T) <= g * aL).all(), n
        x = s.solution(i).double().cpu().numpy()
        assert (np.abs(L @ (L.T @ x) - rhs[i]) <= 3 * n * u * (aL @ np.abs(x)) + u * np.abs(rhs[i])).all(), n


@pytest.mark.parametrize("value", [-1.0, 0.0, float("nan")])
def test_batched_failing_pivots(cuda, value):
    bad = {7: 0, 12: 31, 15: 32, 18: 150, 24: 511}
    mats, rhs = [_spd(n) for n in SIZES], [np.ones(n) for n in SIZES]
    for i, j in bad.items():
        mats[i][j, j] = value
    s = ops.BatchedSystems(mats, rhs)
    s.solve(autotune=False)
    assert s.info.cpu().tolist() == [bad[i] + 1 if i in bad else 0 for i in range(len(SIZES))]
    for i in bad:
        assert torch.equal(s.solution(i).cpu(), torch.ones(SIZES[i], dtype=torch.float64))
