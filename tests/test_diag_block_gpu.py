"""The 128-block of the Cholesky factorisation at the edges of its 16- and 32-row sub-blocks:
every order and element type against Higham's componentwise bound |A - L L^T| <= g |L||L^T|
with g = (n + 1) 2^-53 (plus two roundings to the element type), values next to underflow and
overflow, and the index of a failing pivot."""
from __future__ import annotations

import numpy as np
import pytest
import torch

from remora_b200 import ops

pytestmark = pytest.mark.gpu


def _spd(n: int, seed: int) -> np.ndarray:
    G = np.random.default_rng(seed).standard_normal((n, n))
    return G @ G.T / n + 0.1 * np.eye(n)


@pytest.mark.parametrize("dtype", [torch.float64, torch.float32])
@pytest.mark.parametrize("row_major", [True, False])
@pytest.mark.parametrize("upper", [False, True])
@pytest.mark.parametrize("n", [1, 2, 15, 16, 17, 31, 33, 64, 79, 97, 127, 128])
def test_diag_block_residual(cuda, n, upper, row_major, dtype):
    A = torch.from_numpy(_spd(n, n)).to("cuda", dtype)
    L = A.clone() if row_major else A.t().clone().t()
    assert ops.potrf(L, upper=upper) == 0
    A64, L64 = A.double().cpu().numpy(), L.double().cpu().numpy()
    other = np.tril(L64, -1) - np.tril(A64, -1) if upper else np.triu(L64, 1) - np.triu(A64, 1)
    assert not other.any()
    F = np.triu(L64).T if upper else np.tril(L64)
    S = np.triu(A64) + np.triu(A64, 1).T if upper else np.tril(A64) + np.tril(A64, -1).T
    R = np.abs((S - F.astype(np.longdouble) @ F.T.astype(np.longdouble)).astype(np.float64))
    g = (n + 1) * 2.0 ** -53 + (2.1 * 2.0 ** -24 if dtype == torch.float32 else 0.0)
    assert (R <= g * (np.abs(F) @ np.abs(F).T)).all()


@pytest.mark.parametrize("scale", [2.0 ** -1000, 2.0 ** -500, 2.0 ** 500, 2.0 ** 1000])
def test_diag_block_scales(cuda, scale):
    """Powers of four scale A and its factor exactly, so the same bound holds for the rescaled
    factor: pivots below 1e-300 take another route."""
    A = _spd(128, 5)
    L = torch.from_numpy(A).cuda() * scale
    assert ops.potrf(L) == 0
    F = np.tril(L.cpu().numpy()) / scale ** 0.5
    R = np.abs((A - F.astype(np.longdouble) @ F.T.astype(np.longdouble)).astype(np.float64))
    assert (R <= 129 * 2.0 ** -53 * (np.abs(F) @ np.abs(F).T)).all()


@pytest.mark.parametrize("value", [-1.0, 0.0, float("nan")])
@pytest.mark.parametrize("bad", [1, 16, 17, 32, 33, 100, 113, 128, 129, 300])
def test_diag_block_failing_pivot(cuda, bad, value):
    A = torch.from_numpy(_spd(300, 9)).cuda()
    A[bad - 1, bad - 1] = value
    assert ops.potrf(A) == bad
