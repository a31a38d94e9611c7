"""Matrices of subnormal numbers are positive definite as well. Entries are integers times 2^-1074,
the spacing down there: with F the factor times 2^537, |A - F F^T| is at most (n + 1) 2^-53 |F||F^T|
(Higham) plus the rounding of each of the n updates of an entry to the spacing, half of 1 in these
units."""
from __future__ import annotations

import numpy as np
import pytest
import torch

from remora_b200 import ops

pytestmark = pytest.mark.gpu


def _subnormal(n: int) -> np.ndarray:
    B = np.random.default_rng(n).integers(-8, 9, (n, n)).astype(np.float64)
    return np.tril(B, -1) + np.tril(B, -1).T + 65536.0 * np.eye(n)  # diagonally dominant: positive definite


def _check(A: np.ndarray, L: np.ndarray) -> None:
    n = len(A)
    F = (np.tril(L) * 2.0 ** 537).astype(np.longdouble)
    bound = 0.5 * n + (n + 1) * 2.0 ** -53 * (np.abs(F) @ np.abs(F).T)
    assert (np.abs(A - F @ F.T) <= bound).all(), n


@pytest.mark.parametrize("n", [1, 2, 16, 17, 33, 64, 128, 200])
def test_potrf_of_subnormal_numbers(cuda, n):
    A = _subnormal(n)
    L = torch.from_numpy(A * 2.0 ** -1074).cuda()
    assert ops.potrf(L) == 0
    _check(A, L.cpu().numpy())


def test_batched_of_subnormal_numbers(cuda):
    mats = [_subnormal(n) for n in (1, 16, 31, 32, 33, 70)]
    s = ops.BatchedSystems([m * 2.0 ** -1074 for m in mats], [np.zeros(len(m)) for m in mats])
    s.solve(autotune=False)
    assert not s.info.any()
    for i, m in enumerate(mats):
        _check(m, s.factor(i).cpu().numpy())
