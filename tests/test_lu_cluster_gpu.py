"""The LU panel on a thread-block cluster at the sizes where it can go wrong: rows at the edges of
its CTAs (256 each, up to 16 of them) and beyond them, strips of 16 columns cut short, equal
pivots, a zero pivot and a column of NaN. The factors obey |P A - L U| <= n u |L||U| entry by
entry (Higham's bound for Gaussian elimination, u the element type's unit, and once more for the
product here, in FP64); pivots are in range and, among equals, the lowest row."""
from __future__ import annotations

import pytest
import torch

from remora_b200 import ops

pytestmark = pytest.mark.gpu


def _matrix(n: int, row_major: bool, dtype, seed: int) -> torch.Tensor:
    g = torch.Generator(device="cuda").manual_seed(seed)
    A = torch.rand((n, n), generator=g, device="cuda", dtype=torch.float64) * 2 - 1
    return A.to(dtype) if row_major else A.to(dtype).t()


def _permuted(A: torch.Tensor, piv: torch.Tensor) -> torch.Tensor:
    order = list(range(A.shape[0]))
    for i, p in enumerate(piv.tolist()):
        order[i], order[p] = order[p], order[i]
    return A[torch.tensor(order, device=A.device)]


@pytest.mark.parametrize("dtype,u", [(torch.float64, 2.0 ** -53), (torch.float32, 2.0 ** -24)])
@pytest.mark.parametrize("row_major", [True, False])
@pytest.mark.parametrize("n", [1, 15, 17, 63, 65, 127, 255, 256, 257, 513, 1030, 2049, 4096, 4200])
def test_getrf_cluster_edges(cuda, n, row_major, dtype, u):
    A = _matrix(n, row_major, dtype, n)
    F = A.clone()
    info, piv = ops.getrf(F)
    assert info == 0
    rows = torch.arange(n, device="cuda")
    assert bool(((piv >= rows) & (piv < n)).all())
    F = F.double()
    L, U = torch.tril(F, -1) + torch.eye(n, device="cuda", dtype=torch.float64), torch.triu(F)
    PA = _permuted(A.double(), piv)
    bound = n * (u + 2.0 ** -53) * (L.abs() @ U.abs())
    assert bool(((L @ U - PA).abs() <= bound).all())
    assert float(torch.tril(F, -1).abs().max() if n > 1 else 0.0) <= 1.0


@pytest.mark.parametrize("n", [40, 300, 1100])
def test_getrf_equal_pivots_take_the_lowest_row(cuda, n):
    A = _matrix(n, False, torch.float64, 3)
    A[:, 0] = 1.0 - 2.0 * (torch.arange(n, device="cuda") % 2).double()
    A[0, 0] = 0.5
    F = A.clone()
    info, piv = ops.getrf(F)
    assert info == 0 and int(piv[0]) == 1


@pytest.mark.parametrize("col", [0, 20, 63, 64, 200])
def test_getrf_zero_and_nan_columns(cuda, col):
    A = _matrix(300, True, torch.float64, 4)
    Z = A.clone()
    Z[:, col] = 0.0
    info, piv = ops.getrf(Z)
    assert info == col + 1 and int(piv[col]) == col
    A[:, col] = float("nan")
    info, piv = ops.getrf(A)
    rows = torch.arange(300, device="cuda")
    assert info == 0 and bool(((piv >= rows) & (piv < 300)).all()) and int(piv[col]) == col
    assert not bool(torch.isnan(A[:, :col]).any())
