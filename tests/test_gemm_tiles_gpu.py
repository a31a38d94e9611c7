"""The GEMM's tiles, FP64 and FP32, at the sizes where they can go wrong: tile edges and remainders in
m, n and k, every storage order, operands without 16-byte alignment, both triangle masks and
split K. Entries are small integers, so every product and sum is exact in either type and the
result must equal the integer product."""
from __future__ import annotations

import numpy as np
import pytest
import torch

from remora_b200 import ops

pytestmark = pytest.mark.gpu

SHAPES = [(1, 1, 1), (31, 33, 15), (33, 16, 17), (65, 15, 129), (64, 17, 16), (97, 161, 33), (640, 1100, 31),
          (1500, 1400, 65), (70, 9, 2100), (130, 200, 2049)]


def _dev(M: np.ndarray, row: bool, shift: int, dtype) -> torch.Tensor:
    """M on the device, row- or column-major, `shift` elements past an aligned address and
    with a leading dimension larger than needed by as many."""
    X = M if row else M.T
    r, c = X.shape
    buf = torch.zeros(r * (c + shift) + shift, dtype=dtype, device="cuda")
    V = buf[shift:].view(r, c + shift)[:, :c]
    V.copy_(torch.from_numpy(np.ascontiguousarray(X)))
    return V if row else V.t()


@pytest.mark.parametrize("dtype", [torch.float64, torch.float32])
@pytest.mark.parametrize("shift", [0, 1])
@pytest.mark.parametrize("orders", [(0, 0, 0), (1, 0, 1), (0, 1, 1), (1, 1, 0)])
@pytest.mark.parametrize("shape", SHAPES)
def test_gemm_tiles_exact(cuda, shape, orders, shift, dtype):
    m, n, k = shape
    rs = np.random.default_rng(m * 7 + n * 3 + k)
    A, B, C = (rs.integers(-8, 9, s).astype(np.float64) for s in ((m, k), (k, n), (m, n)))
    Ad, Bd, Cd = (_dev(X, bool(o), shift, dtype) for X, o in zip((A, B, C), orders))
    ops.gemm(Ad, Bd, Cd, 2.0, -3.0)
    assert np.array_equal(Cd.cpu().numpy(), 2.0 * (A @ B) - 3.0 * C)
    ops.gemm(Ad, Bd, Cd, 1.0, 0.0)
    assert np.array_equal(Cd.cpu().numpy(), A @ B)


@pytest.mark.parametrize("dtype", [torch.float64, torch.float32])
@pytest.mark.parametrize("shift", [0, 1])
@pytest.mark.parametrize("upper", [False, True])
@pytest.mark.parametrize("n,k", [(1, 3), (33, 16), (65, 40), (129, 7), (700, 33), (1500, 20)])
def test_syrk_tiles_exact(cuda, n, k, upper, shift, dtype):
    rs = np.random.default_rng(n + k)
    A, C = rs.integers(-8, 9, (n, k)).astype(np.float64), rs.integers(-8, 9, (n, n)).astype(np.float64)
    Ad, Cd = _dev(A, True, shift, dtype), _dev(C, False, shift, dtype)
    ops.syrk(Ad, Cd, -1.0, upper)
    full = C - A @ A.T
    want = np.triu(full) + np.tril(C, -1) if upper else np.tril(full) + np.triu(C, 1)
    assert np.array_equal(Cd.cpu().numpy(), want)


@pytest.mark.parametrize("dtype", [torch.float64, torch.float32])
@pytest.mark.parametrize("n", [5, 33, 64, 500])
def test_gemm_in_place_left(cuda, n, dtype):
    """B <- L B over its own operand with 64 rows, as the factorisations' block rows do: no tile
    may overwrite rows that another one still reads."""
    rs = np.random.default_rng(n)
    L, B = rs.integers(-4, 5, (64, 64)).astype(np.float64), rs.integers(-4, 5, (64, n)).astype(np.float64)
    Ld, Bd = _dev(L, True, 0, dtype), _dev(B, False, 0, dtype)
    ops.gemm(Ld, Bd, Bd, 1.0, 0.0)
    assert np.array_equal(Bd.cpu().numpy(), L @ B)
