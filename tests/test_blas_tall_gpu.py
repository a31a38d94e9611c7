"""Products with more rows than a grid's y extent holds tiles (65535 of 64 rows, FP64; of 128, FP32),
in every storage order. Entries are small integers, so the result must equal the integer product."""
from __future__ import annotations

import pytest
import torch

from remora_b200 import ops

pytestmark = pytest.mark.gpu


def _ints(shape, row: bool, dtype, seed: int) -> torch.Tensor:
    g = torch.Generator(device="cuda").manual_seed(seed)
    r, c = shape if row else shape[::-1]
    X = torch.randint(-8, 9, (r, c), generator=g, device="cuda").to(dtype)
    return X if row else X.t()


@pytest.mark.parametrize("dtype,m", [(torch.float64, 4_200_001), (torch.float32, 8_400_001)])
@pytest.mark.parametrize("orders", [(0, 0, 0), (1, 1, 1), (0, 1, 1), (1, 0, 0)])
def test_gemm_tall(cuda, orders, dtype, m):
    A, B = _ints((m, 8), bool(orders[0]), dtype, 1), _ints((8, 8), bool(orders[1]), dtype, 2)
    C = _ints((m, 8), bool(orders[2]), dtype, 3)
    want = sum(A[:, q:q + 1] * B[q:q + 1, :] for q in range(8)) + C
    ops.gemm(A, B, C, 1.0, 1.0)
    assert torch.equal(C, want)
