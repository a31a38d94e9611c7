"""Fills whose contiguous direction is shorter than a block, at its powers of two and beside them: a
block then takes several steps of the other direction. Words against the oracle, the memory around
the matrix untouched."""
from __future__ import annotations

import numpy as np
import pytest
import torch

from remora_b200 import ops

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("row_major", [True, False])
@pytest.mark.parametrize("short,long", [(1, 1), (1, 4001), (2, 3000), (3, 70001), (5, 257), (8, 1000), (21, 5003),
                                        (64, 300), (127, 129), (129, 1030), (255, 260), (257, 258)])
def test_narrow_fills(cuda, orc, short, long, row_major):
    rows, cols = (long, 4 * short - 3) if row_major else (short, long)  # `short` 4-column groups, or rows
    key = [5, 0xFFFFFFFF, 77, 1 << 31]
    lead = (cols if row_major else rows) + 3
    buf = torch.full(((rows if row_major else cols) + 1, lead), 7, dtype=torch.int32, device="cuda")
    V = buf[:-1, :cols] if row_major else buf[:-1, :rows].t()
    ops.generate_bits(V, key)
    assert np.array_equal(V.cpu().numpy().view(np.uint32), orc.rng_fill("bits", key, rows, cols))
    assert bool((buf[-1] == 7).all()) and bool((buf[:, lead - 3:] == 7).all())
