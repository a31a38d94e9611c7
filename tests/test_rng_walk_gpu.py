"""Fills large enough that a thread walks several rows (column groups), and the normal
transform at the ends of its range, against the oracle."""
from __future__ import annotations

import numpy as np
import pytest
import torch

from remora_b200 import ops

from helpers import to_host

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("row_major,shape", [(True, (10003, 21)), (False, (301, 38002))])
def test_walk(cuda, orc, row_major, shape):
    rows, cols = shape
    key = [0xFFFFFFFF, 3, 0x80000000, 77]
    new = lambda dt: torch.empty((rows, cols), dtype=dt, device="cuda") if row_major else \
        torch.empty((cols, rows), dtype=dt, device="cuda").t()  # noqa: E731
    B = new(torch.int32)
    ops.generate_bits(B, key)
    words = orc.rng_fill("bits", key, rows, cols)
    assert np.array_equal(to_host(B).view(np.uint32), words)
    X = new(torch.float32)
    ops.generate_normal(X, key)
    # the transform of the same words in 64 bits: u is the float next below x 2^-32
    u = words.astype(np.float32) * np.float32(2.0 ** -32)
    u = np.nextafter(u, np.float32(0)).astype(np.float64)
    q, full = np.float32(2.0 * np.pi), cols // 4 * 4
    u = u[:, :full].reshape(rows, -1, 4)
    with np.errstate(divide="ignore"):
        r0, r1 = np.sqrt(-2 * np.log(u[..., 0])), np.sqrt(-2 * np.log(u[..., 1]))
    a0, a1 = ((q * u[..., k].astype(np.float32)).astype(np.float64) for k in (2, 3))
    ref = np.stack([r0 * np.sin(a0), r0 * np.cos(a0), r1 * np.sin(a1), r1 * np.cos(a1)], -1).reshape(rows, full)
    got = to_host(X)[:, :full]
    fin = np.isfinite(ref)
    assert np.array_equal(np.isfinite(got), fin)
    # logarithm 1 ulp, root half of that and 1 ulp of its own, sine 2 ulp, product half: below 4 ulp of
    # the radius (at most 6.7) or of the value
    r = np.repeat(np.stack([r0, r1], -1), 2, axis=-1).reshape(rows, full)
    assert np.all(np.abs(got[fin] - ref[fin]) <= 4 * 2.0 ** -23 * r[fin])
