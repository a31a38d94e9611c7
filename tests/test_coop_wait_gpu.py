"""The LU panel on a cooperative grid with a limit of a nanosecond: a grid barrier's wait runs out, the
factorisation ends with the panel's first column in the status word (the swaps must not use an
incomplete piv), the error word has the site, and the next factorisation is not affected."""
from __future__ import annotations

import ctypes

import pytest
import torch

from remora_b200 import _lib, ops

pytestmark = pytest.mark.gpu


def test_grid_barrier_timeout_stops_the_factorisation(cuda):
    lib = _lib.lib()
    n = 4400  # more rows than the cluster panel takes
    g = torch.Generator(device="cuda").manual_seed(1)
    A = torch.randn((n, n), generator=g, device="cuda", dtype=torch.float64)
    F, site = A.clone(), ctypes.c_int(-1)
    assert lib.rc_device_status(None) == 0 and lib.rc_set_wait_limit_ns(1) == 0
    try:
        info, _ = ops.getrf(F)
        status = lib.rc_device_error_site(None, ctypes.byref(site))
    finally:
        lib.rc_set_wait_limit_ns(2_000_000_000)
    assert (status, site.value) == (5, 500)
    assert info == 1
    assert lib.rc_device_status(None) == 0
    info, piv = ops.getrf(A)
    rows = torch.arange(n, device="cuda")
    assert info == 0 and bool(((piv >= rows) & (piv < n)).all())
