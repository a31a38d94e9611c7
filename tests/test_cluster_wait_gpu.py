"""The LU panel's waits on a thread-block cluster with a limit of a nanosecond, which every wait exceeds:
the panel goes on to the end in all of its CTAs, the factors are those of an unlimited run, and the
error word tells of the wait (site 501) until it is read. A zero pivot ends a panel of many CTAs in
all of them, at any column of a strip."""
from __future__ import annotations

import ctypes

import pytest
import torch

from remora_b200 import _lib, ops

pytestmark = pytest.mark.gpu


def _matrix(n: int) -> torch.Tensor:
    g = torch.Generator(device="cuda").manual_seed(n)
    return torch.randn((n, n), generator=g, device="cuda", dtype=torch.float64)


@pytest.mark.parametrize("n", [200, 1000, 2049])
def test_exceeded_limit_is_reported_and_harmless(cuda, n):
    lib = _lib.lib()
    A = _matrix(n)
    want, site = A.clone(), ctypes.c_int(-1)
    info, want_piv = ops.getrf(want)
    assert info == 0 and lib.rc_device_status(None) == 0
    got = A.clone()
    assert lib.rc_set_wait_limit_ns(1) == 0
    try:
        info, piv = ops.getrf(got)
        status = lib.rc_device_error_site(None, ctypes.byref(site))
    finally:
        lib.rc_set_wait_limit_ns(2_000_000_000)
    assert (status, site.value) == (5, 501) and info == 0
    assert torch.equal(got, want) and torch.equal(piv, want_piv)
    assert lib.rc_device_status(None) == 0


@pytest.mark.parametrize("col", [0, 1, 15, 16, 40, 63, 64])
def test_zero_pivot_ends_a_panel_of_many_ctas(cuda, col):
    A = _matrix(2100)
    A[:, col] = 0.0
    info, piv = ops.getrf(A)
    assert info == col + 1 and int(piv[col]) == col
    B = _matrix(2100)
    info, _ = ops.getrf(B)  # the next factorisation is not affected
    assert info == 0 and _lib.lib().rc_device_status(None) == 0
