"""Triangular solves across the strip kernel's edges (128-row blocks, 512-row panels, 8- and
16-column strips, the change to products a block at a time), aligned and unaligned, against plain
FP64 torch; and the factorisation that shares it."""
from __future__ import annotations

import pytest
import torch

from remora_b200 import ops

pytestmark = pytest.mark.gpu
TOL = {torch.float64: 1e-13, torch.float32: 1e-5}  # the parity bars, relative Frobenius


def _mat(r, c, dtype, row, pad, g):
    big = torch.rand((r, c + pad) if row else (c, r + pad), generator=g, device="cuda", dtype=torch.float64) * 2 - 1
    big = big.to(dtype)
    return big[:, :c] if row else big[:, :r].t()


@pytest.mark.parametrize("dtype", [torch.float64, torch.float32])
@pytest.mark.parametrize("upper,a_row,b_row", [(False, False, False), (True, False, True), (False, True, True),
                                               (True, True, False)])
@pytest.mark.parametrize("m,n,pad", [(1, 1, 0), (127, 9, 1), (129, 8, 0), (512, 17, 0), (513, 40, 3), (640, 1184, 0),
                                     (200, 1185, 1), (384, 4737, 0)])
def test_trsm(cuda, dtype, upper, a_row, b_row, m, n, pad):
    g = torch.Generator(device="cuda").manual_seed(m * n)
    A = _mat(m, m, dtype, a_row, pad, g)
    A.diagonal().add_(m)
    X = _mat(m, n, dtype, b_row, pad, g)
    ref = torch.linalg.solve_triangular(A.double(), X.double(), upper=upper)
    ops.trsm(A, X, upper=upper)
    assert torch.linalg.norm(X.double() - ref) <= TOL[dtype] * torch.linalg.norm(ref)


@pytest.mark.parametrize("dtype", [torch.float64, torch.float32])
@pytest.mark.parametrize("n,row,pad", [(511, False, 0), (513, True, 1), (1100, False, 0), (1409, False, 1)])
def test_potrf_across_panels(cuda, dtype, n, row, pad):
    g = torch.Generator(device="cuda").manual_seed(n)
    G = torch.randn((n, n), generator=g, device="cuda", dtype=torch.float64)
    S = (G @ G.t() / n + torch.eye(n, device="cuda", dtype=torch.float64)).to(dtype)
    A = _mat(n, n, dtype, row, pad, g)
    A.copy_(torch.tril(S, 0) + torch.triu(torch.full_like(S, 7.0), 1))
    assert ops.potrf(A) == 0
    assert torch.all(torch.triu(A, 1) == torch.triu(torch.full_like(S, 7.0), 1))
    L = torch.tril(A).double()
    ref = torch.linalg.cholesky(S.double())
    assert torch.linalg.norm(L - ref) <= TOL[dtype] * torch.linalg.norm(ref)


def test_threads_solve_panels_of_different_heights(cuda):
    """Solves of 128 and of 512 rows from several host threads, each on a stream of its own."""
    import threading

    wrong = []

    def work(m):
        s = torch.cuda.Stream()
        with torch.cuda.stream(s):
            g = torch.Generator(device="cuda").manual_seed(m)
            A = torch.rand((m, m), generator=g, device="cuda", dtype=torch.float64)
            A.diagonal().add_(m)
            B = torch.rand((m, 8), generator=g, device="cuda", dtype=torch.float64)
            ref = torch.linalg.solve_triangular(A, B, upper=False)
            for _ in range(200):
                X = B.clone()
                try:
                    ops.trsm(A, X)
                except Exception as e:  # noqa: BLE001
                    wrong.append(e)
                    return
            if not torch.linalg.norm(X - ref) <= 1e-13 * torch.linalg.norm(ref):
                wrong.append(m)

    threads = [threading.Thread(target=work, args=(m,)) for m in (128, 512, 256, 512)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not wrong
