"""The likelihood's adjoint and the RBF kernels at the edges of their tiles (64 points, 128-row
blocks, 512-row panels), against plain FP64 numpy."""
from __future__ import annotations

import numpy as np
import pytest
import torch

from remora_b200 import ops
from remora_b200._lib import call

from helpers import to_dev, to_host

pytestmark = pytest.mark.gpu
U = 2.0 ** -53


@pytest.mark.parametrize("n", [1, 33, 127, 128, 129, 511, 513, 700, 1030])
def test_nll_adjoint(cuda, n):
    rs = np.random.default_rng(n)
    G = rs.standard_normal((n, n))
    A = G @ G.T / n + np.eye(n)  # condition number about 5
    L = np.linalg.cholesky(A) + np.triu(rs.standard_normal((n, n)), 1)  # the upper part is not read
    a = rs.standard_normal(n)
    Ld, ad = to_dev(L, False), torch.from_numpy(a).cuda()
    out = torch.full((n, n + 3), 7.0, dtype=torch.float64, device="cuda")  # columns of n + 3
    call("rc_nll_adjoint_f64", n, Ld.data_ptr(), n, ad.data_ptr(), out.data_ptr(), n + 3,
         torch.cuda.current_stream().cuda_stream)
    got = out.cpu().numpy()
    assert np.all(got[:, n:] == 7.0)
    got = got[:, :n].T
    assert np.array_equal(got, got.T)
    ref = 0.5 * (np.linalg.inv(A) - np.outer(a, a))
    # an inverse from a factor of condition kappa is good to a small multiple of n kappa u
    assert np.linalg.norm(got - ref) <= 40 * n * U * np.linalg.norm(ref)


@pytest.mark.parametrize("n,d", [(1, 1), (63, 3), (64, 16), (65, 2), (130, 7), (321, 16)])
def test_rbf_matrix_and_gradient(cuda, n, d):
    rs = np.random.default_rng(n + d)
    X, ls = rs.standard_normal((n, d)), rs.uniform(0.5, 2.0, d)
    ls[0] = -ls[0]
    if d > 2:
        ls[1] = 1e300  # a reciprocal outside the fast range
    Xd, ld = torch.from_numpy(X).cuda(), torch.from_numpy(ls).cuda()
    K = to_host(ops.rbf_kernel(Xd, ld, 0.25))
    Z = (X[:, None, :] - X[None, :, :]) / ls
    r2 = (Z * Z).sum(-1)
    ref = np.exp(-0.5 * r2)
    # d squares of rounded quotients and their sum, both sides; the exponential's own rounding
    assert np.all(np.abs(K - (ref + 0.25 * np.eye(n))) <= 2 * U * (r2 * (d + 4) + 8) * (ref + 0.25))
    assert np.array_equal(K, K.T)
    Kbar = rs.standard_normal((n, n))  # not symmetric
    g = torch.empty(d, dtype=torch.float64, device="cuda")
    call("rc_rbf_lengthscale_grad_f64", n, d, Xd.data_ptr(), ld.data_ptr(), to_dev(Kbar, False).data_ptr(), n,
         g.data_ptr(), torch.cuda.current_stream().cuda_stream)
    terms = (Kbar * ref)[:, :, None] * (X[:, None, :] - X[None, :, :]) ** 2
    scale = np.abs(terms).sum((0, 1)) / np.abs(ls * ls * ls)
    assert np.all(np.abs(g.cpu().numpy() - terms.sum((0, 1)) / (ls * ls * ls)) <= 4 * U * (n * n + 200) * scale)


def test_gradient_of_equal_points_far_out(cuda):
    """Distances are zero wherever the points lie, also beside the unused part of a tile."""
    X = torch.full((5, 2), 1e200, dtype=torch.float64, device="cuda")
    ls, Kbar = torch.ones(2, dtype=torch.float64, device="cuda"), torch.ones((5, 5), dtype=torch.float64, device="cuda")
    g = torch.empty(2, dtype=torch.float64, device="cuda")
    call("rc_rbf_lengthscale_grad_f64", 5, 2, X.data_ptr(), ls.data_ptr(), Kbar.data_ptr(), 5, g.data_ptr(),
         torch.cuda.current_stream().cuda_stream)
    assert torch.all(g == 0)
    assert torch.all(ops.rbf_kernel(X, ls, 0.0) == 1)
