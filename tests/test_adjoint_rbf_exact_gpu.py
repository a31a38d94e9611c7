"""The quotients by a lengthscale in the RBF matrix are those of a division. Where every one is a whole
number nothing but the exponential may round, so an entry is off by no more than CUDA's bound for
exp (1 ulp) and the rounding of the value that it is held against. With one coordinate an entry is
exp(-1/2 t t) of the rounded quotient t, which plain torch computes in the same steps, bit for bit."""
from __future__ import annotations

from decimal import Decimal, localcontext

import numpy as np
import pytest
import torch

from remora_b200 import ops

from helpers import to_host

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("lengthscales", [[49.0], [3.0, 49.0, 107.0], [0.1], [1e300, 1e-300]])
def test_whole_quotients(cuda, lengthscales):
    d = len(lengthscales)
    rs = np.random.default_rng(d)
    steps = rs.integers(0, 21, (70, d)).astype(np.float64)
    ls = np.array(lengthscales)
    X = steps * ls
    # differences of multiples round for lengthscales that are no whole number: keep exact quotients
    diff = X[:, None, :] - X[None, :, :]
    whole = steps[:, None, :] - steps[None, :, :]
    exact = np.all(diff / ls == whole, axis=-1)
    assert exact.mean() > 0.2
    K = to_host(ops.rbf_kernel(torch.from_numpy(X).cuda(), torch.from_numpy(ls).cuda(), 0.0))
    r2 = (whole * whole).sum(-1)
    with localcontext() as ctx:
        ctx.prec = 40
        values = {v: float((Decimal(v) / -2).exp()) for v in np.unique(r2).tolist()}
    ref = np.vectorize(values.get)(r2)
    assert np.all(np.abs(K - ref)[exact] <= 1.5 * np.spacing(ref)[exact])


@pytest.mark.parametrize("scale", [1.0, 1e-3, 1e-150, 1e150])
def test_one_coordinate_bit_for_bit(cuda, scale):
    g = torch.Generator(device="cuda").manual_seed(7)
    x = torch.randn(1000, generator=g, device="cuda", dtype=torch.float64) * scale
    for ls in ((torch.rand(20, generator=g, device="cuda", dtype=torch.float64) + 0.5) * scale):
        t = (x[:, None] - x[None, :]) / ls
        assert torch.equal(ops.rbf_kernel(x[:, None], ls.reshape(1), 0.0), torch.exp(-0.5 * (t * t)))


@pytest.mark.parametrize("x,ls", [([1.7e308, -1.7e308, 0.0], 1.0), ([1e300, -1e300, 0.0], 1e-280),
                                  ([float("inf"), 0.0, 1.0], 2.0), ([5e-324, 0.0, 1e-310], 1e-290)])
def test_distances_beyond_the_range(cuda, x, ls):
    X = torch.tensor(x, device="cuda", dtype=torch.float64)
    l = torch.tensor([ls], device="cuda", dtype=torch.float64)
    t = (X[:, None] - X[None, :]) / l
    K = ops.rbf_kernel(X[:, None], l, 0.0)
    assert torch.equal(torch.nan_to_num(K, nan=7.0), torch.nan_to_num(torch.exp(-0.5 * (t * t)), nan=7.0))
