"""The work a program has this library do, as cases that can be timed and compared.

Every case is one call (or one short sequence of calls) of the public entry points in
``remora_b200.ops``, on inputs a program would have in hand on the GPU. ``listed()`` holds
the representative ones, ``draw(rng)`` gives another of the same ranges, ``prepare`` makes
the inputs of one case from a seed, ``run`` is one pass, ``work`` the bytes and operations
the pass cannot do without, and ``exact`` the result of plain FP64 torch code.
"""
from __future__ import annotations

import math

import torch

from remora_b200 import ops

DT = {"f64": torch.float64, "f32": torch.float32}


def listed() -> list[dict]:
    return [
        # C = A B of small odd matrices, all in a program's inner loop: launch latency counts.
        {"name": "gemm_f64_small", "op": "gemm", "dtype": "f64", "m": 61, "n": 37, "k": 53, "a_row": True,
         "b_row": True, "c_row": True, "beta": 0.0},
        # prod(A, B) at a middle size of the BLAS-3 sweep, mixed storage orders.
        {"name": "gemm_f64_4096", "op": "gemm", "dtype": "f64", "m": 4096, "n": 4096, "k": 4096, "a_row": True,
         "b_row": False, "c_row": False, "beta": 0.0},
        # A Gram / covariance matrix in single precision, C += A A^T: the sweep's SYRK.
        {"name": "syrk_f32_8192", "op": "syrk", "dtype": "f32", "n": 8192, "k": 4096, "a_row": True, "c_row": False,
         "upper": False, "beta": 1.0},
        # A triangular solve with many right-hand sides: the sweep's TRSM.
        {"name": "trsm_f64_8192", "op": "trsm", "dtype": "f64", "n": 8192, "nrhs": 1024, "a_row": False,
         "b_row": False, "upper": False, "unit": False, "left": True},
        # The plain SPD solve of a moderate system, cholesky_decomposition(A).solve(B).
        {"name": "chol_f64_1024", "op": "chol_solve", "n": 1024, "nrhs": 16},
        # The same in single precision on a ragged size, with the decomposition kept:
        # potrf, then a forward and a backward triangular solve.
        {"name": "chol_f32_3001", "op": "chol", "dtype": "f32", "n": 3001, "nrhs": 40, "a_row": False},
        # LU with partial pivoting of a general matrix (pivoting_lu_decomposition).
        {"name": "getrf_f64_2048", "op": "getrf", "dtype": "f64", "n": 2048, "a_row": False},
        # The headline: a large SPD solve with a TF32 factor, refined to FP64 backward error.
        {"name": "mixed_tf32_32768", "op": "mixed", "precision": "tf32", "n": 32768, "nrhs": 64, "kappa": 1e2},
        # The refined solve where the conditioning asks for the emulated-FP64 factor.
        {"name": "mixed_emu64_16384", "op": "mixed", "precision": "emu64", "n": 16384, "nrhs": 64, "kappa": 1e4},
        # Many independent uneven SPD systems (RBF kernels of 16 to 512 points), one launch.
        {"name": "batched_f64_1024", "op": "batched", "dtype": "f64", "count": 1024, "max_n": 512},
        # GP marginal likelihood, forward and backward through Cholesky and the solves.
        {"name": "gp_f64_8192", "op": "gp", "n": 8192, "d": 16},
        # A normal fill of 2^28 floats.
        {"name": "rng_normal_16384", "op": "rng", "kind": "normal", "rows": 16384, "cols": 16384, "row_major": True},
    ]


def _size(rng, lo: int, hi: int) -> int:
    """Log-uniform in [lo, hi]; half of them are whatever came out, odd ones included, the
    others the near multiple of 16."""
    v = int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))
    if rng.random() < 0.5:
        v = max(lo, min(hi, (v + 8) // 16 * 16))
    return max(lo, min(hi, v))


def draw(rng) -> dict:
    op = rng.choice(["gemm", "gemm", "syrk", "trsm", "chol_solve", "chol", "getrf", "mixed", "batched", "gp", "rng"])
    dtype = rng.choice(["f64", "f32"])
    flag = lambda: rng.random() < 0.5  # noqa: E731
    if op == "gemm":
        return {"op": op, "dtype": dtype, "m": _size(rng, 24, 4096), "n": _size(rng, 24, 4096),
                "k": _size(rng, 24, 4096), "a_row": flag(), "b_row": flag(), "c_row": flag(),
                "beta": rng.choice([0.0, 1.0])}
    if op == "syrk":
        return {"op": op, "dtype": dtype, "n": _size(rng, 64, 6000), "k": _size(rng, 24, 4096), "a_row": flag(),
                "c_row": flag(), "upper": flag(), "beta": rng.choice([0.0, 1.0])}
    if op == "trsm":
        return {"op": op, "dtype": dtype, "n": _size(rng, 64, 8192), "nrhs": _size(rng, 1, 1024), "a_row": flag(),
                "b_row": flag(), "upper": flag(), "unit": flag(), "left": flag()}
    if op == "chol_solve":
        return {"op": op, "n": _size(rng, 32, 4096), "nrhs": _size(rng, 1, 64)}
    if op == "chol":
        return {"op": op, "dtype": dtype, "n": _size(rng, 32, 6000), "nrhs": _size(rng, 1, 128), "a_row": flag()}
    if op == "getrf":  # in FP64: single-precision runs may differ in a pivot by rounding alone
        return {"op": op, "dtype": "f64", "n": _size(rng, 48, 4096), "a_row": flag()}
    if op == "mixed":
        precision = rng.choice(["tf32", "bf16", "emu64"])
        return {"op": op, "precision": precision, "n": _size(rng, 1500, 16384), "nrhs": _size(rng, 1, 64),
                "kappa": 1e4 if precision == "emu64" else 1e2}
    if op == "batched":
        return {"op": op, "dtype": dtype, "count": _size(rng, 16, 1024), "max_n": _size(rng, 32, 512)}
    if op == "gp":
        return {"op": op, "n": _size(rng, 256, 6000), "d": rng.randint(2, 16)}
    return {"op": op, "kind": rng.choice(["normal", "normal", "uniform", "bits"]), "rows": _size(rng, 100, 16384),
            "cols": _size(rng, 100, 16384), "row_major": flag()}


# -- inputs ---------------------------------------------------------------------------


def _gen(seed: int) -> torch.Generator:
    return torch.Generator(device="cuda").manual_seed(seed)


def _uniform(g, r: int, c: int, dtype, row: bool) -> torch.Tensor:
    """U[-1, 1], row- or column-major."""
    if row:
        return torch.rand((r, c), generator=g, device="cuda", dtype=dtype) * 2 - 1
    return (torch.rand((c, r), generator=g, device="cuda", dtype=dtype) * 2 - 1).t()


def _normal(g, r: int, c: int, dtype, row: bool) -> torch.Tensor:
    if row:
        return torch.randn((r, c), generator=g, device="cuda", dtype=dtype)
    return torch.randn((c, r), generator=g, device="cuda", dtype=dtype).t()


def _hartley_rows(M: torch.Tensor, signs: list[torch.Tensor]) -> None:
    """M <- M Q^T in place for the orthogonal Q = H S_k ... H S_1 (H the discrete Hartley
    transform, S random signs), a few rows at a time."""
    n = M.shape[1]
    step = max(1, (1 << 26) // n)
    for r in range(0, M.shape[0], step):
        x = M[r:r + step]
        for s in signs:
            f = torch.fft.fft(x * s, dim=1)
            x = (f.real - f.imag) / math.sqrt(n)
        M[r:r + step] = x


def _spd_with_spectrum(n: int, kappa: float, g) -> torch.Tensor:
    """Q diag(lambda) Q^T, dense and exactly symmetric, lambda log-spaced to 1 / kappa."""
    signs = [torch.randint(0, 2, (n,), generator=g, device="cuda").double() * 2 - 1 for _ in range(3)]
    A = torch.diag(torch.logspace(0.0, -math.log10(kappa), n, device="cuda", dtype=torch.float64))
    _hartley_rows(A, signs)
    A = A.t().contiguous()
    _hartley_rows(A, signs)
    A.add_(A.t().contiguous()).mul_(0.5)
    return A


def _rbf_systems(case: dict, seed: int):
    """Host matrices and right-hand sides of the batch: RBF kernels on points ~ N(0, I_8),
    lengthscale 1, noise 1e-2, sizes uniform in [16, max_n] (one set of them per case)."""
    g = _gen(seed)
    count, max_n = case["count"], case["max_n"]
    sizes = torch.randint(16, max_n + 1, (count,), generator=torch.Generator().manual_seed(count * 1000 + max_n)).tolist()
    pts = torch.randn((count, max_n, 8), generator=g, device="cuda", dtype=torch.float64)
    rhs = torch.randn((count, max_n), generator=g, device="cuda", dtype=torch.float64).cpu()
    mats = []
    for at in range(0, count, 64):
        P = pts[at:at + 64]
        q = (P * P).sum(-1)
        d2 = (q[:, :, None] + q[:, None, :] - 2 * P @ P.transpose(1, 2)).clamp_min_(0.0)
        K = torch.exp(-0.5 * d2)
        K = 0.5 * (K + K.transpose(1, 2))
        K.diagonal(dim1=1, dim2=2).fill_(1.01)
        mats += [K[i, :n, :n].contiguous().cpu().numpy() for i, n in enumerate(sizes[at:at + 64])]
    return mats, [rhs[i, :n].numpy() for i, n in enumerate(sizes)]


def prepare(case: dict, seed: int) -> dict:
    op = case["op"]
    st: dict = {"case": case}
    g = _gen(seed)
    dt = DT.get(case.get("dtype", "f64"))
    if op == "gemm":
        st["A"] = _uniform(g, case["m"], case["k"], dt, case["a_row"])
        st["B"] = _uniform(g, case["k"], case["n"], dt, case["b_row"])
        st["C0"] = _uniform(g, case["m"], case["n"], dt, case["c_row"])
        st["C"] = st["C0"].clone()
    elif op == "syrk":
        st["A"] = _uniform(g, case["n"], case["k"], dt, case["a_row"])
        st["C0"] = _uniform(g, case["n"], case["n"], dt, case["c_row"])
        st["C"] = st["C0"].clone()
    elif op == "trsm":
        n = case["n"]
        A = _uniform(g, n, n, dt, case["a_row"])
        if case["unit"]:  # small entries beside the ones that the solve puts on the diagonal
            A.mul_(1.0 / n)
        A.diagonal().add_(n)
        st["A"] = A
        shape = (n, case["nrhs"]) if case["left"] else (case["nrhs"], n)
        st["B"] = _uniform(g, *shape, dt, case["b_row"])
    elif op in ("chol_solve", "chol"):
        n = case["n"]
        G = _normal(g, n, n, torch.float64, True)
        A = G @ G.T / n
        A.add_(A.t().contiguous()).mul_(0.5)
        A.diagonal().add_(1e-2 if op == "chol_solve" else 1e-1)
        st["A"] = A.to(dt) if case.get("a_row") else A.to(dt).t()
        st["B"] = _normal(g, n, case["nrhs"], dt, False)
    elif op == "getrf":
        st["A"] = _normal(g, case["n"], case["n"], dt, case["a_row"])
    elif op == "mixed":
        st["A"] = _spd_with_spectrum(case["n"], case["kappa"], g)
        st["B"] = _normal(g, case["n"], case["nrhs"], torch.float64, False)
    elif op == "batched":
        mats, rhs = _rbf_systems(case, seed)
        st["sys"] = ops.BatchedSystems(mats, rhs, dtype=dt)
        st["A0"], st["b0"] = st["sys"].A.clone(), st["sys"].b.clone()
    elif op == "gp":
        st["X"] = _normal(g, case["n"], case["d"], torch.float64, True)
        st["y"] = _normal(g, case["n"], 1, torch.float64, True).reshape(-1)
        st["ls"] = torch.rand(case["d"], generator=g, device="cuda", dtype=torch.float64) * 1.5 + 0.5
    elif op == "rng":
        st["key"] = torch.randint(0, 1 << 31, (4,), generator=g, device="cuda").tolist()
        dtype = torch.int32 if case["kind"] == "bits" else torch.float32
        r, c = case["rows"], case["cols"]
        st["X"] = torch.zeros((r, c), device="cuda", dtype=dtype) if case["row_major"] else \
            torch.zeros((c, r), device="cuda", dtype=dtype).t()
    else:
        raise ValueError(op)
    return st


# -- one pass -------------------------------------------------------------------------


def run(st: dict):
    case = st["case"]
    op = case["op"]
    if op == "gemm":
        if case["beta"]:
            st["C"].copy_(st["C0"])
        ops.gemm(st["A"], st["B"], st["C"], 1.0, case["beta"])
        return st["C"]
    if op == "syrk":
        if case["beta"]:
            st["C"].copy_(st["C0"])
        ops.syrk(st["A"], st["C"], 1.0, case["upper"], case["beta"])
        return st["C"]
    if op == "trsm":
        X = st["B"].clone()
        ops.trsm(st["A"], X, case["upper"], case["unit"], case["left"])
        return X
    if op == "chol_solve":
        X = st["B"].clone()
        ops.cholesky_solve(st["A"], X)
        return X
    if op == "chol":
        L, X = st["A"].clone(), st["B"].clone()
        ops.potrf(L)
        ops.trsm(L, X)
        ops.trsm(L.t(), X, upper=True)
        return {"L": L, "X": X}
    if op == "getrf":
        LU = st["A"].clone()
        _, piv = ops.getrf(LU)
        return {"LU": LU, "piv": piv}
    if op == "mixed":
        X, _, _ = ops.spd_solve_mixed(st["A"], st["B"], case["precision"])
        return X
    if op == "batched":
        s = st["sys"]
        s.A.copy_(st["A0"])
        s.b.copy_(st["b0"])
        s.solve()
        return {"A": s.A, "b": s.b, "info": s.info}
    if op == "gp":
        f, grad, Kbar = ops.gp_nll_and_grad(st["X"], st["y"], st["ls"], 1e-2)
        return {"f": f, "g": grad, "Kbar": Kbar}
    X = st["X"]
    if case["kind"] == "normal":
        ops.generate_normal(X, st["key"])
    elif case["kind"] == "uniform":
        ops.generate_uniform(X, st["key"])
    else:
        ops.generate_bits(X, st["key"])
    return X


def work(case: dict) -> dict:
    op = case["op"]
    e = 4 if case.get("dtype") == "f32" else 8
    n = case.get("n", 0)
    if op == "gemm":
        m, k = case["m"], case["k"]
        return {"bytes": e * (m * k + k * n + m * n * (2 if case["beta"] else 1)), "flops": 2 * m * n * k}
    if op == "syrk":
        k = case["k"]
        return {"bytes": e * (n * k + n * (n + 1) / 2 * (2 if case["beta"] else 1)), "flops": n * (n + 1) * k}
    if op == "trsm":
        return {"bytes": e * (n * (n + 1) / 2 + 2 * n * case["nrhs"]), "flops": n * n * case["nrhs"]}
    if op in ("chol_solve", "chol"):
        q = case["nrhs"]
        out = 0 if op == "chol_solve" else n * (n + 1) / 2
        return {"bytes": e * (n * (n + 1) / 2 + out + 2 * n * q), "flops": n ** 3 / 3 + 2 * n * n * q}
    if op == "getrf":
        return {"bytes": e * 2 * n * n, "flops": 2 * n ** 3 / 3}
    if op == "mixed":
        q = case["nrhs"]
        return {"bytes": 8 * (n * n + 2 * n * q), "flops": n ** 3 / 3 + 2 * n * n * q}
    if op == "batched":  # expectations over sizes uniform in [16, max_n]
        sizes = range(16, case["max_n"] + 1)
        mean = lambda p: sum(s ** p for s in sizes) / len(sizes)  # noqa: E731
        c = case["count"]
        return {"bytes": c * e * (mean(2) + 3 * mean(1)), "flops": c * (mean(3) / 3 + 2 * mean(2))}
    if op == "gp":  # Cholesky, and the inverse its adjoint needs; K is made and its adjoint returned
        return {"bytes": 8 * n * n, "flops": n ** 3 / 3 + 2 * n ** 3 / 3 + 4 * n * n * case["d"]}
    # twelve rounds and four injections of 32-bit integer work, a few float operations each
    return {"bytes": 4 * case["rows"] * case["cols"], "flops": 30 * case["rows"] * case["cols"]}


# -- the same in plain FP64 torch -------------------------------------------------------


def _threefry(rows: torch.Tensor, cols4: torch.Tensor, key) -> list[torch.Tensor]:
    """The four 32-bit words of each (row, 4-column group) block, as int64 tensors."""
    m = 0xFFFFFFFF
    k = [int(v) & m for v in key]
    k4 = 0x1BD11BDA ^ k[0] ^ k[1] ^ k[2] ^ k[3]
    r0 = [10, 11, 13, 23, 6, 17, 25, 18]
    r1 = [26, 21, 27, 5, 20, 11, 10, 20]
    x = (rows & 0xFFFF)[:, None].expand(-1, cols4.numel()).contiguous()
    y = (rows >> 32)[:, None].expand_as(x).contiguous()
    z = (cols4 & 0xFFFF)[None, :].expand_as(x).contiguous()
    w = (cols4 >> 32)[None, :].expand_as(x).contiguous()
    rot = lambda v, r: ((v << r) | (v >> (32 - r))) & m  # noqa: E731

    def mix(x, y, z, w, base):
        for r in range(4):
            s = base + r
            if r % 2 == 0:
                x = (x + y) & m
                y = rot(y, r0[s]) ^ x
                z = (z + w) & m
                w = rot(w, r1[s]) ^ z
            else:
                x = (x + w) & m
                w = rot(w, r0[s]) ^ x
                z = (z + y) & m
                y = rot(y, r1[s]) ^ z
        return x, y, z, w

    x, y, z, w = (x + k[0]) & m, (y + k[1]) & m, (z + k[2]) & m, (w + k[3]) & m
    x, y, z, w = mix(x, y, z, w, 0)
    x, y, z, w = (x + k[1]) & m, (y + k[2]) & m, (z + k[3]) & m, (w + k4 + 1) & m
    x, y, z, w = mix(x, y, z, w, 4)
    x, y, z, w = (x + k[2]) & m, (y + k[3]) & m, (z + k4) & m, (w + k[0] + 2) & m
    x, y, z, w = mix(x, y, z, w, 0)
    return [(x + k[3]) & m, (y + k4) & m, z, (w + k[0] + k[1] + 3) & m]


def _exact_rng(case: dict, key) -> torch.Tensor:
    r, c = case["rows"], case["cols"]
    groups = (c + 3) // 4
    cols4 = torch.arange(groups, device="cuda", dtype=torch.int64) * 4
    out = torch.empty((r, 4 * groups), device="cuda", dtype=torch.int64 if case["kind"] == "bits" else torch.float64)
    step = max(1, (1 << 24) // groups)
    # the stream's uniforms are floats: x rounded to 24 bits, times 2^-32, one float towards 0
    unit = lambda v: torch.nextafter(v.float() * 2.0 ** -32, torch.zeros((), device="cuda")).double()  # noqa: E731
    for at in range(0, r, step):
        rows = torch.arange(at, min(at + step, r), device="cuda", dtype=torch.int64)
        v = _threefry(rows, cols4, key)
        if case["kind"] == "bits":
            v = [torch.where(t >= 1 << 31, t - (1 << 32), t) for t in v]
        else:
            v = [unit(t) for t in v]
            if case["kind"] == "normal":
                a, b = (torch.sqrt(-2.0 * torch.log(t)) for t in v[:2])
                p, q = (2.0 * math.pi * t for t in v[2:])
                v = [a * torch.sin(p), a * torch.cos(p), b * torch.sin(q), b * torch.cos(q)]
        out[at:at + len(rows)] = torch.stack(v, dim=-1).reshape(len(rows), -1)
    return out[:, :c].int() if case["kind"] == "bits" else out[:, :c]


def exact(case: dict, seed: int):
    op = case["op"]
    if op == "batched":
        mats, rhs = _rbf_systems(case, seed)
        A, b = [], []
        for m, v in zip(mats, rhs):
            M = torch.from_numpy(m).cuda().to(DT[case["dtype"]]).double()
            v = torch.from_numpy(v).cuda().to(DT[case["dtype"]]).double()
            L = torch.linalg.cholesky(M)
            b.append(torch.cholesky_solve(v[:, None], L)[:, 0])
            A.append((L + torch.triu(M, 1)).t().reshape(-1))  # column-major, the upper part as it was
        return {"A": torch.cat(A), "b": torch.cat(b), "info": torch.zeros(len(mats), dtype=torch.int32)}
    st = prepare(case, seed)
    st = {k: v.double() if isinstance(v, torch.Tensor) and v.is_floating_point() else v for k, v in st.items()}
    if op == "gemm":
        C = st["A"] @ st["B"]
        return C + st["C0"] if case["beta"] else C
    if op == "syrk":
        C = st["A"] @ st["A"].t()
        if case["beta"]:
            C = C + st["C0"]
        return torch.triu(C) + torch.tril(st["C0"], -1) if case["upper"] else torch.tril(C) + torch.triu(st["C0"], 1)
    if op == "trsm":
        return torch.linalg.solve_triangular(st["A"], st["B"], upper=case["upper"], left=case["left"],
                                             unitriangular=case["unit"])
    if op in ("chol_solve", "chol", "mixed"):
        L = torch.linalg.cholesky(st["A"])
        X = torch.cholesky_solve(st["B"], L)
        return {"L": L + torch.triu(st["A"], 1), "X": X} if op == "chol" else X
    if op == "getrf":
        return {"LU": torch.linalg.lu_factor(st["A"])[0], "piv": None}
    if op == "gp":
        X, y, ls = st["X"], st["y"], st["ls"]
        n = X.shape[0]
        d2 = torch.zeros((n, n), device="cuda", dtype=torch.float64)
        for q in range(X.shape[1]):
            d2 += ((X[:, None, q] - X[None, :, q]) / ls[q]) ** 2
        K = torch.exp(-0.5 * d2)
        L = torch.linalg.cholesky(K + 1e-2 * torch.eye(n, device="cuda", dtype=torch.float64))
        alpha = torch.cholesky_solve(y[:, None], L)
        Kbar = 0.5 * (torch.cholesky_inverse(L) - alpha @ alpha.t())
        W = Kbar * K
        grad = [(W * (X[:, None, q] - X[None, :, q]) ** 2).sum() / ls[q] ** 3 for q in range(X.shape[1])]
        return {"f": float(0.5 * (y @ alpha[:, 0]) + torch.log(torch.diagonal(L)).sum()), "g": torch.stack(grad),
                "Kbar": Kbar}
    return _exact_rng(case, st["key"])
