// Reverse-mode adjoints of the Cholesky factorisation and of the triangular solve
// (extension; the reference has no derivatives of its decompositions).
//
// Cholesky A = L L^T (Murray 2016, "Differentiation of the Cholesky decomposition"):
// with dA = dL L^T + L dL^T, X = L^-1 dL is lower triangular and L^-1 dA L^-T = X + X^T,
// so dL = L Phi(L^-1 dA L^-T) with Phi = lower triangle, diagonal halved. For a scalar
// f(L) with adjoint Lbar = df/dL this gives, for symmetric perturbations dA,
//     Abar = 1/2 L^-T (P + P^T) L^-1,   P = Phi(L^T Lbar).
// Blocked evaluation on the library's kernels, from L alone (the backward pass stores no
// intermediate of the forward factorisation):
//     M = tril(L^T Lbar)          lower-masked GEMM (the upper triangle is never formed)
//     S = M + M^T - diag(M)       = P + P^T
//     T = L^-T S                  blocked TRSM
//     Abar = 1/2 T L^-1           blocked TRSM on the transposed view, then symmetrised.
// Triangular solve X = L^-1 B (and X = L^-T B): Bbar = L^-T Xbar (L^-1 Xbar) and
// Lbar -= tril(Bbar X^T) (tril(X Bbar^T)).
#include "adjoint.cuh"
#include "assign.cuh"
#include "factor.cuh"
#include "gemm.cuh"
#include "strip.cuh"
#include <type_traits>

namespace rc {
namespace {

// dst = tril(src) (upper triangle zeroed), both n x n.
__global__ void tril_copy_kernel(int64_t n, View<const double> src, View<double> dst) {
    for (int64_t j = blockIdx.y; j < n; j += gridDim.y)
        for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
            dst(i, j) = i >= j ? src(i, j) : 0.0;
}

// mode 0: S(i, j) = S(j, i) for i < j (mirror the lower triangle up);
// mode 1: S = (S + S^T) / 2.
__global__ void symmetrize_kernel(int64_t n, View<double> S, int mode) {
    for (int64_t j = blockIdx.y; j < n; j += gridDim.y)
        for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < j; i += (int64_t)gridDim.x * blockDim.x) {
            if (mode == 0) {
                S(i, j) = S(j, i);
            } else {
                const double v = 0.5 * (S(i, j) + S(j, i));
                S(i, j) = v;
                S(j, i) = v;
            }
        }
}

dim3 sq_grid(int64_t n) {
    return dim3(ceil_div(n, 256) < 256u ? ceil_div(n, 256) : 256u, n < 65535 ? (unsigned)n : 65535u);
}

// Kbar = S - 1/2 a a^T from the lower triangle of S, both halves: 32 x 32 tiles, the upper
// one written through shared memory so that both stores run along the columns.
__global__ void __launch_bounds__(256) nll_adjoint_kernel(int64_t n, const double* a, View<double> S) {
    __shared__ double tile[32][33];
    const int64_t i0 = (int64_t)blockIdx.x * 32, j0 = (int64_t)blockIdx.y * 32;
    if (i0 < j0) return;
    const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
    for (int r = ty; r < 32; r += 8) {
        const int64_t i = i0 + tx, j = j0 + r;
        if (i >= n || j >= n || i < j) continue;
        const double v = fma(-0.5 * a[i], a[j], S(i, j));
        S(i, j) = v;
        tile[r][tx] = v;
    }
    __syncthreads();
    for (int r = ty; r < 32; r += 8) {
        const int64_t i = i0 + r, j = j0 + tx;
        if (i < n && j < n && i > j) S(j, i) = tile[tx][r];
    }
}

__global__ void identity_kernel(int64_t n, View<double> X) {
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
        X(i, i) = 1.0;
}

}  // namespace

int potrf_backward(int64_t n, View<const double> L, View<const double> Lbar, View<double> Abar, cudaStream_t s) {
    if (n <= 0) return RC_SUCCESS;
    double* w = static_cast<double*>(workspace(s, (size_t)2 * n * n * sizeof(double), 8));
    if (!w) return RC_ERR_ALLOC;
    const View<double> L0 = colmajor(w, n), Lb0 = colmajor(w + (size_t)n * n, n);
    tril_copy_kernel<<<sq_grid(n), 256, 0, s>>>(n, L, L0);
    tril_copy_kernel<<<sq_grid(n), 256, 0, s>>>(n, Lbar, Lb0);
    RC_TRY(check_launch());
    const View<const double> Lc = {L0.p, L0.rs, L0.cs}, Lbc = {Lb0.p, Lb0.rs, Lb0.cs};
    // M = tril(L^T Lbar) into Abar (lower triangle), S = M + M^T - diag(M).
    RC_TRY(gemm<double>(n, n, n, 1.0, Lc.t(), Lbc, 0.0, Abar, kLower, 0, s));
    symmetrize_kernel<<<sq_grid(n), 256, 0, s>>>(n, Abar, 0);
    RC_TRY(check_launch());
    // T = L^-T S; Abar = 1/2 T L^-1, i.e. L^T Abar^T = 1/2 T^T.
    RC_TRY(trsm_left<double>(true, false, n, n, 1.0, Lc.t(), Abar, nullptr, s));
    RC_TRY(trsm_left<double>(true, false, n, n, 0.5, Lc.t(), Abar.t(), nullptr, s));
    symmetrize_kernel<<<sq_grid(n), 256, 0, s>>>(n, Abar, 1);
    return check_launch();
}

int trsm_backward(bool trans, int64_t n, int64_t nrhs, View<const double> L, View<const double> X, View<double> Xbar,
                  View<double> Lbar, cudaStream_t s) {
    if (n <= 0 || nrhs <= 0) return RC_SUCCESS;
    double* w = static_cast<double*>(workspace(s, (size_t)n * n * sizeof(double), 8));
    if (!w) return RC_ERR_ALLOC;
    const View<double> L0 = colmajor(w, n);
    tril_copy_kernel<<<sq_grid(n), 256, 0, s>>>(n, L, L0);
    RC_TRY(check_launch());
    const View<const double> Lc = {L0.p, L0.rs, L0.cs};
    const View<const double> Bb = {Xbar.p, Xbar.rs, Xbar.cs};
    if (!trans) {
        // X = L^-1 B: Bbar = L^-T Xbar, Lbar -= tril(Bbar X^T)
        RC_TRY(trsm_left<double>(true, false, n, nrhs, 1.0, Lc.t(), Xbar, nullptr, s));
        return gemm<double>(n, n, nrhs, -1.0, Bb, X.t(), 1.0, Lbar, kLower, 0, s);
    }
    // X = L^-T B: Bbar = L^-1 Xbar, Lbar -= tril(X Bbar^T)
    RC_TRY(trsm_left<double>(false, false, n, nrhs, 1.0, Lc, Xbar, nullptr, s));
    return gemm<double>(n, n, nrhs, -1.0, X, Bb.t(), 1.0, Lbar, kLower, 0, s);
}

// 1/2 (L^-T L^-1 - a a^T): the inverse X = L^-1 is built in row panels of kPanel, whose columns
// right of the diagonal block are zero and never touched, and multiplied by itself from each
// tile's diagonal on: 2/3 n^3 operations; through the adjoint of the factorisation (one masked
// product, two triangular solves with n columns) they were 3 n^3. Likelihood and gradient at
// n = 8192, d = 16: 90.2 -> 26.4 ms (27.5 with X^T X a panel at a time), and Kbar's error against a 64-bit
// library result 7.2e-15 -> 3.1e-15.
int nll_adjoint(int64_t n, View<const double> L, const double* a, View<double> Kbar, cudaStream_t s) {
    if (n <= 0) return RC_SUCCESS;
    constexpr int64_t kPanel = kStripRows;  // trailing updates as deep as the factorisation's
    double* w = static_cast<double*>(workspace(s, (size_t)n * n * sizeof(double), 8));
    double* W = static_cast<double*>(workspace(s, (size_t)ceil_div(n, kNB) * kNB * kNB * sizeof(double), 1));
    if (!w || !W) return RC_ERR_ALLOC;
    const View<double> X = colmajor(w, n);
    auto C_ = [](const View<double>& v) { return View<const double>{v.p, v.rs, v.cs}; };
    if (cudaMemsetAsync(w, 0, (size_t)n * n * sizeof(double), s) != cudaSuccess) return RC_ERR_CUDA;
    identity_kernel<<<ceil_div(n, 256), 256, 0, s>>>(n, X);
    RC_TRY(check_launch());
    RC_TRY(trtri_blocks_launch<double>(n, L, false, W, nullptr, nullptr, s));
    for (int64_t p = 0; p < n; p += kPanel) {
        const int64_t pe = n - p < kPanel ? n : p + kPanel;
        RC_TRY(strip_solve<double>(false, pe - p, pe, L.sub(p, p), W + p * kNB, false, X.sub(p, 0), s, nullptr));
        const View<const double> Xp = C_(X.sub(p, 0));
        if (pe < n)
            RC_TRY(gemm<double>(n - pe, pe, pe - p, -1.0, L.sub(pe, p), Xp, 1.0, X.sub(pe, 0), kFull, 0, s));
    }
    RC_TRY(gemm<double>(n, n, n, 0.5, C_(X).t(), C_(X), 0.0, Kbar, kLowerTri, 0, s));
    const unsigned nt = ceil_div(n, 32);
    nll_adjoint_kernel<<<dim3(nt, nt), 256, 0, s>>>(n, a, Kbar);
    return check_launch();
}

}  // namespace rc

extern "C" {

int rc_potrf_backward_f64(size_t n, const double* L, size_t ldl, const double* Lbar, size_t ldlb, double* Abar,
                          size_t ldab, void* stream) {
    if (n == 0) return RC_SUCCESS;
    if (!L || !Lbar || !Abar || ldl < n || ldlb < n || ldab < n) return RC_ERR_INVALID_ARGUMENT;
    return rc::potrf_backward((int64_t)n, rc::colmajor(L, (int64_t)ldl), rc::colmajor(Lbar, (int64_t)ldlb),
                              rc::colmajor(Abar, (int64_t)ldab), static_cast<cudaStream_t>(stream));
}

int rc_trsm_backward_f64(int trans, size_t n, size_t nrhs, const double* L, size_t ldl, const double* X, size_t ldx,
                         double* Xbar, size_t ldxb, double* Lbar, size_t ldlb, void* stream) {
    if (n == 0 || nrhs == 0) return RC_SUCCESS;
    if (!L || !X || !Xbar || !Lbar || ldl < n || ldx < n || ldxb < n || ldlb < n) return RC_ERR_INVALID_ARGUMENT;
    return rc::trsm_backward(trans != 0, (int64_t)n, (int64_t)nrhs, rc::colmajor(L, (int64_t)ldl),
                             rc::colmajor(X, (int64_t)ldx), rc::colmajor(Xbar, (int64_t)ldxb),
                             rc::colmajor(Lbar, (int64_t)ldlb), static_cast<cudaStream_t>(stream));
}

int rc_nll_adjoint_f64(size_t n, const double* L, size_t ldl, const double* a, double* Kbar, size_t ldkb,
                       void* stream) {
    if (n == 0) return RC_SUCCESS;
    // one 32-row tile per index of a grid of at most 65535
    if (!L || !a || !Kbar || ldl < n || ldkb < n || n > (size_t)32 * 65535) return RC_ERR_INVALID_ARGUMENT;
    return rc::nll_adjoint((int64_t)n, rc::colmajor(L, (int64_t)ldl), a, rc::colmajor(Kbar, (int64_t)ldkb),
                           static_cast<cudaStream_t>(stream));
}

}  // extern "C"

// ---------------------------------------------------------------------------------------
// RBF kernel matrix of a Gaussian process and the contraction of its adjoint with the
// lengthscale derivatives: the model around the differentiated Cholesky in the
// marginal-likelihood workload.
namespace rc {
namespace {

// Both kernels work on 64 x 64 tiles of the lower triangle: k(x_i, x_j) is symmetric, so one
// exponential serves two elements, and the d coordinates of 128 points come from shared memory.
// They are bound by FP64 arithmetic, about 7 d + 30 operations a pair (matrix) and 10 d + 30
// (gradient). A quotient by a lengthscale is the product with its reciprocal and one correction by
// the residual, t + (x - t l) (1 / l) (Markstein, IBM Journal of Research and Development, 1990):
// the quotient as a division rounds it, at three operations in place of ten and more (with divisions
// the likelihood and gradient of n = 8192, d = 16 take 0.9 ms longer; without the correction a
// rounding more per quotient, and the entries' error grows). Where the reciprocal or the residual
// would leave the range, divisions.
constexpr int kRbfTile = 64, kRbfDim = 16, kRbfLd = kRbfTile + 1;

struct RbfShared {
    double x[2][kRbfDim][kRbfTile];  // coordinate q of the tile's row and column points
    double ls[kRbfDim], inv[kRbfDim];
};

// Tile t of the lower triangle, column by column: the row and column tile.
__device__ __forceinline__ void rbf_tile(int64_t t, int64_t nt, int64_t* ti, int64_t* tj) {
    // column tj starts at tj nt - tj (tj - 1) / 2
    const double b = 2.0 * nt + 1.0;
    int64_t j = (int64_t)((b - sqrt(b * b - 8.0 * (double)t)) * 0.5);
    while (j > 0 && j * nt - j * (j - 1) / 2 > t) --j;
    while ((j + 1) * nt - (j + 1) * j / 2 <= t) ++j;
    *tj = j;
    *ti = j + t - (j * nt - j * (j - 1) / 2);
}

__device__ __forceinline__ bool rbf_lengthscales(RbfShared& sh, int d, const double* ls) {
    if (threadIdx.x < kRbfDim) {
        sh.ls[threadIdx.x] = threadIdx.x < d ? ls[threadIdx.x] : 1.0;
        sh.inv[threadIdx.x] = 1.0 / sh.ls[threadIdx.x];
    }
    __syncthreads();
    bool plain = true;
    for (int q = 0; q < d; ++q) plain = plain && fabs(sh.ls[q]) >= 1e-290 && fabs(sh.ls[q]) <= 1e290;
    return plain;
}

__device__ __forceinline__ void rbf_points(RbfShared& sh, int64_t n, int d, const double* X, int64_t i0, int64_t j0) {
    for (int e = threadIdx.x; e < 2 * kRbfTile * d; e += 256) {
        const int side = e / (kRbfTile * d), r = e % (kRbfTile * d) / d, q = e % d;
        const int64_t i = (side ? j0 : i0) + r;
        sh.x[side][q][r] = X[(i < n ? i : n - 1) * d + q];  // beyond the end the last point, at weight 0
    }
}

// k of the thread's 4 x 4 pairs (i, j) = (tx + 16 a, ty + 16 b).
__device__ __forceinline__ void rbf_values(const RbfShared& sh, int d, bool plain, int tx, int ty, double (&k)[4][4]) {
    auto distances = [&](auto divide) {
#pragma unroll
        for (int a = 0; a < 4; ++a)
#pragma unroll
            for (int b = 0; b < 4; ++b) k[a][b] = 0.0;
        for (int q = 0; q < d; ++q) {
            double xi[4], xj[4];
#pragma unroll
            for (int a = 0; a < 4; ++a) xi[a] = sh.x[0][q][tx + 16 * a];
#pragma unroll
            for (int b = 0; b < 4; ++b) xj[b] = sh.x[1][q][ty + 16 * b];
            const double inv = sh.inv[q], l = sh.ls[q];
#pragma unroll
            for (int a = 0; a < 4; ++a)
#pragma unroll
                for (int b = 0; b < 4; ++b) {
                    const double x = xi[a] - xj[b];
                    double t;
                    if constexpr (divide.value) {
                        t = x / l;
                    } else {
                        t = x * inv;
                        t = fma(fma(-t, l, x), inv, t);
                    }
                    k[a][b] = fma(t, t, k[a][b]);
                }
        }
    };
    if (plain) {
        distances(std::false_type{});
        bool nan = false;  // an infinite difference or quotient leaves no residual
#pragma unroll
        for (int a = 0; a < 4; ++a)
#pragma unroll
            for (int b = 0; b < 4; ++b) nan = nan || isnan(k[a][b]);
        plain = !nan;
    }
    if (!plain) distances(std::true_type{});
#pragma unroll
    for (int a = 0; a < 4; ++a)
#pragma unroll
        for (int b = 0; b < 4; ++b) k[a][b] = exp(-0.5 * k[a][b]);
}

__global__ void __launch_bounds__(256) rbf_kernel(int64_t n, int d, const double* X, const double* ls, double noise,
                                                  View<double> K) {
    __shared__ union {
        RbfShared sh;
        double t[kRbfTile][kRbfLd];
    } u;
    const int64_t nt = (n + kRbfTile - 1) / kRbfTile;
    int64_t ti, tj;
    rbf_tile(blockIdx.x, nt, &ti, &tj);
    const int64_t i0 = ti * kRbfTile, j0 = tj * kRbfTile;
    const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
    rbf_points(u.sh, n, d, X, i0, j0);
    const bool plain = rbf_lengthscales(u.sh, d, ls);
    double k[4][4];
    rbf_values(u.sh, d, plain, tx, ty, k);
#pragma unroll
    for (int a = 0; a < 4; ++a)
#pragma unroll
        for (int b = 0; b < 4; ++b) {
            const int64_t i = i0 + tx + 16 * a, j = j0 + ty + 16 * b;
            if (i < n && j < n) K(i, j) = k[a][b] + (i == j ? noise : 0.0);
        }
    if (ti == tj) return;
    __syncthreads();
#pragma unroll
    for (int a = 0; a < 4; ++a)
#pragma unroll
        for (int b = 0; b < 4; ++b) u.t[tx + 16 * a][ty + 16 * b] = k[a][b];
    __syncthreads();
    for (int e = threadIdx.x; e < kRbfTile * kRbfTile; e += 256) {
        const int jj = e % kRbfTile, ii = e / kRbfTile;
        if (i0 + ii < n && j0 + jj < n) K(j0 + jj, i0 + ii) = u.t[ii][jj];
    }
}

// g[q] = sum_ij Kbar(i, j) k(i, j) (x_iq - x_jq)^2 / ls_q^3, k without the noise term. A pair
// off the diagonal tiles takes Kbar(i, j) + Kbar(j, i), the latter through shared memory.
__global__ void __launch_bounds__(256) rbf_ls_grad_kernel(int64_t n, int d, const double* X, const double* ls,
                                                          View<const double> Kbar, double* g) {
    __shared__ union {
        RbfShared sh;
        double t[kRbfTile][kRbfLd];
        double red[kRbfDim][8];
    } u;
    const int64_t nt = (n + kRbfTile - 1) / kRbfTile, tiles = nt * (nt + 1) / 2;
    const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
    double acc[kRbfDim];
#pragma unroll
    for (int q = 0; q < kRbfDim; ++q) acc[q] = 0.0;
    for (int64_t tile = blockIdx.x; tile < tiles; tile += gridDim.x) {
        int64_t ti, tj;
        rbf_tile(tile, nt, &ti, &tj);
        const int64_t i0 = ti * kRbfTile, j0 = tj * kRbfTile;
        __syncthreads();
        double w[4][4], k[4][4];
        if (ti != tj) {
            for (int e = threadIdx.x; e < kRbfTile * kRbfTile; e += 256) {
                const int jj = e % kRbfTile, ii = e / kRbfTile;
                u.t[ii][jj] = i0 + ii < n && j0 + jj < n ? Kbar(j0 + jj, i0 + ii) : 0.0;
            }
            __syncthreads();
        }
#pragma unroll
        for (int a = 0; a < 4; ++a)
#pragma unroll
            for (int b = 0; b < 4; ++b) {
                const int64_t i = i0 + tx + 16 * a, j = j0 + ty + 16 * b;
                w[a][b] = i < n && j < n ? Kbar(i, j) : 0.0;
                if (ti != tj) w[a][b] += u.t[tx + 16 * a][ty + 16 * b];
            }
        __syncthreads();
        rbf_points(u.sh, n, d, X, i0, j0);
        const bool plain = rbf_lengthscales(u.sh, d, ls);
        rbf_values(u.sh, d, plain, tx, ty, k);
#pragma unroll
        for (int a = 0; a < 4; ++a)
#pragma unroll
            for (int b = 0; b < 4; ++b) w[a][b] *= k[a][b];
#pragma unroll
        for (int q = 0; q < kRbfDim; ++q) {
            if (q >= d) break;
            double xi[4], xj[4];
#pragma unroll
            for (int a = 0; a < 4; ++a) xi[a] = u.sh.x[0][q][tx + 16 * a];
#pragma unroll
            for (int b = 0; b < 4; ++b) xj[b] = u.sh.x[1][q][ty + 16 * b];
#pragma unroll
            for (int a = 0; a < 4; ++a)
#pragma unroll
                for (int b = 0; b < 4; ++b) {
                    const double dx = xi[a] - xj[b];
                    acc[q] = fma(w[a][b], dx * dx, acc[q]);
                }
        }
    }
    __syncthreads();
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
    for (int q = 0; q < kRbfDim; ++q) {
        double v = acc[q];
        for (int off = 16; off > 0; off >>= 1) v += __shfl_down_sync(0xffffffffu, v, off);
        if (lane == 0) u.red[q][warp] = v;
    }
    __syncthreads();
    if (threadIdx.x < d) {
        double v = 0.0;
        for (int w8 = 0; w8 < 8; ++w8) v += u.red[threadIdx.x][w8];
        const double l = ls[threadIdx.x];
        atomicAdd(&g[threadIdx.x], v / (l * l * l));
    }
}

}  // namespace
}  // namespace rc

extern "C" {

int rc_rbf_kernel_f64(size_t n, int d, const double* X, const double* ls, double noise, double* K, size_t ldk,
                      void* stream) {
    if (n == 0) return RC_SUCCESS;
    if (d < 1 || d > 16 || !X || !ls || !K || ldk < n) return RC_ERR_INVALID_ARGUMENT;
    const size_t nt = rc::ceil_div(n, rc::kRbfTile);
    rc::rbf_kernel<<<(unsigned)(nt * (nt + 1) / 2), 256, 0, static_cast<cudaStream_t>(stream)>>>(
        (int64_t)n, d, X, ls, noise, rc::colmajor(K, (int64_t)ldk));
    return rc::check_launch();
}

int rc_rbf_lengthscale_grad_f64(size_t n, int d, const double* X, const double* ls, const double* Kbar, size_t ldk,
                                double* grad, void* stream) {
    if (n == 0) return RC_SUCCESS;
    if (d < 1 || d > 16 || !X || !ls || !Kbar || !grad || ldk < n) return RC_ERR_INVALID_ARGUMENT;
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    if (cudaMemsetAsync(grad, 0, d * sizeof(double), s) != cudaSuccess) return RC_ERR_CUDA;
    const size_t nt = rc::ceil_div(n, rc::kRbfTile), tiles = nt * (nt + 1) / 2, most = 4 * (size_t)rc::sm_count();
    rc::rbf_ls_grad_kernel<<<(unsigned)(tiles < most ? tiles : most), 256, 0, s>>>(
        (int64_t)n, d, X, ls, rc::View<const double>{Kbar, 1, (int64_t)ldk}, grad);
    return rc::check_launch();
}

}  // extern "C"
