// Warp-level pieces of the small Cholesky factorisations (the 128-block of potrf, the 32-blocks
// of the batched solver), on FP64 blocks in shared memory: DMMA updates, the dependent chain
// of 16 columns, substitution, and the merges of a block inverse. A block has row stride SLD
// with SLD % 16 == 4, so that DMMA fragment loads hit all banks; L stands in its strict lower
// triangle, the reciprocals of L's diagonal on the diagonal and inv(L) transposed in the upper
// triangle (Inv(i, c), i >= c, at S[c * SLD + i]).
#pragma once
#include "common.cuh"

namespace rc {
namespace {

constexpr int kDB = 16;   // columns of a sub-block
constexpr int kLTD = 32;  // column stride of a sub-block's transposed copy

__device__ __forceinline__ void dmma_16x8x4(double (&d)[4], double a0, double a1, double b0) {
    asm("mma.sync.aligned.m16n8k4.row.col.f64.f64.f64.f64 {%0,%1,%2,%3}, {%4,%5}, {%6}, {%0,%1,%2,%3};\n"
        : "+d"(d[0]), "+d"(d[1]), "+d"(d[2]), "+d"(d[3])
        : "d"(a0), "d"(a1), "d"(b0));
}

// Tile (rows i0 .. i0 + 15, columns j0 .. j0 + 7) of S -= L(:, m0 : m0 + 16) L(:, m0 : m0 + 16)^T.
template <int SLD>
__device__ __forceinline__ void syrk_tile(double* S, int i0, int j0, int m0, int lane) {
    const int g = lane >> 2, t = lane & 3;
    double d[4] = {};
#pragma unroll
    for (int k = 0; k < kDB; k += 4)
        dmma_16x8x4(d, S[(i0 + g) * SLD + m0 + k + t], S[(i0 + g + 8) * SLD + m0 + k + t],
                    S[(j0 + g) * SLD + m0 + k + t]);
    double2* lo = reinterpret_cast<double2*>(S + (i0 + g) * SLD + j0 + 2 * t);
    double2* hi = reinterpret_cast<double2*>(S + (i0 + g + 8) * SLD + j0 + 2 * t);
    double2 a = *lo, b = *hi;
    a.x -= d[0];
    a.y -= d[1];
    b.x -= d[2];
    b.y -= d[3];
    *lo = a;
    *hi = b;
}

// One merge of the block inverse: with inv(A) (rows and columns J0 .. J0 + H) and inv(D)
// (I0 .. I0 + H, I0 = J0 + H) in place, the off-diagonal block of inv([A 0; C D]) is
// X = -inv(D) (C inv(A)). merge_t computes tile q of T = C inv(A), merge_x tile q of X (16 x 8
// tiles, down the columns); both skip the zero blocks of the triangular operand and select
// within its diagonal blocks.
template <int H, int SLD>
__device__ __forceinline__ void merge_t(const double* S, double* T, int J0, int q, int lane) {
    constexpr int TD = H + 4, ROWS = H / 16;
    const int ti = 16 * (q % ROWS), tc = 8 * (q / ROWS);
    const int g = lane >> 2, t = lane & 3, c = tc + g;
    const double *a = S + (J0 + H + ti + g) * SLD + J0 + t, *v = S + (J0 + c) * SLD + J0 + t;  // v: inv(A)(k, c)
    double d[4] = {};
#pragma unroll
    for (int k = 0; k < 8; k += 4)
        dmma_16x8x4(d, a[tc + k], a[8 * SLD + tc + k], tc + k + t >= c ? v[tc + k] : 0.0);
#pragma unroll 4
    for (int k = tc + 8; k < H; k += 4) dmma_16x8x4(d, a[k], a[8 * SLD + k], v[k]);
    *reinterpret_cast<double2*>(T + (ti + g) * TD + tc + 2 * t) = make_double2(d[0], d[1]);
    *reinterpret_cast<double2*>(T + (ti + g + 8) * TD + tc + 2 * t) = make_double2(d[2], d[3]);
}
template <int H, int SLD>
__device__ __forceinline__ void merge_x(double* S, const double* T, int J0, int xi, int xc, int lane) {
    constexpr int TD = H + 4;
    const int I0 = J0 + H, g = lane >> 2, t = lane & 3, i = xi + g;
    const double *a = S + (I0 + t) * SLD + I0 + i, *b = T + t * TD + xc + g;  // a: inv(D)(i, k)
    double d[4] = {};
#pragma unroll 4
    for (int k = 0; k < xi; k += 4) dmma_16x8x4(d, a[k * SLD], a[k * SLD + 8], b[k * TD]);
#pragma unroll
    for (int k = 0; k < 16; k += 4) {
        const int kk = xi + k;
        dmma_16x8x4(d, k + t <= g ? a[kk * SLD] : 0.0, k + t <= g + 8 ? a[kk * SLD + 8] : 0.0, b[kk * TD]);
    }
    double* x = S + (J0 + xc + 2 * t) * SLD + I0 + i;  // X(i, c), transposed
    x[0] = -d[0];
    x[SLD] = -d[1];
    x[8] = -d[2];
    x[SLD + 8] = -d[3];
}

// x solved with the 16-block L, each lane its own x: x[m] /= L(m, m), x[q] -= L(q, m) x[m].
// Columns of L in Lt, reciprocal diagonal in rd; wait(h) is called before the first use of
// columns 8 h .. 8 h + 7. With x a unit vector this is a column of inv(L), with x a row of the
// panel below L that row of the panel solve.
template <class Wait>
__device__ __forceinline__ void solve_sub_block(double (&x)[kDB], const double* rd, const double* Lt, Wait wait) {
#pragma unroll
    for (int m = 0; m < kDB; ++m) {
        if (m % 8 == 0) wait(m / 8);
        x[m] *= rd[m];
        const double2* pair = reinterpret_cast<const double2*>(Lt + m * kLTD);
#pragma unroll
        for (int q = (m + 1) & ~1; q < kDB; q += 2) {
            const double2 v = pair[q / 2];
            if (q > m) x[q] = fma(-v.x, x[m], x[q]);
            x[q + 1] = fma(-v.y, x[m], x[q + 1]);
        }
    }
}

// 1 / sqrt(d) for a normal d > 0: the hardware approximation (relative error e below 2^-20)
// and one step of the third-order series of (1 - e)^(-1/2). Straight-line code, so that the
// rank-1 update of the column before is scheduled into its latency; for a subnormal d the
// approximation is infinite and the caller starts over with rsqrt().
__device__ __forceinline__ double rsqrt_normal(double d) {
    double r;
    asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(r) : "d"(d));
    const double e = fma(-(d * r), r, 1.0);
    return fma(r * e, fma(e, fma(e, 0.3125, 0.375), 0.5), r);
}

// Right-looking factorisation of 16 columns of 32 rows by one warp, row `lane` in a (the
// 16 x 16 block to factor and the 16 rows below it): a becomes L's row, column j of L goes to
// Lt + j * kLTD, L(j, j) to ld and its reciprocal to rd; arrive(h) is called once columns
// 8 h .. 8 h + 7 are there. flags[0] = 1 + column of the first non-positive (or NaN)
// pivot, 0 if there is none; after one the values are void. flags[1] = 1 where any pivot is below
// 1e-300, negative ones included, and so perhaps too small for rsqrt_normal: the pivots after it may
// be infinite or NaN whatever the matrix, so the result is void, the failing column included.
template <class Arrive>
__device__ __forceinline__ void factor_sub_block(double (&a)[kDB], double* Lt, double* ld, double* rd, int lane,
                                                 volatile int* flags, Arrive arrive) {
    int bad = 0;
    bool tiny = false;
    auto pivot = [&](double own, int j) {
        const double d = __shfl_sync(0xffffffffu, own, j);
        if (!(d > 0.0) && bad == 0) bad = j + 1;
        tiny |= d < 1e-300;
        return d;
    };
    double d = pivot(a[0], 0), r = rsqrt_normal(d);
#pragma unroll
    for (int j = 0; j < kDB; ++j) {
        const double l = lane == j ? d * r : a[j] * r;  // L(i, j); above the diagonal, unused
        a[j] = l;
        if (lane == j) {
            rd[j] = r;
            ld[j] = l;
        }
        double* colj = Lt + j * kLTD;
        colj[lane] = l;
        if (j + 1 < kDB) {
            d = pivot(fma(-l, l, a[j + 1]), j + 1);  // row j + 1's own update of its diagonal
            r = rsqrt_normal(d);
        } else if (lane == 0) {
            flags[0] = bad;
            flags[1] = tiny;
        }
        __syncwarp();
        if (j % 8 == 7) arrive(j / 8);
        const double2* pair = reinterpret_cast<const double2*>(colj);
#pragma unroll
        for (int c = (j + 1) & ~1; c < kDB; c += 2) {
            const double2 v = pair[c / 2];
            if (c > j) a[c] = fma(-l, v.x, a[c]);
            a[c + 1] = fma(-l, v.y, a[c + 1]);
        }
    }
}

// The same for pivots of any size, on the rows in shared memory (row: this lane's) and with the
// library's rsqrt: the way out for values next to underflow.
template <class Arrive>
__device__ __noinline__ void factor_sub_block_any(double* row, bool own, double* Lt, double* ld, double* rd, int lane,
                                                  volatile int* flags, Arrive arrive) {
    int bad = 0;
#pragma unroll 1
    for (int j = 0; j < kDB; ++j) {
        double d = __shfl_sync(0xffffffffu, own ? row[j] : 0.0, j);
        if (!(d > 0.0)) {
            if (bad == 0) bad = j + 1;
            d = 1.0;
        }
        const double r = rsqrt(d), l = lane == j ? d * r : own ? row[j] * r : 0.0;
        if (lane == j) {
            rd[j] = r;
            ld[j] = l;
        }
        if (own && lane > j) row[j] = l;
        Lt[j * kLTD + lane] = l;
        if (j + 1 == kDB && lane == 0) {
            flags[0] = bad;
            flags[1] = 0;
        }
        __syncwarp();
        if (j % 8 == 7) arrive(j / 8);
        if (own)
            for (int c = j + 1; c < kDB && c <= lane; ++c) row[c] = fma(-l, Lt[j * kLTD + c], row[c]);
    }
}

}  // namespace
}  // namespace rc
