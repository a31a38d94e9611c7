// The triangular solve of one panel, all of its 128-row steps in one launch.
//
// Substitution with a block of right-hand sides is independent per column, so a CTA takes a
// strip of 8 or 16 columns through the whole panel. The strip stays in shared memory in FP64;
// the blocks of the triangle and the inverses of its diagonal blocks go from L2 straight to
// the registers of the warp that multiplies them on DMMA (an element has one user, so staging
// it would only cost shared-memory bandwidth), 32 columns ahead of their use. Left-looking: a
// block row subtracts the products of the blocks before it in one accumulation and is then
// multiplied by its inverse; warps meet only there.
//
// Bound by the load unit: a fragment's four columns (rows, for a row-major block) lie on four
// (two) 128-byte lines per eight lanes, 16 (8) passes a load; DMMA is busy 27% of the time. A panel of 512
// rows with up to 8 columns an SM takes 37 us (30), with 16 columns 43. As launches of one
// product each the seven dependent steps took 62. Tried: the blocks through shared memory by
// cp.async (35 us, more barriers and passes than the loads here) and by bulk copies (49, and 155
// for row-major blocks, whose copies are of 256 bytes).
#include "gemm.cuh"
#include "strip.cuh"
#include <type_traits>

namespace rc {
namespace {

constexpr int SB = 128;   // rows of a block
constexpr int SG = 32;    // depth of a group of loads
constexpr int kStripThreads = 512;

__device__ __forceinline__ void dmma(double (&d)[4], double a0, double a1, double b0) {
    asm("mma.sync.aligned.m16n8k4.row.col.f64.f64.f64.f64 {%0,%1,%2,%3}, {%4,%5}, {%6}, {%0,%1,%2,%3};\n"
        : "+d"(d[0]), "+d"(d[1]), "+d"(d[2]), "+d"(d[3])
        : "d"(a0), "d"(a1), "d"(b0));
}

template <class T>
using Pair = typename std::conditional<sizeof(T) == 8, double2, float2>::type;

// A warp's 16 x 32 share of a block as MMA fragments: v[q][e][h] multiplies row 8 q + 2 t + e of the
// 32 rows of X. Fragment rows g and g + 8 are the block's rows 2 g and 2 g + 1 where columns are
// contiguous, so that a load is a pair of either rows or columns.
template <class T>
struct Frag {
    T v[SG / 8][2][2];
};

// p: the share's first element; rows, depth: what lies inside the matrix from there (zero beyond).
template <class T>
__device__ __forceinline__ void load_frag(Frag<T>& f, const T* p, bool km, int64_t ld, int rows, int depth, bool vec,
                                          int g, int t) {
    if (vec && rows >= 16 && depth >= SG) {
        const T* src = km ? p + g * ld + 2 * t : p + 2 * t * ld + 2 * g;
#pragma unroll
        for (int q = 0; q < SG / 8; ++q) {
            const auto x = __ldg(reinterpret_cast<const Pair<T>*>(src)),
                       y = __ldg(reinterpret_cast<const Pair<T>*>(src + (km ? 8 * ld : ld)));
            f.v[q][0][0] = x.x;
            f.v[q][km ? 1 : 0][km ? 0 : 1] = x.y;
            f.v[q][km ? 0 : 1][km ? 1 : 0] = y.x;
            f.v[q][1][1] = y.y;
            src += km ? 8 : 8 * ld;
        }
    } else {
        const int64_t rs = km ? ld : 1, cs = km ? 1 : ld;
#pragma unroll
        for (int q = 0; q < SG / 8; ++q)
#pragma unroll
            for (int e = 0; e < 2; ++e)
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    const int r = km ? g + 8 * h : 2 * g + h, k = 8 * q + 2 * t + e;
                    f.v[q][e][h] = r < rows && k < depth ? p[r * rs + k * cs] : T(0);
                }
    }
}

template <class T, int COLS, bool AKM, bool WKM>
__global__ void __launch_bounds__(kStripThreads, 1)
    strip_kernel(bool upper, int m, int64_t n, View<const T> A, const T* W, View<T> B, bool vecA, const int* abort) {
    // With this row stride the fragment loads from X (4 rows 2 t x 8 columns) hit all banks.
    constexpr int LDX = COLS + 2, NI = COLS / 8;
    constexpr int GB = SB / 2 / SG;  // groups of a warp per block: half of the block's depth
    extern __shared__ __align__(16) double strip_shared[];
    const int nb = (m + SB - 1) / SB, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5 & 7, half = tid >> 8;
    const int g = lane >> 2, t = lane & 3;
    double *X = strip_shared, *part = X + nb * SB * LDX;  // part: the second half's sums
    if (abort != nullptr && *(volatile const int*)abort != 0) return;
    const int64_t j0 = (int64_t)blockIdx.x * COLS;
    const int64_t lda = AKM ? A.rs : A.cs;
    auto block = [&](int s) { return upper ? nb - 1 - s : s; };  // the s-th block in the order of substitution

    // Groups in order: for each block row those of the blocks left of (right of) its diagonal
    // block, then those of its inverse. Warps 0-7 take the first half of a block's depth, 8-15 the
    // second.
    int ls = 0, lq = 0;
    auto load_next = [&](Frag<T>& f) {
        if (ls >= nb) return;
        const int i = block(ls) * SB + 16 * warp, k = half * (SB / 2) + lq % GB * SG;
        if (lq < GB * ls) {
            const int c = block(lq / GB) * SB + k;
            load_frag<T>(f, A.p + (AKM ? i * lda + c : i + c * lda), AKM, lda, m - i, m - c, vecA, g, t);
        } else {
            const int b0 = block(ls) * SB, sz = m - b0;
            load_frag<T>(f, W + (size_t)b0 * SB + (WKM ? 16 * warp * SB + k : 16 * warp + k * SB), WKM, SB,
                         sz - 16 * warp, sz - k, true, g, t);
        }
        if (++lq == GB * (ls + 1)) {
            ++ls;
            lq = 0;
        }
    };
    Frag<T> fr[2];
    load_next(fr[0]);

    for (int e = tid; e < nb * SB * COLS; e += kStripThreads) {
        const int r = B.cs == 1 ? e / COLS : e % (nb * SB), c = B.cs == 1 ? e % COLS : e / (nb * SB);
        X[r * LDX + c] = r < m && j0 + c < n ? (double)B(r, j0 + c) : 0.0;
    }
    __syncthreads();

    double acc[2][NI][4];  // two chains of alternate steps
    auto clear = [&]() {
#pragma unroll
        for (int h = 0; h < 2; ++h)
#pragma unroll
            for (int ni = 0; ni < NI; ++ni)
#pragma unroll
                for (int c = 0; c < 4; ++c) acc[h][ni][c] = 0.0;
    };
    auto multiply = [&](const Frag<T>& f, int x0) {  // acc += f X[x0 .. x0 + SG)
        const double* x = X + (x0 + 2 * t) * LDX + g;
#pragma unroll
        for (int q = 0; q < SG / 8; ++q)
#pragma unroll
            for (int e = 0; e < 2; ++e)
#pragma unroll
                for (int ni = 0; ni < NI; ++ni)
                    dmma(acc[e][ni], (double)f.v[q][e][0], (double)f.v[q][e][1], x[(8 * q + e) * LDX + 8 * ni]);
    };
    auto product = [&](int x0) {  // the next block's product with X from row x0
        static_assert(GB == 2, "a block is two groups of a warp");
        load_next(fr[1]);
        multiply(fr[0], x0 + half * (SB / 2));
        load_next(fr[0]);
        multiply(fr[1], x0 + half * (SB / 2) + SG);
    };
    // use(row, column, sum) on the first half's warps, once every warp has read X.
    auto gather = [&](bool km, auto use) {
        auto each = [&](auto f) {
#pragma unroll
            for (int ni = 0; ni < NI; ++ni)
#pragma unroll
                for (int c = 0; c < 4; ++c)
                    f(16 * warp + (km ? g + 8 * (c >> 1) : 2 * g + (c >> 1)), 8 * ni + 2 * t + (c & 1),
                      acc[0][ni][c] + acc[1][ni][c]);
        };
        if (half) each([&](int r, int col, double v) { part[r * LDX + col] = v; });
        __syncthreads();
        if (!half) each([&](int r, int col, double v) { use(r, col, v + part[r * LDX + col]); });
        __syncthreads();
    };
    for (int s = 0; s < nb; ++s) {
        const int i0 = block(s) * SB;
        if (s > 0) {
            clear();
            for (int q = 0; q < s; ++q) product(block(q) * SB);
            gather(AKM, [&](int r, int col, double v) { X[(i0 + r) * LDX + col] -= v; });
        }
        clear();
        product(i0);
        gather(WKM, [&](int r, int col, double v) {
            const T x = (T)v;
            X[(i0 + r) * LDX + col] = (double)x;
            if (i0 + r < m && j0 + col < n) B(i0 + r, j0 + col) = x;
        });
    }
}

template <class T, int COLS, bool AKM, bool WKM>
int launch_strip(bool upper, int64_t m, int64_t n, View<const T> A, const T* W, View<T> B, cudaStream_t s,
                 const int* abort) {
    auto smem = [](int64_t rows) { return (size_t)(rows + SB) * (COLS + 2) * sizeof(double); };
    // always the limit of the tallest panel: threads and captured launches share the attribute
    if (cudaFuncSetAttribute(strip_kernel<T, COLS, AKM, WKM>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             (int)smem(kStripRows)) != cudaSuccess)
        return RC_ERR_CUDA;
    const bool vec = reinterpret_cast<uintptr_t>(A.p) % (2 * sizeof(T)) == 0 && (AKM ? A.rs : A.cs) % 2 == 0;
    strip_kernel<T, COLS, AKM, WKM><<<ceil_div(n, COLS), kStripThreads, smem((m + SB - 1) / SB * SB), s>>>(
        upper, (int)m, n, A, W, B, vec, abort);
    return check_launch();
}

template <class T, int COLS>
int launch_strip(bool upper, int64_t m, int64_t n, View<const T> A, const T* W, bool w_row_major, View<T> B,
                 cudaStream_t s, const int* abort) {
    if (A.cs == 1)
        return w_row_major ? launch_strip<T, COLS, true, true>(upper, m, n, A, W, B, s, abort)
                           : launch_strip<T, COLS, true, false>(upper, m, n, A, W, B, s, abort);
    return w_row_major ? launch_strip<T, COLS, false, true>(upper, m, n, A, W, B, s, abort)
                       : launch_strip<T, COLS, false, false>(upper, m, n, A, W, B, s, abort);
}

// The same a block at a time: products in place on a tile that spans the block's rows, and updates
// of the panel's other rows.
template <class T>
int block_solve(bool upper, int64_t m, int64_t n, View<const T> A, const T* W, bool w_row_major, View<T> B,
                cudaStream_t s, const int* abort) {
    const int64_t nblk = (m + SB - 1) / SB;
    for (int64_t step = 0; step < nblk; ++step) {
        const int64_t b = upper ? nblk - 1 - step : step, r0 = b * SB, sz = m - r0 < SB ? m - r0 : SB;
        const View<const T> X = {W + r0 * SB, w_row_major ? SB : 1, w_row_major ? 1 : SB};
        const View<T> Bb = B.sub(r0, 0);
        const View<const T> Bc = {Bb.p, Bb.rs, Bb.cs};
        RC_TRY(gemm<T>(sz, n, sz, T(1), X, Bc, T(0), Bb, kFull, 0, s, abort));
        const int64_t from = upper ? 0 : r0 + sz, rows = upper ? r0 : m - from;
        if (rows > 0)
            RC_TRY(gemm<T>(rows, n, sz, T(-1), A.sub(from, r0), Bc, T(1), B.sub(from, 0), kFull, 0, s, abort));
    }
    return RC_SUCCESS;
}

}  // namespace

template <class T>
int strip_solve(bool upper, int64_t m, int64_t n, View<const T> A, const T* W, bool w_row_major, View<T> B,
                cudaStream_t s, const int* abort) {
    if (m <= 0 || n <= 0) return RC_SUCCESS;
    if (m > kStripRows) return RC_ERR_INVALID_ARGUMENT;
    // Up to two rounds of 16-column strips (43 us each) beat the seven launches of a 512-row panel
    // (about 100 us at 4000 columns, 150 at 8000): 8 columns while every strip has an SM of its own.
    const int64_t sms = sm_count();
    if (n <= 8 * sms) return launch_strip<T, 8>(upper, m, n, A, W, w_row_major, B, s, abort);
    if (n <= 32 * sms) return launch_strip<T, 16>(upper, m, n, A, W, w_row_major, B, s, abort);
    return block_solve<T>(upper, m, n, A, W, w_row_major, B, s, abort);
}

template int strip_solve<double>(bool, int64_t, int64_t, View<const double>, const double*, bool, View<double>,
                                 cudaStream_t, const int*);
template int strip_solve<float>(bool, int64_t, int64_t, View<const float>, const float*, bool, View<float>,
                                cudaStream_t, const int*);

}  // namespace rc
