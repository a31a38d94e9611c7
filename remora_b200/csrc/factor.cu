// Blocked triangular solve (TRSM) and blocked right-looking Cholesky (POTRF).
//
// Replaces kernels::trsm / kernels::potrf for hip_tag (include/remora/kernels/hip/
// trsm.hpp:45-107 -> cublas trsm; include/remora/kernels/hip/potrf.hpp:41-141, a
// recursive split whose 16x16 leaves are factored by a single thread). Here:
//  * TRSM: every 128x128 diagonal block of the triangle is inverted at once (one CTA
//    per block, FP64 in shared memory); the solve then walks panels of 512 rows, each
//    solved in strips of a few right-hand sides per CTA (strip.cu) and followed by one
//    GEMM update of the remaining rows, where nearly all flops are.
//  * POTRF: panels of 512 columns. Inside a panel's diagonal block, per 128 columns, one
//    CTA factors the diagonal block in FP64 shared memory (and inverts it), the rows below
//    it are solved in strips and the rest of the block is updated; then the rows below the
//    panel are solved in strips through all of its 128-column steps, and the trailing
//    matrix is updated by a lower-masked GEMM of depth 512 (the SYRK schedule).
//    A non-positive pivot writes its global index to the status word and every later
//    kernel of the factorization returns at once.
#include "factor.cuh"
#include "assign.cuh"
#include "diag.cuh"
#include "gemm.cuh"
#include "strip.cuh"

namespace rc {
namespace {

constexpr int NB = kNB;
constexpr int SLD = NB + 4;  // shared-memory row stride (doubles): DMMA fragment loads hit all banks
constexpr int DB = kDB;      // diagonal sub-block
constexpr int LTD = kLTD;    // column stride of the sub-block's transposed copy
constexpr int NSUB = NB / DB;
constexpr int kDiagThreads = 512;

// Shared memory of the diagonal-block kernels (doubles): S holds L in its strict lower
// triangle, the reciprocals of L's diagonal on its diagonal and the strict part of inv(L)
// transposed in its upper triangle (Inv(i, c), i >= c, at S[c * SLD + i]); ld L's diagonal,
// rd its reciprocals, Lt the columns of the sub-block being factored, T16 / T32 / T64 the
// scratch of the inverse's merges.
constexpr int kOffLt = NB * SLD, kOffLd = kOffLt + NB * LTD / 2, kOffRd = kOffLd + NB, kOffT64 = kOffRd + NB,
              kOffT32 = kOffT64 + 64 * (64 + 4), kOffT16 = kOffT32 + 32 * (32 + 4), kOffEnd = kOffT16 + 16 * (16 + 4);
constexpr size_t kDiagSmem = kOffEnd * sizeof(double) + 16;

__device__ __forceinline__ bool aborted(const int* abort) { return abort != nullptr && *(volatile const int*)abort != 0; }

// The update of S by columns m0 .. m0 + 15 on the 16-row tiles from r0, columns from r0 up to
// `width` 8-column tiles wide or to the diagonal, spread over n workers (number w).
__device__ __forceinline__ void syrk_tiles(double* S, int r0, int width, int m0, int w, int n, int lane) {
    int e = w;
    for (int i0 = r0; i0 < NB; i0 += 16) {
        const int diag = (i0 - r0) / 8 + 2, cnt = diag < width ? diag : width;
        for (; e < cnt; e += n) syrk_tile<SLD>(S, i0, r0 + 8 * e, m0, lane);
        e -= cnt;
    }
}

// The 32 x 32 blocks (bi, bj) of the lower triangle, by number 0 .. 9.
__device__ __forceinline__ void lower_block(int q, int& bi, int& bj) {
    bi = q < 1 ? 0 : q < 3 ? 1 : q < 6 ? 2 : 3;
    bj = q - bi * (bi + 1) / 2;
}

// Half h (16 elements a lane, all loads before the stores) of block q of inv(L) to the NB x NB
// block W. Row-major W: 8 rows x 4 columns a step (32-byte runs, at most two lanes per bank);
// column-major: 32 rows of a column.
template <class T>
__device__ __forceinline__ void store_inverse(const double* S, T* W, bool row_major, int q, int h, int lane) {
    int bi, bj;
    lower_block(q, bi, bj);
    const int i0 = 32 * bi + (row_major ? 16 * h + (lane >> 2) : lane);
    const int c0 = 32 * bj + (row_major ? lane & 3 : 16 * h);
    double v[16];
#pragma unroll
    for (int u = 0; u < 16; ++u)
        v[u] = row_major ? S[(c0 + (u & 7) * 4) * SLD + i0 + (u >> 3) * 8] : S[(c0 + u) * SLD + i0];
#pragma unroll
    for (int u = 0; u < 16; ++u) {
        const int i = row_major ? i0 + (u >> 3) * 8 : i0, c = row_major ? c0 + (u & 7) * 4 : c0 + u;
        if (i >= c) W[row_major ? i * NB + c : i + c * NB] = (T)v[u];
    }
}

// Zeros above W's diagonal: part p of NSUB - 1, by 96 threads.
template <class T>
__device__ __forceinline__ void zero_upper(T* W, bool row_major, int p, int tid) {
    constexpr int kPart = (NB * NB + NSUB - 2) / (NSUB - 1);
    const int end = (p + 1) * kPart < NB * NB ? (p + 1) * kPart : NB * NB;
#pragma unroll 4
    for (int e = p * kPart + tid; e < end; e += 96) {
        const int i = row_major ? e / NB : e % NB, c = row_major ? e % NB : e / NB;
        if (i < c) W[e] = T(0);
    }
}

// Element (i, c) of step u = 0 .. 31 of a lane in a 32 x 32 block of a matrix of either order:
// 32 columns of a row a step where rows are contiguous, else 8 rows x 4 columns (64-byte runs;
// the 16 lanes of a half-warp, 4 x 4, fall on distinct banks of S).
__device__ __forceinline__ int block_row(bool rowmaj, int u, int lane) {
    return rowmaj ? u : (u & 3) * 8 + (lane & 3) + ((lane >> 4) << 2);
}
__device__ __forceinline__ int block_col(bool rowmaj, int u, int lane) {
    return rowmaj ? lane : (u >> 2) * 4 + ((lane >> 2) & 3);
}

// Block q of the diagonal block's lower triangle (the identity beyond its sz rows) into S by
// one warp, 32 loads a lane in flight; unit: ones on the diagonal, which is not read.
template <class T>
__device__ __forceinline__ void load_block(const View<T>& A, int sz, bool rowmaj, bool unit, int q, double* S,
                                           int lane) {
    int bi, bj;
    lower_block(q, bi, bj);
    // (float columns: 32 rows a step, for the longer runs)
    constexpr bool kRows32 = sizeof(T) == 4;
    const int i0 = 32 * bi + (kRows32 && !rowmaj ? lane : block_row(rowmaj, 0, lane));
    const int c0 = 32 * bj + (kRows32 && !rowmaj ? 0 : block_col(rowmaj, 0, lane));
    auto di = [&](int u) { return rowmaj ? u : kRows32 ? 0 : (u & 3) * 8; };
    auto dc = [&](int u) { return rowmaj ? 0 : kRows32 ? u : (u >> 2) * 4; };
    const T* src = &A(i0, c0);
    double v[32];
#pragma unroll
    for (int u = 0; u < 32; ++u) {
        const int i = i0 + di(u), c = c0 + dc(u);
        v[u] = i == c ? 1.0 : 0.0;
        if (i < sz && (c < i || (c == i && !unit))) v[u] = (double)src[di(u) * A.rs + dc(u) * A.cs];
    }
#pragma unroll
    for (int u = 0; u < 32; ++u) {
        const int i = i0 + di(u), c = c0 + dc(u);
        if (c <= i) S[i * SLD + c] = v[u];
    }
}

// Half h of L's block q from S and ld back to A by one warp.
template <class T>
__device__ __forceinline__ void store_block(const View<T>& A, int sz, bool rowmaj, int q, int h, const double* S,
                                            const double* ld, int lane) {
    int bi, bj;
    lower_block(q, bi, bj);
    const int i0 = 32 * bi + block_row(rowmaj, 16 * h, lane), c0 = 32 * bj + block_col(rowmaj, 16 * h, lane);
    T* dst = &A(i0, c0);
    double v[16];
#pragma unroll
    for (int u = 0; u < 16; ++u) {
        const int i = rowmaj ? i0 + u : i0 + (u & 3) * 8, c = rowmaj ? c0 : c0 + (u >> 2) * 4;
        v[u] = *(i == c ? ld + i : S + i * SLD + c);
    }
    const int64_t r8 = 8 * A.rs, c4 = 4 * A.cs;
#pragma unroll
    for (int u = 0; u < 16; ++u) {
        const int i = rowmaj ? i0 + u : i0 + (u & 3) * 8, c = rowmaj ? c0 : c0 + (u >> 2) * 4;
        if (i < sz && c <= i) dst[rowmaj ? u * A.rs : (u >> 2) * c4 + (u & 3) * r8] = (T)v[u];
    }
}

// The same as calls: inlined, the FP32 instance's conversions took registers from the dependent
// chain of potrf_diag (44 us a block, 36 with calls; 29 in FP64).
__device__ __noinline__ void load_block_call(const View<float>& A, int sz, bool rowmaj, int q, double* S, int lane) {
    load_block(A, sz, rowmaj, false, q, S, lane);
}
__device__ __noinline__ void store_block_call(const View<float>& A, int sz, bool rowmaj, int q, int h, const double* S,
                                              const double* ld, int lane) {
    store_block(A, sz, rowmaj, q, h, S, ld, lane);
}
__device__ __noinline__ void store_inverse_call(const double* S, float* W, bool row_major, int q, int h, int lane) {
    store_inverse(S, W, row_major, q, h, lane);
}
__device__ __forceinline__ void load_block_call(const View<double>& A, int sz, bool rowmaj, int q, double* S, int lane) {
    load_block(A, sz, rowmaj, false, q, S, lane);
}
__device__ __forceinline__ void store_block_call(const View<double>& A, int sz, bool rowmaj, int q, int h,
                                                 const double* S, const double* ld, int lane) {
    store_block(A, sz, rowmaj, q, h, S, ld, lane);
}
__device__ __forceinline__ void store_inverse_call(const double* S, double* W, bool row_major, int q, int h, int lane) {
    store_inverse(S, W, row_major, q, h, lane);
}

// Named barriers of potrf_diag: kBarChunk + h says that columns 8 h .. 8 h + 7 of the
// sub-block being factored are in Lt and rd (warp 0 arrives, their readers wait).
constexpr int kBarBackground = 1, kBarChunk = 2;
__device__ __forceinline__ void named_sync(int id, int threads) {
    asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(threads) : "memory");
}
__device__ __forceinline__ void named_arrive(int id, int threads) {
    asm volatile("bar.arrive %0, %1;" ::"r"(id), "r"(threads) : "memory");
}

// One CTA per diagonal block: W_b = inverse of the lower-triangular block b of L. The 16-blocks
// are inverted by a warp each and merged pairwise on DMMA (16-, 32-, then 64-blocks).
// 64 blocks of an 8192-row FP64 triangle: 15 us (227 us with one thread per column and a
// barrier per row).
template <class T>
__global__ void __launch_bounds__(kDiagThreads, 1) trtri_blocks(int64_t m, View<const T> L, bool unit, T* W, int* info,
                                                                const int* abort) {
    extern __shared__ __align__(16) double S[];
    double *rd = S + kOffRd, *T64 = S + kOffT64, *T32 = S + kOffT32, *T16 = S + kOffT16;
    if (aborted(abort)) return;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int64_t r0 = (int64_t)blockIdx.x * NB;
    const int sz = (int)(m - r0 < NB ? m - r0 : NB);
    T* Wb = W + (size_t)blockIdx.x * NB * NB;
    const View<const T> A = L.sub(r0, r0);
    if (warp < 10) load_block(A, sz, A.cs == 1, unit, warp, S, lane);
    else if (warp < 13)
        for (int p = 0; p < NSUB - 1; ++p) zero_upper(Wb, false, p, tid - 320);
    __syncthreads();
    if (tid < NB) {
        const double d = S[tid * SLD + tid];
        if (!unit && info != nullptr && tid < sz && d == 0.0) record_first(info, (int)(r0 + tid + 1));
        rd[tid] = S[tid * SLD + tid] = 1.0 / d;
    }
    __syncthreads();
    if (warp < NSUB) {
        const int c0 = DB * warp;
        double* Lt = S + kOffLt + warp * DB * 16;  // columns of the sub-block, stride 16
        if (lane < DB) {
#pragma unroll
            for (int p = 0; p < DB; ++p) Lt[p * DB + lane] = S[(c0 + lane) * SLD + c0 + p];
        }
        __syncwarp();
        double x[DB];
#pragma unroll
        for (int q = 0; q < DB; ++q) x[q] = q == lane ? 1.0 : 0.0;
#pragma unroll
        for (int p = 0; p < DB; ++p) {
            x[p] *= rd[c0 + p];
#pragma unroll
            for (int q = p + 1; q < DB; ++q) x[q] = fma(-Lt[p * DB + q], x[p], x[q]);
        }
#pragma unroll
        for (int q = 0; q < DB; ++q)
            if (q > lane) S[(c0 + lane) * SLD + c0 + q] = x[q];
    }
    __syncthreads();
    // four 16-merges (scratch: T16 and, for the others, T64), two 32-merges, the 64-merge
    double* Tq = warp < 2 ? T16 : T64 + (warp >> 1) * 16 * 20;
    if (warp < 8) merge_t<16, SLD>(S, Tq, 32 * (warp >> 1), warp & 1, lane);
    __syncthreads();
    if (warp < 8) merge_x<16, SLD>(S, Tq, 32 * (warp >> 1), 0, 8 * (warp & 1), lane);
    __syncthreads();
    Tq = warp < 8 ? T32 : T64;
    merge_t<32, SLD>(S, Tq, 64 * (warp >> 3), warp & 7, lane);
    __syncthreads();
    merge_x<32, SLD>(S, Tq, 64 * (warp >> 3), 16 * (warp & 1), 8 * ((warp & 7) >> 1), lane);
    __syncthreads();
    for (int q = warp; q < 32; q += 16) merge_t<64, SLD>(S, T64, 0, q, lane);
    __syncthreads();
    for (int q = warp; q < 32; q += 16) merge_x<64, SLD>(S, T64, 0, 16 * (q & 3), 8 * (q >> 2), lane);
    __syncthreads();
    for (int q = warp; q < 20; q += 16) store_inverse(S, Wb, false, q >> 1, q & 1, lane);
}

// Factor the sz x sz lower diagonal block (A already offset to it) in FP64 and store
// inv(L) into W (column-major, or row-major when w_row_major); g0 = global index of the
// block for the pivot status. One CTA; the critical path is warp 0's, over the 16-column
// sub-blocks kb:
//   A. warp 0 factors the 16 x 16 diagonal sub-block and solves the 16 rows below it,
//      right-looking with each lane's row in registers. A column's chain is the shuffle of its
//      pivot, the reciprocal square root, the scaling and the next pivot's own update; the
//      column reaches the other lanes through shared memory and its rank-1 update runs in the
//      shadow of that chain. Eight columns behind, warps 1-3 solve the other rows below (each
//      thread a row, in registers) and warp 5 inverts the sub-block (each lane a column).
//   C. all warps apply the panel's rank-16 update to the next 16 columns (DMMA).
// The rest runs on the other warps in the shadow of A: the first loads, the trailing update
// beyond the next panel, the merges of the block inverse (X = -inv(D) C inv(A) for 16-, 32-,
// 64-blocks), so that after the last sub-block only the part of the inverse that depends on
// it is left.
// No DMMA work runs on the scheduler of warp 0 (warps 4, 8, 12) during A, and each role has a
// loop of its own, so that warp 0's stays in the instruction cache of its scheduler (the same
// schedule with the roles inside one loop ran the chain at half the speed, and on 32-column
// sub-blocks, whose unrolled steps are four times the code, 40% of all stalls were waits for
// instructions). Bound by latency: 128 dependent columns at ~180 cycles, ~1400 cycles a
// sub-block for C and its barriers, 5000 for the first loads and 7000 for the last merges and
// stores. In a factorisation of n = 1024: 26.5 us a block (46.7 with the merges and updates in
// register tiles on the critical path); beside the mixed solve's trailing update 43.5 (61.8).
template <class T>
__global__ void __launch_bounds__(kDiagThreads, 1) potrf_diag(View<T> A, int sz, int64_t g0, T* W, int* info,
                                                              bool w_row_major) {
    extern __shared__ __align__(16) double S[];
    double *Lt = S + kOffLt, *ld = S + kOffLd, *rd = S + kOffRd;
    double *T64 = S + kOffT64, *T32 = S + kOffT32, *T16 = S + kOffT16;
    volatile int* flags = reinterpret_cast<int*>(S + kOffEnd);  // [0]: failing column, [1]: start over
    const bool skip = aborted(info);  // looked at once the block's loads are under way
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const bool rowmaj = A.cs == 1;
    auto sync_all = [] { named_sync(0, kDiagThreads); };
    // The end of A for everybody: whether warp 0 has to start over (then once every thread has
    // read the flag).
    auto redo = [&] {
        sync_all();
        const bool r = flags[1] != 0;
        if (r) sync_all();
        return r;
    };
    // C by warps 1 .. 15: the next panel's update.
    auto next_panel = [&](int c0) {
        if (c0 + DB < NB) syrk_tiles(S, c0 + DB, 2, c0, warp - 1, kDiagThreads / 32 - 1, lane);
        sync_all();
    };
    // Warps 1 .. 3 with rows at sub-block kb, beyond the 32 of warp 0; participants of its
    // chunk barriers.
    auto solvers = [](int kb) { return kb < 6 ? (NB - DB * kb - 1) / 32 : 0; };
    auto participants = [&](int kb) { return 32 * (2 + solvers(kb)); };
    if (warp < 10) load_block_call(A, sz, rowmaj, warp, S, lane);
    if (skip) return;
    sync_all();
    if (warp == 0) {
#pragma unroll 1
        for (int kb = 0; kb < NSUB; ++kb) {
            const int c0 = DB * kb;
            double* row = S + (c0 + lane) * SLD + c0;
            auto arrive = [&](int h) { named_arrive(kBarChunk + h, participants(kb)); };
            double x[DB];
#pragma unroll
            for (int c = 0; c < DB; c += 2) {
                const double2 v = reinterpret_cast<const double2*>(row)[c / 2];
                x[c] = v.x;
                x[c + 1] = v.y;
            }
            factor_sub_block(x, Lt, ld + c0, rd + c0, lane, flags, arrive);
            __syncwarp();
            if (!flags[1] && c0 + lane < NB) {
#pragma unroll
                for (int q = 0; q < DB; ++q)
                    if (q < lane) row[q] = x[q];
            }
            if (redo()) {
                factor_sub_block_any(row, c0 + lane < NB, Lt, ld + c0, rd + c0, lane, flags, arrive);
                redo();
            }
            if (flags[0]) {
                if (lane == 0) record_first(info, (int)(g0 + c0 + flags[0]));
                return;
            }
            sync_all();
        }
    } else if (warp <= 3 || warp == 5) {
#pragma unroll 1
        for (int kb = 0; kb < NSUB; ++kb) {
            const int c0 = DB * kb, row = c0 + 32 * warp + lane;
            do {
                if (warp != 5 && warp > solvers(kb)) continue;
                double x[DB];
                double2* src = reinterpret_cast<double2*>(S + row * SLD + c0);
                if (warp == 5) {
#pragma unroll
                    for (int q = 0; q < DB; ++q) x[q] = q == lane ? 1.0 : 0.0;
                } else if (row < NB) {
#pragma unroll
                    for (int c = 0; c < DB; c += 2) {
                        const double2 v = src[c / 2];
                        x[c] = v.x;
                        x[c + 1] = v.y;
                    }
                }
                const int threads = participants(kb);
                solve_sub_block(x, rd + c0, Lt, [&](int h) { named_sync(kBarChunk + h, threads); });
                if (flags[1]) continue;
                if (warp == 5) {
                    double* dst = S + (c0 + lane) * SLD + c0;
#pragma unroll
                    for (int q = 0; q < DB; ++q)
                        if (q >= lane) dst[q] = x[q];
                } else if (row < NB) {
#pragma unroll
                    for (int c = 0; c < DB; c += 2) src[c / 2] = make_double2(x[c], x[c + 1]);
                }
            } while (redo());
            if (flags[0]) return;
            next_panel(c0);
        }
    } else if (warp % 4 != 0) {  // the eight background warps 6, 7, 9, 10, 11, 13, 14, 15
        constexpr int nbg = 8;
        const int bg = warp - 5 - warp / 4;
#pragma unroll 1
        for (int kb = 0; kb < NSUB; ++kb) {
            const int c0 = DB * kb;
            // panel kb - 1's update right of this panel: rows and columns from c0 + 16
            if (kb > 0) syrk_tiles(S, c0 + DB, NB, c0 - DB, bg, nbg, lane);
            if (kb == 2 || kb == 4 || kb == 6) {  // the 32-block before this sub-block
                if (bg < 2) merge_t<16, SLD>(S, T16, c0 - 32, bg, lane);
                named_sync(kBarBackground, 32 * nbg);
                if (bg < 2) merge_x<16, SLD>(S, T16, c0 - 32, 0, 8 * bg, lane);
                if (kb == 4) {
                    named_sync(kBarBackground, 32 * nbg);
                    merge_x<32, SLD>(S, T32, 0, 16 * (bg & 1), 8 * (bg >> 1), lane);
                }
            } else if (kb == 3 || kb == 7) {
                merge_t<32, SLD>(S, T32, kb == 3 ? 0 : 64, bg, lane);
                if (kb == 7) {
                    if (bg < 2) merge_t<16, SLD>(S, T16, 96, bg, lane);
                    // rows 64 .. 95 of the 64-merge need no part of the last 32 rows
                    for (int q = bg; q < 16; q += nbg) merge_x<64, SLD>(S, T64, 0, 16 * (q & 1), 8 * (q >> 1), lane);
                }
            }
            if (kb == 5 || kb == 6)  // T of the 64-merge, half of its columns each
                for (int q = bg; q < 16; q += nbg) merge_t<64, SLD>(S, T64, 0, 16 * (kb - 5) + q, lane);
            while (redo()) {}
            if (flags[0]) return;
            next_panel(c0);
        }
    } else {  // warps 4, 8, 12
#pragma unroll 1
        for (int kb = 0; kb < NSUB; ++kb) {
            if (kb < NSUB - 1) zero_upper(W, w_row_major, kb, 32 * (warp / 4 - 1) + lane);
            if (kb == NSUB - 1)  // the inverse's final blocks (0, 0), (1, 0), (1, 1), (2, 2)
                for (int q = warp / 4 - 1; q < 8; q += 3) store_inverse_call(S, W, w_row_major, q < 6 ? q >> 1 : 5, q & 1, lane);
            while (redo()) {}
            if (flags[0]) return;
            next_panel(DB * kb);
        }
    }
    // What depends on the last sub-blocks: the last 16-, the last 32-merge and the lower half
    // of the 64-merge (warps 0-7); meanwhile L goes back to global memory.
    if (warp < 8) {
        if (warp < 2) merge_x<16, SLD>(S, T16, 96, 0, 8 * warp, lane);
        named_sync(kBarBackground, 256);
        merge_x<32, SLD>(S, T32, 64, 16 * (warp & 1), 8 * (warp >> 1), lane);
        named_sync(kBarBackground, 256);
        merge_x<64, SLD>(S, T64, 0, 32, 8 * warp, lane);
        merge_x<64, SLD>(S, T64, 0, 48, 8 * warp, lane);
    } else {
        for (int q = warp - 8; q < 20; q += 8) store_block_call(A, sz, rowmaj, q >> 1, q & 1, S, ld, lane);
    }
    __syncthreads();
    if (warp < 12)  // the blocks of the inverse that are not stored yet
        store_inverse_call(S, W, w_row_major, warp < 4 ? 3 + (warp >> 1) : 6 + ((warp - 4) >> 1), warp & 1, lane);
}

template <class K>
int set_smem(K kernel, size_t bytes) {
    return cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes) == cudaSuccess
               ? RC_SUCCESS
               : RC_ERR_CUDA;
}

}  // namespace

// One sweep of substitution with the triangle A, given the inverses W of its diagonal blocks:
// panels solved a strip of columns per CTA, the other rows updated once per panel. 8192 x 1024:
// 2.92 ms (3.81 with a product, a copy and an update of all other rows per 128-row block), 2.28 of it in
// the updates.
template <class T>
int sweep(bool upper, int64_t m, int64_t n, View<const T> A, const T* W, bool w_row_major, View<T> B, cudaStream_t s,
          const int* abort) {
    constexpr int64_t per = kStripRows;
    const int64_t panels = (m + per - 1) / per;
    for (int64_t q = 0; q < panels; ++q) {
        const int64_t p0 = (upper ? panels - 1 - q : q) * per, sz = m - p0 < per ? m - p0 : per;
        const View<T> Bp = B.sub(p0, 0);
        RC_TRY(strip_solve<T>(upper, sz, n, A.sub(p0, p0), W + (size_t)p0 * NB, w_row_major, Bp, s, abort));
        const int64_t from = upper ? 0 : p0 + sz, rows = upper ? p0 : m - from;
        if (rows > 0)
            RC_TRY(gemm<T>(rows, n, sz, T(-1), A.sub(from, p0), View<const T>{Bp.p, Bp.rs, Bp.cs}, T(1),
                           B.sub(from, 0), kFull, 0, s, abort));
    }
    return RC_SUCCESS;
}

template <class T>
int trsm_left(bool upper, bool unit, int64_t m, int64_t n, T alpha, View<const T> A, View<T> B, int* info,
              cudaStream_t s, const int* abort) {
    if (m <= 0 || n <= 0) return RC_SUCCESS;
    const int64_t nblk = (m + NB - 1) / NB;
    T* W = static_cast<T*>(workspace(s, (size_t)nblk * NB * NB * sizeof(T), 1));
    if (!W) return RC_ERR_ALLOC;
    RC_TRY(trtri_blocks_launch<T>(m, upper ? A.t() : A, unit, W, info, abort, s));
    if (alpha != T(1)) RC_TRY(copy2d<T, T>(m, n, alpha, View<const T>{B.p, B.rs, B.cs}, B, s, abort));
    return trsm_preinv<T>(upper, m, n, A, W, false, B, s, abort);
}

template <class T>
int potrf_lower(int64_t n, View<T> A, int* info, cudaStream_t s, T* Winv) {
    if (!info) return RC_ERR_INVALID_ARGUMENT;
    if (cudaMemsetAsync(info, 0, sizeof(int), s) != cudaSuccess) return RC_ERR_CUDA;
    if (n <= 0) return RC_SUCCESS;
    // Outer panels of kOuter columns: 128-column steps factor the panel's diagonal block, the rows
    // below it are solved a strip per CTA (and so are those of a step inside the block), and the
    // trailing matrix gets one update of depth kOuter. SPD solve n = 1024, 16 right-hand sides:
    // 730 -> 568 us; FP32 factor and solves n = 3001: 3.09 -> 2.38 ms.
    constexpr int64_t kOuter = kStripRows;
    T* own = Winv ? nullptr : static_cast<T*>(workspace(s, (size_t)kOuter * NB * sizeof(T), 1));
    if (!Winv && !own) return RC_ERR_ALLOC;
    RC_TRY(set_smem(potrf_diag<T>, kDiagSmem));
    auto C_ = [](const View<T>& v) { return View<const T>{v.p, v.rs, v.cs}; };
    for (int64_t k0 = 0; k0 < n; k0 += kOuter) {
        const int64_t w = (n - k0) < kOuter ? n - k0 : kOuter, end = k0 + w;
        T* Wp = Winv ? Winv + k0 * NB : own;
        for (int64_t j0 = k0; j0 < end; j0 += NB) {
            const int jb = (int)(end - j0 < NB ? end - j0 : NB);
            T* W = Wp + (j0 - k0) * NB;
            potrf_diag<T><<<1, kDiagThreads, kDiagSmem, s>>>(A.sub(j0, j0), jb, j0, W, info, false);
            RC_TRY(check_launch());
            const int64_t rows = end - j0 - jb;
            if (rows <= 0) continue;
            const View<T> P = A.sub(j0 + jb, j0);
            RC_TRY(strip_solve<T>(false, jb, rows, C_(A.sub(j0, j0)), W, false, P.t(), s, info));
            RC_TRY(gemm<T>(rows, rows, jb, T(-1), C_(P), C_(P).t(), T(1), A.sub(j0 + jb, j0 + jb), kLower, 0, s,
                           info));
        }
        const int64_t rows = n - end;
        if (rows <= 0) continue;
        const View<T> Pk = A.sub(end, k0);
        RC_TRY(strip_solve<T>(false, w, rows, C_(A.sub(k0, k0)), Wp, false, Pk.t(), s, info));
        RC_TRY(gemm<T>(rows, rows, w, T(-1), C_(Pk), C_(Pk).t(), T(1), A.sub(end, end), kLower, 0, s, info));
    }
    return RC_SUCCESS;
}

template <class T>
int potrf_diag_block(View<T> A, int sz, int64_t g0, T* W, bool w_row_major, int* info, cudaStream_t s) {
    RC_TRY(set_smem(potrf_diag<T>, kDiagSmem));
    potrf_diag<T><<<1, kDiagThreads, kDiagSmem, s>>>(A, sz, g0, W, info, w_row_major);
    return check_launch();
}

template <class T>
int trsm_preinv(bool upper, int64_t m, int64_t n, View<const T> A, const T* Winv, bool w_row_major, View<T> B,
                cudaStream_t s, const int* abort) {
    if (m <= 0 || n <= 0) return RC_SUCCESS;
    const bool flip = upper != w_row_major;  // an upper triangle's blocks are the transposed inverses
    return sweep<T>(upper, m, n, A, Winv, flip, B, s, abort);
}

template <class T>
int trtri_blocks_launch(int64_t m, View<const T> L, bool unit, T* W, int* info, const int* abort, cudaStream_t s) {
    if (m <= 0) return RC_SUCCESS;
    RC_TRY(set_smem(trtri_blocks<T>, kDiagSmem));
    trtri_blocks<T><<<(unsigned)((m + NB - 1) / NB), kDiagThreads, kDiagSmem, s>>>(m, L, unit, W, info, abort);
    return check_launch();
}

template int trtri_blocks_launch<double>(int64_t, View<const double>, bool, double*, int*, const int*, cudaStream_t);
template int potrf_diag_block<float>(View<float>, int, int64_t, float*, bool, int*, cudaStream_t);
template int potrf_diag_block<double>(View<double>, int, int64_t, double*, bool, int*, cudaStream_t);
template int trsm_preinv<double>(bool, int64_t, int64_t, View<const double>, const double*, bool, View<double>,
                                 cudaStream_t, const int*);
template int trsm_left<double>(bool, bool, int64_t, int64_t, double, View<const double>, View<double>, int*,
                               cudaStream_t, const int*);
template int trsm_left<float>(bool, bool, int64_t, int64_t, float, View<const float>, View<float>, int*,
                              cudaStream_t, const int*);
template int potrf_lower<double>(int64_t, View<double>, int*, cudaStream_t, double*);
template int potrf_lower<float>(int64_t, View<float>, int*, cudaStream_t, float*);

}  // namespace rc

namespace {

template <class T>
int trsm_abi(int left, int upper, int trans, int unit, size_t m, size_t n, T alpha, const T* A, size_t lda, T* B,
             size_t ldb, int* d_info, void* stream) {
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    if (d_info && cudaMemsetAsync(d_info, 0, sizeof(int), s) != cudaSuccess) return RC_ERR_CUDA;
    if (m == 0 || n == 0) return RC_SUCCESS;
    const size_t na = left ? m : n;
    if (!A || !B || lda < na || ldb < m) return RC_ERR_INVALID_ARGUMENT;
    rc::View<const T> a = rc::colmajor(A, (int64_t)lda);
    bool up = upper != 0;
    if (trans) { a = a.t(); up = !up; }
    rc::View<T> b = rc::colmajor(B, (int64_t)ldb);
    if (left) return rc::trsm_left<T>(up, unit != 0, (int64_t)m, (int64_t)n, alpha, a, b, d_info, s);
    // B op(A)^-1: solve op(A)^T X^T = alpha B^T on the left.
    return rc::trsm_left<T>(!up, unit != 0, (int64_t)n, (int64_t)m, alpha, a.t(), b.t(), d_info, s);
}

template <class T>
int potrf_abi(int upper, size_t n, T* A, size_t lda, int* d_info, void* stream) {
    if (!d_info) return RC_ERR_INVALID_ARGUMENT;
    if (n > 0 && (!A || lda < n)) return RC_ERR_INVALID_ARGUMENT;
    rc::View<T> a = rc::colmajor(A, (int64_t)lda);
    if (upper) a = a.t();
    return rc::potrf_lower<T>((int64_t)n, a, d_info, static_cast<cudaStream_t>(stream));
}

}  // namespace

extern "C" {

int rc_trsm_f64(int left, int upper, int trans, int unit, size_t m, size_t n, double alpha, const double* A,
                size_t lda, double* B, size_t ldb, int* d_info, void* stream) {
    return trsm_abi<double>(left, upper, trans, unit, m, n, alpha, A, lda, B, ldb, d_info, stream);
}
int rc_trsm_f32(int left, int upper, int trans, int unit, size_t m, size_t n, float alpha, const float* A,
                size_t lda, float* B, size_t ldb, int* d_info, void* stream) {
    return trsm_abi<float>(left, upper, trans, unit, m, n, alpha, A, lda, B, ldb, d_info, stream);
}
int rc_potrf_f64(int upper, size_t n, double* A, size_t lda, int* d_info, void* stream) {
    return potrf_abi<double>(upper, n, A, lda, d_info, stream);
}
int rc_potrf_f32(int upper, size_t n, float* A, size_t lda, int* d_info, void* stream) {
    return potrf_abi<float>(upper, n, A, lda, d_info, stream);
}

int rc_spd_solve_f64(size_t n, size_t nrhs, const double* A, size_t lda, double* B, size_t ldb, int* d_info,
                     void* stream) {
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    if (!d_info) return RC_ERR_INVALID_ARGUMENT;
    if (n == 0) return cudaMemsetAsync(d_info, 0, sizeof(int), s) == cudaSuccess ? RC_SUCCESS : RC_ERR_CUDA;
    if (!A || lda < n || (nrhs > 0 && (!B || ldb < n))) return RC_ERR_INVALID_ARGUMENT;
    // The reference copies A into the decomposition's own storage (decompositions.hpp:81-84).
    double* L = static_cast<double*>(rc::workspace(s, n * n * sizeof(double), 3));
    if (!L) return RC_ERR_ALLOC;
    const rc::View<double> Lv = rc::colmajor(L, (int64_t)n);
    RC_TRY(rc::copy2d<double, double>((int64_t)n, (int64_t)n, 1.0, rc::colmajor(A, (int64_t)lda), Lv, s));
    // The factorisation's block inverses serve both solves.
    const int64_t nn = (int64_t)n, nblk = rc::ceil_div(n, rc::kNB);
    double* W = static_cast<double*>(rc::workspace(s, (size_t)nblk * rc::kNB * rc::kNB * sizeof(double), 1));
    if (!W) return RC_ERR_ALLOC;
    RC_TRY(rc::potrf_lower<double>(nn, Lv, d_info, s, W));
    if (nrhs == 0) return RC_SUCCESS;
    const rc::View<const double> Lc = {L, 1, nn};
    const rc::View<double> Bv = rc::colmajor(B, (int64_t)ldb);
    RC_TRY(rc::trsm_preinv<double>(false, nn, (int64_t)nrhs, Lc, W, false, Bv, s, d_info));
    return rc::trsm_preinv<double>(true, nn, (int64_t)nrhs, Lc.t(), W, false, Bv, s, d_info);
}

}  // extern "C"
