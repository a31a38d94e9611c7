// Batched uneven SPD solves: POTRF + the two triangular solves of many independent
// small systems (n <= 512) in ONE persistent launch, replayed as a CUDA graph.
//
// Extension on top of the reference's per-system path (cholesky_decomposition + solve,
// include/remora/decompositions.hpp:81-115; no batched counterpart exists there).
//
// Design:
//  * persistent CTAs (a multiple of the SM count) pull systems from an atomic work
//    counter over an order sorted by decreasing n, so the large systems start first and
//    the small ones fill the tail -- no inter-CTA waiting, only one atomicAdd per system;
//  * per system, a left-looking Cholesky in 32-column panels on DMMA, in FP64 also for float
//    matrices: the panel's rows, as 32 x 32 warp tiles in registers, subtract the product of
//    the columns before them (fragments straight from global memory, which L2 and L1 hold:
//    each element of L is read once per panel to its right, where a right-looking update
//    would read and write the whole trailing triangle per panel), and are solved with the
//    inverse of the panel's diagonal block;
//  * one warp factors and inverts the diagonal block (diag.cuh) while the others update the
//    rows below it;
//  * the right-hand side's forward substitution is part of the panels; the backward
//    substitution walks the panels with the kept inverses;
//  * a failing pivot records its 1-based index in info[i] and the CTA moves on.
// The warps per CTA are chosen per (precision, size bucket) by a small autotuner that times
// every candidate on the caller's batch, loaded and warm, and caches the winner.
//
// 1024 systems of 16 to 512 rows: 1.04 ms in FP64, 1.00 ms in FP32 (12.3 and 10.4 ms with FMA
// tiles over a right-looking update and one barrier per column), 11.9 GFLOP of which the DMMA
// pipe could do in 0.35 ms. What is left is latency: a 512-row system alone takes 0.52 ms, its
// 16 panels ~35K cycles each for the loads, the 32 dependent columns and three barriers. Tiles
// kept in registers from their update to their solve (which spill at two CTAs per SM) took
// 1.8 ms; the code is kept small (one form of each tile) because the phases of a panel are
// bound by instruction fetch before anything else.
#include <algorithm>
#include <map>
#include <memory>
#include <tuple>
#include <mutex>
#include <numeric>
#include <vector>

#include "common.cuh"
#include "diag.cuh"

namespace rc {
namespace {

constexpr int kMaxN = 512;

constexpr int PB = 32;      // panel width
constexpr int DLD = PB + 4;  // row stride of the diagonal block in shared memory
constexpr int kPacked = PB * (PB + 1) / 2;

// Shared memory (doubles): two diagonal blocks (this panel's and the next's), the scratch of
// their factorisation, the right-hand side y (then L^-1 b, then the solution), a panel's part
// of it and the packed inverses of the diagonal blocks of a matrix of up to nmax rows.
struct BatchedSmem {
    static constexpr int D = 0, Lt = D + 2 * PB * DLD, T16 = Lt + kDB * kLTD, ld = T16 + 16 * 20, rd = ld + PB,
                         flags = rd + PB, y = flags + 2, t = y + kMaxN + PB, inv = t + PB;
    static size_t bytes(int nmax) { return (size_t)(inv + (nmax + PB - 1) / PB * kPacked) * sizeof(double); }
};

// P = C - L(rows, 0 : k0) L(k0 : k0 + 32, 0 : k0)^T on the 32-row tile at r0 of the panel at k0, in
// place, by one warp. Rows past the matrix stand on its last row and are not stored. The
// fragments of two k-steps ahead are in flight; the last two fetches read columns of the panel
// itself, which exist (n > r0 >= k0 + 32), and are not used.
template <class T>
__device__ __forceinline__ void update_tile(T* A, int n, int k0, int r0, int lane) {
    const int g = lane >> 2, t = lane & 3;
    int row[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) row[u] = r0 + 8 * u + g < n ? r0 + 8 * u + g : n - 1;
    double acc[2][4][4] = {};
    const T *a = A + (int64_t)t * n, *b = a + k0 + g;
    const int64_t step = 4 * (int64_t)n;
    T av[4][4], bv[4][4];  // three of the four stages are live at a time
    auto fetch = [&](int st) {
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            av[st][u] = a[row[u]];
            bv[st][u] = b[8 * u];
        }
        a += step;
        b += step;
    };
    fetch(0);
    fetch(1);
#pragma unroll 1
    for (int k = 0; k < k0; k += 16)
#pragma unroll
        for (int st = 0; st < 4; ++st) {
            fetch((st + 2) & 3);
#pragma unroll
            for (int mi = 0; mi < 2; ++mi)
#pragma unroll
                for (int ni = 0; ni < 4; ++ni)
                    dmma_16x8x4(acc[mi][ni], (double)av[st][2 * mi], (double)av[st][2 * mi + 1], (double)bv[st][ni]);
        }
    T* c = A + (int64_t)(k0 + 2 * t) * n;
#pragma unroll
    for (int ni = 0; ni < 4; ++ni) {
        T old[2][4];
#pragma unroll
        for (int e = 0; e < 2; ++e)
#pragma unroll
            for (int u = 0; u < 4; ++u) old[e][u] = c[e * n + row[u]];
#pragma unroll
        for (int e = 0; e < 2; ++e)
#pragma unroll
            for (int u = 0; u < 4; ++u)
                if (r0 + 8 * u + g < n) c[e * n + row[u]] = (T)((double)old[e][u] - acc[u >> 1][ni][2 * (u & 1) + e]);
        c += 8 * (int64_t)n;
    }
}

// X = P inv(L_kk)^T on one tile, in place (all of it is loaded before any is stored), and
// y(rows) -= X y(k0 : k0 + 32): the forward substitution of the right-hand side. D holds the
// diagonal block's inverse, yp = y + k0.
template <class T>
__device__ __forceinline__ void solve_tile(T* A, const double* D, const double* yp, double* y, int n, int k0, int r0,
                                           int lane) {
    const int g = lane >> 2, t = lane & 3;
    int row[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) row[u] = r0 + 8 * u + g < n ? r0 + 8 * u + g : n - 1;
    T av[8][4];
    const T* p = A + (int64_t)(k0 + t) * n;
#pragma unroll
    for (int q = 0; q < 8; ++q) {
#pragma unroll
        for (int u = 0; u < 4; ++u) av[q][u] = p[row[u]];
        p += 4 * (int64_t)n;
    }
    __syncwarp();
#pragma unroll
    for (int mi = 0; mi < 2; ++mi) {
        double acc[4][4] = {};
#pragma unroll
        for (int q = 0; q < 8; ++q) {
            const int k = 4 * q + t;
#pragma unroll
            for (int ni = q / 2; ni < 4; ++ni) {  // inv(c, k), c = 8 ni + g: zero below the diagonal
                double v = D[k * DLD + 8 * ni + g];
                if (ni == q / 2) v = k <= 8 * ni + g ? v : 0.0;
                dmma_16x8x4(acc[ni], (double)av[q][2 * mi], (double)av[q][2 * mi + 1], v);
            }
        }
        T* c = A + (int64_t)(k0 + 2 * t) * n;
        double dot[2] = {};
#pragma unroll
        for (int ni = 0; ni < 4; ++ni) {
#pragma unroll
            for (int e = 0; e < 2; ++e)
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    dot[h] = fma(acc[ni][2 * h + e], yp[8 * ni + 2 * t + e], dot[h]);
                    if (r0 + 16 * mi + 8 * h + g < n) c[e * n + row[2 * mi + h]] = (T)acc[ni][2 * h + e];
                }
            c += 8 * (int64_t)n;
        }
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            dot[h] += __shfl_xor_sync(0xffffffffu, dot[h], 1);
            dot[h] += __shfl_xor_sync(0xffffffffu, dot[h], 2);
            if (t == 0 && r0 + 16 * mi + 8 * h + g < n) y[r0 + 16 * mi + 8 * h + g] -= dot[h];
        }
    }
}

// Factor the 32 x 32 block in D by one warp and build its inverse: two 16-column sub-blocks, then
// one merge. flags[0]: 1 + the failing column of the block, or 0.
__device__ __forceinline__ void factor_block(double* D, double* Lt, double* T16, double* ld, double* rd,
                                             volatile int* flags, int lane) {
#pragma unroll 1
    for (int c0 = 0; c0 < PB; c0 += kDB) {
        const bool mine = c0 + lane < PB;
        double* row = D + (mine ? c0 + lane : c0) * DLD + c0;
        double x[kDB];
#pragma unroll
        for (int c = 0; c < kDB; c += 2) {
            const double2 v = reinterpret_cast<const double2*>(row)[c / 2];
            x[c] = v.x;
            x[c + 1] = v.y;
        }
        factor_sub_block(x, Lt, ld + c0, rd + c0, lane, flags, [](int) {});
        __syncwarp();
        if (flags[1]) {
            factor_sub_block_any(row, mine, Lt, ld + c0, rd + c0, lane, flags, [](int) {});
        } else if (mine) {
#pragma unroll
            for (int q = 0; q < kDB; ++q)
                if (q < lane) row[q] = x[q];
        }
        __syncwarp();
        if (flags[0]) {
            if (lane == 0) flags[0] = flags[0] + c0;
            return;
        }
        // this sub-block's inverse, and the update of the next one
#pragma unroll
        for (int q = 0; q < kDB; ++q) x[q] = q == lane ? 1.0 : 0.0;
        solve_sub_block(x, rd + c0, Lt, [](int) {});
        if (lane < kDB) {
#pragma unroll
            for (int q = 0; q < kDB; ++q)
                if (q >= lane) row[q] = x[q];
        }
        if (c0 == 0) {
            syrk_tile<DLD>(D, kDB, kDB, 0, lane);
            syrk_tile<DLD>(D, kDB, kDB + 8, 0, lane);
        }
        __syncwarp();
    }
    merge_t<16, DLD>(D, T16, 0, 0, lane);
    merge_t<16, DLD>(D, T16, 0, 1, lane);
    __syncwarp();
    merge_x<16, DLD>(D, T16, 0, 0, 0, lane);
    merge_x<16, DLD>(D, T16, 0, 0, 8, lane);
    __syncwarp();
}

// D -= L(rows, ka : kb) L(rows, ka : kb)^T on tiles q, q + 1 (of the six 16 x 8 tiles on and
// below the diagonal: 0, 1 in rows 0 .. 15, 2 .. 5 in rows 16 .. 31) of the diagonal block at r0;
// first: D starts from the matrix (the identity beyond its n rows).
template <class T>
__device__ __forceinline__ void diag_tiles(const T* A, int n, int r0, int ka, int kb, int q, bool first, double* D,
                                           int lane) {
    const int g = lane >> 2, t = lane & 3, i0 = q < 2 ? 0 : 16, j0 = q < 4 ? 0 : 16;
    auto row = [&](int i) { return A + (r0 + i < n ? r0 + i : n - 1) + (int64_t)(ka + t) * n; };
    const T *a0 = row(i0 + g), *a1 = row(i0 + g + 8), *b0 = row(j0 + g), *b1 = row(j0 + g + 8);
    double acc[2][4] = {};
    const int64_t step = 4 * (int64_t)n;
#pragma unroll 4
    for (int k = ka; k < kb; k += 4) {
        const double x0 = (double)*a0, x1 = (double)*a1, y0 = (double)*b0, y1 = (double)*b1;
        a0 += step;
        a1 += step;
        b0 += step;
        b1 += step;
        dmma_16x8x4(acc[0], x0, x1, y0);
        dmma_16x8x4(acc[1], x0, x1, y1);
    }
#pragma unroll
    for (int h = 0; h < 2; ++h)
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            const int r = i0 + g + 8 * (e >> 1), c = j0 + 8 * h + 2 * t + (e & 1);
            double v = r == c ? 1.0 : 0.0;
            if (!first) v = D[r * DLD + c];
            else if (c <= r && r0 + r < n) v = (double)A[(r0 + r) + (int64_t)(r0 + c) * n];
            D[r * DLD + c] = r0 + r < n ? v - acc[h][e] : v;
        }
}

template <class T, int NW>
__global__ void __launch_bounds__(32 * NW, 16 / NW) batched_chol_solve(int count, const int* __restrict__ order,
                                                                       const int* __restrict__ sizes,
                                                                       T* const* __restrict__ Aptr,
                                                                       T* const* __restrict__ bptr,
                                                                       int* __restrict__ info, int* __restrict__ next) {
    extern __shared__ __align__(16) double sm[];
    using M = BatchedSmem;
    double *D = sm + M::D, *ld = sm + M::ld, *rd = sm + M::rd, *y = sm + M::y, *tv = sm + M::t, *inv = sm + M::inv;
    volatile int* flags = reinterpret_cast<int*>(sm + M::flags);
    __shared__ int s_work;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    constexpr int THREADS = 32 * NW;
    while (true) {
        __syncthreads();
        if (tid == 0) s_work = atomicAdd(next, 1);
        __syncthreads();
        if (s_work >= count) break;
        const int sys = order[s_work];
        const int n = sizes[sys];
        T* A = Aptr[sys];  // column-major, ld = n
        T* b = bptr[sys];
        for (int i = tid; i < n + PB; i += THREADS) y[i] = i < n ? (double)b[i] : 0.0;
        int failed = 0;
        for (int k0 = 0; k0 < n; k0 += PB) {
            // The diagonal block: the last panel's update (the earlier ones' came with that
            // panel's, below).
            double *Dk = D + (k0 / PB & 1) * PB * DLD, *Dn = D + (~(k0 / PB) & 1) * PB * DLD;
            for (int q = warp; q < 3; q += NW)
                diag_tiles(A, n, k0, k0 > 0 ? k0 - PB : 0, k0, 2 * q, k0 == 0, Dk, lane);
            __syncthreads();
            const int r1 = k0 + PB, tiles = r1 < n ? (n - r1 + 31) / 32 : 0;
            if (warp == 0) {
                factor_block(Dk, sm + M::Lt, sm + M::T16, ld, rd, flags, lane);
                double v = 0.0;  // y(k0 : k0 + 32) solved with the block
#pragma unroll 8
                for (int k = 0; k < PB; ++k)
                    if (k <= lane) v = fma(Dk[k * DLD + lane], y[k0 + k], v);
                __syncwarp();
                y[k0 + lane] = v;
            } else if (tiles > 0) {  // the rows below it, and the next diagonal block's update so far
                for (int q = warp - 1; q < tiles + 3; q += NW - 1) {
                    if (q < 3) diag_tiles(A, n, r1, 0, k0, 2 * q, true, Dn, lane);
                    else if (k0 > 0) update_tile(A, n, k0, r1 + 32 * (q - 3), lane);
                }
            }
            __syncthreads();
            if (flags[0]) {
                failed = k0 + flags[0];
                break;
            }
            for (int q = warp; q < tiles; q += NW) solve_tile(A, Dk, y + k0, y, n, k0, r1 + 32 * q, lane);
            // the diagonal block and its inverse (packed by rows)
            double* pk = inv + (k0 / PB) * kPacked;
            for (int e = tid; e < PB * PB; e += THREADS) {
                const int r = e % PB, c = e / PB;
                if (c > r) continue;
                pk[r * (r + 1) / 2 + c] = Dk[c * DLD + r];
                if (k0 + r < n) A[(k0 + r) + (int64_t)(k0 + c) * n] = (T)(r == c ? ld[r] : Dk[r * DLD + c]);
            }
            __syncthreads();
        }
        if (failed) {
            if (tid == 0) info[sys] = failed;
            continue;
        }
        // L^T x = y, panel by panel from the last: x_p = inv(L_pp)^T (y_p - L(below, p)^T x(below)).
        // A warp sums 32 / NW columns, its lanes along the rows.
        for (int k0 = (n - 1) / PB * PB; k0 >= 0; k0 -= PB) {
            constexpr int NC = PB / NW;
            double part[NC] = {};
            const int c0 = k0 + NC * warp;
#pragma unroll 2
            for (int i = k0 + PB + lane; i < n; i += 32) {
                const double xi = y[i];
#pragma unroll
                for (int c = 0; c < NC; ++c) part[c] = fma((double)A[i + (int64_t)(c0 + c) * n], xi, part[c]);
            }
#pragma unroll
            for (int c = 0; c < NC; ++c) {
#pragma unroll
                for (int off = 16; off > 0; off >>= 1) part[c] += __shfl_xor_sync(0xffffffffu, part[c], off);
                if (lane == c) tv[NC * warp + c] = y[c0 + c] - part[c];
            }
            __syncthreads();
            if (warp == 0) {
                const double* pk = inv + (k0 / PB) * kPacked;
                double v = 0.0;
#pragma unroll 8
                for (int r = 0; r < PB; ++r)
                    if (r >= lane) v = fma(pk[r * (r + 1) / 2 + lane], tv[r], v);
                y[k0 + lane] = v;
            }
            __syncthreads();
        }
        for (int i = tid; i < n; i += THREADS) b[i] = (T)y[i];
        if (tid == 0) info[sys] = 0;
    }
}

struct Config {
    int warps;
};

template <class T>
using KernelFn = void (*)(int, const int*, const int*, T* const*, T* const*, int*, int*);

template <class T>
KernelFn<T> kernel_for(Config c) {
    return c.warps == 8 ? batched_chol_solve<T, 8> : batched_chol_solve<T, 4>;
}

const Config kCandidates[] = {{8}, {4}};

// A plan: the device copy of sizes and order, the chosen configuration, the captured
// graph (work-counter reset + the persistent kernel) for one set of pointer arrays.
struct Plan {
    int dev = -1;
    int count = 0;
    const void* A = nullptr;
    const void* b = nullptr;
    const int* info = nullptr;
    std::vector<int> sizes;
    int* d_buf = nullptr;  // [next | order (count) | sizes (count)]
    Config cfg{8};
    cudaGraphExec_t exec = nullptr;
    ~Plan() {
        if (exec) cudaGraphExecDestroy(exec);
        if (d_buf) cudaFree(d_buf);
    }
};

std::mutex g_mutex;
// (device, element size, A pointer array, b pointer array, info, count) -> plan. The element
// size is part of the key: a plan's graph holds a kernel for one element type, and arrays of
// another type can come back at the same addresses.
std::map<std::tuple<int, int, const void*, const void*, const int*, int>, std::unique_ptr<Plan>> g_plans;
std::map<std::pair<int, int>, Config> g_tuned;  // (sizeof(T), bucket of the largest n) -> config

int size_bucket(const std::vector<int>& sizes) {
    const int mx = sizes.empty() ? 0 : *std::max_element(sizes.begin(), sizes.end());
    return mx <= 64 ? 0 : mx <= 128 ? 1 : mx <= 256 ? 2 : 3;
}

template <class T>
int launch_plain(const Plan& p, Config c, cudaStream_t s) {
    const size_t smem = BatchedSmem::bytes(*std::max_element(p.sizes.begin(), p.sizes.end()));
    auto fn = kernel_for<T>(c);
    // always the limit of the tallest batch: kept plans and other threads share the attribute
    if (cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)BatchedSmem::bytes(kMaxN)) !=
        cudaSuccess)
        return RC_ERR_CUDA;
    int per_sm = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, fn, 32 * c.warps, smem) != cudaSuccess || per_sm < 1)
        per_sm = 1;
    const int grid = std::min(sm_count() * per_sm, std::max(p.count, 1));
    if (cudaMemsetAsync(p.d_buf, 0, sizeof(int), s) != cudaSuccess) return RC_ERR_CUDA;
    fn<<<grid, 32 * c.warps, smem, s>>>(p.count, p.d_buf + 1, p.d_buf + 1 + p.count, (T* const*)p.A, (T* const*)p.b,
                                    const_cast<int*>(p.info), p.d_buf);
    return check_launch();
}

// Time each candidate once on the caller's batch (the factorisations happen in place, so
// the caller's matrices are first saved and restored around the tuning runs). A first run of all
// is not timed: it loads the kernels, which takes longer than they run and by chance differs
// between them (1 process of 6 kept 4 warps, 1.47 ms for 1024 systems, where 8 take 1.04).
template <class T>
int autotune(Plan& p, cudaStream_t s) {
    const auto key = std::make_pair((int)sizeof(T), size_bucket(p.sizes));
    {
        auto it = g_tuned.find(key);
        if (it != g_tuned.end()) {
            p.cfg = it->second;
            return RC_SUCCESS;
        }
    }
    // Save the inputs: host copies of the pointer arrays give every system's storage.
    std::vector<T*> hA(p.count), hb(p.count);
    if (cudaMemcpy(hA.data(), p.A, p.count * sizeof(T*), cudaMemcpyDeviceToHost) != cudaSuccess ||
        cudaMemcpy(hb.data(), p.b, p.count * sizeof(T*), cudaMemcpyDeviceToHost) != cudaSuccess)
        return RC_ERR_CUDA;
    size_t total = 0;
    for (int i = 0; i < p.count; ++i) total += (size_t)p.sizes[i] * p.sizes[i] + p.sizes[i];
    T* save = nullptr;
    if (cudaMalloc(&save, total * sizeof(T)) != cudaSuccess) return RC_ERR_ALLOC;
    note_allocation();
    auto copy_all = [&](bool to_save) {
        size_t off = 0;
        for (int i = 0; i < p.count; ++i) {
            const size_t nn = (size_t)p.sizes[i] * p.sizes[i], nb = p.sizes[i];
            if (to_save) {
                cudaMemcpyAsync(save + off, hA[i], nn * sizeof(T), cudaMemcpyDeviceToDevice, s);
                cudaMemcpyAsync(save + off + nn, hb[i], nb * sizeof(T), cudaMemcpyDeviceToDevice, s);
            } else {
                cudaMemcpyAsync(hA[i], save + off, nn * sizeof(T), cudaMemcpyDeviceToDevice, s);
                cudaMemcpyAsync(hb[i], save + off + nn, nb * sizeof(T), cudaMemcpyDeviceToDevice, s);
            }
            off += nn + nb;
        }
    };
    copy_all(true);
    float best = 1e30f;
    Config best_cfg = kCandidates[0];
    cudaEvent_t e0, e1;
    cudaEventCreate(&e0);
    cudaEventCreate(&e1);
    for (const Config& c : kCandidates) launch_plain<T>(p, c, s);  // (the later ones on what the first left)
    copy_all(false);
    for (const Config& c : kCandidates) {
        cudaEventRecord(e0, s);
        const int st = launch_plain<T>(p, c, s);
        cudaEventRecord(e1, s);
        copy_all(false);
        if (st != RC_SUCCESS) continue;
        cudaEventSynchronize(e1);
        float ms = 0.f;
        cudaEventElapsedTime(&ms, e0, e1);
        if (ms < best) {
            best = ms;
            best_cfg = c;
        }
    }
    cudaStreamSynchronize(s);
    cudaEventDestroy(e0);
    cudaEventDestroy(e1);
    cudaFree(save);
    p.cfg = best_cfg;
    g_tuned[key] = best_cfg;
    return RC_SUCCESS;
}

template <class T>
int batched(size_t count, const int* h_n, T* const* d_A, T* const* d_b, int* d_info, int autotune_flag,
            cudaStream_t s) {
    if (count == 0) return RC_SUCCESS;
    if (!h_n || !d_A || !d_b || !d_info || count > (size_t)INT32_MAX) return RC_ERR_INVALID_ARGUMENT;
    for (size_t i = 0; i < count; ++i)
        if (h_n[i] < 1 || h_n[i] > kMaxN) return RC_ERR_NOT_SUPPORTED;
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) return RC_ERR_CUDA;
    std::lock_guard<std::mutex> lock(g_mutex);
    auto key = std::make_tuple(dev, (int)sizeof(T), (const void*)d_A, (const void*)d_b, (const int*)d_info, (int)count);
    std::unique_ptr<Plan>& slot = g_plans[key];
    std::vector<int> sizes(h_n, h_n + count);
    if (slot && slot->sizes != sizes) slot.reset();
    if (!slot) {
        auto p = std::make_unique<Plan>();
        p->dev = dev;
        p->count = (int)count;
        p->A = d_A;
        p->b = d_b;
        p->info = d_info;
        p->sizes = sizes;
        std::vector<int> order(count);
        std::iota(order.begin(), order.end(), 0);
        std::stable_sort(order.begin(), order.end(), [&](int a, int b) { return sizes[a] > sizes[b]; });
        std::vector<int> host(1 + 2 * count, 0);
        std::copy(order.begin(), order.end(), host.begin() + 1);
        std::copy(sizes.begin(), sizes.end(), host.begin() + 1 + count);
        if (cudaMalloc(&p->d_buf, host.size() * sizeof(int)) != cudaSuccess) return RC_ERR_ALLOC;
        note_allocation();
        if (cudaMemcpy(p->d_buf, host.data(), host.size() * sizeof(int), cudaMemcpyHostToDevice) != cudaSuccess)
            return RC_ERR_CUDA;
        if (autotune_flag) RC_TRY(autotune<T>(*p, s));
        // Capture counter reset + kernel once; later calls replay the graph.
        cudaStream_t cs;
        if (cudaStreamCreateWithFlags(&cs, cudaStreamNonBlocking) != cudaSuccess) return RC_ERR_CUDA;
        cudaGraph_t g = nullptr;
        int st = cudaStreamBeginCapture(cs, cudaStreamCaptureModeRelaxed) == cudaSuccess ? RC_SUCCESS : RC_ERR_CUDA;
        if (st == RC_SUCCESS) st = launch_plain<T>(*p, p->cfg, cs);
        if (cudaStreamEndCapture(cs, &g) != cudaSuccess && st == RC_SUCCESS) st = RC_ERR_CUDA;
        cudaStreamDestroy(cs);
        if (st == RC_SUCCESS && cudaGraphInstantiate(&p->exec, g, 0) != cudaSuccess) st = RC_ERR_CUDA;
        if (g) cudaGraphDestroy(g);
        if (st != RC_SUCCESS) {
            cudaGetLastError();
            return st;
        }
        slot = std::move(p);
    }
    if (cudaGraphLaunch(slot->exec, s) != cudaSuccess) return RC_ERR_CUDA;
    count_launch();
    return RC_SUCCESS;
}

}  // namespace
}  // namespace rc

extern "C" {

int rc_potrf_trsm_batched_f64(size_t count, const int* h_n, double* const* d_A, double* const* d_b, int* d_info,
                              int autotune, void* stream) {
    return rc::batched<double>(count, h_n, d_A, d_b, d_info, autotune, static_cast<cudaStream_t>(stream));
}
int rc_potrf_trsm_batched_f32(size_t count, const int* h_n, float* const* d_A, float* const* d_b, int* d_info,
                              int autotune, void* stream) {
    return rc::batched<float>(count, h_n, d_A, d_b, d_info, autotune, static_cast<cudaStream_t>(stream));
}
int rc_batched_release_plans(void) {
    std::lock_guard<std::mutex> lock(rc::g_mutex);
    rc::g_plans.clear();
    return RC_SUCCESS;
}

}  // extern "C"
