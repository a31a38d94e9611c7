// LU with partial pivoting (getrf) and pivoted Cholesky (pstrf) on the GPU, in place on
// any strided view of the logical n x n matrix.
//
// getrf (kernels/getrf.hpp:50-59; CPU algorithm kernels/default/getrf.hpp:41-181):
// blocked right-looking LU with 64-column panels. A panel (of up to 4096 rows on one
// thread-block cluster, beyond that on a cooperative grid or one CTA) is factored column by
// column -- pivot = the row of largest |A(i, j)| at or below the diagonal (the lowest
// row among equals, as the reference's strictly-larger scan), the swap of the two rows
// across the panel, the division of the column by the pivot (in double, as the
// reference), the rank-1 update of the panel -- then the panel's swaps are applied to
// the other columns in order, U12 = L11^-1 A12 (unit lower TRSM) and A22 -= L21 U12 (DMMA
// GEMM). piv[i] is the row swapped with row i at step i (LAPACK order, 0-based, as
// Remora's permutation_matrix). A zero pivot records its 1-based column in *info and
// stops every later kernel (the reference throws).
//
// pstrf (kernels/pstrf.hpp:62-70; CPU algorithm kernels/default/pstrf.hpp:40-147, the
// blocked pivoted Cholesky of LAWN 161): blocks of 32 columns. One CTA runs a block: the
// pivot values (the trailing diagonal, refreshed from the block's finished columns)
// choose the largest remaining pivot (the lowest index among equals, as std::max_element),
// rows and columns of the whole matrix are swapped, the factor stops with rank c when the
// pivot value is below n^2 eps max|A_ii| (the trailing square is cleared), else the
// column is finished by the dot products with the block's earlier columns and a division,
// and the row right of the diagonal is cleared. After the block the whole trailing square
// (both triangles, which later swaps read) is updated by a DMMA GEMM with the block's
// columns. piv as for getrf (identity where no swap happened); the rank goes to *rank.
#include <cooperative_groups.h>

#include <cfloat>
#include <climits>
#include <cmath>

#include "diag.cuh"
#include "factor.cuh"
#include "gemm.cuh"
#include "per_device.cuh"

namespace cg = cooperative_groups;

namespace rc {
namespace {

constexpr int kLuNB = 64;       // getrf panel width
constexpr int kPsNB = 32;       // pstrf block width
constexpr int kLuThreads = 1024;

// Block-wide (value, index) reduction: larger value wins, the smaller index among equals.
__device__ __forceinline__ void argmax_pair(double& v, int64_t& i, double ov, int64_t oi) {
    if (ov > v || (ov == v && oi < i)) {
        v = ov;
        i = oi;
    }
}

__device__ void block_argmax(double& v, int64_t& i, double* sv, int64_t* si) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
    for (int o = 16; o; o >>= 1) argmax_pair(v, i, __shfl_xor_sync(0xffffffffu, v, o),
                                             __shfl_xor_sync(0xffffffffu, i, o));
    if (lane == 0) {
        sv[warp] = v;
        si[warp] = i;
    }
    __syncthreads();
    if (warp == 0) {
        v = lane < (int)(blockDim.x >> 5) ? sv[lane] : -DBL_MAX;
        i = lane < (int)(blockDim.x >> 5) ? si[lane] : INT64_MAX;
#pragma unroll
        for (int o = 16; o; o >>= 1) argmax_pair(v, i, __shfl_xor_sync(0xffffffffu, v, o),
                                                 __shfl_xor_sync(0xffffffffu, i, o));
        if (lane == 0) {
            sv[0] = v;
            si[0] = i;
        }
    }
    __syncthreads();
    v = sv[0];
    i = si[0];
    __syncthreads();
}

template <class T>
__global__ void __launch_bounds__(kLuThreads) getrf_panel_kernel(int64_t n, View<T> A, int64_t k0, int nb, int* piv,
                                                                 int* info) {
    __shared__ double sv[32];
    __shared__ int64_t si[32];
    if (*(volatile int*)info != 0) return;
    for (int j = 0; j < nb; ++j) {
        const int64_t c = k0 + j;
        double best = -1.0;
        int64_t bi = INT64_MAX;
        for (int64_t i = c + threadIdx.x; i < n; i += blockDim.x) {
            const double a = fabs((double)A(i, c));
            if (a > best) {
                best = a;
                bi = i;
            }
        }
        block_argmax(best, bi, sv, si);
        const int64_t p = bi == INT64_MAX ? c : bi;  // nothing but NaN: the row itself
        const double pv = (double)A(p, c);
        if (pv == 0.0) {  // also all-zero columns: the first row is the pivot, value 0
            if (threadIdx.x == 0) {
                piv[c] = (int)c;
                record_first(info, (int)(c + 1));
            }
            return;
        }
        if (threadIdx.x == 0) piv[c] = (int)p;
        if (p != c)
            for (int col = threadIdx.x; col < nb; col += blockDim.x) {
                const T t = A(c, k0 + col);
                A(c, k0 + col) = A(p, k0 + col);
                A(p, k0 + col) = t;
            }
        __syncthreads();
        for (int64_t i = c + 1 + threadIdx.x; i < n; i += blockDim.x) A(i, c) = (T)((double)A(i, c) / pv);
        __syncthreads();
        const int64_t rows = n - c - 1, cols = nb - j - 1;
        for (int64_t e = threadIdx.x; e < rows * cols; e += blockDim.x) {
            const int64_t i = c + 1 + e % rows, col = c + 1 + e / rows;
            A(i, col) -= A(i, c) * A(c, col);
        }
        __syncthreads();
    }
}

// The same panel factorisation spread over a cooperative grid: CTA b holds rows
// [k0 + b chunk, k0 + (b + 1) chunk) of the panel in shared memory (row stride nb + 1), and
// one bounded grid barrier per column exchanges what the next column needs. For column j
// (c = k0 + j), after the barrier every CTA reduces the published candidates in the same
// order (so all agree on the pivot p) and reads p's row; the owners of rows c and p swap
// them; then, with a look-ahead of one column:
//   1. every row below c is divided by the pivot and only its column j + 1 is updated;
//   2. the CTA's candidate for column j + 1 (largest |A(i, c + 1)|, i > c, the lowest row
//      among equals) and row c + 1 are updated in full and published;
//   3. the CTA arrives at the barrier, applies the rest of the rank-1 update to its other
//      rows while the others arrive, and waits.
// Each element sees exactly the operations of getrf_panel_kernel, in the same order.
constexpr int kCoopThreads = 256;
constexpr int kCoopMaxChunk = 384;  // rows per CTA (shared memory: 384 x 65 doubles)

struct CoopScratch {  // indexed by column j; the barrier words live separately
    double* cand_v;   // [nb][G]
    int64_t* cand_i;  // [nb][G]
    double* cand_row; // [nb][G][nb]
    double* crow;     // [nb][nb]: row c before the swap
};

// Grid barrier over nblocks co-resident CTAs (a cooperative launch), split into an arrival
// and a wait so that work can run in between: bar[0] counts arrivals, bar[1] is the
// generation. The wait is bounded by the SM's cycle counter (2 cycles per ns of the
// library's wait limit); a timeout records RC_ERR_TIMEOUT in the error word and the caller
// leaves, with the panel's first column in the status word: piv is not whole, and the later kernels
// would swap by it.
__device__ void grid_arrive(unsigned* bar, unsigned nblocks, unsigned gen) {
    __syncthreads();  // every thread's stores before the arrival
    if (threadIdx.x == 0) {
        __threadfence();
        if (atomicAdd(&bar[0], 1u) == nblocks - 1) {
            atomicExch(&bar[0], 0u);
            __threadfence();
            atomicExch(&bar[1], gen + 1u);
        }
    }
}
__device__ bool grid_wait(unsigned* bar, unsigned& gen, uint64_t limit_ns, int* err, int* pass) {
    if (threadIdx.x == 0) {
        int ok = 1;
        const long long t0 = clock64(), lim = (long long)(limit_ns * 2u);
        while (*(volatile unsigned*)&bar[1] == gen) {
            if (clock64() - t0 > lim) {
                ok = 0;
                if (err && atomicCAS(err, 0, RC_ERR_TIMEOUT) == 0) atomicExch(err + 1, 500);
                break;
            }
            __nanosleep(32);
        }
        __threadfence();
        *pass = ok;
    }
    __syncthreads();
    ++gen;
    return *pass != 0;
}

template <class T>
__global__ void __launch_bounds__(kCoopThreads, 1)
    getrf_panel_coop_kernel(int64_t n, View<T> A, int64_t k0, int nb, int chunk, int* piv, int* info,
                            CoopScratch sc, unsigned* bar, int* err, uint64_t limit_ns, T* linv) {
    extern __shared__ unsigned char coop_smem[];
    T* P = reinterpret_cast<T*>(coop_smem);  // chunk x (nb + 1)
    double* prow = reinterpret_cast<double*>(coop_smem) + ((size_t)chunk * (nb + 1) * sizeof(T) + 7) / 8;  // nb
    double* sv = prow + kLuNB;                                // 32
    int64_t* si = reinterpret_cast<int64_t*>(sv + 32);        // 32
    int* pass = reinterpret_cast<int*>(si + 32);
    const int ld = nb + 1, G = (int)gridDim.x, b = (int)blockIdx.x;
    if (*(volatile int*)info != 0) return;
    const int64_t base = k0 + (int64_t)b * chunk;
    const int myrows = (int)(n - base < chunk ? (n - base > 0 ? n - base : 0) : chunk);
    for (int e = threadIdx.x; e < myrows * nb; e += kCoopThreads) {
        const int r = e / nb, col = e % nb;
        P[r * ld + col] = A(base + r, k0 + col);
    }
    __syncthreads();
    // Publish the candidate for column j (rows >= k0 + j) and row k0 + j; both fully updated.
    auto publish = [&](int j, double best, int64_t bi) {
        const int64_t c = k0 + j;
        if (threadIdx.x == 0) {
            sc.cand_v[(size_t)j * G + b] = best;
            sc.cand_i[(size_t)j * G + b] = bi;
        }
        if (bi != INT64_MAX) {
            double* dst = sc.cand_row + ((size_t)j * G + b) * nb;
            for (int col = threadIdx.x; col < nb; col += kCoopThreads) dst[col] = (double)P[(bi - base) * ld + col];
        }
        if (c >= base && c < base + myrows)
            for (int col = threadIdx.x; col < nb; col += kCoopThreads)
                sc.crow[(size_t)j * nb + col] = (double)P[(c - base) * ld + col];
    };
    auto local_argmax = [&](int j, double& best, int64_t& bi) {
        const int64_t c = k0 + j;
        best = -1.0;
        bi = INT64_MAX;
        for (int r = threadIdx.x; r < myrows; r += kCoopThreads) {
            const int64_t i = base + r;
            if (i < c) continue;
            const double a = fabs((double)P[r * ld + j]);
            if (a > best || (a == best && i < bi)) {
                best = a;
                bi = i;
            }
        }
        block_argmax(best, bi, sv, si);
    };
    auto gave_up = [&] {
        if (threadIdx.x == 0) record_first(info, (int)(k0 + 1));
    };
    unsigned gen = 0;
    {  // column 0 needs no update first
        double best;
        int64_t bi;
        local_argmax(0, best, bi);
        publish(0, best, bi);
        grid_arrive(bar, (unsigned)G, gen);
        if (!grid_wait(bar, gen, limit_ns, err, pass)) {
            gave_up();
            return;
        }
    }
    for (int j = 0; j < nb; ++j) {
        const int64_t c = k0 + j;
        // The pivot: every CTA reduces the G candidates in the same order.
        double best = -1.0;
        int64_t bi = INT64_MAX;
        for (int q = threadIdx.x; q < G; q += kCoopThreads) {
            const double v = __ldcg(sc.cand_v + (size_t)j * G + q);
            const int64_t i = __ldcg(sc.cand_i + (size_t)j * G + q);
            if (v > best || (v == best && i < bi)) {
                best = v;
                bi = i;
            }
        }
        block_argmax(best, bi, sv, si);
        const int64_t p = bi == INT64_MAX ? c : bi;  // nothing but NaN: the row itself
        const int owner = (int)((p - k0) / chunk);
        const double* pr = bi == INT64_MAX ? sc.crow + (size_t)j * nb : sc.cand_row + ((size_t)j * G + owner) * nb;
        for (int col = threadIdx.x; col < nb; col += kCoopThreads) prow[col] = __ldcg(pr + col);
        __syncthreads();
        const double pv = prow[j];
        if (pv == 0.0) {  // also all-zero columns: the first row is the pivot, value 0
            if (b == 0 && threadIdx.x == 0) {
                piv[c] = (int)c;
                record_first(info, (int)(c + 1));
            }
            return;
        }
        if (b == 0 && threadIdx.x == 0) piv[c] = (int)p;
        if (p != c) {
            if (c >= base && c < base + myrows)
                for (int col = threadIdx.x; col < nb; col += kCoopThreads) P[(c - base) * ld + col] = (T)prow[col];
            if (p >= base && p < base + myrows)
                for (int col = threadIdx.x; col < nb; col += kCoopThreads)
                    P[(p - base) * ld + col] = (T)__ldcg(sc.crow + (size_t)j * nb + col);
        }
        __syncthreads();
        // 1. divide, and update column j + 1 only
        for (int r = threadIdx.x; r < myrows; r += kCoopThreads) {
            if (base + r <= c) continue;
            T* row = P + r * ld;
            const T l = (T)((double)row[j] / pv);
            row[j] = l;
            if (j + 1 < nb) row[j + 1] -= l * (T)prow[j + 1];
        }
        __syncthreads();
        if (j + 1 == nb) break;
        // 2. the candidate for column j + 1 and row c + 1, updated in full and published
        local_argmax(j + 1, best, bi);
        const int64_t rc1 = c + 1;
        const bool own_c1 = rc1 >= base && rc1 < base + myrows;
        const int ra = bi != INT64_MAX ? (int)(bi - base) : -1;
        const int rb = own_c1 ? (int)(rc1 - base) : -1;
        for (int col = j + 2 + threadIdx.x; col < nb; col += kCoopThreads) {
            if (ra >= 0) P[ra * ld + col] -= P[ra * ld + j] * (T)prow[col];
            if (rb >= 0 && rb != ra) P[rb * ld + col] -= P[rb * ld + j] * (T)prow[col];
        }
        __syncthreads();
        publish(j + 1, best, bi);
        grid_arrive(bar, (unsigned)G, gen);
        // 3. the rest of the rank-1 update while the other CTAs arrive
        for (int r = threadIdx.x; r < myrows; r += kCoopThreads) {
            if (base + r <= c || r == ra || r == rb) continue;
            T* row = P + r * ld;
            const T l = row[j];
            for (int col = j + 2; col < nb; ++col) row[col] -= l * (T)prow[col];
        }
        if (!grid_wait(bar, gen, limit_ns, err, pass)) {
            gave_up();
            return;
        }
    }
    __syncthreads();
    for (int e = threadIdx.x; e < myrows * nb; e += kCoopThreads) {
        const int r = e / nb, col = e % nb;
        A(base + r, k0 + col) = P[r * ld + col];
    }
    if (b != 0) return;
    // CTA 0 holds L11 (rows k0 .. k0 + nb, unit lower): its inverse, in place over L11 in
    // shared memory, column by column from the last (X L = I gives, for q > j,
    // X(q, j) = -(L(q, j) + sum_{j < m < q} X(q, m) L(m, j)), columns m > j already final),
    // then to linv (row-major nb x nb) for the TRSM of the rows right of the panel.
    __syncthreads();
    for (int j = nb - 2; j >= 0; --j) {
        const int q = j + 1 + threadIdx.x;
        T v = 0;
        if (q < nb) {
            v = P[q * ld + j];
            for (int m = j + 1; m < q; ++m) v += P[q * ld + m] * P[m * ld + j];
        }
        __syncthreads();
        if (q < nb) P[q * ld + j] = -v;
        __syncthreads();
    }
    for (int e = threadIdx.x; e < nb * nb; e += kCoopThreads) {
        const int q = e / nb, m = e % nb;
        linv[e] = q > m ? P[q * ld + m] : (q == m ? T(1) : T(0));
    }
}

// The panel factorisation on one thread-block cluster: CTA r of the G (a power of two, at most
// 16) holds rows [k0 + 256 r, k0 + 256 (r + 1)) of the panel, a thread per row, in shared memory
// P (row stride kClLd). The panel is walked in 16-column strips, whose rows are in registers,
// rotated so that a[0] is the column to eliminate. Per column every CTA sends its candidate
// (largest |a[0]|, the lowest row among equals) and that row into every CTA's shared memory by
// st.async and waits for theirs on its own mbarrier. All that a column writes for other warps or
// CTAs to read (the warps' candidates, their rows, row c, the exchanged keys and rows, the mbarrier)
// exists twice, by the column's parity: a wait ends once one warp of every CTA has sent, so a warp may
// be a column ahead of the others of its CTA, but not two, as the barrier between its candidate and
// its sending lies in between; and what is sent for a column is sent after its reader has read all of
// the column before last. Then all agree on the pivot, the two rows swap within the strip, and
// every row is divided and updated. Per strip, the swaps of the panel's other columns (and of the
// strip's own finished ones) are gathered through distributed shared memory, the strip's 16 rows
// of U are solved, and the columns to the right are updated on DMMA. Each element sees the pivot,
// division and update order of getrf_panel_kernel, a strip's sixteen products summed before they
// are subtracted.
// Bound by latency: of a column's ~2400 cycles (8 CTAs) the two-level search for the candidate
// takes ~1000, sending and waiting ~600 (cluster barriers instead: 860, with 16 CTAs 1400
// instead of 720), the agreed pivot, the division and the update ~700. 2048 x 64: about 105 us (385 on
// the cooperative grid, whose columns cost a grid barrier and two round trips through L2).
//
// Every way out of the column loop is taken by all threads of a CTA at the same barrier, and the
// panel's end by all CTAs at the same cluster barrier, so that none leaves while another writes or
// reads its shared memory: what ends the panel (a zero pivot, a message that does not come) is set
// down in every CTA and looked at after the strip. (It is set down behind the loop: a way back into
// the loop would keep two places for every a[q], 5% of a panel's time.) A wait beyond its limit alone
// ends nothing: the panel goes on, and the error word tells of it.
constexpr int kClThreads = 256, kStrip = 16, kClLd = kLuNB + 4, kClMax = 16;
constexpr int kZeroPivot = 1, kGaveUp = 2;
constexpr long long kClGrace = 4000000000ll;  // cycles beyond its limit after which a wait gives up
constexpr long long kClDrain = 1ll << 20;     // cycles in which a message under way arrives

template <class T>
struct ClusterSmem {
    T P[kClThreads * kClLd];
    T cand_row[2][kClMax][kStrip];  // by column parity and CTA
    T crow[2][kStrip];              // row c before the swap
    uint64_t cand_key[2][kClMax][2];  // (hi, lo) of |a[0]|; the row
    uint64_t bar[2];
    int late;     // a wait took longer than its limit
    int stop[2];  // by column parity: this CTA's column work ends (kZeroPivot or kGaveUp)
    int ends;     // why the cluster's panel ends early, 0 if it does not
    int from_all[2 * kStrip], from_strip[2 * kStrip][kStrip], dest[2 * kStrip];
    T mine[2][8][kStrip], top[2][kStrip];  // by column parity: the warps' candidate rows; row c
    T U[kStrip][kLuNB];
    unsigned whi[2][8], wlo[2][8];  // by column parity: the warps' candidates
    int widx[2][8];
    int pivots[kStrip];
    // the inverse of L11 (read and written in pairs)
    alignas(16) double L[kLuNB * kClLd];
    alignas(16) double Lt[4][kDB * kLTD];
    alignas(16) double T16[2][16 * 20];
    alignas(16) double T32[32 * 36];
    double rd[kLuNB];
};
static_assert(sizeof(ClusterSmem<double>) <= 227 * 1024, "a CTA's shared memory");

// Largest (hi, lo), the smallest idx among equals, over a warp; lanes without a candidate have
// hi = 0 and idx = INT_MAX.
__device__ __forceinline__ void warp_best(unsigned& hi, unsigned& lo, int& idx) {
    const unsigned mh = __reduce_max_sync(0xffffffffu, hi), at = __ballot_sync(0xffffffffu, hi == mh);
    if ((at & (at - 1)) == 0) {  // one lane has it
        const int src = __ffs((int)at) - 1;
        lo = __shfl_sync(0xffffffffu, lo, src);
        idx = __shfl_sync(0xffffffffu, idx, src);
        hi = mh;
        return;
    }
    const unsigned ml = __reduce_max_sync(0xffffffffu, hi == mh ? lo : 0u);
    idx = __reduce_min_sync(0xffffffffu, hi == mh && lo == ml ? idx : INT_MAX);
    hi = mh;
    lo = ml;
}

__device__ __forceinline__ uint32_t peer_address(const void* p, int rank) {
    uint32_t r;
    asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"((uint32_t)__cvta_generic_to_shared(p)), "r"(rank));
    return r;
}
__device__ __forceinline__ void send(uint32_t to, uint64_t v, uint32_t bar) {
    asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.b64 [%0], %1, [%2];" ::"r"(to), "l"(v), "r"(bar)
                 : "memory");
}
__device__ __forceinline__ void send(uint32_t to, double v, uint32_t bar) {
    send(to, (uint64_t)__double_as_longlong(v), bar);
}
__device__ __forceinline__ void send(uint32_t to, float v, uint32_t bar) {
    asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.b32 [%0], %1, [%2];" ::"r"(to),
                 "r"(__float_as_uint(v)), "r"(bar)
                 : "memory");
}
// Waits for phase `parity` of the mbarrier. 0: it completed within `limit` cycles, 1: later, 2: not
// within kClGrace more.
__device__ __forceinline__ int wait_phase(uint64_t* bar, unsigned parity, long long limit) {
    const uint32_t b = (uint32_t)__cvta_generic_to_shared(bar);
    const long long t0 = clock64();
    while (true) {
        uint32_t ok;
        asm volatile(
            "{\n.reg .pred p;\nmbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\nselp.u32 %0, 1, 0, p;\n}"
            : "=r"(ok)
            : "r"(b), "r"(parity)
            : "memory");
        const long long over = clock64() - t0 - limit;
        if (ok) return over > 0;
        if (over > kClGrace) return 2;
    }
}

template <class T>
__global__ void __launch_bounds__(kClThreads, 1)
    getrf_panel_cluster_kernel(int64_t n, View<T> A, int64_t k0, int nb, int* piv, int* info, T* linv, int* err,
                               uint64_t limit_ns) {
    extern __shared__ __align__(16) unsigned char cl_smem[];
    ClusterSmem<T>& sm = *reinterpret_cast<ClusterSmem<T>*>(cl_smem);
    cg::cluster_group cluster = cg::this_cluster();
    const int G = (int)cluster.num_blocks(), rank = (int)cluster.block_rank();
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    if (*(volatile int*)info != 0) return;  // the same for the whole cluster
    const int m = (int)(n - k0);             // rows of the panel; rows are numbered from k0 here
    const int base = rank * kClThreads, row = base + tid;
    const long long limit = (long long)(limit_ns < 1ull << 61 ? limit_ns * 2u : 1ull << 62);
    if (tid == 0) {
        for (int q = 0; q < 2; ++q)
            asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"((uint32_t)__cvta_generic_to_shared(&sm.bar[q])));
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        sm.late = sm.stop[0] = sm.stop[1] = sm.ends = 0;
    }
    auto end_panel = [&](int par, int why) {  // by whole warps
        if (lane != 0) return;
        sm.stop[par] = why;
        for (int q = 0; q < G; ++q) atomicMax(&cluster.map_shared_rank(&sm, q)->ends, why);
    };
    T* const prow_mem = sm.P + tid * kClLd;
    if (A.cs == 1) {  // rows contiguous: lanes along the columns
        for (int r = warp; r < kClThreads; r += 8)
            for (int col = lane; col < kLuNB; col += 32)
                sm.P[r * kClLd + col] = base + r < m && col < nb ? A(k0 + base + r, k0 + col) : T(0);
    } else {
#pragma unroll 32
        for (int col = 0; col < kLuNB; ++col) prow_mem[col] = row < m && col < nb ? A(k0 + row, k0 + col) : T(0);
    }
    cluster.sync();  // every CTA runs before any writes to another's shared memory
    const unsigned bytes = (unsigned)(G * (kStrip * sizeof(T) + 16) + kStrip * sizeof(T));  // sent to a CTA per column
    unsigned turn = 0;                                                                     // columns so far
    int zero_at = 0;  // the zero pivot's column, on the thread that records it
    auto report_late = [&] {
        if (tid == 0 && sm.late && err && atomicCAS(err, 0, RC_ERR_TIMEOUT) == 0) atomicExch(err + 1, 501);
    };
    for (int j0 = 0; j0 < nb; j0 += kStrip) {
        const int w = nb - j0 < kStrip ? nb - j0 : kStrip;
        T a[kStrip];
        {
            const T* src = prow_mem + j0;
#pragma unroll
            for (int q = 0; q < kStrip; ++q) a[q] = src[q];
        }
        int jj = 0, ends = 0;
#pragma unroll 1
        for (; jj < w; ++jj, ++turn) {
            const int c = j0 + jj, par = turn & 1;
            if (tid == 0)
                asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(
                                 (uint32_t)__cvta_generic_to_shared(&sm.bar[par])),
                             "r"(bytes)
                             : "memory");
            // the CTA's candidate
            const unsigned long long bits = (unsigned long long)__double_as_longlong(fabs((double)a[0]));
            const bool valid = row >= c && row < m && bits <= 0x7ff0000000000000ull;  // not NaN
            unsigned hi = valid ? (unsigned)(bits >> 32) + 1u : 0u, lo = valid ? (unsigned)bits : 0u;
            int idx = valid ? row : INT_MAX;
            warp_best(hi, lo, idx);
            if (lane == 0) {
                sm.whi[par][warp] = hi;
                sm.wlo[par][warp] = lo;
                sm.widx[par][warp] = idx;
            }
            if (row == idx) {
#pragma unroll
                for (int q = 0; q < kStrip; ++q) sm.mine[par][warp][q] = a[q];
            }
            if (row == c) {
#pragma unroll
                for (int q = 0; q < kStrip; ++q) sm.top[par][q] = a[q];
            }
            __syncthreads();
            const int stop = sm.stop[par ^ 1];  // set in the column before, by any warp
            hi = lane < 8 ? sm.whi[par][lane] : 0u;
            lo = lane < 8 ? sm.wlo[par][lane] : 0u;
            idx = lane < 8 ? sm.widx[par][lane] : INT_MAX;
            if (stop != 0) break;
            warp_best(hi, lo, idx);
            const int from_warp = idx == INT_MAX ? 0 : (idx - base) >> 5;
            {  // thread (dest, e) sends element e to CTA dest
                const int dest = tid / kStrip, e = tid % kStrip;
                if (dest < G) {
                    const uint32_t bar = peer_address(&sm.bar[par], dest);
                    send(peer_address(&sm.cand_row[par][rank][e], dest), sm.mine[par][from_warp][e], bar);
                    if (rank == 0) send(peer_address(&sm.crow[par][e], dest), sm.top[par][e], bar);
                    if (e == 0) send(peer_address(&sm.cand_key[par][rank][0], dest), (uint64_t)hi << 32 | lo, bar);
                    if (e == 1) send(peer_address(&sm.cand_key[par][rank][1], dest), (uint64_t)idx, bar);
                }
            }
            const int waited = wait_phase(&sm.bar[par], turn >> 1 & 1, limit);
            if (waited != 0) sm.late = 1;
            if (__any_sync(0xffffffffu, waited == 2)) {  // what was sent is not read
                ends = kGaveUp;
                break;
            }
            hi = lane < G ? (unsigned)(sm.cand_key[par][lane][0] >> 32) : 0u;
            lo = lane < G ? (unsigned)sm.cand_key[par][lane][0] : 0u;
            idx = lane < G ? (int)sm.cand_key[par][lane][1] : INT_MAX;
            warp_best(hi, lo, idx);
            const int p = idx == INT_MAX ? c : idx;  // nothing but NaN: the row itself
            const T* pr = idx == INT_MAX ? sm.crow[par] : sm.cand_row[par][p / kClThreads];
            const double pv = (double)pr[0];
            if (pv == 0.0) {  // also all-zero columns: the first row is the pivot, value 0
                if (rank == 0 && tid == 0) {
                    piv[k0 + c] = (int)(k0 + c);
                    zero_at = (int)(k0 + c + 1);
                }
                ends = kZeroPivot;
                break;
            }
            if (tid == 0) {
                sm.pivots[jj] = p;
                if (rank == 0) piv[k0 + c] = (int)(k0 + p);
            }
            if (row == p || row == c) {
                const T* from = row == p ? sm.crow[par] : pr;
#pragma unroll
                for (int q = 0; q < kStrip; ++q) a[q] = from[q];
            }
            T l = a[0];
            if (row > c) {
                l = (T)((double)a[0] / pv);
#pragma unroll
                for (int q = 1; q < kStrip; ++q) a[q] -= l * pr[q];
            }
            // column c is final but for the strip's later swaps; the next one moves to a[0]
            prow_mem[c] = l;
#pragma unroll
            for (int q = 0; q + 1 < kStrip; ++q) a[q] = a[q + 1];
            // (columns past the strip's width rotate in: never a[0], their updates unused)
            if (row == c) {  // U's row right of the diagonal, kept as the rotation leaves it
#pragma unroll
                for (int q = 0; q + 1 < kStrip; ++q)
                    if (jj + 1 + q < w) prow_mem[c + 1 + q] = a[q];
            }
        }
        if (ends != 0) {
            end_panel(turn & 1, ends);
            if (jj + 1 < w) __syncthreads();  // the other warps' next column, where they look at stop
        }
        cluster.sync();  // P's strip and the pivots are final everywhere
        if (sm.ends != 0) {  // the same in every CTA
            if (sm.ends == kGaveUp) {  // the messages that are under way arrive while their CTA is there
                for (const long long t0 = clock64(); clock64() - t0 < kClDrain;) {}
                zero_at = rank == 0 && tid == 0 ? (int)(k0 + 1) : 0;  // stops the later kernels: piv is not whole
            }
            if (zero_at != 0) record_first(info, zero_at);
            report_late();
            return;
        }
        // The swaps of the other columns, and of the strip's own columns by the later pivots
        // (entries right of a row's diagonal were swapped in registers): destination rows are
        // j0 .. j0 + w and the pivots beyond them; each traces its content back through the swaps.
        {
            int pv[kStrip];
#pragma unroll
            for (int i = 0; i < kStrip; ++i) pv[i] = i < w ? sm.pivots[i] : -1;
            for (int e = tid; e < 2 * kStrip * kStrip; e += kClThreads) {
                const int d = e % (2 * kStrip), j = e / (2 * kStrip);
                int r = d < w ? j0 + d : -1;
                if (d >= kStrip) {
                    r = d - kStrip < w ? sm.pivots[d - kStrip] : -1;
                    if (r < j0 + w) r = -1;
#pragma unroll
                    for (int i = 0; i < kStrip; ++i)
                        if (i < d - kStrip && pv[i] == r) r = -1;
                }
                int from = r, from_j = r;
#pragma unroll
                for (int i = kStrip - 1; i >= 0; --i) {
                    if (i == j) from_j = from;  // column j takes the swaps after its own
                    if (i < w) from = from == j0 + i ? pv[i] : from == pv[i] ? j0 + i : from;
                }
                sm.from_strip[d][j] = r >= j0 && r < j0 + j ? r : from_j;  // U's rows are final
                if (j == 0) {
                    sm.from_all[d] = from;
                    sm.dest[d] = r;
                }
            }
        }
        __syncthreads();
        T moved[4][2];
        int dst[4];
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            const int d = warp + 8 * q, r = sm.dest[d];
            dst[q] = r >= 0 && r / kClThreads == rank ? r : -1;
            if (dst[q] < 0) continue;
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const int col = lane + 32 * h;
                const int from = col >= j0 && col < j0 + w ? sm.from_strip[d][col - j0] : sm.from_all[d];
                const ClusterSmem<T>* peer = cluster.map_shared_rank(&sm, from / kClThreads);
                moved[q][h] = peer->P[(from % kClThreads) * kClLd + col];
            }
        }
        cluster.sync();  // all gathered
#pragma unroll
        for (int q = 0; q < 4; ++q)
            if (dst[q] >= 0)
#pragma unroll
                for (int h = 0; h < 2; ++h) sm.P[(dst[q] - base) * kClLd + lane + 32 * h] = moved[q][h];
        __syncthreads();
        const int j1 = j0 + w, right = nb - j1;
        if (right <= 0) break;
        // U(strip, right) = inv(L11) A(strip, right), a thread per column
        if (rank == 0 && tid < right) {
            T u[kStrip];
            T* col = sm.P + j0 * kClLd + j1 + tid;
            const T* l11 = sm.P + j0 * kClLd + j0;
#pragma unroll
            for (int i = 0; i < kStrip; ++i) u[i] = col[i * kClLd];
#pragma unroll
            for (int k = 0; k < kStrip; ++k)
#pragma unroll
                for (int i = k + 1; i < kStrip; ++i) u[i] -= l11[i * kClLd + k] * u[k];
#pragma unroll
            for (int i = 0; i < kStrip; ++i) col[i * kClLd] = sm.U[i][tid] = u[i];
        }
        cluster.sync();
        if (rank != 0) {
            const ClusterSmem<T>* first = cluster.map_shared_rank(&sm, 0);
            for (int e = tid; e < kStrip * right; e += kClThreads) sm.U[e / right][e % right] = first->U[e / right][e % right];
            __syncthreads();
        }
        // P(:, right) -= L(:, strip) U on the rows below the strip: 16 x 8 tiles
        const int g = lane >> 2, t = lane & 3;
        for (int ti = warp; ti < kClThreads / 16; ti += 8) {
            if (base + 16 * ti < j1) continue;
            const T* l0 = sm.P + (16 * ti + g) * kClLd + j0 + t;
            double lf[4][2];
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                lf[k][0] = (double)l0[4 * k];
                lf[k][1] = (double)l0[8 * kClLd + 4 * k];
            }
            for (int tj = 0; tj < right; tj += 8) {
                double d[4] = {};
#pragma unroll
                for (int k = 0; k < 4; ++k) dmma_16x8x4(d, lf[k][0], lf[k][1], (double)sm.U[4 * k + t][tj + g]);
                T* x = sm.P + (16 * ti + g) * kClLd + j1 + tj + 2 * t;
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    T& v = x[(e >> 1) * 8 * kClLd + (e & 1)];
                    if (tj + 2 * t + (e & 1) < right) v = (T)((double)v - d[e]);
                }
            }
        }
        __syncthreads();
    }
    cluster.sync();  // no CTA leaves while its shared memory may be read
    report_late();
    if (A.cs == 1) {
        for (int r = warp; r < kClThreads; r += 8)
            for (int col = lane; col < nb; col += 32)
                if (base + r < m) A(k0 + base + r, k0 + col) = sm.P[r * kClLd + col];
    } else if (row < m) {
#pragma unroll 32
        for (int col = 0; col < kLuNB; ++col)
            if (col < nb) A(k0 + row, k0 + col) = prow_mem[col];
    }
    if (rank != 0 || m == nb) return;  // nothing right of the last panel
    // inv(L11), unit lower (the identity beyond nb), for U12 = inv(L11) A12 right of the panel:
    // 16-blocks by a warp each, then merges (diag.cuh)
#pragma unroll 8
    for (int e = tid; e < kLuNB * kLuNB; e += kClThreads) {
        const int i = e / kLuNB, j = e % kLuNB;
        if (j <= i) sm.L[i * kClLd + j] = i == j ? 1.0 : i < nb ? (double)sm.P[i * kClLd + j] : 0.0;
    }
    if (tid < kLuNB) sm.rd[tid] = 1.0;
    __syncthreads();
    if (warp < 4) {
        const int c0 = kDB * warp;
        double* Lt = sm.Lt[warp];
        if (lane < kDB)
#pragma unroll
            for (int p = 0; p < kDB; ++p) Lt[p * kLTD + lane] = sm.L[(c0 + lane) * kClLd + c0 + p];
        __syncwarp();
        double x[kDB];
#pragma unroll
        for (int q = 0; q < kDB; ++q) x[q] = q == lane ? 1.0 : 0.0;
        solve_sub_block(x, sm.rd, Lt, [](int) {});
        if (lane < kDB)
#pragma unroll
            for (int q = 0; q < kDB; ++q)
                if (q >= lane) sm.L[(c0 + lane) * kClLd + c0 + q] = x[q];
    }
    __syncthreads();
    if (warp < 4) merge_t<16, kClLd>(sm.L, sm.T16[warp >> 1], 32 * (warp >> 1), warp & 1, lane);
    __syncthreads();
    if (warp < 4) merge_x<16, kClLd>(sm.L, sm.T16[warp >> 1], 32 * (warp >> 1), 0, 8 * (warp & 1), lane);
    __syncthreads();
    merge_t<32, kClLd>(sm.L, sm.T32, 0, warp, lane);
    __syncthreads();
    merge_x<32, kClLd>(sm.L, sm.T32, 0, 16 * (warp & 1), 8 * (warp >> 1), lane);
    __syncthreads();
#pragma unroll 8
    for (int e = tid; e < kLuNB * kLuNB; e += kClThreads) {  // (only used when nb == kLuNB)
        const int i = e / kLuNB, j = e % kLuNB;
        linv[e] = i >= j ? (T)sm.L[j * kClLd + i] : T(0);
    }
}

// The row swaps piv[k0 .. k0 + nb) on the columns outside the panel, 32 columns a CTA. The rows
// they touch (the panel's nb and the pivots beyond them) trace their content back through the
// swaps, a thread per row; then all of it is gathered into shared memory and written back.
// 64 swaps on 1984 columns of a column-major matrix: 14 us (49 with a thread per column that makes
// them one after the other).
constexpr int kSwapCols = 32;
template <class T>
__global__ void __launch_bounds__(256) lu_swap_kernel(int64_t n, View<T> A, int64_t k0, int nb, const int* piv,
                                                      const int* info) {
    __shared__ int64_t src[2 * kLuNB], dst[2 * kLuNB];
    __shared__ int64_t p[kLuNB];
    __shared__ T tile[2 * kLuNB][kSwapCols + 1];
    if (*(volatile const int*)info != 0) return;
    const int tid = threadIdx.x;
    if (tid < nb) p[tid] = piv[k0 + tid];
    __syncthreads();
    if (tid < 2 * kLuNB) {
        int64_t r = -1;
        if (tid < nb) r = k0 + tid;
        else if (tid >= kLuNB && tid - kLuNB < nb) {
            r = p[tid - kLuNB];
            if (r < k0 + nb) r = -1;
#pragma unroll 16
            for (int i = 0; i < kLuNB; ++i)
                if (i < tid - kLuNB && p[i] == r) r = -1;
        }
        int64_t from = r;
#pragma unroll 16
        for (int i = kLuNB - 1; i >= 0; --i)
            if (i < nb) from = from == k0 + i ? p[i] : from == p[i] ? k0 + i : from;
        dst[tid] = from == r ? -1 : r;  // rows that keep their content are left alone
        src[tid] = from;
    }
    __syncthreads();
    const int64_t cols = n - nb;
    const bool along_rows = A.cs == 1;  // a row's columns are contiguous
    for (int64_t cb = (int64_t)blockIdx.x * kSwapCols; cb < cols; cb += (int64_t)gridDim.x * kSwapCols) {
        auto each = [&](auto body) {
#pragma unroll 4
            for (int e = tid; e < 2 * kLuNB * kSwapCols; e += 256) {
                const int d = along_rows ? e / kSwapCols : e % (2 * kLuNB);
                const int c = along_rows ? e % kSwapCols : e / (2 * kLuNB);
                if (dst[d] >= 0 && cb + c < cols) body(d, c, cb + c < k0 ? cb + c : cb + c + nb);
            }
        };
        each([&](int d, int c, int64_t col) { tile[d][c] = A(src[d], col); });
        __syncthreads();
        each([&](int d, int c, int64_t col) { A(dst[d], col) = tile[d][c]; });
        __syncthreads();
    }
}

// eps = n^2 epsilon(T) max(A(0, 0), max_i |A(i, i)|); piv = identity; rank = n; stop = 0.
template <class T>
__global__ void pstrf_init_kernel(int64_t n, View<const T> A, double* eps, int* piv, int* rank, int* stop) {
    __shared__ double sv[32];
    __shared__ int64_t si[32];
    double mx = -DBL_MAX;
    int64_t dummy = 0;
    for (int64_t i = threadIdx.x; i < n; i += blockDim.x) {
        mx = fmax(mx, i == 0 ? (double)A(0, 0) : fabs((double)A(i, i)));
        piv[i] = (int)i;
    }
    block_argmax(mx, dummy, sv, si);
    if (threadIdx.x == 0) {
        const double e = sizeof(T) == 8 ? DBL_EPSILON : (double)FLT_EPSILON;
        *eps = (double)(n * n) * e * mx;
        *rank = (int)n;
        *stop = 0;
    }
}

template <class T>
__global__ void __launch_bounds__(kLuThreads) pstrf_block_kernel(int64_t n, View<T> A, int64_t k, int cur, T* pv,
                                                                 const double* eps, int* piv, int* rank,
                                                                 int* stop) {
    __shared__ double sv[32];
    __shared__ int64_t si[32];
    if (*(volatile int*)stop != 0) return;
    const double epsv = *eps;
    for (int j = 0; j < cur; ++j) {
        const int64_t c = k + j;
        for (int64_t i = c + threadIdx.x; i < n; i += blockDim.x) {
            if (j == 0) pv[i] = A(i, i);
            else pv[i] -= A(i, c - 1) * A(i, c - 1);
        }
        __syncthreads();
        double best = -DBL_MAX;
        int64_t bi = INT64_MAX;
        for (int64_t i = c + threadIdx.x; i < n; i += blockDim.x)
            if ((double)pv[i] > best) {
                best = (double)pv[i];
                bi = i;
            }
        block_argmax(best, bi, sv, si);
        const int64_t p = bi;
        if (p != c) {
            if (threadIdx.x == 0) piv[c] = (int)p;
            for (int64_t t = threadIdx.x; t < n; t += blockDim.x) {
                const T x = A(c, t);
                A(c, t) = A(p, t);
                A(p, t) = x;
            }
            __syncthreads();
            for (int64_t t = threadIdx.x; t < n; t += blockDim.x) {
                const T x = A(t, c);
                A(t, c) = A(t, p);
                A(t, p) = x;
            }
            if (threadIdx.x == 0) {
                const T x = pv[c];
                pv[c] = pv[p];
                pv[p] = x;
            }
            __syncthreads();
        }
        const T v = pv[c];
        if ((double)v < epsv) {
            const int64_t m = n - c;
            for (int64_t e = threadIdx.x; e < m * m; e += blockDim.x) A(c + e % m, c + e / m) = T(0);
            if (threadIdx.x == 0) {
                *rank = (int)c;
                *stop = 1;
            }
            return;
        }
        const T d = sqrt(v);
        // Row c's block columns in shared memory; each row's block entries loaded 8 at a time
        // (independent loads in flight), the dot product accumulated in the same order.
        __shared__ T rowc[kPsNB];
        if (threadIdx.x < j) rowc[threadIdx.x] = A(c, k + threadIdx.x);
        __syncthreads();
        for (int64_t i = c + 1 + threadIdx.x; i < n; i += blockDim.x) {
            T s = A(i, c);
            for (int t0 = 0; t0 < j; t0 += 8) {
                T a[8];
#pragma unroll
                for (int u = 0; u < 8; ++u) a[u] = t0 + u < j ? A(i, k + t0 + u) : T(0);
#pragma unroll
                for (int u = 0; u < 8; ++u)
                    if (t0 + u < j) s -= a[u] * rowc[t0 + u];
            }
            A(i, c) = s / d;
        }
        __syncthreads();
        if (threadIdx.x == 0) A(c, c) = d;
        for (int64_t t = c + 1 + threadIdx.x; t < n; t += blockDim.x) A(c, t) = T(0);
        __syncthreads();
    }
}

template <class T>
View<T> view_of(int row_major, T* A, int64_t lda) {
    return row_major ? View<T>{A, lda, 1} : View<T>{A, 1, lda};
}

template <class T>
void cluster_config(int G, cudaLaunchConfig_t* cfg, cudaLaunchAttribute* attr) {
    attr->id = cudaLaunchAttributeClusterDimension;
    attr->val.clusterDim.x = (unsigned)G;
    attr->val.clusterDim.y = attr->val.clusterDim.z = 1;
    cfg->gridDim = dim3((unsigned)G);
    cfg->blockDim = dim3(kClThreads);
    cfg->dynamicSmemBytes = sizeof(ClusterSmem<T>);
    cfg->attrs = attr;
    cfg->numAttrs = 1;
}

// CTAs of the cluster that holds a panel of `rows` rows, 0 where none does: more than 4096 rows,
// or a device that cannot run such a cluster. The kernel's attributes on the device are set with the
// question.
template <class T>
int cluster_size(int64_t rows) {
    static PerDevice<5> fits;  // by the cluster's size, 1 to 16
    int g = 1, lg = 0, dev = 0;
    for (; g < kClMax && (int64_t)g * kClThreads < rows; g *= 2) ++lg;
    if ((int64_t)g * kClThreads < rows || cudaGetDevice(&dev) != cudaSuccess) return 0;
    const bool fit = fits.get(dev, lg, [&] {
        cudaLaunchConfig_t cfg = {};
        cudaLaunchAttribute attr;
        cluster_config<T>(g, &cfg, &attr);
        int num = 0;
        auto kernel = getrf_panel_cluster_kernel<T>;
        const bool ok = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                             (int)sizeof(ClusterSmem<T>)) == cudaSuccess &&
                        cudaFuncSetAttribute(kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) == cudaSuccess &&
                        cudaOccupancyMaxActiveClusters(&num, kernel, &cfg) == cudaSuccess && num > 0;
        if (!ok) cudaGetLastError();
        return ok;
    });
    return fit ? g : 0;
}

// The panel on a cooperative grid of about 256 rows per CTA (a grid barrier costs more the
// more CTAs meet at it, the column work per CTA grows with its rows), at most one CTA per
// SM; on one CTA when the panel's rows do not fit the grid's shared memory (n above ~56K).
constexpr int kCoopRows = 256;
// linv (device, nb x nb): receives inv(L11) when the cooperative form ran (*have_inv).
template <class T>
int getrf_panel(int64_t n, View<T> A, int64_t k0, int nb, int* piv, int* info, T* linv, bool* have_inv,
                cudaStream_t s) {
    *have_inv = false;
    const int64_t rows = n - k0;
    const int sms = sm_count();
    int G = (int)((rows + kCoopRows - 1) / kCoopRows);
    if (G > sms) G = sms;
    const int cl = cluster_size<T>(rows);
    if (cl > 0) {
        cudaLaunchConfig_t cfg = {};
        cudaLaunchAttribute attr;
        cluster_config<T>(cl, &cfg, &attr);
        cfg.stream = s;
        if (cudaLaunchKernelEx(&cfg, getrf_panel_cluster_kernel<T>, n, A, k0, nb, piv, info, linv, error_word(),
                               wait_limit_ns()) != cudaSuccess) {
            cudaGetLastError();
            return RC_ERR_CUDA;
        }
        RC_TRY(check_launch());
        *have_inv = true;
        return RC_SUCCESS;
    }
    const int chunk = (int)((rows + G - 1) / G);
    if (chunk > kCoopMaxChunk || sms <= 0) {
        getrf_panel_kernel<T><<<1, kLuThreads, 0, s>>>(n, A, k0, nb, piv, info);
        return check_launch();
    }
    const size_t panel_bytes = ((size_t)chunk * (nb + 1) * sizeof(T) + 7) / 8 * 8;
    const size_t smem = panel_bytes + (kLuNB + 32) * sizeof(double) + 32 * sizeof(int64_t) + 16;
    const size_t n_cand = (size_t)kLuNB * sms;
    const size_t bytes = 256 + n_cand * (sizeof(double) + sizeof(int64_t)) + n_cand * kLuNB * sizeof(double) +
                         (size_t)kLuNB * kLuNB * sizeof(double);
    char* ws = static_cast<char*>(workspace(s, bytes, 14));
    if (!ws) return RC_ERR_ALLOC;
    unsigned* bar = reinterpret_cast<unsigned*>(ws);
    CoopScratch sc;
    sc.cand_v = reinterpret_cast<double*>(ws + 256);
    sc.cand_i = reinterpret_cast<int64_t*>(sc.cand_v + n_cand);
    sc.cand_row = reinterpret_cast<double*>(sc.cand_i + n_cand);
    sc.crow = sc.cand_row + n_cand * kLuNB;
    if (cudaMemsetAsync(bar, 0, 2 * sizeof(unsigned), s) != cudaSuccess) return RC_ERR_CUDA;
    if (cudaFuncSetAttribute(getrf_panel_coop_kernel<T>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) !=
        cudaSuccess)
        return RC_ERR_CUDA;
    int* err = error_word();
    uint64_t lim = wait_limit_ns();
    void* args[] = {&n, &A, &k0, &nb, const_cast<int*>(&chunk), &piv, &info, &sc, &bar, &err, &lim, &linv};
    if (cudaLaunchCooperativeKernel((const void*)getrf_panel_coop_kernel<T>, dim3((unsigned)G), dim3(kCoopThreads),
                                    args, smem, s) != cudaSuccess) {
        cudaGetLastError();
        return RC_ERR_CUDA;
    }
    count_launch();
    *have_inv = true;
    return RC_SUCCESS;
}

template <class T>
int getrf(int row_major, int64_t n, T* Ap, int64_t lda, int* piv, int* info, cudaStream_t s) {
    if (cudaMemsetAsync(info, 0, sizeof(int), s) != cudaSuccess) return RC_ERR_CUDA;
    const View<T> A = view_of(row_major, Ap, lda);
    T* linv = static_cast<T*>(workspace(s, (size_t)kLuNB * kLuNB * sizeof(T), 16));
    if (!linv) return RC_ERR_ALLOC;
    for (int64_t k0 = 0; k0 < n; k0 += kLuNB) {
        const int nb = (int)(n - k0 < kLuNB ? n - k0 : kLuNB);
        bool have_inv = false;
        RC_TRY(getrf_panel<T>(n, A, k0, nb, piv, info, linv, &have_inv, s));
        if (n > nb) {
            const int64_t cols = n - nb;
            const unsigned grid = ceil_div(cols, kSwapCols) < 4096u ? ceil_div(cols, kSwapCols) : 4096u;
            lu_swap_kernel<T><<<grid, 256, 0, s>>>(n, A, k0, nb, piv, info);
            RC_TRY(check_launch());
        }
        const int64_t r = n - k0 - nb;
        if (r <= 0) continue;
        if (have_inv) {  // U12 = inv(L11) A12, in place (the GEMM's single row tile reads all of A12's k range first)
            const View<T> A12 = A.sub(k0, k0 + nb);
            RC_TRY(gemm<T>(nb, r, nb, T(1), View<const T>{linv, kLuNB, 1}, View<const T>{A12.p, A12.rs, A12.cs},
                           T(0), A12, kFull, 0, s, info));
        } else {
            const View<const T> L11{A.sub(k0, k0).p, A.rs, A.cs};
            RC_TRY(trsm_left<T>(false, true, nb, r, T(1), L11, A.sub(k0, k0 + nb), nullptr, s, info));
        }
        const View<const T> L21{A.sub(k0 + nb, k0).p, A.rs, A.cs}, U12{A.sub(k0, k0 + nb).p, A.rs, A.cs};
        RC_TRY(gemm<T>(r, r, nb, T(-1), L21, U12, T(1), A.sub(k0 + nb, k0 + nb), kFull, 0, s, info));
    }
    return RC_SUCCESS;
}

template <class T>
int pstrf(int row_major, int64_t n, T* Ap, int64_t lda, int* piv, int* rank, cudaStream_t s) {
    const size_t bytes = ((size_t)n * sizeof(T) + 255) / 256 * 256 + 256;
    char* ws = static_cast<char*>(workspace(s, bytes, 12));
    if (!ws) return RC_ERR_ALLOC;
    T* pv = reinterpret_cast<T*>(ws);
    double* eps = reinterpret_cast<double*>(ws + bytes - 256);
    int* stop = reinterpret_cast<int*>(ws + bytes - 128);
    const View<T> A = view_of(row_major, Ap, lda);
    pstrf_init_kernel<T><<<1, kLuThreads, 0, s>>>(n, View<const T>{A.p, A.rs, A.cs}, eps, piv, rank, stop);
    RC_TRY(check_launch());
    for (int64_t k = 0; k < n; k += kPsNB) {
        const int cur = (int)(n - k < kPsNB ? n - k : kPsNB);
        pstrf_block_kernel<T><<<1, kLuThreads, 0, s>>>(n, A, k, cur, pv, eps, piv, rank, stop);
        RC_TRY(check_launch());
        const int64_t r = n - k - cur;
        if (r <= 0) continue;
        const View<const T> L21{A.sub(k + cur, k).p, A.rs, A.cs};
        RC_TRY(gemm<T>(r, r, cur, T(-1), L21, L21.t(), T(1), A.sub(k + cur, k + cur), kFull, 0, s, stop));
    }
    return RC_SUCCESS;
}

}  // namespace
}  // namespace rc

extern "C" {

int rc_getrf_f64(int row_major, size_t n, double* A, size_t lda, int* piv, int* info, void* stream) {
    if (!info) return RC_ERR_INVALID_ARGUMENT;
    if (n == 0) return cudaMemsetAsync(info, 0, sizeof(int), static_cast<cudaStream_t>(stream)) == cudaSuccess
                           ? RC_SUCCESS
                           : RC_ERR_CUDA;
    if (!A || !piv || lda < n) return RC_ERR_INVALID_ARGUMENT;
    if (n > (size_t)INT32_MAX) return RC_ERR_NOT_SUPPORTED;
    return rc::getrf<double>(row_major, (int64_t)n, A, (int64_t)lda, piv, info, static_cast<cudaStream_t>(stream));
}

int rc_getrf_f32(int row_major, size_t n, float* A, size_t lda, int* piv, int* info, void* stream) {
    if (!info) return RC_ERR_INVALID_ARGUMENT;
    if (n == 0) return cudaMemsetAsync(info, 0, sizeof(int), static_cast<cudaStream_t>(stream)) == cudaSuccess
                           ? RC_SUCCESS
                           : RC_ERR_CUDA;
    if (!A || !piv || lda < n) return RC_ERR_INVALID_ARGUMENT;
    if (n > (size_t)INT32_MAX) return RC_ERR_NOT_SUPPORTED;
    return rc::getrf<float>(row_major, (int64_t)n, A, (int64_t)lda, piv, info, static_cast<cudaStream_t>(stream));
}

int rc_pstrf_f64(int row_major, size_t n, double* A, size_t lda, int* piv, int* rank, void* stream) {
    if (!rank) return RC_ERR_INVALID_ARGUMENT;
    if (n == 0) return cudaMemsetAsync(rank, 0, sizeof(int), static_cast<cudaStream_t>(stream)) == cudaSuccess
                           ? RC_SUCCESS
                           : RC_ERR_CUDA;
    if (!A || !piv || lda < n) return RC_ERR_INVALID_ARGUMENT;
    if (n > (size_t)INT32_MAX) return RC_ERR_NOT_SUPPORTED;
    return rc::pstrf<double>(row_major, (int64_t)n, A, (int64_t)lda, piv, rank, static_cast<cudaStream_t>(stream));
}

int rc_pstrf_f32(int row_major, size_t n, float* A, size_t lda, int* piv, int* rank, void* stream) {
    if (!rank) return RC_ERR_INVALID_ARGUMENT;
    if (n == 0) return cudaMemsetAsync(rank, 0, sizeof(int), static_cast<cudaStream_t>(stream)) == cudaSuccess
                           ? RC_SUCCESS
                           : RC_ERR_CUDA;
    if (!A || !piv || lda < n) return RC_ERR_INVALID_ARGUMENT;
    if (n > (size_t)INT32_MAX) return RC_ERR_NOT_SUPPORTED;
    return rc::pstrf<float>(row_major, (int64_t)n, A, (int64_t)lda, piv, rank, static_cast<cudaStream_t>(stream));
}

}  // extern "C"
