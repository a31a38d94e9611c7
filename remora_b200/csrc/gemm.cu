// Dense GEMM / SYRK for Remora's cuda_tag.
//
// Replaces the reference's cuBLAS calls behind kernels::gemm and kernels::syrk
// (include/remora/hip/cublas_backend.hpp:121-166, :389-431, called from
// include/remora/kernels/hip/gemm.hpp:46-112 and kernels/hip/syrk.hpp:44-85).
//
// Two kernels:
//  * gemm_dmma_f64: the FP64 tensor-core path (DMMA, mma.sync m16n8k4 f64), a family of
//    CTA tiles from 128 x 128 down to 32 x 32 over one kernel template. Operand tiles are
//    staged by 16-byte cp.async (8-byte where the alignment asks for it) in the order of
//    their global layout, so all four transpose combinations run at the same rate.
//  * sgemm_simt: FP32 on the FMA units, register tiles of packed pairs.
// Both honour a triangle mask (SYRK writes one triangle; whole tiles outside it exit at
// once) and an abort word (a failed Cholesky pivot stops the trailing updates).
#include "gemm.cuh"
#include "gemm_plan.cuh"
#include "tc_gemm.cuh"
#include <cmath>
#include <type_traits>

namespace rc {
namespace {

__device__ __forceinline__ bool aborted(const int* abort) { return abort != nullptr && *(volatile const int*)abort != 0; }

__device__ __forceinline__ bool tile_outside(Mask mask, int64_t off, int64_t m0, int64_t n0, int bm, int bn) {
    if (mask == kLower) return (m0 + bm - 1) - n0 - off < 0;
    if (mask == kUpper) return m0 - (n0 + bn - 1) - off > 0;
    return false;
}

__device__ __forceinline__ bool in_mask(Mask mask, int64_t off, int64_t i, int64_t j) {
    if (mask == kLower) return i - j >= off;
    if (mask == kUpper) return i - j <= off;
    return true;
}

// First row and column of this CTA's BM x BN tile of an m x n product, all tiles along grid.x (the
// other extents end at 65535, too few for the row tiles of a tall product). Grouped order:
// consecutive CTAs take a group of row tiles (1024 rows) of one column tile before the next
// column tile, so that a wave holds a few A row blocks and B column blocks in L2 instead of
// streaming all of B once per row of tiles.
template <int BM, int BN>
__device__ __forceinline__ void tile_origin(int64_t m, int64_t n, int64_t* m0, int64_t* n0) {
    constexpr int64_t kGroupM = 1024 / BM;
    const int64_t rows = (m + BM - 1) / BM, per = kGroupM * ((n + BN - 1) / BN), lin = blockIdx.x;
    const int64_t first = lin / per * kGroupM, rest = rows - first;
    const int64_t gsz = rest < kGroupM ? rest : kGroupM, r = lin % per;
    *m0 = (first + r % gsz) * BM;
    *n0 = r / gsz * BN;
}

// ------------------------------------------------------------------------------------
// FP32 kernel on the FMA units (68.6 TFLOP/s measured on registers alone), exact FP32
// accumulation in ascending k. Operand tiles go through registers into shared memory as
// [k][m] and [k][n], two buffers, the next tile's loads in flight under the current one's
// products. A thread owns GM x GN groups of 4 x 4 elements of C, so that one 16-byte fragment
// load feeds 4 GN (4 GM) products; a warp is 4 (m) x 8 (n) threads, whose fragment loads cover
// 64 and 128 distinct bytes. Products are packed pairs along n (fma.rn.f32x2): half the issue
// slots, the rest of which hold the fragment loads.
template <int BM_, int BN_, int GM_, int GN_, int OCC_>
struct SimtTile {
    static constexpr int BM = BM_, BN = BN_, GM = GM_, GN = GN_, OCC = OCC_, BK = 16;
    static constexpr int WARPS_M = BM / (16 * GM), WARPS_N = BN / (32 * GN), THREADS = 32 * WARPS_M * WARPS_N;
    static constexpr int LDA = BM + 4, LDB = BN + 4;
};
// 128 x 64 with three CTAs of 4 warps per SM: 4096^3 in 2.65 ms (52 TFLOP/s; the 64 x 64 tile
// of one 4 x 4 group a thread and one barrier-bound buffer took 6.2), 1024^3 in 68 us (153). The
// variants 128 x 128 of 8 warps (2.59-2.75 ms, 115 us), of 4 warps (2.60-2.63, 115) and 64 x 64
// of 2 warps (2.75-2.80, 73) are no better on large products and worse on middle ones. Below
// about a tile per SM the 32 x 32 tile wins: 512^3 in 19 us (37 with 128 x 64).
using SimtL = SimtTile<128, 64, 2, 2, 3>;
using SimtS = SimtTile<32, 32, 1, 1, 12>;

// One thread's share of a 16-deep operand tile: groups of 4 elements along the contiguous
// direction (k when KM, else the row direction), zero outside rows x k. V16: 16-byte loads are
// aligned.
template <bool KM, int ROWS, int THREADS, bool V16>
struct SimtLoader {
    static constexpr int COUNT = ROWS * 16 / 4, PER = (COUNT + THREADS - 1) / THREADS;
    static constexpr int RUN = (KM ? 16 : ROWS) / 4;  // groups per contiguous run
    static __device__ __forceinline__ void load(float4 (&v)[PER], const float* p, int64_t ld, int64_t rows, int64_t k,
                                                int64_t r0, int64_t k0, int tid) {
        const bool inside = r0 + ROWS <= rows && k0 + 16 <= k;
#pragma unroll
        for (int e = 0; e < PER; ++e) {
            const int q = tid + e * THREADS, c = q % RUN * 4, o = q / RUN;
            const int row = KM ? o : c, kk = KM ? c : o;
            v[e] = make_float4(0.f, 0.f, 0.f, 0.f);
            if (COUNT % THREADS != 0 && q >= COUNT) continue;
            const float* src = KM ? p + (r0 + row) * ld + k0 + kk : p + r0 + row + (k0 + kk) * ld;
            if (V16 && inside) {
                v[e] = *reinterpret_cast<const float4*>(src);
            } else {
                const int64_t left = KM ? (r0 + row < rows ? k - (k0 + kk) : 0) : (k0 + kk < k ? rows - (r0 + row) : 0);
                if (left > 0) v[e].x = src[0];
                if (left > 1) v[e].y = src[1];
                if (left > 2) v[e].z = src[2];
                if (left > 3) v[e].w = src[3];
            }
        }
    }
    static __device__ __forceinline__ void store(const float4 (&v)[PER], float* dst, int ldt, int tid) {
#pragma unroll
        for (int e = 0; e < PER; ++e) {
            const int q = tid + e * THREADS, c = q % RUN * 4, o = q / RUN;
            if (COUNT % THREADS != 0 && q >= COUNT) continue;
            if (KM) {
                dst[c * ldt + o] = v[e].x;
                dst[(c + 1) * ldt + o] = v[e].y;
                dst[(c + 2) * ldt + o] = v[e].z;
                dst[(c + 3) * ldt + o] = v[e].w;
            } else {
                *reinterpret_cast<float4*>(dst + o * ldt + c) = v[e];
            }
        }
    }
};

__device__ __forceinline__ uint64_t pack2(float a, float b) {
    uint64_t r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
    return r;
}
__device__ __forceinline__ void fma2(uint64_t& d, uint64_t a, uint64_t b) {
    asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(d) : "l"(a), "l"(b));
}

template <bool A_KMAJOR, bool B_KMAJOR, class Tile, bool V16>
__global__ void __launch_bounds__(Tile::THREADS, Tile::OCC)
    sgemm_simt(int64_t m, int64_t n, int64_t k, float alpha, View<const float> A, View<const float> B, float beta,
               View<float> C, Mask mask, int64_t off, const int* abort) {
    constexpr int BM = Tile::BM, BN = Tile::BN, GM = Tile::GM, GN = Tile::GN, BK = Tile::BK;
    constexpr int LDA = Tile::LDA, LDB = Tile::LDB;
    using LA = SimtLoader<A_KMAJOR, BM, Tile::THREADS, V16>;
    using LB = SimtLoader<B_KMAJOR, BN, Tile::THREADS, V16>;
    __shared__ __align__(16) float sA[2][BK * LDA];
    __shared__ __align__(16) float sB[2][BK * LDB];
    int64_t m0, n0;
    tile_origin<BM, BN>(m, n, &m0, &n0);
    if (aborted(abort) || tile_outside(mask, off, m0, n0, BM, BN)) return;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int tm = (warp / Tile::WARPS_N) * 16 + (lane >> 3) * 4, tn = (warp % Tile::WARPS_N) * 32 + (lane & 7) * 4;
    const int64_t lda = A_KMAJOR ? A.rs : A.cs, ldb = B_KMAJOR ? B.cs : B.rs;
    uint64_t acc[GM * 4][GN * 2];
#pragma unroll
    for (int i = 0; i < GM * 4; ++i)
#pragma unroll
        for (int j = 0; j < GN * 2; ++j) acc[i][j] = 0;
    float4 va[LA::PER], vb[LB::PER];
    LA::load(va, A.p, lda, m, k, m0, 0, tid);
    LB::load(vb, B.p, ldb, n, k, n0, 0, tid);
    LA::store(va, sA[0], LDA, tid);
    LB::store(vb, sB[0], LDB, tid);
    __syncthreads();
    const int KT = (int)((k + BK - 1) / BK);
    for (int kt = 0; kt < KT; ++kt) {
        const bool more = kt + 1 < KT;
        if (more) {
            LA::load(va, A.p, lda, m, k, m0, (int64_t)(kt + 1) * BK, tid);
            LB::load(vb, B.p, ldb, n, k, n0, (int64_t)(kt + 1) * BK, tid);
        }
        const float *a_s = sA[kt & 1] + tm, *b_s = sB[kt & 1] + tn;
#pragma unroll
        for (int kk = 0; kk < BK; ++kk) {
            float4 a[GM];
            ulonglong2 b[GN];
#pragma unroll
            for (int q = 0; q < GM; ++q) a[q] = *reinterpret_cast<const float4*>(a_s + kk * LDA + q * (BM / GM));
#pragma unroll
            for (int q = 0; q < GN; ++q) b[q] = *reinterpret_cast<const ulonglong2*>(b_s + kk * LDB + q * (BN / GN));
#pragma unroll
            for (int q = 0; q < GM; ++q) {
                const float ai[4] = {a[q].x, a[q].y, a[q].z, a[q].w};
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    const uint64_t aa = pack2(ai[i], ai[i]);
#pragma unroll
                    for (int j = 0; j < GN; ++j) {
                        fma2(acc[4 * q + i][2 * j], aa, b[j].x);
                        fma2(acc[4 * q + i][2 * j + 1], aa, b[j].y);
                    }
                }
            }
        }
        if (more) {
            LA::store(va, sA[(kt + 1) & 1], LDA, tid);
            LB::store(vb, sB[(kt + 1) & 1], LDB, tid);
            __syncthreads();
        }
    }
    // Epilogue: 4 x 4 group by group; the old C of a group is fetched before any of it is
    // written; 16-byte accesses along C's contiguous direction where the group lies inside.
    const bool colC = C.rs == 1, vecC = (colC || C.cs == 1) && (colC ? C.cs : C.rs) % 4 == 0 &&
                                        reinterpret_cast<uintptr_t>(C.p) % 16 == 0;
    const int64_t ci = colC ? C.cs : C.rs;
#pragma unroll
    for (int gm = 0; gm < GM; ++gm)
#pragma unroll
        for (int gn = 0; gn < GN; ++gn) {
            const int64_t i0 = m0 + tm + gm * (BM / GM), j0 = n0 + tn + gn * (BN / GN);
            float v[4][4];
#pragma unroll
            for (int i = 0; i < 4; ++i)
#pragma unroll
                for (int j = 0; j < 2; ++j)
                    asm("mov.b64 {%0, %1}, %2;" : "=f"(v[i][2 * j]), "=f"(v[i][2 * j + 1]) : "l"(acc[4 * gm + i][2 * gn + j]));
            const bool inside = i0 + 4 <= m && j0 + 4 <= n &&
                                (mask == kFull || (mask == kLower ? i0 - (j0 + 3) >= off : (i0 + 3) - j0 <= off));
            if (vecC && inside) {
                float4* c4[4];
                float4 old[4];
#pragma unroll
                for (int q = 0; q < 4; ++q) {
                    c4[q] = reinterpret_cast<float4*>(C.p + (colC ? i0 + (j0 + q) * ci : (i0 + q) * ci + j0));
                    if (beta != 0.f) old[q] = *c4[q];
                }
#pragma unroll
                for (int q = 0; q < 4; ++q) {
                    float w[4];
#pragma unroll
                    for (int u = 0; u < 4; ++u) w[u] = alpha * (colC ? v[u][q] : v[q][u]);
                    if (beta != 0.f) {
                        w[0] = fmaf(beta, old[q].x, w[0]);
                        w[1] = fmaf(beta, old[q].y, w[1]);
                        w[2] = fmaf(beta, old[q].z, w[2]);
                        w[3] = fmaf(beta, old[q].w, w[3]);
                    }
                    *c4[q] = make_float4(w[0], w[1], w[2], w[3]);
                }
            } else {
                float old[4][4];
#pragma unroll
                for (int i = 0; i < 4; ++i)
#pragma unroll
                    for (int j = 0; j < 4; ++j)
                        old[i][j] = beta != 0.f && i0 + i < m && j0 + j < n && in_mask(mask, off, i0 + i, j0 + j)
                                        ? C(i0 + i, j0 + j) : 0.f;
#pragma unroll
                for (int i = 0; i < 4; ++i)
#pragma unroll
                    for (int j = 0; j < 4; ++j) {
                        if (i0 + i >= m || j0 + j >= n || !in_mask(mask, off, i0 + i, j0 + j)) continue;
                        float w = alpha * v[i][j];
                        if (beta != 0.f) w = fmaf(beta, old[i][j], w);
                        C(i0 + i, j0 + j) = w;
                    }
            }
        }
}

// ------------------------------------------------------------------------------------
// FP64 DMMA kernel. Tiles of BM x BN by a k-step of 16 staged through a cp.async ring, one
// warp tile of 16 MI x 8 NI per warp. The pipe does 64 FMA per SM and cycle (36.9 TFLOP/s
// measured on registers alone), so what a shape reaches depends on how evenly its tiles
// load the SMs and on what a tile spends outside its k loop; pick_tile (gemm_plan.cuh) weighs both.
// gridDim.z > 1 splits K: slice z covers [z * kchunk, (z + 1) * kchunk) and writes its
// partial product (alpha = 1, beta = 0) to Cz + z * zstride; a second kernel then reduces
// the slices into C.
constexpr int DKP = DK + 4;  // row stride of a K-major tile (doubles)

// Shared-memory tile of an operand with ROWS rows (the m or n direction), in the order of
// its global layout, so that 16-byte copies keep it: K-major tiles are [row][k] with rows
// of 20 doubles, the others [k][row] with rows of ROWS + 4 doubles. With either stride the
// 16 lanes of a half-warp's fragment load (4 rows x 4 k) hit 16 distinct bank pairs.
template <bool KM, int ROWS>
struct OpTile {
    static constexpr int SIZE = KM ? ROWS * DKP : DK * (ROWS + 4);
    static __device__ __forceinline__ int at(int row, int k) { return KM ? row * DKP + k : k * (ROWS + 4) + row; }
};

__device__ __forceinline__ void cp_async8(void* smem, const void* gmem, int bytes) {
    const unsigned s = (unsigned)__cvta_generic_to_shared(smem);
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;\n" ::"r"(s), "l"(gmem), "r"(bytes));
}
__device__ __forceinline__ void cp_async16(void* smem, const void* gmem, int bytes) {
    const unsigned s = (unsigned)__cvta_generic_to_shared(smem);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(s), "l"(gmem), "r"(bytes));
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::); }
template <int N>
__device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;\n" ::"n"(N)); }

__device__ __forceinline__ void dmma_16x8x4(double (&d)[4], double a0, double a1, double b0) {
    asm("mma.sync.aligned.m16n8k4.row.col.f64.f64.f64.f64 {%0,%1,%2,%3}, {%4,%5}, {%6}, {%0,%1,%2,%3};\n"
        : "+d"(d[0]), "+d"(d[1]), "+d"(d[2]), "+d"(d[3])
        : "d"(a0), "d"(a1), "d"(b0));
}

// Copy k-tile k0 of an operand (element (i, k) at p[i * ld + k] when KM, else p[i + k * ld])
// into its shared tile; zero outside rows x k. V16: base and ld allow 16-byte copies (rows
// r0 and k0 are even).
template <bool KM, int ROWS, int THREADS, bool V16>
__device__ __forceinline__ void load_operand(double* dst, const double* p, int64_t ld, int64_t rows, int64_t k,
                                             int64_t r0, int64_t k0, int tid) {
    constexpr int W = V16 ? 2 : 1;               // doubles per copy
    constexpr int PER_ROW = (KM ? DK : ROWS) / W;  // copies per contiguous run
    constexpr int COUNT = ROWS * DK / W;
    const bool inside = r0 + ROWS <= rows && k0 + DK <= k;
#pragma unroll
    for (int e0 = 0; e0 < COUNT; e0 += THREADS) {
        const int e = e0 + tid;
        if (COUNT % THREADS != 0 && e >= COUNT) break;
        const int c = (e % PER_ROW) * W, o = e / PER_ROW;  // along the run, across runs
        const int row = KM ? o : c, kk = KM ? c : o;
        int bytes = 8 * W;
        const double* src = KM ? p + (r0 + row) * ld + k0 + kk : p + r0 + row + (k0 + kk) * ld;
        if (!inside) {
            const int64_t left = KM ? (r0 + row < rows ? k - (k0 + kk) : 0) : (k0 + kk < k ? rows - (r0 + row) : 0);
            bytes = left >= W ? 8 * W : left > 0 ? 8 : 0;
            if (bytes == 0) src = p;
        }
        if (V16) cp_async16(dst + OpTile<KM, ROWS>::at(row, kk), src, bytes);
        else cp_async8(dst + OpTile<KM, ROWS>::at(row, kk), src, bytes);
    }
}

template <bool A_KMAJOR, bool B_KMAJOR, class Tile>
constexpr size_t dmma_smem() {
    return (size_t)Tile::STAGES * (OpTile<A_KMAJOR, Tile::BM>::SIZE + OpTile<B_KMAJOR, Tile::BN>::SIZE) * sizeof(double);
}

// A_KMAJOR: A(i, k) is contiguous along k (A.cs == 1), else along i (A.rs == 1).
// B_KMAJOR: B(k, j) is contiguous along k (B.rs == 1), else along j (B.cs == 1).
template <bool A_KMAJOR, bool B_KMAJOR, class Tile, bool V16>
__global__ void __launch_bounds__(Tile::THREADS, Tile::OCC)
    gemm_dmma_f64(int64_t m, int64_t n, int64_t k, double alpha, View<const double> A, View<const double> B,
                  double beta, View<double> C, Mask mask, int64_t off, const int* abort, int64_t kchunk,
                  int64_t zstride) {
    using TA = OpTile<A_KMAJOR, Tile::BM>;
    using TB = OpTile<B_KMAJOR, Tile::BN>;
    constexpr int BM = Tile::BM, BN = Tile::BN, MI = Tile::MI, NI = Tile::NI, ST = Tile::STAGES, T = Tile::THREADS;
    extern __shared__ __align__(16) double dsmem[];
    double* sA = dsmem;
    double* sB = dsmem + ST * TA::SIZE;
    int64_t m0, n0;
    tile_origin<BM, BN>(m, n, &m0, &n0);
    const bool tri = mask == kLowerTri;
    if (tri) mask = kLower;
    if (aborted(abort) || tile_outside(mask, off, m0, n0, BM, BN)) return;
    if (tri && m0 < k) {
        A = A.sub(0, m0);
        B = B.sub(m0, 0);
        k -= m0;
    }
    if (gridDim.z > 1) {  // K slice of a split-K product
        const int64_t kz = (int64_t)blockIdx.z * kchunk;
        A = A.sub(0, kz);
        B = B.sub(kz, 0);
        k = (k - kz) < kchunk ? k - kz : kchunk;
        C.p += (int64_t)blockIdx.z * zstride;
    }
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int g = lane >> 2, t = lane & 3;
    const int wm = (warp / Tile::WARPS_N) * Tile::WM, wn = (warp % Tile::WARPS_N) * Tile::WN;
    const int64_t lda = A_KMAJOR ? A.rs : A.cs, ldb = B_KMAJOR ? B.cs : B.rs;
    auto load = [&](int kt) {
        const int st = kt % ST;
        load_operand<A_KMAJOR, BM, T, V16>(sA + st * TA::SIZE, A.p, lda, m, k, m0, (int64_t)kt * DK, tid);
        load_operand<B_KMAJOR, BN, T, V16>(sB + st * TB::SIZE, B.p, ldb, n, k, n0, (int64_t)kt * DK, tid);
    };
    double acc[MI][NI][4];
#pragma unroll
    for (int a = 0; a < MI; ++a)
#pragma unroll
        for (int b = 0; b < NI; ++b)
#pragma unroll
            for (int c = 0; c < 4; ++c) acc[a][b][c] = 0.0;

    const int KT = (int)((k + DK - 1) / DK);
#pragma unroll
    for (int s = 0; s < ST - 1; ++s) {
        if (s < KT) load(s);
        cp_async_commit();
    }
    for (int kt = 0; kt < KT; ++kt) {
        cp_async_wait<ST - 2>();
        __syncthreads();
        if (kt + ST - 1 < KT) load(kt + ST - 1);
        cp_async_commit();
        const double* a_s = sA + (kt % ST) * TA::SIZE;
        const double* b_s = sB + (kt % ST) * TB::SIZE;
#pragma unroll
        for (int ks = 0; ks < DK; ks += 4) {
            double af[MI][2], bf[NI];
#pragma unroll
            for (int mi = 0; mi < MI; ++mi) {
                af[mi][0] = a_s[TA::at(wm + mi * 16 + g, ks + t)];
                af[mi][1] = a_s[TA::at(wm + mi * 16 + g + 8, ks + t)];
            }
#pragma unroll
            for (int ni = 0; ni < NI; ++ni) bf[ni] = b_s[TB::at(wn + ni * 8 + g, ks + t)];
#pragma unroll
            for (int mi = 0; mi < MI; ++mi)
#pragma unroll
                for (int ni = 0; ni < NI; ++ni) dmma_16x8x4(acc[mi][ni], af[mi][0], af[mi][1], bf[ni]);
        }
    }
    cp_async_wait<0>();
    // Epilogue: element (g, 2t + c) and (g + 8, 2t + c) of each 16x8 accumulator tile. The
    // old C of 16 rows is fetched before any of it is written, so that its loads are all in
    // flight at once.
#pragma unroll
    for (int mi = 0; mi < MI; ++mi) {
        double old[2][NI][2];
        if (beta != 0.0) {
#pragma unroll
            for (int h = 0; h < 2; ++h)
#pragma unroll
                for (int ni = 0; ni < NI; ++ni)
#pragma unroll
                    for (int c = 0; c < 2; ++c) {
                        const int64_t i = m0 + wm + mi * 16 + g + 8 * h, j = n0 + wn + ni * 8 + 2 * t + c;
                        old[h][ni][c] = i < m && j < n && in_mask(mask, off, i, j) ? C(i, j) : 0.0;
                    }
        }
#pragma unroll
        for (int h = 0; h < 2; ++h)
#pragma unroll
            for (int ni = 0; ni < NI; ++ni)
#pragma unroll
                for (int c = 0; c < 2; ++c) {
                    const int64_t i = m0 + wm + mi * 16 + g + 8 * h, j = n0 + wn + ni * 8 + 2 * t + c;
                    if (i >= m || j >= n || !in_mask(mask, off, i, j)) continue;
                    double v = alpha * acc[mi][ni][2 * h + c];
                    if (beta != 0.0) v = fma(beta, old[h][ni][c], v);
                    C(i, j) = v;
                }
    }
}

// C = alpha * sum_z P_z + beta * C over the split-K slices (column-major m x n, ld m each).
__global__ void splitk_reduce(int64_t m, int64_t n, int nz, const double* P, int64_t zstride, double alpha,
                              double beta, View<double> C) {
    for (int64_t j = blockIdx.y; j < n; j += gridDim.y)
        for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < m; i += (int64_t)gridDim.x * blockDim.x) {
            double acc = 0.0;
            for (int z = 0; z < nz; ++z) acc += P[z * zstride + i + j * m];
            double v = alpha * acc;
            if (beta != 0.0) v = fma(beta, C(i, j), v);
            C(i, j) = v;
        }
}

struct Shape : Problem {
    Mask mask;
    Shape(int64_t m_, int64_t n_, int64_t k_, Mask mask_) : Problem{m_, n_, k_, mask_ != kFull}, mask(mask_) {}
};

// The grid of a product's tiles (tile_origin); false where there are more than a grid holds.
template <class Tile>
bool tile_grid(const Shape& p, dim3* grid) {
    const int64_t tiles = ((p.m + Tile::BM - 1) / Tile::BM) * ((p.n + Tile::BN - 1) / Tile::BN);
    *grid = dim3((unsigned)tiles);
    return tiles <= INT32_MAX;
}

template <bool AK, bool BK, class Tile, bool V16>
int launch_dmma(const Shape& p, double alpha, View<const double> A, View<const double> B, double beta,
                View<double> C, int64_t off, int nz, cudaStream_t s, const int* abort) {
    constexpr size_t smem = dmma_smem<AK, BK, Tile>();
    auto kernel = gemm_dmma_f64<AK, BK, Tile, V16>;
    // 48 KB need no leave; the call is a share of a small product's time
    if (smem > 48 * 1024 &&
        cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) != cudaSuccess)
        return RC_ERR_CUDA;
    dim3 grid;
    if (!tile_grid<Tile>(p, &grid)) return RC_ERR_NOT_SUPPORTED;
    const int64_t zstride = p.m * p.n;
    // Without room for the partial products (or a capture under way, in which none can be made) the
    // same tiles take all of K.
    double* P = nz > 1 ? static_cast<double*>(workspace_if_any(s, (size_t)nz * zstride * sizeof(double), 7)) : nullptr;
    if (P) {
        const int64_t kchunk = ((p.k + nz - 1) / nz + DK - 1) / DK * DK;
        nz = (int)((p.k + kchunk - 1) / kchunk);
        grid.z = nz;
        kernel<<<grid, Tile::THREADS, smem, s>>>(p.m, p.n, p.k, 1.0, A, B, 0.0, colmajor(P, p.m), kFull, 0, abort,
                                                 kchunk, zstride);
        RC_TRY(check_launch());
        dim3 rg(ceil_div(p.m, 256) < 1024u ? ceil_div(p.m, 256) : 1024u, p.n < 65535 ? (unsigned)p.n : 65535u);
        splitk_reduce<<<rg, 256, 0, s>>>(p.m, p.n, nz, P, zstride, alpha, beta, C);
        return check_launch();
    }
    kernel<<<grid, Tile::THREADS, smem, s>>>(p.m, p.n, p.k, alpha, A, B, beta, C, p.mask, off, abort, p.k, 0);
    return check_launch();
}

template <bool AK, bool BK, bool V16>
int launch_tile(TileId id, const Shape& p, double alpha, View<const double> A, View<const double> B, double beta,
                View<double> C, int64_t off, int nz, cudaStream_t s, const int* abort) {
    switch (id) {
    case kTileM: return launch_dmma<AK, BK, TileM, V16>(p, alpha, A, B, beta, C, off, nz, s, abort);
    case kTileS: return launch_dmma<AK, BK, TileS, V16>(p, alpha, A, B, beta, C, off, nz, s, abort);
    case kTileT: return launch_dmma<AK, BK, TileT, V16>(p, alpha, A, B, beta, C, off, nz, s, abort);
    case kTileP: return launch_dmma<AK, BK, TileP, V16>(p, alpha, A, B, beta, C, off, nz, s, abort);
    case kTileR: return launch_dmma<AK, BK, TileR, V16>(p, alpha, A, B, beta, C, off, nz, s, abort);
    default: return launch_dmma<AK, BK, TileQ, V16>(p, alpha, A, B, beta, C, off, nz, s, abort);
    }
}

template <bool AK, bool BK>
int gemm_dmma(int64_t m, int64_t n, int64_t k, double alpha, View<const double> A, View<const double> B, double beta,
              View<double> C, Mask mask, int64_t off, cudaStream_t s, const int* abort) {
    const Shape p(m, n, k, mask);
    TileId id = kTileM;
    int nz = 1;
    pick_tile(p, C.p == A.p, C.p == B.p, mask == kFull && k >= 2048, sm_count(), &id, &nz);
    auto even = [](const double* q, int64_t ld) { return reinterpret_cast<uintptr_t>(q) % 16 == 0 && ld % 2 == 0; };
    if (even(A.p, AK ? A.rs : A.cs) && even(B.p, BK ? B.cs : B.rs))
        return launch_tile<AK, BK, true>(id, p, alpha, A, B, beta, C, off, nz, s, abort);
    return launch_tile<AK, BK, false>(id, p, alpha, A, B, beta, C, off, nz, s, abort);
}

// Cycles an FP32 product takes with a tile (the FMA units do BM BN BK / 128 a k-step, of which
// a tile reaches the share eff: 0.78 measured at 4096^3 and 0.40 at 1024^3; a k-step of a lone tile takes
// `chain` cycles: 1900 and 800 measured at 512^3; see tile_cycles).
template <class Tile>
double simt_cycles(const Shape& s, double eff, double chain) {
    const int64_t tm = (s.m + Tile::BM - 1) / Tile::BM, tn = (s.n + Tile::BN - 1) / Tile::BN;
    double tiles = (double)tm * tn;
    if (s.triangle) tiles = 0.5 * (tiles + (tm > tn ? tm : tn));
    const double per_sm = ceil(tiles / sm_count()), work = Tile::BM * Tile::BN * Tile::BK / 128.0 / eff;
    const double ksteps = ceil((double)s.k / Tile::BK), full = floor(per_sm / Tile::OCC), rest = per_sm - full * Tile::OCC;
    auto round = [&](double c) { return c <= 0 ? 0.0 : ksteps * (c * work > chain ? c * work : chain) + 3000.0; };
    return full * round(Tile::OCC) + round(rest);
}

template <bool AK, bool BK, class Tile>
int launch_sgemm(const Shape& p, float alpha, View<const float> A, View<const float> B, float beta, View<float> C,
                 int64_t off, cudaStream_t s, const int* abort) {
    auto aligned = [](const float* q, int64_t ld) { return reinterpret_cast<uintptr_t>(q) % 16 == 0 && ld % 4 == 0; };
    dim3 grid;
    if (!tile_grid<Tile>(p, &grid)) return RC_ERR_NOT_SUPPORTED;
    if (aligned(A.p, AK ? A.rs : A.cs) && aligned(B.p, BK ? B.cs : B.rs))
        sgemm_simt<AK, BK, Tile, true><<<grid, Tile::THREADS, 0, s>>>(p.m, p.n, p.k, alpha, A, B, beta, C, p.mask, off,
                                                                      abort);
    else
        sgemm_simt<AK, BK, Tile, false><<<grid, Tile::THREADS, 0, s>>>(p.m, p.n, p.k, alpha, A, B, beta, C, p.mask,
                                                                       off, abort);
    return check_launch();
}

template <bool AK, bool BK>
int sgemm(int64_t m, int64_t n, int64_t k, float alpha, View<const float> A, View<const float> B, float beta,
          View<float> C, Mask mask, int64_t off, cudaStream_t s, const int* abort) {
    const Shape p(m, n, k, mask);
    // A product that writes over one of its own operands (C on B with m <= 128, on A with n <= 64)
    // takes the tile that spans that operand's rows or columns, as in pick_tile.
    const bool in_place = C.p == A.p || C.p == B.p;
    if (in_place || simt_cycles<SimtL>(p, 0.78, 1900.0) <= simt_cycles<SimtS>(p, 0.40, 800.0))
        return launch_sgemm<AK, BK, SimtL>(p, alpha, A, B, beta, C, off, s, abort);
    return launch_sgemm<AK, BK, SimtS>(p, alpha, A, B, beta, C, off, s, abort);
}

// Scale (beta != 1) the masked part of C when k == 0 or alpha == 0.
template <class T>
__global__ void scale_masked(int64_t m, int64_t n, T beta, View<T> C, Mask mask, int64_t off, const int* abort) {
    if (aborted(abort)) return;
    for (int64_t j = blockIdx.y; j < n; j += gridDim.y)
        for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < m; i += (int64_t)gridDim.x * blockDim.x)
            if (in_mask(mask, off, i, j)) C(i, j) = beta == T(0) ? T(0) : beta * C(i, j);
}

}  // namespace

template <class T>
int gemm(int64_t m, int64_t n, int64_t k, T alpha, View<const T> A, View<const T> B, T beta, View<T> C, Mask asked,
         int64_t off, cudaStream_t s, const int* abort) {
    if (m <= 0 || n <= 0) return RC_SUCCESS;
    const Mask mask = asked == kLowerTri ? kLower : asked;  // of the kernels that multiply the zeros
    if (k <= 0 || alpha == T(0)) {
        if (beta == T(1)) return RC_SUCCESS;
        dim3 grid(ceil_div(m, 256) < 1024u ? ceil_div(m, 256) : 1024u, n < 65535 ? (unsigned)n : 65535u);
        scale_masked<T><<<grid, 256, 0, s>>>(m, n, beta, C, mask, off, abort);
        return check_launch();
    }
    const bool a_k = A.cs == 1, a_m = A.rs == 1, b_k = B.rs == 1, b_n = B.cs == 1;
    if (!(a_k || a_m) || !(b_k || b_n)) return RC_ERR_NOT_SUPPORTED;
    auto run = [&](auto ak, auto bk) {
        if constexpr (std::is_same<T, double>::value)
            return gemm_dmma<ak.value, bk.value>(m, n, k, alpha, A, B, beta, C, asked, off, s, abort);
        else
            return sgemm<ak.value, bk.value>(m, n, k, alpha, A, B, beta, C, mask, off, s, abort);
    };
    if (a_k && b_k) return run(std::true_type{}, std::true_type{});
    if (a_k) return run(std::true_type{}, std::false_type{});
    if (b_k) return run(std::false_type{}, std::true_type{});
    return run(std::false_type{}, std::false_type{});
}

template int gemm<double>(int64_t, int64_t, int64_t, double, View<const double>, View<const double>, double,
                          View<double>, Mask, int64_t, cudaStream_t, const int*);
template int gemm<float>(int64_t, int64_t, int64_t, float, View<const float>, View<const float>, float,
                         View<float>, Mask, int64_t, cudaStream_t, const int*);

}  // namespace rc

namespace {

template <class T>
int gemm_abi(int transA, int transB, size_t m, size_t n, size_t k, T alpha, const T* A, size_t lda, const T* B,
             size_t ldb, T beta, T* C, size_t ldc, void* stream) {
    if (m == 0 || n == 0) return RC_SUCCESS;
    if (!C || ldc < m) return RC_ERR_INVALID_ARGUMENT;
    if (k > 0) {
        if (!A || !B) return RC_ERR_INVALID_ARGUMENT;
        if (lda < (transA ? k : m) || ldb < (transB ? n : k)) return RC_ERR_INVALID_ARGUMENT;
    }
    rc::View<const T> a = rc::colmajor(A, (int64_t)lda);
    rc::View<const T> b = rc::colmajor(B, (int64_t)ldb);
    if (transA) a = a.t();
    if (transB) b = b.t();
    return rc::gemm<T>((int64_t)m, (int64_t)n, (int64_t)k, alpha, a, b, beta, rc::colmajor(C, (int64_t)ldc),
                       rc::kFull, 0, static_cast<cudaStream_t>(stream));
}

template <class T>
int syrk_abi(int upper, int trans, size_t n, size_t k, T alpha, const T* A, size_t lda, T beta, T* C, size_t ldc,
             void* stream) {
    if (n == 0) return RC_SUCCESS;
    if (!C || ldc < n) return RC_ERR_INVALID_ARGUMENT;
    if (k > 0 && (!A || lda < (trans ? k : n))) return RC_ERR_INVALID_ARGUMENT;
    rc::View<const T> a = rc::colmajor(A, (int64_t)lda);
    if (trans) a = a.t();  // op(A) = A^T, n x k
    return rc::gemm<T>((int64_t)n, (int64_t)n, (int64_t)k, alpha, a, a.t(), beta, rc::colmajor(C, (int64_t)ldc),
                       upper ? rc::kUpper : rc::kLower, 0, static_cast<cudaStream_t>(stream));
}

}  // namespace

extern "C" {

int rc_gemm_f64(int transA, int transB, size_t m, size_t n, size_t k, double alpha, const double* A, size_t lda,
                const double* B, size_t ldb, double beta, double* C, size_t ldc, void* stream) {
    return gemm_abi<double>(transA, transB, m, n, k, alpha, A, lda, B, ldb, beta, C, ldc, stream);
}
int rc_gemm_f32(int transA, int transB, size_t m, size_t n, size_t k, float alpha, const float* A, size_t lda,
                const float* B, size_t ldb, float beta, float* C, size_t ldc, void* stream) {
    return gemm_abi<float>(transA, transB, m, n, k, alpha, A, lda, B, ldb, beta, C, ldc, stream);
}
int rc_syrk_f64(int upper, int trans, size_t n, size_t k, double alpha, const double* A, size_t lda, double beta,
                double* C, size_t ldc, void* stream) {
    return syrk_abi<double>(upper, trans, n, k, alpha, A, lda, beta, C, ldc, stream);
}
int rc_syrk_f32(int upper, int trans, size_t n, size_t k, float alpha, const float* A, size_t lda, float beta,
                float* C, size_t ldc, void* stream) {
    return syrk_abi<float>(upper, trans, n, k, alpha, A, lda, beta, C, ldc, stream);
}

}  // extern "C"
