// The FP64 product's tiles and the choice among them: host arithmetic only.
#pragma once
#include <cmath>
#include <cstdint>

namespace rc {

constexpr int DK = 16;  // depth of a k-step

template <int BM_, int BN_, int WARPS_M_, int WARPS_N_, int STAGES_, int OCC_>
struct DmmaTile {
    static constexpr int BM = BM_, BN = BN_, WARPS_M = WARPS_M_, WARPS_N = WARPS_N_, STAGES = STAGES_;
    static constexpr int OCC = OCC_;  // CTAs per SM, by shared memory and registers
    static constexpr int THREADS = 32 * WARPS_M * WARPS_N;
    static constexpr int WM = BM / WARPS_M, WN = BN / WARPS_N;
    static constexpr int MI = WM / 16, NI = WN / 8;
};
// 64 x 64 with three CTAs per SM is the fastest at every size that fills the GPU: the CTAs'
// barriers, fills and drains fall at different times, so the pipe always has work. 4096^3:
// 4.08-4.12 ms (33.7 TFLOP/s), against 4.47-4.72 for one 128 x 128 CTA of 8 warps per SM,
// 4.10-4.14 for two 128 x 64 of 4 warps, 4.17-4.26 for four 64 x 64 with a two-stage ring
// and 4.71-4.88 for 32 x 32. Below about one tile per SM the smaller tiles win: 512^3 takes
// 16.5 us with 32 x 32 and 32.8 us with 64 x 64.
using TileM = DmmaTile<64, 64, 2, 2, 3, 3>;
using TileS = DmmaTile<32, 32, 2, 2, 4, 5>;   // small products: latency counts
using TileT = DmmaTile<64, 16, 4, 1, 4, 4>;   // up to 16 columns
using TileP = DmmaTile<32, 128, 1, 4, 4, 2>;  // one CTA owns whole rows of a 128-column panel (in place)
using TileQ = DmmaTile<128, 32, 4, 1, 4, 2>;  // one CTA owns whole columns of a 128-row block (in place)
using TileR = DmmaTile<128, 16, 4, 1, 4, 2>;  // the same for few columns: half the serial work per CTA

struct Problem {
    int64_t m, n, k;
    bool triangle;  // one triangle of a square product
};

enum TileId { kTileM, kTileS, kTileT, kTileP, kTileQ, kTileR };

// Cycles a product takes with a tile, per the model behind the choice of tiles: an SM works
// on up to OCC tiles at a time, a k-step of which takes the pipe BM BN / 4 cycles each (it
// reaches 94% of that with 64 x 64 tiles, 80% with the small ones), but never less than one
// warp's own chain (its MMAs and ~400 cycles of barrier and fragment loads: 512^3 on 64 x 64
// tiles, one per SM); a round of tiles pays a fixed fill and drain.
template <class Tile>
double tile_cycles(const Problem& s, int nz, int sms) {
    const int64_t tm = (s.m + Tile::BM - 1) / Tile::BM, tn = (s.n + Tile::BN - 1) / Tile::BN;
    double tiles = (double)tm * tn;
    if (s.triangle) tiles = 0.5 * (tiles + (tm > tn ? tm : tn));  // of a square, tm (tm + 1) / 2 tiles run
    const double per_sm = std::ceil(tiles * nz / sms);
    const double work = Tile::BM * Tile::BN / 4.0 / (Tile::MI * Tile::NI >= 8 ? 0.94 : 0.80);
    const double chain = Tile::MI * Tile::NI * 4 * 32 + 400.0, ksteps = std::ceil((double)s.k / nz / DK);
    const double full = std::floor(per_sm / Tile::OCC), rest = per_sm - full * Tile::OCC;
    auto round = [&](double c) { return c <= 0 ? 0.0 : ksteps * (c * work > chain ? c * work : chain) + 3000.0; };
    return full * round(Tile::OCC) + round(rest);
}

// A K split's partial products, in bytes, and the most that they may take: the buffer stays with
// the stream. By the model a larger one would gain 2.5% at most (20000 shapes drawn from 24 to
// 16000 rows and columns and a depth of 2048 to 60000; up to 256 MB the gain reaches 20%).
inline double split_bytes(const Problem& p, int nz) { return nz > 1 ? 8.0 * nz * p.m * p.n : 0.0; }
constexpr double kSplitMost = 256.0 * 1024 * 1024;

// The tile and K split of least modelled time. A product that writes over one of its own
// operands (C on A with n <= 128, or on B with m <= 128) takes a tile that spans that
// operand's rows or columns: each CTA has then read all of what it overwrites.
inline void pick_tile(const Problem& p, bool c_on_a, bool c_on_b, bool may_split, int sms, TileId* id, int* nz) {
    *nz = 1;
    if (c_on_a || c_on_b) {
        *id = c_on_a ? kTileP : p.n <= 16 * (int64_t)sms ? kTileR : kTileQ;
        return;
    }
    *id = kTileM;
    double best = tile_cycles<TileM>(p, 1, sms);
    auto look = [&](TileId t, double cycles, int z) {
        if (cycles < best) {
            best = cycles;
            *id = t;
            *nz = z;
        }
    };
    // A split pays a second launch and two passes over its partial products.
    const int zmax = may_split ? 8 : 1;
    for (int z = 1; z <= zmax && (z == 1 || ((int64_t)z * 512 <= p.k && split_bytes(p, z) <= kSplitMost)); ++z) {
        const double extra = z > 1 ? 6000.0 + 16.0 * z * p.m * p.n / 2500.0 : 0.0;
        look(kTileM, tile_cycles<TileM>(p, z, sms) + extra, z);
        look(kTileS, tile_cycles<TileS>(p, z, sms) + extra, z);
        if (p.n <= 16) look(kTileT, tile_cycles<TileT>(p, z, sms) + extra, z);
    }
}

}  // namespace rc
