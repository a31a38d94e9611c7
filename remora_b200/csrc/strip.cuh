// Triangular solve of a panel of up to kStripRows rows.
#pragma once
#include "common.cuh"

namespace rc {

constexpr int64_t kStripRows = 512;

// B <- A^-1 B in place for the m x m lower or upper triangle A and m x n B (each row- or
// column-major), m <= kStripRows, given the inverses of A's 128-row diagonal blocks: block b at
// W + b * 128 * 128, column- or row-major.
template <class T>
int strip_solve(bool upper, int64_t m, int64_t n, View<const T> A, const T* W, bool w_row_major, View<T> B,
                cudaStream_t s, const int* abort);

}  // namespace rc
