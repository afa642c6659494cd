/*
 * sor_box.h -- the nodes of one colour of the linear box, host and device.
 */
#pragma once
#include <stdint.h>

#include "espic_world.h"

namespace espic {

/* Entry t of colour c's enumeration is node i = 1 + 2 i2 + ((1 + j + k + c) & 1)
 * of interior row (j, k), i2 = t mod hx; a row of an odd interior has one
 * entry too many in one colour. */
__host__ __device__ inline int sor_row_entries(const Geo &g) { return (g.ni - 1) / 2; }
__host__ __device__ inline int64_t sor_rows(const Geo &g) { return (int64_t)(g.nj - 2) * (g.nk - 2); }

/* Whether 32-bit indices and div_small find every entry: nodes below 2^31,
 * and fewer than 2^24 entries or than 2^22 rows (the quotients).  Thin boxes
 * leave that range long before the largest ones do: 7x3402x3402 nodes are
 * 11.6M rows, and the estimate would miss 46,899 of 34.7M entries. */
inline bool sor_short_indices(const Geo &g) {
    const int64_t rows = sor_rows(g);
    return (int64_t)g.ni * g.nj * g.nk < (1ll << 31) && (sor_row_entries(g) * rows < (1 << 24) || rows < (1 << 22));
}

/* the node u of entry t; false for the entry too many.  int32_t: the box has
 * sor_short_indices */
template <typename I, typename U>
__host__ __device__ __forceinline__ bool sor_entry(const Geo &g, U hx, U t, int c, I &u) {
    int i, j, k;
    if constexpr (sizeof(I) == 4) {
        const U row = div_small(t, hx, 1.f / (float)hx);
        const U kk = div_small(row, (U)(g.nj - 2), 1.f / (float)(g.nj - 2));
        j = 1 + (int)(row - kk * (U)(g.nj - 2));
        k = 1 + (int)kk;
        i = 1 + 2 * (int)(t - row * hx) + ((1 + j + k + c) & 1);
    } else {
        const U row = t / hx, kk = row / (U)(g.nj - 2);
        j = 1 + (int)(row - kk * (U)(g.nj - 2));
        k = 1 + (int)kk;
        i = 1 + 2 * (int)(t - row * hx) + ((1 + j + k + c) & 1);
    }
    if (i > g.ni - 2) return false;
    u = ((I)k * g.nj + j) * g.ni + i;
    return true;
}

}  // namespace espic
