// row_parts.h -- which image rows a warp of the forward projection marches over,
// and how they are divided into parts.  Plain arithmetic, so that a host program
// can go through it without a GPU.
#pragma once

#include <cmath>

#ifdef __CUDACC__
#define ROW_PARTS_FN __host__ __device__ __forceinline__
#else
#define ROW_PARTS_FN inline
#endif

namespace ctprj {

// Rows bottom, ..., top.  "No rows" lies next to the image (half + 1 and
// -half - 1) and not at the ends of the integers, so that no difference or sum
// of the two leaves 32 bits.
struct RowRange {
    int bottom, top;
};

ROW_PARTS_FN RowRange no_rows(int half) { return {half + 1, -half - 1}; }

// The rows in which a ray can meet the image: its crossing xc = A - y S is
// affine in y, and rows with |xc| > half + 2 are skipped anyway; two rows of
// margin cover the division's rounding.
ROW_PARTS_FN RowRange ray_rows(float A, float S, int half)
{
    const float lim = (float)half + 2.0f;
    float lo = (float)-half, hi = (float)half;
    if (fabsf(S) > 1e-6f) {
#ifdef __CUDA_ARCH__
        const float a = __fdividef(A - lim, S), b = __fdividef(A + lim, S);
#else
        const float a = (A - lim) / S, b = (A + lim) / S;
#endif
        lo = fmaxf(lo, fminf(a, b) - 2.0f);
        hi = fminf(hi, fmaxf(a, b) + 2.0f);
    } else if (fabsf(A) > lim + 1.0f) {
        return no_rows(half);
    }
    if (!(lo <= hi)) return no_rows(half);
    return {(int)floorf(lo), (int)ceilf(hi)};
}

// part s of R of the rows `all` (none where there are none)
ROW_PARTS_FN RowRange part_rows(RowRange all, int s, int R)
{
    if (all.top < all.bottom) return all;
    const int M = all.top - all.bottom + 1;
    return {all.top - (int)((long long)M * (s + 1) / R) + 1, all.top - (int)((long long)M * s / R)};
}

}  // namespace ctprj
