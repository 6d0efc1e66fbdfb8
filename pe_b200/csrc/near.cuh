// near.cuh -- the candidate lists of the grid step (dem.cu k_grid_near): per slot of the cell
// order, the slots of the spheres within reach by an FP32 test with a margin.  Used by the step's
// force kernel and by its adjoint.
#pragma once

#include <climits>

#include "internal.cuh"

namespace peb {

constexpr int kNear = 16;   // recorded candidates per sphere; one with more searches its cells

// What a sphere's rounded FP32 record may be off: |d_fp32 - d| stays below ~1e-7 (|x| + |y| + |z| + 2 r +
// d) for any partner closer than r_i + r_j; the margin is 100 times that.
__device__ __forceinline__ float near_margin(float x, float y, float z, float r) {
    return 1e-5f * (1.0f + fabsf(x) + fabsf(y) + fabsf(z) + 4.0f * r);
}

// slot t's recorded candidates in ascending order, the order in which a 27-cell scan visits them
// (a sorting network over registers; the places from cnt on hold INT_MAX and sort last)
__device__ __forceinline__ void load_near(const int32_t *__restrict__ near_idx, int64_t n, int64_t t,
                                          int cnt, int32_t sl[kNear]) {
#pragma unroll
    for (int k = 0; k < kNear; ++k) sl[k] = k < cnt ? near_idx[(int64_t)k * n + t] : INT_MAX;
    if (cnt > 1) {
#pragma unroll
        for (int kk = 2; kk <= kNear; kk <<= 1)
#pragma unroll
            for (int j = kk >> 1; j > 0; j >>= 1)
#pragma unroll
                for (int i = 0; i < kNear; ++i) {
                    const int l = i ^ j;
                    if (l > i) {
                        const int32_t x = sl[i], y = sl[l];
                        const bool up = (i & kk) == 0;
                        if ((x > y) == up) {
                            sl[i] = y;
                            sl[l] = x;
                        }
                    }
                }
    }
}

}  // namespace peb
