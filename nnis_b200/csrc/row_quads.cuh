// Rows of float32 values held whole in registers, four neighbours a load: a warp issues every load of a row before it
// needs the first value, and a norm's second use of the row costs no second trip.  (One value a load and two passes left
// a row-wise kernel waiting for a chain of loads: 10 us for eight rows of 2,048 in four groups, 2.4 us now.)
#pragma once

#include "common.cuh"

namespace nnis {

// Lane `lane` of a warp holds values 4 (lane + 32 j) .. + 3 of a row of 4 n4 values; zeros beyond it.
template <int Q>
struct RowQuads {
    float4 v[Q];
    __device__ __forceinline__ void load(const float* row, int n4, int lane) {
#pragma unroll
        for (int j = 0; j < Q; ++j)
            v[j] = lane + 32 * j < n4 ? load4(row + 4 * (lane + 32 * j)) : make_float4(0.f, 0.f, 0.f, 0.f);
    }
    __device__ __forceinline__ float squares() const {
        float ss = 0.f;
#pragma unroll
        for (int j = 0; j < Q; ++j) {
            ss = fmaf(v[j].x, v[j].x, ss);
            ss = fmaf(v[j].y, v[j].y, ss);
            ss = fmaf(v[j].z, v[j].z, ss);
            ss = fmaf(v[j].w, v[j].w, ss);
        }
        return ss;
    }
};

// out = o / rms(o) * f(i), a warp per head: f gives the four multipliers of values 4 i ..
template <typename T, int Q, typename F>
__device__ __forceinline__ void finish_head(const float* o, T* out, int n4, float eps, int lane, F f) {
    RowQuads<Q> row;
    row.load(o, n4, lane);
    float4 m[Q];
#pragma unroll
    for (int j = 0; j < Q; ++j) m[j] = lane + 32 * j < n4 ? f(lane + 32 * j) : make_float4(0.f, 0.f, 0.f, 0.f);
    const float s = 1.0f / sqrtf(warp_sum(row.squares()) / (float)(4 * n4) + eps);
#pragma unroll
    for (int j = 0; j < Q; ++j)
        if (lane + 32 * j < n4)
            store4(out + 4 * (lane + 32 * j), make_float4((row.v[j].x * s) * m[j].x, (row.v[j].y * s) * m[j].y,
                                                          (row.v[j].z * s) * m[j].z, (row.v[j].w * s) * m[j].w));
}

}  // namespace nnis
