// The merge of split attention: kernels that cut a query's key range into slices
// leave, per (token, head, slice), a record [running max, running sum, unnormalised
// output of d values]; this kernel adds the slices up in ascending order.  With `row_gate`
// (float32, one per row) the row's output is multiplied by it.
#pragma once

#include <float.h>

#include "async_copy.cuh"
#include "common.cuh"

namespace nnis {

// At most 64 slices.  A warp works out the slices' weights exp(m_s - m) / l once (lane s holds slices s and s + 32); then
// every thread sums its output values over the slices, in ascending order of slice.  Rows of at most 64 values take a
// warp each, four to a CTA of 128 threads, rows of up to 128 where they are many and their slices few; others a CTA each
// (32 slices of 128 values, 16 rows: a warp a row 3 us longer; 16,384 rows of 4 slices: a CTA a row 7 us longer of 263
// with the attention).  Eight slices' values of a thread's pair are asked for together: one after another they were a trip
// to L2 each (128 rows of 512 values, 16 slices: 9.5 -> 5.8 us; 9,216 rows of 64 values in a float32 prompt: 11.0
// -> 5.4).  EARLY: few rows, where these trips are the whole time: sixteen slices' values are asked
// for beside the maxima and sums, needed or not, and rows beyond 256 values take 256 threads, a pair each (128 rows of 512 values,
// 16 slices, one launch after another: 3.7 -> 2.4 us; behind latent attention 6.1 -> 2.9).
template <typename T, bool WARP_ROWS, int THREADS, bool EARLY>
__global__ void __launch_bounds__(THREADS)
attn_merge_kernel(const float* __restrict__ partial, T* __restrict__ out, size_t n_rows, int d,
                  int n_splits, const float* __restrict__ row_gate, int pairs) {
    __shared__ float shares[WARP_ROWS ? 4 : 1][64];
    pdl_wait();  // (a no-op unless launched as a programmatic dependent)
    pdl_launch_dependents();
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const size_t row = WARP_ROWS ? blockIdx.x * (size_t)4 + warp : blockIdx.x;
    if (row >= n_rows) return;  // (whole warps)
    float* share = shares[WARP_ROWS ? warp : 0];
    const float* rec = partial + row * n_splits * (size_t)(d + 2);
    const int first = WARP_ROWS ? lane : (int)threadIdx.x;
    constexpr int kThreads = WARP_ROWS ? 32 : THREADS, kMost = EARLY ? 16 : 8;
    float2 v[kMost];
    if (EARLY && pairs) {
#pragma unroll
        for (int k = 0; k < kMost; ++k)
            v[k] = k < n_splits && first * 2 < d ? *reinterpret_cast<const float2*>(rec + (size_t)k * (d + 2) + 2 + first * 2)
                                                 : make_float2(0.f, 0.f);
    }
    if (WARP_ROWS || warp == 0) {
        float ms[2], ls[2];
        float m = -FLT_MAX;
#pragma unroll
        for (int k = 0; k < 2; ++k) {
            int s = lane + 32 * k;
            ms[k] = s < n_splits ? rec[(size_t)s * (d + 2)] : 0.f;
            ls[k] = s < n_splits ? rec[(size_t)s * (d + 2) + 1] : 0.f;
            if (ls[k] != 0.f) m = fmaxf(m, ms[k]);
        }
        m = warp_max(m);
        float l = 0.f;
#pragma unroll
        for (int k = 0; k < 2; ++k) {
            ms[k] = ls[k] != 0.f ? expf(ms[k] - m) : 0.f;
            l += ls[k] * ms[k];
        }
        l = warp_sum(l);
        float inv = l != 0.f ? 1.0f / l : 0.f;  // (a sum that is no number stays one)
        if (row_gate) inv *= row_gate[row];
        share[lane] = ms[0] * inv;
        share[lane + 32] = ms[1] * inv;
    }
    if (WARP_ROWS) __syncwarp();
    else __syncthreads();
    if (pairs) {
        for (int i = first * 2; i < d; i += kThreads * 2) {
            float2 o = make_float2(0.f, 0.f);
            for (int s0 = 0; s0 < n_splits; s0 += kMost) {
                // (slices that hold nothing for the row have weight zero and are never added)
                float w[kMost];
#pragma unroll
                for (int k = 0; k < kMost; ++k) {
                    w[k] = s0 + k < n_splits ? share[s0 + k] : 0.f;
                    if (!EARLY || s0 || i != first * 2)
                        v[k] = w[k] != 0.f ? *reinterpret_cast<const float2*>(rec + (size_t)(s0 + k) * (d + 2) + 2 + i)
                                           : make_float2(0.f, 0.f);
                }
#pragma unroll
                for (int k = 0; k < kMost; ++k) {
                    if (w[k] != 0.f) {
                        o.x = fmaf(w[k], v[k].x, o.x);
                        o.y = fmaf(w[k], v[k].y, o.y);
                    }
                }
            }
            store2(out + row * d + i, o.x, o.y);
        }
        return;
    }
    for (int i = first; i < d; i += kThreads) {
        float o = 0.f;
        for (int s = 0; s < n_splits; ++s) {
            float w = share[s];
            if (w != 0.f) o = fmaf(w, rec[(size_t)s * (d + 2) + 2 + i], o);
        }
        out[row * d + i] = from_float<T>(o);
    }
}

template <typename T>
static cudaError_t launch_merge(const float* partial, T* out, size_t rows, int d, int n_splits, const float* row_gate,
                                cudaStream_t stream) {
    // (records of an even number of floats start on 8-byte boundaries if the first does)
    const int pairs = d % 2 == 0 && (uintptr_t)partial % 8 == 0 && (uintptr_t)out % (2 * sizeof(T)) == 0;
    const bool warp_rows = d <= 64 || (d <= 128 && rows >= 2000 && n_splits <= 16);
    // Early as long as the device holds all rows beside the next kernel's CTAs (float32 outputs take more registers: three
    // instead of four CTAs an SM).  us late -> early, bfloat16 / float32: 16 slices of 128 values, 444 rows 2.66 -> 2.32 /
    // 2.66 -> 2.31, 592 rows 2.75 -> 2.45 / 2.72 -> 2.85, 740 rows 2.85 -> 3.01; of 512 values 444 rows 4.19 -> 3.38 / 4.19
    // -> 3.12, 592 rows 4.41 -> 3.53 / 4.49 -> 4.50, 740 rows 4.66 -> 4.85; of 1,024 values 296 rows 6.28 -> 5.85, 370 rows
    // 6.66 -> 6.83.  From 6 rows an SM on the late form is in its second wave, the early one up to 8 (7) not in its third:
    // 1,036 rows of 256 values 4.67 -> 3.43 / 4.69 -> 3.27, of 512 7.72 -> 5.57 / 7.72 -> 6.45 (level at 128 values; 320
    // values of float32, 9 slices, 5.58 -> 5.84).  Up to eight slices are one trip late too: level or slower up to 256
    // values (592 rows 2.14 -> 2.40), of 512 values 296 rows 2.76 -> 2.55 / 2.76 -> 2.86, 128 rows 2.56 -> 2.20 / 2.56 ->
    // 2.20, of 1,024 slower (3.58 -> 4.04).  More than sixteen are slower (32: 3.6 -> 5.1).
    const bool wide = d > 256, f32 = sizeof(T) == 4;
    bool early = !warp_rows && pairs && n_splits <= 16;
    if (early) {
        const size_t sms = (size_t)device_sms(), held = f32 ? 3 : 4;
        if (n_splits > 8) {
            const bool second = d > 128 && d <= 512 && (d <= 256 || d >= 384) && rows > 6 * sms && rows <= (f32 ? 7 : 8) * sms;
            early = rows <= (d > 512 ? 2 : held) * sms || second;
        } else {
            early = wide && d <= 512 && rows <= held / 2 * sms;
        }
    }
    if (early) {
        return launch_dependent(wide ? attn_merge_kernel<T, false, 256, true> : attn_merge_kernel<T, false, 128, true>, (unsigned)rows,
                                wide ? 256 : 128, 0, stream, partial, out, rows, d, n_splits, row_gate, pairs);
    }
    return warp_rows ? launch_dependent(attn_merge_kernel<T, true, 128, false>, (unsigned)((rows + 3) / 4), 128, 0, stream, partial, out,
                                        rows, d, n_splits, row_gate, pairs)
                     : launch_dependent(attn_merge_kernel<T, false, 128, false>, (unsigned)rows, 128, 0, stream, partial, out, rows,
                                        d, n_splits, row_gate, pairs);
}

}  // namespace nnis
