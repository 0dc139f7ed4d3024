// A float32 value as the sum of three bfloat16 values (h = bfloat16(x), then bfloat16 of what is left, twice), exact from
// 2^-109 on and within 2^-134 below, for products of float32 operands on the tensor cores: see gemm_split_f32.cu.
#pragma once

#include "fma_pairs.cuh"

namespace nnis {

// Eight consecutive floats in one load, in pairs; the address is a multiple of 32 bytes.
__device__ __forceinline__ void load8(const float* p, unsigned long long (&v)[4]) {
    asm volatile("ld.global.v4.b64 {%0, %1, %2, %3}, [%4];" : "=l"(v[0]), "=l"(v[1]), "=l"(v[2]), "=l"(v[3]) : "l"(p));
}

// Eight values in one store; the address is a multiple of 32 bytes.
__device__ __forceinline__ void store8(float* p, const float* v) {
    asm volatile("st.global.v4.b64 [%0], {%1, %2, %3, %4};" ::"l"(p), "l"(pair_of(v[0], v[1])), "l"(pair_of(v[2], v[3])),
                 "l"(pair_of(v[4], v[5])), "l"(pair_of(v[6], v[7]))
                 : "memory");
}

// A pair of values' next bfloat16 parts, packed; what is left of the values stays in x.
__device__ __forceinline__ uint32_t next_part(unsigned long long& x) {
    uint32_t p;
    asm("{\n\t.reg .f32 a, b;\n\t.reg .b32 lo, hi;\n\t.reg .b64 h;\n\t"
        "mov.b64 {a, b}, %1;\n\t"
        "cvt.rn.bf16x2.f32 %0, b, a;\n\t"
        "shl.b32 lo, %0, 16;\n\t"
        "and.b32 hi, %0, 0xffff0000;\n\t"
        "mov.b64 h, {lo, hi};\n\t"
        "sub.rn.f32x2 %1, %1, h;\n\t}"
        : "=r"(p), "+l"(x));
    return p;
}
__device__ __forceinline__ uint32_t last_part(unsigned long long x) {
    const float2 f = halves(x);
    uint32_t p;
    asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(p) : "f"(f.y), "f"(f.x));
    return p;
}

// The three parts of eight values at `dst`, `dst + part` and `dst + 2 part` (16 bytes each; what is left stays in v).
__device__ __forceinline__ void store_parts(unsigned char* dst, uint32_t part, unsigned long long (&v)[4]) {
    uint4 o;
    o.x = next_part(v[0]);
    o.y = next_part(v[1]);
    o.z = next_part(v[2]);
    o.w = next_part(v[3]);
    *reinterpret_cast<uint4*>(dst) = o;
    o.x = next_part(v[0]);
    o.y = next_part(v[1]);
    o.z = next_part(v[2]);
    o.w = next_part(v[3]);
    *reinterpret_cast<uint4*>(dst + part) = o;
    o.x = last_part(v[0]);
    o.y = last_part(v[1]);
    o.z = last_part(v[2]);
    o.w = last_part(v[3]);
    *reinterpret_cast<uint4*>(dst + 2 * part) = o;
}

// Parts of the two operands of the six products that are made, the smallest first.
constexpr int kSplitProducts = 6;
__host__ __device__ constexpr int split_part_a(int p) { return p == 0 ? 2 : p == 2 || p == 3 ? 1 : 0; }
__host__ __device__ constexpr int split_part_b(int p) { return p == 1 ? 2 : p == 2 || p == 4 ? 1 : 0; }

}  // namespace nnis
