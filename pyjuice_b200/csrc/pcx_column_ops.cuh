// Device helpers shared by the kernels of the column program (pcx_column.cu, pcx_column_chain.cu).
#pragma once
#include <cuda_bf16.h>
#include "pcx_common.cuh"

namespace {

enum ColMode { C_FWD = 0, C_ELE = 1 };

// Value rows are written and read inside one launch: plain (coherent) loads, never the read-only path.  Volatile, so that
// none moves over a level's barrier, but without a memory clobber: the loads of tables and parameters (which a launch only
// reads) may move freely between them.
__device__ __forceinline__ float ldv(const float* p) {
    float v;
    asm volatile("ld.global.f32 %0, [%1];" : "=f"(v) : "l"(p));
    return v;
}
template <int N>
__device__ __forceinline__ void ldvec(const float* p, float* v) {
    if (N == 1) {
        asm volatile("ld.global.f32 %0, [%1];" : "=f"(v[0]) : "l"(p));
    } else if (N == 2) {
        asm volatile("ld.global.v2.f32 {%0, %1}, [%2];" : "=f"(v[0]), "=f"(v[1]) : "l"(p));
    } else {
#pragma unroll
        for (int i = 0; i < N; i += 4)
            asm volatile("ld.global.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v[i]), "=f"(v[i + 1]), "=f"(v[i + 2]), "=f"(v[i + 3]) : "l"(p + i));
    }
}
template <int N>
__device__ __forceinline__ void stvec(float* p, const float* v) {
    if (N == 1) *p = v[0];
    else if (N == 2) *reinterpret_cast<float2*>(p) = make_float2(v[0], v[1]);
    else
#pragma unroll
        for (int i = 0; i < N; i += 4) *reinterpret_cast<float4*>(p + i) = make_float4(v[i], v[i + 1], v[i + 2], v[i + 3]);
}

// Two fp32 values as packed bf16 high and low parts.
__device__ __forceinline__ void split2(float x, float y, uint32_t& hi, uint32_t& lo) {
    const __nv_bfloat162 h = __floats2bfloat162_rn(x, y);
    hi = *reinterpret_cast<const uint32_t*>(&h);
    const __nv_bfloat162 l = __floats2bfloat162_rn(x - __uint_as_float(hi << 16), y - __uint_as_float(hi & 0xffff0000u));
    lo = *reinterpret_cast<const uint32_t*>(&l);
}
__device__ __forceinline__ void mma16816(float* d, const uint4& a, uint32_t b0, uint32_t b1) {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
                 : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
                 : "r"(a.x), "r"(a.y), "r"(a.z), "r"(a.w), "r"(b0), "r"(b1));
}
__device__ __forceinline__ float flow_over_value(float f, float m, int logspace) {
    if (!logspace) f = (f > 0.0f) ? logf(f) : PCX_NEG_INF;
    return (m == PCX_NEG_INF) ? PCX_NEG_INF : f - m;       // (a flow of -inf stays -inf)
}
// exp and log as the tensor-core kernels take them (ex2 / lg2 approximations), flushing denormals: two instructions
// each.  An exponential under 2^-126 of its column's maximum is zero beside it; fast_log(0) = -inf.
__device__ __forceinline__ float fast_exp(float x) {
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x * 1.4426950408889634f));
    return y;
}
__device__ __forceinline__ float fast_log_plus(float x, float m) {          // log(x) + m
    float y;
    asm("lg2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return fmaf(y, 0.6931471805599453f, m);
}

}  // namespace
