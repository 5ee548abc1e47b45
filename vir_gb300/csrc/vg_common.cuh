// Shared helpers of libvirgpu: status/error plumbing and small device
// utilities (compensated sums, FP64 arithmetic without contraction).
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>
#include <stdio.h>

#include "../../include/virgpu.h"

namespace vg {

// Last error message of the calling host thread.
void set_error(const char *fmt, ...);

// Turns a CUDA error into a status, recording the message.
int cuda_status(cudaError_t e, const char *where);

// Status of the launch just issued (cudaGetLastError).
inline int launch_status(const char *where) {
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) {
        set_error("%s: launch failed: %s", where, cudaGetErrorString(e));
        return VG_ERR_LAUNCH;
    }
    return VG_OK;
}

inline cudaStream_t as_stream(void *s) { return reinterpret_cast<cudaStream_t>(s); }

#define VG_REQUIRE(cond, ...)                  \
    do {                                        \
        if (!(cond)) {                          \
            ::vg::set_error(__VA_ARGS__);       \
            return VG_ERR_ARG;                  \
        }                                       \
    } while (0)

// Kahan-compensated FP32 accumulator (the per-ray / per-pixel sums).
struct Kahan {
    float s = 0.f, c = 0.f;
    __device__ __forceinline__ void add(float v) {
        float y = __fsub_rn(v, c);
        float t = __fadd_rn(s, y);
        c = __fsub_rn(__fsub_rn(t, s), y);
        s = t;
    }
    // another such sum (s, c); the compensation of an infinite one is NaN, which would
    // make it NaN
    __device__ __forceinline__ void merge(float2 q) {
        add(q.x);
        if (q.y == q.y) add(-q.y);
    }
};

// FP64 helpers that keep every operation separately rounded, matching the
// evaluation order of the numpy expressions they restate.
__device__ __forceinline__ double d_mul(double a, double b) { return __dmul_rn(a, b); }
__device__ __forceinline__ double d_add(double a, double b) { return __dadd_rn(a, b); }
__device__ __forceinline__ double d_sub(double a, double b) { return __dsub_rn(a, b); }
__device__ __forceinline__ double d_div(double a, double b) { return __ddiv_rn(a, b); }

// Packed float32 pairs: one instruction each on sm_100 and later.
__device__ __forceinline__ unsigned long long &pk_bits(float2 &a) {
    return reinterpret_cast<unsigned long long &>(a);
}
__device__ __forceinline__ float2 pk_fma(float2 a, float2 b, float2 c) {
    float2 d;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(pk_bits(d)) : "l"(pk_bits(a)), "l"(pk_bits(b)), "l"(pk_bits(c)));
    return d;
}
__device__ __forceinline__ float2 pk_mul(float2 a, float2 b) {
    float2 d;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(pk_bits(d)) : "l"(pk_bits(a)), "l"(pk_bits(b)));
    return d;
}
__device__ __forceinline__ float2 pk_add(float2 a, float2 b) {
    float2 d;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(pk_bits(d)) : "l"(pk_bits(a)), "l"(pk_bits(b)));
    return d;
}
__device__ __forceinline__ float2 pk_add_rd(float2 a, float2 b) {
    float2 d;
    asm("add.rm.f32x2 %0, %1, %2;" : "=l"(pk_bits(d)) : "l"(pk_bits(a)), "l"(pk_bits(b)));
    return d;
}
__device__ __forceinline__ float2 pk_sub(float2 a, float2 b) {  // a - b: -b is exact
    return pk_fma(b, make_float2(-1.f, -1.f), a);
}
__device__ __forceinline__ float2 dup(float a) { return make_float2(a, a); }

// 1 / d to about half an ulp: the hardware's estimate and one Newton step.
__device__ __forceinline__ float recip_n(float d) {
    float r;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(d));
    return fmaf(fmaf(-d, r, 1.0f), r, r);
}

// *p (shared memory) where w > 0, else 0 without reading: lanes that read
// nothing cause no bank conflicts.
__device__ __forceinline__ float lds_if(const float *p, float w) {
    float x = 0.f;
    asm volatile("{\n\t.reg .pred q;\n\tsetp.gt.f32 q, %2, 0f00000000;\n\t@q ld.shared.f32 %0, [%1];\n\t}"
                 : "+f"(x)
                 : "r"((unsigned)__cvta_generic_to_shared(p)), "f"(w)
                 : "memory");  // it reads what stores before it wrote
    return x;
}

// p + j * stride as one instruction.
__device__ __forceinline__ const char *ptr_at(const char *p, unsigned j, unsigned stride) {
    const char *q;
    asm("mad.wide.u32 %0, %1, %2, %3;" : "=l"(q) : "r"(j), "r"(stride), "l"(p));
    return q;
}

constexpr int NSM = 152;  // SMs of the GPU that grids are sized for

inline int ceil_div(long long a, long long b) { return (int)((a + b - 1) / b); }

}  // namespace vg
