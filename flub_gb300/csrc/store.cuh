// Storage types of the V-cycle levels: FP32, or FP16 for the mixed-precision
// preconditioner (values are converted to FP32 on load and all arithmetic is
// FP32; FP16 rounding happens only on store).
//
// ld*_in load what an earlier kernel of the stream wrote: residuals and
// corrections.  Under programmatic dependent launch a block is resident while
// that kernel still writes them, so they are not read-only for the kernel's
// life, as the read-only path (__ldg, and what the compiler makes of const
// __restrict__ parameters) asks; volatile, they stay behind griddepcontrol.wait.
#pragma once

#include <cuda_fp16.h>

#include <cstdint>

namespace flub {

template <typename T>
struct St;

template <>
struct St<float> {
    static __device__ __forceinline__ float ld(const float *p) { return *p; }
    static __device__ __forceinline__ float ld_in(const float *p) {
        float v;
        asm volatile("ld.global.f32 %0, [%1];" : "=f"(v) : "l"(__cvta_generic_to_global(p)));
        return v;
    }
    static __device__ __forceinline__ void st(float *p, float v) { *p = v; }
    static __device__ __forceinline__ void ld8(const float *p, float o[8]) {
        const float4 a = reinterpret_cast<const float4 *>(p)[0], b = reinterpret_cast<const float4 *>(p)[1];
        o[0] = a.x; o[1] = a.y; o[2] = a.z; o[3] = a.w; o[4] = b.x; o[5] = b.y; o[6] = b.z; o[7] = b.w;
    }
    static __device__ __forceinline__ void ld8_in(const float *p, float o[8]) {
        ld4_in(p, o);
        ld4_in(p + 4, o + 4);
    }
    static __device__ __forceinline__ void ld4_in(const float *p, float *o) {
        asm volatile("ld.global.v4.f32 {%0, %1, %2, %3}, [%4];"
                     : "=f"(o[0]), "=f"(o[1]), "=f"(o[2]), "=f"(o[3])
                     : "l"(__cvta_generic_to_global(p)));
    }
    static __device__ __forceinline__ void ld4(const float *p, float o[4]) {
        const float4 a = *reinterpret_cast<const float4 *>(p);
        o[0] = a.x; o[1] = a.y; o[2] = a.z; o[3] = a.w;
    }
    static __device__ __forceinline__ void ld2_in(const float *p, float o[2]) {
        asm volatile("ld.global.v2.f32 {%0, %1}, [%2];" : "=f"(o[0]), "=f"(o[1]) : "l"(__cvta_generic_to_global(p)));
    }
    static __device__ __forceinline__ void ld2(const float *p, float o[2]) {
        const float2 a = *reinterpret_cast<const float2 *>(p);
        o[0] = a.x; o[1] = a.y;
    }
    // L2-only loads (ld.global.cg) of data other blocks wrote earlier in the
    // same launch (persistent kernels)
    static __device__ __forceinline__ float ld_cg(const float *p) { return __ldcg(p); }
    static __device__ __forceinline__ void ld2_cg(const float *p, float o[2]) {
        const float2 a = __ldcg(reinterpret_cast<const float2 *>(p));
        o[0] = a.x; o[1] = a.y;
    }
    static __device__ __forceinline__ void ld4_cg(const float *p, float o[4]) {
        const float4 a = __ldcg(reinterpret_cast<const float4 *>(p));
        o[0] = a.x; o[1] = a.y; o[2] = a.z; o[3] = a.w;
    }
    static __device__ __forceinline__ void ld8_cg(const float *p, float o[8]) {
        const float4 a = __ldcg(reinterpret_cast<const float4 *>(p)), b = __ldcg(reinterpret_cast<const float4 *>(p) + 1);
        o[0] = a.x; o[1] = a.y; o[2] = a.z; o[3] = a.w; o[4] = b.x; o[5] = b.y; o[6] = b.z; o[7] = b.w;
    }
    static __device__ __forceinline__ void st8(float *p, const float v[8]) {
        reinterpret_cast<float4 *>(p)[0] = make_float4(v[0], v[1], v[2], v[3]);
        reinterpret_cast<float4 *>(p)[1] = make_float4(v[4], v[5], v[6], v[7]);
    }
    static __device__ __forceinline__ void st4(float *p, const float v[4]) {
        *reinterpret_cast<float4 *>(p) = make_float4(v[0], v[1], v[2], v[3]);
    }
    // 32 bytes in one access; p is 32-byte aligned.  A warp whose lanes hold
    // consecutive groups then touches each 128-byte line once, not twice.
    static __device__ __forceinline__ void ld8_wide(const float *p, float o[8]) {
        asm volatile("ld.global.v8.f32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                     : "=f"(o[0]), "=f"(o[1]), "=f"(o[2]), "=f"(o[3]), "=f"(o[4]), "=f"(o[5]), "=f"(o[6]), "=f"(o[7])
                     : "l"(__cvta_generic_to_global(p)));
    }
    static __device__ __forceinline__ void st8_wide(float *p, const float v[8]) {
        asm volatile("st.global.v8.f32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"l"(__cvta_generic_to_global(p)),
                     "f"(v[0]), "f"(v[1]), "f"(v[2]), "f"(v[3]), "f"(v[4]), "f"(v[5]), "f"(v[6]), "f"(v[7])
                     : "memory");
    }
    // the same where p may be a caller's array, 16-byte aligned only
    static __device__ __forceinline__ void ld8_any(const float *p, float o[8]) {
        if (reinterpret_cast<uintptr_t>(p) & 16) ld8(p, o); else ld8_wide(p, o);
    }
    static __device__ __forceinline__ void st8_any(float *p, const float v[8]) {
        if (reinterpret_cast<uintptr_t>(p) & 16) st8(p, v); else st8_wide(p, v);
    }
};

template <>
struct St<__half> {
    static __device__ __forceinline__ float ld(const __half *p) { return __half2float(*p); }
    static __device__ __forceinline__ float ld_in(const __half *p) {
        unsigned short u;
        asm volatile("ld.global.u16 %0, [%1];" : "=h"(u) : "l"(__cvta_generic_to_global(p)));
        return __half2float(__ushort_as_half(u));
    }
    static __device__ __forceinline__ void st(__half *p, float v) { *p = __float2half_rn(v); }
    static __device__ __forceinline__ void unpack8(uint4 u, float o[8]) {
        const __half2 *h = reinterpret_cast<const __half2 *>(&u);
#pragma unroll
        for (int q = 0; q < 4; q++) {
            const float2 f = __half22float2(h[q]);
            o[2 * q] = f.x;
            o[2 * q + 1] = f.y;
        }
    }
    static __device__ __forceinline__ void ld8(const __half *p, float o[8]) {
        unpack8(*reinterpret_cast<const uint4 *>(p), o);
    }
    static __device__ __forceinline__ void ld8_in(const __half *p, float o[8]) {
        uint4 u;
        asm volatile("ld.global.v4.u32 {%0, %1, %2, %3}, [%4];"
                     : "=r"(u.x), "=r"(u.y), "=r"(u.z), "=r"(u.w)
                     : "l"(__cvta_generic_to_global(p)));
        unpack8(u, o);
    }
    static __device__ __forceinline__ void ld8_any(const __half *p, float o[8]) { ld8(p, o); }
    static __device__ __forceinline__ void ld4_in(const __half *p, float o[4]) {
        uint2 u;
        asm volatile("ld.global.v2.u32 {%0, %1}, [%2];" : "=r"(u.x), "=r"(u.y) : "l"(__cvta_generic_to_global(p)));
        const __half2 *h = reinterpret_cast<const __half2 *>(&u);
        const float2 a = __half22float2(h[0]), b = __half22float2(h[1]);
        o[0] = a.x; o[1] = a.y; o[2] = b.x; o[3] = b.y;
    }
    static __device__ __forceinline__ void ld4(const __half *p, float o[4]) {
        const uint2 u = *reinterpret_cast<const uint2 *>(p);
        const __half2 *h = reinterpret_cast<const __half2 *>(&u);
        const float2 a = __half22float2(h[0]), b = __half22float2(h[1]);
        o[0] = a.x; o[1] = a.y; o[2] = b.x; o[3] = b.y;
    }
    static __device__ __forceinline__ void ld2_in(const __half *p, float o[2]) {
        unsigned int u;
        asm volatile("ld.global.u32 %0, [%1];" : "=r"(u) : "l"(__cvta_generic_to_global(p)));
        const float2 a = __half22float2(*reinterpret_cast<const __half2 *>(&u));
        o[0] = a.x; o[1] = a.y;
    }
    static __device__ __forceinline__ void ld2(const __half *p, float o[2]) {
        const float2 a = __half22float2(*reinterpret_cast<const __half2 *>(p));
        o[0] = a.x; o[1] = a.y;
    }
    static __device__ __forceinline__ float ld_cg(const __half *p) {
        const unsigned short u = __ldcg(reinterpret_cast<const unsigned short *>(p));
        return __half2float(__ushort_as_half(u));
    }
    static __device__ __forceinline__ void ld2_cg(const __half *p, float o[2]) {
        const unsigned int u = __ldcg(reinterpret_cast<const unsigned int *>(p));
        const float2 a = __half22float2(*reinterpret_cast<const __half2 *>(&u));
        o[0] = a.x; o[1] = a.y;
    }
    static __device__ __forceinline__ void ld4_cg(const __half *p, float o[4]) {
        const uint2 u = __ldcg(reinterpret_cast<const uint2 *>(p));
        const __half2 *h = reinterpret_cast<const __half2 *>(&u);
        const float2 a = __half22float2(h[0]), b = __half22float2(h[1]);
        o[0] = a.x; o[1] = a.y; o[2] = b.x; o[3] = b.y;
    }
    static __device__ __forceinline__ void ld8_cg(const __half *p, float o[8]) {
        unpack8(__ldcg(reinterpret_cast<const uint4 *>(p)), o);
    }
    static __device__ __forceinline__ void st8(__half *p, const float v[8]) {
        uint4 u;
        __half2 *h = reinterpret_cast<__half2 *>(&u);
#pragma unroll
        for (int q = 0; q < 4; q++) h[q] = __floats2half2_rn(v[2 * q], v[2 * q + 1]);
        *reinterpret_cast<uint4 *>(p) = u;
    }
    static __device__ __forceinline__ void st8_any(__half *p, const float v[8]) { st8(p, v); }
    static __device__ __forceinline__ void st4(__half *p, const float v[4]) {
        uint2 u;
        __half2 *h = reinterpret_cast<__half2 *>(&u);
        h[0] = __floats2half2_rn(v[0], v[1]);
        h[1] = __floats2half2_rn(v[2], v[3]);
        *reinterpret_cast<uint2 *>(p) = u;
    }
};

}  // namespace flub
