// qi_device.cuh — device-side helpers shared by the engine's kernels.
#pragma once
#include <cuda_runtime.h>
#include <cstdint>

namespace qi {

// Complex arithmetic on the CUDA vector types (float2 / double2).
template <typename T> struct Cx;
template <> struct Cx<float> {
    using V2 = float2;
    __host__ __device__ static inline float2 make(float r, float i) { return make_float2(r, i); }
    __device__ static inline float2 add(float2 a, float2 b) { return make_float2(a.x + b.x, a.y + b.y); }
    __device__ static inline float2 sub(float2 a, float2 b) { return make_float2(a.x - b.x, a.y - b.y); }
    __device__ static inline float2 mul(float2 a, float2 b) {
        return make_float2(fmaf(a.x, b.x, -a.y * b.y), fmaf(a.x, b.y, a.y * b.x));
    }
    // acc + a*b
    __device__ static inline float2 fma(float2 a, float2 b, float2 acc) {
        acc.x = fmaf(a.x, b.x, acc.x);
        acc.x = fmaf(-a.y, b.y, acc.x);
        acc.y = fmaf(a.x, b.y, acc.y);
        acc.y = fmaf(a.y, b.x, acc.y);
        return acc;
    }
};
template <> struct Cx<double> {
    using V2 = double2;
    __host__ __device__ static inline double2 make(double r, double i) { return make_double2(r, i); }
    __device__ static inline double2 add(double2 a, double2 b) { return make_double2(a.x + b.x, a.y + b.y); }
    __device__ static inline double2 sub(double2 a, double2 b) { return make_double2(a.x - b.x, a.y - b.y); }
    __device__ static inline double2 mul(double2 a, double2 b) {
        return make_double2(::fma(a.x, b.x, -a.y * b.y), ::fma(a.x, b.y, a.y * b.x));
    }
    __device__ static inline double2 fma(double2 a, double2 b, double2 acc) {
        acc.x = ::fma(a.x, b.x, acc.x);
        acc.x = ::fma(-a.y, b.y, acc.x);
        acc.y = ::fma(a.x, b.y, acc.y);
        acc.y = ::fma(a.y, b.x, acc.y);
        return acc;
    }
};

// exp(2 pi i f / 2^32) for a phase in fixed-point turns: T1[f >> 22] (T1 = exp(2 pi i j / 1024))
// times exp(i x), x = the remaining 22 bits as an angle (< 2 pi / 1024), from the Taylor
// polynomials of sin and cos to x^5 and x^4 (remainder < 1e-16).
__device__ __forceinline__ float2 turn_phase(uint32_t f, const float2 *T1) {
    const float2 t = T1[f >> 22];
    const float x = (float)(f & 0x3FFFFFu) * 1.46291807926715968e-9f;   // 2 pi / 2^32
    const float x2 = x * x;
    const float s = x * (1.0f - x2 * (1.0f / 6.0f) * (1.0f - x2 * 0.05f));
    const float c = 1.0f - x2 * 0.5f * (1.0f - x2 * (1.0f / 12.0f));
    return make_float2(t.x * c - t.y * s, t.x * s + t.y * c);
}

// Streaming loads for data read exactly once (evict-first in L1/L2).
__device__ static inline float4 ldg_stream(const float4 *p) { return __ldcs(p); }
__device__ static inline double2 ldg_stream(const double2 *p) { return __ldcs(p); }
__device__ static inline float2 ldg_stream(const float2 *p) { return __ldcs(p); }

// Block-wide sum of one double (blockDim.x a multiple of 32, <= 1024, or 1, 2, 4, 8 or 16).
__device__ static inline double block_sum(double v) {
    __shared__ double warp_part[32];
    if (blockDim.x < 32) {   // less than a warp: only the lanes that exist take part
        const unsigned lanes = (1u << blockDim.x) - 1u;
        for (unsigned o = blockDim.x >> 1; o > 0; o >>= 1) v += __shfl_xor_sync(lanes, v, o);
        return v;
    }
    for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    __syncthreads();   // warp_part may still be read by a previous call
    if (lane == 0) warp_part[wid] = v;
    __syncthreads();
    const int nw = (blockDim.x + 31) >> 5;
    double r = 0.0;
    if (wid == 0) {
        r = lane < nw ? warp_part[lane] : 0.0;
        for (int o = 16; o > 0; o >>= 1) r += __shfl_down_sync(0xffffffffu, r, o);
    }
    return r;   // valid in thread 0
}

// Sum of FP32 values that keeps about 48 bits, two addends at a time: two lanes of a float and the sum of its
// additions' rounding errors (Knuth's two-sum, exact), seven packed FP32 operations.
struct PairSum {
    uint64_t hi = 0, lo = 0;
    static __device__ __forceinline__ uint64_t add2(uint64_t a, uint64_t b) {
        uint64_t d;
        asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
        return d;
    }
    static __device__ __forceinline__ uint64_t sub2(uint64_t a, uint64_t b) {   // a - b, rounded once
        uint64_t d;
        asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(b), "l"(0xbf800000bf800000ull), "l"(a));
        return d;
    }
    __device__ __forceinline__ void add(float a, float b) {
        uint64_t x;
        asm("mov.b64 %0, {%1, %2};" : "=l"(x) : "f"(a), "f"(b));
        const uint64_t s = add2(hi, x), t = sub2(s, hi);
        lo = add2(lo, add2(sub2(hi, sub2(s, t)), sub2(x, t)));
        hi = s;
    }
    __device__ __forceinline__ double total() const {
        const float h0 = __uint_as_float((uint32_t)hi), h1 = __uint_as_float((uint32_t)(hi >> 32));
        const float l0 = __uint_as_float((uint32_t)lo), l1 = __uint_as_float((uint32_t)(lo >> 32));
        // infinities and NaN have no rounding error
        return ((double)h0 + (isfinite(h0) ? l0 : 0.0f)) + ((double)h1 + (isfinite(h1) ? l1 : 0.0f));
    }
};

// Insert a zero bit at each of the `np` ascending positions `pos[]` of w.
__device__ static inline uint64_t insert_zeros(uint64_t w, const int8_t *pos, int np) {
    for (int k = 0; k < np; ++k) {
        const int p = pos[k];
        const uint64_t lo = w & ((1ull << p) - 1);
        w = ((w >> p) << (p + 1)) | lo;
    }
    return w;
}

}  // namespace qi
