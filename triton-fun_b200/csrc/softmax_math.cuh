// Register-level arithmetic shared by the tensor-core attention kernels: exp2 on the special
// function unit, packed fp32x2 operations, 3-input max, 16-bit packing.
#pragma once

#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <stdint.h>

namespace splat {
namespace sm {

__device__ __forceinline__ float ex2(float x) {
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
__device__ __forceinline__ float fmax3(float a, float b, float c) {
    float d;
    asm("max.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c));
    return d;
}
// packed fp32x2 arithmetic: one issue slot for two lanes of work
__device__ __forceinline__ float2 fma2(float2 a, float2 b, float2 c) {
    uint64_t ua = *reinterpret_cast<uint64_t*>(&a), ub = *reinterpret_cast<uint64_t*>(&b),
             uc = *reinterpret_cast<uint64_t*>(&c), ud;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(ud) : "l"(ua), "l"(ub), "l"(uc));
    return *reinterpret_cast<float2*>(&ud);
}
__device__ __forceinline__ float2 add2(float2 a, float2 b) {
    uint64_t ua = *reinterpret_cast<uint64_t*>(&a), ub = *reinterpret_cast<uint64_t*>(&b), ud;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(ud) : "l"(ua), "l"(ub));
    return *reinterpret_cast<float2*>(&ud);
}
__device__ __forceinline__ float2 mul2(float2 a, float2 b) {
    uint64_t ua = *reinterpret_cast<uint64_t*>(&a), ub = *reinterpret_cast<uint64_t*>(&b), ud;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(ud) : "l"(ua), "l"(ub));
    return *reinterpret_cast<float2*>(&ud);
}

template <typename T> __device__ __forceinline__ uint32_t pack2(float a, float b);
template <> __device__ __forceinline__ uint32_t pack2<__half>(float a, float b) {
    __half2 h = __floats2half2_rn(a, b);
    return *reinterpret_cast<uint32_t*>(&h);
}
template <> __device__ __forceinline__ uint32_t pack2<__nv_bfloat16>(float a, float b) {
    __nv_bfloat162 h = __floats2bfloat162_rn(a, b);
    return *reinterpret_cast<uint32_t*>(&h);
}

// The pieces of a softmax step over a row's N scores in registers (attention_wide.cu, attention_duo.cu).
// Band edge: keys outside [lo, hi) become -inf (exp2 -> 0), 32 at a time.
template <int N>
__device__ __forceinline__ void mask_scores(uint32_t (&r)[N], int lo, int hi) {
#pragma unroll
    for (int c = 0; c < N; c += 32) {
        const int a = min(max(lo - c, 0), 32), b = min(max(hi - c, 0), 32);
        const uint32_t valid = (b >= 32 ? ~0u : (1u << b) - 1) & ~(a >= 32 ? ~0u : (1u << a) - 1);
#pragma unroll
        for (int j = 0; j < 32; ++j) r[c + j] = (valid & (1u << j)) ? r[c + j] : 0xff800000u;
    }
}
template <int N>
__device__ __forceinline__ float max_score(const uint32_t (&r)[N]) {
    float mx[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
#pragma unroll
    for (int j = 0; j < N; j += 8)
#pragma unroll
        for (int i = 0; i < 4; ++i) mx[i] = fmax3(mx[i], __uint_as_float(r[j + 2 * i]), __uint_as_float(r[j + 2 * i + 1]));
    return fmaxf(fmaxf(mx[0], mx[1]), fmaxf(mx[2], mx[3]));
}
// N scores c -> probabilities exp2(c scale + offset), packed into p (which may be c's own front), and two halves of their sum.
template <typename T, int N>
__device__ __forceinline__ void exp_scores(const uint32_t* c, uint32_t* p, float2 scale, float2 offset, float2& sum0, float2& sum1) {
#pragma unroll
    for (int j = 0; j < N; j += 4) {
        float2 a0 = fma2(make_float2(__uint_as_float(c[j]), __uint_as_float(c[j + 1])), scale, offset);
        float2 a1 = fma2(make_float2(__uint_as_float(c[j + 2]), __uint_as_float(c[j + 3])), scale, offset);
        a0.x = ex2(a0.x); a0.y = ex2(a0.y); a1.x = ex2(a1.x); a1.y = ex2(a1.y);
        sum0 = add2(sum0, a0);
        sum1 = add2(sum1, a1);
        p[j >> 1] = pack2<T>(a0.x, a0.y);
        p[(j >> 1) + 1] = pack2<T>(a1.x, a1.y);
    }
}

}  // namespace sm
}  // namespace splat
