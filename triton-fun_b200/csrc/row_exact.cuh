// A row's result from the row's own keys alone, by one warp.
//
// The tile kernels multiply whole steps of keys, with probability 0 outside a row's band.  Where V is not finite at a key
// that only other rows of the tile attend to (padding that was never written, an overflow), that is 0 * inf = NaN in
// rows which have nothing to do with it.  A result that is not finite is rare and is noticed at the end for little, so
// the tile kernels multiply as they did and hand such rows to these functions, which give what the row kernels
// (ops_generic.cu) give, NaN or not.  Masking V or the accumulation itself would cost every step.
#pragma once

#include "common.cuh"
#include "softmax_math.cuh"

namespace splat {

// softmax(scale q . K) V over the columns first, first + step, ... (nnz of them).  q: the row; k, v: the head's arrays,
// element (column, c) of K at column * ksc + c * ksk.  Lane l returns columns l, l + 32, l + 64 and l + 96, and the
// maximum and the sum (both in the log2 domain) in `m` and `sum`.
template <typename T>
__device__ __forceinline__ float4 attention_row_sums(const T* q, const T* k, int64_t ksc, int64_t ksk, const T* v, int64_t first,
                                                     int step, int nnz, int d, float scale_log2, float& m, float& sum) {
    const int lane = threadIdx.x & 31;
    float l = 0.f, acc[4] = {0.f, 0.f, 0.f, 0.f};
    m = -INFINITY;
    for (int j = lane; j < nnz; j += 32)
        m = fmaxf(m, dot_strided<T>(q, k + (first + (int64_t)j * step) * ksc, ksk, d) * scale_log2);
    m = warp_max(m);
    for (int j0 = 0; j0 < nnz; j0 += 32) {
        const int64_t col = first + (int64_t)(j0 + lane) * step;
        const float mine = j0 + lane < nnz ? exp2f(dot_strided<T>(q, k + col * ksc, ksk, d) * scale_log2 - m) : 0.f;
        l += mine;
        for (int t = 0; t < min(32, nnz - j0); ++t) {
            const float pt = __shfl_sync(0xffffffffu, mine, t);
            const T* row = v + (first + (int64_t)(j0 + t) * step) * d;
#pragma unroll
            for (int i = 0; i < 4; ++i)
                if (lane + 32 * i < d) acc[i] = fmaf(pt, DT<T>::to_f(row[lane + 32 * i]), acc[i]);
        }
    }
    sum = warp_sum(l);
    const float inv = 1.f / sum;
    return make_float4(acc[0] * inv, acc[1] * inv, acc[2] * inv, acc[3] * inv);
}
template <typename T>
__device__ __noinline__ float4 attention_row(const T* q, const T* k, int64_t ksc, int64_t ksk, const T* v, int64_t first,
                                             int step, int nnz, int d, float scale_log2) {
    float m, sum;
    return attention_row_sums<T>(q, k, ksc, ksk, v, first, step, nnz, d, scale_log2, m, sum);
}
// ... and the row's log-sum-exp to *lse
template <typename T>
__device__ __noinline__ float4 attention_row_lse(const T* q, const T* k, int64_t ksc, int64_t ksk, const T* v, int64_t first,
                                                 int step, int nnz, int d, float scale_log2, float* lse) {
    float m, sum;
    const float4 o = attention_row_sums<T>(q, k, ksc, ksk, v, first, step, nnz, d, scale_log2, m, sum);
    if ((threadIdx.x & 31) == 0) *lse = lse_from_log2(m, sum);
    return o;
}

// sum_j p[j] V[first + j step], as above.
template <typename T>
__device__ __noinline__ float4 spmm_row(const T* p, const T* v, int64_t first, int step, int nnz, int d) {
    const int lane = threadIdx.x & 31;
    float acc[4] = {0.f, 0.f, 0.f, 0.f};
    for (int j = 0; j < nnz; ++j) {
        const float pj = DT<T>::to_f(p[j]);
        const T* row = v + (first + (int64_t)j * step) * d;
#pragma unroll
        for (int i = 0; i < 4; ++i)
            if (lane + 32 * i < d) acc[i] = fmaf(pj, DT<T>::to_f(row[lane + 32 * i]), acc[i]);
    }
    return make_float4(acc[0], acc[1], acc[2], acc[3]);
}

// Lane l's columns of a row, as returned above, to memory.
template <typename T>
__device__ __forceinline__ void store_row(T* row, int d, float4 x) {
    const int lane = threadIdx.x & 31;
    const float v[4] = {x.x, x.y, x.z, x.w};
#pragma unroll
    for (int i = 0; i < 4; ++i)
        if (lane + 32 * i < d) row[lane + 32 * i] = DT<T>::from_f(v[i]);
}

// so_far plus x[0] x[2] and x[1] x[3]: not finite if one of them is not (nor, in vain, if a product overflows).
__device__ __forceinline__ float2 note_nonfinite(float2 so_far, const uint32_t* x) {
    return sm::fma2(make_float2(__uint_as_float(x[0]), __uint_as_float(x[1])),
                    make_float2(__uint_as_float(x[2]), __uint_as_float(x[3])), so_far);
}

}  // namespace splat
