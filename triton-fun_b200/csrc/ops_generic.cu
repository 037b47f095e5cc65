// CUDA-core kernels for SDDMM, row softmax, SpMM and a fused chain over ACSR.  They consume only
// the per-row affine metadata, so they are correct for every metadata the builder can produce
// (any stride, ragged rows, empty rows) and for fp32 inputs with true fp32 FMA.  The tensor-core
// band kernel covers the regular, 16-bit cases; these kernels are the general path.
//
// Work decomposition: one warp per sparse row.
//   SDDMM  : lanes own slots (slot j -> dense column start + j*stride); the Q row sits in shared
//            memory as fp32 and is broadcast; a lane streams its K row with 16-byte loads when K is
//            row-contiguous, or walks a contiguous K^T with lane-coalesced scalar loads.
//   SpMM   : the warp is split into G groups of d/vec lanes; group g handles slots j == g (mod G)
//            and each lane accumulates one 16-byte chunk of the output row; groups are reduced
//            with shuffles at the end.
//   fused  : 32 slots at a time -- scores as in SDDMM, online max/sum with exp2 and the softmax
//            scale folded into the exponent, then the SpMM accumulation with the probabilities
//            broadcast by shuffle.
#include <limits.h>

#include "common.cuh"
#include "softmax_math.cuh"

namespace splat {

constexpr int kWarpsPerBlock = 4;

// Checked-index mode (splat_debug_check_indices): while a word is registered, every dense column
// these kernels derive from the row metadata is compared with [0, n_cols); a column outside it is
// clamped to the nearest valid one before it is dereferenced and the kernel's code is recorded in
// the word (the first code stays).  Off (null) the comparison is skipped.
static int32_t* g_index_check = nullptr;
bool index_check_on() { return g_index_check != nullptr; }
enum : int32_t { kIndexSddmm = 71, kIndexSpmm = 72, kIndexFused = 73 };

__device__ __forceinline__ int64_t slot_col(const RowAffine& ra, int j, int64_t n_cols, int32_t* check,
                                            int32_t code) {
    int64_t col = (int64_t)ra.start + (int64_t)j * ra.stride;
    if (check != nullptr && (col < 0 || col >= n_cols)) {
        atomicCAS(check, 0, code);
        col = col < 0 ? 0 : n_cols - 1;
    }
    return col;
}

// ---------------------------------------------------------------------------------------------
// dot(Q row in shared memory, K[col, :]).  A column of K^T is read with kAhead loads on their way at a time: 16 in SDDMM
// (fp32 B2 H13 L256 d128 strided 15: 24.7 -> 12.4 us); the fused kernel, which has more registers to keep, loses
// occupancy by it (B3 H15 L1280 d64 strided 118: 140 -> 165 us).
// ---------------------------------------------------------------------------------------------
template <typename T, bool kRowContig, int kAhead = 1>
__device__ __forceinline__ float dot_qk(const float* __restrict__ qs, const T* __restrict__ kbh,
                                        int64_t col, int d, int64_t ksc, int64_t ksk) {
    float acc = 0.f;
    if constexpr (kRowContig) {
        const T* kr = kbh + col * ksc;
        constexpr int V = DT<T>::kVec;
        float tmp[V];
        for (int k0 = 0; k0 < d; k0 += V) {
            load16_as_float(kr + k0, tmp);
#pragma unroll
            for (int t = 0; t < V; ++t) acc = fmaf(qs[k0 + t], tmp[t], acc);
        }
    } else {
        const T* kc = kbh + col * ksc;
        int k0 = 0;
        if constexpr (kAhead > 1) {
            for (; k0 + kAhead <= d; k0 += kAhead) {
                T tmp[kAhead];
#pragma unroll
                for (int u = 0; u < kAhead; ++u) tmp[u] = kc[(int64_t)(k0 + u) * ksk];
#pragma unroll
                for (int u = 0; u < kAhead; ++u) acc = fmaf(qs[k0 + u], DT<T>::to_f(tmp[u]), acc);
            }
        }
        for (; k0 < d; ++k0) acc = fmaf(qs[k0], DT<T>::to_f(kc[(int64_t)k0 * ksk]), acc);
    }
    return acc;
}

template <typename T>
__device__ __forceinline__ void stage_q_row(float* qs, const T* __restrict__ qrow, int d, int lane) {
    for (int k0 = lane; k0 < d; k0 += 32) qs[k0] = DT<T>::to_f(qrow[k0]);
    __syncwarp();
}

// ---------------------------------------------------------------------------------------------
// SDDMM
// ---------------------------------------------------------------------------------------------
template <typename T, bool kRowContig>
__global__ void __launch_bounds__(kWarpsPerBlock * 32)
sddmm_rows_kernel(const T* __restrict__ q, const T* __restrict__ k, int64_t ksb, int64_t ksc,
                  int64_t ksk, T* __restrict__ out, const float* __restrict__ lin,
                  const float* __restrict__ tr, const float* __restrict__ nnzs, int64_t total_rows,
                  int64_t n_rows, int64_t n_cols, int d, int trailing, int32_t* check) {
    depend_wait();
    depend_release();
    extern __shared__ float smem_q[];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int64_t grow = (int64_t)blockIdx.x * kWarpsPerBlock + warp;
    if (grow >= total_rows) return;
    const int64_t bh = grow / n_rows, row = grow % n_rows;
    float* qs = smem_q + (size_t)warp * d;
    stage_q_row(qs, q + grow * d, d, lane);
    const RowAffine ra = row_affine(lin, tr, nnzs, row);
    const T* kbh = k + bh * ksb;
    T* orow = out + grow * trailing;
    for (int j = lane; j < trailing; j += 32) {
        float v = 0.f;
        if (j < ra.nnz) v = dot_qk<T, kRowContig, 16>(qs, kbh, slot_col(ra, j, n_cols, check, kIndexSddmm),
                                                  d, ksc, ksk);
        orow[j] = DT<T>::from_f(v);
    }
}

// ---------------------------------------------------------------------------------------------
// Row softmax.  G lanes hold a row in registers, NV 16-byte pieces each (R rows of short ones); all loads are issued
// before the first reduction, so that enough bytes are in flight to keep HBM busy.  Few lanes per row: the
// shuffles of the two reductions and a row's fixed work (its number of non-zeros, addresses, a division) are per
// lane and row, and with 32 lanes and one piece each they were two thirds of the instructions, at 57 % of the
// issue slots.  Long rows: several warps, which exchange two numbers through shared memory.  The pieces
// are those of the array, not of the row: a row that begins inside a piece (odd trailing dimensions) masks
// the neighbours' elements when reading, and stores its first and last piece element by element.  Rows
// longer than kSoftmaxMaxPieces take the loop kernel, which reads a row three times.
// 262 144 rows, us, with a warp per row -> now: T = 35 fp16 71.5 -> 20.8, 64 60.8 -> 14.9, 256 59.7 -> 41.1
// (6.5 TB/s), 257 99.8 -> 52.2, 1024 184 -> 164; T = 257 fp32 118.5 -> 79.9 (6.7 TB/s); 65 536 rows, T = 4096: fp16
// 339 -> 186, fp32 855 -> 316.
// ---------------------------------------------------------------------------------------------
constexpr int kSoftmaxWarps = 8;
constexpr int kSoftmaxMaxPieces = 8 * 32 * kSoftmaxWarps;

template <typename T, int G, int NV, int R>
__global__ void __launch_bounds__(kSoftmaxWarps * 32)
softmax_rows_kernel(const T* s, T* p, const float* __restrict__ nnzs, int64_t total_rows, int64_t n_rows, int trailing,
                    int lead, float scale_log2e) {
    depend_wait();
    depend_release();
    constexpr int V = DT<T>::kVec;
    constexpr int kRows = kSoftmaxWarps * 32 / G;              // rows side by side in the block
    __shared__ float part[2][kSoftmaxWarps];
    const int lane = threadIdx.x & (G - 1);
    const int64_t grow0 = (int64_t)blockIdx.x * (R * kRows) + threadIdx.x / G;
    // `m` or `sum` of the row's other warps, if it has more than one
    auto across_warps = [&](int which, float x, auto op) {
        if (G <= 32) return x;
        const int warp = threadIdx.x >> 5, first_warp = warp & ~(G / 32 - 1);
        if ((threadIdx.x & 31) == 0) part[which][warp] = x;
        __syncthreads();
        x = part[which][first_warp];
#pragma unroll
        for (int w = 1; w < G / 32; ++w) x = op(x, part[which][first_warp + w]);
        return x;
    };
    const int64_t in_head0 = total_rows <= UINT_MAX ? (uint32_t)grow0 % (uint32_t)n_rows : grow0 % n_rows;
    uint4 raw[R][NV];
    int first[R], nnz[R];       // slot of this lane's first element
#pragma unroll
    for (int r = 0; r < R; ++r) {
        nnz[r] = 0;
        // s and p are rounded down to 16 bytes; `lead` elements were lost by that
        const int64_t e = lead + (grow0 + r * kRows) * trailing;
        first[r] = lane * V - (int)(e & (V - 1));
        if (grow0 + r * kRows < total_rows) {
            int64_t in_head = in_head0 + r * kRows;
            while (in_head >= n_rows) in_head -= n_rows;
            const int n = (int)rintf(__ldg(nnzs + in_head));
            nnz[r] = n < 0 ? 0 : (n > trailing ? trailing : n);
        }
        const T* row = s + (e & ~(int64_t)(V - 1)) + lane * V;
#pragma unroll
        for (int v = 0; v < NV; ++v)
            if (first[r] + v * G * V < nnz[r] && first[r] + v * G * V > -V)
                raw[r][v] = *reinterpret_cast<const uint4*>(row + v * G * V);
    }
    float2 vals[R][NV][V / 2];
    float m[R], sum[R];
    const float2 sc2 = make_float2(scale_log2e, scale_log2e);
    // scaled scores of a piece; elements outside the row's non-zeros -inf (a warp whose pieces are all inside them
    // skips that)
    auto scores = [&](int r, int v, float2 (&x)[V / 2]) {
        const T* e = reinterpret_cast<const T*>(&raw[r][v]);
#pragma unroll
        for (int t = 0; t < V / 2; ++t) x[t] = sm::mul2(make_float2(DT<T>::to_f(e[2 * t]), DT<T>::to_f(e[2 * t + 1])), sc2);
        const int j = first[r] + v * G * V;
        if (!__all_sync(0xffffffffu, j >= 0 && j + V <= nnz[r])) {
#pragma unroll
            for (int t = 0; t < V / 2; ++t) {
                x[t].x = j + 2 * t >= 0 && j + 2 * t < nnz[r] ? x[t].x : -INFINITY;
                x[t].y = j + 2 * t + 1 >= 0 && j + 2 * t + 1 < nnz[r] ? x[t].y : -INFINITY;
            }
        }
    };
    auto exponentials = [&](float2 (&x)[V / 2], float mm) {
        const float2 nm = make_float2(-mm, -mm);
#pragma unroll
        for (int t = 0; t < V / 2; ++t) {
            x[t] = sm::add2(x[t], nm);
            // (16-bit results: flushing exponentials below 2^-126 to zero changes nothing)
            x[t].x = sizeof(T) == 2 ? sm::ex2(x[t].x) : exp2f(x[t].x);
            x[t].y = sizeof(T) == 2 ? sm::ex2(x[t].y) : exp2f(x[t].y);
        }
    };
#pragma unroll
    for (int r = 0; r < R; ++r) {
        m[r] = -INFINITY;
#pragma unroll
        for (int v = 0; v < NV; ++v) {
            float2 (&x)[V / 2] = vals[r][v];
            scores(r, v, x);
#pragma unroll
            for (int t = 0; t < V / 2; ++t) m[r] = sm::fmax3(m[r], x[t].x, x[t].y);
        }
    }
#pragma unroll
    for (int o = (G < 32 ? G : 32) / 2; o > 0; o >>= 1)
#pragma unroll
        for (int r = 0; r < R; ++r) m[r] = fmaxf(m[r], __shfl_xor_sync(0xffffffffu, m[r], o));
#pragma unroll
    for (int r = 0; r < R; ++r) {
        m[r] = across_warps(0, m[r], [](float a, float b) { return fmaxf(a, b); });
        m[r] = m[r] == -INFINITY ? 0.f : m[r];
        float2 acc = make_float2(0.f, 0.f);
#pragma unroll
        for (int v = 0; v < NV; ++v) {
            float2 (&x)[V / 2] = vals[r][v];
            exponentials(x, m[r]);
#pragma unroll
            for (int t = 0; t < V / 2; ++t) acc = sm::add2(acc, x[t]);
        }
        sum[r] = acc.x + acc.y;
    }
#pragma unroll
    for (int o = (G < 32 ? G : 32) / 2; o > 0; o >>= 1)
#pragma unroll
        for (int r = 0; r < R; ++r) sum[r] += __shfl_xor_sync(0xffffffffu, sum[r], o);
#pragma unroll
    for (int r = 0; r < R; ++r) {
        sum[r] = across_warps(1, sum[r], [](float a, float b) { return a + b; });
        const float inv = sum[r] > 0.f ? 1.f / sum[r] : 0.f;
        const float2 inv2 = make_float2(inv, inv);
        const int64_t e = lead + (grow0 + r * kRows) * trailing;
        T* row = p + (e & ~(int64_t)(V - 1)) + lane * V;
#pragma unroll
        for (int v = 0; v < NV; ++v) {
            const int j0 = grow0 + r * kRows < total_rows ? first[r] + v * G * V : trailing;
            float2 (&x)[V / 2] = vals[r][v];
#pragma unroll
            for (int t = 0; t < V / 2; ++t) x[t] = sm::mul2(x[t], inv2);
            const float* out = reinterpret_cast<const float*>(&x[0]);
            if (j0 >= 0 && j0 + V <= trailing) {
                store16_from_float(row + v * G * V, out);
            } else if (j0 > -V && j0 < trailing) {
#pragma unroll
                for (int t = 0; t < V; ++t)
                    if (j0 + t >= 0 && j0 + t < trailing) row[v * G * V + t] = DT<T>::from_f(out[t]);
            }
        }
    }
}

template <typename T>
__global__ void __launch_bounds__(kWarpsPerBlock * 32)
softmax_rows_loop_kernel(const T* s, T* p,
                         const float* __restrict__ nnzs, int64_t total_rows, int64_t n_rows,
                         int trailing, float scale_log2e) {
    depend_wait();
    depend_release();
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int64_t grow = (int64_t)blockIdx.x * kWarpsPerBlock + warp;
    if (grow >= total_rows) return;
    int nnz = (int)rintf(__ldg(nnzs + grow % n_rows));
    nnz = nnz < 0 ? 0 : (nnz > trailing ? trailing : nnz);
    const T* srow = s + grow * trailing;
    T* prow = p + grow * trailing;
    float m = -INFINITY;
    for (int j = lane; j < nnz; j += 32) m = fmaxf(m, DT<T>::to_f(srow[j]) * scale_log2e);
    m = warp_max(m);
    float sum = 0.f;
    for (int j = lane; j < nnz; j += 32) sum += exp2f(DT<T>::to_f(srow[j]) * scale_log2e - m);
    sum = warp_sum(sum);
    const float inv = sum > 0.f ? 1.f / sum : 0.f;
    // s and p may alias: every element is read by the lane that overwrites it
    for (int j = lane; j < trailing; j += 32) {
        float v = 0.f;
        if (j < nnz) v = exp2f(DT<T>::to_f(srow[j]) * scale_log2e - m) * inv;
        prow[j] = DT<T>::from_f(v);
    }
}

// ---------------------------------------------------------------------------------------------
// SpMM accumulation helpers: the warp is G groups of LPG lanes; lane owns one 16-byte chunk.
// ---------------------------------------------------------------------------------------------
template <typename T>
__device__ __forceinline__ void accum_v(float* acc, float pv, const T* __restrict__ vrow_chunk) {
    constexpr int V = DT<T>::kVec;
    float tmp[V];
    load16_as_float(vrow_chunk, tmp);
#pragma unroll
    for (int t = 0; t < V; ++t) acc[t] = fmaf(pv, tmp[t], acc[t]);
}

template <int V>
__device__ __forceinline__ void reduce_groups(float* acc, int lpg) {
    for (int o = lpg; o < 32; o <<= 1)
#pragma unroll
        for (int t = 0; t < V; ++t) acc[t] += __shfl_xor_sync(0xffffffffu, acc[t], o);
}

// lanes-per-group = d / vec must be a power of two <= 32 (host checks).
template <typename T>
__global__ void __launch_bounds__(kWarpsPerBlock * 32)
spmm_rows_kernel(const T* __restrict__ p, const T* __restrict__ v, T* __restrict__ o,
                 const float* __restrict__ lin, const float* __restrict__ tr,
                 const float* __restrict__ nnzs, int64_t total_rows, int64_t n_rows,
                 int64_t n_cols, int d, int trailing, int32_t* check) {
    depend_wait();
    depend_release();
    constexpr int V = DT<T>::kVec;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int64_t grow = (int64_t)blockIdx.x * kWarpsPerBlock + warp;
    if (grow >= total_rows) return;
    const int64_t bh = grow / n_rows, row = grow % n_rows;
    const RowAffine ra = row_affine(lin, tr, nnzs, row);
    const int nnz = ra.nnz > trailing ? trailing : ra.nnz;
    const int lpg = d / V, G = 32 / lpg, g = lane / lpg, c0 = (lane % lpg) * V;
    const T* prow = p + grow * trailing;
    const T* vbh = v + bh * n_cols * d;
    float acc[V];
#pragma unroll
    for (int t = 0; t < V; ++t) acc[t] = 0.f;
    for (int j0 = 0; j0 < nnz; j0 += 32) {
        const int j = j0 + lane;
        const float pj = j < nnz ? DT<T>::to_f(prow[j]) : 0.f;
        const int lim = min(32, nnz - j0);
        // uniform trip count: every lane takes part in every shuffle
        for (int t0 = 0; t0 < lim; t0 += G) {
            const int t = t0 + g;
            const float pv = __shfl_sync(0xffffffffu, pj, t & 31);
            if (t < lim) {
                const int64_t col = slot_col(ra, j0 + t, n_cols, check, kIndexSpmm);
                accum_v<T>(acc, pv, vbh + col * d + c0);
            }
        }
    }
    reduce_groups<V>(acc, lpg);
    if (g == 0) store16_from_float(o + grow * d + c0, acc);
}

// Scalar SpMM for head dimensions the grouped kernel does not take.
template <typename T>
__global__ void __launch_bounds__(kWarpsPerBlock * 32)
spmm_rows_scalar_kernel(const T* __restrict__ p, const T* __restrict__ v, T* __restrict__ o,
                        const float* __restrict__ lin, const float* __restrict__ tr,
                        const float* __restrict__ nnzs, int64_t total_rows, int64_t n_rows,
                        int64_t n_cols, int d, int trailing, int32_t* check) {
    depend_wait();
    depend_release();
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int64_t grow = (int64_t)blockIdx.x * kWarpsPerBlock + warp;
    if (grow >= total_rows) return;
    const int64_t bh = grow / n_rows, row = grow % n_rows;
    const RowAffine ra = row_affine(lin, tr, nnzs, row);
    const int nnz = ra.nnz > trailing ? trailing : ra.nnz;
    const T* prow = p + grow * trailing;
    const T* vbh = v + bh * n_cols * d;
    for (int c = lane; c < d; c += 32) {
        float acc = 0.f;
        for (int j = 0; j < nnz; ++j) {
            const int64_t col = slot_col(ra, j, n_cols, check, kIndexSpmm);
            acc = fmaf(DT<T>::to_f(prow[j]), DT<T>::to_f(vbh[col * d + c]), acc);
        }
        o[grow * d + c] = DT<T>::from_f(acc);
    }
}

// ---------------------------------------------------------------------------------------------
// Fused SDDMM -> softmax -> SpMM, one warp per row, scores stay in registers.
// ---------------------------------------------------------------------------------------------
template <typename T, bool kRowContig>
__global__ void __launch_bounds__(kWarpsPerBlock * 32)
attention_rows_kernel(const T* __restrict__ q, const T* __restrict__ k, int64_t ksb, int64_t ksc,
                      int64_t ksk, const T* __restrict__ v, T* __restrict__ o,
                      const float* __restrict__ lin, const float* __restrict__ tr,
                      const float* __restrict__ nnzs, int64_t total_rows, int64_t n_rows,
                      int64_t n_cols, int d, float scale_log2e, int32_t* check, float* lse) {
    depend_wait();
    depend_release();
    constexpr int V = DT<T>::kVec;
    extern __shared__ float smem_q[];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int64_t grow = (int64_t)blockIdx.x * kWarpsPerBlock + warp;
    if (grow >= total_rows) return;
    const int64_t bh = grow / n_rows, row = grow % n_rows;
    float* qs = smem_q + (size_t)warp * d;
    stage_q_row(qs, q + grow * d, d, lane);
    const RowAffine ra = row_affine(lin, tr, nnzs, row);
    const T* kbh = k + bh * ksb;
    const T* vbh = v + bh * n_cols * d;
    const int lpg = d / V, G = 32 / lpg, g = lane / lpg, c0 = (lane % lpg) * V;
    float acc[V];
#pragma unroll
    for (int t = 0; t < V; ++t) acc[t] = 0.f;
    float m = -INFINITY, l = 0.f;
    for (int j0 = 0; j0 < ra.nnz; j0 += 32) {
        const int j = j0 + lane;
        const bool valid = j < ra.nnz;
        float sc = -INFINITY;
        const int64_t col = valid ? slot_col(ra, j, n_cols, check, kIndexFused) : 0;
        if (valid) sc = dot_qk<T, kRowContig>(qs, kbh, col, d, ksc, ksk) * scale_log2e;
        const float m_new = fmaxf(m, warp_max(sc));      // finite: lane 0 of every chunk is valid
        const float corr = exp2f(m - m_new);              // 0 on the first chunk
        const float pj = valid ? exp2f(sc - m_new) : 0.f;
        l = l * corr + warp_sum(pj);
        m = m_new;
#pragma unroll
        for (int t = 0; t < V; ++t) acc[t] *= corr;
        const int lim = min(32, ra.nnz - j0);
        for (int t0 = 0; t0 < lim; t0 += G) {
            const int t = t0 + g;
            const float pv = __shfl_sync(0xffffffffu, pj, t & 31);
            if (t < lim) {
                const int64_t ct = slot_col(ra, j0 + t, n_cols, check, kIndexFused);
                accum_v<T>(acc, pv, vbh + ct * d + c0);
            }
        }
    }
    reduce_groups<V>(acc, lpg);
    if (lse != nullptr && lane == 0) lse[grow] = lse_from_log2(m, l);
    if (g == 0) {
        const float inv = l > 0.f ? 1.f / l : 0.f;
#pragma unroll
        for (int t = 0; t < V; ++t) acc[t] *= inv;
        store16_from_float(o + grow * d + c0, acc);
    }
}

// ---------------------------------------------------------------------------------------------
// (BH, d, L) -> (BH, L, d), 16-bit elements: 64 columns x all of d per CTA through shared memory, coalesced
// 4-byte (2-byte for odd L) reads along L and 4-byte writes along d.  A row of the staging tile is d + 2
// elements, an odd number of words: neither direction conflicts more than twofold.
// ---------------------------------------------------------------------------------------------
constexpr int kTransCols = 64;
__global__ void __launch_bounds__(256)
transpose_16_kernel(const uint16_t* __restrict__ in, uint16_t* __restrict__ out, int d, int n_cols, int wide) {
    depend_wait();
    depend_release();
    extern __shared__ uint16_t s_t[];
    const int pitch = d + 2;
    const int64_t head = (int64_t)blockIdx.y * d * n_cols;
    const int l0 = blockIdx.x * kTransCols, n = min(kTransCols, n_cols - l0);
    in += head + l0;
    if (wide) {       // n_cols even: row starts are 4-byte aligned
        for (int i = threadIdx.x; i < d * (kTransCols / 2); i += 256) {
            const int c = i / (kTransCols / 2), l = (i % (kTransCols / 2)) * 2;
            if (l < n) {
                const uint32_t v = *reinterpret_cast<const uint32_t*>(in + (int64_t)c * n_cols + l);
                s_t[l * pitch + c] = (uint16_t)v;
                s_t[(l + 1) * pitch + c] = (uint16_t)(v >> 16);
            }
        }
    } else {
        for (int i = threadIdx.x; i < d * kTransCols; i += 256) {
            const int c = i / kTransCols, l = i % kTransCols;
            if (l < n) s_t[l * pitch + c] = in[(int64_t)c * n_cols + l];
        }
    }
    __syncthreads();
    uint32_t* o = reinterpret_cast<uint32_t*>(out + head + (int64_t)l0 * d);
    const int half = d / 2;
    for (int i = threadIdx.x; i < n * half; i += 256) {
        const int l = i / half, c = i % half;
        o[i] = *reinterpret_cast<const uint32_t*>(s_t + l * pitch + 2 * c);
    }
}

// ---------------------------------------------------------------------------------------------
// Host dispatch
// ---------------------------------------------------------------------------------------------
static bool grouped_d_ok(int64_t d, int vec) {
    if (d % vec) return false;
    int64_t lpg = d / vec;
    return lpg >= 1 && lpg <= 32 && (lpg & (lpg - 1)) == 0;
}

template <typename T>
static int32_t sddmm_t(const void* q, const void* k, int64_t ksb, int64_t ksc, int64_t ksk,
                       void* out, const float* lin, const float* tr, const float* nnzs, int64_t bh,
                       int64_t n_rows, int64_t n_cols, int64_t d, int64_t trailing, cudaStream_t st) {
    const int64_t total = bh * n_rows;
    const unsigned grid = (unsigned)((total + kWarpsPerBlock - 1) / kWarpsPerBlock);
    const size_t smem = (size_t)kWarpsPerBlock * d * sizeof(float);
    const bool contig = ksk == 1 && (d % DT<T>::kVec == 0) && aligned16(k) &&
                        (ksc % DT<T>::kVec == 0) && (ksb % DT<T>::kVec == 0);
    if (contig)
        return launch_kernel(sddmm_rows_kernel<T, true>, grid, kWarpsPerBlock * 32, smem, st,
            (const T*)q, (const T*)k, ksb, ksc, ksk, (T*)out, lin, tr, nnzs, total, n_rows, n_cols, (int)d,
            (int)trailing, g_index_check);
    return launch_kernel(sddmm_rows_kernel<T, false>, grid, kWarpsPerBlock * 32, smem, st,
            (const T*)q, (const T*)k, ksb, ksc, ksk, (T*)out, lin, tr, nnzs, total, n_rows, n_cols, (int)d,
            (int)trailing, g_index_check);
}

template <typename T>
static int32_t softmax_t(const void* s, void* p, const float* nnzs, int64_t bh, int64_t n_rows,
                         int64_t trailing, float scale, cudaStream_t st) {
    const int64_t total = bh * n_rows;
    constexpr int V = DT<T>::kVec;
    const uintptr_t sa = reinterpret_cast<uintptr_t>(s), pa = reinterpret_cast<uintptr_t>(p);
    const int lead = (int)(sa & 15) / (int)sizeof(T);
    // pieces a row can reach into: its own, and one more where rows do not begin with a piece
    const int64_t pieces = (trailing + V - 1) / V + (lead != 0 || trailing % V != 0 ? 1 : 0);
    const bool same = (sa & 15) == (pa & 15) && (sa & 15) % sizeof(T) == 0 && pieces <= kSoftmaxMaxPieces;
    const T* sb = reinterpret_cast<const T*>(sa & ~(uintptr_t)15);
    T* pb = reinterpret_cast<T*>(pa & ~(uintptr_t)15);
    auto go = [&](auto kern, int per_block) {
        return launch_kernel(kern, (unsigned)((total + per_block - 1) / per_block), kSoftmaxWarps * 32, 0, st,
            sb, pb, nnzs, total, n_rows, (int)trailing, lead, scale * kLog2e);
    };
    if (!same)
        return launch_kernel(softmax_rows_loop_kernel<T>, (unsigned)((total + kWarpsPerBlock - 1) / kWarpsPerBlock),
                             kWarpsPerBlock * 32, 0, st,
            (const T*)s, (T*)p, nnzs, total, n_rows, (int)trailing, scale * kLog2e);
    // as few lanes per row as hold it in five pieces each, but eight at least (128 contiguous bytes)
    if (pieces <= 8) return go(softmax_rows_kernel<T, 8, 1, 4>, 128);
    if (pieces <= 16) return go(softmax_rows_kernel<T, 8, 2, 2>, 64);
    if (pieces <= 24) return go(softmax_rows_kernel<T, 8, 3, 1>, 32);
    if (pieces <= 32) return go(softmax_rows_kernel<T, 8, 4, 1>, 32);
    if (pieces <= 40) return go(softmax_rows_kernel<T, 8, 5, 1>, 32);
    if (pieces <= 64) return go(softmax_rows_kernel<T, 16, 4, 1>, 16);
    if (pieces <= 80) return go(softmax_rows_kernel<T, 16, 5, 1>, 16);
    if (pieces <= 96) return go(softmax_rows_kernel<T, 32, 3, 1>, 8);
    if (pieces <= 128) return go(softmax_rows_kernel<T, 32, 4, 1>, 8);
    if (pieces <= 160) return go(softmax_rows_kernel<T, 32, 5, 1>, 8);
    if (pieces <= 192) return go(softmax_rows_kernel<T, 64, 3, 1>, 4);
    if (pieces <= 256) return go(softmax_rows_kernel<T, 64, 4, 1>, 4);
    if (pieces <= 384) return go(softmax_rows_kernel<T, 128, 3, 1>, 2);
    if (pieces <= 512) return go(softmax_rows_kernel<T, 128, 4, 1>, 2);
    if (pieces <= 768) return go(softmax_rows_kernel<T, 256, 3, 1>, 1);
    if (pieces <= 1024) return go(softmax_rows_kernel<T, 256, 4, 1>, 1);
    return go(softmax_rows_kernel<T, 256, 8, 1>, 1);
}

template <typename T>
static int32_t spmm_t(const void* p, const void* v, void* o, const float* lin, const float* tr,
                      const float* nnzs, int64_t bh, int64_t n_rows, int64_t n_cols, int64_t d,
                      int64_t trailing, cudaStream_t st) {
    const int64_t total = bh * n_rows;
    const unsigned grid = (unsigned)((total + kWarpsPerBlock - 1) / kWarpsPerBlock);
    if (grouped_d_ok(d, DT<T>::kVec) && aligned16(v) && aligned16(o))
        return launch_kernel(spmm_rows_kernel<T>, grid, kWarpsPerBlock * 32, 0, st,
            (const T*)p, (const T*)v, (T*)o, lin, tr, nnzs, total, n_rows, n_cols, (int)d,
            (int)trailing, g_index_check);
    return launch_kernel(spmm_rows_scalar_kernel<T>, grid, kWarpsPerBlock * 32, 0, st,
            (const T*)p, (const T*)v, (T*)o, lin, tr, nnzs, total, n_rows, n_cols, (int)d,
            (int)trailing, g_index_check);
}

template <typename T>
static int32_t attention_t(const void* q, const void* k, int64_t ksb, int64_t ksc, int64_t ksk,
                           const void* v, void* o, const float* lin, const float* tr,
                           const float* nnzs, int64_t bh, int64_t n_rows, int64_t n_cols, int64_t d,
                           float scale, float* lse, cudaStream_t st) {
    if (!grouped_d_ok(d, DT<T>::kVec) || !aligned16(v) || !aligned16(o))
        return SPLAT_ERR_UNSUPPORTED_SHAPE;
    const int64_t total = bh * n_rows;
    const unsigned grid = (unsigned)((total + kWarpsPerBlock - 1) / kWarpsPerBlock);
    const size_t smem = (size_t)kWarpsPerBlock * d * sizeof(float);
    const bool contig = ksk == 1 && aligned16(k) && (ksc % DT<T>::kVec == 0) &&
                        (ksb % DT<T>::kVec == 0);
    if (contig)
        return launch_kernel(attention_rows_kernel<T, true>, grid, kWarpsPerBlock * 32, smem, st,
            (const T*)q, (const T*)k, ksb, ksc, ksk, (const T*)v, (T*)o, lin, tr, nnzs, total,
            n_rows, n_cols, (int)d, scale * kLog2e, g_index_check, lse);
    return launch_kernel(attention_rows_kernel<T, false>, grid, kWarpsPerBlock * 32, smem, st,
            (const T*)q, (const T*)k, ksb, ksc, ksk, (const T*)v, (T*)o, lin, tr, nnzs, total,
            n_rows, n_cols, (int)d, scale * kLog2e, g_index_check, lse);
}

static bool sizes_ok(int64_t bh, int64_t n_rows, int64_t n_cols, int64_t d, int64_t trailing) {
    return bh >= 0 && n_rows >= 0 && n_cols >= 0 && d >= 1 && trailing >= 0 && d <= 2048 &&
           n_rows <= INT32_MAX && n_cols <= INT32_MAX && trailing <= INT32_MAX &&
           bh * n_rows / kWarpsPerBlock < (int64_t)INT32_MAX;
}

int32_t attention_generic(const void* q, const void* k, int64_t ksb, int64_t ksc, int64_t ksk,
                          const void* v, void* o, const float* lin, const float* tr,
                          const float* nnzs, int64_t bh, int64_t n_rows, int64_t n_cols, int64_t d,
                          float scale, int32_t dtype, float* lse, cudaStream_t st) {
    if (!sizes_ok(bh, n_rows, n_cols, d, 0)) return SPLAT_ERR_BAD_ARG;
    if (bh * n_rows == 0) return SPLAT_OK;   // empty batch: nothing to read or write, pointers may be null
    if (!q || !k || !v || !o || !lin || !tr || !nnzs) return SPLAT_ERR_BAD_ARG;
    switch (dtype) {
        case SPLAT_F32: return attention_t<float>(q, k, ksb, ksc, ksk, v, o, lin, tr, nnzs, bh, n_rows, n_cols, d, scale, lse, st);
        case SPLAT_F16: return attention_t<__half>(q, k, ksb, ksc, ksk, v, o, lin, tr, nnzs, bh, n_rows, n_cols, d, scale, lse, st);
        case SPLAT_BF16: return attention_t<__nv_bfloat16>(q, k, ksb, ksc, ksk, v, o, lin, tr, nnzs, bh, n_rows, n_cols, d, scale, lse, st);
        default: return SPLAT_ERR_UNSUPPORTED_DTYPE;
    }
}

}  // namespace splat

using namespace splat;

extern "C" int32_t splat_transpose_16(const void* in, void* out, int64_t bh, int64_t d, int64_t n_cols, void* stream) {
    if (bh < 0 || n_cols < 0 || d < 1) return SPLAT_ERR_BAD_ARG;
    if (d > 256 || d % 4 != 0 || bh > 65535 || n_cols > INT32_MAX) return SPLAT_ERR_UNSUPPORTED_SHAPE;
    if (bh == 0 || n_cols == 0) return SPLAT_OK;
    if (!in || !out) return SPLAT_ERR_BAD_ARG;
    if ((reinterpret_cast<uintptr_t>(out) & 3u) != 0) return SPLAT_ERR_MISALIGNED;
    const int wide = n_cols % 2 == 0 && (reinterpret_cast<uintptr_t>(in) & 3u) == 0;
    const dim3 grid((unsigned)((n_cols + kTransCols - 1) / kTransCols), (unsigned)bh);
    return launch_kernel(transpose_16_kernel, grid, 256, kTransCols * (d + 2) * 2, (cudaStream_t)stream,
        (const uint16_t*)in, (uint16_t*)out, (int)d, (int)n_cols, wide);
}

extern "C" int32_t splat_debug_check_indices(int32_t* status_word) {
    g_index_check = status_word;
    return SPLAT_OK;
}

extern "C" int32_t splat_sddmm(const void* q, const void* k, int64_t k_stride_bh,
                               int64_t k_stride_col, int64_t k_stride_k, void* s_out,
                               const float* sTod_lin, const float* sTod_tr, const float* nnzs,
                               int64_t bh, int64_t n_rows, int64_t n_cols, int64_t d,
                               int64_t trailing_dim, int32_t dtype, void* stream) {
    if (!sizes_ok(bh, n_rows, n_cols, d, trailing_dim)) return SPLAT_ERR_BAD_ARG;
    if (bh * n_rows * trailing_dim == 0) return SPLAT_OK;   // empty: pointers may be null
    if (!q || !k || !s_out || !sTod_lin || !sTod_tr || !nnzs) return SPLAT_ERR_BAD_ARG;
    cudaStream_t st = (cudaStream_t)stream;
    switch (dtype) {
        case SPLAT_F32: return sddmm_t<float>(q, k, k_stride_bh, k_stride_col, k_stride_k, s_out, sTod_lin, sTod_tr, nnzs, bh, n_rows, n_cols, d, trailing_dim, st);
        case SPLAT_F16: return sddmm_t<__half>(q, k, k_stride_bh, k_stride_col, k_stride_k, s_out, sTod_lin, sTod_tr, nnzs, bh, n_rows, n_cols, d, trailing_dim, st);
        case SPLAT_BF16: return sddmm_t<__nv_bfloat16>(q, k, k_stride_bh, k_stride_col, k_stride_k, s_out, sTod_lin, sTod_tr, nnzs, bh, n_rows, n_cols, d, trailing_dim, st);
        default: return SPLAT_ERR_UNSUPPORTED_DTYPE;
    }
}

extern "C" int32_t splat_softmax(const void* s_in, void* p_out, const float* nnzs, int64_t bh,
                                 int64_t n_rows, int64_t trailing_dim, float scale, int32_t dtype,
                                 void* stream) {
    if (!sizes_ok(bh, n_rows, 0, 1, trailing_dim)) return SPLAT_ERR_BAD_ARG;
    if (bh * n_rows * trailing_dim == 0) return SPLAT_OK;   // empty: pointers may be null
    if (!s_in || !p_out || !nnzs) return SPLAT_ERR_BAD_ARG;
    cudaStream_t st = (cudaStream_t)stream;
    switch (dtype) {
        case SPLAT_F32: return softmax_t<float>(s_in, p_out, nnzs, bh, n_rows, trailing_dim, scale, st);
        case SPLAT_F16: return softmax_t<__half>(s_in, p_out, nnzs, bh, n_rows, trailing_dim, scale, st);
        case SPLAT_BF16: return softmax_t<__nv_bfloat16>(s_in, p_out, nnzs, bh, n_rows, trailing_dim, scale, st);
        default: return SPLAT_ERR_UNSUPPORTED_DTYPE;
    }
}

extern "C" int32_t splat_spmm(const void* p, const void* v, void* o, const float* sTod_lin,
                              const float* sTod_tr, const float* nnzs, int64_t bh, int64_t n_rows,
                              int64_t n_cols, int64_t d, int64_t trailing_dim, int32_t dtype,
                              void* stream) {
    if (!sizes_ok(bh, n_rows, n_cols, d, trailing_dim)) return SPLAT_ERR_BAD_ARG;
    if (bh * n_rows == 0) return SPLAT_OK;   // empty: pointers may be null
    if (!p || !v || !o || !sTod_lin || !sTod_tr || !nnzs) return SPLAT_ERR_BAD_ARG;
    cudaStream_t st = (cudaStream_t)stream;
    switch (dtype) {
        case SPLAT_F32: return spmm_t<float>(p, v, o, sTod_lin, sTod_tr, nnzs, bh, n_rows, n_cols, d, trailing_dim, st);
        case SPLAT_F16: return spmm_t<__half>(p, v, o, sTod_lin, sTod_tr, nnzs, bh, n_rows, n_cols, d, trailing_dim, st);
        case SPLAT_BF16: return spmm_t<__nv_bfloat16>(p, v, o, sTod_lin, sTod_tr, nnzs, bh, n_rows, n_cols, d, trailing_dim, st);
        default: return SPLAT_ERR_UNSUPPORTED_DTYPE;
    }
}
