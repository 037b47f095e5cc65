// fp32 SDDMM, SpMM and fused attention over ACSR on register tiles (CUDA cores, true fp32 FMA).  What is more than a wave or two
// of these tiles runs on the tensor cores (attention_split.cu, ops_split.cu), given a status word.
//
// Applies to patterns whose rows, regrouped by residue class, are contiguous bands: one stride s for
// all rows with more than one non-zero and start_i == i (mod s), as the plan of splat_acsr_classify
// says (the regrouping is described in attention_band.cu).  Here the last row of a class may be
// missing (L need not be a multiple of s), K may have either layout and any L.  d = 32, 64 or 128.
//
// Why tiles: the row kernels (ops_generic.cu) let every lane walk a K row of its own, so each score
// costs a 16-byte load per four FMAs and nothing is reused between the rows of a band that share
// their keys: 4.5 TFLOP/s.  A warp here owns 32 rows x 32 keys, a lane an 8 x 4 block of the scores and
// an 8 x D/8 block of the output.
//
// One CTA = RW x 32 rows of one (bh, class) and RW x KW warps: KW groups take the 32-key steps of
// the rows' bands in turn, each group with key and value buffers of its own, each warp with a running
// maximum, sum and output block of its own; the KW partial results of a row are merged through shared
// memory at the end.  A group of two warps synchronises with a named barrier, a group of one with
// itself.  Three CTAs (two at D = 128) share an SM: a warp's loads are covered by the other warps of its
// scheduler and are not double buffered.
//   RW = 2, KW = 2  the usual split: every K and V tile serves 64 rows.
//   RW = 1, KW = 4 or 8  for problems too small to fill the GPU with 64-row CTAs (see run()).
// The packed FMA (two results per instruction, two cycles of the pipe) leaves the issue slots that the
// shared-memory reads and the operand duplication need; in a loop of nothing but such updates an
// 8 x 8 block takes 75 to 78 cycles instead of 64 (packed) and 77 to 83 (scalar).
// Measured on B2 H16 L4096 d64, causal window 256 (1862 us with the row kernel, 104 on the tensor cores, which take it given a word):
//   64 rows per CTA, 64-key steps, 8 x 8 scores per lane, K and V prefetched    267 us (scalar FMAs 301)
//   the same, 32 rows x 2 keys per lane, the rows read uniformly                 280 us
//   RW = 2, KW = 1, six CTAs per SM                                              258 us
//   RW = 1, KW = 4                                                               278 us
//   RW = 2, KW = 2                                                               259 us; D = 128 510 us (544 / 528 us)
// The FMA pipe is busy 62 % of the time (ncu); the rest is the softmax, operand set-up and barriers.
//
// Shared memory (floats): Qt[D][32 RW rows] and per group Kt[D][32 keys] with the contraction index
// outermost, Vs[32 keys][D] (for RW = 1, D = 128 in Kt's place) and per warp Pt[32 keys][32 rows] (else
// in Kt's place).  Qt and Kt are swizzled in groups of four floats (group ^ 2 (c mod 4)) so that the
// transposing 4-byte copies, 8 rows x 4 columns per warp, do not conflict; Pt by (group ^ (key / 4))
// for its 16-byte writes.
// Lane (r, t) = (lane / 8, lane mod 8) owns rows 4r..4r+3 and 16+4r.., keys 4t..4t+3 and output
// columns 4t..4t+3 of every 32.
#include <limits.h>

#include "common.cuh"
#include "row_exact.cuh"

namespace splat {
namespace tile {

constexpr int kKeys = 32;            // keys of a step

enum class Op { kFused, kSddmm, kSpmm };

struct Params {
    const float* q;       // fused, sddmm: (BH, L, D)
    const float* k;       // fused, sddmm: K in either layout
    const float* v;       // fused, spmm: (BH, L, D)
    float* o;             // fused, spmm: (BH, L, D)
    float* sparse;        // sddmm: S out, spmm: P in, (BH, L, trailing)
    float* lse;           // fused: (BH, L) or null
    const float* lin;
    const float* tr;
    const float* nnzs;
    int n_rows;           // L
    int stride;
    int tiles;            // row tiles of a class
    int trailing;
    int kt;               // K is a contiguous (BH, D, L) array
    int kt_vec;           // ... and four keys are 16 contiguous, aligned bytes
    float scale_log2;
};

__device__ __forceinline__ float2 fma2(float2 a, float2 b, float2 c) {
    uint64_t d;
    asm("fma.rn.f32x2 %0, %1, %2, %3;"
        : "=l"(d)
        : "l"(*reinterpret_cast<uint64_t*>(&a)), "l"(*reinterpret_cast<uint64_t*>(&b)),
          "l"(*reinterpret_cast<uint64_t*>(&c)));
    return *reinterpret_cast<float2*>(&d);
}
__device__ __forceinline__ void cp4(uint32_t dst, const float* src, bool valid) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(dst), "l"(src), "r"(valid ? 4 : 0) : "memory");
}
__device__ __forceinline__ void cp16(uint32_t dst, const float* src, bool valid) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(valid ? 16 : 0)
                 : "memory");
}
__device__ __forceinline__ void cp_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N> __device__ __forceinline__ void cp_wait() {
    asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}

template <int D, int RW, int KW, Op OP> struct Layout {
    static constexpr int kWarps = RW * KW;
    static constexpr int kGroups = KW;
    static constexpr int kRows = 32 * RW;
    static constexpr bool kOneBuffer = D == 128 && RW == 1 && OP == Op::kFused;   // V follows K through one buffer
    static constexpr int kQ = OP == Op::kSpmm ? 0 : D * kRows;
    static constexpr int kTile = D * kKeys;             // a K or V tile
    static constexpr int kPt = kKeys * 32;              // a warp's P tile (sddmm: the output staging)
    // per group: offsets of P and V; K is at 0
    static constexpr int kOffP = kOneBuffer ? kTile : 0;
    static constexpr int kFront = OP == Op::kSpmm || kTile < RW * kPt ? RW * kPt : kTile;
    static constexpr int kOffV = kOneBuffer ? 0 : kFront;
    static constexpr int kGroupFloats = kOneBuffer ? kTile + kPt : kFront + (OP == Op::kSddmm ? 0 : kTile);
    static constexpr int kPart = 32 * D + 64;           // a warp's partial result: O[32][D], maxima, sums
    static constexpr int kMain = kQ + kGroups * kGroupFloats;
    static constexpr int kFloats = OP == Op::kSddmm || kMain > kWarps * kPart ? kMain : kWarps * kPart;
    // CTAs per SM the registers are budgeted for: usually, and where run() wants more.  (The same where a smaller budget
    // changes nothing: D = 128 for lack of shared memory, SpMM at D = 32 needs 114 registers anyway.)
    static constexpr int kPerSm = KW == 8 ? 1 : (D == 128 ? 2 : 3);
    static constexpr int kPerSmMore = OP == Op::kFused || D == 128 || (OP == Op::kSpmm && D == 32) ? kPerSm : kPerSm + 1;
};

// acc[8 rows][NP pairs of columns] += a[8] x b[NP]
template <int NP>
__device__ __forceinline__ void outer(float2 (&acc)[8][NP], const float (&a)[8], const float2 (&b)[NP]) {
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        const float2 aa = make_float2(a[i], a[i]);
#pragma unroll
        for (int j = 0; j < NP; ++j) acc[i][j] = fma2(aa, b[j], acc[i][j]);
    }
}
__device__ __forceinline__ void ld8(float (&x)[8], const float* lo, const float* hi) {
    const float4 u = *reinterpret_cast<const float4*>(lo), w = *reinterpret_cast<const float4*>(hi);
    x[0] = u.x; x[1] = u.y; x[2] = u.z; x[3] = u.w;
    x[4] = w.x; x[5] = w.y; x[6] = w.z; x[7] = w.w;
}

// The loaders are called by W warps, w = 0 .. W - 1, of a group (or of the CTA).
// R rows of D in global memory (row pitch in elements) -> [D][R] transposed and swizzled; rows >= limit
// become zero.
template <int D, int R, int W>
__device__ __forceinline__ void load_transposed(float* smem, const float* base, int64_t pitch, int row0, int limit, int w) {
    const int lane = threadIdx.x & 31;
    // a warp instruction: 8 rows x 4 consecutive columns
    const int r8 = lane & 7, c4 = lane >> 3;
#pragma unroll 4
    for (int it = w; it < (R / 8) * (D / 4); it += W) {
        const int row = (it % (R / 8)) * 8 + r8, c = (it / (R / 8)) * 4 + c4;
        const bool ok = row0 + row < limit;
        const float* src = base + (ok ? (int64_t)(row0 + row) * pitch : 0) + c;
        cp4((uint32_t)__cvta_generic_to_shared(smem + c * R + (((row >> 2) ^ (2 * (c & 3))) << 2) + (row & 3)), src, ok);
    }
}
// K^T (D, L) in global memory -> [D][32 keys]
template <int D, int W>
__device__ __forceinline__ void load_kt(float* smem, const float* base, const Params& p, int res, int u0, int limit, int w) {
    const int tid = w * 32 + (threadIdx.x & 31);
    if (p.kt_vec) {
#pragma unroll 4
        for (int it = tid; it < D * (kKeys / 4); it += W * 32) {
            const int c = it / (kKeys / 4), g = it % (kKeys / 4);
            const int n = limit - (u0 + g * 4);       // keys of this group that exist
            const float* src = base + (int64_t)c * p.n_rows + (n > 0 ? u0 + g * 4 : 0);
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(
                             (uint32_t)__cvta_generic_to_shared(smem + c * kKeys + ((g ^ (2 * (c & 3))) << 2))),
                         "l"(src), "r"(n >= 4 ? 16 : (n > 0 ? 4 * n : 0))
                         : "memory");
        }
        return;
    }
#pragma unroll 4
    for (int it = tid; it < D * kKeys; it += W * 32) {
        const int c = it / kKeys, key = it % kKeys;
        const bool ok = u0 + key < limit;
        const float* src = base + (int64_t)c * p.n_rows + (ok ? (int64_t)(u0 + key) * p.stride + res : 0);
        cp4((uint32_t)__cvta_generic_to_shared(smem + c * kKeys + (((key >> 2) ^ (2 * (c & 3))) << 2) + (key & 3)), src, ok);
    }
}
template <int D, int W>
__device__ __forceinline__ void load_v(float* smem, const float* base, int64_t pitch, int u0, int limit, int w) {
#pragma unroll 4
    for (int it = w * 32 + (threadIdx.x & 31); it < kKeys * (D / 4); it += W * 32) {
        const int key = it / (D / 4), c = (it % (D / 4)) * 4;
        const bool ok = u0 + key < limit;
        cp16((uint32_t)__cvta_generic_to_shared(smem + key * D + c), base + (ok ? (int64_t)(u0 + key) * pitch : 0) + c, ok);
    }
}

// One row of the fused operator that may have come out not finite by keys outside its band: from its own n keys
// (row_exact.cuh).
template <int D>
__device__ __noinline__ void fused_row_again(const Params& p, int64_t head, int64_t row, int start, int n) {
    float* o = p.o + row * D;
    bool odd = false;
#pragma unroll
    for (int c = threadIdx.x & 31; c < D; c += 32) odd = odd || !isfinite(o[c]);
    if (__any_sync(0xffffffffu, odd))
        store_row(o, D, attention_row<float>(p.q + row * D, p.k + head * D, p.kt ? 1 : D, p.kt ? p.n_rows : 1, p.v + head * D,
                                             start, p.stride, n, D, p.scale_log2));
}
// Rows with one non-zero elsewhere, a row per lane that has one: V[start] so far, NaN if the score is not finite.
template <int D>
__device__ __noinline__ void fused_singles_again(const Params& p, int64_t head, int64_t row, int start, bool mine) {
    float s = 0.f;
    if (mine) {
        const float* q = p.q + row * D;
        const float* k = p.k + head * D + (p.kt ? start : (int64_t)start * D);
        const int64_t ksk = p.kt ? p.n_rows : 1;
#pragma unroll 16
        for (int c = 0; c < D; ++c) s = fmaf(q[c], k[c * ksk], s);
    }
    for (unsigned odd = __ballot_sync(0xffffffffu, !isfinite(s * p.scale_log2)); odd != 0; odd &= odd - 1) {
        const int64_t r = __shfl_sync(0xffffffffu, row, __ffs(odd) - 1);
        for (int c = threadIdx.x & 31; c < D; c += 32) p.o[r * D + c] = NAN;
    }
}
// ... of SpMM (parameters by value: see tile_kernel)
template <int D>
__device__ __noinline__ void spmm_row_again(const float* prow, const float* v, float* o, int start, int stride, int n) {
    bool odd = false;
#pragma unroll
    for (int c = threadIdx.x & 31; c < D; c += 32) odd = odd || !isfinite(o[c]);
    if (__any_sync(0xffffffffu, odd)) store_row(o, D, spmm_row<float>(prow, v, start, stride, n, D));
}

template <int D, int RW, int KW, Op OP>
__device__ __forceinline__ void tile_body(const Params& p) {
    using L = Layout<D, RW, KW, OP>;
    constexpr int kRows = L::kRows, kGroups = L::kGroups, kWarps = L::kWarps;
    extern __shared__ __align__(16) float smem[];
    depend_wait();
    depend_release();
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int r = lane >> 3, t = lane & 7;
    float* s_q = smem;
    const int rw = warp % RW, group = warp / RW;          // row block and key group of this warp
    float* s_k = smem + L::kQ + group * L::kGroupFloats;
    float* s_p = s_k + L::kOffP + rw * L::kPt;
    float* s_v = s_k + L::kOffV;
    auto group_sync = [&] {
        if (RW == 1) __syncwarp();
        else asm volatile("bar.sync %0, %1;" ::"r"(1 + group), "n"(RW * 32) : "memory");
    };
    const int tile = blockIdx.x % p.tiles;
    const int rest = blockIdx.x / p.tiles;
    const int res = rest % p.stride;
    const int64_t bh = rest / p.stride;
    const int cta_u0 = tile * kRows, u0 = cta_u0 + rw * 32;           // first row of the CTA, of this warp
    const int rows_v = (p.n_rows - res + p.stride - 1) / p.stride;    // rows of this class
    if (cta_u0 >= rows_v) return;
    const int64_t head = bh * p.n_rows;
    const int64_t pitch = (int64_t)p.stride * D;
    const float* qbase = p.q + (head + res) * D;
    const float* kbase = p.kt ? p.k + head * D : p.k + (head + res) * D;
    const float* vbase = p.v + (head + res) * D;

    // metadata of the rows, one row per lane, in class coordinates: band columns [a, a + n).  Asked for before the copies of
    // Q, which take a thousand cycles to issue; the fused kernel of one row block is faster the other way round (a tiny problem
    // 6.56 against 6.70 us; with two row blocks 254 against 249).
    int my_a = 0, my_n = 0, my_nnz = 0, my_start = 0;   // handed out by shuffles
    RowAffine ra = {0, 1, 0};
    constexpr bool kQFirst = OP == Op::kFused && RW == 1;
    if (!kQFirst && u0 + lane < rows_v) ra = row_affine(p.lin, p.tr, p.nnzs, (int64_t)(u0 + lane) * p.stride + res);
    if (OP != Op::kSpmm) load_transposed<D, kRows, kWarps>(s_q, qbase, pitch, cta_u0, rows_v, warp);
    cp_commit();
    if (kQFirst && u0 + lane < rows_v) ra = row_affine(p.lin, p.tr, p.nnzs, (int64_t)(u0 + lane) * p.stride + res);
    if (u0 + lane < rows_v) {
        my_nnz = ra.nnz;
        my_start = ra.start;
        if (my_nnz > 1) { my_a = (my_start - res) / p.stride; my_n = my_nnz; }
    }
    const int min_a = warp_min_i(my_n > 0 ? my_a : INT_MAX), max_a = warp_max_i(my_a);
    const int min_end = warp_min_i(my_n > 0 ? my_a + my_n : 0);     // 0 when a row has no band
    const int max_end = min(warp_max_i(my_a + my_n), rows_v);
    int k_lo = min_a, k_hi = max_end;                               // over the rows of the CTA
    if (RW > 1) {
        if (lane == 0 && group == 0) reinterpret_cast<int2*>(s_k)[rw] = make_int2(min_a, max_end);
        __syncthreads();
        const int2* ranges = reinterpret_cast<const int2*>(smem + L::kQ);
#pragma unroll
        for (int x = 0; x < RW; ++x) { k_lo = min(k_lo, ranges[x].x); k_hi = max(k_hi, ranges[x].y); }
        __syncthreads();           // the ranges have been read: the key buffers may be filled
    }
    // A row with one non-zero among the warp's keys is a band like any other (its probability comes out as 1).
    if (OP == Op::kFused && my_nnz == 1) {
        const int b = (my_start - res) / p.stride;
        if (b * p.stride == my_start - res && b >= min_a && b < max_end) { my_a = b; my_n = 1; my_nnz = 2; }
    }
    k_lo = k_hi > 0 ? k_lo / kKeys : 0;
    k_hi = (k_hi + kKeys - 1) / kKeys;
    // the first step goes to a group that depends on the CTA, so that no scheduler gets the extra steps
    // of every CTA
    const int c_first = (k_lo + ((group + (int)blockIdx.x) & (kGroups - 1))) * kKeys, c_end = k_hi * kKeys;

    // this warp's first row of the sparse operand, and from one row to the next
    float* const sparse_row = OP == Op::kFused ? nullptr : p.sparse + (head + (int64_t)u0 * p.stride + res) * p.trailing;
    const int64_t sparse_pitch = (int64_t)p.stride * p.trailing;
    auto load_keys = [&](int c0) {
        if (OP != Op::kSpmm) {
            if (p.kt) load_kt<D, RW>(s_k, kbase, p, res, c0, rows_v, rw);
            else load_transposed<D, kKeys, RW>(s_k, kbase, pitch, c0, rows_v, rw);
        }
        if (OP != Op::kSddmm && !L::kOneBuffer) load_v<D, RW>(s_v, vbase, pitch, c0, rows_v, rw);
        if (OP == Op::kSpmm) {     // this warp's rows of P into Pt, one row per round, lanes along the keys
            const float* src = sparse_row;
            const uint32_t dst = (uint32_t)__cvta_generic_to_shared(s_p + lane * 32);
            const int behind = c0 + lane - my_a;       // row `lane`'s slot of column c0 + lane; row rr's: behind(rr) - rr + lane
#pragma unroll 8
            for (int rr = 0; rr < 32; ++rr, src += sparse_pitch) {
                const int slot = __shfl_sync(0xffffffffu, behind, rr) - rr + lane;
                const bool in = (unsigned)slot < (unsigned)__shfl_sync(0xffffffffu, my_n, rr);
                cp4(dst + (((((rr >> 2) ^ (lane >> 2)) << 2) | (rr & 3)) << 2), in ? src + slot : p.sparse, in);
            }
        }
        cp_commit();
    };
    if (c_first < c_end) load_keys(c_first);
    else cp_commit();
    cp_wait<1>();
    __syncthreads();               // Q is complete

    constexpr int NO = D / 16;     // pairs of output columns of a lane
    float2 acc_o[8][NO];
    float m[8], l[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        m[i] = -INFINITY; l[i] = 0.f;
#pragma unroll
        for (int j = 0; j < NO; ++j) acc_o[i][j] = make_float2(0.f, 0.f);
    }
    auto row_of = [&](int i) { return (i >> 2) * 16 + 4 * r + (i & 3); };

    for (int c0 = c_first; c0 < c_end; c0 += kGroups * kKeys) {
        const bool active = RW == 1 || (c0 < max_end && c0 + kKeys > min_a);   // warp-uniform
        const bool edge = max_a > c0 || min_end < c0 + kKeys;           // warp-uniform
        float2 s[8][2];
        cp_wait<0>();
        group_sync();
        if (OP != Op::kSpmm) {
            if (active) {
#pragma unroll
                for (int i = 0; i < 8; ++i) s[i][0] = s[i][1] = make_float2(0.f, 0.f);
#pragma unroll 2
                for (int c = 0; c < D; c += 4) {
#pragma unroll
                    for (int h = 0; h < 4; ++h) {
                        const float* q = s_q + (c + h) * kRows + rw * 32;
                        float a[8];
                        ld8(a, q + ((r ^ (2 * h)) << 2), q + (((r + 4) ^ (2 * h)) << 2));
                        const float4 k4 = *reinterpret_cast<const float4*>(s_k + (c + h) * kKeys + ((t ^ (2 * h)) << 2));
                        const float2 b[2] = {make_float2(k4.x, k4.y), make_float2(k4.z, k4.w)};
                        outer<2>(s, a, b);
                    }
                }
            }
            group_sync();          // Kt is consumed: its memory takes the probabilities, or V
            if (L::kOneBuffer) {
                load_v<D, RW>(s_v, vbase, pitch, c0, rows_v, rw);
                cp_commit();
            }
        }
        if (OP == Op::kFused && active) {
            float mx[8];
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                float(&x)[4] = *reinterpret_cast<float(*)[4]>(&s[i][0]);
#pragma unroll
                for (int j = 0; j < 4; ++j) x[j] *= p.scale_log2;
                if (edge) {
                    const int lo = __shfl_sync(0xffffffffu, my_a, row_of(i)) - c0;
                    const int hi = lo + __shfl_sync(0xffffffffu, my_n, row_of(i));
#pragma unroll
                    for (int j = 0; j < 4; ++j) x[j] = (4 * t + j >= lo && 4 * t + j < hi) ? x[j] : -INFINITY;
                }
                mx[i] = fmaxf(fmaxf(x[0], x[1]), fmaxf(x[2], x[3]));
            }
#pragma unroll
            for (int o = 1; o < 8; o <<= 1)
#pragma unroll
                for (int i = 0; i < 8; ++i) mx[i] = fmaxf(mx[i], __shfl_xor_sync(0xffffffffu, mx[i], o));
            bool moved = false;
#pragma unroll
            for (int i = 0; i < 8; ++i) moved |= mx[i] > m[i];
            if (__any_sync(0xffffffffu, moved)) {
#pragma unroll
                for (int i = 0; i < 8; ++i) {
                    const float mn = fmaxf(m[i], mx[i]);
                    const float corr = mn == -INFINITY ? 1.f : exp2f(m[i] - mn);
                    m[i] = mn;
                    l[i] *= corr;
#pragma unroll
                    for (int j = 0; j < NO; ++j) { acc_o[i][j].x *= corr; acc_o[i][j].y *= corr; }
                }
            }
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                const float me = m[i] == -INFINITY ? 0.f : m[i];
                float(&x)[4] = *reinterpret_cast<float(*)[4]>(&s[i][0]);
#pragma unroll
                for (int j = 0; j < 4; ++j) x[j] = exp2f(x[j] - me);
                l[i] += (x[0] + x[1]) + (x[2] + x[3]);
            }
            // to Pt[key][row]
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                float* row = s_p + (4 * t + j) * 32;
                float x[8];
#pragma unroll
                for (int i = 0; i < 8; ++i) x[i] = (j & 1) ? s[i][j >> 1].y : s[i][j >> 1].x;
                *reinterpret_cast<float4*>(row + ((r ^ t) << 2)) = make_float4(x[0], x[1], x[2], x[3]);
                *reinterpret_cast<float4*>(row + (((r + 4) ^ t) << 2)) = make_float4(x[4], x[5], x[6], x[7]);
            }
        } else if (active && OP == Op::kSddmm) {
            // through the warp's tile [32 rows][32 keys] to row-wise coalesced stores
#pragma unroll
            for (int i = 0; i < 8; ++i)
                *reinterpret_cast<float4*>(s_p + row_of(i) * 32 + 4 * t) =
                    make_float4(s[i][0].x, s[i][0].y, s[i][1].x, s[i][1].y);
            __syncwarp();
            // (a row costs eight instructions: with 64-bit addresses formed for each this was half of a small call)
            float* mem = sparse_row;
            const int behind = c0 + lane - my_a;       // (as in load_keys)
#pragma unroll 8
            for (int rr = 0; rr < 32; ++rr, mem += sparse_pitch) {
                const int slot = __shfl_sync(0xffffffffu, behind, rr) - rr + lane;
                if ((unsigned)slot < (unsigned)__shfl_sync(0xffffffffu, my_n, rr)) mem[slot] = s_p[rr * 32 + lane];
            }
        }
        if (OP != Op::kSddmm) {
            if (L::kOneBuffer) cp_wait<0>();
            __syncwarp();
            if (active) {
#pragma unroll 4
                for (int key = 0; key < kKeys; ++key) {
                    const int f = key >> 2;
                    float a[8];
                    float2 b[NO];
                    ld8(a, s_p + key * 32 + ((r ^ f) << 2), s_p + key * 32 + (((r + 4) ^ f) << 2));
#pragma unroll
                    for (int g = 0; g < D / 32; ++g) {
                        const float4 w = *reinterpret_cast<const float4*>(s_v + key * D + g * 32 + 4 * t);
                        b[2 * g] = make_float2(w.x, w.y);
                        b[2 * g + 1] = make_float2(w.z, w.w);
                    }
                    outer<NO>(acc_o, a, b);
                }
            }
        }
        group_sync();
        if (c0 + kGroups * kKeys < c_end) load_keys(c0 + kGroups * kKeys);
    }

    if (OP == Op::kSddmm) {
        // padding slots, rows with one non-zero (a dot product by hand) and rows with none
        unsigned todo = __ballot_sync(0xffffffffu, (lane & (kGroups - 1)) == group && u0 + lane < rows_v &&
                                                       (my_nnz < p.trailing || my_nnz == 1));
        while (todo) {
            const int rr = __ffs(todo) - 1;
            todo &= todo - 1;
            const int nnz = __shfl_sync(0xffffffffu, my_nnz, rr), start = __shfl_sync(0xffffffffu, my_start, rr);
            const int64_t real = head + (int64_t)(u0 + rr) * p.stride + res;
            float* dst = p.sparse + real * p.trailing;
            for (int j = nnz + lane; j < p.trailing; j += 32) dst[j] = 0.f;
            if (nnz == 1) {
                const float* kr = p.kt ? p.k + head * D + start : p.k + (head + start) * D;
                const int64_t kc = p.kt ? p.n_rows : 1;
                float x = 0.f;
                for (int c = lane; c < D; c += 32) x = fmaf(p.q[real * D + c], kr[(int64_t)c * kc], x);
                x = warp_sum(x);
                if (lane == 0) dst[0] = x;
            }
        }
        return;
    }

    // partial results O[32 rows][D], maxima, sums, over the tiles
    if (OP == Op::kFused) {
#pragma unroll
        for (int o = 1; o < 8; o <<= 1)
#pragma unroll
            for (int i = 0; i < 8; ++i) l[i] += __shfl_xor_sync(0xffffffffu, l[i], o);
    }
    __syncthreads();
    float* s_w = smem + warp * L::kPart;
#pragma unroll
    for (int i = 0; i < 8; ++i) {
#pragma unroll
        for (int g = 0; g < D / 32; ++g)
            *reinterpret_cast<float4*>(s_w + row_of(i) * D + g * 32 + 4 * t) =
                make_float4(acc_o[i][2 * g].x, acc_o[i][2 * g].y, acc_o[i][2 * g + 1].x, acc_o[i][2 * g + 1].y);
        if (OP == Op::kFused && t == 0) {
            s_w[32 * D + row_of(i)] = m[i];
            s_w[32 * D + 32 + row_of(i)] = l[i];
        }
    }
    __syncthreads();
    // a group's warp merges and writes 32 / kGroups of its rows, lanes along D
    float odd = 0.f;               // NaN: a row is not finite, or has its only non-zero elsewhere
    const float* parts = smem + rw * L::kPart;          // of these rows by group 0; the next group RW parts on
    // Weights of the partial results: 32 / kGroups rows with kGroups parts each, one per lane.  (With every lane forming the
    // weights of every row the merge was a quarter of a small call.)
    float w_mine = 1.f, mt = 0.f, lt = 0.f;
    if (OP == Op::kFused) {
        const float* about = parts + (lane % kGroups) * RW * L::kPart + 32 * D + group * (32 / kGroups) + lane / kGroups;
        const float mp = about[0];
        mt = mp;
#pragma unroll
        for (int o = 1; o < kGroups; o <<= 1) mt = fmaxf(mt, __shfl_xor_sync(0xffffffffu, mt, o));
        w_mine = mp == -INFINITY ? 0.f : exp2f(mp - mt);
        lt = w_mine * about[32];
#pragma unroll
        for (int o = 1; o < kGroups; o <<= 1) lt += __shfl_xor_sync(0xffffffffu, lt, o);
        w_mine *= 1.f / lt;            // (rows whose scores are all -inf: NaN; empty ones are zeroed below)
    }
#pragma unroll 4
    for (int i = 0; i < 32 / kGroups; ++i) {
        const int row = group * (32 / kGroups) + i;
        const int nnz = __shfl_sync(0xffffffffu, my_nnz, row), start = __shfl_sync(0xffffffffu, my_start, row);
        if (u0 + row >= rows_v) break;
        const int64_t real = head + (int64_t)(u0 + row) * p.stride + res;
        float w[kGroups];
#pragma unroll
        for (int x = 0; x < kGroups; ++x) w[x] = OP == Op::kFused ? __shfl_sync(0xffffffffu, w_mine, i * kGroups + x) : 1.f;
        // a row with one non-zero is described by the metadata as column `start`, outside the band
        const float w1 = OP == Op::kSpmm && nnz == 1 ? p.sparse[real * p.trailing] : 1.f;
#pragma unroll
        for (int g = 0; g < D / 32; ++g) {
            const int c = g * 32 + lane;
            float y = 0.f;
            if (nnz > 1) {
#pragma unroll
                for (int x = 0; x < kGroups; ++x) y = fmaf(w[x], parts[x * RW * L::kPart + row * D + c], y);
            } else if (nnz == 1) {
                y = w1 * p.v[(head + start) * D + c];
            }
            p.o[real * D + c] = y;
            odd = fmaf(y, 0.f, odd);
        }
        if (OP == Op::kFused && nnz == 1) odd = NAN;
        if (OP == Op::kFused && p.lse != nullptr && lane == i * kGroups) {
            float e = nnz > 1 ? lse_from_log2(mt, lt) : -INFINITY;
            if (nnz == 1) {
                const float* kr = p.kt ? p.k + head * D + start : p.k + (head + start) * D;
                e = dot_strided<float>(p.q + real * D, kr, p.kt ? p.n_rows : 1, D) * p.scale_log2 * kLn2;
            }
            p.lse[real] = e;
        }
    }
    if (__any_sync(0xffffffffu, odd != 0.f)) {
        if (OP == Op::kFused)
            fused_singles_again<D>(p, head, head + (int64_t)(u0 + lane) * p.stride + res, my_start,
                                   my_nnz == 1 && lane / (32 / kGroups) == group);
#pragma unroll 1
        for (int i = 0; i < 32 / kGroups; ++i) {
            const int row = group * (32 / kGroups) + i;
            const int start = __shfl_sync(0xffffffffu, my_start, row);
            const int n = __shfl_sync(0xffffffffu, my_n, row);
            if (n == 0) continue;
            const int64_t real = head + (int64_t)(u0 + row) * p.stride + res;
            const int own = min(n, (p.n_rows - 1 - start) / p.stride + 1);
            if (OP == Op::kFused) fused_row_again<D>(p, head, real, start, own);
            else spmm_row_again<D>(p.sparse + real * p.trailing, p.v + head * D, p.o + real * D, start, p.stride, own);
        }
    }
}

// (Parameters by value, or by reference to where they are: the repair at the end of tile_body changes how the rest is
// compiled.  Fused B2 H16 L4096 d64 270 against 262 us, the three launchers of H8 L1024 32.3 against 33.7 us.)
template <int D, int RW, int KW, Op OP, int kPerSm>
__global__ void __launch_bounds__(32 * RW * KW, kPerSm) tile_kernel(const Params p) {
    tile_body<D, RW, KW, OP>(p);
}
template <int D, int RW, int KW>
__global__ void __launch_bounds__(32 * RW * KW, Layout<D, RW, KW, Op::kFused>::kPerSm)
tile_kernel_fused(const __grid_constant__ Params p) {
    tile_body<D, RW, KW, Op::kFused>(p);
}

}  // namespace tile

namespace band {
bool allow_dynamic_smem(const void* kernel, int bytes);   // attention_band.cu
}
bool index_check_on();                                    // ops_generic.cu

namespace tile {

template <int D, int RW, int KW, Op OP, int kPerSm = Layout<D, RW, KW, OP>::kPerSm>
static int32_t launch(Params p, int64_t bh, cudaStream_t st) {
    constexpr int bytes = Layout<D, RW, KW, OP>::kFloats * (int)sizeof(float);
    void (*kern)(const Params);
    if constexpr (OP == Op::kFused) kern = tile_kernel_fused<D, RW, KW>;
    else kern = tile_kernel<D, RW, KW, OP, kPerSm>;
    if (!band::allow_dynamic_smem(reinterpret_cast<const void*>(kern), bytes)) return SPLAT_ERR_LAUNCH;
    p.tiles = ((p.n_rows + p.stride - 1) / p.stride + 32 * RW - 1) / (32 * RW);
    const int64_t blocks = (int64_t)p.tiles * p.stride * bh;
    if (blocks > INT32_MAX) return SPLAT_ERR_UNSUPPORTED_SHAPE;
    return launch_kernel(kern, (unsigned)blocks, 32 * RW * KW, bytes, st, p);
}

// More than a wave or two of 32-row CTAs come here only without a status word (splat_sddmm_tile, splat_spmm_tile, a null word of the fused
// entry points), with Q off a 16-byte boundary or with a scale below 2^-60: for these the 64-row CTAs, four warps and the
// smaller register budget of more than 296 CTAs are.
// 64-row CTAs unless they leave SMs without their three CTAs: then 32-row CTAs, whose four warps share the
// keys of one row block, finish sooner, while with the GPU full they load every key twice as often; and with
// less than two such CTAs per SM eight warps share them.  Four / eight warps, us, at 256 CTAs (L1024, +-64, where five or
// six steps leave some of the eight groups without any): d64 fused 33.9 / 24.7, SDDMM 16.5 / 16.3, SpMM 16.9 / 14.1;
// d128 42.1 / 43.7, 29.1 / 28.9, 19.8 / 21.5; d32 16.8 / 16.9, 12.0 / 10.9, 8.2 / 8.8; +-400, d64: 98 / 67, 55 / 53, 50 / 35.
// At 192 CTAs +-64 fused d64 30.3 / 24.5, SpMM 11.0 / 13.9.
// SDDMM and SpMM at d <= 64, four CTAs per SM (two of eight warps) instead of three (one), with fewer registers: a wave of
// them takes longer, so it is taken where it saves one.  Three / four, us, SDDMM then SpMM, L1024 d64 +-255: at 448 CTAs of
// 32 rows (those at the ends of a head are short and make room for the few that are left) 48.2 / 60.7, 35.5 / 43.1; 480 57.3 / 60.9,
// 41.6 / 43.6; 512 64.9 / 60.8, 45.0 / 43.5; 576 75.4 / 60.9, 49.3 / 43.9; 608 76.5 / 67.8, 50.2 / 48.7; 736 81.8 / 87.2,
// 57.8 / 58.3; 864 86.1 / 93.5, 62.6 / 64.4; of 64 rows 448 86.8 / 92.3, 67.2 / 76.3; 512 105.6 / 93.1, 84.9 / 77.0; 736
// 130.8 / 136.8, 103.4 / 104.7; 1024 169.0 / 163.3, 133.8 / 131.2; 1536 234.5 / 225.8, 185.5 / 179.9.  With +-64 the lines
// are the same, but for 480 (27.8 / 25.9, 22.2 / 20.4).  Eight warps, one / two, +-64: 128 CTAs 8.7 / 8.9, 7.4 / 7.6; 160 14.9 /
// 14.3, 12.0 / 12.0; 256 16.1 / 14.5, 13.7 / 12.1; SDDMM at d32 +-64 160 11.1 / 9.2.
template <int D, int RW, int KW, Op OP>
static int32_t launch_for(const Params& p, int64_t bh, int64_t blocks, cudaStream_t st) {
    using L = Layout<D, RW, KW, OP>;
    if constexpr (L::kPerSmMore != L::kPerSm)
        if (KW == 8 ? blocks > 148 : (blocks > 470 && blocks <= 614) || blocks > 888)
            return launch<D, RW, KW, OP, L::kPerSmMore>(p, bh, st);
    return launch<D, RW, KW, OP>(p, bh, st);
}
template <int D, Op OP>
static int32_t run(const Params& p, int64_t bh, cudaStream_t st) {
    const int64_t rows = ((int64_t)p.n_rows + p.stride - 1) / p.stride, classes = p.stride * bh;
    const int64_t of64 = (rows + 63) / 64 * classes, of32 = (rows + 31) / 32 * classes;
    if (of64 >= 3 * 148) return launch_for<D, 2, 2, OP>(p, bh, of64, st);
    if (of32 >= 2 * 148) return launch_for<D, 1, 4, OP>(p, bh, of32, st);
    return launch_for<D, 1, 8, OP>(p, bh, of32, st);
}

}  // namespace tile

int32_t attention_split_f32(const void* q, const void* k, int kt, const void* v, void* o, const float* lin, const float* tr,
                            const float* nnzs, int64_t bh, int64_t n_rows, int64_t d, int64_t stride, float scale,
                            int32_t* status_word, float* lse, cudaStream_t st);    // attention_split.cu
int32_t sddmm_split_f32(const void* q, const void* k, int kt, void* s, const float* lin, const float* tr, const float* nnzs, int64_t bh,
                        int64_t n_rows, int64_t d, int64_t stride, int64_t trailing, int32_t* status_word, cudaStream_t st);
int32_t spmm_split_f32(const void* p_in, const void* v, void* o, const float* lin, const float* tr, const float* nnzs, int64_t bh,
                       int64_t n_rows, int64_t d, int64_t stride, int64_t trailing, int32_t* status_word, cudaStream_t st);    // ops_split.cu

// Fills p and says whether the tile kernels take the problem (SPLAT_ERR_UNSUPPORTED_SHAPE if not).
// plan: {max_nnz, stride_min, stride_max, misaligned, n_single, max_col+1, n_empty, n_multi}
static int32_t tile_setup(tile::Params& p, const int32_t* plan, int64_t bh, int64_t n_rows, int64_t n_cols, int64_t d,
                          int64_t ksb, int64_t ksc, int64_t ksk, bool has_k, int64_t min_rows) {
    if (index_check_on()) return SPLAT_ERR_UNSUPPORTED_SHAPE;   // checked columns: the row kernels
    if (plan == nullptr || bh < 1 || n_rows < 1 || n_rows != n_cols || n_rows > INT32_MAX) return SPLAT_ERR_UNSUPPORTED_SHAPE;
    if (d != 32 && d != 64 && d != 128) return SPLAT_ERR_UNSUPPORTED_SHAPE;
    const int64_t stride = plan[7] > 0 ? plan[1] : 1;
    if ((plan[7] > 0 && plan[1] != plan[2]) || plan[3] != 0 || stride < 1 || plan[5] > n_cols)
        return SPLAT_ERR_UNSUPPORTED_SHAPE;
    // Short classes leave most of a tile empty: strided patterns, 16 to 32 heads, tile against row kernel at 16 / 22 /
    // 32 / 43 rows per class 0.7 / 0.9 / 1.5 / 2.1 times as fast (fused, SDDMM), SpMM 0.4 / - / 0.85 / -.
    if ((n_rows + stride - 1) / stride < min_rows && stride > 1) return SPLAT_ERR_UNSUPPORTED_SHAPE;
    p.kt = p.kt_vec = 0;
    if (has_k) {
        const bool k_major = ksk == 1 && ksc == d && ksb == n_cols * d;
        const bool kt_major = ksc == 1 && ksk == n_cols && ksb == n_cols * d;
        if (!k_major && !kt_major) return SPLAT_ERR_UNSUPPORTED_SHAPE;
        p.kt = k_major ? 0 : 1;
        p.kt_vec = stride == 1 && n_cols % 4 == 0;
    }
    p.n_rows = (int)n_rows;
    p.stride = (int)stride;
    return SPLAT_OK;
}

// Tiles of 32 rows.
static int64_t rows32(int64_t n_rows, int64_t stride, int64_t bh) { return ((n_rows + stride - 1) / stride + 31) / 32 * stride * bh; }

template <tile::Op OP>
static int32_t tile_launch(const tile::Params& p, int64_t d, int64_t bh, cudaStream_t st) {
    if (d == 32) return tile::run<32, OP>(p, bh, st);
    if (d == 64) return tile::run<64, OP>(p, bh, st);
    return tile::run<128, OP>(p, bh, st);
}

int32_t attention_tile_f32(const void* q, const void* k, int64_t ksb, int64_t ksc, int64_t ksk, const void* v, void* o,
                           const float* lin, const float* tr, const float* nnzs, int64_t bh, int64_t n_rows,
                           int64_t n_cols, int64_t d, float scale, const int32_t* plan, int32_t* status_word, float* lse,
                           cudaStream_t st) {
    tile::Params p{};
    if (!q || !k || !v || !o || !lin || !tr || !nnzs) return SPLAT_ERR_UNSUPPORTED_SHAPE;   // left to the row kernel
    const int32_t rc = tile_setup(p, plan, bh, n_rows, n_cols, d, ksb, ksc, ksk, true, 24);
    if (rc != SPLAT_OK) return rc;
    if (!aligned16(k) || !aligned16(v) || !aligned16(o)) return SPLAT_ERR_UNSUPPORTED_SHAPE;
    // The tensor cores take what is more than a wave of the tiles here: 128 rows to a CTA are coarser pieces of work.  us, here /
    // there, at 128 and 160 CTAs of 32 rows: +-64 of L1024 d32 9.0 / 9.9, 14.9 / 9.9; d64 12.9 / 15.3, 21.2 / 15.4; d128 22.2 /
    // 17.8, 36.7 / 17.9; window 32 of L200, 147 and 154: d32 7.3 / 7.4, 12.5 / 7.4; d64 9.7 / 11.5, 17.2 / 11.6; d128 15.5 /
    // 13.8, 28.1 / 13.8.  At d = 128 they are the faster for less as well (window 32 of L256, 16 CTAs 15.3 / 14.7), but for a
    // K^T that has to be gathered key by key (strided 16 of L2048, 64 CTAs 21.1 / 21.4).  Scales below 2^-60, 0 among them, stay
    // here: scaled down by another 2^-32 (split_f32.cuh) they would lose bits.
    if (status_word != nullptr && aligned16(q) && fabsf(scale) >= 0x1p-60f && (rows32(n_rows, p.stride, bh) > 148 || (d == 128 && (!p.kt || p.stride == 1))))
        return attention_split_f32(q, k, p.kt, v, o, lin, tr, nnzs, bh, n_rows, d, p.stride, scale, status_word, lse, st);
    p.q = (const float*)q; p.k = (const float*)k; p.v = (const float*)v; p.o = (float*)o; p.lse = lse;
    p.lin = lin; p.tr = tr; p.nnzs = nnzs; p.scale_log2 = scale * kLog2e;
    return tile_launch<tile::Op::kFused>(p, d, bh, st);
}

}  // namespace splat

using namespace splat;

extern "C" int32_t splat_sddmm_tile_status(const void* q, const void* k, int64_t k_stride_bh, int64_t k_stride_col,
                                           int64_t k_stride_k, void* s_out, const float* sTod_lin, const float* sTod_tr,
                                           const float* nnzs, int64_t bh, int64_t n_rows, int64_t n_cols, int64_t d,
                                           int64_t trailing_dim, int32_t dtype, const int32_t* plan_i32, int32_t* status_word,
                                           void* stream) {
    if (bh < 0 || n_rows < 0 || trailing_dim < 0) return SPLAT_ERR_BAD_ARG;
    if (dtype != SPLAT_F32 || trailing_dim < 1 || trailing_dim > INT32_MAX) return SPLAT_ERR_UNSUPPORTED_SHAPE;
    tile::Params p{};
    const int32_t rc = tile_setup(p, plan_i32, bh, n_rows, n_cols, d, k_stride_bh, k_stride_col, k_stride_k, true, 24);
    if (rc != SPLAT_OK) return rc;
    if (!q || !k || !s_out || !sTod_lin || !sTod_tr || !nnzs) return SPLAT_ERR_BAD_ARG;
    if (plan_i32[0] > trailing_dim) return SPLAT_ERR_UNSUPPORTED_SHAPE;
    if (!aligned16(k)) return SPLAT_ERR_MISALIGNED;
    // The tensor cores (ops_split.cu) where there is more than a wave of the tiles here, at d = 32 more than two.  us, here / there,
    // at CTAs of 32 rows: +-64 of L1024 d32 128 6.1 / 8.8, 256 9.2 / 8.9 (contiguous K^T 8.0 / 9.1), 320 11.3 / 9.2; d64 128
    // 8.6 / 9.8, 160 14.3 / 9.8 (11.2 / 9.9); d128 128 13.7 / 13.8 (10.6 / 13.6), 160 22.9 / 13.8; causal 32 of L256 d64 152 9.2 / 8.5;
    // 64 taps by 4 of L1000 d64 160 10.0 / 8.6, d32 256 7.2 / 7.8, 320 9.3 / 7.8.
    if (status_word != nullptr && aligned16(q) && rows32(n_rows, p.stride, bh) > (d == 32 ? 296 : 148))
        return sddmm_split_f32(q, k, p.kt, s_out, sTod_lin, sTod_tr, nnzs, bh, n_rows, d, p.stride, trailing_dim, status_word,
                               (cudaStream_t)stream);
    p.q = (const float*)q; p.k = (const float*)k; p.sparse = (float*)s_out;
    p.lin = sTod_lin; p.tr = sTod_tr; p.nnzs = nnzs; p.trailing = (int)trailing_dim;
    return tile_launch<tile::Op::kSddmm>(p, d, bh, (cudaStream_t)stream);
}

extern "C" int32_t splat_sddmm_tile(const void* q, const void* k, int64_t k_stride_bh, int64_t k_stride_col,
                                    int64_t k_stride_k, void* s_out, const float* sTod_lin, const float* sTod_tr,
                                    const float* nnzs, int64_t bh, int64_t n_rows, int64_t n_cols, int64_t d,
                                    int64_t trailing_dim, int32_t dtype, const int32_t* plan_i32, void* stream) {
    return splat_sddmm_tile_status(q, k, k_stride_bh, k_stride_col, k_stride_k, s_out, sTod_lin, sTod_tr, nnzs, bh, n_rows, n_cols,
                                   d, trailing_dim, dtype, plan_i32, nullptr, stream);
}

extern "C" int32_t splat_spmm_tile_status(const void* p_in, const void* v, void* o, const float* sTod_lin, const float* sTod_tr,
                                          const float* nnzs, int64_t bh, int64_t n_rows, int64_t n_cols, int64_t d,
                                          int64_t trailing_dim, int32_t dtype, const int32_t* plan_i32, int32_t* status_word,
                                          void* stream) {
    if (bh < 0 || n_rows < 0 || trailing_dim < 0) return SPLAT_ERR_BAD_ARG;
    if (dtype != SPLAT_F32 || trailing_dim < 1 || trailing_dim > INT32_MAX) return SPLAT_ERR_UNSUPPORTED_SHAPE;
    tile::Params p{};
    const int32_t rc = tile_setup(p, plan_i32, bh, n_rows, n_cols, d, 0, 0, 0, false, 40);
    if (rc != SPLAT_OK) return rc;
    if (!p_in || !v || !o || !sTod_lin || !sTod_tr || !nnzs) return SPLAT_ERR_BAD_ARG;
    if (plan_i32[0] > trailing_dim) return SPLAT_ERR_UNSUPPORTED_SHAPE;
    if (!aligned16(v) || !aligned16(o)) return SPLAT_ERR_MISALIGNED;
    // As above, but its steps wait for one another: more than two waves at d <= 64.  us: +-64 of L1024 d64 128 7.3 / 11.5, 256
    // 12.1 / 11.6, 320 16.4 / 11.6; +-500 of L2048 d64 256 41.8 / 46.9, 512 76.9 / 47.6; d32 +-64 256 8.2 / 9.5, 320 12.8 / 9.5; 64 taps by 4
    // of L1000 d64 288 8.5 / 9.2, 320 10.3 / 9.2; d128 +-64 128 11.3 / 14.7, 160 18.5 / 14.8; +-500 128 38.4 / 52.7, 192 62.7 / 53.0.
    if (status_word != nullptr && rows32(n_rows, p.stride, bh) > (d == 128 ? 148 : 296))
        return spmm_split_f32(p_in, v, o, sTod_lin, sTod_tr, nnzs, bh, n_rows, d, p.stride, trailing_dim, status_word,
                              (cudaStream_t)stream);
    p.sparse = (float*)const_cast<void*>(p_in); p.v = (const float*)v; p.o = (float*)o;
    p.lin = sTod_lin; p.tr = sTod_tr; p.nnzs = nnzs; p.trailing = (int)trailing_dim;
    return tile_launch<tile::Op::kSpmm>(p, d, bh, (cudaStream_t)stream);
}

extern "C" int32_t splat_spmm_tile(const void* p_in, const void* v, void* o, const float* sTod_lin, const float* sTod_tr,
                                   const float* nnzs, int64_t bh, int64_t n_rows, int64_t n_cols, int64_t d,
                                   int64_t trailing_dim, int32_t dtype, const int32_t* plan_i32, void* stream) {
    return splat_spmm_tile_status(p_in, v, o, sTod_lin, sTod_tr, nnzs, bh, n_rows, n_cols, d, trailing_dim, dtype, plan_i32, nullptr,
                                  stream);
}
