// fp32 SDDMM and SpMM on the tensor cores, band patterns (the same as in tile_f32.cu): operands as three bf16 numbers each, six
// products, the small ones first (attention_split.cu, with the errors measured).
//
//   sddmm_split_kernel   S(j) = Q K(j)^T of 128 rows and 64 keys, Q from tensor memory; a thread reads half of its row, and
//       the warp's 32 x 32 block goes through shared memory to stores along the rows
//   spmm_split_kernel    O += P(j) V(j): 32 x 32 blocks of P by cp.async, a row of the sparse operand at a time, then split and
//       placed in tensor memory; P V of a step is added to the O in registers a step later
// Measured, us, register tiles -> this: B2 H16 L4096 window 256, d32 / d64 / d128 SDDMM 112 / 176 / 326 -> 57 / 69 / 105, SpMM 100 / 146 /
// 279 -> 72 / 88 / 143 (HBM, d64: 31); H64 L1024 +-64 d64 60 -> 26, 52 -> 31.  SDDMM is bound by the instructions that store a row's 32
// scores at a time (rows begin at any element), SpMM by the chain of a step, P V -> O, V -> P V, and the copies of P, 4 bytes at a
// time.  Two places of K and of the scores, or of P, so that a step's MMAs do not wait for the stores or the split of the
// step before: SDDMM of H8 L1024 +-64 10.5 -> 10.0, SpMM 12.7 -> 11.6.
// One CTA = 128 rows of one (bh, class).  Warps 0-7: thread = (row, half of the columns); warp 8 issues the MMAs.
#include <limits.h>

#include "row_exact.cuh"
#include "split_f32.cuh"

namespace splat {
namespace band {
bool allow_dynamic_smem(const void* kernel, int bytes);   // attention_band.cu
}

namespace split {
namespace ops {

constexpr int kThreads = kWorkers + 32;
constexpr int kPitch = 36;               // floats of a staged row of 32: conflict-free 16-byte accesses along and across
constexpr int kBlockBytes = 32 * kPitch * 4;      // a warp's 32 x 32 block

// status-word codes (which wait gave up)
enum : int { kErrK = 91, kErrS = 92, kErrP = 93, kErrO = 94 };

struct Params {
    const float* q;       // sddmm: (BH, L, D)
    const float* k;       // sddmm: K in either layout
    const float* v;       // spmm: (BH, L, D)
    float* o;             // spmm: (BH, L, D)
    float* sparse;        // sddmm: S out, spmm: P in, (BH, L, trailing)
    const float* lin;
    const float* tr;
    const float* nnzs;
    int32_t* status;
    int32_t* mirror;      // host copy of the status word, or null
    int n_rows;           // L
    int stride;
    int tiles;            // row tiles of a class
    int trailing;
    int kt;               // K is a contiguous (BH, D, L) array
    int vec_q, vec_k, vec_v;   // elements that a load may take at a time: 8, 4 or 1
};

struct Control {
    uint64_t in_full[2];  // by step mod 2: operands in their places (a warp arrival each)
    uint64_t done[2];     // ... MMAs complete
    uint64_t drain;
    uint32_t tmem_base;
    int32_t abort_at_entry;
    int32_t gave_up;      // code of a wait that ran out
    int32_t lo[4], hi[4]; // key range of 32 rows' bands
    int2 row[kTile];      // start, non-zeros (-1: no such row)
    int2 band[kTile];     // begin in class coordinates, keys (0: none)
    alignas(16) uint32_t again[4];   // rows whose result is not finite
};

// Where a CTA's tile lies.
struct Place {
    int res, u0, rows_v;
    int64_t head, pitch;
    __device__ __forceinline__ Place(const Params& p, int d) {
        const int tile = blockIdx.x % p.tiles, rest = blockIdx.x / p.tiles;
        res = rest % p.stride;
        u0 = tile * kTile;
        rows_v = (p.n_rows - res + p.stride - 1) / p.stride;
        head = (int64_t)(rest / p.stride) * p.n_rows;
        pitch = (int64_t)p.stride * d;
    }
};

// The MMA warp's share of the prologue; the metadata of row t by one thread.
__device__ __forceinline__ void set_up(const Params& p, Control* ctrl, int lane, int tmem_cols) {
    if (lane == 0) {
        for (int i = 0; i < 2; ++i) {
            mbar_init(&ctrl->in_full[i], 8);
            mbar_init(&ctrl->done[i], 1);
        }
        mbar_init(&ctrl->drain, 1);
        mbar_fence_init();
    }
    __syncwarp();
    depend_wait();
    tmem_alloc(&ctrl->tmem_base, tmem_cols);
    tmem_relinquish();
    if (lane == 0) {
        ctrl->abort_at_entry = entry_status(p.status, p.mirror);
        ctrl->gave_up = 0;
    }
}
__device__ __forceinline__ void row_of_tile(const Params& p, Control* ctrl, const Place& at, int t, int warp, int lane) {
    RowAffine ra = {0, 1, 0};
    const bool exists = at.u0 + t < at.rows_v;
    if (exists) ra = row_affine(p.lin, p.tr, p.nnzs, (int64_t)(at.u0 + t) * p.stride + at.res);
    const int a = ra.nnz > 1 ? (ra.start - at.res) / p.stride : 0, n = ra.nnz > 1 ? ra.nnz : 0;
    ctrl->row[t] = make_int2(ra.start, exists ? ra.nnz : -1);
    ctrl->band[t] = make_int2(a, n);
    const int lo = warp_min_i(n > 0 ? a : INT_MAX), hi = warp_max_i(a + n);
    if (lane == 0) { ctrl->lo[warp] = lo; ctrl->hi[warp] = hi; ctrl->again[warp] = 0; }
}
// First key, and number of 64-key steps, of the tile's bands.
__device__ __forceinline__ int2 steps_of(const Control* ctrl, int rows_v) {
    int lo = INT_MAX, hi = 0;
    for (int w = 0; w < 4; ++w) { lo = min(lo, ctrl->lo[w]); hi = max(hi, ctrl->hi[w]); }
    hi = min(hi, rows_v);
    lo = hi > 0 ? lo & ~7 : 0;
    return make_int2(lo, hi > 0 ? (hi - lo + kKeys - 1) / kKeys : 0);
}
__device__ __forceinline__ void arrive(uint64_t* bar, int lane) {
    tc_fence_before_sync();
    __syncwarp();
    if (lane == 0) mbar_arrive(bar);
}

template <int D> struct SddmmLayout {
    static constexpr int kAhead = D == 128 ? 1 : 2;              // places of K and of scores: as many as two CTAs have room for
    static constexpr int kKBytes = 3 * kPieceBytes<D>;
    static constexpr int kStageOff = kAhead * kKBytes;           // behind K
    static constexpr int kSmemBytes = kStageOff + 8 * kBlockBytes + 1024;
    static constexpr int kS = 3 * D / 2;                         // tensor memory: Q, scores
    static constexpr int kTmemCols = 256;
    static_assert(kS + kAhead * kKeys <= kTmemCols, "tensor memory");
};

template <int D, bool kKt>
__global__ void __launch_bounds__(kThreads, 2)
sddmm_split_kernel(const __grid_constant__ Params p) {
    using L = SddmmLayout<D>;
    constexpr int kHalf = D / 2;         // columns of Q of a thread
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = smem_raw + (((smem_u32(smem_raw) + 1023) & ~1023u) - smem_u32(smem_raw));
    __shared__ Control ctrl_mem;
    Control* const ctrl = &ctrl_mem;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const Place at(p, D);
    if (at.u0 >= at.rows_v) return;
    const int t = threadIdx.x & (kTile - 1), half = warp >> 2;        // workers: row of the tile, half of its columns
    if (warp == kMmaWarp) {
        set_up(p, ctrl, lane, L::kTmemCols);
    } else {
        depend_wait();
        if (half == 0) row_of_tile(p, ctrl, at, t, warp, lane);
    }
    tc_fence_before_sync();
    __syncthreads();
    tc_fence_after_sync();
    depend_release();
    const uint32_t tmem_base = ctrl->tmem_base;
    if (ctrl->abort_at_entry != 0) {   // an earlier launch gave up
        if (warp == kMmaWarp) tmem_dealloc(tmem_base, L::kTmemCols);
        return;
    }
    const int2 range = steps_of(ctrl, at.rows_v);
    const int lo = range.x, steps = range.y;

    if (warp == kMmaWarp) {
        // ------------------------------------------------------------------ MMA issuer
        if (steps > 0) {
            const bool lead = elect_one();
            constexpr uint32_t idesc = instr_desc_f16(1, kTile, kKeys, kKt ? 1u : 0u);
            const uint32_t k_lo = desc_lo(smem, 16);
#pragma unroll 1
            for (int j = 0; j < steps; ++j) {
                if (!wait_all(&ctrl->in_full[j & 1], (uint32_t)(j >> 1) & 1u, &ctrl->gave_up, kErrK)) break;
                tc_fence_after_sync();
                if (lead) {
                    const int place = j % L::kAhead;
                    const uint32_t kl = hidden(k_lo + (uint32_t)(place * L::kKBytes >> 4)), tm = hidden(tmem_base), to = tm + L::kS + place * kKeys;
#pragma unroll
                    for (int i = 0; i < 6; ++i)
#pragma unroll
                        for (int kk = 0; kk < D / 16; ++kk)
                            mma_ts(to, tm + piece_a(i) * (D / 2) + kk * 8,
                                   desc_sw128(kl + ((piece_b(i) * kPieceBytes<D> + (kKt ? kk * 2048 : (kk >> 2) * kSubBytes + (kk & 3) * 32)) >> 4)),
                                   idesc, i > 0 || kk > 0 ? 1u : 0u);
                    mma_commit(&ctrl->done[j & 1]);
                }
                __syncwarp();
            }
            if (lead) mma_commit(&ctrl->drain);      // tensor memory is released only after every MMA has completed
            wait_quiet(&ctrl->drain, 0);
            __syncwarp();
        }
    } else {
        // ------------------------------------------------------------------ copies, stores
        const uint32_t lane_addr = tmem_base + ((uint32_t)((warp & 3) * 32) << 16);
        const int2 about = ctrl->row[t], band = ctrl->band[t];
        const float* kbase = kKt ? p.k + at.head * D : p.k + (at.head + at.res) * D;
        float x[kUnits<D>][8];           // K on its way
        auto ask_k = [&](int j) {
            if constexpr (kKt) ask_kt<D, true>(x, kbase, p.n_rows, p.stride, at.res, lo + j * kKeys, at.rows_v, p.vec_k);
            else ask_rows<D>(x, kbase, at.pitch, lo + j * kKeys, at.rows_v, p.vec_k);
        };
        if (steps > 0) {
            ask_k(0);
            const float* qr = p.q + (at.head + (int64_t)(at.u0 + t) * p.stride + at.res) * D + half * kHalf;
#pragma unroll 2
            for (int c = 0; c < kHalf; c += 8) {       // Q: the A operand
                float xq[8];
                if (at.u0 + t < at.rows_v) {
                    load8(xq, qr + c, p.vec_q);
                } else {
#pragma unroll
                    for (int e = 0; e < 8; ++e) xq[e] = 0.f;
                }
                uint4 h, m, l;
                split8<true, true>(xq, h, m, l);
                const uint32_t to = lane_addr + (half * kHalf + c) / 2;
                tmem_st4(to, h);
                tmem_st4(to + D / 2, m);
                tmem_st4(to + D, l);
            }
            put<D, kKt>(x, smem);
            tmem_st_wait();
            arrive(&ctrl->in_full[0], lane);
            if (steps > 1) ask_k(1);
            if (L::kAhead == 2 && steps > 1) {
                put<D, kKt>(x, smem + L::kKBytes);
                arrive(&ctrl->in_full[1], lane);
                if (steps > 2) ask_k(2);
            }
        }
        float* const stage = reinterpret_cast<float*>(smem + L::kStageOff + warp * kBlockBytes);
        const int2* const bands = ctrl->band + (warp & 3) * 32;
        // the warp's first row of S, and from one row to the next
        float* const first = p.sparse + (at.head + (int64_t)(at.u0 + (warp & 3) * 32) * p.stride + at.res) * p.trailing;
        const int64_t row_pitch = (int64_t)p.stride * p.trailing;
        float2 odd = make_float2(0.f, 0.f);
#pragma unroll 1
        for (int j = 0; j < steps; ++j) {
            if (!wait_all(&ctrl->done[j & 1], (uint32_t)(j >> 1) & 1u, &ctrl->gave_up, kErrS)) break;
            tc_fence_after_sync();
            constexpr int kAhead = L::kAhead;
            const int place = j % kAhead;
            uint32_t r[32];
            tmem_ld32(lane_addr + L::kS + place * kKeys + half * 32, r);
            if (j + kAhead < steps) put<D, kKt>(x, smem + place * L::kKBytes);       // (S(j) is complete: K(j) has been read)
            tmem_ld_wait();
            if (j + kAhead < steps) arrive(&ctrl->in_full[(j + kAhead) & 1], lane);
            if (j + kAhead + 1 < steps) ask_k(j + kAhead + 1);
            const int c0 = lo + j * kKeys + half * 32;
            if (__all_sync(0xffffffffu, band.x >= c0 + 32 || band.x + band.y <= c0)) continue;     // in none of the warp's bands
#pragma unroll
            for (int i = 0; i < 32; i += 4) {
                const float2 a = mul2(make_float2(__uint_as_float(r[i]), __uint_as_float(r[i + 1])), make_float2(kDown, kDown));
                const float2 b = mul2(make_float2(__uint_as_float(r[i + 2]), __uint_as_float(r[i + 3])), make_float2(kDown, kDown));
                odd = fma2(a, make_float2(0.f, 0.f), odd);
                odd = fma2(b, make_float2(0.f, 0.f), odd);
                *reinterpret_cast<float4*>(stage + lane * kPitch + i) = make_float4(a.x, a.y, b.x, b.y);
            }
            __syncwarp();
            float* mem = first;
#pragma unroll 8
            for (int rr = 0; rr < 32; ++rr, mem += row_pitch) {
                const int2 b = bands[rr];
                const int slot = c0 + lane - b.x;
                if ((unsigned)slot < (unsigned)b.y) mem[slot] = stage[rr * kPitch + lane];
            }
            __syncwarp();
        }
        const uint32_t again = __ballot_sync(0xffffffffu, band.y > 0 && !(odd.x + odd.y == 0.f));
        if (again != 0 && lane == 0) atomicOr(&ctrl->again[warp & 3], again);
        // padding slots, rows with one non-zero (a dot product by hand) and rows with none
        uint32_t left = __ballot_sync(0xffffffffu, about.y >= 0 && (about.y < p.trailing || about.y == 1)) & (half ? 0xaaaaaaaau : 0x55555555u);
#pragma unroll 1
        for (; left != 0; left &= left - 1) {
            const int from = __ffs(left) - 1;
            const int start = __shfl_sync(0xffffffffu, about.x, from), n = __shfl_sync(0xffffffffu, about.y, from);
            const int64_t row = at.head + (int64_t)(at.u0 + (warp & 3) * 32 + from) * p.stride + at.res;
            float* dst = p.sparse + row * p.trailing;
            for (int i = n + lane; i < p.trailing; i += 32) dst[i] = 0.f;
            if (n == 1) {
                const float* kr = kKt ? p.k + at.head * D + start : p.k + (at.head + start) * D;
                const int64_t kc = kKt ? p.n_rows : 1;
                float s = 0.f;
#pragma unroll
                for (int c = lane; c < D; c += 32) s = fmaf(p.q[row * D + c], kr[c * kc], s);
                s = warp_sum(s);
                if (lane == 0) dst[0] = s;
            }
        }
    }
    tc_fence_before_sync();
    __syncthreads();
    if (threadIdx.x == 0) publish_gave_up(p.status, &ctrl->gave_up);
    if (warp == kMmaWarp) {
        __syncwarp();
        tc_fence_after_sync();
        tmem_dealloc(tmem_base, L::kTmemCols);
    }
    // rows with scores that are not finite, perhaps by what splitting an infinity gives, or outside their bands
    const uint4 again = *reinterpret_cast<const uint4*>(ctrl->again);
    if ((again.x | again.y | again.z | again.w) == 0) return;
#pragma unroll 1
    for (int i = warp; i < kTile; i += kThreads / 32) {
        if (((ctrl->again[i >> 5] >> (i & 31)) & 1u) == 0) continue;
        const int2 about = ctrl->row[i];
        const int64_t row = at.head + (int64_t)(at.u0 + i) * p.stride + at.res;
        for (int s = lane; s < about.y; s += 32) {
            const int64_t col = about.x + (int64_t)s * p.stride;
            p.sparse[row * p.trailing + s] = dot_strided<float>(p.q + row * D, kKt ? p.k + at.head * D + col : p.k + (at.head + col) * D,
                                                                kKt ? p.n_rows : 1, D);
        }
    }
}

template <int D> struct SpmmLayout {
    static constexpr int kStageOff = 3 * kPieceBytes<D>;         // behind V; two steps' blocks of P per warp
    static constexpr int kSmemBytes = kStageOff + 16 * kBlockBytes + 1024;
    static constexpr int kPerSm = D == 128 ? 1 : 2;
    static constexpr int kP = 3 * kKeys / 2;                     // tensor memory: P (three pieces) of two steps, P V of a step
    static constexpr int kO = 2 * kP;
    static constexpr int kTmemCols = D == 128 ? 512 : 256;
    static_assert(kO + D <= kTmemCols, "tensor memory");
};

template <int D>
__global__ void __launch_bounds__(kThreads, SpmmLayout<D>::kPerSm)
spmm_split_kernel(const __grid_constant__ Params p) {
    using L = SpmmLayout<D>;
    constexpr int kHalf = D / 2;         // columns of O of a thread
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = smem_raw + (((smem_u32(smem_raw) + 1023) & ~1023u) - smem_u32(smem_raw));
    __shared__ Control ctrl_mem;
    Control* const ctrl = &ctrl_mem;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const Place at(p, D);
    if (at.u0 >= at.rows_v) return;
    const int t = threadIdx.x & (kTile - 1), half = warp >> 2;        // workers: row of the tile, half of its columns
    if (warp == kMmaWarp) {
        set_up(p, ctrl, lane, L::kTmemCols);
    } else {
        depend_wait();
        if (half == 0) row_of_tile(p, ctrl, at, t, warp, lane);
    }
    tc_fence_before_sync();
    __syncthreads();
    tc_fence_after_sync();
    depend_release();
    const uint32_t tmem_base = ctrl->tmem_base;
    if (ctrl->abort_at_entry != 0) {   // an earlier launch gave up
        if (warp == kMmaWarp) tmem_dealloc(tmem_base, L::kTmemCols);
        return;
    }
    const int2 range = steps_of(ctrl, at.rows_v);
    const int lo = range.x, steps = range.y;

    if (warp == kMmaWarp) {
        // ------------------------------------------------------------------ MMA issuer
        if (steps > 0) {
            const bool lead = elect_one();
            constexpr uint32_t idesc = instr_desc_f16(1, kTile, D, 1);
            const uint32_t v_lo = desc_lo(smem, kSubBytes);
#pragma unroll 1
            for (int j = 0; j < steps; ++j) {
                if (!wait_all(&ctrl->in_full[j & 1], (uint32_t)(j >> 1) & 1u, &ctrl->gave_up, kErrP)) break;
                tc_fence_after_sync();
                if (lead) {
                    const uint32_t vl = hidden(v_lo), tm = hidden(tmem_base), from = tm + (j & 1) * L::kP;
#pragma unroll
                    for (int i = 0; i < 6; ++i)
#pragma unroll
                        for (int kk = 0; kk < kKeys / 16; ++kk)
                            mma_ts(tm + L::kO, from + piece_a(i) * 32 + kk * 8, desc_sw128(vl + ((piece_b(i) * kPieceBytes<D> + kk * 2048) >> 4)), idesc,
                                   i > 0 || kk > 0 ? 1u : 0u);
                    mma_commit(&ctrl->done[j & 1]);
                }
                __syncwarp();
            }
            if (lead) mma_commit(&ctrl->drain);      // tensor memory is released only after every MMA has completed
            wait_quiet(&ctrl->drain, 0);
            __syncwarp();
        }
    } else {
        // ------------------------------------------------------------------ copies, sums, epilogue
        const uint32_t lane_addr = tmem_base + ((uint32_t)((warp & 3) * 32) << 16);
        const uint32_t p_addr = lane_addr + half * 16, o_addr = lane_addr + L::kO + half * kHalf;
        const int2 about = ctrl->row[t], band = ctrl->band[t];
        const bool banded = band.y > 0;
        const float* vbase = p.v + (at.head + at.res) * D;
        float x[kUnits<D>][8];           // V on its way
        uint8_t* const stage = smem + L::kStageOff + warp * 2 * kBlockBytes;
        const int2* const bands = ctrl->band + (warp & 3) * 32;
        const float* const first = p.sparse + (at.head + (int64_t)(at.u0 + (warp & 3) * 32) * p.stride + at.res) * p.trailing;
        const int64_t row_pitch = (int64_t)p.stride * p.trailing;
        auto none = [&](int j) {         // nothing of the warp's rows
            const int c0 = lo + j * kKeys + half * 32;
            return __all_sync(0xffffffffu, band.x >= c0 + 32 || band.x + band.y <= c0) != 0;
        };
        auto fetch = [&](int j) {        // the warp's block of P, a row at a time, lanes along the keys
            if (j < steps && !none(j)) {
                const uint32_t dst = smem_u32(stage + (j & 1) * kBlockBytes) + lane * 4;
                const int c = lo + j * kKeys + half * 32 + lane;
                const float* src = first;
#pragma unroll 8
                for (int rr = 0; rr < 32; ++rr, src += row_pitch) {
                    const int2 b = bands[rr];
                    const bool in = (unsigned)(c - b.x) < (unsigned)b.y;
                    asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(dst + rr * (kPitch * 4)),
                                 "l"(in ? src + (c - b.x) : p.sparse), "r"(in ? 4 : 0) : "memory");
                }
            }
            asm volatile("cp.async.commit_group;" ::: "memory");
        };
        float2 acc[kHalf / 2];
#pragma unroll
        for (int i = 0; i < kHalf / 2; ++i) acc[i] = make_float2(0.f, 0.f);
        auto add_o = [&] {               // acc += P V of the last step
#pragma unroll
            for (int c = 0; c < kHalf; c += 16) {
                uint32_t y[16];
                tmem_ld16(o_addr + c, y);
                tmem_ld_wait();
#pragma unroll
                for (int i = 0; i < 8; ++i)
                    acc[c / 2 + i] = fma2(make_float2(__uint_as_float(y[2 * i]), __uint_as_float(y[2 * i + 1])), make_float2(kDown, kDown),
                                          acc[c / 2 + i]);
            }
        };
        bool ok = true;
        if (steps > 0) {
            ask_rows<D>(x, vbase, at.pitch, lo, at.rows_v, p.vec_v);
            fetch(0);
            fetch(1);
        }
#pragma unroll 1
        for (int j = 0; j < steps; ++j) {
            asm volatile("cp.async.wait_group 1;" ::: "memory");
            __syncwarp();
            const bool empty = none(j);
            const float* mine = reinterpret_cast<const float*>(stage + (j & 1) * kBlockBytes) + lane * kPitch;
#pragma unroll
            for (int c = 0; c < 32; c += 8) {
                uint4 h = make_uint4(0, 0, 0, 0), m = h, l = h;
                if (!empty) {
                    const float4 a = *reinterpret_cast<const float4*>(mine + c), b = *reinterpret_cast<const float4*>(mine + c + 4);
                    const float y[8] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
                    split8(y, h, m, l);
                }
                const uint32_t to = p_addr + (j & 1) * L::kP + c / 2;       // (P V(j - 2) is complete)
                tmem_st4(to, h);
                tmem_st4(to + 32, m);
                tmem_st4(to + 64, l);
            }
            __syncwarp();                      // every lane has read its row
            fetch(j + 2);
            if (j > 0) {       // P V of the step before is complete: V may be overwritten, and its result be fetched
                ok = wait_all(&ctrl->done[(j - 1) & 1], (uint32_t)((j - 1) >> 1) & 1u, &ctrl->gave_up, kErrO);
                if (!ok) break;
                tc_fence_after_sync();
                add_o();
            }
            put<D, false>(x, smem);
            if (j + 1 < steps) ask_rows<D>(x, vbase, at.pitch, lo + (j + 1) * kKeys, at.rows_v, p.vec_v);
            tmem_st_wait();
            arrive(&ctrl->in_full[j & 1], lane);
        }
        asm volatile("cp.async.wait_all;" ::: "memory");
        __syncwarp();
        if (steps > 0 && ok) {
            ok = wait_all(&ctrl->done[(steps - 1) & 1], (uint32_t)((steps - 1) >> 1) & 1u, &ctrl->gave_up, kErrO);
            tc_fence_after_sync();
        }
        if (steps > 0 && ok) {
            add_o();
            // through the warp's blocks of shared memory to whole rows
            float2 odd = make_float2(0.f, 0.f);
            constexpr int kRowBytes = kHalf * 4, kPer = kHalf / 4, kRows = 32 / kPer;     // float4 of a half row; rows of a store
            static_assert(32 * kRowBytes <= 2 * kBlockBytes, "staging of the output");
#pragma unroll
            for (int i = 0; i < kPer; ++i) {
                const float2 a = acc[2 * i], b = acc[2 * i + 1];
                odd = fma2(a, make_float2(0.f, 0.f), odd);
                odd = fma2(b, make_float2(0.f, 0.f), odd);
                *reinterpret_cast<float4*>(stage + lane * kRowBytes + ((i ^ (lane & (kPer - 1))) << 4)) = make_float4(a.x, a.y, b.x, b.y);
            }
            const uint32_t again = __ballot_sync(0xffffffffu, banded && !(odd.x + odd.y == 0.f));
            if (again != 0 && lane == 0) atomicOr(&ctrl->again[warp & 3], again);
            const uint32_t rows = __ballot_sync(0xffffffffu, banded);
            __syncwarp();
            float* out = p.o + (at.head + (int64_t)(at.u0 + (warp & 3) * 32) * p.stride + at.res) * D + half * kHalf;
#pragma unroll
            for (int r0 = 0; r0 < 32; r0 += kRows) {
                const int row = r0 + lane / kPer, i = lane % kPer;
                const float4 y = *reinterpret_cast<const float4*>(stage + row * kRowBytes + ((i ^ (row & (kPer - 1))) << 4));
                if ((rows >> row) & 1u) *reinterpret_cast<float4*>(out + row * at.pitch + i * 4) = y;
            }
        }
        // rows with one non-zero, P[0] V[start], and without one
        uint32_t left = __ballot_sync(0xffffffffu, about.y == 0 || about.y == 1) & (half ? 0xaaaaaaaau : 0x55555555u);
#pragma unroll 1
        for (; left != 0; left &= left - 1) {
            const int from = __ffs(left) - 1;
            const int start = __shfl_sync(0xffffffffu, about.x, from), n = __shfl_sync(0xffffffffu, about.y, from);
            const int64_t row = at.head + (int64_t)(at.u0 + (warp & 3) * 32 + from) * p.stride + at.res;
            const float w = n == 1 ? p.sparse[row * p.trailing] : 0.f;
#pragma unroll
            for (int c = lane; c < D; c += 32) p.o[row * D + c] = n == 1 ? w * p.v[(at.head + start) * D + c] : 0.f;
        }
    }
    tc_fence_before_sync();
    __syncthreads();
    if (threadIdx.x == 0) publish_gave_up(p.status, &ctrl->gave_up);
    if (warp == kMmaWarp) {
        __syncwarp();
        tc_fence_after_sync();
        tmem_dealloc(tmem_base, L::kTmemCols);
    }
    // rows that are not finite, perhaps by keys outside their bands
    const uint4 again = *reinterpret_cast<const uint4*>(ctrl->again);
    if ((again.x | again.y | again.z | again.w) == 0) return;
#pragma unroll 1
    for (int i = warp; i < kTile; i += kThreads / 32) {
        if (((ctrl->again[i >> 5] >> (i & 31)) & 1u) == 0) continue;
        const int2 about = ctrl->row[i];
        const int64_t row = at.head + (int64_t)(at.u0 + i) * p.stride + at.res;
        const int own = min(about.y, (p.n_rows - 1 - about.x) / p.stride + 1);
        store_row(p.o + row * D, D, spmm_row<float>(p.sparse + row * p.trailing, p.v + at.head * D, about.x, p.stride, own, D));
    }
}

template <int D>
static int32_t launch(Params p, bool sddmm, int64_t bh, cudaStream_t st) {
    void (*kern)(const Params) = !sddmm ? spmm_split_kernel<D> : p.kt ? sddmm_split_kernel<D, true> : sddmm_split_kernel<D, false>;
    const int bytes = sddmm ? SddmmLayout<D>::kSmemBytes : SpmmLayout<D>::kSmemBytes;
    if (!band::allow_dynamic_smem(reinterpret_cast<const void*>(kern), bytes)) return SPLAT_ERR_LAUNCH;
    p.tiles = ((p.n_rows + p.stride - 1) / p.stride + kTile - 1) / kTile;
    const int64_t blocks = (int64_t)p.tiles * p.stride * bh;
    if (blocks > INT32_MAX) return SPLAT_ERR_UNSUPPORTED_SHAPE;
    return launch_kernel(kern, (unsigned)blocks, kThreads, bytes, st, p);
}
static int32_t launch(const Params& p, bool sddmm, int64_t bh, int64_t d, cudaStream_t st) {
    return d == 32 ? launch<32>(p, sddmm, bh, st) : d == 64 ? launch<64>(p, sddmm, bh, st) : launch<128>(p, sddmm, bh, st);
}

}  // namespace ops
}  // namespace split

// Operands checked by splat_sddmm_tile_status() / splat_spmm_tile_status().
int32_t sddmm_split_f32(const void* q, const void* k, int kt, void* s, const float* lin, const float* tr, const float* nnzs, int64_t bh,
                        int64_t n_rows, int64_t d, int64_t stride, int64_t trailing, int32_t* status_word, cudaStream_t st) {
    split::ops::Params p{};
    p.q = (const float*)q; p.k = (const float*)k; p.sparse = (float*)s;
    p.lin = lin; p.tr = tr; p.nnzs = nnzs; p.status = status_word; p.mirror = status_mirror(status_word);
    p.n_rows = (int)n_rows; p.stride = (int)stride; p.trailing = (int)trailing; p.kt = kt;
    p.vec_q = split::vec_of(q); p.vec_k = split::vec_of_k(k, kt, stride, n_rows);
    return split::ops::launch(p, true, bh, d, st);
}
int32_t spmm_split_f32(const void* p_in, const void* v, void* o, const float* lin, const float* tr, const float* nnzs, int64_t bh,
                       int64_t n_rows, int64_t d, int64_t stride, int64_t trailing, int32_t* status_word, cudaStream_t st) {
    split::ops::Params p{};
    p.sparse = (float*)const_cast<void*>(p_in); p.v = (const float*)v; p.o = (float*)o;
    p.lin = lin; p.tr = tr; p.nnzs = nnzs; p.status = status_word; p.mirror = status_mirror(status_word);
    p.n_rows = (int)n_rows; p.stride = (int)stride; p.trailing = (int)trailing;
    p.vec_v = split::vec_of(v);
    return split::ops::launch(p, false, bh, d, st);
}

}  // namespace splat
