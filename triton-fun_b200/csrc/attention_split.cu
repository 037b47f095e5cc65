// Fused attention of fp32 operands on the tensor cores, band patterns (the same as in tile_f32.cu).
//
// An fp32 number is the sum of three bf16 numbers to 2^-26 of itself: h = bf16(x), m = bf16(x - h), l = bf16(x - h - m).  A
// product of two of them is six products on the tensor cores (hh, hm, mh, mm, hl, lh; what is left out is 2^-22 of it at most and
// 2^-25 on average), with fp32 accumulators.  Those round towards zero at every addition, so the order of the additions matters:
//   * the five small products of a score are summed before hh, over all of d: they meet a small accumulator;
//   * Q's h has six bits (split2()), so that most of what hh adds needs no rounding;
//   * P V is summed on the tensor core over one step of 64 keys only; the steps are added up in registers, rounded to nearest.
// Error against 64 bits over that of the register tiles (2-norm; L1024, windows of 31 to 1001 keys, d 32 to 128, the three operators):
//   normal operands of either sign     fused 0.43 to 0.58, log-sum-exp 0.67 to 0.88, SDDMM 0.44 to 0.56, SpMM 0.37 to 1.01
//   all of one sign                    fused 0.42 to 1.25, log-sum-exp 0.73 to 1.8 (it is 8e-8 then), SDDMM 0.24 to 0.66, SpMM 0.68 to 1.39 (9e-8;
//                                      1.25 and 1.39 at 127 keys: sums of so few numbers that FMAs have hardly rounded)
//   ... weights e^N(0,4), unnormalised SpMM 1.2 to 2.3 (1.8e-7)
// for a truncated sum of numbers with one sign is short by half a unit or so, whatever they are.  (Six bits of V as well: SpMM
// 1.39 -> 1.17, 2.3 -> 1.8, fused 1.25 -> 1.1 for 1 to 2 % of the time; of Q: log-sum-exp 2.6 -> 1.8 for nothing.  hh first instead
// of last 7.5e-7 at sums over 64, sums over 1024 on the tensor core alone 6.6e-6.)
// Numbers that are not finite, or too large (split2()), make their rows NaN; such rows, and their log-sum-exps, are computed again
// from their own keys (row_exact.cuh), as in the other tile kernels.
//
// One CTA = 128 rows of one (bh, class).  Warps 0-7: thread = (row, half of the columns).  A step of 64 keys:
//     K(j + 1), V(j) from global memory through registers, split, to shared memory (128-byte swizzle; both layouts of K)
//     S(j)   = Q K(j)^T      24 MMAs 128x64x16 at D = 64, Q from tensor memory (at D = 64 its pieces m, l from shared memory)
//     P(j)   = exp2(S c - m) m: the running maximum, exchanged between the two threads of a row; split, to tensor memory
//     O     += P(j) V(j)     24 MMAs 128xDx16 into a place of its own, added to the O in registers a step later
// Warp 8 issues the MMAs; the three others of its warpgroup are there to hand their registers to the workers.  Two barriers
// say all: k_full (K(j + 1) in its place and S(j) read), p_full (V(j), P(j) in their places and P V(j - 1) fetched).
// Pieces of 16 columns outside all of a warp's bands are not exponentiated.
//
// Measured, us, register tiles -> this: B2 H16 L4096 window 256 d32 166 -> 64, d64 248 -> 104, d128 561 -> 172; B1 H8 L8192
// d128 256 taps by 2 288 -> 99; B3 H8 L3001 d64 +-200 240 -> 81; B1 H2 L8192 d128 +-700 389 -> 69.  At d64 the tensor pipe is
// busy 37 % of the time, issue slots 47 %, ALUs 34 % (the split is seven ALU instructions for two numbers): a CTA's chain S -> max
// -> P -> P V, two CTAs to an SM.  Its MMAs, edges of the bands included, are 41 us of
// tensor time, six times the products themselves 30.
// What lost, at the same d64 problem: softmax warps of a thread per row (four) beside four that copy and issue 120 to 135 us
// (the copying warps are the bottleneck), beside eight 146 (registers); one warp that issues beside eight workers without
// the hand-over of registers 117 (spills); scores kept in registers for their exponentials at d64 117 to 124 (spills; at
// d32 and d128, where there is room, 64 against 70 and 171 against 189).
#include <limits.h>

#include "row_exact.cuh"
#include "split_f32.cuh"

namespace splat {
namespace band {
bool allow_dynamic_smem(const void* kernel, int bytes);   // attention_band.cu
}

namespace split {

using sm::ex2;

constexpr int kThreads = kWorkers + 128;   // (a warpgroup more: registers are handed from it to the others)
// status-word codes (which wait gave up)
enum : int { kErrK = 81, kErrP = 82, kErrS = 83, kErrO = 84, kErrMax = 85 };

struct Params {
    const float* q;       // (BH, L, D)
    const float* k;       // K in either layout
    const float* v;       // (BH, L, D)
    float* o;             // (BH, L, D)
    float* lse;           // (BH, L) or null
    const float* lin;
    const float* tr;
    const float* nnzs;
    int32_t* status;
    int32_t* mirror;      // host copy of the status word, or null
    int n_rows;           // L
    int stride;
    int tiles;            // row tiles of a class
    int kt;               // K is a contiguous (BH, D, L) array
    int vec_q, vec_k, vec_v;   // elements that a load may take at a time: 8, 4 or 1
    float scale_log2;     // > 0
    float score_scale;    // scale_log2 for scores as the tensor core gives them: times kDown
    float sign;           // of the scale: goes to Q
};

struct Control {
    uint64_t k_full;               // K of step j in its place, scores of step j - 1 read (a warp arrival each)
    uint64_t p_full;               // V and P of step j in their places, P V of step j - 1 fetched (a warp arrival each)
    uint64_t s_full, o_full;       // S, P V of step j complete
    uint64_t max_full[4];          // the two halves' maxima of 32 rows (two warp arrivals)
    uint64_t drain;
    uint32_t tmem_base;
    int32_t abort_at_entry;
    int32_t gave_up;               // code of a wait that ran out
    int32_t lo[4], hi[4];          // key range of 32 rows' bands
    int2 row[kTile];               // start, non-zeros (-1: no such row)
    float half[2][2][kTile];       // maxima of the halves, by step mod 2; sums at the end
    alignas(16) uint32_t again[4]; // rows whose result is not finite
};

template <int D> struct Layout {
    static constexpr int kPiece = kPieceBytes<D>;
    static constexpr int kOperand = 3 * kPiece;
    // Q's pieces m and l in shared memory where tensor memory has no room for them beside two CTAs' other operands
    static constexpr bool kQSmem = D == 64;
    static constexpr int kQPiece = kTile * 128;
    static constexpr int kKOff = kQSmem ? 2 * kQPiece : 0, kVOff = kKOff + kOperand;     // one step of K, two of V
    static constexpr int kSmemBytes = kVOff + 2 * kOperand + 1024;
    static constexpr int kPerSm = D == 128 ? 1 : 2;
    // tensor memory: Q, scores, P (three pieces), P V of a step
    static constexpr int kS = kQSmem ? D / 2 : 3 * D / 2;
    static constexpr int kP = kS + kKeys;
    static constexpr int kO = kP + 3 * kKeys / 2;
    static constexpr int kTmemCols = D == 128 ? 512 : 256;
    static_assert(kO + D <= kTmemCols, "tensor memory");
    // Scores are fetched again for their exponentials where the registers of two CTAs do not hold them beside the rest; their
    // place is free, and the next S can begin, the later for it.
    static constexpr bool kAgain = D == 64;
    static constexpr int kWorkerRegs = D == 128 ? 232 : 104, kOtherRegs = D == 128 ? 40 : 32;   // of 168, 80 at the launch
};

// Columns outside [lo, hi) become -inf.
__device__ __forceinline__ void mask16(uint32_t (&r)[16], int lo, int hi) {
    const int a = min(max(lo, 0), 16), b = min(max(hi, 0), 16);
    const uint32_t valid = ((1u << b) - 1) & ~((1u << a) - 1);
#pragma unroll
    for (int j = 0; j < 16; ++j) r[j] = (valid & (1u << j)) ? r[j] : 0xff800000u;
}

template <int D, bool kKt, bool kLse>
__global__ void __launch_bounds__(kThreads, Layout<D>::kPerSm)
attention_split_kernel(const __grid_constant__ Params p) {
    using L = Layout<D>;
    constexpr int kHalf = D / 2;         // columns of Q and O of a thread
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = smem_raw + (((smem_u32(smem_raw) + 1023) & ~1023u) - smem_u32(smem_raw));
    __shared__ Control ctrl_mem;
    Control* const ctrl = &ctrl_mem;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int tile = blockIdx.x % p.tiles;
    const int rest = blockIdx.x / p.tiles;
    const int res = rest % p.stride;
    const int64_t bh = rest / p.stride;
    const int u0 = tile * kTile;
    const int rows_v = (p.n_rows - res + p.stride - 1) / p.stride;    // rows of this class
    if (u0 >= rows_v) return;
    const int64_t head = bh * p.n_rows;
    const int64_t pitch = (int64_t)p.stride * D;
    const int t = threadIdx.x & (kTile - 1), half = warp >> 2;        // workers: row of the tile, half of its columns

    float xq[kHalf / 8][8];
    if (warp == kMmaWarp) {
        if (lane == 0) {
            mbar_init(&ctrl->k_full, 8);
            mbar_init(&ctrl->p_full, 8);
            mbar_init(&ctrl->s_full, 1);
            mbar_init(&ctrl->o_full, 1);
            for (int i = 0; i < 4; ++i) mbar_init(&ctrl->max_full[i], 2);
            mbar_init(&ctrl->drain, 1);
            mbar_fence_init();
        }
        __syncwarp();
        depend_wait();
        tmem_alloc(&ctrl->tmem_base, L::kTmemCols);
        tmem_relinquish();
        if (lane == 0) {
            ctrl->abort_at_entry = entry_status(p.status, p.mirror);
            ctrl->gave_up = 0;
        }
    } else if (warp > kMmaWarp) {
        depend_wait();
    } else {
        depend_wait();
        const int64_t real = (int64_t)(u0 + t) * p.stride + res;
        const float* qr = p.q + (head + real) * D + half * kHalf;
#pragma unroll
        for (int i = 0; i < kHalf / 8; ++i) {
            if (u0 + t < rows_v) {
                load8(xq[i], qr + 8 * i, p.vec_q);
            } else {
#pragma unroll
                for (int e = 0; e < 8; ++e) xq[i][e] = 0.f;
            }
        }
        if (half == 0) {
            RowAffine ra = {0, 1, 0};
            if (u0 + t < rows_v) ra = row_affine(p.lin, p.tr, p.nnzs, real);
            const int a = (ra.start - res) / p.stride;
            ctrl->row[t] = make_int2(ra.start, u0 + t < rows_v ? ra.nnz : -1);
            const int lo = warp_min_i(ra.nnz > 1 ? a : INT_MAX), hi = warp_max_i(ra.nnz > 1 ? a + ra.nnz : 0);
            if (lane == 0) { ctrl->lo[warp] = lo; ctrl->hi[warp] = hi; ctrl->again[warp] = 0; }
        }
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
    int lo = INT_MAX, hi = 0;
    for (int w = 0; w < 4; ++w) { lo = min(lo, ctrl->lo[w]); hi = max(hi, ctrl->hi[w]); }
    hi = min(hi, rows_v);
    lo = hi > 0 ? lo & ~7 : 0;
    const int steps = hi > 0 ? (hi - lo + kKeys - 1) / kKeys : 0;

    if (warp >= kMmaWarp) {
        // ------------------------------------------------------------------ MMA issuer
        asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(L::kOtherRegs));
        if (warp == kMmaWarp && steps > 0) {
            const bool lead = elect_one();
            constexpr uint32_t idesc_s = instr_desc_f16(1, kTile, kKeys, kKt ? 1u : 0u);
            constexpr uint32_t idesc_o = instr_desc_f16(1, kTile, D, 1);
            const uint32_t q_lo = desc_lo(smem, 16), k_lo = desc_lo(smem + L::kKOff, 16), v_lo = desc_lo(smem + L::kVOff, kSubBytes);
            auto issue_s = [&](int j) {
                if (!wait_all(&ctrl->k_full, (uint32_t)j & 1u, &ctrl->gave_up, kErrK)) return false;
                tc_fence_after_sync();
                if (lead) {
                    const uint32_t ql = hidden(q_lo), kl = hidden(k_lo), tm = hidden(tmem_base);
#pragma unroll
                    for (int i = 0; i < 6; ++i)
#pragma unroll
                        for (int kk = 0; kk < D / 16; ++kk) {
                            const uint64_t b = desc_sw128(kl + ((piece_b(i) * L::kPiece + (kKt ? kk * 2048 : (kk >> 2) * kSubBytes + (kk & 3) * 32)) >> 4));
                            const uint32_t add = i > 0 || kk > 0 ? 1u : 0u;
                            if (L::kQSmem && piece_a(i) > 0)
                                mma_ss(tm + L::kS, desc_sw128(ql + (((piece_a(i) - 1) * L::kQPiece + kk * 32) >> 4)), b, idesc_s, add);
                            else
                                mma_ts(tm + L::kS, tm + piece_a(i) * (D / 2) + kk * 8, b, idesc_s, add);
                        }
                    mma_commit(&ctrl->s_full);
                }
                __syncwarp();
                return true;
            };
            bool ok = issue_s(0);
#pragma unroll 1
            for (int j = 0; j < steps && ok; ++j) {
                if (j + 1 < steps) ok = issue_s(j + 1);
                if (ok) ok = wait_all(&ctrl->p_full, (uint32_t)j & 1u, &ctrl->gave_up, kErrP);
                if (!ok) break;
                tc_fence_after_sync();
                if (lead) {
                    const uint32_t vl = hidden(v_lo + ((j & 1) * L::kOperand >> 4)), tm = hidden(tmem_base);
#pragma unroll
                    for (int i = 0; i < 6; ++i)
#pragma unroll
                        for (int kk = 0; kk < kKeys / 16; ++kk)
                            mma_ts(tm + L::kO, tm + L::kP + piece_a(i) * 32 + kk * 8, desc_sw128(vl + ((piece_b(i) * L::kPiece + kk * 2048) >> 4)), idesc_o,
                                   (i > 0 || kk > 0) ? 1u : 0u);
                    mma_commit(&ctrl->o_full);
                }
                __syncwarp();
            }
            // tensor memory is released only after every MMA has completed
            if (lead) mma_commit(&ctrl->drain);
            wait_quiet(&ctrl->drain, 0);
            __syncwarp();
        }
    } else {
        // ------------------------------------------------------------------ copies, softmax, epilogue
        asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(L::kWorkerRegs));
        const uint32_t lane_addr = tmem_base + ((uint32_t)((warp & 3) * 32) << 16);
        const uint32_t s_addr = lane_addr + L::kS + half * 32, p_addr = lane_addr + L::kP + half * 16, o_addr = lane_addr + L::kO + half * kHalf;
        const int2 about = ctrl->row[t];
        const bool banded = about.y > 1;
        const int my_a = banded ? (about.x - res) / p.stride : 0, my_n = banded ? about.y : 0;     // the row's band, in class coordinates
        const float* kbase = kKt ? p.k + head * D : p.k + (head + res) * D;
        const float* vbase = p.v + (head + res) * D;
        float x[kUnits<D>][8];           // K or V on its way
        auto ask_v = [&](int j) { ask_rows<D>(x, vbase, pitch, lo + j * kKeys, rows_v, p.vec_v); };
        auto ask_k = [&](int j) {
            if constexpr (kKt) ask_kt<D, false>(x, kbase, p.n_rows, p.stride, res, lo + j * kKeys, rows_v, p.vec_k);
            else ask_rows<D>(x, kbase, pitch, lo + j * kKeys, rows_v, p.vec_k);
        };
        auto arrive = [&](uint64_t* bar) {
            tc_fence_before_sync();
            __syncwarp();
            if (lane == 0) mbar_arrive(bar);
        };
        bool ok = true;
        float2 acc[kHalf / 2];
        float m_run = -INFINITY, l_sum = 0.f;
        if (steps > 0) {
            ask_k(0);
            // Q: the A operand of S
#pragma unroll
            for (int i = 0; i < kHalf / 8; ++i) {
                const int c = half * kHalf + 8 * i;
                uint4 h, m, l;
#pragma unroll
                for (int e = 0; e < 8; ++e) xq[i][e] *= p.sign;
                split8<true, true>(xq[i], h, m, l);
                tmem_st4(lane_addr + c / 2, h);
                if constexpr (L::kQSmem) {
                    uint8_t* to = smem + t * 128 + (((c / 8) ^ (t & 7)) << 4);
                    *reinterpret_cast<uint4*>(to) = m;
                    *reinterpret_cast<uint4*>(to + L::kQPiece) = l;
                } else {
                    tmem_st4(lane_addr + D / 2 + c / 2, m);
                    tmem_st4(lane_addr + D + c / 2, l);
                }
            }
            put<D, kKt>(x, smem + L::kKOff);
            tmem_st_wait();
            arrive(&ctrl->k_full);
            if (steps > 1) ask_k(1);
        }
#pragma unroll
        for (int i = 0; i < kHalf / 2; ++i) acc[i] = make_float2(0.f, 0.f);
        auto add_o = [&] {              // acc += P V of the last step (2^16 times too large, up to the end)
#pragma unroll
            for (int c = 0; c < kHalf; c += 16) {
                uint32_t y[16];
                tmem_ld16(o_addr + c, y);
                tmem_ld_wait();
#pragma unroll
                for (int i = 0; i < 8; ++i)
                    acc[c / 2 + i] = add2(acc[c / 2 + i], make_float2(__uint_as_float(y[2 * i]), __uint_as_float(y[2 * i + 1])));
            }
        };
        const float2 sc2 = make_float2(p.score_scale, p.score_scale);
#pragma unroll 1
        for (int j = 0; j < steps; ++j) {
            ok = wait_all(&ctrl->s_full, (uint32_t)j & 1u, &ctrl->gave_up, kErrS);
            if (!ok) break;
            tc_fence_after_sync();
            uint32_t r[32];
            if (!L::kAgain) tmem_ld32(s_addr, r);
            if (j + 1 < steps) put<D, kKt>(x, smem + L::kKOff);       // (S(j) is complete: K(j) has been read)
            if (!L::kAgain) {
                tmem_ld_wait();
                if (j + 1 < steps) arrive(&ctrl->k_full);
            }
            ask_v(j);
            if (L::kAgain) {
                tmem_ld32(s_addr, r);
                tmem_ld_wait();
            }
            // Pieces of 16 columns: in none of the warp's bands (their P is 0), in all of them, or at an edge.
            const int v_lo = my_a - (lo + j * kKeys) - half * 32, v_hi = v_lo + my_n;      // valid columns of this half
            bool none[2], whole[2];
            float mine = -INFINITY;
#pragma unroll
            for (int c = 0; c < 2; ++c) {
                none[c] = __all_sync(0xffffffffu, v_lo >= 16 * c + 16 || v_hi <= 16 * c);
                whole[c] = __all_sync(0xffffffffu, v_lo <= 16 * c && v_hi >= 16 * c + 16);
                if (none[c]) continue;
                uint32_t(&part)[16] = *reinterpret_cast<uint32_t(*)[16]>(r + 16 * c);
                if (!whole[c]) mask16(part, v_lo - 16 * c, v_hi - 16 * c);
                mine = fmaxf(mine, sm::max_score(part));
            }
            ctrl->half[j & 1][half][t] = mine;
            arrive(&ctrl->max_full[warp & 3]);
            ok = wait_all(&ctrl->max_full[warp & 3], (uint32_t)j & 1u, &ctrl->gave_up, kErrMax);
            if (!ok) break;
            const float m_new = fmaxf(m_run, fmaxf(mine, ctrl->half[j & 1][half ^ 1][t]) * p.score_scale);
            const float corr = m_new > m_run ? ex2(m_run - m_new) : 1.f;
            const bool moved = __any_sync(0xffffffffu, m_new > m_run);
            m_run = m_new;
            const float me = m_run == -INFINITY ? 0.f : m_run;
            const float2 me2 = make_float2(-me, -me);
            float2 sum0 = make_float2(0.f, 0.f), sum1 = sum0;
            auto exponentials = [&](const uint32_t* from, float* to) {       // of eight scores
#pragma unroll
                for (int i = 0; i < 8; i += 2) {
                    float2 z = fma2(make_float2(__uint_as_float(from[i]), __uint_as_float(from[i + 1])), sc2, me2);
                    z.x = ex2(z.x);
                    z.y = ex2(z.y);
                    if (i & 2) sum1 = add2(sum1, z);
                    else sum0 = add2(sum0, z);
                    to[i] = z.x;
                    to[i + 1] = z.y;
                }
            };
            auto next_v = [&] {
                put<D, false>(x, smem + L::kVOff + (j & 1) * L::kOperand);       // (P V(j - 2) is complete)
                if (j + 2 < steps) ask_k(j + 2);
            };
            if (!L::kAgain) {
#pragma unroll
                for (int c = 0; c < 2; ++c) {
                    if (none[c]) continue;
#pragma unroll
                    for (int e = 16 * c; e < 16 * c + 16; e += 8) exponentials(r + e, reinterpret_cast<float*>(r + e));
                }
                next_v();
            }
            if (j > 0) {       // P V of the step before is complete: its P may be overwritten, and its result be fetched
                ok = wait_all(&ctrl->o_full, (uint32_t)(j - 1) & 1u, &ctrl->gave_up, kErrO);
                if (!ok) break;
                tc_fence_after_sync();
                add_o();
                if (moved) {
                    const float2 corr2 = make_float2(corr, corr);
#pragma unroll
                    for (int i = 0; i < kHalf / 2; ++i) acc[i] = mul2(acc[i], corr2);
                }
            }
#pragma unroll
            for (int c = 0; c < 2; ++c) {
                if (none[c]) {
#pragma unroll
                    for (int e = 16 * c; e < 16 * c + 16; e += 8)
#pragma unroll
                        for (int i = 0; i < 3; ++i) tmem_st4(p_addr + e / 2 + 32 * i, make_uint4(0, 0, 0, 0));
                    continue;
                }
                uint32_t part[16];
                if (L::kAgain) {
                    tmem_ld16(s_addr + 16 * c, part);
                    tmem_ld_wait();
                    if (!whole[c]) mask16(part, v_lo - 16 * c, v_hi - 16 * c);
                }
#pragma unroll
                for (int e = 0; e < 16; e += 8) {
                    float y[8];
                    if (L::kAgain) {
                        exponentials(part + e, y);
                    } else {
#pragma unroll
                        for (int i = 0; i < 8; ++i) y[i] = __uint_as_float(r[16 * c + e + i]);
                    }
                    uint4 h, m, l;
                    split8<false>(y, h, m, l);
                    const uint32_t to = p_addr + (16 * c + e) / 2;
                    tmem_st4(to, h);
                    tmem_st4(to + 32, m);
                    tmem_st4(to + 64, l);
                }
            }
            if (L::kAgain) {
                if (j + 1 < steps) arrive(&ctrl->k_full);
                next_v();
            }
            sum0 = add2(sum0, sum1);
            l_sum = fmaf(l_sum, corr, sum0.x + sum0.y);
            tmem_st_wait();
            arrive(&ctrl->p_full);
        }
        if (steps > 0 && ok) {
            ok = wait_all(&ctrl->o_full, (uint32_t)(steps - 1) & 1u, &ctrl->gave_up, kErrO);
            tc_fence_after_sync();
            if (ok) {
                // O / l through shared memory (everything has been multiplied) to whole rows
                add_o();
                ctrl->half[steps & 1][half][t] = l_sum;
                arrive(&ctrl->max_full[warp & 3]);
                ok = wait_all(&ctrl->max_full[warp & 3], (uint32_t)steps & 1u, &ctrl->gave_up, kErrMax);
            }
        }
        if (steps > 0 && ok) {
            l_sum = ctrl->half[steps & 1][0][t] + ctrl->half[steps & 1][1][t];
            const float inv = 1.f / l_sum * (1.f / kUp);
            const float2 inv2 = make_float2(inv, inv);
            float2 odd = make_float2(0.f, 0.f);
            constexpr int kPitch = kHalf * 4, kPer = kHalf / 4, kRows = 32 / kPer;     // a warp's 32 half rows; float4 of one; rows of a store
            uint8_t* stage = smem + L::kKOff + warp * (32 * kPitch);
#pragma unroll
            for (int i = 0; i < kPer; ++i) {
                const float2 a = mul2(acc[2 * i], inv2), b = mul2(acc[2 * i + 1], inv2);
                odd = fma2(a, make_float2(0.f, 0.f), odd);
                odd = fma2(b, make_float2(0.f, 0.f), odd);
                *reinterpret_cast<float4*>(stage + lane * kPitch + ((i ^ (lane & (kPer - 1))) << 4)) = make_float4(a.x, a.y, b.x, b.y);
            }
            const uint32_t again = __ballot_sync(0xffffffffu, banded && !(odd.x + odd.y == 0.f));
            if (again != 0 && lane == 0) atomicOr(&ctrl->again[warp & 3], again);
            const uint32_t rows = __ballot_sync(0xffffffffu, banded);
            if (kLse && banded && half == 0) p.lse[head + (int64_t)(u0 + t) * p.stride + res] = fmaf(m_run, kLn2, logf(l_sum));
            __syncwarp();
            float* out = p.o + (head + (int64_t)(u0 + (warp & 3) * 32) * p.stride + res) * D + half * kHalf;
#pragma unroll
            for (int r0 = 0; r0 < 32; r0 += kRows) {
                const int row = r0 + lane / kPer, i = lane % kPer;
                const float4 y = *reinterpret_cast<const float4*>(stage + row * kPitch + ((i ^ (row & (kPer - 1))) << 4));
                if ((rows >> row) & 1u) *reinterpret_cast<float4*>(out + row * pitch + i * 4) = y;
            }
        }
        // rows with one non-zero, V[start] -- or NaN if their score is not finite -- and without one
        if (half == 0) {
            uint32_t left = __ballot_sync(0xffffffffu, about.y == 0 || about.y == 1);
#pragma unroll 1
            for (; left != 0; left &= left - 1) {
                const int from = __ffs(left) - 1;
                const int start = __shfl_sync(0xffffffffu, about.x, from), n = __shfl_sync(0xffffffffu, about.y, from);
                const int64_t row = head + (int64_t)(u0 + warp * 32 + from) * p.stride + res;
                float score = 0.f;
                if (n == 1) {
                    const float* kr = kKt ? p.k + head * D + start : p.k + (head + start) * D;
                    const int64_t kc = kKt ? p.n_rows : 1;
#pragma unroll
                    for (int c = lane; c < D; c += 32) score = fmaf(p.q[row * D + c], kr[c * kc], score);
                    score = warp_sum(score) * p.sign * p.scale_log2;
                }
#pragma unroll
                for (int c = lane; c < D; c += 32)
                    p.o[row * D + c] = n == 0 ? 0.f : isfinite(score) ? p.v[(head + start) * D + c] : NAN;
                if (kLse && lane == 0) p.lse[row] = n == 0 ? -INFINITY : score * kLn2;
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
    // rows that are not finite, perhaps by keys outside their bands (by the warps that have the registers)
    const uint4 again = *reinterpret_cast<const uint4*>(ctrl->again);
    if ((again.x | again.y | again.z | again.w) == 0 || warp >= kMmaWarp) return;
#pragma unroll 1
    for (int i = warp; i < kTile; i += kWorkers / 32) {
        if (((ctrl->again[i >> 5] >> (i & 31)) & 1u) == 0) continue;
        const int2 about = ctrl->row[i];
        const int64_t row = head + (int64_t)(u0 + i) * p.stride + res;
        const int own = min(about.y, (p.n_rows - 1 - about.x) / p.stride + 1);
        const float* k = p.k + head * D;
        const int64_t ksc = kKt ? 1 : D, ksk = kKt ? p.n_rows : 1;
        const float scale = p.sign * p.scale_log2;
        float4 o;
        if constexpr (kLse) o = attention_row_lse<float>(p.q + row * D, k, ksc, ksk, p.v + head * D, about.x, p.stride, own, D, scale, p.lse + row);
        else o = attention_row<float>(p.q + row * D, k, ksc, ksk, p.v + head * D, about.x, p.stride, own, D, scale);
        store_row(p.o + row * D, D, o);
    }
}

template <int D>
static int32_t launch(Params p, int64_t bh, cudaStream_t st) {
    using L = Layout<D>;
    auto kern = p.kt ? (p.lse != nullptr ? attention_split_kernel<D, true, true> : attention_split_kernel<D, true, false>)
                     : (p.lse != nullptr ? attention_split_kernel<D, false, true> : attention_split_kernel<D, false, false>);
    if (!band::allow_dynamic_smem(reinterpret_cast<const void*>(kern), L::kSmemBytes)) return SPLAT_ERR_LAUNCH;
    p.tiles = ((p.n_rows + p.stride - 1) / p.stride + kTile - 1) / kTile;
    const int64_t blocks = (int64_t)p.tiles * p.stride * bh;
    if (blocks > INT32_MAX) return SPLAT_ERR_UNSUPPORTED_SHAPE;
    return launch_kernel(kern, (unsigned)blocks, kThreads, L::kSmemBytes, st, p);
}

}  // namespace split

// Operands checked by attention_tile_f32().
int32_t attention_split_f32(const void* q, const void* k, int kt, const void* v, void* o, const float* lin, const float* tr,
                            const float* nnzs, int64_t bh, int64_t n_rows, int64_t d, int64_t stride, float scale,
                            int32_t* status_word, float* lse, cudaStream_t st) {
    split::Params p{};
    p.q = (const float*)q; p.k = (const float*)k; p.v = (const float*)v; p.o = (float*)o; p.lse = lse;
    p.lin = lin; p.tr = tr; p.nnzs = nnzs; p.status = status_word; p.mirror = status_mirror(status_word);
    p.n_rows = (int)n_rows; p.stride = (int)stride; p.kt = kt; p.sign = scale < 0.f ? -1.f : 1.f; p.scale_log2 = p.sign * scale * kLog2e;
    p.score_scale = p.scale_log2 * split::kDown;
    p.vec_q = split::vec_of(q); p.vec_v = split::vec_of(v); p.vec_k = split::vec_of_k(k, kt, stride, n_rows);
    if (d == 32) return split::launch<32>(p, bh, st);
    if (d == 64) return split::launch<64>(p, bh, st);
    return split::launch<128>(p, bh, st);
}

}  // namespace splat
