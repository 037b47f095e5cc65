// Fused band attention, one 128-row Q tile per CTA, two CTAs per SM.  Problem, regrouping by residue class and
// operand layouts: see attention_band.cu.  The default for band patterns of 16-bit operands, but for large problems with
// d = 128 (attention_duo.cu).
//
// A step is 128 keys:
//     S(j)  = Q K(j)^T       tcgen05.mma 128x128x16, operands in shared memory
//     P(j)  = exp2(S c - m)  thread = row = tensor-memory lane: its 128 scores in registers
//     O    += P(j) V(j)      tcgen05.mma 128xDx16, A = P from tensor memory, in two halves of 64 keys
// What this replaced was a kernel with 64-key steps and two score buffers.  Its N = 64 QK MMAs read the whole
// Q tile from shared memory for every 64 keys and run at 0.64 of the tensor rate, and a softmax step paid its
// fixed costs (barrier wait, tensor-memory round trip, maximum chain, arrival: more than half of 1 700
// cycles) per 64 keys.  With 128-key steps a tile has ONE score buffer, so its softmax and its MMAs take
// turns; the other CTA of the SM, which is in no way synchronised with this one, fills the gaps.
//   * P of keys 0-63 goes to the tensor core while keys 64-127 are still being exponentiated.
//   * D = 128: S(128) + O(128) fill the CTA's 256 tensor-memory columns; P(j) (16 bit, two keys per column)
//     overwrites columns 0-63 of the consumed scores, and S(j+1) follows PV(j).
//     D = 64: P has columns of its own, and S(j+1) is computed while P(j) is.
//   * Half steps outside the bands of a warp's rows are not exponentiated, those outside the tile's bands
//     not multiplied.
//   * The tile's key range comes from the band table, which the caller's plan keeps (acsr_meta.cu), so that Q,
//     K and V are on their way some 500 cycles after the start.  Finding it from the row metadata first
//     (gathers, a division per row, a reduction over the block) cost 1 500 cycles of a CTA's 15 000 to
//     30 000 at stride 1 and 3 800 at stride 64; it remains for callers without a table.
//   * Any d that is a multiple of 8 up to 128 runs: the copies fill a tile's columns past d with zeros, and
//     the store clips them.  Any L: see band_classes.cuh.
//   * Classes of up to 64 rows (strided patterns as a rule) have one step of 64 keys at most.  At d <= 64 they have a kernel of
//     their own with half of the tensor memory, 80 registers a thread and four CTAs per SM.  us, 128-key steps -> this, at
//     tiles, bf16 d64 strided 64 of L4096 64 4.68 -> 4.43, 256 5.73 -> 5.08, 512 10.07 -> 6.72, 1024 20.1 -> 11.4; strided 64
//     of L1024 1024 18.4 -> 9.8; L64 causal 1000 19.7 -> 11.0; the same bits.  With two steps it depends on the number of tiles
//     (class of 128 rows 256 5.97 -> 6.72, 512 12.2 -> 9.5), and with more of them the running maximum is another than
//     with 128-key steps, so that shards of a problem would not agree bit for bit.
//   * With d up to 32 the MMAs and the epilogue take the first 32 of a tile's 64 columns (kCols; the others are zero).  us, 64 columns -> 32:
//     bf16 H2 L300 window 32 6.11 -> 5.73; fp16 H16 L512 window 128 6.83 -> 6.31, B4 H16 L4096 window 256 59.9 -> 57.0; bf16 B3 H34
//     L633 strided 19 20.3 -> 17.3, B2 H16 L4096 strided 64 28.0 -> 25.2, H32 L8192 window 1024 122.2 -> 118.9; the same bits.
//   * Few instructions where they are not the point: waits are a try and a counter (looking at the status word, a clock and an
//     atomic in each of 15 of them were a quarter of the code), the control block has constant addresses, an MMA's
//     descriptor is an addition.  us, before -> after: fp16 B4 H16 L4096 d64 window 256 64.1 -> 60.7; bf16 B4 H16 L4096
//     d32 window 256 65.1 -> 60.7, B2 H16 L8000 d64 strided 13 73.7 -> 67.1, H2 L256 d64 window 32 6.04 -> 5.78.
// Softmax step of 128 keys by itself (no MMAs, cycles for one / two warps per scheduler): row in registers
// 1468 / 2262, four chunks with the maximum looked at per chunk 1655 / 2403, a quarter of the exponentials
// by polynomial on the FMA pipe 1414 / 2002; 64-key steps 2 x 900 / 2 x 1140.  In the kernel the chunked
// form is 10 to 15 % slower and the polynomial changes nothing: the special function unit is busy 40 % of
// the time; what a CTA waits for is its own chain softmax -> PV -> QK -> softmax.
#include <limits.h>
#include <type_traits>

#include "band_classes.cuh"
#include "common.cuh"
#include "row_exact.cuh"
#include "softmax_math.cuh"
#include "tc_ptx.cuh"

namespace splat {
namespace band {

using namespace tc;

namespace wide {

using sm::ex2;
using sm::pack2;

constexpr int kTile = 128;               // rows of a Q tile
constexpr int kChunk = 32;               // columns of a tensor-memory load
constexpr int kSubBytes = kTile * 128;   // one 64-element (128-byte) column chunk of a Q tile
constexpr int kTmaWarp = 4;
constexpr int kMmaWarp = 5;
constexpr int kThreads = 192;            // warps 0-3 softmax and epilogue, 4 TMA, 5 MMA issuer and tensor-memory owner
constexpr float kRescaleThreshold = 8.0f;   // log2 domain: P stays below 2^8 between rescales

// status-word codes (which wait gave up)
enum : int { kErrQ = 41, kErrKFull = 42, kErrKFree = 43, kErrVFull = 44, kErrVFree = 45, kErrS = 46, kErrP = 47, kErrO = 48,
             kErrSFree = 50, kErrPv = 51 };

struct Params {
    const float* lin;
    const float* tr;
    const float* nnzs;
    const void* q;     // raw operands: rows with one non-zero are handled through them
    const void* k;
    const void* v;
    void* o;
    const int2* rows;  // band table (see acsr_meta.cu): rows in class order, tiles' key ranges; or null
    const int2* tiles;
    float* lse;        // (BH, L) or null
    int32_t* status;
    int32_t* mirror;   // host copy of the status word, or null
    int64_t n_rows;    // L
    Classes cls;
    int stride;
    int d;             // real head dimension, <= D and a multiple of 8 (the rest of a tile is zero)
    int kt_major;
    float scale_log2;
};

struct Control {
    uint64_t q_full, o_full, drain;
    uint64_t k_full[2], k_free[2], v_full[2], v_free[2];
    uint64_t s_full;           // MMA -> softmax: scores ready (D = 128: and every earlier PV complete)
    uint64_t p_full[2];        // softmax -> MMA: probabilities of keys 0-63 / 64-127 stored (4 warp arrivals)
    uint64_t s_free, pv_done;  // D = 64, 128-key steps.  softmax -> MMA: scores read (4 warp arrivals); MMA -> softmax: PV complete
    uint32_t tmem_base;
    int32_t abort_at_entry;
    int32_t gave_up;           // code of a wait that ran out
    int32_t lo[4], hi[4];      // key range of the rows' bands: of the tile (table), or per softmax warp
    alignas(16) uint32_t again[4];   // rows whose result is not finite
    alignas(16) uint32_t single[4];  // rows with one non-zero; later those of them whose score is not finite
};

// D: columns of a tile.  kKeys: keys of a step; with 64 there is one step (classes of up to 64 rows)
template <int D, int kKeys> struct Layout {
    static constexpr int kSub = D / 64;
    static constexpr int kQBytes = kSub * kSubBytes;
    static constexpr int kKeySub = kKeys * 128;             // one 64-element column chunk of a step's K or V
    static constexpr int kKeyBytes = kSub * kKeySub;
    static constexpr int kSlots = D == 128 || kKeys == 64 ? 1 : 2;      // steps of K, and of V, in shared memory
    static constexpr int kKOff = kQBytes;                   // behind the Q tile
    static constexpr int kVOff = kKOff + kSlots * kKeyBytes;
    static constexpr int kSmemBytes = kVOff + kSlots * kKeyBytes + 1024;    // + alignment slack
    static constexpr int kTmemCols = kKeys == 128 ? 256 : 128;
    static constexpr int kPerSm = kKeys == 128 ? 2 : 4;
};

// O of the warp's rows (n pieces of 16 columns) times corr.  Rare, and kept out of the main loop.
__device__ __forceinline__ void rescale_o(uint32_t o_addr, int n, float corr) {
    uint32_t v[16];
#pragma unroll 1
    for (int i = 0; i < n; ++i) {
        tmem_ld16(o_addr + i * 16, v);
        tmem_ld_wait();
#pragma unroll
        for (int j = 0; j < 16; ++j) v[j] = __float_as_uint(__uint_as_float(v[j]) * corr);
        tmem_st16(o_addr + i * 16, v);
    }
    tmem_st_wait();
}

// Band [begin, end) of a row in class coordinates; end = kSingle for a row with one non-zero (begin = its column),
// kEmpty for one without and past the end of the class.
constexpr int kSingle = -1, kEmpty = INT_MIN / 2;
__device__ __forceinline__ int2 band_of(const Params& p, int res, int u) {
    if (p.rows != nullptr) return __ldg(p.rows + p.cls.first_row(res) + u);
    const RowAffine ra = row_affine(p.lin, p.tr, p.nnzs, (int64_t)u * p.stride + res);
    if (ra.nnz > 1) {
        const int begin = p.stride == 1 ? ra.start : (ra.start - res) / p.stride;
        return make_int2(begin, begin + ra.nnz);
    }
    return ra.nnz == 1 ? make_int2(ra.start, kSingle) : make_int2(0, kEmpty);
}

// Rows of a tile that came out not finite, perhaps by keys outside their bands: from their own keys (row_exact.cuh),
// after the tile has been stored.
template <typename T>
__device__ __noinline__ void rows_again(const Params p, uint4 again, int64_t bh, int res, int u0) {
    const uint32_t mask[4] = {again.x, again.y, again.z, again.w};
    const int64_t head = bh * p.n_rows;
    const T* k = reinterpret_cast<const T*>(p.k) + head * p.d;
    const T* v = reinterpret_cast<const T*>(p.v) + head * p.d;
    for (int t = threadIdx.x >> 5; t < kTile; t += kThreads / 32) {
        if (((mask[t >> 5] >> (t & 31)) & 1u) == 0) continue;
        const int2 band = band_of(p, res, u0 + t);
        const int64_t row = head + (int64_t)(u0 + t) * p.stride + res;
        const bool one = band.y == kSingle;
        const float4 x = attention_row<T>(reinterpret_cast<const T*>(p.q) + row * p.d, k, p.kt_major ? 1 : p.d,
                                          p.kt_major ? p.n_rows : 1, v, one ? band.x : (int64_t)band.x * p.stride + res,
                                          p.stride, one ? 1 : min(band.y, p.cls.rows_of(res)) - band.x, p.d, p.scale_log2);
        store_row<T>(reinterpret_cast<T*>(p.o) + row * p.d, p.d, x);
    }
}

// Rows of a tile with one non-zero whose score is not finite, of those in `single` (a bit per row).  Such a row takes
// V[start] without its score having been formed (the metadata gives column 0 as its place, outside its band as a
// rule).  By the TMA warp, which has requested all it can for now, a row per lane: in the softmax warps it cost 40 us
// of a strided call's 103.
template <typename T>
__device__ __forceinline__ uint4 odd_singles(const Params& p, uint4 single, int64_t bh, int res, int u0) {
    const int lane = threadIdx.x & 31;
    uint32_t rows[4] = {single.x, single.y, single.z, single.w};
#pragma unroll
    for (int w = 0; w < 4; ++w) {
        float s = 0.f;
        if ((rows[w] >> lane) & 1u) {
            const int u = u0 + w * 32 + lane;
            const int64_t col = band_of(p, res, u).x;
            const T* q = reinterpret_cast<const T*>(p.q) + (bh * p.n_rows + (int64_t)u * p.stride + res) * p.d;
            const T* k = reinterpret_cast<const T*>(p.k) + bh * p.n_rows * p.d + (p.kt_major ? col : col * p.d);
#pragma unroll 4
            for (int c = 0; c < p.d; c += 8) {
                const uint4 a = *reinterpret_cast<const uint4*>(q + c);
                uint4 b;
                T* kc = reinterpret_cast<T*>(&b);
                if (p.kt_major) {
#pragma unroll
                    for (int i = 0; i < 8; ++i) kc[i] = k[(int64_t)(c + i) * p.n_rows];
                } else {
                    b = *reinterpret_cast<const uint4*>(k + c);
                }
                const T* qc = reinterpret_cast<const T*>(&a);
#pragma unroll
                for (int i = 0; i < 8; ++i) s = fmaf(DT<T>::to_f(qc[i]), DT<T>::to_f(kc[i]), s);
            }
        }
        rows[w] = __ballot_sync(0xffffffffu, !isfinite(s * p.scale_log2));
    }
    return make_uint4(rows[0], rows[1], rows[2], rows[3]);
}

template <typename T, int D, int kCols, int kKeys, bool kLse, bool kOwn>
__global__ void __launch_bounds__(kThreads, Layout<D, kKeys>::kPerSm)
attention_wide_kernel(const __grid_constant__ Maps<4> maps, const Params p) {
    using L = Layout<D, kKeys>;
    constexpr int kSlots = L::kSlots, kTmemCols = L::kTmemCols;
    constexpr bool kOwnP = D == 64 && kKeys == 128;              // P has tensor-memory columns of its own
    constexpr uint32_t kPCol = kOwnP ? kKeys + D : 0;
    constexpr int kHalves = kKeys / 64;
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = smem_raw + (((smem_u32(smem_raw) + 1023) & ~1023u) - smem_u32(smem_raw));
    __shared__ Control ctrl_mem;             // (static: constant addresses)
    Control* const ctrl = &ctrl_mem;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int real_res = blockIdx.y, res = p.cls.in_part(real_res), rows_v = p.cls.rows_of(real_res);
    const CUtensorMap* map = maps.part[p.cls.part(real_res)];       // Q, K, V, O
    const int64_t bh = blockIdx.z;
    const int u0 = blockIdx.x * kTile;
    if (u0 >= rows_v) return;       // (a class one tile shorter than the longest)

    // Prologue, one block-wide barrier: tensor-memory allocation, row metadata and the first copies proceed
    // side by side.
    int jk = 0, jv = 0;                // TMA warp: K and V tiles requested
    int klo = 0;                       // first 128-key step
    auto load_k = [&]() {
        const int st = jk % kSlots, row = (klo + jk) * kKeys;
        if (jk >= kSlots && !wait_bar(&ctrl->k_free[st], ((uint32_t)(jk / kSlots) & 1u) ^ 1u, &ctrl->gave_up, kErrKFree)) return false;
        mbar_arrive_expect_tx(&ctrl->k_full[st], L::kKeyBytes);
        uint8_t* dst = smem + L::kKOff + st * L::kKeyBytes;
        if (p.kt_major) {
            for (int ch = 0; ch < kHalves; ++ch)       // 64-key chunks of [d][64 keys]
                tma_load_4d(dst + ch * (D * 128), map + 1, &ctrl->k_full[st], row + ch * 64, 0, (int)bh, 0);
        } else {
            for (int sub = 0; sub < L::kSub; ++sub)
                tma_load_4d(dst + sub * L::kKeySub, map + 1, &ctrl->k_full[st], sub * 64, res, row, (int)bh);
        }
        ++jk;
        return true;
    };
    auto load_v = [&]() {
        const int st = jv % kSlots;
        if (jv >= kSlots && !wait_bar(&ctrl->v_free[st], ((uint32_t)(jv / kSlots) & 1u) ^ 1u, &ctrl->gave_up, kErrVFree)) return false;
        mbar_arrive_expect_tx(&ctrl->v_full[st], L::kKeyBytes);
        for (int sub = 0; sub < L::kSub; ++sub)
            tma_load_4d(smem + L::kVOff + st * L::kKeyBytes + sub * L::kKeySub, map + 2, &ctrl->v_full[st], sub * 64, res,
                        (klo + jv) * kKeys, (int)bh);
        ++jv;
        return true;
    };
    int my_begin = 0, my_end = kEmpty;      // band of this thread's row
    if (warp == kMmaWarp) {
        depend_wait();
        tmem_alloc(&ctrl->tmem_base, kTmemCols);
        tmem_relinquish();
    } else if (warp == kTmaWarp) {
        if (lane == 0) {
            for (int i = 0; i < 3; ++i) tma_prefetch_desc(map + i);
            mbar_init(&ctrl->q_full, 1);
            mbar_init(&ctrl->o_full, 1);
            mbar_init(&ctrl->drain, 1);
            mbar_init(&ctrl->s_full, 1);
            mbar_init(&ctrl->s_free, 4);
            mbar_init(&ctrl->pv_done, 1);
            for (int i = 0; i < 2; ++i) {
                mbar_init(&ctrl->k_full[i], 1);
                mbar_init(&ctrl->k_free[i], 1);
                mbar_init(&ctrl->v_full[i], 1);
                mbar_init(&ctrl->v_free[i], 1);
                mbar_init(&ctrl->p_full[i], 4);      // one arrival per softmax warp
            }
            mbar_fence_init();
            depend_wait();
            int2 range = make_int2(0, 0);
            if (p.tiles != nullptr) range = __ldg(p.tiles + real_res * p.cls.tile_pitch + blockIdx.x);
            const int32_t stop = entry_status(p.status, p.mirror);
            ctrl->abort_at_entry = stop;
            ctrl->gave_up = 0;
            if (stop == 0) {
                mbar_arrive_expect_tx(&ctrl->q_full, L::kQBytes);
                for (int sub = 0; sub < L::kSub; ++sub)
                    tma_load_4d(smem + sub * kSubBytes, map, &ctrl->q_full, sub * 64, res, u0, (int)bh);
                if (range.y > 0) {
                    klo = range.x / kKeys;
                    load_k();
                    load_v();
                }
            }
            if (p.tiles != nullptr)
                for (int w = 0; w < 4; ++w) { ctrl->lo[w] = range.x; ctrl->hi[w] = range.y; }
        }
    } else {
        depend_wait();
        const int u = u0 + warp * 32 + lane;
        if (u < rows_v) {
            const int2 band = band_of(p, real_res, u);
            my_begin = band.x;
            my_end = band.y;
            if (my_end == kSingle) {   // its row of V is copied at the end
                const char* vrow = reinterpret_cast<const char*>(p.v) + (bh * p.n_rows + my_begin) * p.d * 2;
                for (int i = 0; i < p.d * 2; i += 128) asm volatile("prefetch.global.L1 [%0];" ::"l"(vrow + i));
            }
        }
        if constexpr (kOwn) {
            const unsigned single = __ballot_sync(0xffffffffu, my_end == kSingle);
            if (lane == 0) ctrl->single[warp] = single;
        }
        if (p.rows == nullptr) {
            const int lo = warp_min_i(my_end > 0 ? my_begin : INT_MAX), hi = warp_max_i(max(my_end, 0));
            if (lane == 0) { ctrl->lo[warp] = lo; ctrl->hi[warp] = hi; }
        }
    }
    tc_fence_before_sync();
    __syncthreads();
    tc_fence_after_sync();
    depend_release();
    const uint32_t tmem_base = ctrl->tmem_base;
    if (ctrl->abort_at_entry != 0) {   // an earlier launch gave up
        if (warp == kMmaWarp) tmem_dealloc(tmem_base, kTmemCols);
        return;
    }
    int lo64 = INT_MAX, hi64 = 0;
    for (int w = 0; w < 4; ++w) { lo64 = min(lo64, ctrl->lo[w]); hi64 = max(hi64, ctrl->hi[w]); }
    hi64 = min(hi64, rows_v);
    if (hi64 <= 0) lo64 = 0;
    lo64 = lo64 / 64;          // in 64-key units from here
    hi64 = (hi64 + 63) / 64;
    klo = lo64 / kHalves;
    const int steps = (hi64 + kHalves - 1) / kHalves - klo;
    auto wait_all = [&](uint64_t* bar, uint32_t parity, int code) { return tc::wait_all(bar, parity, &ctrl->gave_up, code); };

    if (warp == kTmaWarp) {
        // ------------------------------------------------------------------ TMA producer
        if constexpr (kOwn) {
            const uint4 single = *reinterpret_cast<const uint4*>(ctrl->single);
            if ((single.x | single.y | single.z | single.w) != 0) {
                const uint4 odd = odd_singles<T>(p, single, bh, real_res, u0);
                __syncwarp();
                if (lane == 0) *reinterpret_cast<uint4*>(ctrl->single) = odd;
            }
        }
        if (lane == 0) {
            bool ok = true;
            while (ok && jv < steps) {     // K(0) V(0) K(1) V(1) ...: the order in which the slots come free
                if (jk <= jv) ok = load_k();
                if (ok) ok = load_v();
            }
            if (!ok) {                     // leave only after the copies already issued have landed
                wait_quiet(&ctrl->q_full, 0);
                for (int i = max(0, jk - kSlots); i < jk; ++i) wait_quiet(&ctrl->k_full[i % kSlots], (uint32_t)(i / kSlots) & 1u);
                for (int i = max(0, jv - kSlots); i < jv; ++i) wait_quiet(&ctrl->v_full[i % kSlots], (uint32_t)(i / kSlots) & 1u);
            }
        }
    } else if (warp == kMmaWarp) {
        // ------------------------------------------------------------------ MMA issuer
        // (whole warp on warp-uniform values, one elected lane issues)
        if (steps > 0) {
            const bool lead = elect_one();
            constexpr uint32_t fmt = std::is_same<T, __nv_bfloat16>::value ? 1u : 0u;
            const uint32_t idesc_qk = instr_desc_f16(fmt, kTile, kKeys, p.kt_major ? 1u : 0u);
            const uint32_t idesc_qk_half = instr_desc_f16(fmt, kTile, 64, p.kt_major ? 1u : 0u);
            constexpr uint32_t idesc_pv = instr_desc_f16(fmt, kTile, kCols, 1);
            const uint32_t q_lo = desc_lo(smem, 16), k_lo = desc_lo(smem + L::kKOff, p.kt_major ? D * 128 : 16);
            const uint32_t v_lo = desc_lo(smem + L::kVOff, L::kKeySub);
            const uint32_t k_step = (p.kt_major ? 2048 : 32) >> 4, k_sub = (p.kt_major ? 4 * 2048 : L::kKeySub) >> 4;
            const uint32_t o_tmem = tmem_base + kKeys;
            auto commit = [&](uint64_t* bar) { if (lead) mma_commit(bar); };
            auto in_range = [&](int j, int half) { const int i = 2 * (klo + j) + half; return kHalves == 1 || (i >= lo64 && i < hi64); };
            bool ok = wait_all(&ctrl->q_full, 0, kErrQ);
            bool first_pv = true;
            auto k_here = [&](int j) { return wait_all(&ctrl->k_full[j % kSlots], (uint32_t)(j / kSlots) & 1u, kErrKFull); };
            auto issue_s = [&](int j) {                // S(j); half steps outside the range are left out
                const int st = j % kSlots;
                if (!kOwnP) ok = k_here(j);
                if (!ok) return;
                tc_fence_after_sync();
                const bool h0 = in_range(j, 0), both = h0 && in_range(j, 1);
                const uint32_t idesc = kHalves == 1 || both ? idesc_qk : idesc_qk_half;
                const uint32_t skip = h0 ? 0u : 1u;
                if (lead) {
                    const uint32_t to = tmem_base + skip * 64;
                    uint32_t b = k_lo + ((st * L::kKeyBytes + skip * (p.kt_major ? D * 128 : 64 * 128)) >> 4);
#pragma unroll
                    for (int sub = 0; sub < L::kSub; ++sub, b += k_sub)
#pragma unroll
                        for (int kk = 0; kk < (kCols < 64 ? kCols / 16 : 4); ++kk)
                            mma_ss(to, desc_sw128(q_lo + ((sub * kSubBytes + kk * 32) >> 4)), desc_sw128(b + kk * k_step), idesc, sub + kk > 0);
                    mma_commit(&ctrl->s_full);
                    mma_commit(&ctrl->k_free[st]);
                }
                __syncwarp();
            };
            if (ok && kOwnP) ok = k_here(0);
            if (ok) issue_s(0);
            for (int j = 0; j < steps && ok; ++j) {
                if (kOwnP && j + 1 < steps) {          // the next scores as soon as these have been read
                    ok = k_here(j + 1) && wait_all(&ctrl->s_free, (uint32_t)j & 1u, kErrSFree);
                    if (!ok) break;
                    issue_s(j + 1);
                }
                const int st = j % kSlots;
                ok = wait_all(&ctrl->v_full[st], (uint32_t)(j / kSlots) & 1u, kErrVFull);
                if (!ok) break;
#pragma unroll 1
                for (int half = 0; half < kHalves; ++half) {
                    ok = wait_all(&ctrl->p_full[half], (uint32_t)j & 1u, kErrP);
                    if (!ok) break;
                    tc_fence_after_sync();
                    if (in_range(j, half)) {
                        if (lead) {
                            const uint32_t b = v_lo + (uint32_t)(st * L::kKeyBytes >> 4) + half * 512;
#pragma unroll
                            for (int kk = 0; kk < 4; ++kk)
                                mma_ts(o_tmem, tmem_base + kPCol + half * 32 + kk * 8, desc_sw128(b + kk * 128), idesc_pv, (!first_pv || kk > 0) ? 1u : 0u);
                        }
                        __syncwarp();
                        first_pv = false;
                    }
                }
                if (!ok) break;
                commit(j + 1 < steps ? &ctrl->v_free[st] : &ctrl->o_full);
                if (kOwnP) commit(&ctrl->pv_done);
                else if (j + 1 < steps) issue_s(j + 1);
            }
            // tensor memory is released only after every MMA has completed
            commit(&ctrl->drain);
            wait_quiet(&ctrl->drain, 0);
            __syncwarp();
        }
    } else {
        // ------------------------------------------------------------------ softmax + epilogue
        const uint32_t lane_addr = tmem_base + ((uint32_t)(warp * 32) << 16);
        const uint32_t s_addr = lane_addr, o_addr = lane_addr + kKeys, p_addr = lane_addr + kPCol;
        const float sc = p.scale_log2;
        const float2 sc2 = make_float2(sc, sc);
        float m_used = -INFINITY, l_sum = 0.f;
        bool ok = true;
        for (int k = 0; k < steps; ++k) {
            ok = wait_all(&ctrl->s_full, (uint32_t)k & 1u, kErrS);
            if (!ok) break;
            tc_fence_after_sync();
            const int c0 = (klo + k) * kKeys;
            const int v_lo = my_begin - c0, v_hi = my_end - c0;  // valid keys of this step: [v_lo, v_hi)
            // P with columns of its own: before the first store of P or a rescale of O, PV(k-1) has to be complete (it usually is)
            auto pv_wait = [&]() {
                if (!kOwnP || k == 0) return true;
                const bool r = wait_all(&ctrl->pv_done, (uint32_t)(k - 1) & 1u, kErrPv);
                tc_fence_after_sync();
                return r;
            };
            auto offset = [&]() {
                const float m_eff = (m_used == -INFINITY) ? 0.f : m_used;
                return make_float2(-m_eff, -m_eff);
            };
            auto p_stored = [&](int half) {           // on its way to the tensor core
                tmem_st_wait();
                tc_fence_before_sync();
                __syncwarp();
                if (lane == 0) mbar_arrive(&ctrl->p_full[half]);
            };
            float2 acc0 = make_float2(0.f, 0.f), acc1 = make_float2(0.f, 0.f);
            if constexpr (kKeys == 64) {
                // The scores are fetched twice, 32 at a time, for four CTAs per SM (80 registers a thread).  Pieces outside all of
                // a warp's bands are not fetched (their P is 0), pieces inside all of them not masked.
                uint32_t r[32];
                bool none[2], whole[2];
                float mx = -INFINITY;
#pragma unroll
                for (int ch = 0; ch < 2; ++ch) {
                    const int a = v_lo - ch * 32, b = v_hi - ch * 32;
                    none[ch] = __all_sync(0xffffffffu, a >= 32 || b <= 0);
                    whole[ch] = __all_sync(0xffffffffu, a <= 0 && b >= 32);
                    if (none[ch]) continue;
                    tmem_ld32(s_addr + ch * 32, r);
                    tmem_ld_wait();
                    if (!whole[ch]) sm::mask_scores(r, a, b);
                    mx = fmaxf(mx, sm::max_score(r));
                }
                m_used = mx * sc;          // (the only step)
                const float2 nm2 = offset();
#pragma unroll
                for (int ch = 0; ch < 2; ++ch) {
                    if (none[ch]) {
#pragma unroll
                        for (int i = 0; i < 16; ++i) r[i] = 0u;
                    } else {
                        tmem_ld32(s_addr + ch * 32, r);
                        tmem_ld_wait();
                        if (!whole[ch]) sm::mask_scores(r, v_lo - ch * 32, v_hi - ch * 32);
                        sm::exp_scores<T, 32>(r, r, sc2, nm2, acc0, acc1);
                    }
                    tmem_st16(p_addr + ch * 16, r);
                }
                p_stored(0);
            } else {
                uint32_t r[kKeys];
#pragma unroll
                for (int ch = 0; ch < kKeys / kChunk; ++ch) tmem_ld32(s_addr + ch * kChunk, r + ch * kChunk);
                tmem_ld_wait();
                if (kOwnP) {                       // the next scores may be formed
                    tc_fence_before_sync();
                    __syncwarp();
                    if (lane == 0) mbar_arrive(&ctrl->s_free);
                }
                if (!__all_sync(0xffffffffu, v_lo <= 0 && v_hi >= kKeys)) sm::mask_scores(r, v_lo, v_hi);
                // Lazy rescale: only when a row's maximum has grown by more than 2^8 (false when both are -inf).  At D = 128 the
                // maximum and the sum change behind the vote, at D = 64 beside it.  us, behind / beside: d64 window 256 of
                // B4 H16 L4096 60.6 / 59.9, L1024 4 heads 7.23 / 7.17; d128 +-58 of L149 6.93 / 7.02, +-127 of H32 L2048 25.7 / 26.0.
                const float m_new = fmaxf(m_used, sm::max_score(r) * sc);
                const bool need = (m_new - m_used) > kRescaleThreshold;
                const bool any = __any_sync(0xffffffffu, need);
                float corr = 1.f;
                auto raise = [&]() {
                    corr = need ? ex2(m_used - m_new) : 1.f;
                    if (need) m_used = m_new;
                    if (any) l_sum *= corr;
                };
                if (kOwnP) raise();
                if (any && (!kOwnP || k > 0)) {
                    ok = pv_wait();
                    if (!ok) break;
                    if (!kOwnP) raise();
                    if (k > 0) rescale_o(o_addr, kCols / 16, corr);
                }
                const float2 nm2 = offset();
#pragma unroll
                for (int half = 0; half < 2; ++half) {
                    uint32_t* pk = r + half * 32;
                    sm::exp_scores<T, 64>(r + half * 64, pk, sc2, nm2, acc0, acc1);
                    if (kOwnP && half == 0) ok = pv_wait();
                    tmem_st32(p_addr + half * 32, pk);
                    p_stored(half);
                }
            }
            l_sum += (acc0.x + acc0.y) + (acc1.x + acc1.y);
            if (!ok) break;
        }
        const bool have_o = ok && steps > 0;
        if (have_o) {
            ok = wait_all(&ctrl->o_full, 0, kErrO);
            tc_fence_after_sync();
        } else if (ok) {
            ok = wait_all(&ctrl->q_full, 0, kErrQ);   // nothing to multiply; the copy of Q has to have landed all the same
        }
        // epilogue: O / l for band rows, V[start] for single-element rows, zero otherwise.  Rows are staged in
        // the Q tile's memory (every MMA has completed) in the 128-byte-swizzled tile layout and leave
        // through one tiled TMA store per 64 columns and warp (rows and columns past the end are clipped).
        // (all scores of a row -inf: zeros, or NaN like the row kernels)
        const float inv = kOwn || l_sum > 0.f ? 1.f / l_sum : 0.f;
        const int64_t head = bh * p.n_rows;
        const int u = u0 + warp * 32 + lane;
        const int64_t row_real = u < rows_v ? (int64_t)u * p.stride + real_res : -1;
        const int row_nnz = my_end > 0 ? 2 : (my_end == kSingle ? 1 : 0), row_start = my_begin;
        if (kLse && row_real >= 0 && ok) {
            float e = -INFINITY;
            if (row_nnz > 1) {
                e = lse_from_log2(m_used, l_sum);
            } else if (row_nnz == 1) {
                const T* qr = reinterpret_cast<const T*>(p.q) + (head + row_real) * p.d;
                const T* kb = reinterpret_cast<const T*>(p.k);
                const float s = p.kt_major ? dot_strided<T>(qr, kb + head * p.d + row_start, p.n_rows, p.d)
                                           : dot_strided<T>(qr, kb + (head + row_start) * p.d, 1, p.d);
                e = s * p.scale_log2 * kLn2;
            }
            p.lse[head + row_real] = e;
        }
        const T* vrow = reinterpret_cast<const T*>(p.v) + (head + row_start) * p.d;
        const int t = warp * 32 + lane;
        constexpr int kRead = kKeys == 64 ? 32 : kCols;             // columns of O in registers at a time
        uint32_t o_raw[kRead];
        float2 odd0 = make_float2(0.f, 0.f), odd1 = odd0;       // not finite: nor is the row
#pragma unroll
        for (int ch = 0; ch < kCols / 32; ++ch) {
            if (ch * 32 % kRead == 0 && have_o && ok) {
#pragma unroll
                for (int i = 0; i < kRead; i += 32) tmem_ld32(o_addr + ch * 32 + i, o_raw + i);
                tmem_ld_wait();
                if constexpr (kOwn) {
#pragma unroll
                    for (int j = 0; j < kRead; j += 8) {
                        odd0 = note_nonfinite(odd0, o_raw + j);
                        odd1 = note_nonfinite(odd1, o_raw + j + 4);
                    }
                }
            }
            const uint32_t* r = o_raw + ch * 32 % kRead;
            uint4 out[4];
            uint32_t* o32 = reinterpret_cast<uint32_t*>(out);
            if (row_nnz > 1 && have_o && ok) {
#pragma unroll
                for (int j = 0; j < 32; j += 2)
                    o32[j >> 1] = pack2<T>(__uint_as_float(r[j]) * inv, __uint_as_float(r[j + 1]) * inv);
            } else if (row_nnz == 1) {
#pragma unroll
                for (int i = 0; i < 4; ++i)
                    out[i] = ch * 32 + i * 8 < p.d ? *reinterpret_cast<const uint4*>(vrow + ch * 32 + i * 8) : make_uint4(0, 0, 0, 0);
            } else {
#pragma unroll
                for (int i = 0; i < 4; ++i) out[i] = make_uint4(0, 0, 0, 0);
            }
            uint8_t* srow = smem + (ch >> 1) * kSubBytes + t * 128;
#pragma unroll
            for (int i = 0; i < 4; ++i)
                *reinterpret_cast<uint4*>(srow + ((((ch & 1) * 4 + i) ^ (t & 7)) << 4)) = out[i];
        }
        if constexpr (kOwn) {
            const unsigned again = __ballot_sync(0xffffffffu, row_nnz > 1 && !isfinite(odd0.x + odd0.y + (odd1.x + odd1.y)));
            if (lane == 0) ctrl->again[warp] = again;
        }
        fence_proxy_async_smem();
        __syncwarp();
        if (lane == 0 && u0 + warp * 32 < rows_v) {
            for (int sub = 0; sub < L::kSub; ++sub)
                tma_store_4d(map + 3, smem + sub * kSubBytes + warp * 32 * 128, sub * 64, res, u0 + warp * 32, (int)bh);
            tma_store_commit();
            tma_store_wait_read();
        }
    }
    tc_fence_before_sync();
    __syncthreads();
    if (threadIdx.x == 0) publish_gave_up(p.status, &ctrl->gave_up);
    if (warp == kMmaWarp) {
        __syncwarp();
        tc_fence_after_sync();
        tmem_dealloc(tmem_base, kTmemCols);
    }
    if constexpr (kOwn) {
        const uint4 again = *reinterpret_cast<const uint4*>(ctrl->again), odd = *reinterpret_cast<const uint4*>(ctrl->single);
        if ((again.x | again.y | again.z | again.w | odd.x | odd.y | odd.z | odd.w) != 0) {
            if (warp < 4 && lane == 0) tma_store_wait_all();      // the tile is in memory before its rows are written again
            __syncthreads();
            rows_again<T>(p, make_uint4(again.x | odd.x, again.y | odd.y, again.z | odd.z, again.w | odd.w), bh, real_res, u0);
        }
    }
}

// `own`: a row's result depends on its own keys alone, also where Q, K or V is not finite at other ones.  It takes a look at
// every result and code for the rows that need it; that costs 3 % (fp16 B4 H16 L4096 d64 window 256 64.1 -> 66.0 us, bf16
// B8 H64 L32768 d128 window 1024 11.71 -> 12.12 ms).  Problems with d = 64 or 128 and classes of one length do without:
// they have only ever run on tensor cores, with finite V as a condition (splat_b200.h); the others came from the row
// kernels, which read nothing but a row's own keys.
template <typename T, int D, int kCols, int kKeys>
static int32_t launch(const Maps<4>& maps, const Params& prm, int64_t bh, cudaStream_t st) {
    const bool own = (prm.d != 64 && prm.d != 128) || prm.cls.longer != 0;
    auto kern = prm.lse != nullptr ? attention_wide_kernel<T, D, kCols, kKeys, true, true> : attention_wide_kernel<T, D, kCols, kKeys, false, true>;
    if constexpr (kCols == D)
        if (!own) kern = prm.lse != nullptr ? attention_wide_kernel<T, D, D, kKeys, true, false> : attention_wide_kernel<T, D, D, kKeys, false, false>;
    if (!allow_dynamic_smem(reinterpret_cast<const void*>(kern), Layout<D, kKeys>::kSmemBytes)) return SPLAT_ERR_LAUNCH;
    return launch_kernel(kern, prm.cls.grid(prm.stride, bh), kThreads, Layout<D, kKeys>::kSmemBytes, st, maps, prm);
}

}  // namespace wide
}  // namespace band

// Operands checked by attention_band().
int32_t attention_wide(const void* q, const void* k, int kt_major, const void* v, void* o, const float* lin, const float* tr,
                       const float* nnzs, int64_t bh, int64_t n_rows, int64_t d, int64_t stride, float scale, int32_t dtype,
                       int32_t* status_word, const int32_t* band_table, float* lse, cudaStream_t st) {
    using namespace band;
    wide::Params p;
    p.lin = lin; p.tr = tr; p.nnzs = nnzs; p.q = q; p.k = k; p.v = v; p.o = o; p.lse = lse;
    p.status = status_word; p.mirror = status_mirror(status_word);
    p.n_rows = n_rows; p.stride = (int)stride; p.d = (int)d;
    p.kt_major = kt_major; p.scale_log2 = scale * kLog2e;
    p.cls = Classes(n_rows, stride, wide::kTile);
    p.rows = reinterpret_cast<const int2*>(band_table);
    p.tiles = band_table != nullptr ? p.rows + n_rows : nullptr;
    // Classes of up to 64 rows at d <= 64: the kernel with 64-key steps, see above.
    const bool one_step = d <= 64 && p.cls.rows + (p.cls.longer > 0 ? 1 : 0) <= 64;
    const int keys = one_step ? 64 : 128;
    Maps<4> maps;
    for (int part = 0; part < 2; ++part) {
        if (!p.cls.has(part)) continue;
        CUtensorMap* m = maps.part[part];
        if (!p.cls.view(m, q, dtype, bh, n_rows, d, stride, part, wide::kTile) ||
            !(kt_major ? make_map_kt(m + 1, k, dtype, bh, n_rows, d, d > 64 ? 128 : 64)
                       : p.cls.view(m + 1, k, dtype, bh, n_rows, d, stride, part, keys)) ||
            !p.cls.view(m + 2, v, dtype, bh, n_rows, d, stride, part, keys) ||
            !p.cls.view(m + 3, o, dtype, bh, n_rows, d, stride, part, 32))
            return SPLAT_ERR_DRIVER;
    }
    auto launch = [&](auto element) {
        using T = decltype(element);
        if (d > 64) return wide::launch<T, 128, 128, 128>(maps, p, bh, st);
        if (d > 32) return one_step ? wide::launch<T, 64, 64, 64>(maps, p, bh, st) : wide::launch<T, 64, 64, 128>(maps, p, bh, st);
        return one_step ? wide::launch<T, 64, 32, 64>(maps, p, bh, st) : wide::launch<T, 64, 32, 128>(maps, p, bh, st);
    };
    return dtype == SPLAT_BF16 ? launch(__nv_bfloat16()) : launch(__half());
}

}  // namespace splat
