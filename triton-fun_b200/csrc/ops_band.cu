// SDDMM and SpMM over ACSR for patterns whose rows are contiguous bands after regrouping by residue class (the
// same condition and the same tensor-map views as the fused kernel, attention_band.cu / attention_wide.cu):
// TMA-staged tiles, tcgen05 MMAs with the accumulator in tensor memory.  Both kernels are bound by the
// (BH, L, trailing_dim) sparse operand they write or read; the tensor cores only have to keep up with it.
//
//   sddmm_band_kernel   S[i, j'] = Q[i] . K[start_i + j' stride]   (SPLAT/r_sddmm.py:16-114)
//       S(k) = Q K(k)^T (tcgen05.mma 128x64x16) into one of two 64-column buffers; a thread reads the 64 scores
//       of its row, packs them and hands them on as whole 16-byte pieces of the sparse row.
//   spmm_band_kernel    O[i] = sum_j' P[i, j'] V[start_i + j' stride]   (SPLAT/r_spmm.py:14-164)
//       cp.async brings the 16-byte pieces of P that a 64-key step needs; a thread takes its row's pieces,
//       shifts them into place and stores them in tensor memory as the A operand of O += P(k) V(k).
// One CTA = one 128-row tile of one (bh, class).  Row warps: thread = row = tensor-memory lane, one warp to 32 rows or two that
// share a step's columns (see two_warps()); then a TMA and an MMA warp.
//
// The sparse layout shifts every row by its own number of elements against the dense columns, so a row's 64
// columns of a step begin anywhere in a 16-byte piece of the sparse array.  They begin at the SAME place in
// every step (64 elements are eight pieces): with e the element index of the step's first column and
// sft = e mod 8, a step of a row is eight whole pieces made of the last sft elements of the step before and
// the first 64 - sft of this one (with two warps to the rows four pieces of 32 columns, and the columns in front read with
// the warp's own).  The thread forms them in registers (barrel()), and a warp moves them through a swizzled staging tile
// so that global memory sees 128 or 64 contiguous bytes per row.  The kernels before did this
// with 2-byte accesses, or 16-byte ones of 32 different rows per instruction: 70 % of the L1 wavefronts, a
// third of the memory bandwidth.  B4 H16 L4096 d64 fp16 window 256: SDDMM 102 -> 59 us, SpMM 114 -> 65.
// Pieces that a row's band only partly covers (its ends, if trailing_dim is no multiple of 8) are stored element
// by element.  Rows with one non-zero (described by the metadata as column `start`, outside the band) and rows
// with none are fixed up by plain loads, padding slots of S are written as zero like the CUDA-core kernels do.
// Any d that is a multiple of 8 up to 128 and any L, as in attention_wide.cu.
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

namespace ops {

using sm::pack2;

constexpr int kTile = 128;
constexpr int kStep = 64;
constexpr int kSubBytes = kTile * 128;          // 128 rows x 128 bytes
constexpr int kStepBytesPerSub = kStep * 128;   // 64 keys x 128 bytes
// What these kernels are bound by is instructions: with waits of a few of them (tc_ptx.cuh) and the control block at
// constant addresses SDDMM at d = 128 went from 70.1 to 66.2 us, SpMM from 70.1 to 68.7 (B4 H16 L4096 window 256).
constexpr int kStages = 3;                      // K / V ring
constexpr int kSingle = -1, kEmpty = INT_MIN / 2;   // row kinds, as in the band table (acsr_meta.cu)
enum : int { kErrQ = 11, kErrFull = 12, kErrEmpty = 13, kErrReady = 14, kErrFree = 15 };

struct Params {
    const float* lin;
    const float* tr;
    const float* nnzs;
    const int2* rows;    // band table, or null
    const int2* tiles;
    const void* q;       // sddmm: (BH, L, d), for rows with one non-zero
    const void* kv;      // sddmm: K, spmm: V
    void* o;             // spmm: (BH, L, d)
    uint16_t* sparse;    // sddmm: S out, spmm: P in, (BH, L, trailing_dim), rounded down to 16 bytes ...
    int lead;            // ... and the elements lost by that
    int32_t* status;
    int32_t* mirror;     // host copy of the status word, or null
    int64_t n_rows;      // L
    int stride;
    Classes cls;
    int d;
    int trailing_dim;
    int kt_major;        // sddmm: K is a contiguous (BH, d, L) array (keys innermost), stride 1 only
};

template <typename T> __device__ __forceinline__ float to_f(T v);
template <> __device__ __forceinline__ float to_f<__half>(__half v) { return __half2float(v); }
template <> __device__ __forceinline__ float to_f<__nv_bfloat16>(__nv_bfloat16 v) { return __bfloat162float(v); }

struct Control {
    uint64_t q_full;
    uint64_t full[kStages];
    uint64_t empty[kStages];
    uint64_t ready[2];   // sddmm: scores of a step in tensor memory; spmm: P of a step in tensor memory
    uint64_t freed[2];   // the consumer is through with that buffer
    uint64_t drain;
    uint32_t tmem_base;
    int32_t abort_at_entry;
    int32_t gave_up;     // code of a wait that ran out
    int32_t lo[4];
    int32_t hi[4];
    uint32_t again[4];   // spmm: rows whose result is not finite
};

// The row warps' share of the prologue: this thread's band, and without a table the warp's key range.
__device__ __forceinline__ int2 load_band(const Params& p, Control* ctrl, int real_res, int u, int warp, int lane) {
    int2 band = make_int2(0, kEmpty);
    if (u < p.cls.rows_of(real_res)) {
        if (p.rows != nullptr) {
            band = __ldg(p.rows + p.cls.first_row(real_res) + u);
        } else {
            const RowAffine ra = row_affine(p.lin, p.tr, p.nnzs, (int64_t)u * p.stride + real_res);
            if (ra.nnz > 1) {
                band.x = (ra.start - real_res) / p.stride;
                band.y = band.x + ra.nnz;
            } else if (ra.nnz == 1) {
                band = make_int2(ra.start, kSingle);
            }
        }
    }
    if (p.rows == nullptr && warp < 4) {
        const int lo = warp_min_i(band.y > 0 ? band.x : INT_MAX), hi = warp_max_i(max(band.y, 0));
        if (lane == 0) { ctrl->lo[warp] = lo; ctrl->hi[warp] = hi; }
    }
    return band;
}
__device__ __forceinline__ void key_range(int rows_v, const Control* ctrl, int* klo, int* khi) {
    int lo = INT_MAX, hi = 0;
    for (int w = 0; w < 4; ++w) { lo = min(lo, ctrl->lo[w]); hi = max(hi, ctrl->hi[w]); }
    hi = min(hi, rows_v);
    *klo = hi > 0 ? lo / kStep : 0;
    *khi = (hi + kStep - 1) / kStep;
}

// out = 2 kWords elements (two per word) of the eight more in x from element t on, 0 <= t <= kMax.
template <int kMax, int kWords>
__device__ __forceinline__ void barrel(uint32_t (&x)[kWords + 4], int t, uint32_t (&out)[kWords]) {
    const int s = t >> 1;
    if (kMax == 8 && (s & 4)) {
#pragma unroll
        for (int i = 0; i < kWords; ++i) x[i] = x[i + 4];
    }
    if (s & 2) {
#pragma unroll
        for (int i = 0; i < kWords + 2; ++i) x[i] = x[i + 2];
    }
    if (s & 1) {
#pragma unroll
        for (int i = 0; i < kWords + 3; ++i) x[i] = x[i + 1];
    }
    const uint32_t shift = (t & 1) * 16;
#pragma unroll
    for (int i = 0; i < kWords; ++i) out[i] = __funnelshift_r(x[i], x[i + 1], shift);
}
// 32 bit, 8 consecutive columns of tensor memory
__device__ __forceinline__ void tmem_ld8(uint32_t taddr, uint32_t* r) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]) : "r"(taddr) : "memory");
}

// ---------------------------------------------------------------------------------------------
// SDDMM
// ---------------------------------------------------------------------------------------------
template <int D, int kRowWarps> struct SddmmLayout {
    static constexpr int kSub = D / 64;
    static constexpr int kQBytes = kSub * kSubBytes;
    static constexpr int kItemBytes = kSub * kStepBytesPerSub;
    static constexpr int kRingOff = kQBytes;
    static constexpr int kStageOff = kRingOff + kStages * kItemBytes;
    static constexpr int kSmemBytes = kStageOff + kTile * 128 + 1024;   // + alignment slack
    static constexpr int kPerSm = D == 128 || kRowWarps == 8 ? 2 : 3;
    static constexpr int kThreads = (kRowWarps + 2) * 32;
};

template <typename T, int D, int kRowWarps>
__global__ void __launch_bounds__(SddmmLayout<D, kRowWarps>::kThreads, SddmmLayout<D, kRowWarps>::kPerSm)
sddmm_band_kernel(const __grid_constant__ Maps<2> maps, const Params p) {
    using L = SddmmLayout<D, kRowWarps>;
    constexpr int kTmaWarp = kRowWarps, kMmaWarp = kRowWarps + 1;
    constexpr int kHalves = kRowWarps / 4, kCols = kStep / kHalves;      // warps that share 32 rows, columns of a step of each
    constexpr int kTmemCols = 128;   // two 64-column score buffers
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = smem_raw + (((smem_u32(smem_raw) + 1023) & ~1023u) - smem_u32(smem_raw));
    uint8_t* s_ring = smem + L::kRingOff;
    __shared__ Control ctrl_mem;             // (static: constant addresses)
    Control* const ctrl = &ctrl_mem;
    __shared__ int4 about_mem[kRowWarps * 32];      // what a lane knows of its row, for the lanes that store it

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int real_res = blockIdx.y, res = p.cls.in_part(real_res), rows_v = p.cls.rows_of(real_res);
    const CUtensorMap* map = maps.part[p.cls.part(real_res)];       // Q, K
    const int64_t bh = blockIdx.z;
    const int u0 = blockIdx.x * kTile;
    if (u0 >= rows_v) return;       // (a class one tile shorter than the longest)

    int2 band = make_int2(0, kEmpty);
    int klo = 0, khi = 0, item = 0;
    auto load_item = [&]() {
        const int stage = item % kStages, k = klo + item;
        if (item >= kStages && !wait_bar(&ctrl->empty[stage], ((uint32_t)(item / kStages) & 1u) ^ 1u, &ctrl->gave_up, kErrEmpty)) return false;
        mbar_arrive_expect_tx(&ctrl->full[stage], L::kItemBytes);
        if (p.kt_major)      // one [d][64 keys] block (K layouts: see attention_band.cu)
            tma_load_4d(s_ring + stage * L::kItemBytes, map + 1, &ctrl->full[stage], k * kStep, 0, (int)bh, 0);
        else
            for (int sub = 0; sub < L::kSub; ++sub)
                tma_load_4d(s_ring + stage * L::kItemBytes + sub * kStepBytesPerSub, map + 1, &ctrl->full[stage], sub * 64, res,
                            k * kStep, (int)bh);
        ++item;
        return true;
    };
    if (warp == kMmaWarp) {
        depend_wait();
        tmem_alloc(&ctrl->tmem_base, kTmemCols);
        tmem_relinquish();
    } else if (warp == kTmaWarp) {
        if (lane == 0) {
            tma_prefetch_desc(map);
            tma_prefetch_desc(map + 1);
            mbar_init(&ctrl->q_full, 1);
            for (int i = 0; i < kStages; ++i) {
                mbar_init(&ctrl->full[i], 1);
                mbar_init(&ctrl->empty[i], 1);
            }
            for (int b = 0; b < 2; ++b) {
                mbar_init(&ctrl->ready[b], 1);
                mbar_init(&ctrl->freed[b], kRowWarps);
            }
            mbar_init(&ctrl->drain, 1);
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
                    klo = range.x / kStep;
                    khi = (range.y + kStep - 1) / kStep;
                    while (item < kStages && klo + item < khi) load_item();
                }
            }
            if (p.tiles != nullptr)
                for (int w = 0; w < 4; ++w) { ctrl->lo[w] = range.x; ctrl->hi[w] = range.y; }
        }
    } else {
        depend_wait();
        band = load_band(p, ctrl, real_res, u0 + (warp & 3) * 32 + lane, warp, lane);
    }
    tc_fence_before_sync();
    __syncthreads();
    tc_fence_after_sync();
    depend_release();
    const uint32_t tmem_base = ctrl->tmem_base;
    if (ctrl->abort_at_entry != 0) {
        if (warp == kMmaWarp) tmem_dealloc(tmem_base, kTmemCols);
        return;
    }
    key_range(rows_v, ctrl, &klo, &khi);

    if (warp == kTmaWarp) {
        // ------------------------------------------------------------------ TMA producer
        if (lane == 0) {
            bool ok = true;
            while (ok && klo + item < khi) ok = load_item();
            if (!ok)   // leave only after the copies already issued have landed
                for (int i = max(0, item - kStages); i < item; ++i) wait_quiet(&ctrl->full[i % kStages], (uint32_t)(i / kStages) & 1u);
            wait_quiet(&ctrl->q_full, 0);
        }
    } else if (warp == kMmaWarp) {
        // ------------------------------------------------------------------ MMA issuer
        // (the whole warp walks the loop on warp-uniform values and one elected lane issues)
        if (khi > klo) {
            constexpr uint32_t fmt = std::is_same<T, __nv_bfloat16>::value ? 1u : 0u;
            const uint32_t idesc = instr_desc_f16(fmt, kTile, kStep, p.kt_major ? 1u : 0u);
            const bool lead = elect_one();
            const uint32_t ring_addr = smem_u32(s_ring), q_base = smem_u32(smem);
            bool ok = wait_all(&ctrl->q_full, 0, &ctrl->gave_up, kErrQ);
            for (int k = klo; k < khi && ok; ++k) {
                const int it = k - klo, b = it & 1;
                ok = wait_all(&ctrl->full[it % kStages], (uint32_t)(it / kStages) & 1u, &ctrl->gave_up, kErrFull);
                if (ok && it >= 2) ok = wait_all(&ctrl->freed[b], (uint32_t)((it >> 1) - 1) & 1u, &ctrl->gave_up, kErrFree);
                if (!ok) break;
                tc_fence_after_sync();
                const uint32_t b_base = ring_addr + (it % kStages) * L::kItemBytes;
#pragma unroll
                for (int kk = 0; kk < D / 16; ++kk) {
                    const uint64_t da = smem_desc_sw128(q_base + (kk >> 2) * kSubBytes + (kk & 3) * 32, 16, 1024);
                    const uint64_t db = p.kt_major
                        ? smem_desc_sw128(b_base + kk * 2048, D * 128, 1024)
                        : smem_desc_sw128(b_base + (kk >> 2) * kStepBytesPerSub + (kk & 3) * 32, 16, 1024);
                    if (lead) mma_ss(tmem_base + b * kStep, da, db, idesc, kk > 0);
                }
                if (lead) {
                    mma_commit(&ctrl->ready[b]);
                    mma_commit(&ctrl->empty[it % kStages]);
                }
            }
            // let the tensor pipe drain before tensor memory is released
            if (lead) mma_commit(&ctrl->drain);
            wait_quiet(&ctrl->drain, 0);
            __syncwarp();
        }
    } else {
        // ------------------------------------------------------------------ row warps
        const int rw = warp & 3, half = warp >> 2;
        const uint32_t s_addr = tmem_base + ((uint32_t)(rw * 32) << 16);
        uint8_t* stage = smem + L::kStageOff + warp * 32 * (kCols * 2);
        const int64_t head = bh * p.n_rows;
        // element index (in p.sparse) of class column 0 of this row, were its band to reach that far
        const int64_t e_row = p.lead + (head + (int64_t)(u0 + rw * 32 + lane) * p.stride + real_res) * p.trailing_dim - band.x;
        const int sft = (int)(e_row & 7);
        constexpr int kPieces = kCols / 8, kRows = 32 / kPieces;       // 16-byte pieces of a row, rows of a warp's store
        // The rows whose pieces this lane stores: row kRows i + lane / kPieces, piece lane mod kPieces.  Byte offset of the piece of
        // class column 0's step, and the column range in which the piece's first column is inside the band.
        // (what a lane knows of its row reaches the others through shared memory: five shuffles per row took 1 300 cycles)
        const int64_t e_base = __shfl_sync(0xffffffffu, e_row + band.x, 0) & ~(int64_t)7;
        uint8_t* base = reinterpret_cast<uint8_t*>(p.sparse + e_base);
        const int e_rel = (int)(e_row - e_base);
        int4* about = about_mem + warp * 32;
        about[lane] = make_int4(e_rel, u0 + rw * 32 + lane < rows_v ? 1 : 0, band.x, max(band.y, -64));     // (-64, below every step: no band)
        __syncwarp();
        int32_t off[kPieces];
        int lo8[kPieces], hi8[kPieces];
#pragma unroll
        for (int i = 0; i < kPieces; ++i) {
            const int4 r = about[kRows * i + lane / kPieces];
            const int behind = lane % kPieces * 8 - (r.x & 7);       // first column - the warp's first of the step
            off[i] = (r.x + behind) * 2;
            lo8[i] = r.z - behind;
            hi8[i] = r.w - behind;
        }
        // this warp's first and last columns of its rows' bands
        const int w_lo = warp_min_i(band.y > 0 ? band.x : INT_MAX), w_hi = warp_max_i(band.y > 0 ? band.y + sft : 0);
        uint32_t tail[4] = {0, 0, 0, 0};       // the eight elements before the warp's columns of the step
        bool ok = true;
        for (int k = klo; k <= khi && khi > klo; ++k) {      // khi: what is left of the last step
            const int it = k - klo, b = it & 1, c0 = k * kStep + half * kCols;
            const bool active = c0 < w_hi && c0 + kCols > w_lo;
            if (k < khi) {
                ok = wait_all(&ctrl->ready[b], (uint32_t)(it >> 1) & 1u, &ctrl->gave_up, kErrReady);
                if (!ok) break;
                tc_fence_after_sync();
            }
            const uint32_t from = s_addr + b * kStep + half * kCols;
            uint32_t x[kCols / 2 + 4], out[kCols / 2];
            if (active && k < khi) {
                uint32_t r[kCols];
#pragma unroll
                for (int c = 0; c < kCols; c += 32) tmem_ld32(from + c, r + c);
                tmem_ld_wait();
#pragma unroll
                for (int i = 0; i < kCols / 2; ++i) x[4 + i] = pack2<T>(__uint_as_float(r[2 * i]), __uint_as_float(r[2 * i + 1]));
            } else {
#pragma unroll
                for (int i = 4; i < kCols / 2 + 4; ++i) x[i] = 0u;
            }
            // The eight columns in front: the warp's own last ones, or, of two warps that share the rows, columns 24-31 for the
            // second one's 32, and columns 56-63 for the first one's of the next step.
            if constexpr (kHalves == 2) {
                if (!half) {
#pragma unroll
                    for (int i = 0; i < 4; ++i) x[i] = tail[i];
                }
                if (k < khi) {
                    uint32_t t[8];
                    tmem_ld8(s_addr + b * kStep + (half ? kCols : kStep) - 8, t);
                    tmem_ld_wait();
#pragma unroll
                    for (int i = 0; i < 4; ++i) tail[i] = pack2<T>(__uint_as_float(t[2 * i]), __uint_as_float(t[2 * i + 1]));
                }
                if (half) {
#pragma unroll
                    for (int i = 0; i < 4; ++i) x[i] = tail[i];
                }
            }
            if (k < khi) {
                tc_fence_before_sync();
                __syncwarp();
                if (lane == 0) mbar_arrive(&ctrl->freed[b]);   // the buffer may take the scores of step k + 2
            }
            if (!active) continue;
            if constexpr (kHalves == 1) {
#pragma unroll
                for (int i = 0; i < 4; ++i) x[i] = tail[i];
#pragma unroll
                for (int i = 0; i < 4; ++i) tail[i] = x[kCols / 2 + i];
            }
            barrel<8>(x, 8 - sft, out);
#pragma unroll
            for (int q4 = 0; q4 < kPieces; ++q4)
                *reinterpret_cast<uint4*>(stage + lane * (kCols * 2) + ((q4 ^ (kHalves == 2 ? (lane >> 1) & 3 : lane & 7)) << 4)) =
                    make_uint4(out[4 * q4], out[4 * q4 + 1], out[4 * q4 + 2], out[4 * q4 + 3]);
            __syncwarp();
            uint8_t* to = base + (int64_t)c0 * 2;
#pragma unroll
            for (int i = 0; i < kPieces; ++i) {
                const int row = kRows * i + lane / kPieces;
                const uint4 v = *reinterpret_cast<const uint4*>(
                    stage + row * (kCols * 2) + ((lane % kPieces ^ (kHalves == 2 ? (row >> 1) & 3 : row & 7)) << 4));
                if (c0 >= lo8[i] && c0 + 8 <= hi8[i]) {
                    *reinterpret_cast<uint4*>(to + off[i]) = v;
                } else if (c0 + 8 > lo8[i] && c0 < hi8[i]) {
                    const uint16_t* e = reinterpret_cast<const uint16_t*>(&v);
#pragma unroll
                    for (int j = 0; j < 8; ++j)
                        if (c0 + j >= lo8[i] && c0 + j < hi8[i]) reinterpret_cast<uint16_t*>(to + off[i])[j] = e[j];
                }
            }
            __syncwarp();   // the staging tile is rewritten in the next step
        }
        // padding slots, rows with one non-zero (a dot product by hand) and rows with none
        // (eight lanes per row: one element each of the pieces at either end, 16-byte stores between; a warp per row,
        // element by element, took 2 to 3 us of a small call; either warp of the rows has half of them)
        const int4 mine = about[lane];
        const int nnz = mine.w > 0 ? mine.w - mine.z : (mine.w == kSingle ? 1 : 0);
        if (__any_sync(0xffffffffu, mine.y != 0 && nnz < p.trailing_dim)) {
            uint16_t* to = reinterpret_cast<uint16_t*>(base);
#pragma unroll 1
            for (int i = 8 / kHalves * half; i < 8 / kHalves * (half + 1); ++i) {
                const int4 r = about[4 * i + (lane >> 3)];
                const int l = lane & 7, slot0 = r.x + r.z, end = slot0 + p.trailing_dim;
                const int from = r.y == 0 ? end : slot0 + (r.w > 0 ? r.w - r.z : (r.w == kSingle ? 1 : 0));
                const int first = (from + 7) & ~7, last = end & ~7;      // whole pieces
                if (from + l < min(first, end)) to[from + l] = 0;
                for (int e = first + l * 8; e < last; e += 64) *reinterpret_cast<uint4*>(to + e) = make_uint4(0, 0, 0, 0);
                if (last >= first && last + l < end) to[last + l] = 0;
            }
        }
        unsigned todo = half == 0 ? __ballot_sync(0xffffffffu, mine.y != 0 && mine.w == kSingle) : 0;
        const T* qg = reinterpret_cast<const T*>(p.q);
        const T* kg = reinterpret_cast<const T*>(p.kv);
        while (todo) {
            const int rr = __ffs(todo) - 1;
            todo &= todo - 1;
            const int start = about[rr].z;
            const int64_t row_real = head + (int64_t)(u0 + rw * 32 + rr) * p.stride + real_res;
            uint16_t* row = p.sparse + p.lead + row_real * p.trailing_dim;
            float acc = 0.f;
            const T* qr = qg + row_real * p.d;
            // K[bh][start][c]: rows of d elements, or column `start` of the (d, L) array
            const int64_t k0 = p.kt_major ? head * p.d + start : (head + start) * p.d;
            const int64_t kc = p.kt_major ? p.n_rows : 1;
            for (int c = lane; c < p.d; c += 32) acc += to_f<T>(qr[c]) * to_f<T>(kg[k0 + c * kc]);
            acc = warp_sum(acc);
            if (lane == 0) *reinterpret_cast<T*>(row) = DT<T>::from_f(acc);
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
}

// ---------------------------------------------------------------------------------------------
// SpMM
// ---------------------------------------------------------------------------------------------
// kPerSm CTAs share an SM: two with three steps of P on their way, or, at D = 64 and with more than two CTAs per SM to
// run, three with two steps each (with one warp to 32 rows 112 registers and some spills): B3 H44 L7680 +-224 294 -> 270 us, B2 H116 L4032
// +-17 165 -> 144 us; a single wave (H8 L1024) is faster with two, 7.5 against 8.3 us.
template <int D, int kPerSm, int kRowWarps> struct SpmmLayout {
    static constexpr int kThreads = (kRowWarps + 2) * 32;
    static constexpr int kPieces = kStep * 4 / kRowWarps / 8 + 1;      // 16-byte pieces of a row's columns of a step (of one warp)
    static constexpr int kPPitch = kPieces * 16;                  // (an odd number of pieces: conflict-free 16-byte reads)
    static constexpr int kSub = D / 64;
    static constexpr int kItemBytes = kSub * kStepBytesPerSub;    // 64 keys of V
    static constexpr int kPBytes = kRowWarps * 32 * kPPitch;      // a step's pieces of P
    static constexpr int kPStages = kPerSm == 2 ? 3 : 2;          // steps of P on their way
    static constexpr int kPOff = 0;                               // later reused as the output's staging
    static constexpr int kFront = (kPStages * kPBytes + 1023) / 1024 * 1024;
    static constexpr int kRingOff = kFront;
    static constexpr int kSmemBytes = kRingOff + kStages * kItemBytes + 1024;   // + alignment slack
    static_assert(kFront >= kSub * kSubBytes, "output staging");
};

template <typename T, int D, int kPerSm, int kRowWarps>
__global__ void __launch_bounds__((kRowWarps + 2) * 32, kPerSm)
spmm_band_kernel(const __grid_constant__ Maps<2> maps, const Params p) {
    using L = SpmmLayout<D, kPerSm, kRowWarps>;
    constexpr int kPStages = L::kPStages, kPPitch = L::kPPitch, kPieces = L::kPieces, kTmaWarp = kRowWarps, kMmaWarp = kRowWarps + 1;
    constexpr int kHalves = kRowWarps / 4, kCols = kStep / kHalves;      // warps that share 32 rows, columns of a step of each
    constexpr int kTmemCols = D == 128 ? 256 : 128;   // the output accumulator, two steps of P (32 columns each)
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = smem_raw + (((smem_u32(smem_raw) + 1023) & ~1023u) - smem_u32(smem_raw));
    uint8_t* s_ring = smem + L::kRingOff;
    __shared__ Control ctrl_mem;             // (static: constant addresses)
    Control* const ctrl = &ctrl_mem;

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int real_res = blockIdx.y, res = p.cls.in_part(real_res), rows_v = p.cls.rows_of(real_res);
    const CUtensorMap* map = maps.part[p.cls.part(real_res)];       // V, O
    const int64_t bh = blockIdx.z;
    const int u0 = blockIdx.x * kTile;
    if (u0 >= rows_v) return;       // (a class one tile shorter than the longest)

    int2 band = make_int2(0, kEmpty);
    int klo = 0, khi = 0, item = 0;
    auto load_item = [&]() {
        const int stage = item % kStages, k = klo + item;
        if (item >= kStages && !wait_bar(&ctrl->empty[stage], ((uint32_t)(item / kStages) & 1u) ^ 1u, &ctrl->gave_up, kErrEmpty)) return false;
        mbar_arrive_expect_tx(&ctrl->full[stage], L::kItemBytes);
        for (int sub = 0; sub < L::kSub; ++sub)
            tma_load_4d(s_ring + stage * L::kItemBytes + sub * kStepBytesPerSub, map, &ctrl->full[stage], sub * 64, res, k * kStep,
                        (int)bh);
        ++item;
        return true;
    };
    if (warp == kMmaWarp) {
        depend_wait();
        tmem_alloc(&ctrl->tmem_base, kTmemCols);
        tmem_relinquish();
    } else if (warp == kTmaWarp) {
        if (lane == 0) {
            tma_prefetch_desc(map);
            for (int i = 0; i < kStages; ++i) {
                mbar_init(&ctrl->full[i], 1);
                mbar_init(&ctrl->empty[i], 1);
            }
            for (int b = 0; b < 2; ++b) {
                mbar_init(&ctrl->ready[b], kRowWarps);
                mbar_init(&ctrl->freed[b], 1);
            }
            mbar_init(&ctrl->drain, 1);
            mbar_fence_init();
            depend_wait();
            int2 range = make_int2(0, 0);
            if (p.tiles != nullptr) range = __ldg(p.tiles + real_res * p.cls.tile_pitch + blockIdx.x);
            const int32_t stop = entry_status(p.status, p.mirror);
            ctrl->abort_at_entry = stop;
            ctrl->gave_up = 0;
            for (int w = 0; w < 4; ++w) ctrl->again[w] = 0;
            if (stop == 0 && range.y > 0) {
                klo = range.x / kStep;
                khi = (range.y + kStep - 1) / kStep;
                while (item < kStages && klo + item < khi) load_item();
            }
            if (p.tiles != nullptr)
                for (int w = 0; w < 4; ++w) { ctrl->lo[w] = range.x; ctrl->hi[w] = range.y; }
        }
    } else {
        depend_wait();
        band = load_band(p, ctrl, real_res, u0 + (warp & 3) * 32 + lane, warp, lane);
    }
    tc_fence_before_sync();
    __syncthreads();
    tc_fence_after_sync();
    depend_release();
    const uint32_t tmem_base = ctrl->tmem_base;
    if (ctrl->abort_at_entry != 0) {
        if (warp == kMmaWarp) tmem_dealloc(tmem_base, kTmemCols);
        return;
    }
    key_range(rows_v, ctrl, &klo, &khi);
    const uint32_t p_col = D;        // tensor-memory columns of P behind the accumulator

    if (warp == kTmaWarp) {
        // ------------------------------------------------------------------ TMA producer (V)
        if (lane == 0) {
            bool ok = true;
            while (ok && klo + item < khi) ok = load_item();
            if (!ok)
                for (int i = max(0, item - kStages); i < item; ++i) wait_quiet(&ctrl->full[i % kStages], (uint32_t)(i / kStages) & 1u);
        }
    } else if (warp == kMmaWarp) {
        // ------------------------------------------------------------------ MMA issuer
        if (khi > klo) {
            constexpr uint32_t fmt = std::is_same<T, __nv_bfloat16>::value ? 1u : 0u;
            constexpr uint32_t idesc = instr_desc_f16(fmt, kTile, D, 1);   // A (P) from tensor memory, B (V) MN-major
            const bool lead = elect_one();
            const uint32_t ring_addr = smem_u32(s_ring);
            bool ok = true;
            for (int k = klo; k < khi && ok; ++k) {
                const int it = k - klo, b = it & 1;
                ok = wait_all(&ctrl->full[it % kStages], (uint32_t)(it / kStages) & 1u, &ctrl->gave_up, kErrFull);
                if (ok) ok = wait_all(&ctrl->ready[b], (uint32_t)(it >> 1) & 1u, &ctrl->gave_up, kErrReady);
                if (!ok) break;
                tc_fence_after_sync();
                const uint32_t b_base = ring_addr + (it % kStages) * L::kItemBytes;
#pragma unroll
                for (int kk = 0; kk < kStep / 16; ++kk) {
                    const uint64_t db = smem_desc_sw128(b_base + kk * 2048, kStepBytesPerSub, 1024);
                    if (lead) mma_ts(tmem_base, tmem_base + p_col + b * 32 + kk * 8, db, idesc, (it > 0 || kk > 0) ? 1u : 0u);
                }
                if (lead) {
                    mma_commit(&ctrl->freed[b]);
                    mma_commit(&ctrl->empty[it % kStages]);
                }
            }
            if (lead) mma_commit(&ctrl->drain);   // every MMA complete: O final
            wait_quiet(&ctrl->drain, 0);
            __syncwarp();
        }
    } else {
        // ------------------------------------------------------------------ P loaders + epilogue
        const int rw = warp & 3, half = warp >> 2;
        const uint32_t lane_addr = tmem_base + ((uint32_t)(rw * 32) << 16);
        const int64_t head = bh * p.n_rows;
        const int64_t e_row = p.lead + (head + (int64_t)(u0 + rw * 32 + lane) * p.stride + real_res) * p.trailing_dim - band.x;
        const int sft = (int)((e_row + (int64_t)klo * kStep) & 7);
        // Pieces of a step: kPieces per row, piece idx = lane + 32 i of row idx / kPieces: byte offset of the
        // piece in class column 0's step, and the range of the warp's first column in which it holds some of the band.
        const int64_t e_base = __shfl_sync(0xffffffffu, e_row + band.x, 0) & ~(int64_t)7;
        const uint8_t* base = reinterpret_cast<const uint8_t*>(p.sparse + e_base);
        int4* about = reinterpret_cast<int4*>(smem + L::kPOff + warp * 32 * kPPitch);      // (as in SDDMM)
        about[lane] = make_int4((int)(e_row - e_base), sft, band.x, band.y);
        __syncwarp();
        int32_t off[kPieces];
        int first[kPieces], last[kPieces];
#pragma unroll
        for (int i = 0; i < kPieces; ++i) {
            const int idx = lane + 32 * i, row = idx / kPieces, piece = idx - row * kPieces;
            const int4 r = about[row];
            const int behind = piece * 8 - r.y;
            off[i] = ((r.x & ~7) + piece * 8) * 2;
            first[i] = r.z - behind - 7;
            last[i] = r.w > 0 ? r.w - behind : INT_MIN;
        }
        __syncwarp();
        auto fetch = [&](int it) {
            if (klo + it < khi) {
                const uint32_t dst = smem_u32(smem + L::kPOff) + (it % kPStages) * L::kPBytes + warp * 32 * kPPitch + lane * 16;
                const int c0 = (klo + it) * kStep + half * kCols;
                const uint8_t* from = base + (int64_t)c0 * 2;
#pragma unroll
                for (int i = 0; i < kPieces; ++i)
                    if (c0 >= first[i] && c0 < last[i])
                        asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst + i * 512), "l"(from + off[i]) : "memory");
            }
            asm volatile("cp.async.commit_group;" ::: "memory");
        };
        const int w_lo = warp_min_i(band.y > 0 ? band.x : INT_MAX), w_hi = warp_max_i(band.y > 0 ? band.y : 0);
        for (int it = 0; it < kPStages; ++it) fetch(it);
        bool ok = true;
        for (int k = klo; k < khi; ++k) {
            const int it = k - klo, b = it & 1;
            asm volatile("cp.async.wait_group %0;" ::"n"(kPStages - 1) : "memory");
            __syncwarp();
            const int c0 = k * kStep + half * kCols;
            const int lo = band.x - c0, hi = band.y - c0;       // valid columns of the warp's: [lo, hi)
            uint32_t out[kCols / 2];
            if (c0 < w_hi && c0 + kCols > w_lo) {
                const uint8_t* mine = smem + L::kPOff + (it % kPStages) * L::kPBytes + (warp * 32 + lane) * kPPitch;
                uint32_t x[kCols / 2 + 4];
#pragma unroll
                for (int i = 0; i < kPieces; ++i) {
                    const uint4 v = *reinterpret_cast<const uint4*>(mine + i * 16);
                    x[4 * i] = v.x; x[4 * i + 1] = v.y; x[4 * i + 2] = v.z; x[4 * i + 3] = v.w;
                }
                barrel<7>(x, sft, out);          // the warp's columns begin sft elements into the pieces
                if (!__all_sync(0xffffffffu, lo <= 0 && hi >= kCols)) {
                    // pairs of columns: a mask bit per column, two per word
#pragma unroll
                    for (int c = 0; c < kCols; c += 32) {
                        const int l = min(max(lo - c, 0), 32), h = min(max(hi - c, 0), 32);
                        const uint32_t valid = (h >= 32 ? ~0u : (1u << h) - 1) & ~(l >= 32 ? ~0u : (1u << l) - 1);
#pragma unroll
                        for (int i = 0; i < 16; ++i) {
                            uint32_t& w = out[c / 2 + i];
                            w = ((valid >> (2 * i)) & 1u ? w & 0xffffu : 0u) | ((valid >> (2 * i + 1)) & 1u ? w & 0xffff0000u : 0u);
                        }
                    }
                }
            } else {
#pragma unroll
                for (int i = 0; i < kCols / 2; ++i) out[i] = 0u;
            }
            __syncwarp();
            fetch(it + kPStages);
            if (it >= 2) {   // the MMAs that read this buffer two steps ago are complete
                ok = wait_all(&ctrl->freed[b], (uint32_t)((it >> 1) - 1) & 1u, &ctrl->gave_up, kErrFree);
                if (!ok) break;
                tc_fence_after_sync();
            }
            if constexpr (kHalves == 1) tmem_st32(lane_addr + p_col + b * 32, out);
            else tmem_st16(lane_addr + p_col + b * 32 + half * 16, out);
            tmem_st_wait();
            tc_fence_before_sync();
            __syncwarp();
            if (lane == 0) mbar_arrive(&ctrl->ready[b]);
        }
        asm volatile("cp.async.wait_all;" ::: "memory");
        const bool have_o = ok && khi > klo;
        if (have_o) {
            ok = wait_all(&ctrl->drain, 0, &ctrl->gave_up, kErrReady);
            tc_fence_after_sync();
        }
        // every warp is through with its pieces of P before their memory becomes the staging of the output
        asm volatile("bar.sync 1, %0;" ::"n"(kRowWarps * 32) : "memory");
        // epilogue: O for band rows, P[i,0] * V[start] for single-element rows, zero otherwise, staged in the
        // 128-byte-swizzled tile layout (either warp of the rows half of the columns), one TMA store per 64 columns and 32 rows
        const int t = rw * 32 + lane;
        const bool single = band.y == kSingle;
        const T* vrow = reinterpret_cast<const T*>(p.kv) + (head + band.x) * p.d;
        const float p0 = single ? to_f<T>(*reinterpret_cast<const T*>(p.sparse + e_row + band.x)) : 0.f;
        float2 odd = make_float2(0.f, 0.f);       // not finite: nor is the row
#pragma unroll
        for (int n = 0; n < D / 32 / kHalves; ++n) {
            const int ch = half * (D / 32 / kHalves) + n;
            uint32_t r[32];
            if (have_o && ok) {
                tmem_ld32(lane_addr + ch * 32, r);
                tmem_ld_wait();
#pragma unroll
                for (int j = 0; j < 32; j += 4) odd = note_nonfinite(odd, r + j);
            }
            uint4 outv[4];
            uint32_t* o32 = reinterpret_cast<uint32_t*>(outv);
            if (band.y > 0 && have_o && ok) {
#pragma unroll
                for (int j = 0; j < 32; j += 2) o32[j >> 1] = pack2<T>(__uint_as_float(r[j]), __uint_as_float(r[j + 1]));
            } else if (single) {
#pragma unroll
                for (int q4 = 0; q4 < 4; ++q4) {
                    const int c = ch * 32 + q4 * 8;
                    outv[q4] = c < p.d ? *reinterpret_cast<const uint4*>(vrow + c) : make_uint4(0, 0, 0, 0);
                }
#pragma unroll
                for (int j = 0; j < 16; ++j) {
                    const T* e = reinterpret_cast<const T*>(o32 + j);
                    o32[j] = pack2<T>(p0 * to_f<T>(e[0]), p0 * to_f<T>(e[1]));
                }
            } else {
#pragma unroll
                for (int q4 = 0; q4 < 4; ++q4) outv[q4] = make_uint4(0, 0, 0, 0);
            }
            uint8_t* srow = smem + (ch >> 1) * kSubBytes + t * 128;
#pragma unroll
            for (int q4 = 0; q4 < 4; ++q4)
                *reinterpret_cast<uint4*>(srow + ((((ch & 1) * 4 + q4) ^ (t & 7)) << 4)) = outv[q4];
        }
        const unsigned odd_rows = __ballot_sync(0xffffffffu, band.y > 0 && !isfinite(odd.x + odd.y));
        unsigned again = odd_rows;
        fence_proxy_async_smem();
        if constexpr (kHalves == 2) {          // the first warp of the rows stores them
            if (odd_rows != 0 && lane == 0) atomicOr(&ctrl->again[rw], odd_rows);
            asm volatile("bar.sync 1, %0;" ::"n"(kRowWarps * 32) : "memory");
            again = half == 0 ? ctrl->again[rw] : 0;
        } else {
            __syncwarp();
        }
        if (half == 0 && lane == 0 && u0 + rw * 32 < rows_v) {
            for (int sub = 0; sub < L::kSub; ++sub)
                tma_store_4d(map + 1, smem + sub * kSubBytes + rw * 32 * 128, sub * 64, res, u0 + rw * 32, (int)bh);
            tma_store_commit();
            if (again == 0) tma_store_wait_read();
            else tma_store_wait_all();
        }
        while (again) {        // rows that are not finite, perhaps by keys outside their bands
            __syncwarp();
            const int rr = __ffs(again) - 1;
            again &= again - 1;
            const int begin = __shfl_sync(0xffffffffu, band.x, rr), end = min(__shfl_sync(0xffffffffu, band.y, rr), rows_v);
            const int64_t row = head + (int64_t)(u0 + rw * 32 + rr) * p.stride + real_res;
            const float4 x = spmm_row<T>(reinterpret_cast<const T*>(p.sparse + p.lead + row * p.trailing_dim),
                                         reinterpret_cast<const T*>(p.kv) + head * p.d, (int64_t)begin * p.stride + real_res,
                                         p.stride, end - begin, p.d);
            store_row<T>(reinterpret_cast<T*>(p.o) + row * p.d, p.d, x);
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
}

// ---------------------------------------------------------------------------------------------
// host
// ---------------------------------------------------------------------------------------------
template <typename T, int D, int kRowWarps>
static int32_t launch_sddmm(const Maps<2>& maps, const Params& prm, int64_t bh, cudaStream_t st) {
    using L = SddmmLayout<D, kRowWarps>;
    auto kern = sddmm_band_kernel<T, D, kRowWarps>;
    if (!allow_dynamic_smem(reinterpret_cast<const void*>(kern), L::kSmemBytes)) return SPLAT_ERR_LAUNCH;
    return launch_kernel(kern, prm.cls.grid(prm.stride, bh), L::kThreads, L::kSmemBytes, st, maps, prm);
}
// Two warps to 32 rows halve what a step costs the warp that is in the way of the next, and leave twice as many to hide one
// another's latencies; a warp to 32 rows moves 128 bytes of a row at a time instead of 64.  So the latter where rows are long and
// the GPU is full.  us, one / two, SDDMM then SpMM: fp16 B4 H16 L4096 d64 window 256 55.3 / 51.5, 56.2 / 52.1; bf16 H16 L4096 d128
// +-100 22.5 / 20.1, 20.0 / 18.7; fp16 H8 L1024 d64 +-64 8.3 / 5.9, 5.9 / 5.6; bf16 H4 L2048 d64 window 512 12.9 / 8.7, 10.2 / 8.9; B2 H16 L8192
// d128 strided 64 55.5 / 46.6, 52.7 / 51.9; d64, H1 L8192 +-1000 (64 tiles) 39.1 / 25.0, 24.2 / 21.0; H4 (256) 58.0 / 58.7, 33.2 / 36.2; H24 L2048
// +-500 (384) 35.5 / 40.7, 30.8 / 32.0; d128, H1 L8192 +-1000 33.3 / 28.2, 25.1 / 22.8; H4 56.5 / 65.4, 35.8 / 39.7; H8 L4096 +-600 (256) 32.4 / 33.6,
// 25.0 / 27.1; H24 L2048 +-500 48.6 / 48.7, 36.8 / 38.2.
// SDDMM at d <= 64 up to two waves: H3 L8192 +-1000 (192) 50.1 / 42.3, H4 +-700 (256) 37.0 / 30.1.
static bool two_warps(const Params& prm, int64_t bh, int64_t tiles) { return prm.trailing_dim <= 512 || prm.cls.tiles(prm.stride, bh) <= tiles; }
template <typename T, int D>
static int32_t launch_sddmm(const Maps<2>& maps, const Params& prm, int64_t bh, cudaStream_t st) {
    return two_warps(prm, bh, D == 64 ? 296 : 148) ? launch_sddmm<T, D, 8>(maps, prm, bh, st) : launch_sddmm<T, D, 4>(maps, prm, bh, st);
}
template <typename T, int D, int kPerSm, int kRowWarps>
static int32_t launch_spmm(const Maps<2>& maps, const Params& prm, int64_t bh, cudaStream_t st) {
    using L = SpmmLayout<D, kPerSm, kRowWarps>;
    auto kern = spmm_band_kernel<T, D, kPerSm, kRowWarps>;
    if (!allow_dynamic_smem(reinterpret_cast<const void*>(kern), L::kSmemBytes)) return SPLAT_ERR_LAUNCH;
    return launch_kernel(kern, prm.cls.grid(prm.stride, bh), L::kThreads, L::kSmemBytes, st, maps, prm);
}
template <typename T>
static int32_t launch_spmm(const Maps<2>& maps, const Params& prm, int64_t bh, cudaStream_t st) {
    if (two_warps(prm, bh, 148)) {
        if (prm.d > 64) return launch_spmm<T, 128, 2, 8>(maps, prm, bh, st);
        return prm.cls.tiles(prm.stride, bh) > 2 * 148 ? launch_spmm<T, 64, 3, 8>(maps, prm, bh, st) : launch_spmm<T, 64, 2, 8>(maps, prm, bh, st);
    }
    if (prm.d > 64) return launch_spmm<T, 128, 2, 4>(maps, prm, bh, st);
    return prm.cls.tiles(prm.stride, bh) > 2 * 148 ? launch_spmm<T, 64, 3, 4>(maps, prm, bh, st) : launch_spmm<T, 64, 2, 4>(maps, prm, bh, st);
}

// Checks shared by both operators; fills stride.  plan as written by splat_acsr_classify:
// {max_nnz, stride_min, stride_max, misaligned, n_single, max_col+1, n_empty, n_multi}
static int32_t band_applies(const int32_t* plan, int64_t bh, int64_t n_rows, int64_t n_cols, int64_t d,
                            int64_t trailing_dim, int32_t dtype, int64_t* stride_out) {
    if (bh < 0 || n_rows < 0 || trailing_dim < 0) return SPLAT_ERR_BAD_ARG;
    if (bh == 0 || n_rows == 0 || trailing_dim == 0) return SPLAT_ERR_UNSUPPORTED_SHAPE;
    if (dtype != SPLAT_F16 && dtype != SPLAT_BF16) return SPLAT_ERR_UNSUPPORTED_SHAPE;
    if (d < 8 || d > 128 || d % 8 != 0) return SPLAT_ERR_UNSUPPORTED_SHAPE;
    if (n_rows != n_cols) return SPLAT_ERR_UNSUPPORTED_SHAPE;
    const int64_t stride = plan[7] > 0 ? plan[1] : 1;
    if (plan[7] > 0 && plan[1] != plan[2]) return SPLAT_ERR_UNSUPPORTED_SHAPE;
    if (plan[3] != 0 || stride < 1 || stride > 65535) return SPLAT_ERR_UNSUPPORTED_SHAPE;
    if (plan[5] > n_cols || plan[0] > trailing_dim || bh > 65535 || n_rows > INT32_MAX ||
        trailing_dim > INT32_MAX)
        return SPLAT_ERR_UNSUPPORTED_SHAPE;
    // (the kernels address the sparse rows of a warp with signed 32-bit byte offsets)
    if ((32 * stride * trailing_dim + n_rows) * 2 >= INT32_MAX) return SPLAT_ERR_UNSUPPORTED_SHAPE;
    *stride_out = stride;
    return SPLAT_OK;
}

static Params params(const void* sparse, const float* lin, const float* tr, const float* nnzs, int64_t n_rows, int64_t d,
                     int64_t trailing_dim, int64_t stride, const int32_t* band_table, int32_t* status_word) {
    Params p{};
    p.lin = lin; p.tr = tr; p.nnzs = nnzs;
    const uintptr_t a = reinterpret_cast<uintptr_t>(sparse);
    p.sparse = reinterpret_cast<uint16_t*>(a & ~(uintptr_t)15);
    p.lead = (int)(a & 15) / 2;
    p.status = status_word; p.mirror = status_mirror(status_word);
    p.n_rows = n_rows; p.stride = (int)stride; p.d = (int)d; p.trailing_dim = (int)trailing_dim;
    p.cls = Classes(n_rows, stride, kTile);
    p.rows = reinterpret_cast<const int2*>(band_table);
    p.tiles = band_table != nullptr ? p.rows + n_rows : nullptr;
    return p;
}

}  // namespace ops
}  // namespace band
}  // namespace splat

using namespace splat;
using namespace splat::band;

extern "C" int32_t splat_sddmm_band_table(const void* q, const void* k, int64_t k_stride_bh, int64_t k_stride_col,
                                          int64_t k_stride_k, void* s_out, const float* sTod_lin,
                                          const float* sTod_tr, const float* nnzs, int64_t bh, int64_t n_rows,
                                          int64_t n_cols, int64_t d, int64_t trailing_dim, int32_t dtype,
                                          const int32_t* plan_i32, const int32_t* band_table, int32_t* status_word,
                                          void* stream) {
    if (!plan_i32) return SPLAT_ERR_BAD_ARG;
    int64_t stride = 1;
    int32_t rc = ops::band_applies(plan_i32, bh, n_rows, n_cols, d, trailing_dim, dtype, &stride);
    if (rc != SPLAT_OK) return rc;
    if (!q || !k || !s_out || !sTod_lin || !sTod_tr || !nnzs || !status_word) return SPLAT_ERR_BAD_ARG;
    const bool k_major = k_stride_k == 1 && k_stride_col == d && k_stride_bh == n_cols * d;
    const bool kt_major = k_stride_col == 1 && k_stride_k == n_cols && k_stride_bh == n_cols * d;
    if (!k_major && !(kt_major && stride == 1 && n_cols % 8 == 0)) return SPLAT_ERR_UNSUPPORTED_SHAPE;
    if (!aligned16(q) || !aligned16(k)) return SPLAT_ERR_MISALIGNED;
    ops::Params p = ops::params(s_out, sTod_lin, sTod_tr, nnzs, n_rows, d, trailing_dim, stride, band_table, status_word);
    p.q = q; p.kv = k; p.kt_major = k_major ? 0 : 1;
    cudaStream_t st = (cudaStream_t)stream;
    Maps<2> maps;
    for (int part = 0; part < 2; ++part) {
        CUtensorMap* m = maps.part[part];
        if (p.cls.has(part) &&
            (!p.cls.view(m, q, dtype, bh, n_rows, d, stride, part, ops::kTile) ||
             !(k_major ? p.cls.view(m + 1, k, dtype, bh, n_rows, d, stride, part, ops::kStep)
                       : make_map_kt(m + 1, k, dtype, bh, n_cols, d, d > 64 ? 128 : 64))))
            return SPLAT_ERR_DRIVER;
    }
    if (dtype == SPLAT_BF16)
        return d > 64 ? ops::launch_sddmm<__nv_bfloat16, 128>(maps, p, bh, st) : ops::launch_sddmm<__nv_bfloat16, 64>(maps, p, bh, st);
    return d > 64 ? ops::launch_sddmm<__half, 128>(maps, p, bh, st) : ops::launch_sddmm<__half, 64>(maps, p, bh, st);
}

extern "C" int32_t splat_spmm_band_table(const void* p_in, const void* v, void* o, const float* sTod_lin,
                                         const float* sTod_tr, const float* nnzs, int64_t bh, int64_t n_rows,
                                         int64_t n_cols, int64_t d, int64_t trailing_dim, int32_t dtype,
                                         const int32_t* plan_i32, const int32_t* band_table, int32_t* status_word,
                                         void* stream) {
    if (!plan_i32) return SPLAT_ERR_BAD_ARG;
    int64_t stride = 1;
    int32_t rc = ops::band_applies(plan_i32, bh, n_rows, n_cols, d, trailing_dim, dtype, &stride);
    if (rc != SPLAT_OK) return rc;
    if (!p_in || !v || !o || !sTod_lin || !sTod_tr || !nnzs || !status_word) return SPLAT_ERR_BAD_ARG;
    if (!aligned16(v) || !aligned16(o)) return SPLAT_ERR_MISALIGNED;
    ops::Params p = ops::params(p_in, sTod_lin, sTod_tr, nnzs, n_rows, d, trailing_dim, stride, band_table, status_word);
    p.kv = v; p.o = o;
    cudaStream_t st = (cudaStream_t)stream;
    Maps<2> maps;
    for (int part = 0; part < 2; ++part) {
        CUtensorMap* m = maps.part[part];
        if (p.cls.has(part) && (!p.cls.view(m, v, dtype, bh, n_rows, d, stride, part, ops::kStep) ||
                                !p.cls.view(m + 1, o, dtype, bh, n_rows, d, stride, part, 32)))
            return SPLAT_ERR_DRIVER;
    }
    return dtype == SPLAT_BF16 ? ops::launch_spmm<__nv_bfloat16>(maps, p, bh, st) : ops::launch_spmm<__half>(maps, p, bh, st);
}

extern "C" int32_t splat_sddmm_band(const void* q, const void* k, int64_t k_stride_bh, int64_t k_stride_col,
                                    int64_t k_stride_k, void* s_out, const float* sTod_lin,
                                    const float* sTod_tr, const float* nnzs, int64_t bh, int64_t n_rows,
                                    int64_t n_cols, int64_t d, int64_t trailing_dim, int32_t dtype,
                                    const int32_t* plan_i32, int32_t* status_word, void* stream) {
    return splat_sddmm_band_table(q, k, k_stride_bh, k_stride_col, k_stride_k, s_out, sTod_lin, sTod_tr, nnzs, bh, n_rows,
                                  n_cols, d, trailing_dim, dtype, plan_i32, nullptr, status_word, stream);
}

extern "C" int32_t splat_spmm_band(const void* p, const void* v, void* o, const float* sTod_lin,
                                   const float* sTod_tr, const float* nnzs, int64_t bh, int64_t n_rows,
                                   int64_t n_cols, int64_t d, int64_t trailing_dim, int32_t dtype,
                                   const int32_t* plan_i32, int32_t* status_word, void* stream) {
    return splat_spmm_band_table(p, v, o, sTod_lin, sTod_tr, nnzs, bh, n_rows, n_cols, d, trailing_dim, dtype, plan_i32,
                                 nullptr, status_word, stream);
}
