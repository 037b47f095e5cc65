// Fused band attention for d = 128: a persistent CTA per SM with two 128-row Q tiles ("pipes") side by
// side.  Problem, regrouping by residue class and operand layouts: see attention_band.cu; a step's arithmetic: see
// attention_wide.cu, which has the other problems (other d, classes of unequal length, no band table).
//
// What bounds a tile is its own chain S -> softmax -> P -> PV -> S: with the exponentials left out the kernel gains 10 %,
// with the MMAs left out 18 %.  So there are two independent tiles per SM here as in attention_wide.cu, but
//   * the next tile's Q, K and V are on their way, and its first S is computed, while a tile ends.  A CTA per tile spent
//     9.3 of 28.7 thousand cycles (five steps) on launch, prologue, first copies, epilogue and exit;
//   * two tiles of one class share every K and V block of the union of their key ranges: 1.84 GB read from L2 instead of
//     2.94 (B1 H16 L32768 window 1024), which had come to 8 TB/s;
//   * S(j + 1) does not wait for PV(j): P has columns of its own, and the 128 columns that are left hold one S, that of either
//     tile in turn.  It is read into registers within some 200 cycles of its completion.
// Tensor memory: P of pipe 0 (64 columns), S (128), P of pipe 1 (64), O of pipe 0 and of pipe 1 (128 each).
//
// Work: an item is two neighbouring tiles (of the list head by head, class by class), or one in a short last wave.  A CTA begins with the item of its
// index and then takes over CTAs that have not started (clusterlaunchcontrol), two items ahead.  The K / V blocks of an
// item travel as a stream of entries through a ring of two slots each; every role derives the same numbering of the
// entries from the items.
// Warps: 0-3 softmax and epilogue of pipe 0 (thread = row = tensor-memory lane), 4-7 of pipe 1; 8 TMA; 9 issues S = Q K^T
// and thereby sets the order of the steps; 10 issues O += P V in the same order; 11 fetches items.
//
// Instruction fetch matters: with inlined polling loops that looked at the status word, unrolled epilogue and generic
// addresses the same kernel had 85 KB of code and stalled for thousands of cycles at a time (B1 H37 L16384 window 128 / 512
// 223 / 314 us against 116 / 200 us with 49 KB).  Hence waits of a few instructions, rolled loops and out-of-range checks.
// Measured, bf16, us, a CTA per tile -> this: B1 H37 L16384 window 128 / 256 / 512 / 1024 147 / 176 / 236 / 363 -> 116 /
// 144 / 200 / 320; B2 H32 L8192 strided 64 109.9 -> 92.1 (HBM: 82); B1 H32 L16384 512 taps by 2 242 -> 206; B8 H64 L32768
// window 1024 11.79 -> 10.13 ms; B3 H12 L3000 +-200 with log-sum-exp 58.1 -> 48.8.
// Variants that lost: one warp that issues all MMAs 2.3-2.4 thousand cycles per step and tile (here 1.75); two threads per
// row (16 softmax warps) 2.0; PV issued for whichever pipe has its P first 2.4; K ring of three slots with 32-byte
// stores straight from registers: strided 87, dilated 181.
#include <limits.h>
#include <type_traits>

#include "band_classes.cuh"
#include "common.cuh"
#include "softmax_math.cuh"
#include "tc_ptx.cuh"

namespace splat {
namespace band {

using namespace tc;

namespace duo {

using sm::ex2;
using sm::mul2;
using sm::pack2;

constexpr int kD = 128;                  // columns of a tile
constexpr int kTile = 128;               // rows of a Q tile, keys of a block
constexpr int kChunk = 32;               // columns of a tensor-memory load
constexpr int kChunks = kTile / kChunk;
constexpr int kSub = kD / 64;
constexpr int kSubBytes = kTile * 128;   // one 64-element (128-byte) column chunk of a tile
constexpr int kTileBytes = kSub * kSubBytes;
constexpr int kTmaWarp = 8;
constexpr int kQkWarp = 9;
// (warp 10: PV)
constexpr int kPlanWarp = 11;
constexpr int kThreads = 384;
constexpr int kSoftmaxRegs = 208, kOtherRegs = 88;   // 2 x 208 + 88 = 3 x 168, the registers of the launch
constexpr int kTmemCols = 512;
constexpr int kTmemP = 0, kTmemPPitch = 192, kTmemS = 64, kTmemO = 256;
constexpr int kSlots = 2;                // K blocks, and V blocks, in shared memory
constexpr int kItems = 2;                // items known ahead
constexpr int kItemReaders = 8 + 2 + 1;  // softmax warps, the QK warp once per pipe, the TMA thread
constexpr int kOrders = 8;               // S issued whose PV has not been: never more than three per pipe, and the end
constexpr float kRescaleThreshold = 8.0f;   // log2 domain: P stays below 2^8 between rescales
constexpr uint32_t kIdlePolls = 1u << 22;   // of the QK warp without an S to issue: less than a second

// shared memory
constexpr int kKOff = 2 * kTileBytes;            // behind the Q tiles
constexpr int kVOff = kKOff + kSlots * kTileBytes;
constexpr int kStageOff = kVOff + kSlots * kTileBytes;    // 2 KB per softmax warp
constexpr int kSmemBytes = kStageOff + 8 * 2048 + 1024;   // + alignment slack

// status-word codes (which wait gave up)
enum : int { kErrOrder = 59, kErrV = 60, kErrQFree = 61, kErrKFree = 62, kErrVFree = 63, kErrItem = 64, kErrItemFree = 65, kErrClc = 66,
             kErrS = 67, kErrP = 68, kErrO = 69, kErrSFree = 70, kErrPv = 74, kErrIdle = 75 };

struct Maps3 { CUtensorMap m[3]; };       // Q, K, V

struct Params {
    const void* q;     // raw operands: rows with one non-zero are handled through them
    const void* k;
    const void* v;
    void* o;
    const int2* bands; // band table (see acsr_meta.cu): of the rows in class order, tiles' key ranges
    const int2* tiles;
    float* lse;        // (BH, L) or null
    int32_t* status;
    int32_t* mirror;   // host copy of the status word, or null
    int64_t n_rows;    // L
    int stride;        // classes of a head
    int rows;          // ... rows of each
    uint32_t pitch;    // ... tiles of each
    uint32_t total;    // tiles of all heads and classes
    uint32_t pairs;    // items of two tiles; the rest have one
    int kt_major;
    float scale_log2;
};

// what the QK warp tells the PV warp of a step
enum : int { kHalf0 = 1, kHalf1 = 2, kFirst = 4, kLast = 8, kBoth = 16, kPipe1 = 32, kStop = 64 };

// A tile of an item; lo, hi: key range of its rows' bands in 64-key units.  u0 < 0: none.
struct Tile {
    int u0, res, bh, lo, hi;
    __device__ __forceinline__ int first() const { return lo >> 1; }                       // 128-key blocks
    __device__ __forceinline__ int blocks() const { return ((hi + 1) >> 1) - (lo >> 1); }
};
struct Item {
    Tile t[2];
    int stop;
};

// The K / V blocks of an item in the order in which they travel.  Two tiles of one class whose ranges meet share every
// block of the union; otherwise their blocks alternate.  (Far apart ranges share too, although one tile then waits: with
// sharing only up to two blocks apart blocks of 1000 keys, L8000, 756 tiles, took 157 us instead of 134.)
struct Stream {
    bool shared;
    int first, count;
    __device__ __forceinline__ Stream(const Tile& a, const Tile& b) {
        const int na = a.blocks(), nb = b.blocks(), ea = a.first() + na, eb = b.first() + nb;
        shared = na > 0 && nb > 0 && a.bh == b.bh && a.res == b.res && a.first() <= eb && b.first() <= ea;
        first = min(a.first(), b.first());
        count = shared ? max(ea, eb) - first : na + nb;
    }
};

struct Control {
    uint64_t q_full[2], q_free[2], o_full[2], s_full[2], p_full[2][2], pv_done[2];     // by pipe
    uint64_t s_free;                      // the scores have been read
    uint64_t k_full[kSlots], k_free[kSlots], v_full[kSlots], v_free[kSlots];
    uint64_t order_full[kOrders];
    uint64_t item_full[kItems], item_free[kItems];
    uint64_t clc_full, drain[2];
    alignas(16) uint4 clc;                // answer of the work distributor
    Item item[kItems];
    int2 order[kOrders];                  // QK -> PV warp: stream entry, flags
    uint32_t tmem_base;
    int32_t abort_at_entry;
    int32_t gave_up;                      // code of a wait that ran out
};
static_assert(kSmemBytes + sizeof(Control) <= 232448, "shared memory of a CTA");

__device__ __forceinline__ bool test_all(uint64_t* bar, uint32_t parity) {
    return __all_sync(0xffffffffu, mbar_test_wait(bar, parity)) != 0;
}
// O of the warp's rows times corr.
__device__ __forceinline__ void rescale_o(uint32_t o_addr, float corr) {
    uint32_t v[16];
#pragma unroll 1
    for (int i = 0; i < kD / 16; ++i) {
        tmem_ld16(o_addr + i * 16, v);
        tmem_ld_wait();
#pragma unroll
        for (int j = 0; j < 16; ++j) v[j] = __float_as_uint(__uint_as_float(v[j]) * corr);
        tmem_st16(o_addr + i * 16, v);
    }
    tmem_st_wait();
}

// Row kinds in the band table: end of the band for a row with one non-zero (begin = its column), without one and past the
// end of the class.
constexpr int kSingle = -1, kEmpty = INT_MIN / 2;

// Log-sum-exp of a row with one non-zero: its score, summed in the order of the other kernels.  Every head has such a row as a
// rule, every class of a strided pattern.  With the loop rolled and a load of either operand per round trip they were
// most of the call (us, a CTA per tile / rolled / this: H320 L512 window 128 K^T as rows 46.5 / 64.0 / 40.7, contiguous 49.0 / 189 /
// 44.0; H216 L1280 567 taps by 4 84.9 / 106.9 / 70.5).
template <typename T>
__device__ __forceinline__ float single_lse(const Params& p, int64_t head, int64_t row, int start) {
    const T* q = reinterpret_cast<const T*>(p.q) + (head + row) * kD;
    const T* k = reinterpret_cast<const T*>(p.k) + head * kD + (p.kt_major ? start : (int64_t)start * kD);
    float acc = 0.f;
    auto add = [&](const uint4& a, const T* kc) {
        const T* qc = reinterpret_cast<const T*>(&a);
#pragma unroll
        for (int i = 0; i < 8; ++i) acc = fmaf(DT<T>::to_f(qc[i]), DT<T>::to_f(kc[i]), acc);
    };
    if (p.kt_major) {
#pragma unroll 4
        for (int c = 0; c < kD; c += 8) {
            T kc[8];
#pragma unroll
            for (int i = 0; i < 8; ++i) kc[i] = k[(c + i) * p.n_rows];
            add(*reinterpret_cast<const uint4*>(q + c), kc);
        }
    } else {
#pragma unroll 4
        for (int c = 0; c < kD; c += 8) {
            const uint4 b = *reinterpret_cast<const uint4*>(k + c);
            add(*reinterpret_cast<const uint4*>(q + c), reinterpret_cast<const T*>(&b));
        }
    }
    return acc * p.scale_log2 * kLn2;
}

// Tile n of the list.
__device__ __forceinline__ Tile tile_of(const Params& p, uint32_t n) {
    Tile t = {-1, 0, 0, 0, 0};
    if (n >= p.total) return t;
    const uint32_t rest = n / p.pitch, tile = n - rest * p.pitch;
    t.bh = (int)(rest / (uint32_t)p.stride);
    t.res = (int)(rest - (uint32_t)t.bh * (uint32_t)p.stride);
    t.u0 = (int)tile * kTile;
    const int2 range = __ldg(p.tiles + t.res * (int64_t)p.pitch + tile);
    const int hi = min(range.y, p.rows);
    if (hi > 0) { t.lo = range.x / 64; t.hi = (hi + 63) / 64; }
    return t;
}

// Asks the work distributor for a CTA of this grid that has not started; the answer (16 bytes) counts on the barrier.
__device__ __forceinline__ void clc_request(uint4* answer, uint64_t* bar) {
    asm volatile("clusterlaunchcontrol.try_cancel.async.shared::cta.mbarrier::complete_tx::bytes.b128 [%0], [%1];" ::"r"(
                     smem_u32(answer)), "r"(smem_u32(bar)) : "memory");
}
// Its blockIdx.x, or -1: all have started.
__device__ __forceinline__ int64_t clc_answer(const uint4* answer) {
    uint32_t got, x = 0;
    asm volatile(
        "{\n"
        ".reg .pred p;\n"
        ".reg .b128 h;\n"
        "ld.shared.b128 h, [%2];\n"
        "clusterlaunchcontrol.query_cancel.is_canceled.pred.b128 p, h;\n"
        "selp.u32 %0, 1, 0, p;\n"
        "mov.u32 %1, 0;\n"
        "@p clusterlaunchcontrol.query_cancel.get_first_ctaid::x.b32.b128 %1, h;\n"
        "}\n"
        : "=r"(got), "=r"(x) : "r"(smem_u32(answer)) : "memory");
    return got ? (int64_t)x : -1;
}

template <typename T, bool kLse>
__global__ void __launch_bounds__(kThreads, 1)
attention_duo_kernel(const __grid_constant__ Maps3 maps, const Params p) {
    constexpr uint32_t kFmt = std::is_same<T, __nv_bfloat16>::value ? 1u : 0u;
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = smem_raw + (((smem_u32(smem_raw) + 1023) & ~1023u) - smem_u32(smem_raw));
    __shared__ Control ctrl_mem;             // (static: constant addresses)
    Control* const ctrl = &ctrl_mem;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;

    if (warp == kQkWarp) {
        depend_wait();
        tmem_alloc(&ctrl->tmem_base, kTmemCols);
        tmem_relinquish();
    } else if (warp == kTmaWarp) {
        if (lane == 0) {
#pragma unroll 1
            for (int i = 0; i < 3; ++i) tma_prefetch_desc(&maps.m[i]);
#pragma unroll 1
            for (int i = 0; i < 2; ++i) {
                mbar_init(&ctrl->q_full[i], 1);
                mbar_init(&ctrl->q_free[i], 1);
                mbar_init(&ctrl->o_full[i], 1);
                mbar_init(&ctrl->s_full[i], 1);
                mbar_init(&ctrl->pv_done[i], 1);
                mbar_init(&ctrl->p_full[i][0], 4);       // one arrival per softmax warp
                mbar_init(&ctrl->p_full[i][1], 4);
                mbar_init(&ctrl->k_full[i], 1);
                mbar_init(&ctrl->k_free[i], 2);          // both pipes
                mbar_init(&ctrl->v_full[i], 1);
                mbar_init(&ctrl->v_free[i], 2);
                mbar_init(&ctrl->item_full[i], 1);
                mbar_init(&ctrl->item_free[i], kItemReaders);
                mbar_init(&ctrl->drain[i], 1);
            }
#pragma unroll 1
            for (int i = 0; i < kOrders; ++i) mbar_init(&ctrl->order_full[i], 1);
            mbar_init(&ctrl->s_free, 4);
            mbar_init(&ctrl->clc_full, 1);
            mbar_fence_init();
            ctrl->gave_up = 0;
            depend_wait();
            ctrl->abort_at_entry = entry_status(p.status, p.mirror);
        }
    } else {
        depend_wait();
    }
    tc_fence_before_sync();
    __syncthreads();
    tc_fence_after_sync();
    depend_release();
    const uint32_t tmem_base = ctrl->tmem_base;
    if (ctrl->abort_at_entry != 0) {   // an earlier launch gave up
        if (warp == kQkWarp) tmem_dealloc(tmem_base, kTmemCols);
        return;
    }

    if (warp >= 8) {
        asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(kOtherRegs));
        if (warp == kPlanWarp) {
            // -------------------------------------------------------------- items
            int64_t next = blockIdx.x;
            for (int n = 0;; ++n) {
                const int slot = n % kItems;
                if (n >= kItems && !wait_all(&ctrl->item_free[slot], ((uint32_t)(n / kItems) & 1u) ^ 1u, &ctrl->gave_up, kErrItemFree)) break;
                // (once a CTA has given up no other is taken over, as none that starts then does anything)
                if (n > 0 && __any_sync(0xffffffffu, *(const volatile int32_t*)p.status != 0)) next = -1;
                if (next >= 0) {
#pragma unroll 1
                    for (int x = 0; x < 2; ++x) {
                        const uint32_t i = (uint32_t)next;
                        const Tile t = tile_of(p, i < p.pairs ? 2 * i + x : x == 0 ? i + p.pairs : p.total);
                        if (lane == 0) ctrl->item[slot].t[x] = t;
                    }
                }
                if (lane == 0) {
                    ctrl->item[slot].stop = next < 0;
                    mbar_arrive(&ctrl->item_full[slot]);
                }
                if (next < 0) break;
                if (lane == 0) {
                    mbar_arrive_expect_tx(&ctrl->clc_full, 16);
                    clc_request(&ctrl->clc, &ctrl->clc_full);
                }
                __syncwarp();
                if (!wait_all(&ctrl->clc_full, (uint32_t)n & 1u, &ctrl->gave_up, kErrClc)) {
                    wait_quiet(&ctrl->clc_full, (uint32_t)n & 1u);     // leave only after the answer has been written
                    break;
                }
                next = clc_answer(&ctrl->clc);
                fence_proxy_async_smem();      // read before the next answer is written
                __syncwarp();
            }
        } else if (warp == kTmaWarp) {
            // -------------------------------------------------------------- TMA producer
            if (lane == 0) {
                int entry = 0, k_asked = 0, q0_asked = 0, q1_asked = 0;   // stream entries, K blocks and Q tiles requested
                bool ok = true;
                auto load = [&](uint64_t* bar, uint8_t* dst, const CUtensorMap* map, int res, int row, int bh) {
                    mbar_arrive_expect_tx(bar, kTileBytes);
#pragma unroll 1
                    for (int sub = 0; sub < kSub; ++sub) tma_load_4d(dst + sub * kSubBytes, map, bar, sub * 64, res, row, bh);
                };
                auto load_q = [&](const Tile& t, int x, int& asked) {
                    if (asked > 0) ok = wait_bar(&ctrl->q_free[x], ((uint32_t)asked & 1u) ^ 1u, &ctrl->gave_up, kErrQFree);
                    if (!ok) return;
                    load(&ctrl->q_full[x], smem + x * kTileBytes, &maps.m[0], t.res, t.u0, t.bh);
                    ++asked;
                };
                for (int n = 0; ok; ++n) {
                    const int slot = n % kItems;
                    ok = wait_bar(&ctrl->item_full[slot], (uint32_t)(n / kItems) & 1u, &ctrl->gave_up, kErrItem);
                    if (!ok || ctrl->item[slot].stop) break;
                    const Tile a = ctrl->item[slot].t[0], b = ctrl->item[slot].t[1];
                    mbar_arrive(&ctrl->item_free[slot]);
                    const Stream s(a, b);
                    const int na = a.blocks(), nb = b.blocks(), twice = 2 * min(na, nb);
#pragma unroll 1
                    for (int i = 0; i < s.count; ++i) {
                        // a Q tile travels in front of the first block that it meets
                        int x = 0, block = s.first + i;
                        bool q0 = block == a.first(), q1 = block == b.first();
                        if (!s.shared) {
                            const int k = i < twice ? i >> 1 : i - twice / 2;
                            x = i < twice ? (i & 1) : (na > nb ? 0 : 1);
                            block = (x ? b.first() : a.first()) + k;
                            q0 = x == 0 && k == 0;
                            q1 = x == 1 && k == 0;
                        }
                        if (q0) load_q(a, 0, q0_asked);
                        if (q1 && ok) load_q(b, 1, q1_asked);
                        if (!ok) break;
                        const int res = x ? b.res : a.res, bh = x ? b.bh : a.bh, st = entry % kSlots;
                        const uint32_t parity = ((uint32_t)(entry / kSlots) & 1u) ^ 1u;
                        uint8_t* dst = smem + kKOff + st * kTileBytes;
                        if (entry >= kSlots) ok = wait_bar(&ctrl->k_free[st], parity, &ctrl->gave_up, kErrKFree);
                        if (!ok) break;
                        if (p.kt_major) {
                            mbar_arrive_expect_tx(&ctrl->k_full[st], kTileBytes);
#pragma unroll 1
                            for (int ch = 0; ch < kTile / 64; ++ch)       // 64-key chunks of [d][64 keys]
                                tma_load_4d(dst + ch * (kD * 128), &maps.m[1], &ctrl->k_full[st], block * kTile + ch * 64, 0, bh, 0);
                        } else {
                            load(&ctrl->k_full[st], dst, &maps.m[1], res, block * kTile, bh);
                        }
                        ++k_asked;
                        if (entry >= kSlots) ok = wait_bar(&ctrl->v_free[st], parity, &ctrl->gave_up, kErrVFree);
                        if (!ok) break;
                        load(&ctrl->v_full[st], smem + kVOff + st * kTileBytes, &maps.m[2], res, block * kTile, bh);
                        ++entry;
                    }
                }
                if (!ok) {                     // leave only after the copies already issued have landed
                    if (q0_asked > 0) wait_quiet(&ctrl->q_full[0], (uint32_t)(q0_asked - 1) & 1u);
                    if (q1_asked > 0) wait_quiet(&ctrl->q_full[1], (uint32_t)(q1_asked - 1) & 1u);
#pragma unroll 1
                    for (int i = max(0, k_asked - kSlots); i < k_asked; ++i) {
                        wait_quiet(&ctrl->k_full[i % kSlots], (uint32_t)(i / kSlots) & 1u);
                        if (i < entry) wait_quiet(&ctrl->v_full[i % kSlots], (uint32_t)(i / kSlots) & 1u);
                    }
                }
            }
        } else if (warp == kQkWarp) {
            // -------------------------------------------------------------- S = Q K^T
            // (whole warp on warp-uniform values, one elected lane issues)
            const bool lead = elect_one();
            const uint32_t idesc_full = instr_desc_f16(kFmt, kTile, kTile, p.kt_major ? 1u : 0u);
            const uint32_t idesc_half = instr_desc_f16(kFmt, kTile, 64, p.kt_major ? 1u : 0u);
            const uint64_t q_desc = smem_desc_sw128(smem_u32(smem), 16, 1024);
            const uint64_t k_desc = smem_desc_sw128(smem_u32(smem + kKOff), p.kt_major ? kD * 128 : 16, 1024);
            const uint32_t k_step = (p.kt_major ? 2048 : 32) >> 4, k_sub = (p.kt_major ? 4 * 2048 : kSubBytes) >> 4;
            const uint32_t k_skip = (p.kt_major ? kD * 128 : 64 * 128) >> 4;
            struct Pipe {
                int items = 0;                 // items opened
                bool done = false;             // none will follow
                int n = 0, k = 0;              // blocks of the tile, those whose scores have been issued
                int lo = 0, hi = 0;            // its range in 64-key units
                int base = 0, count = 0;       // stream entries before the item, of the item
                int next = 0;                  // no entry before this one is still to be issued
                bool shared = false;
                int first_entry = 0;           // shared: entry of the tile's first block
                int other_n = 0, other_first = 0;
                int tiles = 0, scores = 0;     // tiles whose last S has been issued, S issued
            };
            Pipe me, other;
            int x = 0, last_x = -1;            // me is pipe x; pipe of the last S
            int issued = 0;
            uint32_t polls = 0;
            // The pipes take turns, so that their softmax steps run half a period apart; a pipe gets two S in a row only
            // if the other is not ready by the time that half of the first has been exponentiated.  Nothing is
            // waited for here that the other pipe may hold up.
            for (;;) {
                // the next item with blocks for this pipe
                while (!me.done && me.k == me.n) {
                    const int slot = me.items % kItems;
                    if (!test_all(&ctrl->item_full[slot], (uint32_t)(me.items / kItems) & 1u)) break;
                    const bool stop = ctrl->item[slot].stop != 0;
                    const Tile t = ctrl->item[slot].t[x], o = ctrl->item[slot].t[x ^ 1];
                    __syncwarp();
                    if (lead) mbar_arrive(&ctrl->item_free[slot]);
                    if (stop) { me.done = true; me.next = INT_MAX; break; }
                    const Stream s(t, o);
                    me.base += me.count;
                    me.count = s.count;
                    me.shared = s.shared;
                    me.n = t.blocks(); me.k = 0;
                    me.lo = t.lo; me.hi = t.hi;
                    me.first_entry = t.first() - s.first;
                    me.other_n = o.blocks(); me.other_first = o.first();
                    me.next = me.base + (me.n == 0 ? me.count : me.shared ? me.first_entry : me.other_n == 0 ? 0 : x);
                    ++me.items;
                }
                bool go = me.k < me.n;
                int e = 0, st = 0;
                if (go) {
                    const int k = me.k;
                    e = me.base + (me.shared ? me.first_entry + k : (k < me.other_n ? 2 * k + x : me.other_n + k));
                    st = e % kSlots;
                    // (entry e - kSlots has been issued in both pipes: its phase of the slot's barrier is not mistaken for e's)
                    go = e - kSlots < other.next && (k > 0 || test_all(&ctrl->q_full[x], (uint32_t)me.tiles & 1u)) &&
                         test_all(&ctrl->k_full[st], (uint32_t)(e / kSlots) & 1u);
                    // (s_free first: once the last S, this pipe's, has been read, p_full can be no more than one phase behind, and its
                    // parity tells which)
                    if (go && last_x == x)
                        go = test_all(&ctrl->s_free, (uint32_t)(issued - 1) & 1u) && test_all(&ctrl->p_full[x][0], (uint32_t)(me.scores - 1) & 1u);
                }
                if (go) {
                    const int block = (me.lo >> 1) + me.k;
                    const bool h0 = 2 * block >= me.lo, h1 = 2 * block + 1 < me.hi;     // half blocks outside the range are left out
                    const bool last = me.k + 1 == me.n;
                    const bool both = me.shared && block >= me.other_first && block < me.other_first + me.other_n;
                    const uint32_t idesc = h0 && h1 ? idesc_full : idesc_half;
                    uint64_t da = q_desc + (uint32_t)(x * kTileBytes >> 4);
                    uint64_t db = k_desc + (uint32_t)(st * kTileBytes >> 4) + (h0 ? 0u : k_skip);
                    const uint32_t to = tmem_base + kTmemS + (h0 ? 0 : 64);
                    const int2 order = make_int2(e, (h0 ? kHalf0 : 0) | (h1 ? kHalf1 : 0) | (me.k == 0 ? kFirst : 0) |
                                                    (last ? kLast : 0) | (both ? kBoth : 0) | (x ? kPipe1 : 0));
                    // the scores before have been read
                    if (issued > 0 && !wait_all(&ctrl->s_free, (uint32_t)(issued - 1) & 1u, &ctrl->gave_up, kErrSFree)) break;
                    tc_fence_after_sync();
                    if (lead) {
#pragma unroll 1
                        for (int sub = 0; sub < kSub; ++sub, da += kSubBytes >> 4, db += k_sub)
#pragma unroll
                            for (int kk = 0; kk < 4; ++kk) mma_ss(to, da + (uint32_t)(kk * 2), db + kk * k_step, idesc, sub + kk > 0);
                        mma_commit(&ctrl->s_full[x]);
                        mma_commit(&ctrl->k_free[st]);
                        if (last) mma_commit(&ctrl->q_free[x]);
                        if (!both) mbar_arrive(&ctrl->k_free[st]);
                        ctrl->order[issued % kOrders] = order;
                        mbar_arrive(&ctrl->order_full[issued % kOrders]);
                    }
                    __syncwarp();
                    ++issued;
                    last_x = x;
                    if (last) ++me.tiles;
                    me.next = last ? me.base + me.count : e + 1;
                    ++me.k;
                    ++me.scores;
                    polls = 0;
                } else if (me.done && other.done) {
                    break;
                } else if (++polls == kIdlePolls) {
                    ctrl->gave_up = kErrIdle;
                    break;
                } else {
                    __nanosleep(20);
                }
                const Pipe was = me;
                me = other;
                other = was;
                x ^= 1;
            }
            if (lead) {
                ctrl->order[issued % kOrders] = make_int2(0, kStop);
                mbar_arrive(&ctrl->order_full[issued % kOrders]);
                mma_commit(&ctrl->drain[0]);     // tensor memory is released only after every MMA has completed
            }
            wait_quiet(&ctrl->drain[0], 0);
            __syncwarp();
        } else {
            // -------------------------------------------------------------- O += P V, in the order of the S
            const bool lead = elect_one();
            constexpr uint32_t idesc = instr_desc_f16(kFmt, kTile, kD, 1);
            const uint64_t v_desc = smem_desc_sw128(smem_u32(smem + kVOff), kSubBytes, 1024);
            uint32_t phase = 0;                // bit x: parity of pipe x's next P
            for (int n = 0;; ++n) {
                if (!wait_all(&ctrl->order_full[n % kOrders], (uint32_t)(n / kOrders) & 1u, &ctrl->gave_up, kErrOrder)) break;
                const int2 order = ctrl->order[n % kOrders];
                if (order.y & kStop) break;
                const int x = (order.y & kPipe1) ? 1 : 0, st = order.x % kSlots;
                const uint32_t o_tmem = tmem_base + kTmemO + x * kD;
                uint32_t p_tmem = tmem_base + kTmemP + x * kTmemPPitch;
                uint64_t db = v_desc + (uint32_t)(st * kTileBytes >> 4);
                uint32_t add = (order.y & kFirst) ? 0u : 1u;
                bool ok = wait_all(&ctrl->v_full[st], (uint32_t)(order.x / kSlots) & 1u, &ctrl->gave_up, kErrV);
#pragma unroll 1
                for (int half = 0; half < 2 && ok; ++half, p_tmem += 32, db += 512) {
                    ok = wait_all(&ctrl->p_full[x][half], (phase >> x) & 1u, &ctrl->gave_up, kErrP);
                    tc_fence_after_sync();
                    if (ok && (order.y & (half ? kHalf1 : kHalf0))) {
                        if (lead) {
#pragma unroll
                            for (int kk = 0; kk < 4; ++kk) mma_ts(o_tmem, p_tmem + kk * 8, db + (uint32_t)(kk * 128), idesc, kk > 0 ? 1u : add);
                        }
                        add = 1;
                    }
                }
                if (!ok) break;
                if (lead) {
                    mma_commit(&ctrl->pv_done[x]);
                    mma_commit(&ctrl->v_free[st]);
                    if (order.y & kLast) mma_commit(&ctrl->o_full[x]);
                    if (!(order.y & kBoth)) mbar_arrive(&ctrl->v_free[st]);
                }
                __syncwarp();
                phase ^= 1u << x;
            }
            if (lead) mma_commit(&ctrl->drain[1]);
            wait_quiet(&ctrl->drain[1], 0);
            __syncwarp();
        }
    } else {
        // ------------------------------------------------------------------ softmax + epilogue
        asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(kSoftmaxRegs));
        const int x = warp >> 2, w4 = warp & 3;
        const uint32_t lane_addr = tmem_base + ((uint32_t)(w4 * 32) << 16);
        const uint32_t s_addr = lane_addr + kTmemS, o_addr = lane_addr + kTmemO + x * kD, p_addr = lane_addr + kTmemP + x * kTmemPPitch;
        uint8_t* stage = smem + kStageOff + warp * 2048;
        const float sc = p.scale_log2;
        const float2 sc2 = make_float2(sc, sc);
        bool ok = true, more = true;
        uint32_t g = 0, tiles = 0;         // steps and tiles (with steps) so far
        Tile now = {-1, 0, 0, 0, 0};
        int begin = 0, end = kEmpty;       // band of this thread's row
        for (int n = 0; more; ++n) {       // the steps of tile n - 1, tile n's band, the epilogue of tile n - 1
            const int steps = now.blocks();
            float m_used = -INFINITY, l_sum = 0.f;
            for (int k = 0; k < steps; ++k, ++g) {
                ok = wait_all(&ctrl->s_full[x], g & 1u, &ctrl->gave_up, kErrS);
                if (!ok) break;
                tc_fence_after_sync();
                const int c0 = (now.first() + k) * kTile;
                const int v_lo = begin - c0, v_hi = end - c0;  // valid keys of this step: [v_lo, v_hi)
                uint32_t r[kTile];
#pragma unroll
                for (int ch = 0; ch < kChunks; ++ch) tmem_ld32(s_addr + ch * kChunk, r + ch * kChunk);
                tmem_ld_wait();
                tc_fence_before_sync();
                __syncwarp();
                if (lane == 0) mbar_arrive(&ctrl->s_free);
                if (!__all_sync(0xffffffffu, v_lo <= 0 && v_hi >= kTile)) sm::mask_scores(r, v_lo, v_hi);
                const float m_new = fmaxf(m_used, sm::max_score(r) * sc);
                // lazy rescale: only when a row's maximum has grown by more than 2^8 (false when both are -inf)
                const bool need = (m_new - m_used) > kRescaleThreshold;
                // before a rescale of O or the first store of P, the PV before has to be complete (it usually is)
                auto pv_wait = [&]() {
                    ok = g == 0 || wait_all(&ctrl->pv_done[x], (g - 1) & 1u, &ctrl->gave_up, kErrPv);
                    tc_fence_after_sync();
                };
                if (__any_sync(0xffffffffu, need)) {
                    const float corr = need ? ex2(m_used - m_new) : 1.f;
                    if (need) m_used = m_new;
                    l_sum *= corr;
                    if (k > 0) {
                        pv_wait();
                        if (ok) rescale_o(o_addr, corr);
                    }
                }
                const float m_eff = (m_used == -INFINITY) ? 0.f : m_used;
                const float2 nm2 = make_float2(-m_eff, -m_eff);
                float2 acc0 = make_float2(0.f, 0.f), acc1 = make_float2(0.f, 0.f);
#pragma unroll
                for (int half = 0; half < 2; ++half) {
                    uint32_t* pk = r + half * (kTile / 4);
                    sm::exp_scores<T, kTile / 2>(r + half * (kTile / 2), pk, sc2, nm2, acc0, acc1);
                    if (half == 0) pv_wait();
                    tmem_st32(p_addr + half * 32, pk);
                    tmem_st_wait();
                    tc_fence_before_sync();
                    __syncwarp();
                    if (lane == 0) mbar_arrive(&ctrl->p_full[x][half]);      // half 0: on its way to the tensor core
                }
                l_sum += (acc0.x + acc0.y) + (acc1.x + acc1.y);
                if (!ok) break;
            }
            if (!ok) break;
            const Tile was = now;
            const int row_start = begin, row_end = end;
            // the next item's tile and the row's band: on their way during the epilogue
            ok = wait_all(&ctrl->item_full[n % kItems], (uint32_t)(n / kItems) & 1u, &ctrl->gave_up, kErrItem);
            if (!ok) break;
            more = ctrl->item[n % kItems].stop == 0;
            now = ctrl->item[n % kItems].t[x];
            __syncwarp();
            if (lane == 0) mbar_arrive(&ctrl->item_free[n % kItems]);
            begin = 0; end = kEmpty;
            const int u = now.u0 + w4 * 32 + lane;
            if (more && now.u0 >= 0 && u < p.rows) {
                const int2 band = __ldg(p.bands + (int64_t)now.res * p.rows + u);
                begin = band.x; end = band.y;
            }
            if (was.u0 < 0) continue;
            if (steps > 0) {
                ok = wait_all(&ctrl->o_full[x], tiles & 1u, &ctrl->gave_up, kErrO);
                if (!ok) break;
                tc_fence_after_sync();
                ++tiles;
            }
            // epilogue: O / l for band rows, V[start] for single-element rows, zero otherwise.
            // (all scores of a row -inf: zeros)
            const float inv = l_sum > 0.f ? 1.f / l_sum : 0.f;
            const int64_t head = was.bh * p.n_rows;
            const int u_warp = was.u0 + w4 * 32;
            const int64_t row_real = (int64_t)(u_warp + lane) * p.stride + was.res;
            const bool exists = u_warp + lane < p.rows;
            if (kLse && exists) {
                float e = -INFINITY;
                if (row_end > 0) e = lse_from_log2(m_used, l_sum);
                else if (row_end == kSingle) e = single_lse<T>(p, head, row_real, row_start);
                p.lse[head + row_real] = e;
            }
            // through the warp's staging memory to stores of 64 contiguous bytes, 32 columns at a time
            const uint32_t in_band = __ballot_sync(0xffffffffu, row_end > 0);
            if (in_band != 0) {
                const float2 inv2 = make_float2(inv, inv);
                const int piece = lane & 3;
                char* to = reinterpret_cast<char*>(p.o) + ((head + (int64_t)(u_warp + (lane >> 2)) * p.stride + was.res) * kD + piece * 8) * 2;
                const int64_t to_step = (int64_t)8 * p.stride * kD * 2;
#pragma unroll 1
                for (int c = 0; c < kD; c += 32) {
                    uint32_t r[32];
                    tmem_ld32(o_addr + c, r);
                    tmem_ld_wait();
#pragma unroll
                    for (int i = 0; i < 4; ++i) {
                        uint4 out;
                        uint32_t* o32 = reinterpret_cast<uint32_t*>(&out);
                        const uint32_t* f = r + 8 * i;
#pragma unroll
                        for (int j = 0; j < 4; ++j) {
                            const float2 y = mul2(make_float2(__uint_as_float(f[2 * j]), __uint_as_float(f[2 * j + 1])), inv2);
                            o32[j] = pack2<T>(y.x, y.y);
                        }
                        *reinterpret_cast<uint4*>(stage + lane * 64 + ((i ^ ((lane >> 1) & 3)) << 4)) = out;
                    }
                    __syncwarp();
#pragma unroll
                    for (int i = 0; i < 4; ++i) {
                        const int row = 8 * i + (lane >> 2);
                        const uint4 v = *reinterpret_cast<const uint4*>(stage + row * 64 + ((piece ^ ((row >> 1) & 3)) << 4));
                        if ((in_band >> row) & 1u) *reinterpret_cast<uint4*>(to + i * to_step + c * 2) = v;
                    }
                    __syncwarp();
                }
            }
            // the other rows, one per half warp at a time
#pragma unroll 1
            for (uint32_t left = __ballot_sync(0xffffffffu, exists) & ~in_band; left != 0;) {
                const int r0 = __ffs(left) - 1;
                left &= left - 1;
                const int r1 = left != 0 ? __ffs(left) - 1 : r0;
                left &= left - 1;
                const int at = lane < 16 ? r0 : r1, c = (lane & 15) * 8;
                const int start = __shfl_sync(0xffffffffu, row_start, at), kind = __shfl_sync(0xffffffffu, row_end, at);
                uint4 v = make_uint4(0, 0, 0, 0);
                if (kind == kSingle) v = *reinterpret_cast<const uint4*>(reinterpret_cast<const T*>(p.v) + (head + start) * kD + c);
                *reinterpret_cast<uint4*>(reinterpret_cast<T*>(p.o) + (head + (int64_t)(u_warp + at) * p.stride + was.res) * kD + c) = v;
            }
        }
    }
    tc_fence_before_sync();
    __syncthreads();
    if (threadIdx.x == 0) publish_gave_up(p.status, &ctrl->gave_up);
    if (warp == kQkWarp) {
        __syncwarp();
        tc_fence_after_sync();
        tmem_dealloc(tmem_base, kTmemCols);
    }
}

template <typename T>
static int32_t launch(const Maps3& maps, const Params& prm, cudaStream_t st) {
    auto kern = prm.lse != nullptr ? attention_duo_kernel<T, true> : attention_duo_kernel<T, false>;
    if (!allow_dynamic_smem(reinterpret_cast<const void*>(kern), kSmemBytes)) return SPLAT_ERR_LAUNCH;
    return launch_kernel(kern, prm.pairs + (prm.total > 2 * prm.pairs ? prm.total - 2 * prm.pairs : 0), kThreads, kSmemBytes, st, maps, prm);
}

}  // namespace duo
}  // namespace band

// Operands checked by attention_band(): d = 128, a stride that divides n_rows, a band table, and the tiles of all heads
// and classes fit 31 bits.
int32_t attention_duo(const void* q, const void* k, int kt_major, const void* v, void* o, int64_t bh, int64_t n_rows, int64_t stride,
                      float scale, int32_t dtype, int32_t* status_word, const int32_t* band_table, float* lse, cudaStream_t st) {
    using namespace band;
    duo::Params p;
    p.q = q; p.k = k; p.v = v; p.o = o; p.lse = lse;
    p.status = status_word; p.mirror = status_mirror(status_word);
    p.n_rows = n_rows; p.stride = (int)stride; p.rows = (int)(n_rows / stride);
    p.pitch = (uint32_t)((p.rows + duo::kTile - 1) / duo::kTile);
    p.kt_major = kt_major; p.scale_log2 = scale * kLog2e;
    p.bands = reinterpret_cast<const int2*>(band_table);
    p.tiles = p.bands + n_rows;
    p.total = (uint32_t)(bh * stride * p.pitch);
    // A last wave of no more tiles than SMs goes one tile to an SM: alone a tile takes two thirds of the time of two.
    const uint32_t rest = p.total % (2 * 148);
    p.pairs = rest <= 148 ? (p.total - rest) / 2 : (p.total + 1) / 2;
    duo::Maps3 maps;
    auto view = [&](CUtensorMap* m, const void* base) {
        return make_map_view(m, base, dtype, bh, n_rows, duo::kD, stride, 0, stride, p.rows, duo::kTile);
    };
    if (!view(&maps.m[0], q) || !(kt_major ? make_map_kt(&maps.m[1], k, dtype, bh, n_rows, duo::kD, 128) : view(&maps.m[1], k)) ||
        !view(&maps.m[2], v))
        return SPLAT_ERR_DRIVER;
    return dtype == SPLAT_BF16 ? duo::launch<__nv_bfloat16>(maps, p, st) : duo::launch<__half>(maps, p, st);
}

}  // namespace splat
