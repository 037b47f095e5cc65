// fp32 operands as three bf16 numbers each for the tensor cores (attention_split.cu, ops_split.cu; why, and what it costs in
// accuracy: see there).
//
// K and V are multiplied 64 keys at a time.  kWorkers threads bring a step's block from global memory through registers, split it
// and place it in shared memory: three pieces one behind the other, each rows of 128 bytes (64 numbers) with the 128-byte
// swizzle, columns past 64 in a second half.
#pragma once

#include "common.cuh"
#include "softmax_math.cuh"
#include "tc_ptx.cuh"

namespace splat {
namespace split {

using namespace tc;
using sm::add2;
using sm::fma2;
using sm::mul2;

constexpr int kTile = 128;               // rows of a tile
constexpr int kKeys = 64;                // keys of a step
constexpr int kWorkers = 256;            // warps 0-7: thread = (row, half of the columns)
constexpr int kMmaWarp = 8;
constexpr int kSubBytes = kKeys * 128;   // 64 rows x 64 bf16
// bytes of one piece of a step's K or V, pieces of 8 elements per thread
template <int D> constexpr int kPieceBytes = (D == 128 ? 2 : 1) * kSubBytes;
template <int D> constexpr int kUnits = kKeys * D / 8 / kWorkers;

__device__ __forceinline__ void load8(float (&x)[8], const float* p, int vec) {
    if (vec == 8) {
        asm volatile("ld.global.nc.v8.f32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
            : "=f"(x[0]), "=f"(x[1]), "=f"(x[2]), "=f"(x[3]), "=f"(x[4]), "=f"(x[5]), "=f"(x[6]), "=f"(x[7]) : "l"(p));
    } else {
        const float4 a = __ldg(reinterpret_cast<const float4*>(p)), b = __ldg(reinterpret_cast<const float4*>(p) + 1);
        x[0] = a.x; x[1] = a.y; x[2] = a.z; x[3] = a.w;
        x[4] = b.x; x[5] = b.y; x[6] = b.z; x[7] = b.w;
    }
}
// Two numbers, times 2^16 -> their three bf16 pieces, packed.  fp32's smallest number is 2^-149, bf16's 2^-133: unscaled, an
// operand below 2^-110 would lose its last bits.  A product is 2^32 times too large (kDown); operands above 2^111 and sums above
// 2^96 become infinite by it, and their rows are computed again like those of other infinities.
//   kScale  false for the weights of a softmax: beside their row's largest, 1, those below 2^-110 are known to 2^-17 at most
//   kShort  the first piece has six bits instead of eight (6 + 8 + 8 and a sign for each are 24 all the same), so that the products
//           of first pieces are of 14 bits and sums of them have room in 24: see attention_split.cu
constexpr float kUp = 65536.f, kDown = 1.f / (65536.f * 65536.f);
template <bool kScale, bool kShort>
__device__ __forceinline__ void split2(float2 x, uint32_t& h, uint32_t& m, uint32_t& l) {
    const float2 minus = make_float2(-1.f, -1.f);
    if (kScale) x = mul2(x, make_float2(kUp, kUp));
    uint32_t a, b;
    if (kShort) {
        a = (__float_as_uint(x.x) + 0x20000u) & 0xfffc0000u;
        b = (__float_as_uint(x.y) + 0x20000u) & 0xfffc0000u;
        h = __byte_perm(a, b, 0x7632);
    } else {
        h = sm::pack2<__nv_bfloat16>(x.x, x.y);
        a = h << 16;
        b = h & 0xffff0000u;
    }
    x = fma2(make_float2(__uint_as_float(a), __uint_as_float(b)), minus, x);
    m = sm::pack2<__nv_bfloat16>(x.x, x.y);
    x = fma2(make_float2(__uint_as_float(m << 16), __uint_as_float(m & 0xffff0000u)), minus, x);
    l = sm::pack2<__nv_bfloat16>(x.x, x.y);
}
template <bool kScale = true, bool kShort = false>
__device__ __forceinline__ void split8(const float (&x)[8], uint4& h, uint4& m, uint4& l) {
    split2<kScale, kShort>(make_float2(x[0], x[1]), h.x, m.x, l.x);
    split2<kScale, kShort>(make_float2(x[2], x[3]), h.y, m.y, l.y);
    split2<kScale, kShort>(make_float2(x[4], x[5]), h.z, m.z, l.z);
    split2<kScale, kShort>(make_float2(x[6], x[7]), h.w, m.w, l.w);
}
__device__ __forceinline__ void tmem_st4(uint32_t taddr, uint4 r) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x4.b32 [%0], {%1, %2, %3, %4};" ::"r"(taddr), "r"(r.x), "r"(r.y), "r"(r.z), "r"(r.w)
                 : "memory");
}
// Hides from the compiler where a descriptor's low word (desc_lo()) or a tensor-memory address comes from: it otherwise keeps the sums
// of all 48 MMAs of a step in registers.
__device__ __forceinline__ uint32_t hidden(uint32_t x) {
    asm volatile("" : "+r"(x));
    return x;
}

// The six products: piece (0 h, 1 m, 2 l) of A and of B, the largest product last.
__host__ __device__ constexpr int piece_a(int i) { return (0x001102 >> (4 * i)) & 15; }
__host__ __device__ constexpr int piece_b(int i) { return (0x010120 >> (4 * i)) & 15; }

// Of a step's block of a (rows, D) array, class rows u .. u + 63 (rows from rows_v on: 0); base: the class's first row.
template <int D>
__device__ __forceinline__ void ask_rows(float (&x)[kUnits<D>][8], const float* base, int64_t pitch, int u, int rows_v, int vec) {
#pragma unroll
    for (int i = 0; i < kUnits<D>; ++i) {
        const int unit = threadIdx.x + i * kWorkers, row = u + unit / (D / 8), c = unit % (D / 8) * 8;
        if (row < rows_v) {
            load8(x[i], base + (int64_t)row * pitch + c, vec);
        } else {
#pragma unroll
            for (int e = 0; e < 8; ++e) x[i][e] = 0.f;
        }
    }
}
// ... of a (D, n_rows) K^T, eight keys of a row at a time where they are contiguous and aligned (vec > 1).  One branch for all units of a
// thread: with one for each the fused kernel at d = 128 spilled where it counted, us, each / one: H8 L21120 window 25 161 / 150,
// L8606 +-318 48.8 / 43.6, H22 L1152 window 96 39.7 / 38.4; d64 104.1 / 103.5 (B2 H16 L4096 window 256).  kAnew: the row addresses are
// formed at every step instead of kept, which SDDMM has no registers for (us, kept / anew: d128 H6 L2944 +-38 17.4 / 16.2).
template <int D, bool kAnew>
__device__ __forceinline__ void ask_kt(float (&x)[kUnits<D>][8], const float* base, int n_rows, int stride, int res, int u, int rows_v,
                                       int vec) {
    // (a thread's units are at the same keys, kWorkers * 8 / kKeys rows apart)
    const int key = u + (int)threadIdx.x % (kKeys / 8) * 8;
    const int rows = kAnew ? (int)hidden((uint32_t)n_rows) : n_rows;
    const float* src = base + (int64_t)(threadIdx.x / (kKeys / 8)) * rows;
    const int64_t pitch = (int64_t)(kWorkers * 8 / kKeys) * rows;
    if (vec > 1 && key + 8 <= rows_v) {
        src += key;
#pragma unroll
        for (int i = 0; i < kUnits<D>; ++i, src += pitch) load8(x[i], src, vec);
    } else {
        src += (int64_t)key * stride + res;
#pragma unroll
        for (int i = 0; i < kUnits<D>; ++i, src += pitch)
#pragma unroll
            for (int e = 0; e < 8; ++e) x[i][e] = key + e < rows_v ? __ldg(src + (int64_t)e * stride) : 0.f;
    }
}
// kKt: the block came from ask_kt()
template <int D, bool kKt>
__device__ __forceinline__ void put(const float (&x)[kUnits<D>][8], uint8_t* dst) {
#pragma unroll
    for (int i = 0; i < kUnits<D>; ++i) {
        const int unit = threadIdx.x + i * kWorkers;
        constexpr int kPerRow = kKt ? kKeys / 8 : D / 8;
        const int row = unit / kPerRow, piece = unit % kPerRow;
        uint8_t* to = dst + (kKt ? 0 : (piece >> 3) * kSubBytes) + row * 128 + (((piece & 7) ^ (row & 7)) << 4);
        uint4 h, m, l;
        split8(x[i], h, m, l);
        *reinterpret_cast<uint4*>(to) = h;
        *reinterpret_cast<uint4*>(to + kPieceBytes<D>) = m;
        *reinterpret_cast<uint4*>(to + 2 * kPieceBytes<D>) = l;
    }
    fence_proxy_async_smem();
}
// elements that a load of an array's rows (multiples of 32 bytes long) may take at a time, of K^T's
inline int vec_of(const void* base) { return (reinterpret_cast<uintptr_t>(base) & 31u) == 0 ? 8 : 4; }
inline int vec_of_k(const void* base, int kt, int64_t stride, int64_t n_rows) {
    return !kt ? vec_of(base) : stride != 1 || n_rows % 4 != 0 ? 1 : n_rows % 8 != 0 ? 4 : vec_of(base);
}

}  // namespace split
}  // namespace splat
