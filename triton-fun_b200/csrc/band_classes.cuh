// Residue classes of a band pattern as one launch (attention_wide.cu, ops_band.cu).
//
// Class r of L rows and stride s has L / s rows, the first L mod s classes one more.  A tensor map describes classes of
// one length, so a stride that does not divide L needs two sets of them; the launch carries both and a CTA
// takes the one of its class (blockIdx.y).  With a launch per length the second waited for the first to end:
// B3 H1 L1740 strided 13 bf16 (fused, us): 12.4 -> 6.6; B2 H8 L10000 d64 dilated by 3: 65.0 -> 58.3; SDDMM, softmax
// and SpMM of B3 H7 L513 strided 14: 36.5 -> 21.3.
#pragma once
#include <cuda.h>

#include "common.cuh"

namespace splat {
namespace band {

// defined in attention_band.cu
bool allow_dynamic_smem(const void* kernel, int bytes);
bool make_map_view(CUtensorMap* map, const void* base, int32_t dtype, int64_t bh, int64_t n_rows, int64_t d, int64_t stride,
                   int64_t res0, int64_t count, int64_t rows, int box_rows);
bool make_map_kt(CUtensorMap* map, const void* base, int32_t dtype, int64_t bh, int64_t n_cols, int64_t d, int64_t box_d);

template <int N> struct Maps { CUtensorMap part[2][N]; };    // of the longer classes, of the others

struct Classes {
    int longer;          // classes of rows + 1 rows: the first L mod stride
    int rows;            // of the others
    int tile_pitch;      // tiles of a class in the band table

    Classes() = default;
    Classes(int64_t n_rows, int64_t stride, int tile)
        : longer((int)(n_rows % stride)), rows((int)(n_rows / stride)),
          tile_pitch((int)(((n_rows + stride - 1) / stride + tile - 1) / tile)) {}
    dim3 grid(int64_t stride, int64_t bh) const {
        return dim3((unsigned)tile_pitch, (unsigned)(rows > 0 ? stride : longer), (unsigned)bh);
    }
    int64_t tiles(int64_t stride, int64_t bh) const { return (int64_t)tile_pitch * (rows > 0 ? stride : longer) * bh; }     // of the grid
    bool has(int part) const { return part == 0 ? longer > 0 : rows > 0; }
    // view of a (BH, L, d) array: rows of `part`'s classes
    bool view(CUtensorMap* map, const void* base, int32_t dtype, int64_t bh, int64_t n_rows, int64_t d, int64_t stride,
              int part, int box_rows) const {
        return make_map_view(map, base, dtype, bh, n_rows, d, stride, part == 0 ? 0 : longer, part == 0 ? longer : stride - longer,
                             part == 0 ? rows + 1 : rows, box_rows);
    }
    __device__ __forceinline__ int part(int res) const { return res < longer ? 0 : 1; }
    __device__ __forceinline__ int rows_of(int res) const { return res < longer ? rows + 1 : rows; }
    __device__ __forceinline__ int in_part(int res) const { return res < longer ? res : res - longer; }
    __device__ __forceinline__ int first_row(int res) const { return res * rows + min(res, longer); }    // in class order
};

}  // namespace band
}  // namespace splat
