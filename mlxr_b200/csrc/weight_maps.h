// TMA descriptions of packed weights and activations, shared by the tensor-core launchers.
#pragma once
#include <cuda.h>
#include <stddef.h>

namespace mlxr {

// The maps of one packed matrix [N, K] for tiles of `tile_rows` of its rows, a super-block (256 weights)
// per box.  NF4 rows are 136 bytes per 256 weights, so with an odd number of super-blocks every
// other row starts 8 bytes off a 16-byte boundary: even and odd rows get a map each (out[0], out[1]), with
// twice the row stride, the odd one starting at the 16-byte boundary at or below row 1 (*odd_shift bytes
// before it).  Rows past the end read as zero.
int weight_maps(int qt, const void* w, int N, int K, int tile_rows, CUtensorMap* out, int* odd_shift);
// Packed rows of `row_bytes`, boxes of box_bytes x box_rows; rows past the end and bytes past a row's read as zero
int rows_map(const void* w, int rows, size_t row_bytes, int box_bytes, int box_rows, CUtensorMap* out);
// X [M, K] of a 16-bit type, boxes of 64 x `rows` with the 128-byte swizzle; rows past M read as zero
int activation_map(const void* x, int M, int K, int dtype, int rows, CUtensorMap* out);
// The same with `blocks` consecutive 64-wide k-blocks in a box, one [rows][64] tile behind the other: coordinates (0, row, k-block)
int activation_blocks_map(const void* x, int M, int K, int dtype, int rows, int blocks, CUtensorMap* out);
// Y [M, N] of a 16-bit type for stores, boxes of box_cols (16: plain, 32: 64-byte swizzle) x box_rows
int result_map(void* y, int M, int N, int dtype, int box_cols, int box_rows, CUtensorMap* out);
int device_sms(int* out);

}  // namespace mlxr
