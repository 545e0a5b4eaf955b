// fcs_infer_layout.h -- where the inference kernel (fcs_mlp.cu) puts a tile's
// activations in shared memory: 128 rows of 256 BF16 in four chunks of 64
// columns, K-major with 128-byte swizzle, and who writes which bytes.
//
// Eight warps work on a tile, two to a group q of 32 rows.  Warp (q, part)
//   * writes the input of rows 32 q + 16 part + 0..15, every column;
//   * writes a hidden layer's outputs of all 32 rows, columns 128 part + 0..127;
//   * stages the last layer's outputs, 16 columns of the 32 rows at a time.
// A layer's MMAs order one layer's writes after the other's, but nothing
// orders the two warps of a group between the last layer and the next tile's
// input.  So a warp stages in bytes that it alone writes as that input.
#pragma once

namespace fcs {

constexpr int kActChunkBytes = 128 * 64 * 2;

// Byte offset of element (r, k)
constexpr int act_offset(int r, int k) {
    return (k >> 6) * kActChunkBytes + r * 128 + ((((k & 63) >> 3) ^ (r & 7)) << 4) + (k & 7) * 2;
}

// First of the 16 rows whose input warp (q, part) writes
constexpr int input_row(int q, int part) { return 32 * q + 16 * part; }

// Where it stages: floats from its input rows' first bytes on, column u (of 16)
// of row 32 q + r at stage_index(r, u), rows r and r + 1 in 128 bytes.  The lanes
// of a column, and of rows r and r + 1, fall on 32 different banks.
constexpr int stage_offset(int q, int part) { return input_row(q, part) * 128; }
constexpr int stage_index(int r, int u) { return (r & 31) * 16 + ((u ^ (r >> 1)) & 15); }

}  // namespace fcs
