// Dense products for the dense fold and the device entry points.
#pragma once

#include <cuda.h>
#include <cuda_runtime.h>

#include <cstdint>

#include "common.h"

namespace ef {

constexpr int kDefaultSlices = 6;
constexpr int kMinSlices = 2;
constexpr int kMaxSlices = 7;

// C[w] = A[w] · B[w] for w < batches: A [batches][m][k] row-major, B either
// natural [batches][k][n] (b_natural) or transposed [batches][n][k], C
// [batches][m][n]. Every value of A and B must be finite: each row of A and
// each column of B is cut into `slices` int8 digits under a power-of-two
// scale, the digit products are summed exactly in int32 on the tensor cores,
// level by level, and the levels are combined in FP64.
void split_gemm(Context& ctx, const double* a, const double* b, bool b_natural, double* c, int64_t batches,
                int64_t m, int64_t n, int64_t k, int slices, cudaStream_t stream);

// The gradients of C = A · B (B natural) for d_c [batches][m][n]: d_a = d_c · Bᵀ
// [batches][m][k] and d_b = Aᵀ · d_c [batches][k][n], either null to leave out.
// The same digits and products as two split_gemm calls, Aᵀ given as an array.
void split_gradients(Context& ctx, const double* a, const double* b, const double* d_c, double* d_a, double* d_b,
                     int64_t batches, int64_t m, int64_t n, int64_t k, int slices, cudaStream_t stream);

// C[w] = A[w] · B[w] in FP64 on the CUDA cores, B natural [batches][k][n],
// each cell's terms added in k order from +0.0 with unfused multiply and add,
// skipping cells of A whose 2-bit `held` code (16 per word, if given) isn't 2.
// With zblock > 0, the terms of each block of `zblock` values of k are summed
// apart and the blocks added in order (the reference's accumulate for small
// outputs, dense.rs:752-768).
void fp64_gemm(Context& ctx, const double* a, const uint32_t* held, const double* b, double* c, int64_t batches,
               int64_t m, int64_t n, int64_t k, int64_t batch_of_row, int64_t zblock, bool fused_multiply_add,
               cudaStream_t stream);

// A TMA map over digit planes [planes][rows][k_pad] (uint8), boxes of 64
// bytes of k by box_rows rows by box_planes planes, 64-byte swizzle.
CUtensorMap digit_planes_map(const int8_t* digits, int64_t k_pad, int64_t rows, int64_t planes, int box_rows,
                             int box_planes);

// A TMA map over doubles [batches][rows][cols] (cols a multiple of 2),
// boxes of box_cols (at most 16) by box_rows in the 128-byte swizzle.
CUtensorMap f64_boxes_map(const double* x, int64_t cols, int64_t rows, int64_t batches, int box_cols, int box_rows);

// BT[w][j][i] = B[w][i][j] for a [batches][rows][cols] array.
void transpose(const double* b, double* bt, int64_t batches, int64_t rows, int64_t cols, cudaStream_t stream);

}  // namespace ef
