// What an attention pass needs of its operands before its tile kernels, in one
// reading of each: row digits, column maxima and digits, exponent ranges,
// value statistics, D = rowsum(d_out∘out).
#pragma once

#include <cstdint>

#include "attention.cuh"
#include "common.h"

namespace ef {

// The smallest and largest exponents of a set of rows, as maxima of e and -e
// plus this (so that a pair starts at zero).
constexpr int kExponentBias = 1 << 16;

// One operand x [batches][rows][cols], rows past lens[w] (or `rows`) taken as
// zeros up to rows_pad (a multiple of 64). Null outputs are left out.
struct RowSet {
  const double* x = nullptr;
  int64_t rows = 0, rows_pad = 0, cols = 0;
  const int64_t* lens = nullptr;
  // Row digits [w·S + s][rows_pad][k_pad] and exponents [w][rows_pad] (cols <=
  // k_pad, 64 or 128); with skip_padding the padding rows' digits stay unwritten.
  int8_t* digits = nullptr;
  int32_t* e = nullptr;
  int k_pad = 64;
  bool skip_padding = false;
  int* range = nullptr;  // (max e, max -e) over the padded rows, both biased, folded in
  unsigned long long* colmax = nullptr;  // [w][cols], the bits of the largest magnitudes, folded in
  // Value statistics by position (as value_stats gives them), and each block of
  // 64 positions' extrema of them, [w][rows_pad / 64].
  uint8_t* flag = nullptr;
  double* largest = nullptr;
  double* smallest = nullptr;
  double* block_largest = nullptr;
  double* block_smallest = nullptr;
  // Row dots with `other` [batches][rows][cols]: [w][rows], and with zeros up to
  // rows_pad; and a row value copied to rows_pad likewise.
  const double* other = nullptr;
  double* dots = nullptr;
  double* dots_pad = nullptr;
  const double* value = nullptr;
  double* value_pad = nullptr;
  int bad = 1;  // ORed into *status where a live value isn't finite
};

// Columns of x [batches][rows][cols] as K-major digits [w·S + s][cols_pad][rows_pad]
// under their maxima's powers of two, e [w][cols_pad].
struct ColumnSet {
  const double* x = nullptr;
  int64_t rows = 0, rows_pad = 0, cols = 0, cols_pad = 0;
  const int64_t* lens = nullptr;
  const unsigned long long* colmax = nullptr;
  bool skip_padding = false;  // tiles of rows all past their length stay unwritten
  int8_t* digits = nullptr;
  int32_t* e = nullptr;
};

constexpr int kPrepareSets = 4;

// One launch each over every set (six slices).
void prepare_rows(Context& ctx, const RowSet* sets, int n, int64_t batches, int* status, cudaStream_t s);
void prepare_columns(Context& ctx, const ColumnSet* sets, int n, int64_t batches, cudaStream_t s);

// The extrema of blocks of 64 positions, [w][(lnj + 63) / 64], from the positions'
// statistics (where prepare_rows didn't give them).
void block_extrema(Context& ctx, int64_t batches, int64_t lnj, const double* largest, const double* smallest,
                   double* block_largest, double* block_smallest, cudaStream_t s);
// Each row's largest and smallest nonzero value magnitude over its allowed
// keys (the bounds of Bounds::hold, fused.rs:1058-1086), from the positions'
// statistics and their blocks' extrema ([w][blocks]).
void row_bounds(Context& ctx, const Mask& m, int64_t nx, int64_t blocks, const double* largest, const double* smallest,
                const double* block_largest, const double* block_smallest, double* rl, double* rs, cudaStream_t s);

// Whether the status words say that a split pass may run with normal powers of
// two: no value that isn't finite (word 0), and each pair of ranges (words 2 p ..,
// biased) keeping eq + ek within [-low, top].
struct Ready {
  const int* status = nullptr;  // null: no question
  int pairs = 1;                // (words 2..5), 2: and (words 6..9)
  int top = 1023, low = 1022;
  __host__ __device__ bool ok() const {
    if (!status) return true;
    if (status[0]) return false;
    for (int p = 0; p < pairs; p++) {
      const int* r = status + 2 + 4 * p;
      if (r[0] + r[2] - 2 * kExponentBias > top || r[1] + r[3] - 2 * kExponentBias > low) return false;
    }
    return true;
  }
};

}  // namespace ef
