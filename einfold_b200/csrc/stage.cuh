// Staging Arrow columns into HBM, once per call, and small device helpers
// shared by the folds.
#pragma once

#include <cuda_runtime.h>

#include <vector>

#include "arrow.h"
#include "common.h"
#include "fold.h"

namespace ef {

// One column of a relation, every batch concatenated, in HBM.
struct DeviceColumn {
  Kind kind = Kind::Other;
  int width = 0;
  int64_t rows = 0;
  int64_t nulls = 0;
  DeviceBuffer<uint8_t> data;   // fixed-width values (rows * width)
  const uint8_t* alias = nullptr;  // the caller's device buffer, used in place of `data`
  const uint8_t* ptr() const { return alias ? alias : data.get(); }
  DeviceBuffer<uint8_t> valid;  // one byte per row, 1 = valid; empty when nulls == 0
  // var-length kinds
  DeviceBuffer<int64_t> offsets;  // rows + 1
  DeviceBuffer<uint8_t> bytes;
};

// Copies column `col` of every batch into HBM; validity as bytes.
DeviceColumn stage_column(Context& ctx, const Relation& r, int col, bool with_validity = true);

// Keys of an integer column as int64, with the largest value and whether any
// is negative or too large for int64 (an unsigned 2^63 or more).
struct KeyStats {
  int64_t max = -1;
  bool negative = false;
  bool too_large = false;
};
DeviceBuffer<int64_t> keys_as_i64(Context& ctx, const DeviceColumn& c, KeyStats* stats);

// Exclusive prefix sum of n flags (uint8) into int64 positions; returns the total.
int64_t exclusive_scan_flags(Context& ctx, const uint8_t* flags, int64_t n, int64_t* out);

// Packs n bytes (0/1) into an Arrow validity bitmap of (n + 7) / 8 bytes.
void pack_bits(Context& ctx, const uint8_t* bytes, int64_t n, uint8_t* bits);

// Device to host, into a fresh host buffer.
HostBuffer to_host(Context& ctx, const void* dev, size_t bytes);

// A result buffer from a device buffer: moved into the result as it is when
// the result stays in device memory, else copied to host memory.
template <class T>
Buffer result_buffer(Context& ctx, DeviceBuffer<T>& dev, size_t bytes, bool on_device) {
  if (!on_device) return Buffer(to_host(ctx, dev.get(), bytes));
  Buffer b;
  b.ptr = dev.ptr;
  b.bytes = bytes;
  b.device = ctx.device;
  b.capacity = dev.count * sizeof(T);
  dev.ptr = nullptr;
  dev.count = 0;
  return b;
}

constexpr int kMaxDims = 8;

// A row's cell in a matrix: Σ_i key[i][row]·stride[i].
struct CellKeys {
  int n = 0;
  const int64_t* key[2 * kMaxDims] = {};
  int64_t stride[2 * kMaxDims] = {};
};

// Where output keys come from: position x (in_x) or y, their stride and extent.
struct KeyAt {
  int in_x;
  int64_t stride, extent;
  __device__ __forceinline__ int64_t at(int64_t x, int64_t y) const { return ((in_x ? x : y) / stride) % extent; }
};

// The output's key columns: where each key comes from, its width in bytes
// and its device buffer.
struct OutKeys {
  int n = 0;
  KeyAt key[kMaxDims];
  int width[kMaxDims];
  void* out[kMaxDims];
};

// n / d for 32-bit n by a multiplication: q = (hi32(n·m) + n) >> s with
// s = ceil(log2 d) and m = floor(2^32·(2^s - d)/d) + 1 (T. Granlund and
// P. L. Montgomery, "Division by invariant integers using multiplication",
// PLDI 1994). A divisor of 2^32 or more gives 0.
struct Divisor {
  uint32_t m = 1, s = 0;
  uint64_t d = 1;
  Divisor() = default;
  explicit Divisor(uint64_t by) : d(by) {
    if (by > UINT32_MAX) {
      m = 0;
      s = 32;
      return;
    }
    while ((1ull << s) < by) s++;
    m = (uint32_t)(((((1ull << s) - by) << 32) / by) + 1);
  }
  __host__ __device__ __forceinline__ uint32_t operator()(uint32_t n) const {
    return (uint32_t)((((uint64_t)n * m >> 32) + n) >> s);
  }
};

// The key columns of a result holding every cell (x, y) of nx rows of ny
// cells in order (below 2^32 in all), written to keys.out: the result's values
// are then the matrix of cells itself.
void emit_keys(Context& ctx, const OutKeys& keys, uint64_t nx, uint64_t ny);

// The keys of output dimensions along x (or y), one table per key:
// table[k][p] = (p / stride) % extent, so that emitting needs no division.
__global__ void key_tables(int64_t n, OutKeys keys, int in_x, int64_t* __restrict__ tables);

// An int64 key narrowed to an output column of `width` bytes (Arrow's cast
// of an in-range value).
__device__ __forceinline__ void store_key(void* base, int width, int64_t i, int64_t v) {
  switch (width) {
    case 1: ((uint8_t*)base)[i] = (uint8_t)v; break;
    case 2: ((uint16_t*)base)[i] = (uint16_t)v; break;
    case 4: ((uint32_t*)base)[i] = (uint32_t)v; break;
    default: ((int64_t*)base)[i] = v; break;
  }
}

// Keys of every batch of a relation for one operand, staged as int64, with
// extents.
struct StagedKeys {
  std::vector<DeviceColumn> cols;           // staged columns (int64 ones read in place)
  std::vector<DeviceBuffer<int64_t>> wide;  // other integer columns widened to int64
  std::vector<const int64_t*> keys;         // per key of the operand, in op.keys order
  std::vector<int64_t> extent;              // per key
};

// Stages operands' key columns, all read in one launch and one wait; declines
// where dense::keys (crates/einfold-kernels/src/dense.rs:97-111) returns None: a
// key column that isn't integers, a NULL key, a negative one.
std::vector<StagedKeys> stage_keys(Context& ctx, const std::vector<std::pair<const OperandD*, const Relation*>>& ops);
inline StagedKeys stage_keys(Context& ctx, const OperandD& op, const Relation& r) {
  return std::move(stage_keys(ctx, {{&op, &r}})[0]);
}

// Where `op`'s rows go in a matrix whose rows are the positions of `rows` and
// whose columns those of `cols`, first dimension slowest.
CellKeys cell_keys(const std::vector<int>& rows, const std::vector<int>& cols, const OperandD& op,
                   const StagedKeys& s, const std::vector<int64_t>& extent);

// Scatters a column's rows into `mat` by their cells (below 2^32) and marks
// each in `held`: `bits` bits a cell, 1 for presence, or 2 for a code (1 a NULL
// value, 2 a value). A cell marked twice sets `dup` in *flags, a value that
// isn't finite `nonfinite`; NULL values (valid 0) aren't written.
void scatter_cells(Context& ctx, const CellKeys& k, int64_t rows, const double* vals, const uint8_t* valid,
                   double* mat, uint32_t* held, int bits, unsigned* flags, unsigned dup, unsigned nonfinite);

}  // namespace ef
