// The operands of an attention pass, read once: prepare_rows, prepare_columns,
// row_bounds.
//
// Bound by issue slots at large sizes (72% of them busy, 108 instructions a value;
// DRAM 34%), by launches at small ones. With a kernel an operand and purpose (row digits,
// column maxima, value statistics or dots, exponent ranges) there were 12
// launches and 3 waits before the forward's tiles, 22 and 2 before the
// backward's. Here all operands share a launch and one reading, and the
// exponents' ranges stay on the device for the tile kernels to judge (Ready).
// Forward and backward of 6 batches of 100 rows of 32: 730 to 450 us a step.
// 64 batches of 128 to 8192 rows of 128, forward: 2.81 to 2.56 ms
// (prepare_rows 237 us; chunks past a batch's length are told apart first,
// 667 us without). 64 batches of 4096 x 64: prepare_rows 222 us for 0.6 GB
// (forward), 362 for 1.0 GB (backward), at three blocks an SM; 259 and 432
// at two, 237 and 377 at four.
#include <algorithm>

#include "levels.cuh"
#include "prepare.cuh"
#include "ptx.cuh"

namespace ef {
namespace {

constexpr int S = 6;
constexpr int kRowsChunk = 64;
constexpr double kLargestDouble = 1.7976931348623157e308;

struct RowSets {
  RowSet set[kPrepareSets];
};
struct ColumnSets {
  ColumnSet set[kPrepareSets];
  int n;
};

// LANES lanes a row (16: up to 64 columns, 32: up to 128, four a lane); wider
// operands (without row digits) take their columns LANES·4 at a time, their
// maxima straight to memory. A block takes 64 rows of one batch, two a group of
// lanes at a time.
template <int LANES>
__global__ void __launch_bounds__(256, 3) prepare_rows_kernel(const __grid_constant__ RowSets sets, int64_t batches, int* __restrict__ status) {
  constexpr int GROUPS = 256 / LANES, STEP = 2 * GROUPS, COLS = LANES * 4;
  __shared__ double s_col[GROUPS][COLS];
  __shared__ double s_lg[GROUPS], s_sm[GROUPS];
  const RowSet& s = sets.set[blockIdx.y];
  const int l = threadIdx.x % LANES, grp = threadIdx.x / LANES;
  const int64_t chunks = s.rows_pad / kRowsChunk;
  const bool narrow = s.cols <= COLS;
  int top = 0, low = 0;  // biased
  bool bad = false;
  for (int64_t chunk = blockIdx.x; chunk < batches * chunks; chunk += gridDim.x) {
    const int64_t w = chunk / chunks, r0 = (chunk - w * chunks) * kRowsChunk;
    const int64_t live_rows = s.lens ? min(s.rows, s.lens[w]) : s.rows;
    double cm[4] = {0.0, 0.0, 0.0, 0.0};
    double block_lg = 0.0, block_sm = INFINITY;
    if (r0 >= live_rows && !s.other && !s.value && (!s.digits || s.skip_padding)) {
      // A chunk past its batch's length: what rows of zeros give.
      const int64_t r = r0 + threadIdx.x;
      if (threadIdx.x < kRowsChunk) {
        if (s.digits) {
          s.e[w * s.rows_pad + r] = 0;
          top = max(top, kExponentBias);
          low = max(low, kExponentBias);
        }
        if (s.largest && r < s.rows) {
          s.flag[w * s.rows + r] = 1;
          s.largest[w * s.rows + r] = 0.0;
          s.smallest[w * s.rows + r] = INFINITY;
        }
      }
      if (s.block_largest && threadIdx.x == 0) {
        s.block_largest[chunk] = 0.0;
        s.block_smallest[chunk] = INFINITY;
      }
      continue;
    }
#pragma unroll 1
    for (int i = grp; i < kRowsChunk; i += STEP) {
      double lg[2] = {0.0, 0.0}, sm[2] = {INFINITY, INFINITY}, dot[2] = {0.0, 0.0};
      unsigned odd[2] = {0, 0};  // bit 0: a value not finite, 1: an infinity
      for (int64_t c0 = 4 * l; c0 < (narrow ? COLS : s.cols); c0 += COLS) {
        double v[2][4];
#pragma unroll
        for (int u = 0; u < 2; u++) {
          const int64_t r = r0 + i + u * GROUPS;
          const double* row = s.x + (w * s.rows + r) * s.cols;
          const bool live = r < live_rows;
          if (live && c0 + 3 < s.cols && (((uintptr_t)(row + c0)) & 15) == 0) {
            const double2 a = *(const double2*)(row + c0), b = *(const double2*)(row + c0 + 2);
            v[u][0] = a.x; v[u][1] = a.y; v[u][2] = b.x; v[u][3] = b.y;
          } else {
#pragma unroll
            for (int j = 0; j < 4; j++) v[u][j] = live && c0 + j < s.cols ? row[c0 + j] : 0.0;
          }
        }
        if (s.other)
#pragma unroll
          for (int u = 0; u < 2; u++) {
            const int64_t r = r0 + i + u * GROUPS, at = (w * s.rows + r) * s.cols;
            // (Rows past their length too: the caller's D has every row.)
            if (r < s.rows)
#pragma unroll
              for (int j = 0; j < 4; j++)
                if (c0 + j < s.cols)
                  dot[u] = fma(r < live_rows ? v[u][j] : s.x[at + c0 + j], s.other[at + c0 + j], dot[u]);
          }
#pragma unroll
        for (int u = 0; u < 2; u++) {
          const int64_t r = r0 + i + u * GROUPS;
          double m = 0.0;
#pragma unroll
          for (int j = 0; j < 4; j++) {
            const double a = fabs(v[u][j]);
            if (!(a <= kLargestDouble)) {
              odd[u] |= 1u | (isinf(a) ? 2u : 0u);
              v[u][j] = 0.0;
            } else {
              m = fmax(m, a);
              cm[j] = fmax(cm[j], a);
              if (a != 0.0) sm[u] = fmin(sm[u], a);
            }
          }
          lg[u] = fmax(lg[u], m);
          if (s.digits) {
#pragma unroll
            for (int o = LANES / 2; o; o >>= 1) m = fmax(m, __shfl_xor_sync(0xffffffffu, m, o));
            const int ex = slice_exponent(m);
            if (l == 0) s.e[w * s.rows_pad + r] = ex;
            top = max(top, kExponentBias + ex);
            low = max(low, kExponentBias - ex);
            // x · 2^(8S - ex) in two exact factors (8S - ex may leave the normal range).
            const int shift = 8 * S - ex;
            const double f1 = ptx::pow2(shift >> 1), f2 = ptx::pow2(shift - (shift >> 1));
            double xs[4];
#pragma unroll
            for (int j = 0; j < 4; j++) xs[j] = v[u][j] * f1 * f2;
            uint32_t planes[S];
            digit_planes4<S>(xs, planes);
            if (4 * l < s.k_pad && (r < live_rows || !s.skip_padding))
#pragma unroll
              for (int d = 0; d < S; d++)
                *(uint32_t*)(s.digits + ((w * S + d) * s.rows_pad + r) * s.k_pad + 4 * l) = planes[d];
          }
        }
        if (s.colmax && !narrow)
#pragma unroll
          for (int j = 0; j < 4; j++) {
            if (cm[j] > 0.0 && c0 + j < s.cols)
              atomicMax(&s.colmax[w * s.cols + c0 + j], (unsigned long long)__double_as_longlong(cm[j]));
            cm[j] = 0.0;
          }
      }
#pragma unroll
      for (int u = 0; u < 2; u++) {
        const int64_t r = r0 + i + u * GROUPS;
        bad |= odd[u] != 0;
        if (s.largest || s.block_largest) {
#pragma unroll
          for (int o = LANES / 2; o; o >>= 1) {
            lg[u] = fmax(lg[u], __shfl_xor_sync(0xffffffffu, lg[u], o));
            sm[u] = fmin(sm[u], __shfl_xor_sync(0xffffffffu, sm[u], o));
            odd[u] |= __shfl_xor_sync(0xffffffffu, odd[u], o);
          }
          if (s.largest && l == 0 && r < s.rows) {
            s.flag[w * s.rows + r] = (uint8_t)((odd[u] & 1u ? 0u : 1u) | (odd[u] & 2u));
            s.largest[w * s.rows + r] = lg[u];
            s.smallest[w * s.rows + r] = sm[u];
          }
          block_lg = fmax(block_lg, lg[u]);
          block_sm = fmin(block_sm, sm[u]);
        }
        if (s.other) {
#pragma unroll
          for (int o = LANES / 2; o; o >>= 1) dot[u] += __shfl_xor_sync(0xffffffffu, dot[u], o);
          if (l == 0) {
            if (r < s.rows) s.dots[w * s.rows + r] = dot[u];
            s.dots_pad[w * s.rows_pad + r] = r < s.rows ? dot[u] : 0.0;
          }
        }
        if (s.value && l == 0) s.value_pad[w * s.rows_pad + r] = r < s.rows ? s.value[w * s.rows + r] : 0.0;
      }
    }
    if ((s.colmax && narrow) || s.block_largest) {
      __syncthreads();
#pragma unroll
      for (int j = 0; j < 4; j++) s_col[grp][4 * l + j] = cm[j];
      if (l == 0) {
        s_lg[grp] = block_lg;
        s_sm[grp] = block_sm;
      }
      __syncthreads();
      if (s.colmax && narrow && threadIdx.x < s.cols) {
        double m = 0.0;
#pragma unroll
        for (int g = 0; g < GROUPS; g++) m = fmax(m, s_col[g][threadIdx.x]);
        if (m > 0.0) atomicMax(&s.colmax[w * s.cols + threadIdx.x], (unsigned long long)__double_as_longlong(m));
      }
      if (s.block_largest && threadIdx.x == 0) {
        for (int g = 1; g < GROUPS; g++) {
          block_lg = fmax(block_lg, s_lg[g]);
          block_sm = fmin(block_sm, s_sm[g]);
        }
        s.block_largest[chunk] = block_lg;
        s.block_smallest[chunk] = block_sm;
      }
    }
  }
  if (s.range) {
    top = __reduce_max_sync(0xffffffffu, top);
    low = __reduce_max_sync(0xffffffffu, low);
    if ((threadIdx.x & 31) == 0 && top) {
      atomicMax(&s.range[0], top);
      atomicMax(&s.range[1], low);
    }
  }
  if (__any_sync(0xffffffffu, bad) && (threadIdx.x & 31) == 0) atomicOr(status, s.bad);
}

// A 64 x 64 tile staged in shared memory, read along the columns and cut along
// the rows; each thread cuts 16 rows of one column.
__global__ void __launch_bounds__(256) prepare_columns_kernel(const __grid_constant__ ColumnSets sets) {
  __shared__ double tile[kColumnTile];
  const ColumnSet& s = sets.set[blockIdx.y % sets.n];
  const int64_t w = blockIdx.z, k0 = (int64_t)blockIdx.x * 64, n0 = (int64_t)(blockIdx.y / sets.n) * 64;
  if (k0 >= s.rows_pad || n0 >= s.cols_pad) return;
  const double* X = s.x + w * s.rows * s.cols;
  const int64_t live = s.lens ? min(s.rows, s.lens[w]) : s.rows;
  if (s.skip_padding && k0 >= live && k0 > 0) return;  // (the first block gives the exponents)
#pragma unroll
  for (int i0 = 0; i0 < 64 * 64; i0 += 256) {
    const int i = i0 + threadIdx.x;
    const int kr = i / 64, nc = i % 64;
    const int64_t gk = k0 + kr, gn = n0 + nc;
    double v = (gk < live && gn < s.cols) ? X[gk * s.cols + gn] : 0.0;
    if (!(fabs(v) <= kLargestDouble)) v = 0.0;
    tile[column_tile_at(kr, nc)] = v;
  }
  __syncthreads();
  const int nl = threadIdx.x / 4, kc = threadIdx.x % 4;
  const int64_t col = n0 + nl;
  const int ex = col < s.cols ? slice_exponent(__longlong_as_double((long long)s.colmax[w * s.cols + col])) : 0;
  if (blockIdx.x == 0 && kc == 0) s.e[w * s.cols_pad + col] = ex;
  const int shift = 8 * S - ex;
  const double f1 = ptx::pow2(shift >> 1), f2 = ptx::pow2(shift - (shift >> 1));
  uint32_t word[S][4];
#pragma unroll
  for (int q = 0; q < 4; q++) {
    double xs[4];
#pragma unroll
    for (int i = 0; i < 4; i++) xs[i] = tile[column_tile_at(kc * 16 + q * 4 + i, nl)] * f1 * f2;
    uint32_t planes[S];
    digit_planes4<S>(xs, planes);
#pragma unroll
    for (int d = 0; d < S; d++) word[d][q] = planes[d];
  }
#pragma unroll
  for (int d = 0; d < S; d++)
    *(uint4*)(s.digits + ((w * S + d) * s.cols_pad + col) * s.rows_pad + k0 + kc * 16) =
        make_uint4(word[d][0], word[d][1], word[d][2], word[d][3]);
}

// A warp a block of 64 positions.
__global__ void __launch_bounds__(256) block_extrema_kernel(int64_t batches, int64_t lnj, int64_t blocks,
                                                            const double* __restrict__ largest,
                                                            const double* __restrict__ smallest,
                                                            double* __restrict__ block_largest,
                                                            double* __restrict__ block_smallest) {
  const int lane = threadIdx.x & 31;
  for (int64_t x = ((int64_t)blockIdx.x * 256 + threadIdx.x) >> 5; x < batches * blocks; x += (int64_t)gridDim.x * 8) {
    const int64_t w = x / blocks, b = x - w * blocks;
    double mx = 0.0, mn = INFINITY;
    for (int64_t j = b * 64 + lane; j < min(lnj, b * 64 + 64); j += 32) {
      mx = fmax(mx, largest[w * lnj + j]);
      mn = fmin(mn, smallest[w * lnj + j]);
    }
#pragma unroll
    for (int o = 16; o; o >>= 1) {
      mx = fmax(mx, __shfl_xor_sync(0xffffffffu, mx, o));
      mn = fmin(mn, __shfl_xor_sync(0xffffffffu, mn, o));
    }
    if (lane == 0) {
      block_largest[x] = mx;
      block_smallest[x] = mn;
    }
  }
}

// A warp `rows` (up to 32) rows: each lane finds one's keys (128-bit arithmetic), and the warp
// takes the rows that join any in turn: the positions before its first whole
// block and after its last, and the blocks between.
__global__ void __launch_bounds__(256) row_bounds_kernel(int64_t nx, int rows, Mask m, int64_t blocks,
                                                         const double* __restrict__ largest,
                                                         const double* __restrict__ smallest,
                                                         const double* __restrict__ block_largest,
                                                         const double* __restrict__ block_smallest,
                                                         double* __restrict__ rl, double* __restrict__ rs) {
  const int lane = threadIdx.x & 31;
  for (int64_t x0 = (((int64_t)blockIdx.x * 256 + threadIdx.x) >> 5) * rows; x0 < nx;
       x0 += (int64_t)gridDim.x * 8 * rows) {
    const int64_t x = x0 + lane;
    int64_t lo = 0, hi = 0, w = 0;
    if (lane < rows && x < nx) {
      allowed(m, x, lo, hi);
      w = x / m.lnx;
      lo -= w * m.lnj;
      hi -= w * m.lnj;
    }
    double row_mx = 0.0, row_mn = INFINITY;
    for (unsigned left = __ballot_sync(0xffffffffu, lo < hi); left; left &= left - 1) {
      const int r = __ffs(left) - 1;
      const int64_t a = __shfl_sync(0xffffffffu, lo, r), b = __shfl_sync(0xffffffffu, hi, r);
      const int64_t wr = __shfl_sync(0xffffffffu, w, r), base = wr * m.lnj;
      double mx = 0.0, mn = INFINITY;
      auto positions = [&](int64_t from, int64_t to) {
        for (int64_t j = from + lane; j < to; j += 32) {
          mx = fmax(mx, largest[base + j]);
          mn = fmin(mn, smallest[base + j]);
        }
      };
      // Whole blocks [b0, b1); the last block of the batch counts as whole
      // when the row joins its every position.
      const int64_t b0 = (a + 63) >> 6, b1 = b == m.lnj ? (b + 63) >> 6 : b >> 6;
      if (b0 < b1) {
        positions(a, b0 << 6);
        for (int64_t i = b0 + lane; i < b1; i += 32) {
          mx = fmax(mx, block_largest[wr * blocks + i]);
          mn = fmin(mn, block_smallest[wr * blocks + i]);
        }
        positions(b1 << 6, b);
      } else {
        positions(a, b);
      }
#pragma unroll
      for (int o = 16; o; o >>= 1) {
        mx = fmax(mx, __shfl_xor_sync(0xffffffffu, mx, o));
        mn = fmin(mn, __shfl_xor_sync(0xffffffffu, mn, o));
      }
      if (lane == r) {
        row_mx = mx;
        row_mn = mn;
      }
    }
    if (lane < rows && x < nx) {
      rl[x] = row_mx;
      rs[x] = row_mn;
    }
  }
}

}  // namespace

void prepare_rows(Context& ctx, const RowSet* sets, int n, int64_t batches, int* status, cudaStream_t s) {
  RowSets a;
  int64_t chunks = 0;
  bool wide = false;
  for (int i = 0; i < n; i++) {
    a.set[i] = sets[i];
    chunks = std::max(chunks, sets[i].rows_pad / kRowsChunk);
    wide = wide || sets[i].cols > 64;
  }
  const dim3 grid((unsigned)std::min<int64_t>(std::max<int64_t>(batches * chunks, 1), (int64_t)ctx.sm_count * 8),
                  (unsigned)n);
  if (wide) prepare_rows_kernel<32><<<grid, 256, 0, s>>>(a, batches, status);
  else prepare_rows_kernel<16><<<grid, 256, 0, s>>>(a, batches, status);
  ctx.kernels++;
  EF_LAUNCH_CHECK();
}

void prepare_columns(Context& ctx, const ColumnSet* sets, int n, int64_t batches, cudaStream_t s) {
  ColumnSets a;
  a.n = n;
  int64_t k = 0, c = 0;
  for (int i = 0; i < n; i++) {
    a.set[i] = sets[i];
    k = std::max(k, sets[i].rows_pad / 64);
    c = std::max(c, sets[i].cols_pad / 64);
  }
  prepare_columns_kernel<<<dim3((unsigned)k, (unsigned)(c * n), (unsigned)batches), 256, 0, s>>>(a);
  ctx.kernels++;
  EF_LAUNCH_CHECK();
}

void block_extrema(Context& ctx, int64_t batches, int64_t lnj, const double* largest, const double* smallest,
                   double* block_largest, double* block_smallest, cudaStream_t s) {
  const int64_t blocks = (lnj + 63) / 64;
  block_extrema_kernel<<<blocks_for((uint64_t)(batches * blocks), 8), 256, 0, s>>>(batches, lnj, blocks, largest,
                                                                                  smallest, block_largest,
                                                                                  block_smallest);
  ctx.kernels++;
  EF_LAUNCH_CHECK();
}

void row_bounds(Context& ctx, const Mask& m, int64_t nx, int64_t blocks, const double* largest, const double* smallest,
                const double* block_largest, const double* block_smallest, double* rl, double* rs, cudaStream_t s) {
  // A row a warp where that fills the device (3.5 us against 8.5 by eights at 4096
  // rows), up to eight (85 us against 230 one at a time at 524,288 rows, a
  // quarter of them live).
  const int rows = (int)std::clamp<int64_t>(nx / (ctx.sm_count * 32), 1, 8);
  row_bounds_kernel<<<blocks_for((uint64_t)(nx + rows - 1) / rows, 8, (unsigned)ctx.sm_count * 16), 256, 0, s>>>(
      nx, rows, m, blocks, largest, smallest, block_largest, block_smallest, rl, rs);
  ctx.kernels++;
  EF_LAUNCH_CHECK();
}

}  // namespace ef
