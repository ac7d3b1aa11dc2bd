// Attention of a few queries against many keys (a decoding step, a lookup):
// product scores, the softmax shifted by the row's maximum, a normalised
// average, in FP64 on the CUDA cores.
//
// Bound by HBM: k and v are read once and nothing of their size is written.
// The tensor-core form computes 128 query rows whatever their number, cuts k
// and v into digits first, and gives a batch's queries one block that walks
// the key tiles one after another: 16 groups of one query by 8,191 keys of
// d = 64 took it 956 us and its slicing 140 more (1300 a call). Here the keys
// are cut into chunks of kKeys, a block each, whatever the number of queries
// and groups, and a second kernel joins a row's chunks in order under their
// common maximum: 102 us a call, 42 in the kernels (20 us at the measured
// HBM rate). A chunk that none of a block's rows joins is neither read nor written
// (64 groups of 32 queries by 8,192 keys of d = 128 in a window of 100: 0.37 ms, 2.3
// with every chunk), and a row's chunks are joined over its interval.
//
// A block: eight lanes a key read its k row (128 contiguous bytes a load) and
// form its scores with the block's R rows of q in shared memory; a warp a row
// turns them into weights; eight warps take the keys in turn, a lane two (or
// four) value columns, and their sums meet in order in shared memory.
//
// The row guards take bounds of the values' magnitudes over the chunks' keys
// (their high words, an integer maximum and minimum a value): a row that
// passes with them passes with its exact ones. A row that doesn't, a score or a
// value that isn't finite, sets *retry and the caller takes another form.
#include <algorithm>
#include <cmath>

#include "attention.cuh"

namespace ef {
namespace {

constexpr int kRowsThreads = 256;
constexpr int kKeys = 128;          // keys a block
constexpr int kMaxChunks = 4096;
constexpr int64_t kMaxRows = 32;    // queries a group
constexpr int64_t kMinKeys = 512;   // keys a group

struct RowsArgs {
  Mask mask;
  const double* q;
  const double* k;
  const double* v;
  int64_t lnx, lnj;
  int ne, ny, n_chunks, scale_kind;
  double scale_c;
  // Per row and chunk: its maximum, sum of weights and smallest score; its weighted
  // sums; per block of rows and chunk the values' high words. Chunks that no row of
  // the block joins stay unwritten.
  double* stats;   // [row][3][chunk]
  double* sums;    // [row][chunk][ny]
  unsigned* high;  // [batch][block of rows][2][chunk]: the largest and the smallest nonzero value's
  int row_blocks, block_shift;  // blocks of 2^block_shift rows
  double* out;
  double* lse;
  unsigned* retry;
};

// A row's doubles 2·i and 2·i + 1 (0 past its n).
__device__ __forceinline__ double2 load_pair(const double* row, int i, int n, bool pairs) {
  if (pairs) return 2 * i < n ? *reinterpret_cast<const double2*>(row + 2 * i) : make_double2(0.0, 0.0);
  return make_double2(2 * i < n ? row[2 * i] : 0.0, 2 * i + 1 < n ? row[2 * i + 1] : 0.0);
}

// R: rows of q a block; DI: d in units of 16; YI: value columns in units of 64.
template <int R, int DI, int YI>
__global__ void __launch_bounds__(kRowsThreads) attn_rows(const RowsArgs a) {
  __shared__ __align__(16) double sq[R][DI * 16];
  __shared__ double ss[R][kKeys];
  __shared__ double red[kRowsThreads / 32][YI * 64];
  __shared__ int s_lo[R], s_hi[R];
  __shared__ unsigned s_top, s_low;
  const int t = threadIdx.x, warp = t >> 5, lane = t & 31;
  const int chunk = blockIdx.x;
  const int64_t w = blockIdx.y, row0 = (int64_t)blockIdx.z * R;
  const int64_t j0 = (int64_t)chunk * kKeys;
  const int width = (int)min((long long)kKeys, (long long)(a.lnj - j0));
  const double* kb = a.k + (w * a.lnj + j0) * a.ne;
  const double* vb = a.v + (w * a.lnj + j0) * a.ny;

  for (int i = t; i < R * DI * 16; i += kRowsThreads) {
    const int r = i / (DI * 16), e = i % (DI * 16);
    sq[r][e] = row0 + r < a.lnx && e < a.ne ? a.q[(w * a.lnx + row0 + r) * a.ne + e] : 0.0;
  }
  bool joins = false;
  if (t < R) {
    int lo = 0, hi = 0;
    if (row0 + t < a.lnx) {
      int64_t l, h;
      allowed(a.mask, w * a.lnx + row0 + t, l, h);
      l -= w * a.lnj + j0;
      h -= w * a.lnj + j0;
      lo = (int)(l < 0 ? 0 : l > width ? width : l);
      hi = (int)(h < 0 ? 0 : h > width ? width : h);
    }
    s_lo[t] = lo;
    s_hi[t] = hi;
    joins = lo < hi;
  }
  if (t == 0) {
    s_top = 0;
    s_low = 0xffffffffu;
  }
  if (!__syncthreads_or(joins)) return;  // no row joins a key here: nothing is read or written

  // Scores.
  const bool k_pairs = (a.ne & 1) == 0 && ((uintptr_t)a.k & 15) == 0;
  const int l8 = t & 7;
#pragma unroll
  for (int it = 0; it < kKeys / (kRowsThreads / 8); it++) {
    const int j = it * (kRowsThreads / 8) + (t >> 3);
    const double* row = kb + (int64_t)(j < width ? j : 0) * a.ne;
    double2 kv[DI];
#pragma unroll
    for (int i = 0; i < DI; i++) kv[i] = load_pair(row, l8 + 8 * i, a.ne, k_pairs);
#pragma unroll
    for (int r = 0; r < R; r++) {
      double s = 0.0;
#pragma unroll
      for (int i = 0; i < DI; i++) {
        const double2 qv = *reinterpret_cast<const double2*>(&sq[r][2 * (l8 + 8 * i)]);
        s = fma(qv.x, kv[i].x, s);
        s = fma(qv.y, kv[i].y, s);
      }
#pragma unroll
      for (int o = 4; o; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
      if (l8 == 0) ss[r][j] = a.scale_kind == 1 ? s * a.scale_c : a.scale_kind == 2 ? __ddiv_rn(s, a.scale_c) : s;
    }
  }
  __syncthreads();

  // Weights under the chunk's maximum, a warp a row.
  bool retry = false;
  for (int r = warp; r < R; r += kRowsThreads / 32) {
    const int lo = s_lo[r], hi = s_hi[r];
    double s[kKeys / 32], m = -INFINITY, light = INFINITY, z = 0.0;
#pragma unroll
    for (int i = 0; i < kKeys / 32; i++) {
      const int j = lane + 32 * i;
      s[i] = ss[r][j];
      if (j >= lo && j < hi) {
        if (!isfinite(s[i])) retry = true;
        m = fmax(m, s[i]);
        light = fmin(light, s[i]);
      }
    }
#pragma unroll
    for (int o = 16; o; o >>= 1) {
      m = fmax(m, __shfl_xor_sync(0xffffffffu, m, o));
      light = fmin(light, __shfl_xor_sync(0xffffffffu, light, o));
    }
#pragma unroll
    for (int i = 0; i < kKeys / 32; i++) {
      const int j = lane + 32 * i;
      const double x = j >= lo && j < hi ? exp(s[i] - m) : 0.0;
      ss[r][j] = x;
      z += x;
    }
#pragma unroll
    for (int o = 16; o; o >>= 1) z += __shfl_xor_sync(0xffffffffu, z, o);
    if (lane == 0 && row0 + r < a.lnx) {
      double* st = a.stats + (w * a.lnx + row0 + r) * 3 * a.n_chunks + chunk;
      st[0] = m;
      st[a.n_chunks] = z;
      st[2 * a.n_chunks] = light;
    }
  }
  __syncthreads();

  // Weighted values.
  const bool v_pairs = (a.ny & 1) == 0 && ((uintptr_t)a.v & 15) == 0;
  double acc[R][2 * YI];
#pragma unroll
  for (int r = 0; r < R; r++)
#pragma unroll
    for (int u = 0; u < 2 * YI; u++) acc[r][u] = 0.0;
  unsigned top = 0, low = 0xffffffffu;
  auto bounds = [&](double x) {
    const unsigned h = (unsigned)__double2hiint(x) & 0x7fffffffu;
    top = max(top, h);
    low = min(low, x != 0.0 ? h : 0xffffffffu);
  };
#pragma unroll 4
  for (int i = 0; i < kKeys / 8; i++) {
    const int j = warp + 8 * i;
    if (j >= width) break;
    double2 x[YI];
#pragma unroll
    for (int u = 0; u < YI; u++) {
      x[u] = load_pair(vb + (int64_t)j * a.ny, lane + 32 * u, a.ny, v_pairs);
      bounds(x[u].x);
      bounds(x[u].y);
    }
#pragma unroll
    for (int r = 0; r < R; r++) {
      const double wt = ss[r][j];
#pragma unroll
      for (int u = 0; u < YI; u++) {
        acc[r][2 * u] = fma(wt, x[u].x, acc[r][2 * u]);
        acc[r][2 * u + 1] = fma(wt, x[u].y, acc[r][2 * u + 1]);
      }
    }
  }
  top = __reduce_max_sync(0xffffffffu, top);
  low = __reduce_min_sync(0xffffffffu, low);
  if (lane == 0) {
    atomicMax(&s_top, top);
    atomicMin(&s_low, low);
  }
#pragma unroll
  for (int r = 0; r < R; r++) {
    if (row0 + r >= a.lnx) break;
    __syncthreads();
#pragma unroll
    for (int u = 0; u < YI; u++) {
      red[warp][2 * (lane + 32 * u)] = acc[r][2 * u];
      red[warp][2 * (lane + 32 * u) + 1] = acc[r][2 * u + 1];
    }
    __syncthreads();
    if (t < a.ny) {
      double s = red[0][t];
#pragma unroll
      for (int i = 1; i < kRowsThreads / 32; i++) s += red[i][t];
      a.sums[((w * a.lnx + row0 + r) * a.n_chunks + chunk) * a.ny + t] = s;
    }
  }
  __syncthreads();
  if (t == 0) {
    if (s_top >= 0x7ff00000u) retry = true;
    unsigned* high = a.high + (w * a.row_blocks + blockIdx.z) * 2 * a.n_chunks + chunk;
    high[0] = s_top;
    high[a.n_chunks] = s_low;
  }
  if (retry) atomicOr(a.retry, 1u);
}

// A block a row: its chunks' maxima, sums and weighted sums under one maximum,
// the row's guards (Bounds::hold, fused.rs:1058-1086, the heaviest weight
// being exp(high - m) = 1) and its output.
__global__ void __launch_bounds__(kRowsThreads) join_chunks(const RowsArgs a) {
  __shared__ double f[kMaxChunks];
  __shared__ double red[3][kRowsThreads / 32];
  __shared__ unsigned red_u[2][kRowsThreads / 32];
  __shared__ double part[4][128];
  const int t = threadIdx.x, warp = t >> 5, lane = t & 31;
  const int64_t x = blockIdx.x, w = x / a.lnx;
  int64_t lo, hi;
  allowed(a.mask, x, lo, hi);
  if (lo >= hi) return;
  const int c0 = (int)((lo - w * a.lnj) / kKeys), c1 = (int)((hi - 1 - w * a.lnj) / kKeys) + 1;  // the row's chunks
  const double* st = a.stats + x * 3 * a.n_chunks;
  const unsigned* high = a.high + (w * a.row_blocks + ((x - w * a.lnx) >> a.block_shift)) * 2 * a.n_chunks;
  double m = -INFINITY, light = INFINITY;
  unsigned top = 0, low = 0xffffffffu;
  auto joined = [&](int c) { return c >= c0 && c < c1; };
  for (int c = t; c < a.n_chunks; c += kRowsThreads) {
    if (!joined(c)) continue;
    m = fmax(m, st[c]);
    light = fmin(light, st[2 * a.n_chunks + c]);
    top = max(top, high[c]);
    low = min(low, high[a.n_chunks + c]);
  }
#pragma unroll
  for (int o = 16; o; o >>= 1) {
    m = fmax(m, __shfl_xor_sync(0xffffffffu, m, o));
    light = fmin(light, __shfl_xor_sync(0xffffffffu, light, o));
  }
  top = __reduce_max_sync(0xffffffffu, top);
  low = __reduce_min_sync(0xffffffffu, low);
  if (lane == 0) {
    red[0][warp] = m;
    red[1][warp] = light;
    red_u[0][warp] = top;
    red_u[1][warp] = low;
  }
  __syncthreads();
  for (int i = 0; i < kRowsThreads / 32; i++) {
    m = fmax(m, red[0][i]);
    light = fmin(light, red[1][i]);
    top = max(top, red_u[0][i]);
    low = min(low, red_u[1][i]);
  }
  double z = 0.0;
  for (int c = t; c < a.n_chunks; c += kRowsThreads) {
    if (!joined(c)) continue;
    f[c] = exp(st[c] - m);
    z += f[c] * st[a.n_chunks + c];
  }
#pragma unroll
  for (int o = 16; o; o >>= 1) z += __shfl_xor_sync(0xffffffffu, z, o);
  if (lane == 0) red[2][warp] = z;
  __syncthreads();
  z = 0.0;
  for (int i = 0; i < kRowsThreads / 32; i++) z += red[2][i];
  // Four groups of 64 threads take the chunks in turn.
  const int g = t >> 6;
  const double* sums = a.sums + x * a.n_chunks * a.ny;
  for (int y = t & 63; y < a.ny; y += 64) {
    double s = 0.0;
    for (int b = c0 & ~31; b < c1; b += 32) {
      double v[8];  // (chunks the row doesn't join may be unwritten)
#pragma unroll
      for (int u = 0; u < 8; u++) {
        const int c = b + 4 * u + g;
        v[u] = c < a.n_chunks ? sums[(int64_t)c * a.ny + y] : 0.0;
      }
#pragma unroll
      for (int u = 0; u < 8; u++) {
        const int c = b + 4 * u + g;
        s = joined(c) ? fma(f[c], v[u], s) : s;
      }
    }
    part[g][y] = s;
  }
  __syncthreads();
  // The values' largest magnitude from above, the smallest from below.
  const double rl = __hiloint2double((int)top, -1), rs = low == 0xffffffffu ? INFINITY : __hiloint2double((int)low, 0);
  const double normal = 2.0 * 2.2250738585072014e-308, t2 = 2.0 * (double)(hi - lo);
  const double inverse = 1.0 / fabs(z), lightest = exp(light - m);
  bool over = !isfinite(z) || !isfinite(rl * t2) || !isfinite(inverse) || !isfinite(inverse * rl * t2);
  const double lost = (t2 * 4.9406564584124654e-324) * ((inverse + rl) + 1.0);
  bool no_underflow = rs == INFINITY;
  if (!no_underflow) {
    const double quotient = lightest / fabs(z);
    no_underflow = lightest * rs >= normal && quotient >= normal && quotient * rs >= normal;
  }
  const double rounding = 2.220446049250313e-16 / 4.0;
  if (t < a.ny) {
    const double s = (part[0][t] + part[1][t]) + (part[2][t] + part[3][t]);
    const double o = __ddiv_rn(s, z);
    if (!isfinite(s) || !isfinite(o) || (!no_underflow && !(lost <= rounding * fabs(o)))) over = true;
    a.out[x * a.ny + t] = o;
  }
  if (t == 0 && a.lse) a.lse[x] = m + log(z);
  if (over) atomicOr(a.retry, 1u);
}

template <int R>
auto rows_kernel(int64_t d, int64_t dv) {
  return d <= 64 ? (dv <= 64 ? attn_rows<R, 4, 1> : attn_rows<R, 4, 2>)
                 : (dv <= 64 ? attn_rows<R, 8, 1> : attn_rows<R, 8, 2>);
}

}  // namespace

// At most 32 queries a group and 512 keys or more: the tensor-core form computes
// 128 rows in any case and its one block a group takes 7.5 us a tile of 64 keys.
// Ragged groups keep the form their full ones have been given (the same bits
// alone and together).
//
// The chunks' work grows with the rows, in blocks of 16, and the joined keys; the
// FP64 tensor pipe computes 64 rows for any number and fills the device with some
// 300 groups. So chunks always up to 8 queries (2,000 groups by 512 keys, d = 16:
// 0.54 ms against 1.05), up to 16 but for many groups of narrow rows (2,000 by 512,
// d = 16: 1.26 against 1.14; d = 32: 1.20 against 1.23); and beyond, two blocks of
// rows, while the groups leave SMs idle or (d = 64) don't share them evenly (100 of
// 32 by 4,096, d = 64: 0.87 against 1.10; 148: 1.20 against 1.15; 160: 1.28 against
// 1.39; 200: 1.56 against 1.45), or up to twice as many by few keys or in wide rows
// (300 of 32 by 512, d = 64: 0.47 against 0.49, d = 128: 0.87 against 0.96; by 4,096,
// d = 16: 2.28 against 1.97; 148 by 4,096, d = 128: 2.65 against 1.96 in the split
// form). 2,000 groups of 32 by 512, d = 64: 2.3 ms in chunks, 1.4 on the tensor pipe,
// 1.8 in the split form; d = 128: 4.9, 4.4 and 3.7 (hence left to the caller's
// precision).
FewQueries few_queries(const Context& ctx, const AttentionProblem& p) {
  const int64_t chunks = (p.lnj + kKeys - 1) / kKeys, W = p.batches, sms = ctx.sm_count;
  if (p.lnx < 1 || p.lnx > kMaxRows || p.lnj < kMinKeys || chunks > kMaxChunks || p.ne < 1 || p.ne > 128 || p.ny < 1 ||
      p.ny > 128 || W < 1 || W > 65535 || p.mask.xlen || p.mask.jlen)
    return FEW_NONE;
  const int64_t wide = std::max(p.ne, p.ny);
  bool rows;
  if (p.lnx <= 16) {
    rows = p.lnx <= 8 || wide > 16 || W <= 8 * sms;
  } else if (W * 10 <= sms * 7 || (wide > 32 && wide <= 64 && W * 8 <= sms * 9)) {
    rows = true;
  } else {
    int64_t first = p.lnj, last = 0;  // the keys joined
    for (int64_t x = 0; x < p.lnx; x++) {
      int64_t lo, hi;
      allowed(p.mask, x, lo, hi);
      if (lo >= hi) continue;
      first = std::min(first, lo);
      last = std::max(last, hi);
    }
    const int64_t keys = std::max<int64_t>(last - first, 0);
    rows = W * 4 <= sms * 9 && (keys <= 1024 ? wide > 32 || W * keys <= 160 << 10 : wide > 64 && W > sms);
  }
  return rows ? FEW_CHUNKS : wide > 64 ? FEW_NONE : FEW_MMA;
}

AttentionOutcome attention_rows(Context& ctx, const AttentionProblem& p, cudaStream_t s) {
  const int64_t chunks = (p.lnj + kKeys - 1) / kKeys;
  const int64_t nx = p.batches * p.lnx;
  DeviceBuffer<double> stats((size_t)(nx * 3 * chunks), s), sums((size_t)(nx * chunks * p.ny), s);
  int shift = 0;
  while (shift < 4 && (1 << shift) < p.lnx) shift++;
  const int rows = 1 << shift;
  const int64_t row_blocks = (p.lnx + rows - 1) / rows;
  DeviceBuffer<unsigned> high((size_t)(p.batches * row_blocks * 2 * chunks), s), retry(1, s);
  retry.zero();
  RowsArgs a{};
  a.mask = p.mask;
  a.q = p.q;
  a.k = p.k;
  a.v = p.v;
  a.lnx = p.lnx;
  a.lnj = p.lnj;
  a.ne = (int)p.ne;
  a.ny = (int)p.ny;
  a.n_chunks = (int)chunks;
  a.scale_kind = p.scale_kind;
  a.scale_c = p.scale_c;
  a.stats = stats.get();
  a.sums = sums.get();
  a.high = high.get();
  a.out = p.out;
  a.lse = p.lse;
  a.retry = retry.get();
  a.row_blocks = (int)row_blocks;
  a.block_shift = shift;
  auto kernel = rows == 1   ? rows_kernel<1>(p.ne, p.ny)
                : rows == 2 ? rows_kernel<2>(p.ne, p.ny)
                : rows == 4 ? rows_kernel<4>(p.ne, p.ny)
                : rows == 8 ? rows_kernel<8>(p.ne, p.ny)
                            : rows_kernel<16>(p.ne, p.ny);
  kernel<<<dim3((unsigned)chunks, (unsigned)p.batches, (unsigned)row_blocks), kRowsThreads, 0, s>>>(a);
  join_chunks<<<(unsigned)nx, kRowsThreads, 0, s>>>(a);
  EF_LAUNCH_CHECK();
  ctx.kernels += 2;
  unsigned again = 0;
  ReadBack back(ctx, s);
  back.add(&again, retry.get());
  back.wait();
  ctx.phase("attention: few queries");
  return again ? ATTENTION_INELIGIBLE : ATTENTION_DONE;
}

}  // namespace ef
