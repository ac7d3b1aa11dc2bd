// Combining the exact level sums of a split product in FP64, and cutting
// values into balanced base-256 digits.
#pragma once

#include "ptx.cuh"

namespace ef {

// The S levels of one TMEM column, combined: Σ_l L_l 2^{-8(l+2)}, in groups
// of three summed exactly in int64 (|L_l| < 2^31, so three of them shifted
// by 8 bits fit in 2^48) and added from the smallest group up.
template <int S, int N>
__device__ __forceinline__ double combine_levels(const int32_t (&L)[S][N], int i) {
  double v = 0.0;
#pragma unroll
  for (int g = (S - 1) / 3; g >= 0; g--) {
    long long part = 0;
    const int l0 = 3 * g, l1 = (3 * g + 3 < S ? 3 * g + 3 : S);
#pragma unroll
    for (int l = l0; l < l1; l++) part = part * 256 + (long long)L[l][i];
    v += (double)part * ptx::pow2(-8 * (l1 + 1));
  }
  return v;
}

// An integer |x| < 2^51 as a double, exactly, from x + kInt51: the bits of
// 1.5·2^52 + x.
constexpr long long kInt51 = 0x4338000000000000ll;
__device__ __forceinline__ double int51(long long biased) {
  return __longlong_as_double(biased) - 6755399441055744.0;
}
__device__ __forceinline__ long long mad_wide(int a, int b, long long c) {
  long long d;
  asm("mad.wide.s32 %0, %1, %2, %3;" : "=l"(d) : "r"(a), "r"(b), "l"(c));
  return d;
}

// The same for six levels small enough that two of them, one shifted by 8
// bits, fit in int32 (|L_l| < 2^23): the first four summed exactly in int64,
// the last two beside them, and one rounding. In units of 2^kLevelUnit, which
// callers fold into a power of two they apply anyway. Nine instructions (three
// of them FP64) against fifteen (six) for pairs converted one by one.
constexpr int kLevelUnit = -40;
template <int N>
__device__ __forceinline__ double combine_levels_small(const int32_t (&L)[6][N], int i) {
  const int a = L[0][i] * 256 + L[1][i], b = L[2][i] * 256 + L[3][i], c = L[4][i] * 256 + L[5][i];
  const double high = int51(mad_wide(a, 65536, mad_wide(b, 1, kInt51)));
  const double low = int51(mad_wide(c, 1, kInt51));
  return fma(low, 1.0 / 65536.0, high);
}

// The S digit planes of four values x·f (f a power of two, |x·f| < 2^(8S-2),
// S <= 6): x·f rounds to the nearest integer W (ties to even, as llrint) by
// adding 1.5·2^52 + 0x80…80 (even, and 48 bits), and W's balanced base-256
// digits d_s in [-128, 127] are the bytes of W + 0x80…80 with their top bits
// flipped (byte s of W + Σ 128·256^s is d_s + 128). planes[s] holds digit s
// (most significant first) of the four values, byte c for value c: the bytes
// the split product's digit planes hold.
template <int S>
__device__ __forceinline__ void digit_planes4(const double (&x)[4], double f, uint32_t (&planes)[S]) {
  static_assert(S <= 6, "six digits or fewer fit the 48-bit window");
  uint32_t lo[4], hi[4];
#pragma unroll
  for (int c = 0; c < 4; c++) {
    const long long u = __double_as_longlong(fma(x[c], f, 6755399441055744.0 + (double)0x808080808080ll));
    lo[c] = (uint32_t)u;
    hi[c] = (uint32_t)(u >> 32);
  }
#pragma unroll
  for (int s = 0; s < S; s++) {
    const int b = S - 1 - s;  // byte of W holding digit s
    const uint32_t* h = b < 4 ? lo : hi;
    const uint32_t sel = (uint32_t)((b & 3) | (((b & 3) + 4) << 4));
    const uint32_t t01 = __byte_perm(h[0], h[1], sel), t23 = __byte_perm(h[2], h[3], sel);
    planes[s] = __byte_perm(t01, t23, 0x5410) ^ 0x80808080u;
  }
}
template <int S>
__device__ __forceinline__ void digit_planes4(const double (&x)[4], uint32_t (&planes)[S]) {
  digit_planes4<S>(x, 1.0, planes);
}

// The exponent e with |x| < 2^(e-2) for the largest magnitude x of a row
// (0 for a row of zeros): digits of x / 2^e then start below 64.
__device__ __forceinline__ int slice_exponent(double largest) {
  int e = 0;
  if (largest > 0.0) {
    frexp(largest, &e);
    e += 2;
  }
  return e;
}

// A 64 x 64 tile written row by row and read by warps of 8 columns x 4 runs of 16
// rows: rows 65 apart, each run of 16 shifted by 8 more, so that a warp's 32
// doubles cover the banks twice (four to a bank without the shift).
constexpr int kColumnTile = 64 * 65 + 3 * 8;
__device__ __forceinline__ int column_tile_at(int row, int col) { return row * 65 + (row >> 4) * 8 + col; }

}  // namespace ef
