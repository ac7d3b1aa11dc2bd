// The backward pass of an attention-shaped pipeline: the gradients of the
// forward pass's average with respect to q, k and v, with the scores
// recomputed tile by tile from the saved log-sum-exp rather than stored.
//
// One kernel shape serves the three gradients. A CTA owns 128 rows of one
// batch and walks the column tiles of 64 its rows may pair with; per tile
//   s  = scale · (A1_r · B1_c)                  (product 1)
//   p  = exp(s - lse_x) on allowed pairs, else 0
//   dp = A2_r · B2_c, ds = p · (dp - D_x)       (product 2; not for d_v)
//   out_r += Σ_c w_rc · B3_c,  w = p (d_v) or ds (d_k, d_q)
// with x the query of the pair and D_x = Σ_y d_out_xy · out_xy:
//   d_v: rows keys,    A1 = k, B1 = q,                         B3 = d_out
//   d_k: rows keys,    A1 = k, B1 = q, A2 = v,     B2 = d_out, B3 = q
//   d_q: rows queries, A1 = q, B1 = k, A2 = d_out, B2 = v,     B3 = k
// (d_k and d_q then times scale). Each output row is summed by one CTA in
// column order: no atomics, the same bits on every run.
//
// The split form runs every product on tcgen05 kind::i8 over six int8
// digit planes, as the forward pass does, into TMEM columns 0..383; the
// weights w are cut into digits under a power of two per row and tile, and
// the rows' FP64 sums live in TMEM columns 384..511. Sixteen epilogue warps
// take a quarter of the columns each. The FP64 form runs the same tiles on
// the CUDA cores.
//
// Bound by the epilogue's instructions, as the forward pass (24,600 clocks a tile
// of d_k, the three products' 4,000 among them). Each operand's columns have
// stages of their own, so that a tile's load as soon as the product that read the
// last ones has run; the products run beside epilogue work (5.56 to 5.49 ms at 64
// x 4096 x 64, causal); P's export leaves through shared memory in whole lines
// (5.86 to 5.56 ms); dS is cut for d_q while the tile before is multiplied (2.21 to
// 1.76 ms). d_v, 1.25 ms, waits for P: 3.3 GB and as much again from L2, 1.04 ms
// with no arithmetic on its levels; its outputs multiplied by halves: 1.24 ms.
#include <algorithm>
#include <climits>
#include <cstdlib>
#include <cmath>
#include <type_traits>

#include "attention.cuh"
#include "fastexp.cuh"
#include "gemm.cuh"
#include "levels.cuh"
#include "prepare.cuh"
#include "ptx.cuh"

namespace ef {
namespace {

using namespace ptx;

enum GradMode { GRAD_V = 0, GRAD_K = 1, GRAD_Q = 2 };

constexpr int GM = 128, GJ = 64, GY = 64;
constexpr int CW = 16;            // columns an epilogue thread takes of its row
constexpr int kGroups = 64 / CW;  // groups of four epilogue warps, a row per TMEM lane
constexpr int kEpi = 128 * kGroups;
constexpr int kGradThreads = 64 + kEpi;
constexpr int kSumCol = 384;
constexpr int kMaxSmem = 232448;
constexpr int S = 6;

template <int MODE>
struct GradShape {
  static constexpr bool kTwo = MODE != GRAD_V;
  static constexpr int kA1 = S * GM * 64;            // rows' digits, product 1 (64 B of features)
  static constexpr int kA2 = kTwo ? S * GM * 64 : 0;  // rows' digits, product 2
  static constexpr int kB1 = S * GJ * 64;            // per stage
  static constexpr int kB2 = kTwo ? S * GJ * 64 : 0;
  static constexpr int kB3 = S * GY * 64;
  static constexpr int kE = 2 * GJ * 4;              // the columns' exponents of products 1 and 2
  // Rows of keys: the columns' (queries') lse, and for d_k their D.
  static constexpr int kL = (MODE == GRAD_V ? 1 : (MODE == GRAD_K ? 2 : 0)) * GJ * 8;
  static constexpr int kP = S * GM * 64;
  static constexpr int kStage = kB1 + kB2 + kB3;
  static constexpr int kStages = kA1 + kA2 + kP + 16384 + 2 * kStage <= kMaxSmem ? 2 : 1;
  // The columns' values are read after the first product frees its stage for
  // another tile's: they go round in two slots a stage.
  static constexpr int kCols = 2 * kStages;
  static constexpr int kAux = 6144 + kCols * (kE + kL);
  static constexpr int kSmem = kA1 + kA2 + kP + kAux + 1024 + kStages * kStage;
  static_assert(kSmem <= kMaxSmem, "the tiles must fit in shared memory");
};

struct GradArgs {
  Mask mask;  // the columns each row may pair with
  int64_t lr, lc, lr_pad, lc_pad, dy, dy_pad;
  int y0;
  double scale, out_factor;
  const int32_t* e_a1;  // [w][lr_pad]
  const int32_t* e_b1;  // [w][lc_pad]
  const int32_t* e_a2;
  const int32_t* e_b2;
  const int32_t* e_b3;  // [w][dy_pad]
  const double* lse;    // per query: [w·lq + x]
  const double* dd;     // D per query
  const double* lse_pad;  // the same, [w][lq_pad] (zeros past lq), for stages of keys' rows
  const double* dd_pad;
  const double* exp_table;
  double* out;  // [w·lr + r][dy]
  int* status;
  unsigned long long* tiles;
  int w0;  // the first batch of this launch (blockIdx.y counts from it)
  int reverse;  // row blocks from the last one (whose rows join the most columns) down
  // The d_k kernel's exports for the tile kernels (null: none), only for
  // the tiles some pair of is allowed: P's digit tiles as the d_v kernel cuts
  // them, [tile][S][128 rows][64 B] in the MMA's 64-byte swizzle, with their
  // rows' powers of two [tile][128], a key block's tiles from p_off[batch ·
  // n_rb + block] - p_base on, one a query tile it joins; and dS in tiles of
  // 128 queries by 64 keys, [tile][128][64], a query block's from
  // dq_off[batch · n_qb + block] - dq_base on, one a key tile from
  // dq_ct0[...] on (dq_n of them). Batches count from the launch's first.
  uint8_t* p_tiles;
  int32_t* p_exp;
  double* ds_out;
  const int64_t* p_off;
  const int64_t* dq_off;
  const int32_t* dq_ct0;
  const int32_t* dq_n;
  int64_t p_base, dq_base;
  int64_t n_rb, n_qb;  // key blocks and query blocks of a batch
  Ready ready;         // judged first: a launch that may not run does nothing
};


// The S levels of this thread's 4 TMEM columns at `col`, on their
// way; and landed.
__device__ __forceinline__ void load_levels(uint32_t lane_addr, int col, int32_t (&L)[S][4]) {
#pragma unroll
  for (int l = 0; l < S; l++) tmem_ld4(lane_addr + (uint32_t)(l * 64 + col), L[l]);
}
__device__ __forceinline__ void landed(int32_t (&L)[S][4]) {
#pragma unroll
  for (int l = 0; l < S; l++) tmem_landed(L[l]);
}

// `each(c, l)` for this thread's 16 columns from `col` on with their levels' sums l
// (in units of 2^kLevelUnit), the next four columns' levels loading meanwhile.
template <class F>
__device__ __forceinline__ void each_level_sum(uint32_t lane_addr, int col, F&& each) {
  int32_t L[S][4];
  load_levels(lane_addr, col, L);
#pragma unroll
  for (int c4 = 0; c4 < CW / 4; c4++) {
    tmem_wait_ld();
    landed(L);
    double l[4];
#pragma unroll
    for (int i = 0; i < 4; i++) l[i] = combine_levels_small(L, i);
    if (c4 + 1 < CW / 4) load_levels(lane_addr, col + c4 * 4 + 4, L);
#pragma unroll
    for (int i = 0; i < 4; i++) each(c4 * 4 + i, l[i]);
  }
}

// slice_exponent of the largest magnitude of w, INT_MIN if all are zeros: from the
// largest high word (an integer maximum a value, a third of a double's) unless
// that is a zero's or a subnormal's.
__device__ __forceinline__ int row_exponent(const double (&w)[CW]) {
  int h = 0;
#pragma unroll
  for (int c = 0; c < CW; c++) h = max(h, __double2hiint(w[c]) & 0x7fffffff);
  if (h >= 0x00100000) return (h >> 20) - 1020;
  double m = 0.0;
#pragma unroll
  for (int c = 0; c < CW; c++) m = fmax(m, fabs(w[c]));
  return m > 0.0 ? slice_exponent(m) : INT_MIN;
}

// The row's exponent from its groups' (0: all zeros).
__device__ __forceinline__ int row_maximum(const int* parts, int r) {
  int e = parts[r];
#pragma unroll
  for (int i = 1; i < kGroups; i++) e = max(e, parts[i * GM + r]);
  return e == INT_MIN ? 0 : e;
}

// The digit planes of w · 2^(8S - e), sixteen bytes a plane: the power of two in
// one factor where it is a normal double for the whole warp, else in two exact
// ones (8S - e lies in [-978, 1119]).
__device__ __forceinline__ void cut_digits(const double (&w)[CW], int e, uint32_t (&chunk)[S][CW / 4]) {
  const int shift = 8 * S - e;
  auto cut = [&](auto one) {
    const double f1 = pow2(decltype(one)::value ? shift : shift >> 1), f2 = pow2(shift - (shift >> 1));
#pragma unroll
    for (int c4 = 0; c4 < CW / 4; c4++) {
      double x[4];
#pragma unroll
      for (int i = 0; i < 4; i++) x[i] = decltype(one)::value ? w[c4 * 4 + i] : w[c4 * 4 + i] * f2;
      uint32_t planes[S];
      digit_planes4<S>(x, f1, planes);
#pragma unroll
      for (int s = 0; s < S; s++) chunk[s][c4] = planes[s];
    }
  };
  if (__all_sync(0xffffffffu, shift <= 1023)) cut(std::true_type{});
  else cut(std::false_type{});
}
// A row's digits into a tile of digit planes, in the MMA's 64-byte swizzle.
__device__ __forceinline__ void store_digits(const uint32_t (&chunk)[S][CW / 4], uint8_t* tile, int r, int col) {
#pragma unroll
  for (int b = 0; b < CW / 16; b++) {
    uint8_t* dst = tile + sw64_offset((uint32_t)r, (uint32_t)(col + b * 16));
#pragma unroll
    for (int s = 0; s < S; s++)
      *(uint4*)(dst + s * GM * 64) =
          make_uint4(chunk[s][b * 4], chunk[s][b * 4 + 1], chunk[s][b * 4 + 2], chunk[s][b * 4 + 3]);
  }
}

// sums += the levels · 2^(ew + e3): one rounding either way, the power of two a
// normal double on the first path (e3lo and e3hi bound e3). `first`: sums start here.
__device__ __forceinline__ void add_levels(uint32_t lane_addr, uint32_t sum_addr, int col, int ew, const int* e3, int e3lo,
                                           int e3hi, bool first) {
  auto add = [&](auto normal) {
    int32_t L[S][4], sum[8];
    load_levels(lane_addr, col, L);
    if (!first) tmem_ld8(sum_addr, sum);
    const int base = (ew + 1023 + kLevelUnit) << 20;
#pragma unroll
    for (int c4 = 0; c4 < CW / 4; c4++) {
      tmem_wait_ld();
      landed(L);
      if (!first) tmem_landed(sum);
      uint32_t next[8];
#pragma unroll
      for (int i = 0; i < 4; i++) {
        const int e = e3[c4 * 4 + i];
        const double prev = first ? 0.0 : __hiloint2double(sum[2 * i + 1], sum[2 * i]);
        const double l = combine_levels_small(L, i);
        const double v = decltype(normal)::value ? fma(l, __hiloint2double((e << 20) + base, 0), prev)
                                                 : prev + scale2(l, ew + e + kLevelUnit);
        next[2 * i] = (uint32_t)__double2loint(v);
        next[2 * i + 1] = (uint32_t)__double2hiint(v);
      }
      if (c4 + 1 < CW / 4) {
        load_levels(lane_addr, col + c4 * 4 + 4, L);
        if (!first) tmem_ld8(sum_addr + c4 * 8 + 8, sum);
      }
      tmem_st8(sum_addr + c4 * 8, next);
    }
  };
  if (__all_sync(0xffffffffu, ew + e3lo + kLevelUnit >= -1022 && ew + e3hi + kLevelUnit <= 1023)) add(std::true_type{});
  else add(std::false_type{});
}

constexpr int kPTile = S * GM * 64;  // bytes of one tile of weight digits

// FAST: every pair of row and column exponents of products 1 and 2 sums to
// a normal double's power of two.
template <int MODE, bool FAST>
__global__ void __launch_bounds__(kGradThreads, 1)
    grad_split(const __grid_constant__ CUtensorMap ta1, const __grid_constant__ CUtensorMap tb1,
               const __grid_constant__ CUtensorMap ta2, const __grid_constant__ CUtensorMap tb2,
               const __grid_constant__ CUtensorMap tb3, const GradArgs a) {
  using Sh = GradShape<MODE>;
  constexpr bool kTwo = Sh::kTwo;
  if (!a.ready.ok()) return;  // the same for every thread
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = (uint8_t*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  uint8_t* sA1 = smem;
  uint8_t* sA2 = sA1 + Sh::kA1;
  uint8_t* sP = sA2 + Sh::kA2;
  uint8_t* sB = sP + Sh::kP;  // stages of [B1 | B2 | B3]
  uint8_t* aux = sB + Sh::kStages * Sh::kStage;
  uint64_t* bars = (uint64_t*)aux;
  uint64_t* a_full = bars + 0;
  // Stages' [2] of each operand: loaded as soon as the product that reads it has
  // run on the tile before.
  uint64_t* b1_full = bars + 1;
  uint64_t* b1_empty = bars + 3;
  uint64_t* b2_full = bars + 5;
  uint64_t* b2_empty = bars + 7;
  uint64_t* b3_full = bars + 9;
  uint64_t* b3_empty = bars + 11;
  uint64_t* s1_full = bars + 13;
  uint64_t* t1_free = bars + 14;
  uint64_t* s2_full = bars + 15;
  uint64_t* p_full = bars + 16;
  uint64_t* o_full = bars + 17;
  uint64_t* o_free = bars + 18;
  uint64_t* s2_free = bars + 19;  // the second product's levels are read (without one: the sums are added)
  uint32_t* tmem_slot = (uint32_t*)(bars + 20);
  int* failed = (int*)(tmem_slot + 1);
  long long* span = (long long*)(tmem_slot + 4);
  int* row_lo = (int*)(aux + 256);
  int* row_hi = row_lo + GM;
  int* e3_s = row_hi + GM;               // [64]
  double* texp = (double*)(aux + 1536);  // [64]
  int* red = (int*)(aux + 2048);         // [4][128] the quarters' exponents
  int* redp = (int*)(aux + 4096);        // [4][128] the same for P (d_k's export)
  uint8_t* cols = aux + 6144;            // a tile's exponents, lse and D of its columns

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int rt = a.reverse ? (int)(gridDim.x - 1 - blockIdx.x) : (int)blockIdx.x;
  const int w = a.w0 + (int)blockIdx.y;
  const int64_t r_base = (int64_t)w * a.lr, c_base = (int64_t)w * a.lc;

  if (threadIdx.x == 0) {
    for (int i = 0; i < 18; i++) mbar_init(&bars[i], 1);
    // Each epilogue warp arrives on the barriers that free TMEM or shared memory.
    mbar_init(t1_free, kEpi / 32);
    mbar_init(p_full, kEpi / 32);
    mbar_init(o_free, kEpi / 32);
    mbar_init(s2_free, kEpi / 32);
    *failed = 0;
    span[0] = LLONG_MAX;
    span[1] = LLONG_MIN;
    mbar_fence_init();
  }
  if (warp == 1) {
    tmem_alloc(tmem_slot, 512);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  if (threadIdx.x < GM) {
    const int64_t rl = (int64_t)rt * GM + threadIdx.x;
    int lo = 0, hi = 0;
    if (rl < a.lr) {
      int64_t l, h;
      allowed(a.mask, r_base + rl, l, h);
      lo = (int)(l - c_base);
      hi = (int)(h - c_base);
      if (lo < hi) {
        atomicMin(&span[0], (long long)lo);
        atomicMax(&span[1], (long long)hi);
      }
    }
    row_lo[threadIdx.x] = lo;
    row_hi[threadIdx.x] = hi;
  } else if (threadIdx.x < GM + GY) {
    const int c = threadIdx.x - GM;
    e3_s[c] = a.y0 + c < a.dy_pad ? a.e_b3[(int64_t)w * a.dy_pad + a.y0 + c] : 0;
  } else if (threadIdx.x < GM + GY + 64) {
    texp[threadIdx.x - GM - GY] = a.exp_table[threadIdx.x - GM - GY];
  }
  __syncthreads();
  const uint32_t tmem = *tmem_slot;
  const long long first = span[0], last = span[1];
  const int ct0 = first < last ? (int)(first / GJ) : 0;
  const int n_tiles = first < last ? (int)((last + GJ - 1) / GJ) - ct0 : 0;
  if (threadIdx.x == 0 && n_tiles > 0) atomicAdd(a.tiles, (unsigned long long)n_tiles);

  if (warp == 0) {
    if (lane == 0 && n_tiles > 0) {
      prefetch_map(&ta1);
      prefetch_map(&tb1);
      prefetch_map(&tb3);
      mbar_expect_tx(a_full, (uint32_t)(Sh::kA1 + Sh::kA2));
      tma_load_3d(sA1, &ta1, a_full, 0, rt * GM, w * S);
      if (kTwo) tma_load_3d(sA2, &ta2, a_full, 0, rt * GM, w * S);
      // Each operand's tiles issued, and one of them (false once a wait ran out).
      int n1 = 0, n2 = 0, n3 = 0;
      auto slot = [&](uint64_t* empty, int it) {
        if (*(volatile int*)failed) return false;
        if (mbar_wait(&empty[it % Sh::kStages], ((uint32_t)(it / Sh::kStages) & 1) ^ 1)) return true;
        atomicOr(a.status, 2);
        *(volatile int*)failed = 1;
        return false;
      };
      auto load1 = [&](int it) {
        if (!slot(b1_empty, it)) return false;
        const int st = it % Sh::kStages, cl0 = (ct0 + it) * GJ;
        uint64_t* full = &b1_full[st];
        mbar_expect_tx(full, (uint32_t)(Sh::kB1 + (kTwo ? 2 : 1) * GJ * 4 + Sh::kL));
        tma_load_3d(sB + st * Sh::kStage, &tb1, full, 0, cl0, w * S);
        int* es = (int*)(cols + (it % Sh::kCols) * (Sh::kE + Sh::kL));
        bulk_load(es, a.e_b1 + (int64_t)w * a.lc_pad + cl0, GJ * 4, full);
        if (kTwo) bulk_load(es + GJ, a.e_b2 + (int64_t)w * a.lc_pad + cl0, GJ * 4, full);
        if (MODE != GRAD_Q) {
          double* ls = (double*)(es + 2 * GJ);
          bulk_load(ls, a.lse_pad + (int64_t)w * a.lc_pad + cl0, GJ * 8, full);
          if (MODE == GRAD_K) bulk_load(ls + GJ, a.dd_pad + (int64_t)w * a.lc_pad + cl0, GJ * 8, full);
        }
        n1 = it + 1;
        return true;
      };
      auto load2 = [&](int it) {
        if (!slot(b2_empty, it)) return false;
        const int st = it % Sh::kStages;
        mbar_expect_tx(&b2_full[st], (uint32_t)Sh::kB2);
        tma_load_3d(sB + st * Sh::kStage + Sh::kB1, &tb2, &b2_full[st], 0, (ct0 + it) * GJ, w * S);
        n2 = it + 1;
        return true;
      };
      auto load3 = [&](int it) {
        if (!slot(b3_empty, it)) return false;
        const int st = it % Sh::kStages;
        mbar_expect_tx(&b3_full[st], (uint32_t)Sh::kB3);
        tma_load_3d(sB + st * Sh::kStage + Sh::kB1 + Sh::kB2, &tb3, &b3_full[st], (ct0 + it) * GJ, a.y0, w * S);
        n3 = it + 1;
        return true;
      };
      // In the order in which the products free them: tile it + 1's first, tile
      // it's third, tile it + 1's second.
      auto within = [&](int it) { return it < n_tiles; };
      bool ok = load1(0) && (!kTwo || load2(0)) && load3(0);
      if (within(1)) ok = ok && load1(1) && (!kTwo || load2(1));
      for (int it = 0; ok && within(it + 1); it++) {
        if (within(it + 2)) ok = load1(it + 2);
        ok = ok && load3(it + 1);
        if (kTwo && within(it + 2)) ok = ok && load2(it + 2);
      }
      mbar_wait(a_full, 0);
      auto drain = [&](uint64_t* full, int issued) {
        for (int it = std::max(0, issued - Sh::kStages); it < issued; it++)
          mbar_wait(&full[it % Sh::kStages], (uint32_t)((it / Sh::kStages) & 1));
      };
      drain(b1_full, n1);
      drain(b2_full, n2);
      drain(b3_full, n3);
    }
  } else if (warp == 1) {
    if (lane == 0 && n_tiles > 0) {
      uint64_t* last_bar = nullptr;
      uint32_t last_parity = 0;
      bool ok = mbar_wait(a_full, 0);
      // D (+)= A · B over S digit planes, the level scheme of the forward pass.
      auto product = [&](uint32_t a_base, uint32_t b_base, int n) {
        const uint64_t a0 = desc_sw64(a_base), b0 = desc_sw64(b_base);
#pragma unroll
        for (int kk = 0; kk < 2; kk++)
#pragma unroll
          for (int s = 1; s <= S; s++) {
            const int total = (S + 1 - s) * n;
#pragma unroll
            for (int nn0 = 0; nn0 < total; nn0 += 256) {
              const int nn = total - nn0 < 256 ? total - nn0 : 256;
              umma_i8(tmem + (uint32_t)((s - 1) * n + nn0), desc_further(a0, (s - 1) * GM * 64 + kk * 32),
                      desc_further(b0, nn0 * 64 + kk * 32), idesc_i8(GM, nn), (kk > 0 || s > 1) ? 1u : 0u);
            }
          }
      };
      auto wait = [&](uint64_t* bar, int phase) {
        return mbar_wait(bar, (uint32_t)(phase & 1)) && !*(volatile int*)failed;
      };
      // Tile `it`'s product number `i` once its columns are there.
      auto run = [&](int it, int i, uint64_t* full, uint64_t* empty, uint64_t* done, const uint8_t* a_digits) {
        const int st = it % Sh::kStages;
        if (!wait(&full[st], it / Sh::kStages)) return false;
        tc_fence_after();
        product(smem_u32(a_digits), smem_u32(sB + st * Sh::kStage + (i > 1 ? Sh::kB1 : 0) + (i > 2 ? Sh::kB2 : 0)), 64);
        umma_commit(done);
        umma_commit(&empty[st]);
        last_bar = done;
        last_parity = (uint32_t)(it & 1);
        return true;
      };
      static_assert(GJ == 64 && GY == 64, "the products' columns");
      // Each product runs beside epilogue work that needs none of the levels:
      // the next tile's scores while the weights' digits are cut, the weighted
      // values while the next tile's exponentials are taken, d_out·v while P's
      // digits are cut.
      ok = ok && run(0, 1, b1_full, b1_empty, s1_full, sA1) && wait(t1_free, 0);
      for (int it = 0; ok && it < n_tiles; it++) {
        if (kTwo) ok = (it == 0 || wait(o_free, it - 1)) && run(it, 2, b2_full, b2_empty, s2_full, sA2);
        ok = ok && wait(s2_free, it);
        if (it + 1 < n_tiles) ok = ok && run(it + 1, 1, b1_full, b1_empty, s1_full, sA1) && wait(t1_free, it + 1);
        ok = ok && wait(p_full, it) && run(it, 3, b3_full, b3_empty, o_full, sP);
      }
      if (!ok) {
        atomicOr(a.status, 2);
        *(volatile int*)failed = 1;
      }
      if (last_bar) mbar_wait(last_bar, last_parity);
    }
  } else {
    // Epilogue: warp w reads TMEM lanes 32·(w % 4) .. +31 and a quarter of
    // the columns; the four warps of a lane quarter exchange row maxima over
    // their own named barrier, and each warp signals the MMA warp by itself.
    const int h = (warp - 2) >> 2;
    const int quarter = warp & 3;
    const int r = quarter * 32 + lane;
    const int64_t rl = (int64_t)rt * GM + r;
    const bool valid = rl < a.lr;
    const int lo = row_lo[r], hi = row_hi[r];
    // Column c of a tile starting at cl0 is allowed iff (unsigned)(cl0 + c - lo) < span.
    const unsigned span = (valid && lo < hi) ? (unsigned)(hi - lo) : 0u;
    const int e1r = valid ? a.e_a1[(int64_t)w * a.lr_pad + rl] : 0;
    const int e2r = (kTwo && valid) ? a.e_a2[(int64_t)w * a.lr_pad + rl] : 0;
    // FAST: a score's scale times its powers of two, but for the column's; and
    // d_out·v's.
    const int factor_hi = __double2hiint(a.scale) + ((e1r + kLevelUnit) << 20), factor_lo = __double2loint(a.scale);
    const int base2 = (e2r + 1023 + kLevelUnit) << 20;
    // A row of queries reads its own lse and D; a row of keys its columns'.
    const int64_t p_first =
        MODE == GRAD_K && a.p_tiles ? a.p_off[(int64_t)blockIdx.y * a.n_rb + rt] - a.p_base : 0;
    const double lse_r = (MODE == GRAD_Q && valid) ? a.lse[r_base + rl] : 0.0;
    const double dd_r = (MODE == GRAD_Q && valid) ? a.dd[r_base + rl] : 0.0;
    const uint32_t lane_addr = tmem + ((uint32_t)(quarter * 32) << 16);
    const uint32_t sum_addr = lane_addr + (uint32_t)(kSumCol + h * 2 * CW);
    int e3lo = INT_MAX, e3hi = INT_MIN;
    for (int c = 0; c < GY; c++) {
      e3lo = min(e3lo, e3_s[c]);
      e3hi = max(e3hi, e3_s[c]);
    }
    auto wait = [&](uint64_t* bar, uint32_t parity) {
      if (*(volatile int*)failed) return;
      if (!mbar_wait(bar, parity)) {
        *(volatile int*)failed = 1;
        atomicOr(a.status, 2);
      }
    };
    // This warp is done with TMEM or shared memory: one arrival.
    auto arrive = [&](uint64_t* bar) {
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(bar);
    };
    auto columns = [&](int it) { return cols + (it % Sh::kCols) * (Sh::kE + Sh::kL); };
    double wv[CW];
    // Tile `it`'s scaled scores.
    auto read_scores = [&](int it) {
      const int* es = (const int*)columns(it) + h * CW;
      wait(s1_full, (uint32_t)(it & 1));
      tc_fence_after();
      each_level_sum(lane_addr, h * CW, [&](int c, double l) {
        wv[c] = FAST ? l * __hiloint2double((es[c] << 20) + factor_hi, factor_lo)
                     : a.scale * scale2(l, e1r + es[c] + kLevelUnit);
      });
      arrive(t1_free);
    };
    int ew = 0;  // the row's power of two of the weights cut last
    auto add = [&](int it) {
      wait(o_full, (uint32_t)(it & 1));
      tc_fence_after();
      add_levels(lane_addr, sum_addr, h * CW, ew, e3_s + h * CW, e3lo, e3hi, it == 0);
      tmem_wait_st();
      arrive(o_free);
    };
    if (n_tiles > 0) read_scores(0);
    for (int it = 0; it < n_tiles; it++) {
      const int cl0 = (ct0 + it) * GJ + h * CW;
      const int* es = (const int*)columns(it) + h * CW;
      const double* ls = (const double*)(columns(it) + Sh::kE) + h * CW;
      const uint32_t par = (uint32_t)(it & 1);
      const int off = cl0 - lo;
      // d_k's export of dS: into the d_q kernel's tile of this tile's query
      // block and the row's key tile, row (query) cl0 + c, the keys
      // contiguous; nothing for a key tile the query block's rows don't join
      // (every pair there is masked).
      double* ds_col = nullptr;
      if (MODE == GRAD_K && a.ds_out) {
        const int64_t qbi = (int64_t)blockIdx.y * a.n_qb + cl0 / GM;
        const int64_t kt = ((int64_t)rt * GM + r) / GJ - a.dq_ct0[qbi];
        const int64_t tiles_q = a.dq_n[qbi], first_q = a.dq_off[qbi];
        if (kt >= 0 && kt < tiles_q) ds_col = a.ds_out + ((first_q - a.dq_base + kt) * GM + cl0 % GM) * GJ + r % GJ;
      }
      // Every pair of the warp's rows and columns allowed: no selects.
      const bool whole = __all_sync(0xffffffffu, off >= 0 && (unsigned)off + CW <= span);
#pragma unroll
      for (int c = 0; c < CW; c++) wv[c] = exp_weight(wv[c] - (MODE == GRAD_Q ? lse_r : ls[c]), texp, 0);
      if (!whole)
#pragma unroll
        for (int c = 0; c < CW; c++) wv[c] = (unsigned)(off + c) < span ? wv[c] : 0.0;
      if (it > 0) add(it - 1);
      if (!kTwo) arrive(s2_free);
      if (kTwo) {
        if (MODE == GRAD_K && a.p_tiles) {
          // While d_out·v runs: P's digits for the d_v tile kernel, cut as
          // that kernel's own epilogue would (W = p · 2^(8S - ep), ep the
          // row's exponent over these 64 columns), swizzled rows through sP and
          // from there in one copy a plane and quarter (sixteen bytes a row
          // straight from registers wrote half sectors).
          redp[h * GM + r] = row_exponent(wv);
          named_bar(2 + quarter, 32 * kGroups);
          const int ep = row_maximum(redp, r);
          const int64_t tile = p_first + it;
          uint32_t chunk[S][CW / 4];
          cut_digits(wv, ep, chunk);
          store_digits(chunk, sP, r, h * CW);  // (the tile before's MMAs have read it)
          fence_proxy_async();
          if (h == 0) a.p_exp[tile * GM + r] = ep;
          named_bar(2 + quarter, 32 * kGroups);
          if (h == 0 && lane == 0) {
#pragma unroll
            for (int s = 0; s < S; s++) {
              const int at = s * GM * 64 + quarter * 32 * 64;
              bulk_store(a.p_tiles + tile * kPTile + at, sP + at, 32 * 64);
            }
            bulk_commit();
          }
        }
        wait(s2_full, par);
        tc_fence_after();
        each_level_sum(lane_addr, h * CW, [&](int c, double l) {
          const double dp = FAST ? l * __hiloint2double((es[GJ + c] << 20) + base2, 0)
                                 : scale2(l, e2r + es[GJ + c] + kLevelUnit);
          const double t = wv[c] * (dp - (MODE == GRAD_Q ? dd_r : ls[GJ + c]));
          wv[c] = whole || wv[c] != 0.0 ? t : 0.0;
          if (ds_col) ds_col[(int64_t)c * GJ] = wv[c];
        });
        arrive(s2_free);
      }
      // The row's power of two for this tile, over the four quarters.
      if (MODE == GRAD_K && a.p_tiles && h == 0 && lane == 0) bulk_wait_read();  // P's export has left sP
      red[h * GM + r] = row_exponent(wv);
      named_bar(2 + quarter, 32 * kGroups);
      ew = row_maximum(red, r);
      // The weights' digits: W = w · 2^(8S - ew), |W| < 2^(8S-2).
      {
        uint32_t chunk[S][CW / 4];
        cut_digits(wv, ew, chunk);
        store_digits(chunk, sP, r, h * CW);
      }
      fence_proxy_async();
      arrive(p_full);
      if (it + 1 < n_tiles) read_scores(it + 1);
    }
    if (n_tiles > 0) add(n_tiles - 1);
    if (MODE == GRAD_K && a.p_tiles && h == 0 && lane == 0) bulk_wait();
    // Every lane of the warp reads TMEM (the loads are warp-wide); the rows
    // past the batch's end write nothing.
    tc_fence_after();
    const bool store = valid && !*(volatile int*)failed;
    double* orow = a.out + (r_base + rl) * a.dy;
#pragma unroll
    for (int c4 = 0; c4 < CW / 4; c4++) {
      uint32_t sum[8];
      if (n_tiles > 0) {
        tmem_ld8(sum_addr + c4 * 8, (int32_t*)sum);
        tmem_wait_ld();
      }
#pragma unroll
      for (int i = 0; i < 4; i++) {
        const int64_t y = (int64_t)a.y0 + h * CW + c4 * 4 + i;
        const double v = n_tiles > 0 ? __hiloint2double((int)sum[2 * i + 1], (int)sum[2 * i]) : 0.0;
        if (store && y < a.dy) orow[y] = a.out_factor * v;
      }
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem, 512);
  }
}

// The d_v and d_q tiles from the weights the d_k kernel exported: one
// product a tile (the weights' digits against the columns' B3 digits) and
// the rows' sums, with no scores, exponentials or d_out·v recomputed. d_v
// reads P's digit tiles and their rows' powers of two as they are; d_q reads
// dS (query-major, four 128-byte-swizzled boxes of 16 keys a tile), applies
// the mask and cuts its digits under the row's power of two over the tile,
// as grad_split's epilogue does, so that both gradients come out with the
// same bits as there.
template <int MODE>
struct TileShape {
  static constexpr bool kQ = MODE == GRAD_Q;
  static constexpr int kDs = kQ ? GM * GJ * 8 : 0;  // one dS tile
  static constexpr int kDsBufs = kQ ? 2 : 0;        // d_q: dS tiles double-buffered
  static constexpr int kBufs = kQ ? 1 : 2;          // weight digit tiles (d_v: one a stage)
  static constexpr int kB3 = S * GY * 64;
  static constexpr int kStage = kB3 + (kQ ? 0 : 1024);  // B3, and for d_v the rows' exponents
  static constexpr int kStages = kQ ? 1 : 2;
  static constexpr int kAux = 8192;
  static constexpr int kSmem = kDsBufs * kDs + kBufs * kPTile + kStages * kStage + kAux + 1024;
  static_assert(kSmem <= kMaxSmem, "the tiles must fit in shared memory");
};

template <int MODE>
__global__ void __launch_bounds__(kGradThreads, 1)
    grad_tiles(const __grid_constant__ CUtensorMap tds, const __grid_constant__ CUtensorMap tb3, const GradArgs a) {
  using Sh = TileShape<MODE>;
  constexpr bool kQ = Sh::kQ;
  if (!a.ready.ok()) return;  // the same for every thread
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = (uint8_t*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  uint8_t* sDs = smem;  // d_q: [2] dS tiles
  uint8_t* sP = sDs + Sh::kDsBufs * Sh::kDs;
  uint8_t* sB = sP + Sh::kBufs * kPTile;  // stages of [B3 | rows' exponents]
  uint8_t* aux = sB + Sh::kStages * Sh::kStage;
  uint64_t* bars = (uint64_t*)aux;
  uint64_t* kv_full = bars + 0;   // [2] B3 stages (d_v: with the weights' tile)
  uint64_t* kv_empty = bars + 2;  // [2]
  uint64_t* ds_full = bars + 4;   // [2] d_q: dS tiles
  uint64_t* ds_empty = bars + 6;  // [2]
  uint64_t* p_full = bars + 8;
  uint64_t* o_full = bars + 9;
  uint64_t* tmem_free = bars + 10;
  uint32_t* tmem_slot = (uint32_t*)(bars + 16);
  int* failed = (int*)(tmem_slot + 1);
  long long* span = (long long*)(tmem_slot + 4);
  int* row_lo = (int*)(aux + 256);
  int* row_hi = row_lo + GM;
  int* e3_s = row_hi + GM;        // [64]
  int* red = (int*)(aux + 4096);  // [2][4][128]

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int rt = a.reverse ? (int)(gridDim.x - 1 - blockIdx.x) : (int)blockIdx.x;
  const int w = a.w0 + (int)blockIdx.y;
  const int64_t r_base = (int64_t)w * a.lr, c_base = (int64_t)w * a.lc;

  if (threadIdx.x == 0) {
    for (int i = 0; i < 2; i++) {
      mbar_init(&kv_full[i], 1);
      // d_v: the MMAs' commit and every epilogue warp (which reads the
      // stage's exponents) free a stage.
      mbar_init(&kv_empty[i], kQ ? 1 : 1 + kEpi / 32);
    }
    for (int i = 0; i < 2; i++) {
      mbar_init(&ds_full[i], 1);
      mbar_init(&ds_empty[i], kEpi / 32);
    }
    mbar_init(p_full, kEpi / 32);
    mbar_init(o_full, 1);
    mbar_init(tmem_free, kEpi / 32);
    *failed = 0;
    span[0] = LLONG_MAX;
    span[1] = LLONG_MIN;
    mbar_fence_init();
  }
  if (warp == 1) {
    tmem_alloc(tmem_slot, 512);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  if (threadIdx.x < GM) {
    const int64_t rl = (int64_t)rt * GM + threadIdx.x;
    int lo = 0, hi = 0;
    if (rl < a.lr) {
      int64_t l, h;
      allowed(a.mask, r_base + rl, l, h);
      lo = (int)(l - c_base);
      hi = (int)(h - c_base);
      if (lo < hi) {
        atomicMin(&span[0], (long long)lo);
        atomicMax(&span[1], (long long)hi);
      }
    }
    row_lo[threadIdx.x] = lo;
    row_hi[threadIdx.x] = hi;
  } else if (threadIdx.x < GM + GY) {
    const int c = threadIdx.x - GM;
    e3_s[c] = a.y0 + c < a.dy_pad ? a.e_b3[(int64_t)w * a.dy_pad + a.y0 + c] : 0;
  }
  __syncthreads();
  const uint32_t tmem = *tmem_slot;
  const long long first = span[0], last = span[1];
  const int ct0 = first < last ? (int)(first / GJ) : 0;
  const int n_tiles = first < last ? (int)((last + GJ - 1) / GJ) - ct0 : 0;
  if (threadIdx.x == 0 && n_tiles > 0) atomicAdd(a.tiles, (unsigned long long)n_tiles);
  // d_v: this key block's P tiles; d_q: this query block's dS tiles.
  auto tile_of = [&](int it) {
    return kQ ? a.dq_off[(int64_t)blockIdx.y * a.n_qb + rt] - a.dq_base + it
              : a.p_off[(int64_t)blockIdx.y * a.n_rb + rt] - a.p_base + it;
  };

  if (warp == 0) {
    if (lane == 0 && n_tiles > 0) {
      prefetch_map(&tb3);
      if (kQ) prefetch_map(&tds);
      int issued = 0;
      for (int it = 0; it < n_tiles; it++) {
        const int st = it & 1;
        const uint32_t round = (uint32_t)(it >> 1);
        const int cl0 = (ct0 + it) * GJ;
        if (*(volatile int*)failed) break;
        bool ok;
        if (kQ) {
          // dS two tiles ahead; B3 (one stage) once the previous tile's MMAs are done.
          ok = mbar_wait(&ds_empty[st], (round & 1) ^ 1);
          if (ok) {
            mbar_expect_tx(&ds_full[st], (uint32_t)Sh::kDs);
            for (int j = 0; j < 4; j++)
              tma_load_3d(sDs + st * Sh::kDs + j * GM * 128, &tds, &ds_full[st], 16 * j, (int)(tile_of(it) * GM),
                          0);
          }
          ok = ok && (it == 0 || mbar_wait(&kv_empty[0], (uint32_t)((it - 1) & 1)));
          if (ok) {
            mbar_expect_tx(&kv_full[0], (uint32_t)Sh::kB3);
            tma_load_3d(sB, &tb3, &kv_full[0], cl0, a.y0, w * S);
          }
        } else {
          ok = mbar_wait(&kv_empty[st], (round & 1) ^ 1);
          if (ok) {
            uint8_t* stage = sB + st * Sh::kStage;
            mbar_expect_tx(&kv_full[st], (uint32_t)(Sh::kB3 + kPTile + GM * 4));
            tma_load_3d(stage, &tb3, &kv_full[st], cl0, a.y0, w * S);
            bulk_load(sP + st * kPTile, a.p_tiles + tile_of(it) * kPTile, kPTile, &kv_full[st]);
            bulk_load(stage + Sh::kB3, a.p_exp + tile_of(it) * GM, GM * 4, &kv_full[st]);
          }
        }
        if (!ok) {
          atomicOr(a.status, 2);
          *(volatile int*)failed = 1;
          break;
        }
        issued = it + 1;
      }
      // Copies still in flight complete before the CTA may exit.
      for (int it = std::max(0, issued - 2); it < issued; it++) {
        if (kQ) {
          mbar_wait(&ds_full[it & 1], (uint32_t)((it >> 1) & 1));
          if (it == issued - 1) mbar_wait(&kv_full[0], (uint32_t)(it & 1));
        } else {
          mbar_wait(&kv_full[it & 1], (uint32_t)((it >> 1) & 1));
        }
      }
    }
  } else if (warp == 1) {
    if (lane == 0 && n_tiles > 0) {
      int last = -1;  // the last tile whose MMAs were committed
      bool ok = true;
      for (int it = 0; ok && it < n_tiles; it++) {
        const int st = kQ ? 0 : (it & 1);
        const uint32_t par = (uint32_t)(it & 1);
        const uint32_t a_base = smem_u32(sP + (kQ ? 0 : st * kPTile)), b_base = smem_u32(sB + st * Sh::kStage);
        ok = mbar_wait(&kv_full[st], kQ ? par : (uint32_t)((it >> 1) & 1)) &&
             (it == 0 || mbar_wait(tmem_free, par ^ 1)) && (!kQ || mbar_wait(p_full, par));
        if (!ok || *(volatile int*)failed) break;
        const uint64_t a0 = desc_sw64(a_base), b0 = desc_sw64(b_base);
        tc_fence_after();
#pragma unroll
        for (int kk = 0; kk < 2; kk++)
#pragma unroll
          for (int s = 1; s <= S; s++) {
            const int total = (S + 1 - s) * GY;
#pragma unroll
            for (int nn0 = 0; nn0 < total; nn0 += 256) {
              const int nn = total - nn0 < 256 ? total - nn0 : 256;
              umma_i8(tmem + (uint32_t)((s - 1) * GY + nn0), desc_further(a0, (s - 1) * GM * 64 + kk * 32),
                      desc_further(b0, nn0 * 64 + kk * 32), idesc_i8(GM, nn), (kk > 0 || s > 1) ? 1u : 0u);
            }
          }
        umma_commit(o_full);
        umma_commit(&kv_empty[st]);
        last = it;
      }
      if (!ok) {
        atomicOr(a.status, 2);
        *(volatile int*)failed = 1;
      }
      // MMAs still running complete before TMEM is freed.
      if (last >= 0) mbar_wait(o_full, (uint32_t)(last & 1));
    }
  } else {
    const int h = (warp - 2) >> 2;
    const int quarter = warp & 3;
    const int r = quarter * 32 + lane;
    const int64_t rl = (int64_t)rt * GM + r;
    const bool valid = rl < a.lr;
    const int lo = row_lo[r], hi = row_hi[r];
    const unsigned span_r = (valid && lo < hi) ? (unsigned)(hi - lo) : 0u;
    const uint32_t lane_addr = tmem + ((uint32_t)(quarter * 32) << 16);
    const uint32_t sum_addr = lane_addr + (uint32_t)(kSumCol + h * 2 * CW);
    int e3lo = INT_MAX, e3hi = INT_MIN;
    for (int c = 0; c < GY; c++) {
      e3lo = min(e3lo, e3_s[c]);
      e3hi = max(e3hi, e3_s[c]);
    }
    auto wait = [&](uint64_t* bar, uint32_t parity) {
      if (*(volatile int*)failed) return;
      if (!mbar_wait(bar, parity)) {
        *(volatile int*)failed = 1;
        atomicOr(a.status, 2);
      }
    };
    // d_q: tile `it`'s digits in registers, cut while the tile before is
    // multiplied; its row's power of two.
    uint32_t chunk[S][CW / 4];
    auto cut = [&](int it) {
      const int st = it & 1;
      wait(&ds_full[st], (uint32_t)((it >> 1) & 1));
      // This row's 16 keys of the tile: box h, 128-byte row r, its 16-byte
      // chunks permuted by r mod 8.
      const uint8_t* row = sDs + st * Sh::kDs + h * (CW / 16) * GM * 128 + r * 128;
      const int off = (ct0 + it) * GJ + h * CW - lo;
      double wv[CW];
#pragma unroll
      for (int j = 0; j < CW / 2; j++) {
        const double2 v = *(const double2*)(row + (j >> 3) * GM * 128 + (((j & 7) ^ (r & 7)) << 4));
        wv[2 * j] = (unsigned)(off + 2 * j) < span_r ? v.x : 0.0;
        wv[2 * j + 1] = (unsigned)(off + 2 * j + 1) < span_r ? v.y : 0.0;
      }
      __syncwarp();
      if (lane == 0) mbar_arrive(&ds_empty[st]);
      int* parts = red + st * 4 * GM;
      parts[h * GM + r] = row_exponent(wv);
      named_bar(2 + quarter, 32 * kGroups);
      const int ew = row_maximum(parts, r);
      cut_digits(wv, ew, chunk);
      return ew;
    };
    auto put = [&]() {
      store_digits(chunk, sP, r, h * CW);
      fence_proxy_async();
      __syncwarp();
      if (lane == 0) mbar_arrive(p_full);
    };
    int ew = 0, ew_next = 0;
    if (kQ && n_tiles > 0) {
      ew_next = cut(0);
      put();
    }
    for (int it = 0; it < n_tiles; it++) {
      const int st = it & 1;
      const uint32_t par = (uint32_t)(it & 1);
      if (kQ) {
        ew = ew_next;
        if (it + 1 < n_tiles) ew_next = cut(it + 1);
      } else {
        wait(&kv_full[st], (uint32_t)((it >> 1) & 1));
        ew = ((const int*)(sB + st * Sh::kStage + Sh::kB3))[r];
        __syncwarp();
        if (lane == 0) mbar_arrive(&kv_empty[st]);
      }
      wait(o_full, par);
      tc_fence_after();
      add_levels(lane_addr, sum_addr, h * CW, ew, e3_s + h * CW, e3lo, e3hi, it == 0);
      tmem_wait_st();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(tmem_free);
      if (kQ && it + 1 < n_tiles) put();  // (the tile's MMAs have read its digits)
    }
    tc_fence_after();
    const bool store = valid && !*(volatile int*)failed;
    double* orow = a.out + (r_base + rl) * a.dy;
#pragma unroll
    for (int c4 = 0; c4 < CW / 4; c4++) {
      uint32_t sum[8];
      if (n_tiles > 0) {
        tmem_ld8(sum_addr + c4 * 8, (int32_t*)sum);
        tmem_wait_ld();
      }
#pragma unroll
      for (int i = 0; i < 4; i++) {
        const int64_t y = (int64_t)a.y0 + h * CW + c4 * 4 + i;
        const double v = n_tiles > 0 ? __hiloint2double((int)sum[2 * i + 1], (int)sum[2 * i]) : 0.0;
        if (store && y < a.dy) orow[y] = a.out_factor * v;
      }
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem, 512);
  }
}

// The same tiles in FP64 on the CUDA cores: 64 rows by 64 outputs per CTA,
// a 4 x 4 block of (row, output) per thread.
constexpr int FT = 64;
struct GradFp64Args {
  Mask mask;
  int64_t lr, lc, d1, d2, dy;  // rows, columns per batch; widths of products 1, 2 and the values
  double scale, out_factor;
  const double* a1;  // [w·lr + r][d1]
  const double* b1;  // [w·lc + c][d1]
  const double* a2;  // [w·lr + r][d2]
  const double* b2;  // [w·lc + c][d2]
  const double* b3;  // [w·lc + c][dy]
  const double* lse;
  const double* dd;
  double* out;  // [w·lr + r][dy]
};

constexpr size_t kFp64Smem = sizeof(double) * (FT * (FT + 1) + 2 * 32 * (FT + 1));

template <int MODE>
__global__ void __launch_bounds__(256) grad_fp64(const GradFp64Args a) {
  extern __shared__ __align__(16) unsigned char smem_fp64[];
  double(*blk)[FT + 1] = reinterpret_cast<double(*)[FT + 1]>(smem_fp64);
  double(*sa)[FT + 1] = reinterpret_cast<double(*)[FT + 1]>(smem_fp64 + sizeof(double) * FT * (FT + 1));
  double(*sb)[FT + 1] = sa + 32;
  __shared__ int s_lo[FT], s_hi[FT];
  __shared__ long long s_first, s_last;
  const int t = threadIdx.x, tx = t & 15, ty = t >> 4;
  const int w = blockIdx.z;
  const int64_t r0 = (int64_t)blockIdx.x * FT, y0 = (int64_t)blockIdx.y * FT;
  const int64_t r_base = (int64_t)w * a.lr, c_base = (int64_t)w * a.lc;
  const int rows = (int)std::min<int64_t>(FT, a.lr - r0);
  if (t == 0) {
    s_first = LLONG_MAX;
    s_last = LLONG_MIN;
  }
  __syncthreads();
  if (t < FT) {
    int lo = 0, hi = 0;
    if (t < rows) {
      int64_t l, h;
      allowed(a.mask, r_base + r0 + t, l, h);
      lo = (int)(l - c_base);
      hi = (int)(h - c_base);
      if (lo < hi) {
        atomicMin(&s_first, (long long)lo);
        atomicMax(&s_last, (long long)hi);
      }
    }
    s_lo[t] = lo;
    s_hi[t] = hi;
  }
  __syncthreads();
  const long long first = s_first, last = s_last;
  double acc[4][4] = {};
  // Σ_e A[r][e] B[c][e] for this thread's 4 x 4 (row, column) pairs.
  auto product = [&](const double* A, const double* B, int64_t dk, int64_t c0, int width, double (&o)[4][4]) {
    for (int i = 0; i < 4; i++)
      for (int j = 0; j < 4; j++) o[i][j] = 0.0;
    for (int64_t e0 = 0; e0 < dk; e0 += 32) {
      const int ec = (int)std::min<int64_t>(32, dk - e0);
      for (int idx = t; idx < FT * 32; idx += 256) {
        const int rr = idx >> 5, e = idx & 31;
        sa[e][rr] = (rr < rows && e < ec) ? A[(r_base + r0 + rr) * dk + e0 + e] : 0.0;
        sb[e][rr] = (rr < width && e < ec) ? B[(c_base + c0 + rr) * dk + e0 + e] : 0.0;
      }
      __syncthreads();
      for (int e = 0; e < ec; e++)
        for (int i = 0; i < 4; i++)
          for (int j = 0; j < 4; j++) o[i][j] = fma(sa[e][ty + 16 * i], sb[e][tx + 16 * j], o[i][j]);
      __syncthreads();
    }
  };
  for (long long c0 = first < last ? first - first % FT : 0; c0 < last; c0 += FT) {
    const int width = (int)std::min<long long>(FT, a.lc - c0);
    double s[4][4];
    product(a.a1, a.b1, a.d1, c0, width, s);
    double dp[4][4];
    if (MODE != GRAD_V) product(a.a2, a.b2, a.d2, c0, width, dp);
    for (int i = 0; i < 4; i++)
      for (int j = 0; j < 4; j++) {
        const int rr = ty + 16 * i, cc = tx + 16 * j;
        const int64_t cl = c0 + cc;
        double wgt = 0.0;
        if (rr < rows && cc < width && cl >= s_lo[rr] && cl < s_hi[rr]) {
          const int64_t xq = MODE == GRAD_Q ? r_base + r0 + rr : c_base + cl;
          wgt = exp(a.scale * s[i][j] - a.lse[xq]);
          if (MODE != GRAD_V) wgt = wgt * (dp[i][j] - a.dd[xq]);
        }
        blk[rr][cc] = wgt;
      }
    __syncthreads();
    for (int cc = 0; cc < width; cc++) {
      double bv[4];
      for (int j = 0; j < 4; j++) {
        const int64_t y = y0 + tx + 16 * j;
        bv[j] = y < a.dy ? a.b3[(c_base + c0 + cc) * a.dy + y] : 0.0;
      }
      for (int i = 0; i < 4; i++) {
        const double wgt = blk[ty + 16 * i][cc];
        for (int j = 0; j < 4; j++) acc[i][j] = fma(wgt, bv[j], acc[i][j]);
      }
    }
    __syncthreads();
  }
  for (int i = 0; i < 4; i++) {
    const int rr = ty + 16 * i;
    if (rr >= rows) continue;
    for (int j = 0; j < 4; j++) {
      const int64_t y = y0 + tx + 16 * j;
      if (y < a.dy) a.out[(r_base + r0 + rr) * a.dy + y] = a.out_factor * acc[i][j];
    }
  }
}

// D_x = Σ_y d_out[x][y] · out[x][y], a warp per row.
__global__ void row_dots(int64_t n, int64_t dv, const double* __restrict__ d_out, const double* __restrict__ out,
                         double* __restrict__ dd) {
  const int lane = threadIdx.x & 31;
  for (int64_t x = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5; x < n;
       x += ((int64_t)gridDim.x * blockDim.x) >> 5) {
    double s = 0.0;
    for (int64_t y = lane; y < dv; y += 32) s = fma(d_out[x * dv + y], out[x * dv + y], s);
    for (int o = 16; o; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    if (lane == 0) dd[x] = s;
  }
}

inline int64_t round_up(int64_t x, int64_t m) { return (x + m - 1) / m * m; }

// Each block of 128 rows' first column tile and number of tiles, a warp a
// block; with `off`, also where its tiles go, `stride` tiles a block (for
// exports small enough to hold every block's most). A thread a block took 31 us
// at any size, a warp takes 3 to 4.
__global__ void __launch_bounds__(128) export_plan(Mask m, int64_t lr, int64_t lc, int64_t batches, int64_t blocks,
                                                   int32_t* __restrict__ ct0, int32_t* __restrict__ n,
                                                   int64_t* __restrict__ off, int64_t stride) {
  const int lane = threadIdx.x & 31;
  for (int64_t x = ((int64_t)blockIdx.x * 128 + threadIdx.x) >> 5; x < batches * blocks; x += (int64_t)gridDim.x * 4) {
    const int64_t w = x / blocks, b = x - w * blocks;
    int first = INT_MAX, last = INT_MIN;  // positions are below 2^30
    for (int64_t r = b * GM + lane; r < min(lr, b * GM + GM); r += 32) {
      int64_t lo, hi;
      allowed(m, w * lr + r, lo, hi);
      if (lo < hi) {
        first = min(first, (int)(lo - w * lc));
        last = max(last, (int)(hi - w * lc));
      }
    }
    first = __reduce_min_sync(0xffffffffu, first);
    last = __reduce_max_sync(0xffffffffu, last);
    if (lane == 0) {
      ct0[x] = first < last ? first / GJ : 0;
      n[x] = first < last ? (last + GJ - 1) / GJ - first / GJ : 0;
      if (off) off[x] = x * stride;
    }
  }
}

// The mask of keys as rows: each condition x <cmp> j + off as j <cmp'> x - off.
Mask transposed(const Mask& m) {
  static const int mirror[4] = {2, 3, 0, 1};
  Mask t;
  t.n = m.n;
  for (int i = 0; i < m.n; i++) {
    if (m.off[i] == INT64_MIN) fail(EINFOLD_INVALID, "a condition offset of -2^63 has no mirror");
    t.cmp[i] = mirror[m.cmp[i]];
    t.off[i] = -m.off[i];
  }
  t.lnx = m.lnj > 0 ? m.lnj : 1;
  t.lnj = m.lnx;
  t.xlen = m.jlen;
  t.jlen = m.xlen;
  return t;
}

// One operand's digits: rows (or columns) sliced, with exponents.
struct Digits {
  int8_t* d = nullptr;
  int32_t* e = nullptr;
};

template <int MODE>
void launch_split(const CUtensorMap* maps, const GradArgs& args, dim3 grid, bool fast, cudaStream_t stream) {
  using Sh = GradShape<MODE>;
  if (fast) {
    EF_CUDA(cudaFuncSetAttribute(grad_split<MODE, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, Sh::kSmem));
    grad_split<MODE, true><<<grid, kGradThreads, Sh::kSmem, stream>>>(maps[0], maps[1], maps[2], maps[3], maps[4],
                                                                       args);
  } else {
    EF_CUDA(cudaFuncSetAttribute(grad_split<MODE, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, Sh::kSmem));
    grad_split<MODE, false><<<grid, kGradThreads, Sh::kSmem, stream>>>(maps[0], maps[1], maps[2], maps[3], maps[4],
                                                                        args);
  }
  EF_LAUNCH_CHECK();
}

template <int MODE>
void launch_tiles(const CUtensorMap& tds, const CUtensorMap& tb3, const GradArgs& args, dim3 grid,
                  cudaStream_t stream) {
  using Sh = TileShape<MODE>;
  EF_CUDA(cudaFuncSetAttribute(grad_tiles<MODE>, cudaFuncAttributeMaxDynamicSharedMemorySize, Sh::kSmem));
  grad_tiles<MODE><<<grid, kGradThreads, Sh::kSmem, stream>>>(tds, tb3, args);
  EF_LAUNCH_CHECK();
}

// The split backward; false if it doesn't apply or an operand isn't finite (no
// gradient written). D = rowsum(d_out∘out) goes to dd where `*have_dd` is set on
// return.
bool backward_split(Context& ctx, const AttentionGradients& g, double* dd, bool* have_dd, cudaStream_t s) {
  const AttentionProblem& f = g.f;
  const int64_t W = f.batches, lq = f.lnx, lk = f.lnj, d = f.ne, dv = f.ny;
  if (d > 64 || dv > 64 || d <= 0 || dv <= 0 || lq <= 0 || lk <= 0) return false;
  if (lq > (1 << 30) || lk > (1 << 30) || W > 65535) return false;
  const int64_t lq_pad = round_up(lq, GM), lk_pad = round_up(lk, GM);
  auto al = [](size_t x) { return (x + 255) & ~(size_t)255; };
  // Row digits of q, k, v, d_out (64 B of features each) and column digits
  // of d_out, q, k (K-major along the batch's positions).
  const size_t rq = al((size_t)(W * S * lq_pad * 64)), rk = al((size_t)(W * S * lk_pad * 64));
  const size_t cq = al((size_t)(W * S * 64 * lq_pad)), ck = al((size_t)(W * S * 64 * lk_pad));
  const size_t eqs = al((size_t)(W * lq_pad) * 4), eks = al((size_t)(W * lk_pad) * 4), ecs = al((size_t)(W * 64) * 4);
  const size_t cm = al((size_t)(3 * W * 64) * 8), lp = al((size_t)(W * lq_pad) * 8);
  const size_t total = 2 * rq + 2 * rk + 2 * cq + ck + 2 * eqs + 2 * eks + 3 * ecs + cm + 2 * lp + 256;
  DeviceBuffer<uint8_t> scratch(total, s);
  uint8_t* p = scratch.get();
  auto take = [&](size_t n) {
    uint8_t* q = p;
    p += n;
    return q;
  };
  Digits Qr{(int8_t*)take(rq), nullptr}, dOr{(int8_t*)take(rq), nullptr}, Kr{(int8_t*)take(rk), nullptr},
      Vr{(int8_t*)take(rk), nullptr}, dOc{(int8_t*)take(cq), nullptr}, Qc{(int8_t*)take(cq), nullptr},
      Kc{(int8_t*)take(ck), nullptr};
  Qr.e = (int32_t*)take(eqs);
  dOr.e = (int32_t*)take(eqs);
  Kr.e = (int32_t*)take(eks);
  Vr.e = (int32_t*)take(eks);
  dOc.e = (int32_t*)take(ecs);
  Qc.e = (int32_t*)take(ecs);
  Kc.e = (int32_t*)take(ecs);
  double* lse_pad = (double*)take(lp);
  double* dd_pad = (double*)take(lp);
  unsigned long long* colmax = (unsigned long long*)take(cm);  // d_out's, q's, k's
  // [0] an operand isn't finite, [1] kernels, [2..9] (max e, max -e) of q's, k's,
  // v's and d_out's rows, [10..15] tile pairs of the three kernels
  int* status = (int*)take(256);
  unsigned long long* tiles = (unsigned long long*)(status + 10);
  EF_CUDA(cudaMemsetAsync(colmax, 0, cm + 64, s));  // and status behind it
  // Ragged batches: the padding rows are not read (their digits are zeros).
  auto row_set = [&](const double* x, int64_t rows, int64_t rows_pad, int64_t cols, const int64_t* lens,
                     const Digits& to, int range) {
    RowSet r;
    r.x = x;
    r.rows = rows;
    r.rows_pad = rows_pad;
    r.cols = cols;
    r.lens = lens;
    r.digits = to.d;
    r.e = to.e;
    r.range = status + 2 + 2 * range;
    return r;
  };
  const int64_t *xl = f.mask.xlen, *jl = f.mask.jlen;
  RowSet sets[4] = {row_set(f.q, lq, lq_pad, d, xl, Qr, 0), row_set(f.k, lk, lk_pad, d, jl, Kr, 1),
                    row_set(f.v, lk, lk_pad, dv, jl, Vr, 2), row_set(g.d_out, lq, lq_pad, dv, xl, dOr, 3)};
  sets[0].colmax = colmax + W * 64;
  sets[1].colmax = colmax + 2 * W * 64;
  sets[3].colmax = colmax;
  sets[3].other = g.out;
  sets[3].dots = dd;
  sets[3].dots_pad = dd_pad;
  sets[3].value = g.lse;
  sets[3].value_pad = lse_pad;
  prepare_rows(ctx, sets, 4, W, status, s);
  *have_dd = true;
  auto column_set = [&](const double* x, int64_t rows, int64_t rows_pad, int64_t cols, const int64_t* lens,
                        const unsigned long long* cmax, const Digits& to) {
    ColumnSet c;
    c.x = x;
    c.rows = rows;
    c.rows_pad = rows_pad;
    c.cols = cols;
    c.cols_pad = 64;
    c.lens = lens;
    c.colmax = cmax;
    c.digits = to.d;
    c.e = to.e;
    return c;
  };
  const ColumnSet columns[3] = {column_set(g.d_out, lq, lq_pad, dv, xl, sets[3].colmax, dOc),
                                column_set(f.q, lq, lq_pad, d, xl, sets[0].colmax, Qc),
                                column_set(f.k, lk, lk_pad, d, jl, sets[1].colmax, Kc)};
  prepare_columns(ctx, columns, 3, W, s);
  // Products 1 (q·k) and 2 (d_out·v) with normal powers of two 2^(e_r + e_c): the
  // tile kernels judge by themselves where their exports need no counting.
  Ready ready;
  ready.status = status;
  ready.pairs = 2;
  const double scale = std::fabs(f.scale_kind == 1 ? f.scale_c : 1.0);
  const int scale_exp = std::isnormal(scale) ? std::ilogb(scale) : 0;
  ready.top = std::isnormal(scale) ? 1023 - std::max(0, scale_exp) : INT_MIN / 2;
  ready.low = 1022 + kLevelUnit + std::min(0, scale_exp);
  int sts[16] = {};
  auto read_status = [&]() {
    ReadBack back(ctx, s);
    back.add(sts, status, 16);
    back.wait();
  };
  auto normal_powers = [&]() {
    Ready host = ready;
    host.status = sts;
    return host.ok();
  };
  ctx.phase("attention backward: sliced");
  auto rows_map = [&](const Digits& x, int64_t rows_pad, int box) {
    return digit_planes_map(x.d, 64, rows_pad, W * S, box, S);
  };
  auto cols_map = [&](const Digits& x, int64_t k_pad) { return digit_planes_map(x.d, k_pad, 64, W * S, GY, S); };
  const Mask keys_mask = transposed(f.mask);
  const double* table = exp_table(ctx.device);
  GradArgs args[3];
  CUtensorMap mode_maps[3][5];
  for (int mode = 0; mode < 3; mode++) {
    GradArgs& a = args[mode];
    a = GradArgs{};
    CUtensorMap* maps = mode_maps[mode];
    const bool keys = mode != GRAD_Q;
    a.mask = keys ? keys_mask : f.mask;
    a.lr = keys ? lk : lq;
    a.lc = keys ? lq : lk;
    a.lr_pad = keys ? lk_pad : lq_pad;
    a.lc_pad = keys ? lq_pad : lk_pad;
    a.scale = f.scale_kind == 1 ? f.scale_c : 1.0;
    a.lse = g.lse;
    a.dd = dd;
    a.lse_pad = lse_pad;
    a.dd_pad = dd_pad;
    a.exp_table = table;
    a.status = status + 1;
    a.tiles = tiles + mode;
    if (mode == GRAD_V) {
      maps[0] = rows_map(Kr, lk_pad, GM);
      maps[1] = rows_map(Qr, lq_pad, GJ);
      maps[2] = maps[0];
      maps[3] = maps[1];
      maps[4] = cols_map(dOc, lq_pad);
      a.e_a1 = Kr.e;
      a.e_b1 = Qr.e;
      a.e_b3 = dOc.e;
      a.dy = dv;
      a.out = g.d_v;
      a.out_factor = 1.0;
    } else if (mode == GRAD_K) {
      maps[0] = rows_map(Kr, lk_pad, GM);
      maps[1] = rows_map(Qr, lq_pad, GJ);
      maps[2] = rows_map(Vr, lk_pad, GM);
      maps[3] = rows_map(dOr, lq_pad, GJ);
      maps[4] = cols_map(Qc, lq_pad);
      a.e_a1 = Kr.e;
      a.e_b1 = Qr.e;
      a.e_a2 = Vr.e;
      a.e_b2 = dOr.e;
      a.e_b3 = Qc.e;
      a.dy = d;
      a.out = g.d_k;
      a.out_factor = a.scale;
    } else {
      maps[0] = rows_map(Qr, lq_pad, GM);
      maps[1] = rows_map(Kr, lk_pad, GJ);
      maps[2] = rows_map(dOr, lq_pad, GM);
      maps[3] = rows_map(Vr, lk_pad, GJ);
      maps[4] = cols_map(Kc, lk_pad);
      a.e_a1 = Qr.e;
      a.e_b1 = Kr.e;
      a.e_a2 = dOr.e;
      a.e_b2 = Vr.e;
      a.e_b3 = Kc.e;
      a.dy = d;
      a.out = g.d_q;
      a.out_factor = a.scale;
    }
    a.dy_pad = 64;
    a.y0 = 0;
    a.n_rb = a.lr_pad / GM;
    a.reverse = last_rows_longest(a.mask, a.lr);
  }
  // The tile path: d_k first, exporting P's digits and dS; then d_v and d_q
  // from them, one product a tile each. The exports cover only the tiles
  // some pair of is allowed (export_plan counts them per block), 14 bytes a
  // pair of those. Batches go in chunks whose exports fit the export limit
  // (EINFOLD_BACKWARD_EXPORT_MB, 4096 by default): all in one when they fit,
  // else in chunks of at most half of it in two buffers, the chunks
  // alternating between the call's stream and the context's second stream,
  // so that one chunk's kernels run beside the other's and a chunk's last
  // wave of blocks leaves no SM idle. The buffers are freed at the end of
  // the call. A batch whose exports alone exceed half the limit takes the
  // three kernels that each recompute the scores.
  const int64_t n_kb = lk_pad / GM, n_qb = lq_pad / GM;
  // Once the kernels have run and the status is read: their failures and counts.
  auto finish = [&](cudaEvent_t from, cudaEvent_t to, bool exported) {
    float ms = 0;
    cudaEventElapsedTime(&ms, from, to);
    cudaEventDestroy(from);
    cudaEventDestroy(to);
    if (sts[1] & 2) fail(EINFOLD_TIMEOUT, "a bounded wait in the attention backward ran out");
    // Digit products executed: per pair of tiles, S(S+1)/2 digit pairs of a
    // 128 x 64 x 64 product, three for d_k, and for d_v and d_q one on the
    // tile path (else two and three).
    unsigned long long pairs[3];
    std::memcpy(pairs, sts + 10, 24);
    ctx.product_ms += ms;
    const double per = (S * (S + 1) / 2) * 2.0 * GM * GJ * 64;
    const double pv = exported ? 1.0 : 2.0, pq = exported ? 1.0 : 3.0;
    ctx.product_ops += per * (pv * (double)pairs[0] + 3.0 * (double)pairs[1] + pq * (double)pairs[2]);
    ctx.phase("attention backward: tiles");
  };
  static const size_t limit = [] {
    const char* e = std::getenv("EINFOLD_BACKWARD_EXPORT_MB");
    const long long mb = e ? std::atoll(e) : 4096;
    return (size_t)std::max(0ll, mb) << 20;
  }();
  DeviceBuffer<int32_t> plan((size_t)(2 * W * (n_kb + n_qb)), s);
  int32_t* pk_ct0 = plan.get();
  int32_t* pk_n = pk_ct0 + W * n_kb;
  int32_t* pq_ct0 = pk_n + W * n_kb;
  int32_t* pq_n = pq_ct0 + W * n_qb;
  // Exports of at most kSmallExports whatever the mask joins: every block gets room
  // for its most tiles, and nothing needs counting before the kernels run (a wait
  // and four copies fewer: 232 to 189 us for 6 batches of 100 rows, 368 to 327 for
  // 16 of 512, 855 to 812 at 450 MB, 8 of 2048). Above, the gain is below 4% and
  // the room a causal mask leaves unused would grow with the batches.
  constexpr size_t kSmallExports = (size_t)512 << 20;
  const int64_t p_most = lq_pad / GJ, q_most = lk_pad / GJ;
  const double most = (double)W * ((double)n_kb * p_most * (kPTile + GM * 4) + (double)n_qb * q_most * GM * GJ * 8);
  const bool small = !g.budget && most <= (double)std::min(limit, kSmallExports);
  DeviceBuffer<int64_t> small_off;
  if (small) small_off.allocate((size_t)(W * (n_kb + n_qb)), s);
  int64_t* const pk_off = small_off.get();
  int64_t* const pq_off = small ? pk_off + W * n_kb : nullptr;
  export_plan<<<blocks_for((uint64_t)(W * n_kb), 4), 128, 0, s>>>(keys_mask, lk, lq, W, n_kb, pk_ct0, pk_n, pk_off,
                                                                 p_most);
  export_plan<<<blocks_for((uint64_t)(W * n_qb), 4), 128, 0, s>>>(f.mask, lq, lk, W, n_qb, pq_ct0, pq_n, pq_off, q_most);
  ctx.kernels += 2;
  EF_LAUNCH_CHECK();
  bool fast = true;
  cudaEvent_t e0, e1, joined = nullptr;
  if (small) {
    DeviceBuffer<uint8_t> exports((size_t)most + 512, s);
    EF_CUDA(cudaEventCreate(&e0));
    EF_CUDA(cudaEventCreate(&e1));
    auto run = [&]() {
      EF_CUDA(cudaEventRecord(e0, s));
      const int64_t np = W * n_kb * p_most, nq = W * n_qb * q_most;
      double* ds = (double*)exports.get();
      uint8_t* p_tiles = exports.get() + (size_t)nq * GM * GJ * 8;
      const CUtensorMap tds = f64_boxes_map(ds, GJ, nq * GM, 1, 16, GM);
      GradArgs k = args[GRAD_K], v = args[GRAD_V], q = args[GRAD_Q];
      for (GradArgs* g2 : {&k, &v, &q}) {
        g2->w0 = 0;
        g2->p_tiles = p_tiles;
        g2->p_exp = (int32_t*)(p_tiles + (size_t)np * kPTile);
        g2->p_off = pk_off;
        g2->dq_off = pq_off;
        g2->dq_ct0 = pq_ct0;
        g2->dq_n = pq_n;
        g2->n_rb = n_kb;
        g2->n_qb = n_qb;
        g2->ready = ready;
      }
      k.ds_out = ds;
      launch_split<GRAD_K>(mode_maps[GRAD_K], k, dim3((unsigned)n_kb, (unsigned)W), fast, s);
      launch_tiles<GRAD_V>(tds, mode_maps[GRAD_V][4], v, dim3((unsigned)n_kb, (unsigned)W), s);
      launch_tiles<GRAD_Q>(tds, mode_maps[GRAD_Q][4], q, dim3((unsigned)n_qb, (unsigned)W), s);
      ctx.kernels += 3;
      EF_CUDA(cudaEventRecord(e1, s));
    };
    run();
    read_status();
    if (sts[0]) {
      cudaEventDestroy(e0);
      cudaEventDestroy(e1);
      return false;
    }
    if (!normal_powers()) {  // the launches did nothing
      fast = false;
      ready.status = nullptr;
      run();
      read_status();
    }
    finish(e0, e1, true);
    return true;
  }
  std::vector<int32_t> hk_n((size_t)(W * n_kb)), hq_n((size_t)(W * n_qb));
  EF_CUDA(cudaMemcpyAsync(hk_n.data(), pk_n, hk_n.size() * 4, cudaMemcpyDeviceToHost, s));
  EF_CUDA(cudaMemcpyAsync(hq_n.data(), pq_n, hq_n.size() * 4, cudaMemcpyDeviceToHost, s));
  read_status();
  if (sts[0]) return false;
  fast = normal_powers();
  // Each block's first tile (exclusive over all batches), and each batch's tiles.
  std::vector<int64_t> hp_off((size_t)(W * n_kb) + 1), hq_off((size_t)(W * n_qb) + 1);
  for (size_t x = 0; x < hk_n.size(); x++) hp_off[x + 1] = hp_off[x] + hk_n[x];
  for (size_t x = 0; x < hq_n.size(); x++) hq_off[x + 1] = hq_off[x] + hq_n[x];
  constexpr size_t kDsBytes = (size_t)GM * GJ * 8;
  auto bytes_of = [&](int64_t w0, int64_t w1) {
    const int64_t np = hp_off[(size_t)(w1 * n_kb)] - hp_off[(size_t)(w0 * n_kb)];
    const int64_t nq = hq_off[(size_t)(w1 * n_qb)] - hq_off[(size_t)(w0 * n_qb)];
    return al((size_t)np * kPTile) + al((size_t)np * GM * 4) + (size_t)nq * kDsBytes;
  };
  // The chunks and buffers under a limit: one chunk when every batch's
  // exports fit it, else chunks of at most half of it in two buffers; none
  // when one batch's exports exceed half of it.
  std::vector<std::pair<int64_t, int64_t>> chunks;
  int buffers = 1;
  auto plan_under = [&](size_t lim) {
    chunks.clear();
    buffers = 1;
    if (bytes_of(0, W) <= lim) {
      chunks.push_back({0, W});
      return;
    }
    buffers = 2;
    int64_t w0 = 0;
    while (w0 < W) {
      if (bytes_of(w0, w0 + 1) > lim / 2) {
        chunks.clear();
        return;
      }
      int64_t w1 = w0 + 1;
      while (w1 < W && bytes_of(w0, w1 + 1) <= lim / 2) w1++;
      chunks.push_back({w0, w1});
      w0 = w1;
    }
  };
  auto biggest_chunk = [&]() {
    size_t b = 0;
    for (auto& c : chunks) b = std::max(b, bytes_of(c.first, c.second));
    return std::max<size_t>(b, 256);
  };
  // With a budget, the plan's buffers are asked of it, and a refusal halves
  // the limit until a plan is granted or none is left.
  struct Granted {
    Budget* budget = nullptr;
    uint64_t bytes = 0;
    ~Granted() {
      if (budget && bytes) budget->release(bytes);
    }
  } granted;
  for (size_t lim = limit;; lim /= 2) {
    plan_under(lim);
    if (chunks.empty() || !g.budget) break;
    const uint64_t want = (uint64_t)buffers * biggest_chunk();
    if (g.budget->try_reserve(want)) {
      granted.budget = g.budget;
      granted.bytes = want;
      break;
    }
    if (lim == 0) {
      chunks.clear();
      break;
    }
  }
  DeviceBuffer<int64_t> offs;
  if (!chunks.empty()) {
    offs.allocate(hp_off.size() + hq_off.size(), s);
    EF_CUDA(cudaMemcpyAsync(offs.get(), hp_off.data(), hp_off.size() * 8, cudaMemcpyHostToDevice, s));
    EF_CUDA(cudaMemcpyAsync(offs.get() + hp_off.size(), hq_off.data(), hq_off.size() * 8, cudaMemcpyHostToDevice, s));
  }
  const int64_t* p_off = offs.get();
  const int64_t* q_off = offs.get() + hp_off.size();
  DeviceBuffer<uint8_t> exports[2];
  cudaStream_t streams[2] = {s, s};
  EF_CUDA(cudaEventCreate(&e0));
  EF_CUDA(cudaEventCreate(&e1));
  EF_CUDA(cudaEventRecord(e0, s));
  if (!chunks.empty() && buffers == 2) {
    if (!ctx.aux) EF_CUDA(cudaStreamCreateWithFlags(&ctx.aux, cudaStreamNonBlocking));
    streams[1] = ctx.aux;
    EF_CUDA(cudaEventCreateWithFlags(&joined, cudaEventDisableTiming));
    EF_CUDA(cudaEventRecord(joined, s));  // the slicing above, before the second stream starts
    EF_CUDA(cudaStreamWaitEvent(ctx.aux, joined, 0));
  }
  if (!chunks.empty()) {
    const size_t biggest = biggest_chunk();
    for (int b = 0; b < buffers; b++) exports[b].allocate(biggest, streams[b]);
    for (size_t c = 0; c < chunks.size(); c++) {
      const int b = (int)(c % (size_t)buffers);
      cudaStream_t st = streams[b];
      const int64_t w0 = chunks[c].first, w1 = chunks[c].second;
      const int64_t np = hp_off[(size_t)(w1 * n_kb)] - hp_off[(size_t)(w0 * n_kb)];
      const int64_t nq = hq_off[(size_t)(w1 * n_qb)] - hq_off[(size_t)(w0 * n_qb)];
      uint8_t* p_tiles = exports[b].get();
      int32_t* p_exp = (int32_t*)(p_tiles + al((size_t)np * kPTile));
      double* ds = (double*)((uint8_t*)p_exp + al((size_t)np * GM * 4));
      const CUtensorMap tds = f64_boxes_map(ds, GJ, std::max<int64_t>(nq, 1) * GM, 1, 16, GM);
      const unsigned wc = (unsigned)(w1 - w0);
      GradArgs k = args[GRAD_K], v = args[GRAD_V], q = args[GRAD_Q];
      for (GradArgs* g2 : {&k, &v, &q}) {
        g2->w0 = (int)w0;
        g2->p_tiles = p_tiles;
        g2->p_exp = p_exp;
        g2->p_off = p_off + w0 * n_kb;
        g2->p_base = hp_off[(size_t)(w0 * n_kb)];
        g2->dq_off = q_off + w0 * n_qb;
        g2->dq_ct0 = pq_ct0 + w0 * n_qb;
        g2->dq_n = pq_n + w0 * n_qb;
        g2->dq_base = hq_off[(size_t)(w0 * n_qb)];
        g2->n_rb = n_kb;
        g2->n_qb = n_qb;
      }
      k.ds_out = ds;
      launch_split<GRAD_K>(mode_maps[GRAD_K], k, dim3((unsigned)n_kb, wc), fast, st);
      launch_tiles<GRAD_V>(tds, mode_maps[GRAD_V][4], v, dim3((unsigned)n_kb, wc), st);
      launch_tiles<GRAD_Q>(tds, mode_maps[GRAD_Q][4], q, dim3((unsigned)n_qb, wc), st);
      ctx.kernels += 3;
    }
    if (joined) {
      EF_CUDA(cudaEventRecord(joined, ctx.aux));  // the second stream's chunks, before the call's stream goes on
      EF_CUDA(cudaStreamWaitEvent(s, joined, 0));
    }
  } else {
    for (int mode = 0; mode < 3; mode++) {
      const dim3 grid((unsigned)(args[mode].lr_pad / GM), (unsigned)W);
      if (mode == GRAD_V) launch_split<GRAD_V>(mode_maps[mode], args[mode], grid, fast, s);
      else if (mode == GRAD_K) launch_split<GRAD_K>(mode_maps[mode], args[mode], grid, fast, s);
      else launch_split<GRAD_Q>(mode_maps[mode], args[mode], grid, fast, s);
      ctx.kernels++;
    }
  }
  EF_CUDA(cudaEventRecord(e1, s));
  read_status();
  if (joined) cudaEventDestroy(joined);
  finish(e0, e1, !chunks.empty());
  return true;
}

void backward_fp64(Context& ctx, const AttentionGradients& g, const double* dd, cudaStream_t s) {
  const AttentionProblem& f = g.f;
  const int64_t W = f.batches, lq = f.lnx, lk = f.lnj, d = f.ne, dv = f.ny;
  const Mask keys_mask = transposed(f.mask);
  for (int mode = 0; mode < 3; mode++) {
    GradFp64Args a{};
    const bool keys = mode != GRAD_Q;
    a.mask = keys ? keys_mask : f.mask;
    a.lr = keys ? lk : lq;
    a.lc = keys ? lq : lk;
    a.scale = f.scale_kind == 1 ? f.scale_c : 1.0;
    a.lse = g.lse;
    a.dd = dd;
    if (mode == GRAD_V) {
      a.a1 = f.k; a.b1 = f.q; a.d1 = d; a.b3 = g.d_out; a.dy = dv; a.out = g.d_v; a.out_factor = 1.0;
    } else if (mode == GRAD_K) {
      a.a1 = f.k; a.b1 = f.q; a.d1 = d; a.a2 = f.v; a.b2 = g.d_out; a.d2 = dv; a.b3 = f.q; a.dy = d;
      a.out = g.d_k; a.out_factor = a.scale;
    } else {
      a.a1 = f.q; a.b1 = f.k; a.d1 = d; a.a2 = g.d_out; a.b2 = f.v; a.d2 = dv; a.b3 = f.k; a.dy = d;
      a.out = g.d_q; a.out_factor = a.scale;
    }
    if (a.lr == 0 || a.dy == 0 || W == 0) continue;
    const dim3 grid((unsigned)((a.lr + FT - 1) / FT), (unsigned)((a.dy + FT - 1) / FT), (unsigned)W);
    if (mode == GRAD_V) {
      EF_CUDA(cudaFuncSetAttribute(grad_fp64<GRAD_V>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kFp64Smem));
      grad_fp64<GRAD_V><<<grid, 256, kFp64Smem, s>>>(a);
    } else if (mode == GRAD_K) {
      EF_CUDA(cudaFuncSetAttribute(grad_fp64<GRAD_K>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kFp64Smem));
      grad_fp64<GRAD_K><<<grid, 256, kFp64Smem, s>>>(a);
    } else {
      EF_CUDA(cudaFuncSetAttribute(grad_fp64<GRAD_Q>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kFp64Smem));
      grad_fp64<GRAD_Q><<<grid, 256, kFp64Smem, s>>>(a);
    }
    EF_LAUNCH_CHECK();
    ctx.kernels++;
  }
  EF_CUDA(cudaStreamSynchronize(s));
  ctx.phase("attention backward: fp64 tiles");
}

}  // namespace

void attention_backward(Context& ctx, const AttentionGradients& g, int precision, cudaStream_t s) {
  const AttentionProblem& f = g.f;
  const int64_t W = f.batches, lq = f.lnx;
  if (W <= 0) return;
  if (W > 65535) fail(EINFOLD_INVALID, "more than 65535 batches");
  DeviceBuffer<double> dd((size_t)std::max<int64_t>(W * lq, 1), s);
  bool have_dd = false;
  if (precision == 0 && backward_split(ctx, g, dd.get(), &have_dd, s)) return;
  if (W * lq > 0 && !have_dd) {
    row_dots<<<blocks_for((uint64_t)(W * lq) * 32, 256), 256, 0, s>>>(W * lq, f.ny, g.d_out, g.out, dd.get());
    EF_LAUNCH_CHECK();
    ctx.kernels++;
  }
  if (backward_f64_mma(ctx, g, transposed(f.mask), dd.get(), s)) return;
  backward_fp64(ctx, g, dd.get(), s);
}

}  // namespace ef
