// The split forward pass of an attention-shaped pipeline on the B200: the
// tile of fused.rs:694-1019 for product scores, a softmax shifted by the
// running maximum and a normalised average, with both products on the
// tensor cores.
//
// A CTA owns 128 query rows of one batch and walks the batch's key tiles of
// 64 that its rows may join. Per tile:
//   1. q·k: the rows' and keys' S int8 digit planes (sliced once, staged by
//      TMA) multiply on tcgen05 kind::i8, each digit s of q against digits
//      1..S+1-s of k stacked along N, so that digit pair (s, t) accumulates
//      in TMEM columns (s + t - 2)·64: level l's exact int32 sum.
//   2. Sixteen epilogue warps read the levels (a row per TMEM lane, a
//      quarter of the columns per warp group), combine them in FP64 under
//      the row's and key's powers of two, apply the mask, update the running
//      maximum (shared between the quarters), and turn the weights
//      exp(s - m) in [0, 1] into S digit planes of a fixed scale 2^2,
//      written to shared memory in the MMA's 64-byte swizzle.
//   3. w·v: the weights' digits against v's column-scaled digits, the same
//      level scheme, into the same TMEM columns (q·k's levels were read).
//   4. The epilogue rescales the row's FP64 running sums and adds the
//      levels to them, in units of each value column's power of two (applied
//      once, at the end). The sums live in the 128 TMEM columns the six
//      slices' 384 level columns leave free, two 32-bit columns a value, so
//      that a thread's registers hold only its 16 scores.
// The four warps sharing a row exchange its maximum over a named barrier of
// their own; every other hand-off is an mbarrier each warp arrives on.
// A TMA producer warp double-buffers k and v tiles; an MMA warp issues both
// products, each beside epilogue work that needs none of the levels: the next
// tile's q·k while the second half of this tile's exponentials are taken, a
// tile's w·v while the first half of the next one's are. Every wait is bounded (2 s); on a timeout the kernel sets a
// status bit, waits for its copies and MMAs in flight, frees TMEM and
// returns.
//
// Bound by the epilogue's instructions: some 100 a score, a quarter of them FP64,
// which share their pipe with the MMAs (FP64 20% of it and the MMAs 19% at 8 x
// 2048 x 64, issue slots 46%), so that running them side by side gives little
// (3.29 to 3.19 ms at 64 x 4096 x 64, and 3.58 with 130 instructions a score).
// Eight warps of 32 columns in place of sixteen: 3.36 ms.
//
// Launch forms: a block per (query tile, batch) item, or persistent blocks
// (one an SM) that claim the items of a work list in its order from a
// counter, keeping their barriers and TMEM across items: the barriers'
// phases count the block's key tiles and q loads since the launch.
//
// Accuracy: each operand value carries 8S - 2 bits under its row's (or
// column's) power of two, levels above S + 1 are dropped, and every level
// sum is exact, so a score's error is about ne · 2^(3-8S) · max|q| · max|k|
// and a weight's about 2^(1-8S): with S = 6, scores to ~1e-14 of their scale
// and averages to ~1e-14 of max|v|.
#include <algorithm>
#include <cmath>
#include <cstdlib>
#include <cstring>
#include <map>
#include <memory>
#include <mutex>

#include "attention.cuh"
#include "fastexp.cuh"
#include "gemm.cuh"
#include "levels.cuh"
#include "prepare.cuh"
#include "ptx.cuh"

namespace ef {
namespace {

using namespace ptx;

constexpr int AM = 128;  // query rows per CTA (TMEM lanes)
constexpr int AJ = 64;   // key positions per tile
constexpr int AY = 64;   // value columns per CTA
constexpr int CW = 16;            // columns an epilogue thread takes of its row
constexpr int kGroups = 64 / CW;  // groups of four epilogue warps, a row per TMEM lane
constexpr int kEpi = 128 * kGroups;
constexpr int kAttnThreads = 64 + kEpi;
constexpr int kSumCol = 384;  // TMEM columns of the rows' FP64 running sums, two per value
constexpr int kMaxSmem = 232448;

template <int S, int KB>
struct AttnShape {
  static constexpr int kQ = KB * S * AM * 64;  // q digits [kb][s][128][64 B]
  static constexpr int kK = KB * S * AJ * 64;  // k digits per stage [kb][t][64][64 B]
  static constexpr int kV = S * AY * 64;       // v digits per stage [t][64 y][64 B of j]
  static constexpr int kP = S * AM * 64;       // weight digits [s][128][64 B of j]
  static constexpr int kAux = 8192;            // barriers, row spans, exponents, exchanges
  static constexpr int kFixed = kQ + kP + kAux + 1024;
  static constexpr int kStages = kFixed + 2 * (kK + kV) <= kMaxSmem ? 2 : 1;
  static constexpr int kSmem = kFixed + kStages * (kK + kV);
  static_assert(kSmem <= kMaxSmem, "the tiles must fit in shared memory");
  static_assert(S * 64 <= kSumCol, "the levels and the running sums must fit in TMEM");
};

struct AttnArgs {
  Mask mask;
  int64_t lnx, lnj, lnx_pad, lnj_pad, ny, ny_pad;
  int y0;
  int scale_kind;
  double scale_c;
  const int32_t* eq;  // [w][lnx_pad]
  const int32_t* ek;  // [w][lnj_pad]
  const int32_t* ev;  // [w][ny_pad]
  const double* rl;   // [w·lnx + x]: the largest magnitude of the values the row weighs
  const double* rs;   // and the smallest nonzero one (+inf if none)
  const double* exp_table;
  double* out;  // [w·lnx + x][ny]
  double* lse;  // [w·lnx + x] or null
  int* status;  // bit 0: a guard fired; bit 1: a wait ran out; bit 2: only exact maxima tell (FAST)
  unsigned long long* tiles;  // (row tile, key tile) pairs computed
  const int2* items;  // a work list of (query tile, batch) items; null: the grid's (x: tile, y: batch)
  int n_items;
  // Persistent blocks: the next item of the list no block has claimed (zero
  // at the launch). Null: block i runs items[i].
  unsigned* next;
  int reverse;        // the grid's query tiles from the last one (whose rows join the most keys) down
  Ready ready;        // judged first: a launch that may not run does nothing
};

// The S levels of this thread's 4 TMEM columns at `col`, on their way.
template <int S>
__device__ __forceinline__ void load_levels(uint32_t lane_addr, int col, int32_t (&L)[S][4]) {
#pragma unroll
  for (int l = 0; l < S; l++) tmem_ld4(lane_addr + (uint32_t)(l * 64 + col), L[l]);
}
template <int S>
__device__ __forceinline__ void landed(int32_t (&L)[S][4]) {
#pragma unroll
  for (int l = 0; l < S; l++) tmem_landed(L[l]);
}

// The sum of a score's levels in units of 2^kScoreUnit<KB>.
template <int KB>
constexpr int kScoreUnit = KB == 1 ? kLevelUnit : 0;
template <int S, int KB>
__device__ __forceinline__ double level_sum(const int32_t (&L)[S][4], int i) {
  // Level sums of products over 64 values of k fit the int32 pairs.
  if constexpr (KB == 1) return combine_levels_small(L, i);
  else return combine_levels<S, 4>(L, i);
}

// A double's high word as a float: orders as the doubles do (sign and
// magnitude), within their high words, for magnitudes below 2^1016; -inf reads
// as a NaN, which fmaxf and fminf pass over. One instruction a value (or half
// of one) where a double's maximum takes three.
__device__ __forceinline__ float high_float(double x) { return __int_as_float(__double2hiint(x)); }
// The least double no smaller, the largest no larger than any of that high word.
__device__ __forceinline__ double high_above(float f) {
  const int h = __float_as_int(f);
  return __hiloint2double(h, ~(h >> 31));
}
__device__ __forceinline__ double high_below(float f) {
  const int h = __float_as_int(f);
  return __hiloint2double(h, h >> 31);
}
constexpr float kLowestFloat = -3.4028234663852886e38f;

// The high word of 1024, from which on a running maximum is taken exactly.
constexpr float kExactHigh = 4.5f;  // 0x40900000

// FAST: every q row's and k row's exponents keep a score's power of two (times
// the scale) a normal double and the scaled scores below 2^1016. The running
// maximum and the lightest score are then bounds taken from the scores' high words
// (above by at most 2^-20 of it, below likewise). The shift by the maximum cancels
// in the quotient of doubles, but the weights are cut to 46 bits once shifted: a
// bound x above the maximum costs them x·log2(e) bits. So a maximum of 1024 or more
// in magnitude is taken exactly, by a second exchange of its low word (a bound 2^-20
// of 1e8 above it left no digit of any weight; below 1024 it is 2^-10 at most, a
// seven-hundredth of a bit). That costs ordinary tiles a vote (a training step of 64
// x 4096 x 64, causal, 12.9 ms with and without). A row whose guards hold under one
// end of the bounds and not under the other asks for the variant that keeps both
// exactly (status bit 2).
template <int S, int KB, bool FAST>
__global__ void __launch_bounds__(kAttnThreads, 1)
    attn_fwd_split(const __grid_constant__ CUtensorMap tq, const __grid_constant__ CUtensorMap tk,
                   const __grid_constant__ CUtensorMap tv, const AttnArgs a) {
  using Sh = AttnShape<S, KB>;
  extern __shared__ uint8_t smem_raw[];
  if (!a.ready.ok()) return;  // the same for every thread
  uint8_t* smem = (uint8_t*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  uint8_t* sQ = smem;
  uint8_t* sP = sQ + Sh::kQ;
  uint8_t* sK = sP + Sh::kP;
  uint8_t* sV = sK + Sh::kStages * Sh::kK;
  uint8_t* aux = sV + Sh::kStages * Sh::kV;
  uint64_t* bars = (uint64_t*)aux;  // 16 barriers
  uint64_t* q_full = bars + 0;
  uint64_t* k_full = bars + 1;   // [2]
  uint64_t* k_empty = bars + 3;  // [2]
  uint64_t* v_full = bars + 5;   // [2]
  uint64_t* v_empty = bars + 7;  // [2]
  uint64_t* qk_full = bars + 9;
  uint64_t* s_free = bars + 10;  // a tile's scores are read
  uint64_t* p_full = bars + 11;  // its weights' digits written
  uint64_t* pv_full = bars + 12;
  uint64_t* o_free = bars + 13;  // its weighted values are read
  uint32_t* tmem_slot = (uint32_t*)(bars + 16);
  int* failed = (int*)(tmem_slot + 1);
  int* item_slot = (int*)(tmem_slot + 2);         // the item the block runs next
  long long* span = (long long*)(tmem_slot + 4);  // first, last
  int* row_lo = (int*)(aux + 256);                // [128]
  int* row_hi = row_lo + AM;                      // [128]
  int* ev_s = row_hi + AM;                        // [64]
  double* texp = (double*)(aux + 2048);           // [64]
  // [4][64], tiles' key exponents: a tile's are read after its product frees its
  // stage for another, so they go round in four.
  int* ek_s = (int*)(aux + 2560);
  double* red = (double*)(aux + 4096);            // [4][128]; FAST: floats [2][4][128]

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;

  if (threadIdx.x == 0) {
    mbar_init(q_full, 1);
    for (int i = 0; i < 2; i++) {
      mbar_init(&k_full[i], 1);
      mbar_init(&k_empty[i], 1);
      mbar_init(&v_full[i], 1);
      mbar_init(&v_empty[i], 1);
    }
    mbar_init(qk_full, 1);
    mbar_init(pv_full, 1);
    mbar_init(s_free, kEpi / 32);  // each epilogue warp arrives
    mbar_init(p_full, kEpi / 32);
    mbar_init(o_free, kEpi / 32);
    *failed = 0;
    mbar_fence_init();
  }
  if (warp == 1) {
    tmem_alloc(tmem_slot, 512);
    tmem_relinquish();
  }
  if (threadIdx.x < 64) texp[threadIdx.x] = a.exp_table[threadIdx.x];
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *tmem_slot;
  // The barriers' completed phases before the current item: one per key
  // tile (the k and v ones by stage) and one per q load.
  int tiles_before = 0, q_loads = 0;
  for (int round_ = 0;; round_++) {
    if (threadIdx.x == 0) {
      *item_slot = a.next ? (int)atomicAdd(a.next, 1u) : round_ == 0 ? 0 : INT_MAX;
      span[0] = LLONG_MAX;
      span[1] = LLONG_MIN;
    }
    __syncthreads();
    // Every thread reads the same item and failure flag: all leave together.
    const int item = *item_slot;
    if (*(volatile int*)failed || item >= (a.next ? a.n_items : 1)) break;
    // The longest rows of a causal mask first; work lists in their order.
    int xt, w;
    if (a.items) {
      const int2 wk = a.items[a.next ? item : (int)blockIdx.x];
      xt = wk.x;
      w = wk.y;
    } else {
      xt = a.reverse ? (int)(gridDim.x - 1 - blockIdx.x) : (int)blockIdx.x;
      w = (int)blockIdx.y;
    }
    const int64_t x_base = (int64_t)w * a.lnx;
    // Each row's allowed keys, local to the batch.
    if (threadIdx.x < AM) {
      const int64_t xl = (int64_t)xt * AM + threadIdx.x;
      int lo = 0, hi = 0;
      if (xl < a.lnx) {
        int64_t l, h;
        allowed(a.mask, x_base + xl, l, h);
        lo = (int)(l - (int64_t)w * a.lnj);
        hi = (int)(h - (int64_t)w * a.lnj);
        if (lo < hi) {
          atomicMin(&span[0], (long long)lo);
          atomicMax(&span[1], (long long)hi);
        }
      }
      row_lo[threadIdx.x] = lo;
      row_hi[threadIdx.x] = hi;
    } else if (threadIdx.x < AM + AY) {
      const int c = threadIdx.x - AM;
      ev_s[c] = a.y0 + c < a.ny_pad ? a.ev[(int64_t)w * a.ny_pad + a.y0 + c] : 0;
    }
    __syncthreads();
    const long long first = span[0], last = span[1];
    const int jt0 = first < last ? (int)(first / AJ) : 0;
    const int n_tiles = first < last ? (int)((last + AJ - 1) / AJ) - jt0 : 0;
    if (threadIdx.x == 0 && n_tiles > 0) atomicAdd(a.tiles, (unsigned long long)n_tiles);

    if (warp == 0) {
      if (lane == 0 && n_tiles > 0) {
        // Producer: q's digits once, then k's and v's per tile, with the
        // keys' exponents.
        prefetch_map(&tq);
        prefetch_map(&tk);
        prefetch_map(&tv);
        mbar_expect_tx(q_full, (uint32_t)Sh::kQ);
        for (int kb = 0; kb < KB; kb++) tma_load_3d(sQ + kb * S * AM * 64, &tq, q_full, kb * 64, xt * AM, w * S);
        // k's digits run a tile ahead of v's: the next scores are computed
        // while this tile's weights are.
        int k_issued = 0, v_issued = 0;
        auto slot = [&](uint64_t* empty, int g) {
          if (*(volatile int*)failed) return false;
          if (mbar_wait(&empty[g % Sh::kStages], ((uint32_t)(g / Sh::kStages) & 1) ^ 1)) return true;
          atomicOr(a.status, 2);
          *(volatile int*)failed = 1;
          return false;
        };
        auto load_k = [&](int it) {
          const int g = tiles_before + it, st = g % Sh::kStages, jl0 = (jt0 + it) * AJ;
          if (!slot(k_empty, g)) return false;
          mbar_expect_tx(&k_full[st], (uint32_t)(Sh::kK + AJ * 4));
          for (int kb = 0; kb < KB; kb++)
            tma_load_3d(sK + st * Sh::kK + kb * S * AJ * 64, &tk, &k_full[st], kb * 64, jl0, w * S);
          bulk_load(ek_s + (g & 3) * AJ, a.ek + (int64_t)w * a.lnj_pad + jl0, AJ * 4, &k_full[st]);
          k_issued = it + 1;
          return true;
        };
        auto load_v = [&](int it) {
          const int g = tiles_before + it, st = g % Sh::kStages;
          if (!slot(v_empty, g)) return false;
          mbar_expect_tx(&v_full[st], (uint32_t)Sh::kV);
          tma_load_3d(sV + st * Sh::kV, &tv, &v_full[st], (jt0 + it) * AJ, a.y0, w * S);
          v_issued = it + 1;
          return true;
        };
        bool ok = load_k(0);
        for (int it = 0; ok && it < n_tiles; it++) ok = (it + 1 == n_tiles || load_k(it + 1)) && load_v(it);
        // Copies still in flight complete before the item ends.
        mbar_wait(q_full, (uint32_t)(q_loads & 1));
        auto drain = [&](uint64_t* full, int issued) {
          for (int it = std::max(0, issued - Sh::kStages); it < issued; it++) {
            const int g = tiles_before + it;
            mbar_wait(&full[g % Sh::kStages], (uint32_t)((g / Sh::kStages) & 1));
          }
        };
        drain(k_full, k_issued);
        drain(v_full, v_issued);
      }
    } else if (warp == 1) {
      if (lane == 0 && n_tiles > 0) {
        // MMA issuer. q·k of tile t + 1 follows the reading of tile t - 1's
        // weighted values, and w·v of tile t that of tile t + 1's scores. The
        // item's first tile needs no wait for TMEM: the block's barrier
        // between items follows the epilogue's last TMEM read.
        uint64_t* last_bar = nullptr;
        uint32_t last_parity = 0;
        auto wait = [&](uint64_t* bar, uint32_t parity) {
          return mbar_wait(bar, parity) && !*(volatile int*)failed;
        };
        auto commit = [&](uint64_t* bar, uint64_t* empty, int g) {
          umma_commit(bar);
          umma_commit(empty);
          last_bar = bar;
          last_parity = (uint32_t)(g & 1);
        };
        // One digit of A (64 B of k at a_base) against digits 1.. of B stacked
        // along N, as many as keep the pair's level.
        auto product = [&](uint32_t a_base, uint32_t b_base, bool first) {
          const uint64_t a0 = desc_sw64(a_base), b0 = desc_sw64(b_base);
  #pragma unroll
          for (int kk = 0; kk < 2; kk++)
  #pragma unroll
            for (int s = 1; s <= S; s++) {
              const int total = (S + 1 - s) * 64;
  #pragma unroll
              for (int nn0 = 0; nn0 < total; nn0 += 256) {
                const int nn = total - nn0 < 256 ? total - nn0 : 256;
                const uint64_t ad = desc_further(a0, (s - 1) * AM * 64 + kk * 32);
                const uint64_t bd = desc_further(b0, nn0 * 64 + kk * 32);
                umma_i8(tmem + (uint32_t)((s - 1) * 64 + nn0), ad, bd, idesc_i8(AM, nn),
                        (!first || kk > 0 || s > 1) ? 1u : 0u);
              }
            }
        };
        static_assert(AJ == 64 && AY == 64, "the products' columns");
        auto scores = [&](int it) {
          const int g = tiles_before + it, st = g % Sh::kStages;
          if (!wait(&k_full[st], (uint32_t)(g / Sh::kStages) & 1)) return false;
          tc_fence_after();
  #pragma unroll
          for (int kb = 0; kb < KB; kb++)
            product(smem_u32(sQ) + kb * S * AM * 64, smem_u32(sK + st * Sh::kK) + kb * S * AJ * 64, kb == 0);
          commit(qk_full, &k_empty[st], g);
          return true;
        };
        auto values = [&](int it) {
          const int g = tiles_before + it, st = g % Sh::kStages;
          if (!wait(p_full, (uint32_t)(g & 1)) || !wait(&v_full[st], (uint32_t)(g / Sh::kStages) & 1)) return false;
          tc_fence_after();
          product(smem_u32(sP), smem_u32(sV + st * Sh::kV), true);
          commit(pv_full, &v_empty[st], g);
          return true;
        };
        bool ok = wait(q_full, (uint32_t)(q_loads & 1)) && scores(0);
        for (int it = 0; ok && it < n_tiles; it++) {
          const int g = tiles_before + it;
          ok = wait(s_free, (uint32_t)(g & 1));
          if (ok && it > 0) ok = values(it - 1) && wait(o_free, (uint32_t)((g - 1) & 1));
          if (ok && it + 1 < n_tiles) ok = scores(it + 1);
        }
        ok = ok && values(n_tiles - 1);
        if (!ok) {
          atomicOr(a.status, 2);
          *(volatile int*)failed = 1;
        }
        // MMAs still running complete before TMEM is freed.
        if (last_bar) mbar_wait(last_bar, last_parity);
      }
    } else {
      // Epilogue: warp w reads TMEM lanes 32·(w % 4) .. +31; warps 2..5 take
      // columns 0..15 of each tile and of the sums, 6..9 columns 16..31, and
      // so on. The four warps of a lane quarter exchange row maxima over their
      // own named barrier; each warp signals the MMA warp by itself.
      constexpr int kShift = 8 * S - 2;
      const int h = (warp - 2) >> 2;
      const int quarter = warp & 3;
      const int r = quarter * 32 + lane;
      const int64_t xl = (int64_t)xt * AM + r;
      const bool valid = xl < a.lnx;
      const int lo = row_lo[r], hi = row_hi[r];
      // Column c of a tile starting at jl0 is allowed iff (unsigned)(jl0 + c - lo) < span.
      const unsigned span = (valid && lo < hi) ? (unsigned)(hi - lo) : 0u;
      const int eqr = valid ? a.eq[(int64_t)w * a.lnx_pad + xl] : 0;
      const uint32_t lane_addr = tmem + ((uint32_t)(quarter * 32) << 16);
      const uint32_t sum_addr = lane_addr + (uint32_t)(kSumCol + h * 2 * CW);
      const double NEG_INF = -INFINITY;
      // z sums the weights times 2^(8S-2); the running sums are in units of
      // their columns' powers of two 2^(2 + kLevelUnit + ev).
      double m = NEG_INF, z = 0.0, light = INFINITY;
      float light_f = INFINITY;
      // FAST: a score's scale times its powers of two, but for the key's.
      const double factor = a.scale_kind == 1 ? a.scale_c : 1.0;
      const int factor_hi = __double2hiint(factor) + ((eqr + kScoreUnit<KB>) << 20), factor_lo = __double2loint(factor);
      auto wait = [&](uint64_t* bar, uint32_t parity) {
        if (*(volatile int*)failed) return;
        if (!mbar_wait(bar, parity)) {
          *(volatile int*)failed = 1;
          atomicOr(a.status, 2);
        }
      };
      uint32_t chunk[S][CW / 4];
      // sums = sums · by + tile `it`'s weighted values, four at a time.
      auto add_values = [&](int it, double by) {
        wait(pv_full, (uint32_t)((tiles_before + it) & 1));
        tc_fence_after();
        int32_t L[S][4], sum[8];
        load_levels<S>(lane_addr, h * CW, L);
        if (it > 0) tmem_ld8(sum_addr, sum);
  #pragma unroll
        for (int c4 = 0; c4 < CW / 4; c4++) {
          tmem_wait_ld();
          landed<S>(L);
          if (it > 0) tmem_landed(sum);
          uint32_t next[8];
  #pragma unroll
          for (int i = 0; i < 4; i++) {
            const double l = combine_levels_small(L, i);
            const double v = it > 0 ? fma(__hiloint2double(sum[2 * i + 1], sum[2 * i]), by, l) : l;
            next[2 * i] = (uint32_t)__double2loint(v);
            next[2 * i + 1] = (uint32_t)__double2hiint(v);
          }
          if (c4 + 1 < CW / 4) {
            load_levels<S>(lane_addr, h * CW + c4 * 4 + 4, L);
            if (it > 0) tmem_ld8(sum_addr + c4 * 8 + 8, sum);
          }
          tmem_st8(sum_addr + c4 * 8, next);
        }
        tmem_wait_st();
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(o_free);
      };
      double last_rescale = 1.0;
      for (int it = 0; it < n_tiles; it++) {
        const int g = tiles_before + it;
        const int jl0 = (jt0 + it) * AJ + h * CW;
        const int* eks = ek_s + (g & 3) * AJ + h * CW;
        wait(qk_full, (uint32_t)(g & 1));
        tc_fence_after();
        double sc[CW];
        {
          // The next four columns' levels load while these are scaled.
          int32_t L[S][4];
          load_levels<S>(lane_addr, h * CW, L);
  #pragma unroll
          for (int c4 = 0; c4 < CW / 4; c4++) {
            tmem_wait_ld();
            landed<S>(L);
            double l[4];
  #pragma unroll
            for (int i = 0; i < 4; i++) l[i] = level_sum<S, KB>(L, i);
            if (c4 + 1 < CW / 4) load_levels<S>(lane_addr, h * CW + c4 * 4 + 4, L);
  #pragma unroll
            for (int i = 0; i < 4; i++) {
              const int c = c4 * 4 + i;
              sc[c] = FAST ? l[i] * __hiloint2double((eks[c] << 20) + factor_hi, factor_lo)
                           : scale2(l[i], eqr + eks[c] + kScoreUnit<KB>);
            }
          }
        }
        // (Without the row maxima's second buffer, once those are exchanged.)
        auto scores_read = [&]() {
          tc_fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive(s_free);
        };
        if constexpr (FAST) scores_read();
        if (!FAST && a.scale_kind == 1) {
  #pragma unroll
          for (int c = 0; c < CW; c++) sc[c] *= a.scale_c;
        } else if (a.scale_kind == 2) {
  #pragma unroll
          for (int c = 0; c < CW; c++) sc[c] = __ddiv_rn(sc[c], a.scale_c);
        }
        // The mask, and the row's largest and smallest allowed scores.
        const int off = jl0 - lo;
        const bool whole = __all_sync(0xffffffffu, off >= 0 && (unsigned)off + CW <= span);
        double m_new;
        if constexpr (FAST) {
          float mx = kLowestFloat;
          if (whole) {
  #pragma unroll
            for (int c = 0; c < CW; c++) {
              const float f = high_float(sc[c]);
              mx = fmaxf(mx, f);
              light_f = fminf(light_f, f);
            }
          } else {
  #pragma unroll
            for (int c = 0; c < CW; c++) {
              if ((unsigned)(off + c) < span) {
                const float f = high_float(sc[c]);
                mx = fmaxf(mx, f);
                light_f = fminf(light_f, f);
              } else {
                sc[c] = NEG_INF;
              }
            }
          }
          float* redf = (float*)red + (it & 1) * 4 * AM;
          redf[h * AM + r] = mx;
          named_bar(2 + quarter, 32 * kGroups);
  #pragma unroll
          for (int i = 0; i < kGroups; i++) mx = fmaxf(mx, redf[i * AM + r]);
          const bool any = mx != kLowestFloat, large = any && fabsf(mx) >= kExactHigh;
          double top = high_above(mx);
          // (The row's four warps hold the same maxima: they vote alike.)
          if (__any_sync(0xffffffffu, large)) {
            // The low words under that high word, ordered by sign.
            const int high = __float_as_int(mx);
            unsigned low = 0;
  #pragma unroll
            for (int c = 0; c < CW; c++)
              if (__double2hiint(sc[c]) == high) low = max(low, (unsigned)(__double2loint(sc[c]) ^ (high >> 31)));
            named_bar(2 + quarter, 32 * kGroups);  // the high words are read
            unsigned* lows = (unsigned*)redf;
            lows[h * AM + r] = low;
            named_bar(2 + quarter, 32 * kGroups);
  #pragma unroll
            for (int i = 0; i < kGroups; i++) low = max(low, lows[i * AM + r]);
            if (large) top = __hiloint2double(high, (int)low ^ (high >> 31));
          }
          m_new = any ? fmax(m, top) : m;
        } else {
          double mx = NEG_INF;
          if (whole) {
  #pragma unroll
            for (int c = 0; c < CW; c++) {
              mx = fmax(mx, sc[c]);
              light = fmin(light, sc[c]);
            }
          } else {
  #pragma unroll
            for (int c = 0; c < CW; c++) {
              const bool in = (unsigned)(off + c) < span;
              light = fmin(light, in ? sc[c] : INFINITY);
              sc[c] = in ? sc[c] : NEG_INF;
              mx = fmax(mx, sc[c]);
            }
          }
          red[h * AM + r] = mx;
          named_bar(2 + quarter, 32 * kGroups);
  #pragma unroll
          for (int i = 0; i < kGroups; i++) mx = fmax(mx, red[i * AM + r]);
          m_new = fmax(m, mx);
          scores_read();
        }
        double rescale = 1.0;
        if (m_new != m) {
          rescale = m == NEG_INF ? 0.0 : exp_tang(m - m_new, texp);
          z *= rescale;
          m = m_new;
        }
        // Weights and their digits: W = exp(s - m) · 2^(8S-2) < 2^(8S-2),
        // balanced base-256 digits, most significant first, sixteen columns a
        // store. A masked score's -inf clamps to a weight below 2^-974 (also
        // before the row's first key, when nothing is shifted yet): no digit
        // keeps it, and z drops it with its first real weight.
        const double shift = m == NEG_INF ? 0.0 : m;
        auto weigh = [&](int c4) {
          double x[4];
  #pragma unroll
          for (int i = 0; i < 4; i++) {
            x[i] = exp_weight(sc[c4 * 4 + i] - shift, texp, kShift);
            z += x[i];
          }
          uint32_t planes[S];
          digit_planes4<S>(x, planes);
  #pragma unroll
          for (int s = 0; s < S; s++) chunk[s][c4] = planes[s];
        };
        // The tile before's w·v runs beside the first half, the next one's q·k
        // beside the second.
  #pragma unroll
        for (int c4 = 0; c4 < CW / 8; c4++) weigh(c4);
        if (it > 0) add_values(it - 1, last_rescale);
        last_rescale = rescale;
  #pragma unroll
        for (int c4 = CW / 8; c4 < CW / 4; c4++) weigh(c4);
  #pragma unroll
        for (int b = 0; b < CW / 16; b++) {
          uint8_t* prow = sP + sw64_offset((uint32_t)r, (uint32_t)(h * CW + b * 16));
  #pragma unroll
          for (int s = 0; s < S; s++)
            *(uint4*)(prow + s * AM * 64) =
                make_uint4(chunk[s][b * 4], chunk[s][b * 4 + 1], chunk[s][b * 4 + 2], chunk[s][b * 4 + 3]);
        }
        fence_proxy_async();
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(p_full);
      }
      if (n_tiles > 0) add_values(n_tiles - 1, last_rescale);
      if (n_tiles > 0) {
        // The four quarters' sums of weights and lightest scores (P's digits
        // are no longer read).
        double* xz = (double*)sP;
        double* xlg = xz + kGroups * AM;
        xz[h * AM + r] = z;
        xlg[h * AM + r] = FAST ? (light_f == INFINITY ? INFINITY : high_below(light_f)) : light;
        named_bar(2 + quarter, 32 * kGroups);
        z = 0.0;
        light = INFINITY;
  #pragma unroll
        for (int i = 0; i < kGroups; i++) {
          z += xz[i * AM + r];
          light = fmin(light, xlg[i * AM + r]);
        }
        z *= pow2(-kShift);
        tc_fence_after();
        double o[CW];
  #pragma unroll
        for (int c4 = 0; c4 < CW / 4; c4++) {
          uint32_t sum[8];
          tmem_ld8(sum_addr + c4 * 8, (int32_t*)sum);
          tmem_wait_ld();
  #pragma unroll
          for (int i = 0; i < 4; i++)
            o[c4 * 4 + i] = scale2(__hiloint2double((int)sum[2 * i + 1], (int)sum[2 * i]), 2 + kLevelUnit + ev_s[h * CW + c4 * 4 + i]);
        }
        if (valid && lo < hi && !*(volatile int*)failed) {
          // Bounds::hold (fused.rs:1058-1086): the heaviest weight is
          // exp(high - m) = 1, the row's largest score being m.
          const double rl = a.rl[x_base + xl], rs = a.rs[x_base + xl];
          const double normal = 2.0 * 2.2250738585072014e-308, rounding = 2.220446049250313e-16 / 4.0;
          const double t2 = 2.0 * (double)(hi - lo);
          bool odd = !(z <= 1.7976931348623157e308);
          double least = INFINITY;  // the smallest magnitude of the outputs
          double* orow = a.out + (x_base + xl) * a.ny;
  #pragma unroll
          for (int c = 0; c < CW; c++) {
            const int64_t y = (int64_t)a.y0 + h * CW + c;
            if (y >= a.ny) continue;
            if (!isfinite(o[c])) odd = true;
            const double v = __ddiv_rn(o[c], z);
            if (!isfinite(v)) odd = true;
            least = fmin(least, fabs(v));
            orow[y] = v;
          }
          auto holds = [&](double lightest, double sum, double slack) {
            const double inverse = 1.0 / fabs(sum);
            if (!isfinite(rl * t2) || !isfinite(inverse) || !isfinite(inverse * rl * t2)) return false;
            if (rs == INFINITY) return true;
            const double quotient = lightest / fabs(sum);
            if (lightest * rs >= normal && quotient >= normal && quotient * rs >= normal) return true;
            return (t2 * 4.9406564584124654e-324) * ((inverse + rl) + 1.0) <= slack * rounding * least;
          };
          if (odd || !holds(exp(light - m), z, 1.0)) {
            // A guard fired. FAST: under the bounds' far ends (high words as they
            // are) too, with twice the room for the outputs' rounding, or only
            // the exact maxima can tell.
            bool unsure = FAST;
            if (FAST && !odd) {
              const double lowest = high_below(high_float(m)), lightest = high_above(high_float(light));
              unsure = holds(exp(lightest - lowest), z * exp(m - lowest), 2.0);
            }
            atomicOr(a.status, unsure ? 4 : 1);
          }
          if (h == 0 && a.lse && a.y0 == 0) a.lse[x_base + xl] = m + log(z);
        }
      }
    }
    tiles_before += n_tiles;
    q_loads += n_tiles > 0 ? 1 : 0;
    // The item's TMEM reads and shared-memory uses end before the next
    // item's setup and MMAs.
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem, 512);
  }
}

inline int64_t round_up(int64_t x, int64_t m) { return (x + m - 1) / m * m; }

// The kernel variant for d <= 64 (KB 1) or <= 128 (KB 2), with or without
// the fast powers of two.
using AttnKernel = void (*)(CUtensorMap, CUtensorMap, CUtensorMap, AttnArgs);

AttnKernel attn_kernel(int kb, bool fast, int* smem) {
  *smem = kb == 1 ? AttnShape<6, 1>::kSmem : AttnShape<6, 2>::kSmem;
  if (kb == 1) return fast ? attn_fwd_split<6, 1, true> : attn_fwd_split<6, 1, false>;
  return fast ? attn_fwd_split<6, 2, true> : attn_fwd_split<6, 2, false>;
}

// How the (query tile, batch) items of a forward pass reach the SMs.
enum Schedule : int {
  kGridSchedule = 0,   // a block per item: the grid's order, or the work list's by key tiles
  kTilesSchedule = 1,  // persistent blocks claiming the items by key tiles, most first
  kBatchSchedule = 2,  // persistent, batch by batch (the most key tiles first), in a batch by key tiles
  kSchedules = 3,
};

// A problem's work lists (the items that join some key).
struct WorkLists {
  std::vector<int2> by_tiles, both;  // by_tiles, and by_tiles then by batch
};

std::mutex g_work_lock;

// The schedules timed fastest, by padded shape and conditions (not by the
// ragged lengths, which a training loop may change at every step).
std::vector<int64_t> tuning_key(const AttentionProblem& p, int kb, bool fast) {
  std::vector<int64_t> key = {p.batches, p.lnx, p.lnj, p.ne, p.ny, kb, fast,
                              (int64_t)(!p.xlen_host.empty() || !p.jlen_host.empty()), p.mask.n};
  for (int i = 0; i < p.mask.n; i++) {
    key.push_back(p.mask.cmp[i]);
    key.push_back(p.mask.off[i]);
  }
  return key;
}
std::map<std::vector<int64_t>, int>& tuned_schedules() {
  static std::map<std::vector<int64_t>, int> tuned;
  return tuned;
}

// The work lists of a problem. Those of the last few shapes (lengths,
// extents, conditions) are kept: a training loop over the same batches
// asks for the same ones at every step.
std::shared_ptr<WorkLists> work_lists(const AttentionProblem& p) {
  std::vector<int64_t> key = {p.batches, p.lnx, p.lnj, p.ne, p.ny, p.mask.n, (int64_t)p.xlen_host.size(),
                              (int64_t)p.jlen_host.size()};
  for (int i = 0; i < p.mask.n; i++) {
    key.push_back(p.mask.cmp[i]);
    key.push_back(p.mask.off[i]);
  }
  key.insert(key.end(), p.xlen_host.begin(), p.xlen_host.end());
  key.insert(key.end(), p.jlen_host.begin(), p.jlen_host.end());
  static std::vector<std::pair<std::vector<int64_t>, std::shared_ptr<WorkLists>>> kept;  // most recent last
  {
    std::lock_guard<std::mutex> g(g_work_lock);
    for (size_t i = 0; i < kept.size(); i++)
      if (kept[i].first == key) {
        auto hit = kept[i];
        kept.erase(kept.begin() + (int64_t)i);
        kept.push_back(hit);
        return hit.second;
      }
  }
  Mask hm = p.mask;
  hm.xlen = p.xlen_host.empty() ? nullptr : p.xlen_host.data();
  hm.jlen = p.jlen_host.empty() ? nullptr : p.jlen_host.data();
  const bool ragged = hm.xlen || hm.jlen;
  // A query tile's key tiles (0: it joins none); without lengths every
  // batch has batch 0's.
  auto key_tiles = [&](int64_t w, int64_t xt) -> int64_t {
    const int64_t rows = hm.xlen ? hm.xlen[w] : p.lnx;
    int64_t first = INT64_MAX, last = INT64_MIN;
    for (int64_t r = xt * AM; r < std::min(rows, xt * AM + AM); r++) {
      int64_t lo, hi;
      allowed(hm, w * p.lnx + r, lo, hi);
      if (lo < hi) {
        first = std::min(first, lo - w * p.lnj);
        last = std::max(last, hi - w * p.lnj);
      }
    }
    return first < last ? (last + AJ - 1) / AJ - first / AJ : 0;
  };
  const int64_t n_xt = (p.lnx + AM - 1) / AM;
  std::vector<int64_t> first_batch;
  if (!ragged)
    for (int64_t xt = 0; xt < n_xt; xt++) first_batch.push_back(key_tiles(0, xt));
  std::vector<std::pair<int64_t, int2>> work;
  std::vector<std::pair<int64_t, int64_t>> batch_total;  // (key tiles, batch)
  for (int64_t w = 0; w < p.batches; w++) {
    int64_t total = 0;
    const int64_t rows = hm.xlen ? hm.xlen[w] : p.lnx;
    for (int64_t xt = 0; xt * AM < rows; xt++) {
      const int64_t n = ragged ? key_tiles(w, xt) : first_batch[(size_t)xt];
      if (n > 0) work.push_back({n, make_int2((int)xt, (int)w)});
      total += n;
    }
    batch_total.push_back({total, w});
  }
  auto most_first = [](const auto& a, const auto& b) { return a.first > b.first; };
  auto lists = std::make_shared<WorkLists>();
  std::stable_sort(work.begin(), work.end(), most_first);
  for (auto& x : work) lists->by_tiles.push_back(x.second);
  std::stable_sort(batch_total.begin(), batch_total.end(), most_first);
  std::vector<int64_t> place((size_t)p.batches);
  for (size_t i = 0; i < batch_total.size(); i++) place[(size_t)batch_total[i].second] = (int64_t)i;
  std::vector<int2> by_batch = lists->by_tiles;
  std::stable_sort(by_batch.begin(), by_batch.end(),
                   [&](const int2& a, const int2& b) { return place[(size_t)a.y] < place[(size_t)b.y]; });
  lists->both = lists->by_tiles;
  lists->both.insert(lists->both.end(), by_batch.begin(), by_batch.end());
  std::lock_guard<std::mutex> g(g_work_lock);
  kept.emplace_back(std::move(key), lists);
  if (kept.size() > 8) kept.erase(kept.begin());
  return lists;
}

// EINFOLD_ATTENTION_SCHEDULE = grid | tiles | batches forces a schedule;
// unset, the first call of a shape times them all.
int forced_schedule() {
  const char* s = std::getenv("EINFOLD_ATTENTION_SCHEDULE");
  if (!s || !*s) return -1;
  if (!std::strcmp(s, "grid")) return kGridSchedule;
  if (!std::strcmp(s, "tiles")) return kTilesSchedule;
  if (!std::strcmp(s, "batches")) return kBatchSchedule;
  fail(EINFOLD_INVALID, "EINFOLD_ATTENTION_SCHEDULE is %s, not grid, tiles or batches", s);
  return -1;
}

// EINFOLD_GRAPHS=0 launches directly instead of through CUDA graphs.
bool graphs_enabled() {
  const char* s = std::getenv("EINFOLD_GRAPHS");
  return !(s && !std::strcmp(s, "0"));
}

template <class T>
void put(std::vector<uint8_t>& key, const T& v) {
  const uint8_t* b = (const uint8_t*)&v;
  key.insert(key.end(), b, b + sizeof v);
}

}  // namespace

AttentionOutcome attention_split(Context& ctx, const AttentionProblem& p, int slices, cudaStream_t stream) {
  // Six slices: their levels (384 TMEM columns) and the rows' FP64 sums
  // (128) fill TMEM.
  const int S = slices;
  if (S != 6) return ATTENTION_INELIGIBLE;
  const int KB = p.ne <= 64 ? 1 : (p.ne <= 128 ? 2 : 0);
  if (KB == 0) return ATTENTION_INELIGIBLE;
  if (p.batches <= 0 || p.lnx <= 0 || p.lnj <= 0 || p.ny <= 0) return ATTENTION_INELIGIBLE;
  if (p.lnx > (1 << 30) || p.lnj > (1 << 30) || p.batches > 65535 || p.batches * S > INT32_MAX) return ATTENTION_INELIGIBLE;
  const int64_t W = p.batches;
  const int64_t lnx_pad = round_up(p.lnx, AM), lnj_pad = round_up(p.lnj, AJ), d_pad = 64 * KB;
  const int64_t ny_pad = round_up(p.ny, AY);
  auto al = [](size_t x) { return (x + 255) & ~(size_t)255; };
  const size_t szq = al((size_t)(W * S * lnx_pad * d_pad)), szk = al((size_t)(W * S * lnj_pad * d_pad)),
               szv = al((size_t)(W * S * ny_pad * lnj_pad));
  const size_t sze = al((size_t)(W * (lnx_pad + lnj_pad + ny_pad)) * 4), szc = al((size_t)(W * p.ny) * 8);
  DeviceBuffer<uint8_t> scratch(szq + szk + szv + sze + szc + 256, stream);
  uint8_t* b = scratch.get();
  int8_t* qd = (int8_t*)b;
  int8_t* kd = (int8_t*)(b + szq);
  int8_t* vd = (int8_t*)(b + szq + szk);
  int32_t* eq = (int32_t*)(b + szq + szk + szv);
  int32_t* ek = eq + W * lnx_pad;
  int32_t* ev = ek + W * lnj_pad;
  unsigned long long* colmax = (unsigned long long*)(b + szq + szk + szv + sze);
  // [0] 1: q or k not finite, 4: v; [1] kernel; [2..3] q's range, [4..5] k's,
  // [6..7] tile pairs
  int* status = (int*)(b + szq + szk + szv + sze + szc);
  unsigned long long* tiles = (unsigned long long*)(status + 6);
  EF_CUDA(cudaMemsetAsync(colmax, 0, szc + 32, stream));  // and status behind it
  const int64_t nx = W * p.lnx, nj = W * p.lnj, n_blocks = lnj_pad / 64;
  DeviceBuffer<double> bounds((size_t)(2 * nx + 2 * W * n_blocks), stream);
  double* rl = bounds.get();
  double* rs = rl + nx;
  double* bmax = rs + nx;
  double* bmin = bmax + W * n_blocks;
  const double *largest = p.largest, *smallest = p.smallest;
  // Ragged batches: the padding rows are neither read nor given digits. A
  // padding query joins no key and a padding key no query, so their digits
  // only meet masked scores (weights exactly 0) in exact integer sums, and
  // their rows' exponents (0) still bound the scores.
  RowSet sets[3];
  sets[0].x = p.q;
  sets[0].rows = p.lnx;
  sets[0].rows_pad = lnx_pad;
  sets[0].cols = p.ne;
  sets[0].lens = p.mask.xlen;
  sets[0].digits = qd;
  sets[0].e = eq;
  sets[0].k_pad = (int)d_pad;
  sets[0].skip_padding = p.mask.xlen != nullptr;
  sets[0].range = status + 2;
  sets[1] = sets[0];
  sets[1].x = p.k;
  sets[1].rows = p.lnj;
  sets[1].rows_pad = lnj_pad;
  sets[1].lens = p.mask.jlen;
  sets[1].digits = kd;
  sets[1].e = ek;
  sets[1].skip_padding = p.mask.jlen != nullptr;
  sets[1].range = status + 4;
  sets[2].x = p.v;
  sets[2].rows = p.lnj;
  sets[2].rows_pad = lnj_pad;
  sets[2].cols = p.ny;
  sets[2].lens = p.mask.jlen;
  sets[2].colmax = colmax;
  sets[2].block_largest = bmax;
  sets[2].block_smallest = bmin;
  sets[2].bad = 4;
  if (p.values) {
    p.values->flag.allocate((size_t)nj, stream);
    p.values->largest.allocate((size_t)nj, stream);
    p.values->smallest.allocate((size_t)nj, stream);
    p.values->known = true;
    sets[2].flag = p.values->flag.get();
    largest = sets[2].largest = p.values->largest.get();
    smallest = sets[2].smallest = p.values->smallest.get();
  }
  prepare_rows(ctx, sets, 3, W, status, stream);
  ColumnSet vc;
  vc.x = p.v;
  vc.rows = p.lnj;
  vc.rows_pad = lnj_pad;
  vc.cols = p.ny;
  vc.cols_pad = ny_pad;
  vc.lens = p.mask.jlen;
  vc.skip_padding = p.mask.jlen != nullptr;
  vc.colmax = colmax;
  vc.digits = vd;
  vc.e = ev;
  prepare_columns(ctx, &vc, 1, W, stream);
  row_bounds(ctx, p.mask, nx, n_blocks, largest, smallest, bmax, bmin, rl, rs, stream);
  // Every operand finite, no score near overflow (|s| < ne · 2^(eq+ek-4)), and
  // (FAST) every score's power of two 2^(eq + ek) a normal double: the tile kernel
  // judges by itself, and the host once it has run.
  const int top = 1000 - 8 - (int)std::ceil(std::log2((double)p.ne + 1));
  const double scale = std::fabs(p.scale_kind == 1 ? p.scale_c : p.scale_kind == 2 ? 1.0 / p.scale_c : 1.0);
  Ready ready;
  ready.status = status;
  ready.pairs = 1;
  const int scale_exp = std::isnormal(scale) ? std::ilogb(scale) : 0;
  ready.top = std::isnormal(scale) ? top - std::max(0, 1 + scale_exp) : INT_MIN / 2;
  ready.low = 1022 + (KB == 1 ? kLevelUnit : 0) + std::min(0, scale_exp);
  int st[8] = {};
  auto read_status = [&]() {
    ReadBack back(ctx, stream);
    back.add(st, status, 8);
    back.wait();
  };
  auto eligible = [&]() {
    if (p.values) p.values->all_finite = !(st[0] & 4);
    return st[0] == 0 && st[2] + st[4] - 2 * kExponentBias <= top;
  };
  auto normal_powers = [&]() {
    Ready host = ready;
    host.status = st;
    return host.ok();
  };
  bool fast = true;

  const CUtensorMap tq = digit_planes_map(qd, d_pad, lnx_pad, W * S, AM, S);
  const CUtensorMap tk = digit_planes_map(kd, d_pad, lnj_pad, W * S, AJ, S);
  const CUtensorMap tv = digit_planes_map(vd, lnj_pad, ny_pad, W * S, AY, S);
  AttnArgs args{};
  args.mask = p.mask;
  args.lnx = p.lnx;
  args.lnj = p.lnj;
  args.lnx_pad = lnx_pad;
  args.lnj_pad = lnj_pad;
  args.ny = p.ny;
  args.ny_pad = ny_pad;
  args.scale_kind = p.scale_kind;
  args.scale_c = p.scale_c;
  args.eq = eq;
  args.ek = ek;
  args.ev = ev;
  args.rl = rl;
  args.rs = rs;
  args.exp_table = exp_table(ctx.device);
  args.out = p.out;
  args.lse = p.lse;
  args.status = status + 1;
  args.tiles = tiles;
  // The query tiles whose rows join the most keys first: the last ones
  // under a causal mask, the first ones when the mask runs the other way.
  args.reverse = last_rows_longest(p.mask, p.lnx);
  // The items that join some key, by key tiles and batch by batch.
  const std::shared_ptr<WorkLists> lists = work_lists(p);
  const int n_items = (int)lists->by_tiles.size();
  if (n_items == 0) {
    if (p.values) {
      read_status();
      return eligible() ? ATTENTION_DONE : ATTENTION_INELIGIBLE;
    }
    return ATTENTION_DONE;
  }
  const bool ragged = !p.xlen_host.empty() || !p.jlen_host.empty();
  const int n_y = (int)((p.ny + AY - 1) / AY);
  // (The lists' order of batches lies behind that of tiles, copied in one.)
  DeviceBuffer<int2> items((size_t)n_items * 2, stream);
  EF_CUDA(cudaMemcpyAsync(items.get(), lists->both.data(), (size_t)n_items * 2 * sizeof(int2), cudaMemcpyHostToDevice,
                          stream));
  DeviceBuffer<unsigned> counters((size_t)n_y, stream);
  int smem = 0;
  AttnKernel kernel = attn_kernel(KB, true, &smem);
  EF_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
  const int persistent_blocks = std::min(n_items, ctx.sm_count);
  // The tile phase under a schedule: a launch per block of 64 value columns
  // (persistent ones after zeroing their item counters).
  auto enqueue = [&](int schedule, cudaStream_t st) {
    AttnArgs ar = args;
    ar.ready = ready;
    dim3 grid((unsigned)(lnx_pad / AM), (unsigned)W);
    if (schedule == kGridSchedule) {
      if (ragged) {
        ar.items = items.get();
        ar.n_items = n_items;
        grid = dim3((unsigned)n_items, 1);
      }
    } else {
      ar.items = items.get() + (schedule == kBatchSchedule ? n_items : 0);
      ar.n_items = n_items;
      grid = dim3((unsigned)persistent_blocks, 1);
      EF_CUDA(cudaMemsetAsync(counters.get(), 0, (size_t)n_y * sizeof(unsigned), st));
    }
    for (int yb = 0; yb < n_y; yb++) {
      ar.y0 = yb * AY;
      ar.next = schedule == kGridSchedule ? nullptr : counters.get() + yb;
      kernel<<<grid, kAttnThreads, smem, st>>>(tq, tk, tv, ar);
      EF_LAUNCH_CHECK();
    }
  };
  cudaEvent_t e0, e1;
  EF_CUDA(cudaEventCreate(&e0));
  EF_CUDA(cudaEventCreate(&e1));
  struct Events {
    cudaEvent_t a, b;
    ~Events() {
      cudaEventDestroy(a);
      cudaEventDestroy(b);
    }
  } events{e0, e1};
  const int forced = forced_schedule();
  int schedule = forced;
  auto tuned_schedule = [&]() {
    if (forced >= 0) return forced;
    std::lock_guard<std::mutex> g(g_work_lock);
    const auto it = tuned_schedules().find(tuning_key(p, KB, fast));
    return it != tuned_schedules().end() ? it->second : -1;
  };
  schedule = tuned_schedule();
  // A shape whose schedule is known launches FAST at once under `ready`; a new
  // one, or one whose powers of two turn out not to be normal, waits for the
  // status first.
  bool judged = false, exact = false;
  auto judge = [&]() -> bool {
    read_status();
    judged = true;
    if (!eligible()) return false;
    fast = !exact && normal_powers();
    if (!fast) ready.status = nullptr;
    kernel = attn_kernel(KB, fast, &smem);
    EF_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
    schedule = tuned_schedule();
    return true;
  };
  if (schedule < 0 && !judge()) return ATTENTION_INELIGIBLE;
  const auto tune = [&]() {
    if (schedule < 0) {
      // The first call of this shape: each schedule twice (the same results
      // each time), the fastest by its shorter run.
      float best = INFINITY;
      for (int sc = 0; sc < kSchedules; sc++) {
        for (int rep = 0; rep < 2; rep++) {
          EF_CUDA(cudaEventRecord(e0, stream));
          enqueue(sc, stream);
          EF_CUDA(cudaEventRecord(e1, stream));
          EF_CUDA(cudaEventSynchronize(e1));
          float ms = 0;
          EF_CUDA(cudaEventElapsedTime(&ms, e0, e1));
          ctx.kernels += (uint64_t)n_y;
          if (ms < best) {
            best = ms;
            schedule = sc;
          }
        }
      }
      {
        std::lock_guard<std::mutex> g(g_work_lock);
        auto& tuned = tuned_schedules();
        if (tuned.size() >= 256) tuned.clear();
        tuned[tuning_key(p, KB, fast)] = schedule;
      }
      EF_CUDA(cudaMemsetAsync(tiles, 0, sizeof(unsigned long long), stream));
    }
  };
  const auto run = [&]() {
    tune();
    EF_CUDA(cudaEventRecord(e0, stream));
    if (graphs_enabled()) {
      // Replayed while every argument of the launches is the same (pointers
      // included); else captured again and updated in place.
      std::vector<uint8_t> shape, key;
      put(shape, ctx.device);
      put(shape, KB);
      put(shape, fast);
      put(shape, schedule);
      put(shape, n_y);
      put(shape, ragged);
      put(shape, persistent_blocks);
      for (const void* ptr : {(const void*)scratch.get(), (const void*)items.get(), (const void*)counters.get(),
                              (const void*)rl, (const void*)p.out, (const void*)p.lse, (const void*)args.exp_table,
                              (const void*)p.mask.xlen, (const void*)p.mask.jlen})
        put(key, ptr);
      for (int64_t x : {W, p.lnx, p.lnj, p.ne, p.ny, lnx_pad, lnj_pad, ny_pad, (int64_t)n_items, (int64_t)p.scale_kind,
                        (int64_t)args.reverse, (int64_t)p.mask.n, p.mask.lnx, p.mask.lnj})
        put(key, x);
      put(key, p.scale_c);
      for (int i = 0; i < p.mask.n; i++) {
        put(key, p.mask.cmp[i]);
        put(key, p.mask.off[i]);
      }
      ctx.graph = ctx.graphs.run(shape, key, stream, [&](cudaStream_t st) { enqueue(schedule, st); });
    } else {
      enqueue(schedule, stream);
    }
    ctx.kernels += (uint64_t)n_y;
    ctx.schedule = schedule;
    EF_CUDA(cudaEventRecord(e1, stream));
  };
  run();
  read_status();
  if (!judged && !eligible()) return ATTENTION_INELIGIBLE;
  // The launch did nothing, or met guards that only exact maxima decide (and none
  // that fire in any case: a refused call doesn't run twice, 3.6 ms against 7.3 at
  // 64 x 4096 x 64). A call whose rows lie between the bounds runs twice every
  // time: starting such shapes with the exact variant would make a call's bits
  // depend on the calls before it.
  if (fast && (!normal_powers() || ((st[1] & 4) && !(st[1] & 1)))) {
    exact = st[1] & 4;
    EF_CUDA(cudaMemsetAsync(status + 1, 0, 4, stream));
    EF_CUDA(cudaMemsetAsync(tiles, 0, sizeof(unsigned long long), stream));
    judge();
    run();
    read_status();
  }
  unsigned long long pairs = 0;
  std::memcpy(&pairs, st + 6, 8);
  float ms = 0;
  cudaEventElapsedTime(&ms, e0, e1);
  // Digit products executed: per pair of tiles, S(S+1)/2 digit pairs of a
  // 128 x 64 x d_pad product (scores) and of a 128 x 64 x 64 one (values).
  ctx.product_ms += ms;
  ctx.product_ops += (double)pairs * (S * (S + 1) / 2) * 2.0 * AM * AJ * (double)(d_pad + AY);
  ctx.phase("attention: tiles");
  if (st[1] & 2) fail(EINFOLD_TIMEOUT, "a bounded wait in the attention kernel ran out");
  return (st[1] & 1) ? ATTENTION_GUARDED : ATTENTION_DONE;
}

}  // namespace ef
