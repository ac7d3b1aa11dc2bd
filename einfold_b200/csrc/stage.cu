// Staging Arrow columns into HBM, and the scan/pack helpers.
#include <cub/cub.cuh>

#include "stage.cuh"

namespace ef {
namespace {

struct Segment {
  int64_t row;       // first row of the batch in the concatenation
  int64_t byte;      // where its bitmap bytes start in the staged bitmap
  int32_t shift;     // bit of its first row in the first byte
  int32_t pad;
};

__global__ void expand_validity(const uint8_t* __restrict__ bits, const Segment* __restrict__ seg, int n_seg,
                                int64_t rows, uint8_t* __restrict__ out) {
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < rows; i += (int64_t)gridDim.x * blockDim.x) {
    int lo = 0, hi = n_seg - 1;
    while (lo < hi) {
      int mid = (lo + hi + 1) >> 1;
      if (seg[mid].row <= i) lo = mid; else hi = mid - 1;
    }
    const Segment s = seg[lo];
    if (s.byte < 0) { out[i] = 1; continue; }
    const int64_t b = (int64_t)s.shift + (i - s.row);
    out[i] = (bits[s.byte + (b >> 3)] >> (b & 7)) & 1;
  }
}

template <class T>
__global__ void widen(const T* __restrict__ in, int64_t n, int64_t* __restrict__ out, unsigned long long* max,
                      int* flags) {
  int64_t local = -1;
  int f = 0;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    T v = in[i];
    int64_t w;
    if constexpr (sizeof(T) == 8 && !std::is_signed<T>::value) {
      if ((uint64_t)v >= (1ull << 63)) { f |= 2; w = -1; } else w = (int64_t)v;
    } else {
      w = (int64_t)v;
    }
    if (w < 0) f |= 1;
    if (out) out[i] = w;
    if (w > local) local = w;
  }
  for (int o = 16; o; o >>= 1) {
    long long other = __shfl_xor_sync(0xffffffffu, (long long)local, o);
    if (other > local) local = other;
    f |= __shfl_xor_sync(0xffffffffu, f, o);
  }
  if ((threadIdx.x & 31) == 0) {
    if (local >= 0) atomicMax(max, (unsigned long long)local);
    if (f) atomicOr(flags, f);
  }
}

__global__ void pack_bits_kernel(const uint8_t* __restrict__ in, int64_t n, uint8_t* __restrict__ out) {
  const int64_t bytes = (n + 7) / 8;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < bytes; i += (int64_t)gridDim.x * blockDim.x) {
    uint8_t v = 0;
    for (int j = 0; j < 8; j++) {
      const int64_t r = i * 8 + j;
      if (r < n && in[r]) v |= (uint8_t)(1u << j);
    }
    out[i] = v;
  }
}

}  // namespace

DeviceColumn stage_column(Context& ctx, const Relation& r, int col, bool with_validity) {
  DeviceColumn d;
  cudaStream_t s = ctx.stream;
  if (col < 0 || col >= (int)r.fields.size()) fail(EINFOLD_INVALID, "column %d of a relation with %zu", col, r.fields.size());
  d.kind = r.fields[col].kind;
  d.rows = r.rows();
  const cudaMemcpyKind from = r.device >= 0 ? cudaMemcpyDeviceToDevice : cudaMemcpyHostToDevice;
  if (r.device >= 0 && r.device != ctx.device)
    fail(EINFOLD_INVALID, "a relation on device %d given to a context on device %d", r.device, ctx.device);
  for (auto& b : r.batches) {
    const Column& c = b.columns[col];
    if (c.dictionary) fail(EINFOLD_INVALID, "dictionary columns are not staged here");
    d.nulls += c.nulls();
  }
  if (is_var(d.kind)) {
    if (r.device >= 0) fail(EINFOLD_INVALID, "variable-length columns must be in host memory");
    bool large = d.kind == Kind::LargeUtf8 || d.kind == Kind::LargeBinary;
    // Offsets rebased per batch on the host (one pass over the offsets), bytes copied as they are.
    std::vector<int64_t> off((size_t)d.rows + 1);
    int64_t total = 0, row = 0;
    std::vector<std::pair<const uint8_t*, int64_t>> spans;
    for (auto& b : r.batches) {
      const Column& c = b.columns[col];
      if (c.length == 0) continue;
      int64_t first, last;
      if (large) { first = ((const int64_t*)c.values)[c.offset]; last = ((const int64_t*)c.values)[c.offset + c.length]; }
      else { first = ((const int32_t*)c.values)[c.offset]; last = ((const int32_t*)c.values)[c.offset + c.length]; }
      for (int64_t i = 0; i < c.length; i++) {
        int64_t o = large ? ((const int64_t*)c.values)[c.offset + i] : ((const int32_t*)c.values)[c.offset + i];
        off[(size_t)(row + i)] = total + (o - first);
      }
      spans.push_back({c.data + first, last - first});
      total += last - first;
      row += c.length;
    }
    off[(size_t)d.rows] = total;
    d.offsets.allocate((size_t)d.rows + 1, s);
    EF_CUDA(cudaMemcpyAsync(d.offsets.get(), off.data(), off.size() * 8, cudaMemcpyHostToDevice, s));
    d.bytes.allocate((size_t)(total ? total : 1), s);
    int64_t pos = 0;
    for (auto& sp : spans) {
      if (sp.second) EF_CUDA(cudaMemcpyAsync(d.bytes.get() + pos, sp.first, (size_t)sp.second, cudaMemcpyHostToDevice, s));
      pos += sp.second;
    }
    EF_CUDA(cudaStreamSynchronize(s));  // `off` is a host temporary
  } else if (d.kind == Kind::Bool) {
    // Booleans are bit-packed; expanded to bytes with the validity machinery.
    d.width = 1;
    d.data.allocate((size_t)(d.rows ? d.rows : 1), s);
    std::vector<Segment> seg;
    int64_t nbytes = 0, row = 0;
    for (auto& b : r.batches) {
      const Column& c = b.columns[col];
      int64_t first = c.offset / 8, last = (c.offset + c.length + 7) / 8;
      seg.push_back({row, nbytes, (int32_t)(c.offset % 8), 0});
      nbytes += last - first;
      row += c.length;
    }
    DeviceBuffer<uint8_t> bits((size_t)(nbytes ? nbytes : 1), s);
    int64_t pos = 0;
    for (auto& b : r.batches) {
      const Column& c = b.columns[col];
      int64_t first = c.offset / 8, last = (c.offset + c.length + 7) / 8;
      if (last > first) EF_CUDA(cudaMemcpyAsync(bits.get() + pos, c.values + first, (size_t)(last - first), from, s));
      pos += last - first;
    }
    if (seg.empty()) seg.push_back({0, -1, 0, 0});
    DeviceBuffer<Segment> dseg(seg.size(), s);
    EF_CUDA(cudaMemcpyAsync(dseg.get(), seg.data(), seg.size() * sizeof(Segment), cudaMemcpyHostToDevice, s));
    if (d.rows) expand_validity<<<blocks_for(d.rows, 256), 256, 0, s>>>(bits.get(), dseg.get(), (int)seg.size(), d.rows, d.data.get());
    EF_CUDA(cudaStreamSynchronize(s));
  } else if (d.kind != Kind::Null) {
    d.width = fixed_width(r.fields[col].format);
    if (!d.width) fail(EINFOLD_INVALID, "a column of an unsupported type");
    if (r.device >= 0 && r.batches.size() == 1) {
      // One batch already in HBM: read in place.
      const Column& c = r.batches[0].columns[col];
      d.alias = c.values + c.offset * d.width;
    } else {
      d.data.allocate((size_t)(d.rows * d.width ? d.rows * d.width : 1), s);
      int64_t row = 0;
      for (auto& b : r.batches) {
        const Column& c = b.columns[col];
        if (c.length)
          EF_CUDA(cudaMemcpyAsync(d.data.get() + row * d.width, c.values + c.offset * d.width,
                                  (size_t)(c.length * d.width), from, s));
        row += c.length;
      }
    }
  }
  if (with_validity && d.nulls > 0) {
    d.valid.allocate((size_t)d.rows, s);
    std::vector<Segment> seg;
    int64_t nbytes = 0, row = 0;
    for (auto& b : r.batches) {
      const Column& c = b.columns[col];
      if (c.validity && c.nulls() > 0) {
        int64_t first = c.offset / 8, last = (c.offset + c.length + 7) / 8;
        seg.push_back({row, nbytes, (int32_t)(c.offset % 8), 0});
        nbytes += last - first;
      } else {
        seg.push_back({row, -1, 0, 0});
      }
      row += c.length;
    }
    DeviceBuffer<uint8_t> bits((size_t)(nbytes ? nbytes : 1), s);
    int64_t pos = 0;
    for (auto& b : r.batches) {
      const Column& c = b.columns[col];
      if (c.validity && c.nulls() > 0) {
        int64_t first = c.offset / 8, last = (c.offset + c.length + 7) / 8;
        EF_CUDA(cudaMemcpyAsync(bits.get() + pos, c.validity + first, (size_t)(last - first), from, s));
        pos += last - first;
      }
    }
    DeviceBuffer<Segment> dseg(seg.size(), s);
    EF_CUDA(cudaMemcpyAsync(dseg.get(), seg.data(), seg.size() * sizeof(Segment), cudaMemcpyHostToDevice, s));
    expand_validity<<<blocks_for(d.rows, 256), 256, 0, s>>>(bits.get(), dseg.get(), (int)seg.size(), d.rows, d.valid.get());
    EF_LAUNCH_CHECK();
    ctx.kernels++;
    EF_CUDA(cudaStreamSynchronize(s));  // `seg` is a host temporary
  }
  return d;
}

DeviceBuffer<int64_t> keys_as_i64(Context& ctx, const DeviceColumn& c, KeyStats* stats) {
  cudaStream_t s = ctx.stream;
  DeviceBuffer<int64_t> out((size_t)(c.rows ? c.rows : 1), s);
  DeviceBuffer<unsigned long long> mx(1, s);
  DeviceBuffer<int> flags(1, s);
  mx.zero();
  flags.zero();
  unsigned g = blocks_for(c.rows, 256);
  switch (c.kind) {
    case Kind::Int8: widen<int8_t><<<g, 256, 0, s>>>((const int8_t*)c.ptr(), c.rows, out.get(), mx.get(), flags.get()); break;
    case Kind::UInt8: widen<uint8_t><<<g, 256, 0, s>>>((const uint8_t*)c.ptr(), c.rows, out.get(), mx.get(), flags.get()); break;
    case Kind::Int16: widen<int16_t><<<g, 256, 0, s>>>((const int16_t*)c.ptr(), c.rows, out.get(), mx.get(), flags.get()); break;
    case Kind::UInt16: widen<uint16_t><<<g, 256, 0, s>>>((const uint16_t*)c.ptr(), c.rows, out.get(), mx.get(), flags.get()); break;
    case Kind::Int32: widen<int32_t><<<g, 256, 0, s>>>((const int32_t*)c.ptr(), c.rows, out.get(), mx.get(), flags.get()); break;
    case Kind::UInt32: widen<uint32_t><<<g, 256, 0, s>>>((const uint32_t*)c.ptr(), c.rows, out.get(), mx.get(), flags.get()); break;
    case Kind::Int64: widen<int64_t><<<g, 256, 0, s>>>((const int64_t*)c.ptr(), c.rows, out.get(), mx.get(), flags.get()); break;
    case Kind::UInt64: widen<uint64_t><<<g, 256, 0, s>>>((const uint64_t*)c.ptr(), c.rows, out.get(), mx.get(), flags.get()); break;
    default: fail(EINFOLD_INVALID, "keys_as_i64 of a non-integer column");
  }
  EF_LAUNCH_CHECK();
  ctx.kernels++;
  unsigned long long m = 0;
  int f = 0;
  EF_CUDA(cudaMemcpyAsync(&m, mx.get(), 8, cudaMemcpyDeviceToHost, s));
  EF_CUDA(cudaMemcpyAsync(&f, flags.get(), 4, cudaMemcpyDeviceToHost, s));
  EF_CUDA(cudaStreamSynchronize(s));
  stats->max = c.rows ? (int64_t)m : -1;
  stats->negative = f & 1;
  stats->too_large = (f & 2) != 0;
  return out;
}

void key_stats_i64(Context& ctx, const int64_t* keys, int64_t n, KeyStats* stats) {
  cudaStream_t s = ctx.stream;
  DeviceBuffer<unsigned long long> mx(1, s);
  DeviceBuffer<int> flags(1, s);
  mx.zero();
  flags.zero();
  widen<int64_t><<<blocks_for(n, 256), 256, 0, s>>>(keys, n, nullptr, mx.get(), flags.get());
  EF_LAUNCH_CHECK();
  ctx.kernels++;
  unsigned long long m = 0;
  int f = 0;
  EF_CUDA(cudaMemcpyAsync(&m, mx.get(), 8, cudaMemcpyDeviceToHost, s));
  EF_CUDA(cudaMemcpyAsync(&f, flags.get(), 4, cudaMemcpyDeviceToHost, s));
  EF_CUDA(cudaStreamSynchronize(s));
  stats->max = n ? (int64_t)m : -1;
  stats->negative = f & 1;
  stats->too_large = (f & 2) != 0;
}

int64_t exclusive_scan_flags(Context& ctx, const uint8_t* flags, int64_t n, int64_t* out) {
  cudaStream_t s = ctx.stream;
  if (n <= 0) return 0;
  size_t temp = 0;
  cub::TransformInputIterator<int64_t, cub::CastOp<int64_t>, const uint8_t*> it(flags, cub::CastOp<int64_t>());
  EF_CUDA(cub::DeviceScan::ExclusiveSum(nullptr, temp, it, out, n, s));
  DeviceBuffer<uint8_t> t(temp ? temp : 1, s);
  EF_CUDA(cub::DeviceScan::ExclusiveSum(t.get(), temp, it, out, n, s));
  int64_t last = 0;
  uint8_t lastf = 0;
  EF_CUDA(cudaMemcpyAsync(&last, out + n - 1, 8, cudaMemcpyDeviceToHost, s));
  EF_CUDA(cudaMemcpyAsync(&lastf, flags + n - 1, 1, cudaMemcpyDeviceToHost, s));
  EF_CUDA(cudaStreamSynchronize(s));
  ctx.kernels += 2;
  return last + (lastf ? 1 : 0);
}

void pack_bits(Context& ctx, const uint8_t* bytes, int64_t n, uint8_t* bits) {
  if (n <= 0) return;
  pack_bits_kernel<<<blocks_for((n + 7) / 8, 256), 256, 0, ctx.stream>>>(bytes, n, bits);
  EF_LAUNCH_CHECK();
  ctx.kernels++;
}

HostBuffer to_host(Context& ctx, const void* dev, size_t bytes) {
  HostBuffer h = HostBuffer::page_locked(bytes ? bytes : 1);
  if (bytes) {
    EF_CUDA(cudaMemcpyAsync(h.ptr, dev, bytes, cudaMemcpyDeviceToHost, ctx.stream));
    EF_CUDA(cudaStreamSynchronize(ctx.stream));
  }
  h.bytes = bytes;
  return h;
}

__global__ void key_tables(int64_t n, OutKeys keys, int in_x, int64_t* __restrict__ tables) {
  for (int64_t p = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; p < n; p += (int64_t)gridDim.x * blockDim.x)
    for (int k = 0; k < keys.n; k++)
      if (keys.key[k].in_x == in_x) tables[(int64_t)k * n + p] = keys.key[k].at(p, p);
}

StagedKeys stage_keys(Context& ctx, const OperandD& op, const Relation& r) {
  StagedKeys s;
  for (auto& k : op.keys) {
    const Field& f = r.fields[k.col];
    if (f.dictionary || !is_integer(f.kind)) decline("a key column that isn't integers");
    for (auto& b : r.batches)
      if (b.columns[k.col].nulls() > 0) decline("a NULL key");
    s.cols.push_back(stage_column(ctx, r, k.col, false));
    DeviceColumn& c = s.cols.back();
    KeyStats st;
    if (c.kind == Kind::Int64) {
      key_stats_i64(ctx, (const int64_t*)c.ptr(), c.rows, &st);
      s.keys.push_back((const int64_t*)c.ptr());
    } else {
      s.wide.push_back(keys_as_i64(ctx, c, &st));
      s.keys.push_back(s.wide.back().get());
    }
    if (st.negative || st.too_large) decline("a negative key, or one too large for int64");
    if (st.max == INT64_MAX) decline("a key whose extent doesn't fit");
    s.extent.push_back(st.max + 1);
  }
  return s;
}

CellKeys cell_keys(const std::vector<int>& rows, const std::vector<int>& cols, const OperandD& op,
                   const StagedKeys& s, const std::vector<int64_t>& extent) {
  if (rows.size() > (size_t)kMaxDims || cols.size() > (size_t)kMaxDims) decline("more than 8 dimensions in one role");
  std::vector<int> dims = rows;
  dims.insert(dims.end(), cols.begin(), cols.end());
  CellKeys k;
  uint64_t stride = 1;  // of the last dimension; an extent of 0 leaves no rows
  k.n = (int)dims.size();
  for (int i = k.n - 1; i >= 0; i--) {
    int slot = -1;
    for (size_t j = 0; j < op.keys.size(); j++)
      if (op.keys[j].dim == dims[(size_t)i]) slot = (int)j;
    k.key[i] = s.keys[(size_t)slot];
    k.stride[i] = (int64_t)stride;
    stride *= (uint64_t)extent[(size_t)dims[(size_t)i]];
  }
  return k;
}

namespace {

// Bound by HBM: (8·keys + 8) bytes read and 8 written a row. What keeps it
// there:
// - Every key of kScatterRows rows a thread is loaded before any is used (the
//   number of keys is a template argument): a loop over the keys waits a DRAM
//   latency for each.
// - A warp whose 32 rows fall on consecutive cells (a table in key order) marks
//   them with an atomic OR a word of `held`, found from the first row's cell. A
//   warp where neighbouring rows share a word (rows partly in order) ORs the codes
//   of the lanes that share one first (a match and a reduction), one atomic a
//   word. Others (shuffled rows) issue an atomic a row: a match of 32 different
//   words takes longer.
// Measured (one B200): 67.1M rows of two keys in order 671 us (2-bit codes) and
// 552 us (1-bit) when every warp matched and loaded key by key, 439 and 429 now
// (6548 GB/s would take 328); 67.1M rows of three keys 1123 us, 472 now.
// Four rows a thread from kManyRows rows on, which still fills the SMs; below,
// one (262,144 shuffled rows: 8.5 us against 23 with four, and 67 before).
constexpr int kScatterRows = 4;
constexpr int64_t kManyRows = 148 * 2048 * 4;

template <int NK, int BITS, int U>
__global__ void __launch_bounds__(256) scatter_cells_kernel(CellKeys k, int64_t rows, const double* __restrict__ vals,
                                                            const uint8_t* __restrict__ valid,
                                                            double* __restrict__ mat, uint32_t* __restrict__ held,
                                                            unsigned* flags, unsigned dup, unsigned nonfinite) {
  constexpr unsigned CELLS = 32 / BITS, LOG = BITS == 1 ? 5 : 4, CODE = (1u << BITS) - 1;
  unsigned f = 0;
  const unsigned lane = threadIdx.x & 31;
  for (int64_t base = (int64_t)blockIdx.x * (256 * U); base < rows; base += (int64_t)gridDim.x * (256 * U)) {
    int64_t kv[U][NK];
    double val[U];
    bool on[U], ok[U];
#pragma unroll
    for (int u = 0; u < U; u++) {
      const int64_t r = base + u * 256 + threadIdx.x;
      on[u] = r < rows;
#pragma unroll
      for (int i = 0; i < NK; i++) kv[u][i] = on[u] && i < k.n ? k.key[i][r] : 0;
      val[u] = on[u] ? vals[r] : 0.0;
      ok[u] = on[u] && (!valid || valid[r]);
    }
    uint32_t cell[U];
#pragma unroll
    for (int u = 0; u < U; u++) {
      int64_t c = 0;
#pragma unroll
      for (int i = 0; i < NK; i++) c += kv[u][i] * k.stride[i];
      cell[u] = (uint32_t)c;
      if (ok[u]) {
        mat[c] = val[u];
        if (!isfinite(val[u])) f |= nonfinite;
      }
    }
#pragma unroll
    for (int u = 0; u < U; u++) {
      const unsigned active = __ballot_sync(0xffffffffu, on[u]);
      if (active == 0) continue;
      const uint32_t c0 = __shfl_sync(0xffffffffu, cell[u], 0);
      if (__all_sync(0xffffffffu, ok[u] && cell[u] == c0 + lane)) {
        // Cells c0 .. c0 + 31, all valued: lane i marks its word, cells
        // [first, last) of it.
        const unsigned off = c0 & (CELLS - 1), words = (off + 31) / CELLS + 1;
        if (lane < words) {
          const unsigned first = lane == 0 ? off : 0, last = min(CELLS, off + 32 - lane * CELLS);
          const unsigned n = (last - first) * BITS;
          const unsigned cells = (n == 32 ? 0xffffffffu : (1u << n) - 1) << (first * BITS);
          const unsigned codes = cells & (BITS == 1 ? 0xffffffffu : 0xaaaaaaaau);
          if (atomicOr(&held[(c0 >> LOG) + lane], codes) & cells) f |= dup;
        }
        continue;
      }
      if (!on[u]) continue;
      const unsigned sh = (cell[u] & (CELLS - 1)) * BITS;
      const uint32_t word = cell[u] >> LOG;
      const uint32_t before = __shfl_up_sync(active, word, 1);
      if (!__any_sync(active, lane != 0 && before == word)) {
        const unsigned code = BITS == 1 || !ok[u] ? 1u : 2u;
        if ((atomicOr(&held[word], code << sh) >> sh) & CODE) f |= dup;
        continue;
      }
      const unsigned same = __match_any_sync(active, word);
      const unsigned codes = __reduce_or_sync(same, (BITS == 1 || !ok[u] ? 1u : 2u) << sh);
      // A cell twice in the warp leaves fewer distinct cells than lanes.
      if (__popc(__reduce_or_sync(same, 1u << (cell[u] & (CELLS - 1)))) != __popc(same)) f |= dup;
      const unsigned leader = __ffs(same) - 1;
      unsigned old = 0;
      if (lane == leader) old = atomicOr(&held[word], codes);
      old = __shfl_sync(same, old, leader);
      if ((old >> sh) & CODE) f |= dup;
    }
  }
  if (f) atomicOr(flags, f);
}

}  // namespace

void scatter_cells(Context& ctx, const CellKeys& k, int64_t rows, const double* vals, const uint8_t* valid,
                   double* mat, uint32_t* held, int bits, unsigned* flags, unsigned dup, unsigned nonfinite) {
  if (rows <= 0) return;
  auto launch = [&](auto one, auto two, int per_thread) {
    const unsigned g = blocks_for((uint64_t)(rows + per_thread - 1) / per_thread, 256, 148 * 16);
    (bits == 1 ? one : two)<<<g, 256, 0, ctx.stream>>>(k, rows, vals, valid, mat, held, flags, dup, nonfinite);
  };
  constexpr int R = kScatterRows;
  if (k.n > 4) launch(scatter_cells_kernel<2 * kMaxDims, 1, 1>, scatter_cells_kernel<2 * kMaxDims, 2, 1>, 1);
  else if (rows < kManyRows) launch(scatter_cells_kernel<4, 1, 1>, scatter_cells_kernel<4, 2, 1>, 1);
  else if (k.n <= 2) launch(scatter_cells_kernel<2, 1, R>, scatter_cells_kernel<2, 2, R>, R);
  else if (k.n == 3) launch(scatter_cells_kernel<3, 1, R>, scatter_cells_kernel<3, 2, R>, R);
  else launch(scatter_cells_kernel<4, 1, R>, scatter_cells_kernel<4, 2, R>, R);
  ctx.kernels++;
  EF_LAUNCH_CHECK();
}

}  // namespace ef
