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

// A key column read by key_columns: its values widened to int64 (or left where
// they are: int64 ones), their largest value and what makes them no positions.
struct KeyColumn {
  const void* in;
  int64_t rows;
  int64_t* out;  // null: not written
  int kind;      // Kind
};
constexpr int kKeyColumns = 24;
constexpr int kKeysRead = 2048;  // keys a block reads at a time
struct KeyColumns {
  KeyColumn col[kKeyColumns];
};
struct KeyColumnStats {
  unsigned long long max;
  unsigned long long flags;  // 1: a negative key, 2: one of 2^63 or more
};

template <class T>
__device__ void read_keys(const KeyColumn& c, int64_t& top, int& f) {
  const T* in = (const T*)c.in;
  auto take = [&](T v, int64_t i) {
    int64_t w = (int64_t)v;
    if constexpr (sizeof(T) == 8 && !std::is_signed<T>::value) {
      if ((uint64_t)v >= (1ull << 63)) { f |= 2; w = -1; }
    }
    if (w < 0) f |= 1;
    if (c.out) c.out[i] = w;
    if (w > top) top = w;
  };
  // Blocks of kKeysRead keys, 16 bytes a load for 8-byte keys at an aligned
  // address (a caller's column may start at any key).
  constexpr int PER = kKeysRead / 256;
  const bool pairs = sizeof(T) == 8 && ((uintptr_t)in & 15) == 0;
  for (int64_t base = (int64_t)blockIdx.x * kKeysRead; base < c.rows; base += (int64_t)gridDim.x * kKeysRead) {
    if (sizeof(T) == 8 && pairs && base + kKeysRead <= c.rows) {
      longlong2 v[PER / 2];
#pragma unroll
      for (int u = 0; u < PER / 2; u++) v[u] = ((const longlong2*)(in + base))[u * 256 + threadIdx.x];
#pragma unroll
      for (int u = 0; u < PER / 2; u++) {
        take((T)v[u].x, base + 2 * (u * 256 + threadIdx.x));
        take((T)v[u].y, base + 2 * (u * 256 + threadIdx.x) + 1);
      }
      continue;
    }
    T v[PER];
#pragma unroll
    for (int u = 0; u < PER; u++) {
      const int64_t i = base + u * 256 + threadIdx.x;
      v[u] = i < c.rows ? in[i] : T(0);
    }
#pragma unroll
    for (int u = 0; u < PER; u++) {
      const int64_t i = base + u * 256 + threadIdx.x;
      if (i < c.rows) take(v[u], i);
    }
  }
}

// A call's key columns, a grid row a column: bound by HBM beyond a few MB, by
// its launch below. One atomic a block (one a warp made 12 us of a column of
// 512,000 keys, 3 us' worth of bytes), and one launch and one wait for all
// columns of all operands (twelve of each for a pipeline of three 4-key tables:
// 480 us of its 1150, 40 now). 268 million keys in four columns: 308 us, 7.0 TB/s;
// 8-byte loads a grid apart took 509, a launch a column 400.
__global__ void __launch_bounds__(256) key_columns(KeyColumns a, KeyColumnStats* __restrict__ stats) {
  __shared__ long long s_top[8];
  __shared__ int s_flags[8];
  const KeyColumn& c = a.col[blockIdx.y];
  int64_t top = -1;
  int f = 0;
  switch ((Kind)c.kind) {
    case Kind::Int8: read_keys<int8_t>(c, top, f); break;
    case Kind::UInt8: read_keys<uint8_t>(c, top, f); break;
    case Kind::Int16: read_keys<int16_t>(c, top, f); break;
    case Kind::UInt16: read_keys<uint16_t>(c, top, f); break;
    case Kind::Int32: read_keys<int32_t>(c, top, f); break;
    case Kind::UInt32: read_keys<uint32_t>(c, top, f); break;
    case Kind::UInt64: read_keys<uint64_t>(c, top, f); break;
    default: read_keys<int64_t>(c, top, f); break;
  }
  for (int o = 16; o; o >>= 1) {
    const long long other = __shfl_xor_sync(0xffffffffu, (long long)top, o);
    if (other > top) top = other;
  }
  f = __reduce_or_sync(0xffffffffu, (unsigned)f);
  if ((threadIdx.x & 31) == 0) {
    s_top[threadIdx.x >> 5] = top;
    s_flags[threadIdx.x >> 5] = f;
  }
  __syncthreads();
  if (threadIdx.x) return;
  for (int i = 1; i < 8; i++) {
    if (s_top[i] > top) top = s_top[i];
    f |= s_flags[i];
  }
  if (top >= 0) atomicMax(&stats[blockIdx.y].max, (unsigned long long)top);
  if (f) atomicOr(&stats[blockIdx.y].flags, (unsigned long long)f);
}

// key_columns over `cols`, and each column's statistics.
std::vector<KeyStats> read_key_columns(Context& ctx, const std::vector<KeyColumn>& cols) {
  cudaStream_t s = ctx.stream;
  std::vector<KeyStats> out(cols.size());
  for (size_t at = 0; at < cols.size(); at += kKeyColumns) {
    const int n = (int)std::min<size_t>(kKeyColumns, cols.size() - at);
    KeyColumns a;
    int64_t rows = 0;
    for (int i = 0; i < n; i++) {
      a.col[i] = cols[at + (size_t)i];
      rows = std::max(rows, a.col[i].rows);
    }
    DeviceBuffer<KeyColumnStats> stats((size_t)n, s);
    stats.zero();
    // Up to eight blocks an SM a column (a short column's spare blocks end at once).
    const unsigned g = blocks_for((uint64_t)rows, kKeysRead, (unsigned)ctx.sm_count * 8);
    key_columns<<<dim3(g, (unsigned)n), 256, 0, s>>>(a, stats.get());
    EF_LAUNCH_CHECK();
    ctx.kernels++;
    KeyColumnStats got[kKeyColumns];
    ReadBack back(ctx, s);
    back.add(got, stats.get(), (size_t)n);
    back.wait();
    for (int i = 0; i < n; i++) {
      KeyStats& k = out[at + (size_t)i];
      k.max = a.col[i].rows ? (int64_t)got[i].max : -1;
      k.negative = (got[i].flags & 1) != 0;
      k.too_large = (got[i].flags & 2) != 0;
    }
  }
  return out;
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
  if (!is_integer(c.kind)) fail(EINFOLD_INVALID, "keys_as_i64 of a non-integer column");
  DeviceBuffer<int64_t> out((size_t)(c.rows ? c.rows : 1), ctx.stream);
  *stats = read_key_columns(ctx, {KeyColumn{c.ptr(), c.rows, out.get(), (int)c.kind}})[0];
  return out;
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
  ReadBack back(ctx, s);
  back.add(&last, out + n - 1);
  back.add(&lastf, flags + n - 1);
  back.wait();
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

namespace {

struct CellDivisors {
  Divisor ny, stride[kMaxDims], extent[kMaxDims];
};

// Bound by HBM writes: 8 bytes a key and cell, two cells a thread (16 bytes a
// store), keys by multiplications. 67.1M cells of two keys: emitting them with
// a copy of the values, their validity bytes and keys from tables took 542 us,
// 162 now; 67.1M rows of a pipeline with one value column, tables of 1 GB, row
// numbers and their scan 1260 us, 162 now.
__global__ void __launch_bounds__(256) emit_keys_kernel(OutKeys keys, CellDivisors by, uint32_t ny, uint64_t cells) {
  for (uint64_t c = 2 * ((uint64_t)blockIdx.x * 256 + threadIdx.x); c < cells; c += 2ull * gridDim.x * 256) {
    const uint32_t x0 = by.ny((uint32_t)c), y0 = (uint32_t)c - x0 * ny;
    const bool wraps = y0 + 1 == ny, two = c + 1 < cells;
    const uint32_t x1 = x0 + wraps, y1 = wraps ? 0 : y0 + 1;
    for (int k = 0; k < keys.n; k++) {
      const bool in_x = keys.key[k].in_x != 0;
      auto key = [&](uint32_t p) {
        const uint32_t q = by.stride[k](p);
        return (int64_t)(q - by.extent[k](q) * (uint32_t)by.extent[k].d);
      };
      const int64_t k0 = key(in_x ? x0 : y0);
      const int64_t k1 = key(in_x ? x1 : y1);
      if (keys.width[k] == 8 && two) {
        *(longlong2*)((int64_t*)keys.out[k] + c) = make_longlong2(k0, k1);
      } else {
        store_key(keys.out[k], keys.width[k], (int64_t)c, k0);
        if (two) store_key(keys.out[k], keys.width[k], (int64_t)c + 1, k1);
      }
    }
  }
}

}  // namespace

void emit_keys(Context& ctx, const OutKeys& keys, uint64_t nx, uint64_t ny) {
  if (!nx || !ny || !keys.n) return;
  CellDivisors by;
  by.ny = Divisor(ny);
  for (int k = 0; k < keys.n; k++) {
    by.stride[k] = Divisor((uint64_t)keys.key[k].stride);
    by.extent[k] = Divisor((uint64_t)keys.key[k].extent);
  }
  emit_keys_kernel<<<blocks_for((nx * ny + 1) / 2, 256, (unsigned)ctx.sm_count * 32), 256, 0, ctx.stream>>>(
      keys, by, (uint32_t)ny, nx * ny);
  EF_LAUNCH_CHECK();
  ctx.kernels++;
}

std::vector<StagedKeys> stage_keys(Context& ctx, const std::vector<std::pair<const OperandD*, const Relation*>>& ops) {
  std::vector<StagedKeys> staged(ops.size());
  std::vector<KeyColumn> cols;
  for (size_t o = 0; o < ops.size(); o++) {
    StagedKeys& s = staged[o];
    const Relation& r = *ops[o].second;
    for (auto& k : ops[o].first->keys) {
      const Field& f = r.fields[k.col];
      if (f.dictionary || !is_integer(f.kind)) decline("a key column that isn't integers");
      for (auto& b : r.batches)
        if (b.columns[k.col].nulls() > 0) decline("a NULL key");
      s.cols.push_back(stage_column(ctx, r, k.col, false));
      DeviceColumn& c = s.cols.back();
      int64_t* out = nullptr;
      if (c.kind != Kind::Int64) {
        s.wide.emplace_back((size_t)(c.rows ? c.rows : 1), ctx.stream);
        out = s.wide.back().get();
      }
      s.keys.push_back(out ? out : (const int64_t*)c.ptr());
      cols.push_back(KeyColumn{c.ptr(), c.rows, out, (int)c.kind});
    }
  }
  const std::vector<KeyStats> stats = read_key_columns(ctx, cols);
  size_t at = 0;
  for (auto& s : staged)
    for (size_t i = 0; i < s.keys.size(); i++) {
      const KeyStats& st = stats[at++];
      if (st.negative || st.too_large) decline("a negative key, or one too large for int64");
      if (st.max == INT64_MAX) decline("a key whose extent doesn't fit");
      s.extent.push_back(st.max + 1);
    }
  return staged;
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
// Four rows a thread from kManyRows rows an SM on, which still fills the SMs; below,
// one (262,144 shuffled rows: 8.5 us against 23 with four, and 67 before).
constexpr int kScatterRows = 4;
constexpr int64_t kManyRows = 2048 * 4;

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
    const unsigned g = blocks_for((uint64_t)(rows + per_thread - 1) / per_thread, 256,
                                  (unsigned)ctx.sm_count * 16);
    (bits == 1 ? one : two)<<<g, 256, 0, ctx.stream>>>(k, rows, vals, valid, mat, held, flags, dup, nonfinite);
  };
  constexpr int R = kScatterRows;
  if (k.n > 4) launch(scatter_cells_kernel<2 * kMaxDims, 1, 1>, scatter_cells_kernel<2 * kMaxDims, 2, 1>, 1);
  else if (rows < kManyRows * ctx.sm_count) launch(scatter_cells_kernel<4, 1, 1>, scatter_cells_kernel<4, 2, 1>, 1);
  else if (k.n <= 2) launch(scatter_cells_kernel<2, 1, R>, scatter_cells_kernel<2, 2, R>, R);
  else if (k.n == 3) launch(scatter_cells_kernel<3, 1, R>, scatter_cells_kernel<3, 2, R>, R);
  else launch(scatter_cells_kernel<4, 1, R>, scatter_cells_kernel<4, 2, R>, R);
  ctx.kernels++;
  EF_LAUNCH_CHECK();
}

}  // namespace ef
