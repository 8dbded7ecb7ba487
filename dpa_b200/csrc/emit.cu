// emit.cu -- curve emission: prune, index pairs and angular-velocity colors of
// one round, one warp per particle, compacted with ballot/popc.
//
// Restates, data-parallel, particle_advector::prune_integral_curves
// (particle_advector.cpp:402-408), index_generator::generate
// (index_generator.cpp:10-39) and color_generator::
// generate_from_angular_velocities (color_generator.cpp:37-58). The output is
// the reference's round curve: vertices in round-particle order, invalid
// sentinels removed, index pairs (i, i + 1) for consecutive vertices neither
// of which is the terminal sentinel, and one color per vertex.
#include <cmath>

#include "kernels.cuh"
#include "sample.cuh"

namespace dpa {

namespace {

constexpr int kEmitWarps = 8;

struct V3 {
  float x, y, z;
};

__device__ __forceinline__ V3 load3(const float* p) { return {p[0], p[1], p[2]}; }

__device__ __forceinline__ void store3(float* p, const V3& v) {
  p[0] = v.x;
  p[1] = v.y;
  p[2] = v.z;
}

// Eigen 3.3 squaredNorm / dot on 3 elements: c0 + (c1 + c2).
__device__ __forceinline__ float sum3(float a, float b, float c) {
  return __fadd_rn(a, __fadd_rn(b, c));
}

// Eigen normalized(): v / sqrt(|v|^2), or v unchanged when |v|^2 == 0.
__device__ __forceinline__ V3 normalized(V3 v) {
  const float z = sum3(__fmul_rn(v.x, v.x), __fmul_rn(v.y, v.y), __fmul_rn(v.z, v.z));
  if (z > 0.0f) {
    const float n = __fsqrt_rn(z);
    v.x = __fdiv_rn(v.x, n);
    v.y = __fdiv_rn(v.y, n);
    v.z = __fdiv_rn(v.z, n);
  }
  return v;
}

// atan2(|prev x next|, prev . next) (color_generator.cpp:51-54).
__device__ __forceinline__ float angular_velocity(const V3& a, const V3& b) {
  const float cx = __fsub_rn(__fmul_rn(a.y, b.z), __fmul_rn(a.z, b.y));
  const float cy = __fsub_rn(__fmul_rn(a.z, b.x), __fmul_rn(a.x, b.z));
  const float cz = __fsub_rn(__fmul_rn(a.x, b.y), __fmul_rn(a.y, b.x));
  const float norm = __fsqrt_rn(sum3(__fmul_rn(cx, cx), __fmul_rn(cy, cy), __fmul_rn(cz, cz)));
  const float dot = sum3(__fmul_rn(a.x, b.x), __fmul_rn(a.y, b.y), __fmul_rn(a.z, b.z));
  return atan2f(norm, dot);
}

// Sum of counts[0 .. n) over a warp.
__device__ __forceinline__ uint64_t warp_sum(const uint32_t* counts, uint64_t n, unsigned lane) {
  uint64_t sum = 0;
  for (uint64_t i = lane; i < n; i += 32) sum += counts[i];
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
  return sum;
}

template <bool kIndex64, bool kColors, bool kScan>
__global__ void __launch_bounds__(kEmitWarps * 32) emit_kernel(const EmitArgs e) {
  const uint64_t k = uint64_t(blockIdx.x) * kEmitWarps + (threadIdx.x >> 5);
  if (k >= e.count) return;
  const unsigned lane = threadIdx.x & 31u;
  const unsigned lanes_below = (1u << lane) - 1u;

  // Pass 1: copy the particle's surviving raw vertices to their pruned slots.
  const float* raw = e.raw_vertices + 3 * e.raw_offsets[k];
  const uint64_t raw_in = e.remaining_in ? e.remaining_in[k] + 2 : e.raw_offsets[k + 1] - e.raw_offsets[k];
  const uint64_t raw_count = raw_in - e.remaining[k];
  uint64_t first, segment;
  if constexpr (kScan) {
    first = warp_sum(e.kept_vertices, k, lane);
    segment = warp_sum(e.kept_segments, k, lane);
    if (k + 1 == e.count && lane == 0) {
      e.totals[0] = first + e.kept_vertices[k];
      e.totals[1] = segment + e.kept_segments[k];
    }
  } else {
    first = e.vertex_offsets[k];
    segment = e.segment_offsets[k];
  }
  uint64_t cursor = first;
  for (uint64_t j0 = 0; j0 < raw_count; j0 += 32) {
    const uint64_t j = j0 + lane;
    V3 v = {0.0f, 0.0f, 0.0f};
    bool keep = false;
    if (j < raw_count) {
      v = load3(raw + 3 * j);
      keep = !equals3(v.x, v.y, v.z, kInvalid);
    }
    const unsigned mask = __ballot_sync(0xffffffffu, keep);
    if (keep) store3(e.vertices + 3 * (cursor + __popc(mask & lanes_below)), v);
    cursor += __popc(mask);
  }
  __syncwarp();

  // Pass 2: index pairs and colors over the particle's pruned vertices. The
  // last one is always the terminal sentinel, so no pair or neighbour reaches
  // into another particle's curve; the reference's "vertex_index > 1" test
  // (color_generator.cpp:50) is applied to the round-level index.
  const uint64_t kept = e.kept_vertices[k];
  for (uint64_t m0 = 0; m0 < kept; m0 += 32) {
    const uint64_t m = m0 + lane;
    const bool valid = m < kept;
    const uint64_t local = first + m;
    const uint64_t global = e.vertex_base + local;
    bool pair = false;
    V3 y = {0.0f, 0.0f, 0.0f};
    bool terminal = true, next_open = false, prev_open = false;
    V3 yn = y, yp = y;
    if (valid) {
      y = load3(e.vertices + 3 * local);
      terminal = equals3(y.x, y.y, y.z, kTerminal);
      if (m + 1 < kept) {
        yn = load3(e.vertices + 3 * (local + 1));
        next_open = !equals3(yn.x, yn.y, yn.z, kTerminal);
      }
      if (m > 0 && global > 1) {
        yp = load3(e.vertices + 3 * (local - 1));
        prev_open = !equals3(yp.x, yp.y, yp.z, kTerminal);
      }
      pair = !terminal && next_open;
    }
    const unsigned mask = __ballot_sync(0xffffffffu, pair);
    if (pair) {
      const uint64_t slot = 2 * (segment + __popc(mask & lanes_below));
      if constexpr (kIndex64) {
        uint64_t* out = static_cast<uint64_t*>(e.indices);
        out[slot] = global;
        out[slot + 1] = global + 1;
      } else {
        uint32_t* out = static_cast<uint32_t*>(e.indices);
        out[slot] = uint32_t(global);
        out[slot + 1] = uint32_t(global + 1);
      }
    }
    segment += __popc(mask);
    if constexpr (kColors) {
      if (valid) {
        float color = 0.0f;
        if (!terminal) {
          V3 a = {0.0f, 0.0f, 0.0f}, b = {0.0f, 0.0f, 0.0f};
          if (prev_open)
            a = normalized({__fsub_rn(y.x, yp.x), __fsub_rn(y.y, yp.y), __fsub_rn(y.z, yp.z)});
          if (next_open)
            b = normalized({__fsub_rn(yn.x, y.x), __fsub_rn(yn.y, y.y), __fsub_rn(yn.z, y.z)});
          color = angular_velocity(a, b);
        }
        e.colors[local] = color;
      }
    }
  }
}

// Curve offsets: the exclusive scans of the per-particle kept-vertex and
// kept-segment counts (uint32) into uint64 offsets, the data-parallel form of
// the running positions that index_generator::generate (index_generator.cpp:
// 10-39) and prune_integral_curves walk serially. Three passes over tiles of
// kScanTileItems particles: tile sums, one block's scan of the tile sums
// (which also writes the two totals), and each tile's scan plus its prefix.
constexpr int kScanThreads = 256;
constexpr int kScanItems = 8;  // consecutive particles per thread
constexpr uint64_t kScanTileItems = uint64_t(kScanThreads) * kScanItems;

// Block-wide exclusive scan of one pair of values per thread; returns the
// block's totals through total.
__device__ __forceinline__ ulonglong2 block_exclusive_scan2(ulonglong2 v, ulonglong2* warp_sums,
                                                           ulonglong2* total) {
  const unsigned lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
  ulonglong2 x = v;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const unsigned long long a = __shfl_up_sync(0xffffffffu, x.x, o);
    const unsigned long long b = __shfl_up_sync(0xffffffffu, x.y, o);
    if (lane >= unsigned(o)) {
      x.x += a;
      x.y += b;
    }
  }
  if (lane == 31) warp_sums[warp] = x;
  __syncthreads();
  ulonglong2 before = make_ulonglong2(0, 0), all = make_ulonglong2(0, 0);
  for (unsigned w = 0; w < blockDim.x / 32; ++w) {
    const ulonglong2 ws = warp_sums[w];
    if (w < warp) {
      before.x += ws.x;
      before.y += ws.y;
    }
    all.x += ws.x;
    all.y += ws.y;
  }
  __syncthreads();  // warp_sums may be reused by the caller's next scan
  *total = all;
  return make_ulonglong2(before.x + x.x - v.x, before.y + x.y - v.y);
}

__device__ __forceinline__ ulonglong2 load_counts(const uint32_t* a, const uint32_t* b,
                                                  uint64_t n, uint64_t i) {
  return i < n ? make_ulonglong2(a[i], b[i]) : make_ulonglong2(0, 0);
}

__global__ void __launch_bounds__(kScanThreads) offsets_tile_sums_kernel(
    const uint32_t* a, const uint32_t* b, uint64_t n, ulonglong2* tile_sums) {
  __shared__ ulonglong2 warp_sums[kScanThreads / 32];
  const uint64_t first = uint64_t(blockIdx.x) * kScanTileItems;
  ulonglong2 sum = make_ulonglong2(0, 0);
#pragma unroll
  for (int j = 0; j < kScanItems; ++j) {  // coalesced: item j * threads + t
    const ulonglong2 v = load_counts(a, b, n, first + uint64_t(j) * kScanThreads + threadIdx.x);
    sum.x += v.x;
    sum.y += v.y;
  }
  ulonglong2 total;
  block_exclusive_scan2(sum, warp_sums, &total);
  if (threadIdx.x == 0) tile_sums[blockIdx.x] = total;
}

// One block: tile sums -> exclusive tile prefixes in place, in chunks of
// kScanThreads with a running carry; totals receives the grand totals.
__global__ void __launch_bounds__(kScanThreads) offsets_tile_prefix_kernel(
    ulonglong2* tile_sums, uint64_t tiles, unsigned long long* totals) {
  __shared__ ulonglong2 warp_sums[kScanThreads / 32];
  ulonglong2 carry = make_ulonglong2(0, 0);
  for (uint64_t base = 0; base < tiles; base += kScanThreads) {
    const uint64_t i = base + threadIdx.x;
    const ulonglong2 v = i < tiles ? tile_sums[i] : make_ulonglong2(0, 0);
    ulonglong2 total;
    const ulonglong2 ex = block_exclusive_scan2(v, warp_sums, &total);
    if (i < tiles) tile_sums[i] = make_ulonglong2(carry.x + ex.x, carry.y + ex.y);
    carry.x += total.x;
    carry.y += total.y;
  }
  if (threadIdx.x == 0) {
    totals[0] = carry.x;
    totals[1] = carry.y;
  }
}

__global__ void __launch_bounds__(kScanThreads) offsets_tiles_kernel(
    const uint32_t* a, const uint32_t* b, uint64_t n, const ulonglong2* tile_prefix,
    uint64_t* out_a, uint64_t* out_b) {
  __shared__ ulonglong2 warp_sums[kScanThreads / 32];
  const uint64_t first = uint64_t(blockIdx.x) * kScanTileItems + uint64_t(threadIdx.x) * kScanItems;
  ulonglong2 v[kScanItems];
  ulonglong2 sum = make_ulonglong2(0, 0);
#pragma unroll
  for (int j = 0; j < kScanItems; ++j) {
    v[j] = load_counts(a, b, n, first + j);
    sum.x += v[j].x;
    sum.y += v[j].y;
  }
  ulonglong2 total;
  const ulonglong2 ex = block_exclusive_scan2(sum, warp_sums, &total);
  const ulonglong2 prefix = tile_prefix[blockIdx.x];
  ulonglong2 run = make_ulonglong2(prefix.x + ex.x, prefix.y + ex.y);
#pragma unroll
  for (int j = 0; j < kScanItems; ++j) {
    const uint64_t i = first + j;
    if (i < n) {
      out_a[i] = run.x;
      out_b[i] = run.y;
    }
    run.x += v[j].x;
    run.y += v[j].y;
  }
}

// The three passes as one block's, for few particles: launches cost more there
// than the scan (kOneBlockOffsets).
constexpr int kOneBlockThreads = 1024;
__global__ void __launch_bounds__(kOneBlockThreads) offsets_one_block_kernel(
    const uint32_t* a, const uint32_t* b, uint64_t n, uint64_t* out_a, uint64_t* out_b,
    unsigned long long* totals) {
  __shared__ ulonglong2 warp_sums[kOneBlockThreads / 32];
  ulonglong2 carry = make_ulonglong2(0, 0);
  for (uint64_t base = 0; base < n; base += kOneBlockThreads) {
    const uint64_t i = base + threadIdx.x;
    const ulonglong2 v = load_counts(a, b, n, i);
    ulonglong2 total;
    const ulonglong2 ex = block_exclusive_scan2(v, warp_sums, &total);
    if (i < n) {
      out_a[i] = carry.x + ex.x;
      out_b[i] = carry.y + ex.y;
    }
    carry.x += total.x;
    carry.y += total.y;
  }
  if (threadIdx.x == 0) {
    totals[0] = carry.x;
    totals[1] = carry.y;
  }
}

// Node layouts: one float4 (F32) or (x, y, z, 0) half/bfloat quad per node.
// F32_EDGES: record t holds nodes t and t + 1 along axis 2, each component's
// pair side by side (sample.cuh); the last node of a row repeats itself, and
// no cell reads that record's second half. In a tiled layout of nodes the first
// node of a tile's row also ends the row of the tile before it.
template <int kStorage, bool kTiled>
__global__ void repack_kernel(const float* xyzv, uint64_t nodes, const FieldView f, void* out) {
  const uint64_t t = uint64_t(blockIdx.x) * blockDim.x + threadIdx.x;
  if (t >= nodes) return;
  const float x = xyzv[3 * t], y = xyzv[3 * t + 1], z = xyzv[3 * t + 2];
  const uint32_t n2 = uint32_t(f.n[2]);
  uint64_t at = t, copy = t;
  if constexpr (kTiled) {  // one slice of fewer than 2^32 nodes
    const uint32_t row = uint32_t(t) / n2, i2 = uint32_t(t) - row * n2;
    const uint32_t i0 = row / uint32_t(f.n[1]), i1 = row - i0 * uint32_t(f.n[1]);
    at = copy = tiled_node(f.tile, i0, i1, i2);
    if (kStorage != DPA_STORAGE_F32_EDGES && i2 > 0 &&
        tile_bits(f.tile, 2, float(i2)) != tile_bits(f.tile, 2, float(i2 - 1)))
      copy = uint64_t(tiled_node(f.tile, i0, i1, i2 - 1)) + 1;
  }
  auto store = [&](auto* o, auto v) {
    o[at] = v;
    if (kTiled && copy != at) o[copy] = v;
  };
  if constexpr (kStorage == DPA_STORAGE_F32_EDGES) {
    const uint64_t u = (t % n2) + 1 < n2 ? t + 1 : t;
    float4* o = reinterpret_cast<float4*>(out) + 2 * at;
    o[0] = make_float4(x, xyzv[3 * u], y, xyzv[3 * u + 1]);
    o[1] = make_float4(z, xyzv[3 * u + 2], 0.0f, 0.0f);
  } else if constexpr (kStorage == DPA_STORAGE_F32) {
    store(reinterpret_cast<float4*>(out), make_float4(x, y, z, 0.0f));
  } else if constexpr (kStorage == DPA_STORAGE_F16) {
    const __half2 a = __floats2half2_rn(x, y);
    const __half2 b = __floats2half2_rn(z, 0.0f);
    store(reinterpret_cast<uint2*>(out), make_uint2(*reinterpret_cast<const unsigned*>(&a),
                                                    *reinterpret_cast<const unsigned*>(&b)));
  } else {
    const __nv_bfloat162 a = __floats2bfloat162_rn(x, y);
    const __nv_bfloat162 b = __floats2bfloat162_rn(z, 0.0f);
    store(reinterpret_cast<uint2*>(out), make_uint2(*reinterpret_cast<const unsigned*>(&a),
                                                    *reinterpret_cast<const unsigned*>(&b)));
  }
}

template <int kStorage>
cudaError_t launch_repack_as(const float* xyzv, uint64_t nodes, const FieldView& f, void* out,
                             cudaStream_t stream) {
  const unsigned grid = unsigned((nodes + 255) / 256);
  if (f.tiled) repack_kernel<kStorage, true><<<grid, 256, 0, stream>>>(xyzv, nodes, f, out);
  else repack_kernel<kStorage, false><<<grid, 256, 0, stream>>>(xyzv, nodes, f, out);
  return cudaGetLastError();
}

inline unsigned blocks_for(uint64_t n, unsigned block) { return unsigned((n + block - 1) / block); }

}  // namespace

cudaError_t launch_emit(const EmitArgs& e, bool index64, bool colors, cudaStream_t stream) {
  if (e.count == 0) return cudaSuccess;
  const dim3 grid(blocks_for(e.count, kEmitWarps)), block(kEmitWarps * 32);
  auto launch = [&](auto scan) {
    constexpr bool kScan = decltype(scan)::value;
    if (index64) {
      if (colors) emit_kernel<true, true, kScan><<<grid, block, 0, stream>>>(e);
      else emit_kernel<true, false, kScan><<<grid, block, 0, stream>>>(e);
    } else {
      if (colors) emit_kernel<false, true, kScan><<<grid, block, 0, stream>>>(e);
      else emit_kernel<false, false, kScan><<<grid, block, 0, stream>>>(e);
    }
  };
  if (e.vertex_offsets) launch(std::false_type{});
  else launch(std::true_type{});
  return cudaGetLastError();
}

uint64_t curve_offsets_scratch_bytes(uint64_t count) {
  return ((count + kScanTileItems - 1) / kScanTileItems) * sizeof(ulonglong2) + 16;
}

cudaError_t launch_curve_offsets(const uint32_t* kept_vertices, const uint32_t* kept_segments,
                                 uint64_t count, void* scratch, uint64_t* vertex_offsets,
                                 uint64_t* segment_offsets, unsigned long long* totals,
                                 cudaStream_t stream) {
  if (count == 0) return cudaMemsetAsync(totals, 0, 16, stream);
  if (count <= kOneBlockOffsets) {
    offsets_one_block_kernel<<<1, kOneBlockThreads, 0, stream>>>(
        kept_vertices, kept_segments, count, vertex_offsets, segment_offsets, totals);
    return cudaGetLastError();
  }
  const uint64_t tiles = (count + kScanTileItems - 1) / kScanTileItems;
  if (tiles > 0x7fffffffull) return cudaErrorInvalidValue;
  ulonglong2* sums = static_cast<ulonglong2*>(scratch);
  offsets_tile_sums_kernel<<<unsigned(tiles), kScanThreads, 0, stream>>>(
      kept_vertices, kept_segments, count, sums);
  DPA_CUDA_TRY(cudaGetLastError());
  offsets_tile_prefix_kernel<<<1, kScanThreads, 0, stream>>>(sums, tiles, totals);
  DPA_CUDA_TRY(cudaGetLastError());
  offsets_tiles_kernel<<<unsigned(tiles), kScanThreads, 0, stream>>>(
      kept_vertices, kept_segments, count, sums, vertex_offsets, segment_offsets);
  return cudaGetLastError();
}

uint64_t field_node_bytes(int storage) {
  return storage == DPA_STORAGE_F32_EDGES ? 32 : storage == DPA_STORAGE_F32 ? 16 : 8;
}

cudaError_t launch_repack(const float* xyzv, uint64_t nodes, const FieldView& f, void* out,
                          cudaStream_t stream) {
  if (nodes == 0) return cudaSuccess;
  switch (f.storage) {
    case DPA_STORAGE_F32: return launch_repack_as<DPA_STORAGE_F32>(xyzv, nodes, f, out, stream);
    case DPA_STORAGE_F16: return launch_repack_as<DPA_STORAGE_F16>(xyzv, nodes, f, out, stream);
    case DPA_STORAGE_BF16: return launch_repack_as<DPA_STORAGE_BF16>(xyzv, nodes, f, out, stream);
    case DPA_STORAGE_F32_EDGES:
      return launch_repack_as<DPA_STORAGE_F32_EDGES>(xyzv, nodes, f, out, stream);
    default: return cudaErrorInvalidValue;
  }
}

namespace {

constexpr int kSpeedBlocks = 64, kSpeedThreads = 256, kSpeedNodes = 4;  // per thread

// The sampled nodes are the golden-ratio sequence over the field: evenly spread and in no
// step with its rows.
__global__ void __launch_bounds__(kSpeedThreads) field_speed_kernel(
    const float* xyzv, uint64_t nodes, uint32_t n2, float s0, float s1, float s2, double* sums) {
  const float per_cell[3] = {1.0f / s2, 1.0f / s1, 1.0f / s0};  // components in reversed order
  double sum[2] = {0.0, 0.0};
  for (int j = 0; j < kSpeedNodes; ++j) {
    const uint64_t i = (uint64_t(blockIdx.x) * kSpeedThreads + threadIdx.x) * kSpeedNodes + j;
    uint64_t node = __umul64hi(i * 0x9E3779B97F4A7C15ull, nodes);
    if (node % n2 + 1 == n2) --node;  // a row's last node has none behind it
    const float* at = xyzv + 3 * node;
    for (int c = 0; c < 3; ++c) {
      const double v = double(at[c]) * double(per_cell[c]);
      const double next = double(at[3 + c]) * double(per_cell[c]);
      if (!isfinite(v) || !isfinite(next)) continue;
      sum[0] += v * v;
      sum[1] += (next - v) * (next - v);
    }
  }
  __shared__ double warps[2][kSpeedThreads / 32];
  for (int k = 0; k < 2; ++k) {
    for (int o = 16; o > 0; o >>= 1) sum[k] += __shfl_xor_sync(0xffffffffu, sum[k], o);
    if ((threadIdx.x & 31u) == 0) warps[k][threadIdx.x >> 5] = sum[k];
  }
  __syncthreads();
  if (threadIdx.x >= 2) return;
  double total = 0.0;
  for (double w : warps[threadIdx.x]) total += w;
  atomicAdd(sums + threadIdx.x, total);
  if (threadIdx.x == 0) atomicAdd(sums + 2, double(kSpeedThreads * kSpeedNodes));
}

}  // namespace

cudaError_t launch_field_speed(const float* xyzv, uint64_t nodes, uint32_t n2,
                               const float spacing[3], double* sums, cudaStream_t stream) {
  field_speed_kernel<<<kSpeedBlocks, kSpeedThreads, 0, stream>>>(
      xyzv, nodes, n2, spacing[0], spacing[1], spacing[2], sums);
  return cudaGetLastError();
}

// Where the lines lie, measured on curl noise with 2 million seeds of up to 1000
// steps of a quarter cell (rows, tiles; threads per SM in brackets, ms):
//   F32 320^3, 0.5 GB   9.0 [1024]             9.0 [1024]
//   F32 400^3, 1.0 GB  20.8 [1024], 12.4 [512]  10.0 [1024]
//   F32 512^3, 2.1 GB  29.1 [1024], 14.2 [512]  13.8 [1024], 11.9 [768], 14.2 [512]
//   F32 768^3, 7.2 GB                           32.5 [1024], 16.8 [768], 17.0 [512]
//   F16 512^3, 1.1 GB  15.9 [1024], 11.1 [768]  10.4 [1024], 11.3 [768]
//   F16 768^3, 3.6 GB                           15.5 [1024], 13.6 [768]
// and 500 steps of curl noise / of a field that varies over 8 nodes only:
//   F32 330^3, 0.6 GB   6.6 / 5.8 [1024]        6.6 / 5.9 [1024]
//   F16 420^3, 0.6 GB   6.0 / 5.5 [1024]        6.3 / 6.0 [1024]
//   F16 512^3, 1.1 GB  12.0 / 5.6 [1024]        7.1 / 6.1 [1024],  7.7 / 6.3 [768]
//   F16 640^3, 2.1 GB  18.0 / 5.8 [1024]        8.7 / 6.3 [1024],  9.1 / 6.6 [768]
//   F16 768^3, 3.6 GB                          10.6 / 6.4 [1024],  9.9 / 6.9 [768]
//   edges 260^3, 0.6 GB 5.1 / 4.5 [1024]        5.3 / 4.8 [1024],  5.8 / 5.0 [768]
//   edges 400^3, 2.0 GB 16.7 / 4.7 [1024]       8.5 / 5.1 [1024],  8.6 / 5.5 [768]
//   edges 450^3, 2.9 GB                         9.2 / 5.2 [1024],  9.0 / 5.6 [768]
//   edges 500^3, 4.0 GB 19.4 / 5.2 [1024]      10.1 / 5.3 [1024],  9.5 / 5.8 [768]
// (a lattice of 2 million seeds in edge records of 256^3, 0.5 GB: 2.6 in rows, 2.35 in
// tiles). Beyond about half a gigabyte the gathers of a full SM miss the address
// translation cache: random 16-byte gathers fall from 2079 GB/s in a table of
// 256 MB to 892 in one of 2 GB. Tiles keep a particle's path in fewer pages, and
// fewer warps in flight leave room for their misses: above 1.25 GiB for F32 nodes, above
// 3 GiB for the others, whose gathers are half as many or half as large. Between those
// the others gain by it where a step is long, and lose where particles stay in a cell
// (launch_shape.hpp): 300 steps of 2 million seeds, ms in rows and at
// 1024 and 768 threads, of curl noise at 0.6 cells a step, F16 580^3 20.7, 13.3, 9.0, edges
// 400^3 19.8, 13.2, 8.5; of noise over 8 nodes at 0.25, 4.7, 4.5, 5.0 and 4.5, 4.1, 4.6. F32
// nodes at 450^3, 1.5 GB: 24.8, 16.8, 11.9 and 6.2, 4.2, 4.6.
uint64_t choose_layout(FieldView& v, uint32_t slices, bool rows) {
  constexpr uint64_t kTileBytes = 512ull << 20;
  constexpr uint64_t kFewerThreadsBytes = 1280ull << 20, kAlwaysFewerBytes = 3072ull << 20;
  const uint64_t node_bytes = field_node_bytes(v.storage);
  const uint64_t nodes = uint64_t(v.n[0]) * uint64_t(v.n[1]) * uint64_t(v.n[2]);
  v.tiled = 0;
  v.tile = TileLayout{};
  v.threads_per_sm = 0;
  v.limit_speed = 0.0f;
  if (slices != 1 || nodes * node_bytes < kTileBytes) return nodes * slices;
  // About 64 nodes an axis, of a 2 MiB page for F32 nodes (axis 2: 32); tiles of
  // one axis are as even as they can be, and a row of one tile ends in no node of the
  // next, so that at most an eighth is allocated beyond the field (a field of
  // 65 x 15,645 x 33 F32 nodes 11 %, 512^3 3 %). A field that finds no room for that
  // lies in rows.
  const bool edges = v.storage == DPA_STORAGE_F32_EDGES;
  const uint32_t want[3] = {64u, edges ? 32u : 64u, v.storage == DPA_STORAGE_F32 || edges ? 32u : 64u};
  uint64_t size[3], tiles[3];
  for (int i = 0; i < 3; ++i) {
    tiles[i] = (uint64_t(v.n[i]) + want[i] - 1) / want[i];
    size[i] = (uint64_t(v.n[i]) + tiles[i] - 1) / tiles[i];
  }
  const uint64_t row = size[2] + (edges || tiles[2] == 1 ? 0 : 1);
  const uint64_t tile = size[0] * size[1] * row;
  const uint64_t total = tile * tiles[0] * tiles[1] * tiles[2];
  v.threads_per_sm = 512;
  // The index is 32 bits wide; an axis of one node has no cells.
  if (rows || size[0] < 2 || size[1] < 2 || size[2] < 2 || total >= (1ull << 32)) return nodes;
  const uint64_t bytes = total * node_bytes;
  v.threads_per_sm = bytes > kFewerThreadsBytes ? 768 : 0;
  if (v.threads_per_sm && v.storage != DPA_STORAGE_F32 && bytes <= kAlwaysFewerBytes)
    v.limit_speed = 1.0f;
  v.tiled = 1;
  for (int i = 0; i < 3; ++i) {
    v.tile.inverse[i] = 1.0f / float(size[i]);
    if (double(v.tile.inverse[i]) * double(size[i]) < 1.0)
      v.tile.inverse[i] = std::nextafter(v.tile.inverse[i], 2.0f);
    v.tile.magic[i] = uint32_t((1ull << 32) / size[i] + 1);
  }
  v.tile.stride[0] = uint32_t(size[1] * row);
  v.tile.stride[1] = uint32_t(row);
  v.tile.jump[0] = uint32_t(tiles[1] * tiles[2] * tile - size[0] * size[1] * row);
  v.tile.jump[1] = uint32_t(tiles[2] * tile - size[1] * row);
  v.tile.jump[2] = uint32_t(tile - size[2]);
  v.tile.bias = 0u - 0x4B000000u * (v.tile.jump[0] + v.tile.jump[1] + v.tile.jump[2]);
  return total;
}

}  // namespace dpa
