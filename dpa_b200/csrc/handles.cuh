// handles.cuh -- definitions of the opaque handles of include/dpa_b200.h
// (dpa_context, dpa_field) and the device/pinned buffers they own.
#pragma once

#include <algorithm>
#include <atomic>
#include <mutex>
#include <string>
#include <vector>

#include "kernels.cuh"

namespace dpa {

// Device blocks of destroyed fields, kept for the next field of about their size:
// a program that makes a field of each time step would otherwise spend more on
// allocating and freeing it than on using it. At most limit_ bytes in kMost blocks
// stay (a larger block is freed at once); the oldest go first, all when the context goes
// or when an allocation of any context of the process finds no memory. Blocks are given
// back only when the device has finished with them.
class SpareBlocks {
 public:
  static constexpr size_t kMost = 4;
  SpareBlocks() {
    std::lock_guard<std::mutex> guard(registry().lock);
    registry().all.push_back(this);
  }
  ~SpareBlocks() {
    std::lock_guard<std::mutex> guard(registry().lock);
    auto& all = registry().all;
    all.erase(std::remove(all.begin(), all.end(), this), all.end());
    release();
  }
  SpareBlocks(const SpareBlocks&) = delete;
  SpareBlocks& operator=(const SpareBlocks&) = delete;

  // A kept block of n bytes or up to an eighth more, or null.
  void* take(size_t n, size_t* bytes) {
    std::lock_guard<std::mutex> guard(lock_);
    for (size_t i = 0; i < count_; ++i) {
      if (blocks_[i].bytes < n || blocks_[i].bytes - n > n / 8) continue;
      *bytes = blocks_[i].bytes;
      return remove(i);
    }
    return nullptr;
  }
  void give(void* ptr, size_t bytes) {
    std::lock_guard<std::mutex> guard(lock_);
    if (bytes > limit_) {
      cudaFree(ptr);
      return;
    }
    shrink(limit_ - bytes, kMost - 1);
    blocks_[count_++] = {ptr, bytes};
  }
  void release() {
    std::lock_guard<std::mutex> guard(lock_);
    shrink(0, 0);
  }
  void set_limit(size_t bytes) {
    std::lock_guard<std::mutex> guard(lock_);
    limit_ = bytes;
    shrink(bytes, kMost);
  }
  // Returns what every context of the process keeps.
  static void release_everywhere() {
    std::lock_guard<std::mutex> guard(registry().lock);
    for (SpareBlocks* s : registry().all) s->release();
  }

 private:
  struct block {
    void* ptr;
    size_t bytes;
  };
  struct registry_type {
    std::mutex lock;
    std::vector<SpareBlocks*> all;
  };
  static registry_type& registry() {
    static registry_type* r = new registry_type;  // outlives every context
    return *r;
  }
  void* remove(size_t i) {
    void* ptr = blocks_[i].ptr;
    std::copy(blocks_ + i + 1, blocks_ + count_, blocks_ + i);
    --count_;
    return ptr;
  }
  // Frees the oldest until at most this many bytes and blocks are left.
  void shrink(size_t bytes, size_t blocks) {
    size_t held = 0;
    for (size_t i = 0; i < count_; ++i) held += blocks_[i].bytes;
    while (count_ && (held > bytes || count_ > blocks)) {
      held -= blocks_[0].bytes;
      cudaFree(remove(0));
    }
  }
  std::mutex lock_;
  size_t limit_ = size_t(1) << 30;
  block blocks_[kMost];
  size_t count_ = 0;
};

// Grow-only device buffer; freed by release() or when it goes out of scope
// (with its device current).
struct DeviceBuffer {
  void* ptr = nullptr;
  size_t bytes = 0;
  DeviceBuffer() = default;
  DeviceBuffer(const DeviceBuffer&) = delete;
  DeviceBuffer& operator=(const DeviceBuffer&) = delete;
  ~DeviceBuffer() { release(); }
  cudaError_t reserve(size_t n) {
    if (n <= bytes && ptr) return cudaSuccess;
    release();
    if (n == 0) n = 16;
    cudaError_t e = cudaMalloc(&ptr, n);
    if (e == cudaErrorMemoryAllocation) {
      cudaGetLastError();
      SpareBlocks::release_everywhere();
      e = cudaMalloc(&ptr, n);
    }
    if (e != cudaSuccess) {
      cudaGetLastError();  // not the next launch's error
      ptr = nullptr;
      return e;
    }
    bytes = n;
    return cudaSuccess;
  }
  // reserve() from the spare blocks where one fits, and release() to them.
  cudaError_t reserve_from(SpareBlocks& spare, size_t n, bool* kept = nullptr) {
    release();
    if (n) ptr = spare.take(n, &bytes);
    if (kept) *kept = ptr != nullptr;
    return ptr ? cudaSuccess : reserve(n);
  }
  void release_to(SpareBlocks& spare) {
    if (ptr) spare.give(ptr, bytes);
    ptr = nullptr;
    bytes = 0;
  }
  void release() {
    if (ptr) cudaFree(ptr);
    ptr = nullptr;
    bytes = 0;
  }
  template <class T>
  T* as() const { return static_cast<T*>(ptr); }
};

struct PinnedBuffer {
  void* ptr = nullptr;
  size_t bytes = 0;
  PinnedBuffer() = default;
  PinnedBuffer(const PinnedBuffer&) = delete;
  PinnedBuffer& operator=(const PinnedBuffer&) = delete;
  ~PinnedBuffer() { release(); }
  cudaError_t reserve(size_t n) {
    if (n <= bytes && ptr) return cudaSuccess;
    release();
    if (n == 0) n = 16;
    cudaError_t e = cudaMallocHost(&ptr, n);
    if (e != cudaSuccess) {
      ptr = nullptr;
      return e;
    }
    bytes = n;
    return cudaSuccess;
  }
  void release() {
    if (ptr) cudaFreeHost(ptr);
    ptr = nullptr;
    bytes = 0;
  }
  template <class T>
  T* as() const { return static_cast<T*>(ptr); }
};

}  // namespace dpa

using dpa::DeviceBuffer;
using dpa::PinnedBuffer;
using dpa::SpareBlocks;

// Launch parameters an autotuner may change per context.
struct dpa_tuning_state {
  uint32_t claim = 16;        // order entries a warp claims at once
  uint32_t blocks_per_sm = 0; // persistent grid: 0 = as many as fit
  uint32_t order = 64;        // processing order: Morton buckets of an order^3
                              // coarsening of the grid (1..64); 0: input order
  uint32_t block = 0;         // threads per block (multiple of 32, <= 256); 0: the
                              // rules of launch_shape.hpp
  uint32_t particles_per_thread = 1;  // 1 or 2 (steady fields without recording)
};

namespace dpa {
// The launch parameters of a tuning.
inline void apply_tuning(const dpa_tuning_state& t, AdvectArgs& a) {
  a.claim = t.claim;
  a.blocks_per_sm = t.blocks_per_sm;
  a.block = t.block;
  a.particles_per_thread = t.particles_per_thread;
}
}  // namespace dpa

// Scratch of one processing-order + advection launch sequence: bucket ids,
// the order, the counting sort's counters and the claim counter. A context
// keeps one for its calls; a CUDA graph keeps its own, because a later call
// with more particles reallocates the context's.
struct dpa_launch_scratch {
  DeviceBuffer keys, values, sort_temp, work_counter;
  void release() {
    keys.release();
    values.release();
    sort_temp.release();
    work_counter.release();
  }
};

struct dpa_context {
  int device = 0;
  cudaStream_t stream = nullptr;
  std::string error;
  uint64_t staging_limit = 1ull << 30;
  uint64_t host_chunk_bytes = 256ull << 20;  // per pinned half (vertices + colors; indices)
  cudaEvent_t chunk_events[2] = {nullptr, nullptr};
  bool ieee_division = false;  // fields created now divide by __fdiv_rn only

  SpareBlocks spare;  // of destroyed fields
  DeviceBuffer round;       // a round's arrays (round_arrays, capi.cu)
  PinnedBuffer host_round;  // a staged round's
  DeviceBuffer remaining_in;
  dpa_launch_scratch scratch;
  uint64_t launches = 0;  // kernels this context launched (advection path)
  bool profiling = false;
  // order begin, advect begin, advect end, emission begin, emission end
  cudaEvent_t events[5] = {nullptr, nullptr, nullptr, nullptr, nullptr};
  bool timed_order = false;
  // A profiled recording round: its pieces' times, summed as they finish.
  bool timed_round = false;
  float round_order_ms = 0.0f, round_advect_ms = 0.0f, round_emit_ms = 0.0f;
  dpa_tuning_state tuning;
  DeviceBuffer raw, raw_offsets, kept_vertices, kept_segments;
  DeviceBuffer wide, vertex_offsets, segment_offsets, scan_temp;
  DeviceBuffer out_vertices, out_colors, out_indices;
  PinnedBuffer host_vertices, host_colors, host_indices, host_totals, host_offsets;
  DeviceBuffer ftle_winners, ftle_out, ftle_original, ftle_final;

  void release_all() {
    scratch.release();
    spare.release();
    DeviceBuffer* d[] = {&round, &remaining_in, &raw, &raw_offsets,
                         &kept_vertices, &kept_segments, &wide, &vertex_offsets,
                         &segment_offsets, &scan_temp, &out_vertices, &out_colors,
                         &out_indices, &ftle_winners, &ftle_out, &ftle_original,
                         &ftle_final};
    for (DeviceBuffer* b : d) b->release();
    PinnedBuffer* h[] = {&host_round, &host_vertices, &host_colors, &host_indices, &host_totals,
                         &host_offsets};
    for (PinnedBuffer* b : h) b->release();
  }
};

struct dpa_field {
  dpa_context* owner = nullptr;
  DeviceBuffer nodes;
  uint64_t node_bytes = 0;  // of nodes, a kept block being up to an eighth larger
  dpa::FieldView view{};
  uint64_t shape[3] = {0, 0, 0};
  float offset[3] = {0, 0, 0};
  float spacing[3] = {0, 0, 0};
  int32_t storage = DPA_STORAGE_F32;
  uint32_t slices = 1;  // > 1: a time-varying field
  float time_origin = 0.0f;
  float time_spacing = 0.0f;
  // Whether work elsewhere than in the context's stream may read the nodes: a caller's
  // stream, a graph or a server. Such a field's block is freed, not kept: only cudaFree
  // waits for that work without a device-wide wait, which CUDA forbids while any thread
  // captures a stream of the device.
  mutable std::atomic<bool> elsewhere{false};
};

namespace dpa {
// Notes that work reading the field's nodes goes to stream s.
inline cudaError_t note_stream(const dpa_context* ctx, const dpa_field* field, cudaStream_t s) {
  cudaStreamCaptureStatus status = cudaStreamCaptureStatusNone;
  if (s == ctx->stream) DPA_CUDA_TRY(cudaStreamIsCapturing(s, &status));
  if (s != ctx->stream || status != cudaStreamCaptureStatusNone)
    field->elsewhere.store(true, std::memory_order_relaxed);
  return cudaSuccess;
}
}  // namespace dpa

