// advect_kernel.cuh -- the advection kernel template and its launchers:
// every step of a particle in registers (particle_advector.cpp:325-396), one
// or two particles per lane. advect_f32.cu, advect_f32e.cu, advect_f16.cu and
// advect_bf16.cu instantiate it per field storage, for steady and
// time-varying fields.
#pragma once

#include <algorithm>
#include <atomic>
#include <type_traits>

#include "kernels.cuh"
#include "sample.cuh"

namespace dpa {
namespace {

// Appends one vertex to the count of the pruned curve: invalid-sentinel
// vertices are dropped by prune_integral_curves (particle_advector.cpp:402-408),
// and index_generator (index_generator.cpp:10-39) pairs consecutive kept
// vertices of which neither equals the terminal sentinel.
struct CurveCounter {
  uint32_t kept = 0;
  uint32_t segments = 0;
  bool prev_open = false;  // previous kept vertex is not terminal-valued

  __device__ __forceinline__ void append(float x, float y, float z, bool taken = true) {
    const bool valid = taken && !equals3(x, y, z, kInvalid);
    const bool terminal = equals3(x, y, z, kTerminal);
    segments += valid && !terminal && prev_open ? 1u : 0u;
    prev_open = valid ? !terminal : prev_open;
    kept += valid ? 1u : 0u;
  }
};

template <int kIntegrator, bool kRecord, bool kUnsteady, int kPPT>
constexpr int advect_min_blocks() {
  return kPPT == 2                                       ? kAdvectPpt2MinBlocks
         : kRecord && !kUnsteady                         ? kAdvectRecordMinBlocks
         : kUnsteady                                     ? kAdvectUnsteadyMinBlocks
         : kIntegrator == DPA_INTEGRATOR_RUNGE_KUTTA_4_TRUE ? kAdvectTrueRk4MinBlocks
                                                         : kAdvectMinBlocks;
}

// Pathlines of F32 nodes by Euler and RK4 also come as narrow kernels (kNarrowBit
// of the mode): held to 96 registers, with four words spilled around the gather, and
// launched in blocks of 64, which gives each of an SM's register files 5 warps
// instead of 4. Issue was busy 57 % of the time at 4. 250,000 pathlines of 1000 steps
// 3054 -> 2654 us, from edge records 2930 -> 2685; F16 fields, issue-bound at 67 to
// 72 %, gain nothing (2926 -> 3007), the four-sample stepper spills (2863 -> 2943).
template <int kIntegrator, int kStorage, bool kRecord, bool kUnsteady>
constexpr bool advect_has_narrow() {
  return kUnsteady && !kRecord &&
         (kStorage == DPA_STORAGE_F32 || kStorage == DPA_STORAGE_F32_EDGES) &&
         (kIntegrator == DPA_INTEGRATOR_EULER || kIntegrator == DPA_INTEGRATOR_RUNGE_KUTTA_4);
}

// Registers per thread: what the block count leaves (allocated by eights).
template <int kIntegrator, int kLocate, bool kRecord, bool kUnsteady, int kPPT>
constexpr int advect_registers() {
  return kLocate & kNarrowBit
             ? 96
             : 65536 / (kAdvectBlock * advect_min_blocks<kIntegrator, kRecord, kUnsteady, kPPT>()) / 8 * 8;
}

// Persistent advection. Every lane owns kPPT slots, each holding one particle
// at a time; a slot whose particle finishes takes the next one from its
// warp's claim of a.claim consecutive entries of the processing order, and
// the warp claims a new batch with one atomic when its batch runs out. A launch
// with a slot for every particle needs no claims: each warp is given its own
// a.own_entries entries (work_counter null). Lanes
// therefore stay busy while particles of one warp end after very different
// numbers of steps. A particle takes at most a.max_steps steps per launch;
// one stopped by that budget alone is reported as in flight and resumes in a
// later launch.
//
// Between hand-outs the warp runs stretches: every slot steps until one of
// the warp's particles stops or has no step left, with one vote per step and one
// count for the warp (a stretch ends at 2^32 - 1 steps at the latest). The
// kPPT slots of a lane step in lock-step, so one particle's corner gather is
// in flight while the other's arithmetic issues. An empty slot holds a parked
// position, the centre of the first cell (never NaN, which would send the
// division of a step into its slow path for the whole warp) at the middle of the
// first time slice. With one particle per lane the branch-free Euler and RK4
// steppers step a parked slot and discard the result; otherwise an empty slot
// takes no steps.
template <int kIntegrator, int kStorage, int kLocate, bool kRecord, bool kUnsteady, int kPPT>
__global__ void __maxnreg__((advect_registers<kIntegrator, kLocate, kRecord, kUnsteady, kPPT>()))
advect_kernel(const FieldView f, const AdvectArgs a) {
  using Sampler = std::conditional_t<kUnsteady, TimeSampler<kStorage, kLocate & ~kNarrowBit>,
                                     CellSampler<kStorage, kLocate>>;
  constexpr unsigned kFull = 0xffffffffu;
  // State touched only when particles are handed out or finish lives in
  // shared memory, leaving the registers to the stepping loop: the warp's
  // claim [next, end) of the order and, per slot, the particle index, its
  // remaining iterations and the steps it may still take in this launch
  // (its remaining iterations or the launch's step budget).
  __shared__ uint64_t claims[kAdvectBlock / 32][2];
  __shared__ uint64_t particle[kPPT][kAdvectBlock];
  __shared__ uint64_t remaining[kPPT][kAdvectBlock];
  __shared__ uint64_t budget[kPPT][kAdvectBlock];
  const uint32_t claim = a.claim;
  const unsigned tid = threadIdx.x;
  const unsigned lane = tid & 31u;
  uint64_t* const warp_claim = claims[tid >> 5];
  if (lane == 0) {
    const uint64_t size = a.work_counter ? 0 : a.own_entries;
    const uint64_t own = (uint64_t(blockIdx.x) * (blockDim.x >> 5) + (tid >> 5)) * size;
    warp_claim[0] = own < a.count ? own : a.count;
    warp_claim[1] = own + size < a.count ? own + size : a.count;
  }
  __syncwarp();
  bool exhausted = false;
  // Where an empty slot waits: the centre of the first cell, so that a step
  // run for it (branch-free steppers) divides normal numbers and loads its
  // corners once.
  const Position parked{__fmaf_rn(0.5f, f.spacing[0], f.offset[0]),
                        make_float2(__fmaf_rn(0.5f, f.spacing[2], f.offset[2]),
                                    __fmaf_rn(0.5f, f.spacing[1], f.offset[1]))};
  const float parked_time = __fmaf_rn(0.5f, f.time_spacing, f.time_origin);
  // (One particle per lane only: with two, skipping a pair's empty slot by a
  // branch measured 1.7x faster on the 512^3 batch than stepping it.)
  constexpr bool kStepAll = kPPT == 1 &&
                            (kIntegrator == DPA_INTEGRATOR_EULER ||
                             kIntegrator == DPA_INTEGRATOR_RUNGE_KUTTA_4);

  bool active[kPPT];
  Position p[kPPT];
  Sampler sampler[kPPT];
  StepHistory history[kPPT];
  float t[kPPT];          // particle time (a.times)
  float* curve[kPPT];     // the particle's last written vertex
  CurveCounter counter[kPPT];
#pragma unroll
  for (int j = 0; j < kPPT; ++j) {
    active[j] = false;
    p[j] = parked;
    history[j] = StepHistory{};
    t[j] = parked_time;
    curve[j] = nullptr;
  }

  while (true) {
    // Hand new particles to idle slots.
#pragma unroll
    for (int j = 0; j < kPPT; ++j) {
      unsigned idle = __ballot_sync(kFull, !active[j]);
      while (idle && !exhausted) {
        uint64_t next = warp_claim[0], end = warp_claim[1];
        if (next == end) {
          unsigned long long base = a.count;
          if (lane == 0 && a.work_counter)
            base = atomicAdd(a.work_counter, (unsigned long long)claim);
          base = __shfl_sync(kFull, base, 0);
          if (base >= a.count) {
            exhausted = true;
            break;
          }
          next = base;
          end = base + claim < a.count ? base + claim : a.count;
        }
        const uint32_t avail = uint32_t(end - next);
        const uint32_t take = uint32_t(__popc(idle)) < avail ? uint32_t(__popc(idle)) : avail;
        const uint32_t rank = __popc(idle & ((1u << lane) - 1u));
        // Lanes still in the idle set take entries next + rank. (A slot that
        // drew a finished particle earlier in this round is inactive but no
        // longer idle, and must not take one again.)
        const bool took = ((idle >> lane) & 1u) && rank < take;
        bool mine = took;
        uint64_t k = 0;
        if (mine) {
          const uint64_t e = next + rank;
          k = a.order ? a.order[e] : e;
          // Serving: a finished particle stays finished.
          if (a.resume_only && a.termination[k] != DPA_TERMINATION_IN_FLIGHT) mine = false;
        }
        if (mine) {
          particle[j][tid] = k;
          p[j].p0 = a.positions[3 * k];
          p[j].p21 = make_float2(a.positions[3 * k + 2], a.positions[3 * k + 1]);
          const uint64_t rem = a.remaining[k];
          remaining[j][tid] = rem;
          budget[j][tid] = rem < a.max_steps ? rem : a.max_steps;
          if (a.times) t[j] = a.times[k];
          sampler[j].reset();
          history[j].started = false;
          active[j] = true;
          if constexpr (kRecord) {
            // A particle resumed from an earlier launch continues its curve
            // where that launch left it.
            const uint64_t done = a.remaining_initial ? a.remaining_initial[k] - rem : 0;
            curve[j] = a.raw_vertices + 3 * (a.raw_offsets[k] + done);
            counter[j] = CurveCounter();
            if (done == 0) {
              curve[j][0] = p[j].p0;
              curve[j][1] = p[j].p21.y;
              curve[j][2] = p[j].p21.x;
              counter[j].append(p[j].p0, p[j].p21.y, p[j].p21.x);
            } else {
              counter[j].kept = a.kept_vertices[k];
              counter[j].segments = a.kept_segments[k];
              counter[j].prev_open = a.curve_open[k] != 0;
            }
          }
        }
        __syncwarp();
        if (lane == 0) {
          warp_claim[0] = next + take;
          warp_claim[1] = end;
        }
        __syncwarp();
        // Every lane that took an entry leaves this round of hand-outs; one
        // that drew a finished particle (serving) stays inactive until the next.
        idle &= ~__ballot_sync(kFull, took);
      }
    }
    bool any = false;
#pragma unroll
    for (int j = 0; j < kPPT; ++j) any = any || active[j];
    if (!__any_sync(kFull, any)) {
      if (exhausted) break;
      continue;  // every lane drew a finished particle (serving): claim again
    }

    // One stretch: as many steps as every particle of the warp may still take.
    uint32_t steps = 0xffffffffu;
    int r[kPPT];
#pragma unroll
    for (int j = 0; j < kPPT; ++j) {
      const uint64_t allowed = active[j] ? budget[j][tid] : ~0ull;
      steps = allowed < steps ? uint32_t(allowed) : steps;
      r[j] = kStepTaken;
    }
    steps = __reduce_min_sync(kFull, steps);
    uint32_t n = 0;
    bool halt = false;
    while (n != steps && !halt) {
      // Branch-free steppers run every slot, an empty one without moving it;
      // the others skip empty slots.
#pragma unroll
      for (int j = 0; j < kPPT; ++j) {
        if constexpr (kStepAll)
          r[j] = step<kIntegrator>(f, a.coefficients, sampler[j], p[j], t[j], history[j],
                                   active[j]);
        else
          r[j] = active[j]
                     ? step<kIntegrator>(f, a.coefficients, sampler[j], p[j], t[j], history[j])
                     : int(kStepOutOfBounds);
      }
      ++n;
#pragma unroll
      for (int j = 0; j < kPPT; ++j) {
        const bool taken = r[j] == kStepTaken;  // never for an empty slot
        if constexpr (kUnsteady) t[j] = taken ? __fadd_rn(t[j], a.coefficients.dt) : t[j];
        if constexpr (kRecord) {
          // The step's vertex, stored by predicated stores rather than a
          // branch (a launch of few particles waits on each step's chain).
          float* v = curve[j] + 3 * uint64_t(n);
          asm volatile(
              "{\n\t.reg .pred p;\n\tsetp.ne.u32 p, %4, 0;\n\t"
              "@p st.global.f32 [%0], %1;\n\t@p st.global.f32 [%0+4], %2;\n\t"
              "@p st.global.f32 [%0+8], %3;\n\t}" ::"l"(v),
              "f"(p[j].p0), "f"(p[j].p21.y), "f"(p[j].p21.x), "r"(taken ? 1u : 0u));
          counter[j].append(p[j].p0, p[j].p21.y, p[j].p21.x, taken);
        }
        halt = halt || (active[j] && !taken);
      }
      halt = __any_sync(kFull, halt);
    }

#pragma unroll
    for (int j = 0; j < kPPT; ++j) {
      if (!active[j]) continue;
      const uint32_t taken = r[j] == kStepTaken ? n : n - 1;
      const uint64_t rem = remaining[j][tid] - taken;
      const uint64_t left = budget[j][tid] - taken;
      remaining[j][tid] = rem;
      budget[j][tid] = left;
      if constexpr (!kUnsteady) {
        // A steady field's particles carry their time only when asked to; it
        // advances by dt per step taken, rounded step by step as a
        // time-varying field's does.
        if (a.times)
          for (uint32_t i = 0; i < taken; ++i) t[j] = __fadd_rn(t[j], a.coefficients.dt);
      }
      if constexpr (kRecord) curve[j] += 3 * uint64_t(taken);
      // A particle that only reached the end of a stretch carries on.
      if (r[j] == kStepTaken && left > 0) continue;

      const uint64_t k = particle[j][tid];
      const int reason = r[j] == kStepOutOfBounds    ? DPA_TERMINATION_OUT_OF_BOUNDS
                         : r[j] == kStepZeroVelocity ? DPA_TERMINATION_ZERO_VELOCITY
                         : rem == 0                  ? DPA_TERMINATION_COMPLETE
                                                     : DPA_TERMINATION_IN_FLIGHT;
      if constexpr (kRecord) {
        if (reason != DPA_TERMINATION_IN_FLIGHT) {
          float* v = curve[j] + 3;
          v[0] = kTerminal;
          v[1] = kTerminal;
          v[2] = kTerminal;
          counter[j].append(kTerminal, kTerminal, kTerminal);
        } else {
          a.curve_open[k] = counter[j].prev_open ? 1 : 0;
        }
        a.kept_vertices[k] = counter[j].kept;
        a.kept_segments[k] = counter[j].segments;
      }
      a.positions[3 * k] = p[j].p0;
      a.positions[3 * k + 1] = p[j].p21.y;
      a.positions[3 * k + 2] = p[j].p21.x;
      a.remaining[k] = rem;
      if (a.times) a.times[k] = t[j];
      if (a.termination) a.termination[k] = uint8_t(reason);
      if (a.in_flight && reason != DPA_TERMINATION_IN_FLIGHT)
        atomicSub(a.in_flight + a.request_of[k], 1u);
      active[j] = false;
      p[j] = parked;
      if constexpr (kUnsteady) t[j] = parked_time;
    }
  }
}

// Resident blocks per SM of one instantiation at one block size, and the SM
// count, looked up once per process (every device of a process is a B200
// here) and published as one atomic value, so that threads making their
// first launches at once each see either nothing or both figures.
template <int kIntegrator, int kStorage, int kLocate, bool kRecord, bool kUnsteady, int kPPT>
cudaError_t resident_blocks(uint32_t block, int* blocks_per_sm, int* sms) {
  static std::atomic<uint64_t> cache[kAdvectBlock / 32 + 1] = {};
  std::atomic<uint64_t>& slot = cache[block / 32];
  uint64_t packed = slot.load(std::memory_order_acquire);
  if (packed == 0) {
    int device = 0, count = 0, r = 0;
    DPA_CUDA_TRY(cudaGetDevice(&device));
    DPA_CUDA_TRY(cudaDeviceGetAttribute(&count, cudaDevAttrMultiProcessorCount, device));
    DPA_CUDA_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(
        &r, advect_kernel<kIntegrator, kStorage, kLocate, kRecord, kUnsteady, kPPT>, int(block),
        0));
    packed = (uint64_t(uint32_t(count)) << 32) | uint32_t(r < 1 ? 1 : r);
    slot.store(packed, std::memory_order_release);
  }
  *blocks_per_sm = int(uint32_t(packed));
  *sms = int(packed >> 32);
  return cudaSuccess;
}

template <int kIntegrator, int kStorage, int kLocate, bool kRecord, bool kUnsteady, int kPPT>
cudaError_t launch_typed(const FieldView& f, const AdvectArgs& a, cudaStream_t stream) {
  // Persistent grid: as many blocks as fit on the device at once (or as the
  // tuning asks), fewer when there are fewer particles than lanes.
  const uint64_t lanes = (a.count + kPPT - 1) / kPPT;
  int sms = 0, resident = 0;
  DPA_CUDA_TRY((resident_blocks<kIntegrator, kStorage, kLocate, kRecord, kUnsteady, kPPT>(
      kAdvectBlock, &resident, &sms)));
  const bool free_shape = kPPT == 1 && !a.block && !a.blocks_per_sm;
  const uint32_t limit = limited_threads(f.threads_per_sm, f.limit_speed, a.coefficients.dt);
  const uint32_t own = free_shape ? particles_per_warp(a.count, sms) : 32u * kPPT;
  constexpr uint32_t threads = kLocate & kNarrowBit ? 64 : kAdvectBlock;
  const uint32_t block =
      own < 32 ? 32
               : advect_block(a.block, a.blocks_per_sm, threads, lanes, sms,
                              limit ? 0 : resident);
  if (block == 0 || block % 32 != 0 || block > uint32_t(kAdvectBlock)) return cudaErrorInvalidValue;
  DPA_CUDA_TRY((resident_blocks<kIntegrator, kStorage, kLocate, kRecord, kUnsteady, kPPT>(
      block, &resident, &sms)));
  if (a.count == 0) return cudaSuccess;  // nothing to do, or preparation only
  if (a.blocks_per_sm && int(a.blocks_per_sm) < resident) resident = int(a.blocks_per_sm);
  if (!a.blocks_per_sm && limit) resident = std::min(resident, std::max(1, int(limit / block)));
  const uint64_t per_block = uint64_t(block / 32) * own;
  const uint64_t needed = (a.count + per_block - 1) / per_block;
  const uint64_t blocks = std::min<uint64_t>(needed, uint64_t(resident) * uint64_t(sms));
  if (blocks == 0) return cudaSuccess;
  AdvectArgs launch = a;
  launch.own_entries = own;
  if (blocks == needed)
    launch.work_counter = nullptr;
  else
    DPA_CUDA_TRY(cudaMemsetAsync(a.work_counter, 0, sizeof(unsigned long long), stream));
  advect_kernel<kIntegrator, kStorage, kLocate, kRecord, kUnsteady, kPPT>
      <<<dim3(unsigned(blocks)), dim3(block), 0, stream>>>(f, launch);
  return cudaGetLastError();
}

// Two particles per lane for steady fields without recording; everything
// else runs one.
template <int kIntegrator, int kStorage, int kLocate, bool kRecord, bool kUnsteady>
cudaError_t launch_ppt(const FieldView& f, const AdvectArgs& a, cudaStream_t s) {
  if constexpr (!kRecord && !kUnsteady && kIntegrator != DPA_INTEGRATOR_RUNGE_KUTTA_4_TRUE) {
    if (a.particles_per_thread == 2)
      return launch_typed<kIntegrator, kStorage, kLocate, kRecord, kUnsteady, 2>(f, a, s);
  }
  if constexpr (advect_has_narrow<kIntegrator, kStorage, kRecord, kUnsteady>()) {
    // Narrow where the wide kernel cannot hold every particle at once; where it can,
    // a launch lasts as long as its longest chain of steps, and the spills lengthen
    // that (8000 pathlines 600 -> 608 us; of 300 steps, wide and narrow: 60,000 292 and
    // 294, edge records 75,776 295 and 303). Beyond it 76,000 take 409 and 340 us, edge
    // records 411 and 342, 100,000 505 and 486, 470 and 459, 300,000 1135 and 1058, 1020
    // and 907. A tuning's launch shape is the wide kernel's. A launch of nothing prepares
    // both.
    int sms = 0, resident = 0;
    DPA_CUDA_TRY((resident_blocks<kIntegrator, kStorage, kLocate, kRecord, kUnsteady, 1>(
        kAdvectBlock, &resident, &sms)));
    const uint64_t held = uint64_t(resident) * uint64_t(sms) * kAdvectBlock;
    if (a.count == 0 || (a.count > held && !a.block && !a.blocks_per_sm)) {
      const cudaError_t e =
          launch_typed<kIntegrator, kStorage, kLocate | kNarrowBit, kRecord, kUnsteady, 1>(f, a, s);
      if (a.count != 0 || e != cudaSuccess) return e;
    }
  }
  return launch_typed<kIntegrator, kStorage, kLocate, kRecord, kUnsteady, 1>(f, a, s);
}

template <int kIntegrator, int kStorage, int kMode, bool kUnsteady>
cudaError_t launch_record(const FieldView& f, const AdvectArgs& a, bool record, cudaStream_t s) {
  return record ? launch_ppt<kIntegrator, kStorage, kMode, true, kUnsteady>(f, a, s)
                : launch_ppt<kIntegrator, kStorage, kMode, false, kUnsteady>(f, a, s);
}

template <int kIntegrator, int kStorage, bool kUnsteady>
cudaError_t launch_locate(const FieldView& f, const AdvectArgs& a, bool record, cudaStream_t s) {
  if constexpr (!kUnsteady) {
    if (f.tiled) {
      switch (f.locate) {
        case kLocatePow2:
          return launch_record<kIntegrator, kStorage, kLocatePow2 | kTiledBit, false>(f, a, record,
                                                                                      s);
        case kLocateReciprocal:
          return launch_record<kIntegrator, kStorage, kLocateReciprocal | kTiledBit, false>(
              f, a, record, s);
        default:
          return launch_record<kIntegrator, kStorage, kLocateDivide | kTiledBit, false>(
              f, a, record, s);
      }
    }
  }
  switch (f.locate) {
    case kLocatePow2:
      return launch_record<kIntegrator, kStorage, kLocatePow2, kUnsteady>(f, a, record, s);
    case kLocateReciprocal:
      return launch_record<kIntegrator, kStorage, kLocateReciprocal, kUnsteady>(f, a, record, s);
    default:
      return launch_record<kIntegrator, kStorage, kLocateDivide, kUnsteady>(f, a, record, s);
  }
}

}  // namespace

// Every integrator for one storage and kind of field (steady or time-varying).
template <int kStorage, bool kUnsteady>
cudaError_t launch_advect_storage(const FieldView& f, const AdvectArgs& a, int integrator,
                                  bool record, cudaStream_t stream) {
  switch (integrator) {
    case DPA_INTEGRATOR_EULER:
      return launch_locate<DPA_INTEGRATOR_EULER, kStorage, kUnsteady>(f, a, record, stream);
    case DPA_INTEGRATOR_RUNGE_KUTTA_4:
      return launch_locate<DPA_INTEGRATOR_RUNGE_KUTTA_4, kStorage, kUnsteady>(f, a, record, stream);
    case DPA_INTEGRATOR_RUNGE_KUTTA_4_TRUE:
      return launch_locate<DPA_INTEGRATOR_RUNGE_KUTTA_4_TRUE, kStorage, kUnsteady>(f, a, record,
                                                                                  stream);
    case DPA_INTEGRATOR_MODIFIED_MIDPOINT:
    case DPA_INTEGRATOR_RUNGE_KUTTA_CASH_KARP_54:
    case DPA_INTEGRATOR_RUNGE_KUTTA_DORMAND_PRINCE_5:
    case DPA_INTEGRATOR_RUNGE_KUTTA_FEHLBERG_78:
    case DPA_INTEGRATOR_ADAMS_BASHFORTH_2:
    case DPA_INTEGRATOR_ADAMS_BASHFORTH_MOULTON_2:
      // The coefficients in a.coefficients.g select the stepper.
      return launch_locate<kGeneralIntegrator, kStorage, kUnsteady>(f, a, record, stream);
    default:
      return cudaErrorInvalidValue;
  }
}

}  // namespace dpa
