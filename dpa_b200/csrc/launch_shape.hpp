// launch_shape.hpp -- how an advection launch is dealt out over the device: particles
// per warp and threads per block. Host code without CUDA, so that the rules are tested
// on their own.
#pragma once

#include <algorithm>
#include <cmath>
#include <cstdint>

#ifndef DPA_ADVECT_BLOCK
#define DPA_ADVECT_BLOCK 256
#endif
// Launches whose particles would fill fewer blocks than the device has SMs
// use smaller blocks (1) or keep their own threads per block (0).
#ifndef DPA_ADVECT_SPREAD
#define DPA_ADVECT_SPREAD 1
#endif

namespace dpa {

constexpr int kAdvectBlock = DPA_ADVECT_BLOCK;

// Threads per block of a launch: the tuning's choice, else the kernel's own, or
// fewer (a multiple of 32) when the particles would fill fewer blocks than
// the device has SMs, so that a small launch still spreads over every SM. A launch
// whose blocks all fit at once (resident of them to an SM) but would leave the
// fullest SM more than a quarter above the average takes blocks of 64: 50,000 seeds
// are 196 blocks of 256, two on 48 SMs and one on the others. us at 256 and 64:
// 47,172 seeds of the four-sample stepper, F16, 612 -> 520; 50,000 F16 258 -> 237, F32
// in 96^3 284 -> 226; 60,000 pathlines 1010 -> 951. More even ones gain little or lose
// a percent (100,000 F16 seeds, 391 blocks: 329 -> 335). Not where a tuning limits the
// blocks per SM, which counts blocks of the kernel's own size: 50,000 seeds at 2 blocks
// of 256 per SM take 250 us, of 64 (a quarter of the lanes) 396.
inline uint32_t advect_block(uint32_t tuned_block, uint32_t tuned_blocks_per_sm, uint32_t own,
                             uint64_t lanes, int sms, int resident) {
  if (tuned_block) return tuned_block;
  uint32_t block = own;
#if DPA_ADVECT_SPREAD
  const uint64_t per_sm = (lanes + uint64_t(sms) - 1) / uint64_t(sms);
  if (per_sm < uint64_t(own)) block = uint32_t(std::max<uint64_t>(32, (per_sm + 31) / 32 * 32));
  const uint64_t blocks = (lanes + own - 1) / own, n = uint64_t(sms);
  if (!tuned_blocks_per_sm && blocks > n && blocks <= uint64_t(resident) * n &&
      4 * n * ((blocks + n - 1) / n) > 5 * blocks)
    block = std::min(block, 64u);
#else
  (void)tuned_blocks_per_sm;
  (void)lanes;
  (void)sms;
  (void)resident;
#endif
  return block;
}

// Threads per SM that a launch of steps of dt keeps resident (0: as many as fit), by the
// field's limit and, where that depends on the steps, a speed in cells per time. A third
// of a cell a step is where nodes of 16 bits and edge records between 1.25 and 3 GiB begin
// to gain by fewer threads while neighbouring particles stay together. 200 steps of 2
// million seeds, us at 1024 and 768 threads:
//   F16 580^3, curl noise      0.3 cells 3899 and 4089, 0.35 4341 and 4250, 0.5 6451 and 4889
//   F16 700^3                  0.3 4755 and 4576, 0.35 5671 and 4824
//   edges 350^3                0.3 3467 and 3712, 0.35 3713 and 3876, 0.4 4040 and 4042
//   edges 450^3                0.3 4587 and 4413, 0.35 5160 and 4666, 0.5 7418 and 5714
//   F16 580^3, noise over 8 nodes only
//                              0.3 3390 and 3729, 0.35 3537 and 3792, 0.5 4007 and 3961
inline uint32_t limited_threads(uint32_t limit, float speed, float dt) {
  return speed == 0.0f || std::fabs(dt) * speed > 1.0f / 3.0f ? limit : 0;
}

// That speed, of a field's RMS speed and the RMS change of its velocity from a node to the
// next. Where the velocity changes by more than a twentieth in a cell, particles part on
// their way and gather from everywhere: the line lies at a fifth of a cell a step. Curl
// noise, 400 and 2000 steps of 2 million seeds, ms at 1024 and 768 threads:
//   F16 580^3    0.16 cells 5.8 and 6.6, 24.2 and 27.5; 0.22 6.3 and 6.9, 28.9 and 28.3
//   F16 700^3    0.16 6.4 and 7.1, 26.8 and 29.6; 0.22 7.1 and 7.6, 40.0 and 31.2
//   edges 450^3  0.16 6.0 and 6.6, 24.5 and 26.0; 0.22 6.9 and 7.1, 31.3 and 27.9
// and at 0.3 cells, 2000 steps, 52 and 33, 67 and 42, 61 and 33; noise over 8 nodes only, 0.25
// cells, 2000 steps, 19.4 and 21.2, 20.5 and 22.9, 15.8 and 17.7.
inline double limit_speed(double speed, double change) {
  return change > 0.05 * speed ? speed * (5.0 / 3.0) : speed;
}

// Particles per warp of a small launch: as few as keep every SM at 8 warps or
// less (1, 2, 4, 8, 16; else 32). A warp waits at every step for the slowest of its
// lanes' gathers, and such a launch leaves the SMs' issue slots idle; more warps per
// SM than that take turns instead. B200, us at 32 lanes and as chosen: 100 recorded
// seeds 33 -> 21 (1 lane), 1000 216 -> 168 (1), 4096 245 -> 200 (4), 16,384 202 ->
// 178 (16); end positions of 8000 seeds in a 256^3 field 227 -> 191 (8), in F16 fields
// that L2 holds 119 -> 121; pathlines of 8000 seeds 262 -> 214.
inline uint32_t particles_per_warp(uint64_t count, int sms) {
  uint32_t lanes = 1;
  while (lanes < 32 && count > uint64_t(lanes) * 8u * uint64_t(sms)) lanes *= 2;
  return lanes;
}

}  // namespace dpa
