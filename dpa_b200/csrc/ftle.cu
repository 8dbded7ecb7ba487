// ftle.cu -- flow-map claims, central-difference Jacobian, C = J^T J,
// FP64 largest eigenvalue and ln(sqrt(lambda)) / T per lattice cell
// (ftle_estimator.cpp:7-65 with regular_grid::gradient, regular_grid.hpp:87-108).
#include <type_traits>

#include "kernels.cuh"

namespace dpa {

namespace {

inline unsigned blocks_for(uint64_t n, unsigned block) { return unsigned((n + block - 1) / block); }

__device__ __forceinline__ bool reference_cell(const FtleArgs& a, uint64_t p, uint64_t& cell) {
  uint64_t sub[3];
#pragma unroll
  for (int i = 0; i < 3; ++i) {
    // regular_grid::cell_index (regular_grid.hpp:28-34) on the flow map.
    const float s = floorf(__fdiv_rn(__fsub_rn(a.original_positions[3 * p + i], a.offset[i]),
                                     a.spacing[i]));
    if (!(s >= 0.0f) || !(s < float(a.shape[i]))) return false;
    sub[i] = uint64_t(s);
  }
  cell = (sub[0] * a.shape[1] + sub[1]) * a.shape[2] + sub[2];
  return true;
}

// Reference mapping, first pass: every particle claims its cell; the largest
// particle index wins. kIndex holds an index + 1 (0: nobody): 32 bits for all
// but the largest counts, half the clearing and the atomics' traffic.
template <class kIndex>
__global__ void ftle_claim_kernel(const FtleArgs a) {
  const uint64_t p = uint64_t(blockIdx.x) * blockDim.x + threadIdx.x;
  if (p >= a.count) return;
  uint64_t cell;
  if (reference_cell(a, p, cell)) atomicMax(static_cast<kIndex*>(a.winners) + cell, kIndex(p + 1));
}

// The flow map at a cell: the particle of that index (lattice mapping, kIndex
// void), or the winner's final position, zero where no particle landed (the
// reference's zero-initialized multi_array).
template <class kIndex>
__device__ __forceinline__ void flow_at(const FtleArgs& a, uint64_t cell, float v[3]) {
  const float* at = a.final_positions + 3 * cell;
  if constexpr (!std::is_void_v<kIndex>) {
    const kIndex w = static_cast<const kIndex*>(a.winners)[cell];
    v[0] = v[1] = v[2] = 0.0f;
    if (!w) return;
    at = a.final_positions + 3 * uint64_t(w - 1);
  }
#pragma unroll
  for (int r = 0; r < 3; ++r) v[r] = at[r];
}

// Largest eigenvalue of a symmetric 3x3 matrix by cyclic Jacobi rotations, in registers
// (as a function of its own, which keeps the matrix in memory: 2 million cells that all
// need it, 1e-5 from the identity, 213 us, inlined 197; 40 and 45 registers).
__device__ __forceinline__ double max_eigenvalue_jacobi(double a[3][3]) {
  for (int sweep = 0; sweep < 32; ++sweep) {
    const double off = a[0][1] * a[0][1] + a[0][2] * a[0][2] + a[1][2] * a[1][2];
    const double diag = a[0][0] * a[0][0] + a[1][1] * a[1][1] + a[2][2] * a[2][2];
    if (off == 0.0 || off <= 1e-32 * diag) break;
#pragma unroll
    for (int p = 0; p < 2; ++p) {
#pragma unroll
      for (int q = p + 1; q < 3; ++q) {
        const double apq = a[p][q];
        if (apq == 0.0) continue;
        const double theta = (a[q][q] - a[p][p]) / (2.0 * apq);
        const double t = (theta >= 0.0 ? 1.0 : -1.0) / (fabs(theta) + sqrt(theta * theta + 1.0));
        const double c = 1.0 / sqrt(t * t + 1.0);
        const double s = t * c;
#pragma unroll
        for (int r = 0; r < 3; ++r) {
          const double arp = a[r][p], arq = a[r][q];
          a[r][p] = c * arp - s * arq;
          a[r][q] = s * arp + c * arq;
        }
#pragma unroll
        for (int r = 0; r < 3; ++r) {
          const double apr = a[p][r], aqr = a[q][r];
          a[p][r] = c * apr - s * aqr;
          a[q][r] = s * apr + c * aqr;
        }
      }
    }
  }
  return fmax(a[0][0], fmax(a[1][1], a[2][2]));
}

// Largest eigenvalue of a symmetric 3x3 matrix from its characteristic cubic
// (Smith, "Eigenvalues of a symmetric 3 x 3 matrix", Comm. ACM 4(4), 1961):
// with q the mean of the diagonal, B = A - q I, p^2 = |B|^2 / 6 and
// r = det(B) / (2 p^3), the eigenvalues are q + p x for the roots x of
// x^3 - 3 x = 2 r. For r >= 0 the largest root lies apart, in [sqrt 3, 2], where
// the cubic's slope is at least 6. It is found by Newton steps, two in 32 bits
// from the chord of [sqrt 3, 2] (1e-7) and two in 64 with the 32-bit slope there, which
// leave rounding errors only. For r < 0 that root is the smallest eigenvalue's, with
// its sign changed, and the largest is -x / 2 away from it plus half the gap of
// the other two, sqrt(3 - 3/4 x^2). The gap loses digits as it closes: the rounding of
// q alone, 2^-53 q, moves the eigenvalue by 2^-54 q / gap. The FTLE is the logarithm,
// which is nearly |1 - largest| where that is small (a flow map near the identity), so
// cells with gap * |1 - largest| below 2^-16 (1 + q) return false, as matrices that are
// not finite do, and the Jacobi rotations answer. What is left is a relative error of
// 1e-11 in the logarithm, beside what the rotations have too (random matrices I + s S, s
// from 1e-6 to 1, the two largest eigenvalues 1e-4 to 1 of s apart, against 80 bits),
// where the 32-bit result has 6e-8.
//
// The rotations throughout took 1900 warp instructions for 32 cells, 800 of them in
// 64 bits: 132 us for 1.5 million cells at 70 % of the issue slots; this took 480
// and 32 us, and 430 and 27 us with the divisions of cauchy_green(). In a stream of
// calls that is 21.8 us, and 22.8 with the test of the gap.
__device__ __forceinline__ bool max_eigenvalue(const double a[3][3], double& largest) {
  const double q = (a[0][0] + a[1][1] + a[2][2]) * (1.0 / 3.0);
  const double b0 = a[0][0] - q, b1 = a[1][1] - q, b2 = a[2][2] - q;
  const double u = a[0][1], v = a[0][2], w = a[1][2];
  const double p2 = (b0 * b0 + b1 * b1 + b2 * b2 + 2.0 * (u * u + v * v + w * w)) * (1.0 / 6.0);
  largest = q;
  if (p2 == 0.0) return true;
  const double inverse = rsqrt(p2), p = p2 * inverse;
  const double half_det =
      0.5 * (b0 * (b1 * b2 - w * w) - u * (u * b2 - w * v) + v * (u * w - b1 * v));
  const double r = half_det * inverse * inverse * inverse;
  if (!(p2 < 1e300)) return false;
  const double two_r = fmin(2.0 * fabs(r), 2.0);
  constexpr float kRoot3 = 1.7320508f;
  float x0 = fmaf(0.5f * (2.0f - kRoot3), float(two_r), kRoot3);
  float slope = __fdividef(1.0f, fmaf(3.0f * x0, x0, -3.0f));
#pragma unroll
  for (int i = 0; i < 2; ++i) {
    x0 -= fmaf(fmaf(x0, x0, -3.0f), x0, -float(two_r)) * slope;
    slope = __fdividef(1.0f, fmaf(3.0f * x0, x0, -3.0f));
  }
  double x = x0;
#pragma unroll
  for (int i = 0; i < 2; ++i) x -= fma(fma(x, x, -3.0), x, -two_r) * double(slope);
  double gap = 2.0;
  if (r < 0.0) {
    gap = sqrt(fmax(fma(-0.75 * x, x, 3.0), 0.0));
    x = 0.5 * x + gap;
  }
  largest = fma(p, x, q);
  return r >= 0.0 || gap * fabs(largest - 1.0) >= fma(0x1p-16, q, 0x1p-16);
}

// C = J^T J of a lattice cell in FP32 (Eigen's 3x3 lazy product, c0 + (c1 + c2)),
// widened: J[r][d] = (flow[next_d] - flow[prev_d])[r] / (2 h_d) with prev/next
// clamped at the border (bit d of `border`: no cell before this one along d, bit
// 3 + d: none behind it) while the divisor stays 2 h_d. The neighbours come straight
// from the particles' final positions (a pass that laid the flow map out first took
// 9 to 14 us more).
//
// kReciprocal divides by a product with the rounded reciprocal and one correction by
// its remainder (Markstein, "Computation of elementary functions on the IBM RISC
// System/6000", IBM J. Res. Dev. 34(1), 1990): 3 instructions instead of about 10,
// nine times a cell. Its quotients are IEEE's while the remainder's last bits are
// representable; where they are not (differences below 2^-101) the squares vanish in
// FP32 for the divisors it is used with, [2^-26, 2^26]. Infinities come out as NaN,
// which sends the cell to the other form.
template <class kIndex, bool kReciprocal>
__device__ __forceinline__ void cauchy_green(const FtleArgs& a, uint64_t flat, unsigned border,
                                             double C[3][3]) {
  const uint64_t step[3] = {a.shape[1] * a.shape[2], a.shape[2], 1};
  float J[3][3];
#pragma unroll
  for (int d = 0; d < 3; ++d) {
    float prev[3], next[3];
    flow_at<kIndex>(a, border >> d & 1u ? flat : flat - step[d], prev);
    flow_at<kIndex>(a, border >> (3 + d) & 1u ? flat : flat + step[d], next);
#pragma unroll
    for (int r = 0; r < 3; ++r) {
      const float n = __fsub_rn(next[r], prev[r]);
      if constexpr (kReciprocal) {
        const float q = __fmul_rn(n, a.reciprocal[d]);
        J[r][d] = __fmaf_rn(__fmaf_rn(-q, a.two_spacing[d], n), a.reciprocal[d], q);
      } else {
        J[r][d] = __fdiv_rn(n, a.two_spacing[d]);
      }
    }
  }
#pragma unroll
  for (int i = 0; i < 3; ++i)
#pragma unroll
    for (int j = i; j < 3; ++j)
      C[i][j] = C[j][i] =
          double(__fadd_rn(__fmul_rn(J[0][i], J[0][j]),
                           __fadd_rn(__fmul_rn(J[1][i], J[1][j]), __fmul_rn(J[2][i], J[2][j]))));
}

// The cells that the closed form leaves.
template <class kIndex>
__device__ __noinline__ double max_eigenvalue_general(const FtleArgs& a, uint64_t flat,
                                                      unsigned border) {
  double C[3][3];
  cauchy_green<kIndex, false>(a, flat, border, C);
  return max_eigenvalue_jacobi(C);
}

// The eigenvalue and the logarithm in FP64. kSize holds a cell index: 32-bit
// divisions unless the lattice needs more.
template <class kIndex, class kSize, bool kReciprocal>
__global__ void __launch_bounds__(128) ftle_kernel(const __grid_constant__ FtleArgs a,
                                                   uint64_t cells) {
  const uint64_t flat = uint64_t(blockIdx.x) * blockDim.x + threadIdx.x;
  if (flat >= cells) return;
  const kSize n[3] = {kSize(a.shape[0]), kSize(a.shape[1]), kSize(a.shape[2])};
  const kSize row = kSize(flat) / n[2];
  const kSize sub[3] = {row / n[1], row % n[1], kSize(flat) - row * n[2]};
  unsigned border = 0;
#pragma unroll
  for (int d = 0; d < 3; ++d)
    border |= (sub[d] == 0 ? 1u << d : 0u) | (sub[d] + 1 == n[d] ? 8u << d : 0u);
  double C[3][3], largest;
  cauchy_green<kIndex, kReciprocal>(a, flat, border, C);
  if (!max_eigenvalue(C, largest)) largest = max_eigenvalue_general<kIndex>(a, flat, border);
  a.ftle[flat] = float(0.5 * log(largest) * a.inverse_horizon);
}

template <class kIndex, bool kReciprocal>
cudaError_t launch_ftle_kernel(const FtleArgs& a, uint64_t cells, cudaStream_t stream) {
  const unsigned blocks = blocks_for(cells, 128);
  if (cells <= 0xffffffffull)
    ftle_kernel<kIndex, uint32_t, kReciprocal><<<blocks, 128, 0, stream>>>(a, cells);
  else
    ftle_kernel<kIndex, uint64_t, kReciprocal><<<blocks, 128, 0, stream>>>(a, cells);
  return cudaGetLastError();
}

template <class kIndex>
cudaError_t launch_ftle_cells(const FtleArgs& a, uint64_t cells, cudaStream_t stream) {
  bool reciprocal = true;
  for (float h : a.two_spacing) reciprocal = reciprocal && h >= 0x1p-26f && h <= 0x1p26f;
  return reciprocal ? launch_ftle_kernel<kIndex, true>(a, cells, stream)
                    : launch_ftle_kernel<kIndex, false>(a, cells, stream);
}

template <class kIndex>
cudaError_t launch_ftle_claims(const FtleArgs& a, uint64_t cells, cudaStream_t stream) {
  DPA_CUDA_TRY(cudaMemsetAsync(a.winners, 0, cells * sizeof(kIndex), stream));
  if (a.count) {
    ftle_claim_kernel<kIndex><<<blocks_for(a.count, 256), 256, 0, stream>>>(a);
    DPA_CUDA_TRY(cudaGetLastError());
  }
  return launch_ftle_cells<kIndex>(a, cells, stream);
}

__global__ void lattice_kernel(float o0, float o1, float o2, float s0, float s1, float s2,
                               uint64_t n0, uint64_t n1, uint64_t n2, float* out) {
  const uint64_t t = uint64_t(blockIdx.x) * blockDim.x + threadIdx.x;
  const uint64_t count = n0 * n1 * n2;
  if (t >= count) return;
  // unravel_index (indexing.hpp:11-20): last axis fastest.
  const uint64_t i2 = t % n2, i1 = (t / n2) % n1, i0 = t / (n1 * n2);
  out[3 * t] = __fadd_rn(o0, __fmul_rn(s0, float(i0)));
  out[3 * t + 1] = __fadd_rn(o1, __fmul_rn(s1, float(i1)));
  out[3 * t + 2] = __fadd_rn(o2, __fmul_rn(s2, float(i2)));
}

// Counter-based seed stream: splitmix64 (Steele, Lea and Flood, "Fast
// splittable pseudorandom number generators", 2014) of key ^ (3 i + axis).
__device__ __forceinline__ uint64_t splitmix64(uint64_t x) {
  x += 0x9e3779b97f4a7c15ull;
  x = (x ^ (x >> 30)) * 0xbf58476d1ce4e5b9ull;
  x = (x ^ (x >> 27)) * 0x94d049bb133111ebull;
  return x ^ (x >> 31);
}

__global__ void random_seeds_kernel(float o0, float o1, float o2, float s0, float s1, float s2,
                                    uint64_t count, uint64_t key, float* out) {
  const uint64_t t = uint64_t(blockIdx.x) * blockDim.x + threadIdx.x;
  if (t >= count) return;
  const float o[3] = {o0, o1, o2}, s[3] = {s0, s1, s2};
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    const uint64_t r = splitmix64(key ^ (3 * t + uint64_t(a)));
    const float u = float(uint32_t(r >> 40)) * 0x1p-24f;  // [0, 1), 24 random bits
    out[3 * t + a] = __fadd_rn(o[a], __fmul_rn(s[a], u));
  }
}

}  // namespace

cudaError_t launch_random_seeds(const float offset[3], const float size[3], uint64_t count,
                                uint64_t key, float* out, cudaStream_t stream) {
  if (count == 0) return cudaSuccess;
  random_seeds_kernel<<<blocks_for(count, 256), 256, 0, stream>>>(
      offset[0], offset[1], offset[2], size[0], size[1], size[2], count, key, out);
  return cudaGetLastError();
}

cudaError_t launch_ftle(const FtleArgs& args, cudaStream_t stream) {
  FtleArgs a = args;
  a.inverse_horizon = 1.0 / a.horizon;
  for (int i = 0; i < 3; ++i) a.reciprocal[i] = 1.0f / a.two_spacing[i];
  const uint64_t cells = a.shape[0] * a.shape[1] * a.shape[2];
  if (cells == 0) return cudaSuccess;
  if (a.mapping == DPA_FTLE_MAPPING_LATTICE) return launch_ftle_cells<void>(a, cells, stream);
  return a.count < 0xffffffffull ? launch_ftle_claims<unsigned int>(a, cells, stream)
                                 : launch_ftle_claims<unsigned long long>(a, cells, stream);
}

cudaError_t launch_lattice_seeds(const float offset[3], const float stride[3],
                                 const uint64_t shape[3], float* out, cudaStream_t stream) {
  const uint64_t count = shape[0] * shape[1] * shape[2];
  if (count == 0) return cudaSuccess;
  lattice_kernel<<<blocks_for(count, 256), 256, 0, stream>>>(
      offset[0], offset[1], offset[2], stride[0], stride[1], stride[2], shape[0], shape[1],
      shape[2], out);
  return cudaGetLastError();
}

}  // namespace dpa
