// sample.cuh -- grid location, trilinear sampling and integrator steps.
//
// Restates, per particle step, regular_grid::contains / interpolate
// (include/dpa/types/regular_grid.hpp:41-75, corner order of
// include/dpa/math/permute_for.hpp:12-34) and the odeint euler /
// runge_kutta4 updates that particle_advector.cpp:369-385 performs, with the
// same rounding as the reference's FP32 build.
#pragma once

#include <type_traits>

#include "common.cuh"


namespace dpa {

// One node of the repacked field, widened to FP32.
template <int kStorage>
__device__ __forceinline__ void load_node(const void* nodes, int64_t index, float& x, float& y,
                                          float& z) {
  if constexpr (kStorage == DPA_STORAGE_F32) {
    const float4 v = __ldg(reinterpret_cast<const float4*>(nodes) + index);
    x = v.x;
    y = v.y;
    z = v.z;
  } else if constexpr (kStorage == DPA_STORAGE_F16) {
    const uint2 r = __ldg(reinterpret_cast<const uint2*>(nodes) + index);
    const float2 xy = __half22float2(*reinterpret_cast<const __half2*>(&r.x));
    x = xy.x;
    y = xy.y;
    z = __low2float(*reinterpret_cast<const __half2*>(&r.y));
  } else {
    const uint2 r = __ldg(reinterpret_cast<const uint2*>(nodes) + index);
    const float2 xy = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&r.x));
    x = xy.x;
    y = xy.y;
    z = __low2float(*reinterpret_cast<const __nv_bfloat162*>(&r.y));
  }
}

// Two FP32 lanes. Products use sm_100's packed multiply (FMUL2), whose
// lanes round exactly as __fmul_rn does. The compiler fuses a packed multiply
// feeding a packed add into one packed FMA even when both carry explicit
// round-to-nearest, and the fused result differs from the reference's
// separately rounded product and sum. A sum that may take such a product as an
// operand is therefore a * unit + b in one packed FMA whose multiplier, 1.0,
// comes with the launch (FieldView::unit): the product by 1 is exact, so the
// FMA rounds a + b once, and a multiplier unknown when compiling leaves nothing
// to fuse.
__device__ __forceinline__ float2 add2(float2 a, float2 b, float2 unit) {
  return __ffma2_rn(a, unit, b);
}
__device__ __forceinline__ float2 mul2(float2 a, float2 b) { return __fmul2_rn(a, b); }
__device__ __forceinline__ float2 splat(float a) { return make_float2(a, a); }
// t * a + u * b, every operation rounded on its own.
__device__ __forceinline__ float2 blend2(float2 a, float2 b, float2 t, float2 u, float2 unit) {
  return add2(mul2(t, a), mul2(u, b), unit);
}
__device__ __forceinline__ float blend(float a, float b, float t, float u) {
  return __fadd_rn(__fmul_rn(t, a), __fmul_rn(u, b));
}

// A particle position is held as p0 and the pair p21 = (p2, p1): the
// derivative of (p2, p1) is (v0, v1), the first two components of a sample,
// because of the reversed components of particle_advector.cpp:369.
struct Position {
  float p0;
  float2 p21;
};

// Weights of one sample: w = fmod(p - offset, h) / h per axis, as (w0, (w2, w1)).
struct Weights {
  float w0;
  float2 w21;
};

// fmod(a, h) from the floor s of the rounded quotient a / h. (A negative a is
// inside only where a / h underflows to -0; fmod(a, h) is then a itself.)
__device__ __forceinline__ float remainder_general(float a, float s, float h) {
  float r = fmaf(-s, h, a);
  if (r < 0.0f && a > 0.0f) r = __fadd_rn(r, h);
  if (r == 0.0f) r = copysignf(0.0f, a);
  return r;
}

// Subscripts of a cell's first node, and the same as floats.
struct Cell {
  uint32_t i0, i1, i2;
  float s[3];
};

// Where a position falls in the grid, per axis: the rounded quotient
// q = (p - offset) / h, its floor s (the cell subscript) and the weight
// w = fmod(p - offset, h) / h, all as the reference rounds them. The position
// is inside iff 0 <= s <= n - 2 on every axis (regular_grid::contains), which
// for any float q (NaN included) is 0 <= q < n - 1.
//
// kLocatePow2: q is one FMA of the exact p / h and offset / h, and
// fmod(a, h) / h = q - s, whose difference is representable; a zero weight
// takes q's sign as fmod's takes a's (q - s is -0 - (+0) = -0 for q = -0).
//
// Other spacings: the rounded quotient is either the true integer quotient N
// or N + 1 (only when a / h lies within half an ulp below N + 1, so that
// fmod(a, h) >= h / 2). In both cases a - s * h is exactly representable, so
// one FMA gives it exactly; adding h back in the N + 1 case is exact too.
// Both divisions are IEEE division (kLocateDivide) or by the verified
// reciprocal pair (kLocateReciprocal), which gives the same bits.
//
// kLocateReciprocal's fields have spacings in [2^-40, 2^40]. One test, every
// a >= 2^-64, then covers both divisions: a quotient beyond divide_by_
// reciprocal's upper bound is outside whatever its last bits; a remainder is
// zero (+0 on both paths, a being positive) or a multiple of half an ulp of h,
// hence at least 2^-64. Anything else (a start on the grid's lower faces, a
// position that left through one) takes the guarded divisions.
//
// The floor and its integer come from one round-down add: for 0 <= q < 2^23,
// RD(q + 2^23) is 2^23 + floor(q), whose low mantissa bits are floor(q), and
// subtracting 2^23 again is exact. Inside the grid q < n - 1 <= 2^23 (the
// field's axes hold at most 2^23 nodes); outside it neither value is used.
__device__ __forceinline__ void floor_bits(const float q[3], float s[3], Cell& c) {
  constexpr uint32_t kTwo23 = 0x4B000000u;  // the bits of 2^23
  uint32_t i[3];
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    const float b = __fadd_rd(q[k], 0x1p23f);
    s[k] = __fsub_rn(b, 0x1p23f);
    i[k] = __float_as_uint(b) - kTwo23;
  }
  c = {i[0], i[1], i[2], {s[0], s[1], s[2]}};
}

// Locates p; c receives its cell (meaningful only when p is inside).
template <int kLocate>
__device__ __forceinline__ bool locate(const FieldView& f, const Position& p, Cell& c,
                                       Weights& w) {
  const float x[3] = {p.p0, p.p21.y, p.p21.x};
  float q[3], s[3], v[3];
  if constexpr (kLocate == kLocatePow2) {
    // q = p / h - offset / h in one rounding: p / h and offset / h are exact,
    // so this is the reference's rounded (p - offset) scaled by 1 / h.
#pragma unroll
    for (int k = 0; k < 3; ++k) q[k] = __fmaf_rn(x[k], f.reciprocal[k], -f.scaled_offset[k]);
    floor_bits(q, s, c);
#pragma unroll
    for (int k = 0; k < 3; ++k) v[k] = __fsub_rn(q[k], s[k]);
  } else {
    float a[3];
#pragma unroll
    for (int k = 0; k < 3; ++k) a[k] = __fsub_rn(x[k], f.offset[k]);
    if (kLocate == kLocateReciprocal && a[0] >= 0x1p-64f && a[1] >= 0x1p-64f &&
        a[2] >= 0x1p-64f) {
      auto divide = [&](float n, int k) {
        return __fmaf_rn(n, f.reciprocal[k], __fmul_rn(n, f.reciprocal_lo[k]));
      };
#pragma unroll
      for (int k = 0; k < 3; ++k) q[k] = divide(a[k], k);
      floor_bits(q, s, c);
#pragma unroll
      for (int k = 0; k < 3; ++k) {
        float r = __fmaf_rn(-s[k], f.spacing[k], a[k]);
        if (r < 0.0f) r = __fadd_rn(r, f.spacing[k]);
        v[k] = divide(r, k);
      }
    } else {
#pragma unroll
      for (int k = 0; k < 3; ++k)
        q[k] = divide_spacing<kLocate>(a[k], f.spacing[k], f.reciprocal[k], f.reciprocal_lo[k]);
      floor_bits(q, s, c);
#pragma unroll
      for (int k = 0; k < 3; ++k)
        v[k] = divide_spacing<kLocate>(remainder_general(a[k], s[k], f.spacing[k]), f.spacing[k],
                                       f.reciprocal[k], f.reciprocal_lo[k]);
    }
  }
  w.w0 = v[0];
  w.w21 = make_float2(v[2], v[1]);
  // 0 <= q < n - 1 iff 0 <= floor(q) < n - 1, and a negative, NaN, infinite
  // or too large q gives a difference of n - 1 or more as an unsigned value
  // (-0 gives 0, inside, as the reference has it).
  return (c.i0 < f.cells[0]) & (c.i1 < f.cells[1]) & (c.i2 < f.cells[2]);
}

// The tile of a subscript along an axis, plus the bits of 2^23 (TileLayout::bias takes
// them off): s * inverse + 2^23 rounded down, as in floor_bits. inverse is 1 / size
// rounded up, too large by less than 2^-23 / size, so that s * inverse never reaches the
// next integer for s < 2^23.
__device__ __forceinline__ uint32_t tile_bits(const TileLayout& t, int axis, float s) {
  return __float_as_uint(__fmaf_rd(s, t.inverse[axis], 0x1p23f));
}

// Index, within its slice, of a node in tile order.
__device__ __forceinline__ uint32_t tiled_node(const TileLayout& t, uint32_t i0, uint32_t i1,
                                               uint32_t i2) {
  return i0 * t.stride[0] + tile_bits(t, 0, float(i0)) * t.jump[0] + i1 * t.stride[1] +
         tile_bits(t, 1, float(i1)) * t.jump[1] + i2 + tile_bits(t, 2, float(i2)) * t.jump[2] +
         t.bias;
}

// Index of a cell's first node in row order: tells cells apart also in a tiled field, where
// the node's own index would cost three more products a sample.
__device__ __forceinline__ uint32_t first_node(const FieldView& f, const Cell& c) {
  return c.i0 * f.stride0 + c.i1 * f.stride1 + c.i2;
}

// Indices, within their slice, of the first nodes of a cell's four edges along
// axis 2: e = dx * 2 + dy.
struct CellRows {
  uint32_t at[4];
};

// Rows as they lie in memory, tiles with their numbers from tile_bits, and from products'
// high words.
enum class Rows { kInRow, kTiled, kTiledProducts };

template <Rows kRows>
__device__ __forceinline__ CellRows cell_rows(const FieldView& f, const Cell& c) {
  if constexpr (kRows == Rows::kTiled) {
    const TileLayout& t = f.tile;
    const uint32_t z = c.i2 + tile_bits(t, 2, c.s[2]) * t.jump[2] + t.bias;
    const uint32_t r0 = c.i0 * t.stride[0] + z, r1 = c.i1 * t.stride[1];
    const uint32_t a0 = r0 + tile_bits(t, 0, c.s[0]) * t.jump[0];
    const uint32_t a1 = r0 + t.stride[0] + tile_bits(t, 0, c.s[0] + 1.0f) * t.jump[0];
    const uint32_t b0 = r1 + tile_bits(t, 1, c.s[1]) * t.jump[1];
    const uint32_t b1 = r1 + t.stride[1] + tile_bits(t, 1, c.s[1] + 1.0f) * t.jump[1];
    return {a0 + b0, a0 + b1, a1 + b0, a1 + b1};
  } else if constexpr (kRows == Rows::kTiledProducts) {
    const TileLayout& t = f.tile;
    auto along = [&](int axis, uint32_t i) {
      return i * t.stride[axis] + __umulhi(i, t.magic[axis]) * t.jump[axis];
    };
    const uint32_t a0 = along(0, c.i0), a1 = along(0, c.i0 + 1);
    const uint32_t z = c.i2 + __umulhi(c.i2, t.magic[2]) * t.jump[2];
    const uint32_t b0 = along(1, c.i1) + z, b1 = along(1, c.i1 + 1) + z;
    return {a0 + b0, a0 + b1, a1 + b0, a1 + b1};
  } else {
    const uint32_t n = first_node(f, c);
    return {n, n + f.stride1, n + f.stride0, n + f.stride0 + f.stride1};
  }
}

// The eight corners of one cell are corner j = dx * 4 + dy * 2 + dz (the
// permute_for order of permute_for.hpp:12-34). Three register layouts of them
// serve the trilinear reduction of regular_grid.hpp:71-73 (axis 2, then 1,
// then 0, with c[j] = (1 - w) * c[2j] + w * c[2j+1]); all give the same bits,
// and each storage takes the one that its loads fill without register moves.
//
// CornerNodes (F32 nodes): xy[j] = (v0, v1) of corner j as the 16-byte node
// load leaves them, blended in packed form, and the third component beside
// them in scalar form. (Scalar lerps throughout: 6.6e9 warp instructions
// against 5.7e9 on a million seeds of 2000 steps; the launch, bound by the L1
// data pipe there, takes 10.4 and 10.2 ms.)
struct CornerNodes {
  float2 xy[8];
  float z[8];
};

// CornerPairs (F16 / BF16 nodes): p[k][c] = (component c of corner k, of
// corner k + 4), the two ends of an edge along axis 0, formed as 16-bit values
// are widened. Blends along axes 2 and 1 are packed over the two ends; the
// last, along axis 0, is one packed multiply and one scalar sum. (Pairs along
// axis 2, one packed multiply and one scalar sum for each of the 21 lerps: 224
// warp instructions a step against 202, 542 against 515 us a call of 200,003
// seeds and 400 steps in a stream of calls.)
struct CornerPairs {
  float2 p[4][3];
};

// CornerEdges (F32 edge records): z[e][c] = (component c of corner 2e,
// component c of corner 2e + 1), the two ends of edge e = dx * 2 + dy along
// axis 2, loaded as they are from an edge record. Each lerp is one packed
// multiply of (lo, hi) by the weight pair (1 - w, w) and one scalar sum.
struct CornerEdges {
  float2 z[4][3];
};

template <int kStorage>
using CornersOf = std::conditional_t<
    kStorage == DPA_STORAGE_F32, CornerNodes,
    std::conditional_t<kStorage == DPA_STORAGE_F32_EDGES, CornerEdges, CornerPairs>>;

// Node layouts (F32, F16, BF16): one 16-byte float4 (F32) or 8-byte uint2
// per node.
template <int kStorage>
using NodeOf = std::conditional_t<kStorage == DPA_STORAGE_F32, float4, uint2>;

// Edge records (F32_EDGES): record n holds node n and node n + 1 along axis
// 2 with each component's two values side by side, (x_n, x_n+1, y_n, y_n+1,
// z_n, z_n+1, 0, 0), 32 bytes read by one 256-bit load whose registers are
// already the (lo, hi) pairs the packed lerps take.
constexpr int kEdgeRecordBytes = 32;

__device__ __forceinline__ void load_edge_record(const char* record, float2 out[3]) {
  float v[8];
  asm("ld.global.nc.v8.f32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
      : "=f"(v[0]), "=f"(v[1]), "=f"(v[2]), "=f"(v[3]), "=f"(v[4]), "=f"(v[5]), "=f"(v[6]),
        "=f"(v[7])
      : "l"(record));
  out[0] = make_float2(v[0], v[1]);
  out[1] = make_float2(v[2], v[3]);
  out[2] = make_float2(v[4], v[5]);
}

template <int kStorage>
__device__ __forceinline__ const NodeOf<kStorage>* row_pointer(const FieldView& f, uint32_t row,
                                                               int64_t slice_base) {
  return reinterpret_cast<const NodeOf<kStorage>*>(f.nodes) + slice_base + row;
}

template <int kStorage>
__device__ __forceinline__ void gather(const FieldView& f, const CellRows& rows, CornerNodes& k,
                                       int64_t slice_base = 0) {
#pragma unroll
  for (int e = 0; e < 4; ++e) {
    const NodeOf<kStorage>* at = row_pointer<kStorage>(f, rows.at[e], slice_base);
    load_node<kStorage>(at, 0, k.xy[2 * e].x, k.xy[2 * e].y, k.z[2 * e]);
    load_node<kStorage>(at, 1, k.xy[2 * e + 1].x, k.xy[2 * e + 1].y, k.z[2 * e + 1]);
  }
}

// gather() of F32 nodes into CornerNodes only where `need` holds, by
// predicated loads instead of a branch: elsewhere the corners keep their
// values and no load is made.
__device__ __forceinline__ void load_node_if(bool need, const float4* at, float2& xy, float& z) {
  asm("{\n\t.reg .pred p;\n\t.reg .f32 pad;\n\tsetp.ne.u32 p, %4, 0;\n\t"
      "@p ld.global.nc.v4.f32 {%0, %1, %2, pad}, [%3];\n\t}"
      : "+f"(xy.x), "+f"(xy.y), "+f"(z)
      : "l"(at), "r"(need ? 1u : 0u));
}

__device__ __forceinline__ void gather_if(const FieldView& f, const CellRows& rows, bool need,
                                          CornerNodes& k) {
#pragma unroll
  for (int e = 0; e < 4; ++e) {
    const float4* at = row_pointer<DPA_STORAGE_F32>(f, rows.at[e], 0);
    load_node_if(need, at, k.xy[2 * e], k.z[2 * e]);
    load_node_if(need, at + 1, k.xy[2 * e + 1], k.z[2 * e + 1]);
  }
}

template <int kStorage>
__device__ __forceinline__ void gather(const FieldView& f, const CellRows& rows, CornerPairs& k,
                                       int64_t slice_base = 0) {
  const NodeOf<kStorage>* at[4];
#pragma unroll
  for (int e = 0; e < 4; ++e) at[e] = row_pointer<kStorage>(f, rows.at[e], slice_base);
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    float a[3], b[3];
    load_node<kStorage>(at[j >> 1], j & 1, a[0], a[1], a[2]);
    load_node<kStorage>(at[2 + (j >> 1)], j & 1, b[0], b[1], b[2]);
#pragma unroll
    for (int i = 0; i < 3; ++i) k.p[j][i] = make_float2(a[i], b[i]);
  }
}

template <int kStorage>
__device__ __forceinline__ void gather(const FieldView& f, const CellRows& rows, CornerEdges& k,
                                       int64_t slice_base = 0) {
#pragma unroll
  for (int e = 0; e < 4; ++e)
    load_edge_record(static_cast<const char*>(f.nodes) +
                         (uint64_t(slice_base) + rows.at[e]) * uint64_t(kEdgeRecordBytes),
                     k.z[e]);
}

__device__ __forceinline__ void trilinear(const FieldView& f, const CornerNodes& k,
                                          const Weights& w, float2& v01, float& v2) {
  const float2 unit = make_float2(f.unit[0], f.unit[1]);
  const float w2 = w.w21.x, t2 = __fsub_rn(1.0f, w2);
  const float w1 = w.w21.y, t1 = __fsub_rn(1.0f, w1);
  const float w0 = w.w0, t0 = __fsub_rn(1.0f, w0);
  float2 e[4];
  float z[4];
#pragma unroll
  for (int r = 0; r < 4; ++r) {
    e[r] = blend2(k.xy[2 * r], k.xy[2 * r + 1], splat(t2), splat(w2), unit);
    z[r] = blend(k.z[2 * r], k.z[2 * r + 1], t2, w2);
  }
  const float2 f0 = blend2(e[0], e[1], splat(t1), splat(w1), unit);
  const float2 f1 = blend2(e[2], e[3], splat(t1), splat(w1), unit);
  v01 = blend2(f0, f1, splat(t0), splat(w0), unit);
  v2 = blend(blend(z[0], z[1], t1, w1), blend(z[2], z[3], t1, w1), t0, w0);
}

// (1 - w) * lo + w * hi for the pair lohi = (lo, hi) and tw = (1 - w, w).
__device__ __forceinline__ float lerp_pair(float2 lohi, float2 tw) {
  const float2 m = mul2(tw, lohi);
  return __fadd_rn(m.x, m.y);
}

__device__ __forceinline__ void trilinear(const FieldView& f, const CornerPairs& k,
                                          const Weights& w, float2& v01, float& v2) {
  const float2 unit = make_float2(f.unit[0], f.unit[1]);
  const float2 w2 = splat(w.w21.x), t2 = splat(__fsub_rn(1.0f, w.w21.x));
  const float2 w1 = splat(w.w21.y), t1 = splat(__fsub_rn(1.0f, w.w21.y));
  const float2 tw0 = make_float2(__fsub_rn(1.0f, w.w0), w.w0);
  float v[3];
#pragma unroll
  for (int i = 0; i < 3; ++i) {
    const float2 e0 = blend2(k.p[0][i], k.p[1][i], t2, w2, unit);
    const float2 e1 = blend2(k.p[2][i], k.p[3][i], t2, w2, unit);
    v[i] = lerp_pair(blend2(e0, e1, t1, w1, unit), tw0);
  }
  v01 = make_float2(v[0], v[1]);
  v2 = v[2];
}

__device__ __forceinline__ void trilinear(const FieldView&, const CornerEdges& k,
                                          const Weights& w, float2& v01, float& v2) {
  const float2 tw2 = make_float2(__fsub_rn(1.0f, w.w21.x), w.w21.x);
  const float2 tw1 = make_float2(__fsub_rn(1.0f, w.w21.y), w.w21.y);
  const float2 tw0 = make_float2(__fsub_rn(1.0f, w.w0), w.w0);
  float v[3];
#pragma unroll
  for (int c = 0; c < 3; ++c) {
    const float e0 = lerp_pair(k.z[0][c], tw2), e1 = lerp_pair(k.z[1][c], tw2);
    const float e2 = lerp_pair(k.z[2][c], tw2), e3 = lerp_pair(k.z[3][c], tw2);
    const float f0 = lerp_pair(make_float2(e0, e1), tw1);
    const float f1 = lerp_pair(make_float2(e2, e3), tw1);
    v[c] = lerp_pair(make_float2(f0, f1), tw0);
  }
  v01 = make_float2(v[0], v[1]);
  v2 = v[2];
}

// A per-thread cache of the current cell's corners: a particle usually stays
// in one cell for several steps, and the sampled values do not depend on
// whether the corners came from the cache or from memory. kMode is the field's
// LocateMode, with kTiledBit for a tiled field.
template <int kStorage, int kMode>
struct CellSampler {
  static constexpr int kLocate = kMode & ~kTiledBit;
  static constexpr bool kTiled = (kMode & kTiledBit) != 0;
  CornersOf<kStorage> corners;
  // What tells the cached cell: where its first node lies, or its first_node in sample()
  // of a tiled field. No cell starts at ~0.
  uint32_t cached = ~0u;

  // Samples at p (a steady field: the time t is not used); returns false
  // when p is outside the grid. The sample is returned as v01 = (v0, v1)
  // and v2.
  __device__ __forceinline__ bool sample(const FieldView& f, const Position& p, float /*t*/,
                                         float2& v01, float& v2) {
    Cell c;
    Weights w;
    if (!locate<kLocate>(f, p, c, w)) return false;
    if constexpr (kTiled) {
      const uint32_t cell = first_node(f, c);
      if (cell != cached) {
        gather<kStorage>(f, cell_rows<Rows::kTiled>(f, c), corners);
        cached = cell;
      }
    } else {
      const CellRows rows = cell_rows<Rows::kInRow>(f, c);
      if (rows.at[0] != cached) {
        gather<kStorage>(f, rows, corners);
        cached = rows.at[0];
      }
    }
    trilinear(f, corners, w, v01, v2);
    return true;
  }

  // A branch-free step forms its rows whether it gathers or not. For F32 nodes and edge
  // records tile_bits saves 1 to 3 % of a launch whose particles stay in a cell, but where
  // address translations bind it loses: curl noise, 2 million seeds, ms by products and by
  // tile_bits, F32 512^3, 2000 steps of 0.25 cells 29.3 and 31.6, 560^3 of 0.3 68.3 and 71.8,
  // edge records of 330^3, 800 steps of 0.4 15.4 and 18.0, 450^3, 2000 of 0.3 32.1 and 35.2.
  // 16-bit nodes gain 4 to 7 % (420^3, 300 steps of 0.1 cells 4.16 and 3.92 ms, in rows 3.81)
  // and lose at the largest only (700^3, 2000 of 0.25 32.3 and 33.0, of 0.3 39.8 and 49.8).
  static constexpr Rows kStepRows =
      !kTiled ? Rows::kInRow
      : kStorage == DPA_STORAGE_F32 || kStorage == DPA_STORAGE_F32_EDGES ? Rows::kTiledProducts
                                                                         : Rows::kTiled;

  // sample() without the early return, for a caller that selects its result:
  // an outside position loads no corners, and its sample (from the cached
  // ones) is to be discarded.
  __device__ __forceinline__ bool sample_selected(const FieldView& f, const Position& p,
                                                  float /*t*/, float2& v01, float& v2) {
    Cell c;
    Weights w;
    const bool inside = locate<kLocate>(f, p, c, w);
    const CellRows rows = cell_rows<kStepRows>(f, c);
    const bool need = inside && rows.at[0] != cached;
    if constexpr (kStorage == DPA_STORAGE_F32) {
      gather_if(f, rows, need, corners);
      cached = need ? rows.at[0] : cached;
    } else if (need) {
      gather<kStorage>(f, rows, corners);
      cached = rows.at[0];
    }
    trilinear(f, corners, w, v01, v2);
    return inside;
  }

  // (An edge-record field's kernels are at their register limit.)
  static constexpr bool kPackedSums = kStorage != DPA_STORAGE_F32_EDGES;

  __device__ __forceinline__ void reset() { cached = ~0u; }
};

// The time axis of a time-varying field, located by the spatial rule: slice
// k = floor((t - t0) / dt) of the rounded quotient, weight fmod(t - t0, dt) / dt,
// inside iff 0 <= k <= slices - 2. time_fast fields (spacing in [2^-40, 2^40], at
// most 2^23 slices) divide and take the floor as locate() does, without the
// conversions and the branches of the guarded divisions.
__device__ __forceinline__ bool locate_time(const FieldView& f, float t, uint32_t& k, float& w) {
  const float a = __fsub_rn(t, f.time_origin);
  const float y = f.time_reciprocal, yl = f.time_reciprocal_lo, h = f.time_spacing;
  if (f.time_fast && a >= 0x1p-64f) {
    const float b = __fadd_rd(__fmaf_rn(a, y, __fmul_rn(a, yl)), 0x1p23f);
    k = __float_as_uint(b) - 0x4B000000u;
    float r = __fmaf_rn(-__fsub_rn(b, 0x1p23f), h, a);
    if (r < 0.0f) r = __fadd_rn(r, h);
    w = __fmaf_rn(r, y, __fmul_rn(r, yl));
    return k < f.time_cells;
  }
  const float q = f.time_fast ? divide_by_reciprocal(a, h, y, yl) : __fdiv_rn(a, h);
  if (!(q >= 0.0f && q < f.time_upper)) return false;
  const float s = floorf(q);
  const float r = remainder_general(a, s, h);
  w = f.time_fast ? divide_by_reciprocal(r, h, y, yl) : __fdiv_rn(r, h);
  k = uint32_t(s);
  return true;
}

// Sampler of a time-varying field: the trilinear samples of the two slices
// around t at p, blended as (1 - w) * a + w * b per component. It caches the
// corners of both slices for the current cell and slice pair: a pathline
// usually stays in one cell for many steps and in one slice pair for many
// more, and the sampled values do not depend on whether the corners came
// from the cache or from memory.
template <int kStorage, int kLocate>
struct TimeSampler {
  CornersOf<kStorage> lo, hi;  // slices s and s + 1
  uint32_t cached = ~0u, cached_slice = 0;

  // Samples at p and time t without an early return, as CellSampler's; outside the
  // grid or the slices it returns false and loads nothing.
  __device__ __forceinline__ bool sample_selected(const FieldView& f, const Position& p, float t,
                                                  float2& v01, float& v2) {
    Cell c;
    Weights w;
    uint32_t slice = 0;
    float wt = 0.0f;
    const bool here = locate<kLocate>(f, p, c, w);
    const bool now = locate_time(f, t, slice, wt);
    const CellRows rows = cell_rows<Rows::kInRow>(f, c);
    if (here && now && (rows.at[0] != cached || slice != cached_slice)) {
      const int64_t base = int64_t(uint64_t(slice) * uint32_t(f.slice_stride));
      gather<kStorage>(f, rows, lo, base);
      gather<kStorage>(f, rows, hi, base + f.slice_stride);
      cached = rows.at[0];
      cached_slice = slice;
    }
    float2 a01, b01;
    float a2, b2;
    trilinear(f, lo, w, a01, a2);
    trilinear(f, hi, w, b01, b2);
    const float u = __fsub_rn(1.0f, wt);
    v01 = blend2(a01, b01, splat(u), splat(wt), make_float2(f.unit[0], f.unit[1]));
    v2 = blend(a2, b2, u, wt);
    return here && now;
  }

  __device__ __forceinline__ bool sample(const FieldView& f, const Position& p, float t,
                                         float2& v01, float& v2) {
    return sample_selected(f, p, t, v01, v2);
  }

  static constexpr bool kPackedSums = true;

  __device__ __forceinline__ void reset() { cached = ~0u; }
};

__device__ __forceinline__ bool is_zero(float2 v01, float v2) {
  return fabsf(v01.x) <= kZeroPrecision && fabsf(v01.y) <= kZeroPrecision &&
         fabsf(v2) <= kZeroPrecision;
}

enum StepResult : int { kStepTaken = 0, kStepOutOfBounds = 1, kStepZeroVelocity = 2 };

// What the general steppers keep of a particle's previous step: its
// derivative (as v01, v2) and whether the particle has taken a step yet.
// Every particle starts fresh, as the reference copies its integrator per
// particle (particle_advector.cpp:335).
struct StepHistory {
  float2 d01;
  float d2;
  bool started;
};

// odeint modified_midpoint with kSteps sub-steps and the state-independent
// derivative d, one component: m_x1 = x + h d; kSteps - 1 times
// (m_x1, m_x0) = (m_x0 + h2 d, m_x1); out = 0.5 m_x0 + 0.5 m_x1 + (0.5 h) d.
// mm = {h, h2, 0.5 h}.
template <int kSteps>
__device__ __forceinline__ float modified_midpoint(float x, float d, const float* mm) {
  float x1 = __fadd_rn(x, __fmul_rn(mm[0], d));
  float x0 = x;
#pragma unroll
  for (int i = 1; i < kSteps; ++i) {
    const float t = x1;
    x1 = __fadd_rn(x0, __fmul_rn(mm[1], d));
    x0 = t;
  }
  return __fadd_rn(__fadd_rn(__fmul_rn(0.5f, x0), __fmul_rn(0.5f, x1)), __fmul_rn(mm[2], d));
}

// The Adams methods' initialising stepper (an order-4 extrapolation
// stepper): modified midpoints with 2 and 4 sub-steps, one polynomial
// extrapolation x = (1 + c) mm4 + (-c) mm2, c = 1/3.
__device__ __forceinline__ float extrapolated_start(float x, float d, const GeneralCoefficients& g) {
  const float a = modified_midpoint<2>(x, d, g.mm2);
  const float b = modified_midpoint<4>(x, d, g.mm4);
  return __fadd_rn(__fmul_rn(g.ex[0], b), __fmul_rn(g.ex[1], a));
}

// One step of a general stepper (kGeneralIntegrator) given this step's
// derivative; updates the history.
__device__ __forceinline__ void general_step(const GeneralCoefficients& g, float2 v01, float v2,
                                             StepHistory& h, Position& p) {
  if (g.kind == kGeneralMidpoint) {
    p.p0 = modified_midpoint<2>(p.p0, v2, g.mm2);
    p.p21 = make_float2(modified_midpoint<2>(p.p21.x, v01.x, g.mm2),
                        modified_midpoint<2>(p.p21.y, v01.y, g.mm2));
  } else if (g.extrapolated_start && !h.started) {
    p.p0 = extrapolated_start(p.p0, v2, g);
    p.p21 = make_float2(extrapolated_start(p.p21.x, v01.x, g),
                        extrapolated_start(p.p21.y, v01.y, g));
  } else {
    float x0 = p.p0, xa = p.p21.x, xb = p.p21.y;
#pragma unroll
    for (int i = 0; i < 13; ++i) {
      if (i < g.terms) {
        const bool prev = h.started && ((g.prev_mask >> i) & 1u);
        x0 = __fadd_rn(x0, __fmul_rn(g.s[i], prev ? h.d2 : v2));
        xa = __fadd_rn(xa, __fmul_rn(g.s[i], prev ? h.d01.x : v01.x));
        xb = __fadd_rn(xb, __fmul_rn(g.s[i], prev ? h.d01.y : v01.y));
      }
    }
    p.p0 = x0;
    p.p21 = make_float2(xa, xb);
  }
  h.d01 = v01;
  h.d2 = v2;
  h.started = true;
}

// a + b for the sum of a position and a product: packed (add2), or for
// samplers that hold no unit pair two scalar sums.
template <bool kPacked>
__device__ __forceinline__ float2 advance(float2 a, float2 b, float2 unit) {
  if constexpr (kPacked) return add2(a, b, unit);
  else return make_float2(__fadd_rn(a.x, b.x), __fadd_rn(a.y, b.y));
}

// One integrator step in place. The derivative of p0 is v2 and that of
// (p2, p1) is (v0, v1) (particle_advector.cpp:369).
// t is the particle's time (used by time-varying fields only); the caller
// advances it by dt after a step is taken.
// active: false for an empty slot, which the branch-free steps below run
// through without moving it (its position is parked inside the grid).
template <int kIntegrator, class Sampler>
__device__ __forceinline__ int step(const FieldView& f, const StepCoefficients& k,
                                   Sampler& sampler, Position& p, float t,
                                   StepHistory& history, bool active = true) {
  constexpr bool kPacked = Sampler::kPackedSums;
  const float2 unit = make_float2(f.unit[0], f.unit[1]);
  float2 v01;
  float v2;
  if constexpr (kIntegrator == DPA_INTEGRATOR_EULER ||
                kIntegrator == DPA_INTEGRATOR_RUNGE_KUTTA_4) {
    // Without branches on the outcome: the step is computed whatever the
    // sample, and kept only when the position was inside and the velocity
    // not zero (a step's latency is a dependent chain; the launch's end and
    // launches of few particles wait for it).
    const bool inside = sampler.sample_selected(f, p, t, v01, v2);
    const bool zero = is_zero(v01, v2);
    Position n = p;
    if constexpr (kIntegrator == DPA_INTEGRATOR_EULER) {
      // odeint euler: x = 1 * x + dt * dxdt
      n.p0 = __fadd_rn(p.p0, __fmul_rn(k.dt, v2));
      n.p21 = advance<kPacked>(p.p21, mul2(splat(k.dt), v01), unit);
    } else {
      // odeint runge_kutta4, final stage with four equal stage derivatives:
      // x = 1 * x + (b0 dt) d + (b1 dt) d + (b2 dt) d + (b3 dt) d, left to right.
      const float m0 = __fmul_rn(k.c0, v2), m1 = __fmul_rn(k.c1, v2);
      n.p0 = __fadd_rn(__fadd_rn(__fadd_rn(__fadd_rn(p.p0, m0), m1), m1), m0);
      const float2 n0 = mul2(splat(k.c0), v01), n1 = mul2(splat(k.c1), v01);
      n.p21 = advance<kPacked>(n.p21, n0, unit);
      n.p21 = advance<kPacked>(n.p21, n1, unit);
      n.p21 = advance<kPacked>(n.p21, n1, unit);
      n.p21 = advance<kPacked>(n.p21, n0, unit);
    }
    const bool taken = active && inside && !zero;
    p.p0 = taken ? n.p0 : p.p0;
    p.p21 = make_float2(taken ? n.p21.x : p.p21.x, taken ? n.p21.y : p.p21.y);
    return !(active && inside) ? int(kStepOutOfBounds)
           : zero              ? int(kStepZeroVelocity)
                               : int(kStepTaken);
  } else {
    if (!sampler.sample(f, p, t, v01, v2)) return kStepOutOfBounds;
    if (is_zero(v01, v2)) return kStepZeroVelocity;
    if constexpr (kIntegrator == kGeneralIntegrator) {
      general_step(k.g, v01, v2, history, p);
    } else {
      // Four-sample RK4; a stage outside the grid ends the particle without
      // taking the step.
      float2 k2_01, k3_01, k4_01;
      float k2_2, k3_2, k4_2;
      Position x;
      x.p0 = __fadd_rn(p.p0, __fmul_rn(k.half, v2));
      x.p21 = advance<kPacked>(p.p21, mul2(splat(k.half), v01), unit);
      const float t_half = __fadd_rn(t, k.half), t_end = __fadd_rn(t, k.dt);
      if (!sampler.sample(f, x, t_half, k2_01, k2_2)) return kStepOutOfBounds;
      x.p0 = __fadd_rn(p.p0, __fmul_rn(k.half, k2_2));
      x.p21 = advance<kPacked>(p.p21, mul2(splat(k.half), k2_01), unit);
      if (!sampler.sample(f, x, t_half, k3_01, k3_2)) return kStepOutOfBounds;
      x.p0 = __fadd_rn(p.p0, __fmul_rn(k.dt, k3_2));
      x.p21 = advance<kPacked>(p.p21, mul2(splat(k.dt), k3_01), unit);
      if (!sampler.sample(f, x, t_end, k4_01, k4_2)) return kStepOutOfBounds;
      p.p0 = __fadd_rn(__fadd_rn(__fadd_rn(__fadd_rn(p.p0, __fmul_rn(k.c0, v2)),
                                           __fmul_rn(k.c1, k2_2)),
                                 __fmul_rn(k.c1, k3_2)),
                       __fmul_rn(k.c0, k4_2));
      const float2 c0 = splat(k.c0), c1 = splat(k.c1);
      p.p21 = advance<kPacked>(p.p21, mul2(c0, v01), unit);
      p.p21 = advance<kPacked>(p.p21, mul2(c1, k2_01), unit);
      p.p21 = advance<kPacked>(p.p21, mul2(c1, k3_01), unit);
      p.p21 = advance<kPacked>(p.p21, mul2(c0, k4_01), unit);
    }
    return kStepTaken;
  }
}

}  // namespace dpa
