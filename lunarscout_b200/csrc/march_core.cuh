// The per-ray core of the horizon march, shared by the per-tile production
// kernel (march.cu) and the persistent multi-site kernel (march_batch.cu).
//
// Semantics follow src/lunarscout/_numba_horizon/cuda_backend.py:
//   subpatch_hierarchy_kernel :1007-1134 (segment interpolation, observer)
//   hierarchy_maximum          :656-874  (the march)
//   helpers                    :43-132
//
// Arithmetic contract.  The including files are compiled with --fmad=false,
// so every written multiply and add rounds separately, and the multiply-adds
// that the reference's GPU compiler fuses are written as explicit __fmaf_rn:
//   * every "x + a*b" / "x - a*b" whose product feeds the add is fused;
//   * for "a*b + c*d" the first product is fused, except local_x^2 =
//     dist*dist - local_z^2, which fuses local_z^2.
// That is the reference's Numba-CUDA kernel as NVVM compiles it on the B200
// (its slopes on the same GPU are the golden file numba_cuda_b200.npz of the
// tests).  Division, reciprocal and square root are IEEE round-to-nearest;
// the tangent's reciprocals come from rcp.approx plus one Newton step, which
// equals the IEEE reciprocal on every input it receives (see rcp_approx).
// The x and y arithmetic of a step (path position and tangent, planar
// offset, cell-exit slab) is issued as f32x2 pairs, whose lanes round as the
// scalar intrinsics do.  No shift amount comes from stored state unclamped:
// an amount out of range is undefined even on a path that is never taken
// (slow_step clamps the level that it loads).
// With the same segment inputs the results are bit-identical to the CPU
// oracle's FP32 restatement under its production mask.
//
// The march is bound by the latency of a step's chain and by instruction issue
// (71 % of the slots; its gathers hit L1/L2), so the work per node visit is kept
// small without changing any rounded value or decision:
//   * cells come from a sanitized copy of level 0 (invalid -> -32000) packed
//     with the mips, so validity is one comparison and the four-cell bound
//     is a plain maximum;
//   * per-level constants (cell side, step and fallback advances, offsets)
//     come from a table computed once per DEM;
//   * the tangent and its reciprocals depend only on the ray position and are
//     computed once per position, not per level;
//   * the cull test decides with a cheap bound outside a guard band and with
//     the reference arithmetic inside it (bound_culled);
//   * in the reference traversal most far-field culls are settled by a step
//     of 55 instructions that computes exactly only what moves the ray
//     (FarRay, march_dem_far), most other steps by level0_step, and the
//     first 500 m of a ray by march_near.
//
// The skip ladder (kLadder, the batched traversal; no reference counterpart)
// extends a cull to the largest culled ancestor cell, see ladder_advance.
//
// The relative arithmetic (kRelative; no reference counterpart) marches the
// same algorithm in FP32 on coordinates and heights relative to a local
// origin: positions as an integer origin (near the ray start) plus small
// offsets, level-0 heights as differences from the observer's z taken
// before interpolation, and the far-field local z from that difference
// (never rounding R + height on its own).  The FP32 reference arithmetic
// rounds absolute coordinates (an ulp of 5e-4 px at 4096 px) and absolute
// heights, which at the 1 m first sample moves the slope by up to ~0.02 deg;
// the relative march stays within ~1e-4 deg of the FP64 restatement.
#pragma once

#include "internal.cuh"

namespace ls200 {

// Per-level constants of one DEM.
struct LevelTable {
    float side[kMaxLevels];      // float(4^l) * resolution: the level choice
    float fallback[kMaxLevels];  // ((side * 0.5) * 0.001)
    float out_step[kMaxLevels];  // max(0.001, side * 0.001)
    int4 cells[kMaxLevels];      // (cell offset, width, height, fallback bits)
};

// Everything the march of one DEM pass needs about the DEM.
struct DemView {
    const float *cells;   // sanitized level 0 + packed mips
    const float *bounds;  // four-cell bound of every cell, the layout of cells
    int width, height, level_count;
    float resolution;    // mean pixel size of the DEM (m)
    float column_res;    // hypot of the column axis of the geotransform
    float radius;
};

// The ladder acts from this distance on (m); nearer, steep crater walls make
// the reference's slope formula sensitive to where samples fall.
constexpr float kLadderMinimumDistance = 1000.0f;

// Warp-aggregated counter update over the lanes that reach it together
// (counting launches are diagnostics, never timed).
__device__ __forceinline__ void add_counters(unsigned long long *counters, unsigned visits,
                                             unsigned samples, unsigned steps) {
    const unsigned mask = __activemask();
    const unsigned v = __reduce_add_sync(mask, visits);
    const unsigned n = __reduce_add_sync(mask, samples);
    const unsigned t = __reduce_add_sync(mask, steps);
    if ((threadIdx.x & 31) == __ffs(mask) - 1) {
        atomicAdd(counters, static_cast<unsigned long long>(v));
        atomicAdd(counters + 1, static_cast<unsigned long long>(n));
        atomicAdd(counters + 2, static_cast<unsigned long long>(t));
    }
}

// Correctly rounded reciprocal: the hardware approximation plus one
// Newton-Raphson correction whose residual an FMA forms exactly,
// y' = y + y (1 - x y) with y ~ 1/x (P. W. Markstein, "Computation of
// elementary functions on the IBM RISC System/6000 processor", IBM J. Res.
// Develop. 34(1), 1990).  For 2^-64 <= |x| < 2^64 it equals __frcp_rn bit for
// bit; |x| >= 2^64, infinities and NaN take __frcp_rn itself.
// ls200_check_arithmetic compares every pattern with |x| >= 2^-64.
__device__ __forceinline__ float rcp_approx(float x) {
    float y;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}

__device__ __forceinline__ float hypot_fused(float a, float b) {
    return __fsqrt_rn(__fmaf_rn(a, a, __fmul_rn(b, b)));
}

// Mean pixel size (m) from the geotransform terms m6, m7 (column axis) and
// m9, m10 (row axis) (cuda_backend.py:1036-1040).
__device__ __forceinline__ float mean_resolution(float m6, float m7, float m9, float m10) {
    return __fmul_rn(__fadd_rn(hypot_fused(m6, m9), hypot_fused(m7, m10)), 0.5f);
}

// Fill entry `l` of a level table (block_m = float(4^l) * resolution).
__device__ __forceinline__ void fill_level(LevelTable &table, int l, float resolution,
                                           int4 cells) {
    const float block_m = __fmul_rn(static_cast<float>(1 << (2 * l)), resolution);
    const float step_km = __fmul_rn(block_m, 0.001f);
    table.side[l] = block_m;
    table.fallback[l] = __fmul_rn(__fmul_rn(block_m, 0.5f), 0.001f);
    table.out_step[l] = 0.001f > step_km ? 0.001f : step_km;
    // w carries the fallback's bits: a visit reads its cells and its
    // fallback with one 16-byte load.
    table.cells[l] = make_int4(cells.x, cells.y, cells.z, __float_as_int(table.fallback[l]));
}

// 2^shift as a float (exact; shift <= 38), from the exponent bits.
__device__ __forceinline__ float power_of_two(int shift) {
    return __int_as_float((127 + shift) << 23);
}

// Two FP32 lanes per instruction (the f32x2 operations of sm_100): each
// lane rounds exactly as the scalar __fadd_rn / __fmul_rn / __fmaf_rn does, so
// the march pairs its x and y arithmetic without changing a bit.
__device__ __forceinline__ float2 pair(float x, float y) { return make_float2(x, y); }
__device__ __forceinline__ float2 sub2(float2 a, float2 b) {
    float2 d;
    asm("sub.rn.f32x2 %0, %1, %2;"
        : "=l"(reinterpret_cast<unsigned long long &>(d))
        : "l"(reinterpret_cast<const unsigned long long &>(a)),
          "l"(reinterpret_cast<const unsigned long long &>(b)));
    return d;
}

__device__ __forceinline__ float2 add2_down(float2 a, float2 b) {  // rounding down
    float2 d;
    asm("add.rm.f32x2 %0, %1, %2;"
        : "=l"(reinterpret_cast<unsigned long long &>(d))
        : "l"(reinterpret_cast<const unsigned long long &>(a)),
          "l"(reinterpret_cast<const unsigned long long &>(b)));
    return d;
}
__device__ __forceinline__ float sqrt_approx(float x) {
    float y;
    asm("sqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}

// The quartic path polynomial of both axes at once: lane x with
// (start_x, a1..a4), lane y with (start_y, b1..b4); d2, d3, d4 are the powers
// of the path offset d (cuda_backend.py:62-73).
__device__ __forceinline__ float2 quartic2(float2 x0, float2 k1, float2 k2, float2 k3,
                                           float2 k4, float2 d, float2 d2, float2 d3,
                                           float2 d4) {
    float2 r = __ffma2_rn(k1, d, x0);
    r = __ffma2_rn(k2, d2, r);
    r = __ffma2_rn(k3, d3, r);
    return __ffma2_rn(k4, d4, r);
}

// The negated Newton reciprocal -1/x of both lanes without the range
// fallback (the caller handles |x| >= 2^64).  Starting from y ~ 1/(-x) the
// residual 1 - x/x is fma(x, y, 1) without negating x first, and every
// rounding is that of the positive reciprocal with its sign turned.
__device__ __forceinline__ float2 newton_minus_reciprocal_pair(float2 x) {
    const float2 y = pair(rcp_approx(-x.x), rcp_approx(-x.y));
    const float2 e = __ffma2_rn(x, y, pair(1.0f, 1.0f));
    return __ffma2_rn(y, e, y);
}

// The correctly rounded reciprocal of both lanes (see rcp_approx), the
// Newton step issued as f32x2 pairs; each lane needs |x| >= 2^-64.  The
// march inlines the same choice with one branch for both lanes.
__device__ __forceinline__ float2 reciprocal_pair(float2 x) {
    float2 y = newton_minus_reciprocal_pair(x);
    y = pair(-y.x, -y.y);
    if (!(fabsf(x.x) < 0x1p64f)) y.x = __frcp_rn(x.x);
    if (!(fabsf(x.y) < 0x1p64f)) y.y = __frcp_rn(x.y);
    return y;
}

// Its derivative: a1 + 2 a2 d + 3 a3 d^2 + 4 a4 d^3 per lane
// (cuda_backend.py:76-84).
__device__ __forceinline__ float2 quartic_tangent2(float2 k1, float2 k2, float2 k3, float2 k4,
                                                   float2 d, float2 d2, float2 d3) {
    float2 r = __ffma2_rn(__fmul2_rn(pair(2.0f, 2.0f), k2), d, k1);
    r = __ffma2_rn(__fmul2_rn(pair(3.0f, 3.0f), k3), d2, r);
    return __ffma2_rn(__fmul2_rn(pair(4.0f, 4.0f), k4), d3, r);
}

// Clamped bilinear sample of sanitized level-0 cells; -32000 when any corner
// is invalid (cuda_backend.py:107-132).
__device__ __forceinline__ float bilinear(const float *__restrict__ cells, int width,
                                          int height, float column, float row) {
    const float cmax = __fsub_rn(static_cast<float>(width), 1.0001f);
    const float rmax = __fsub_rn(static_cast<float>(height), 1.0001f);
    column = column > 0.0f ? column : 0.0f;
    column = column < cmax ? column : cmax;
    row = row > 0.0f ? row : 0.0f;
    row = row < rmax ? row : rmax;
    const int x0 = static_cast<int>(floorf(column));
    const int y0 = static_cast<int>(floorf(row));
    const int x1 = min(x0 + 1, width - 1);
    const int y1 = min(y0 + 1, height - 1);
    const float *r0 = cells + static_cast<size_t>(y0) * width;
    const float *r1 = cells + static_cast<size_t>(y1) * width;
    const float q00 = __ldg(r0 + x0), q10 = __ldg(r0 + x1);
    const float q01 = __ldg(r1 + x0), q11 = __ldg(r1 + x1);
    if (!(q00 > -20000.0f && q10 > -20000.0f && q01 > -20000.0f && q11 > -20000.0f))
        return -32000.0f;
    const float tx = __fsub_rn(column, static_cast<float>(x0));
    const float ty = __fsub_rn(row, static_cast<float>(y0));
    const float top = __fmaf_rn(tx, __fsub_rn(q10, q00), q00);
    const float bottom = __fmaf_rn(tx, __fsub_rn(q11, q01), q01);
    return __fmaf_rn(ty, __fsub_rn(bottom, top), top);
}

// The relative arithmetic's level-0 sample: the height above `base` (the
// observer's z) at column origin_x + offset_x, row origin_y + offset_y.  The
// rounded absolute coordinates only decide the clamp; inside the clamp range
// the cell comes from the origin plus the offset's integer part and the
// fraction from the offset, and the corners are taken relative to `base`
// before they are interpolated.  Returns false (no data) when a corner is
// invalid.
__device__ __forceinline__ bool bilinear_above(const float *__restrict__ cells, int width,
                                               int height, int origin_x, float offset_x,
                                               float absolute_x, int origin_y, float offset_y,
                                               float absolute_y, float base, float &above) {
    const float cmax = __fsub_rn(static_cast<float>(width), 1.0001f);
    const float rmax = __fsub_rn(static_cast<float>(height), 1.0001f);
    int x0, y0;
    float tx, ty;
    if (absolute_x >= 0.0f && absolute_x <= cmax && absolute_y >= 0.0f && absolute_y <= rmax) {
        const float fx = floorf(offset_x), fy = floorf(offset_y);
        x0 = origin_x + static_cast<int>(fx);
        y0 = origin_y + static_cast<int>(fy);
        tx = __fsub_rn(offset_x, fx);
        ty = __fsub_rn(offset_y, fy);
    } else {
        float column = absolute_x > 0.0f ? absolute_x : 0.0f;
        column = column < cmax ? column : cmax;
        float row = absolute_y > 0.0f ? absolute_y : 0.0f;
        row = row < rmax ? row : rmax;
        x0 = static_cast<int>(floorf(column));
        y0 = static_cast<int>(floorf(row));
        tx = __fsub_rn(column, static_cast<float>(x0));
        ty = __fsub_rn(row, static_cast<float>(y0));
    }
    const int x1 = min(x0 + 1, width - 1);
    const int y1 = min(y0 + 1, height - 1);
    const float *r0 = cells + static_cast<size_t>(y0) * width;
    const float *r1 = cells + static_cast<size_t>(y1) * width;
    float q00 = __ldg(r0 + x0), q10 = __ldg(r0 + x1);
    float q01 = __ldg(r1 + x0), q11 = __ldg(r1 + x1);
    if (!(q00 > -20000.0f && q10 > -20000.0f && q01 > -20000.0f && q11 > -20000.0f))
        return false;
    q00 = __fsub_rn(q00, base);
    q10 = __fsub_rn(q10, base);
    q01 = __fsub_rn(q01, base);
    q11 = __fsub_rn(q11, base);
    const float top = __fmaf_rn(tx, __fsub_rn(q10, q00), q00);
    const float bottom = __fmaf_rn(tx, __fsub_rn(q11, q01), q01);
    above = __fmaf_rn(ty, __fsub_rn(bottom, top), top);
    return true;
}

// The relative arithmetic's far-field slope of a sample `above` metres above
// the observer's z: the four-cell bound's local-z formula (bound_slope) with
// the height difference given directly.
__device__ __forceinline__ float above_slope(float dist, float above, float radius,
                                             float observer_z, float observer_radius) {
    const float squared = __fmul_rn(dist, dist);
    float radius_sum = __fadd_rn(__fmul_rn(2.0f, radius), __fadd_rn(observer_z, above));
    radius_sum = __fadd_rn(radius_sum, observer_z);
    const float numerator = __fmaf_rn(above, radius_sum, -squared);
    const float local_z = __fdiv_rn(numerator, __fmul_rn(2.0f, observer_radius));
    const float lx2 = __fmaf_rn(-local_z, local_z, squared);
    const float local_x = lx2 > 0.0f ? __fsqrt_rn(lx2) : 1e-6f;
    return __fdiv_rn(local_z, local_x);
}

// Local-z slope of a terrain point seen over the chord `dist`
// (cuda_backend.py:812-830): numerator fused on its first product, local_x^2
// = dist*dist - local_z^2 fused on local_z*local_z (dist*dist rounded), as
// the reference's Numba-CUDA kernel computes it on the B200.
__device__ __forceinline__ float sample_slope(float dist, float height, float radius,
                                              float observer_radius) {
    const float squared = __fmul_rn(dist, dist);
    const float point_radius = __fadd_rn(radius, height);
    const float radius_delta = __fsub_rn(point_radius, observer_radius);
    const float radius_sum = __fadd_rn(point_radius, observer_radius);
    const float numerator = __fmaf_rn(radius_delta, radius_sum, -squared);
    const float local_z = __fdiv_rn(numerator, __fmul_rn(2.0f, observer_radius));
    const float lx2 = __fmaf_rn(-local_z, local_z, squared);
    const float local_x = lx2 > 0.0f ? __fsqrt_rn(lx2) : 1e-6f;
    return __fdiv_rn(local_z, local_x);
}

// The same for the four-cell culling bound (cuda_backend.py:777-795).
__device__ __forceinline__ float bound_slope(float dist, float height, float radius,
                                             float observer_z, float observer_radius) {
    const float squared = __fmul_rn(dist, dist);
    const float height_delta = __fsub_rn(height, observer_z);
    float radius_sum = __fadd_rn(__fmul_rn(2.0f, radius), height);
    radius_sum = __fadd_rn(radius_sum, observer_z);
    const float numerator = __fmaf_rn(height_delta, radius_sum, -squared);
    const float local_z = __fdiv_rn(numerator, __fmul_rn(2.0f, observer_radius));
    const float lx2 = __fmaf_rn(-local_z, local_z, squared);
    const float local_x = lx2 > 0.0f ? __fsqrt_rn(lx2) : 1e-6f;
    return __fdiv_rn(local_z, local_x);
}

// Exactly `possible <= current` for the four-cell bound `possible` of the
// reference (near field: fl((h - oz) / tn); far field: bound_slope), at a
// fraction of its cost.  The cull test is the most frequent operation of the
// march and `possible` only feeds this comparison, so an approximation may
// decide it whenever it lies outside a guard band around `current`:
//   near: __fdividef has at most 2 ulp error;
//   far:  the numerator is the exact one; z = num * rcp(den) is within 3 ulp
//         of fl(num / den); with local_x^2 > tn^2 / 4 (bound below 60 deg)
//         the cancellation in local_x^2 amplifies that by at most 3, and
//         rsqrtf adds 2 ulp: the approximation is within 2e-6 (relative) of
//         the exact FP32 value.
// The band is 1e-5 relative, five times that bound; inside it, and for
// steeper bounds, the exact arithmetic of the reference decides.
__device__ __forceinline__ bool bound_culled(bool near, float true_near, float height,
                                             float radius, float observer_z,
                                             float observer_radius, float inverse_denominator,
                                             float current) {
    float approx;
    if (near) {
        approx = __fdividef(__fsub_rn(height, observer_z), true_near);
    } else {
        const float squared = __fmul_rn(true_near, true_near);
        const float height_delta = __fsub_rn(height, observer_z);
        float radius_sum = __fadd_rn(__fmul_rn(2.0f, radius), height);
        radius_sum = __fadd_rn(radius_sum, observer_z);
        const float numerator = __fmaf_rn(height_delta, radius_sum, -squared);
        const float local_z = __fmul_rn(numerator, inverse_denominator);
        const float lx2 = __fmaf_rn(true_near, true_near, -__fmul_rn(local_z, local_z));
        if (!(lx2 > 0.25f * squared)) {
            return bound_slope(true_near, height, radius, observer_z, observer_radius) <= current;
        }
        approx = __fmul_rn(local_z, rsqrtf(lx2));
    }
    const float band = 1e-5f * fmaxf(fabsf(approx), fabsf(current));
    if (approx < current - band) return true;
    if (approx > current + band) return false;
    const float possible =
        near ? __fdiv_rn(__fsub_rn(height, observer_z), true_near)
             : bound_slope(true_near, height, radius, observer_z, observer_radius);
    return possible <= current;
}

__device__ __forceinline__ int clamp_center(int requested, int dem_size, int subpatch) {
    const int half = subpatch / 2;
    int maximum = dem_size - half;
    if (maximum < half) maximum = half;
    if (requested < half) return half;
    if (requested > maximum) return maximum;
    return requested;
}

// Four-cell bound of the level cell (cx, cy): the maximum of the cell and its
// right / lower / diagonal neighbours, -32000 standing in for a missing one.
__device__ __forceinline__ float four_cell_bound(const float *__restrict__ cells, int4 L,
                                                 int cx, int cy) {
    const int index = L.x + cy * L.y + cx;
    const bool has_right = cx + 1 < L.y, has_down = cy + 1 < L.z;
    const float v00 = __ldg(cells + index);
    const float v10 = has_right ? __ldg(cells + index + 1) : -32000.0f;
    const float v01 = has_down ? __ldg(cells + index + L.y) : -32000.0f;
    const float v11 = has_right && has_down ? __ldg(cells + index + L.y + 1) : -32000.0f;
    return fmaxf(fmaxf(v00, v10), fmaxf(v01, v11));
}

// The same value read from the precomputed bound table (one load per visit).
__device__ __forceinline__ float cell_bound(const float *__restrict__ bounds, int4 L, int cx,
                                            int cy) {
    return __ldg(bounds + L.x + cy * L.y + cx);
}

// Advance (km) to the exit of the cell (cx, cy) of side 4^level pixels along
// the tangent, or `fallback` when the exit is not ahead, + 1e-4 km
// (cuda_backend.py:733-762).  Of max(t1, t2) only the far edge can win:
// (min_x - px) <= 0 < (max_x - px), so the product with inv_x keeps that
// order's sign pattern and the larger t is the edge ahead of the ray
// (bitwise the same value, including the -0.0 of a ray starting on the edge).
// (ux, uy) is the position relative to the integer origin (origin_x,
// origin_y); the reference arithmetic is origin 0 with u the absolute position.
// minus_inv is the negated reciprocal of the tangent: (u - edge) * -1/t rounds
// to the same value as (edge - u) * 1/t.
__device__ __forceinline__ float cell_exit_advance(int shift, int cx, int cy, float ux, float uy,
                                                   int origin_x, int origin_y,
                                                   float2 minus_inv, float fallback) {
    const float scale_f = power_of_two(shift);
    const float2 low = pair(static_cast<float>((cx << shift) - origin_x),
                            static_cast<float>((cy << shift) - origin_y));
    const float2 high = __fadd2_rn(low, pair(scale_f, scale_f));
    const float2 edge = pair(minus_inv.x < 0.0f ? high.x : low.x,
                             minus_inv.y < 0.0f ? high.y : low.y);
    const float2 tm = __fmul2_rn(sub2(pair(ux, uy), edge), minus_inv);
    const float tmx = tm.x, tmy = tm.y;
    const float exit_distance = tmx < tmy ? tmx : tmy;
    // The reference returns `fallback` when the distance it adds 1e-4 km to
    // is not positive; that distance is the exit or, behind the ray, the
    // fallback, which is positive on every DEM that marches (the host
    // refuses pixel sizes too small for the ray length).  With a fallback of
    // zero the reference would not advance and its ray would never end.
    return __fadd_rn(exit_distance > 0.0f ? exit_distance : fallback, 0.0001f);
}

// The skip ladder.  After a cull at `level`, climb to the ancestors of the
// cell while each is culled by a conservative test, and return the advance
// to the exit of the largest culled one (`advance` when none is).  Every
// ancestor of an in-range cell is in range.  The test bounds the slope of
// every sample the skip passes over: heights are <= the ancestor's four-cell
// bound h, distances lie in [d0, d1] with d0 = true_m (distance grows along
// the ray) and d1 = d0 + 1010 m per km of advance + 1 m (a chord never
// outgrows the path).  With dh = h - observer_z >= 0 the slope falls with
// distance, so the bound is the slope formula at d0; with dh < 0 every slope
// is below dh / d1 (the curvature drop only lowers it).  The cull needs the
// bound below `current` by a relative 4e-6, which covers its rounding.
//
// The decision is made on a cheap approximation of the bound whenever it lies
// outside a guard band around `current` (as in bound_culled: the far-field
// approximation is within 2e-6 relative of the exact float32 bound, the
// divisions within 2 ulp; the band is 1e-5 relative), and with the exact
// arithmetic inside it, so the decision is always that of the exact test.
// ladder_culled tests the level-m ancestor and sets `step` to its exit
// advance; ladder_advance climbs from `level`, returns the advance and sets
// `reached` to the largest culled level (`level` if none).
template <class Table>
__device__ __forceinline__ bool ladder_culled(const Table &table, const float *__restrict__ bounds,
                                              int m, int ipx, int ipy, float ux, float uy,
                                              int origin_x, int origin_y, float2 minus_inv,
                                              bool near, float true_m, float radius, float observer_z,
                                              float observer_radius, float inverse_denominator,
                                              float current, float &step) {
    const int shift = 2 * m;
    const int cx = ipx >> shift, cy = ipy >> shift;
    const int4 L = table.cells(m);
    const float maximum_height = cell_bound(bounds, L, cx, cy);
    step = cell_exit_advance(shift, cx, cy, ux, uy, origin_x, origin_y, minus_inv,
                             __int_as_float(L.w));
    if (maximum_height < -20000.0f) return true;
    const float dh = __fsub_rn(maximum_height, observer_z);
    const float far_distance = __fadd_rn(__fadd_rn(true_m, __fmul_rn(step, 1010.0f)), 1.0f);
    float approx;
    bool exact = false;
    if (dh < 0.0f) {
        approx = __fdividef(dh, far_distance);
    } else if (near) {
        approx = __fdividef(dh, true_m);
    } else {
        const float squared = __fmul_rn(true_m, true_m);
        float radius_sum = __fadd_rn(__fmul_rn(2.0f, radius), maximum_height);
        radius_sum = __fadd_rn(radius_sum, observer_z);
        const float numerator = __fmaf_rn(dh, radius_sum, -squared);
        const float local_z = __fmul_rn(numerator, inverse_denominator);
        const float lx2 = __fmaf_rn(true_m, true_m, -__fmul_rn(local_z, local_z));
        exact = !(lx2 > 0.25f * squared);
        approx = exact ? 0.0f : __fmul_rn(local_z, rsqrtf(lx2));
    }
    if (!exact) {
        const float size = fmaxf(fabsf(approx), fabsf(current));
        const float decided = __fadd_rn(approx, __fmul_rn(4e-6f, size));
        const float band = 1e-5f * size + 1e-30f;
        if (decided < current - band) return true;
        if (decided > current + band) return false;
    }
    float bound;
    if (dh < 0.0f) {
        bound = __fdiv_rn(dh, far_distance);
    } else {
        bound = near ? __fdiv_rn(dh, true_m)
                     : bound_slope(true_m, maximum_height, radius, observer_z, observer_radius);
    }
    const float size = fmaxf(fabsf(bound), fabsf(current));
    return __fadd_rn(bound, __fmul_rn(4e-6f, size)) <= current;
}

template <bool kCount, class Table>
__device__ __forceinline__ float ladder_advance(const Table &table, const float *__restrict__ bounds,
                                                int level, int top, int ipx, int ipy, float ux,
                                                float uy, int origin_x, int origin_y,
                                                float2 minus_inv, bool near, float true_m,
                                                float radius, float observer_z,
                                                float observer_radius, float inverse_denominator,
                                                float current, float advance, unsigned &visits,
                                                int &reached) {
    reached = level;
    if (true_m < kLadderMinimumDistance) return advance;
    float best = advance;
    for (int m = level + 1; m <= top; ++m) {
        float step;
        if (kCount) ++visits;
        if (!ladder_culled(table, bounds, m, ipx, ipy, ux, uy, origin_x, origin_y, minus_inv,
                           near, true_m, radius, observer_z, observer_radius,
                           inverse_denominator, current, step))
            break;
        best = step;
        reached = m;
    }
    return best;
}

// One interpolated segment (fields 0,1,4..17 of the reference layout).
// With the relative arithmetic start_x, start_y are relative to the integer
// origin (origin_x, origin_y); otherwise the origin is 0.
struct RaySegment {
    float2 start;           // (start_x, start_y)
    float2 k1, k2, k3, k4;  // (a1, b1) .. (a4, b4)
    float s_start, s_end, s_start_chord, c1, c2, c3;
    int origin_x, origin_y;
};

// Subpatch interpolation of one ray's segment (cuda_backend.py:1032-1119):
// four centres around the pixel, their start points shifted to the pixel.
// kRelative: the origin is the integer part of the upper-left centre's start,
// and the four starts are taken relative to it before the shift and the
// interpolation (exact: they lie within a few pixels of each other).
template <bool kRelative = false>
__device__ __forceinline__ RaySegment interpolate_segment(
    const float *__restrict__ segments, int center_count, int dem_count, int pass_index,
    int azimuth, int column, int row, int tile_column, int tile_row, int tile_width,
    int subpatch, int primary_width, int primary_height, float ratio) {
    const int count = tile_width / subpatch + 2;
    const float gx = __fadd_rn(__fdiv_rn(static_cast<float>(column - subpatch / 2),
                                         static_cast<float>(subpatch)), 1.0f);
    const float gy = __fadd_rn(__fdiv_rn(static_cast<float>(row - subpatch / 2),
                                         static_cast<float>(subpatch)), 1.0f);
    int left = static_cast<int>(gx), top = static_cast<int>(gy);
    float tx = __fsub_rn(gx, static_cast<float>(left));
    float ty = __fsub_rn(gy, static_cast<float>(top));
    if (left < 0) { left = 0; tx = 0.0f; }
    if (top < 0) { top = 0; ty = 0.0f; }
    if (left > count - 2) { left = count - 2; tx = 1.0f; }
    if (top > count - 2) { top = count - 2; ty = 1.0f; }
    const int i00 = top * count + left, i10 = i00 + 1;
    const int i01 = (top + 1) * count + left, i11 = i01 + 1;
    const int req_left = tile_column + (left - 1) * subpatch + subpatch / 2;
    const int req_top = tile_row + (top - 1) * subpatch + subpatch / 2;
    const float d_left = static_cast<float>(
        column - (clamp_center(req_left, primary_width, subpatch) - tile_column));
    const float d_right = static_cast<float>(
        column - (clamp_center(req_left + subpatch, primary_width, subpatch) - tile_column));
    const float d_top = static_cast<float>(
        row - (clamp_center(req_top, primary_height, subpatch) - tile_row));
    const float d_bottom = static_cast<float>(
        row - (clamp_center(req_top + subpatch, primary_height, subpatch) - tile_row));

    const size_t stride_c = static_cast<size_t>(dem_count) * kSegmentFields;
    const float *base = segments + static_cast<size_t>(azimuth) * center_count * stride_c +
                        static_cast<size_t>(pass_index) * kSegmentFields;
    const float *s00 = base + i00 * stride_c, *s10 = base + i10 * stride_c;
    const float *s01 = base + i01 * stride_c, *s11 = base + i11 * stride_c;
    float seg[kMarchFields];
    int origin[2] = {0, 0};
    if (kRelative) {
        origin[0] = static_cast<int>(floorf(__ldg(s00 + 0)));
        origin[1] = static_cast<int>(floorf(__ldg(s00 + 1)));
    }
#pragma unroll
    for (int k = 0; k < kMarchFields; ++k) {
        const int f = k < 2 ? k : k + 2;
        float v00 = __ldg(s00 + f), v10 = __ldg(s10 + f);
        float v01 = __ldg(s01 + f), v11 = __ldg(s11 + f);
        if (kRelative && f < 2) {
            const float o = static_cast<float>(origin[f]);
            v00 = __fsub_rn(v00, o);
            v10 = __fsub_rn(v10, o);
            v01 = __fsub_rn(v01, o);
            v11 = __fsub_rn(v11, o);
        }
        if (f == 0) {
            v00 = __fmaf_rn(d_left, ratio, v00);
            v10 = __fmaf_rn(d_right, ratio, v10);
            v01 = __fmaf_rn(d_left, ratio, v01);
            v11 = __fmaf_rn(d_right, ratio, v11);
        } else if (f == 1) {
            v00 = __fmaf_rn(d_top, ratio, v00);
            v10 = __fmaf_rn(d_top, ratio, v10);
            v01 = __fmaf_rn(d_bottom, ratio, v01);
            v11 = __fmaf_rn(d_bottom, ratio, v11);
        }
        const float upper = __fmaf_rn(__fsub_rn(v10, v00), tx, v00);
        const float lower = __fmaf_rn(__fsub_rn(v11, v01), tx, v01);
        seg[k] = __fmaf_rn(__fsub_rn(lower, upper), ty, upper);
    }
    return RaySegment{pair(seg[0], seg[1]), pair(seg[2], seg[6]), pair(seg[3], seg[7]),
                      pair(seg[4], seg[8]), pair(seg[5], seg[9]), seg[10], seg[11],
                      seg[12], seg[13], seg[14], seg[15], origin[0], origin[1]};
}

// The state of one ray within one DEM pass of hierarchy_maximum.
struct MarchState {
    float s;            // path position (km)
    float current;      // maximum slope so far (-1e30 for none)
    int level_hint;     // level of the previous step
    // side(level_hint + 1) (NaN at the top level) and side(level_hint)
    // (-inf at level 0): the level search keeps level_hint whenever
    // !(side_up <= footprint) && side_here <= footprint.
    float side_up, side_here;
};

// side_here = +inf sends the first step through the full level search.
__device__ __forceinline__ MarchState begin_pass(const DemView &dem, const RaySegment &g,
                                                 float current) {
    return MarchState{g.s_start > 0.001f ? g.s_start : 0.001f, current, dem.level_count - 1,
                      __int_as_float(0x7fffffff), INFINITY};
}

// Traversals of march_step, a bit set: the reference's (0), the skip ladder
// (bit 0) and the relative arithmetic (bit 1).
enum Traversal { kReference = 0, kLadderClimb = 1, kRelative = 2 };


// Which level-0 sample set the running maximum: nothing (NoArgmax, the
// production kernels) or its position, distance and slope (Argmax, the
// checkpoint of the DEM adjoint; `pass` is set by the caller).
struct NoArgmax {
    __device__ __forceinline__ void record(float, float, float, float, bool) {}
};
struct Argmax {
    float px = 0.0f, py = 0.0f, true_m = 0.0f, slope = -1e30f;
    int near = 0, pass = -1;
    int current_pass = 0;
    __device__ __forceinline__ void record(float x, float y, float distance, float value,
                                           bool is_near) {
        px = x;
        py = y;
        true_m = distance;
        slope = value;
        near = is_near ? 1 : 0;
        pass = current_pass;
    }
};

// Where a ray stands at path position s: DEM position p, the position u
// relative to the integer origin (p itself in the reference arithmetic), the
// tangent and its negated reciprocals, which depend on s alone.
struct StepPoint {
    float2 p, u;
    float2 r;  // relative arithmetic: offset from the ray's start
    float2 tangent, minus_inv;
};

template <bool kRelativeArithmetic>
__device__ __forceinline__ StepPoint step_point(const RaySegment &g, float s) {
    StepPoint at;
    const float delta = __fsub_rn(s, g.s_start);
    const float2 d1 = pair(delta, delta);
    const float2 d2 = __fmul2_rn(d1, d1);
    const float2 d3 = __fmul2_rn(d2, d1);
    const float2 d4 = __fmul2_rn(d2, d2);
    // Relative arithmetic: offsets along the ray without the start, added
    // to the start relative to the origin; the absolute position (origin
    // + offset, rounded) only takes the bounds decisions.
    if (kRelativeArithmetic) {
        at.r = quartic2(pair(0.0f, 0.0f), g.k1, g.k2, g.k3, g.k4, d1, d2, d3, d4);
        at.u = __fadd2_rn(g.start, at.r);
        at.p = __fadd2_rn(pair(static_cast<float>(g.origin_x), static_cast<float>(g.origin_y)),
                          at.u);
    } else {
        at.p = quartic2(g.start, g.k1, g.k2, g.k3, g.k4, d1, d2, d3, d4);
        at.u = at.p;
    }
    // The Newton reciprocal is exact for 2^-64 <= |d| < 2^64 and used only
    // for |d| > 1e-8; march_step replaces the others.
    at.tangent = quartic_tangent2(g.k1, g.k2, g.k3, g.k4, d1, d2, d3);
    at.minus_inv = newton_minus_reciprocal_pair(at.tangent);
    return at;
}

// Far-field culls settled without the reference's full step.
//
// Nine steps in ten of a ray are one culled visit beyond 500 m.  Such a step
// needs exactly only what moves the ray (position, tangent reciprocals, cell
// exit); the chord distance, the level and the bound's slope feed comparisons,
// so a bound on their error may decide those.  With d the distance at the
// cell's near side, dh = h - observer_z, E = 2 (R + observer_z) and sin the
// sine of the running maximum's elevation, the reference's
//   (dh (2R + h + observer_z) - d^2) / E / local_x <= current
// is, local_x being sqrt(d^2 - local_z^2),
//   dh (E + dh) <= d (d + E sin):
// no division, no root.  The margins below cover every rounding of both
// sides: the reference's slope is within 7e-7 (|dh| (E + |dh|) + d^2) / E of
// its real value in local z; the approximate d within 2e-6 of the
// reference's (8 roundings each, the chord's higher terms at most a fifth of
// the linear one: see far_range), so with dn >= true_m / 2 the right side
// moves by at most 4e-6 d (2d + E |sin|).
//
// The exit: the edges ahead are chosen by the signs of the tangent that the
// last full step saw (`ahead`).  A wrong sign makes that axis' exit negative
// or -0, and the step is not settled; +0 is a position on the edge itself,
// which advances by the fallback.  A component within 1e-8 of zero, for which
// the reference takes the reciprocal 1e30, is not settled either; at exactly
// zero its exit is NaN, which the minimum drops as it would 1e30 pixels.
//
// A step that is not settled here (the bound too high or too close to tell,
// another level, a wrong sign) goes to level0_step or the reference's step.
// Half of the values sit in shared memory (RayStore) and are loaded at each
// step: four 16-byte loads cost less than the resident warps that their
// registers would.
struct FarRay {
    float end;            // s below which steps may settle (km; -inf: none)
    float height_base;    // observer_z lowered by 5e-6 (32768 + |observer_z|)
    float double_radius;  // E, raised by 4e-6
    float sine;           // E sin, lowered by 8e-6; -inf when nothing culls
};
// Of the level of the previous step:
struct FarLevel {
    float chord_base;  // start chord (m) less the cell's side (m)
    float low, high;   // dn range over which the level stays the reference's
    float fallback;    // the level's advance when no edge lies ahead (km)
};
struct FarCell {
    float rounder;       // 2^23 4^level: adding it rounds down to a cell edge
    float2 ahead;        // 4^level - rounder where the tangent rises, else -rounder
    unsigned row, base;  // index = bits(rounded y) * row + bits(rounded x) + base
};

// Per-ray values outside the registers, one column per thread of a 128-thread
// block.  Volatile accesses: the compiler must not carry them in registers.
struct RayStore {
    static constexpr int kQuads = 2;
    enum Field { kCurrent, kSideUp, kSideHere, kLevel, kEnd, kChord, kObserver, kLimit, kFields };
    struct Block {
        float4 quads[kQuads][128];
        float fields[kFields][128];
    };
    unsigned quad;           // shared address of the thread's first quad
    volatile float *column;  // the thread's first field
    __device__ __forceinline__ explicit RayStore(Block &block)
        : quad(static_cast<unsigned>(__cvta_generic_to_shared(&block.quads[0][threadIdx.x]))),
          column(&block.fields[0][threadIdx.x]) {}
    __device__ __forceinline__ float get(Field f) const { return column[f * 128]; }
    __device__ __forceinline__ void set(Field f, float v) const { column[f * 128] = v; }
    __device__ __forceinline__ float4 load(int i) const {
        float4 v;
        asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];"
                     : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w)
                     : "r"(quad + i * 2048u) : "memory");
        return v;
    }
    __device__ __forceinline__ void save(int i, float x, float y, float z, float w) const {
        asm volatile("st.shared.v4.f32 [%0], {%1, %2, %3, %4};"
                     :: "r"(quad + i * 2048u), "f"(x), "f"(y), "f"(z), "f"(w) : "memory");
    }
    __device__ __forceinline__ FarRay ray() const {
        const float4 v = load(0);
        return FarRay{v.x, v.y, v.z, v.w};
    }
    __device__ __forceinline__ FarLevel level() const {
        const float4 v = load(1);
        return FarLevel{v.x, v.y, v.z, v.w};
    }
};

__device__ __forceinline__ float far_sine(float observer_radius, float current) {
    const float slope = fminf(current, 1e4f);
    const float scaled = 2.0f * observer_radius * (slope * rsqrtf(1.0f + slope * slope));
    // Nothing settles before the first sample.  A steep maximum needs no
    // limit: with the sine lowered by 8e-6 the slopes that settle stay below
    // 400, where local_x^2 is still 20 times its rounding.
    return current >= -30.0f ? scaled - 8e-6f * fabsf(scaled) : -INFINITY;
}

// The values of `level`, and the edges ahead for a tangent.
template <class Table>
__device__ __forceinline__ void far_level(FarCell &far, const RayStore &store, const Table &table,
                                          const DemView &dem, float start_chord_km, int level) {
    const int4 cells = table.cells(level);
    far.rounder = power_of_two(2 * level + 23);
    const unsigned bits = __float_as_uint(far.rounder);
    far.row = static_cast<unsigned>(cells.y);
    far.base = static_cast<unsigned>(cells.x) - bits * (far.row + 1u);
    const float side = power_of_two(2 * level) * dem.resolution;
    // side <= footprint(true_m) < side above, footprint = true_m * 0.25 deg.
    constexpr float kReach = 229.1831180523293f;
    const float least = level > 0 ? table.side(level) * kReach * 1.00001f : 0.0f;
    store.save(1, start_chord_km * 1000.0f - side, fmaxf(least, 2.0f * side + 2.0f) - side,
               level < dem.level_count - 1 ? table.side(level + 1) * kReach * 0.99999f - side
                                           : INFINITY,
               __int_as_float(cells.w));
}

__device__ __forceinline__ void far_ahead(FarCell &far, float2 tangent) {
    const float cell = far.rounder * 0x1p-23f;
    far.ahead = pair((tangent.x < -1e-8f ? 0.0f : cell) - far.rounder,
                     (tangent.y < -1e-8f ? 0.0f : cell) - far.rounder);
}

// The s range in which steps may settle.  The segment must keep the
// approximations' error bounds (finite, of ordinary size, starting at or
// after the observer: march_near bounds the tangent from there; the chord
// polynomial's higher terms within a fifth of its linear one, the path
// bounded by its coefficients), the DEM must be small enough for exact float
// cell edges, and the path must stay inside the DEM by more than its
// rounding: the Bernstein coefficients of the quartic over the range enclose
// it.  A segment usually ends at the DEM's edge, so the range stops 1/256
// short of it, or 1/16 where the path leaves at a shallow angle; a path that
// hugs an edge gets an empty range.
struct FarRange {
    bool tame;  // the error bounds hold on the whole segment
    float end;  // steps may settle from 500 m up to here (km; -inf: none)
};

__device__ __forceinline__ float path_reach(const RaySegment &g) {
    const float span = g.s_end - g.s_start;
    return span * (fabsf(g.k1.x) + fabsf(g.k1.y) +
                   span * (fabsf(g.k2.x) + fabsf(g.k2.y) +
                           span * (fabsf(g.k3.x) + fabsf(g.k3.y) +
                                   span * (fabsf(g.k4.x) + fabsf(g.k4.y)))));
}

__device__ __forceinline__ bool far_tame(const DemView &dem, const RaySegment &g,
                                         float observer_z) {
    const float reach = path_reach(g);
    const float planar = reach * dem.resolution * 1.0001f;
    return g.s_start >= 0.0f && g.s_end - g.s_start >= 1e-3f && reach < 4e6f &&
           fabsf(g.start.x) < 4e6f && fabsf(g.start.y) < 4e6f && g.s_start_chord >= 0.0f &&
           g.s_start_chord < 1e6f && g.c1 >= 0.1f && g.c1 <= 10.0f &&
           planar * (fabsf(g.c2) + planar * fabsf(g.c3)) <= 0.2f * g.c1 &&
           dem.width <= (1 << 22) && dem.height <= (1 << 22) && fabsf(observer_z) < 1e6f &&
           dem.radius > 1e5f && dem.radius < 1e9f;
}

__device__ __forceinline__ FarRange far_range(const DemView &dem, const RaySegment &g,
                                              float observer_z) {
    const float span = g.s_end - g.s_start, reach = path_reach(g);
    const bool tame = far_tame(dem, g, observer_z);
    const float a = fmaxf(0.5f - g.s_start, 0.0f);
    const float2 a2 = pair(a, a);
    const float2 t0 = __ffma2_rn(a2, __ffma2_rn(a2, __ffma2_rn(a2, __ffma2_rn(a2, g.k4, g.k3),
                                                               g.k2), g.k1), g.start);
    // Derivatives at `a` over 1!, 2! and 3!.
    const float2 p3 = __fmul2_rn(pair(3.0f, 3.0f), g.k3), p4 = __fmul2_rn(a2, g.k4);
    const float2 d1 = __ffma2_rn(a2, __ffma2_rn(a2, __ffma2_rn(pair(4.0f, 4.0f), p4, p3),
                                                __fadd2_rn(g.k2, g.k2)), g.k1);
    const float2 d2 = __ffma2_rn(a2, __ffma2_rn(pair(6.0f, 6.0f), p4, p3), g.k2);
    const float2 d3 = __ffma2_rn(pair(4.0f, 4.0f), p4, g.k3);
    const float margin = 1.0f + 1e-5f * (reach + fabsf(g.start.x) + fabsf(g.start.y));
    FarRange range{tame, -INFINITY};
    if (!tame) return range;
    for (float part = 0.00390625f; part < 0.5f; part *= 16.0f) {
        const float w = (span - a) * (1.0f - part);
        if (!(w > 0.0f)) break;
        const float2 w2 = pair(w, w), w3 = pair(w * w, w * w);
        const float2 t1 = __fmul2_rn(w2, d1), t2 = __fmul2_rn(w3, d2);
        const float2 t3 = __fmul2_rn(__fmul2_rn(w3, w2), d3);
        const float2 t4 = __fmul2_rn(__fmul2_rn(w3, w3), g.k4);
        const float2 b1 = __ffma2_rn(pair(0.25f, 0.25f), t1, t0);
        const float2 b2 = __ffma2_rn(pair(1.0f / 6, 1.0f / 6), t2,
                                     __ffma2_rn(pair(0.5f, 0.5f), t1, t0));
        const float2 b3 = __ffma2_rn(pair(0.25f, 0.25f), t3,
                                     __ffma2_rn(pair(0.5f, 0.5f), t2,
                                                __ffma2_rn(pair(0.75f, 0.75f), t1, t0)));
        const float2 b4 = __fadd2_rn(__fadd2_rn(__fadd2_rn(t0, t1), __fadd2_rn(t2, t3)), t4);
        const float least_x = fminf(fminf(fminf(t0.x, b1.x), fminf(b2.x, b3.x)), b4.x);
        const float least_y = fminf(fminf(fminf(t0.y, b1.y), fminf(b2.y, b3.y)), b4.y);
        const float most_x = fmaxf(fmaxf(fmaxf(t0.x, b1.x), fmaxf(b2.x, b3.x)), b4.x);
        const float most_y = fmaxf(fmaxf(fmaxf(t0.y, b1.y), fmaxf(b2.y, b3.y)), b4.y);
        if (least_x > margin && least_y > margin &&
            most_x < static_cast<float>(dem.width - 1) - margin &&
            most_y < static_cast<float>(dem.height - 1) - margin) {
            range.end = fminf(g.s_start + a + w, g.s_end);
            break;
        }
    }
    return range;
}

// The step from path position `s` at DEM position `p`: true when it is a
// cull that could be settled; `s` then is the next path position.
__device__ __forceinline__ bool far_step(const FarCell &far, const RayStore &store,
                                         const DemView &dem, const RaySegment &g, float2 p,
                                         float2 minus_inv, float &s) {
    const FarRay ray = store.ray();
    const bool in = s < ray.end;
    const float2 down = add2_down(p, pair(far.rounder, far.rounder));
    const unsigned index =
        __float_as_uint(down.y) * far.row + __float_as_uint(down.x) + far.base;
    float height = INFINITY;  // settles nothing
    if (in) height = __ldg(dem.bounds + static_cast<int>(index));
    const FarLevel at = store.level();
    const float2 r = sub2(p, g.start);
    const float planar = sqrt_approx(__fmaf_rn(r.x, r.x, r.y * r.y)) * dem.resolution;
    const float dn = __fmaf_rn(
        planar, __fmaf_rn(planar, __fmaf_rn(planar, g.c3, g.c2), g.c1), at.chord_base);
    // down + (4^level - rounder) and down - rounder are exact.
    const float2 exits = __fmul2_rn(sub2(p, __fadd2_rn(down, far.ahead)), minus_inv);
    const float exit = fminf(exits.x, exits.y);
    const float dh = height - ray.height_base;
    const float left = dh * (dh + ray.double_radius);
    const float right = dn * __fmaf_rn(dn, 0.999988f, ray.sine);
    const float next = __fadd_rn(s, __fadd_rn(exit > 0.0f ? exit : at.fallback, 0.0001f));
    const bool settled = left < right && dn > at.low && dn < at.high &&
                         __float_as_int(exit) >= 0 &&
                         fmaxf(fabsf(minus_inv.x), fabsf(minus_inv.y)) < 9e7f;
    if (settled) s = next;
    return settled;
}

// x / 1000 correctly rounded (for normal x and quotient): a faithful quotient
// corrected by its exact residual (Markstein, as rcp_approx).  Equal to the IEEE
// division on every pattern from 2^-64 to 2^64 (ls200_check_arithmetic).  Its
// operand is a path advance (m): 0 or at most a few kilometres, and a value too
// small for the check loses to the floor step.
__device__ __forceinline__ float over_1000(float x) {
    const float q = __fmul_rn(x, 0.001f);
    return __fmaf_rn(__fmaf_rn(-1000.0f, q, x), 0.001f, q);
}

// The chord distance of a far-field position in the reference's rounding.
__device__ __forceinline__ float chord_distance_m(const RaySegment &g, float2 r,
                                                  float resolution) {
    const float2 planar = __fmul2_rn(r, pair(resolution, resolution));
    const float planar_m = hypot_fused(planar.x, planar.y);
    const float pm2 = __fmul_rn(planar_m, planar_m);
    // (c2 * pm2, pm2 * planar_m) in one instruction.
    const float2 terms = __fmul2_rn(pair(g.c2, pm2), pair(pm2, planar_m));
    float chord = __fmaf_rn(g.c1, planar_m, terms.x);
    chord = __fmaf_rn(g.c3, terms.y, chord);
    return __fmaf_rn(g.s_start_chord, 1000.0f, chord);
}

// The level-0 sample of a step, in the reference's arithmetic: its slope, the
// running maximum and the advance.  q.. are the cell's corners, `corner` its
// integer position; which of pixel, angular and floor step is the largest is
// decided by a bound where that is clear.
template <class Tracker>
__device__ __forceinline__ void sample_step(const DemView &dem, int pass_index, float observer_z,
                                            float observer_radius, bool near, float2 p,
                                            float2 corner, float2 tangent, float true_m,
                                            float q00, float q10, float q01, float q11,
                                            MarchState &st, Tracker &tracker) {
    const float current = st.current, resolution = dem.resolution;
    const bool valid = q00 > -20000.0f && q10 > -20000.0f && q01 > -20000.0f && q11 > -20000.0f;
    const float2 t = sub2(p, corner);
    const float top = __fmaf_rn(t.x, __fsub_rn(q10, q00), q00);
    const float bottom = __fmaf_rn(t.x, __fsub_rn(q11, q01), q01);
    const float height = __fmaf_rn(t.y, __fsub_rn(bottom, top), top);
    float slope = -1e30f;
    if (valid) {
        slope = near ? __fdiv_rn(__fsub_rn(height, observer_z), true_m)
                     : sample_slope(true_m, height, dem.radius, observer_radius);
        if (slope > current) {
            st.current = slope;
            tracker.record(p.x, p.y, true_m, slope, near);
        }
    }
    // The smaller of the margin's and the angular product, over 1000 (see
    // march_step).
    const float angular = __fmul_rn(true_m, 0.00151f);
    const float margin = __fsub_rn(st.current, slope);
    float product = 0.0f;
    if (margin > 0.0f) {
        const float margin_product = __fmul_rn(__fmul_rn(margin, true_m), 1.732f);
        product = margin_product < angular ? margin_product : angular;
    }
    const float floor_step = pass_index == 0 && true_m >= 100.0f
                                 ? __fmul_rn(__fmul_rn(0.8f, resolution), 0.001f)
                                 : __fmul_rn(__fmul_rn(0.5f, resolution), 0.001f);
    const float scale = near ? 0.25f : 1.0f;
    float advance = over_1000(product);
    const float squared = tangent.x * tangent.x + tangent.y * tangent.y;
    const float pixel_most = rsqrtf(squared) * 1.00001f;
    if (!(squared > 1e-11f) ||
        !(advance > pixel_most || pixel_most * scale < floor_step * 0.99999f)) {
        const float magnitude = hypot_fused(tangent.x, tangent.y);
        const float pixel_step = magnitude > 1e-6f ? __frcp_rn(magnitude) : 0.0005f;
        advance = pixel_step > advance ? pixel_step : advance;
    }
    advance = __fmul_rn(advance, scale);
    advance = advance > floor_step ? advance : floor_step;
    st.s = __fadd_rn(st.s, advance);
}

// One step at level 0 in the reference's arithmetic, for the rays far_range
// found tame and positions whose clamps do not act: most steps that far_step
// leaves over.  Returns false, having done nothing, when the step is another
// one.  The cull (one product per side) and which
// of pixel, angular and floor step is the largest are again decided by a
// bound on the error where that is clear.
template <bool kCount, bool kAhead, class Table, class Tracker>
__device__ __forceinline__ bool level0_step(const Table &table, const DemView &dem,
                                            const RaySegment &g, const StepPoint &at,
                                            int pass_index, float observer_z, MarchState &st,
                                            unsigned &samples, Tracker &tracker) {
    const float2 p = at.p, tangent = at.tangent, minus_inv = at.minus_inv;
    const float s = st.s, current = st.current;
    const float resolution = dem.resolution;
    const float xmax = fminf(static_cast<float>(dem.width) - 1.0001f,
                             static_cast<float>(dem.width - 1) - 0.5f);
    const float ymax = fminf(static_cast<float>(dem.height) - 1.0001f,
                             static_cast<float>(dem.height - 1) - 0.5f);
    if (!(st.level_hint == 0 && p.x >= 0.0f && p.y >= 0.0f && p.x < xmax &&
          p.y < ymax && fabsf(tangent.x) > 1e-8f && fabsf(tangent.y) > 1e-8f))
        return false;
    const bool near = s < 0.5f;
    const float true_m =
        near ? __fmul_rn(s, 1000.0f) : chord_distance_m(g, sub2(p, g.start), resolution);
    if (st.side_up <= __fmul_rn(true_m, 0.004363323129985824f)) return false;
    const float2 down = add2_down(p, pair(0x1p23f, 0x1p23f));
    const float2 corner = __fadd2_rn(down, pair(-0x1p23f, -0x1p23f));
    const int index = (__float_as_int(down.y) - 0x4b000000) * dem.width +
                      (__float_as_int(down.x) - 0x4b000000);
    // kAhead: the corners are loaded along with the bound, before it is known
    // whether they are needed: one memory latency per step instead of two.
    const float *r0 = dem.cells + index, *r1 = r0 + dem.width;
    float q00, q10, q01, q11;
    if (kAhead) {
        q00 = __ldg(r0), q10 = __ldg(r0 + 1);
        q01 = __ldg(r1), q11 = __ldg(r1 + 1);
    }
    const float maximum_height = __ldg(dem.bounds + index);
    const float observer_radius = __fadd_rn(dem.radius, observer_z);
    const float denominator = __fmul_rn(2.0f, observer_radius);
    bool culled = maximum_height < -20000.0f;
    if (!culled) {
        float true_near = __fsub_rn(true_m, resolution);
        true_near = true_near > 1.0f ? true_near : 1.0f;
        const float dh = __fsub_rn(maximum_height, observer_z);
        float left, right, band;
        if (near) {
            left = dh;
            right = current * true_near;
            band = 1e-5f * fabsf(right) + 1e-30f;
        } else {
            const float sine = denominator * (current * rsqrtf(1.0f + current * current));
            left = dh * (denominator + dh);
            right = true_near * (true_near + sine);
            band = 2e-5f * (fabsf(left) + true_near * (true_near + fabsf(sine)));
            if (!(fabsf(current) <= 30.0f)) band = INFINITY;
        }
        culled = left < right - band;
        if (!culled && !(left > right + band)) {
            const float possible =
                near ? __fdiv_rn(dh, true_near)
                     : bound_slope(true_near, maximum_height, dem.radius, observer_z,
                                   observer_radius);
            culled = possible <= current;
        }
    }
    if (culled) {
        const float2 edge = __fadd2_rn(corner, pair(tangent.x > 0.0f ? 1.0f : 0.0f,
                                                    tangent.y > 0.0f ? 1.0f : 0.0f));
        const float2 exits = __fmul2_rn(sub2(p, edge), minus_inv);
        const float exit = fminf(exits.x, exits.y);
        st.s = __fadd_rn(s, __fadd_rn(exit > 0.0f ? exit : table.fallback(0), 0.0001f));
        return true;
    }
    if (kCount) ++samples;
    if (!kAhead) {
        q00 = __ldg(r0), q10 = __ldg(r0 + 1);
        q01 = __ldg(r1), q11 = __ldg(r1 + 1);
    }
    sample_step(dem, pass_index, observer_z, observer_radius, near, p, corner, tangent, true_m,
                q00, q10, q01, q11, st, tracker);
    return true;
}

// The sample of a far step at level 0 that is known not to be culled.  Returns
// false, having done nothing, where the bilinear clamps may act.
template <bool kCount, class Tracker>
__device__ __forceinline__ bool far_sample_step(const DemView &dem, const RaySegment &g,
                                                const StepPoint &at, int pass_index,
                                                float observer_z, MarchState &st,
                                                unsigned &samples, Tracker &tracker) {
    const float2 p = at.p;
    const float xmax = fminf(static_cast<float>(dem.width) - 1.0001f,
                             static_cast<float>(dem.width - 1) - 0.5f);
    const float ymax = fminf(static_cast<float>(dem.height) - 1.0001f,
                             static_cast<float>(dem.height - 1) - 0.5f);
    if (!(p.x < xmax && p.y < ymax)) return false;
    const float2 down = add2_down(p, pair(0x1p23f, 0x1p23f));
    const float2 corner = __fadd2_rn(down, pair(-0x1p23f, -0x1p23f));
    const int index = (__float_as_int(down.y) - 0x4b000000) * dem.width +
                      (__float_as_int(down.x) - 0x4b000000);
    const float *r0 = dem.cells + index, *r1 = r0 + dem.width;
    const float q00 = __ldg(r0), q10 = __ldg(r0 + 1);
    const float q01 = __ldg(r1), q11 = __ldg(r1 + 1);
    if (kCount) ++samples;
    sample_step(dem, pass_index, observer_z, __fadd_rn(dem.radius, observer_z), false, p, corner,
                at.tangent, chord_distance_m(g, sub2(p, g.start), dem.resolution), q00, q10, q01,
                q11, st, tracker);
    return true;
}

// One outer iteration of hierarchy_maximum (cuda_backend.py:672-867) at a
// position s <= s_end: the level descent (and with the ladder the climb) and
// the advance.  Returns false, leaving `st` untouched, when the pass is over
// (outside the DEM, or the cell left the level grid).
template <bool kCount, int kLadder, class Table, class Tracker>
__device__ __forceinline__ bool march_step(const Table &table, const DemView &dem,
                                           const RaySegment &g, const StepPoint &at,
                                           int pass_index, float observer_z, MarchState &st,
                                           unsigned &visits, unsigned &samples,
                                           unsigned &steps, Tracker &tracker) {
    const float radius = dem.radius;
    const float resolution = dem.resolution;
    const float observer_radius = __fadd_rn(radius, observer_z);
    const float inverse_denominator = __frcp_rn(__fmul_rn(2.0f, observer_radius));
    const float *__restrict__ cells = dem.cells;
    const float minimum_step = __fmul_rn(__fmul_rn(0.5f, resolution), 0.001f);
    const float primary_far_step = __fmul_rn(__fmul_rn(0.8f, resolution), 0.001f);
    const float last_x = static_cast<float>(dem.width - 1);
    const float last_y = static_cast<float>(dem.height - 1);
    const int top_level = dem.level_count - 1;
    float s = st.s;
    float current = st.current;
    int level_hint = st.level_hint;
    float side_up = st.side_up, side_here = st.side_here;
    constexpr bool relative = (kLadder & kRelative) != 0;
    {
        if (kCount) ++steps;
        const float2 u = at.u, p = at.p;
        const float dx = at.tangent.x, dy = at.tangent.y;
        float2 minus_inv = at.minus_inv;
        const float ax = fabsf(dx), ay = fabsf(dy);
        if (!(ax > 1e-8f)) minus_inv.x = -1e30f;
        if (!(ay > 1e-8f)) minus_inv.y = -1e30f;
        if (!(ax < 0x1p64f && ay < 0x1p64f)) {
            minus_inv.x = ax > 1e-8f ? -__frcp_rn(dx) : -1e30f;
            minus_inv.y = ay > 1e-8f ? -__frcp_rn(dy) : -1e30f;
        }
        const float ux = u.x, uy = u.y, px = p.x, py = p.y;
        // NaN fails every comparison, as the reference's isnan tests do.
        if (!(px >= 0.0f && py >= 0.0f && px < last_x && py < last_y)) return false;
        const bool near = s < 0.5f;
        float true_m;
        if (near) {
            true_m = __fmul_rn(s, 1000.0f);
        } else {
            // The planar distance only feeds the far-field chord.
            true_m = chord_distance_m(g, relative ? at.r : sub2(p, g.start), resolution);
        }
        const float footprint = __fmul_rn(true_m, 0.004363323129985824f);
        // The reference scans down from the top level to the largest level
        // whose side fits the footprint (or 0).  Sides grow with the level,
        // so that level is also found by moving up or down from the previous
        // step's level, which usually takes one comparison.
        // The two sides around the previous level sit in registers, so the
        // usual step decides with two comparisons and no table read.
        int level = level_hint;
        if (side_up <= footprint || !(side_here <= footprint)) {
            while (level < top_level && table.side(level + 1) <= footprint) ++level;
            while (level > 0 && !(table.side(level) <= footprint)) --level;
            level_hint = level;
            side_up = level < top_level ? table.side(level + 1) : __int_as_float(0x7fffffff);
            side_here = level > 0 ? table.side(level) : -INFINITY;
        }
        const int origin_x = relative ? g.origin_x : 0;
        const int origin_y = relative ? g.origin_y : 0;
        const int ipx = relative ? origin_x + static_cast<int>(floorf(ux)) : static_cast<int>(px);
        const int ipy = relative ? origin_y + static_cast<int>(floorf(uy)) : static_cast<int>(py);
        bool ray_out = false;
        for (;;) {
            const int4 L = table.cells(level);
            const int shift = level * 2;
            const int cx = ipx >> shift, cy = ipy >> shift;
            if (kCount) ++visits;
            if (cx >= L.y || cy >= L.z) {  // cx, cy >= 0 since px, py >= 0
                s = __fadd_rn(s, table.out_step(level));
                ray_out = true;
                break;
            }
            const float maximum_height = cell_bound(dem.bounds, L, cx, cy);
            const float skip = cell_exit_advance(shift, cx, cy, ux, uy, origin_x, origin_y, minus_inv,
                                                 __int_as_float(L.w));
            bool culled = maximum_height < -20000.0f;
            if (!culled) {
                const float scale_f = power_of_two(shift);
                float true_near = __fmaf_rn(-scale_f, resolution, true_m);
                true_near = true_near > 1.0f ? true_near : 1.0f;
                culled = bound_culled(near, true_near, maximum_height, radius, observer_z,
                                      observer_radius, inverse_denominator, current);
            }
            if (culled) {
                float advance = skip;
                if (kLadder & kLadderClimb) {
                    int reached;
                    advance = ladder_advance<kCount>(table, dem.bounds, level, top_level, ipx, ipy,
                                                     ux, uy, origin_x, origin_y, minus_inv,
                                                     near, true_m, radius, observer_z,
                                                     observer_radius, inverse_denominator,
                                                     current, skip, visits, reached);
                }
                s = __fadd_rn(s, advance);
                break;
            }
            if (level == 0) {
                if (kCount) ++samples;
                float slope = -1e30f;
                if (relative) {
                    float above;
                    if (bilinear_above(cells, dem.width, dem.height, origin_x, ux, px, origin_y,
                                       uy, py, observer_z, above)) {
                        slope = near ? __fdiv_rn(above, true_m)
                                     : above_slope(true_m, above, radius, observer_z,
                                                   observer_radius);
                        if (slope > current) {
                            current = slope;
                            tracker.record(px, py, true_m, slope, near);
                        }
                    }
                } else {
                    const float height = bilinear(cells, dem.width, dem.height, px, py);
                    if (height > -20000.0f) {
                        slope = near ? __fdiv_rn(__fsub_rn(height, observer_z), true_m)
                                     : sample_slope(true_m, height, radius, observer_radius);
                        if (slope > current) {
                            current = slope;
                            tracker.record(px, py, true_m, slope, near);
                        }
                    }
                }
                const float magnitude = hypot_fused(dx, dy);
                const float pixel_step = magnitude > 1e-6f ? __frcp_rn(magnitude) : 0.0005f;
                // inner = min(margin_step, angular_step), both a product
                // divided by 1000 (the margin one 0 unless margin > 0).  A
                // correctly rounded division by a positive constant is
                // monotone, so the smaller quotient is the quotient of the
                // smaller product: one division gives the same value.
                const float margin = __fsub_rn(current, slope);
                const float angular_product = __fmul_rn(true_m, 0.00151f);
                float inner = 0.0f;
                if (margin > 0.0f) {
                    const float margin_product = __fmul_rn(__fmul_rn(margin, true_m), 1.732f);
                    inner = __fdiv_rn(margin_product < angular_product ? margin_product
                                                                       : angular_product,
                                      1000.0f);
                }
                float advance = pixel_step > inner ? pixel_step : inner;
                if (near) advance = __fmul_rn(advance, 0.25f);
                const float floor_step =
                    (pass_index == 0 && true_m >= 100.0f) ? primary_far_step : minimum_step;
                advance = advance > floor_step ? advance : floor_step;
                s = __fadd_rn(s, advance);
                break;
            }
            --level;
        }
        if (ray_out) return false;
    }
    st.s = s;
    st.current = current;
    st.level_hint = level_hint;
    st.side_up = side_up;
    st.side_here = side_here;
    return true;
}

// hierarchy_maximum (cuda_backend.py:656-874): the maximum slope along one
// ray over one DEM, starting from `current` (-1e30 for none).  Table gives
// side(l), fallback(l), out_step(l) and cells(l).
template <bool kCount, int kLadder, class Table, class Tracker>
__device__ __forceinline__ float march_dem_tracked(const Table &table, const DemView &dem,
                                                   const RaySegment &g, int pass_index,
                                                   float observer_z, float current,
                                                   unsigned &visits, unsigned &samples,
                                                   unsigned &steps, Tracker &tracker) {
    MarchState st = begin_pass(dem, g, current);
    while (st.s <= g.s_end &&
           march_step<kCount, kLadder>(table, dem, g,
                                       step_point<(kLadder & kRelative) != 0>(g, st.s),
                                       pass_index, observer_z, st, visits, samples, steps,
                                       tracker)) {
    }
    return st.current;
}

// The near field (the first 500 m) of one ray: at level 0 throughout, and its
// samples advance by the floor step whatever the slope, because a quarter of a
// pixel's step and of the angular step stay below it (checked for the segment).
// So a sample needs its slope only when it may raise the maximum, and a step
// needs the tangent only when its cell is culled: 60 instructions where
// level0_step takes 200 (a site-scale tile 183 -> 174.5 ms, a preview tile of
// 5 km rays 265 -> 255 us).  A ray meets a step it does not cover (the DEM's edge,
// an axis-parallel exit) by leaving; the caller's loop goes on from there.
// Returns the path position reached; every lane of the warp calls it.
template <bool kCount, class Table, class Tracker>
__device__ __forceinline__ float march_near(const Table &table, const DemView &dem,
                                            const RaySegment &g, bool tame, int pass_index,
                                            float observer_z, float s, float &current,
                                            unsigned &visits, unsigned &samples,
                                            unsigned &steps, Tracker &tracker) {
    const float resolution = dem.resolution;
    const float floor_step = __fmul_rn(__fmul_rn(0.5f, resolution), 0.001f);
    const float far_floor = pass_index == 0
                                ? __fmul_rn(__fmul_rn(0.8f, resolution), 0.001f) : floor_step;
    // The tangent's least length over the near field, in pixels per km.
    const float bend = (fabsf(g.k2.x) + fabsf(g.k2.y)) +
                       0.75f * (fabsf(g.k3.x) + fabsf(g.k3.y)) +
                       0.5f * (fabsf(g.k4.x) + fabsf(g.k4.y));
    const float least = 0.9999f * sqrt_approx(g.k1.x * g.k1.x + g.k1.y * g.k1.y) - bend;
    const bool covered = tame && least * floor_step > 0.2501f && floor_step > 1.89e-4f &&
                         (dem.level_count < 2 || table.side(1) > 2.2f);
    const float xmax = fminf(static_cast<float>(dem.width) - 1.0001f,
                             static_cast<float>(dem.width - 1) - 0.5f);
    const float ymax = fminf(static_cast<float>(dem.height) - 1.0001f,
                             static_cast<float>(dem.height - 1) - 0.5f);
    bool live = covered && s < 0.5f && s <= g.s_end;
    while (__any_sync(0xffffffffu, live)) {
        if (live) {
            const float delta = __fsub_rn(s, g.s_start);
            const float2 d1 = pair(delta, delta);
            const float2 d2 = __fmul2_rn(d1, d1);
            const float2 d3 = __fmul2_rn(d2, d1);
            const float2 d4 = __fmul2_rn(d2, d2);
            const float2 p = quartic2(g.start, g.k1, g.k2, g.k3, g.k4, d1, d2, d3, d4);
            live = p.x >= 0.0f && p.y >= 0.0f && p.x < xmax && p.y < ymax;
            if (live) {
                const float true_m = __fmul_rn(s, 1000.0f);
                const float2 down = add2_down(p, pair(0x1p23f, 0x1p23f));
                const float2 corner = __fadd2_rn(down, pair(-0x1p23f, -0x1p23f));
                const int index = (__float_as_int(down.y) - 0x4b000000) * dem.width +
                                  (__float_as_int(down.x) - 0x4b000000);
                const float *r0 = dem.cells + index, *r1 = r0 + dem.width;
                const float maximum_height = __ldg(dem.bounds + index);
                const float q00 = __ldg(r0), q10 = __ldg(r0 + 1);
                const float q01 = __ldg(r1), q11 = __ldg(r1 + 1);
                const float dh = __fsub_rn(maximum_height, observer_z);
                float true_near = __fsub_rn(true_m, resolution);
                true_near = true_near > 1.0f ? true_near : 1.0f;
                const float limit = current * true_near;
                const float band = 1e-5f * fabsf(limit) + 1e-30f;
                bool culled = maximum_height < -20000.0f || dh < limit - band;
                if (!culled && !(dh > limit + band)) culled = __fdiv_rn(dh, true_near) <= current;
                if (culled) {
                    const float2 tangent = quartic_tangent2(g.k1, g.k2, g.k3, g.k4, d1, d2, d3);
                    if (fabsf(tangent.x) > 1e-8f && fabsf(tangent.y) > 1e-8f) {
                        const float2 edge =
                            __fadd2_rn(corner, pair(tangent.x > 0.0f ? 1.0f : 0.0f,
                                                    tangent.y > 0.0f ? 1.0f : 0.0f));
                        const float2 exits = __fmul2_rn(sub2(p, edge),
                                                        newton_minus_reciprocal_pair(tangent));
                        const float exit = fminf(exits.x, exits.y);
                        s = __fadd_rn(s, __fadd_rn(exit > 0.0f ? exit : table.fallback(0),
                                                   0.0001f));
                        if (kCount) ++steps, ++visits;
                    } else {
                        live = false;
                    }
                } else {
                    if (q00 > -20000.0f && q10 > -20000.0f && q01 > -20000.0f &&
                        q11 > -20000.0f) {
                        const float2 t = sub2(p, corner);
                        const float top = __fmaf_rn(t.x, __fsub_rn(q10, q00), q00);
                        const float bottom = __fmaf_rn(t.x, __fsub_rn(q11, q01), q01);
                        const float height = __fmaf_rn(t.y, __fsub_rn(bottom, top), top);
                        const float rise = __fsub_rn(height, observer_z);
                        const float least_rise = current * true_m;
                        if (!(rise < least_rise - 1e-6f * fabsf(least_rise))) {
                            const float slope = __fdiv_rn(rise, true_m);
                            if (slope > current) {
                                current = slope;
                                tracker.record(p.x, p.y, true_m, slope, true);
                            }
                        }
                    }
                    s = __fadd_rn(s, true_m >= 100.0f ? far_floor : floor_step);
                    if (kCount) ++steps, ++visits, ++samples;
                }
                live = live && s < 0.5f && s <= g.s_end;
            }
        }
    }
    return s;
}

// The last path position of a ray that RayStore holds.  Finite (or NaN): a ray
// that has ended stands at +inf, which must lie past every end, also that of a
// caller's segment without one.
__device__ __forceinline__ float ray_end(const RaySegment &g) {
    constexpr float kLargest = 0x1.fffffep127f;
    return g.s_end > kLargest ? kLargest : g.s_end;
}

// The step of a lane that far_step left over: level0_step or the reference's
// full step, and what they change for the next fast steps.
template <bool kCount, bool kAhead, class Table, class Tracker>
__device__ __forceinline__ void slow_step(FarCell &far, const RayStore &store, const Table &table,
                                          const DemView &dem, const RaySegment &g,
                                          const StepPoint &at, int pass_index, float s_end,
                                          float &s, unsigned &visits, unsigned &samples,
                                          unsigned &steps, Tracker &tracker) {
    RaySegment own = g;
    own.s_end = s_end;
    own.s_start_chord = store.get(RayStore::kChord);
    const float z = store.get(RayStore::kObserver);
    const float limit = store.get(RayStore::kLimit);
    const float before = store.get(RayStore::kCurrent);
    // Clamped: march_step shifts by it and indexes the level table with it.
    const int level = min(max(__float_as_int(store.get(RayStore::kLevel)), 0),
                          dem.level_count - 1);
    MarchState st{s, before, level, store.get(RayStore::kSideUp),
                  store.get(RayStore::kSideHere)};
    bool alive = true;
    if (limit < INFINITY &&
        level0_step<kCount, kAhead>(table, dem, own, at, pass_index, z, st, samples, tracker)) {
        if (kCount) ++steps, ++visits;
    } else {
        alive = march_step<kCount, kReference>(table, dem, own, at, pass_index, z, st, visits,
                                               samples, steps, tracker);
    }
    if (st.level_hint != level) {
        far_level(far, store, table, dem, own.s_start_chord, st.level_hint);
        store.set(RayStore::kLevel, __int_as_float(st.level_hint));
        store.set(RayStore::kSideUp, st.side_up);
        store.set(RayStore::kSideHere, st.side_here);
    }
    far_ahead(far, at.tangent);
    s = alive ? st.s : INFINITY;
    FarRay ray = store.ray();
    ray.end = s >= 0.5f && limit < INFINITY ? limit : -INFINITY;
    if (st.current != before) {
        ray.sine = far_sine(dem.radius + z, st.current);
        store.set(RayStore::kCurrent, st.current);
    }
    store.save(0, ray.end, ray.height_base, ray.double_radius, ray.sine);
}

// The reference traversal with its far-field culls settled by far_step.
// Every lane of the warp calls it; `marches` is false for a lane without a
// ray.  The fast step has no branch; the lanes it leaves over step together.
// The votes also keep the warp together: without one per step the settled
// lanes ran ahead while the others waited (4.3 times slower).
template <bool kCount, bool kAhead, class Table, class Tracker>
__device__ __forceinline__ float march_dem_far(const Table &table, const DemView &dem,
                                               const RaySegment &g, int pass_index,
                                               float observer_z, float current, bool marches,
                                               const RayStore &store, unsigned &visits,
                                               unsigned &samples, unsigned &steps,
                                               Tracker &tracker) {
    const MarchState first = begin_pass(dem, g, current);
    const FarRange range = far_range(dem, g, observer_z);
    // A lane whose ray has ended (or never was) stands at +inf.
    float s = march_near<kCount>(table, dem, g, range.tame, pass_index, observer_z,
                                 marches ? first.s : INFINITY, current, visits, samples, steps,
                                 tracker);
    const float height_base = observer_z - 5e-6f * (32768.0f + fabsf(observer_z));
    const float double_radius = 2.0f * (dem.radius + observer_z) * 1.000004f;
    FarCell far;
    far_level(far, store, table, dem, g.s_start_chord, first.level_hint);
    far_ahead(far, pair(-1.0f, -1.0f));
    store.save(0, s >= 0.5f ? range.end : -INFINITY, height_base, double_radius,
               far_sine(dem.radius + observer_z, current));
    store.set(RayStore::kCurrent, current);
    store.set(RayStore::kSideUp, first.side_up);
    store.set(RayStore::kSideHere, first.side_here);
    store.set(RayStore::kLevel, __int_as_float(first.level_hint));
    store.set(RayStore::kEnd, ray_end(g));
    store.set(RayStore::kChord, g.s_start_chord);
    store.set(RayStore::kObserver, observer_z);
    store.set(RayStore::kLimit, range.tame ? range.end : INFINITY);  // +inf: not tame
    for (;;) {
        const StepPoint at = step_point<false>(g, s);
        const bool settled = far_step(far, store, dem, g, at.p, at.minus_inv, s);
        if (kCount && settled) ++steps, ++visits;
        if (__any_sync(0xffffffffu, !settled)) {
            const float s_end = store.get(RayStore::kEnd);
            if (!settled && s <= s_end)
                slow_step<kCount, kAhead>(far, store, table, dem, g, at, pass_index, s_end, s,
                                          visits, samples, steps, tracker);
            if (!__any_sync(0xffffffffu, s <= s_end)) break;
        }
    }
    return store.get(RayStore::kCurrent);
}

// The skip ladder's steps settled as far_step settles the reference's: a cull
// at the footprint's level and the climb from it (ladder_culled), decided by
// the same comparison of products.  The level comes from the exponent of the
// footprint in cells, since a skip often changes it.  For an ancestor whose
// bound lies above the observer the climb's test is
//   dh (E + dh) <= d (d + E sin)
// at d = true_m, one product and one comparison a level; below the observer it
// is dh <= current * far.  Both decisions of a test must be clear by 3e-5 of
// their terms (the reference's own 4e-6 allowance, 4e-6 d (2d + E |sin|) for the
// approximate d and the roundings of both sides); otherwise the step is not
// settled.  (A maximum beyond 1e4, where the reference's slopes end in its
// 1e-6 m local_x, leaves every bound above it unclear.)  The exit is computed
// once, for the level reached.  It is bound by lanes that differ and by issue:
// 19.2 of 32 lanes active, 165 instructions a lane's step, 77 % of the slots (four
// sites of 512^2 to 1500^2 pixels).  Eight sites 426 -> 390 ms, two of 2048^2
// pixels 71.4 -> 62.7 ms, the checkpointing march of one tile 55.5 -> 49.8 ms.
struct LadderRay {
    float end;            // s up to which steps may settle (km; -inf: none)
    float observer_z;
    float double_radius;  // E
    float sine;           // E sin of the running maximum; -inf when nothing culls
};
struct LadderScale {
    float chord_base;  // start chord (m)
    float footprint;   // cells of level 0 per metre of true_m
    float current;
};

__device__ __forceinline__ float ladder_sine(float observer_radius, float current) {
    const float slope = fminf(current, 1e4f);
    return current >= -30.0f
               ? 2.0f * observer_radius * (slope * rsqrtf(1.0f + slope * slope))
               : -INFINITY;
}

// What ladder_step found: the step is done; the level-0 cell under the ray is
// not culled (a sample follows); neither is clear.
enum LadderFound { kSettled, kSample, kUnclear };

template <bool kCount, class Table>
__device__ __forceinline__ LadderFound ladder_step(const RayStore &store, const Table &table,
                                                   const DemView &dem, const RaySegment &g,
                                                   const StepPoint &at, float &s,
                                                   unsigned &visits) {
    const float4 quad0 = store.load(0), quad1 = store.load(1);
    const LadderRay ray{quad0.x, quad0.y, quad0.z, quad0.w};
    const LadderScale scale{quad1.x, quad1.y, quad1.z};
    const float2 p = at.p;
    const float2 last = table.last();
    if (!(s <= ray.end && p.x >= 0.0f && p.y >= 0.0f && p.x < last.x && p.y < last.y))
        return kUnclear;
    const float2 r = sub2(p, g.start);
    const float planar = sqrt_approx(__fmaf_rn(r.x, r.x, r.y * r.y)) * dem.resolution;
    const float d = __fmaf_rn(
        planar, __fmaf_rn(planar, __fmaf_rn(planar, g.c3, g.c2), g.c1), scale.chord_base);
    // The largest level whose side, 4^level cells, fits the footprint.
    const float cells = d * scale.footprint;
    const int top = dem.level_count - 1;
    int level = min(max(((__float_as_int(cells) >> 23) - 127) >> 1, 0), top);
    const float inside = cells * __int_as_float((127 - 2 * level) << 23);
    const float dn = __fmaf_rn(-power_of_two(2 * level), dem.resolution, d);
    // The level is clear, and so is which side of the ladder's least distance.
    if (!((level == 0 || inside > 1.00001f) && (level == top || inside < 3.99996f) &&
          dn > d * 0.5f && dn > 1.0f && fabsf(d - kLadderMinimumDistance) > 0.02f &&
          fmaxf(fabsf(at.minus_inv.x), fabsf(at.minus_inv.y)) < 9e7f))
        return kUnclear;
    auto height_at = [&](int l) {
        const int4 L = table.cells(l);
        const float rounder = power_of_two(2 * l + 23);
        const unsigned bits = __float_as_uint(rounder);
        const float2 down = add2_down(p, pair(rounder, rounder));
        const unsigned index =
            (__float_as_uint(down.y) - bits) * static_cast<unsigned>(L.y) +
            (__float_as_uint(down.x) - bits) + static_cast<unsigned>(L.x);
        return __ldg(dem.bounds + static_cast<int>(index));
    };
    auto exit_advance = [&](int l) {
        const float rounder = power_of_two(2 * l + 23), side = power_of_two(2 * l);
        const float2 down = add2_down(p, pair(rounder, rounder));
        const float2 edge =
            __fadd2_rn(down, pair((at.tangent.x > 0.0f ? side : 0.0f) - rounder,
                                  (at.tangent.y > 0.0f ? side : 0.0f) - rounder));
        const float2 exits = __fmul2_rn(sub2(p, edge), at.minus_inv);
        const float exit = fminf(exits.x, exits.y);
        return __fadd_rn(exit > 0.0f ? exit : table.fallback(l), 0.0001f);
    };
    {
        const float height = height_at(level);
        const float dh = height - ray.observer_z;
        const float left = dh * (ray.double_radius + dh);
        const float right = dn * (dn + ray.sine);
        const float band = 2e-5f * (fabsf(left) + dn * (dn + fabsf(ray.sine)));
        if (!(height < -20000.0f || left < right - band))
            return level == 0 && left > right + band && scale.current <= 1e4f ? kSample
                                                                              : kUnclear;
    }
    // Climb from level to level while the ancestor's cell is culled.
    if (kCount) ++visits;
    bool clear = true;
    if (d > kLadderMinimumDistance) {
        // dh (E + dh) <= w solved for the height above the observer.
        const float w = d * (d + ray.sine);
        const float root = sqrt_approx(
            __fmaf_rn(ray.double_radius, ray.double_radius, fmaxf(4.0f * w, 0.0f)));
        const float inverse = rcp_approx(ray.double_radius + root);
        const float height_limit = 2.0f * w * inverse;
        const float height_band =
            6e-5f * __fmaf_rn(d * (d + fabsf(ray.sine)), inverse, fabsf(height_limit));
        const float above_low = height_limit - height_band;
        const float above_high =
            scale.current <= 1e4f ? height_limit + height_band : INFINITY;
        // Below the observer: dh against current * far.  far lies between d and
        // the furthest exit's, a side along the faster axis (or the fallback,
        // half a side); a maximum above the horizontal culls every such cell.
        const float falling = fminf(scale.current, 0.0f);
        float side = power_of_two(2 * level);
        const float across = fmaxf(fminf(fabsf(at.minus_inv.x), fabsf(at.minus_inv.y)),
                                   5.1e-4f * dem.resolution) * 1010.1f * falling;
        const float below_base = __fmaf_rn(falling, d, 3.0f * falling) * 1.00006f;
        const float below_high = falling < 0.0f ? falling * d * 0.99994f + 1e-3f : INFINITY;
        while (level < top) {
            if (kCount) ++visits;
            side *= 4.0f;
            const float height = height_at(level + 1);
            const float dh = height - ray.observer_z;
            const bool above = dh >= 0.0f;
            const float below_low =
                falling < 0.0f ? __fmaf_rn(across, side, below_base) - 1e-3f : INFINITY;
            bool culled = dh < (above ? above_low : below_low) || height < -20000.0f;
            if (!culled && !(dh > (above ? above_high : below_high))) {
                // Between the limits: below the observer the exit decides.
                clear = false;
                if (!above) {
                    const float limit =
                        scale.current *
                        (__fmaf_rn(exit_advance(level + 1), 1010.0f, d) + 1.0f);
                    const float band = 3e-5f * (fabsf(dh) + fabsf(limit)) + 1e-30f;
                    culled = dh < limit - band;
                    clear = culled || dh > limit + band;
                }
            }
            if (!culled) break;
            ++level;
        }
    }
    if (!clear) return kUnclear;
    s = __fadd_rn(s, exit_advance(level));
    return kSettled;
}

// The skip ladder with its culls settled by ladder_step (as march_dem_far).
template <bool kCount, class Table, class Tracker>
__device__ __forceinline__ float march_dem_ladder(const Table &table, const DemView &dem,
                                                  const RaySegment &g, int pass_index,
                                                  float observer_z, float current, bool marches,
                                                  const RayStore &store, unsigned &visits,
                                                  unsigned &samples, unsigned &steps,
                                                  Tracker &tracker) {
    const MarchState first = begin_pass(dem, g, current);
    const bool tame = far_tame(dem, g, observer_z);
    float s = march_near<kCount>(table, dem, g, tame, pass_index, observer_z,
                                 marches ? first.s : INFINITY, current, visits, samples, steps,
                                 tracker);
    const float double_radius = 2.0f * (dem.radius + observer_z);
    store.save(0, tame && s >= 0.5f ? g.s_end : -INFINITY, observer_z, double_radius,
               ladder_sine(dem.radius + observer_z, current));
    store.save(1, g.s_start_chord * 1000.0f, 0.004363323129985824f / dem.resolution, current,
               0.0f);
    store.set(RayStore::kEnd, ray_end(g));
    store.set(RayStore::kChord, g.s_start_chord);
    store.set(RayStore::kLimit, tame ? 0.0f : INFINITY);  // +inf: not tame
    for (;;) {
        const StepPoint at = step_point<false>(g, s);
        unsigned tests = 0;
        const LadderFound found = ladder_step<kCount>(store, table, dem, g, at, s, tests);
        const bool settled = found == kSettled;
        if (kCount && settled) ++steps, visits += tests;
        if (__any_sync(0xffffffffu, !settled)) {
            const float s_end = store.get(RayStore::kEnd);
            if (!settled && s <= s_end) {
                RaySegment own = g;
                own.s_end = s_end;
                own.s_start_chord = store.get(RayStore::kChord);
                const float4 ray = store.load(0), scale = store.load(1);
                const float z = ray.y, before = scale.z;
                const float limit = store.get(RayStore::kLimit);
                // The level search may start anywhere: at level 0.
                const bool mips = dem.level_count > 1;
                MarchState st{s, before, 0, mips ? table.side(1) : __int_as_float(0x7fffffff),
                              -INFINITY};
                bool alive = true;
                if (found == kSample && far_sample_step<kCount>(dem, own, at, pass_index, z, st,
                                                                samples, tracker)) {
                    if (kCount) ++steps, ++visits;
                } else {
                    alive = march_step<kCount, kLadderClimb>(table, dem, own, at, pass_index, z,
                                                             st, visits, samples, steps, tracker);
                }
                s = alive ? st.s : INFINITY;
                store.save(0, s >= 0.5f && limit < INFINITY ? s_end : -INFINITY, z, ray.z,
                           st.current != before ? ladder_sine(dem.radius + z, st.current) : ray.w);
                if (st.current != before) store.save(1, scale.x, scale.y, st.current, 0.0f);
            }
            if (!__any_sync(0xffffffffu, s <= s_end)) break;
        }
    }
    return store.load(1).z;
}

}  // namespace ls200
