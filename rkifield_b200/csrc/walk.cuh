// walk.cuh — what the march and the settling passes before it share: the launch
// parameters, the bounds of objects outside the EMPTY samples (balls, boxes,
// half-spaces), the walk of a ray through EMPTY boxes, ray generation and the
// outputs of a ray that misses.
#pragma once

#include "march.h"
#include "sampler.cuh"
#include "tiled.h"

namespace rkf {

namespace detail {

constexpr uint32_t kFull = 0xFFFFFFFFu;

// Object set of a launch: several objects, exactly one, or exactly one that
// qualifies for the empty-space path (voxelized, translation-only
// inverse_world, verified exact quotient, fewer than 2^20 voxels per axis).
// OBJ_SINGLE_EMPTY_TILED: the empty-space path of a tiled launch (EMPTY runs
// on the tiled empty-space field, tiled full steps elsewhere).
// OBJ_MULTI_EMPTY: one object that qualifies for the empty-space path plus
// analytic objects that each fit a ball (FarBall) and objects of no type; its
// EMPTY runs and settling chains stay outside every ball.
// OBJ_MULTI_EMPTY_TILED: the same under the tiled strategy (EMPTY runs on
// the tiled empty-space field, for rays whose object list holds the
// voxelized object; tiled full steps elsewhere).
enum : int {
  OBJ_MULTI = 0,
  OBJ_SINGLE = 1,
  OBJ_SINGLE_EMPTY = 2,
  OBJ_SINGLE_EMPTY_TILED = 3,
  OBJ_MULTI_EMPTY = 4,
  OBJ_MULTI_EMPTY_TILED = 5
};

// Multi-object empty-space path.  Each analytic primitive lies inside a ball
// of radius R around its local origin (sphere r, box |b|, capsule |r|+|h|,
// torus |R|+|r|, cylinder |(r, h)|), and its exact distance is at least |l|-R
// at a local position l.  With c the local origin in world space, sigma a
// lower bound of the smallest singular value of inverse_world's linear part
// and s the object's min_scale, the FP32 value of evaluate_object at a world
// position p is at least (sigma*|p - c| - R - rounding)*s.  The host folds
// the voxelized object's largest EMPTY value and bounds of every rounding
// (the object's own evaluation, the ray's position, this centre's rounding)
// into a radius a + b*P, P = |o| + |d|*|tmax| bounding the magnitude of a
// ray's positions: outside that ball the object's value exceeds every EMPTY
// value, so wherever the voxelized object samples EMPTY, the minimum over
// the scene is that sample, bit for bit.
struct FarBall {
  float c[3];     // world-space centre (half-space: the coefficients G)
  float a, b;     // radius a + b * P (box: margin a + b * P beyond the half extents;
                  // half-space: G.w + H <= a + b * P)
  uint32_t path;  // the object's index in the empty-space path (KParams::ev), or ~0u
  float h[3];     // box: world-space half extents (half-space: h[0] = H)
  uint32_t box;   // 1: an axis-aligned box around c instead of a ball; 2: a half-space
};

// One voxelized object of the multi-object empty-space path.  Wherever the
// ray lies in EMPTY cubes of a set of these objects (each on its own field)
// and outside the balls of every other object (analytic or voxelized), each
// object of the set samples its EMPTY value and every other object a larger
// value, so the scene's minimum is the least EMPTY value of the set.
constexpr uint32_t kMaxEmptyVox = 8;
constexpr uint32_t kWalkLinks = 64;  // boxes a walk may add
struct EmptyVox {
  uint32_t obj;       // object index
  uint32_t plain;     // zero translation and unit scale
  float probe_min;    // probe for a cube once a sample was at least this
  float empty_lo;     // lower bound of every EMPTY value (times the scale)
  float empty_lo_t, empty_hi;  // tight bounds of an EMPTY step
};

struct KParams {
  ObjDev objs[kMaxObjectsFast];  // object table in the constant parameter bank
  SceneDev s;
  const Segment* segs;
  uint32_t nseg;
  uint32_t tile_w, tile_h;
  uint32_t interval;
  uint32_t refill_idle;    // a warp refills once this many of its lanes are done
  uint64_t total;          // work ids of this launch: id0 .. id0 + total - 1
  uint64_t id0;
  unsigned long long* counter;
  rkf_march_params p;
  float probe_min;  // empty-space path: walk ahead once a sample was at least this
  uint32_t budget;     // empty-space path: steps per run before the warp re-converges
  uint32_t plain_obj;  // object 0 has zero translation and unit scale
  TiledDev td;             // tiled strategy inputs (views of a tiled launch)
  uint32_t tiled;
  // empty-space path: a lower bound of every EMPTY value of the path's
  // objects, and tight bounds of the steps a ray takes over EMPTY samples (a
  // tiled launch's coarse skips, of more than 0.5, included in the lower one)
  float empty_lo, empty_lo_t, empty_hi;
  const uint8_t* brute_field;  // empty-space field of the objects alone (s.empty_dist: the tiled launch's)
  const rkf_bvh_node* bvh; // BVH strategy: the imported tree, root first
  const uint32_t* bvh_next;  // per node: the walk's next node (bits 0-30), descend (bit 31)
  // multi-object empty-space path: the voxelized objects that take EMPTY
  // runs, and a ball for every object that needs one (bounding the largest
  // EMPTY value of the path)
  EmptyVox ev[kMaxEmptyVox];
  uint32_t n_ev;
  FarBall ball[kMaxObjectsFast];
  uint32_t n_ball;
  // the rays that the settling passes (settle.cu) left of the launch's views,
  // whose ids come first: {id, end of the EMPTY samples seen (NaN: none)}, and
  // their number; null when no such pass ran
  const uint2* list;
  const uint32_t* list_n;
  uint64_t view_ids;
};
static_assert(sizeof(KParams) <= 32000, "the launch parameters must fit the kernel parameter space");

// Interval helpers in directed rounding: each result interval contains the
// exact result for every value of the operand intervals.
__device__ __forceinline__ void iv_mul(float x, float lo, float hi, float& rlo, float& rhi) {  // x * [lo, hi]
  if (x >= 0.0f) {
    rlo = __fmul_rd(x, lo);
    rhi = __fmul_ru(x, hi);
  } else {
    rlo = __fmul_rd(x, hi);
    rhi = __fmul_ru(x, lo);
  }
}
__device__ __forceinline__ void iv_sq(float lo, float hi, float& rlo, float& rhi) {  // [lo, hi]^2
  const float mlo = lo > 0.0f ? lo : (hi < 0.0f ? -hi : 0.0f);
  const float mhi = fmaxf(fabsf(lo), fabsf(hi));
  rlo = __fmul_rd(mlo, mlo);
  rhi = __fmul_ru(mhi, mhi);
}

// Largest t' >= t such that every position of the ray o + d*u, u in [t, t'],
// lies outside every ball (kMaxFloat when no ball lies ahead), skipping the
// balls of the path objects in `skip` (those the run's set samples), with pad
// added to every ball's reach (rays that stay that near this one); -1 when the
// position at t may lie inside one, with *recheck set to the earliest time
// the ray may leave the balls that may hold it (else -1).  Per ball, with
// w = o - c: the line's squared distance to the centre is |w|^2 - (d.w)^2/|d|^2,
// its closest approach is at -(d.w)/|d|^2, and the chord within the ball
// spans sqrt((rho^2 - h^2)/|d|^2) on each side.  Every quantity is an interval
// evaluated in directed rounding, so the entry time used is a lower bound
// and the exit time an upper bound of the exact ones.  A non-finite ray (or
// a zero direction) makes every ball near.  Out of line: the march loop
// calls it about once per ray, and its code would otherwise sit among the
// loop's hot paths (measured 3% faster out of line).
static __device__ __noinline__ float far_limit(const FarBall* __restrict__ far, uint32_t n, uint32_t skip, float ox,
                                               float oy, float oz, float dx, float dy, float dz, float tmax, float t,
                                               float pad, float& recheck) {
  const float a_lo = __fadd_rd(__fadd_rd(__fmul_rd(dx, dx), __fmul_rd(dy, dy)), __fmul_rd(dz, dz));
  const float a_hi = __fadd_ru(__fadd_ru(__fmul_ru(dx, dx), __fmul_ru(dy, dy)), __fmul_ru(dz, dz));
  // P >= |o| + |d| |tmax| (an L1 norm bounds the L2 norm)
  const float P = __fadd_ru(__fadd_ru(__fadd_ru(fabsf(ox), fabsf(oy)), fabsf(oz)),
                            __fmul_ru(__fsqrt_ru(a_hi), fabsf(tmax)));
  float lim = kMaxFloat;
  bool inside = false;
  recheck = kMaxFloat;
  for (uint32_t j = 0; j < n; ++j) {
    const FarBall& f = far[j];
    if (f.path < 32u && ((skip >> f.path) & 1u)) continue;  // an object of the run's set
    if (f.box == 2) {
      // half-space G.w + H <= m, m = a + b*P (a plane's small values lie in
      // it): along the ray its coordinate G.(o + d u) + H - m is at least
      // s0 + s1 u for u >= 0, both rounded down
      const float m = __fadd_ru(__fadd_ru(f.a, __fmul_ru(f.b, P)),
                                __fmul_ru(pad, __fadd_ru(__fadd_ru(fabsf(f.c[0]), fabsf(f.c[1])), fabsf(f.c[2]))));
      const float s0 = __fsub_rd(__fadd_rd(__fadd_rd(__fadd_rd(__fmul_rd(f.c[0], ox), __fmul_rd(f.c[1], oy)),
                                                     __fmul_rd(f.c[2], oz)), f.h[0]), m);
      const float s1 = __fadd_rd(__fadd_rd(__fmul_rd(f.c[0], dx), __fmul_rd(f.c[1], dy)), __fmul_rd(f.c[2], dz));
      const float now = __fadd_rd(s0, __fmul_rd(s1, t));  // t >= 0
      if (s1 >= 0.0f) {
        if (now > 0.0f) continue;  // outside and not approaching: never inside
        inside = true;             // may be inside now
        // s0 <= now <= 0: outside again for u > -s0 / s1
        if (s1 > 0.0f) recheck = fminf(recheck, __fdiv_ru(-s0, s1));
      } else if (s1 < 0.0f && now > 0.0f) {
        // approaching, outside now (s0 > 0): inside no earlier than s0 / -s1
        lim = fminf(lim, fmaxf(t, __fdiv_rd(s0, -s1)));
      } else {  // inside from now on, or NaN
        inside = true;
      }
      continue;
    }
    if (f.box) {
      // slab test of the box [c - h - m, c + h + m], m = a + b*P: the entry
      // time rounded down and the exit time rounded up
      const float m = __fadd_ru(__fadd_ru(f.a, __fmul_ru(f.b, P)), pad);
      const float o3[3] = {ox, oy, oz}, d3[3] = {dx, dy, dz};
      float e = -kMaxFloat, x = kMaxFloat;
      bool miss = false;
#pragma unroll
      for (int k = 0; k < 3; ++k) {
        const float hw = __fadd_ru(f.h[k], m);
        const float lo = __fsub_rd(f.c[k], hw), hi = __fadd_ru(f.c[k], hw);
        if (d3[k] > 0.0f) {
          e = fmaxf(e, __fdiv_rd(__fsub_rd(lo, o3[k]), d3[k]));
          x = fminf(x, __fdiv_ru(__fsub_ru(hi, o3[k]), d3[k]));
        } else if (d3[k] < 0.0f) {
          e = fmaxf(e, __fdiv_rd(__fsub_ru(hi, o3[k]), d3[k]));
          x = fminf(x, __fdiv_ru(__fsub_rd(lo, o3[k]), d3[k]));
        } else if (!(o3[k] >= lo && o3[k] <= hi)) {
          miss = true;  // parallel to this slab and outside it (NaN: not a miss)
        }
      }
      if (miss || e > x) continue;
      if (t < e) {
        lim = fminf(lim, e);
      } else if (!(t > x)) {  // may be inside now (or NaN)
        inside = true;
        recheck = fminf(recheck, x);
      }
      continue;
    }
    const float rho = __fadd_ru(__fadd_ru(f.a, __fmul_ru(f.b, P)), pad);
    const float rho2 = __fmul_ru(rho, rho);
    const float wxl = __fsub_rd(ox, f.c[0]), wxh = __fsub_ru(ox, f.c[0]);
    const float wyl = __fsub_rd(oy, f.c[1]), wyh = __fsub_ru(oy, f.c[1]);
    const float wzl = __fsub_rd(oz, f.c[2]), wzh = __fsub_ru(oz, f.c[2]);
    float sxl, sxh, syl, syh, szl, szh;
    iv_sq(wxl, wxh, sxl, sxh);
    iv_sq(wyl, wyh, syl, syh);
    iv_sq(wzl, wzh, szl, szh);
    const float W_lo = __fadd_rd(__fadd_rd(sxl, syl), szl);
    float pxl, pxh, pyl, pyh, pzl, pzh;  // d.w
    iv_mul(dx, wxl, wxh, pxl, pxh);
    iv_mul(dy, wyl, wyh, pyl, pyh);
    iv_mul(dz, wzl, wzh, pzl, pzh);
    const float b_lo = __fadd_rd(__fadd_rd(pxl, pyl), pzl), b_hi = __fadd_ru(__fadd_ru(pxh, pyh), pzh);
    float b2l, b2h;
    iv_sq(b_lo, b_hi, b2l, b2h);
    const float h2_lo = __fsub_rd(W_lo, __fdiv_ru(b2h, a_lo));
    if (h2_lo > rho2) continue;  // the line never comes within rho (NaN: not skipped)
    const float half = __fsqrt_ru(__fdiv_ru(__fsub_ru(rho2, h2_lo), a_lo));
    const float nb_lo = -b_hi, nb_hi = -b_lo;  // closest approach -(d.w)/|d|^2
    const float tc_lo = __fdiv_rd(nb_lo, nb_lo < 0.0f ? a_lo : a_hi);
    const float tc_hi = __fdiv_ru(nb_hi, nb_hi > 0.0f ? a_lo : a_hi);
    const float e = __fsub_rd(tc_lo, half), x = __fadd_ru(tc_hi, half);
    if (t < e) {
      lim = fminf(lim, e);
    } else if (!(t > x)) {  // may be inside now (or NaN)
      inside = true;
      recheck = fminf(recheck, x);
    }
  }
  if (inside) return -1.0f;
  recheck = -1.0f;
  return lim;
}

// Grid coordinate (position + half grid size, object-local) of the ray at t,
// rounded exactly as eval_obj -> sample_vox round it for a translation-only
// object.
__device__ __forceinline__ float grid_coord(float o, float d, float t, float m, float half) {
  return __fadd_rn(__fadd_rn(__fadd_rn(o, __fmul_rn(d, t)), m), half);
}

// The EMPTY sampling value of sample_vox at a grid coordinate whose trilinear
// cell lies in EMPTY blocks inside the grid and the geometry box (no clamp,
// no outside term), times the object's scale: eval_obj's result there.
__device__ __forceinline__ float empty_value(const ObjDev& o, float gx, float gy, float gz) {
  const float vx = __fsub_rn(exact_div_vs(gx, o.vs, o.rcp_vs), 0.5f);
  const float vy = __fsub_rn(exact_div_vs(gy, o.vs, o.rcp_vs), 0.5f);
  const float vz = __fsub_rn(exact_div_vs(gz, o.vs, o.rcp_vs), 0.5f);
  const float v = mix3_const(o.be, frac_of(vx), frac_of(vy), frac_of(vz));
  return __fmul_rn(v, o.min_scale);
}

// Conversions by adding 1.5 * 2^23, where floats are the integers: two
// full-rate instructions each, where the conversion instructions issue at a
// quarter of that rate.  near_int: an integer within 1 of x, 0 <= x < 2^22.
__device__ __forceinline__ int near_int(float x) { return __float_as_int(__fadd_rn(x, kIntMagic)) - 0x4B400000; }
__device__ __forceinline__ float small_float(int i) {  // |i| < 2^22, exact
  return __fsub_rn(__int_as_float(i + 0x4B400000), kIntMagic);
}
// Square root within an ulp or two, for bounds with a margin.
__device__ __forceinline__ float sqrt_approx(float x) {
  float r;
  asm("sqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
}
// 1/x within an ulp (infinite for a subnormal x): for bounds with a margin.
__device__ __forceinline__ float rcp_approx(float x) {
  float r;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
}

// A ray as the walk through EMPTY boxes sees it, in voxels: on axis a the
// sampler's voxel-centre coordinate at time t is g[a] + d[a] * t.  The walk
// mirrors the axes the ray runs down (d[a]'s sign bit): with M =
// ObjDev::mirror, a power of two less one that no voxel index exceeds, the
// mirrored coordinate M - v only grows, indices mirror by an exclusive or with
// M, and blocks and bricks map onto blocks and bricks.  The ray passes a face
// at mirrored coordinate x, moved inwards by the margin, at x * inv - cin
// where it enters and at (x - 2 margin) * inv - cin where it leaves.  margin
// covers every rounding between t and the sampler's grid coordinate and every
// rounding made here: 0.1 voxel plus 2^-18 of the magnitudes involved, a wide
// multiple of the few 2^-24 roundings.  It is infinite for a direction that is
// NaN, infinite or beyond kMaxRate voxels per unit of t, of which face times say
// nothing (the reciprocal underflows to zero): no walk starts then.
struct ProbeRay {
  float g[3], d[3], inv[3], cin[3], margin;
};
constexpr float kMaxRate = 1.152921504606847e18f;  // 2^60

__device__ __forceinline__ int down_mask(const ProbeRay& r, int a) { return __float_as_int(r.d[a]) >> 31; }
__device__ __forceinline__ float mirrored(const ObjDev& o, const ProbeRay& r, int a, float v) {
  return r.d[a] < 0.0f ? small_float(o.mirror) - v : v;
}

__device__ __forceinline__ ProbeRay probe_ray(const ObjDev& o, float ox, float oy, float oz, float dx, float dy,
                                              float dz) {
  ProbeRay r;
  const float og[3] = {ox, oy, oz}, dir[3] = {dx, dy, dz};
  float mag = 1.0f;
#pragma unroll
  for (int a = 0; a < 3; ++a) mag += fabsf(og[a]) + o.mag[a];
  r.margin = 0.1f + mag * o.rcp_vs * 3.814697265625e-6f;
#pragma unroll
  for (int a = 0; a < 3; ++a)
    if (!(fabsf(dir[a]) * o.rcp_vs <= kMaxRate)) r.margin = INFINITY;
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    r.g[a] = (og[a] + o.m[12 + a] + o.half_gs[a]) * o.rcp_vs - 0.5f;
    // (an axis the ray does not move on: no position of interest moves by a
    // millionth of a voxel)
    r.d[a] = copysignf(fmaxf(fabsf(dir[a]) * o.rcp_vs, 1.0e-15f), dir[a]);
    r.inv[a] = fabsf(rcp_approx(r.d[a]));
    r.cin[a] = (mirrored(o, r, a, r.g[a]) - r.margin) * r.inv[a];
  }
  return r;
}

// A box of EMPTY bricks as the times the ray enters and leaves it on each
// axis, its faces moved inwards by the margin: between max(in) and min(out)
// the trilinear corners of every sample lie in EMPTY bricks.  A face at the
// grid's border lies at infinity: beyond it the sampler clamps the coordinate
// to the border voxel, which is in the box.
struct EmptyBox {
  float in[3], out[3];
};

// The EMPTY box around the (clamped) position at t: the cube of EMPTY blocks
// the empty-space field promises there or, in a leaf block (bricks), the cube
// of EMPTY bricks its leaf distances promise.  Which block the position falls
// into only chooses the box (its EMPTY-ness holds for any).  false: the
// position's brick is not EMPTY (or, without bricks, its block).
__device__ __forceinline__ bool empty_box(const ObjDev& o, const SceneDev& s, const uint8_t* __restrict__ field,
                                          bool bricks, const ProbeRay& r, float t, EmptyBox& b) {
  int v[3];
#pragma unroll
  for (int a = 0; a < 3; ++a)
    v[a] = near_int(fminf(fmaxf(__fmaf_rn(r.d[a], t, r.g[a]) - 0.5f, 0.0f), o.last[a]));
  const uint32_t blk = o.top_off + (v[0] >> 6) + ((v[1] >> 6) + (v[2] >> 6) * o.tdim[1]) * o.tdim[0];
  uint32_t d = __ldg(field + blk);
  int shift = 6;
  if (d == 0) {
    if (!bricks) return false;
    const uint32_t leaf = __ldg(s.top + blk);
    if (leaf >= RKF_INTERIOR_SLOT) return false;
    d = load_leaf_dist(s.leaf_dist + static_cast<size_t>(leaf) * 512 +
                       (((v[0] >> 3) & 7) + (v[1] & 56) + (v[2] & 56) * 8));
    if (d == 0) return false;
    shift = 3;
  }
  // every block (brick) within d - 1 is EMPTY
  const int above = static_cast<int>(d) << shift, unit = 1 << shift;
  const float two_m = 2.0f * r.margin;
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    const int down = down_mask(r, a);
    const int base = (v[a] ^ (down & o.mirror)) & -unit;  // mirrored from here on
    const int first = down & (o.mirror - o.tv[a] + 1);    // the grid's border voxels: first, first + tv - 1
    const int lo = base + unit - above, hi = base + above - 1;
    b.in[a] = lo <= first ? -INFINITY : __fmaf_rn(small_float(lo), r.inv[a], -r.cin[a]);
    b.out[a] = hi - first >= o.tv[a] - 1 ? INFINITY : __fmaf_rn(small_float(hi) - two_m, r.inv[a], -r.cin[a]);
  }
  return true;
}

// A walk of the ray from t through EMPTY boxes: every sample at a time in
// [t, end] has all its corners in EMPTY bricks (clamped to the grid as the
// sampler clamps them), so its value is at least the EMPTY value -- that value
// inside the grid and the geometry box, the distance to either where that is
// larger.  out: the times the ray leaves the last box on each axis.
//
// walk_start: the box at t.  false when the position at t lies in none.
__device__ __forceinline__ bool walk_start(const ObjDev& o, const SceneDev& s, const uint8_t* __restrict__ field,
                                           bool bricks, const ProbeRay& r, float t, float& end, float* out) {
  EmptyBox A;
  if (!empty_box(o, s, field, bricks, r, t, A)) return false;
#pragma unroll
  for (int a = 0; a < 3; ++a) out[a] = A.out[a];
  end = fminf(fminf(A.out[0], A.out[1]), A.out[2]);
  // (a margin beyond two voxels, or none that would do: a seam would span more
  // than a brick)
  return fmaxf(fmaxf(A.in[0], A.in[1]), A.in[2]) <= t && end >= t && r.margin < 2.0f;
}

// Whether every brick that a sample between times t0 < t1 can touch is EMPTY,
// where these lie in at most two bricks on each axis (the ray's voxels from t0
// to t1, a margin to each side).
__device__ __forceinline__ bool seam_empty(const ObjDev& o, const SceneDev& s, const uint8_t* __restrict__ field,
                                           bool bricks, const ProbeRay& r, float t0, float t1) {
  int b0[3], b1[3];
  bool two = true;
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    const float p0 = __fmaf_rn(r.d[a], t0, r.g[a]), p1 = __fmaf_rn(r.d[a], t1, r.g[a]);
    const float lo = fminf(p0, p1) - r.margin - 0.5f, hi = fmaxf(p0, p1) + r.margin + 1.5f;  // near_int: at most lo + 0.5
    b0[a] = near_int(fminf(fmaxf(lo, 0.0f), o.last[a])) >> 3;
    b1[a] = near_int(fminf(fmaxf(hi, 0.0f), o.last[a])) >> 3;
    two = two && b1[a] - b0[a] <= 1;
  }
  if (!two) return false;
#pragma unroll 1
  for (uint32_t i = 0; i < 8u; ++i) {
    if (((i & 1u) && b1[0] == b0[0]) || ((i & 2u) && b1[1] == b0[1]) || ((i & 4u) && b1[2] == b0[2])) continue;
    const int x = (i & 1u) ? b1[0] : b0[0], y = (i & 2u) ? b1[1] : b0[1], z = (i & 4u) ? b1[2] : b0[2];
    const uint32_t blk = o.top_off + (x >> 3) + ((y >> 3) + (z >> 3) * o.tdim[1]) * o.tdim[0];
    if (__ldg(field + blk)) continue;
    const uint32_t leaf = bricks ? __ldg(s.top + blk) : RKF_INTERIOR_SLOT;
    if (leaf >= RKF_INTERIOR_SLOT ||
        !load_leaf_dist(s.leaf_dist + static_cast<size_t>(leaf) * 512 + ((x & 7) + (y & 7) * 8 + (z & 7) * 64)))
      return false;
  }
  return true;
}

// walk_link: on to the next box.  false when there is none.  The next box B is
// found just past the last one's end: a voxel and both margins beyond the face
// the ray leaves through (and beyond another it leaves through within that
// stretch).  Either B already holds the end, so the boxes overlap, or B begins
// where the last box's voxels end on that one axis, and both hold the ray
// across the seam on the other two; then the cells that straddle the seam touch
// voxels of these two boxes only.  Where neither holds (the ray leaves near an
// edge, about one link in 28) the bricks around the seam are looked up.
__device__ __forceinline__ bool walk_link(const ObjDev& o, const SceneDev& s, const uint8_t* __restrict__ field,
                                          bool bricks, const ProbeRay& r, float& end, float* out) {
  const float seam = (1.0f + 2.0f * r.margin) * 1.01f;
  const bool x0 = out[0] == end, x1 = !x0 && out[1] == end;  // the exit axis: 0, 1, else 2
  float tn = __fmaf_rn(seam, x0 ? r.inv[0] : x1 ? r.inv[1] : r.inv[2], end);
  float tm = tn;
#pragma unroll
  for (int a = 0; a < 3; ++a)
    if (out[a] <= tn) tm = fmaxf(tm, __fmaf_rn(seam, r.inv[a], out[a]));
  tn = tm;
  EmptyBox B;
  if (!empty_box(o, s, field, bricks, r, tn, B)) return false;
  const float e = fminf(fminf(B.out[0], B.out[1]), B.out[2]);
  const float in2 = fmaxf(fmaxf(x0 ? -INFINITY : B.in[0], x1 ? -INFINITY : B.in[1]), x0 || x1 ? B.in[2] : -INFINITY);
  const float out2 = fminf(fminf(x0 ? INFINITY : out[0], x1 ? INFINITY : out[1]), x0 || x1 ? out[2] : INFINITY);
  const float in1 = x0 ? B.in[0] : x1 ? B.in[1] : B.in[2];  // the exit axis
  const bool held = in2 <= end && (in1 <= end || (in1 <= tn && out2 >= tn && e >= tn));
  if (!(e > end)) return false;
  if (!held && !(fmaxf(in1, in2) <= tn && e >= tn && seam_empty(o, s, field, bricks, r, end, tn))) return false;
  end = e;
#pragma unroll
  for (int a = 0; a < 3; ++a) out[a] = B.out[a];
  return true;
}

// The whole walk towards target, over at most `links` further boxes: its end,
// or -1 when the position at t lies in no box.
__device__ __forceinline__ float walk_empty(const ObjDev& o, const SceneDev& s, const uint8_t* __restrict__ field,
                                            bool bricks, const ProbeRay& r, float t, float target, uint32_t links) {
  float end, out[3];
  if (!walk_start(o, s, field, bricks, r, t, end, out)) return -1.0f;
#pragma unroll 1
  while (links && end < target && walk_link(o, s, field, bricks, r, end, out)) --links;
  return end;
}

// The interval in which the ray lies between the border voxel centres of the
// grid and inside the geometry box (both moved inwards by the margin), where a
// sample in EMPTY bricks is exactly empty_value(): true when t lies in it.
__device__ __forceinline__ bool core_interval(const ObjDev& o, const ProbeRay& r, float t, float& t_in,
                                              float& t_out) {
  t_in = -INFINITY;
  t_out = INFINITY;
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    const float l = mirrored(o, r, a, r.d[a] < 0.0f ? o.core_hi[a] : o.core_lo[a]);
    const float h = mirrored(o, r, a, r.d[a] < 0.0f ? o.core_lo[a] : o.core_hi[a]);
    t_in = fmaxf(t_in, __fmaf_rn(l, r.inv[a], -r.cin[a]));
    t_out = fminf(t_out, __fmaf_rn(h - 2.0f * r.margin, r.inv[a], -r.cin[a]));
  }
  return t >= t_in && t <= t_out;
}

// Where a ray is after n <= k steps of [lo, hi] each: each sum rounds by at most
// 2^-24 of t, so t lies between (t + n lo) (1 - grow) and (t + n hi) (1 + grow)
// (2^-22 a step, and 4 more, leaves room for these bounds' own rounding).
// Turned round, t is surely at most T while t + n hi <= T (1 - grow), and at least
// T from t + n lo >= T (1 + 2 grow) on (grow <= 1/2: at most 2^20 steps).
__device__ __forceinline__ float steps_grow(float k) { return (k + 4.0f) * 2.384185791015625e-7f; }

// How a ray whose every sample ahead is at least the EMPTY value ends when it
// leaves the grid before it could run out of steps (one voxelized object): 1
// past tmax, 2 out of steps, 0 undecided.  The ray runs out of steps exactly
// when t after the k steps left is still <= tmax.
//
// From inside the core interval (t <= t_out) every step up to t_out lies in
// [lo, hi], so t after n steps is known to a few millimetres; from the last
// step that surely ends before t_out the interval [L, U] of t is carried on
// step by step.  There the sampler returns the distance to the grid's clamp box
// where that exceeds two brick extents, else the distance to the geometry box
// where that exceeds one, else an EMPTY value plus the former; both distances
// are 0 inside and do not fall along a ray that leaves convex boxes, so their
// values at L and U bound them in between (widened by 2^-12, which covers the
// margin by which the faces are known and every rounding).
//
// Before that, and from anywhere: up to where the ray leaves the clamp box on
// some axis each step is at least lo; from there the distance to it grows by c
// per unit of t, so once it exceeds two brick extents (at most 2/c more steps
// of lo) every step multiplies the time since the exit by at least 1 + c.
// (c > 0; approximate logarithms and quotients, with 0.1% and 3 steps to spare.)
__device__ __forceinline__ uint32_t leaves_grid(const ObjDev& o, const ProbeRay& r, float t, float tmax, bool core,
                                                float t_out, float k, float lo, float hi) {
  const float M = small_float(o.mirror);
  float t_o = INFINITY, c = 0.0f;
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    // the clamp box ends half a voxel beyond the border voxel's centre
    const float e = ((r.d[a] < 0.0f ? M : o.last[a]) + 0.5f + r.margin - mirrored(o, r, a, r.g[a])) * r.inv[a];
    if (e < t_o) {
      t_o = e;
      c = fabsf(r.d[a]) * o.vs;  // world units per unit of t
    }
  }
  c *= o.min_scale * 0.998f;
  const float grow = steps_grow(k);
  const float most =
      __fdividef(fmaxf(t_o * (1.0f + 2.0f * grow) - t, 0.0f), lo) + __fdividef(2.0f, c) +
      __fdividef(__logf(fmaxf(__fdividef((tmax - t_o) * c, lo), 1.0f)), __logf(1.0f + c)) * 1.001f + 7.0f;
  if (most < k) return 1u;
  if (!core || !(t_out < tmax)) return 0u;
  const float n0 = fmaxf(floorf(__fdividef(t_out * (1.0f - grow) - t, hi)) - 3.0f, 0.0f);
  if (n0 >= k) return 2u;
  float L = (t + n0 * lo) * (1.0f - steps_grow(n0));
  float U = (t + n0 * hi) * (1.0f + steps_grow(n0));
  const float be = o.be, be2 = o.be2, e_lo = be * (1.0f - 1.52587890625e-5f), e_hi = be * (1.0f + 1.52587890625e-5f);
  const float wide = 2.44140625e-4f, slack = r.margin * o.vs;
  float n = k - n0;
#pragma unroll 1
  for (uint32_t it = 0; n > 0.0f; ++it) {
    if (it == 96u) return 0u;  // (a grazing exit: step it)
    float oL = 0.0f, oU = 0.0f, gL = 0.0f, gU = 0.0f;
#pragma unroll
    for (int a = 0; a < 3; ++a) {
      // it left through upper faces only (its mirrored coordinates grow)
      const float d = fabsf(r.d[a]), g = mirrored(o, r, a, r.g[a]);
      const float ch = (r.d[a] < 0.0f ? M : o.last[a]) + 0.49f - g;
      const float xL = fmaxf(__fmaf_rn(d, L, -ch), 0.0f), xU = fmaxf(__fmaf_rn(d, U, -ch), 0.0f);
      oL += xL * xL;
      oU += xU * xU;
      if (o.has_geom) {
        const float gh = mirrored(o, r, a, ((r.d[a] < 0.0f ? o.gmin[a] : o.gmax[a]) + o.half_gs[a]) * o.rcp_vs - 0.5f) - g;
        const float yL = fmaxf(__fmaf_rn(d, L, -gh), 0.0f), yU = fmaxf(__fmaf_rn(d, U, -gh), 0.0f);
        gL += yL * yL;
        gU += yU * yU;
      }
    }
    oL = fmaxf(sqrt_approx(oL) * o.vs * (1.0f - wide) - 2.0f * slack, 0.0f), oU = sqrt_approx(oU) * o.vs * (1.0f + wide) + 2.0f * slack;
    gL = fmaxf(sqrt_approx(gL) * o.vs * (1.0f - wide) - 2.0f * slack, 0.0f), gU = sqrt_approx(gU) * o.vs * (1.0f + wide) + 2.0f * slack;
    // the values the three cases can take anywhere in [L, U]
    float v_lo = INFINITY, v_hi = 0.0f;
    if (oU > be2) {
      v_lo = fmaxf(oL, be2);
      v_hi = oU;
    }
    if (oL <= be2) {
      if (gU > be) {
        v_lo = fminf(v_lo, fmaxf(gL, be));
        v_hi = fmaxf(v_hi, gU);
      }
      if (gL <= be) {
        v_lo = fminf(v_lo, e_lo + oL);
        v_hi = fmaxf(v_hi, e_hi + fminf(oU, be2));
      }
    }
    L = (L + v_lo * o.min_scale * (1.0f - 3.0517578125e-5f)) * (1.0f - 2.384185791015625e-7f);
    U = (U + v_hi * o.min_scale * (1.0f + 3.0517578125e-5f)) * (1.0f + 2.384185791015625e-7f);
    n -= 1.0f;
    if (L > tmax) return 1u;  // t only grows
  }
  return U <= tmax ? 2u : 0u;
}

// The next float above a time (t >= 0); NaN above infinity, and every t
// compares false with it: a lane's "no walk before this t" is always past t
// after a walk, so a walk is followed by a step.
__device__ __forceinline__ float after(float t) { return __uint_as_float(__float_as_uint(t) + 1u); }

__device__ __forceinline__ uint32_t find_segment(const Segment* segs, uint32_t nseg, uint64_t id) {
  uint32_t lo = 0, hi = nseg;  // last segment with first <= id
  while (hi - lo > 1) {
    const uint32_t mid = (lo + hi) >> 1;
    if (segs[mid].first <= id) lo = mid; else hi = mid;
  }
  return lo;
}

// The ray of pixel (px, py) of a view (ray_march.wgsl:1046-1053).
__device__ __forceinline__ void view_ray(const Segment& sg, uint32_t px, uint32_t py, float& dx, float& dy, float& dz) {
  const float u = __fdiv_rn(__fadd_rn(__fadd_rn(static_cast<float>(px), 0.5f), sg.jitter[0]), static_cast<float>(sg.w));
  const float v = __fdiv_rn(__fadd_rn(__fadd_rn(static_cast<float>(py), 0.5f), sg.jitter[1]), static_cast<float>(sg.h));
  const float nx = __fsub_rn(__fmul_rn(u, 2.0f), 1.0f);
  const float ny = __fsub_rn(1.0f, __fmul_rn(v, 2.0f));
  const float vx = __fadd_rn(__fadd_rn(sg.fwd[0], __fmul_rn(sg.right[0], nx)), __fmul_rn(sg.up[0], ny));
  const float vy = __fadd_rn(__fadd_rn(sg.fwd[1], __fmul_rn(sg.right[1], nx)), __fmul_rn(sg.up[1], ny));
  const float vz = __fadd_rn(__fadd_rn(sg.fwd[2], __fmul_rn(sg.right[2], nx)), __fmul_rn(sg.up[2], ny));
  const float l = len3(vx, vy, vz);
  dx = __fdiv_rn(vx, l);
  dy = __fdiv_rn(vy, l);
  dz = __fdiv_rn(vz, l);
}

// The march steps along the safe direction (ray_march.wgsl:784).
__device__ __forceinline__ float safe_dir(float d) { return fabsf(d) < 1e-10f ? 1e-10f : d; }

// The outputs of a closest-hit ray that ends unhit.
__device__ __forceinline__ void write_miss(const Segment& sg, uint32_t idx, uint16_t flags) {
  sg.t[idx] = kMaxFloat;
  if (sg.flags) sg.flags[idx] = flags;
  if (sg.normal) {
    sg.normal[3 * static_cast<size_t>(idx)] = 0.0f;
    sg.normal[3 * static_cast<size_t>(idx) + 1] = 0.0f;
    sg.normal[3 * static_cast<size_t>(idx) + 2] = 0.0f;
  }
  if (sg.slot) sg.slot[idx] = RKF_EMPTY_SLOT;
  if (sg.material) sg.material[idx] = 0;
  if (sg.position) reinterpret_cast<float4*>(sg.position)[idx] = make_float4(0.f, 0.f, 0.f, kMaxFloat);
  if (sg.packed) sg.packed[idx] = 0u;
  if (sg.motion) reinterpret_cast<float4*>(sg.motion)[idx] = make_float4(0.f, 0.f, 0.f, 0.f);
}

}  // namespace detail

}  // namespace rkf
