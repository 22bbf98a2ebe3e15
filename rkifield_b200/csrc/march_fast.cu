// march_fast.cu — the B200 march: one persistent, work-fetching kernel for
// views (primary rays) and ray batches (closest / any-hit / soft shadow).
//
// Reference algorithm: crates/rkf-render/shaders/ray_march.wgsl:776-858
// (ray_march_brute), :641-773 (ray_march_bvh), :874-985 (ray_march_tiled),
// :941-964 (bisection), :1003-1032
// (normals), :1036-1112 (ray generation and G-buffer), and
// shade_common_shading.wgsl:9-33 (soft_shadow).
//
// Execution model.  Each lane owns one ray at a time and a warp takes one phase at a
// time, the one most of its lanes are ready for:
//   refill  once enough lanes are done, they write their outputs and take the next
//           work ids from a global counter (one warp-aggregated atomic); ids walk
//           views tile by tile, so a warp's rays stay spatially coherent;
//   walk    lanes whose last sample was about the EMPTY value find how far their rays
//           cross EMPTY boxes (walk.cuh), which settles a ray or starts a run;
//   run     steps over EMPTY samples, without the sampler;
//   eval    samples of the scene, whatever they are for: a step, a bisection, a
//           normal's differences.
// The hit material is read once, from the position that decided it.  Large views come
// through the passes of settle.cu first, which leave the rays that may hit.
#include <algorithm>
#include <cmath>
#include <cstring>
#include <limits>
#include <vector>

#include "../../include/rkf_cuda_testing.h"
#include "ctx.h"
#include "march.h"
#include "f32x2.cuh"
#include "sampler.cuh"
#include "walk.cuh"
#include "settle.h"
#include "tiled.h"
#include "tile_order.h"

namespace rkf {

namespace detail {

// What a lane's ray is doing: nothing, marching (towards a surface, or a
// light), bisecting an overstep, taking the samples of a hit's normal, or done
// with its outputs still to write.
enum : uint32_t { ST_IDLE = 0, ST_MARCH, ST_SHADOW, ST_BISECT, ST_NORMAL, ST_EPI };

// Per-lane ray state that is read or written only when a ray starts, hits
// or ends.
struct ColdState {
  uint32_t seg, idx, hit_obj, sub;
  float lo, hi, mat_t, gpos, shadow;
  uint32_t tile_base, tile_count;  // tiled strategy: the ray's object list (kNoTiles: every object)
  float g[3];                // the normal's central differences
  float sdf_hit;             // the hit's own sample (motion plane)
  bool hit, bisected, mat_ok;
  // multi-object empty-space path: bits 0-7, the voxelized objects of the
  // path (KParams::ev) whose EMPTY runs the ray may take (under the tiled
  // strategy, those its object list holds); bits 8-15, the one whose cube
  // the ray is in (its last successful probe). 
  // (An odd number of words per lane: a warp's accesses hit 32 distinct banks.)
  uint32_t vox_listed;
};
static_assert(sizeof(ColdState) % 8 == 4, "ColdState must span an odd number of 32-bit words");

// The candidate loop of ray_march_bvh (ray_march.wgsl:672-721): a stack walk
// of the tree from the root that skips every node whose AABB lies farther
// from the position than the best distance so far, evaluates the objects of
// the leaves it reaches (object indices beyond the object count are skipped),
// and pushes the left then the right child while fewer than 31 entries are on
// the stack (so the right child is visited first).  On the trees the import
// admits the stack's content at each node is fixed by the tree, so the same
// walk runs from the per-node links bvh.cu derives (next node after the
// subtree, whether to descend), without a stack.  The distance to a box is
// length(clamp(pos, min, max) - pos); its square root is taken only where the
// comparison needs it (an exact zero stays zero, and any length exceeds a
// negative best).
//
// The next object of that walk for position w and the best value so far; node: where
// the walk stands (0 at first).  kBvhEnd: none is left.
constexpr uint32_t kBvhEnd = 0x7FFFFFFFu;
__device__ __forceinline__ uint32_t bvh_candidate(const rkf_bvh_node* nodes, const uint32_t* __restrict__ next,
                                                  uint32_t nobj, float wx, float wy, float wz, float best,
                                                  uint32_t& node) {
  while (node != kBvhEnd) {
    const float4* nd = reinterpret_cast<const float4*>(nodes + node);
    const float4 a = __ldg(nd), b = __ldg(nd + 1);
    const uint32_t link = __ldg(next + node);
    const float ex = __fsub_rn(fminf(fmaxf(wx, a.x), b.x), wx);
    const float ey = __fsub_rn(fminf(fmaxf(wy, a.y), b.y), wy);
    const float ez = __fsub_rn(fminf(fmaxf(wz, a.z), b.z), wz);
    const float d2 = __fadd_rn(__fadd_rn(__fmul_rn(ex, ex), __fmul_rn(ey, ey)), __fmul_rn(ez, ez));
    bool skip;
    if (d2 == 0.0f) skip = 0.0f > best;
    else if (best < 0.0f && d2 == d2) skip = true;
    else skip = __fsqrt_rn(d2) > best;
    const uint32_t left = __float_as_uint(a.w), ro = __float_as_uint(b.w);
    const bool leaf = left == RKF_BVH_INVALID;
    node = !skip && !leaf && (link >> 31) ? ro : (link & kBvhEnd);
    if (!skip && leaf && ro < nobj) return ro;
  }
  return kBvhEnd;
}

// Up to n march steps of a ray through positions covered by EMPTY boxes: each
// sample is empty_value().  The run stops before a step whose sample is below
// brk or whose t is past tmax (the full step decides those), after the step
// that makes max_near samples below near_thr, and at the end of the covered
// interval (t > box_t); stop_full tells whether the next step must be a full
// one.
// PLAIN: the object's translation is zero and its scale one, where adding the
// translation and multiplying by the scale are exact identities.
// Returns the number of steps taken.
template <bool PLAIN>
__device__ __forceinline__ uint32_t empty_run(const ObjDev& o, float ox, float oy, float oz, float dx, float dy,
                                              float dz, float tmax, uint32_t n, float brk, float near_thr,
                                              float min_step, uint32_t max_near, float& t, float box_t,
                                              float& prev_t, float& prev_dist, uint32_t& near, bool& stop_full) {
  uint32_t c = 0;
  const float lim = fminf(box_t, tmax);
  stop_full = false;
#pragma unroll 2
  for (; c < n; ++c) {
    if (t > lim) {
      stop_full = t > tmax;
      break;
    }
    float gx, gy, gz;
    if (PLAIN) {
      gx = __fadd_rn(__fadd_rn(ox, __fmul_rn(dx, t)), o.half_gs[0]);
      gy = __fadd_rn(__fadd_rn(oy, __fmul_rn(dy, t)), o.half_gs[1]);
      gz = __fadd_rn(__fadd_rn(oz, __fmul_rn(dz, t)), o.half_gs[2]);
    } else {
      gx = grid_coord(ox, dx, t, o.m[12], o.half_gs[0]);
      gy = grid_coord(oy, dy, t, o.m[13], o.half_gs[1]);
      gz = grid_coord(oz, dz, t, o.m[14], o.half_gs[2]);
    }
    const float vx = __fsub_rn(exact_div_vs(gx, o.vs, o.rcp_vs), 0.5f);
    const float vy = __fsub_rn(exact_div_vs(gy, o.vs, o.rcp_vs), 0.5f);
    const float vz = __fsub_rn(exact_div_vs(gz, o.vs, o.rcp_vs), 0.5f);
    float d = mix3_const(o.be, frac_of(vx), frac_of(vy), frac_of(vz));
    if (!PLAIN) d = __fmul_rn(d, o.min_scale);
    if (!(d >= brk)) {  // no step: the full step redoes this sample
      stop_full = true;
      break;
    }
    prev_t = t;
    prev_dist = d;
    t = __fadd_rn(t, fmax_(d, min_step));
    if (d < near_thr && ++near >= max_near) {
      stop_full = true;
      return c + 1;
    }
  }
  return c;
}

// The EMPTY value of a plain object (zero translation, unit scale) at the
// ray's position at t: empty_run<PLAIN=true>'s step with the x and y chains
// packed into two-wide FP32 instructions (z stays scalar) -- the same
// operations on the same values, so the same bits.
__device__ __forceinline__ float empty_value_x2(f2 o01, f2 d01, f2 h01, f2 r2, f2 nvs2, f2 half2, float oz, float dz,
                                                float hz, float vs, float rcp, float be, float t) {
  // (the products one at a time: the assembler joins a packed product and the packed
  // sum that takes it into one instruction, which rounds once)
  float dx, dy;
  f2_unpack(d01, dx, dy);
  const f2 g01 = f2_add(f2_add(o01, f2_pack(__fmul_rn(dx, t), __fmul_rn(dy, t))), h01);
  const f2 q0 = f2_mul(g01, r2);
  const f2 v01 = f2_sub(f2_fma(f2_fma(q0, nvs2, g01), r2, q0), half2);
  const float vz = __fsub_rn(exact_div_vs(__fadd_rn(__fadd_rn(oz, __fmul_rn(dz, t)), hz), vs, rcp), 0.5f);
  const f2 magic = f2_pack(kIntMagic, kIntMagic);
  float tx, ty;
  f2_unpack(f2_sub(v01, f2_sub(f2_add(v01, magic), magic)), tx, ty);  // frac_of
  return mix3_const(be, up_frac(tx), up_frac(ty), frac_of(vz));
}

// The run of a plain object whose every EMPTY value is at least brk, near_thr
// and min_step (the caller checks this against a lower bound, so those
// comparisons are known), two steps at a time.  Each step is
// t' = t + E(t), a chain in which every step waits for the last.  E(t)
// equals the brick extent c (the EMPTY constant) exactly for most positions
// (the three nested mix(c, c, f) round back to c for about 93% of
// positions), so the position of the next step is taken to be t + c (the
// rounding the step would make) and both E values are computed
// independently.  The second step is accepted when the first value was
// exactly c -- then its position is the one the serial march reaches, bit
// for bit -- and when it passes the serial loop's checks (budget, box end,
// tmax); otherwise the first step is taken alone, with its value.  (Four
// steps at a time measured 3-4% slower on the 1080p view: the longer code
// raised instruction-fetch stalls by more than it cut dependency stalls.)
__device__ __forceinline__ uint32_t empty_run_x2(const ObjDev& o, float ox, float oy, float oz, float dx, float dy,
                                                 float dz, float tmax, uint32_t n, float& t, float box_t,
                                                 float& prev_t, float& prev_dist, bool& stop_full) {
  uint32_t c = 0;
  const float lim = fminf(box_t, tmax);
  stop_full = false;
  const f2 o01 = f2_pack(ox, oy), d01 = f2_pack(dx, dy), h01 = f2_pack(o.half_gs[0], o.half_gs[1]);
  const f2 r2 = f2_pack(o.rcp_vs, o.rcp_vs), nvs2 = f2_pack(-o.vs, -o.vs), half2 = f2_pack(0.5f, 0.5f);
  const float hz = o.half_gs[2], vs = o.vs, rcp = o.rcp_vs, be = o.be;
  while (c < n) {
    if (t > lim) {
      stop_full = t > tmax;
      break;
    }
    // the position of the next step if this value is c
    const float t1 = __fadd_rn(t, be);
    const float e0 = empty_value_x2(o01, d01, h01, r2, nvs2, half2, oz, dz, hz, vs, rcp, be, t);
    const float e1 = empty_value_x2(o01, d01, h01, r2, nvs2, half2, oz, dz, hz, vs, rcp, be, t1);
    // step 0 passed the checks above; step 1 needs the first value to be c
    // (so that t1 is the serial position) and the serial checks
    float pt = t, pd = e0;
    ++c;
    if (e0 == be && c < n && t1 <= lim) {
      pt = t1;
      pd = e1;
      ++c;
    }
    prev_t = pt;
    prev_dist = pd;
    t = __fadd_rn(pt, pd);
  }
  return c;
}

// Up to n march steps through positions where every object of the set
// (path objects, at least two) samples its EMPTY value and every other
// object lies beyond its ball: each step's value is the least of the set's
// EMPTY values, computed as eval_obj -> sample_vox would round it.  The run
// stops at the end of the nearest cube (box_t, already clipped at the first
// ball ahead), before a step whose value is below brk, and after the step
// that makes max_near values below near_thr; CLEAN: the values clear every
// threshold (a lower bound checked by the caller).  Returns the steps taken.
template <bool CLEAN>
__device__ __noinline__ uint32_t empty_run_set(const ObjDev* objs, const EmptyVox* ev, uint32_t set, uint32_t n_ev,
                                               float ox, float oy, float oz, float dx, float dy, float dz, float tmax,
                                               uint32_t n, float brk, float near_thr, float min_step,
                                               uint32_t max_near, float& t, float box_t, float& prev_t,
                                               float& prev_dist, uint32_t& near, bool& stop_full) {
  uint32_t c = 0;
  const float lim = fminf(box_t, tmax);
  stop_full = false;
  for (; c < n; ++c) {
    if (t > lim) {
      stop_full = t > tmax;
      break;
    }
    float d = kMaxFloat;
    for (uint32_t e = 0; e < n_ev; ++e) {
      if (!((set >> e) & 1u)) continue;
      const ObjDev& o = objs[ev[e].obj];
      const float v = empty_value(o, grid_coord(ox, dx, t, o.m[12], o.half_gs[0]),
                                  grid_coord(oy, dy, t, o.m[13], o.half_gs[1]),
                                  grid_coord(oz, dz, t, o.m[14], o.half_gs[2]));
      if (v < d) d = v;
    }
    if (!CLEAN && !(d >= brk)) {  // no step: the full step redoes this sample
      stop_full = true;
      break;
    }
    prev_t = t;
    prev_dist = d;
    if (CLEAN) {
      t = __fadd_rn(t, d);
      continue;
    }
    t = __fadd_rn(t, fmax_(d, min_step));
    if (d < near_thr && ++near >= max_near) {
      stop_full = true;
      return c + 1;
    }
  }
  return c;
}

constexpr uint32_t kRefillRounds = 8;

// What a hit's outputs are made of.
struct HitRay {
  float ox, oy, oz, rdx, rdy, rdz, t, mat_t, g0, g1, g2, sdf_hit;
  uint32_t idx;
  bool bisected, mat_ok;
};

// The G-buffer entry of a hit (ray_march.wgsl:1003-1032, :1068-1105).  Out of
// line: few rays hit, and its divisions are a large part of a kernel's code.
static __device__ __noinline__ void write_hit(const SceneDev& s, const ObjDev& o, const Segment& sg, const HitRay h) {
  LaneCache lc;
  const uint16_t flags = RKF_FLAG_HIT | (h.bisected ? RKF_FLAG_BISECTED : 0);
  const float hx = __fadd_rn(h.ox, __fmul_rn(h.rdx, h.t)), hy = __fadd_rn(h.oy, __fmul_rn(h.rdy, h.t)),
              hz = __fadd_rn(h.oz, __fmul_rn(h.rdz, h.t));
  float gx = h.g0, gy = h.g1, gz = h.g2, sdf_hit = 0;
  uint32_t slot = RKF_EMPTY_SLOT, mat = 0, sec = 0, blend = 0;
  const bool vox = o.sdf_type == RKF_SDF_VOXELIZED;
  if (vox) {
    // world_grad = transpose(inverse_world) * (g, 0)  (:1014)
    gx = __fadd_rn(__fadd_rn(__fadd_rn(__fmul_rn(o.m[0], h.g0), __fmul_rn(o.m[1], h.g1)), __fmul_rn(o.m[2], h.g2)),
                   __fmul_rn(o.m[3], 0.0f));
    gy = __fadd_rn(__fadd_rn(__fadd_rn(__fmul_rn(o.m[4], h.g0), __fmul_rn(o.m[5], h.g1)), __fmul_rn(o.m[6], h.g2)),
                   __fmul_rn(o.m[7], 0.0f));
    gz = __fadd_rn(__fadd_rn(__fadd_rn(__fmul_rn(o.m[8], h.g0), __fmul_rn(o.m[9], h.g1)), __fmul_rn(o.m[10], h.g2)),
                   __fmul_rn(o.m[11], 0.0f));
    float lpx, lpy, lpz;
    to_local_fast(o, hx, hy, hz, lpx, lpy, lpz);
    uint32_t vi = 0;
    slot = nearest_slot(s, o, lpx, lpy, lpz, vi, lc);
    if (slot < RKF_INTERIOR_SLOT) {
      const size_t v = static_cast<size_t>(slot) * 512 + vi;
      sec = (__ldg(s.mat + v) >> 6) & 0x3Fu;
      blend = __ldg(s.blend + v);
    }
    sdf_hit = h.sdf_hit;  // taken when the motion plane is asked for
  }
  const float l = len3(gx, gy, gz);
  float nx = 0, ny = 1.0f, nz = 0;
  if (!(vox && l < 1e-10f)) {
    nx = __fdiv_rn(gx, l);
    ny = __fdiv_rn(gy, l);
    nz = __fdiv_rn(gz, l);
  }
  if (h.mat_ok || o.sdf_type == RKF_SDF_ANALYTICAL)
    mat = material_at(s, o, __fadd_rn(h.ox, __fmul_rn(safe_dir(h.rdx), h.mat_t)),
                      __fadd_rn(h.oy, __fmul_rn(safe_dir(h.rdy), h.mat_t)),
                      __fadd_rn(h.oz, __fmul_rn(safe_dir(h.rdz), h.mat_t)), lc);
  const size_t i = h.idx;
  sg.t[i] = h.t;
  if (sg.normal) {
    sg.normal[3 * i] = nx;
    sg.normal[3 * i + 1] = ny;
    sg.normal[3 * i + 2] = nz;
  }
  if (sg.slot) sg.slot[i] = slot;
  if (sg.material) sg.material[i] = static_cast<uint16_t>(mat);
  if (sg.flags) sg.flags[i] = flags;
  if (sg.position) reinterpret_cast<float4*>(sg.position)[i] = make_float4(hx, hy, hz, h.t);
  if (sg.packed) sg.packed[i] = (mat & 0x3Fu) | (sec << 6) | (blend << 12) | (o.object_id << 24);
  if (sg.motion) {
    const float* m = sg.prev_vp;  // ray_march.wgsl:1094-1105
    const float cx = __fadd_rn(__fadd_rn(__fadd_rn(__fmul_rn(m[0], hx), __fmul_rn(m[4], hy)), __fmul_rn(m[8], hz)),
                               __fmul_rn(m[12], 1.0f));
    const float cy = __fadd_rn(__fadd_rn(__fadd_rn(__fmul_rn(m[1], hx), __fmul_rn(m[5], hy)), __fmul_rn(m[9], hz)),
                               __fmul_rn(m[13], 1.0f));
    const float cw = __fadd_rn(__fadd_rn(__fadd_rn(__fmul_rn(m[3], hx), __fmul_rn(m[7], hy)), __fmul_rn(m[11], hz)),
                               __fmul_rn(m[15], 1.0f));
    float mox = 0.f, moy = 0.f;
    if (cw > 0.0f) {
      const float ndx = __fdiv_rn(cx, cw), ndy = __fdiv_rn(cy, cw);
      const float pu = __fadd_rn(__fmul_rn(ndx, 0.5f), 0.5f);
      const float pv = __fsub_rn(0.5f, __fmul_rn(ndy, 0.5f));
      const uint32_t px = h.idx % sg.w, py = h.idx / sg.w;
      const float cu = __fdiv_rn(__fadd_rn(static_cast<float>(px), 0.5f), static_cast<float>(sg.w));
      const float cv = __fdiv_rn(__fadd_rn(static_cast<float>(py), 0.5f), static_cast<float>(sg.h));
      mox = __fsub_rn(cu, pu);
      moy = __fsub_rn(cv, pv);
    }
    reinterpret_cast<float4*>(sg.motion)[i] = make_float4(mox, moy, 1.0f, sdf_hit);
  }
}

// The outputs of a ray that ends at its first check, unhit, with no step
// taken (its tmax is below its starting t): what the epilogue writes for it.
__device__ __noinline__ void write_unmarched(const Segment& sg, uint32_t idx, uint32_t mode,
                                             const rkf_march_params& p) {
  if (mode == RKF_TRACE_SHADOW) {
    sg.t[idx] = 1.0f;  // clampf(1, 0, 1)
    if (sg.flags) sg.flags[idx] = 0;
    return;
  }
  const uint16_t flags = (0u >= p.hard_max_steps || 0u >= p.scene.max_steps) ? RKF_FLAG_STEPS_OUT : 0;
  if (mode == RKF_TRACE_ANY) {
    sg.t[idx] = kMaxFloat;
    if (sg.flags) sg.flags[idx] = flags;
    return;
  }
  write_miss(sg, idx, flags);
}

// The march kernel is bound by issue slots and by instruction fetch: its lanes
// are in different phases of their rays (walking ahead, running over EMPTY
// samples, evaluating a sample, done), what one lane does the other lanes of
// its warp wait for, and every phase's code has to come through the
// instruction cache.  So a warp takes one phase at a time, the one that most of
// its lanes are ready for, and hands out new rays as soon as kRefillLanes of its
// lanes are done.  All samples of a ray -- its steps, its bisection, its normal
// -- go through the one evaluation phase, so the kernel holds one copy of the
// sampler: 76 KB of code instead of 209 KB.  1920x1080 over the 1.1M-brick
// scene: 1.45 ms for the kernel that took the phases in lockstep, 0.99 ms with
// the settling passes (settle.cu) before this one.
//
// Measured choices (us: that view / 960x540 of the same scene / 4 views of it
// with their shadow and occlusion rays / 256x256, f32, of the 32 m scene):
//   new rays at 16 lanes done 990 / 605 / 3,300 / 417, at 20 986 / 601 / 3,286 /
//   412, at 24 989 / 596 / 3,235 / 413; waiting for all 32: 1,390 and more.
//   3 blocks an SM 986 / 601 / 3,286 / 412, 4 (64 registers, which spill)
//   1,062 / 659 / 3,112 / 431, 2 1,007 / 547 / 3,659 / 432.
//   A walk that brought no run of kShortRun EMPTY steps puts the next one off by
//   kPutOff: 8 and 8 1,069 / 659 / 3,165 / 426, no putting off 1,157 / 675 /
//   3,691 / 425, 16 and 16 1,092 / 654 / 3,173 / 432 (with 4 blocks).
// The variants of several objects and of the tiled strategy hold more state, and
// spill at 4 blocks, but in large views have more samples to wait for (1920x1080 of the 1.1M-brick
// scene plus 3 voxelized objects and 2 others, brute / tiled / BVH, ms: 4 blocks 6.9 /
// 7.4 / 7.9, 3 7.8 / 8.0 / 8.3, 2 7.9 / 8.4 / 9.0, 5 7.9 / 7.7 / 8.2; plus 9 others 4.66 / 4.81 /
// 5.65, 5.10 / 5.02 / 5.57, 5.23 / 4.94 / 6.01, 5.63 / 5.28 / 5.70).  In smaller views the longest
// rays decide: of the latter 400x225 1.85 / 1.43 / 1.94 with 4, 1.60 / 1.08 / 1.68 with 2, and
// 960x540 2.53 / 2.25 / 2.63 with 4, 2.39 / 2.16 / 2.62 with 2.  Their plain kin run 4 (u8,
// 1920x1080 of the 32 m scene: 1.64 ms with 4 against 1.85 with 5 and 1.73 with 3).
constexpr uint32_t kRefillLanes = 24;
constexpr float kShortRun = 8.0f, kPutOff = 8.0f;  // in EMPTY steps
constexpr uint32_t kLeastLanes = 4;   // lanes a warp fills however few rays there are
constexpr uint64_t kManyIds = 1u << 20;  // work ids of views that count as many
constexpr int march_blocks(int obj, bool many) {
  return obj == OBJ_SINGLE_EMPTY ? 3 : obj > OBJ_SINGLE_EMPTY && !many ? 2 : 4;
}
// How a warp is paced: the lanes done before new rays, and the samples a lane takes in
// one phase (on while half of those that began do).  Without the EMPTY path nearly
// every lane samples, and a warp does best to stay with it: one rotated object,
// 1920x1080 of the 32 m scene, f16 / u8, 2.02 / 1.77 ms at 16 lanes and 8 samples, 1.77 / 1.59
// at 28 and 128; the scene and four more objects, brute / tiled / BVH, 3.30 / 2.57 / 4.88 ms
// to 3.00 / 2.25 / 4.43 at 28 and 16 to 128.  Of several objects the rays that the settling
// passes left (listed) go best at 16 lanes: 2.42 ms, at 28 lanes 2.49.
constexpr uint32_t march_refill(int obj, bool listed) {
  return obj != OBJ_MULTI && obj != OBJ_SINGLE ? kRefillLanes : obj == OBJ_MULTI && listed ? 16u : 28u;
}
constexpr uint32_t eval_reps(int obj) { return obj == OBJ_MULTI ? 16u : obj == OBJ_SINGLE ? 128u : 8u; }
#define kNoBox __int_as_float(0x7fc00000)  // compares false with every time

// A warp's lanes' share of the ids left to hand out.
__device__ __forceinline__ uint32_t lane_share(uint64_t total, uint64_t handed, uint32_t warps) {
  const uint64_t left = total > handed ? total - handed : 0u;
  if (left >= static_cast<uint64_t>(warps) * 32u) return 32u;
  return max((static_cast<uint32_t>(left) + warps - 1u) / warps, kLeastLanes);
}

template <int PREC, int OBJ, bool TREE, bool MANY>
__global__ void __launch_bounds__(256, march_blocks(OBJ, MANY)) k_march_persistent(const __grid_constant__ KParams kp) {
  constexpr bool MULTI_TILED = OBJ == OBJ_MULTI_EMPTY_TILED;
  constexpr bool MULTI_EMPTY = OBJ == OBJ_MULTI_EMPTY || MULTI_TILED;
  constexpr bool SINGLE = OBJ != OBJ_MULTI && !MULTI_EMPTY;
  constexpr bool EMPTY_PATH = OBJ == OBJ_SINGLE_EMPTY || OBJ == OBJ_SINGLE_EMPTY_TILED || MULTI_EMPTY;
  constexpr bool PLAIN_VOX = OBJ == OBJ_SINGLE_EMPTY || OBJ == OBJ_SINGLE_EMPTY_TILED;
  // tile bookkeeping of tiled launches
  constexpr bool TILES = OBJ != OBJ_SINGLE_EMPTY && OBJ != OBJ_MULTI_EMPTY;
  // the object table: the launch parameters hold up to kMaxObjectsFast
  // records; a larger scene (the plain multi-object variant only) reads the
  // device copy
  const ObjDev* sh_objs = (OBJ == OBJ_MULTI && kp.s.n_objs > kMaxObjectsFast) ? kp.s.objs : kp.objs;
  const SceneDev& s = kp.s;
  const rkf_march_params& p = kp.p;
  const uint32_t lane = threadIdx.x & 31;
  const uint32_t nobj = s.n_objs;
  const float hit_thr = p.scene.hit_threshold;

  LaneCache lc;
  uint32_t state = ST_IDLE;
  uint32_t mode = RKF_TRACE_CLOSEST;
  // state a lane touches only when a ray starts, hits or ends lives in shared
  // memory, which keeps the march loop's register footprint small
  __shared__ ColdState cold_all[256];
  ColdState& cs = cold_all[threadIdx.x];
  float ox = 0, oy = 0, oz = 0, rdx = 0, rdy = 0, rdz = 0;
  float t = 0, prev_t = 0, prev_dist = kMaxFloat, tmax = 0;
  // empty-space path: positions up to here sample the EMPTY value (kNoBox: none)
  float box_t = kNoBox;
  float far_t = -1.0f;   // multi-object empty-space path: positions up to here lie outside every ball
  float probe_t = 0.0f;  // empty-space path: no walk before this t
  uint32_t near = 0, step = 0;
  uint32_t since = 0;  // phases since the warp last took new rays
  // Lanes a warp fills: all of them while there is work for every warp's, else
  // its share of what is left, so that a small launch, and the end of a large
  // one, spreads its rays over the chip's warps instead of packing 32 rays in
  // different phases into each of a few.
  const uint32_t n_list = kp.list ? __ldg(kp.list_n) : 0u;
  const uint64_t total = kp.list ? kp.total - kp.view_ids + n_list : kp.total;
  uint32_t lanes = lane_share(total, 0, gridDim.x * (blockDim.x >> 5));
  bool exhausted = false;

  for (;;) {
    const bool march = state == ST_MARCH || state == ST_SHADOW;
    // the march steps along the safe direction (ray_march.wgsl:784); hit
    // positions use the raw direction (:1068), as shadow rays do
    const bool sh = state == ST_SHADOW;
    const float dx = sh ? rdx : safe_dir(rdx), dy = sh ? rdy : safe_dir(rdy), dz = sh ? rdz : safe_dir(rdz);
    // what ends a ray, and what its samples are compared with: a sample below
    // brk is decided by the evaluation phase
    const uint32_t max_step = sh ? 256u : p.hard_max_steps;
    const uint32_t max_near = sh ? 32u : p.scene.max_steps;
    const float brk = sh ? 0.02f : fmaxf(hit_thr, 0.0f);
    const float near_thr = sh ? -1.0f : p.near_surface_threshold;
    const float min_step = sh ? 0.005f : p.min_step;

    // ---- the phase most lanes are ready for -----------------------------------
    const bool run = EMPTY_PATH && march && t <= box_t;
    const bool walk = EMPTY_PATH && march && !run && t >= probe_t && prev_dist >= kp.probe_min;
    const bool done = state == ST_IDLE || state == ST_EPI;
    const uint32_t n_done = __popc(__ballot_sync(kFull, done));
    const uint32_t n_walk = EMPTY_PATH ? __popc(__ballot_sync(kFull, walk)) : 0u;
    const uint32_t n_run = EMPTY_PATH ? __popc(__ballot_sync(kFull, run)) : 0u;
    const uint32_t n_eval = 32u - n_done - n_walk - n_run;
    ++since;

    if (n_done == 32u || (!exhausted && (n_done >= kp.refill_idle + 32u - lanes ||
                                         (n_done > 32u - lanes && since >= kp.interval)))) {
      // ---- outputs of finished rays --------------------------------------------
      if (state == ST_EPI) {
        const Segment& sg = kp.segs[cs.seg];
        if (mode == RKF_TRACE_SHADOW) {
          sg.t[cs.idx] = clampf(cs.shadow, 0.0f, 1.0f);
          if (sg.flags) sg.flags[cs.idx] = cs.hit ? RKF_FLAG_HIT : 0;
        } else if (mode == RKF_TRACE_ANY) {
          sg.t[cs.idx] = cs.hit ? t : kMaxFloat;
          if (sg.flags)
            sg.flags[cs.idx] = cs.hit ? RKF_FLAG_HIT
                                : ((step >= p.hard_max_steps || near >= p.scene.max_steps) ? RKF_FLAG_STEPS_OUT : 0);
        } else {
          if (!cs.hit) {
            write_miss(sg, cs.idx,
                       step >= p.hard_max_steps || near >= p.scene.max_steps ? RKF_FLAG_STEPS_OUT : uint16_t(0));
          } else {
            const HitRay h{ox, oy, oz, rdx, rdy, rdz, t, cs.mat_t, cs.g[0], cs.g[1], cs.g[2], cs.sdf_hit,
                           cs.idx, cs.bisected, cs.mat_ok};
            write_hit(s, sh_objs[cs.hit_obj], sg, h);
          }
        }
        state = ST_IDLE;
      }
      if (exhausted) break;  // every lane is done and no work is left
      since = 0;
      // ---- new rays for the idle lanes -------------------------------------------
      // A ray that ends before its first sample (tmax below its starting t:
      // the secondary rays of pixels that missed) takes its outputs here and
      // its lane takes the next id at once, for up to kRefillRounds rounds, so
      // that such rays do not leave lanes idle through the march loop.
      for (uint32_t round = 0; round < kRefillRounds; ++round) {
        const bool idle = state == ST_IDLE;
        uint32_t need = __ballot_sync(kFull, idle);
        // (the first of the idle lanes, up to the warp's share)
        const uint32_t busy = 32u - __popc(need);
        const uint32_t room = lanes > busy ? lanes - busy : 0u;
        const bool take = idle && __popc(need & ((1u << lane) - 1u)) < room;
        need = __ballot_sync(kFull, take);
        bool again = false;  // this lane's id ended at once (or is off the view)
        if (need && !exhausted) {
          const uint32_t leader = __ffs(need) - 1;
          unsigned long long base = 0;
          if (lane == leader) base = atomicAdd(kp.counter, static_cast<unsigned long long>(__popc(need)));
          base = __shfl_sync(kFull, base, leader);
          if (base + __popc(need) >= total) exhausted = true;
          lanes = lane_share(total, base + __popc(need), gridDim.x * (blockDim.x >> 5));
          if (take) {
            const uint64_t k = base + __popc(need & ((1u << lane) - 1u));
            if (k < total) {
              // the rays the settling passes left, then the ray batches
              const bool listed = kp.list && k < n_list;
              const uint2 entry = listed ? __ldg(kp.list + k) : make_uint2(0u, 0x7fc00000u);
              const uint64_t id = listed ? entry.x : kp.list ? kp.view_ids + (k - n_list) : kp.id0 + k;
              cs.seg = find_segment(kp.segs, kp.nseg, id);
              const Segment& sg = kp.segs[cs.seg];
              const uint64_t local = id - sg.first;
              bool valid = true;
              if (sg.kind == 0) {  // view: tile-ordered pixel ids
                const uint32_t per = kp.tile_w * kp.tile_h;
                // (32-bit division where the view's ids fit it)
                uint32_t tile = (sg.n_ids >> 32) ? static_cast<uint32_t>(local / per) : static_cast<uint32_t>(local) / per;
                const uint32_t r = static_cast<uint32_t>(local - static_cast<uint64_t>(tile) * per);
                if (sg.tile_perm) tile = __ldg(sg.tile_perm + tile);  // heaviest-first order
                const uint32_t px = (tile % sg.tiles_x) * kp.tile_w + r % kp.tile_w;
                const uint32_t py = (tile / sg.tiles_x) * kp.tile_h + r / kp.tile_w;
                valid = px < sg.w && py < sg.h;
                if (valid) {
                  cs.idx = py * sg.w + px;
                  view_ray(sg, px, py, rdx, rdy, rdz);
                  ox = sg.pos[0];
                  oy = sg.pos[1];
                  oz = sg.pos[2];
                  tmax = p.scene.max_distance;
                  mode = RKF_TRACE_CLOSEST;
                  if (TILES) {
                    cs.tile_count = kNoTiles;
                    if (kp.tiled) {  // the pixel's tile (ray_march.wgsl:884-893)
                      const uint32_t tl = sg.tile_off + (py / 16) * ((sg.w + 15) / 16) + px / 16;
                      cs.tile_base = tl * kTileObjects;
                      cs.tile_count = __ldg(kp.td.tile_cnt + tl);
                    }
                    if (MULTI_TILED) {
                      uint32_t listed = 0;
                      for (uint32_t e = 0; e < kp.n_ev; ++e) {
                        bool in = cs.tile_count == kNoTiles;
                        for (uint32_t j = 0; !in && j < cs.tile_count; ++j)
                          in = __ldg(kp.td.tile_list + cs.tile_base + j) == kp.ev[e].obj;
                        if (in) listed |= 1u << e;
                      }
                      cs.vox_listed = listed;
                    }
                  }
                }
              } else {
                if (TILES) cs.tile_count = kNoTiles;
                if (MULTI_TILED) cs.vox_listed = (1u << kp.n_ev) - 1u;
                cs.idx = static_cast<uint32_t>(local);
                const size_t i3 = 3 * static_cast<size_t>(cs.idx);
                tmax = __ldg(sg.tmax + cs.idx);
                mode = sg.mode;
                ox = __ldg(sg.origins + i3);
                oy = __ldg(sg.origins + i3 + 1);
                oz = __ldg(sg.origins + i3 + 2);
                rdx = __ldg(sg.dirs + i3);
                rdy = __ldg(sg.dirs + i3 + 1);
                rdz = __ldg(sg.dirs + i3 + 2);
              }
              if (valid) {
                near = 0;
                step = 0;
                box_t = __uint_as_float(entry.y);  // how far the settling pass saw EMPTY samples
                probe_t = box_t == box_t ? after(0.0f) : 0.0f;
                if (MULTI_EMPTY) {
                  far_t = -1.0f;
                  // (the normal's until then: no settling attempt before this t,
                  // and the first ball ahead)
                  cs.gpos = box_t == box_t ? box_t : 0.0f;
                  cs.g[0] = -1.0f;
                  cs.g[1] = 2.0f * kp.empty_hi;
                  box_t = kNoBox;
                  probe_t = 0.0f;
                  if (!MULTI_TILED) cs.vox_listed = (1u << kp.n_ev) - 1u;
                }
                prev_dist = kMaxFloat;
                cs.hit = cs.bisected = cs.mat_ok = false;
                if (mode == RKF_TRACE_SHADOW) {
                  t = 0.005f;  // SHADOW_EPSILON (shade_common.wgsl:274)
                  cs.shadow = 1.0f;
                  state = ST_SHADOW;
                } else {
                  t = 0.0f;
                  prev_t = 0.0f;
                  // a tile with no objects is sky (ray_march.wgsl:895-897); a
                  // step limit of 0 ends the ray at its first check
                  state = ((TILES && cs.tile_count == 0) || p.scene.max_steps == 0 || p.hard_max_steps == 0)
                              ? ST_EPI : ST_MARCH;
                }
                if (state != ST_EPI && t > tmax) {
                  // its first check ends it unhit with no step taken: the
                  // epilogue's outputs for that (shadow 1; t max, normal 0,
                  // EMPTY slot, material 0, the miss position and motion)
                  write_unmarched(sg, cs.idx, mode, p);
                  state = ST_IDLE;
                  again = true;
                }
              } else {
                again = true;
              }
            }
          }
        }
        if (!__any_sync(kFull, again)) break;
      }
      continue;
    }

    if (EMPTY_PATH && n_walk && n_walk >= n_run && n_walk >= n_eval) {
      // ---- walk: where the samples ahead are known to be EMPTY -------------------
      // A lane whose last sample was (close to) the EMPTY value walks its ray
      // ahead through EMPTY boxes.  If every sample the ray has left is at
      // least the EMPTY value and that clears every threshold, no decision is
      // left to take: the ray misses, its outputs do not depend on its exact t,
      // and it is settled here.  Otherwise the walk's end bounds the run.
      if (walk) {
        uint32_t outcome = 0;  // 1: ends past tmax; 2: runs out of steps
        // The last sample is the (max_step-step-1)th ahead: the ray ends past
        // tmax (with no step flag) if even its smallest t exceeds tmax by then,
        // and runs out of steps if even its largest t stays <= tmax.
        const float k = static_cast<float>(max_step - step - 1);
        const float grow = steps_grow(k);
        const float t_lo = (t + k * kp.empty_lo_t) * (1.0f - grow);
        const float t_hi = (t + k * kp.empty_hi) * (1.0f + grow);
        const bool can = kp.empty_lo >= brk && kp.empty_lo >= near_thr && kp.empty_lo >= min_step;
        if (!MULTI_EMPTY) {
          const ObjDev& o = sh_objs[0];
          const ProbeRay r = probe_ray(o, ox, oy, oz, dx, dy, dz);
          float t_in, t_out;
          const bool core = core_interval(o, r, t, t_in, t_out);
          const float run_end = core ? t_out : -1.0f;
          float target = run_end;
          uint32_t ends = 0;  // the outcome if the walk reaches its target
          if (can) {
            if (t_lo > tmax) {
              ends = 1;
              target = tmax;
            } else if (t_hi <= tmax && core && t_out >= t_hi) {
              ends = 2;
              target = t_hi;
            } else if (OBJ == OBJ_SINGLE_EMPTY) {
              ends = leaves_grid(o, r, t, tmax, core, t_out, k, kp.empty_lo_t, kp.empty_hi);
              if (ends) target = tmax;
            }
          }
          // outside: nothing to walk for before the ray enters
          probe_t = core || (t_in < t_out && t < t_out && !(t_in > t)) ? after(t)
                    : t_in < t_out && t_in > t ? t_in : after(INFINITY);
          // a tiled step is a coarse skip of more than 0.5 (empty_lo_t is at
          // most that) or evaluates the object: the brute field bounds the
          // ray's samples from below, the tiled one gives their value
          const bool brute = OBJ == OBJ_SINGLE_EMPTY || ends == 1u;
          float end = -1.0f;
          if (target >= t) end = walk_empty(o, s, brute ? kp.brute_field : s.empty_dist, brute, r, t, target, kWalkLinks);
          if (end >= target) outcome = ends;
          if (OBJ == OBJ_SINGLE_EMPTY_TILED && ends == 1u && !outcome) {
            // not settled: the tiled field's walk, for a run
            end = run_end >= t ? walk_empty(o, s, s.empty_dist, false, r, t, run_end, kWalkLinks) : -1.0f;
          }
          box_t = end >= t && run_end >= t ? fminf(end, run_end) : kNoBox;
          // a walk that brought no run of some length puts the next one off
          const float from = box_t == box_t ? box_t : t;
          if (probe_t == probe_t && from - t < kShortRun * kp.empty_hi)
            probe_t = fmaxf(probe_t, from + kPutOff * kp.empty_hi);
        } else {
          box_t = kNoBox;
          probe_t = after(t);
          const uint32_t all = (1u << kp.n_ev) - 1u;
          // ---- how far every object off the path keeps its distance: the first
          // entry into the ball (box, half-space) of one ahead.  It stays valid
          // until the ray passes it: balls ahead stay ahead, balls behind stay
          // behind.  A ray that may be inside one takes full steps until it may
          // have left.
          float far_all = cs.g[0];
          if (t > far_all) {
            float again;
            far_all = far_limit(kp.ball, kp.n_ball, all, ox, oy, oz, dx, dy, dz, tmax, t, 0.0f, again);
            cs.g[0] = far_all < 0.0f ? -1.0f : far_all;
            if (far_all < 0.0f && again > t) probe_t = again;
          }
          // ---- settle: no object below its EMPTY value or ball bound ahead.  Under
          // the tiled strategy running out of steps needs the exact EMPTY value
          // of an object every step evaluates: one the tile lists, on the field of
          // blocks no coarse skip can reach; what it does not list is not evaluated.
          const bool past = t_lo > tmax;
          const bool masked = MULTI_TILED && !past;
          const float target = past ? tmax : t_hi;
          bool exact = past, ok = can && t >= cs.gpos && far_all >= target &&
                                  (past || (t_hi <= tmax && (!MULTI_TILED || (cs.vox_listed & 0xFFu) != 0u)));
          const bool tried = ok;
          // ---- run: the set of voxelized objects of the path (that the ray may
          // take runs on) whose EMPTY boxes hold the ray; the run lasts while it
          // is in all of them, and outside every ball: no walk goes on beyond
          uint32_t set = 0;
          float b = kMaxFloat, walk_at = cs.gpos > t ? cs.gpos : after(INFINITY);  // when to walk again
          for (uint32_t e = 0; e < kp.n_ev && far_all >= 0.0f; ++e) {
            const bool listed = (cs.vox_listed >> e) & 1u;
            if (!listed && (!ok || masked)) continue;
            const ObjDev& o = sh_objs[kp.ev[e].obj];
            const ProbeRay r = probe_ray(o, ox, oy, oz, dx, dy, dz);
            float t_in, t_out;
            const bool core = core_interval(o, r, t, t_in, t_out);
            if (listed && core) walk_at = after(t);
            else if (listed && t_in < t_out && t < t_out) walk_at = fminf(walk_at, fmaxf(t_in, after(t)));
            float end = -1.0f;
            // (the tiled strategy's runs need its own field)
            for (uint32_t pass = ok ? 0u : 1u; pass < 2u; ++pass) {
              const bool own = pass || masked;
              if (pass && !(listed && core)) break;
              end = walk_empty(o, s, own ? s.empty_dist : kp.brute_field, !MULTI_TILED || !own, r, t,
                               pass ? fminf(fminf(t_out, b), far_all) : target, kWalkLinks);
              if (!pass) {
                ok = end >= target;
                exact = exact || (core && t_out >= target);
                if (!ok) cs.gpos = fmaxf(end, after(t));
                if (!MULTI_TILED || ok) break;  // (the brute strategy runs on the same field)
              }
            }
            const float bt = listed && core ? fminf(t_out, end) : -1.0f;
            if (t <= bt) {
              set |= 1u << e;
              b = fminf(b, bt);
            }
          }
          if (tried && ok && exact) {
            outcome = past ? 1u : 2u;
          } else if (far_all >= 0.0f) {
            if (!(walk_at > after(t)) && walk_at == walk_at) walk_at = after(t);
            probe_t = walk_at;
            if (set) {
              if (set != (cs.vox_listed >> 8)) {
                // other objects in the set: the balls that bound the run are others
                cs.vox_listed = (cs.vox_listed & 0xFFu) | (set << 8);
                far_t = -1.0f;
              }
              // only positions outside the balls of every object not in the
              // set sample the set's EMPTY values
              if (set == all) {
                far_t = far_all;
              } else if (t > far_t) {
                float again;
                far_t = far_limit(kp.ball, kp.n_ball, set, ox, oy, oz, dx, dy, dz, tmax, t, 0.0f, again);
                if (far_t < 0.0f && again > t) probe_t = again;
              }
              box_t = far_t >= t ? fminf(b, far_t) : kNoBox;
            }
            // a walk that brought no run of some length puts the next one off
            const float from = box_t == box_t ? box_t : t;
            const float back = from - t >= 8.0f * kp.empty_hi ? 2.0f * kp.empty_hi
                                                              : fminf(2.0f * cs.g[1], 16.0f * kp.empty_hi);
            cs.g[1] = back;
            if (probe_t == probe_t) probe_t = fmaxf(probe_t, from + back);
          }
        }
        if (outcome) {
          if (!sh && outcome == 2) step = max_step;
          state = ST_EPI;
        }
      }
      continue;
    }

    if (EMPTY_PATH && n_run && n_run >= n_eval) {
      // ---- run: up to kp.budget steps over EMPTY samples, without the sampler ------
      if (run) {
        // several objects: the set's EMPTY values (of one object, its constants)
        const uint32_t set = MULTI_EMPTY ? (cs.vox_listed >> 8) : 1u;
        const bool one = (set & (set - 1u)) == 0u;
        const EmptyVox& ev = kp.ev[MULTI_EMPTY && set ? (__ffs(set) - 1) : 0];  // (the one of a set of one)
        const ObjDev& o0 = sh_objs[MULTI_EMPTY ? ev.obj : 0u];
        const uint32_t plain = MULTI_EMPTY ? (one ? ev.plain : 0u) : kp.plain_obj;
        // (the path's least lower bound: no set's is below it)
        const bool clean = kp.empty_lo >= brk && kp.empty_lo >= near_thr && kp.empty_lo >= min_step;
        const uint32_t n = min(kp.budget, max_step - step);
        uint32_t c = 0;
        bool stop_full = true;
        if (MULTI_EMPTY && !one) {
          // several objects: the least of their EMPTY values, to the end of
          // the nearest cube
          c = clean ? empty_run_set<true>(sh_objs, kp.ev, set, kp.n_ev, ox, oy, oz, dx, dy, dz, tmax, n, brk,
                                          near_thr, min_step, max_near, t, box_t, prev_t, prev_dist, near, stop_full)
                    : empty_run_set<false>(sh_objs, kp.ev, set, kp.n_ev, ox, oy, oz, dx, dy, dz, tmax, n, brk,
                                           near_thr, min_step, max_near, t, box_t, prev_t, prev_dist, near,
                                           stop_full);
        } else if (plain && clean) {
          c = empty_run_x2(o0, ox, oy, oz, dx, dy, dz, tmax, n, t, box_t, prev_t, prev_dist, stop_full);
        } else if (plain) {
          c = empty_run<true>(o0, ox, oy, oz, dx, dy, dz, tmax, n, brk, near_thr, min_step, max_near, t, box_t,
                              prev_t, prev_dist, near, stop_full);
        } else {
          c = empty_run<false>(o0, ox, oy, oz, dx, dy, dz, tmax, n, brk, near_thr, min_step, max_near, t, box_t,
                               prev_t, prev_dist, near, stop_full);
        }
        step += c;
        if (step >= max_step || t > tmax || near >= max_near) {
          state = ST_EPI;
        } else if (stop_full || t > box_t) {
          // past the covered interval (or at a sample a threshold acts on)
          // comes an evaluated step
          box_t = kNoBox;
          probe_t = after(t);
        }
      }
      continue;
    }

    // ---- eval: a sample of each lane that needs one, and on while most do --------
    bool eval = !done && !walk && !run;
#pragma unroll 1
    for (uint32_t rep = 0; rep < eval_reps(OBJ); ++rep) {
    if (eval) {
      if (state == ST_BISECT && cs.sub >= p.bisect_steps) {
        // bisection done (or a direct hit): t = (lo+hi)/2, on to the normal
        if (cs.bisected) t = __fmul_rn(__fadd_rn(cs.lo, cs.hi), 0.5f);
        cs.sub = 0;
        state = ST_NORMAL;
      }
      float best = kMaxFloat, best_un = kMaxFloat;
      uint32_t best_i = 0;
      bool skipped = false;
      float px, py, pz;       // the position: world space, or object-local for a voxelized object's normal
      bool local = false;     // px..pz are object-local
      bool grad = false;      // the gradient's sampler
      bool only = false;      // the hit object alone, whatever its value
      uint32_t jb = 0, je = SINGLE ? 1u : nobj;
      if (state == ST_NORMAL) {
        px = __fadd_rn(ox, __fmul_rn(rdx, t));
        py = __fadd_rn(oy, __fmul_rn(rdy, t));
        pz = __fadd_rn(oz, __fmul_rn(rdz, t));
        const ObjDev& o = sh_objs[SINGLE ? 0u : cs.hit_obj];
        float eps = __fmul_rn(hit_thr, 10.0f);
        if (PLAIN_VOX || o.sdf_type == RKF_SDF_VOXELIZED) {
          to_local_fast(o, px, py, pz, px, py, pz);
          eps = __fmul_rn(o.vs, 2.0f);
          local = true;
          grad = cs.sub < 6u;  // the 7th sample: the hit's own distance (motion plane)
        }
        const uint32_t ax = cs.sub >> 1;
        if (cs.sub & 1u) eps = -eps;  // x + (-eps) is x - eps
        if (ax == 0) px = __fadd_rn(px, eps);
        if (ax == 1) py = __fadd_rn(py, eps);
        if (ax == 2) pz = __fadd_rn(pz, eps);
        only = true;
      } else {
        const float ts = state == ST_BISECT ? __fmul_rn(__fadd_rn(cs.lo, cs.hi), 0.5f) : t;
        px = __fadd_rn(ox, __fmul_rn(dx, ts));
        py = __fadd_rn(oy, __fmul_rn(dy, ts));
        pz = __fadd_rn(oz, __fmul_rn(dz, ts));
        only = state == ST_BISECT;
      }
      bool list = false;
      if (!SINGLE && only) {
        jb = cs.hit_obj;
        je = jb + 1u;
      }
      if (TILES && kp.tiled && state == ST_MARCH && cs.tile_count != kNoTiles) {
        // ray_march_tiled (:899-938): a coarse empty-space skip, else the
        // tile's objects only
        const Segment& sg = kp.segs[cs.seg];
        const float cd = coarse_sample(kp.td, sg.coarse_ocr, __fsub_rn(px, sg.pos[0]), __fsub_rn(py, sg.pos[1]),
                                       __fsub_rn(pz, sg.pos[2]));
        if (cd > kCoarseNear) {
          prev_dist = kMaxFloat;
          t = __fadd_rn(t, cd);
          step++;
          skipped = true;
          je = 0;
        } else {
          list = true;
          je = cs.tile_count;
        }
      }
      // one object's sample counts whatever its value (a NaN, too)
      const bool take = only || ((SINGLE || (!TREE && nobj == 1u)) && !list);
      const bool tree = TREE && state == ST_MARCH;
      if (tree) jb = 0u;
      for (uint32_t j = jb; tree || j < je; ++j) {
        uint32_t oi = j;
        if (list) oi = __ldg(kp.td.tile_list + cs.tile_base + j);
        if (tree) {  // (j: where the walk of the tree stands)
          oi = bvh_candidate(kp.bvh, kp.bvh_next, nobj, px, py, pz, best, j);
          if (oi == kBvhEnd) break;
          --j;
        }
        const ObjDev& o = sh_objs[SINGLE ? 0u : oi];
        float d = kMaxFloat, du = kMaxFloat;
        if (PLAIN_VOX) {  // one voxelized object, translation only
          const float lx = local ? px : __fadd_rn(px, o.m[12]), ly = local ? py : __fadd_rn(py, o.m[13]),
                      lz = local ? pz : __fadd_rn(pz, o.m[14]);
          du = sample_vox<PREC, true>(s, o, lx, ly, lz, grad, lc);
          d = local ? du : __fmul_rn(du, o.min_scale);
        } else if (o.sdf_type != RKF_SDF_NONE) {
          float lx = px, ly = py, lz = pz;
          if (!local) to_local_fast(o, px, py, pz, lx, ly, lz);
          du = o.sdf_type == RKF_SDF_ANALYTICAL ? analytic_sdf(o, lx, ly, lz)
                                                : sample_vox<PREC>(s, o, lx, ly, lz, grad, lc);
          d = local ? du : __fmul_rn(du, o.min_scale);
        }
        if (take || d < best) {
          best = d;
          best_un = du;
          best_i = oi;
        }
      }
      // ---- what the sample decides ------------------------------------------------
      if (state == ST_MARCH) {
        if (skipped) {
        } else if (best < 0.0f && prev_dist > hit_thr) {  // overstep (ray_march.wgsl:816)
          cs.hit_obj = best_i;
          cs.hit = true;
          cs.lo = prev_t;
          cs.hi = t;
          cs.mat_t = t;
          cs.mat_ok = best_un < sh_objs[best_i].vs16;
          cs.sub = 0;
          cs.bisected = true;
          state = mode == RKF_TRACE_ANY ? ST_EPI : ST_BISECT;
        } else if (best < hit_thr) {  // :842
          // a direct hit: the bisection is done
          cs.hit_obj = best_i;
          cs.hit = true;
          cs.mat_t = t;
          cs.mat_ok = best_un < sh_objs[best_i].vs16;
          cs.sub = p.bisect_steps;
          state = mode == RKF_TRACE_ANY ? ST_EPI : ST_BISECT;
        } else {
          if (best < p.near_surface_threshold) near++;
          prev_t = t;
          prev_dist = best;
          t = __fadd_rn(t, fmax_(best, p.min_step));
          step++;
        }
        if (state == ST_MARCH && (step >= p.hard_max_steps || t > tmax || near >= p.scene.max_steps)) state = ST_EPI;
      } else if (state == ST_SHADOW) {
        // soft_shadow (shade_common_shading.wgsl:9-33)
        prev_dist = best;
        if (best < 0.005f) {
          cs.shadow = 0.0f;
          cs.hit = true;
          state = ST_EPI;
        } else {
          if (best < 0.02f) {
            cs.shadow = fmin_(cs.shadow, __fdiv_rn(__fmul_rn(16.0f, best), t));
            near++;
          }
          t = __fadd_rn(t, fmax_(best, 0.005f));
          step++;
          if (step >= 256u || near >= 32u || t > tmax) state = ST_EPI;
        }
      } else if (state == ST_BISECT) {
        const float mid = __fmul_rn(__fadd_rn(cs.lo, cs.hi), 0.5f);
        if (best < 0.0f) {
          cs.hi = mid;
        } else {
          cs.lo = mid;
          cs.mat_t = mid;
          cs.mat_ok = best_un < sh_objs[SINGLE ? 0u : cs.hit_obj].vs16;
        }
        ++cs.sub;
      } else {  // ST_NORMAL
        const uint32_t sub = cs.sub;
        if (sub >= 6u) {
          cs.sdf_hit = best;
          state = ST_EPI;
        } else if (sub & 1u) {
          cs.g[sub >> 1] = __fsub_rn(cs.gpos, best);
          if (sub == 5u && !(local && kp.segs[cs.seg].motion)) state = ST_EPI;
        } else {
          cs.gpos = best;
        }
        cs.sub = sub + 1u;
      }
      eval = state == ST_BISECT || state == ST_NORMAL ||
             ((state == ST_MARCH || state == ST_SHADOW) &&
              !(EMPTY_PATH && t >= probe_t && prev_dist >= kp.probe_min));
    }
    if (2 * __popc(__ballot_sync(kFull, eval)) < n_eval) break;
    }
  }
}

// Where a kernel reads the object table: the launch parameters (a scene of one
// object), a copy in shared memory (up to kMaxObjectsShared records, a word a
// thread: a record a thread cost a block of a small scene as long as a sample), or
// the device table.
enum : int { TABLE_ONE = 0, TABLE_SHARED = 1, TABLE_DEVICE = 2 };
template <int TABLE>
struct TableArg {};
template <>
struct TableArg<TABLE_ONE> {
  ObjSample one;
};
template <int TABLE>
__device__ __forceinline__ void load_table(ObjSample* sh, const SceneDev& s) {
  if (TABLE != TABLE_SHARED) return;
  constexpr uint32_t kWords = sizeof(ObjSample) / 4, kStride = sizeof(ObjDev) / 4;
  static_assert(sizeof(ObjSample) % 4 == 0 && sizeof(ObjDev) % 4 == 0, "whole words");
  const uint32_t* src = reinterpret_cast<const uint32_t*>(s.objs);
  uint32_t* dst = reinterpret_cast<uint32_t*>(sh);
  for (uint32_t i = threadIdx.x; i < s.n_objs * kWords; i += blockDim.x)
    dst[i] = __ldg(src + i / kWords * kStride + i % kWords);
  __syncthreads();
}

constexpr uint32_t kPointLanes = 8;
constexpr uint32_t kAoLanes = 4;  // one per tap

// SdfQueryable::evaluate / gradient over the pool, eight lanes a point: each
// evaluates its share of the objects, then six of them one sample of the
// gradient each -- of a single object beside the seventh's sample of the point
// itself.  All samples go through one copy of the evaluator.  A thread per point
// took its 7 samples one after the other, through a copy each (246 KB of code):
// bound by instruction fetch and by that chain, 54 us for 300 points near
// surfaces (20 so) and, as a call, 72 us for 65,536 over the 1.1M-brick scene (56
// so; there the bound is the samples' loads).
// A block serves 16 points, and with more than kPointFewObjects objects a copy of
// the table for these costs more than reading the device table, which the
// first-level cache holds: 65,536 points, 60 / 100 / 163 / 198 objects: 80 / 98 / 120 /
// 133 us so, 89 / 123 / 226 / 282 with the copy (a thread per point, 128 to a copy: 97 /
// 115 / 139 / 144); 2 / 5 / 8 / 12 / 24 objects: 56.2 / 57.2 / 57.1 / 60.3 / 63.8
// against 53.9 / 56.0 / 56.3 / 60.3 / 65.9.  One object from the launch parameters:
// 49 us for the 65,536 over the 1.1M-brick scene, 57 with the copy.
constexpr uint32_t kPointFewObjects = 12;
template <int PREC, int TABLE, uint32_t LANES>
__global__ void __launch_bounds__(128) k_query_points(SceneDev s, const __grid_constant__ TableArg<TABLE> arg,
                                                     const float* __restrict__ pts, uint32_t n, float* dist,
                                                     float* grad, uint16_t* material) {
  extern __shared__ ObjSample sh_objs[];
  load_table<TABLE>(sh_objs, s);
  const ObjDev* const table = s.objs;
  const auto object = [&](uint32_t k) -> const ObjSample& {
    if constexpr (TABLE == TABLE_ONE) return arg.one;
    else if constexpr (TABLE == TABLE_SHARED) return sh_objs[k];
    else return table[k];
  };
  const uint32_t id = blockIdx.x * (blockDim.x / LANES) + threadIdx.x / LANES;
  const uint32_t j = threadIdx.x % LANES;
  const uint32_t i = min(id, n - 1);  // (every lane takes part in the exchange)
  LaneCache lc;
  const float px = pts[3 * static_cast<size_t>(i)], py = pts[3 * static_cast<size_t>(i) + 1],
              pz = pts[3 * static_cast<size_t>(i) + 2];
  float best = kMaxFloat, best_un = kMaxFloat, g = 0.0f;
  uint32_t bi = 0;
  const bool taps = LANES > 1u && grad != nullptr;  // (a thread per point takes none)
  const bool diff = taps && j < 6u;
  const uint32_t n_objs = TABLE == TABLE_ONE ? 1u : s.n_objs;
  const uint32_t rounds = (n_objs + LANES - 1u) / LANES;
#pragma unroll 1
  for (uint32_t r = 0; r <= rounds; ++r) {
    if (r == rounds) {
      // the point's object: the smallest value, the first of equal ones
#pragma unroll
      for (int m = LANES / 2; m; m >>= 1) {
        const float d2 = __shfl_xor_sync(kFull, best, m), u2 = __shfl_xor_sync(kFull, best_un, m);
        const uint32_t b2 = __shfl_xor_sync(kFull, bi, m);
        if (d2 < best || (d2 == best && b2 < bi)) {
          best = d2;
          best_un = u2;
          bi = b2;
        }
      }
      if (n_objs <= 1u || !taps) break;
    }
    const bool tap = r == rounds || (n_objs == 1u && diff);
    const uint32_t ob = tap ? bi : r * LANES + (j + 2u) % LANES;
    if (tap ? !diff : ob >= n_objs) continue;
    const ObjSample& o = object(ob);
    float x = px, y = py, z = pz, lx, ly, lz, du;
    // voxelized: central differences of the sampler, eps = 2 voxels, in the
    // object's frame; else of the object, eps = 10 * hit_threshold(0.001)
    const bool vox = o.sdf_type == RKF_SDF_VOXELIZED;
    float e = vox ? __fmul_rn(o.vs, 2.0f) : __fmul_rn(0.001f, 10.0f);
    if (j & 1u) e = -e;  // x + (-e) is x - e
    if (tap && !vox) {
      if (j < 2u) x = __fadd_rn(x, e);
      else if (j < 4u) y = __fadd_rn(y, e);
      else z = __fadd_rn(z, e);
    }
    to_local_fast(o, x, y, z, lx, ly, lz);
    if (tap && vox) {
      if (j < 2u) lx = __fadd_rn(lx, e);
      else if (j < 4u) ly = __fadd_rn(ly, e);
      else lz = __fadd_rn(lz, e);
    }
    float d = kMaxFloat;
    du = kMaxFloat;
    if (o.sdf_type != RKF_SDF_NONE) {
      du = o.sdf_type == RKF_SDF_ANALYTICAL ? analytic_sdf(o, lx, ly, lz)
                                            : sample_vox<PREC>(s, o, lx, ly, lz, tap && vox, lc);
      d = __fmul_rn(du, o.min_scale);
    }
    if (tap) {
      g = vox ? du : d;
    } else if (d < best) {
      best = d;
      best_un = du;
      bi = ob;
    }
  }
  g = __fsub_rn(g, __shfl_down_sync(kFull, g, 1, LANES));  // lanes 0, 2, 4
  const float g0 = __shfl_sync(kFull, g, 0, LANES), g1 = __shfl_sync(kFull, g, 2, LANES),
              g2 = __shfl_sync(kFull, g, 4, LANES);
  if (id >= n) return;
  // lane 6: distance and gradient; lane 7: the material
  if (material && (LANES == 1u || j == 7u)) {
    uint32_t m = 0;
    if (n_objs) {
      const ObjSample& o = object(bi);
      if (o.sdf_type == RKF_SDF_ANALYTICAL || best_un < o.vs16) m = material_at(s, o, px, py, pz, lc);
    }
    material[i] = static_cast<uint16_t>(m);
  }
  if (LANES > 1u && j != 6u) return;
  if (dist) dist[i] = best;
  if (!taps) return;
  float nx = 0.0f, ny = 1.0f, nz = 0.0f;
  if (n_objs) {
    const ObjSample& o = object(bi);
    const bool vox = o.sdf_type == RKF_SDF_VOXELIZED;
    float wx = g0, wy = g1, wz = g2;
    if (vox) {
      wx = __fadd_rn(__fadd_rn(__fadd_rn(__fmul_rn(o.m[0], g0), __fmul_rn(o.m[1], g1)), __fmul_rn(o.m[2], g2)),
                     __fmul_rn(o.m[3], 0.0f));
      wy = __fadd_rn(__fadd_rn(__fadd_rn(__fmul_rn(o.m[4], g0), __fmul_rn(o.m[5], g1)), __fmul_rn(o.m[6], g2)),
                     __fmul_rn(o.m[7], 0.0f));
      wz = __fadd_rn(__fadd_rn(__fadd_rn(__fmul_rn(o.m[8], g0), __fmul_rn(o.m[9], g1)), __fmul_rn(o.m[10], g2)),
                     __fmul_rn(o.m[11], 0.0f));
    }
    const float l = len3(wx, wy, wz);
    if (!vox || l >= 1e-10f) {
      nx = __fdiv_rn(wx, l);
      ny = __fdiv_rn(wy, l);
      nz = __fdiv_rn(wz, l);
    }
  }
  grad[3 * static_cast<size_t>(i)] = nx;
  grad[3 * static_cast<size_t>(i) + 1] = ny;
  grad[3 * static_cast<size_t>(i) + 2] = nz;
}

// sdf_ao (shade_common_shading.wgsl:37-47), four taps along the normal at
// AO_STEP_SIZE * i (0.12 m) through sample_sdf, which for points inside the
// objects' bounds is the minimum of evaluate_object over the objects
// (shade_common.wgsl:521-572); ao = clamp(1 - AO_STRENGTH * sum, 0, 1) with
// AO_STRENGTH 0.7 and tap weights 1, 1/2, 1/4, 1/8.
// A lane per tap, added up in the taps' order: bound by the chain of a tap's
// loads, of which a thread per point took four in a row.  Call times over the
// 32 m scene, 64 / 30,000 / 200,003 / 500,000 points: 32 / 35 / 58 / 86 us for a
// thread per point, 19 / 21 / 44 / 81 us so; 12 blocks an SM (40 registers), as
// 10 take 46 and 85 for the last two.
// Every lane of a warp evaluates the same object, from a copy of the table where it
// fits.  A block takes its points in turns, so that a launch copies the table for
// the blocks that fit the chip alone (ao_blocks).
template <int PREC, int TABLE>
__global__ void __launch_bounds__(128, 12) k_sdf_ao(SceneDev s, const float* __restrict__ pos,
                                                   const float* __restrict__ nrm, uint32_t n,
                                                   float* __restrict__ ao) {
  extern __shared__ ObjSample sh_objs[];
  load_table<TABLE>(sh_objs, s);
  const uint32_t k = 1u + threadIdx.x % kAoLanes, per = blockDim.x / kAoLanes;
#pragma unroll 1
  for (uint64_t first = static_cast<uint64_t>(blockIdx.x) * per; first < n; first += static_cast<uint64_t>(gridDim.x) * per) {
    const uint64_t id = first + threadIdx.x / kAoLanes;
    const uint32_t i = id < n ? static_cast<uint32_t>(id) : n - 1u;  // (every lane takes part in the exchange)
    LaneCache lc;
    const size_t i3 = 3 * static_cast<size_t>(i);
    const float px = pos[i3], py = pos[i3 + 1], pz = pos[i3 + 2];
    const float nx = nrm[i3], ny = nrm[i3 + 1], nz = nrm[i3 + 2];
    const float dist = __fmul_rn(0.12f, static_cast<float>(k));
    const float qx = __fadd_rn(px, __fmul_rn(nx, dist)), qy = __fadd_rn(py, __fmul_rn(ny, dist)),
                qz = __fadd_rn(pz, __fmul_rn(nz, dist));
    float d = kMaxFloat;
    for (uint32_t oi = 0; oi < s.n_objs; ++oi) {
      const ObjSample* o = s.objs + oi;
      if (TABLE == TABLE_SHARED) o = sh_objs + oi;
      float du;
      const float v = eval_obj<PREC>(s, *o, qx, qy, qz, &du, lc);
      if (v < d) d = v;
    }
    const float tap = __fsub_rn(dist, d);
    float acc = 0.0f, scale = 1.0f;
#pragma unroll
    for (int a = 0; a < static_cast<int>(kAoLanes); ++a) {  // in the taps' order
      acc = __fadd_rn(acc, __fmul_rn(scale, __shfl_sync(kFull, tap, a, kAoLanes)));
      scale = __fmul_rn(scale, 0.5f);
    }
    if (id < n && k == 1u) ao[i] = clampf(__fsub_rn(1.0f, __fmul_rn(0.7f, acc)), 0.0f, 1.0f);
  }
}

// The kernel of a launch.  tree: it walks the imported tree (of one object, as of
// several); the walk's code in the loop of the others cost them 6-10%.  many: views of
// kManyIds work ids or more (march_blocks).
template <int PREC, bool MANY>
const void* persistent_fn(int obj, bool tree) {
#define RKF_MARCH(OBJ, TREE, MANY) reinterpret_cast<const void*>(&k_march_persistent<PREC, OBJ, TREE, MANY>)
  if (obj == OBJ_MULTI_EMPTY) return tree ? RKF_MARCH(OBJ_MULTI_EMPTY, true, MANY) : RKF_MARCH(OBJ_MULTI_EMPTY, false, MANY);
  if (tree) return RKF_MARCH(OBJ_MULTI, true, false);
  if (obj == OBJ_MULTI_EMPTY_TILED) return RKF_MARCH(OBJ_MULTI_EMPTY_TILED, false, MANY);
  if (obj == OBJ_SINGLE_EMPTY_TILED) return RKF_MARCH(OBJ_SINGLE_EMPTY_TILED, false, MANY);
  if (obj == OBJ_SINGLE_EMPTY) return RKF_MARCH(OBJ_SINGLE_EMPTY, false, false);
  if (obj == OBJ_SINGLE) return RKF_MARCH(OBJ_SINGLE, false, false);
  return RKF_MARCH(OBJ_MULTI, false, false);
#undef RKF_MARCH
}
template <int PREC>
const void* persistent_fn(int obj, bool tree, bool many) {
  return many ? persistent_fn<PREC, true>(obj, tree) : persistent_fn<PREC, false>(obj, tree);
}

}  // namespace detail

namespace {
// A voxelized object the empty-space path can march: translation-only
// inverse_world, verified exact quotient, fewer than 2^20 voxels per axis.
bool empty_object(const Ctx* c, const ObjDev& o) {
  return o.sdf_type == RKF_SDF_VOXELIZED && o.translate_only && o.div_ok && c->empty_dist.p != nullptr &&
         o.tv[0] < (1 << 20) && o.tv[1] < (1 << 20) && o.tv[2] < (1 << 20);
}

// Upper bound of every EMPTY value of a voxelized object: mix(c, c, t) three
// times stays within 12 roundings of c = brick extent * min_scale (relative
// 2^-24 each), far inside 2^-16.
float empty_hi_of(const ObjDev& o) { return o.be * o.min_scale * (1.0f + 1.52587890625e-5f); }

// Radius of the ball around the local origin that holds an analytic
// primitive (analytic_sdf, ray_march.wgsl:182-264): its value is at least
// |l| - R everywhere.  -1 for a plane (unbounded) or non-finite parameters.
double prim_radius(const ObjDev& o) {
  const double a0 = std::fabs(static_cast<double>(o.params[0])), a1 = std::fabs(static_cast<double>(o.params[1])),
               a2 = std::fabs(static_cast<double>(o.params[2]));
  double r = -1.0;
  switch (o.prim_type) {
    case RKF_PRIM_SPHERE: r = a0; break;
    case RKF_PRIM_BOX: r = std::sqrt(a0 * a0 + a1 * a1 + a2 * a2); break;
    case RKF_PRIM_CAPSULE: r = a0 + a1; break;
    case RKF_PRIM_TORUS: r = a0 + a1; break;
    case RKF_PRIM_CYLINDER: r = std::sqrt(a0 * a0 + a1 * a1); break;
    default: return -1.0;
  }
  return std::isfinite(r) ? r : -1.0;
}

double up_float(double v) {  // a float >= v
  const float f = static_cast<float>(v);
  return static_cast<double>(f) >= v ? f : std::nextafter(f, std::numeric_limits<float>::infinity());
}

// The FarBall of an analytic object for EMPTY values up to empty_hi (the
// bound FarBall describes, with every FP32 rounding of evaluate_object held
// to 2^-16 of the magnitudes involved, a wide margin over the few 2^-24
// roundings each step makes).  false when the object has no usable ball.
bool far_ball(const ObjDev& o, float empty_hi, detail::FarBall* out) {
  // A voxelized object's sampler returns the distance to its clamped grid
  // box (a box inside |l| <= |half_gs|) wherever that distance exceeds two
  // brick extents (ray_march.wgsl:371-376), so beyond the ball of radius
  // |half_gs| + max(2 * brick extent, EMPTY value / scale) its value is at
  // least that distance times its scale, above every EMPTY value.  With a
  // translation-only transform the grid box is axis-aligned in world space,
  // and the same holds outside the box widened by that distance (a position
  // beyond it along one axis is that far from the box): the tighter bound.
  const bool vox = o.sdf_type == RKF_SDF_VOXELIZED;
  std::memset(out, 0, sizeof(*out));
  out->path = ~0u;
  if (vox && o.translate_only) {
    const double s = o.min_scale;
    if (!(s > 0.0) || !std::isfinite(s)) return false;
    const double e16 = 0x1p-16, e20 = 0x1p-20;
    const double need = std::max(static_cast<double>(empty_hi) * (1.0 + e16) / s,
                                 static_cast<double>(o.be2) * (1.0 + e16));
    double tn = 0.0, hn = 0.0;
    for (int i = 0; i < 3; ++i) {
      out->c[i] = -o.m[12 + i];  // local = world + m: the local origin (grid centre) in world space
      out->h[i] = static_cast<float>(up_float(static_cast<double>(o.half_gs[i]) * (1.0 + e16)));
      tn += static_cast<double>(o.m[12 + i]) * o.m[12 + i];
      hn += static_cast<double>(o.half_gs[i]) * o.half_gs[i];
    }
    out->a = static_cast<float>(up_float(need + e16 * (std::sqrt(tn) + std::sqrt(hn)) + e20 * std::sqrt(tn)));
    out->b = static_cast<float>(up_float(3.0 * e16 + e20));
    out->box = 1;
    return std::isfinite(out->a) && std::isfinite(out->h[0]) && std::isfinite(out->h[1]) &&
           std::isfinite(out->h[2]) && std::isfinite(out->c[0]) && std::isfinite(out->c[1]) &&
           std::isfinite(out->c[2]);
  }
  const double R = vox ? std::sqrt(static_cast<double>(o.half_gs[0]) * o.half_gs[0] +
                                   static_cast<double>(o.half_gs[1]) * o.half_gs[1] +
                                   static_cast<double>(o.half_gs[2]) * o.half_gs[2])
                       : prim_radius(o);
  const double s = o.min_scale;
  if (R < 0.0 || !std::isfinite(R) || !(s > 0.0) || !std::isfinite(s)) return false;
  double A[3][3], t[3];  // l_i = sum_k A[i][k] p_k + t_i (to_local)
  for (int i = 0; i < 3; ++i) {
    for (int k = 0; k < 3; ++k) A[i][k] = o.m[4 * k + i];
    t[i] = o.m[12 + i];
  }
  const double det = A[0][0] * (A[1][1] * A[2][2] - A[1][2] * A[2][1]) -
                     A[0][1] * (A[1][0] * A[2][2] - A[1][2] * A[2][0]) +
                     A[0][2] * (A[1][0] * A[2][1] - A[1][1] * A[2][0]);
  if (!std::isfinite(det) || det == 0.0) return false;
  double inv[3][3];
  for (int i = 0; i < 3; ++i)
    for (int k = 0; k < 3; ++k) {
      const int i1 = (k + 1) % 3, i2 = (k + 2) % 3, k1 = (i + 1) % 3, k2 = (i + 2) % 3;
      inv[i][k] = (A[i1][k1] * A[i2][k2] - A[i1][k2] * A[i2][k1]) / det;
    }
  double nf = 0.0, nif = 0.0, tn = 0.0, c[3], cn = 0.0;
  for (int i = 0; i < 3; ++i) {
    c[i] = -(inv[i][0] * t[0] + inv[i][1] * t[1] + inv[i][2] * t[2]);
    cn += c[i] * c[i];
    tn += t[i] * t[i];
    for (int k = 0; k < 3; ++k) {
      nf += A[i][k] * A[i][k];
      nif += inv[i][k] * inv[i][k];
    }
  }
  const double N = std::sqrt(nf), sigma = 1.0 / std::sqrt(nif);  // |A x| >= sigma |x|
  const double e16 = 0x1p-16, e20 = 0x1p-20;
  if (!(sigma > 0.0) || !(N / sigma <= 1024.0)) return false;
  double need = static_cast<double>(empty_hi) * (1.0 + e16) / s;  // local distance beyond R
  if (vox) need = std::max(need, static_cast<double>(o.be2) * (1.0 + e16));
  const double a = (R * (1.0 + e16) + e16 * std::sqrt(tn) + need) / sigma + e20 * std::sqrt(cn);
  const double b = e16 * N / sigma + e20;
  for (int i = 0; i < 3; ++i) out->c[i] = static_cast<float>(c[i]);
  out->a = static_cast<float>(up_float(a));
  out->b = static_cast<float>(up_float(b));
  return std::isfinite(out->c[0]) && std::isfinite(out->c[1]) && std::isfinite(out->c[2]) && std::isfinite(out->a) &&
         std::isfinite(out->b);
}

// The half-space of an analytic plane for EMPTY values up to empty_hi.  The
// plane's value (ray_march.wgsl:206-208, 257-258) is s * n.l with n the
// normalised normal and l = A w + t the local position: exactly G.w + H with
// G = s A^T n, H = s n.t.  The computed value differs from that by at most
// 2^-16 s (|A|_F |w| + |t|) -- about twenty roundings of 2^-24 each over the
// local transform, the normalisation and the dot product -- and the sample
// positions from the line by 2^-16 |w|, so wherever G.w + H exceeds
// empty_hi (1 + 2^-16) + 2^-16 (s |t| + (s |A|_F + |G|) |w|) the plane's value
// exceeds every EMPTY value; |w| <= P along the ray.  Refused for a zero or
// non-finite normal or transform.
bool far_plane(const ObjDev& o, float empty_hi, detail::FarBall* out) {
  std::memset(out, 0, sizeof(*out));
  out->path = ~0u;
  const double s = o.min_scale;
  const double nl = std::sqrt(static_cast<double>(o.params[0]) * o.params[0] +
                              static_cast<double>(o.params[1]) * o.params[1] +
                              static_cast<double>(o.params[2]) * o.params[2]);
  if (!(nl > 0.0) || !std::isfinite(nl) || !(s > 0.0) || !std::isfinite(s)) return false;
  double n[3], G[3] = {0.0, 0.0, 0.0}, H = 0.0, fa = 0.0, tn = 0.0, gn = 0.0;
  for (int i = 0; i < 3; ++i) n[i] = static_cast<double>(o.params[i]) / nl;
  for (int i = 0; i < 3; ++i) {  // l_i = sum_k m[4k + i] w_k + m[12 + i]
    for (int k = 0; k < 3; ++k) {
      const double aik = o.m[4 * k + i];
      G[k] += s * n[i] * aik;
      fa += aik * aik;
    }
    H += s * n[i] * o.m[12 + i];
    tn += static_cast<double>(o.m[12 + i]) * o.m[12 + i];
  }
  for (int k = 0; k < 3; ++k) gn += G[k] * G[k];
  const double e16 = 0x1p-16, e20 = 0x1p-20;
  const double a = static_cast<double>(empty_hi) * (1.0 + e16) + e16 * s * std::sqrt(tn) + e20;
  const double b = e16 * (s * std::sqrt(fa) + std::sqrt(gn)) + e20;
  for (int k = 0; k < 3; ++k) out->c[k] = static_cast<float>(G[k]);
  out->h[0] = static_cast<float>(H);
  out->a = static_cast<float>(up_float(a));
  out->b = static_cast<float>(up_float(b));
  out->box = 2;
  return std::isfinite(out->c[0]) && std::isfinite(out->c[1]) && std::isfinite(out->c[2]) &&
         std::isfinite(out->h[0]) && std::isfinite(out->a) && std::isfinite(out->b);
}

// A scene of several objects the multi-object empty-space path can march:
// one to kMaxEmptyVox voxelized objects that qualify for the empty-space path
// (the first ones by index), each of which takes EMPTY runs on its own field,
// and every object -- analytic, voxelized (on the path or not) or of no type
// -- either bounded by a ball outside which its value exceeds every EMPTY
// value of the path, or (no type, unknown primitives) never below them.
// Fills ev and the balls (with each ball's path index) when given.
bool multi_empty_scene(const Ctx* c, detail::EmptyVox* ev, uint32_t* n_ev, detail::FarBall* balls,
                       uint32_t* n_ball) {
  const uint32_t n = c->obj_count();
  if (n < 2 || n > kMaxObjectsFast) return false;
  uint32_t q[detail::kMaxEmptyVox];
  uint32_t path_of[kMaxObjectsFast];
  uint32_t nq = 0;
  for (uint32_t i = 0; i < n; ++i) {
    path_of[i] = ~0u;
    if (nq < detail::kMaxEmptyVox && empty_object(c, c->objdev_host[i])) {
      path_of[i] = nq;
      q[nq++] = i;
    }
  }
  if (nq == 0) return false;
  float hi = 0.0f;  // the largest EMPTY value of the path
  for (uint32_t j = 0; j < nq; ++j) hi = std::max(hi, empty_hi_of(c->objdev_host[q[j]]));
  uint32_t nb = 0;
  for (uint32_t i = 0; i < n; ++i) {
    const ObjDev& o = c->objdev_host[i];
    if (o.sdf_type == RKF_SDF_NONE) continue;  // no type: kMaxFloat
    if (o.sdf_type == RKF_SDF_ANALYTICAL && o.prim_type > RKF_PRIM_PLANE) {
      // an unknown primitive: kMaxFloat * min_scale
      if (static_cast<double>(kMaxFloat) * o.min_scale * (1.0 - 0x1p-20) >= hi) continue;
      return false;
    }
    detail::FarBall b;
    const bool plane = o.sdf_type == RKF_SDF_ANALYTICAL && o.prim_type == RKF_PRIM_PLANE;
    if (!(plane ? far_plane(o, hi, &b) : far_ball(o, hi, &b))) return false;
    b.path = path_of[i];
    if (balls) balls[nb] = b;
    ++nb;
  }
  for (uint32_t j = 0; ev && j < nq; ++j) {
    const ObjDev& a = c->objdev_host[q[j]];
    detail::EmptyVox e;
    std::memset(&e, 0, sizeof(e));
    e.obj = q[j];
    e.probe_min = 0.99f * a.be * a.min_scale;
    // mix(c, c, t) three times stays within 12 roundings of c (relative
    // 2^-24 each); 0.999 leaves a wide margin, 2^-16 a tight one
    e.empty_lo = 0.999f * a.be * a.min_scale;
    e.empty_lo_t = a.be * a.min_scale * (1.0f - 1.52587890625e-5f);
    e.empty_hi = empty_hi_of(a);
    e.plain = (a.m[12] == 0.0f && a.m[13] == 0.0f && a.m[14] == 0.0f && a.min_scale == 1.0f) ? 1u : 0u;
    ev[j] = e;
  }
  if (n_ev) *n_ev = nq;
  if (n_ball) *n_ball = nb;
  return true;
}

// The BVH walk (eval_bvh) evaluates object vi at every position inside its
// grid (the clamp range every EMPTY cube lies in): some leaf naming vi has
// every node on its path from the root containing that box, and every
// internal node on it descends (the shader's stack had room for its
// children: bit 31 of its walk link).  The walk skips a node only when its
// box distance exceeds the best value so far; inside such nodes that
// distance is 0, and along EMPTY runs outside every ball no value is
// negative, so the leaf is reached and the walk's minimum is the brute one.
bool bvh_reaches(const Ctx* c, uint32_t vi) {
  const std::vector<rkf_bvh_node>& nd = c->bvh_host;
  const std::vector<uint32_t>& link = c->bvh_next_host;
  if (nd.empty() || link.size() != nd.size()) return false;
  const ObjDev& o = c->objdev_host[vi];
  float lo[3], hi[3];
  for (int a = 0; a < 3; ++a) {
    const float base = -o.half_gs[a] - o.m[12 + a];
    lo[a] = 0.5f * o.vs + base;
    hi[a] = (static_cast<float>(o.tv[a] - 1) + 0.5f) * o.vs + base;
  }
  std::vector<uint32_t> stack{0u};
  while (!stack.empty()) {
    const uint32_t i = stack.back();
    stack.pop_back();
    if (i >= nd.size()) continue;
    const rkf_bvh_node& b = nd[i];
    bool holds = true;
    for (int a = 0; a < 3; ++a) holds = holds && b.aabb_min[a] <= lo[a] && b.aabb_max[a] >= hi[a];
    if (!holds) continue;
    if (b.left == RKF_BVH_INVALID) {
      if (b.right_or_object == vi) return true;
    } else if (link[i] >> 31) {
      stack.push_back(b.left);
      stack.push_back(b.right_or_object);
    }
  }
  return false;
}

// The objects of the multi-object empty-space path of a launch, with their
// balls, into kp.ev: those the BVH walk reaches everywhere in their grids
// when the launch walks the tree.  false when none remains.
bool fill_multi_empty(const Ctx* c, bool walk, detail::KParams& kp) {
  detail::EmptyVox ev[detail::kMaxEmptyVox];
  uint32_t n = 0;
  if (!multi_empty_scene(c, ev, &n, kp.ball, &kp.n_ball)) return false;
  // an object the walk may not reach leaves the path (its ball still bounds
  // the others' runs)
  uint32_t remap[detail::kMaxEmptyVox];
  kp.n_ev = 0;
  kp.probe_min = kMaxFloat;
  for (uint32_t j = 0; j < n; ++j) {
    remap[j] = ~0u;
    if (walk && !bvh_reaches(c, ev[j].obj)) continue;
    remap[j] = kp.n_ev;
    kp.ev[kp.n_ev] = ev[j];
    kp.probe_min = std::min(kp.probe_min, ev[j].probe_min);
    ++kp.n_ev;
  }
  for (uint32_t b = 0; b < kp.n_ball; ++b)
    if (kp.ball[b].path < n) kp.ball[b].path = remap[kp.ball[b].path];
  return kp.n_ev > 0;
}

// The bounds of the EMPTY values of the launch's path: of object 0, or of the
// path's objects together (filled by fill_multi_empty).  mix(c, c, t) three
// times stays within 12 roundings of c (relative 2^-24 each): 0.999 leaves a
// wide margin, 2^-16 a tight one.  A tiled launch also steps by coarse skips,
// each of more than kCoarseNear.
void empty_bounds(detail::KParams& kp, bool empty, bool multi, bool tiled) {
  const ObjDev& e0 = kp.objs[0];
  kp.probe_min = empty ? (multi ? kp.probe_min : 0.99f * e0.be * e0.min_scale) : kMaxFloat;
  kp.empty_lo = empty ? 0.999f * e0.be * e0.min_scale : 0.0f;
  kp.empty_lo_t = e0.be * e0.min_scale * (1.0f - 1.52587890625e-5f);
  kp.empty_hi = empty_hi_of(e0);
  for (uint32_t e = 0; multi && e < kp.n_ev; ++e) {
    const detail::EmptyVox& v = kp.ev[e];
    kp.empty_lo = e ? std::min(kp.empty_lo, v.empty_lo) : v.empty_lo;
    kp.empty_lo_t = e ? std::min(kp.empty_lo_t, v.empty_lo_t) : v.empty_lo_t;
    kp.empty_hi = e ? std::max(kp.empty_hi, v.empty_hi) : v.empty_hi;
  }
  if (tiled) kp.empty_lo_t = std::min(kp.empty_lo_t, kCoarseNear);
}

constexpr float kFewSteps = 150.0f, kFewStepsTiled = 250.0f;
// Every grid of the path at most `steps` EMPTY steps long.
bool few_empty_steps(const detail::KParams& kp, bool multi, float steps) {
  for (uint32_t e = 0; e < (multi ? kp.n_ev : 1u); ++e) {
    const ObjDev& o = kp.objs[multi ? kp.ev[e].obj : 0u];
    if (2.0f * std::max({o.half_gs[0], o.half_gs[1], o.half_gs[2]}) > steps * o.be) return false;
  }
  return true;
}

// Which kernel variant a launch over this context's objects uses.
int object_set(const Ctx* c) {
  if (c->obj_count() != 1)
    return multi_empty_scene(c, nullptr, nullptr, nullptr, nullptr) ? detail::OBJ_MULTI_EMPTY : detail::OBJ_MULTI;
  return empty_object(c, c->objdev_host[0]) ? detail::OBJ_SINGLE_EMPTY : detail::OBJ_SINGLE;
}
}  // namespace

bool launch_settles(const Ctx* c, uint64_t view_ids) {
  const int objs = object_set(c);
  return (objs == detail::OBJ_SINGLE_EMPTY || objs == detail::OBJ_MULTI_EMPTY) && view_ids >= kSettleIds &&
         view_ids < (1ull << 32);
}

bool empty_order_source(const Ctx* c, const rkf_march_params* p, const rkf_batch_tuning& tu, ObjDev* o) {
  if (tu.no_empty_path || p->strategy == RKF_STRATEGY_TILED || c->obj_count() == 0 ||
      c->obj_count() > kMaxObjectsFast)
    return false;
  const bool use_bvh = p->strategy == RKF_STRATEGY_BVH;
  const int objs = object_set(c);
  if (objs == detail::OBJ_SINGLE_EMPTY) {
    if (use_bvh && !c->bvh_one_leaf0) return false;
    *o = c->objdev_host[0];
    return true;
  }
  if (objs == detail::OBJ_MULTI_EMPTY) {
    // the estimate walks the field of the path's first object
    detail::KParams kp;
    if (!fill_multi_empty(c, use_bvh, kp)) return false;
    *o = c->objdev_host[kp.ev[0].obj];
    return true;
  }
  return false;
}

float order_reach(const ObjDev& o, const rkf_march_params* p) {
  return std::min(p->scene.max_distance, static_cast<float>(p->hard_max_steps) * o.be * o.min_scale);
}

rkf_status launch_persistent(Ctx* c, const std::vector<Segment>& segs_host, uint64_t total,
                             const rkf_march_params* p, const rkf_batch_tuning& tu,
                             cudaStream_t st, DevBuf* seg_buf, unsigned long long* counter, uint64_t id0,
                             bool segs_resident) {
  if (c->obj_count() == 0) return fail(RKF_INVALID_ARG, "march: the scene has no objects");
  const bool tiled = p->strategy == RKF_STRATEGY_TILED;
  const bool use_bvh = p->strategy == RKF_STRATEGY_BVH;
  if (use_bvh && c->bvh_n == 0) return fail(RKF_INVALID_ARG, "march: the BVH strategy needs an imported BVH");
  std::vector<Segment> tiled_segs;
  TiledDev td;
  std::memset(&td, 0, sizeof(td));
  int objs = object_set(c);
  if (tu.no_empty_path) {  // the same outputs through the full sampler only
    if (objs == detail::OBJ_SINGLE_EMPTY) objs = detail::OBJ_SINGLE;
    if (objs == detail::OBJ_MULTI_EMPTY) objs = detail::OBJ_MULTI;
  }
  if (tiled) {
    tiled_segs = segs_host;
    rkf_status s2 = prepare_tiled(c, tiled_segs, st, &td);
    if (s2 != RKF_OK) return s2;
    // the tiled empty-space field of every object of the path
    std::vector<uint32_t> path{0u};
    if (objs == detail::OBJ_MULTI_EMPTY) {
      detail::EmptyVox ev[detail::kMaxEmptyVox];
      uint32_t n = 0;
      multi_empty_scene(c, ev, &n, nullptr, nullptr);
      path.clear();
      for (uint32_t j = 0; j < n; ++j) path.push_back(ev[j].obj);
    }
    if ((objs == detail::OBJ_SINGLE_EMPTY || objs == detail::OBJ_MULTI_EMPTY) &&
        (s2 = prepare_tiled_empty(c, st, path)) != RKF_OK)
      return s2;
  }
  // heaviest-first order of the views' tiles (a whole launch only: a band of
  // a view is ordered by its caller, which plans all bands at once)
  ObjDev order_obj;
  OrderTable order_tbl;
  bool ordered = false;
  std::vector<Segment> ordered_segs;
  // the settling passes take the place of that order: what they leave is an
  // even list of rays
  uint64_t view_ids = 0;
  for (const Segment& sg : segs_host)
    if (sg.kind == 0) view_ids += sg.n_ids;
  const bool settle = !tu.no_empty_path && launch_settles(c, view_ids) && id0 == 0 && !segs_resident;
  if (tu.order_tiles && !settle && id0 == 0 && !segs_resident && !tiled && empty_order_source(c, p, tu, &order_obj)) {
    ordered_segs = segs_host;
    rkf_status s2 = tile_order_prepare(c, ordered_segs, tu.tile_w, tu.tile_h, nullptr, 0, &order_tbl, &ordered);
    if (s2 != RKF_OK) return s2;
  }
  const std::vector<Segment>& segs_dev = tiled ? tiled_segs : (ordered ? ordered_segs : segs_host);
  const size_t sb = segs_dev.size() * sizeof(Segment);
  if (!segs_resident || seg_buf->bytes < sb) {
    if (seg_buf->bytes < sb) {
      rkf_status s2 = seg_buf->alloc(sb);
      if (s2 != RKF_OK) return s2;
    }
    // a pageable source: the call returns once the stream has taken the data
    RKF_CUDA_TRY(cudaMemcpyAsync(seg_buf->p, segs_dev.data(), sb, cudaMemcpyHostToDevice, st));
  }
  if (ordered) {
    rkf_status s2 = tile_order_enqueue(c, order_tbl, seg_buf->as<Segment>(), order_obj, c->empty_dist.as<uint8_t>(),
                                       order_reach(order_obj, p), order_obj.be * order_obj.min_scale, st);
    if (s2 != RKF_OK) return s2;
  }
  RKF_CUDA_TRY(cudaMemsetAsync(counter, 0, sizeof(unsigned long long), st));
  detail::KParams kp;
  std::memset(&kp, 0, sizeof(kp));
  // beyond kMaxObjectsFast objects the kernel reads the device table
  std::memcpy(kp.objs, c->objdev_host.data(), sizeof(ObjDev) * std::min<uint32_t>(c->obj_count(), kMaxObjectsFast));
  kp.s = c->scene_dev();
  kp.segs = seg_buf->as<Segment>();
  kp.nseg = static_cast<uint32_t>(segs_host.size());
  kp.tile_w = tu.tile_w ? tu.tile_w : 8;
  kp.tile_h = tu.tile_h ? tu.tile_h : 4;
  kp.interval = tu.compact_interval ? tu.compact_interval : 64;
  kp.total = total;
  kp.id0 = id0;
  kp.counter = counter;
  kp.p = *p;
  kp.p.scene.num_objects = c->obj_count();
  // A BVH of one leaf naming the only, voxelized, object makes every step
  // evaluate exactly what the brute step evaluates (the one box test passes
  // for every finite distance, and where it would not, the object's own
  // distance is not finite either), so that walk is the brute march.
  const bool walk = use_bvh && !(objs == detail::OBJ_SINGLE_EMPTY && c->bvh_one_leaf0);
  int obj = objs;
  if (objs == detail::OBJ_SINGLE_EMPTY && walk) obj = detail::OBJ_SINGLE;
  if (objs == detail::OBJ_SINGLE_EMPTY && tiled) {
    obj = detail::OBJ_SINGLE_EMPTY_TILED;
    kp.s.empty_dist = c->tiled_empty_dist.as<uint8_t>();
  }
  // the multi-object empty-space path marches the brute and tiled
  // strategies, and the BVH strategy for the objects whose grids the tree's
  // walk reaches everywhere
  if (objs == detail::OBJ_MULTI_EMPTY && !fill_multi_empty(c, walk, kp)) obj = detail::OBJ_MULTI;
  if (obj == detail::OBJ_MULTI_EMPTY && tiled) {
    obj = detail::OBJ_MULTI_EMPTY_TILED;
    kp.s.empty_dist = c->tiled_empty_dist.as<uint8_t>();
  }
  const bool multi_empty = obj == detail::OBJ_MULTI_EMPTY || obj == detail::OBJ_MULTI_EMPTY_TILED;
  const bool empty = obj == detail::OBJ_SINGLE_EMPTY || obj == detail::OBJ_SINGLE_EMPTY_TILED || multi_empty;
  kp.td = td;
  kp.tiled = tiled ? 1u : 0u;
  kp.bvh = walk ? c->bvh.as<rkf_bvh_node>() : nullptr;
  kp.bvh_next = walk ? c->bvh_next.as<uint32_t>() : nullptr;
  const ObjDev& e0 = kp.objs[0];  // the object of the single-object empty-space path
  empty_bounds(kp, empty, multi_empty, tiled);
  kp.budget = tu.step_budget ? tu.step_budget : 32;
  kp.brute_field = c->empty_dist.as<uint8_t>();
  kp.plain_obj = (e0.m[12] == 0.0f && e0.m[13] == 0.0f && e0.m[14] == 0.0f && e0.min_scale == 1.0f) ? 1u : 0u;
  const uint32_t threads = tu.threads_per_block ? tu.threads_per_block : 256;
  if (threads > 256 || threads % 32)
    return fail(RKF_INVALID_ARG, "march: threads_per_block must be a multiple of 32 <= 256");
  // Several objects whose grids are few EMPTY steps across leave few of them to
  // a run: after the settling passes the rays that are left march the plain
  // kernel, whose loop is the shorter one (1277x717, five objects, grids 100
  // EMPTY steps a side: 1.86 / 1.72 / 2.27 ms against 2.72 / 3.44 / 3.55 under
  // brute / tiled / BVH; 200 steps: 1.77 / 1.43 / 1.79 against 1.46 / 1.76 /
  // 1.77; 400 steps: 7.5 / 4.3 / 7.1 against 2.7 / 1.8 / 2.7).  Else the tiled
  // strategy goes without the passes: its coarse skips leave the misses cheap
  // (grids of 1,600 steps: 1.75 ms against 2.22 with them).  One object: u8,
  // 1920x1080, 100 steps: 1.64 ms plain against 2.29; 200 steps: 0.90 either way;
  // 400 steps: 1.15 against 0.59.  Tiled (plain also without the passes):
  // 100 steps 1.30 ms against 5.9, 200 steps 1.08 against 1.47, 400 steps 3.1
  // against 1.0.  Views below kSettleIds and ray batches keep the EMPTY variants
  // (one object, f16, 100 steps; EMPTY / plain us): 160x90 249 / 311, 256x144 372 / 415,
  // 480x270 544 / 509; 64 / 2,000 / 30,000 / 250,000 rays 88 / 141 / 254 / 694 against 178 /
  // 239 / 308 / 776.
  const bool few = empty && few_empty_steps(kp, multi_empty, tiled ? kFewStepsTiled : kFewSteps);
  const bool tiled_empty = tiled && empty;
  // (march timing covers the passes too)
  rkf_status se = c->march_event(st, false);
  if (se != RKF_OK) return se;
  // (no room for the lists: the march alone)
  const uint64_t part = settle && empty && (!tiled_empty || few) ? settle_part(c, view_ids, kp.tile_w * kp.tile_h) : 0;
  const int path = obj;  // the variant the passes settle for
  if (part && few) obj = multi_empty ? detail::OBJ_MULTI : detail::OBJ_SINGLE;
  if (few && obj == detail::OBJ_SINGLE_EMPTY_TILED) obj = detail::OBJ_SINGLE;
  c->last_variant = obj;
  const uint32_t refill = detail::march_refill(obj, part != 0);
  const bool many = view_ids >= detail::kManyIds;
  // A view of one object off the EMPTY path, f16 or f32, is faster in the kernel of
  // several: that of one spills (f16, rotated, 1920x1080 of the 32 m scene 1.68 against
  // 1.77 ms; u8, which does not, 1.73 against 1.59; 2,000 rays f16 224 against 207 us).
  if (obj == detail::OBJ_SINGLE && view_ids && c->cfg.precision != RKF_PRECISION_U8) obj = detail::OBJ_MULTI;
  const void* fn = nullptr;
  switch (c->cfg.precision) {
    case RKF_PRECISION_F32:
      fn = detail::persistent_fn<RKF_PRECISION_F32>(obj, walk, many);
      break;
    case RKF_PRECISION_U8:
      fn = detail::persistent_fn<RKF_PRECISION_U8>(obj, walk, many);
      break;
    default:
      fn = detail::persistent_fn<RKF_PRECISION_F16>(obj, walk, many);
  }
  kp.refill_idle = tu.refill_idle && tu.refill_idle < 32u ? tu.refill_idle : refill;
  const size_t smem = 0;
  uint32_t bps = tu.blocks_per_sm;
  if (bps == 0) {
    int occ = 0;
    RKF_CUDA_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, fn, threads, smem));
    bps = occ > 0 ? static_cast<uint32_t>(occ) : 1;
  }
  const uint64_t block_rays = threads / 32 * detail::kLeastLanes;  // (lane_share spreads them)
  for (uint64_t first = 0;;) {
    // the next part of the views, with the ray batches after the last; or all at once
    const uint64_t end = part ? std::min(first + part, view_ids) : total;
    const bool last = !part || end == view_ids;
    if (part) {
      if (first) RKF_CUDA_TRY(cudaMemsetAsync(counter, 0, sizeof(unsigned long long), st));
      const rkf_status s2 = settle_enqueue(c, kp, path, first, end, st);
      if (s2 != RKF_OK) return s2;
      kp.total = last ? total : end;
    }
    uint64_t blocks = static_cast<uint64_t>(c->sm_count) * bps;
    const uint64_t need_blocks = ((last ? total : end) - first + block_rays - 1) / block_rays;
    if (blocks > need_blocks) blocks = need_blocks ? need_blocks : 1;
    void* args[] = {&kp};
    RKF_CUDA_TRY(cudaLaunchKernel(fn, dim3(static_cast<unsigned>(blocks)), dim3(threads), args, smem, st));
    c->counted();
    if (last) break;
    first = end;
  }
  return c->march_event(st, true);
}

rkf_status check_persistent_scratch(const Ctx* c, const rkf_march_params* p, const rkf_batch_tuning& tu) {
  if (p->strategy != RKF_STRATEGY_BRUTE)
    return fail(RKF_UNSUPPORTED, "march: this launch path runs the brute strategy only");
  if (c->obj_count() == 0) return fail(RKF_INVALID_ARG, "march: the scene has no objects");
  const uint32_t threads = tu.threads_per_block ? tu.threads_per_block : 256;
  if (threads > 256 || threads % 32)
    return fail(RKF_INVALID_ARG, "march: threads_per_block must be a multiple of 32 <= 256");
  return RKF_OK;
}

rkf_status launch_persistent_scratch(Ctx* c, const Segment* segs_host, uint32_t nseg, uint64_t total,
                                     const rkf_march_params* p, const rkf_batch_tuning& tu,
                                     cudaStream_t st, Segment* dev_segs, unsigned long long* dev_counter,
                                     bool segs_uploaded, bool multi_empty) {
  // every refusal comes before anything is enqueued on the stream
  const rkf_status chk = check_persistent_scratch(c, p, tu);
  if (chk != RKF_OK) return chk;
  if (!segs_uploaded)
    RKF_CUDA_TRY(cudaMemcpyAsync(dev_segs, segs_host, sizeof(Segment) * nseg, cudaMemcpyHostToDevice, st));
  RKF_CUDA_TRY(cudaMemsetAsync(dev_counter, 0, sizeof(unsigned long long), st));
  detail::KParams kp;
  std::memset(&kp, 0, sizeof(kp));
  // beyond kMaxObjectsFast objects the kernel reads the device table
  std::memcpy(kp.objs, c->objdev_host.data(), sizeof(ObjDev) * std::min<uint32_t>(c->obj_count(), kMaxObjectsFast));
  kp.s = c->scene_dev();
  kp.segs = dev_segs;
  kp.nseg = nseg;
  kp.tile_w = tu.tile_w ? tu.tile_w : 8;
  kp.tile_h = tu.tile_h ? tu.tile_h : 4;
  kp.interval = tu.compact_interval ? tu.compact_interval : 64;
  kp.total = total;
  kp.counter = dev_counter;
  kp.p = *p;
  kp.p.scene.num_objects = c->obj_count();
  // without multi_empty, several objects march the plain multi-object kernel
  int obj = object_set(c);
  if (obj == detail::OBJ_MULTI_EMPTY && (!multi_empty || !fill_multi_empty(c, false, kp))) obj = detail::OBJ_MULTI;
  const bool memp = obj == detail::OBJ_MULTI_EMPTY;
  const ObjDev& e0 = kp.objs[0];  // the object of the single-object empty-space path
  const bool empty = obj == detail::OBJ_SINGLE_EMPTY || memp;
  empty_bounds(kp, empty, memp, false);
  kp.budget = tu.step_budget ? tu.step_budget : 32;
  kp.refill_idle = tu.refill_idle && tu.refill_idle < 32u ? tu.refill_idle : detail::march_refill(obj, false);
  kp.brute_field = c->empty_dist.as<uint8_t>();
  kp.plain_obj = (e0.m[12] == 0.0f && e0.m[13] == 0.0f && e0.m[14] == 0.0f && e0.min_scale == 1.0f) ? 1u : 0u;
  const void* fn = nullptr;
  switch (c->cfg.precision) {
    case RKF_PRECISION_F32:
      fn = detail::persistent_fn<RKF_PRECISION_F32>(obj, false, false);
      break;
    case RKF_PRECISION_U8:
      fn = detail::persistent_fn<RKF_PRECISION_U8>(obj, false, false);
      break;
    default:
      fn = detail::persistent_fn<RKF_PRECISION_F16>(obj, false, false);
  }
  c->last_variant = obj;
  const uint32_t threads = tu.threads_per_block ? tu.threads_per_block : 256;  // checked above
  uint32_t bps = tu.blocks_per_sm;
  if (bps == 0) {
    int occ = 0;
    RKF_CUDA_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, fn, threads, 0));
    bps = occ > 0 ? static_cast<uint32_t>(occ) : 1;
  }
  uint64_t blocks = static_cast<uint64_t>(c->sm_count) * bps;
  const uint64_t block_rays = threads / 32 * detail::kLeastLanes;  // (lane_share spreads them)
  const uint64_t need_blocks = (total + block_rays - 1) / block_rays;
  if (blocks > need_blocks) blocks = need_blocks ? need_blocks : 1;
  void* args[] = {&kp};
  rkf_status se = c->march_event(st, false);
  if (se != RKF_OK) return se;
  RKF_CUDA_TRY(cudaLaunchKernel(fn, dim3(static_cast<unsigned>(blocks)), dim3(threads), args, 0, st));
  c->counted();
  return c->march_event(st, true);
}

namespace {
template <int PREC, uint32_t LANES>
void query_points(const Ctx* c, const float* pts, uint32_t n, float* d, float* g, uint16_t* m, cudaStream_t st) {
  using namespace detail;
  const SceneDev s = c->scene_dev();
  const unsigned blocks = (n - 1) / (128 / LANES) + 1;
  if (s.n_objs == 1)
    k_query_points<PREC, TABLE_ONE, LANES><<<blocks, 128, 0, st>>>(s, {c->objdev_host[0]}, pts, n, d, g, m);
  else if (s.n_objs <= (LANES == 1 ? kMaxObjectsShared : kPointFewObjects))
    k_query_points<PREC, TABLE_SHARED, LANES><<<blocks, 128, sizeof(ObjSample) * s.n_objs, st>>>(s, {}, pts, n, d, g, m);
  else
    k_query_points<PREC, TABLE_DEVICE, LANES><<<blocks, 128, 0, st>>>(s, {}, pts, n, d, g, m);
}

// A query of distances (and materials) alone has one sample a point and object, for
// which a thread does: eight lanes serve it while they fit the chip.  16,000 /
// 65,536 / 500,000 points, 1 object: 27.5 / 35 / 97 us for eight lanes, 27 / 28.7 / 40
// for a thread; 12 objects 29.8 / 42 / 148 against 29.4 / 31 / 53; 24 objects 28.7 /
// 45.5 / 168 against 32.5 / 34 / 67; 120 objects 42 / 87 / 425 against 58 / 63 / 202.
constexpr uint32_t kWidePoints = 1u << 14, kWidePointsMany = 1u << 15;
template <int PREC>
void query_points(const Ctx* c, const float* pts, uint32_t n, float* d, float* g, uint16_t* m, cudaStream_t st) {
  const uint32_t n_objs = c->obj_count();
  if (!g && n >= (n_objs <= detail::kPointFewObjects ? kWidePoints : kWidePointsMany) && n_objs <= kMaxObjectsShared)
    query_points<PREC, 1>(c, pts, n, d, g, m, st);
  else
    query_points<PREC, detail::kPointLanes>(c, pts, n, d, g, m, st);
}

// Blocks of an occlusion launch: one for every 32 of its points or, where they copy
// the table and it holds more than kAoFewObjects objects, those that fit the chip
// (65,536 points, 60 / 100 / 163 / 198 objects: 68 / 94 / 177 / 257 us for a block per 32
// points, 62 / 90 / 152 / 209 so; but 1,000,000 points, 24 / 60 / 163 objects: 268 / 559 /
// 2,901 against 283 / 564 / 1,645).
constexpr uint32_t kAoFewObjects = 64;
unsigned ao_blocks(const Ctx* c, uint32_t n, uint32_t n_objs) {
  const unsigned all = (n - 1) / (128 / detail::kAoLanes) + 1;
  if (n_objs <= kAoFewObjects || n_objs > kMaxObjectsShared) return all;
  const unsigned fit = static_cast<unsigned>((227u << 10) / (sizeof(ObjSample) * n_objs + 1024u));
  return std::min(all, static_cast<unsigned>(c->sm_count) * std::max(1u, std::min(12u, fit)));
}

template <int PREC>
void sdf_ao(const Ctx* c, const SceneDev& s, const float* pos, const float* nrm, uint32_t n, float* ao,
            cudaStream_t st) {
  const unsigned blocks = ao_blocks(c, n, s.n_objs);
  if (s.n_objs <= kMaxObjectsShared)
    detail::k_sdf_ao<PREC, detail::TABLE_SHARED><<<blocks, 128, sizeof(ObjSample) * s.n_objs, st>>>(s, pos, nrm, n, ao);
  else
    detail::k_sdf_ao<PREC, detail::TABLE_DEVICE><<<blocks, 128, 0, st>>>(s, pos, nrm, n, ao);
}
}  // namespace

rkf_status launch_query(Ctx* c, const float* pts, uint32_t n, float* d, float* g, uint16_t* m,
                        cudaStream_t st) {
  if (n == 0) return RKF_OK;
  switch (c->cfg.precision) {
    case RKF_PRECISION_F32: query_points<RKF_PRECISION_F32>(c, pts, n, d, g, m, st); break;
    case RKF_PRECISION_U8: query_points<RKF_PRECISION_U8>(c, pts, n, d, g, m, st); break;
    default: query_points<RKF_PRECISION_F16>(c, pts, n, d, g, m, st);
  }
  c->counted();
  RKF_CUDA_TRY(cudaGetLastError());
  return RKF_OK;
}

rkf_status launch_ao(Ctx* c, const float* pos, const float* nrm, uint32_t n, float* ao, cudaStream_t st) {
  if (n == 0) return RKF_OK;
  const SceneDev s = c->scene_dev();
  switch (c->cfg.precision) {
    case RKF_PRECISION_F32: sdf_ao<RKF_PRECISION_F32>(c, s, pos, nrm, n, ao, st); break;
    case RKF_PRECISION_U8: sdf_ao<RKF_PRECISION_U8>(c, s, pos, nrm, n, ao, st); break;
    default: sdf_ao<RKF_PRECISION_F16>(c, s, pos, nrm, n, ao, st);
  }
  c->counted();
  RKF_CUDA_TRY(cudaGetLastError());
  return RKF_OK;
}

Segment view_segment(const rkf_camera* cam, uint32_t w, uint32_t h, uint32_t tile_w, uint32_t tile_h,
                     const rkf_gbuffer& out) {
  Segment sg;
  std::memset(&sg, 0, sizeof(sg));
  sg.kind = 0;
  sg.mode = RKF_TRACE_CLOSEST;
  sg.w = w;
  sg.h = h;
  if (!tile_w) tile_w = 8;
  if (!tile_h) tile_h = 4;
  sg.tiles_x = (w + tile_w - 1) / tile_w;
  const uint32_t tiles_y = (h + tile_h - 1) / tile_h;
  sg.n_ids = static_cast<uint64_t>(sg.tiles_x) * tiles_y * tile_w * tile_h;
  for (int a = 0; a < 3; ++a) {
    sg.pos[a] = cam->position[a];
    sg.fwd[a] = cam->forward[a];
    sg.right[a] = cam->right[a];
    sg.up[a] = cam->up[a];
  }
  sg.jitter[0] = cam->jitter[0];
  sg.jitter[1] = cam->jitter[1];
  std::memcpy(sg.prev_vp, cam->prev_vp, sizeof(sg.prev_vp));
  sg.t = out.t;
  sg.normal = out.normal;
  sg.slot = out.slot;
  sg.material = out.material;
  sg.flags = out.flags;
  sg.position = out.position;
  sg.packed = out.packed_material;
  sg.motion = out.motion;
  return sg;
}

Segment ray_segment(const float* o, const float* d, const float* tmax, uint32_t n, uint32_t mode,
                    const rkf_hits& out) {
  Segment sg;
  std::memset(&sg, 0, sizeof(sg));
  sg.kind = 1;
  sg.mode = mode;
  sg.n_ids = n;
  sg.origins = o;
  sg.dirs = d;
  sg.tmax = tmax;
  sg.t = out.t;
  sg.normal = out.normal;
  sg.slot = out.slot;
  sg.material = out.material;
  sg.flags = out.flags;
  return sg;
}

}  // namespace rkf

extern "C" int rkf_testing_last_variant(rkf_ctx* ctx) {
  return ctx ? reinterpret_cast<rkf::Ctx*>(ctx)->last_variant : -1;
}

extern "C" int rkf_testing_far_plane(const rkf_gpu_object* obj, float empty_hi, float out[6]) {
  if (!obj || !out) return 0;
  const rkf::ObjDev od = rkf::make_objdev(*obj, 0, 0);
  if (od.sdf_type != RKF_SDF_ANALYTICAL || od.prim_type != RKF_PRIM_PLANE) return 0;
  rkf::detail::FarBall b;
  if (!rkf::far_plane(od, empty_hi, &b)) return 0;
  out[0] = b.c[0];
  out[1] = b.c[1];
  out[2] = b.c[2];
  out[3] = b.h[0];
  out[4] = b.a;
  out[5] = b.b;
  return 1;
}

extern "C" int rkf_testing_far_ball(const rkf_gpu_object* obj, float empty_hi, float out[5]) {
  if (!obj || !out) return 0;
  const rkf::ObjDev od = rkf::make_objdev(*obj, 0, 0);
  rkf::detail::FarBall b;
  if (!rkf::far_ball(od, empty_hi, &b)) return 0;
  out[0] = b.c[0];
  out[1] = b.c[1];
  out[2] = b.c[2];
  out[3] = b.a;
  out[4] = b.b;
  return 1;
}
