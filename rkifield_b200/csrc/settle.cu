// settle.cu — views' misses before the march.
//
// Most rays of a view cross EMPTY space only: every sample they take clears
// every threshold, so they miss, with outputs that do not depend on the exact
// t at which they end (walk.cuh, walk_link).  The march's own walk settles such
// a ray in about 10 links of 100-200 instructions; these two passes do it for
// 32 rays at a time where they can, in kernels whose code is the walk alone (the
// march's many phases compete for the instruction caches), and hand the march
// full warps of the rays that have something to find.
//
//   k_settle_tiles  one lane per ray tile: a walk of the tile's whole beam (the
//                   centre ray and a bound of how far the tile's rays stray
//                   from it).  A settled tile's outputs are written by its
//                   warp; the others are listed.
//   k_settle_rays   one warp per listed tile: a walk per ray; what is not
//                   settled is listed for the march with how far its samples
//                   are EMPTY.
//
// Outputs are those of the march, bit for bit: t = MAX_FLOAT, zero normal and
// material, EMPTY slot, and STEPS_OUT exactly for the rays that run out of
// steps, which the walk's bounds decide (else the ray goes to the march).
#include "settle.h"

#include <algorithm>

#include "empty_dist.h"
#include "walk.cuh"

namespace rkf {

namespace detail {

struct SettleLists {
  uint32_t* counts;   // [0] tiles listed, [1] rays listed
  uint32_t* tiles;    // tile numbers (view ids / tile area)
  uint2* rays;        // {id, end of the EMPTY samples seen (NaN: none; several objects: no settling before this t)}
  uint32_t tile0, n_tiles;  // this part of the views' tiles
};

// A tile's rays: the centre ray's voxel coordinate g + d t on each axis, and d
// within `spread` for each of the tile's rays.  Mirrored like ProbeRay, the
// beam's upper edge moves at |d| + spread and its lower edge at |d| - spread
// (backwards when negative).
struct Beam {
  float g[3], d[3], spread, margin;
};

__device__ __forceinline__ int down_mask(const Beam& b, int a) { return __float_as_int(b.d[a]) >> 31; }
__device__ __forceinline__ float up_g(const ObjDev& o, const Beam& b, int a) {
  return b.d[a] < 0.0f ? small_float(o.mirror) - b.g[a] : b.g[a];
}

struct BeamBox {
  float in[3], out[3];
  float face[3];   // the box's upper face (mirrored voxel; infinite at the border)
  bool back;       // it leaves through a lower face first
};

// The EMPTY box around a voxel position (see empty_box), as the times the whole
// beam enters and any of it leaves.
__device__ __forceinline__ bool beam_box(const ObjDev& o, const SceneDev& s, const uint8_t* __restrict__ field,
                                         const Beam& b, const float* pos, BeamBox& x) {
  int v[3];
#pragma unroll
  for (int a = 0; a < 3; ++a) v[a] = near_int(fminf(fmaxf(pos[a] - 0.5f, 0.0f), o.last[a]));
  const uint32_t blk = o.top_off + (v[0] >> 6) + ((v[1] >> 6) + (v[2] >> 6) * o.tdim[1]) * o.tdim[0];
  uint32_t d = __ldg(field + blk);
  int shift = 6;
  if (d == 0) {
    const uint32_t leaf = __ldg(s.top + blk);
    if (leaf >= RKF_INTERIOR_SLOT) return false;
    d = load_leaf_dist(s.leaf_dist + static_cast<size_t>(leaf) * 512 +
                       (((v[0] >> 3) & 7) + (v[1] & 56) + (v[2] & 56) * 8));
    if (d == 0) return false;
    shift = 3;
  }
  const int above = static_cast<int>(d) << shift, unit = 1 << shift;
  float up_end = INFINITY, back_end = INFINITY;
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    const int down = down_mask(b, a);
    const int base = (v[a] ^ (down & o.mirror)) & -unit;
    const int first = down & (o.mirror - o.tv[a] + 1);
    const int lo = base + unit - above, hi = base + above - 1;
    const float g = up_g(o, b, a), fast = fabsf(b.d[a]) + b.spread, slow = fabsf(b.d[a]) - b.spread;
    const bool open_lo = lo <= first, open_hi = hi - first >= o.tv[a] - 1;
    const float t_lo = (small_float(lo) + b.margin - g) * rcp_approx(slow);  // the lower edge at the lower face
    const float t_hi = (small_float(hi) - b.margin - g) * rcp_approx(fast);
    x.face[a] = open_hi ? INFINITY : small_float(hi);
    x.in[a] = open_lo || !(slow > 0.0f) ? -INFINITY : t_lo;
    const float back = open_lo || slow > 0.0f ? INFINITY : t_lo;  // (slow = 0: t_lo infinite of either sign)
    x.out[a] = fminf(open_hi ? INFINITY : t_hi, back);
    up_end = fminf(up_end, open_hi ? INFINITY : t_hi);
    back_end = fminf(back_end, back);
  }
  x.back = back_end <= up_end;
  return true;
}

// The walk of a beam from t = 0 (walk_start, walk_link): true when EMPTY boxes
// hold it up to target.
__device__ __forceinline__ bool beam_walk(const ObjDev& o, const SceneDev& s, const uint8_t* __restrict__ field,
                                          const Beam& b, float target, uint32_t links) {
  BeamBox A;
  if (!(b.margin < 2.0f) || !beam_box(o, s, field, b, b.g, A)) return false;
  float end = fminf(fminf(A.out[0], A.out[1]), A.out[2]);
  if (!(fmaxf(fmaxf(A.in[0], A.in[1]), A.in[2]) <= 0.0f && end >= 0.0f)) return false;
#pragma unroll 1
  for (; end < target; --links) {
    if (!links || A.back) return false;
    const bool x0 = A.out[0] == end, x1 = !x0 && A.out[1] == end;  // the exit axis: 0, 1, else 2
    // just past the face on the exit axis, beside the centre ray on the others
    float pos[3];
#pragma unroll
    for (int a = 0; a < 3; ++a) {
      const bool exit = a == 0 ? x0 : a == 1 ? x1 : !(x0 || x1);
      const float past = A.face[a] + 2.0f;
      pos[a] = exit ? (b.d[a] < 0.0f ? small_float(o.mirror) - past : past) : __fmaf_rn(b.d[a], end, b.g[a]);
    }
    BeamBox B;
    if (!beam_box(o, s, field, b, pos, B)) return false;
    const float e = fminf(fminf(B.out[0], B.out[1]), B.out[2]);
    const float in2 = fmaxf(fmaxf(x0 ? -INFINITY : B.in[0], x1 ? -INFINITY : B.in[1]), x0 || x1 ? B.in[2] : -INFINITY);
    const float out2 = fminf(fminf(x0 ? INFINITY : A.out[0], x1 ? INFINITY : A.out[1]), x0 || x1 ? A.out[2] : INFINITY);
    // the exit axis: B begins where A's voxels end (it holds the voxel past
    // them); the whole beam has crossed the seam at in1
    const float in1 = x0 ? B.in[0] : x1 ? B.in[1] : B.in[2];
    const float slow = (x0 ? fabsf(b.d[0]) : x1 ? fabsf(b.d[1]) : fabsf(b.d[2])) - b.spread;
    const bool held = in2 <= end && (in1 <= end ? true : slow > 0.0f && out2 >= in1 && e >= in1);
    if (!held || !(e > end)) return false;
    end = e;
    A = B;
  }
  return true;
}

// How a view ray ends, from its start, when no sample ahead is below the EMPTY
// value: 1 past tmax, 2 out of steps, 0 undecided; target: the time up to
// which that must be known.  See the march's walk phase.
struct Ending {
  uint32_t kind;
  float target;
};

__device__ __forceinline__ bool thresholds_clear(const KParams& kp) {
  const rkf_march_params& p = kp.p;
  return kp.empty_lo >= fmaxf(p.scene.hit_threshold, 0.0f) && kp.empty_lo >= p.near_surface_threshold &&
         kp.empty_lo >= p.min_step && p.scene.max_steps > 0u && p.hard_max_steps > 0u && p.scene.max_distance >= 0.0f;
}

// The latest the last step can begin.
__device__ __forceinline__ float last_step(const KParams& kp) {
  const float k = static_cast<float>(kp.p.hard_max_steps - 1u);
  return k * kp.empty_hi * (1.0f + steps_grow(k));
}

// SINGLE: one voxelized object, brute strategy (or its equal); else any scene
// and strategy of the empty-space path (tiled launches only past tmax).
template <bool SINGLE>
__device__ __forceinline__ Ending tile_ending(const KParams& kp, const Beam& b, const ObjDev& o) {
  const float k = static_cast<float>(kp.p.hard_max_steps - 1u), tmax = kp.p.scene.max_distance;
  const float grow = steps_grow(k);
  const float t_lo = k * kp.empty_lo_t * (1.0f - grow), t_hi = last_step(kp);
  if (t_lo > tmax) return {1u, tmax};
  if (kp.tiled) return {0u, 0.0f};
  // the whole beam in the core interval (core_interval), and past the clamp box
  float t_out = INFINITY, t_o = INFINITY, c = 0.0f;
  bool core = true;
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    const float M = small_float(o.mirror), g = up_g(o, b, a);
    const bool dn = b.d[a] < 0.0f;
    const float lo = (dn ? M - o.core_hi[a] : o.core_lo[a]) + b.margin - g, hi = (dn ? M - o.core_lo[a] : o.core_hi[a]) - b.margin - g;
    const float fast = fabsf(b.d[a]) + b.spread, slow = fabsf(b.d[a]) - b.spread;
    core = core && lo <= 0.0f && hi >= 0.0f;
    t_out = fminf(t_out, hi * rcp_approx(fast));
    if (slow < 0.0f) t_out = fminf(t_out, lo * rcp_approx(slow));
    if (slow > 0.0f) {
      const float e = ((dn ? M : o.last[a]) + 0.5f + b.margin - g) * rcp_approx(slow);
      if (e < t_o) {
        t_o = e;
        c = slow * o.vs;
      }
    }
  }
  if (t_hi <= tmax && core && t_out >= t_hi) return {2u, t_hi};
  if (!SINGLE) return {0u, 0.0f};
  // leaves_grid, from t = 0, for every ray of the beam
  c *= o.min_scale * 0.998f;
  const float most =
      __fdividef(fmaxf(t_o * (1.0f + 2.0f * grow), 0.0f), kp.empty_lo_t) + __fdividef(2.0f, c) +
      __fdividef(__logf(fmaxf(__fdividef((tmax - t_o) * c, kp.empty_lo_t), 1.0f)), __logf(1.0f + c)) * 1.001f + 7.0f;
  if (most < k) return {1u, tmax};
  if (core && t_out < tmax && floorf(t_out * (1.0f - grow) / kp.empty_hi) - 2.0f >= k) return {2u, tmax};
  return {0u, 0.0f};
}

// One lane per tile of the launch's views.
template <bool SINGLE>
__global__ void __launch_bounds__(128) k_settle_tiles(const __grid_constant__ KParams kp, SettleLists ls) {
  const uint32_t at = blockIdx.x * blockDim.x + threadIdx.x, lane = threadIdx.x & 31u;
  const uint32_t tile = ls.tile0 + at, area = kp.tile_w * kp.tile_h;
  const bool live = at < ls.n_tiles;
  const uint32_t seg = live ? find_segment(kp.segs, kp.nseg, static_cast<uint64_t>(tile) * area) : 0u;
  const Segment& sg = kp.segs[seg];
  const uint32_t local = live ? tile - static_cast<uint32_t>(sg.first / area) : 0u;
  const uint32_t x0 = local % sg.tiles_x * kp.tile_w, y0 = local / sg.tiles_x * kp.tile_h;
  uint32_t kind = 0;
  if (live && thresholds_clear(kp)) {
    // the centre ray, and the most a ray of the tile differs from it: with w
    // the unnormalised direction and |w - wc| <= r over the tile, the unit
    // directions differ by at most r / (|wc| - r) (and the roundings of the
    // generated ones)
    const float u = (static_cast<float>(x0) + 0.5f * static_cast<float>(kp.tile_w) + sg.jitter[0]) / static_cast<float>(sg.w);
    const float v = (static_cast<float>(y0) + 0.5f * static_cast<float>(kp.tile_h) + sg.jitter[1]) / static_cast<float>(sg.h);
    const float nx = 2.0f * u - 1.0f, ny = 1.0f - 2.0f * v;
    float w[3], ww = 0.0f, rr = 0.0f, uu = 0.0f;
#pragma unroll
    for (int a = 0; a < 3; ++a) {
      w[a] = sg.fwd[a] + sg.right[a] * nx + sg.up[a] * ny;
      ww += w[a] * w[a];
      rr += sg.right[a] * sg.right[a];
      uu += sg.up[a] * sg.up[a];
    }
    const float len = sqrtf(ww);
    const float r = (sqrtf(rr) * static_cast<float>(kp.tile_w) / static_cast<float>(sg.w) +
                     sqrtf(uu) * static_cast<float>(kp.tile_h) / static_cast<float>(sg.h)) * 1.0001f;
    const float spread = r / (len - r) * 1.0001f + 4.0e-6f;
    if (len > 2.0f * r && len < kMaxRate && spread < 0.25f) {  // (a finite camera)
      // one walk per voxelized object of the path
      const uint32_t n_ev = SINGLE ? 1u : kp.n_ev;
      bool ok = true, exact = false;
      Ending end = {0u, 0.0f};
      for (uint32_t e = 0; ok && e < n_ev; ++e) {
        const ObjDev& o = kp.objs[SINGLE ? 0u : kp.ev[e].obj];
        Beam b;
        float mag = 1.0f;
#pragma unroll
        for (int a = 0; a < 3; ++a) mag += fabsf(sg.pos[a]) + o.mag[a];
        b.margin = 0.1f + mag * o.rcp_vs * 3.814697265625e-6f;
        b.spread = spread * o.rcp_vs;
#pragma unroll
        for (int a = 0; a < 3; ++a) {
          b.g[a] = (sg.pos[a] + o.m[12 + a] + o.half_gs[a]) * o.rcp_vs - 0.5f;
          b.d[a] = w[a] / len * o.rcp_vs;
        }
        const Ending here = tile_ending<SINGLE>(kp, b, o);
        if (e == 0) end = here;
        // several objects: out of steps needs one whose steps are exact so far
        exact = exact || here.kind != 0u;
        if (!SINGLE && here.kind) end = here;
        const float target = SINGLE || end.kind ? end.target : kp.tiled ? -1.0f : last_step(kp);
        ok = target >= 0.0f && beam_walk(o, kp.s, kp.brute_field, b, target, kWalkLinks);
      }
      ok = ok && exact && end.kind;
      if (!SINGLE && ok) {
        float again;
        const float lim = far_limit(kp.ball, kp.n_ball, (1u << kp.n_ev) - 1u, sg.pos[0], sg.pos[1], sg.pos[2],
                                    w[0] / len, w[1] / len, w[2] / len, kp.p.scene.max_distance, 0.0f,
                                    spread * end.target, again);
        ok = lim >= end.target;
      }
      if (ok) kind = end.kind;
    }
  }
  // ---- outputs of the settled tiles, a tile at a time ---------------------------
  for (uint32_t todo = __ballot_sync(kFull, kind != 0u); todo; todo &= todo - 1u) {
    const uint32_t L = __ffs(todo) - 1u;
    const uint32_t tseg = __shfl_sync(kFull, seg, L), tx = __shfl_sync(kFull, x0, L), ty = __shfl_sync(kFull, y0, L);
    const uint16_t flags = __shfl_sync(kFull, kind, L) == 2u ? RKF_FLAG_STEPS_OUT : 0;
    const Segment& ts = kp.segs[tseg];
    for (uint32_t i = lane; i < area; i += 32u) {
      const uint32_t px = tx + i % kp.tile_w, py = ty + i / kp.tile_w;
      if (px < ts.w && py < ts.h) write_miss(ts, py * ts.w + px, flags);
    }
  }
  // ---- the others, listed -------------------------------------------------------
  const bool left = live && kind == 0u;
  const uint32_t m = __ballot_sync(kFull, left);
  if (m) {
    uint32_t base = 0;
    if (lane == 0) base = atomicAdd(ls.counts, static_cast<uint32_t>(__popc(m)));
    base = __shfl_sync(kFull, base, 0);
    if (left) ls.tiles[base + __popc(m & ((1u << lane) - 1u))] = tile;
  }
}

// One warp per listed tile, in turn.
template <int OBJ>
__global__ void __launch_bounds__(256) k_settle_rays(const __grid_constant__ KParams kp, SettleLists ls) {
  constexpr bool SINGLE = OBJ == OBJ_SINGLE_EMPTY || OBJ == OBJ_SINGLE_EMPTY_TILED;
  const uint32_t lane = threadIdx.x & 31u, area = kp.tile_w * kp.tile_h;
  const uint32_t warps = gridDim.x * (blockDim.x >> 5), n = __ldcg(ls.counts);
  const bool clear = thresholds_clear(kp);
  const float tmax = kp.p.scene.max_distance;
  for (uint32_t li = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5); li < n; li += warps) {
    const uint32_t tile = __ldcg(ls.tiles + li);
    const Segment& sg = kp.segs[find_segment(kp.segs, kp.nseg, static_cast<uint64_t>(tile) * area)];
    const uint32_t local = tile - static_cast<uint32_t>(sg.first / area);
    const uint32_t x0 = local % sg.tiles_x * kp.tile_w, y0 = local / sg.tiles_x * kp.tile_h;
    for (uint32_t i0 = 0; i0 < area; i0 += 32u) {
      const uint32_t i = i0 + lane, px = x0 + i % kp.tile_w, py = y0 + i / kp.tile_w;
      const bool live = i < area && px < sg.w && py < sg.h;
      uint32_t kind = 0;
      float seen = __uint_as_float(0x7fc00000u);
      if (live && clear) {
        float dx, dy, dz;
        view_ray(sg, px, py, dx, dy, dz);
        dx = safe_dir(dx), dy = safe_dir(dy), dz = safe_dir(dz);
        const float k = static_cast<float>(kp.p.hard_max_steps - 1u);
        const float t_lo = k * kp.empty_lo_t * (1.0f - steps_grow(k)), t_hi = last_step(kp);
        if (SINGLE) {
          const ObjDev& o = kp.objs[0];
          const ProbeRay r = probe_ray(o, sg.pos[0], sg.pos[1], sg.pos[2], dx, dy, dz);
          float t_in, t_out;
          const bool core = core_interval(o, r, 0.0f, t_in, t_out);
          float target = core && !kp.tiled ? t_out : -1.0f;
          if (t_lo > tmax) {
            kind = 1;
            target = tmax;
          } else if (!kp.tiled) {
            if (t_hi <= tmax && core && t_out >= t_hi) {
              kind = 2;
              target = t_hi;
            } else {
              kind = leaves_grid(o, r, 0.0f, tmax, core, t_out, k, kp.empty_lo_t, kp.empty_hi);
              if (kind) target = tmax;
            }
          }
          if (target >= 0.0f) {
            const float end = walk_empty(o, kp.s, kp.brute_field, true, r, 0.0f, target, kWalkLinks);
            if (!(end >= target)) kind = 0;
            // (the tiled strategy's steps are EMPTY values on its own field only)
            if (!kp.tiled && core && end >= 0.0f) seen = fminf(end, t_out);
          }
        } else if (t_lo > tmax || (!kp.tiled && t_hi <= tmax)) {
          const uint32_t all = (1u << kp.n_ev) - 1u;
          const bool past = t_lo > tmax;
          const float target = past ? tmax : t_hi;
          float again;
          const float lim = far_limit(kp.ball, kp.n_ball, all, sg.pos[0], sg.pos[1], sg.pos[2], dx, dy, dz, tmax, 0.0f,
                                      0.0f, again);
          bool ok = lim >= target;
          seen = fmaxf(lim < 0.0f ? again : lim, after(0.0f));
          bool exact = past;
          for (uint32_t e = 0; ok && e < kp.n_ev; ++e) {
            const ObjDev& o = kp.objs[kp.ev[e].obj];
            const ProbeRay r = probe_ray(o, sg.pos[0], sg.pos[1], sg.pos[2], dx, dy, dz);
            const float end = walk_empty(o, kp.s, kp.brute_field, true, r, 0.0f, target, kWalkLinks);
            ok = end >= target;
            if (!ok) seen = fmaxf(end, after(0.0f));
            float t_in, t_out;
            exact = exact || (core_interval(o, r, 0.0f, t_in, t_out) && t_out >= target);
          }
          if (ok && exact) kind = past ? 1u : 2u;
        }
        if (kind) write_miss(sg, py * sg.w + px, kind == 2u ? RKF_FLAG_STEPS_OUT : 0);
      }
      const bool left = live && kind == 0u;
      const uint32_t m = __ballot_sync(kFull, left);
      if (m) {
        uint32_t base = 0;
        if (lane == 0) base = atomicAdd(ls.counts + 1, static_cast<uint32_t>(__popc(m)));
        base = __shfl_sync(kFull, base, 0);
        if (left) ls.rays[base + __popc(m & ((1u << lane) - 1u))] = make_uint2(tile * area + i, __float_as_uint(seen));
      }
    }
  }
}

}  // namespace detail

namespace {
size_t tile_bytes(uint64_t ids, uint32_t area) { return (ids / area * 4 + 255) & ~static_cast<size_t>(255); }
}  // namespace

size_t settle_bytes(uint64_t ids, uint32_t area) { return 256 + tile_bytes(ids, area) + ids * 8; }

uint64_t settle_part(Ctx* c, uint64_t view_ids, uint32_t area) {
  const uint64_t want = std::min(view_ids, kSettlePart / area * area);
  const size_t need = settle_bytes(want, area);
  if (c->settle_buf.bytes < need) {
    // (twice the last size at least, so that views that grow rarely come here; the
    // last buffer may be in use by a launch under way)
    const size_t most = settle_bytes(kSettlePart, area);
    auto grown = std::make_unique<DevBuf>();
    if (grown->alloc(std::min(std::max(need, 2 * c->settle_buf.bytes), std::max(most, need))) == RKF_OK) {
      std::swap(grown->p, c->settle_buf.p);
      std::swap(grown->bytes, c->settle_buf.bytes);
      if (grown->p) c->settle_old.push_back(std::move(grown));
    } else {
      cudaGetLastError();
    }
  }
  if (c->settle_buf.bytes >= need) return want;
  // (what is left of the buffer: 8 bytes an id, 4 a tile, 512 for the counts and the rounding)
  const uint64_t tiles = c->settle_buf.bytes > 512 ? (c->settle_buf.bytes - 512) / (8ull * area + 4) : 0;
  return tiles * area < want / kSettleParts ? 0 : tiles * area;
}

rkf_status settle_enqueue(Ctx* c, detail::KParams& kp, int obj, uint64_t first, uint64_t end, cudaStream_t st) {
  const uint32_t area = kp.tile_w * kp.tile_h;
  detail::SettleLists ls;
  ls.tile0 = static_cast<uint32_t>(first / area);
  ls.n_tiles = static_cast<uint32_t>((end - first) / area);
  char* b = c->settle_buf.as<char>();
  ls.counts = reinterpret_cast<uint32_t*>(b);
  ls.tiles = reinterpret_cast<uint32_t*>(b + 256);
  ls.rays = reinterpret_cast<uint2*>(b + 256 + tile_bytes(end - first, area));
  RKF_CUDA_TRY(cudaMemsetAsync(ls.counts, 0, 8, st));
  kp.list = nullptr;
  const unsigned blocks = (ls.n_tiles + 127u) / 128u;
  const bool single = obj == detail::OBJ_SINGLE_EMPTY || obj == detail::OBJ_SINGLE_EMPTY_TILED;
  if (single) detail::k_settle_tiles<true><<<blocks, 128, 0, st>>>(kp, ls);
  else detail::k_settle_tiles<false><<<blocks, 128, 0, st>>>(kp, ls);
  c->counted();
  RKF_CUDA_TRY(cudaGetLastError());
  const unsigned rb = std::min<unsigned>(static_cast<unsigned>(c->sm_count) * 8u, (ls.n_tiles + 7u) / 8u);
  if (single) detail::k_settle_rays<detail::OBJ_SINGLE_EMPTY><<<rb, 256, 0, st>>>(kp, ls);
  else detail::k_settle_rays<detail::OBJ_MULTI_EMPTY><<<rb, 256, 0, st>>>(kp, ls);
  c->counted();
  RKF_CUDA_TRY(cudaGetLastError());
  kp.list = ls.rays;
  kp.list_n = ls.counts + 1;
  kp.view_ids = end;
  return RKF_OK;
}

}  // namespace rkf
