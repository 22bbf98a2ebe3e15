// secondary.cu — shadow and ambient-occlusion rays from a view's G-buffer.
//
// The reference's shading pass (shade_main.wgsl, shade_common_shading.wgsl:
// 9-47) turns every hit pixel into shadow queries towards the lights and
// ambient-occlusion queries about the normal.  This kernel builds those
// queries as ray batches for the batched march: per pixel, n_lights shadow
// rays (origin = hit + normal * shadow_bias, towards each point light,
// tmax = distance to it) and ao_per_hit cosine-weighted hemisphere rays
// (origin = hit + normal * ao_bias, tmax = ao_radius).  Pixel p owns ray
// slots [p*n, p*n + n); pixels that missed get tmax = -1, which ends the ray
// on its first iteration, so the layout needs no compaction and is
// deterministic.  Directions come from a counter-based hash of
// (seed, pixel, ray), so the rays do not depend on launch order.
#include <cstring>

#include "ctx.h"

namespace rkf {
namespace detail {

__device__ __forceinline__ uint32_t hash32(uint32_t x) {
  // integer finaliser of MurmurHash3 (Appleby)
  x ^= x >> 16;
  x *= 0x85ebca6bu;
  x ^= x >> 13;
  x *= 0xc2b2ae35u;
  x ^= x >> 16;
  return x;
}

__device__ __forceinline__ float unit_float(uint32_t h) {
  return static_cast<float>(h >> 8) * (1.0f / 16777216.0f);  // [0, 1)
}

struct SecParams {
  float pos[3], fwd[3], right[3], up[3];
  uint32_t w, h;
  const float* t;
  const float* normal;
  const uint16_t* flags;
  float lights[3 * 16];
  uint32_t n_lights, ao_per_hit;
  uint32_t pixels, shadow_blocks;
  float ao_radius, shadow_bias, ao_bias;
  uint32_t seed;
  float* so;
  float* sd;
  float* st;
  float* ao;
  float* ad;
  float* at;
  unsigned int* hits;
};

// A pixel's surface point and normal.
struct SecHit {
  float x, y, z, nx, ny, nz;
  bool hit;
};
__device__ __forceinline__ SecHit load_hit(const SecParams& k, uint32_t i, bool live) {
  SecHit h{0, 0, 0, 0, 1, 0, live && (k.flags[i] & RKF_FLAG_HIT) != 0};
  if (h.hit) {
    const uint32_t px = i % k.w, py = i / k.w;
    const float u = (static_cast<float>(px) + 0.5f) / static_cast<float>(k.w);
    const float v = (static_cast<float>(py) + 0.5f) / static_cast<float>(k.h);
    float dx = k.fwd[0] + (u * 2.0f - 1.0f) * k.right[0] + (1.0f - v * 2.0f) * k.up[0];
    float dy = k.fwd[1] + (u * 2.0f - 1.0f) * k.right[1] + (1.0f - v * 2.0f) * k.up[1];
    float dz = k.fwd[2] + (u * 2.0f - 1.0f) * k.right[2] + (1.0f - v * 2.0f) * k.up[2];
    const float il = rsqrtf(dx * dx + dy * dy + dz * dz);
    dx *= il;
    dy *= il;
    dz *= il;
    const float t = k.t[i];
    h.x = k.pos[0] + dx * t;
    h.y = k.pos[1] + dy * t;
    h.z = k.pos[2] + dz * t;
    h.nx = k.normal[3 * static_cast<size_t>(i)];
    h.ny = k.normal[3 * static_cast<size_t>(i) + 1];
    h.nz = k.normal[3 * static_cast<size_t>(i) + 2];
  }
  return h;
}

// The ray to light l.
__device__ __forceinline__ float shadow_ray(const SecParams& k, const SecHit& h, uint32_t l, float* o, float* d) {
  const float ox = h.x + h.nx * k.shadow_bias, oy = h.y + h.ny * k.shadow_bias, oz = h.z + h.nz * k.shadow_bias;
  float dx = k.lights[3 * l] - ox, dy = k.lights[3 * l + 1] - oy, dz = k.lights[3 * l + 2] - oz;
  const float len = sqrtf(dx * dx + dy * dy + dz * dz);
  const float il = len > 0.0f ? 1.0f / len : 0.0f;
  o[0] = ox;
  o[1] = oy;
  o[2] = oz;
  d[0] = dx * il;
  d[1] = dy * il;
  d[2] = dz * il;
  return h.hit ? len : -1.0f;
}

// Tangent frame of a normal.
struct SecFrame {
  float tx, ty, tz, bx, by, bz;
};
__device__ __forceinline__ SecFrame frame_of(const SecHit& h) {
  const float ax = fabsf(h.nx) < 0.9f ? 1.0f : 0.0f, ay = fabsf(h.nx) < 0.9f ? 0.0f : 1.0f;
  float tx = ay * h.nz, ty = -ax * h.nz, tz = ax * h.ny - ay * h.nx;  // a x n
  const float itl = rsqrtf(fmaxf(tx * tx + ty * ty + tz * tz, 1e-20f));
  tx *= itl;
  ty *= itl;
  tz *= itl;
  return {tx, ty, tz, h.ny * tz - h.nz * ty, h.nz * tx - h.nx * tz, h.nx * ty - h.ny * tx};
}

// Ambient-occlusion ray a of pixel i.
__device__ __forceinline__ float ao_ray(const SecParams& k, const SecHit& h, const SecFrame& f, uint32_t i, uint32_t a,
                                        float* o, float* d) {
  const uint32_t h0 = hash32(k.seed ^ hash32(i * 0x9E3779B9u + a));
  const float r1 = unit_float(h0), r2 = unit_float(hash32(h0 ^ 0x68bc21ebu));
  const float rr = sqrtf(r1), phi = 6.28318530718f * r2;
  const float lx = rr * cosf(phi), ly = rr * sinf(phi), lz = sqrtf(fmaxf(0.0f, 1.0f - r1));
  o[0] = h.x + h.nx * k.ao_bias;
  o[1] = h.y + h.ny * k.ao_bias;
  o[2] = h.z + h.nz * k.ao_bias;
  d[0] = lx * f.tx + ly * f.bx + lz * h.nx;
  d[1] = lx * f.ty + ly * f.by + lz * h.ny;
  d[2] = lx * f.tz + ly * f.bz + lz * h.nz;
  return h.hit ? k.ao_radius : -1.0f;
}

// One thread per ray, in the order of the output arrays: blocks below
// shadow_blocks write shadow rays, the others ambient-occlusion rays.  Bound by
// its stores (28 bytes a ray), which a thread per pixel spread over 12-byte
// pieces n_lights * 12 (ao_per_hit * 12) bytes apart: the block's vectors go
// through shared memory to whole lines instead, and a block adds its hits with
// one atomic.  Four views of 1.25M pixels together, 28 bytes a ray: 494 us for a
// thread per pixel, 178 us so, now bound by its arithmetic (90% issue).
constexpr uint32_t kSecRays = 256;

__global__ void __launch_bounds__(kSecRays) k_secondary(SecParams k) {
  __shared__ float sh_o[3 * kSecRays], sh_d[3 * kSecRays];
  const bool shadow = blockIdx.x < k.shadow_blocks;
  const uint32_t per = shadow ? k.n_lights : k.ao_per_hit;  // rays per pixel
  // the block's first ray, its pixel and its place among the pixel's rays
  const uint64_t r0 = static_cast<uint64_t>(shadow ? blockIdx.x : blockIdx.x - k.shadow_blocks) * kSecRays;
  const uint64_t n = static_cast<uint64_t>(k.pixels) * per;
  const uint64_t i0 = r0 / per;
  const uint32_t at = static_cast<uint32_t>(r0 - i0 * per) + threadIdx.x;
  const uint32_t i = static_cast<uint32_t>(i0) + at / per;
  const uint32_t l = at % per;
  const bool live = r0 + threadIdx.x < n;
  const SecHit h = load_hit(k, i, live);
  // (the first kind of ray there is counts a pixel)
  const int hits = __syncthreads_count(h.hit && l == 0 && (shadow || k.shadow_blocks == 0));
  if (threadIdx.x == 0 && hits) atomicAdd(k.hits, static_cast<unsigned int>(hits));
  float* so = sh_o + 3 * threadIdx.x;
  float* sd = sh_d + 3 * threadIdx.x;
  const float tmax = shadow ? shadow_ray(k, h, l, so, sd) : ao_ray(k, h, frame_of(h), i, l, so, sd);
  if (live) (shadow ? k.st : k.at)[r0 + threadIdx.x] = tmax;
  __syncthreads();
  const uint32_t words = 3 * static_cast<uint32_t>(n - r0 < kSecRays ? n - r0 : kSecRays);
  float* o = (shadow ? k.so : k.ao) + 3 * r0;
  float* d = (shadow ? k.sd : k.ad) + 3 * r0;
  for (uint32_t e = threadIdx.x; e < words; e += kSecRays) {
    o[e] = sh_o[e];
    d[e] = sh_d[e];
  }
}

// A thread per pixel, which takes its point and its tangent frame once: where a
// pixel has one or two occlusion rays, and at most two shadow rays, its pieces of a
// line are few enough.  1920x1080, 0+1 / 0+2 / 1+1 / 1+2 / 2+1 / 2+2 lights and occlusion
// rays: 55 / 76 / 64 / 80 / 85 / 113 us so, 60 / 88 / 76 / 103 / 101 / 126 for a thread per
// ray; 3+2 225 against 151, 1+4 252 against 163; no occlusion, 1 / 2 / 4 lights 55 / 76 / 250
// against 51 / 76 / 113.  (A ray's values are stored when all are known: through the
// functions' pointers 2+1 took 93.)
constexpr uint32_t kFewRays = 2;

__device__ __forceinline__ void store_ray(float* o, float* d, float* t, size_t r, const float* vo, const float* vd,
                                          float vt) {
#pragma unroll
  for (int c = 0; c < 3; ++c) o[3 * r + c] = vo[c];
#pragma unroll
  for (int c = 0; c < 3; ++c) d[3 * r + c] = vd[c];
  t[r] = vt;
}

__global__ void k_secondary_pixels(SecParams k) {
  const uint64_t id = static_cast<uint64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
  if (id >= k.pixels) return;
  const uint32_t i = static_cast<uint32_t>(id);
  const SecHit h = load_hit(k, i, true);
  if (h.hit) atomicAdd(k.hits, 1u);
  float o[3], d[3];
  for (uint32_t l = 0; l < k.n_lights; ++l) {
    const float t = shadow_ray(k, h, l, o, d);
    store_ray(k.so, k.sd, k.st, static_cast<size_t>(i) * k.n_lights + l, o, d, t);
  }
  const SecFrame f = frame_of(h);
  for (uint32_t a = 0; a < k.ao_per_hit; ++a) {
    const float t = ao_ray(k, h, f, i, a, o, d);
    store_ray(k.ao, k.ad, k.at, static_cast<size_t>(i) * k.ao_per_hit + a, o, d, t);
  }
}

// The hits alone, of a call that asks for no rays.
__global__ void k_count_hits(SecParams k) {
  const uint64_t i = static_cast<uint64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
  const int hits = __syncthreads_count(i < k.pixels && (k.flags[i] & RKF_FLAG_HIT) != 0);
  if (threadIdx.x == 0 && hits) atomicAdd(k.hits, static_cast<unsigned int>(hits));
}

}  // namespace detail
}  // namespace rkf

using namespace rkf;

extern "C" rkf_status rkf_secondary_rays(rkf_ctx* ctx, const rkf_camera* cam, uint32_t w, uint32_t h,
                                         const rkf_gbuffer* gb, const float* lights, uint32_t n_lights,
                                         uint32_t ao_per_hit, float ao_radius, uint32_t seed,
                                         float* shadow_o, float* shadow_d, float* shadow_tmax,
                                         float* ao_o, float* ao_d, float* ao_tmax,
                                         uint32_t* hit_pixels, void* stream) {
  if (!ctx || !cam || !gb || (n_lights && !lights) || !hit_pixels)
    return fail(RKF_INVALID_ARG, "rkf_secondary_rays: null argument");
  if (gb->mem != RKF_MEM_DEVICE || !gb->t || !gb->normal || !gb->flags)
    return fail(RKF_INVALID_ARG, "rkf_secondary_rays: device G-buffer required");
  if (n_lights > 16) return fail(RKF_INVALID_ARG, "rkf_secondary_rays: at most 16 lights");
  if ((n_lights && (!shadow_o || !shadow_d || !shadow_tmax)) || (ao_per_hit && (!ao_o || !ao_d || !ao_tmax)))
    return fail(RKF_INVALID_ARG, "rkf_secondary_rays: missing output array");
  if (w == 0 || h == 0) return fail(RKF_INVALID_ARG, "rkf_secondary_rays: empty view");
  Ctx* c = reinterpret_cast<Ctx*>(ctx);
  RKF_CUDA_TRY(cudaSetDevice(c->device));
  cudaStream_t st = stream ? static_cast<cudaStream_t>(stream) : c->stream;
  detail::SecParams k;
  std::memset(&k, 0, sizeof(k));
  for (int a = 0; a < 3; ++a) {
    k.pos[a] = cam->position[a];
    k.fwd[a] = cam->forward[a];
    k.right[a] = cam->right[a];
    k.up[a] = cam->up[a];
  }
  k.w = w;
  k.h = h;
  k.t = gb->t;
  k.normal = gb->normal;
  k.flags = gb->flags;
  std::memcpy(k.lights, lights, sizeof(float) * 3 * n_lights);
  k.n_lights = n_lights;
  k.ao_per_hit = ao_per_hit;
  k.ao_radius = ao_radius;
  k.shadow_bias = 0.08f;  // SHADOW_BIAS (shade_common.wgsl:276)
  k.ao_bias = 0.02f;
  k.seed = seed;
  k.so = shadow_o;
  k.sd = shadow_d;
  k.st = shadow_tmax;
  k.ao = ao_o;
  k.ad = ao_d;
  k.at = ao_tmax;
  unsigned int* dh = reinterpret_cast<unsigned int*>(c->counters.as<char>() + 256);
  RKF_CUDA_TRY(cudaMemsetAsync(dh, 0, 4, st));
  k.hits = dh;
  k.pixels = w * h;
  const uint64_t n = k.pixels;
  const uint64_t shadow_blocks = (n * n_lights + detail::kSecRays - 1) / detail::kSecRays;
  const uint64_t blocks = shadow_blocks + (n * ao_per_hit + detail::kSecRays - 1) / detail::kSecRays;
  if (blocks > 0x7FFFFFFFull) return fail(RKF_INVALID_ARG, "rkf_secondary_rays: too many rays");
  k.shadow_blocks = static_cast<uint32_t>(shadow_blocks);
  if (ao_per_hit && ao_per_hit <= detail::kFewRays && n_lights <= detail::kFewRays) {
    detail::k_secondary_pixels<<<static_cast<unsigned>((n + 255) / 256), 256, 0, st>>>(k);
  } else if (blocks) {
    detail::k_secondary<<<static_cast<unsigned>(blocks), detail::kSecRays, 0, st>>>(k);
  } else {
    detail::k_count_hits<<<static_cast<unsigned>((n + 255) / 256), 256, 0, st>>>(k);
  }
  c->counted();
  RKF_CUDA_TRY(cudaGetLastError());
  RKF_CUDA_TRY(cudaMemcpyAsync(hit_pixels, dh, 4, cudaMemcpyDeviceToHost, st));
  RKF_CUDA_TRY(cudaStreamSynchronize(st));
  return RKF_OK;
}
