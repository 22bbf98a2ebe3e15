// empty_dist.cu — the empty-space distance field over each object's top grid.
//
// For every block (8^3 bricks = 64^3 voxels) of an object's top grid the
// field holds 0 when the block is not EMPTY, else the Chebyshev distance, in
// blocks, to the nearest block that is not EMPTY, capped at kEmptyDistCap.
// Cells beyond the grid count as EMPTY.  So every block within distance
// (value - 1) of an EMPTY block is EMPTY too, and a ray position whose
// trilinear cell lies inside that cube samples the EMPTY constant: the march
// uses this to run those steps without touching the index.
//
// The L-infinity distance transform is separable: the distance along x, then
// the min over dy of max(|dy|, d_x), then the same over dz.  Edits only turn
// EMPTY blocks into leaf blocks, so after an edit the field is lowered around
// the touched blocks (a conservative bound that never overstates a distance).
#include <algorithm>

#include "ctx.h"
#include "empty_dist.h"

namespace rkf {

namespace detail {

struct GridDims {
  uint32_t off, nx, ny, nz;
};

// distance along x to the nearest non-EMPTY block of the row
__global__ void k_empty_dist_x(const uint32_t* __restrict__ top, uint8_t* __restrict__ out, GridDims g) {
  const uint64_t n = static_cast<uint64_t>(g.nx) * g.ny * g.nz;
  const uint64_t i = static_cast<uint64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const uint32_t x = static_cast<uint32_t>(i % g.nx);
  const uint32_t* row = top + g.off + (i - x);
  uint32_t d = 0;
  if (row[x] == RKF_EMPTY_SLOT) {
    for (d = 1; d < kEmptyDistCap; ++d) {
      if (x >= d && row[x - d] != RKF_EMPTY_SLOT) break;
      if (x + d < g.nx && row[x + d] != RKF_EMPTY_SLOT) break;
    }
  }
  out[i] = static_cast<uint8_t>(d);
}

// out = min over |k| of max(|k|, in at offset k along the axis)
__global__ void k_empty_dist_axis(const uint8_t* __restrict__ in, uint8_t* __restrict__ out, GridDims g,
                                  uint32_t axis) {
  const uint64_t n = static_cast<uint64_t>(g.nx) * g.ny * g.nz;
  const uint64_t i = static_cast<uint64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const uint32_t y = static_cast<uint32_t>((i / g.nx) % g.ny);
  const uint32_t z = static_cast<uint32_t>(i / (static_cast<uint64_t>(g.nx) * g.ny));
  const uint32_t pos = axis == 1 ? y : z;
  const uint32_t len = axis == 1 ? g.ny : g.nz;
  const uint64_t stride = axis == 1 ? g.nx : static_cast<uint64_t>(g.nx) * g.ny;
  uint32_t best = in[i];
  for (uint32_t k = 1; k < best; ++k) {
    if (pos >= k) best = min(best, max(k, static_cast<uint32_t>(in[i - k * stride])));
    if (pos + k < len) best = min(best, max(k, static_cast<uint32_t>(in[i + k * stride])));
  }
  out[i] = static_cast<uint8_t>(best);
}

// Lower the field around newly non-EMPTY blocks: field = min(field, distance
// to the nearest of them).  Cells cover the box [lo, hi] of the grid.
__global__ void k_empty_dist_lower(uint8_t* __restrict__ field, GridDims g, const uint32_t* __restrict__ blocks,
                                   uint32_t nb, uint3 lo, uint3 ext) {
  const uint64_t n = static_cast<uint64_t>(ext.x) * ext.y * ext.z;
  const uint64_t i = static_cast<uint64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const uint32_t x = lo.x + static_cast<uint32_t>(i % ext.x);
  const uint32_t y = lo.y + static_cast<uint32_t>((i / ext.x) % ext.y);
  const uint32_t z = lo.z + static_cast<uint32_t>(i / (static_cast<uint64_t>(ext.x) * ext.y));
  const uint64_t cell = g.off + x + static_cast<uint64_t>(y) * g.nx + static_cast<uint64_t>(z) * g.nx * g.ny;
  uint32_t v = field[cell];
  for (uint32_t b = 0; b < nb && v > 0; ++b) {
    const uint32_t l = blocks[b] - g.off;
    const int bx = static_cast<int>(l % g.nx), by = static_cast<int>((l / g.nx) % g.ny),
              bz = static_cast<int>(l / (g.nx * g.ny));
    const uint32_t d = static_cast<uint32_t>(
        max(abs(bx - static_cast<int>(x)), max(abs(by - static_cast<int>(y)), abs(bz - static_cast<int>(z)))));
    v = min(v, d);
  }
  field[cell] = static_cast<uint8_t>(v);
}

// One block per leaf block: the occupancy of the 24^3 bricks around it (its
// own block and the 26 next to it), then the separable Chebyshev transform
// over the block's own 8^3 bricks.  Shared memory bound; 14,500 leaf blocks
// (the 1.1M-brick scene) take about as long as k_empty_dist_x over that
// scene's 8.6M top cells.  The bytes of a block that an edit did not copy are
// read by older epochs' marches meanwhile: they only ever fall (edits turn
// EMPTY bricks into allocated ones), a lower value is valid for the older
// epoch too, and both sides use relaxed accesses.
__global__ void __launch_bounds__(256) k_leaf_dist(const uint32_t* __restrict__ top,
                                                   const uint32_t* __restrict__ leaves, uint8_t* leaf_dist,
                                                   GridDims g, const uint32_t* __restrict__ blocks, uint32_t n) {
  __shared__ uint8_t occ[24 * 24 * 24];
  __shared__ uint8_t dx[24 * 24 * 8];
  __shared__ uint8_t dy[24 * 8 * 8];
  if (blockIdx.x >= n) return;
  const uint32_t l = blocks[blockIdx.x] - g.off;
  const uint32_t leaf = top[g.off + l];
  if (leaf >= RKF_INTERIOR_SLOT) return;
  const int kx = static_cast<int>(l % g.nx), ky = static_cast<int>((l / g.nx) % g.ny),
            kz = static_cast<int>(l / (g.nx * g.ny));
  for (uint32_t w = threadIdx.x >> 5; w < 27; w += 8) {  // a warp per neighbouring block
    const int ax = static_cast<int>(w % 3), ay = static_cast<int>((w / 3) % 3), az = static_cast<int>(w / 9);
    const int x = kx + ax - 1, y = ky + ay - 1, z = kz + az - 1;
    uint32_t tv = RKF_EMPTY_SLOT;
    if (x >= 0 && y >= 0 && z >= 0 && x < static_cast<int>(g.nx) && y < static_cast<int>(g.ny) &&
        z < static_cast<int>(g.nz))
      tv = top[g.off + x + y * g.nx + z * g.nx * g.ny];
    for (uint32_t e = threadIdx.x & 31; e < 512; e += 32) {
      const uint32_t s = tv >= RKF_INTERIOR_SLOT ? tv : leaves[static_cast<size_t>(tv) * 512 + e];
      occ[(ax * 8 + (e & 7)) + (ay * 8 + ((e >> 3) & 7)) * 24 + (az * 8 + (e >> 6)) * 576] = s != RKF_EMPTY_SLOT;
    }
  }
  __syncthreads();
  for (uint32_t i = threadIdx.x; i < 24 * 24 * 8; i += 256) {
    const uint8_t* row = occ + (i >> 3) * 24 + 8 + (i & 7);
    uint32_t d = 0;
    if (!*row)
      for (d = 1; d < kLeafDistCap; ++d)
        if (row[-static_cast<int>(d)] || row[d]) break;
    dx[i] = static_cast<uint8_t>(d);
  }
  __syncthreads();
  for (uint32_t i = threadIdx.x; i < 24 * 64; i += 256) {
    const uint32_t x = i & 7, y = 8 + ((i >> 3) & 7), z = i >> 6;
    const uint8_t* col = dx + (z * 24 + y) * 8 + x;
    uint32_t best = *col;
    for (int k = 1; k < static_cast<int>(best); ++k)
      best = min(best, max(static_cast<uint32_t>(k), min(static_cast<uint32_t>(col[-8 * k]),
                                                         static_cast<uint32_t>(col[8 * k]))));
    dy[i] = static_cast<uint8_t>(best);
  }
  __syncthreads();
  for (uint32_t i = threadIdx.x; i < 512; i += 256) {
    const uint8_t* col = dy + i + 512;  // z + 8
    uint32_t best = *col;
    for (int k = 1; k < static_cast<int>(best); ++k)
      best = min(best, max(static_cast<uint32_t>(k), min(static_cast<uint32_t>(col[-64 * k]),
                                                         static_cast<uint32_t>(col[64 * k]))));
    store_leaf_dist(leaf_dist + static_cast<size_t>(leaf) * 512 + i, best);
  }
}

}  // namespace detail

rkf_status enqueue_leaf_dist(const ObjDev& o, const uint32_t* top, const uint32_t* leaves, uint8_t* leaf_dist,
                             const uint32_t* d_blocks, uint32_t n, cudaStream_t st) {
  if (n == 0) return RKF_OK;
  const detail::GridDims g{o.top_off, o.tdim[0], o.tdim[1], o.tdim[2]};
  detail::k_leaf_dist<<<n, 256, 0, st>>>(top, leaves, leaf_dist, g, d_blocks, n);
  RKF_CUDA_TRY(cudaGetLastError());
  return RKF_OK;
}

rkf_status build_leaf_dist(const ObjDev& o, const uint32_t* top, const uint32_t* leaves, uint8_t* leaf_dist,
                           const std::vector<uint32_t>& blocks, cudaStream_t st) {
  if (blocks.empty()) return RKF_OK;
  DevBuf list;
  rkf_status s = list.alloc(blocks.size() * 4);
  if (s != RKF_OK) return s;
  RKF_CUDA_TRY(cudaMemcpyAsync(list.p, blocks.data(), blocks.size() * 4, cudaMemcpyHostToDevice, st));
  s = enqueue_leaf_dist(o, top, leaves, leaf_dist, list.as<uint32_t>(), static_cast<uint32_t>(blocks.size()), st);
  RKF_CUDA_TRY(cudaStreamSynchronize(st));  // the list is freed on return
  return s;
}

std::vector<uint32_t> blocks_around(const ObjDev& o, const std::vector<uint32_t>& blocks) {
  std::vector<uint32_t> out;
  const int nx = static_cast<int>(o.tdim[0]), ny = static_cast<int>(o.tdim[1]), nz = static_cast<int>(o.tdim[2]);
  for (uint32_t b : blocks) {
    const int l = static_cast<int>(b - o.top_off), x = l % nx, y = (l / nx) % ny, z = l / (nx * ny);
    for (int c = std::max(z - 1, 0); c <= std::min(z + 1, nz - 1); ++c)
      for (int r = std::max(y - 1, 0); r <= std::min(y + 1, ny - 1); ++r)
        for (int q = std::max(x - 1, 0); q <= std::min(x + 1, nx - 1); ++q)
          out.push_back(o.top_off + static_cast<uint32_t>(q + r * nx + c * nx * ny));
  }
  std::sort(out.begin(), out.end());
  out.erase(std::unique(out.begin(), out.end()), out.end());
  return out;
}

rkf_status build_empty_dist(const ObjDev& o, const uint32_t* top, uint8_t* field, cudaStream_t st) {
  if (o.sdf_type != RKF_SDF_VOXELIZED) return RKF_OK;
  const detail::GridDims g{o.top_off, o.tdim[0], o.tdim[1], o.tdim[2]};
  const uint64_t n = static_cast<uint64_t>(g.nx) * g.ny * g.nz;
  if (n == 0) return RKF_OK;
  DevBuf tmp;
  rkf_status s = tmp.alloc(n);
  if (s != RKF_OK) return s;
  uint8_t* f = field + o.top_off;
  const unsigned blocks = static_cast<unsigned>((n + 255) / 256);
  detail::k_empty_dist_x<<<blocks, 256, 0, st>>>(top, f, g);
  detail::k_empty_dist_axis<<<blocks, 256, 0, st>>>(f, tmp.as<uint8_t>(), g, 1);
  detail::k_empty_dist_axis<<<blocks, 256, 0, st>>>(tmp.as<uint8_t>(), f, g, 2);
  RKF_CUDA_TRY(cudaGetLastError());
  // tmp is freed on return: finish its readers first
  RKF_CUDA_TRY(cudaStreamSynchronize(st));
  return RKF_OK;
}

rkf_status lower_empty_dist(const ObjDev& o, uint8_t* field, const uint32_t* d_blocks,
                            const std::vector<uint32_t>& blocks, cudaStream_t st) {
  if (o.sdf_type != RKF_SDF_VOXELIZED || blocks.empty()) return RKF_OK;
  const detail::GridDims g{o.top_off, o.tdim[0], o.tdim[1], o.tdim[2]};
  int lo[3] = {1 << 30, 1 << 30, 1 << 30}, hi[3] = {-1, -1, -1};
  for (uint32_t b : blocks) {
    const uint32_t l = b - g.off;
    const int c[3] = {static_cast<int>(l % g.nx), static_cast<int>((l / g.nx) % g.ny),
                      static_cast<int>(l / (g.nx * g.ny))};
    for (int a = 0; a < 3; ++a) {
      lo[a] = std::min(lo[a], c[a]);
      hi[a] = std::max(hi[a], c[a]);
    }
  }
  const int dims[3] = {static_cast<int>(g.nx), static_cast<int>(g.ny), static_cast<int>(g.nz)};
  const int reach = static_cast<int>(kEmptyDistCap) - 1;  // farther cells keep a value <= their distance
  uint3 l3, e3;
  uint32_t* lp = &l3.x;
  uint32_t* ep = &e3.x;
  for (int a = 0; a < 3; ++a) {
    const int a0 = std::max(0, lo[a] - reach), a1 = std::min(dims[a] - 1, hi[a] + reach);
    lp[a] = static_cast<uint32_t>(a0);
    ep[a] = static_cast<uint32_t>(a1 - a0 + 1);
  }
  const uint64_t n = static_cast<uint64_t>(e3.x) * e3.y * e3.z;
  detail::k_empty_dist_lower<<<static_cast<unsigned>((n + 255) / 256), 256, 0, st>>>(
      field, g, d_blocks, static_cast<uint32_t>(blocks.size()), l3, e3);
  RKF_CUDA_TRY(cudaGetLastError());
  return RKF_OK;
}

}  // namespace rkf
