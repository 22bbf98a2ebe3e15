// empty_dist.h — empty-space distance field over the top grids (empty_dist.cu).
#pragma once

#include <cuda_runtime.h>

#include <vector>

#include "device_common.cuh"

namespace rkf {

// Field values are capped here: a block this far from any non-EMPTY block
// only promises an EMPTY cube of radius kEmptyDistCap - 1 blocks.
constexpr uint32_t kEmptyDistCap = 64;

// Compute the field of object o's top grid (top[o.top_off ...]) into
// field[o.top_off ...].  Synchronises st.
rkf_status build_empty_dist(const ObjDev& o, const uint32_t* top, uint8_t* field, cudaStream_t st);

// Lower field[o.top_off ...] around `blocks` (global top indices, also on
// the device at d_blocks), which have just stopped being EMPTY.  Enqueued on
// st; d_blocks must stay valid until st reaches it.
rkf_status lower_empty_dist(const ObjDev& o, uint8_t* field, const uint32_t* d_blocks,
                            const std::vector<uint32_t>& blocks, cudaStream_t st);

// The same at brick resolution, inside the leaf blocks: one byte per leaf
// entry (leaf_dist[leaf * 512 + entry]), 0 for a brick that is not EMPTY, else
// the Chebyshev distance in bricks to the nearest one that is not, capped at
// kLeafDistCap, which looks into the 26 blocks around the leaf's own.  Every
// brick within (value - 1) of an EMPTY brick is EMPTY.
constexpr uint32_t kLeafDistCap = 8;

// Compute leaf_dist of the listed leaf blocks (global top indices; entries
// that are no leaf blocks are skipped) of object o from its top grid and
// leaves.  d_blocks: the list on the device.  Enqueued on st.
rkf_status enqueue_leaf_dist(const ObjDev& o, const uint32_t* top, const uint32_t* leaves, uint8_t* leaf_dist,
                             const uint32_t* d_blocks, uint32_t n, cudaStream_t st);
// The same for a list on the host.  Synchronises st.
rkf_status build_leaf_dist(const ObjDev& o, const uint32_t* top, const uint32_t* leaves, uint8_t* leaf_dist,
                           const std::vector<uint32_t>& blocks, cudaStream_t st);

// The listed blocks and every block next to one of them, each once: the
// blocks whose leaf_dist a change inside the listed ones can touch.
std::vector<uint32_t> blocks_around(const ObjDev& o, const std::vector<uint32_t>& blocks);

}  // namespace rkf
