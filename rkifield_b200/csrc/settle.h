// settle.h — the passes that settle a launch's views before the march.
#pragma once

#include "ctx.h"

namespace rkf {

namespace detail {
struct KParams;
}

// A launch's views, when they hold at least this many work ids, go through two
// passes before the march: one settles whole ray tiles, one the rays of the
// tiles that are left, and the march takes what remains.  Below it the march
// alone is as fast: its warps then have no second ray to go on to, so the
// passes' launches (about 4 us each) cost what they save.
constexpr uint64_t kSettleIds = 1u << 17;

// Device bytes the passes need for views of view_ids work ids in tiles of
// `area` of them.
size_t settle_bytes(uint64_t view_ids, uint32_t area);

// Enqueues the passes for the launch kp describes (an empty-space variant whose
// views' ids come first, view_ids of them below 2^32) on st, with their lists
// in ws, and points kp at what they leave.  obj: the launch's kernel variant.
rkf_status settle_enqueue(Ctx* c, detail::KParams& kp, int obj, uint64_t view_ids, void* ws, cudaStream_t st);

}  // namespace rkf
