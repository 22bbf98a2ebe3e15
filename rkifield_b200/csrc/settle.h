// settle.h — the passes that settle a launch's views before the march.
#pragma once

#include "ctx.h"

namespace rkf {

namespace detail {
struct KParams;
}

// A launch's views, when they hold at least this many work ids, go through two
// passes before the march: one settles whole ray tiles, one the rays of the
// tiles that are left, and the march takes what remains.  Below it the march alone
// is faster: its warps have no second ray to go on to, so what the passes take is
// added.  us with / without them (default tuning; mean of three cameras), 32 m scene seen
// from outside: 160x90 413 / 249, 256x144 480 / 372, 400x225 509 / 496, 480x270 557 / 551, 640x360
// 613 / 599, 960x540 770 / 847, 1280x720 995 / 1,178.  Cameras inside the 1.1M-brick
// scene, where few tiles settle: 256x144 331 / 268, 480x270 439 / 385, 960x540 643 / 544,
// 1280x720 717 / 666 -- for such views the line lies too low.
constexpr uint64_t kSettleIds = 1u << 17;

// A launch's views are settled and marched in parts of at most this many ids, which
// bounds the passes' lists (604 MB in tiles of 32 ids): 32 views of 1920x1080.
constexpr uint64_t kSettlePart = 1u << 26;

// Device bytes the passes need for `ids` work ids in tiles of `area` of them.
size_t settle_bytes(uint64_t ids, uint32_t area);

// The ids of a part for views of view_ids work ids, a multiple of area or all of
// them: the context's lists grow for it, or, where there is no room, it is what they
// hold.  0: no lists, or so small that the views would take more than kSettleParts.
constexpr uint64_t kSettleParts = 8;
uint64_t settle_part(Ctx* c, uint64_t view_ids, uint32_t area);

// Enqueues the passes over work ids [first, end) of the launch kp describes (an
// empty-space variant whose views' ids come first, below 2^32; first a multiple of
// the tiles' ids) on st, with the context's lists, and points kp at what they leave.
// obj: the launch's kernel variant.
rkf_status settle_enqueue(Ctx* c, detail::KParams& kp, int obj, uint64_t first, uint64_t end, cudaStream_t st);

}  // namespace rkf
