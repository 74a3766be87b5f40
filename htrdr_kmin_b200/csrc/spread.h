/* How many lanes of each warp of a launch take paths. */
#ifndef HTRDR_SPREAD_H
#define HTRDR_SPREAD_H

#include <stdint.h>

#ifdef __CUDACC__
#define HG_HOST_DEVICE __host__ __device__
#else
#define HG_HOST_DEVICE
#endif

namespace hg {

/* Lanes of warp `warp' (of `warps') that run, with `left' paths to go and room
 * for `room' in flight.  Few paths are spread over all warps, as a warp with a
 * single path takes its bounces fastest.  The warps' shares of the room add up
 * to it and do not depend on `left', which the warps of a launch may read
 * differently while others take work: never more than `room' lanes in all, and
 * no fewer than min(left, room). */
HG_HOST_DEVICE inline uint32_t
warp_lanes(uint64_t warp, uint64_t warps, uint64_t room, uint64_t left)
{
  const uint64_t share = room / warps + (warp < room % warps ? 1 : 0);
  const uint64_t want = (left + warps - 1) / warps;
  const uint64_t n = share < want ? share : want;
  return n < 32 ? (uint32_t)n : 32u;
}

}  // namespace hg

#endif /* HTRDR_SPREAD_H */
