/* A node that waits on the stack of a mesh traversal: 8 bytes. */
#ifndef HTRDR_BVH_ENTRY_H
#define HTRDR_BVH_ENTRY_H

#include <stdint.h>

#ifdef __CUDACC__
#define HG_HOST_DEVICE __host__ __device__
#else
#define HG_HOST_DEVICE
#endif

namespace hg {

struct BvhEntry {
  uint32_t first; /* first triangle, or the first child (any index of 32 bits) */
  uint32_t rest;  /* distance at which the ray enters, its last 3 bits the triangle count
                   * (0 to 7): less by a millionth part, far inside the slack of the
                   * test that drops entries */
};

HG_HOST_DEVICE inline BvhEntry
bvh_entry(uint32_t first, uint32_t count, uint32_t enter_bits)
{
  return BvhEntry{first, (enter_bits & ~7u) | count};
}
HG_HOST_DEVICE inline uint32_t bvh_count(BvhEntry e) { return e.rest & 7u; }
HG_HOST_DEVICE inline uint32_t bvh_enter_bits(BvhEntry e) { return e.rest & ~7u; }

}  // namespace hg

#endif /* HTRDR_BVH_ENTRY_H */
