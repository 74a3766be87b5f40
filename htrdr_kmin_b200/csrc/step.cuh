/* The step loop: a lane per path, the paths of a warp kept in step.
 *
 * A shortwave bounce is a free path, the absorption along it, the scattering
 * and a transmissivity towards the sun; the loop goes through these phases
 * with all paths of the warp, so that the events of a phase and its trace run
 * with every lane that bounces.  Longwave paths have the first phase only.
 * A lane whose path ends takes the next one from its Work (the work queue, a
 * saved pool, a caller's rays).
 *
 * What bounds it: the instruction stream of a shortwave bounce (some 3500
 * instructions, run once from end to end: half of the stalls of a full SM wait
 * for instructions) and, in the last third of a run, the latency of the
 * longest path's bounces (~9 us each).  Hence one copy of every routine in the
 * loop, all lanes of a warp in one phase, and the traces' frequent part apart
 * (cell_walk).  Lanes regrouped at every voxel step instead, in whatever state
 * they are, took 41 us a bounce at the tail of a small image and 72 us at the
 * tail of a flux map; 47 and 128 ms against 12 and 27 ms for the whole calls. */
#ifndef HTRDR_STEP_CUH
#define HTRDR_STEP_CUH

#include "engine.cuh"
#include "walk.cuh"

namespace {

/* Registers of the kernels that run the loop.  Shortwave: all of them (8 warps
 * per SM) against 168 (12): a batch of 32 images 293 against 341 ms, a flux map
 * of 88 000 realisations 27.3 against 28.0, a CIE image 15.3 against 15.6.
 * Longwave, whose bounces are short: 128 (16 warps) against 96, 112 and 168:
 * 13.9, 15.7, 14.7 and 18.0 ms for a flux map of 4.2 M realisations, 11.1, 12.5,
 * 11.7 and 12.8 for an image of 2.3 M. */
__host__ __device__ constexpr int
step_registers(unsigned v)
{
  return (v & HV_SW) ? 255 : 128;
}
/* A phase's trace goes on until a quarter of the warp's paths is left in it;
 * these go on when the phase comes round again.  1/4, 1/8 and 1/16: a batch of
 * 32 images 293, 297 and 308 ms, single maps within 2 %. */
constexpr uint32_t kStepLag = 4;
/* Idle lanes that make a warp take new work (the sensor and spectral sampling
 * is the longest piece of code, so it waits for a few lanes), and the lanes of
 * a longwave warp that go on scattering without the others.  Measured on the
 * longwave flux map and image (idle lanes, lanes): 8, 24 16.0 and 12.7 ms; 8, 16
 * 13.8 and 11.2; 16, 12 13.9 and 11.1; 20, 5 17.1 and 12.3. */
__host__ __device__ constexpr uint32_t
step_refill(unsigned v)
{
  return (v & HV_SW) ? 8 : 16;
}
constexpr uint32_t kStepLwLanes = 12;
/* Lanes of a longwave warp that take a gas region together: several times the
 * code of a cell, reached by a lane or two at a step.  Measured (1 / 2 / 4 / 6 /
 * 8 / 14): a flux map of 4.2 M realisations 15.1 / 14.5 / 14.2 / 14.3 / 14.9 /
 * 18.7 ms, an image of 2.3 M 11.4 / 11.2 / 10.9 / 10.9 / 11.1 / 12.3 ms. */
constexpr uint32_t kStepLwGas = 4;
/* Cloud voxels of a longwave trace at a turn of the warp where there is no
 * majorant grid to walk: a turn's other work is worth a voxel of the tree's
 * descent.  Measured (1 / 2 / 4 / 16) without any grid: a flux map of 4.2 M
 * realisations 25.7 / 24.1 / 26.7 / 27.2 ms (a wavefront of stage kernels took
 * 24.0), an image of 2.3 M 21.5 / 19.3 / 21.0 / 21.3 ms. */
constexpr int kStepLwVoxels = 2;

/* Event part of a lane's path: in shared memory, an odd number of 8-byte
 * words apart, so that a warp's 8-byte accesses to one field do not conflict */
static_assert(sizeof(PathEvent) % 16 == 8, "odd number of 8-byte words per slot");
__host__ __device__ constexpr size_t
step_event_bytes(uint32_t threads)
{
  return (sizeof(PathEvent) * threads + 15) & ~(size_t)15;
}

/* Runs paths until `work' has no more, or asks to stop: then the lanes' paths
 * are handed to work.save().  Work:
 *   scenes, request(e)  the tables of a path
 *   stop(n)             whether to stop, with n live paths (warp-uniform)
 *   take(want, p, e)    gives the lanes of `want' a path each, or leaves them
 *                       idle when there is none left (all lanes call it);
 *                       returns whether this lane may ask again
 *   done(p, e)          a path in ST_DONE */
template <unsigned V, class Work>
__device__ __forceinline__ void
step_loop(Work& work, PathTrace& p, PathEvent& e, bool drained)
{
  p.state = ST_IDLE;
  p.flags = 0;
  p.c_seg = p.c_node = p.c_tc = 0;
  p.si = 0;
  for(;;) {
    const unsigned live = __ballot_sync(HG_FULL, p.state != ST_IDLE);
    if(work.stop((uint32_t)__popc(live))) { work.save(p, e); return; }
    const unsigned idle = __ballot_sync(HG_FULL, p.state == ST_IDLE && !drained);
    if(idle && (!live || __popc(idle) >= step_refill(V))) {
      const bool more = work.take(p.state == ST_IDLE && !drained, p, e);
      drained = drained || !more;
    }
    const uint32_t n = (uint32_t)__popc(__ballot_sync(HG_FULL, p.state != ST_IDLE));
    if(!n) {
      if(__all_sync(HG_FULL, drained)) return;
      continue;
    }
    uint32_t lag = n / kStepLag;
    if constexpr(!(V & HV_SW))
      if(!__any_sync(HG_FULL, drained)) lag = kStepLwLanes;
    for(int ph = 0; ph < ((V & HV_SW) ? 3 : 1); ++ph) {
      const int evph = p.state == ST_SW_SCAT_END ? 1 : (p.state == ST_SW_ABS_END ? 2 : 0);
      if(p.state != ST_IDLE && p.state != ST_TRACE && p.state != ST_DONE && evph == ph)
        path_event<V>(p, e, work.scenes[p.si], work.request(e));
      const int trph = p.tr.kind != TK_TRANS ? 0 : (p.tr.prop == HG_KA ? 1 : 2);
      for(uint32_t it = 0;; ++it) {
        const bool act = p.state == ST_TRACE && trph == ph;
        const uint32_t na = (uint32_t)__popc(__ballot_sync(HG_FULL, act));
        if(!na || (it && na <= lag)) break;
        bool walk = false;
        if(act) {
          trace_enter(p.tr, work.scenes[p.si]);
          /* an absorption trace crosses one merged leaf most often */
          walk = (ph != 1 || it) && p.tr.has_cloud && p.tr.region == 1 && walk_fits(p.tr, work.scenes[p.si]);
        }
        if(ph == 0) cell_walk<V, false>(p, work.scenes, walk);
        else if(V & HV_SW) cell_walk<V, true>(p, work.scenes, walk);
        __syncwarp();
        bool go = act && p.state == ST_TRACE;
        if constexpr(!(V & HV_SW)) {
          /* lanes at a gas region wait for others, as long as there is anything
           * else to do */
          const bool gas = go && !(p.tr.has_cloud && p.tr.region == 1);
          const unsigned waits = __ballot_sync(HG_FULL, gas);
          const unsigned others = __ballot_sync(HG_FULL, act && !gas);
          if(others && __popc(waits) < kStepLwGas) go = go && !gas;
        }
        if(go) {
          const DScene& S = work.scenes[p.si];
          int voxels = (V & HV_SW) || S.maj_grid ? 1 : kStepLwVoxels;
          do trace_step<V>(p, S);
          while(--voxels && p.state == ST_TRACE && p.tr.has_cloud && p.tr.region == 1);
        }
        if constexpr(!(V & HV_SW)) {
          /* a longwave scattering over a plane ground: on with the walk */
          if(act && p.state == ST_LW_END && p.tr.hit && p.tr.event == 1 && p.bounces < HG_MAX_BOUNCES
          && lw_plane_ground<V>(work.scenes[p.si])) {
            TraceArgs q;
            lw_scatter_plane(p, work.scenes[p.si], q);
            e.pos = q.o;
            e.dir = q.d;
            trace_begin(p, work.scenes[p.si], q);
          }
        }
      }
    }
    if(p.state == ST_DONE) {
      work.done(p, e);
      p.c_seg = p.c_node = p.c_tc = 0;
      p.state = ST_IDLE;
    }
  }
}

/* A block's event counters, in shared memory (ten registers less than a
 * lane's own) */
struct StepSums {
  unsigned long long seg, node, tc, real, fail;

  __device__ __forceinline__ void add(const PathTrace& p)
  {
    atomicAdd(&seg, (unsigned long long)p.c_seg);
    if(p.c_node) atomicAdd(&node, (unsigned long long)p.c_node);
    atomicAdd(&tc, (unsigned long long)p.c_tc);
    if(!(p.flags & (PF_REJECTED | PF_FAILED))) atomicAdd(&real, 1ull);
    if(p.flags & PF_FAILED) atomicAdd(&fail, 1ull);
  }
};

}  // namespace

#endif /* HTRDR_STEP_CUH */
