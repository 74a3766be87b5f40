/* The step loop with two warps a path: for runs, and ends of runs, with so few
 * paths that a bounce's latency decides.
 *
 * The sun transmissivity of a bounce (the longest trace of it) is only summed
 * at the path's end; the next free path needs nothing of it but the state of
 * the random stream, and that is known as long as the trace meets no tentative
 * collision (it draws one optical depth; only leaves that span gas layers or
 * merged cells have null collisions to look for).  So a main warp hands the
 * trace to its partner and goes on with the next free path as if one draw had
 * been taken; the partner's transmissivity is added one bounce later, in the
 * order of the walk.  Where the trace did draw more, the bounce made meanwhile
 * is dropped: the path goes back to where it handed the trace over, with the
 * partner's stream, and takes the event it would have taken.  Same draws, same
 * sums, same weights as the step loop.
 *
 * Measured on a B200, a lone path's bounce: 9 us (18 000 cycles) in the step
 * loop, of which the trace 6 100 cycles; 7.5 us in a pair. */
#ifndef HTRDR_PAIR_CUH
#define HTRDR_PAIR_CUH

#include "step.cuh"

namespace {

/* What a lane hands to its partner, and gets back in the same place */
struct PairJob {
  PathTrace t;        /* the trace, its counters from zero */
  PathEvent e;        /* the path's event part when it was handed over */
  double factor;      /* weight of the transmissivity: ksi L_sun, R and 1/pdf apart */
  double Tr;          /* back: the transmissivity */
  uint32_t n;         /* draws when it was handed over */
  uint32_t c_seg, c_node, c_tc, c_grid; /* the path's counters then */
  uint32_t busy;      /* 1: to trace; 0: none or done */
  uint64_t pad;
};
/* an odd number of 8-byte words, as the event part */
static_assert(sizeof(PairJob) % 16 == 8, "a warp's accesses to one field do not conflict");

/* Pairs of warps of a block (its threads hold all registers of an SM), and the
 * shared memory of their paths and jobs */
constexpr uint32_t kPairs = 4;
__host__ __device__ constexpr size_t
pair_bytes()
{
  return step_event_bytes(32 * kPairs) + 32 * kPairs * sizeof(PairJob);
}

/* The main warp and its partner, and nobody else, wait for each other; both
 * reach every wait, as the main warp's flag tells the partner when to leave */
__device__ __forceinline__ void
pair_sync(int pair)
{
  __syncwarp();
  asm volatile("bar.sync %0, 64;" ::"r"(pair + 1) : "memory");
}

template <unsigned V, class Work>
__device__ __forceinline__ void
pair_partner(const Work& work, PairJob& job, volatile uint32_t& live, int pair)
{
  for(;;) {
    pair_sync(pair); /* the traces are done */
    pair_sync(pair); /* new ones are there */
    if(!live) return;
    PathTrace p;
    p.state = ST_IDLE;
    if(job.busy) p = job.t;
    while(__any_sync(HG_FULL, p.state == ST_TRACE)) {
      const bool act = p.state == ST_TRACE;
      bool walk = false;
      if(act) {
        trace_enter(p.tr, work.scenes[p.si]);
        walk = p.tr.has_cloud && p.tr.region == 1 && walk_fits(p.tr, work.scenes[p.si]);
      }
      cell_walk<V, true>(p, work.scenes, walk);
      __syncwarp();
      if(act && p.state == ST_TRACE) trace_step<V>(p, work.scenes[p.si]);
    }
    if(job.busy) {
      job.Tr = p.tr.hit ? 0.0 : (p.tr.Tmin != 0.0 ? exp(-p.tr.Tmin) : 1.0);
      job.t = p;
      job.busy = 0;
    }
  }
}

template <unsigned V, class Work>
__device__ __forceinline__ void
pair_main(Work& work, PathTrace& p, PathEvent& e, PairJob& job, volatile uint32_t& live_flag, int pair,
          bool drained)
{
  p.state = ST_IDLE;
  p.flags = 0;
  p.c_seg = p.c_node = p.c_tc = 0;
  p.si = 0;
  job.busy = 0;
  bool pending = false; /* a trace is with the partner */
  for(;;) {
    const unsigned live = __ballot_sync(HG_FULL, p.state != ST_IDLE);
    const unsigned idle = __ballot_sync(HG_FULL, p.state == ST_IDLE && !drained);
    if(idle && (!live || __popc(idle) >= step_refill(V))) {
      const bool more = work.take(p.state == ST_IDLE && !drained, p, e);
      drained = drained || !more;
    }
    /* a bounce up to its sun transmissivity */
    for(int ph = 0; ph < 3; ++ph) {
      const int evph = p.state == ST_SW_SCAT_END ? 1 : (p.state == ST_SW_ABS_END ? 2 : 0);
      if(p.state != ST_IDLE && p.state != ST_TRACE && p.state != ST_DONE && evph == ph)
        path_event<V>(p, e, work.scenes[p.si], work.request(e));
      if(ph == 2) break;
      const int trph = p.tr.kind != TK_TRANS ? 0 : (p.tr.prop == HG_KA ? 1 : 2);
      for(uint32_t it = 0;; ++it) {
        const bool act = p.state == ST_TRACE && trph == ph;
        if(!__any_sync(HG_FULL, act)) break;
        bool walk = false;
        if(act) {
          trace_enter(p.tr, work.scenes[p.si]);
          walk = ph == 0 && p.tr.has_cloud && p.tr.region == 1 && walk_fits(p.tr, work.scenes[p.si]);
        }
        cell_walk<V, false>(p, work.scenes, walk);
        __syncwarp();
        if(act && p.state == ST_TRACE) trace_step<V>(p, work.scenes[p.si]);
      }
    }
    pair_sync(pair);
    if(pending) {
      pending = false;
      const uint32_t seg = job.t.c_seg, node = job.t.c_node, tc = job.t.c_tc, grid = job.t.c_grid;
      if(job.t.ret == ST_SW_DIRECT_END || job.t.rng.n != job.n) {
        /* the trace the path waits for, or more draws than one: on from there */
        p = job.t;
        e = job.e;
        p.c_seg = job.c_seg; p.c_node = job.c_node; p.c_tc = job.c_tc; p.c_grid = job.c_grid;
      } else {
        e.w += job.factor * job.Tr * (double)job.e.R * (double)job.e.sun_ipdf;
        p.flags |= job.t.flags & PF_FAILED;
        if(p.state == ST_DONE) { /* its weight again, with this term */
          p.state = ST_RAD_END;
          path_event<V>(p, e, work.scenes[p.si], work.request(e));
        }
      }
      p.c_seg += seg;
      p.c_node += node;
      p.c_tc += tc;
      p.c_grid += grid;
    }
    if(p.state == ST_TRACE && p.tr.kind == TK_TRANS && p.tr.prop == HG_KEXT) {
      job.c_seg = p.c_seg; job.c_node = p.c_node; job.c_tc = p.c_tc; job.c_grid = p.c_grid;
      p.c_seg = p.c_node = p.c_tc = p.c_grid = 0;
      job.t = p;
      job.e = e;
      job.n = p.rng.n;
      job.busy = 1;
      p.c_seg = job.c_seg; p.c_node = job.c_node; p.c_tc = job.c_tc; p.c_grid = job.c_grid;
      pending = true;
      if(p.ret == ST_SW_NEE_END) {
        /* ST_SW_NEE_END without the term */
        p.flags &= ~PF_TRACED;
        e.ksi *= e.tr_abs;
        job.factor = (double)e.ksi * e.L_sun;
        if((p.flags & PF_SURFACE) && p.rng.uf() >= e.refl) {
          p.state = ST_RAD_END;
        } else {
          e.pos = e.pnext;
          e.dir = e.dnext;
          p.state = ST_SW_WALK;
        }
      }
    } else if(p.state == ST_DONE) {
      work.done(p, e);
      p.c_seg = p.c_node = p.c_tc = 0;
      p.state = ST_IDLE;
    }
    const bool any = __any_sync(HG_FULL, p.state != ST_IDLE || !drained);
    if((threadIdx.x & 31u) == 0) live_flag = any;
    pair_sync(pair);
    if(!any) return;
  }
}

}  // namespace

#endif /* HTRDR_PAIR_CUH */
