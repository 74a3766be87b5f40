/* Kernels and launchers of the step loop (step.cuh) over the work queue: one
 * launch that renders all queued realisations (the persistent and wavefront
 * engines of the one-shot calls, graph batches and serving rounds), and the
 * serving pool, whose launches end after a set time with the live paths
 * saved, so that newly admitted requests join them in the next one. */
#include "pair.cuh"
#include "spread.h"

#include <algorithm>
#include <map>
#include <memory>
#include <mutex>
#include <set>

namespace hg {

namespace {

constexpr uint32_t kPathV4 = (uint32_t)((sizeof(Path) + 15) / 16);
constexpr uint32_t kTraceV4 = (uint32_t)(sizeof(PathTrace) / 16);
static_assert(sizeof(PathTrace) % 16 == 0, "the trace part is whole vectors");

/* A saved path: kPathV4 consecutive 16-byte vectors */
__device__ __forceinline__ void
load_path(PathTrace& p, PathEvent& e, const uint4* v)
{
  uint4 t[kTraceV4], u[kPathV4 - kTraceV4];
#pragma unroll
  for(uint32_t i = 0; i < kTraceV4; ++i) t[i] = v[i];
#pragma unroll
  for(uint32_t i = kTraceV4; i < kPathV4; ++i) u[i - kTraceV4] = v[i];
  memcpy(&p, t, sizeof(PathTrace));
  memcpy(&e, u, sizeof(PathEvent));
}

__device__ __forceinline__ void
save_path(const PathTrace& p, const PathEvent& e, uint4* v)
{
  uint4 t[kTraceV4], u[kPathV4 - kTraceV4];
  u[kPathV4 - kTraceV4 - 1] = make_uint4(0, 0, 0, 0);
  memcpy(t, &p, sizeof(PathTrace));
  memcpy(u, &e, sizeof(PathEvent));
#pragma unroll
  for(uint32_t i = 0; i < kTraceV4; ++i) v[i] = t[i];
#pragma unroll
  for(uint32_t i = kTraceV4; i < kPathV4; ++i) v[i] = u[i - kTraceV4];
}

/* Where a launch's paths come from and go to: the queue alone; a pool, whose
 * saved paths come before the queue and which saves the live ones when the
 * launch's time is over (launch_end); the queue, and the last paths saved for another
 * launch when it has run dry (LAST_OUT) and taken up by that one (LAST_IN) */
enum { WK_QUEUE = 0, WK_POOL, WK_LAST_OUT, WK_LAST_IN };

/* Live paths of a warp that has found the queue dry at which it hands them
 * over.  Measured (6 / 12 / 20 / 24 / 32, and none handed over): SW image of
 * 131 000 realisations 13.0 / 12.7 / 12.0 / 12.0 / 12.5, 12.8 ms; flux map 29.0 /
 * 27.7 / 26.6 / 26.8 / 26.9, 28.0; CIE image 16.4 / 16.2 / 14.6 / 15.0 / 15.1,
 * 16.6; mesh image 33.2 / 31.2 / 30.1 / 30.6 / 29.7, 32.7. */
constexpr uint32_t kLastPaths = 20;

template <int Kind>
struct QueueWork {
  static constexpr bool kReads = Kind == WK_POOL || Kind == WK_LAST_IN;
  const DScene* scenes;
  PTables T;
  StepSums* sums;
  /* Pool: saved paths read and written, their counters, the end of the launch,
   * whether this block started before it and has not taken its first turn */
  const uint4* in;
  uint4* out;
  StepCtl* ctl;
  uint32_t n_in, turn, room;
  unsigned long long until;
  bool saved_left, dry, fresh;

  __device__ __forceinline__ const DRequest& request(const PathEvent& e) const { return T.reqs[e.ri]; }

  __device__ __forceinline__ bool stop(uint32_t live)
  {
    if(Kind == WK_POOL) {
      const bool over = __shfl_sync(HG_FULL, (int)(gtimer() >= until), 0) != 0 && !fresh;
      fresh = false;
      return over;
    }
    return Kind == WK_LAST_OUT && live <= kLastPaths && __any_sync(HG_FULL, dry);
  }

  __device__ __forceinline__ bool take(bool want, PathTrace& p, PathEvent& e)
  {
    const unsigned lane = threadIdx.x & 31u;
    if(kReads && __any_sync(HG_FULL, saved_left)) {
      const unsigned m = __ballot_sync(HG_FULL, want && saved_left);
      if(m) {
        const unsigned leader = __ffs(m) - 1;
        uint32_t i0 = 0;
        if(lane == leader) i0 = atomicAdd(&ctl->fetch, (uint32_t)__popc(m));
        i0 = __shfl_sync(HG_FULL, i0, leader);
        if(m & (1u << lane)) {
          const uint32_t i = i0 + __popc(m & ((1u << lane) - 1u));
          if(i < n_in) {
            /* a pool's from the end: first those that the launch before left */
            load_path(p, e, in + (size_t)(Kind == WK_POOL ? n_in - 1 - i : i) * kPathV4);
            p.t0 = gtimer() - p.t0; /* saved: busy time so far */
            want = false;
          } else {
            saved_left = false;
          }
        }
      }
    }
    const unsigned m = __ballot_sync(HG_FULL, want);
    if(!m) return true;
    const unsigned leader = __ffs(m) - 1;
    unsigned long long g0 = 0;
    unsigned got = 0;
    if(lane == leader) g0 = queue_take(T, (unsigned)__popc(m), &got);
    g0 = __shfl_sync(HG_FULL, g0, leader);
    got = __shfl_sync(HG_FULL, got, leader);
    if(got < (unsigned)__popc(m)) dry = true;
    if(!want) return true;
    const unsigned rank = __popc(m & ((1u << lane) - 1u));
    if(rank >= got) return false;
    path_assign(p, e.ri, T, g0 + rank);
    return true;
  }

  __device__ __forceinline__ void done(PathTrace& p, PathEvent& e)
  {
    accumulate_b(p, e.weight, T.reqs[e.ri]);
    count_grid(T.cnt, p);
    sums->add(p);
  }

  /* The warp's paths to the pool.  They fit: a lane holds one path, and takes
   * one from the queue only when no saved path is left, so a launch that took
   * from the queue has every path it saves in one of its `lanes' lanes, and one
   * that did not has as many as it read.  (Saved paths that no lane took stay
   * where they are until the launch has ended, in whatever order its blocks
   * start and end: k_step_turn.) */
  __device__ __forceinline__ void save(PathTrace& p, PathEvent& e)
  {
    if(Kind != WK_POOL && Kind != WK_LAST_OUT) return;
    const unsigned lane = threadIdx.x & 31u;
    const bool keep = p.state != ST_IDLE;
    const unsigned m = __ballot_sync(HG_FULL, keep);
    uint32_t o = 0;
    if(lane == 0 && m) o = atomicAdd(&ctl->n[turn ^ 1u], (uint32_t)__popc(m));
    o = __shfl_sync(HG_FULL, o, 0) + __popc(m & ((1u << lane) - 1u));
    if(keep && (Kind != WK_POOL || o < room)) { /* else: counted, for the host to see */
      p.t0 = gtimer() - p.t0;
      save_path(p, e, out + (size_t)o * kPathV4);
    }
  }
};

/* Whether this lane stays empty: few paths are spread over all warps, as a
 * warp with a single path takes its bounces fastest.  A pool's lanes have their
 * limit besides (warp_lanes), the warps counted across the blocks first, so
 * that a pool of few paths runs on all SMs. */
template <int Kind>
__device__ __forceinline__ bool
lane_unused(const PTables& T, uint32_t saved, uint32_t warps_per_block, uint32_t room)
{
  const unsigned long long next = *(volatile unsigned long long*)T.next;
  const unsigned long long left = saved + (T.total > next ? T.total - next : 0ull);
  const unsigned long long warps = (unsigned long long)gridDim.x * warps_per_block;
  if(Kind != WK_POOL) return (threadIdx.x & 31u) >= (left + warps - 1) / warps;
  return (threadIdx.x & 31u) >= warp_lanes((uint64_t)(threadIdx.x >> 5) * gridDim.x + blockIdx.x, warps, room, left);
}

template <int Kind>
__device__ __forceinline__ QueueWork<Kind>
queue_work(const PTables& T, StepSums* sums, const StepPool& P, unsigned long long until = 0, bool fresh = true)
{
  QueueWork<Kind> work;
  work.T = T;
  work.scenes = T.scenes;
  work.sums = sums;
  work.dry = false;
  work.saved_left = false;
  if(Kind != WK_QUEUE) {
    work.in = P.paths[P.turn];
    work.out = P.paths[P.turn ^ 1u];
    work.ctl = P.ctl;
    work.turn = P.turn;
    work.room = Kind == WK_POOL ? P.lanes : 0u;
    work.n_in = work.kReads ? P.ctl->n[P.turn] : 0u;
    if(Kind == WK_POOL) work.n_in = min(work.n_in, P.lanes);
    work.until = until;
    work.fresh = fresh;
    work.saved_left = work.n_in != 0;
  }
  return work;
}

__device__ __forceinline__ void
flush_sums(const PTables& T, const StepSums& sums)
{
  Counters* c = (Counters*)T.cnt;
  atomicAdd(&c->seg, sums.seg);
  atomicAdd(&c->node, sums.node);
  atomicAdd(&c->tc, sums.tc);
  atomicAdd(&c->real, sums.real);
  atomicAdd(&c->fail, sums.fail);
}

/* The end of a pool's launch, the same for all of its blocks: counted from the
 * first one that starts.  A block that starts after it takes nothing; the first
 * one always takes a turn, so a launch advances whatever its length. */
__device__ __forceinline__ unsigned long long
launch_end(const StepPool& P, bool* in_time)
{
  const unsigned long long now = gtimer(), mine = now + P.ns;
  const unsigned long long first = atomicCAS(&P.ctl->until, 0ull, mine);
  *in_time = !first || now < first;
  return first ? first : mine;
}

template <unsigned V, int Kind>
__device__ __forceinline__ void
step_block(PTables& T, const StepPool& P, int tables_in_smem)
{
  extern __shared__ __align__(16) unsigned char smem[];
  __shared__ StepSums sums;
  const bool unused = lane_unused<Kind>(T, QueueWork<Kind>::kReads ? P.ctl->n[P.turn] : 0u, blockDim.x >> 5, P.lanes);
  __shared__ unsigned long long until;
  __shared__ bool fresh;
  if(threadIdx.x == 0) {
    sums = StepSums{0, 0, 0, 0, 0};
    if(Kind == WK_POOL) until = launch_end(P, &fresh);
  }
  if(tables_in_smem) tables_to_smem(T, smem + step_event_bytes(blockDim.x));
  __syncthreads();
  QueueWork<Kind> work = Kind == WK_POOL ? queue_work<Kind>(T, &sums, P, until, fresh)
                                         : queue_work<Kind>(T, &sums, P);
  PathTrace p;
  step_loop<V>(work, p, ((PathEvent*)smem)[threadIdx.x], unused);
  __syncthreads();
  if(threadIdx.x == 0) flush_sums(T, sums);
}

}  // namespace

template <unsigned V>
__global__ void __maxnreg__(step_registers(V))
k_step(PTables T, int tables_in_smem)
{
  step_block<V, WK_QUEUE>(T, StepPool{}, tables_in_smem);
}

template <unsigned V>
__global__ void __maxnreg__(step_registers(V))
k_step_pool(PTables T, StepPool P, int tables_in_smem)
{
  step_block<V, WK_POOL>(T, P, tables_in_smem);
}

/* All but the last paths of a run */
template <unsigned V>
__global__ void __maxnreg__(step_registers(V))
k_step_most(PTables T, StepPool P, int tables_in_smem)
{
  step_block<V, WK_LAST_OUT>(T, P, tables_in_smem);
}

/* The last paths of a run, or a small run: two warps a path (pair.cuh) */
template <unsigned V>
__global__ void __launch_bounds__(64 * kPairs, 1)
k_pair(PTables T, StepPool P, int tables_in_smem)
{
  extern __shared__ __align__(16) unsigned char smem[];
  __shared__ StepSums sums;
  __shared__ uint32_t live[kPairs];
  const bool unused = lane_unused<WK_LAST_IN>(T, P.ctl->n[P.turn], kPairs, 0u);
  if(threadIdx.x == 0) sums = StepSums{0, 0, 0, 0, 0};
  PairJob* jobs = (PairJob*)(smem + step_event_bytes(32 * kPairs));
  if(tables_in_smem) tables_to_smem(T, smem + pair_bytes());
  __syncthreads();
  QueueWork<WK_LAST_IN> work = queue_work<WK_LAST_IN>(T, &sums, P);
  const uint32_t pair = (threadIdx.x >> 5) % kPairs, slot = threadIdx.x % (32 * kPairs);
  if(threadIdx.x < 32 * kPairs) {
    PathTrace p;
    pair_main<V>(work, p, ((PathEvent*)smem)[slot], jobs[slot], live[pair], (int)pair, unused);
  } else {
    pair_partner<V>(work, jobs[slot], live[pair], (int)pair);
  }
  __syncthreads();
  if(threadIdx.x == 0) flush_sums(T, sums);
}

/* After a launch of a pool: the saved paths that no lane took join those it
 * saved, those it read are free, and the queue's head goes back to the queued
 * total, so that work appended later starts there.  Paths are left over where
 * blocks of the launch started late (another stream held their SMs) or where
 * it had fewer lanes than the one before it (another variant): the launch's own
 * blocks cannot move them, as a lane that has yet to start would take work from
 * the queue beside them.  One block: there is nothing to move most often, and
 * 76 000 paths (34 MB) at most. */
__global__ void
k_step_turn(PTables T, StepPool P)
{
  const uint32_t n_in = min(P.ctl->n[P.turn], P.lanes);
  const uint32_t taken = min(P.ctl->fetch, n_in), at = P.ctl->n[P.turn ^ 1u];
  const uint32_t left = n_in - taken;
  if(at + left <= P.lanes) {
    const uint4* from = P.paths[P.turn];
    uint4* to = P.paths[P.turn ^ 1u] + (size_t)at * kPathV4;
    for(uint32_t i = threadIdx.x; i < left * kPathV4; i += blockDim.x) to[i] = from[i];
  }
  __syncthreads();
  if(threadIdx.x) return;
  P.ctl->n[P.turn] = 0;
  P.ctl->n[P.turn ^ 1u] = at + left;
  P.ctl->fetch = 0;
  P.ctl->until = 0;
  queue_clamp(T);
}

namespace {

using StepFn = void (*)(PTables, int);
using StepPoolFn = void (*)(PTables, StepPool, int);
StepFn
step_fn(uint32_t v)
{
  HG_PICK_VARIANT(v, k_step)
}
StepPoolFn
step_pool_fn(uint32_t v)
{
  HG_PICK_VARIANT(v, k_step_pool)
}
/* Those with shortwave paths */
StepPoolFn
step_most_fn(uint32_t v)
{
  switch(v) {
    case 2u: return k_step_most<2u>;
    case 3u: return k_step_most<3u>;
    case 6u: return k_step_most<6u>;
    default: return k_step_most<7u>;
  }
}
StepPoolFn
pair_fn(uint32_t v)
{
  switch(v) {
    case 2u: return k_pair<2u>;
    case 3u: return k_pair<3u>;
    case 6u: return k_pair<6u>;
    default: return k_pair<7u>;
  }
}

/* Grid of a kernel of `*threads' threads a block that fills the device; blocks
 * that its registers do not allow become the largest that they do */
template <class Fn>
cudaError_t
step_shape(Fn kern, const PTables& T, uint32_t* threads, uint32_t blocks_per_sm, int device, size_t* smem,
           int* in_smem, unsigned* grid, size_t own = 0)
{
  cudaFuncAttributes attr;
  const cudaError_t ea = cudaFuncGetAttributes(&attr, kern);
  if(ea != cudaSuccess) return ea;
  *threads = std::min(*threads, (uint32_t)attr.maxThreadsPerBlock & ~31u);
  const size_t tables = ((T.nscenes * sizeof(DScene) + 15) & ~(size_t)15) + T.nreqs * sizeof(DRequest);
  *in_smem = tables <= 96 * 1024;
  *smem = (own ? own : step_event_bytes(*threads)) + (*in_smem ? tables : 0);
  if(*smem > 48 * 1024) {
    const cudaError_t e = allow_shared((const void*)kern, device);
    if(e != cudaSuccess) return e;
  }
  int nsm = 0, per_sm = 0;
  cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, device);
  cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, (int)*threads, *smem);
  if(blocks_per_sm) per_sm = std::min(per_sm, (int)blocks_per_sm);
  *grid = (unsigned)(nsm * std::max(per_sm, 1));
  return cudaSuccess;
}

}  // namespace

cudaError_t
allow_shared(const void* kern, int device)
{
  static std::mutex mtx;
  static std::set<std::pair<const void*, int>> allowed;
  std::lock_guard<std::mutex> lock(mtx);
  if(allowed.count({kern, device})) return cudaSuccess;
  cudaFuncAttributes attr;
  int most = 0;
  cudaError_t e = cudaFuncGetAttributes(&attr, kern);
  if(e == cudaSuccess) e = cudaDeviceGetAttribute(&most, cudaDevAttrMaxSharedMemoryPerBlockOptin, device);
  if(e == cudaSuccess)
    e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, most - (int)attr.sharedSizeBytes);
  if(e == cudaSuccess) allowed.insert({kern, device});
  return e;
}

/* The buffer of the last paths of a run (17 MB), one a host thread and device */
StepBufs&
thread_last(int device)
{
  static thread_local std::map<int, std::unique_ptr<StepBufs>> bufs;
  std::unique_ptr<StepBufs>& b = bufs[device];
  if(!b) b = std::make_unique<StepBufs>();
  return *b;
}

cudaError_t
launch_step(const PTables& T, uint32_t block_size, uint32_t blocks_per_sm, int device, cudaStream_t st,
            bool may_keep)
{
  if(!T.total) return cudaSuccess;
  size_t smem;
  int in_smem;
  unsigned grid;
  cudaError_t e;
  if(!may_keep || !(T.variant & HV_SW)) {
    auto kern = step_fn(T.variant);
    if((e = step_shape(kern, T, &block_size, blocks_per_sm, device, &smem, &in_smem, &grid))) return e;
    kern<<<grid, block_size, smem, st>>>(T, in_smem);
    note_launches(1);
    return cudaGetLastError();
  }
  /* Shortwave: a lone path's bounce takes 7.5 us in k_pair and 9 in k_step, but
   * a full device's takes a fifth more, as half of the warps hold no path: a
   * run that fits in k_pair's lanes goes there (1024 realisations 4.33 -> 3.56
   * ms), of another only the last paths (all of a flux map of 88 000: 31.4 ms,
   * its last paths 26.6, none 28.0). */
  auto pair = pair_fn(T.variant);
  uint32_t pair_threads = 64 * kPairs;
  size_t pair_smem;
  int pair_in_smem;
  unsigned pair_grid;
  if((e = step_shape(pair, T, &pair_threads, 0, device, &pair_smem, &pair_in_smem, &pair_grid, pair_bytes())))
    return e;
  StepBufs& B = thread_last(device);
  if(!B.ctl.ptr && !B.ctl.alloc(sizeof(StepCtl))) return cudaErrorMemoryAllocation;
  if((e = cudaMemsetAsync(B.ctl.ptr, 0, sizeof(StepCtl), st))) return e;
  StepPool P{};
  P.ctl = (StepCtl*)B.ctl.ptr;
  if(T.total > (uint64_t)pair_grid * 32 * kPairs) {
    auto most = step_most_fn(T.variant);
    if((e = step_shape(most, T, &block_size, blocks_per_sm, device, &smem, &in_smem, &grid))) return e;
    const uint32_t lanes = grid * block_size;
    if(B.lanes < lanes) {
      if(B.paths[0].ptr) { cudaFree(B.paths[0].ptr); B.paths[0].ptr = nullptr; }
      B.lanes = 0;
      if(!B.paths[0].alloc((size_t)lanes * kPathV4 * 16)) return cudaErrorMemoryAllocation;
      B.lanes = lanes;
    }
    P.paths[0] = (uint4*)B.paths[0].ptr;
    P.turn = 1; /* saves into paths[0] */
    most<<<grid, block_size, smem, st>>>(T, P, in_smem);
    note_launches(1);
    if((e = cudaGetLastError())) return e;
  }
  P.turn = 0;
  pair<<<pair_grid, pair_threads, pair_smem, st>>>(T, P, pair_in_smem);
  note_launches(1);
  return cudaGetLastError();
}

uint64_t
step_capacity(uint32_t block_size, uint32_t blocks_per_sm, int device)
{
  PTables T{};
  size_t smem;
  int in_smem;
  unsigned grid;
  if(step_shape(k_step<HV_ALL>, T, &block_size, blocks_per_sm, device, &smem, &in_smem, &grid)) return 0;
  return (uint64_t)grid * block_size;
}

/* ---- serving pool ---- */

/* Threads a block of the pool's launches, and lanes an SM at most (any variant
 * takes 64 registers or more) */
constexpr uint32_t kPoolThreads = 128, kPoolLanesPerSm = 1024;

bool
step_pool_create(StepBufs& B, uint32_t lanes, int device, cudaStream_t st)
{
  /* room for the lanes of any variant: a launch carries over what the one
   * before it saved */
  int nsm = 0;
  cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, device);
  const size_t most = (size_t)nsm * kPoolLanesPerSm;
  B.lanes = lanes ? (uint32_t)std::min<size_t>(lanes, most) : (uint32_t)most;
  for(int i = 0; i < 2; ++i)
    if(!B.paths[i].alloc((size_t)B.lanes * kPathV4 * 16)) return false;
  return B.ctl.alloc(sizeof(StepCtl)) && cuda_ok(cudaMemsetAsync(B.ctl.ptr, 0, sizeof(StepCtl), st), "memset");
}

cudaError_t
step_pool_launch(const PTables& T, StepBufs& B, uint64_t ns, uint32_t blocks_per_sm, int device, cudaStream_t st)
{
  StepPool P;
  P.paths[0] = (uint4*)B.paths[0].ptr;
  P.paths[1] = (uint4*)B.paths[1].ptr;
  P.ctl = (StepCtl*)B.ctl.ptr;
  P.turn = B.turn;
  P.lanes = B.lanes;
  P.ns = ns;
  auto kern = step_pool_fn(T.variant);
  uint32_t threads = kPoolThreads;
  size_t smem;
  int in_smem;
  unsigned grid;
  const cudaError_t e = step_shape(kern, T, &threads, blocks_per_sm, device, &smem, &in_smem, &grid);
  if(e != cudaSuccess) return e;
  kern<<<grid, threads, smem, st>>>(T, P, in_smem);
  k_step_turn<<<1, 1024, 0, st>>>(T, P);
  B.turn ^= 1u;
  note_launches(2);
  return cudaGetLastError();
}

}  // namespace hg
