/* Batched engine: many draw_map requests (images, flux maps, spectral
 * domains, scenes) in ONE launch fed by a device work queue.
 *
 * A launch covers items -- ranges of realisations of requests -- whose
 * realisations form one index space (item-major, realisation-major inside a
 * request).  The step loop (step.cuh) runs them: each resident thread owns one
 * path and takes the next realisation when it ends.  Paths of very different
 * lengths therefore never leave lanes idle while work remains (path
 * regeneration), and the weight of each realisation is the same as in the
 * one-thread-per-realisation kernel because both run the same state machine on
 * the same stream.  The block-sorted kernel, kept as an option, regroups the
 * paths of a block by stage at every step instead.
 *
 * Entry points: one-shot htrdr_gpu_draw_maps_batched(_device), the reusable
 * htrdr_gpu_batch_* object whose launch sequence is captured once in a CUDA
 * graph and replayed, and the autotuner. */
#include "engine.cuh"

#include <algorithm>
#include <map>
#include <memory>
#include <cstring>

namespace hg {

template <unsigned V>
__global__ void __maxnreg__(HG_PERSIST_MAXNREG)
k_sorted(PTables T, int tables_in_smem)
{
  extern __shared__ __align__(16) unsigned char smem[];
  PathSlot* slots = (PathSlot*)smem;
  uint32_t* lists = (uint32_t*)(smem + path_slots_bytes(blockDim.x));
  if(tables_in_smem)
    tables_to_smem(T, smem + path_slots_bytes(blockDim.x) + sorted_lists_bytes(blockDim.x));
  sorted_loop<V>(T, slots, lists);
}

using SortedFn = void (*)(PTables, int);
static SortedFn
sorted_fn(uint32_t v)
{
  HG_PICK_VARIANT(v, k_sorted)
}

bool
valid_tuning(const htrdr_gpu_tuning& t)
{
  return t.block_size && t.block_size <= 512 && !(t.block_size & 31) && t.queue_chunk
      && (t.engine == HTRDR_GPU_ENGINE_PERSISTENT || t.engine == HTRDR_GPU_ENGINE_WAVEFRONT
          || t.engine == HTRDR_GPU_ENGINE_SORTED);
}

cudaError_t
launch_sorted(const PTables& T, uint32_t block_size, uint32_t blocks_per_sm, int device, cudaStream_t st)
{
  static_assert(sizeof(DScene) % 4 == 0 && sizeof(DRequest) % 4 == 0, "word copies");
  if(!T.total) return cudaSuccess;
  const size_t tables = ((T.nscenes * sizeof(DScene) + 15) & ~(size_t)15) + T.nreqs * sizeof(DRequest);
  const int in_smem = tables <= 96 * 1024;
  const size_t smem = (in_smem ? tables : 0) + path_slots_bytes(block_size) + sorted_lists_bytes(block_size);
  auto kern = sorted_fn(T.variant);
  if(smem > 227 * 1024) return cudaErrorInvalidConfiguration; /* block too large for its paths */
  if(smem > 48 * 1024) {
    const cudaError_t e = allow_shared((const void*)kern, device);
    if(e != cudaSuccess) return e;
  }
  int nsm = 0, per_sm = 0;
  cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, device);
  cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, (int)block_size, smem);
  if(blocks_per_sm) per_sm = std::min(per_sm, (int)blocks_per_sm);
  per_sm = std::max(per_sm, 1);
  kern<<<(unsigned)(nsm * per_sm), block_size, smem, st>>>(T, in_smem);
  note_launches(1);
  return cudaGetLastError();
}

struct SingleTables {
  DScene scene;
  DRequest req;
  PItem item;
  uint64_t offsets[2];
};

size_t
single_tables_bytes()
{
  return sizeof(SingleTables);
}

cudaError_t
launch_workqueue(const PTables& T0, const htrdr_gpu_tuning& tun, int device, cudaStream_t st, bool may_keep)
{
  PTables T = T0;
  T.regroup_period = tun.regroup_period;
  return tun.engine == HTRDR_GPU_ENGINE_SORTED
    ? launch_sorted(T, tun.block_size, tun.blocks_per_sm, device, st)
    : launch_step(T, tun.block_size, tun.blocks_per_sm, device, st, may_keep);
}

cudaError_t
launch_workqueue_single(const DScene& S, const DRequest& R, void* tables, void* cnt,
                        const htrdr_gpu_tuning& tun, int device, cudaStream_t st)
{
  SingleTables h;
  h.scene = S;
  h.req = R;
  h.item = PItem{0, 0, 0};
  h.offsets[0] = 0;
  h.offsets[1] = (uint64_t)R.width * R.height * R.nreal_pp;
  /* a pageable source is staged before the call returns: `h' may go */
  cudaError_t e = cudaMemcpyAsync(tables, &h, sizeof(h), cudaMemcpyHostToDevice, st);
  if(e != cudaSuccess) return e;
  const SingleTables* d = (const SingleTables*)tables;
  PTables T{};
  T.scenes = &d->scene;
  T.reqs = &d->req;
  T.items = &d->item;
  T.offsets = d->offsets;
  T.nscenes = 1;
  T.variant = hv_make(S.g_ntris != 0, hv_kind(R.mode));
  T.nreqs = 1;
  T.nitems = 1;
  T.total = h.offsets[1];
  T.cnt = cnt;
  T.next = (unsigned long long*)((char*)cnt + 64);
  return launch_workqueue(T, tun, device, st, true);
}

/* Device buffers of a plan: tables, accumulators, counters, output staging */
struct PlanBufs {
  DevBuf d_scenes, d_reqs, d_items, d_offsets, d_acc, d_cnt, d_out;
};

/* Grow-only buffers of the one-shot calls of a host thread on a device (one
 * call at a time per thread): a call reuses those of the last one, as
 * freeing device memory after every call cost up to 0.6 s of host time */
PlanBufs&
thread_plan_bufs(int device)
{
  static thread_local std::map<int, std::unique_ptr<PlanBufs>> bufs;
  std::unique_ptr<PlanBufs>& b = bufs[device];
  if(!b) b = std::make_unique<PlanBufs>();
  return *b;
}

/* `b' holding at least `n' bytes (its contents are not kept) */
bool
reserve(DevBuf& b, size_t n)
{
  if(b.ptr && b.bytes >= n) return true;
  if(b.ptr) { cudaFree(b.ptr); b.ptr = nullptr; b.bytes = 0; }
  return b.alloc(n);
}

bool
fill(DevBuf& b, const void* src, size_t n)
{
  return reserve(b, n) && (!n || cuda_ok(cudaMemcpy(b.ptr, src, n, cudaMemcpyHostToDevice), "cudaMemcpy H2D"));
}

/* Device state of a set of items: tables, accumulators, counters */
struct Plan {
  int device = 0;
  std::vector<DRequest> reqs;
  std::vector<DScene> scenes;
  std::vector<PItem> items;
  std::vector<uint64_t> offsets;
  std::vector<size_t> out_off;
  PlanBufs own;           /* a reusable batch's buffers (its graph holds their addresses) */
  PlanBufs* B = &own;     /* the buffers in use: `own', or the thread's for a one-shot call */
  size_t acc_bytes = 0;
  bool accum_out = false; /* the items' buffers receive the accumulators */
  std::vector<size_t> item_acc_bytes;
  PTables T{};
};

static htrdr_gpu_res_T
plan_build(Plan& P, const htrdr_gpu_batch_item* items, size_t n, bool host_out,
           bool accum_out = false, bool one_shot = true)
{
  const int device = items[0].scene ? items[0].scene->device : -1;
  for(size_t i = 0; i < n; ++i) {
    if(!items[i].scene || items[i].scene->device != device || !items[i].buffer)
      return HTRDR_GPU_RES_BAD_ARG;
    const htrdr_gpu_buffer_layout& L = items[i].layout;
    const htrdr_gpu_request& q = items[i].req;
    if(!accum_out && check_layout(&q, &L) != HTRDR_GPU_RES_OK) return HTRDR_GPU_RES_BAD_ARG;
    if(accum_out && (q.mode < 0 || q.mode > 4 || !q.width || !q.height)) return HTRDR_GPU_RES_BAD_ARG;
  }
  P.accum_out = accum_out;
  if(!cuda_ok(cudaSetDevice(device), "cudaSetDevice")) return HTRDR_GPU_RES_BAD_OP;
  P.device = device;
  if(one_shot) P.B = &thread_plan_bufs(device);
  PlanBufs& B = *P.B;
  P.reqs.resize(n);
  P.items.resize(n);
  P.offsets.assign(n + 1, 0);
  P.out_off.assign(n, 0);
  std::vector<htrdr_gpu_scene*> scene_ptrs;
  std::vector<uint64_t> acc_off(n);
  uint64_t acc_total = 0;
  size_t out_bytes = 0;
  for(size_t i = 0; i < n; ++i) {
    htrdr_gpu_res_T res = make_drequest(items[i].scene, &items[i].req, &P.reqs[i]);
    if(res != HTRDR_GPU_RES_OK) return res;
    auto it = std::find(scene_ptrs.begin(), scene_ptrs.end(), items[i].scene);
    uint32_t si;
    if(it == scene_ptrs.end()) {
      si = (uint32_t)scene_ptrs.size();
      scene_ptrs.push_back(items[i].scene);
      P.scenes.push_back(items[i].scene->d);
    } else {
      si = (uint32_t)(it - scene_ptrs.begin());
    }
    const uint64_t npix = (uint64_t)P.reqs[i].width * P.reqs[i].height;
    const uint32_t nch = P.reqs[i].mode == HG_IMAGE_CIE ? 3u : 1u;
    acc_off[i] = acc_total;
    acc_total += npix * (nch + 1);
    P.items[i] = PItem{(uint32_t)i, si, 0};
    P.out_off[i] = out_bytes;
    if(host_out) out_bytes += (items[i].layout.pitch * items[i].layout.height + 255) & ~(size_t)255;
  }
  /* The work queue takes the shortwave requests first: their walks are tens
   * of times longer, so the longwave ones fill the lanes that run dry, and
   * until then a warp's paths are of one kind. */
  std::stable_partition(P.items.begin(), P.items.end(),
                        [&](const PItem& it) { return hv_kind(P.reqs[it.req].mode) == HV_SW; });
  for(size_t k = 0; k < n; ++k) {
    const DRequest& r = P.reqs[P.items[k].req];
    P.offsets[k + 1] = P.offsets[k] + (uint64_t)r.width * r.height * r.nreal_pp;
  }
  P.acc_bytes = accum_out ? 0 : acc_total * sizeof(DAccum);
  if((!accum_out && !reserve(B.d_acc, P.acc_bytes)) || !reserve(B.d_cnt, 128) || !reserve(B.d_out, out_bytes))
    return HTRDR_GPU_RES_MEM_ERR;
  P.item_acc_bytes.assign(n, 0);
  for(size_t i = 0; i < n; ++i) {
    const uint64_t npix = (uint64_t)P.reqs[i].width * P.reqs[i].height;
    const uint32_t nch = P.reqs[i].mode == HG_IMAGE_CIE ? 3u : 1u;
    P.reqs[i].acc = accum_out ? (DAccum*)items[i].buffer : (DAccum*)B.d_acc.ptr + acc_off[i];
    P.reqs[i].tacc = P.reqs[i].acc + npix * nch;
    P.item_acc_bytes[i] = npix * (nch + 1) * sizeof(DAccum);
  }
  if(!fill(B.d_scenes, P.scenes.data(), P.scenes.size() * sizeof(DScene))
  || !fill(B.d_reqs, P.reqs.data(), n * sizeof(DRequest))
  || !fill(B.d_items, P.items.data(), n * sizeof(PItem))
  || !fill(B.d_offsets, P.offsets.data(), (n + 1) * 8))
    return HTRDR_GPU_RES_MEM_ERR;
  PTables& T = P.T;
  T.scenes = (const DScene*)B.d_scenes.ptr;
  T.reqs = (const DRequest*)B.d_reqs.ptr;
  T.items = (const PItem*)B.d_items.ptr;
  T.offsets = (const uint64_t*)B.d_offsets.ptr;
  T.nscenes = (uint32_t)P.scenes.size();
  T.variant = tables_variant(P.scenes, P.reqs);
  T.nreqs = (uint32_t)n;
  T.nitems = (uint32_t)n;
  T.total = P.offsets[n];
  T.cnt = B.d_cnt.ptr;
  T.next = (unsigned long long*)((char*)B.d_cnt.ptr + 64);
  return HTRDR_GPU_RES_OK;
}

/* Launch sequence of a plan: clear, work-queue engine, finalize into the
 * items' output buffers (device) or the plan's staging (host copies after). */
static bool
plan_enqueue(Plan& P, const htrdr_gpu_batch_item* items, size_t n, const htrdr_gpu_tuning& tun,
             bool host_out, cudaStream_t st, cudaEvent_t k0, cudaEvent_t k1, bool capturing = false)
{
  bool ok = cuda_ok(cudaMemsetAsync(P.B->d_cnt.ptr, 0, 128, st), "memset");
  if(!P.accum_out)
    ok = ok && cuda_ok(cudaMemsetAsync(P.B->d_acc.ptr, 0, P.acc_bytes, st), "memset");
  for(size_t i = 0; ok && P.accum_out && i < n; ++i)
    ok = cuda_ok(cudaMemsetAsync(P.reqs[i].acc, 0, P.item_acc_bytes[i], st), "memset");
  /* inside a stream capture an event record must be an external node to time
   * the replays */
  const unsigned evf = capturing ? cudaEventRecordExternal : cudaEventRecordDefault;
  if(ok && k0) ok = cuda_ok(cudaEventRecordWithFlags(k0, st, evf), "event");
  if(ok) ok = cuda_ok(launch_workqueue(P.T, tun, P.device, st, !capturing), "k_step");
  if(ok && k1) ok = cuda_ok(cudaEventRecordWithFlags(k1, st, evf), "event");
  for(size_t i = 0; ok && !P.accum_out && i < n; ++i) {
    char* dout = host_out ? (char*)P.B->d_out.ptr + P.out_off[i] : (char*)items[i].buffer;
    ok = cuda_ok(launch_finalize(P.reqs[i], P.reqs[i].acc, P.reqs[i].tacc, dout,
                                 items[i].layout.pitch, st), "k_finalize");
    if(ok && host_out)
      ok = cuda_ok(cudaMemcpyAsync(items[i].buffer, dout, items[i].layout.pitch * items[i].layout.height,
                                   cudaMemcpyDeviceToHost, st), "D2H");
  }
  return ok;
}

static void
read_stats(const unsigned long long c[6], float kms, float tms, uint64_t launches,
           htrdr_gpu_stats* stats)
{
  if(!stats) return;
  stats->segments = c[0]; stats->nodes = c[1]; stats->collisions = c[2];
  stats->realisations = c[3]; stats->failures = c[4]; stats->grid_bytes = c[5];
  stats->kernel_ms = kms; stats->total_ms = tms;
  stats->launches = launches;
}

}  // namespace hg

using namespace hg;

extern "C" HTRDR_GPU_API void
htrdr_gpu_default_tuning(htrdr_gpu_tuning* t)
{
  if(!t) return;
  t->block_size = 128;
  t->queue_chunk = 4;
  t->regroup_period = 1;
  t->blocks_per_sm = 0;
  t->engine = HTRDR_GPU_ENGINE_PERSISTENT;
  t->wave_slots = 0;
  t->trace_budget = 0;
  t->wave_tail = 0;
}

/* The step loop for every mode, blocks of 256 (one an SM for shortwave, two
 * for longwave; 128 measured the same).  Of the other fields regroup_period
 * matters to the block-sorted engine and wave_slots to a server's pool; nothing
 * reads queue_chunk, trace_budget and wave_tail, whose values stay as callers
 * know them. */
extern "C" HTRDR_GPU_API void
htrdr_gpu_mode_tuning(int mode, htrdr_gpu_tuning* t)
{
  if(!t) return;
  htrdr_gpu_default_tuning(t);
  const bool lw = mode == HG_XWAVE_LW || mode == HG_FLUX_LW;
  t->engine = HTRDR_GPU_ENGINE_WAVEFRONT;
  t->block_size = 256;
  t->queue_chunk = 1;
  t->regroup_period = mode == HG_IMAGE_CIE ? 16 : 64;
  t->trace_budget = 256;
  t->wave_tail = lw || mode == HG_IMAGE_CIE ? 100000 : 25000;
}

/* `tuning' if given, else the default of the items' modes (SW/CIE if any) */
static htrdr_gpu_tuning
items_tuning(const htrdr_gpu_batch_item* items, size_t n, const htrdr_gpu_tuning* tuning)
{
  htrdr_gpu_tuning tun;
  if(tuning) return *tuning;
  int sw = 0;
  for(size_t i = 0; i < n; ++i)
    sw |= items[i].req.mode != HG_XWAVE_LW && items[i].req.mode != HG_FLUX_LW;
  htrdr_gpu_mode_tuning(sw ? HG_XWAVE_SW : HG_FLUX_LW, &tun);
  return tun;
}

static htrdr_gpu_res_T
batched_impl(htrdr_gpu_batch_item* items, size_t n, const htrdr_gpu_tuning* tuning,
             htrdr_gpu_stats* stats, bool host, bool accum = false)
{
  if(!items || !n) return HTRDR_GPU_RES_BAD_ARG;
  const htrdr_gpu_tuning tun = items_tuning(items, n, tuning);
  if(!valid_tuning(tun)) return HTRDR_GPU_RES_BAD_ARG;
  take_launches();
  Plan P;
  htrdr_gpu_res_T res = plan_build(P, items, n, host, accum);
  if(res != HTRDR_GPU_RES_OK) return res;
  cudaStream_t st = items[0].scene->stream;
  cudaEvent_t e0, e1, e2, e3;
  cudaEventCreate(&e0); cudaEventCreate(&e1); cudaEventCreate(&e2); cudaEventCreate(&e3);
  cudaEventRecord(e0, st);
  bool ok = plan_enqueue(P, items, n, tun, host, st, e1, e2);
  cudaEventRecord(e3, st);
  unsigned long long c[6] = {0, 0, 0, 0, 0, 0};
  if(ok) ok = cuda_ok(cudaMemcpyAsync(c, P.B->d_cnt.ptr, sizeof(c), cudaMemcpyDeviceToHost, st), "D2H");
  /* also after an error: the launches before it use the thread's buffers */
  ok = cuda_ok(cudaStreamSynchronize(st), "sync") && ok;
  if(ok) {
    float k = 0, t = 0;
    cudaEventElapsedTime(&k, e1, e2);
    cudaEventElapsedTime(&t, e0, e3);
    read_stats(c, k, t, take_launches(), stats);
  }
  cudaEventDestroy(e0); cudaEventDestroy(e1); cudaEventDestroy(e2); cudaEventDestroy(e3);
  return ok ? HTRDR_GPU_RES_OK : HTRDR_GPU_RES_UNKNOWN_ERR;
}

extern "C" HTRDR_GPU_API htrdr_gpu_res_T
htrdr_gpu_draw_maps_batched(htrdr_gpu_batch_item* items, size_t n, const htrdr_gpu_tuning* tuning,
                            htrdr_gpu_stats* stats)
try {
  return batched_impl(items, n, tuning, stats, true);
}
HG_API_CATCH("htrdr_gpu_draw_maps_batched")

extern "C" HTRDR_GPU_API htrdr_gpu_res_T
htrdr_gpu_draw_maps_batched_device(htrdr_gpu_batch_item* items, size_t n,
                                   const htrdr_gpu_tuning* tuning, htrdr_gpu_stats* stats)
try {
  return batched_impl(items, n, tuning, stats, false);
}
HG_API_CATCH("htrdr_gpu_draw_maps_batched_device")

extern "C" HTRDR_GPU_API htrdr_gpu_res_T
htrdr_gpu_draw_maps_batched_accum_device(htrdr_gpu_batch_item* items, size_t n,
                                         const htrdr_gpu_tuning* tuning, htrdr_gpu_stats* stats)
try {
  return batched_impl(items, n, tuning, stats, false, true);
}
HG_API_CATCH("htrdr_gpu_draw_maps_batched_accum_device")

/* Autotuner: times the step loop with every candidate block size on the given
 * items (device buffers) with CUDA events and returns the fastest.  Results do
 * not depend on the tuning.  Both names of the step loop's engine run the same
 * kernels here; the persistent one is also what a graph batch takes. */
extern "C" HTRDR_GPU_API htrdr_gpu_res_T
htrdr_gpu_autotune(htrdr_gpu_batch_item* items, size_t n, htrdr_gpu_tuning* best, double* best_ms)
try {
  if(!items || !n || !best) return HTRDR_GPU_RES_BAD_ARG;
  static const uint32_t blocks[] = {64, 128, 256};
  htrdr_gpu_stats st;
  double best_t = 1e300;
  htrdr_gpu_tuning t = items_tuning(items, n, nullptr);
  t.engine = HTRDR_GPU_ENGINE_PERSISTENT;
  htrdr_gpu_res_T res = batched_impl(items, n, &t, &st, false); /* warm-up */
  if(res != HTRDR_GPU_RES_OK) return res;
  for(uint32_t b : blocks) {
    t.block_size = b;
    if((res = batched_impl(items, n, &t, &st, false)) != HTRDR_GPU_RES_OK) return res;
    if(st.kernel_ms < best_t) { best_t = st.kernel_ms; *best = t; }
  }
  if(best_ms) *best_ms = best_t;
  return HTRDR_GPU_RES_OK;
}
HG_API_CATCH("htrdr_gpu_autotune")

/*******************************************************************************
 * Reusable batch: the whole launch sequence (clear, step loop,
 * finalize of every item) captured once in a CUDA graph and replayed.
 ******************************************************************************/
struct htrdr_gpu_batch {
  Plan plan;
  std::vector<htrdr_gpu_batch_item> items;
  cudaStream_t stream = nullptr;
  cudaGraph_t graph = nullptr;
  cudaGraphExec_t exec = nullptr;
  cudaEvent_t e0 = nullptr, e1 = nullptr, e2 = nullptr, e3 = nullptr;
};

extern "C" HTRDR_GPU_API void
htrdr_gpu_batch_release(htrdr_gpu_batch* b)
{
  if(!b) return;
  cudaSetDevice(b->plan.device);
  if(b->stream) cudaStreamSynchronize(b->stream);
  if(b->exec) cudaGraphExecDestroy(b->exec);
  if(b->graph) cudaGraphDestroy(b->graph);
  if(b->e0) cudaEventDestroy(b->e0);
  if(b->e1) cudaEventDestroy(b->e1);
  if(b->e2) cudaEventDestroy(b->e2);
  if(b->e3) cudaEventDestroy(b->e3);
  if(b->stream) cudaStreamDestroy(b->stream);
  delete b;
}

extern "C" HTRDR_GPU_API htrdr_gpu_res_T
htrdr_gpu_batch_create(const htrdr_gpu_batch_item* items, size_t n, const htrdr_gpu_tuning* tuning,
                       htrdr_gpu_batch** out)
try {
  if(!items || !n || !out) return HTRDR_GPU_RES_BAD_ARG;
  htrdr_gpu_tuning tun = items_tuning(items, n, tuning);
  if(!tuning) tun.engine = HTRDR_GPU_ENGINE_PERSISTENT; /* a mode default names the wavefront */
  if(!valid_tuning(tun)) return HTRDR_GPU_RES_BAD_ARG;
  if(tun.engine != HTRDR_GPU_ENGINE_PERSISTENT && tun.engine != HTRDR_GPU_ENGINE_SORTED) {
    set_error("graph batches run the persistent engines");
    return HTRDR_GPU_RES_BAD_ARG;
  }
  auto b = new htrdr_gpu_batch();
  b->items.assign(items, items + n);
  htrdr_gpu_res_T res = plan_build(b->plan, b->items.data(), n, false, false, false);
  if(res != HTRDR_GPU_RES_OK) { htrdr_gpu_batch_release(b); return res; }
  bool ok = cuda_ok(cudaStreamCreateWithFlags(&b->stream, cudaStreamNonBlocking), "stream")
         && cuda_ok(cudaEventCreate(&b->e0), "event") && cuda_ok(cudaEventCreate(&b->e1), "event")
         && cuda_ok(cudaEventCreate(&b->e2), "event") && cuda_ok(cudaEventCreate(&b->e3), "event");
  /* the occupancy query and the smem attribute are set outside the capture */
  if(ok) ok = cuda_ok(cudaStreamBeginCapture(b->stream, cudaStreamCaptureModeThreadLocal), "capture");
  if(ok) {
    const bool enq = plan_enqueue(b->plan, b->items.data(), n, tun, false, b->stream, b->e1, b->e2, true);
    ok = cuda_ok(cudaStreamEndCapture(b->stream, &b->graph), "end capture") && enq;
  }
  if(ok) ok = cuda_ok(cudaGraphInstantiate(&b->exec, b->graph, 0), "graph instantiate");
  if(!ok) { htrdr_gpu_batch_release(b); return HTRDR_GPU_RES_UNKNOWN_ERR; }
  *out = b;
  return HTRDR_GPU_RES_OK;
}
HG_API_CATCH("htrdr_gpu_batch_create")

/* Replays the captured launch: the items' device buffers receive the maps. */
extern "C" HTRDR_GPU_API htrdr_gpu_res_T
htrdr_gpu_batch_run(htrdr_gpu_batch* b, htrdr_gpu_stats* stats)
try {
  if(!b) return HTRDR_GPU_RES_BAD_ARG;
  cudaSetDevice(b->plan.device);
  unsigned long long c[6] = {0, 0, 0, 0, 0, 0};
  bool ok = cuda_ok(cudaEventRecord(b->e0, b->stream), "event")
         && cuda_ok(cudaGraphLaunch(b->exec, b->stream), "graph launch")
         && cuda_ok(cudaEventRecord(b->e3, b->stream), "event")
         && cuda_ok(cudaMemcpyAsync(c, b->plan.B->d_cnt.ptr, sizeof(c), cudaMemcpyDeviceToHost, b->stream), "D2H")
         && cuda_ok(cudaStreamSynchronize(b->stream), "sync");
  if(!ok) return HTRDR_GPU_RES_UNKNOWN_ERR;
  float k = 0, t = 0;
  cudaEventElapsedTime(&k, b->e1, b->e2);
  cudaEventElapsedTime(&t, b->e0, b->e3);
  read_stats(c, k, t, 1 + b->items.size(), stats); /* k_step + finalizes */
  return HTRDR_GPU_RES_OK;
}
HG_API_CATCH("htrdr_gpu_batch_run")
