/* Majorant octrees built on the GPU (the htsky_create acceleration structure,
 * src/atmosphere/htrdr_atmosphere.c:366-382), node arrays byte-identical to
 * the host definition in scene.cpp:
 *
 *  - level 0: one thread per cloud cell, k_cloud = fl(lwc * sigma) plus the
 *    [min, max] of k_gas over the layers the cell overlaps (single precision,
 *    no contraction);
 *  - level L: one thread per node, min/max over its valid children and the
 *    leaf test all-children-leaves && (L <= L_force || (kmax - kmin) 2^L
 *    cmax <= tau) in FP64;
 *  - breadth-first storage: the internal node of rank r of a depth has its 8
 *    children at base(depth + 1) + 8 r in octant order.  A queue-driven walk
 *    visits a depth's nodes in the order of their octant paths, that is in
 *    Morton order, so the rank is an exclusive sum of the internal flags laid
 *    out in Morton order: every node is then written by itself, without the
 *    depths' lists and the host's look at each one's length.
 *
 * All trees of a batch go through each kernel together (as many as fit in a
 * quarter of the free device memory, at most 16 GB; all of them for most
 * scenes), with one scratch allocation and one host wait.  Measured on a B200,
 * 96 trees of 112x90x40 cells (44 M nodes): 2.2 ms, of which 0.8 on the device.
 * A tree at a time on 8 host threads, each with its stream and 8 buffers, took
 * 26 to 70 ms: 9 of build, the rest allocations and their release. */
#include "internal.h"

#include <cub/cub.cuh>

#include <algorithm>
#include <cfloat>
#include <cmath>

namespace hg {

namespace {

/* Scratch of a batch of trees at most */
#ifndef HG_BUILD_BYTES
#define HG_BUILD_BYTES ((size_t)16 << 30)
#endif

struct LevelDims {
  uint32_t D;
  uint32_t n[32][3];
  uint8_t bits[32][3]; /* of the coordinates of level L */
  uint64_t off[33];    /* level L in a tree's row-major arrays; [D + 1]: their size */
  uint64_t moff[33];   /* level L >= 1 in a tree's Morton arrays; [D + 1]: their size */
};

/* One tree of a batch */
struct TreeTask {
  uint32_t q;
  int prop;
  float sig;
  uint32_t pad;
};
/* Where its nodes go: the pool, and the first node of the children of depth d */
struct TreeOut {
  uint64_t base;
  uint32_t child[32];
};

/* Place of (i, j, k) of level L among the octant paths of that level: the
 * coordinate bits from the highest down, z before y before x, without those
 * that are zero for every node of the level */
__device__ __forceinline__ uint32_t
morton(const LevelDims& dims, uint32_t L, uint32_t i, uint32_t j, uint32_t k)
{
  const uint32_t bx = dims.bits[L][0], by = dims.bits[L][1], bz = dims.bits[L][2];
  uint32_t m = 0;
  for(int t = (int)max(bx, max(by, bz)) - 1; t >= 0; --t) {
    if(t < (int)bz) m = (m << 1) | ((k >> t) & 1u);
    if(t < (int)by) m = (m << 1) | ((j >> t) & 1u);
    if(t < (int)bx) m = (m << 1) | ((i >> t) & 1u);
  }
  return m;
}

__global__ void
k_level0(const float* __restrict__ lwc, const int2* __restrict__ cl, const float2* __restrict__ gas,
         uint32_t nlayers, const TreeTask* __restrict__ tasks, LevelDims dims, float* kmin, float* kmax,
         uint8_t* leaf)
{
  const uint64_t c = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const uint64_t nxy = (uint64_t)dims.n[0][0] * dims.n[0][1];
  if(c >= nxy * dims.n[0][2]) return;
  const TreeTask t = tasks[blockIdx.y];
  const int2 lr = cl[c / nxy];
  float gmin = 0.f, gmax = 0.f;
  if(lr.x >= 0) {
    for(int l = lr.x; l <= lr.y; ++l) {
      const float2 as = gas[(size_t)t.q * nlayers + l];
      const float g = t.prop == HG_KA ? as.x : (t.prop == HG_KS ? as.y : __fadd_rn(as.x, as.y));
      if(l == lr.x) { gmin = gmax = g; continue; }
      if(g < gmin) gmin = g;
      if(g > gmax) gmax = g;
    }
  }
  const float kc = __fmul_rn(lwc[c], t.sig);
  const uint64_t o = (uint64_t)blockIdx.y * dims.off[dims.D + 1] + c;
  kmin[o] = __fadd_rn(kc, gmin);
  kmax[o] = __fadd_rn(kc, gmax);
  leaf[o] = 1;
}

__global__ void
k_level(uint32_t L, LevelDims dims, float* kmin, float* kmax, uint8_t* leaf, uint32_t level_force,
        double size, double tau, uint32_t* internal)
{
  const uint32_t* pn = dims.n[L];
  const uint32_t* cn = dims.n[L - 1];
  const uint64_t idx = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if(idx >= (uint64_t)pn[0] * pn[1] * pn[2]) return;
  const uint32_t i = (uint32_t)(idx % pn[0]);
  const uint32_t j = (uint32_t)((idx / pn[0]) % pn[1]);
  const uint32_t k = (uint32_t)(idx / ((uint64_t)pn[0] * pn[1]));
  const uint64_t tree = (uint64_t)blockIdx.y * dims.off[dims.D + 1];
  const float* cmin = kmin + tree + dims.off[L - 1];
  const float* cmax = kmax + tree + dims.off[L - 1];
  const uint8_t* cleaf = leaf + tree + dims.off[L - 1];
  float mn = FLT_MAX, mx = -FLT_MAX;
  int all_leaf = 1;
  for(int oct = 0; oct < 8; ++oct) {
    const uint32_t ci = 2 * i + (oct & 1), cj = 2 * j + ((oct >> 1) & 1), ck = 2 * k + (oct >> 2);
    if(ci >= cn[0] || cj >= cn[1] || ck >= cn[2]) continue;
    const uint64_t cc = ((uint64_t)ck * cn[1] + cj) * cn[0] + ci;
    if(cmin[cc] < mn) mn = cmin[cc];
    if(cmax[cc] > mx) mx = cmax[cc];
    all_leaf &= cleaf[cc];
  }
  const bool lf = all_leaf
    && (L <= level_force || __dmul_rn(__dsub_rn((double)mx, (double)mn), size) <= tau);
  const uint64_t o = tree + dims.off[L] + idx;
  kmin[o] = mn;
  kmax[o] = mx;
  leaf[o] = lf ? 1 : 0;
  if(!lf) internal[(uint64_t)blockIdx.y * dims.moff[dims.D + 1] + dims.moff[L] + morton(dims, L, i, j, k)] = 1u;
}

/* Internal nodes of each level of each tree, from the exclusive sums of the
 * batch's flags */
__global__ void
k_counts(LevelDims dims, uint32_t ntrees, const uint32_t* __restrict__ sum, uint32_t* counts)
{
  const uint32_t x = blockIdx.x * blockDim.x + threadIdx.x;
  const uint32_t t = x / 32, L = x % 32;
  if(t >= ntrees) return;
  uint32_t n = 0;
  if(L >= 1 && L <= dims.D) {
    const uint64_t m = (uint64_t)t * dims.moff[dims.D + 1];
    n = sum[m + dims.moff[L + 1]] - sum[m + dims.moff[L]]; /* the level after the last: the next tree's first */
  }
  counts[x] = n;
}

/* The children of the internal nodes of level L, a thread for each */
__global__ void
k_emit(uint32_t L, LevelDims dims, const float* __restrict__ kmin, const float* __restrict__ kmax,
       const uint8_t* __restrict__ leaf, const uint32_t* __restrict__ sum, const TreeOut* __restrict__ outs,
       uint4* nodes)
{
  const uint64_t x = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const uint32_t* n = dims.n[L];
  const uint64_t idx = x >> 3;
  const uint32_t oct = (uint32_t)x & 7u;
  if(idx >= (uint64_t)n[0] * n[1] * n[2]) return;
  const uint64_t tree = (uint64_t)blockIdx.y * dims.off[dims.D + 1];
  const uint64_t mtree = (uint64_t)blockIdx.y * dims.moff[dims.D + 1];
  const TreeOut* out = outs + blockIdx.y;
  const uint32_t d = dims.D - L;
  const uint64_t c = tree + dims.off[L] + idx;
  const bool inner = L > 0 && !leaf[c];
  if(d == 0 && oct == 0) /* the root */
    nodes[out->base] = make_uint4(__float_as_uint(kmin[c]), __float_as_uint(kmax[c]),
                                  inner ? out->child[0] : HG_LEAF, 0u);
  if(!inner) return;
  const uint32_t i = (uint32_t)(idx % n[0]), j = (uint32_t)((idx / n[0]) % n[1]);
  const uint32_t k = (uint32_t)(idx / ((uint64_t)n[0] * n[1]));
  const uint64_t m = mtree + dims.moff[L];
  const uint32_t rank = sum[m + morton(dims, L, i, j, k)] - sum[m];
  uint4 nd = make_uint4(0u, 0u, HG_LEAF, 0u);
  const uint32_t* cn = dims.n[L - 1];
  const uint32_t ci = 2 * i + (oct & 1u), cj = 2 * j + ((oct >> 1) & 1u), ck = 2 * k + (oct >> 2);
  if(ci < cn[0] && cj < cn[1] && ck < cn[2]) {
    const uint64_t cc = tree + dims.off[L - 1] + ((uint64_t)ck * cn[1] + cj) * cn[0] + ci;
    nd.x = __float_as_uint(kmin[cc]);
    nd.y = __float_as_uint(kmax[cc]);
    if(!leaf[cc]) {
      const uint64_t cm = mtree + dims.moff[L - 1];
      nd.z = out->child[d + 1] + 8u * (sum[cm + morton(dims, L - 1, ci, cj, ck)] - sum[cm]);
    }
  }
  nodes[out->base + out->child[d] + 8ull * rank + oct] = nd;
}

inline unsigned
grid_of(uint64_t n, unsigned bs) { return (unsigned)((n + bs - 1) / bs); }

/* Leaf of every cell of one tree: a descent from the root by the cell's
 * coordinate bits, written as (node index in the tree) << 5 | level */
__global__ void
k_leafgrid(const uint4* __restrict__ nodes, uint32_t depth, uint32_t nx, uint32_t ny, uint32_t nz,
           uint32_t* grid)
{
  const uint64_t c = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if(c >= (uint64_t)nx * ny * nz) return;
  const uint32_t x = (uint32_t)(c % nx), y = (uint32_t)((c / nx) % ny), z = (uint32_t)(c / ((uint64_t)nx * ny));
  uint32_t n = 0, L = depth;
  uint32_t child = nodes[0].z;
  while(child != HG_LEAF && L > 0) {
    --L;
    n = child + (((x >> L) & 1u) | (((y >> L) & 1u) << 1) | (((z >> L) & 1u) << 2));
    child = nodes[n].z;
  }
  grid[c] = (n << 5) | L;
}

/* Majorants and level of the leaf of every cell of one tree (the same
 * descent): the trace reads a cell's kmin/kmax and voxel size with two
 * independent loads instead of the grid entry, then the node.  Cells are laid
 * out by `stride' (ax0 the axis of consecutive entries).  flag: the sign of
 * kmax marks a leaf larger than a cell, so that a walk through single-cell
 * leaves needs one load; *negative is set where that sign is taken. */
__global__ void
k_majgrid(const uint4* __restrict__ nodes, uint32_t depth, uint3 def, uint32_t ax0, uint32_t ax1, int flag,
          float2* maj, uint8_t* lvl, int* negative)
{
  const uint64_t c = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const uint32_t n[3] = {def.x, def.y, def.z};
  if(c >= (uint64_t)n[0] * n[1] * n[2]) return;
  const uint32_t n0 = n[ax0], n1 = n[ax1], ax2 = 3u - ax0 - ax1;
  uint32_t at[3];
  at[ax0] = (uint32_t)(c % n0);
  at[ax1] = (uint32_t)((c / n0) % n1);
  at[ax2] = (uint32_t)(c / ((uint64_t)n0 * n1));
  uint32_t i = 0, L = depth;
  uint32_t child = nodes[0].z;
  while(child != HG_LEAF && L > 0) {
    --L;
    i = child + (((at[0] >> L) & 1u) | (((at[1] >> L) & 1u) << 1) | (((at[2] >> L) & 1u) << 2));
    child = nodes[i].z;
  }
  const uint4 v = nodes[i];
  if((int)v.y < 0) *negative = 1;
  maj[c] = make_float2(__uint_as_float(v.x), __uint_as_float(flag && L ? v.y | 0x80000000u : v.y));
  lvl[c] = (uint8_t)L;
}

}  // namespace

/* Leaf grids of the built trees (tree_count[i] > 0, in index order) into
 * `grids'; rank[i] is the grid of tree i.  Returns false (no grid built, no
 * error) when they would not fit in half of the free device memory or a tree
 * is too large for the 27-bit node index of an entry. */
bool
build_leaf_grids(DScene& S, const std::vector<uint64_t>& tree_base,
                 const std::vector<uint64_t>& tree_count, DevBuf& grids, std::vector<uint32_t>& rank,
                 bool majorants)
{
  const uint64_t ncell = (uint64_t)S.def[0] * S.def[1] * S.def[2];
  rank.assign(tree_base.size(), 0);
  uint32_t ntrees = 0;
  for(size_t i = 0; i < tree_count.size(); ++i) {
    if(!tree_count[i]) continue;
    if(tree_count[i] >= (1ull << 27)) return false;
    rank[i] = ntrees++;
  }
  if(!ntrees || !ncell) return false;
  size_t free_b = 0, total_b = 0;
  if(cudaMemGetInfo(&free_b, &total_b) != cudaSuccess) return false;
  const uint64_t bytes = (uint64_t)ntrees * ncell * (majorants ? 9 : 4);
  if(bytes > free_b / 2) return false;
  if(!grids.alloc(bytes)) return false;
  if(!majorants) {
    for(size_t i = 0; i < tree_count.size(); ++i)
      if(tree_count[i])
        k_leafgrid<<<grid_of(ncell, 256), 256>>>(S.nodes + tree_base[i], S.depth, S.def[0], S.def[1], S.def[2],
                                                  (uint32_t*)grids.ptr + (uint64_t)rank[i] * ncell);
    return cuda_ok(cudaGetLastError(), "leaf grids") && cuda_ok(cudaDeviceSynchronize(), "leaf grids");
  }
  /* most voxels of a cloudy scene are crossed by rays towards the sun, so the
   * axis whose faces these cross most often holds the consecutive entries
   * (four cells of it in one 32-byte sector); then x, y, z in order */
  uint32_t ax0 = 2;
  double most = -1.0;
  for(uint32_t a = 0; a < 3; ++a) {
    const double r = std::fabs(S.sun_dir_d[a]) * (double)S.inv_cell[a];
    if(r > most) { most = r; ax0 = a; }
  }
  const uint32_t ax1 = ax0 == 0 ? 1 : 0, ax2 = 3 - ax0 - ax1;
  S.gstride[ax0] = 1;
  S.gstride[ax1] = S.def[ax0];
  S.gstride[ax2] = S.def[ax0] * S.def[ax1];
  DevBuf neg;
  if(!neg.alloc(sizeof(int)) || !cuda_ok(cudaMemset(neg.ptr, 0, sizeof(int)), "memset")) return false;
  float2* maj = (float2*)grids.ptr;
  uint8_t* lvl = (uint8_t*)(maj + (uint64_t)ntrees * ncell);
  for(S.maj_flag = ncell < (1ull << 32) ? 1 : 0;; S.maj_flag = 0) {
    for(size_t i = 0; i < tree_count.size(); ++i) {
      if(!tree_count[i]) continue;
      const uint64_t off = (uint64_t)rank[i] * ncell;
      k_majgrid<<<grid_of(ncell, 256), 256>>>(S.nodes + tree_base[i], S.depth,
                                               make_uint3(S.def[0], S.def[1], S.def[2]), ax0, ax1, S.maj_flag,
                                               maj + off, lvl + off, (int*)neg.ptr);
    }
    int negative = 0;
    if(!cuda_ok(cudaGetLastError(), "leaf grids")
    || !cuda_ok(cudaMemcpy(&negative, neg.ptr, sizeof(int), cudaMemcpyDeviceToHost), "leaf grids"))
      return false;
    if(!negative || !S.maj_flag) return true;
  }
}

/* Builds the trees of `tasks' ((quad, property) pairs) on the device into one
 * pool; base/count are filled per task index.  Returns false on a CUDA error
 * (message in the last error). */
bool
build_octrees_gpu(const DScene& S, const std::vector<float>& sig3, const std::vector<uint32_t>& band_of,
                  const std::vector<std::pair<uint32_t, int>>& tasks, uint32_t level_force, double tau,
                  double cmax, DevBuf& pool, std::vector<uint64_t>& base, std::vector<uint64_t>& count,
                  cudaStream_t st)
{
  const uint32_t D = S.depth;
  const size_t nt = tasks.size();
  LevelDims dims{};
  dims.D = D;
  uint64_t total = 0, mtotal = 0;
  for(uint32_t L = 0; L <= D; ++L) {
    uint32_t bits = 0;
    for(int a = 0; a < 3; ++a) {
      dims.n[L][a] = (S.def[a] + (1u << L) - 1) >> L;
      while((1u << dims.bits[L][a]) < dims.n[L][a]) ++dims.bits[L][a];
      bits += dims.bits[L][a];
    }
    dims.off[L] = total;
    total += (uint64_t)dims.n[L][0] * dims.n[L][1] * dims.n[L][2];
    dims.moff[L] = mtotal;
    if(L >= 1) mtotal += 1ull << bits;
  }
  dims.off[D + 1] = total;
  dims.moff[D + 1] = mtotal;
  const uint64_t ncell = (uint64_t)S.def[0] * S.def[1] * S.def[2];

  /* trees of a batch, and its scratch: kmin, kmax, leaf; flags, their sums */
  if(!cuda_ok(cudaStreamSynchronize(st), "sync")) return false;
  size_t free_b = 0, total_b = 0;
  if(!cuda_ok(cudaMemGetInfo(&free_b, &total_b), "cudaMemGetInfo")) return false;
  const size_t budget = std::min<size_t>(free_b / 4, HG_BUILD_BYTES);
  const size_t per_tree = total * 9 + mtotal * 8 + 256;
  size_t nb = std::min<size_t>(nt, budget / per_tree);
  nb = std::min<size_t>(nb, 65535);                                          /* grid.y */
  if(mtotal) nb = std::min<size_t>(nb, ((1ull << 31) - 2) / mtotal);        /* 32-bit sums */
  nb = std::max<size_t>(nb, 1);
  const size_t nflags = nb * mtotal + 1;
  size_t cub_bytes = 0;
  cub::DeviceScan::ExclusiveSum(nullptr, cub_bytes, (uint32_t*)nullptr, (uint32_t*)nullptr, (int)nflags, st);
  size_t size = 0;
  auto place = [&](size_t bytes) { const size_t at = size; size += (bytes + 255) & ~(size_t)255; return at; };
  const size_t at_kmin = place(nb * total * 4), at_kmax = place(nb * total * 4), at_leaf = place(nb * total);
  const size_t at_flags = place(nflags * 4), at_sum = place(nflags * 4), at_cub = place(cub_bytes);
  const size_t at_tasks = place(std::max<size_t>(nt, 1) * sizeof(TreeTask));
  const size_t at_outs = place(std::max<size_t>(nt, 1) * sizeof(TreeOut));
  const size_t at_counts = place(std::max<size_t>(nt, 1) * 32 * 4);
  DevBuf scratch;
  if(!scratch.alloc(size)) return false;
  char* w = (char*)scratch.ptr;
  float *kmin = (float*)(w + at_kmin), *kmax = (float*)(w + at_kmax);
  uint8_t* leaf = (uint8_t*)(w + at_leaf);
  uint32_t *flags = (uint32_t*)(w + at_flags), *sum = (uint32_t*)(w + at_sum);
  TreeTask* d_tasks = (TreeTask*)(w + at_tasks);
  TreeOut* d_outs = (TreeOut*)(w + at_outs);
  uint32_t* d_counts = (uint32_t*)(w + at_counts);

  std::vector<TreeTask> host_tasks(nt);
  for(size_t t = 0; t < nt; ++t)
    host_tasks[t] = TreeTask{tasks[t].first, tasks[t].second, sig3[band_of[tasks[t].first] * 3 + tasks[t].second], 0};
  if(nt && !cuda_ok(cudaMemcpyAsync(d_tasks, host_tasks.data(), nt * sizeof(TreeTask), cudaMemcpyHostToDevice, st), "H2D"))
    return false;

  /* the levels of trees [t0, t0 + n) and the sums of their internal flags */
  auto levels = [&](size_t t0, size_t n) -> bool {
    const unsigned y = (unsigned)n;
    if(!cuda_ok(cudaMemsetAsync(flags, 0, (n * mtotal + 1) * 4, st), "memset")) return false;
    k_level0<<<dim3(grid_of(ncell, 256), y), 256, 0, st>>>(S.lwc, S.cell_layers, S.gas, S.nlayers, d_tasks + t0,
                                                            dims, kmin, kmax, leaf);
    for(uint32_t L = 1; L <= D; ++L) {
      const uint64_t np = (uint64_t)dims.n[L][0] * dims.n[L][1] * dims.n[L][2];
      k_level<<<dim3(grid_of(np, 256), y), 256, 0, st>>>(L, dims, kmin, kmax, leaf, level_force,
                                                          (double)(1u << L) * cmax, tau, flags);
    }
    size_t tb = cub_bytes;
    if(!cuda_ok(cub::DeviceScan::ExclusiveSum(w + at_cub, tb, flags, sum, (int)(n * mtotal + 1), st), "scan"))
      return false;
    k_counts<<<grid_of(n * 32, 256), 256, 0, st>>>(dims, y, sum, d_counts + t0 * 32);
    return cuda_ok(cudaGetLastError(), "octree levels");
  };

  /* pass 1: node counts */
  for(size_t t0 = 0; t0 < nt; t0 += nb)
    if(!levels(t0, std::min(nb, nt - t0))) return false;
  std::vector<uint32_t> internal(std::max<size_t>(nt, 1) * 32, 0);
  if(nt && (!cuda_ok(cudaMemcpyAsync(internal.data(), d_counts, nt * 32 * 4, cudaMemcpyDeviceToHost, st), "D2H")
            || !cuda_ok(cudaStreamSynchronize(st), "sync")))
    return false;
  base.assign(nt, 0);
  count.assign(nt, 0);
  std::vector<TreeOut> outs(nt);
  uint64_t total_nodes = 0;
  for(size_t t = 0; t < nt; ++t) {
    uint64_t at = 1; /* first node of depth 1 */
    for(uint32_t d = 0; d < 32; ++d) {
      outs[t].child[d] = (uint32_t)at;
      if(d < D) at += 8ull * internal[t * 32 + (D - d)];
    }
    outs[t].base = total_nodes;
    base[t] = total_nodes;
    count[t] = at;
    total_nodes += at;
  }
  if(!pool.alloc(total_nodes * 16)) return false;
  if(nt && !cuda_ok(cudaMemcpyAsync(d_outs, outs.data(), nt * sizeof(TreeOut), cudaMemcpyHostToDevice, st), "H2D"))
    return false;

  /* pass 2: the nodes (the levels again where one batch did not hold all) */
  for(size_t t0 = 0; t0 < nt; t0 += nb) {
    const size_t n = std::min(nb, nt - t0);
    if(nb < nt && !levels(t0, n)) return false;
    for(uint32_t L = D > 0 ? 1 : 0; L <= D; ++L) {
      const uint64_t np = (uint64_t)dims.n[L][0] * dims.n[L][1] * dims.n[L][2];
      k_emit<<<dim3(grid_of(8 * np, 256), (unsigned)n), 256, 0, st>>>(L, dims, kmin, kmax, leaf, sum, d_outs + t0,
                                                                      (uint4*)pool.ptr);
    }
    if(!cuda_ok(cudaGetLastError(), "octree emission")) return false;
  }
  return cuda_ok(cudaStreamSynchronize(st), "sync");
}

}  // namespace hg
