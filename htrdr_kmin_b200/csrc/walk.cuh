/* Walk through the cloud grid in the lanes of a warp together: the part of a
 * trace that crosses single-cell leaves, 95 % of the voxels of a cloudy
 * shortwave image. */
#ifndef HTRDR_WALK_CUH
#define HTRDR_WALK_CUH

#include "transport.cuh"

namespace {

#define HG_FULL 0xffffffffu

/* Voxels a walk takes at most before the trace's step guard is looked at
 * again */
#define HG_WALK_STEPS (HG_MAX_STEPS / 2)
/* Cell indices up to here (and the planes around them) are exact in FP32 and
 * so is their sum with a tile offset */
#define HG_WALK_INDEX_MAX (1 << 23)

/* Distance along the ray to plane g (a cell index along one axis, tiles
 * included) */
__device__ __forceinline__ float
cell_plane(float g, float cell, float lower, float o, float inv)
{
  return __fmul_rn(__fsub_rn(__fmaf_rn(g, cell, lower), o), inv);
}

/* Whether cell_walk() can take a trace, set up in its cloud region: the scene
 * has the majorant grid, and no plane is beyond exact integers or finite
 * distances */
__device__ __forceinline__ bool
walk_fits(const Trace& T, const DScene& S)
{
  if(!S.maj_grid || !S.maj_flag || T.steps + HG_WALK_STEPS > HG_MAX_STEPS) return false;
  const float big = 1e30f;
  if(!(fabsf(T.o.x) < big && fabsf(T.o.y) < big && fabsf(T.o.z) < big)) return false;
  if(!((T.d.x == 0.f || fabsf(T.inv.x) < big) && (T.d.y == 0.f || fabsf(T.inv.y) < big)
       && (T.d.z == 0.f || fabsf(T.inv.z) < big)))
    return false;
  if(T.d.x == 0.f && T.d.y == 0.f && T.d.z == 0.f) return false;
  const long long gx = (long long)T.tile[0] * S.def[0] + T.c[0];
  const long long gy = (long long)T.tile[1] * S.def[1] + T.c[1];
  const long long lim = HG_WALK_INDEX_MAX - (long long)HG_WALK_STEPS - 64;
  return gx > -lim && gx < lim && gy > -lim && gy < lim && S.def[2] < (uint32_t)lim;
}

/* Cells of the cloud region, one after another, in the lanes of `run' (traces
 * that walk_fits() and that are set up in their cloud region).  A lane stops
 * before a voxel that needs trace_step() -- a leaf larger than a cell, a
 * tentative collision -- or when it leaves the region.
 *
 * What bounds it: a lone path, the ~50 instructions of a cell (410 cycles,
 * 200 ns); many paths, the latency of its one majorant load.  trace_step()
 * takes ~250 instructions and two loads.  Inside a one-cell leaf the way out
 * depends on the three next planes only, whose distances come from their
 * indices with the operations of trace_step(), so the next cell's majorants
 * are asked for before the present ones are used, and the sign of a kmax says
 * that the leaf is larger without another load.  A loop for each kind of
 * trace: a transmissivity through cells of one gas layer (kmin = kmax) has no
 * null collisions to look for, a free path no transmissivity to sum.
 * Measured on a B200, 32 uneven images on clouds of up to 256x256x64 cells,
 * every warp's shortwave paths in step: 540 ms with trace_step() alone, 411 ms
 * with a loop of ~75 instructions and the x axis consecutive in the grid,
 * 325 ms with the axis nearest to the sun consecutive, 317 ms with this loop;
 * 1024 realisations (all latency) 5.1 ms before it, 4.65 ms with it. */
template <unsigned V, bool Trans>
__device__ __forceinline__ void
cell_walk(PathTrace& p, const DScene* scenes, bool run)
{
  if(!run) return;
  Trace& T = p.tr;
  const DScene& S = scenes[p.si];
  const int nx = (int)S.def[0], ny = (int)S.def[1], nz = (int)S.def[2];
  const bool repeat = S.repeat != 0;
  const bool ux = T.d.x > 0.f, uy = T.d.y > 0.f, uz = T.d.z > 0.f;
  /* next plane of each axis, as its index, and the distance to it; an axis
   * the ray does not move along is never the way out */
  const float sx = ux ? 1.f : -1.f, sy = uy ? 1.f : -1.f, sz = uz ? 1.f : -1.f;
  float gx = (float)(T.tile[0] * nx + (int)T.c[0] + ux), gy = (float)(T.tile[1] * ny + (int)T.c[1] + uy);
  float gz = (float)((int)T.c[2] + uz);
  float tx = T.d.x != 0.f ? cell_plane(gx, S.cell[0], S.lower[0], T.o.x, T.inv.x) : INFINITY;
  float ty = T.d.y != 0.f ? cell_plane(gy, S.cell[1], S.lower[1], T.o.y, T.inv.y) : INFINITY;
  float tz = T.d.z != 0.f ? cell_plane(gz, S.cell[2], S.lower[2], T.o.z, T.inv.z) : INFINITY;
  /* cells left before the border of the grid, and the cell's place in it */
  int kx = ux ? nx - 1 - (int)T.c[0] : (int)T.c[0], ky = uy ? ny - 1 - (int)T.c[1] : (int)T.c[1];
  int kz = uz ? nz - 1 - (int)T.c[2] : (int)T.c[2];
  const int ix = ux ? (int)S.gstride[0] : -(int)S.gstride[0], iy = uy ? (int)S.gstride[1] : -(int)S.gstride[1];
  const int iz = uz ? (int)S.gstride[2] : -(int)S.gstride[2];
  uint32_t ci = T.c[0] * S.gstride[0] + T.c[1] * S.gstride[1] + T.c[2] * S.gstride[2];
  const float2* maj = S.maj_grid + (uint64_t)T.grank * S.ncell;
  float2 mm = __ldg(maj + ci);
  const float re = T.cb1;
  float t = T.t;
  double td = (double)t, ts = T.Ts, tmin = T.Tmin;
  uint32_t n = 0, nulls = 0;
  bool out = false, black = false, hit = false, skip = false;
  for(;;) {
    bool go, meet = false; /* meet: a tentative collision of a free path */
    do {
      const float te = fminf(tx, fminf(ty, tz));
      const bool ax = tx == te, ay = !ax && ty == te;
      uint32_t cn = ci + (uint32_t)(ax ? ix : (ay ? iy : iz));
      int kn = (ax ? kx : (ay ? ky : kz)) - 1;
      out = te >= re;
      int turn = 0; /* tiles crossed */
      if(kn < 0) { /* the border */
        if(repeat && (ax || ay)) {
          kn = (ax ? nx : ny) - 1;
          cn -= (uint32_t)((kn + 1) * (ax ? ix : iy));
          turn = (ax ? ux : uy) ? 1 : -1;
        } else {
          out = true;
        }
      }
      float2 nm = mm;
      if(!out) nm = __ldg(maj + cn);
      /* the voxel's filter; a segment that rounding turned round is left to
       * trace_step() */
      const double e = (double)fminf(te, re);
      const double l = e - td;
      bool pass = __float_as_int(mm.y) >= 0 && te >= t;
      if(Trans) {
        const double tn = fma(l, (double)mm.x, tmin);
        double sn = ts;
        /* the filter looks at the transmissivity before the collisions */
        black = pass && tn >= HG_TMIN_ZERO;
        if(mm.x != mm.y) { /* null collisions: not where a cell overlaps one gas layer */
          const double k = (double)mm.y - (double)mm.x;
          sn = sub_tau(ts, l, k);
          if(!(ts > __dmul_rn(l, k))) pass = false;
        } else if(!(ts > 0.0)) {
          pass = false;
        }
        if(pass || black) { tmin = tn; ts = sn; }
      } else {
        const double k = (double)mm.y;
        const bool far = skip || ts > __dmul_rn(l, k);
        meet = pass && !far && te > t;
        if(pass && far && !skip) ts = sub_tau(ts, l, k);
        pass = pass && !meet;
        skip = false;
      }
      if(pass || black) ++n;
      go = pass && !black && !out;
      out = out && pass;
      if(go) {
        if(ax) {
          gx += sx; kx = kn; T.tile[0] += turn;
          tx = cell_plane(gx, S.cell[0], S.lower[0], T.o.x, T.inv.x);
        } else if(ay) {
          gy += sy; ky = kn; T.tile[1] += turn;
          ty = cell_plane(gy, S.cell[1], S.lower[1], T.o.y, T.inv.y);
        } else {
          gz += sz; kz = kn;
          tz = cell_plane(gz, S.cell[2], S.lower[2], T.o.z, T.inv.z);
        }
        ci = cn;
        t = te;
        td = e;
        mm = nm;
        nulls = 0;
      }
    } while(go && n < HG_WALK_STEPS - 64u);
    T.c[0] = (uint32_t)(ux ? nx - 1 - kx : kx);
    T.c[1] = (uint32_t)(uy ? ny - 1 - ky : ky);
    T.c[2] = (uint32_t)(uz ? nz - 1 - kz : kz);
    if(Trans || !meet) break;
    /* the lanes that met a collision, together: the voxel_filter() of a cell */
    if(nulls >= HG_MAX_NULL) { p.flags |= PF_FAILED; skip = true; continue; }
    const double tc = td + ts / (double)mm.y;
    T.tcur = (float)tc;
    if(tc > (double)HG_MAX_DIST) { skip = true; continue; }
    const int cell = (int)((T.c[2] * S.def[1] + T.c[1]) * S.def[0] + T.c[0]);
    const int layer = cell_layer(S, (int)T.c[2], fmaf(T.d.z, T.tcur, T.o.z));
    ++p.c_tc;
    const float r = p.rng.uf();
    if(real_collision<V>(p, S, cell, layer, mm.y, r)) {
      ++n;
      hit = true;
      break;
    }
    ts = p.rng.exp1(); /* a null one: on from there */
    td = tc;
    ++nulls;
  }
  p.c_seg += n;
  p.c_grid += 9u * n;
  T.steps += n;
  T.Ts = ts;
  if(Trans) T.Tmin = tmin;
  T.t = t;
  T.start = 0;
  if(black || hit) trace_finish(p, true);
  else if(out) region_leave(p);
}

}  // namespace

#endif /* HTRDR_WALK_CUH */
