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

/* Distance along the ray to plane g (a global cell index along one axis) */
__device__ __forceinline__ float
cell_plane(int g, float cell, float lower, float o, float inv)
{
  return __fmul_rn(__fsub_rn(__fmaf_rn((float)g, cell, lower), o), inv);
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
 * What bounds it: the latency of one majorant load per cell and the ~60
 * instructions around it (trace_step() takes ~250 and two loads).  Inside a
 * one-cell leaf the way out depends on the three next planes only, whose
 * distances come from their indices with the operations of trace_step(), so
 * the next cell's majorants are asked for before the present ones are used,
 * and the sign of a kmax says that the leaf is larger without another load.
 * Measured on a B200, 32 uneven images on clouds of up to 256x256x64 cells,
 * every warp's shortwave paths in step: 540 ms with trace_step() alone, 411 ms
 * with this loop and the x axis consecutive in the grid, 325 ms with the axis
 * nearest to the sun consecutive. */
template <unsigned V>
__device__ __forceinline__ void
cell_walk(PathTrace& p, const DScene* scenes, bool run)
{
  Trace& T = p.tr;
  if(!__any_sync(HG_FULL, run)) return;
  const DScene& S = scenes[run ? p.si : 0u];
  const int nx = (int)S.def[0], ny = (int)S.def[1], nz = (int)S.def[2];
  const bool repeat = S.repeat != 0;
  const bool trans = (V & HV_SW) && T.kind == TK_TRANS;
  int cx = (int)T.c[0], cy = (int)T.c[1], cz = (int)T.c[2];
  const int sx = T.d.x > 0.f ? 1 : -1, sy = T.d.y > 0.f ? 1 : -1, sz = T.d.z > 0.f ? 1 : -1;
  int gx = T.tile[0] * nx + cx + (sx > 0), gy = T.tile[1] * ny + cy + (sy > 0), gz = cz + (sz > 0);
  /* an axis the ray does not move along is never the way out */
  const float qx = T.d.x != 0.f ? 0.f : INFINITY, qy = T.d.y != 0.f ? 0.f : INFINITY;
  const float qz = T.d.z != 0.f ? 0.f : INFINITY;
  const float re = T.cb1;
  const uint32_t stx = S.gstride[0], sty = S.gstride[1], stz = S.gstride[2];
  const float2* maj = S.maj_grid;
  float2 mm = make_float2(0.f, 0.f);
  if(run) {
    maj += (uint64_t)T.grank * S.ncell;
    mm = __ldg(maj + ((uint32_t)cx * stx + (uint32_t)cy * sty + (uint32_t)cz * stz));
  }
  float t = T.t;
  double ts = T.Ts, tmin = T.Tmin;
  uint32_t n = 0;
  bool left = false, black = false;
  const bool ran = run;
  do {
    if(run) {
      const float tx = qx != 0.f ? qx : cell_plane(gx, S.cell[0], S.lower[0], T.o.x, T.inv.x);
      const float ty = qy != 0.f ? qy : cell_plane(gy, S.cell[1], S.lower[1], T.o.y, T.inv.y);
      const float tz = qz != 0.f ? qz : cell_plane(gz, S.cell[2], S.lower[2], T.o.z, T.inv.z);
      const float te = fminf(tx, fminf(ty, tz));
      const bool ax = tx == te, ay = !ax && ty == te, az = !ax && !ay;
      int x = cx + (ax ? sx : 0), y = cy + (ay ? sy : 0), z = cz + (az ? sz : 0);
      bool out = te >= re || (uint32_t)z >= (uint32_t)nz;
      if((uint32_t)x >= (uint32_t)nx) { out |= !repeat; x -= sx * nx; }
      if((uint32_t)y >= (uint32_t)ny) { out |= !repeat; y -= sy * ny; }
      float2 nm = mm;
      if(!out) nm = __ldg(maj + ((uint32_t)x * stx + (uint32_t)y * sty + (uint32_t)z * stz));
      /* the voxel's filter */
      const float t1 = fmaxf(fminf(te, re), t);
      bool pass = __float_as_int(mm.y) >= 0; /* a leaf of one cell */
      double ts1 = ts, tmin1 = tmin;
      if(t1 > t) {
        const double l = (double)t1 - (double)t;
        double k = (double)mm.y;
        if(trans) {
          tmin1 = fma(l, (double)mm.x, tmin);
          k -= (double)mm.x;
        }
        black = pass && trans && tmin1 >= HG_TMIN_ZERO;
        pass = pass && ts > __dmul_rn(l, k);
        ts1 = sub_tau(ts, l, k);
      }
      if(pass || black) {
        ++n;
        ts = ts1;
        tmin = tmin1;
        left = out;
        if(!out) {
          cx = x; cy = y; cz = z;
          gx += ax ? sx : 0; gy += ay ? sy : 0; gz += az ? sz : 0;
          t = te;
          mm = nm;
        }
      }
      run = pass && !black && !out && n < HG_WALK_STEPS - 64u;
    }
  } while(__any_sync(HG_FULL, run));
  if(ran) {
    p.c_seg += n;
    p.c_grid += 9u * n;
    T.steps += n;
    T.Ts = ts;
    T.Tmin = tmin;
    T.t = t;
    T.c[0] = (uint32_t)cx;
    T.c[1] = (uint32_t)cy;
    T.c[2] = (uint32_t)cz;
    /* plane index = tile * cells + cell + (1 upwards) */
    T.tile[0] = (gx - (sx > 0) - cx) / nx;
    T.tile[1] = (gy - (sy > 0) - cy) / ny;
    T.start = 0;
    if(black) trace_finish(p, true);
    else if(left) region_leave(p);
  }
}

}  // namespace

#endif /* HTRDR_WALK_CUH */
