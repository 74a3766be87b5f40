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

/* Cells of a block of cell_walk().  Measured (none / 2 / 3 / 4 / 6 / 8): a
 * batch of 32 images 319 / 295 / 289 / 292 / 298 / 312 ms, a CIE image 17.8 /
 * 17.0 / 16.8 / 16.6 / 16.6 / 17.7 ms, a mesh image 34.9 / 34.1 / 31.8 / 34.6 /
 * 35.7 / 37.9 ms. */
constexpr int kWalkBlock = 3;

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
 * What bounds it: a lone path, the ~50 instructions of a cell (360 cycles,
 * 180 ns); many paths, the latency of its one majorant load.  trace_step()
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
 * 325 ms with the axis nearest to the sun consecutive, 317 ms with one loop per
 * kind, 289 ms with blocks: a transmissivity's next cells laid out together,
 * their loads in flight at once, where nothing but the sum can happen in them.
 * 1024 realisations (all latency): 5.1, 4.65 and 4.35 ms for the last three. */
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
    uint32_t careful = 0;  /* cells to take one by one before another block */
    do {
      if constexpr(Trans) {
        /* a block of kWalkBlock cells: no border, no end of the region, no null
         * collision and a transmissivity above 0.0, or else cell by cell */
        bool block = careful == 0 && ts > 0.0;
        while(block) {
          float bx = gx, by = gy, bz = gz, dx = tx, dy = ty, dz = tz, te[kWalkBlock];
          uint32_t c[kWalkBlock + 1];
          c[0] = ci;
          bool up = true;
#pragma unroll
          for(int j = 0; j < kWalkBlock; ++j) {
            te[j] = fminf(dx, fminf(dy, dz));
            const bool ax = dx == te[j], ay = !ax && dy == te[j], az = !ax && !ay;
            c[j + 1] = c[j] + (uint32_t)(ax ? ix : (ay ? iy : iz));
            bx += ax ? sx : 0.f;
            by += ay ? sy : 0.f;
            bz += az ? sz : 0.f;
            if(ax) dx = cell_plane(bx, S.cell[0], S.lower[0], T.o.x, T.inv.x);
            if(ay) dy = cell_plane(by, S.cell[1], S.lower[1], T.o.y, T.inv.y);
            if(az) dz = cell_plane(bz, S.cell[2], S.lower[2], T.o.z, T.inv.z);
            up = up && te[j] >= (j ? te[j - 1] : t);
          }
          const int lx = kx - (int)fabsf(bx - gx), ly = ky - (int)fabsf(by - gy), lz = kz - (int)fabsf(bz - gz);
          block = up && te[kWalkBlock - 1] < re && (lx | ly | lz) >= 0 && n < HG_WALK_STEPS - 64u;
          if(block) {
            float2 m[kWalkBlock + 1];
            m[0] = mm;
#pragma unroll
            for(int j = 1; j <= kWalkBlock; ++j) m[j] = __ldg(maj + c[j]);
            double a = td, sum = tmin;
            int differ = 0;
#pragma unroll
            for(int j = 0; j < kWalkBlock; ++j) {
              const double e = (double)te[j];
              sum = fma(e - a, (double)m[j].x, sum);
              a = e;
              /* the same bits: a flagged leaf without extinction (0 and -0) is
               * larger than its cell */
              differ |= __float_as_int(m[j].x) ^ __float_as_int(m[j].y);
            }
            block = !differ && sum < HG_TMIN_ZERO;
            if(block) {
              gx = bx; gy = by; gz = bz;
              tx = dx; ty = dy; tz = dz;
              kx = lx; ky = ly; kz = lz;
              ci = c[kWalkBlock];
              t = te[kWalkBlock - 1];
              td = a;
              tmin = sum;
              mm = m[kWalkBlock];
              n += kWalkBlock;
            }
          }
          if(!block) careful = kWalkBlock;
        }
        if(careful) --careful;
      }
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
  p.c_grid += 8u * n;
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
