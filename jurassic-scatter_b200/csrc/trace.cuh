// Lines of sight of one-dimensional atmospheres (IP 1): the refracted ray
// march (src/lineofsight.c:5-190) once per ray, and everything that a LOS
// point needs beside it in parallel over the points.
//
//   march_kernel     the march: per ray the number of points, the surface
//                    temperature and, per point, its position, step and
//                    smoothed step, in chunks of 32 points
//   march_fit_kernel fixed-capacity runs: the rays cut to the capacity
//   edge_count_kernel  points that the aerosol/cloud layer edges add
//                    (src/lineofsight.c:193-372), a warp per ray
//   expand_kernel    the LOS records (state, columns, table brackets, layer
//                    edges) from the chunks, a warp per ray, a lane per point
//
// A march cannot know its length, so it stores as it goes: the first chunk
// of ray r is chunk r of a pool, further ones are taken from a counter and
// linked.  The prefix sum of the counts then places the records.
#pragma once
#include <limits.h>

#include "device_math.cuh"
#include "kernels.cuh"

#define JSC_CHUNK 32     // points per chunk
#define JSC_CHUNK_REC 5  // doubles per point: position (3), step, smoothed step

struct MarchPool {
  double *pts;      // [cap][JSC_CHUNK][JSC_CHUNK_REC]
  int *next;        // [cap] following chunk of the same ray, -1: none
  unsigned *count;  // [3] chunks taken beyond the first of each ray; points of the longest ray;
                    // chunks taken by march_fit_kernel
  int cap, first;   // chunks of the pool; chunks 0 .. first-1 are the rays' first ones
};

// Pressure and temperature at altitude x (src/atmosphere.c:298-315) from the
// level records that hydro_kernel builds: the quotients log(p1/p0)/(z1-z0)
// and (t1-t0)/(z1-z0) that the reference's EXP and LIN evaluate first depend
// on the level only.  h: level guess; on a strictly ascending profile the
// level whose altitudes bracket x is the one that jsc_locate finds, so the
// guess is moved level by level, else (or after four moves) it is searched.
__device__ __forceinline__ void level_state(const double *__restrict__ lev,
                                            const double *__restrict__ zl, int n, double x, int &h,
                                            double *p, double *t) {
  const double2 *q = reinterpret_cast<const double2 *>(lev) + 4 * (size_t)h;
  double2 zz = __ldg(q), pt = __ldg(q + 1), sl = __ldg(q + 2), fl = __ldg(q + 3);
  int moves = 0;
  while (!(fl.y != 0 && (!(zz.x > x) || h == 0) && (zz.y > x || h == n - 2))) {
    if (fl.y != 0 && x == x && ++moves <= 4) h += zz.x > x ? -1 : 1;
    else h = jsc_locate(zl, n, x);
    q = reinterpret_cast<const double2 *>(lev) + 4 * (size_t)h;
    zz = __ldg(q);
    pt = __ldg(q + 1);
    sl = __ldg(q + 2);
    fl = __ldg(q + 3);
    if (fl.y == 0 || !(x == x)) break;  // searched: nothing to verify
  }
  const double dz = x - zz.x;
  *p = fl.x != 0 ? pt.x * exp(sl.x * dz) : pt.x + sl.x * dz;
  *t = pt.y + sl.y * dz;
}

// Where the segment from g0 to g1 (z, lon, lat) crosses altitude z
// (intersection_point, src/lineofsight.c:385-407).
__device__ __forceinline__ void segment_point(const double *g0, const double *g1, double z,
                                              double *go) {
  double x1[3], x2[3];
  const double frac = (g0[0] - z) / (g0[0] - g1[0]);
  jsc_geo2cart(g0[0], g0[1], g0[2], x1);
  jsc_geo2cart(g1[0], g1[1], g1[2], x2);
  for (int i = 0; i < 3; i++) x2[i] = x1[i] + frac * (x2[i] - x1[i]);
  jsc_cart2geo(x2, &go[0], &go[1], &go[2]);
}

__device__ __forceinline__ double radius_of(const double *x) {
  return sqrt(x[0] * x[0] + x[1] * x[1] + x[2] * x[2]);
}

// Level guess of altitude z: from the spacing (zf: lowest altitude, zs: levels
// per km) on evenly spaced profiles, else (zs 0) the level h of the lookup
// before.
__device__ __forceinline__ int level_guess(double zf, double zs, int n, double z, int h) {
  return zs > 0 ? min(max(__double2int_rz((z - zf) * zs), 0), n - 2) : h;
}

// The march of one ray.  LANES 8: a group of eight lanes per ray (gmask:
// the group's lanes, role: the lane's number in it) holds the same ray
// state; a refracted step needs the state at five positions (the point, the
// middle of the step, and that displaced along each axis), and each lane
// looks up one.  LANES 1: a thread per ray looks them up one after another.
// ENDS: store nothing, report the last two points in *end (the solar
// direction search).  FIT: store the first `limit` points only.  Returns the
// number of points.
template <int LANES, bool ENDS, bool FIT = false>
__device__ __forceinline__ int march_ray(const RayArgs &A, const MarchPool &M, int ai, int r,
                                         const RayIn &in, unsigned gmask, int role, RayEnd *end,
                                         double *tsurf, int limit = 0) {
  const int lo = A.atm_off[ai], n = A.atm_off[ai + 1] - lo;
  const double *__restrict__ lev = A.lev + 8 * (size_t)lo;
  const double *__restrict__ zl = A.z + lo;
  const double zmin = A.zmin[ai], zmax = A.zmax[ai];
  const double zf = zl[0], zs = lev[7] == 2 ? (n - 1) / (zl[n - 1] - zf) : 0.0;
  *tsurf = -999;
  if (in.obsz < zmin) {
    if (role == 0) atomicOr(A.status, JSC_DEV_ERR_OBSERVER);
    return 0;
  }
  if (in.vpz > zmax - 0.001) return 0;

  double x[3], ex0[3], xp[3] = {0, 0, 0}, xpp[3] = {0, 0, 0};
  {
    double xobs[3], xvp[3];
    jsc_geo2cart(in.obsz, in.obslon, in.obslat, xobs);
    jsc_geo2cart(in.vpz, in.vplon, in.vplat, xvp);
    for (int i = 0; i < 3; i++) ex0[i] = xvp[i] - xobs[i];
    const double norm = radius_of(ex0);
    for (int i = 0; i < 3; i++) ex0[i] /= norm;
    for (int i = 0; i < 3; i++) x[i] = xobs[i];
    // Observer above the atmosphere: bisect for the entry point.
    if (in.obsz > zmax) {
      double dmin = 0, dmax = norm;
      while (fabs(dmin - dmax) > 0.001) {
        const double d = (dmax + dmin) / 2;
        for (int i = 0; i < 3; i++) x[i] = xobs[i] + d * ex0[i];
        const double z = radius_of(x) - JSC_RE;
        if (z <= zmax && z > zmax - 0.001) break;
        if (z < zmax - 0.0005) dmax = d; else dmin = d;
      }
    }
  }

  int np = 0, chunk = r, h0 = n - 2, h1 = n - 2;
  double rprev = 0, dprev = 0, tlast = 0, zlast = 0;
  bool bent = true;  // tlast holds the temperature looked up last
  while (1) {
    if (np >= NLOS) {
      if (role == 0) atomicOr(A.status, JSC_DEV_ERR_NLOS);
      return np;
    }
    const double norm = radius_of(x), z = norm - JSC_RE;
    double *rec = nullptr;
    if (!ENDS && (!FIT || np < limit)) {
      if ((np & (JSC_CHUNK - 1)) == 0 && np > 0 && chunk >= 0) {  // the next chunk
        int id = 0;
        if (role == 0) {
          id = M.first + (int)atomicAdd(M.count, 1u);
          if (id >= M.cap || id < 0) id = -1;
          M.next[chunk] = id;
        }
        chunk = LANES == 1 ? id : __shfl_sync(gmask, id, 0, LANES);
      }
      if (chunk >= 0)
        rec = M.pts + ((size_t)chunk * JSC_CHUNK + (np & (JSC_CHUNK - 1))) * JSC_CHUNK_REC;
    }
    if (z < zmin + 0.001 || z > zmax + 0.001) {
      // Last point: where the segment from the previous point crosses the
      // boundary.  It is stored as (z, lon, lat) with a step of 0.
      const int stop = z < zmin + 0.001 ? 2 : 1;
      double g0[3], g1[3], g[3];
      jsc_cart2geo(x, &g1[0], &g1[1], &g1[2]);
      if (np > 0) jsc_cart2geo(xp, &g0[0], &g0[1], &g0[2]);
      else for (int i = 0; i < 3; i++) g0[i] = g1[i];
      segment_point(g0, g1, stop == 2 ? zmin : zmax, g);
      if (rec && role == 0) {
        rec[0] = g[0];
        rec[1] = g[1];
        rec[2] = g[2];
        rec[3] = 0.;
        rec[4] = np == 0 ? 0. : 0.5 * (dprev + 0.);
      }
      np++;
      if (stop == 2) {
        if (!bent) {
          double p;
          level_state(lev, zl, n, zlast, h0, &p, &tlast);
        }
        *tsurf = tlast;
      }
      // A last point that follows a too-short step is dropped
      // (src/lineofsight.c:170-171).
      const bool dropped = np >= 3 && rprev < 1e-3;
      if (dropped) np--;
      if (ENDS) {
        end->tsurf = *tsurf;
        if (dropped) jsc_cart2geo(xpp, &end->g[0][0], &end->g[0][1], &end->g[0][2]);
        for (int i = 0; i < 3; i++) {
          if (!dropped) end->g[0][i] = g0[i];
          end->g[1][i] = dropped ? g0[i] : g[i];
        }
      }
      break;
    }
    double ds = A.rayds;
    if (A.raydz > 0) {
      double xh[3];
      const double rn = 1 / norm;
      for (int i = 0; i < 3; i++) xh[i] = div_known(x[i], norm, rn);
      const double cosa = fabs(ex0[0] * xh[0] + ex0[1] * xh[1] + ex0[2] * xh[2]);
      if (cosa != 0) {
        const double dz = A.raydz / cosa;
        ds = (A.rayds < dz ? A.rayds : dz);  // GSL_MIN
      }
    }
    // Steps are smoothed along the ray (src/lineofsight.c:177-179).
    const double dsm = np == 0 ? 0.5 * ds : 0.5 * (dprev + ds);
    if (rec) {
      if (LANES == 1) {
        rec[0] = x[0];
        rec[1] = x[1];
        rec[2] = x[2];
        rec[3] = ds;
        rec[4] = dsm;
      } else if (role < JSC_CHUNK_REC) {
        rec[role] = role == 0 ? x[0] : role == 1 ? x[1] : role == 2 ? x[2] : role == 3 ? ds : dsm;
      }
    }
    np++;
    rprev = ds;
    dprev = dsm;
    if (ENDS)
      for (int i = 0; i < 3; i++) xpp[i] = xp[i];
    for (int i = 0; i < 3; i++) xp[i] = x[i];

    // Refraction (src/lineofsight.c:122-166).
    bent = A.refrac && z <= JSC_ZREFRAC;
    double ex1[3], ng[3] = {0, 0, 0}, nr = 1;
    if (bent) {
      double xm[3];
      for (int i = 0; i < 3; i++) xm[i] = x[i] + 0.5 * ds * ex0[i];
      double p, t;
      if (LANES > 1) {
        // lane 0 the point, 1 the middle, 2-4 the middle displaced; the
        // reference displaces in place, so an axis displaced before keeps
        // the rounding of + step - step
        for (int i = 0; i < 3; i++) {
          const double up = xm[i] + JSC_FD_STEP;
          if (role == 2 + i) xm[i] = up;
          else if (role > 2 + i) xm[i] = up - JSC_FD_STEP;
        }
        if (role == 0 || role > 4)
          for (int i = 0; i < 3; i++) xm[i] = x[i];
        const double zm = radius_of(xm) - JSC_RE;
        h0 = level_guess(zf, zs, n, zm, h0);
        level_state(lev, zl, n, zm, h0, &p, &t);
        const double rf = jsc_refractivity(p, t);
        nr = 1 + __shfl_sync(gmask, rf, 0, LANES);
        const double g = div_known(rf - __shfl_sync(gmask, rf, 1, LANES), JSC_FD_STEP,
                                   1 / JSC_FD_STEP);
        for (int i = 0; i < 3; i++) ng[i] = __shfl_sync(gmask, g, 2 + i, LANES);
        tlast = __shfl_sync(gmask, t, 4, LANES);
      } else {
        level_state(lev, zl, n, z, h0, &p, &t);
        nr = 1 + jsc_refractivity(p, t);
        level_state(lev, zl, n, radius_of(xm) - JSC_RE, h1, &p, &t);
        const double rm = jsc_refractivity(p, t);
        int h2 = h1;
#pragma unroll
        for (int i = 0; i < 3; i++) {
          xm[i] += JSC_FD_STEP;
          level_state(lev, zl, n, radius_of(xm) - JSC_RE, h2, &p, &t);
          ng[i] = div_known(jsc_refractivity(p, t) - rm, JSC_FD_STEP, 1 / JSC_FD_STEP);
          xm[i] -= JSC_FD_STEP;
        }
        tlast = t;
      }
    } else {
      zlast = z;
    }
    for (int i = 0; i < 3; i++) ex1[i] = ex0[i] * nr;
    for (int i = 0; i < 3; i++) ex1[i] += ds * ng[i];
    const double en = radius_of(ex1), re = 1 / en;
    for (int i = 0; i < 3; i++) ex1[i] = div_known(ex1[i], en, re);
    for (int i = 0; i < 3; i++) x[i] += 0.5 * ds * (ex0[i] + ex1[i]);
    for (int i = 0; i < 3; i++) ex0[i] = ex1[i];
  }
  return np;
}

template <int LANES>
__device__ __forceinline__ void march_one(const RayArgs &A, const MarchPool &M, int r,
                                          unsigned gmask, int role) {
  const RayIn in = {A.obsz[r], A.obslon[r], A.obslat[r], A.vpz[r], A.vplon[r], A.vplat[r]};
  double tsurf;
  const int np = march_ray<LANES, false>(A, M, A.ray_atm[r], r, in, gmask, role, nullptr, &tsurf);
  if (role == 0) {
    A.nlos[r] = np;
    A.tsurf[r] = tsurf;
    if ((unsigned)np > *(volatile unsigned *)(M.count + 1)) atomicMax(M.count + 1, (unsigned)np);
    A.tp[r] = in.vpz;  // where no tangent point is found
    A.tp[A.n_rays + r] = in.vplon;
    A.tp[2 * A.n_rays + r] = in.vplat;
  }
}

template <int LANES>
__global__ void __launch_bounds__(128) march_kernel(RayArgs A, MarchPool M) {
  const int tid = blockIdx.x * blockDim.x + threadIdx.x, r = tid / LANES;
  const int role = LANES == 1 ? 0 : (int)(threadIdx.x & (LANES - 1));
  const unsigned gmask = LANES == 1 ? 0u : ((1u << LANES) - 1u) << ((threadIdx.x & 31) - role);
  if (r >= A.n_rays) return;  // whole groups leave together
  march_one<LANES>(A, M, r, gmask, role);
}

// The pencils of one round of a fixed-capacity scattering run as a device
// work queue: a persistent grid pulls them a warp (32 pencils) at a time
// from the queue head until the round's live count, which only the device
// knows; slots past it are never traced (their nlos stays 0, cleared
// before).  Pulling balances the uneven pencil lengths across the SMs.
static __global__ void __launch_bounds__(128) march_queue_kernel(RayArgs A, MarchPool M,
                                                                 unsigned *head, const int *live) {
  const int lane = threadIdx.x & 31;
  const int n = *live < A.n_rays ? *live : A.n_rays;
  for (;;) {
    int r0 = 0;
    if (lane == 0) r0 = (int)atomicAdd(head, 32u);
    r0 = __shfl_sync(0xffffffffu, r0, 0);
    if (r0 >= n) break;
    if (r0 + lane < n) march_one<1>(A, M, r0 + lane, 0u, 0);
  }
}

// Fixed-capacity runs, a thread per ray, after the prefix sum A.los_off of
// the marched counts A.nlos: a ray that reaches past the max_seg points of
// the LOS buffers keeps the points inside them and no surface, and the run
// reports it.  The pool holds every chain inside the buffers, but the march
// takes chunks as it goes, so rays past their end may have taken those of rays
// before: where the pool ran out, the rays inside march once more, up to that
// end and on a counter of their own (first chunks and at most one per 32
// points of the buffers: the pool's size).  The chains of the others are not
// read again.
static __global__ void __launch_bounds__(128) march_fit_kernel(RayArgs A, MarchPool M,
                                                               int64_t max_seg) {
  const int r = blockIdx.x * blockDim.x + threadIdx.x;
  if (r >= A.n_rays) return;
  const int np = A.nlos[r];
  const int64_t room = max_seg - A.los_off[r];
  if (np > room) {
    atomicOr(A.status, JSC_DEV_ERR_NLOS);
    A.nlos[r] = room > 0 ? (int)room : 0;
    A.tsurf[r] = -999;
  }
  if (np == 0 || room <= 0 || (int64_t)M.count[0] + M.first <= M.cap) return;
  const RayIn in = {A.obsz[r], A.obslon[r], A.obslat[r], A.vpz[r], A.vplon[r], A.vplat[r]};
  double tsurf;
  M.count += 2;
  march_ray<1, false, true>(A, M, A.ray_atm[r], r, in, 0u, 0, nullptr, &tsurf,
                            room < np ? (int)room : np);
}

// ------------------------------------------------------ aerosol layers --

// Layer edges as the refinement sees them (n_alti altitudes, top down).
struct EdgeSet {
  int n_alti;
  double altimax, altimin;
  const double *alti;
};

// Crossings of the segment from altitude zp to zc with the edges
// (src/lineofsight.c:252-290).
__device__ __forceinline__ bool edge_window(const EdgeSet &E, double zp, double zc) {
  return (zp < E.altimax || zc < E.altimax) && (zp > E.altimin || zc > E.altimin);
}

__device__ __forceinline__ int edge_crossings(const EdgeSet &E, double zp, double zc) {
  int c = 0;
  if (edge_window(E, zp, zc))
    for (int il = 0; il < E.n_alti; il++) {
      const double z1 = E.alti[il], z2 = E.alti[E.n_alti - il - 1];
      c += (zp > z1 && zc < z1) + (zp < z2 && zc > z2);
    }
  return c;
}

__device__ __forceinline__ double chunk_altitude(const double *rec) {
  return rec[3] == 0. ? rec[0] : radius_of(rec) - JSC_RE;
}

struct ExpandArgs {
  int n_rays, ng, nw, W, n_levels, ig_h2o;
  const int *ray_atm, *atm_off;
  const double *z, *lev, *q, *k, *qs;  // profiles
  MarchPool M;
  const int *nlos_b;               // points of the march
  int *nlos;                       // points with the layer edges
  const int64_t *off;
  const int64_t *raw;              // prefix sum of the marched counts (fixed-capacity runs), or null
  double *geo, *pts, *tp;
  int64_t max_seg, max_count;      // points of the buffers; most points of a ray
  EdgeSet E;
  int nl;                          // aerosol/cloud layers
  double transs;
  const double *top, *bottom, *trans;
  int grid_np;                     // (p, T) grid shared by every table
  const double *grid_p, *grid_t;
  const int *grid_nt;
  unsigned *status;
};

// Points of each ray with the layer edges: its marched points plus the
// crossings of its segments.
static __global__ void __launch_bounds__(128) edge_count_kernel(ExpandArgs A) {
  const int r = (int)(((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5);
  const int lane = threadIdx.x & 31;
  if (r >= A.n_rays) return;  // whole warps leave together
  const int nb = A.nlos_b[r];
  int o = 0, chunk = r;
  double carry = 0;  // altitude of the point before the chunk
  for (int c0 = 0; c0 < nb && chunk >= 0; c0 += JSC_CHUNK) {
    const int ip = c0 + lane;
    double zc = 0;
    if (ip < nb) zc = chunk_altitude(A.M.pts + ((size_t)chunk * JSC_CHUNK + lane) * JSC_CHUNK_REC);
    double zp = __shfl_up_sync(0xffffffffu, zc, 1);
    if (lane == 0) zp = carry;
    carry = __shfl_sync(0xffffffffu, zc, 31);
    if (ip < nb) o += 1 + (ip > 0 ? edge_crossings(A.E, zp, zc) : 0);
    if (c0 + JSC_CHUNK < nb) chunk = A.M.next[chunk];
  }
  o = __reduce_add_sync(0xffffffffu, o);
  if (lane) return;
  if (o > NLOS || o > A.max_count) {
    atomicOr(A.status, JSC_DEV_ERR_NLOS);
    o = 0;
  }
  A.nlos[r] = o;
}

// Ray r reaches past the LOS buffers: it has no tangent point.
__device__ __forceinline__ bool past_buffers(const ExpandArgs &A, int r) {
  return A.raw && A.raw[r + 1] > A.max_seg;
}

// Geography to position and back as calls: they are used at several places
// of the kernels below, whose instructions would not stay in the
// instruction cache if each were inlined.
struct Vec3 {
  double v[3];
};

static __device__ __noinline__ Vec3 cart_of(double z, double lon, double lat) {
  Vec3 x;
  jsc_geo2cart(z, lon, lat, x.v);
  return x;
}

static __device__ __noinline__ Vec3 geo_of(double x0, double x1, double x2) {
  const double x[3] = {x0, x1, x2};
  Vec3 g;
  jsc_cart2geo(x, &g.v[0], &g.v[1], &g.v[2]);
  return g;
}

// The point of segment_point.
__device__ __forceinline__ Vec3 crossing_of(const double *g0, const double *g1, double z) {
  const double frac = (g0[0] - z) / (g0[0] - g1[0]);
  const Vec3 a = cart_of(g0[0], g0[1], g0[2]), b = cart_of(g1[0], g1[1], g1[2]);
  double x[3];
  for (int i = 0; i < 3; i++) x[i] = a.v[i] + frac * (b.v[i] - a.v[i]);
  return geo_of(x[0], x[1], x[2]);
}

// Record of a LOS point: the state at its altitude z, the column densities
// over its step ds (src/lineofsight.c:182-185), the table brackets, and the
// layer factor (af, ai).  The LIN quotients of a level are in qs.
static __device__ __noinline__ void write_record(const ExpandArgs &A, int lo, int n, double *rec,
                                                 double z, double ds, double af, double ai) {
  const double *zl = A.z + lo, *lev = A.lev + 8 * (size_t)lo;
  const double zf = zl[0];
  int h = level_guess(zf, (n - 1) / (zl[n - 1] - zf), n, z, n - 2);
  double p, t;
  level_state(lev, zl, n, z, h, &p, &t);
  const double dz = z - zl[h];
  const size_t nl = (size_t)A.n_levels, l = (size_t)lo + h;
  rec[REC_P] = p;
  rec[REC_T] = t;
  rec[REC_DS] = ds;
  rec[REC_QH2O] = A.ig_h2o >= 0 ? A.q[A.ig_h2o * nl + l] + A.qs[A.ig_h2o * nl + l] * dz : 0.0;
  rec[REC_GRID] = A.grid_p ? (double)grid_code(A.grid_np, A.grid_p, A.grid_nt, A.grid_t, p, t) : -1.0;
  rec[REC_PLK] = (double)planck_index(t);
  rec[REC_AF] = af;
  rec[REC_AI] = ai;
#pragma unroll 1
  for (int w = 0; w < A.nw; w++)
    rec[REC_K + w] = A.k[w * nl + l] + A.qs[(A.ng + w) * nl + l] * dz;
#pragma unroll 1
  for (int g = 0; g < A.ng; g++) {
    const double q = A.q[g * nl + l] + A.qs[g * nl + l] * dz;
    rec[REC_K + A.nw + g] = 10 * q * p / (JSC_KBOLTZ * t) * ds;
  }
}

// Aerosol/cloud layer and factor of a point at altitude z whose predecessor
// lies at zprev (src/lineofsight.c:332-372).
__device__ __forceinline__ void layer_factor(const ExpandArgs &A, double zprev, double z,
                                             double *af, double *ai) {
  int aeroi = -999;
  double aerofac = 0.;
  if (edge_window(A.E, zprev, z)) {
    for (int il = 0; il < A.nl; il++) {
      if (z <= A.top[il] && z >= A.bottom[il]) {
        aeroi = il;
        aerofac = 1.;
      }
      if (A.trans[il] > A.transs && z <= (A.top[il] + A.trans[il]) && z > A.top[il]) {
        aeroi = il;
        aerofac = (A.top[il] + A.trans[il] - z) / A.trans[il];
      }
      if (A.trans[il] > A.transs && z < A.bottom[il] && z >= (A.bottom[il] - A.trans[il])) {
        aeroi = il;
        aerofac = fabs(A.bottom[il] - A.trans[il] - z) / A.trans[il];
      }
    }
  }
  *af = aerofac;
  *ai = (double)aeroi;
}

// Geometry and step of marched point ip of ray r (walks the ray's chunks).
__device__ inline double marched_point(const MarchPool &M, int r, int ip, double *g) {
  int chunk = r;
  for (int c = ip / JSC_CHUNK; c > 0 && chunk >= 0; c--) chunk = M.next[chunk];
  if (chunk < 0) {
    g[0] = g[1] = g[2] = 0;
    return 0;
  }
  const double *rec = M.pts + ((size_t)chunk * JSC_CHUNK + (ip & (JSC_CHUNK - 1))) * JSC_CHUNK_REC;
  const Vec3 x = rec[3] == 0. ? Vec3{{rec[0], rec[1], rec[2]}} : geo_of(rec[0], rec[1], rec[2]);
  for (int i = 0; i < 3; i++) g[i] = x.v[i];
  return rec[3];
}

// Tangent point of each ray, a thread per ray, from its marched points;
// rays without records are cut.
// (src/lineofsight.c:411-452); tp[r] holds the number of the lowest one.
static __global__ void __launch_bounds__(128) tangent_kernel(ExpandArgs A) {
  const int r = blockIdx.x * blockDim.x + threadIdx.x;
  if (r >= A.n_rays) return;
  const int np = A.nlos_b[r];
  if (np == 0) return;
  if (A.off[r] + A.nlos[r] > A.max_seg)  // expand_kernel<true> has written nothing
    cut_ray(lines_of(A), r, 0, 1, A.off[r], A.nlos[r]);
  if (past_buffers(A, r)) return;
  const int m = (int)A.tp[r];
  double g0[3], g1[3], g2[3], tp[3];
  if (m <= 0 || m >= np - 1) {
    marched_point(A.M, r, np - 1, tp);
  } else {
    marched_point(A.M, r, m - 1, g0);
    const double d1 = marched_point(A.M, r, m, g1), d2 = marched_point(A.M, r, m + 1, g2);
    const double yy0 = g0[0], yy1 = g1[0], yy2 = g2[0];
    const double x1 = sqrt(d1 * d1 - (yy1 - yy0) * (yy1 - yy0));
    const double x2 = x1 + sqrt(d2 * d2 - (yy2 - yy1) * (yy2 - yy1));
    const double aa = 1 / (x1 - x2) * (-(yy0 - yy1) / x1 + (yy0 - yy2) / x2);
    const double bb = -(yy0 - yy1) / x1 - aa * x1;
    const double cc = yy0;
    const double xx = -bb / (2 * aa);
    const Vec3 v0 = cart_of(g0[0], g0[1], g0[2]), v2 = cart_of(g2[0], g2[1], g2[2]);
    double v[3];
    for (int i = 0; i < 3; i++) v[i] = jsc_lin(0.0, v0.v[i], x2, v2.v[i], xx);
    const Vec3 g = geo_of(v[0], v[1], v[2]);
    tp[0] = aa * xx * xx + bb * xx + cc;
    tp[1] = g.v[1];
    tp[2] = g.v[2];
  }
  for (int i = 0; i < 3; i++) A.tp[(size_t)i * A.n_rays + r] = tp[i];
}

// LOS records of a ray by one warp.  EDGES: the points where segments cross
// layer edges go in between (add_aerosol_layers, src/lineofsight.c:193-372).
// Lanes take 32 marched points at a time; a warp scan of their output counts
// (crossings of the segment before the point, then the point) numbers the
// output points, and lanes then take output points, so that the crossings of
// one segment (a dozen where it enters a layer with a transition zone) run in
// parallel.  A second pass takes 32 output points at a time for the records,
// with the neighbours' Cartesian positions passed by shuffles for the chord
// steps.  Bound by instruction issue; with the crossings in the lane of
// their segment, every function inlined and the tangent point in lane 0 the
// warps waited for instructions (9.9 of 17 cycles an issue, 11.7 lanes
// active), 9.6 ms for 232,000 pencils, 3.28 after that, 3.03 since the last lane
// no longer converts its following point by itself.
// A ray whose records do not fit (a fixed-capacity run, EDGES) gets none, and
// tangent_kernel cuts it; without edges march_fit_kernel has.
template <bool EDGES>
__global__ void __launch_bounds__(128, EDGES ? 6 : 8) expand_kernel(const __grid_constant__ ExpandArgs A) {
  const int r = (int)(((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5);
  const int lane = threadIdx.x & 31;
  const unsigned full = 0xffffffffu;
  if (r >= A.n_rays) return;  // whole warps leave together
  const int nb = A.nlos_b[r];
  if (nb == 0) return;
  const int ai = A.ray_atm[r], lo = A.atm_off[ai], nlev = A.atm_off[ai + 1] - lo;
  const int64_t base = A.off[r];
  // points to write; none where they do not fit
  const int nmax = !EDGES ? nb : base + A.nlos[r] <= A.max_seg ? A.nlos[r] : -1;
  // lowest marched point: the first NaN, else the first smallest altitude
  double zlow = 0;
  int mlow = INT_MAX, mnan = INT_MAX;
  double prev[3] = {0, 0, 0};  // geometry of the point before the chunk
  int chunk = r, o = 0;
  for (int c0 = 0; c0 < nb; c0 += JSC_CHUNK) {
    if (chunk < 0) {  // cannot be: the pool holds the chains of a run's last march
      if (lane == 0) {
        atomicOr(A.status, JSC_DEV_ERR_NLOS);
        A.nlos[r] = 0;
      }
      return;
    }
    const int ip = c0 + lane;
    const double *rec = A.M.pts + ((size_t)chunk * JSC_CHUNK + lane) * JSC_CHUNK_REC;
    double g[3] = {0, 0, 0}, raw = 0, ds = 0;
    if (ip < nb) {
      raw = rec[3];
      ds = rec[4];
      const Vec3 x = raw == 0. ? Vec3{{rec[0], rec[1], rec[2]}} : geo_of(rec[0], rec[1], rec[2]);
      for (int i = 0; i < 3; i++) g[i] = x.v[i];
      if (isnan(g[0])) mnan = min(mnan, ip);
      else if (mlow == INT_MAX || g[0] < zlow) {
        zlow = g[0];
        mlow = ip;
      }
    }
    if (!EDGES) {
      if (ip < nb) {
        if (base + ip >= A.max_seg) {
          atomicOr(A.status, JSC_DEV_ERR_NLOS);
        } else {
          double *go = A.geo + (base + ip) * 4;
          go[0] = g[0];
          go[1] = g[1];
          go[2] = g[2];
          go[3] = raw;
          write_record(A, lo, nlev, A.pts + (base + ip) * A.W, g[0], ds, 0.0, -999.0);
        }
      }
    } else {
      double gp[3];
      for (int i = 0; i < 3; i++) {
        gp[i] = __shfl_up_sync(full, g[i], 1);
        if (lane == 0) gp[i] = prev[i];
        prev[i] = __shfl_sync(full, g[i], 31);
      }
      const int cnt = ip < nb ? 1 + (ip > 0 ? edge_crossings(A.E, gp[0], g[0]) : 0) : 0;
      int incl = cnt;
      for (int d = 1; d < 32; d <<= 1) {
        const int v = __shfl_up_sync(full, incl, d);
        if (lane >= d) incl += v;
      }
      const int total = __shfl_sync(full, incl, 31);
#pragma unroll 1
      for (int s0 = 0; s0 < total && o + total <= nmax; s0 += 32) {
        // output point s of the chunk: the k-th crossing before marched point
        // src, or (k = its crossings) that point
        const int s = s0 + lane;
        int src = 0;
        for (int d = 16; d > 0; d >>= 1)
          if (__shfl_sync(full, incl, src + d - 1) <= s) src += d;
        src = min(src, 31);
        const int cs = __shfl_sync(full, cnt, src);
        int k = s - (__shfl_sync(full, incl, src) - cs);
        double a[3], b[3];
        for (int i = 0; i < 3; i++) {
          a[i] = __shfl_sync(full, gp[i], src);
          b[i] = __shfl_sync(full, g[i], src);
        }
        if (s < total) {
          if (k < cs - 1) {
            double znew = 0;
            for (int il = 0; il < A.E.n_alti && k >= 0; il++) {
              const double z1 = A.E.alti[il], z2 = A.E.alti[A.E.n_alti - il - 1];
              if (a[0] > z1 && b[0] < z1 && k-- == 0) znew = z1;
              if (a[0] < z2 && b[0] > z2 && k-- == 0) znew = z2;
            }
            const Vec3 x = crossing_of(a, b, znew);
            for (int i = 0; i < 3; i++) b[i] = x.v[i];
          }
          double *go = A.geo + (base + o + s) * 4;
          go[0] = b[0];
          go[1] = b[1];
          go[2] = b[2];
        }
      }
      o += total;
    }
    if (c0 + JSC_CHUNK < nb) chunk = A.M.next[chunk];
  }
  for (int d = 16; d > 0; d >>= 1) {
    const double oz = __shfl_xor_sync(full, zlow, d);
    const int om = __shfl_xor_sync(full, mlow, d);
    if (om != INT_MAX && (mlow == INT_MAX || oz < zlow || (oz == zlow && om < mlow))) {
      zlow = oz;
      mlow = om;
    }
  }
  mnan = __reduce_min_sync(full, mnan);
  if (lane == 0 && !past_buffers(A, r)) A.tp[r] = (double)(mnan != INT_MAX ? mnan : mlow);
  if (!EDGES) return;
  if (o != nmax) return;
  __syncwarp();  // the geometry written above, for every lane
  const double *go = A.geo + base * 4;
  double carry[3] = {0, 0, 0};  // position of the point before the 32
  // Position of output point i.  The next 32 are converted ahead, so that the
  // last lane has its following point without a conversion of its own.
  auto position = [&](int i) {
    return i < o ? cart_of(go[(size_t)i * 4], go[(size_t)i * 4 + 1], go[(size_t)i * 4 + 2])
                 : Vec3{{0, 0, 0}};
  };
  Vec3 xq = position(lane);
#pragma unroll 1
  for (int i0 = 0; i0 < o; i0 += 32) {
    const int i = i0 + lane;
    double xp[3], xn[3];
    const Vec3 xc = xq;
    xq = position(i + 32);
    for (int c = 0; c < 3; c++) {
      const double up = __shfl_up_sync(full, xc.v[c], 1);
      xp[c] = lane == 0 ? carry[c] : up;
      // lane 0 hands the first of the next 32 to lane 31
      xn[c] = __shfl_sync(full, lane == 0 ? xq.v[c] : xc.v[c], (lane + 1) & 31);
      carry[c] = __shfl_sync(full, xc.v[c], 31);
    }
    if (i < o) {
      const double z = go[(size_t)i * 4];
      // chord step (src/lineofsight.c:300-330)
      double ds = 0;
      if (o > 1) {
        const double *c = xc.v;
        const double back = sqrt((xp[0] - c[0]) * (xp[0] - c[0]) + (xp[1] - c[1]) * (xp[1] - c[1]) +
                                 (xp[2] - c[2]) * (xp[2] - c[2]));
        const double ahead = sqrt((c[0] - xn[0]) * (c[0] - xn[0]) + (c[1] - xn[1]) * (c[1] - xn[1]) +
                                  (c[2] - xn[2]) * (c[2] - xn[2]));
        ds = i == 0 ? 0.5 * ahead : i == o - 1 ? 0.5 * back : 0.5 * (back + ahead);
      }
      A.geo[(base + i) * 4 + 3] = ds;
      // At i = 0 the reference compares z[-1]; the first point, at the top
      // of the atmosphere and outside every layer, stands in for it.
      double af, la;
      layer_factor(A, go[(size_t)(i > 0 ? i - 1 : 0) * 4], z, &af, &la);
      write_record(A, lo, nlev, A.pts + (base + i) * A.W, z, ds, af, la);
    }
  }
}
