// Device kernels of the scattering source (srcfunc_sca, src/scatter.c:643-807
// for thermal radiation in 1-D atmospheres, :899-1041 for the sun).
//
//   sp_count_kernel     scattering points per ray (LOS points with aerosol
//                       factor > 0, src/forwardmodel.c:317)
//   sp_list_kernel      one record per scattering point: position, LOS
//                       direction, layer, observation time, profile
//   sp_spawn_kernel     the secondary pencils of a chunk of points, written
//                       as the rays of a child batch (src/scatter.c:698-735)
//   sp_weights_kernel, sp_integral_kernel
//                       phase-function weighted integral of the secondary
//                       radiances over 180 x 180 directions (:737-800)
//   sun_kernel          solar direction search by repeated ray tracing and
//                       the solar pencil of each point (:899-995)
//   sun_add_kernel      adds the attenuated solar term to the source
//
// A batch whose rays scatter runs, bottom up: its own ray tracing and
// layer refinement, these kernels (the secondary and solar pencils run as
// child batches of one scattering order less), then the radiative transfer
// with the scattering source at every scattering point.
#pragma once
#include "trace.cuh"

#define JSC_SP_REC 10     // doubles per scattering point record
#define JSC_NPHI_SCA 180  // azimuth steps of the source integral
#define JSC_NTH_SCA 180   // polar steps of the source integral
#define JSC_NALPHA_MAX 32 // secondary pencils per scattering point

// Scattering point record (doubles): x[3], dx[3], layer, time, pressure,
// temperature.
enum { SP_X = 0, SP_DX = 3, SP_IL = 6, SP_TIME = 7, SP_P = 8, SP_T = 9 };

// Orthonormal basis with ez along dz and ey in the plane of dy and dz
// (bascoord, src/scatter.c:6-52).
__device__ inline void jsc_bascoord(const double *dz, const double *dy, double *ex, double *ey,
                                    double *ez) {
  double dotp, norm = sqrt(dz[0] * dz[0] + dz[1] * dz[1] + dz[2] * dz[2]);
  for (int i = 0; i < 3; i++) ez[i] = dz[i] / norm;
  norm = sqrt(dy[0] * dy[0] + dy[1] * dy[1] + dy[2] * dy[2]);
  for (int i = 0; i < 3; i++) ey[i] = dy[i] / norm;
  dotp = ey[0] * ez[0] + ey[1] * ez[1] + ey[2] * ez[2];
  if (dotp == 1) {
    ey[0] = 1;
    ey[1] = 0;
    ey[2] = 0;
    dotp = ez[0];
    if (dotp == 1) {
      ey[0] = 0;
      ey[1] = 1;
      dotp = ez[1];
    }
  }
  for (int i = 0; i < 3; i++) ey[i] -= dotp * ez[i];
  norm = sqrt(ey[0] * ey[0] + ey[1] * ey[1] + ey[2] * ey[2]);
  for (int i = 0; i < 3; i++) ey[i] /= norm;
  ex[0] = ey[1] * ez[2] - ey[2] * ez[1];
  ex[1] = ey[2] * ez[0] - ey[0] * ez[2];
  ex[2] = ey[0] * ez[1] - ey[1] * ez[0];
}

// Angle between two vectors (the ANGLE macro, src/jurassic.h:33-34).
__device__ __forceinline__ double jsc_angle(const double *a, const double *b) {
  const double c = (a[0] * b[0] + a[1] * b[1] + a[2] * b[2]) /
                   sqrt(a[0] * a[0] + a[1] * a[1] + a[2] * a[2]) /
                   sqrt(b[0] * b[0] + b[1] * b[1] + b[2] * b[2]);
  return acos(fmin(fmax(c, -1.0), 1.0));
}

// Local frame at x: lz up, ly towards north (src/scatter.c:690-693).
__device__ __forceinline__ void local_frame(const double *x, double *lx, double *ly, double *lz) {
  double dnorth[3];
  dnorth[0] = -x[0];
  dnorth[1] = -x[1];
  dnorth[2] = 2 * JSC_RE - x[2];
  jsc_bascoord(x, dnorth, lx, ly, lz);
}

// --------------------------------------------------------- point list --

// Points of a chunk [first, first + n_pts) of a point list whose total
// count is on the device (n_total; null: all n_pts are real).  Fixed-
// capacity scattering runs launch every chunk up to the list's capacity;
// slots past the real count become null pencils (observer and view point
// far above the atmosphere: no LOS point, no work) and their sources are
// never read.
__device__ __forceinline__ int live_points(const int64_t *n_total, int64_t first, int n_pts) {
  if (!n_total) return n_pts;
  const int64_t left = *n_total - first;
  return left <= 0 ? 0 : (left < n_pts ? (int)left : n_pts);
}

#define JSC_NULL_Z 1.0e4  // altitude of a null pencil's observer and view point [km]

struct SpArgs {
  int n_rays, W;
  const int *nlos;
  const int64_t *los_off;
  const double *geo, *pts;
  const double *time;       // [n_rays]
  const int *ray_atm;
  int *nsp;                 // [n_rays] scattering points per ray
  const int64_t *sp_off;    // [n_rays+1]
  double *sp;               // [n_sp][JSC_SP_REC]
  int *sp_atm;              // [n_sp] profile of the point
  int *sp_idx;              // [LOS points] number of a point that scatters
  int64_t max_sp;           // capacity of sp (fixed-capacity runs; 0: unbounded)
  int *nlos_mut;            // rays whose points do not fit: their LOS is emptied
  unsigned *status;
  unsigned long long *n_listed;  // points actually listed (fixed-capacity runs)
};

// Points a fixed-capacity run lists: all of them, or up to the first ray
// whose points do not fit (sp_list_kernel lowers it with atomicMin).
static __global__ void sp_listed_init_kernel(const int64_t *sp_total, int64_t max_sp,
                                             unsigned long long *n_listed) {
  const int64_t t = *sp_total;
  *n_listed = (unsigned long long)(t < max_sp ? t : max_sp);
}

// A warp per ray, a lane per LOS point: with a thread per ray one chain of
// dependent loads and conversions ran along each line of sight (615 us, now
// 29, for 4000 limb rays through one layer).
static __global__ void __launch_bounds__(128) sp_count_kernel(SpArgs A) {
  const int r = (int)(blockIdx.x * 4 + (threadIdx.x >> 5)), lane = threadIdx.x & 31;
  if (r >= A.n_rays) return;
  const double *rec = A.pts + A.los_off[r] * A.W;
  int n = 0;
  for (int ip = lane; ip < A.nlos[r]; ip += 32)
    if (rec[(size_t)ip * A.W + REC_AF] > 0) n++;
  n = __reduce_add_sync(0xffffffffu, n);
  if (lane == 0) A.nsp[r] = n;
}

static __global__ void __launch_bounds__(128) sp_list_kernel(SpArgs A) {
  const int r = (int)(blockIdx.x * 4 + (threadIdx.x >> 5)), lane = threadIdx.x & 31;
  if (r >= A.n_rays) return;
  const int np = A.nlos[r];
  if (A.max_sp > 0 && A.sp_off[r + 1] > A.max_sp) {
    // more scattering points than the fixed capacity: the run reports the
    // overflow and this ray keeps no LOS point, so nothing reads past sp
    __syncwarp();  // every lane has read nlos
    if (lane == 0) {
      atomicOr(A.status, JSC_DEV_ERR_QUEUE);
      atomicMin(A.n_listed, (unsigned long long)A.sp_off[r]);
      A.nlos_mut[r] = 0;
    }
    return;
  }
  const double *rec = A.pts + A.los_off[r] * A.W;
  const double *geo = A.geo + A.los_off[r] * 4;
  int64_t k0 = A.sp_off[r];
  for (int i0 = 0; i0 < np; i0 += 32) {
    const int ip = i0 + lane;
    const double *rc = rec + (size_t)ip * A.W;
    const bool on = ip < np && rc[REC_AF] > 0;
    const unsigned mask = __ballot_sync(0xffffffffu, on);
    if (on) {
      const int64_t k = k0 + __popc(mask & ((1u << lane) - 1u));
      const int ip0 = ip > 0 ? ip - 1 : ip, ip1 = ip + 1 < np ? ip + 1 : ip;
      double x[3], x0[3], x1[3];
      jsc_geo2cart(geo[(size_t)ip * 4], geo[(size_t)ip * 4 + 1], geo[(size_t)ip * 4 + 2], x);
      jsc_geo2cart(geo[(size_t)ip0 * 4], geo[(size_t)ip0 * 4 + 1], geo[(size_t)ip0 * 4 + 2], x0);
      jsc_geo2cart(geo[(size_t)ip1 * 4], geo[(size_t)ip1 * 4 + 1], geo[(size_t)ip1 * 4 + 2], x1);
      double *o = A.sp + (size_t)k * JSC_SP_REC;
      for (int i = 0; i < 3; i++) {
        o[SP_X + i] = x[i];
        o[SP_DX + i] = x1[i] - x0[i];
      }
      o[SP_IL] = rc[REC_AI];
      o[SP_TIME] = A.time[r];
      o[SP_P] = rc[REC_P];
      o[SP_T] = rc[REC_T];
      A.sp_atm[k] = A.ray_atm[r];
      A.sp_idx[A.los_off[r] + ip] = (int)k;
    }
    k0 += __popc(mask);
  }
}

// ------------------------------------------------------- secondary rays --

struct SpawnArgs {
  int n_pts, nalpha;        // points of this chunk, pencils per point
  const int64_t *n_total;   // device count of the whole list (null: all real)
  int64_t first;            // index of the chunk's first point in the list
  const double *sp;         // first record of the chunk
  const int *sp_atm;
  double alpha[JSC_NALPHA_MAX];
  int *ray_atm;             // child batch inputs, n_pts * nalpha rays
  double *ray;              // [7][n_pts * nalpha]: time obsz obslon obslat vpz vplon vplat
};

// Secondary pencil ir of point k: from x towards the view point 10 km away
// at zenith angle alpha[ir] in the north-up plane (src/scatter.c:722-735).
static __global__ void sp_spawn_kernel(SpawnArgs A) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  const int n = A.n_pts * A.nalpha;
  if (t >= n) return;
  const int k = t / A.nalpha, ir = t - k * A.nalpha;
  if (k >= live_points(A.n_total, A.first, A.n_pts)) {  // null pencil
    A.ray_atm[t] = 0;
    for (int i = 0; i < 7; i++) A.ray[(size_t)i * n + t] = (i == 1 || i == 4) ? JSC_NULL_Z : 0.0;
    return;
  }
  const double *o = A.sp + (size_t)k * JSC_SP_REC;
  const double x[3] = {o[SP_X], o[SP_X + 1], o[SP_X + 2]};
  double lx[3], ly[3], lz[3], xv[3];
  local_frame(x, lx, ly, lz);
  const double al = A.alpha[ir];
  for (int i = 0; i < 3; i++) xv[i] = x[i] + 10. * cos(al) * (-1) * lz[i] + 10. * sin(al) * ly[i];
  double oz, olon, olat, vz, vlon, vlat;
  jsc_cart2geo(x, &oz, &olon, &olat);
  jsc_cart2geo(xv, &vz, &vlon, &vlat);
  A.ray_atm[t] = A.sp_atm[k];
  A.ray[t] = 0;  // the reference leaves the secondary observation time at 0
  A.ray[(size_t)n + t] = oz;
  A.ray[2 * (size_t)n + t] = olon;
  A.ray[3 * (size_t)n + t] = olat;
  A.ray[4 * (size_t)n + t] = vz;
  A.ray[5 * (size_t)n + t] = vlon;
  A.ray[6 * (size_t)n + t] = vlat;
}

// --------------------------------------------------------- source integral --

#define JSC_INT_THREADS 256    // sp_integral3_kernel
#define JSC_INT_CH 16          // channels per pass over the directions
#define JSC_INT1_THREADS 192   // sp_integral_kernel: a thread per polar step, 12 groups of 16 (20 of 8)
#define JSC_INT1_SL 29         // odd row stride of the interval sums (28 pencils, 27 intervals)
static_assert(JSC_INT1_THREADS >= JSC_NTH_SCA, "block shape");
static_assert(JSC_INT1_SL >= JSC_NALPHA_REF, "interval sums");

// Polar weights sin(theta2) phase(theta2) of layer blockIdx.y and channel
// blockIdx.x on the 180 polar steps (phase interpolated on its 1-degree
// grid), wt[nl][180][nd], and their sum over all directions, wsum[nl][nd]
// (src/scatter.c:760-800).
static __global__ void __launch_bounds__(JSC_INT1_THREADS)
sp_weights_kernel(int nd, const double *phase, double *wt, double *wsum) {
  __shared__ double sh[JSC_NTH_SCA];
  const int id = blockIdx.x, il = blockIdx.y, it = threadIdx.x;
  const double *ph = phase + ((size_t)il * nd + id) * NTHETA;
  if (it < JSC_NTH_SCA) {
    const double th = (0.5 + it) * M_PI / 180.;
    // locate(theta, NTHETA, theta2) on theta[i] = i * pi / 180
    int j = 0, hi = NTHETA - 1;
    while (hi > j + 1) {
      const int mid = (hi + j) >> 1;
      if ((double)mid * M_PI / 180. > th) hi = mid; else j = mid;
    }
    const double a0 = (double)j * M_PI / 180., a1 = (double)(j + 1) * M_PI / 180.;
    const double w = sin(th) * jsc_lin(a0, ph[j], a1, ph[j + 1], th);
    sh[it] = w;
    wt[((size_t)il * JSC_NTH_SCA + it) * nd + id] = w;
  }
  __syncthreads();
  if (it == 0) {
    double s = 0;
    for (int i = 0; i < JSC_NTH_SCA; i++) s += sh[i];
    wsum[(size_t)il * nd + id] = s * JSC_NPHI_SCA;
  }
}

struct IntegralArgs {
  int n_pts, nalpha, nd;
  const int64_t *n_total;   // device count of the whole list (null: all real)
  int64_t first;
  const double *sp;          // first record of the chunk
  double alpha[JSC_NALPHA_MAX];
  const double *rad;         // [n_pts * nalpha][nd] secondary radiances
  const double *wt, *wsum;   // polar weights (sp_weights_kernel)
  double *src;               // [n_pts][nd] of the chunk
};

// Source integral of one scattering point per block (src/scatter.c:737-805).
// The secondary radiance of a direction is linear in its angle alpha to the
// zenith between two pencils, and its weight depends on the polar step only.
// So the sum over the azimuth of a polar step needs, per pencil interval,
// the number of its directions and the sum of their alpha - alpha[lo]: a
// thread per polar step walks the azimuth once for all channels and keeps
// them (run sums in registers, added to shared memory when the interval
// changes).  The channels then take 180 x 27 of these sums each instead of
// 32,400 directions.  The zenith has no component across the plane of the
// zenith and the line of sight, so alpha is even in the azimuth and half of
// it suffices (all of it should the component exceed rounding).
// A direction and its opposite share one acos, which leaves 8100 a point.
// Bound by instruction issue at 24 warps an SM (four blocks of 56 KB shared
// memory; at three blocks, with an acos for every direction and passes of 16
// channels only, 1.52 and 11.2 ms in the two cases below).  Evaluating every
// channel in every direction took 9.0 ms for 11,600 points of 16 channels
// and 61.8 ms for a depth-2 batch of 12 rays and 8 channels, this form 1.03
// and 8.0.
#define JSC_INT1_SHMEM (JSC_NTH_SCA * JSC_INT1_SL * 9)

template <int CH>
__global__ void __launch_bounds__(JSC_INT1_THREADS, 4) sp_integral_kernel(IntegralArgs A) {
  extern __shared__ double ss[];  // [180][JSC_INT1_SL] sums of alpha - alpha[lo]
  unsigned char *sn =             // [180][JSC_INT1_SL] directions (at most 180)
      reinterpret_cast<unsigned char *>(ss + JSC_NTH_SCA * JSC_INT1_SL);
  // radiances and slopes of the pencils; before, the azimuths' cosines (with
  // an array of their own only three blocks fit an SM)
  __shared__ double rd[JSC_NALPHA_REF][CH], slp[JSC_NALPHA_REF][CH];
  static_assert(JSC_NALPHA_REF * CH >= JSC_NPHI_SCA, "azimuths");
  double *cph = &rd[0][0];
  __shared__ double alf[JSC_NALPHA_MAX];
  __shared__ double red[JSC_INT1_THREADS];
  const int k = blockIdx.x;
  if (k >= live_points(A.n_total, A.first, A.n_pts)) return;
  const int nd = A.nd, na = A.nalpha, tid = threadIdx.x;
  const double *o = A.sp + (size_t)k * JSC_SP_REC;
  const int il = (int)o[SP_IL];
  for (int i = tid; i < JSC_NPHI_SCA; i += JSC_INT1_THREADS)
    cph[i] = cos(2. * (0.5 + i) * M_PI / 180.);
  for (int i = tid; i < na; i += JSC_INT1_THREADS) alf[i] = A.alpha[i];
  for (int i = tid; i < JSC_NTH_SCA * JSC_INT1_SL; i += JSC_INT1_THREADS) {
    ss[i] = 0;
    sn[i] = 0;
  }
  // components of the downward zenith (-lz) along the axes of the scattering frame
  double ax, ay, az;
  {
    const double x[3] = {o[SP_X], o[SP_X + 1], o[SP_X + 2]};
    const double dx[3] = {o[SP_DX], o[SP_DX + 1], o[SP_DX + 2]};
    double lx[3], ly[3], lz[3], sx[3], sy[3], sz[3];
    local_frame(x, lx, ly, lz);
    jsc_bascoord(dx, x, sx, sy, sz);
    ax = -(lz[0] * sx[0] + lz[1] * sx[1] + lz[2] * sx[2]);
    ay = -(lz[0] * sy[0] + lz[1] * sy[1] + lz[2] * sy[2]);
    az = -(lz[0] * sz[0] + lz[1] * sz[1] + lz[2] * sz[2]);
  }
  const bool even = fabs(ax) <= 1e-14;
  __syncthreads();
  // Polar step of this thread; the lanes 2 j and 2 j + 1 hold steps that are
  // opposite, th and pi - th.
  const int pol = tid & 1 ? JSC_NTH_SCA - 1 - (tid >> 1) : tid >> 1;
  const double th = (0.5 + pol) * M_PI / 180.;
  const double st = sin(th), ct = cos(th);
  const double c1 = st * ay, c0 = ct * az, c2 = st * ax;
  const int row = pol * JSC_INT1_SL;
  // directions in the interval lo of the pencils, and the sum of their alpha
  struct Run {
    int lo, n;
    double s;
  };
  auto store = [&](const Run &r) {
    ss[row + r.lo] += r.s;
    sn[row + r.lo] += (unsigned char)r.n;
  };
  auto add = [&](Run &r, double al) {
    // locate(alpha, nalpha, alpha2) from the interval before
    int l = r.lo;
    while (l < na - 2 && !(alf[l + 1] > al)) l++;
    while (l > 0 && alf[l] > al) l--;
    if (l != r.lo) {
      store(r);
      r = Run{l, 0, 0};
    }
    r.s += al - alf[l];
    r.n++;
  };
  const bool own = tid < JSC_NTH_SCA;
  Run fwd = {0, 0, 0};
  // three azimuths at a time: their acos run in parallel and share constants
  static_assert(JSC_NPHI_SCA / 4 % 3 == 0 && JSC_NTH_SCA % 2 == 0, "azimuths");
  if (even) {
    // a direction's opposite lies in the other lane's polar step, at the
    // azimuth pi - phi, with pi - alpha: one acos for the two
    Run bwd = {0, 0, 0};
    for (int iq = 0; iq < JSC_NPHI_SCA / 4; iq += 3) {
      double al[3];
#pragma unroll
      for (int q = 0; q < 3; q++) al[q] = acos(fmin(fmax(c1 * cph[iq + q] + c0, -1.0), 1.0));
#pragma unroll
      for (int q = 0; q < 3; q++) {
        const double opp = M_PI - __shfl_xor_sync(0xffffffffu, al[q], 1);
        if (own) {
          add(fwd, al[q]);
          add(bwd, opp);
        }
      }
    }
    if (own) store(bwd);
  } else if (own) {
    for (int iq = 0; iq < JSC_NPHI_SCA; iq += 3) {
      double al[3];
#pragma unroll
      for (int q = 0; q < 3; q++)
        al[q] = c1 * cph[iq + q] + c0 + c2 * sin(2. * (0.5 + (iq + q)) * M_PI / 180.);
#pragma unroll
      for (int q = 0; q < 3; q++) al[q] = acos(fmin(fmax(al[q], -1.0), 1.0));
      for (int q = 0; q < 3; q++) add(fwd, al[q]);
    }
  }
  if (own) store(fwd);
  const int c = tid & (CH - 1), grp = tid / CH;
  constexpr int NG = CH == 8 ? 20 : 12, PER = JSC_NTH_SCA / NG;
  static_assert(PER * NG == JSC_NTH_SCA && NG * CH <= JSC_INT1_THREADS, "polar steps per group");
  for (int ch0 = 0; ch0 < nd; ch0 += CH) {
    __syncthreads();
    for (int i = tid; i < na * CH; i += JSC_INT1_THREADS) {
      const int lo = i / CH, cc = i - lo * CH;
      if (ch0 + cc < nd) {
        const double *r = A.rad + ((size_t)k * na + lo) * nd + ch0 + cc;
        rd[lo][cc] = r[0];
        if (lo + 1 < na) slp[lo][cc] = (r[nd] - r[0]) / (alf[lo + 1] - alf[lo]);
      }
    }
    __syncthreads();
    double acc = 0;
    const int id = ch0 + c;
    if (id < nd && grp < NG) {
      double v[PER];  // polar steps grp, grp + NG, ... of this channel
#pragma unroll
      for (int j = 0; j < PER; j++) v[j] = 0;
      for (int lo = 0; lo < na - 1; lo++) {
        const double r0 = rd[lo][c], s0 = slp[lo][c];
#pragma unroll
        for (int j = 0; j < PER; j++) {
          const int q = (grp + j * NG) * JSC_INT1_SL + lo;
          v[j] += (double)sn[q] * r0 + ss[q] * s0;
        }
      }
      const double *w = A.wt + ((size_t)il * JSC_NTH_SCA + grp) * nd + id;
#pragma unroll
      for (int j = 0; j < PER; j++) acc += w[(size_t)j * NG * nd] * v[j];
    }
    red[tid] = acc;
    __syncthreads();
    if (tid < CH && id < nd) {
      double t = 0;
      for (int g = 0; g < NG; g++) t += red[g * CH + c];
      A.src[(size_t)k * nd + id] = (even ? 2 * t : t) / A.wsum[(size_t)il * nd + id];
    }
  }
}

// Channels per pass: a pass of 8 takes 9 polar steps a thread, one of 16
// takes 15, so 8 where that is less in all (up to 8 channels, and 17 to 24).
static inline void sp_integral_launch(const IntegralArgs &ia, int blocks, cudaStream_t s) {
  if ((ia.nd + 7) / 8 * 9 < (ia.nd + 15) / 16 * 15)
    sp_integral_kernel<8><<<blocks, JSC_INT1_THREADS, JSC_INT1_SHMEM, s>>>(ia);
  else
    sp_integral_kernel<16><<<blocks, JSC_INT1_THREADS, JSC_INT1_SHMEM, s>>>(ia);
}

// ------------------------------------------------------------------ sun --

struct SunArgs {
  RayArgs ra;                // profiles, tracing switches, status word
  int n_pts;
  const int64_t *n_total;    // device count of the whole list (null: all real)
  int64_t first;
  const double *sp;          // first record of the chunk
  const int *sp_atm;
  // aerosol refinement edges (the last segment of each solar ray)
  int n_alti;
  double altimax, altimin;
  const double *alti;
  // outputs: the solar pencil of each point as a child-batch ray
  int *ray_atm;
  double *ray;               // [7][n_pts]
  double *theta2;            // [n_pts] scattering angle, or -1: no solar term
};

// Solar position (src/scatter.c:999-1041).
__device__ inline void jsc_suncoord(double sec, double lon, double lat, double *azi, double *sza) {
  const double D = sec / 86400 - 0.5;
  const double g = (357.529 + 0.98560028 * D) * M_PI / 180;
  const double q = 280.459 + 0.98564736 * D;
  const double L = (q + 1.915 * sin(g) + 0.020 * sin(2 * g)) * M_PI / 180;
  const double e = (23.439 - 0.00000036 * D) * M_PI / 180;
  const double dec = asin(sin(e) * sin(L));
  const double ra = atan2(cos(e) * sin(L), cos(L));
  const double GMST = 18.697374558 + 24.06570982441908 * D;
  const double LST = GMST + lon / 15;
  const double h = LST / 12 * M_PI - ra;
  lat *= M_PI / 180;
  *azi = atan2(-sin(h), cos(lat) * tan(dec) - sin(lat) * cos(h)) * 180 / M_PI;
  *sza = acos(sin(lat) * sin(dec) + cos(lat) * cos(dec) * cos(h)) * 180 / M_PI;
}

// The point before the last of the refined line of sight: the last layer
// edge inserted between the last two traced points (add_aerosol_layers,
// src/lineofsight.c:210-290, applied to the final segment), else the
// traced point before the last.
__device__ inline void refined_prev(const SunArgs &A, const double *g0, const double *g1,
                                    double *out) {
  const double zp = g0[0], zc = g1[0];
  out[0] = g0[0];
  out[1] = g0[1];
  out[2] = g0[2];
  if (!((zp < A.altimax || zc < A.altimax) && (zp > A.altimin || zc > A.altimin))) return;
  for (int il = 0; il < A.n_alti; il++) {
    const double z1 = A.alti[il], z2 = A.alti[A.n_alti - il - 1];
    double znew;
    if (zp > z1 && zc < z1) znew = z1;
    else if (zp < z2 && zc > z2) znew = z2;
    else continue;
    segment_point(g0, g1, znew, out);
  }
}

// Solar pencil of each scattering point: search the zenith angle whose
// refracted ray arrives from the sun's direction (up to 10 corrections),
// then, when that ray does not end on the ground, hand it to the solar
// child batch with the scattering angle to the LOS direction.  LANES (IP 1):
// lanes of the march per point, as in march_kernel.
template <int IP, int LANES>
__global__ void __launch_bounds__(128) sun_kernel(SunArgs A) {
  const int k = (blockIdx.x * blockDim.x + threadIdx.x) / LANES;
  const int role = LANES == 1 ? 0 : (int)(threadIdx.x & (LANES - 1));
  const unsigned gmask = LANES == 1 ? 0u : ((1u << LANES) - 1u) << ((threadIdx.x & 31) - role);
  if (k >= A.n_pts) return;  // whole groups leave together
  if (k >= live_points(A.n_total, A.first, A.n_pts)) {  // null solar pencil, no term
    const int n = A.n_pts;
    if (role) return;
    A.ray_atm[k] = 0;
    for (int i = 0; i < 7; i++) A.ray[(size_t)i * n + k] = (i == 1 || i == 4) ? JSC_NULL_Z : 0.0;
    A.theta2[k] = -1.0;
    return;
  }
  const double *o = A.sp + (size_t)k * JSC_SP_REC;
  const double x[3] = {o[SP_X], o[SP_X + 1], o[SP_X + 2]};
  const double dx[3] = {o[SP_DX], o[SP_DX + 1], o[SP_DX + 2]};
  const int ai = A.sp_atm[k];
  double lx[3], ly[3], lz[3], ek[3] = {0, 0, 0}, x1[3], azi, sza;
  local_frame(x, lx, ly, lz);
  RayIn in;
  jsc_cart2geo(x, &in.obsz, &in.obslon, &in.obslat);
  jsc_suncoord(o[SP_TIME], in.obslon, in.obslat, &azi, &sza);
  double sza_cor = sza;
  RayEnd end = {};
  end.tsurf = -999;
  for (int i2 = 0; i2 < 10; i2++) {
    for (int i = 0; i < 3; i++) {
      ek[i] = sin(sza_cor * M_PI / 180) * sin(azi * M_PI / 180) * lx[i] +
              sin(sza_cor * M_PI / 180) * cos(azi * M_PI / 180) * ly[i] +
              cos(sza_cor * M_PI / 180) * lz[i];
      x1[i] = x[i] + 10 * ek[i];
    }
    jsc_cart2geo(x1, &in.vpz, &in.vplon, &in.vplat);
    int np;
    if constexpr (IP == 1) {
      double ts;
      end.tsurf = -999;
      np = march_ray<LANES, true>(A.ra, MarchPool(), ai, 0, in, gmask, role, &end, &ts);
    } else {
      np = trace_core<2, IP>(A.ra, ai, 0, in, &end);
    }
    if (np < 2) break;
    double g0[3], xa[3], xb[3], dout[3];
    refined_prev(A, end.g[0], end.g[1], g0);
    jsc_geo2cart(g0[0], g0[1], g0[2], xa);
    jsc_geo2cart(end.g[1][0], end.g[1][1], end.g[1][2], xb);
    for (int i = 0; i < 3; i++) dout[i] = xb[i] - xa[i];
    const double sza_beam = jsc_angle(x, dout) * 180 / M_PI;
    if (fabs(sza_beam - sza) < 0.01) break;
    sza_cor -= 0.61803 * (sza_beam - sza);
    sza_cor = fmin(fmax(sza_cor, 0.0), 180.0);
  }
  if (role) return;
  const int n = A.n_pts;
  A.ray_atm[k] = ai;
  A.ray[k] = 0;
  A.ray[(size_t)n + k] = in.obsz;
  A.ray[2 * (size_t)n + k] = in.obslon;
  A.ray[3 * (size_t)n + k] = in.obslat;
  A.ray[4 * (size_t)n + k] = in.vpz;
  A.ray[5 * (size_t)n + k] = in.vplon;
  A.ray[6 * (size_t)n + k] = in.vplat;
  A.theta2[k] = end.tsurf < 0 ? jsc_angle(ek, dx) : -1.0;
}

struct SunAddArgs {
  int n_pts, nd;
  const double *sp;          // first record of the chunk
  const double *theta2;      // [n_pts]
  const double *tau;         // [n_pts][nd] transmittance of the solar pencils
  const double *phase;       // [nl][nd][NTHETA]
  const double *planck_sun;  // [nd] Planck radiance at the solar temperature
  double *src;               // [n_pts][nd] of the chunk
};

// src_sca += 6.764e-5 (solid angle of the sun) x phase x B(TSUN) x tau
// (src/scatter.c:980-990).
static __global__ void sun_add_kernel(SunAddArgs A) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= A.n_pts * A.nd) return;
  const int k = t / A.nd, id = t - k * A.nd;
  const double th2 = A.theta2[k];
  if (th2 < 0) return;
  const int il = (int)A.sp[(size_t)k * JSC_SP_REC + SP_IL];
  // locate(theta, NTHETA, theta2) on theta[i] = pi * i / (NTHETA - 1)
  int lo = 0, hi = NTHETA - 1;
  while (hi > lo + 1) {
    const int mid = (hi + lo) >> 1;
    if (M_PI * (double)mid / (NTHETA - 1) > th2) hi = mid; else lo = mid;
  }
  const double *ph = A.phase + ((size_t)il * A.nd + id) * NTHETA;
  const double phase2 = jsc_lin(M_PI * (double)lo / (NTHETA - 1), ph[lo],
                                M_PI * (double)(lo + 1) / (NTHETA - 1), ph[lo + 1], th2);
  A.src[t] += 6.764e-5 * phase2 * A.planck_sun[id] * A.tau[t];
}

// ------------------------------------------------- 3-D scattering source --
// srcfunc_sca_3d (src/scatter.c:811-895), used with horizontally varying
// atmospheres (IP 2/3): a secondary pencil in every direction of the
// 180 x 180 (polar, azimuth) grid around the line of sight, cast 10 km
// towards its view point, and the phase-function weighted sum of their
// radiances.

#define JSC_NDIR3 (JSC_NTH_SCA * JSC_NPHI_SCA)

struct Spawn3Args {
  int n_pts;
  const double *sp;          // first record of the chunk
  const int *sp_atm;
  int *ray_atm;              // child batch inputs, n_pts * JSC_NDIR3 rays
  double *ray;               // [7][n_pts * JSC_NDIR3]
};

static __global__ void sp_spawn3_kernel(Spawn3Args A) {
  const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const int64_t n = (int64_t)A.n_pts * JSC_NDIR3;
  if (t >= n) return;
  const int k = (int)(t / JSC_NDIR3), dir = (int)(t - (int64_t)k * JSC_NDIR3);
  const int it = dir / JSC_NPHI_SCA, iq = dir - it * JSC_NPHI_SCA;
  const double *o = A.sp + (size_t)k * JSC_SP_REC;
  const double x[3] = {o[SP_X], o[SP_X + 1], o[SP_X + 2]};
  const double dx[3] = {o[SP_DX], o[SP_DX + 1], o[SP_DX + 2]};
  double sx[3], sy[3], sz[3], xv[3];
  jsc_bascoord(dx, x, sx, sy, sz);
  const double theta2 = (0.5 + it) / JSC_NTH_SCA * M_PI;
  const double phi = (0.5 + iq) / JSC_NPHI_SCA * 2 * M_PI;
  for (int i = 0; i < 3; i++)
    xv[i] = x[i] + 10 * sin(theta2) * sin(phi) * sx[i] + 10 * sin(theta2) * cos(phi) * sy[i] +
            10 * cos(theta2) * sz[i];
  double oz, olon, olat, vz, vlon, vlat;
  jsc_cart2geo(x, &oz, &olon, &olat);
  jsc_cart2geo(xv, &vz, &vlon, &vlat);
  A.ray_atm[t] = A.sp_atm[k];
  A.ray[t] = 0;  // the secondary observation time stays 0, as in the reference
  A.ray[(size_t)n + t] = oz;
  A.ray[2 * (size_t)n + t] = olon;
  A.ray[3 * (size_t)n + t] = olat;
  A.ray[4 * (size_t)n + t] = vz;
  A.ray[5 * (size_t)n + t] = vlon;
  A.ray[6 * (size_t)n + t] = vlat;
}

struct Integral3Args {
  int n_pts, nd;
  const double *sp;          // first record of the chunk
  const double *rad;         // [n_pts * JSC_NDIR3][nd] secondary radiances
  const double *phase;       // [nl][nd][NTHETA]
  double *src;               // [n_pts][nd] of the chunk
};

// One block per scattering point, channels in passes of JSC_INT_CH: the
// weight pi/180 * 2 pi sin(theta2)/180 * phase(theta2) of each (polar
// angle, channel) in shared memory, directions spread over the threads.
// The reference divides every channel by one sum of the weights over all
// directions *and* channels (src/scatter.c:872-891); so does this.
static __global__ void __launch_bounds__(JSC_INT_THREADS) sp_integral3_kernel(Integral3Args A) {
  __shared__ double wt[JSC_NTH_SCA][JSC_INT_CH];
  __shared__ double red[JSC_INT_THREADS / 32][JSC_INT_CH + 1];
  __shared__ double total;
  const int k = blockIdx.x;
  if (k >= A.n_pts) return;
  const int nd = A.nd;
  const double *o = A.sp + (size_t)k * JSC_SP_REC;
  const int il = (int)o[SP_IL];
  const double *ph = A.phase + (size_t)il * nd * NTHETA;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if (threadIdx.x == 0) total = 0;
  for (int c0 = 0; c0 < nd; c0 += JSC_INT_CH) {
    __syncthreads();
    for (int i = threadIdx.x; i < JSC_NTH_SCA * JSC_INT_CH; i += blockDim.x) {
      const int it = i / JSC_INT_CH, c = i - it * JSC_INT_CH, id = c0 + c;
      double w = 0;
      if (id < nd) {
        const double theta2 = (0.5 + it) / JSC_NTH_SCA * M_PI;
        // locate(theta, NTHETA, theta2) on theta[i] = pi i / (NTHETA - 1)
        int j = 0, hi = NTHETA - 1;
        while (hi > j + 1) {
          const int mid = (hi + j) >> 1;
          if (M_PI * (double)mid / (NTHETA - 1) > theta2) hi = mid; else j = mid;
        }
        const double a0 = M_PI * (double)j / (NTHETA - 1), a1 = M_PI * (double)(j + 1) / (NTHETA - 1);
        const double phase2 = jsc_lin(a0, ph[(size_t)id * NTHETA + j], a1,
                                      ph[(size_t)id * NTHETA + j + 1], theta2);
        w = M_PI / JSC_NTH_SCA * 2 * M_PI * sin(theta2) / JSC_NPHI_SCA * phase2;
      }
      wt[it][c] = w;
    }
    __syncthreads();
    double acc[JSC_INT_CH], ws = 0;
#pragma unroll
    for (int c = 0; c < JSC_INT_CH; c++) acc[c] = 0;
    for (int dir = threadIdx.x; dir < JSC_NDIR3; dir += blockDim.x) {
      const int it = dir / JSC_NPHI_SCA;
      const double *r = A.rad + ((size_t)k * JSC_NDIR3 + dir) * nd + c0;
#pragma unroll
      for (int c = 0; c < JSC_INT_CH; c++)
        if (c0 + c < nd) {
          acc[c] += wt[it][c] * r[c];
          ws += wt[it][c];
        }
    }
#pragma unroll
    for (int c = 0; c <= JSC_INT_CH; c++) {
      double v = c < JSC_INT_CH ? acc[c] : ws;
      for (int off = 16; off > 0; off >>= 1) v += __shfl_down_sync(0xffffffffu, v, off);
      if (lane == 0) red[warp][c] = v;
    }
    __syncthreads();
    if (threadIdx.x <= JSC_INT_CH) {
      double v = 0;
      for (int w = 0; w < JSC_INT_THREADS / 32; w++) v += red[w][threadIdx.x];
      if (threadIdx.x == JSC_INT_CH) total += v;
      else if (c0 + (int)threadIdx.x < nd) A.src[(size_t)k * nd + c0 + threadIdx.x] = v;
    }
  }
  __syncthreads();
  for (int id = threadIdx.x; id < nd; id += blockDim.x) A.src[(size_t)k * nd + id] /= total;
}
