// The EGA, and the radiative transfer as passes of its own.
//
//   ega_gas_kernel     gas transmittance of every (LOS point, channel): a
//                      block takes a tile of ordered rays and a channel, a
//                      warp an emitter (src/forwardmodel.c:409-502)
//   segment_kernel     continua, Planck source, aerosol and scattering terms
//                      of every (LOS point, channel): the transmittance of
//                      the segment and its source
//   transfer_kernel    the recurrence along each ray (:302-399)
//
// Only an emitter's path transmittance ties one LOS point to the next; the
// radiance, whose exponentials depend on the segment only, leaves that chain.
#pragma once
#include "device_math.cuh"
#include "ega_lane.cuh"

struct GasArgs {
  EgaArgs e;
  double *tg;  // [points][nd] gas transmittance
};

// Node at byte offset o of the node array (gas variants run on tables below
// 4 GB: one 32-bit offset, and neighbours by immediate offsets).
__device__ __forceinline__ float2 node_at(const jsc_node *nodes, unsigned o) {
  return __ldg(reinterpret_cast<const float2 *>(reinterpret_cast<const char *>(nodes) + o));
}

// Interval of x (xf: x rounded down) in a row of strictly increasing keys
// that begins at byte offset row: the largest i <= last with key[i] <= x, or
// 0; the guess k and its nodes in, the interval and its nodes out.  A guess
// that is off moves by one or two intervals at a time towards x, from two
// loads on that side, at most three times (a new (p, T) bracket begins one to
// three intervals off); what is further is searched.  NaN compares false and
// so ends at last, as in the searches.
template <bool U>
__device__ __forceinline__ void fix_node(const jsc_node *__restrict__ nodes, unsigned row,
                                         int last, double x, float xf, int &k, float2 &a,
                                         float2 &b) {
#pragma unroll 1
  for (int it = 0;; it++) {
    const bool below = key2<U>(a) > xf && k > 0;
    const bool above = !(key2<U>(b) > xf) && k < last;
    if (!below && !above) break;
    if (it == 3) {
      k = find_interval<U>(nodes + row / 8u, last + 2, true, x, k);
      const unsigned o = row + 8u * (unsigned)k;
      a = node_at(nodes, o);
      b = node_at(nodes, o + 8);
      break;
    }
    const int s = below ? -1 : 1;
    const int i1 = below ? k - 1 : k + 2, i2 = below ? max(k - 2, 0) : min(k + 3, last + 1);
    const float2 n1 = node_at(nodes, row + 8u * (unsigned)i1);
    const float2 n2 = node_at(nodes, row + 8u * (unsigned)i2);
    const bool one = (key2<U>(n1) > xf) != below || k + s == (below ? 0 : last);
    const float2 near = one ? n1 : n2, far = one ? (below ? a : b) : n1;
    k += one ? s : 2 * s;
    a = below ? near : far;
    b = below ? far : near;
  }
}

// Emissivity of the extended path at one (p, T) node, as ega_node (the same
// operations and intervals), on a table of strictly increasing rows.  k: the
// guess of the inverse interval and a, b its nodes.  The forward interval is
// guessed from log2 of the extended column where the table's columns are
// evenly spaced in it (il > 0), else from the distance dj to the inverse
// interval.
__device__ __forceinline__ double gas_node(const jsc_node *__restrict__ nodes, jsc_row rd,
                                           float l0, float il, double x1, float x1f, double useg,
                                           int k, int dj, float2 a, float2 b, int *kout,
                                           int *jout) {
  const int last = (rd.nf & 0xffff) - 2;
  const unsigned row = 8u * (unsigned)rd.off;
  fix_node<false>(nodes, row, last, x1, x1f, k, a, b);
  const double x2 = lin_node(a.y, a.x, float_slope(a.x, a.y, b.x, b.y), x1) + useg;
  const float x2f = __double2float_rd(x2);
  int j = il > 0 ? __float2int_rd((__log2f(x2f) - l0) * il) : k + dj;
  j = min(max(j, 0), last);
  const unsigned o = row + 8u * (unsigned)j;
  a = node_at(nodes, o);
  b = node_at(nodes, o + 8);
  fix_node<true>(nodes, row, last, x2, x2f, j, a, b);
  *kout = k;
  *jout = j;
  return jsc_clamp01(lin_node(a.x, a.y, float_slope(a.y, a.x, b.y, b.x), x2));
}

// The same on any table.
static __device__ __noinline__ double node_general(const jsc_node *nodes, jsc_row rd, double x1,
                                                   double useg, int hint, int dj, int *kout,
                                                   int *jout) {
  unsigned long long none = 0;
  return ega_node<false>(nodes, rd, x1, useg, hint, dj, kout, jout, &none);
}

// Shared memory of a block with nw emitter warps on tiles of `rays` rays and
// pb points between barriers.
static inline size_t gas_shmem(int nw, int rays, int pb) {
  return sizeof(double) * 2 * pb * nw * rays;
}

// What a block keeps of its tile of R rays besides the factors.
template <int R>
struct GasTile {
  int64_t off[R];
  int np[R];
};

// Gas transmittance of the n points that end at LOS point ip: the product of
// the emitters' factors in emitter order, a warp per point.
template <int R>
__device__ __forceinline__ void gas_product(const GasArgs &A, const GasTile<R> &tile,
                                            const double *buf, int nw, int w, int lane, int d,
                                            int ip, int n) {
  for (int q = w * (32 / R) + lane / R; q < n; q += nw * (32 / R)) {
    const int ii = lane & (R - 1), pt = ip - n + 1 + q;
    if (pt < tile.np[ii]) {
      const double *fp = buf + (size_t)q * nw * R + ii;
      double t = fp[0];
      for (int g = 1; g < A.e.m.ng; g++) t *= fp[g * R];
      A.tg[(size_t)(tile.off[ii] + pt) * A.e.m.nd + d] = t;
    }
  }
}

// Evaluation count and, with DIG, the per-channel digest: the fold of the
// per-emitter digests in emitter order.  One lane per ray and emitter calls
// with own = true.
template <int R, bool DIG>
__device__ __forceinline__ void gas_finish(const GasArgs &A, double *sf, int w, int lane, int i,
                                           int r, int d, bool own, unsigned n_ega,
                                           unsigned long long dig) {
  const unsigned tot = __reduce_add_sync(0xffffffffu, own ? n_ega : 0u);
  if (lane == 0 && tot) atomicAdd(&A.e.counters[1], (unsigned long long)tot);
  if (DIG) {
    unsigned long long *sd = reinterpret_cast<unsigned long long *>(sf);
    __syncthreads();
    if (own) sd[w * R + i] = dig;
    __syncthreads();
    if (w == 0 && own && r >= 0) {
      unsigned long long dd = 0;
      for (int g = 0; g < A.e.m.ng; g++) dd = dd * 1000003ull + sd[g * R + i];
      A.e.digest[(size_t)r * A.e.m.nd + d] = dd;
    }
  }
}

// A lane per ray and emitter: a block takes a tile of 32 rays and a channel,
// a warp an emitter.  Every PB points the emitters' factors, in shared
// memory, are multiplied; in between the emitters do not wait for one
// another.  Bound by instruction issue and the gathers' latency together
// (61 % issue).  Against the ray-tile kernel (variant 17), with its barrier
// and transfer step at every point, guesses of each corner by itself,
// branches for every neighbour and divisions by the grids' widths: 65.5 ms
// for 84.9 ms on 20,000 rays x 64 channels x 8 emitters.
template <bool DIG, int PB, int MAXT, int MINB>
__global__ void __launch_bounds__(MAXT, MINB) ega_gas_kernel(const __grid_constant__ GasArgs A) {
  constexpr int R = 32;
  extern __shared__ double sf[];  // [2][PB][nw][R] transmittance factors
  __shared__ GasTile<R> tl;
  const jsc_dev_model &m = A.e.m;
  const int nd = m.nd, ng = m.ng, nw = blockDim.x >> 5;
  const int tile = (int)(blockIdx.x / (unsigned)nd), d = (int)(blockIdx.x - (unsigned)tile * nd);
  const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int slot = tile * R + lane;
  const int r = slot < A.e.n_rays ? A.e.order[slot] : -1;
  const int np = r >= 0 ? A.e.nlos[r] : 0;
  const int npmax = __reduce_max_sync(0xffffffffu, np);  // the same in every warp
  const int64_t off = r >= 0 ? A.e.los_off[r] : 0;
  if (w == 0) {
    tl.off[lane] = off;
    tl.np[lane] = np;
  }
  __syncthreads();
  const EgaTable tb = ega_table(m, d, w);
  const double2 *__restrict__ dt = reinterpret_cast<const double2 *>(m.grid_dt) + (tb.gt - m.grid_t);
  const double2 *__restrict__ dp = reinterpret_cast<const double2 *>(m.grid_dp) + (tb.gp - m.grid_p);
  const jsc_tab_info ti = tb.ok ? m.tab_info[d * ng + w] : jsc_tab_info{0.f, 0.f, 0.f, 0.f};
  const bool strict = ti.strict != 0.f;  // the same in the whole warp
  const int W = A.e.W;
  const double *__restrict__ rec = A.e.pts + off * W;
  double tp = 1;
  // Interval guesses: the last forward interval of each corner, moved by the
  // step to the inverse interval that the first corner takes (its own last
  // step for the first corner): right or one off in 98 % of the lookups,
  // beyond two in 0.1 %.  dj: distance of the forward from the inverse
  // interval of the first corner.
  int k[4] = {0, 0, 0, 0}, dj = 0, sh = 0, hcode = -1;
  unsigned long long dig = 0;
  unsigned n_ega = 0;
  for (int ip = 0; ip < npmax; ip++, rec += W) {
    double f = 1;
    if (ip < np) {
      double eps = 0;
      if (tb.ok) {
        if (tp < 1e-9) {
          eps = 1;
        } else {
          const double P = rec[REC_P], T = rec[REC_T], useg = rec[REC_K + m.nw + w];
          const int code = A.e.single_grid
                               ? (int)rec[REC_GRID]
                               : grid_code(m.grid_np[tb.gid], tb.gp,
                                           m.grid_nt + (size_t)tb.gid * TBLNPMAX, tb.gt, P, T);
          if (code & (1 << 16)) {
            const int ipr = (code >> 10) & 63, it0 = (code >> 5) & 31, it1 = code & 31;
            const int g0 = ipr * TBLNTMAX + it0, g1 = (ipr + 1) * TBLNTMAX + it1;
            jsc_row r4[4];
            r4[0] = tb.rows_dg[(size_t)g0 * tb.rs];
            r4[1] = tb.rows_dg[(size_t)(g0 + 1) * tb.rs];
            r4[2] = tb.rows_dg[(size_t)g1 * tb.rs];
            r4[3] = tb.rows_dg[(size_t)(g1 + 1) * tb.rs];
            if ((r4[0].nf & 0xffff) >= 2 && (r4[1].nf & 0xffff) >= 2 &&
                (r4[2].nf & 0xffff) >= 2 && (r4[3].nf & 0xffff) >= 2) {
              const double x1 = 1 - tp;
              const float x1f = __double2float_rd(x1);
              if (hcode >= 0 && hcode != code) {
                // hints of the new corners, as remap_hints
                const int pi = (hcode >> 10) & 63, p0 = (hcode >> 5) & 31, p1 = hcode & 31;
                int kn[4];
#pragma unroll
                for (int q = 0; q < 4; q++) {
                  const int t = (q >> 1 ? it1 : it0) + (q & 1);
                  kn[q] = ipr + (q >> 1) <= pi ? (t <= p0 ? k[0] : k[1]) : (t <= p1 ? k[2] : k[3]);
                }
#pragma unroll
                for (int q = 0; q < 4; q++) k[q] = kn[q];
              }
              hcode = code;
              if (DIG) dig = dig * 1000003ull + (unsigned long long)(ipr * 961 + it0 * 31 + it1);
              double e[4];
#pragma unroll
              for (int q = 0; q < 4; q++) {
                int kk, jj;
                if (strict) {
                  const int h = min(max(k[q] + sh, 0), (r4[q].nf & 0xffff) - 2);
                  const unsigned o = 8u * (unsigned)(r4[q].off + h);
                  e[q] = gas_node(m.nodes, r4[q], ti.l0, ti.il, x1, x1f, useg, h, dj,
                                  node_at(m.nodes, o), node_at(m.nodes, o + 8), &kk, &jj);
                } else {
                  e[q] = node_general(m.nodes, r4[q], x1, useg, k[q] + sh, dj, &kk, &jj);
                }
                if (DIG)
                  dig = (dig * 1000003ull + (unsigned long long)kk) * 1000003ull +
                        (unsigned long long)jj;
                if (q == 0) {
                  sh = kk - k[0];
                  dj = jj - kk;
                }
                k[q] = jj;
              }
              const double e0 = jsc_clamp01(lin_known(tb.gt[g0], e[0], e[1], T, __ldg(dt + g0)));
              const double e1 = jsc_clamp01(lin_known(tb.gt[g1], e[2], e[3], T, __ldg(dt + g1)));
              const double ea = jsc_clamp01(lin_known(tb.gp[ipr], e0, e1, P, __ldg(dp + ipr)));
              eps = 1 - (1 - ea) / tp;
              n_ega++;
            }
          }
        }
      }
      tp = tp * (1 - eps);
      f = 1 - eps;
    }
    const int b = ip & (PB - 1);
    double *buf = sf + (size_t)((ip / PB) & 1) * PB * nw * R;
    buf[(b * nw + w) * R + lane] = f;
    if (b == PB - 1 || ip == npmax - 1) {
      // the other buffer is filled next; this one again after the barrier
      // that follows these reads
      __syncthreads();
      gas_product<R>(A, tl, buf, nw, w, lane, d, ip, b + 1);
    }
  }
  gas_finish<R, DIG>(A, sf, w, lane, lane, r, d, true, n_ega, dig);
}

// A lane per table corner, four to a ray and emitter, tiles of 8 rays: for
// launches whose LOS chains leave the SMs idle.  A point is two lookups on
// the chain instead of eight; the interpolations and the division are done
// four times over.  The warp stays together: what a lane has not to do it
// leaves out by predicate, and every exchange between corners is a shuffle of
// the whole warp.  The next point's state, and its row, are loaded ahead of
// the chain.  Bound by the latency of the chain, 0.42 ms for 61 limb rays of
// about 290 points with 4 channels and 2 emitters (0.95 ms with a lane per
// ray, 1.09 ms for the ray-tile kernel); at many rays it takes 1.7 times the
// instructions of a lane per ray.
template <bool DIG, int PB, int MAXT, int MINB>
__global__ void __launch_bounds__(MAXT, MINB) ega_gas4_kernel(const __grid_constant__ GasArgs A) {
  constexpr int R = 8;
  constexpr unsigned full = 0xffffffffu;
  extern __shared__ double sf[];  // [2][PB][nw][R] transmittance factors
  __shared__ GasTile<R> tl;
  const jsc_dev_model &m = A.e.m;
  const int nd = m.nd, ng = m.ng, nw = blockDim.x >> 5;
  const int tile = (int)(blockIdx.x / (unsigned)nd), d = (int)(blockIdx.x - (unsigned)tile * nd);
  const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int i = lane >> 2, c = lane & 3, up = c >> 1;
  const int slot = tile * R + i;
  const int r = slot < A.e.n_rays ? A.e.order[slot] : -1;
  const int np = r >= 0 ? A.e.nlos[r] : 0;
  const int npmax = __reduce_max_sync(full, np);  // the same in every warp
  const int64_t off = r >= 0 ? A.e.los_off[r] : 0;
  if (w == 0 && c == 0) {
    tl.off[i] = off;
    tl.np[i] = np;
  }
  __syncthreads();
  const EgaTable tb = ega_table(m, d, w);  // of the whole warp
  const double2 *__restrict__ dt = reinterpret_cast<const double2 *>(m.grid_dt) + (tb.gt - m.grid_t);
  const double2 *__restrict__ dp = reinterpret_cast<const double2 *>(m.grid_dp) + (tb.gp - m.grid_p);
  const jsc_tab_info ti = tb.ok ? m.tab_info[d * ng + w] : jsc_tab_info{0.f, 0.f, 0.f, 0.f};
  const bool strict = ti.strict != 0.f;
  const int W = A.e.W;
  const double *__restrict__ rec = A.e.pts + off * W;
  double tp = 1;
  // Current point: state, bracket code, this corner's row; k: the last
  // forward interval, which belongs to the corner of bracket kcode, sh: the
  // last step from there to the inverse interval, dj: from that to the next
  // forward interval.
  double P = 0, T = 0, useg = 0;
  int code = 0, kcode = -1, k = 0, sh = 0, dj = 0;
  jsc_row rd = {0, 0};
  unsigned long long dig = 0;
  unsigned n_ega = 0;
  const int live = tb.ok ? np : 0;  // points this lane evaluates
  auto load_state = [&](double &p, double &t, double &u, double &g) {
    p = rec[REC_P];
    t = rec[REC_T];
    u = rec[REC_K + m.nw + w];
    g = rec[REC_GRID];
  };
  auto bracket = [&](double g, double p, double t) {
    return A.e.single_grid ? (int)g
                           : grid_code(m.grid_np[tb.gid], tb.gp,
                                       m.grid_nt + (size_t)tb.gid * TBLNPMAX, tb.gt, p, t);
  };
  auto row_of = [&](int cd) {
    const int tlow = up ? cd & 31 : (cd >> 5) & 31;
    return tb.rows_dg[(size_t)((((cd >> 10) & 63) + up) * TBLNTMAX + tlow + (c & 1)) * tb.rs];
  };
  if (live > 0) {
    double g;
    load_state(P, T, useg, g);
    code = bracket(g, P, T);
    if (code & (1 << 16)) rd = row_of(code);
  }
  for (int ip = 0; ip < npmax; ip++) {
    const bool more = ip + 1 < live;
    double P2 = 0, T2 = 0, u2 = 0, g2 = 0;
    if (more) {
      rec += W;
      load_state(P2, T2, u2, g2);
    }
    // all four corners of the ray have a row?
    const bool two = (code & (1 << 16)) && (rd.nf & 0xffff) >= 2;
    const unsigned vote = __ballot_sync(full, two);
    const bool dark = tp < 1e-9;
    const bool ev = ip < live && !dark && ((vote >> (lane & ~3)) & 15u) == 15u;
    // Interval guess of a corner: that of the corner at the same pressure
    // level (else the nearest) and the nearest temperature (remap_hints).
    const int ipr = (code >> 10) & 63, tlow = up ? code & 31 : (code >> 5) & 31;
    int src = c;
    if (code != kcode) {
      const int t = tlow + (c & 1);
      src = ipr + up <= ((kcode >> 10) & 63) ? (t <= ((kcode >> 5) & 31) ? 0 : 1)
                                             : (t <= (kcode & 31) ? 2 : 3);
    }
    const int kh = __shfl_sync(full, k, (lane & ~3) | src);
    int kk = 0, jj = 0;
    double e = 0;
    if (ev) {
      const double x1 = 1 - tp;
      if (strict) {
        const int h = min(max(kh + sh, 0), (rd.nf & 0xffff) - 2);
        const unsigned o = 8u * (unsigned)(rd.off + h);
        e = gas_node(m.nodes, rd, ti.l0, ti.il, x1, __double2float_rd(x1), useg, h, dj,
                     node_at(m.nodes, o), node_at(m.nodes, o + 8), &kk, &jj);
      } else {
        e = node_general(m.nodes, rd, x1, useg, kh + sh, dj, &kk, &jj);
      }
      sh = kk - kh;
      dj = jj - kk;
      k = jj;
      kcode = code;
      n_ega++;
    }
    const int code2 = more ? bracket(g2, P2, T2) : 0;
    if (code2 & (1 << 16)) rd = row_of(code2);
    if (DIG) {
      if (ev) dig = dig * 1000003ull + (unsigned long long)(ipr * 961 + ((code >> 5) & 31) * 31 + (code & 31));
      for (int q = 0; q < 4; q++) {
        const unsigned long long kq = (unsigned long long)__shfl_sync(full, kk, (lane & ~3) | q);
        const unsigned long long jq = (unsigned long long)__shfl_sync(full, jj, (lane & ~3) | q);
        if (ev) dig = (dig * 1000003ull + kq) * 1000003ull + jq;
      }
    }
    const int gi = ev ? (ipr + up) * TBLNTMAX + tlow : 0, gq = ev ? ipr : 0;
    const double eo = __shfl_xor_sync(full, e, 1);
    const double et =
        jsc_clamp01(lin_known(tb.gt[gi], c & 1 ? eo : e, c & 1 ? e : eo, T, __ldg(dt + gi)));
    const double ep = __shfl_xor_sync(full, et, 2);
    const double ea =
        jsc_clamp01(lin_known(tb.gp[gq], up ? ep : et, up ? et : ep, P, __ldg(dp + gq)));
    double eps = ip < live && dark ? 1.0 : 0.0;
    if (ev) eps = 1 - (1 - ea) / tp;
    if (ip < np) tp = tp * (1 - eps);
    const double f = 1 - eps;
    P = P2;
    T = T2;
    useg = u2;
    code = code2;
    const int s = ip & (PB - 1);
    double *buf = sf + (size_t)((ip / PB) & 1) * PB * nw * R;
    if (c == 0) buf[(s * nw + w) * R + i] = f;
    if (s == PB - 1 || ip == npmax - 1) {
      __syncthreads();
      gas_product<R>(A, tl, buf, nw, w, lane, d, ip, s + 1);
    }
  }
  gas_finish<R, DIG>(A, sf, w, lane, i, r, d, c == 0, n_ega, dig);
}

struct SegmentArgs {
  jsc_dev_model m;
  jsc_run_cfg cfg;
  int64_t n_points;
  const int64_t *n_live;  // LOS points on the device (fixed-capacity runs), or null
  int W;
  const double *pts;
  double *x, *src;        // [n_points][nd]; x holds the gas transmittance
  const double *beta;     // aerosol beta_e/beta_s/beta_a [3][nl][nd]
  int aero_nl;
  const double *src_sca;  // scattering sources [n_sp][nd], or null
  const int *sp_idx;      // scattering point of a LOS point
  int64_t n_sp;
  int step;               // points per block and step, at most JSC_SEG_POINTS
};

// What the channels of a LOS point share of jsc_continuum and of the segment
// terms: the subexpressions in the order of that function.
struct SegPoint {
  double T, DS, rDS, P, pp;    // rDS: 1 / DS, or 0 where dividing by it needs more
  double co2, d1, d2, d3;      // u / N_A / 1000 * P / P0; the three T polynomials
  double u_h2o, q, h2o_y, h2o_v, h2o_a2;
  double dtp, af;              // T above its Planck node; layer factor
  int plk, ia, sp;             // Planck node, layer, scattering point
};

#define JSC_SEG_POINTS 128
#define JSC_SEG_THREADS 256

// ctm / DS (div_known within its range).
__device__ __forceinline__ double per_length(double ctm, const SegPoint &p) {
  return p.rDS != 0 && (ctm == 0 || fabs(ctm) > 1e-250) ? div_known(ctm, p.DS, p.rDS) : ctm / p.DS;
}

// jsc_continuum of channel coefficients c at point p.
__device__ __forceinline__ double segment_continuum(const jsc_dev_model &m, const jsc_run_cfg &cfg,
                                                    const jsc_ctm_coef *__restrict__ c, double nu,
                                                    double kwin, const SegPoint &p) {
  double beta = kwin;
  if (cfg.ctm_co2) {
    double ctm = 0;
    if (m.ig_co2 >= 0 && c->co2_on)
      ctm = p.co2 * (p.d1 * c->co2_c230 - p.d2 * c->co2_c260 + p.d3 * c->co2_c296);
    beta += per_length(ctm, p);
  }
  if (cfg.ctm_h2o) {
    double ctm = 0;
    if (m.ig_h2o >= 0 && c->h2o_on) {
      const double ctwslf = c->h2o_self296 * pow(c->h2o_ratio, p.h2o_y);
      const double a1 = nu * p.u_h2o * tanh(p.h2o_v * nu);
      const double a3 = p.pp * (p.q * ctwslf + (1 - p.q) * c->h2o_frn) * 1e-20;
      ctm = a1 * p.h2o_a2 * a3;
    }
    beta += per_length(ctm, p);
  }
  if (cfg.ctm_n2 && c->n2_on) {
    const double t0 = 273, tr = 296, q_n2 = 0.79, tt = t0 / p.T;
    beta += 0.1 * (p.pp * p.pp) * (tt * tt) * q_n2 * c->n2_b *
            exp(c->n2_beta * (1 / tr - 1 / p.T)) *
            (q_n2 + (1 - q_n2) * (1.294 - 0.4545 * p.T / tr));
  }
  if (cfg.ctm_o2 && c->o2_on) {
    const double t0 = 273, tr = 296, q_o2 = 0.21, tt = t0 / p.T;
    beta += 0.1 * (p.pp * p.pp) * (tt * tt) * q_o2 * c->o2_b *
            exp(c->o2_beta * (1 / tr - 1 / p.T));
  }
  return beta;
}

// Transmittance x and source of a segment: x = the gas transmittance times
// the continuum (and aerosol) attenuation, or, at a scattering point
// (src/forwardmodel.c:317-363), minus the attenuation by bext, whose
// radiance is accumulated in another order; the sign tells them apart.
// Gas transmittance 0 leaves the radiance alone: x = 1, source 0.
// A block takes 64 or 128 points at a time: what their channels share (nine
// divisions) is computed once per point into shared memory, then threads
// take (point, channel) pairs.  Bound by instruction issue (pow, tanh and exp
// in FP64): 5.3 ms for 20,000 rays x 64 channels, 7.0 ms with the shared part
// in every pair.
static __global__ void __launch_bounds__(JSC_SEG_THREADS)
segment_kernel(const __grid_constant__ SegmentArgs A) {
  __shared__ SegPoint sp[JSC_SEG_POINTS];
  const int nd = A.m.nd;
  int64_t pts = A.n_points;
  if (A.n_live && *A.n_live < pts) pts = *A.n_live;
  for (int64_t p0 = (int64_t)blockIdx.x * A.step; p0 < pts; p0 += (int64_t)gridDim.x * A.step) {
    const int n = (int)(pts - p0 < A.step ? pts - p0 : A.step);
    __syncthreads();  // the pairs of the step before
    if ((int)threadIdx.x < n) {
      const double *rec = A.pts + (p0 + threadIdx.x) * A.W, *u = rec + REC_K + A.m.nw;
      const double P = rec[REC_P], T = rec[REC_T], DS = rec[REC_DS];
      SegPoint p;
      p.T = T;
      p.DS = DS;
      p.rDS = DS > 1e-50 && DS < 1e50 ? 1 / DS : 0.0;
      p.P = P;
      p.pp = P / JSC_P0;
      const double u_co2 = A.m.ig_co2 >= 0 ? u[A.m.ig_co2] : 0.0;
      p.co2 = u_co2 / JSC_AVOGADRO / 1000 * P / JSC_P0;
      const double dt230 = T - 230, dt260 = T - 260, dt296 = T - 296;
      p.d1 = dt260 * 5.050505e-4 * dt296;
      p.d2 = dt230 * 9.259259e-4 * dt296;
      p.d3 = dt230 * 4.208754e-4 * dt260;
      p.u_h2o = A.m.ig_h2o >= 0 ? u[A.m.ig_h2o] : 0.0;
      p.q = rec[REC_QH2O];
      p.h2o_y = (296 - T) / (296 - 260);
      p.h2o_v = .7193876 / T;
      p.h2o_a2 = 296 / T;
      p.plk = (int)rec[REC_PLK];
      p.dtp = T - planck_temp(p.plk);
      p.af = rec[REC_AF];
      p.ia = (int)rec[REC_AI];
      p.sp = A.src_sca && p.af > 0 ? A.sp_idx[p0 + threadIdx.x] : -1;
      sp[threadIdx.x] = p;
    }
    __syncthreads();
    for (int i = threadIdx.x; i < n * nd; i += JSC_SEG_THREADS) {
      const int k = i / nd, d = i - k * nd;
      const SegPoint &p = sp[k];
      const int64_t t = p0 * nd + i;
      const double tau_gas = A.x[t];
      double x = 1, s = 0;
      if (tau_gas > 0) {
        const int w = A.m.window[d];
        const double kwin = w < A.m.nw ? A.pts[(p0 + k) * A.W + REC_K + w] : 0.0;
        const double beta = segment_continuum(A.m, A.cfg, A.m.ctm + d, A.m.nu[d], kwin, p);
        const size_t o = (size_t)d * JSC_NPLANCK + p.plk;
        s = A.m.planck_b[o] + A.m.planck_s[o] * p.dtp;
        if (A.src_sca && p.af > 0) {
          const double ss =
              p.sp >= 0 && p.sp < A.n_sp ? A.src_sca[(size_t)p.sp * nd + d] : 0.0;
          const double be = A.beta[p.ia * nd + d], bs = A.beta[A.aero_nl * nd + p.ia * nd + d];
          const double bext = (-1.) * log(tau_gas) / p.DS + beta + p.af * be;
          x = -exp(-1 * bext * p.DS);
          s = ((bext - p.af * bs) * s + p.af * bs * ss) / bext;
        } else {
          double b = beta;
          if (A.cfg.sca_n != 0 && p.af != 0)
            b = beta + p.af * A.beta[(A.cfg.sca_ext_beta_a ? 2 : 0) * A.aero_nl * nd + p.ia * nd + d];
          x = tau_gas * exp(-1. * b * p.DS);
        }
      }
      A.x[t] = x;
      A.src[t] = s;
    }
  }
}

// Radiance and transmittance of each (ray, channel), a thread each, the
// channels of a ray side by side; the loads of several points are in flight
// at a time.
static __global__ void __launch_bounds__(128) transfer_kernel(EgaArgs A, const double *x,
                                                              const double *src) {
  const int nd = A.m.nd;
  const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= (int64_t)A.n_rays * nd) return;
  const int r = (int)(t / nd), d = (int)(t - (int64_t)r * nd);
  const int np = A.nlos[r];
  x += A.los_off[r] * nd + d;
  src += A.los_off[r] * nd + d;
  double rad = 0, tau = 1;
  constexpr int U = 8;
  for (int i0 = 0; i0 < np; i0 += U) {
    double xs[U], ss[U];
#pragma unroll
    for (int u = 0; u < U; u++) {
      const int i = i0 + u < np ? i0 + u : np - 1;
      xs[u] = x[(size_t)i * nd];
      ss[u] = src[(size_t)i * nd];
    }
#pragma unroll
    for (int u = 0; u < U; u++)
      if (i0 + u < np) {
        if (signbit(xs[u])) {  // scattering point
          const double v = -xs[u], e = 1 - v;
          rad += tau * e * ss[u];
          tau *= v;
        } else {
          const double e = 1 - xs[u];
          rad += ss[u] * e * tau;
          tau *= (1 - e);
        }
      }
  }
  const double ts = A.tsurf[r];
  if (ts > 0) rad += planck_src(A.m, d, planck_index(ts), ts) * tau;
  A.rad[t] = rad;
  A.tau[t] = tau;
}

// lanes: 1 or 4 a ray
void jsc_ega_gas_launch(const GasArgs &ga, int lanes, cudaStream_t s);
void jsc_segment_launch(SegmentArgs sa, cudaStream_t s);
void jsc_transfer_launch(const EgaArgs &ea, const double *x, const double *src, cudaStream_t s);
