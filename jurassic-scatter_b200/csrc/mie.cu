// Mie scattering of homogeneous spheres on the GPU, for the aerosol/cloud
// optical properties of get_opt_prop (src/scatter.c:330-512).
//
// The series is the Bohren-Huffman one (C. F. Bohren and D. R. Huffman,
// "Absorption and Scattering of Light by Small Particles", 1983, appendix
// A), which the reference evaluates in bhmie (src/scatter.c:56-234):
// logarithmic derivative D_n(mx) by downward recurrence from D_nmx = 0,
// Riccati-Bessel functions psi_n(x), chi_n(x) by upward recurrence, the
// coefficients a_n, b_n, and the amplitudes S1, S2 at (NTHETA+1)/2 angles
// in [0, 90] degrees plus their mirror images in (90, 180], with
// nstop = x + 4 x^0.3333 + 2 terms and nmx = max(nstop, |mx|) + 15.
//
// mie_kernel: a block per task (a size parameter and a refractive index;
// opt_prop_mie_log has one per Gauss-Hermite radius node and channel).  Only
// three recurrences are serial: D_n downwards, and psi_n and chi_n upwards;
// two warps run them at the same time.  The coefficients a_n, b_n then take a
// thread per order, and the amplitudes a thread per angle, whose loop over
// the orders is multiply-adds on what the threads before prepared.  Output
// per task: Q_ext, Q_sca and the normalised phase function at NTHETA angles.
#include <math.h>
#include <stdint.h>

#include <vector>

#include "cuda_util.cuh"
#include "device_math.cuh"
#include "jsc_internal.h"

namespace {

struct cplx {
  double re, im;
};

__device__ __forceinline__ cplx cmake(double r, double i) { return cplx{r, i}; }
__device__ __forceinline__ cplx cadd(cplx a, cplx b) { return cplx{a.re + b.re, a.im + b.im}; }
__device__ __forceinline__ cplx csub(cplx a, cplx b) { return cplx{a.re - b.re, a.im - b.im}; }
__device__ __forceinline__ cplx cmul(cplx a, cplx b) {
  return cplx{a.re * b.re - a.im * b.im, a.re * b.im + a.im * b.re};
}
__device__ __forceinline__ cplx cscale(cplx a, double s) { return cplx{a.re * s, a.im * s}; }
__device__ __forceinline__ double cabs_(cplx a) { return hypot(a.re, a.im); }
// a / b; b scaled by its modulus first where its square leaves the range.
__device__ __forceinline__ cplx cdiv(cplx a, cplx b) {
  const double d = b.re * b.re + b.im * b.im;
  if (d > 1e-280 && d < 1e280) {
    const double r = 1.0 / d;
    return cplx{(a.re * b.re + a.im * b.im) * r, (a.im * b.re - a.re * b.im) * r};
  }
  const double s = 1.0 / cabs_(b);
  const double br = s * b.re, bi = s * b.im;
  return cplx{(a.re * br + a.im * bi) * s, (a.im * br - a.re * bi) * s};
}

constexpr int kHalf = (NTHETA + 1) / 2;   // angles 0..90 degrees
constexpr int kThreads = 128;
static_assert(kHalf < kThreads, "a thread per angle and one for Q_sca");

// What a task keeps per order n.
struct MieTerm {
  cplx d;           // D_n
  double psi, chi;
  cplx a, b;        // (2 n + 1) / (n (n + 1)) times a_n, b_n
  double c1, c2;    // (2 n + 1) / n, (n + 1) / n
  double q;         // (2 n + 1) (|a_n|^2 + |b_n|^2)
};

struct MieArgs {
  int n;
  const double *x, *nr, *ni;  // [n] size parameter, refractive index
  const int64_t *doff;        // [n + 1] first term of each task
  MieTerm *term;
  double *out;                // [n][2 + NTHETA]: Q_ext, Q_sca, phase
  unsigned *status;
};

// Bound by the serial recurrences (one complex quotient an order).  With a
// warp per task that ran the upward recurrence, both coefficients and three
// angles a lane in one loop: 916 us for an ice cloud of 1360 tasks (up to 830
// orders), now 199 us.
__global__ void __launch_bounds__(kThreads) mie_kernel(MieArgs A) {
  const int task = blockIdx.x, tid = threadIdx.x;
  const double x = A.x[task];
  const cplx m = cmake(A.nr[task], A.ni[task]);
  const cplx y = cmul(cmake(x, 0.0), m);
  const double xstop = x + 4.0 * pow(x, 0.3333) + 2.0;
  const int nstop = (int)xstop;
  const double ymod = cabs_(y);
  const int nmx = (int)((xstop > ymod ? xstop : ymod) + 15);
  MieTerm *term = A.term + A.doff[task];
  if (nmx + 1 > A.doff[task + 1] - A.doff[task] || nstop >= nmx) {
    if (tid == 0) atomicOr(A.status, 1u);  // the host sized the scratch otherwise
    return;
  }
  if (tid == 0) {
    cplx d = cmake(0.0, 0.0);
    const cplx ry = cdiv(cmake(1.0, 0.0), y);
    for (int k = nmx; k >= 2; k--) {
      const cplx q = cscale(ry, (double)k);
      d = csub(q, cdiv(cmake(1.0, 0.0), cadd(d, q)));
      if (k - 1 <= nstop) term[k - 1].d = d;
    }
  } else if (tid == 32) {
    double psi0 = cos(x), psi1 = sin(x), chi0 = -sin(x), chi1 = cos(x);
    const double rx = 1.0 / x;
    term[0].psi = psi1;
    term[0].chi = chi1;
    for (int n = 1; n <= nstop; n++) {
      const double f = 2.0 * n - 1.0;
      const double psi = div_known(f * psi1, x, rx) - psi0;
      const double chi = div_known(f * chi1, x, rx) - chi0;
      term[n].psi = psi;
      term[n].chi = chi;
      psi0 = psi1;
      psi1 = psi;
      chi0 = chi1;
      chi1 = chi;
    }
  }
  __syncthreads();
  for (int n = 1 + tid; n <= nstop; n += kThreads) {
    MieTerm &t = term[n];
    const double rn = (double)n, psi1 = term[n - 1].psi;
    const cplx xi = cmake(t.psi, -t.chi), xi1 = cmake(psi1, -term[n - 1].chi);
    const cplx ga = cadd(cdiv(t.d, m), cmake(rn / x, 0.0));
    const cplx an = cdiv(csub(cscale(ga, t.psi), cmake(psi1, 0.0)), csub(cmul(ga, xi), xi1));
    const cplx gb = cadd(cmul(m, t.d), cmake(rn / x, 0.0));
    const cplx bn = cdiv(csub(cscale(gb, t.psi), cmake(psi1, 0.0)), csub(cmul(gb, xi), xi1));
    const double fn = (2.0 * rn + 1.0) / (rn * (rn + 1.0));
    t.a = cscale(an, fn);
    t.b = cscale(bn, fn);
    t.c1 = (2.0 * rn + 1.0) / rn;
    t.c2 = (rn + 1.0) / rn;
    t.q = (2.0 * rn + 1.0) * (an.re * an.re + an.im * an.im + bn.re * bn.re + bn.im * bn.im);
  }
  __syncthreads();
  __shared__ double qs_s;
  if (tid == kHalf) {
    double q = 0.0;
#pragma unroll 8
    for (int n = 1; n <= nstop; n++) q += term[n].q;
    qs_s = (2.0 / (x * x)) * q;
  }
  // Sums of a_n p, b_n t, a_n t and b_n p over the odd and the even orders:
  // S1 = sum (a p + b t), S2 = sum (a t + b p), and at the mirror angle
  // 180 - theta, where p and t have the signs (-1)^(n-1) and (-1)^n, the
  // same sums with other signs.
  cplx ap[2], bt[2], at[2], bp[2];
  for (int e = 0; e < 2; e++) ap[e] = bt[e] = at[e] = bp[e] = cmake(0.0, 0.0);
  if (tid < kHalf) {
    const double mu = cos((double)tid * (0.5 * M_PI / (double)(kHalf - 1)));
    double p = 1.0, pprev = 0.0;
    auto order = [&](int n, cplx &sap, cplx &sbt, cplx &sat, cplx &sbp) {
      const MieTerm &t = term[n];
      const cplx a = t.a, b = t.b;
      const double rn = (double)n, c1 = t.c1, c2 = t.c2;
      const double tau = __fma_rn(rn * mu, p, -((rn + 1.0) * pprev));
      sap.re = __fma_rn(a.re, p, sap.re);
      sap.im = __fma_rn(a.im, p, sap.im);
      sbt.re = __fma_rn(b.re, tau, sbt.re);
      sbt.im = __fma_rn(b.im, tau, sbt.im);
      sat.re = __fma_rn(a.re, tau, sat.re);
      sat.im = __fma_rn(a.im, tau, sat.im);
      sbp.re = __fma_rn(b.re, p, sbp.re);
      sbp.im = __fma_rn(b.im, p, sbp.im);
      const double next = __fma_rn(c1 * mu, p, -(c2 * pprev));
      pprev = p;
      p = next;
    };
    int n = 1;
#pragma unroll 2
    for (; n + 1 <= nstop; n += 2) {
      order(n, ap[0], bt[0], at[0], bp[0]);
      order(n + 1, ap[1], bt[1], at[1], bp[1]);
    }
    if (n <= nstop) order(n, ap[0], bt[0], at[0], bp[0]);
  }
  __syncthreads();  // Q_sca
  if (tid >= kHalf) return;
  const double qs = qs_s;
  const cplx s1 = cadd(cadd(ap[0], ap[1]), cadd(bt[0], bt[1]));
  const cplx s2 = cadd(cadd(at[0], at[1]), cadd(bp[0], bp[1]));
  const cplx s1m = cadd(csub(ap[0], ap[1]), csub(bt[1], bt[0]));
  const cplx s2m = cadd(csub(at[1], at[0]), csub(bp[0], bp[1]));
  double *o = A.out + (size_t)task * (2 + NTHETA);
  if (tid == 0) {
    o[0] = (4.0 / (x * x)) * s1.re;  // forward amplitude: extinction theorem
    o[1] = qs;
  }
  const double f = 2.0 / (x * x * qs);
  o[2 + tid] = f * (s1.re * s1.re + s1.im * s1.im + s2.re * s2.re + s2.im * s2.im);
  if (tid != kHalf - 1)
    o[2 + (NTHETA - 1 - tid)] = f * (s1m.re * s1m.re + s1m.im * s1m.im + s2m.re * s2m.re + s2m.im * s2m.im);
}

}  // namespace

// Terms of the D_n recurrence of size parameter x and refractive index
// (nr, ni), as mie_kernel counts them, plus slack for a last-bit difference
// of pow between host and device.
static int64_t mie_slots(double x, double nr, double ni) {
  const double xstop = x + 4.0 * pow(x, 0.3333) + 2.0;
  const double ymod = hypot(x * nr, x * ni);
  return (int64_t)((xstop > ymod ? xstop : ymod) + 15) + 3;
}

extern "C" int jsc_mie_eval(int device, int n, const double *x, const double *nr,
                            const double *ni, double *out) {
  if (n <= 0) return JSC_OK;
  {
    const cudaError_t e = cudaSetDevice(device);
    if (e != cudaSuccess) {
      jsc_set_error(JSC_ERR_CUDA, "Mie: cudaSetDevice(%d): %s", device, cudaGetErrorString(e));
      return JSC_ERR_CUDA;
    }
  }
  std::vector<int64_t> off((size_t)n + 1, 0);
  for (int i = 0; i < n; i++) {
    const int64_t s = mie_slots(x[i], nr[i], ni[i]);
    if (!(x[i] > 0) || s > 10000 + 3) {
      jsc_set_error(JSC_ERR_ARG, "Mie: size parameter %g needs more than 10000 terms", x[i]);
      return JSC_ERR_ARG;
    }
    off[i + 1] = off[i] + s;
  }
  double *dx = nullptr, *dnr = nullptr, *dni = nullptr, *dout = nullptr;
  int64_t *doff = nullptr;
  MieTerm *dterm = nullptr;
  unsigned *dst = nullptr;
  int st = JSC_OK;
  auto fail = [&](cudaError_t e, const char *what) {
    if (e != cudaSuccess && !st) {
      jsc_set_error(JSC_ERR_CUDA, "Mie: %s: %s", what, cudaGetErrorString(e));
      st = JSC_ERR_CUDA;
    }
  };
  fail(cudaMalloc(&dx, 3 * (size_t)n * sizeof(double)), "cudaMalloc");
  fail(cudaMalloc(&dout, (size_t)n * (2 + NTHETA) * sizeof(double)), "cudaMalloc");
  fail(cudaMalloc(&doff, ((size_t)n + 1) * sizeof(int64_t)), "cudaMalloc");
  fail(cudaMalloc(&dterm, (size_t)off[n] * sizeof(MieTerm)), "cudaMalloc");
  fail(cudaMalloc(&dst, sizeof(unsigned)), "cudaMalloc");
  if (!st) {
    dnr = dx + n;
    dni = dx + 2 * (size_t)n;
    fail(cudaMemcpy(dx, x, n * sizeof(double), cudaMemcpyHostToDevice), "copy");
    fail(cudaMemcpy(dnr, nr, n * sizeof(double), cudaMemcpyHostToDevice), "copy");
    fail(cudaMemcpy(dni, ni, n * sizeof(double), cudaMemcpyHostToDevice), "copy");
    fail(cudaMemcpy(doff, off.data(), ((size_t)n + 1) * sizeof(int64_t), cudaMemcpyHostToDevice),
         "copy");
    fail(cudaMemset(dst, 0, sizeof(unsigned)), "memset");
  }
  if (!st) {
    MieArgs a;
    a.n = n;
    a.x = dx;
    a.nr = dnr;
    a.ni = dni;
    a.doff = doff;
    a.term = dterm;
    a.out = dout;
    a.status = dst;
    mie_kernel<<<(unsigned)n, kThreads>>>(a);
    jsc_count_launch();
    fail(cudaGetLastError(), "mie_kernel launch");
    unsigned hs = 0;
    fail(cudaMemcpy(&hs, dst, sizeof(unsigned), cudaMemcpyDeviceToHost), "mie_kernel");
    if (!st && hs) {
      jsc_set_error(JSC_ERR_ARG, "Mie: recurrence scratch too small");
      st = JSC_ERR_ARG;
    }
    fail(cudaMemcpy(out, dout, (size_t)n * (2 + NTHETA) * sizeof(double), cudaMemcpyDeviceToHost),
         "copy back");
  }
  cudaFree(dx);
  cudaFree(dout);
  cudaFree(doff);
  cudaFree(dterm);
  cudaFree(dst);
  return st;
}
