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
#include <string.h>

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

// What a task keeps per order n: D_n, then (2 n + 1) / (n (n + 1)) a_n in its
// place; psi_n and chi_n, then the same of b_n; and (2 n + 1) (|a_n|^2 +
// |b_n|^2).
constexpr int kTerm = 5;                  // doubles per order
constexpr int kSharedOrders = 5000;       // most orders kept in shared memory (200 KB)
constexpr int kScratchTasks = 1184;       // tasks per launch above that: 8 blocks an SM

struct MieArgs {
  int n, cap;                 // tasks; orders 0 .. cap - 1 of the largest
  const int *task;            // [n] the tasks, long ones first
  const double *x, *nr, *ni;  // [n] size parameter, refractive index
  const cplx *c;              // [cap] (2 n + 1) / n, (n + 1) / n
  double *term;               // [blocks][kTerm * cap] where shared memory is too small
  double *out;                // [n][2 + NTHETA]: Q_ext, Q_sca, phase
  unsigned *status;
};

// Bound by the serial recurrences (one complex quotient an order).  With a
// warp per task that ran the upward recurrence, both coefficients and three
// angles a lane in one loop: 916 us for an ice cloud of 1360 tasks (up to 830
// orders), now 146 us.  The orders lie in shared memory (33 KB a block there),
// long tasks start first: in device memory, allocated for the call and 88 bytes
// an order, the kernel took 199 us and the allocation 0.6 ms more than before.
// SHARED false: more than kSharedOrders.
template <bool SHARED>
__global__ void __launch_bounds__(kThreads) mie_kernel(MieArgs A) {
  extern __shared__ __align__(16) double mie_sh[];
  const int task = A.task[blockIdx.x], tid = threadIdx.x;
  double *base = SHARED ? mie_sh : A.term + (size_t)blockIdx.x * kTerm * A.cap;
  cplx *td = reinterpret_cast<cplx *>(base);                         // D_n, a_n
  cplx *tr = reinterpret_cast<cplx *>(base) + A.cap;                 // psi_n and chi_n, b_n
  double *tq = base + 4 * (size_t)A.cap;
  const double x = A.x[task];
  const cplx m = cmake(A.nr[task], A.ni[task]);
  const cplx y = cmul(cmake(x, 0.0), m);
  const double xstop = x + 4.0 * pow(x, 0.3333) + 2.0;
  const int nstop = (int)xstop;
  const double ymod = cabs_(y);
  const int nmx = (int)((xstop > ymod ? xstop : ymod) + 15);
  if (nstop + 1 > A.cap || nstop >= nmx) {
    if (tid == 0) atomicOr(A.status, 1u);  // the host counted otherwise
    return;
  }
  if (tid == 0) {
    cplx d = cmake(0.0, 0.0);
    const cplx ry = cdiv(cmake(1.0, 0.0), y);
    for (int k = nmx; k >= 2; k--) {
      const cplx q = cscale(ry, (double)k);
      d = csub(q, cdiv(cmake(1.0, 0.0), cadd(d, q)));
      if (k - 1 <= nstop) td[k - 1] = d;
    }
  } else if (tid == 32) {
    double psi0 = cos(x), psi1 = sin(x), chi0 = -sin(x), chi1 = cos(x);
    const double rx = 1.0 / x;
    tr[0] = cmake(psi1, chi1);
    for (int n = 1; n <= nstop; n++) {
      const double f = 2.0 * n - 1.0;
      const double psi = div_known(f * psi1, x, rx) - psi0;
      const double chi = div_known(f * chi1, x, rx) - chi0;
      tr[n] = cmake(psi, chi);
      psi0 = psi1;
      psi1 = psi;
      chi0 = chi1;
      chi1 = chi;
    }
  }
  __syncthreads();
  // from the top, so that the order below a chunk is still psi and chi
  for (int n0 = (nstop - 1) / kThreads * kThreads; n0 >= 0; n0 -= kThreads) {
    const int n = n0 + 1 + tid;
    cplx an, bn;
    double q = 0;
    if (n <= nstop) {
      const double rn = (double)n, psi = tr[n].re, psi1 = tr[n - 1].re;
      const cplx xi = cmake(psi, -tr[n].im), xi1 = cmake(psi1, -tr[n - 1].im), d = td[n];
      const cplx ga = cadd(cdiv(d, m), cmake(rn / x, 0.0));
      an = cdiv(csub(cscale(ga, psi), cmake(psi1, 0.0)), csub(cmul(ga, xi), xi1));
      const cplx gb = cadd(cmul(m, d), cmake(rn / x, 0.0));
      bn = cdiv(csub(cscale(gb, psi), cmake(psi1, 0.0)), csub(cmul(gb, xi), xi1));
      q = (2.0 * rn + 1.0) * (an.re * an.re + an.im * an.im + bn.re * bn.re + bn.im * bn.im);
      const double fn = (2.0 * rn + 1.0) / (rn * (rn + 1.0));
      an = cscale(an, fn);
      bn = cscale(bn, fn);
    }
    __syncthreads();
    if (n <= nstop) {
      td[n] = an;
      tr[n] = bn;
      tq[n] = q;
    }
  }
  __syncthreads();
  __shared__ double qs_s;
  if (tid == kHalf) {
    double q = 0.0;
#pragma unroll 8
    for (int n = 1; n <= nstop; n++) q += tq[n];
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
      const cplx a = td[n], b = tr[n], c = A.c[n];
      const double rn = (double)n, c1 = c.re, c2 = c.im;
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
  int cap = 0;
  std::vector<int> orders((size_t)n);
  for (int i = 0; i < n; i++) {
    const int64_t s = mie_slots(x[i], nr[i], ni[i]);
    if (!(x[i] > 0) || s > 10000 + 3) {
      jsc_set_error(JSC_ERR_ARG, "Mie: size parameter %g needs more than 10000 terms", x[i]);
      return JSC_ERR_ARG;
    }
    orders[i] = (int)(x[i] + 4.0 * pow(x[i], 0.3333) + 2.0) + 3;  // and slack, as mie_slots
    if (orders[i] > cap) cap = orders[i];
  }
  // one buffer: x, nr, ni, the factors of the orders, the tasks by length
  // (64 classes, long ones first); then the status word and the output
  const size_t nin = 3 * (size_t)n + 2 * (size_t)cap + ((size_t)n + 1) / 2;
  const size_t nout = 1 + (size_t)n * (2 + NTHETA);
  std::vector<double> in(nin, 0.0);
  memcpy(in.data(), x, n * sizeof(double));
  memcpy(in.data() + n, nr, n * sizeof(double));
  memcpy(in.data() + 2 * (size_t)n, ni, n * sizeof(double));
  double *c = in.data() + 3 * (size_t)n;
  for (int k = 1; k < cap; k++) {
    c[2 * k] = (2.0 * k + 1.0) / k;
    c[2 * k + 1] = (k + 1.0) / k;
  }
  int *task = reinterpret_cast<int *>(c + 2 * (size_t)cap), first[65] = {0};
  auto cls = [&](int i) { return 63 - (int)((int64_t)orders[i] * 63 / cap); };
  for (int i = 0; i < n; i++) first[cls(i) + 1]++;
  for (int k = 0; k < 64; k++) first[k + 1] += first[k];
  for (int i = 0; i < n; i++) task[first[cls(i)]++] = i;
  double *d = nullptr, *dterm = nullptr;
  int st = JSC_OK;
  auto fail = [&](cudaError_t e, const char *what) {
    if (e != cudaSuccess && !st) {
      jsc_set_error(JSC_ERR_CUDA, "Mie: %s: %s", what, cudaGetErrorString(e));
      st = JSC_ERR_CUDA;
    }
  };
  const bool shared = cap <= kSharedOrders;
  const size_t sh = shared ? sizeof(double) * kTerm * cap : 0;
  fail(cudaMalloc(&d, (nin + nout + 1) * sizeof(double)), "cudaMalloc");
  if (!shared) fail(cudaMalloc(&dterm, sizeof(double) * kTerm * cap * (size_t)(n < kScratchTasks ? n : kScratchTasks)), "cudaMalloc");
  // the largest size always: the attribute is shared by all threads of the process
  if (sh > 48 * 1024)
    fail(cudaFuncSetAttribute(mie_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                              kSharedOrders * kTerm * (int)sizeof(double)),
         "shared memory");
  if (!st) {
    double *dc = d + ((3 * (size_t)n + 1) & ~(size_t)1);  // 16-byte aligned, as in the copies below
    double *dt = dc + 2 * (size_t)cap, *dres = dt + ((size_t)n + 1) / 2;
    fail(cudaMemcpy(d, in.data(), 3 * (size_t)n * sizeof(double), cudaMemcpyHostToDevice), "copy");
    fail(cudaMemcpy(dc, c, (nin - 3 * (size_t)n) * sizeof(double), cudaMemcpyHostToDevice), "copy");
    fail(cudaMemset(dres, 0, sizeof(double)), "memset");
    MieArgs a;
    a.n = n;
    a.cap = cap;
    a.task = reinterpret_cast<const int *>(dt);
    a.x = d;
    a.nr = d + n;
    a.ni = d + 2 * (size_t)n;
    a.c = reinterpret_cast<const cplx *>(dc);
    a.term = dterm;
    a.out = dres + 1;
    a.status = reinterpret_cast<unsigned *>(dres);
    const int step = shared || n < kScratchTasks ? n : kScratchTasks;
    for (int o = 0; o < n && !st; o += step, a.task += step) {
      const unsigned blocks = (unsigned)(n - o < step ? n - o : step);
      if (shared) mie_kernel<true><<<blocks, kThreads, sh>>>(a);
      else mie_kernel<false><<<blocks, kThreads>>>(a);
      jsc_count_launch();
      fail(cudaGetLastError(), "mie_kernel launch");
    }
    unsigned hs = 0;
    if (!st) fail(cudaMemcpy(&hs, dres, sizeof(unsigned), cudaMemcpyDeviceToHost), "mie_kernel");
    if (!st && hs) {
      jsc_set_error(JSC_ERR_ARG, "Mie: recurrence scratch too small");
      st = JSC_ERR_ARG;
    }
    if (!st)
      fail(cudaMemcpy(out, dres + 1, (nout - 1) * sizeof(double), cudaMemcpyDeviceToHost), "copy back");
  }
  cudaFree(d);
  cudaFree(dterm);
  return st;
}
