// Launchers of the gas transmittance, the segment pass and the transfer pass.
#include "ega_gas.cuh"

// A warp per emitter; the register budget follows the block size.  Up to four
// emitters 72 registers (28 warps an SM, no spills) beat 64 (32 warps): 43.5
// against 44.6 ms for the pencils of depth-2 scattering, 2.75 against 2.83 ms
// for 5000 rays x 16 channels x 4 emitters; 80 (24 warps) only do while the
// rays fill less than the chip, and with eight emitters 64 stay best (71.6 ms
// against 75.3 with 80 and 75.8 with 48).
template <bool DIG>
static void gas_launch(const GasArgs &ga, cudaStream_t s) {
  const int nw = ga.e.m.ng > 0 ? ga.e.m.ng : 1;
  const unsigned blocks = (unsigned)(((int64_t)ga.e.n_rays + 31) / 32 * ga.e.m.nd);
  const size_t sh = gas_shmem(nw, 32, nw <= 8 ? 4 : 2);
  if (nw <= 2) ega_gas_kernel<DIG, 4, 64, 14><<<blocks, 32 * nw, sh, s>>>(ga);
  else if (nw <= 4) ega_gas_kernel<DIG, 4, 128, 7><<<blocks, 32 * nw, sh, s>>>(ga);
  else if (nw <= 8) ega_gas_kernel<DIG, 4, 256, 4><<<blocks, 32 * nw, sh, s>>>(ga);
  else ega_gas_kernel<DIG, 2, 1024, 1><<<blocks, 32 * nw, sh, s>>>(ga);
}

template <bool DIG>
static void gas4_launch(const GasArgs &ga, cudaStream_t s) {
  const int nw = ga.e.m.ng > 0 ? ga.e.m.ng : 1;
  const unsigned blocks = (unsigned)(((int64_t)ga.e.n_rays + 7) / 8 * ga.e.m.nd);
  const size_t sh = gas_shmem(nw, 8, 4);
  if (nw <= 2) ega_gas4_kernel<DIG, 4, 64, 16><<<blocks, 32 * nw, sh, s>>>(ga);
  else if (nw <= 4) ega_gas4_kernel<DIG, 4, 128, 8><<<blocks, 32 * nw, sh, s>>>(ga);
  else if (nw <= 8) ega_gas4_kernel<DIG, 4, 256, 4><<<blocks, 32 * nw, sh, s>>>(ga);
  else ega_gas4_kernel<DIG, 4, 1024, 1><<<blocks, 32 * nw, sh, s>>>(ga);
}

void jsc_ega_gas_launch(const GasArgs &ga, int lanes, cudaStream_t s) {
  if (lanes == 4) {
    if (ga.e.digest) gas4_launch<true>(ga, s);
    else gas4_launch<false>(ga, s);
  } else {
    if (ga.e.digest) gas_launch<true>(ga, s);
    else gas_launch<false>(ga, s);
  }
}

// Points per step: 64 fill a block's threads from 32 channels on; with fewer
// channels 128 do better (16: 7.3 against 7.6 ms in single scattering, 8: 8.9
// against 10.8 ms in depth 2, 64: 5.6 against 5.3 ms).
void jsc_segment_launch(SegmentArgs sa, cudaStream_t s) {
  if (sa.n_points <= 0) return;
  sa.step = sa.m.nd >= 32 ? 64 : JSC_SEG_POINTS;
  int64_t blocks = (sa.n_points + sa.step - 1) / sa.step;
  // a count known only on the device: a grid of a few blocks per SM walks it
  if (sa.n_live && blocks > 148 * 16) blocks = 148 * 16;
  segment_kernel<<<(unsigned)blocks, JSC_SEG_THREADS, 0, s>>>(sa);
}

void jsc_transfer_launch(const EgaArgs &ea, const double *x, const double *src, cudaStream_t s) {
  const int64_t n = (int64_t)ea.n_rays * ea.m.nd;
  transfer_kernel<<<(unsigned)((n + 127) / 128), 128, 0, s>>>(ea, x, src);
}
