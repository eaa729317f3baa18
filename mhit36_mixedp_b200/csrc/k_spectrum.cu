// Shell-summed kinetic-energy spectrum of the velocity on the device.  The reference has no
// three-dimensional spectrum tool (its post-processing computes dissipation and drop statistics,
// post/compute_diss, post/unionfind_periodic); this is the textbook definition
//   E(k) = 1/2 sum over |kappa| in [k - 1/2, k + 1/2) of |u_kappa|^2 + |v_kappa|^2 + |w_kappa|^2,
//   u_kappa = (1/N) sum_x u(x) exp(-i kappa.x),   N = nx ny nz,
// so that sum_k E(k) = 1/2 <u.u> (Parseval), the kinetic energy of multi/main.f90's diagnostics.
// Wavenumbers are in units of 2 pi / Lx: kappa_x = m_x, kappa_y = m_y nx/ny, kappa_z = m_z nx/nz
// for a box of nx dx by ny dx by nz dx with Lx = 2 pi.
//
// Each component is transformed by the Poisson solver's own FP64 passes (x real-to-complex, then
// y and z forward) into the x-half spectrum [nz][ny][pitch]; k_spec_bin adds each element's
// energy (weight 2 for 0 < kx < nx/2, the conjugate half) to a block histogram in shared memory,
// and k_spec_reduce sums the block histograms in block order.  The shared-memory atomics make the
// last bits depend on scheduling.
#include "common.cuh"
#include "kernels.h"

namespace mhit {

// A warp takes 32 consecutive kx of one row: the shell number never falls along kx, so equal shells
// sit in adjacent lanes.  A segmented sum by shuffles leaves each run's total in its first lane,
// and those lanes add to the warp's own histogram in shared memory, distinct shells each: no
// atomics, and sums in a fixed order.  (One double atomic per element into a histogram per block
// took 2.10 ms per component at 512^3, where reading the spectrum takes 0.17 ms.)
constexpr int SWARPS = 8;  // warps per block, fewer where their histograms do not fit

__global__ void __launch_bounds__(32 * SWARPS) k_spec_bin(const Cx<double>* __restrict__ spec, Geo g,
                                                         const DevScalars* __restrict__ sc, int comp, int nbins,
                                                         double* __restrict__ partials) {
  extern __shared__ double hist[];
  const int nwarps = blockDim.x >> 5, lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  double* mine = hist + (size_t)wid * nbins;
  for (int b = lane; b < nbins; b += 32) mine[b] = 0.0;
  __syncwarp();
  const int nx = g.nx, ny = g.ny, nz = g.nz, nkx = g.nkx, pitch = g.pitch;
  const double ntot = (double)nx * ny * nz, invn = 1.0 / ntot;
  const double sy = (double)nx / ny, sz = (double)nx / nz;
  const double mean = sc->mean[comp];  // the stored field still carries the lazily removed mean
  const int rows = ny * nz;
  for (int row = blockIdx.x * nwarps + wid; row < rows; row += gridDim.x * nwarps) {
    const int j = row % ny, k = row / ny;
    const double my = (double)(2 * j <= ny ? j : j - ny) * sy;
    const double mz = (double)(2 * k <= nz ? k : k - nz) * sz;
    const double kyz = my * my + mz * mz;
    const Cx<double>* src = spec + (size_t)row * pitch;
    for (int kx0 = 0; kx0 < nkx; kx0 += 32) {
      const int kx = kx0 + lane;
      int shell = 0x7fffffff;  // past the row's end: a run of its own, never added
      double e = 0.0;
      if (kx < nkx) {
        Cx<double> c = src[kx];
        if (row == 0 && kx == 0) c.x -= mean * ntot;
        const double re = c.x * invn, im = c.y * invn;
        const double w = (kx == 0 || 2 * kx == nx) ? 0.5 : 1.0;
        shell = (int)rint(sqrt((double)kx * kx + kyz));
        e = w * (re * re + im * im);
      }
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const double eo = __shfl_down_sync(0xffffffffu, e, o);
        const int so = __shfl_down_sync(0xffffffffu, shell, o);
        if (lane + o < 32 && so == shell) e += eo;
      }
      const int before = __shfl_up_sync(0xffffffffu, shell, 1);
      if ((lane == 0 || before != shell) && shell < nbins) mine[shell] += e;
      __syncwarp();
    }
  }
  __syncthreads();
  for (int b = threadIdx.x; b < nbins; b += blockDim.x) {
    double s = 0.0;
    for (int q = 0; q < nwarps; ++q) s += hist[(size_t)q * nbins + b];
    partials[(size_t)blockIdx.x * nbins + b] = s;
  }
}

// one warp per shell: its lanes stride over the blocks' histograms, then a shuffle tree
__global__ void __launch_bounds__(256) k_spec_reduce(const double* __restrict__ partials, int nblocks, int nbins,
                                                     double* __restrict__ E) {
  const int lane = threadIdx.x & 31;
  const int b = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  if (b >= nbins) return;
  double s = 0.0;
  for (int q = lane; q < nblocks; q += 32) s += partials[(size_t)q * nbins + b];
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) s += __shfl_down_sync(0xffffffffu, s, o);
  if (lane == 0) E[b] += s;
}

int spectrum_blocks(const Geo& g) {
  const int rows = g.ny * g.nz;
  return rows < 148 * 7 ? rows : 148 * 7;
}

cudaError_t launch_spectrum_bin(const Cx<double>* spec, const Geo& g, const DevScalars* sc, int comp, int nbins,
                                double* partials, double* E, cudaStream_t st) {
  const int nb = spectrum_blocks(g);
  // one histogram per warp: eight up to 1500 shells (every box up to 1024 points), fewer beyond
  const size_t one = (size_t)nbins * sizeof(double);
  int warps = SWARPS;
  while (warps > 1 && warps * one > 96 * 1024) warps /= 2;
  const size_t smem = warps * one;
  if (smem > 48 * 1024) {
    cudaError_t e = cudaFuncSetAttribute(k_spec_bin, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
  }
  k_spec_bin<<<nb, 32 * warps, smem, st>>>(spec, g, sc, comp, nbins, partials);
  k_spec_reduce<<<(nbins + 7) / 8, 256, 0, st>>>(partials, nb, nbins, E);
  return cudaGetLastError();
}

}  // namespace mhit
