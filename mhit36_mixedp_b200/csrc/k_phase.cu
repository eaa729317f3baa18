// ACDI phase-field transport: multi/main.f90:522-636 in one kernel.
//
// The reference makes five passes with three stored intermediates (psidi, tanh_psi and the
// three normal components) and six halo exchanges.  Here a block owns a PTX x PTY column of
// cells and marches up a chunk of z planes.  It has one thread per vertical pair of positions of
// the tile plus its x/y halo of 2, and each thread keeps its two z columns in registers:
//   phi  planes k-1..k+3 (k+3 loaded one plane ahead)
//   psi  = eps log((min(phi,1)+1e-16)/(1-min(phi,1)+1e-16))            (:527-528), k..k+2
//   Fz   of F = 1/4 (1 - t^2) n/(|n|+1e-16), n = central psi differences (:559-561,
//        :586-589, :609-614), t = tanh(psi/(2 eps)) (:530),               planes k-1..k+1
// Only x/y neighbours go through shared memory: psi(k+1), phi(k) and Fx, Fy(k), each
// double-buffered, and the output cells' u, v, w and rhsphi_o, copied there with cp.async one
// plane ahead.  Every shared read of plane k's iteration reads what the previous iteration wrote
// or fetched, so one barrier per plane suffices.  psi is evaluated on the halo of 2 and F on the
// halo of 1; threads are numbered so that the output pairs fill whole warps, then the F ring,
// then the outer psi-only ring.  The kernel writes only phi^{n+1} and rhsphi_o.
//
// t is evaluated in closed form: tanh(log(r)/2) = (r-1)/(r+1) with r = (val+1e-16)/(1-val+1e-16)
// gives t = (2 val - 1)/(1 + 2e-16) exactly in real arithmetic; in float64 it agrees with the
// reference's tanh(0.5*psi/eps) to 2.2e-16 over the whole range of phi (a NaN psi, from
// phi < -1e-16, still gives a NaN t as in the reference).
//
// With PhaseArgs::clamp (opt-in, off by default) phi is also clamped below at 0 before the
// log, so a cell undershooting to phi < -1e-16 no longer turns psi into NaN.
//
// gamma = 1.0*gumax is read from the device scalars written by the previous projection
// (:536, :998-1002); u, v, w are the stored fields minus the lazily removed mean.
#include <cuda_pipeline.h>

#include <type_traits>

#include "common.cuh"
#include "kernels.h"
#include "phase_math.cuh"

namespace mhit {

// 32 x 24 output cells per block, one block per SM, two vertically adjacent cells per thread.  The
// kernel is bound by the latency of its FP64 chains (reciprocal, logarithm polynomial, reciprocal
// square root) and of its loads at the 16 to 24 warps an SM holds.  One cell per thread and loads
// in the iteration that uses them (32 x 16 tiles, 23 warps) issued 62% of the cycles and took
// 2.34 ms at 512^3 and 331 us at 256^3.  Now each thread carries two independent chains, psi is
// evaluated on 1.31 instead of 1.41 and F on 1.15 instead of 1.20 cells per output cell, the y
// neighbours inside a pair come from registers, one barrier serves half again as many cells, and
// the fields of the next plane are fetched a whole plane ahead: 1.97 ms and 264 us (without the
// fetch 2.18 ms and 288 us).  ncu at 256^3: 12.3 -> 8.3 warp instructions per cell, FP64 pipe 43%,
// issue 54%.  504 threads leave 128 registers: 32 x 32 tiles (648 threads, 80 registers) spill and
// take 2.01 ms, two 32 x 12 blocks per SM 2.29 ms (without the fetch).  The branch-free log_ratio and
// rsqrt_fast are what lets the two chains interleave: with CUDA's log and rsqrt, whose special cases
// branch, this layout takes 2.66 ms where it takes 2.09 and the one-cell layout 2.41 (one box).
// (These are times without the clamp before F_of's conditions were those of now: 1.89 ms and 250 us, with
// the clamp 1.81 ms and 241 us.)
template <int TX, int TY> struct PhaseTile {
  static constexpr int PTX = TX, PTY = TY;             // output cells per block in x, y
  static constexpr int PHX = PTX + 4, PHY = PTY + 4;   // positions with the halo of 2
  static constexpr int PPOS = PHX * PHY;               // positions of a shared plane
  static constexpr int PNT = PHX * PHY / 2;            // threads per block: one per pair of rows
  static constexpr int PNO = PTX * PTY / 2;            // threads with two output cells
  static constexpr int PNF = PNO + 2 * PTX + 4 + 2 * (PTY / 2);  // ... plus those that evaluate F on the halo of 1
  // one plane of the output cells' u (one column more), v (one row more), w(k+1) and rhs_o in shared
  // memory, fetched with cp.async one plane ahead
  static constexpr int PUX = PTX + 2;
  static constexpr int PSU = 0, PSV = PSU + PTY * PUX, PSW = PSV + (PTY + 1) * PTX, PSR = PSW + PTY * PTX,
                       PSTG = PSR + PTY * PTX;
  // psi, phi, Fx, Fy and the staged fields, twice each
  static constexpr size_t PSMEM = sizeof(double) * (8 * PPOS + 2 * PSTG);
};
// The tiles above, and two of 16 rows for the boxes of 16 or 32 rows, where a third to a half of 24-row
// tiles lies outside the box: 48 cells wide (520 threads, 96 registers) from nx = 192 on, where the
// last tile of a row loses little, 32 wide (360 threads) below.  us with 24-row, 32 x 16, 48 x 16 tiles:
//   1024x32x1024 695, 570, 528   512x16x512 96, 83, 78   192x32x1024 139, 116, 107
//   128x32x128    21,  18,  19   64x32x512  31, 25, 31   32^3         12,  11,  13
// and (whole steps) 16 boxes of 64x32x64 226, 214, 226, 8 of 256x32x256 1459, 1401, 1372.  At 64 rows
// 24-row tiles lose an eighth and take 76 against 82 us at 256x64x256 (32 x 16).
using Tall = PhaseTile<32, 24>;
using Flat = PhaseTile<32, 16>;
using Wide = PhaseTile<48, 16>;
constexpr int PMINB = 1;    // resident blocks per SM
constexpr int PUNROLL = 2;  // two-plane bodies per loop iteration (1: 2.07 ms at 512^3)
constexpr double ENUM = 1.0e-16;
constexpr double TNORM = 1.0 / (1.0 + 2.0 * ENUM);

__device__ __forceinline__ int pmodi(int x, int n) {
  x %= n;
  return x < 0 ? x + n : x;
}

// One z column of PTX x PTY cells, tile (bx, by), chunk bz, of the box a; dta, dtb = dt alpha,
// dt beta of the AB2 update.
template <bool CLAMP, typename L>
__device__ __forceinline__ void phase_tile(const PhaseArgs& a, double dta, double dtb, int bx, int by, int bz,
                                           unsigned char* smraw) {
  constexpr int PTX = L::PTX, PTY = L::PTY, PHX = L::PHX, PHY = L::PHY, PPOS = L::PPOS, PNO = L::PNO, PNF = L::PNF;
  constexpr int PUX = L::PUX, PSU = L::PSU, PSV = L::PSV, PSW = L::PSW, PSR = L::PSR, PSTG = L::PSTG;
  // thread -> column hx and row pair (rows 2 r, 2 r + 1) of the (PHX x PHY) grid of the tile with
  // its halo: first the output pairs (whole warps), then the pairs that add F on the halo of 1
  // (bottom and top row pair, of which only the inner row does; columns 1 and PTX + 2), then the
  // psi-only columns 0 and PTX + 3
  const int tid = threadIdx.x;
  int hx, r;
  if (tid < PNO) {
    hx = 2 + tid % PTX;
    r = 1 + tid / PTX;
  } else if (tid < PNO + 2 * (PTX + 2)) {
    const int e = tid - PNO;
    hx = 1 + e % (PTX + 2);
    r = e < PTX + 2 ? 0 : PHY / 2 - 1;
  } else if (tid < PNF) {
    const int e = tid - PNO - 2 * (PTX + 2);
    hx = e < PTY / 2 ? 1 : PTX + 2;
    r = 1 + e % (PTY / 2);
  } else {
    const int e = tid - PNF;
    hx = e < PHY / 2 ? 0 : PTX + 3;
    r = e % (PHY / 2);
  }
  const int q = 2 * r * PHX + hx;  // lower cell's position in a shared plane; the upper one's is q + PHX
  // shared planes at this position: psi[2], phi[2], Fx[2], Fy[2]
  double* sps = reinterpret_cast<double*>(smraw) + q;
  double* sph = sps + 2 * PPOS;
  double* sfx = sph + 2 * PPOS;
  double* sfy = sfx + 2 * PPOS;

  const Geo& g = a.g;
  const int nx = g.nx, ny = g.ny, nz = g.nz;
  const int plane = nx * ny, ntot = plane * nz;
  const int i0 = bx * PTX, j0 = by * PTY;
  const int zc = a.zchunk;
  const int k0 = bz * zc, k1 = min(k0 + zc, nz);
  const int i = i0 - 2 + hx, j = j0 - 2 + 2 * r;  // lower cell; j and ny are even
  const int ic = pmodi(i, nx), jc = pmodi(j, ny);
  const int col = jc * nx + ic;                   // the upper cell's column is col + nx
  const bool frole = tid < PNF;
  const bool fa = frole && r >= 1, fb = frole && r < PHY / 2 - 1;
  const bool orole = tid < PNO && i < nx && j < ny;
  const double* __restrict__ phig = a.phi;

  auto clampv = [](double ph) {
    double val = fmin(ph, 1.0);
    if (CLAMP) val = fmax(val, 0.0);
    return val;
  };
  // psi / eps of multi/main.f90:527-528 (only the direction of its gradient is used)
  auto psi_of = [&](double ph) {
    const double val = clampv(ph);
    return log_ratio<CLAMP>(val + ENUM, 1.0 - val + ENUM);
  };
  // F of one cell at one plane (multi/main.f90:530, 559-561, 586-589, 609-614) from the psi
  // differences dx, dy, dz and its phi, psi.  n/(|n| + 1e-16) is n rsqrt(|n|^2), 0 for n = 0: it
  // differs from the reference's quotient by 1e-16/|n| relative, far below rounding where the
  // interface makes |n| large, and where psi is flat (|n| tiny) 1/4 (1 - t^2) ~ phi (1 - phi) ~ 0
  // multiplies it.  The fused multiply-adds are written out, so the rounding does not depend on
  // how the compiler contracts each copy of the loop body.
  auto F_of = [&](double dx, double dy, double dz, double ph, double ps, double& fx, double& fy, double& fz) {
    const double n2 = __fma_rn(dz, dz, __fma_rn(dy, dy, __dmul_rn(dx, dx)));
    // clamped, psi is finite; else an infinite n2 gives 0 and NaN stays NaN
    const double normag = (CLAMP ? n2 > 0.0 : n2 != 0.0 && n2 != INFINITY) ? rsqrt_fast(n2) : 0.0;
    const double val = clampv(ph);
    const double tt = (ps == ps) ? __fma_rn(2.0, val, -1.0) * TNORM : ps;
    const double fac = __dmul_rn(__dmul_rn(0.25, __fma_rn(-tt, tt, 1.0)), normag);
    fx = __dmul_rn(dx, fac);
    fy = __dmul_rn(dy, fac);
    fz = __dmul_rn(dz, fac);
  };

  const double gamma = 1.0 * a.sc->gumax;
  const double mu_ = a.sc->mean[0], mv_ = a.sc->mean[1], mw_ = a.sc->mean[2];
  const double dxi = g.dxi, ddxi = g.ddxi;
  const double hdxi = 0.5 * dxi;  // (x*0.5)*dxi == x*(0.5*dxi) exactly
  // the right-hand side's constant factors, applied once per sum of terms (see the output block)
  const double c_lap = gamma * (g.eps * ddxi), c_shp = gamma * -hdxi;
  int c = k0 * plane + col;  // lower cell (output role)
  const int dux = (i + 1 == nx) ? 1 - nx : 1;
  const int dvy = (j + 2 == ny) ? (2 - ny) * nx : 2 * nx;  // the row above the pair
  // staged fields of this pair; the pairs at the tile's or the box's upper edges also fetch the
  // column (row) beyond it
  const int lx = hx - 2, ly = 2 * (r - 1);
  double* const stg = reinterpret_cast<double*>(smraw) + 8 * PPOS;
  const bool uedge = lx == PTX - 1 || i + 1 == nx, vedge = ly + 2 == PTY || j + 2 == ny;
  const int su = PSU + ly * PUX + lx, sv = PSV + ly * PTX + lx, sw = PSW + ly * PTX + lx, sr = PSR + ly * PTX + lx;
  auto stage = [&](double* d, int k, int cc) {  // plane k, whose lower cell is cc, into the slot at d
    const int cw = (k + 1 == nz) ? cc - (nz - 1) * plane : cc + plane;
    __pipeline_memcpy_async(d + su, a.u + cc, 8);
    __pipeline_memcpy_async(d + su + PUX, a.u + cc + nx, 8);
    if (uedge) {
      __pipeline_memcpy_async(d + su + 1, a.u + cc + dux, 8);
      __pipeline_memcpy_async(d + su + PUX + 1, a.u + cc + nx + dux, 8);
    }
    __pipeline_memcpy_async(d + sv, a.v + cc, 8);
    __pipeline_memcpy_async(d + sv + PTX, a.v + cc + nx, 8);
    if (vedge) __pipeline_memcpy_async(d + sv + 2 * PTX, a.v + cc + dvy, 8);
    __pipeline_memcpy_async(d + sw, a.w + cw, 8);
    __pipeline_memcpy_async(d + sw + PTX, a.w + cw + nx, 8);
    __pipeline_memcpy_async(d + sr, a.rphio + cc, 8);
    __pipeline_memcpy_async(d + sr + PTX, a.rphio + cc + nx, 8);
  };
  double wa0 = orole ? __ldg(a.w + c) : 0.0, wb0 = orole ? __ldg(a.w + c + nx) : 0.0;

  // Right-hand side and update of one output cell: p its phi and its six neighbours', the face
  // velocities, and the sum of the F differences.  multi/main.f90:551-557 and :609-614 with each
  // group's constant factor taken out of its sum (the same expression up to rounding: a few ulp
  // of the terms, far inside the 1e-12 parity bound):
  //   rhs = -dxi/2 sum_d (u_d+ (phi+ + phi) - u_d (phi + phi-))                 advection
  //         + gamma eps ddxi (sum of the six neighbours - 6 phi)                diffusion
  //         - gamma dxi/2 sum_d (F_d+ - F_d-)                                   sharpening
  auto out_cell = [&](int cc, double p0, double pxp, double pxm, double pyp, double pym, double pzp, double pzm,
                      double u_0, double u_x, double v_0, double v_y, double w_0, double w_z, double shp, double ro) {
    const double adv = (__fma_rn(u_x, pxp + p0, -u_0 * (p0 + pxm)) + __fma_rn(v_y, pyp + p0, -v_0 * (p0 + pym))) +
                       __fma_rn(w_z, pzp + p0, -w_0 * (p0 + pzm));
    const double lap = ((pxp + pxm) + (pyp + pym)) + __fma_rn(-6.0, p0, pzp + pzm);
    const double rhs = __fma_rn(-hdxi, adv, __fma_rn(c_lap, lap, c_shp * shp));
    // :625-626
    a.phin[cc] = __fma_rn(dta, rhs, __fma_rn(-dtb, ro, p0));
    a.rphio[cc] = rhs;
  };

  // Iteration k computes psi(k+2), F(k+1) and the output plane k.  The loop starts four planes
  // below the chunk: k0-4 and k0-3 only fill psi(k0-2), psi(k0-1), k0-2 and k0-1 add F(k0-1),
  // F(k0).  Every psi and F is thus evaluated by the loop body, so the values of a plane do
  // not depend on where a z chunk starts.  Register state of each cell entering iteration k: phi
  // k-1..k+2, psi k, k+1, Fz k-1, k and Fy k.
  int o3 = pmodi(k0 - 2, nz) * plane + col;
  double fam1 = 0.0, fa0 = 0.0, fap1 = 0.0, fap2 = phig[o3];
  double fbm1 = 0.0, fb0 = 0.0, fbp1 = 0.0, fbp2 = phig[o3 + nx];
  double sa0 = 0.0, sap1 = 0.0, zam1 = 0.0, za0 = 0.0, ya0 = 0.0;
  double sb0 = 0.0, sbp1 = 0.0, zbm1 = 0.0, zb0 = 0.0, yb0 = 0.0;
  o3 = pmodi(k0 - 1, nz) * plane + col;  // phi(k+3) of the first iteration

  // One plane of the loop; P is the parity of k, so the double-buffer slots are compile-time
  // offsets: slot(k) = slot(k + 2) = P PPOS, slot(k + 1) = (1 - P) PPOS.
  auto plane_iter = [&](auto par, int k) {
    constexpr int P = decltype(par)::value;
    constexpr int SK = P * PPOS, SK1 = (1 - P) * PPOS;
    const bool out = orole && k >= k0;
    double fap3 = 0.0, fbp3 = 0.0;
    if (k + 1 < k1) {
      fap3 = phig[o3];
      fbp3 = phig[o3 + nx];
    }
    o3 += plane;
    if (o3 >= ntot) o3 -= ntot;
    // plane k+1's fields go out now; they land before the barrier that ends this iteration
    if (orole && k + 1 >= k0 && k + 1 < k1) stage(stg + (1 - P) * PSTG, k + 1, k >= k0 ? c + plane : c);
    __pipeline_commit();
    // psi(k+2) of both cells; phi(k+1) for the next plane's neighbours
    const double sap2 = psi_of(fap2), sbp2 = psi_of(fbp2);
    sps[SK] = sap2;
    sps[SK + PHX] = sbp2;
    sph[SK1] = fap1;
    sph[SK1 + PHX] = fbp1;
    // F(k+1) from the shared psi(k+1) (written last iteration) and the own psi(k+2) - psi(k)
    double zap1 = 0.0, zbp1 = 0.0, yap1 = 0.0, ybp1 = 0.0;
    if (k >= k0 - 2) {
      const double* Q = sps + SK1;
      double fx;
      if (fa) {
        F_of(Q[1] - Q[-1], sbp1 - Q[-PHX], sap2 - sa0, fap1, sap1, fx, yap1, zap1);
        sfx[SK1] = fx;
        sfy[SK1] = yap1;
      }
      if (fb) {
        F_of(Q[PHX + 1] - Q[PHX - 1], Q[2 * PHX] - sap1, sbp2 - sb0, fbp1, sbp1, fx, ybp1, zbp1);
        sfx[SK1 + PHX] = fx;
        sfy[SK1 + PHX] = ybp1;
      }
    }
    // output plane k from the shared phi(k), Fx/Fy(k) and the own columns
    if (out) {
      const double* P0 = sph + SK;
      const double* Fx = sfx + SK;
      const double* Fy = sfy + SK;
      const double* G = stg + P * PSTG;
      const double va = G[sv], vc = G[sv + 2 * PTX], ua = G[su], uax = G[su + 1], ub = G[su + PUX], ubx = G[su + PUX + 1];
      const double waz = G[sw], wbz = G[sw + PTX], roa = G[sr], rob = G[sr + PTX];
      const double v_b = G[sv + PTX] - mv_;
      out_cell(c, fa0, P0[1], P0[-1], fb0, P0[-PHX], fap1, fam1, ua - mu_, uax - mu_, va - mv_, v_b, wa0 - mw_,
               waz - mw_, ((Fx[1] - Fx[-1]) + (yb0 - Fy[-PHX])) + (zap1 - zam1), roa);
      out_cell(c + nx, fb0, P0[PHX + 1], P0[PHX - 1], P0[2 * PHX], fa0, fbp1, fbm1, ub - mu_, ubx - mu_, v_b, vc - mv_,
               wb0 - mw_, wbz - mw_, ((Fx[PHX + 1] - Fx[PHX - 1]) + (Fy[2 * PHX] - ya0)) + (zbp1 - zbm1), rob);
      wa0 = waz;
      wb0 = wbz;
      c += plane;
    }
    __pipeline_wait_prior(0);
    __syncthreads();
    fam1 = fa0, fa0 = fap1, fap1 = fap2, fap2 = fap3;
    fbm1 = fb0, fb0 = fbp1, fbp1 = fbp2, fbp2 = fbp3;
    sa0 = sap1, sap1 = sap2, sb0 = sbp1, sbp1 = sbp2;
    zam1 = za0, za0 = zap1, zbm1 = zb0, zb0 = zbp1;
    ya0 = yap1, yb0 = ybp1;
  };
  // k0 and the chunk are even (launch_phase), so k0 - 4 is even and the trip count too; two
  // planes per iteration
#pragma unroll PUNROLL
  for (int k = k0 - 4; k < k1; k += 2) {
    plane_iter(std::integral_constant<int, 0>{}, k);
    plane_iter(std::integral_constant<int, 1>{}, k + 1);
  }
}

template <bool CLAMP, typename L>
__global__ void __launch_bounds__(L::PNT, PMINB) k_phase(const __grid_constant__ PhaseArgs a) {
  extern __shared__ __align__(16) unsigned char smraw[];
  phase_tile<CLAMP, L>(a, a.dta, a.dtb, blockIdx.x, blockIdx.y, blockIdx.z, smraw);
}

// The phase step of many boxes in one launch: persistent blocks (one per SM) take work items
// (box, tile x, tile y, z chunk) from a device queue until it is empty.  A box's arguments
// (including its resolved z chunk) come from b.args; alpha, beta are the step's.  The boxes of
// one launch share the psi clamp (CLAMP).
template <bool CLAMP, typename L>
__global__ void __launch_bounds__(L::PNT, PMINB) k_phase_batch(const __grid_constant__ BatchArgs<PhaseArgs> b) {
  extern __shared__ __align__(16) unsigned char smraw[];
  __shared__ int s_item;
  for (;;) {
    if (threadIdx.x == 0) s_item = atomicAdd(b.counter, 1);
    __syncthreads();
    const int it = s_item;
    __syncthreads();  // every thread has the item before thread 0 takes the next one
    if (it >= b.nitems) break;
    const int4 w = b.items[it];
    const PhaseArgs& a = b.args[w.x];
    phase_tile<CLAMP, L>(a, a.g.dt * b.alpha, a.g.dt * b.beta, w.y, w.z, w.w, smraw);
  }
}

PhaseTiles phase_tiles(const Geo& g) {
  return g.ny > 32 ? PhaseTiles::Tall : (g.nx < 192 ? PhaseTiles::Flat : PhaseTiles::Wide);
}

// f(tile) of the box's tiles
template <typename F> static auto with_tiles(PhaseTiles t, F f) {
  return t == PhaseTiles::Tall ? f(Tall{}) : (t == PhaseTiles::Flat ? f(Flat{}) : f(Wide{}));
}

int phase_zchunk(const Geo& g, int requested, double share) {
  if (requested > 0) return requested;
  const dim3 t = phase_grid(g, g.nz);
  const long long cols = (long long)t.x * t.y;
  // The even chunk with the fewest planes in sequence on an SM: waves of one block on each of the
  // 148 SMs times the chunk with its four planes of warm-up (the shorter list of chunks on a tie).
  // With the 32 x 16 tiles of before and chunks of 64, then of the rule: 128^3 87 -> 50 us (32
  // planes), 192x64x128 83 -> 37 us (22), 256^3 345 -> 331 us (32); with the 32 x 24 tiles 45 us
  // (22), 36 us (16) and 254 us (52), 512^3 104 planes.
  // The boxes of an ensemble share the chip: the rule takes the columns of all of them, as if they were
  // boxes like this one.  A chunk of 64 whatever the number of boxes left SMs idle (steps, from 64
  // to the rule's: 16 boxes of 64^3 432 -> 405 us, 4 of 64^3 224 -> 142, 2 of 128^3 423 -> 392).
  // Results do not depend on the chunk.
  return best_zchunk(g.nz, (long long)(cols * share), 148, 4);
}

dim3 phase_grid(const Geo& g, int zc) {
  return with_tiles(phase_tiles(g), [&](auto t) {
    return dim3((g.nx + t.PTX - 1) / t.PTX, (g.ny + t.PTY - 1) / t.PTY, (g.nz + zc - 1) / zc);
  });
}

template <typename L>
static cudaError_t launch_batch(const BatchArgs<PhaseArgs>& b, bool clamp, int nsm, cudaStream_t st) {
  constexpr size_t smem = L::PSMEM;
  auto kern = clamp ? k_phase_batch<true, L> : k_phase_batch<false, L>;
  cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return e;
  e = cudaMemsetAsync(b.counter, 0, sizeof(int), st);
  if (e != cudaSuccess) return e;
  kern<<<b.nitems < nsm ? b.nitems : nsm, L::PNT, smem, st>>>(b);
  return cudaGetLastError();
}

cudaError_t launch_phase_batch(const BatchArgs<PhaseArgs>& b, PhaseTiles tiles, bool clamp, int nsm, cudaStream_t st) {
  return with_tiles(tiles, [&](auto t) { return launch_batch<decltype(t)>(b, clamp, nsm, st); });
}

template <typename L> static cudaError_t launch_one(const PhaseArgs& a, cudaStream_t st) {
  constexpr size_t smem = L::PSMEM;
  auto kern = a.clamp ? k_phase<true, L> : k_phase<false, L>;
  static int attr_set[64][2] = {};
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev >= 64 || !attr_set[dev][a.clamp ? 1 : 0]) {
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
    if (dev < 64) attr_set[dev][a.clamp ? 1 : 0] = 1;
  }
  PhaseArgs b = a;
  b.dta = a.g.dt * a.alpha;
  b.dtb = a.g.dt * a.beta;
  b.zchunk = phase_zchunk(a.g, a.zchunk, a.share);
  const int zc = b.zchunk;
  if (zc % 2 || a.g.nz % 2) return cudaErrorInvalidValue;  // the plane loop runs two planes at a time
  kern<<<phase_grid(a.g, zc), L::PNT, smem, st>>>(b);
  return cudaGetLastError();
}

cudaError_t launch_phase(const PhaseArgs& a, cudaStream_t st) {
  return with_tiles(phase_tiles(a.g), [&](auto t) { return launch_one<decltype(t)>(a, st); });
}

}  // namespace mhit
