// Droplet labelling: the connected components of phi >= thresh with periodic boundaries and
// their statistics, as post/unionfind_periodic/main.f90 computes them (mask :137-151, 6- or
// 26-neighbour connectivity :33-48, periodic halos :152-157/:251-258, per-drop volume, circular
// mean centre and mean velocity :276-336, volume = cells dx^3 :436).
//
// The reference iterates min-label propagation over 16^3 tiles until nothing changes.  Here the
// components come from a lock-free union-find over the cell indices (Playne and Hawick, "A New
// Algorithm for Parallel Connected-Component Labelling on GPUs", IEEE TPDS 2018): every masked
// cell starts as its own root; for each masked neighbour pair the two roots are joined by an
// atomicMin that hangs the larger root under the smaller, so the final root of a component is its
// smallest cell index (k, j, i order) whatever the scheduling; a flatten pass points every cell at
// its root.  Drops are numbered by that smallest index, so the order is deterministic.
//
// Every loop that follows parent pointers or retries a link is bounded (a chain or a retry
// sequence can never be longer than the number of cells); hitting the bound sets an error flag
// that the host turns into an error status instead of looping.
//
// Most cells are background, so every pass is a scan of the label field (0.08 ms at 512^3, 4 bytes
// per cell), and with one cell per thread and iteration the latency of those loads bounds it.  The
// mask and the statistics take four consecutive cells per thread (nx is a multiple of 16) with one
// 16-byte load and skip the groups without a masked cell; the merge and the flatten pass have four
// loads of consecutive lanes in flight, because there the masked cells' work counts: with four
// consecutive cells per thread, one after the other, they took up to four times as long.  Merge and
// flatten, us, one cell per thread / four consecutive / now (64 drops at 64^3 and 256^3, all of
// 64^3, a 256^3 box filled to a third, 64 drops at 512^3):
//   18 / 58 / 19    157 / 224 / 138    97 / 473 / 107    503 / 1193 / 611    837 / 706 / 601
// and the statistics 14 / 8, 184 / 82, 92 / 25, 1790 / 460, 1099 / 417 (the first and the last two).
#include "common.cuh"
#include "kernels.h"

namespace mhit {

// forward half of the neighbourhood (dz, dy, dx): the other half is reached from the neighbour
__constant__ int8_t c_fwd[13][3] = {{0, 0, 1},  {0, 1, 0},  {1, 0, 0},  {0, 1, 1},  {0, 1, -1},
                                    {1, 0, 1},  {1, 0, -1}, {1, 1, 0},  {1, -1, 0}, {1, 1, 1},
                                    {1, 1, -1}, {1, -1, 1}, {1, -1, -1}};

// Root of x with path halving: each visited node is re-pointed at its grandparent.  A node's
// ancestors stay its ancestors (roots are only ever hung under smaller roots) and parents only
// decrease, so a plain store of the grandparent is safe under concurrent links and halvings.
// ATOMIC: stored by an atomicMin (k_lab_flatten).
template <bool ATOMIC = false>
__device__ __forceinline__ int find_root(int* lab, int x, long long bound, int* err) {
  volatile int* vl = lab;  // parents change under concurrent links: read them from L2
  for (long long it = 0; it < bound; ++it) {
    const int y = vl[x];
    if (y == x) return x;
    const int z = vl[y];
    if (z == y) return y;
    if (ATOMIC) atomicMin(&lab[x], z);
    else vl[x] = z;
    x = z;
  }
  atomicExch(err, 1);
  return x;
}

__device__ __forceinline__ void unite(int* lab, int a, int b, long long bound, int* err) {
  for (long long it = 0; it < bound; ++it) {
    a = find_root(lab, a, bound, err);
    b = find_root(lab, b, bound, err);
    if (a == b) return;
    if (a > b) {
      const int t = a;
      a = b;
      b = t;
    }
    const int old = atomicMin(&lab[b], a);
    if (old == b) return;  // b was still a root and now hangs under a
    b = old;               // b was linked meanwhile: continue from its new parent
  }
  atomicExch(err, 1);
}

__global__ void k_lab_init(const double* __restrict__ phi, double thresh, int* __restrict__ lab, int n) {
  for (int c = 4 * (blockIdx.x * blockDim.x + threadIdx.x); c < n; c += 4 * gridDim.x * blockDim.x) {
    const double2 p = *reinterpret_cast<const double2*>(phi + c), q = *reinterpret_cast<const double2*>(phi + c + 2);
    // post/unionfind_periodic/main.f90:141
    *reinterpret_cast<int4*>(lab + c) = make_int4(p.x >= thresh ? c : -1, p.y >= thresh ? c + 1 : -1,
                                                  q.x >= thresh ? c + 2 : -1, q.y >= thresh ? c + 3 : -1);
  }
}

// R: cells per lane and iteration, each a row of 32 cells of the warp.  Four from 2^22 cells on (512^3
// 605 -> 494 us, 256^3 122 -> 106 for 64 drops); below, where that leaves too few warps, one (128^3 87 ->
// 71, 64^3 28 -> 14).
template <int R>
__global__ void k_lab_merge(int* lab, int nx, int ny, int nz, int nfwd, long long bound, int* err) {
  const int n = nx * ny * nz;
  const int lane = threadIdx.x & 31, warps = gridDim.x * (blockDim.x >> 5);
  for (int c0 = 32 * R * (blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5)) + lane; c0 < n; c0 += 32 * R * warps) {
    int l[R];
#pragma unroll
    for (int r = 0; r < R; ++r) l[r] = __ldcg(lab + c0 + 32 * r);  // n is a multiple of 128
#pragma unroll
    for (int r = 0; r < R; ++r) {
      // parents change under concurrent links, masked (>= 0) or not does not
      if (l[r] < 0) continue;
      const int c = c0 + 32 * r;
      const int i = c % nx, j = (c / nx) % ny, k = c / (nx * ny);
      for (int q = 0; q < nfwd; ++q) {
        int ii = i + c_fwd[q][2], jj = j + c_fwd[q][1], kk = k + c_fwd[q][0];
        ii = ii < 0 ? ii + nx : (ii >= nx ? ii - nx : ii);
        jj = jj < 0 ? jj + ny : (jj >= ny ? jj - ny : jj);
        kk = kk >= nz ? kk - nz : kk;
        const int d = (kk * ny + jj) * nx + ii;
        if (d != c && lab[d] >= 0) unite(lab, c, d, bound, err);
      }
    }
  }
}

constexpr int LTHREADS = 256, LCHUNK = 8192;  // threads and cells of a block of the chunked passes

// Every masked cell points at its root afterwards; adds the roots of each chunk of LCHUNK consecutive
// cells to its count (zero before).  A block takes `part` cells, a divisor of LCHUNK.  Halvings store
// with an atomicMin: a plain store could put back a grandparent over a root that the cell's own
// thread has just stored.  Without halving, a chain is walked by every cell on it (rods of 64 cells
// at 64^3 50 us, now 14).
__global__ void __launch_bounds__(LTHREADS) k_lab_flatten(int* lab, int n, int part, long long bound, int* err,
                                                          int* __restrict__ counts) {
  __shared__ int s;
  if (threadIdx.x == 0) s = 0;
  __syncthreads();
  const int p0 = blockIdx.x * part, p1 = min(p0 + part, n);
  int local = 0;
  for (int c = p0 + threadIdx.x; c < p1; c += 4 * LTHREADS) {
    int l[4];
#pragma unroll
    for (int r = 0; r < 4; ++r) l[r] = c + r * LTHREADS < p1 ? __ldcg(lab + c + r * LTHREADS) : -1;
#pragma unroll
    for (int r = 0; r < 4; ++r) {
      if (l[r] < 0) continue;
      const int e = c + r * LTHREADS;
      if (l[r] == e) ++local;  // roots stay roots in this pass
      else lab[e] = find_root<true>(lab, l[r], bound, err);
    }
  }
  if (local) atomicAdd(&s, local);
  __syncthreads();
  if (threadIdx.x == 0 && s) atomicAdd(&counts[p0 / LCHUNK], s);
}

// Number the roots in index order (offsets: the first number of each chunk and the total; chunks
// without a root, nearly all of them, have nothing to do): the root of drop d (0-based) gets
// -(d + 2), so that any cell finds its drop as -lab[lab[c]] - 2 (or -lab[c] - 2 at the root itself)
__global__ void k_lab_number(int* __restrict__ lab, int n, const int* __restrict__ offsets) {
  __shared__ int warp_tot[LTHREADS / 32];
  __shared__ int base;
  if (offsets[blockIdx.x + 1] == offsets[blockIdx.x]) return;
  if (threadIdx.x == 0) base = offsets[blockIdx.x];
  __syncthreads();
  const int c0 = blockIdx.x * LCHUNK, c1 = min(c0 + LCHUNK, n);
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  for (int t0 = c0; t0 < c1; t0 += LTHREADS) {
    const int c = t0 + threadIdx.x;
    const int root = (c < c1 && lab[c] == c) ? 1 : 0;
    const unsigned bal = __ballot_sync(0xffffffffu, root);
    const int before = __popc(bal & ((1u << lane) - 1u));
    if (lane == 0) warp_tot[wid] = __popc(bal);
    __syncthreads();
    int wbase = 0;
    for (int q = 0; q < wid; ++q) wbase += warp_tot[q];
    if (root) lab[c] = -(base + wbase + before + 2);
    __syncthreads();
    if (threadIdx.x == 0) {
      int tot = 0;
      for (int q = 0; q < LTHREADS / 32; ++q) tot += warp_tot[q];
      base += tot;
    }
    __syncthreads();
  }
}

__device__ __forceinline__ int drop_of(const int* lab, int c) {
  const int r = lab[c];
  if (r == -1) return -1;
  return r < -1 ? -r - 2 : -lab[r] - 2;
}

// per drop: cells, sums of sin/cos of the cell centre per axis, sums of u, v, w
// (post/unionfind_periodic/main.f90:302-315); acc is [ndrops][9].  Cells of one drop are
// contiguous along x, so the 128 cells a warp visits (four per lane) mostly belong to one or two
// drops: each lane adds up its cells of one drop, the lanes of a drop are grouped (match_any) and
// sum their values with shuffles, and one lane per group does the atomics -- a drop of 10^5 cells
// would otherwise serialise 10^6 atomics on nine addresses.
__global__ void k_lab_stats(const int* __restrict__ lab, int nx, int ny, int nz, const double* __restrict__ u,
                            const double* __restrict__ v, const double* __restrict__ w,
                            const double* __restrict__ trig, const DevScalars* __restrict__ sc,
                            double* __restrict__ acc, unsigned long long* __restrict__ cells) {
  const int n = nx * ny * nz;
  const double mu_ = sc->mean[0], mv_ = sc->mean[1], mw_ = sc->mean[2];
  // trig: sin x (nx), cos x (nx), sin y (ny), cos y (ny), sin z (nz), cos z (nz)
  const double* sx = trig;
  const double* cxs = sx + nx;
  const double* sy = cxs + nx;
  const double* cys = sy + ny;
  const double* sz = cys + ny;
  const double* czs = sz + nz;
  const int lane = threadIdx.x & 31;
  const int warps = gridDim.x * (blockDim.x >> 5);
  // warp-uniform loops: all 32 lanes take part in every match and shuffle
  for (int base = (blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5)) * 128; base < n; base += warps * 128) {
    const int c = base + 4 * lane;
    int4 l = make_int4(-1, -1, -1, -1);
    if (c < n) l = __ldg(reinterpret_cast<const int4*>(lab + c));
    int d4[4] = {l.x, l.y, l.z, l.w};
    bool some = d4[0] != -1 || d4[1] != -1 || d4[2] != -1 || d4[3] != -1;
    if (!__any_sync(0xffffffffu, some)) continue;  // background only (most warps)
    const int i = c % nx, j = (c / nx) % ny, k = c / (nx * ny);
#pragma unroll
    for (int e = 0; e < 4; ++e) d4[e] = d4[e] == -1 ? -1 : (d4[e] < -1 ? -d4[e] - 2 : -lab[d4[e]] - 2);
    // one drop of each lane per round (a second round only where a lane's four cells meet two drops)
    while (__any_sync(0xffffffffu, some)) {
      int d = -1, cnt = 0;
      double sum[9];
#pragma unroll
      for (int q = 0; q < 9; ++q) sum[q] = 0.0;
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        if (d4[e] < 0 || (d >= 0 && d4[e] != d)) continue;
        d = d4[e];
        d4[e] = -1;
        ++cnt;
        sum[0] += sx[i + e];
        sum[1] += cxs[i + e];
        sum[6] += u[c + e] - mu_;
        sum[7] += v[c + e] - mv_;
        sum[8] += w[c + e] - mw_;
      }
      if (cnt) {
        sum[2] = cnt * sy[j];
        sum[3] = cnt * cys[j];
        sum[4] = cnt * sz[k];
        sum[5] = cnt * czs[k];
      }
      some = d4[0] >= 0 || d4[1] >= 0 || d4[2] >= 0 || d4[3] >= 0;
      const unsigned grp = __match_any_sync(0xffffffffu, d), with = __ballot_sync(0xffffffffu, d >= 0);
      const bool lead = d >= 0 && lane == __ffs(grp) - 1;
      if (__popc(__ballot_sync(0xffffffffu, lead)) == 1) {
        // one drop in the warp: a shuffle tree over all lanes (the others hold zeros)
        const int first = __ffs(with) - 1;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
          cnt += __shfl_xor_sync(0xffffffffu, cnt, o);
#pragma unroll
          for (int q = 0; q < 9; ++q) sum[q] += __shfl_xor_sync(0xffffffffu, sum[q], o);
        }
        if (lane == first) {
          double* a = acc + (size_t)d * 9;
          atomicAdd(&cells[d], (unsigned long long)cnt);
#pragma unroll
          for (int q = 0; q < 9; ++q) atomicAdd(a + q, sum[q]);
        }
      } else {
        double all[9];
        int nall = 0;
#pragma unroll
        for (int q = 0; q < 9; ++q) all[q] = 0.0;
        // every lane of a group walks the same lanes in the same order: the sums are identical
        for (unsigned m = grp; m; m &= m - 1) {
          const int from = __ffs(m) - 1;
          nall += __shfl_sync(grp, cnt, from);
#pragma unroll
          for (int q = 0; q < 9; ++q) all[q] += __shfl_sync(grp, sum[q], from);
        }
        __syncwarp();
        if (lead) {
          double* a = acc + (size_t)d * 9;
          atomicAdd(&cells[d], (unsigned long long)nall);
#pragma unroll
          for (int q = 0; q < 9; ++q) atomicAdd(a + q, all[q]);
        }
      }
    }
  }
}

// label field for the host: 0 background, 1.. drop number
__global__ void k_lab_final(const int* __restrict__ lab, int* __restrict__ out, int n) {
  for (int c = blockIdx.x * blockDim.x + threadIdx.x; c < n; c += gridDim.x * blockDim.x) out[c] = drop_of(lab, c) + 1;
}

int label_chunks(int n) { return (n + LCHUNK - 1) / LCHUNK; }

cudaError_t launch_label_components(const LabelArgs& a, cudaStream_t st) {
  const int n = a.nx * a.ny * a.nz;
  const int grid = 148 * 8;
  k_lab_init<<<grid, 256, 0, st>>>(a.phi, a.thresh, a.lab, n);
  // the loops' bound: the cell count (no chain or retry sequence is longer), or a smaller test
  // bound that makes a legitimate chain run out and exercises the error path
  const long long bound = a.bound > 0 ? a.bound : n;
  const auto merge = n >= (1 << 22) ? k_lab_merge<4> : k_lab_merge<1>;
  merge<<<grid, 256, 0, st>>>(a.lab, a.nx, a.ny, a.nz, a.connectivity == 26 ? 13 : 3, bound, a.err);
  // whole chunks where they fill the chip (eight blocks per SM); 64^3 has 32 of them
  const int part = label_chunks(n) >= 148 * 8 ? LCHUNK : LCHUNK / 8;
  k_lab_flatten<<<(n + part - 1) / part, LTHREADS, 0, st>>>(a.lab, n, part, bound, a.err, a.counts);
  return cudaGetLastError();
}

cudaError_t launch_label_number(const LabelArgs& a, cudaStream_t st) {
  const int n = a.nx * a.ny * a.nz;
  k_lab_number<<<label_chunks(n), LTHREADS, 0, st>>>(a.lab, n, a.counts);
  return cudaGetLastError();
}

cudaError_t launch_label_stats(const LabelArgs& a, cudaStream_t st) {
  const int n = a.nx * a.ny * a.nz;
  k_lab_stats<<<148 * 8, 256, 0, st>>>(a.lab, a.nx, a.ny, a.nz, a.u, a.v, a.w, a.trig, a.sc, a.acc, a.cells);
  if (a.out) k_lab_final<<<148 * 8, 256, 0, st>>>(a.lab, a.out, n);
  return cudaGetLastError();
}

}  // namespace mhit
