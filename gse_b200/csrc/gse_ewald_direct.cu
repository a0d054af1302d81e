// gse_ewald_direct.cu -- FP64 Ewald direct (real-space) sum on the GPU.
//
// CpuEwaldDirect::calcForceEnergy (CpuEwaldDirect.cpp:45-131): over the
// pairs (i, j) at minimum-image distance r < rcut that are not excluded,
//   E    = sum ccelec q_i q_j erfc(r / (sqrt2 sigma)) / r
//          - ccelec / sqrt(2 pi sigma^2) sum_i q_i^2,
//   f_ij = -ccelec q_i q_j (2 / sqrt(pi) / (sqrt2 sigma) exp(-r^2 / 2 sigma^2)
//          + erfc(r / (sqrt2 sigma)) / r) / r^2,
//   F_i  = sum_j f_ij (x_i - x_j)            (the gradient dE/dx_i).
// The pair (a, b), a < b, is excluded when b + 1 = |inb14[k]| for some k in
// [iblo14[a - 1], iblo14[a]) (CpuEwaldDirect.cpp:31-40, :71-85); the host
// turns those lists into one sorted list per atom holding both partners.
//
// Atoms are binned into cells of side >= rcut, stably (original order within
// a cell).  A CTA takes up to 32 of a cell's atoms as i and stages the atoms of
// the neighbouring cells (the 3 nearest along an axis with at least 3 cells,
// every cell along a shorter one) in shared memory as j.  A warp tests all of
// them against two atoms at a time, lane by lane, and queues the ones inside
// the cut-off; whenever a queue holds 32, all lanes form one pair term each.
// Every pair term is formed by both partners, so each atom's force and half of
// its pair energies are summed by one warp in a fixed order: the results do
// not depend on scheduling.
//
// Bound: FP64 arithmetic.  A tenth of the staged atoms lie inside the cut-off
// (the sphere in 27 cells), so with a lane per i nearly every step of a warp
// took the whole erfc/exp/division path for a few lanes, at 216 blocks for
// 23,559 charges: 3.20 ms; with queues 0.55 ms.
#include <cuda_runtime.h>
#include <math.h>

#include <algorithm>

#include "gse_ewald.cuh"
#include "gse_internal.cuh"
#include "gse_reduce.cuh"
#include "gse_tiled.cuh"

namespace gse {

constexpr int kEwdThreads = 256;
constexpr int kEwdI = 32;     // atoms i per block and round
constexpr int kEwdTile = 3072;  // staged atoms j (112 KB: two blocks per SM)

// Cell index of a coordinate along one axis: the position taken into
// [0, box) and scaled by nc / box, clamped to [0, nc).
__device__ __forceinline__ int ewd_cell_axis(double x, double box, double inv_box, int nc) {
  const double w = x - box * floor(x * inv_box);
  const int c = (int)(w * inv_box * (double)nc);
  return c < 0 ? 0 : (c >= nc ? nc - 1 : c);
}

// Also lists the cells that hold atoms, in any order, and clears the partial energies.
__global__ void k_ewd_cell_count(const double4* __restrict__ xyzq, int n, EwdGeom g,
                                 int* __restrict__ key, int* __restrict__ counts,
                                 int* __restrict__ rank, int* __restrict__ cells,
                                 unsigned* __restrict__ used, double* __restrict__ partials) {
  pdl_trigger();
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    const double4 p = xyzq[i];
    const int cx = ewd_cell_axis(p.x, g.box[0], g.inv_box[0], g.nc[0]);
    const int cy = ewd_cell_axis(p.y, g.box[1], g.inv_box[1], g.nc[1]);
    const int cz = ewd_cell_axis(p.z, g.box[2], g.inv_box[2], g.nc[2]);
    const int k = cx + g.nc[0] * (cy + g.nc[1] * cz);
    key[i] = k;
    const int r = atomicAdd(&counts[k], 1);
    rank[i] = r;
    if (r == 0) cells[atomicAdd(used, 1u)] = k;
    partials[i] = 0.0;
  }
}

// The minimum image of d as the reference's while loops leave it: within
// [-box/2, box/2], a difference of exactly +-box/2 kept as it is.
__device__ __forceinline__ double ewd_min_image(double d, double box, double hbox,
                                                double inv_box) {
  if (fabs(d) > hbox) {
    d -= box * rint(d * inv_box);
    if (d < -hbox) d += box;
    if (d > hbox) d -= box;
  }
  return d;
}

__global__ void __launch_bounds__(kEwdThreads, 2)
    k_ewd_pairs(const double4* __restrict__ sorted, const int* __restrict__ perm,
                const int* __restrict__ start, const int* __restrict__ cells,
                const unsigned* __restrict__ used, int n, EwdGeom g, int split,
                const int* __restrict__ ex_start, const int* __restrict__ ex_idx,
                double* __restrict__ fx, double* __restrict__ fy, double* __restrict__ fz,
                double* __restrict__ partials, unsigned* done, double* __restrict__ energy_out) {
  constexpr int NW = kEwdThreads / 32;
  extern __shared__ __align__(16) double ewd_sm[];
  double *sx = ewd_sm, *sy = sx + kEwdTile, *sz = sy + kEwdTile, *sq = sz + kEwdTile;
  int* sid = reinterpret_cast<int*>(sq + kEwdTile);
  __shared__ double facc[kEwdI][3];
  __shared__ unsigned short queue[NW][2][64];
  __shared__ int nbr_a[27], nbr_p[28];  // neighbour cells' first atoms, their prefix
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int part = blockIdx.x % split;
  const bool on = blockIdx.x / split < *used;
  const int cell = on ? cells[blockIdx.x / split] : 0;
  const int i0 = on ? start[cell] + kEwdI * part : 0, i1 = on ? start[cell + 1] : 0;
  double esum = 0.0;
  if (i0 < i1) {
    const int c[3] = {cell % g.nc[0], (cell / g.nc[0]) % g.nc[1], cell / (g.nc[0] * g.nc[1])};
    int lo[3], cnt[3];
#pragma unroll
    for (int d = 0; d < 3; d++) {
      lo[d] = g.nc[d] >= 3 ? c[d] - 1 + g.nc[d] : 0;
      cnt[d] = g.nc[d] >= 3 ? 3 : g.nc[d];
    }
    const int nnb = cnt[0] * cnt[1] * cnt[2];
    if (tid < 32) {  // one warp: ranges of the neighbour cells and their prefix
      int a = 0, m = 0;
      if (tid < nnb) {
        const int ox = tid % cnt[0], oy = tid / cnt[0] % cnt[1], oz = tid / (cnt[0] * cnt[1]);
        const int nb = (lo[0] + ox) % g.nc[0] +
                       g.nc[0] * ((lo[1] + oy) % g.nc[1] + g.nc[1] * ((lo[2] + oz) % g.nc[2]));
        a = start[nb];
        m = start[nb + 1] - a;
      }
      int run = m;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int y = __shfl_up_sync(0xffffffffu, run, o);
        if (lane >= o) run += y;
      }
      if (tid < nnb) {
        nbr_a[tid] = a;
        nbr_p[tid] = run - m;
      }
      if (tid == nnb - 1) nbr_p[nnb] = run;
    }
    __syncthreads();
    const int total = nbr_p[nnb];
    for (int ib = i0; ib < i1; ib += kEwdI * split) {
      const int ni = min(kEwdI, i1 - ib);
      for (int t0 = 0; t0 < total; t0 += kEwdTile) {
        const int nt = min(kEwdTile, total - t0);
        __syncthreads();  // the previous tile is consumed
        if (t0 == 0 && tid < kEwdI) facc[tid][0] = facc[tid][1] = facc[tid][2] = 0.0;
        if (t0 > 0 || ib == i0 || total > kEwdTile)
          for (int r = warp; r < nnb; r += NW) {
            const int p0 = max(nbr_p[r], t0), p1 = min(nbr_p[r + 1], t0 + nt);
            for (int p = p0 + lane; p < p1; p += 32) {
              const int src = nbr_a[r] + (p - nbr_p[r]);
              const double4 v = sorted[src];
              sx[p - t0] = v.x;
              sy[p - t0] = v.y;
              sz[p - t0] = v.z;
              sq[p - t0] = v.w;
              sid[p - t0] = perm[src];
            }
          }
        __syncthreads();
        for (int k = 2 * warp; k < ni; k += 2 * NW) {
          double4 pi[2];
          int oi[2], e0[2] = {0, 0}, e1[2] = {0, 0};
#pragma unroll
          for (int u = 0; u < 2; u++) {
            const int i = ib + min(k + u, ni - 1);
            pi[u] = sorted[i];
            oi[u] = perm[i];
            if (ex_start) {
              e0[u] = ex_start[oi[u]];
              e1[u] = ex_start[oi[u] + 1];
            }
          }
          double f[2][3] = {{0.0, 0.0, 0.0}, {0.0, 0.0, 0.0}};
          // the term of pair (i, tile entry j)
          auto term = [&](int u, int j) {
            const int oj = sid[j];
            if (oj == oi[u]) return;
            bool excl = false;
            for (int e = e0[u]; e < e1[u]; e++) excl |= ex_idx[e] == oj;
            if (excl) return;
            const double dx = ewd_min_image(pi[u].x - sx[j], g.box[0], g.hbox[0], g.inv_box[0]);
            const double dy = ewd_min_image(pi[u].y - sy[j], g.box[1], g.hbox[1], g.inv_box[1]);
            const double dz = ewd_min_image(pi[u].z - sz[j], g.box[2], g.hbox[2], g.inv_box[2]);
            const double r2 = dx * dx + dy * dy + dz * dz;
            const double qq = g.ccelec * pi[u].w * sq[j];
            const double r = sqrt(r2);
            const double erfcval = erfc(r * g.inv_sqrt2sigma);
            const double expval = exp(-r2 * g.inv_2sigmasq);
            const double w = -qq * (g.two_sqrtpi * g.inv_sqrt2sigma * expval + erfcval / r) / r2;
            f[u][0] += w * dx;
            f[u][1] += w * dy;
            f[u][2] += w * dz;
            esum += 0.5 * (qq * erfcval / r);
          };
          int nq[2] = {0, 0};
          for (int base = 0; base < nt; base += 32) {
            const int j = base + lane;
            bool hit[2] = {false, false};
            if (j < nt) {
              const double x = sx[j], y = sy[j], z = sz[j];
#pragma unroll
              for (int u = 0; u < 2; u++) {
                const double dx = ewd_min_image(pi[u].x - x, g.box[0], g.hbox[0], g.inv_box[0]);
                const double dy = ewd_min_image(pi[u].y - y, g.box[1], g.hbox[1], g.inv_box[1]);
                const double dz = ewd_min_image(pi[u].z - z, g.box[2], g.hbox[2], g.inv_box[2]);
                hit[u] = dx * dx + dy * dy + dz * dz < g.rcut2 && k + u < ni;
              }
            }
#pragma unroll
            for (int u = 0; u < 2; u++) {
              const unsigned m = __ballot_sync(0xffffffffu, hit[u]);
              unsigned short* q = queue[warp][u];
              if (hit[u]) q[nq[u] + __popc(m & ((1u << lane) - 1u))] = (unsigned short)j;
              nq[u] += __popc(m);
              if (nq[u] >= 32) {  // uniform in the warp
                nq[u] -= 32;
                __syncwarp();
                const int jj = q[lane], rest = lane < nq[u] ? q[32 + lane] : 0;
                __syncwarp();
                // only what is left moves: the next step's lanes write from q[nq] on,
                // with no barrier between
                if (lane < nq[u]) q[lane] = (unsigned short)rest;
                term(u, jj);
              }
            }
          }
          __syncwarp();
#pragma unroll
          for (int u = 0; u < 2; u++) {
            if (lane < nq[u]) term(u, queue[warp][u][lane]);
            const double ax = warp_sum(f[u][0]), ay = warp_sum(f[u][1]), az = warp_sum(f[u][2]);
            if (lane == 0 && k + u < ni) {
              facc[k + u][0] += ax;
              facc[k + u][1] += ay;
              facc[k + u][2] += az;
            }
          }
          __syncwarp();
        }
      }
      __syncthreads();
      if (tid < ni) {
        const double q = sorted[ib + tid].w;
        if (fx) {
          const int o = perm[ib + tid];
          fx[o] = facc[tid][0];
          fy[o] = facc[tid][1];
          fz[o] = facc[tid][2];
        }
        esum += g.self * q * q;
      }
    }
  }
  // the block's energy at the place of one of its cell's atoms, whichever block took
  // the cell: the order of the sum does not depend on the list's
  if (i0 < i1) block_sum_at(esum, partials + start[cell] + part);
  last_block_sum_n(partials, n, done, 1.0, energy_out);
}

EwdGeom ewald_direct_geom(double sigma, double rcut, const double box[3], double ccelec) {
  EwdGeom g;
  long long cells = 1;
  for (int d = 0; d < 3; d++) {
    g.box[d] = box[d];
    g.hbox[d] = 0.5 * box[d];
    g.inv_box[d] = 1.0 / box[d];
    // a relative margin keeps the side >= rcut through the rounding of the
    // cell index
    const double q = box[d] / (rcut * (1.0 + 1e-9));
    g.nc[d] = q >= (double)kEwdMaxCellsPerAxis ? kEwdMaxCellsPerAxis : (q < 1.0 ? 1 : (int)q);
    cells *= g.nc[d];
  }
  g.ncell = (int)cells;
  g.rcut2 = rcut * rcut;
  g.inv_sqrt2sigma = 1.0 / (std::sqrt(2.0) * sigma);
  g.inv_2sigmasq = 1.0 / (2.0 * sigma * sigma);
  g.two_sqrtpi = 2.0 / std::sqrt(kPi);
  g.self = -ccelec / std::sqrt(2.0 * kPi * sigma * sigma);
  g.ccelec = ccelec;
  return g;
}

// Blocks per cell: one per 32 atoms of a cell of mean size; a fuller cell's blocks
// take several rounds.
static int ewald_direct_split(int n, const EwdGeom& g) {
  const long long per = ((long long)n + g.ncell - 1) / g.ncell;
  return (int)std::max<long long>(1, std::min<long long>((per + kEwdI - 1) / kEwdI, 64));
}

cudaError_t launch_ewald_direct(const double4* xyzq, int n, const EwdGeom& g, EwdScratch w,
                                const int* ex_start, const int* ex_idx, double* fx, double* fy,
                                double* fz, double* energy_out, cudaStream_t st) {
  cudaError_t e = cudaMemsetAsync(w.counts, 0, sizeof(int) * g.ncell, st);
  if (e != cudaSuccess) return e;
  e = cudaMemsetAsync(w.done, 0, 2 * sizeof(unsigned), st);  // done, used
  if (e != cudaSuccess) return e;
  const int gb = (int)std::min<long long>(sm_count() * 8, ((long long)n + 255) / 256);
  k_ewd_cell_count<<<gb, 256, 0, st>>>(xyzq, n, g, w.key, w.counts, w.perm, w.cells,
                                       w.done + 1, w.partials);
  BinScratch b = {};
  b.key = w.key;
  b.counts = w.counts;
  b.start = w.start;
  b.tile_sums = w.tile_sums;
  b.tmp = w.tmp;
  b.lstart = w.lstart;
  e = launch_bin_scan_place<double>(xyzq, n, g.ncell, b, w.sorted, w.perm, st);
  if (e != cudaSuccess) return e;
  const size_t smem = kEwdTile * (4 * sizeof(double) + sizeof(int));
  e = cudaFuncSetAttribute(k_ewd_pairs, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return e;
  // no more cells than atoms hold any: a block per cell of a wide, empty box (1.4 million
  // for 1000 atoms in 100 A at a cut-off of 0.9) took 7.2 ms of launches, 3.8 with the
  // former kernel's smaller blocks; now 0.13
  const int split = ewald_direct_split(n, g);
  k_ewd_pairs<<<std::min(n, g.ncell) * split, kEwdThreads, smem, st>>>(
      w.sorted, w.perm, w.start, w.cells, w.done + 1, n, g, split, ex_start, ex_idx, fx, fy, fz,
      w.partials, w.done, energy_out);
  return cudaGetLastError();
}

}  // namespace gse
