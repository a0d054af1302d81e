// gse_tiled.cu -- the tiled spread and gather kernels of the GSE-k path.
//
//  binning   atoms are counting-sorted by (z cell, y cell, x-bin of 4 or 16 cells)
//            of their stencil centre round(x/h) mod M; the FP64 form keeps the
//            original order within a bin so that its sums run in a fixed
//            order, the mixed form's integer sums need no order.
//  spread    CpuGaussCharge::spreadChargeToGrid (CpuGaussCharge.cpp:235-384),
//            mixed form: atom-stationary scatter into an int32 shared brick
//            tile, added into an int64 grid (scatter_brick).  The FP64 form's
//            output-stationary spread is in gse_spread64.cu.
//  gather    CpuGaussCharge::interpolateLoop (CpuGaussCharge.cpp:105-172): a
//            CTA owns the atoms of a kGX x kGY x kGZ-cell brick and stages the
//            potential of the brick plus its n-cell halo in shared memory;
//            kGatherLanes lanes per atom, over one list per block of the
//            (y, z) rows that an atom's sphere can reach.
#include <atomic>
#include <type_traits>

#include <cooperative_groups.h>

#include "gse_internal.cuh"
#include "gse_smallfft.cuh"
#include "gse_tiled.cuh"
#include "gse_tiled_dev.cuh"

namespace gse {

// ===========================================================================
// Binning
// ===========================================================================
template <typename V>
__device__ __forceinline__ int bin_of(const V& a, const BinLayout& b, decltype(V::x) inv_hx,
                                      decltype(V::x) inv_hy, decltype(V::x) inv_hz,
                                      int* __restrict__ bad) {
  if (bad && !(isfinite(a.x) && isfinite(a.y) && isfinite(a.z) && isfinite(a.w)))
    *bad = kFlagNonFinite;  // the bin below is still in range (wrap1 of any int)
  const int cx = wrap1(centre_cell(a.x, inv_hx), b.M[0]);
  const int cy = wrap1(centre_cell(a.y, inv_hy), b.M[1]);
  const int cz = wrap1(centre_cell(a.z, inv_hz), b.M[2]);
  return (cz * b.M[1] + cy) * b.nbx + (cx >> b.bxs);
}

template <typename CT>
__global__ void k_bin_count(const typename Vec4<CT>::type* __restrict__ xyzq, int n, BinLayout b,
                            CT inv_hx, CT inv_hy, CT inv_hz, int* __restrict__ key,
                            int* __restrict__ counts, int* __restrict__ bad, long long* __restrict__ clear,
                            long long clear_n, int* __restrict__ rank) {
  pdl_trigger();
  if (clear) {
    const long long stride = (long long)gridDim.x * blockDim.x;
    const long long first = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    for (long long i = first; i < clear_n / 2; i += stride)
      reinterpret_cast<int4*>(clear)[i] = make_int4(0, 0, 0, 0);
    if ((clear_n & 1) && first == 0) clear[clear_n - 1] = 0;
  }
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    const int k = bin_of(xyzq[i], b, inv_hx, inv_hy, inv_hz, bad);
    key[i] = k;
    // the atom's place among its bin's atoms (in counting order), so the placement
    // needs no atomics
    rank[i] = atomicAdd(&counts[k], 1);
  }
}

// Exclusive scan of counts[0..nb) within tiles of kScanTile bins, and the tiles' sums.
constexpr int kScanPer = 4;
constexpr int kScanThreads = 1024;
constexpr int kScanTile = kScanPer * kScanThreads;

__global__ void __launch_bounds__(kScanThreads)
    k_scan_tiles(const int* __restrict__ counts, int nb, int* __restrict__ start,
                 int* __restrict__ tile_sums) {
  pdl_trigger();
  pdl_wait();
  const int base = blockIdx.x * kScanTile + threadIdx.x * kScanPer;
  int v[kScanPer];
  int s = 0;
#pragma unroll
  for (int j = 0; j < kScanPer; j++) {
    v[j] = (base + j < nb) ? counts[base + j] : 0;
    s += v[j];
  }
  int total;
  int run = block_exclusive_scan(s, &total);
#pragma unroll
  for (int j = 0; j < kScanPer; j++) {
    if (base + j < nb) start[base + j] = run;
    run += v[j];
  }
  if (threadIdx.x == 0) tile_sums[blockIdx.x] = total;
}

// Placement after a tile-local scan: the block's copy of the tile offsets (exclusive
// prefix of the tile sums) turns the local bin starts into global ones; each atom
// goes to its bin's start plus the rank the counting kernel gave it, the global
// starts are written for the kernels that read the bins, and counts[] is cleared
// for the next call.  sorted: the mixed form's records, in any order within a bin;
// NULL: only the indices into `perm`, which k_bin_place_stable puts in order.
__global__ void __launch_bounds__(256)
    k_bin_place_final(const float4* __restrict__ xyzq, int n, const int* __restrict__ key,
                      const int* __restrict__ lstart, const int* __restrict__ tile_sums,
                      int ntiles, int* __restrict__ counts, float4* __restrict__ sorted,
                      int* __restrict__ perm, int* __restrict__ start, int nb,
                      const int* __restrict__ rank) {
  pdl_trigger();
  pdl_wait();
  __shared__ int off[kScanTile];
  constexpr int PER = kScanTile / 256;
  {
    const int base = threadIdx.x * PER;
    int v[PER];
    int s = 0;
#pragma unroll
    for (int j = 0; j < PER; j++) {
      v[j] = base + j < ntiles ? tile_sums[base + j] : 0;
      s += v[j];
    }
    int run = block_exclusive_scan(s, nullptr);
#pragma unroll
    for (int j = 0; j < PER; j++) {
      off[base + j] = run;
      run += v[j];
    }
  }
  __syncthreads();
  const int gtid = blockIdx.x * blockDim.x + threadIdx.x, gs = gridDim.x * blockDim.x;
  for (int i = gtid; i < n; i += gs) {
    const int k = key[i];
    const int slot = lstart[k] + off[k / kScanTile] + rank[i];
    if (sorted) sorted[slot] = xyzq[i];
    perm[slot] = i;
  }
  for (int i = gtid; i < nb; i += gs) {
    start[i] = lstart[i] + off[i / kScanTile];
    counts[i] = 0;  // zero for the next call's counting
  }
  if (gtid == 0) start[nb] = off[ntiles - 1] + tile_sums[ntiles - 1];
}

// The spread weights' basis of atom `a` into slot `slot` of sb.out.
__device__ __forceinline__ void store_basis(const double4& a, int slot, const BinLayout& b,
                                            const double3& inv_h, const SpreadBasis& sb) {
  const double x[3] = {a.x, a.y, a.z}, ih[3] = {inv_h.x, inv_h.y, inv_h.z};
  double v[kBasis64];
#pragma unroll
  for (int d = 0; d < 3; d++) {
    const int c = centre_cell(x[d], ih[d]);
    // offset of the centre point, from the first point's offset as the reference
    // rounds it (d0 = (c - n) h - x, CpuGaussCharge.cpp:311-329)
    const double h = sb.h[d], hh = h * h;
    const double dc = sub_rn(mul_rn((double)(c - sb.nst), h), x[d]) + (double)sb.nst * h;
    const double wc = exp(mul_rn(mul_rn(-dc, dc), sb.inv_2s2));
    v[3 * d] = d == 0 ? a.w * sb.pref * wc : wc;
    v[3 * d + 1] = exp(-(2 * dc * h + hh) * sb.inv_2s2);
    v[3 * d + 2] = exp(-(hh - 2 * dc * h) * sb.inv_2s2);
    if (d == 0) v[9] = (double)wrap1(c, b.M[0]);
  }
  double2* o = reinterpret_cast<double2*>(sb.out + (long long)slot * kBasis64);
#pragma unroll
  for (int k = 0; k < kBasis64 / 2; k++) o[k] = make_double2(v[2 * k], v[2 * k + 1]);
}

// Stable placement (FP64 form): an atom's rank in its bin is the number of bin
// members (tmp, in any order) with a smaller original index.
__global__ void k_bin_place_stable(const double4* __restrict__ xyzq, int n,
                                   const int* __restrict__ key, const int* __restrict__ start,
                                   const int* __restrict__ tmp, double4* __restrict__ sorted,
                                   int* __restrict__ perm, BinLayout b, double3 inv_h,
                                   SpreadBasis sb) {
  pdl_wait();
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    const int k = key[i];
    const int s = start[k], e = start[k + 1];
    int r = 0;
    for (int j = s; j < e; j++) r += (tmp[j] < i);
    const double4 a = xyzq[i];
    sorted[s + r] = a;
    perm[s + r] = i;
    if (sb.out) store_basis(a, s + r, b, inv_h, sb);
  }
}

// The whole binning of few atoms in one launch (bin_small): block 0, an atom per
// thread, counts, scans and places them with the bins in shared memory (nb ints);
// the other blocks clear the mixed form's grid.  The result is that of the kernels
// above; their global counts stay zero.
template <typename CT>
__global__ void __launch_bounds__(kBinSmall)
    k_bin_small(const typename Vec4<CT>::type* __restrict__ xyzq, int n, BinLayout b, CT inv_hx,
                CT inv_hy, CT inv_hz, int nb, typename Vec4<CT>::type* __restrict__ sorted,
                int* __restrict__ perm, int* __restrict__ start, int* __restrict__ bad,
                long long* __restrict__ clear, long long clear_n, SpreadBasis sb) {
  pdl_trigger();
  const int tid = threadIdx.x;
  if (blockIdx.x > 0) {
    for (long long i = (blockIdx.x - 1) * (long long)kBinSmall + tid; i < clear_n;
         i += (gridDim.x - 1) * (long long)kBinSmall)
      clear[i] = 0;
    return;
  }
  extern __shared__ int bins[];  // [nb] counts, then starts
  __shared__ int tmp[kBinSmall];
  typename Vec4<CT>::type a = {};
  if (tid < n) a = xyzq[tid];
  for (int i = tid; i < nb; i += kBinSmall) bins[i] = 0;
  __syncthreads();
  int k = 0, r = 0;
  if (tid < n) {
    k = bin_of(a, b, inv_hx, inv_hy, inv_hz, bad);
    r = atomicAdd(&bins[k], 1);
  }
  __syncthreads();
  const int per = (nb + kBinSmall - 1) / kBinSmall, i0 = min(tid * per, nb),
            i1 = min(i0 + per, nb);
  int s = 0;
  for (int i = i0; i < i1; i++) s += bins[i];
  int run = block_exclusive_scan(s, nullptr);
  for (int i = i0; i < i1; i++) {
    const int c = bins[i];
    bins[i] = run;
    run += c;
  }
  __syncthreads();
  if (tid < n) {
    r += bins[k];
    if (sizeof(CT) == 8) tmp[r] = tid;
  }
  for (int i = tid; i <= nb; i += kBinSmall) start[i] = i < nb ? bins[i] : n;
  if constexpr (sizeof(CT) == 8) {
    __syncthreads();
    if (tid < n) {
      r = bins[k];
      const int e = k + 1 < nb ? bins[k + 1] : n;
      for (int j = bins[k]; j < e; j++) r += (tmp[j] < tid);
    }
  }
  if (tid < n) {
    sorted[r] = a;
    perm[r] = tid;
    if constexpr (sizeof(CT) == 8) {
      if (sb.out) store_basis(a, r, b, make_double3(inv_hx, inv_hy, inv_hz), sb);
    }
  }
}

// ===========================================================================
// Mixed-form spread: atom-stationary scatter into a shared int32 brick tile
// ===========================================================================
// A CTA owns the atoms of one kSB^3-cell brick and a shared tile of the brick
// plus its n-cell halo, T = kSB + 2n points per axis, in int32 fixed point at
// a power-of-two scale 2^S chosen for this brick so that no partial sum can
// overflow (|q| pref summed over the brick's atoms, times 2^S, stays below
// 2^30, and every single contribution below 2^22).  One warp per atom: lanes
// take (x, z) pairs of the (2n+1)^2 plane, form t = q pref wx wz 2^S and add
// round(t wy) for each of the 2n+1 y values -- one fma (rounding by the
// 1.5 * 2^23 magic constant) and one shared-memory integer reduction per cube
// point.  The z-plane pitch is congruent to 2n+1 mod 32, so the 32 lanes of an
// instruction (consecutive (x, z) pairs) hit 32 different banks.
// The finished tile is added into an int64 grid at the common scale
// 2^kFlushBits (S <= kFlushBits, so the shift is exact) by integer
// reductions; integer sums do not depend on their order, so the grid is the
// same bit for bit on every run.
// SPLIT: the block takes the atoms of one of nparts parts.  Whole bricks keep the constant
// step through their atoms: with the step read from a register a droplet, whose few
// full bricks are bound by one block's chain, took 2305 instead of 2170 us (90,000
// charges in 6 A of a 98 A box).
template <int W, bool SPLIT = false>
__device__ __forceinline__ void scatter_brick(const float4* __restrict__ sorted,
                                              const int* __restrict__ start, const BinLayout& b,
                                              const Stencil<float>& s, int bxi, int byi, int bzi,
                                              int* __restrict__ tile,
                                              long long* __restrict__ grid64, int part = 0,
                                              int nparts = 1) {
  typedef ScatterGeom<W> G;
  constexpr int n = G::n;
  constexpr int NT = kScatterThreads, NW = NT / 32;
  constexpr int NPASS = (W * W + 31) / 32;
  __shared__ int rng_a[kSB * kSB], rng_p[kSB * kSB];
  __shared__ int alist[kScatterList];
  __shared__ __align__(16) float wys[NW][16];  // each warp's atom's y weights

  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int x0 = bxi * kSB, y0 = byi * kSB, z0 = bzi * kSB;
  const float apref = fabsf(s.pref);
  int total;
  const int shift = brick_prologue<W, NT>(
      start, b, x0, y0, z0, tile, rng_a, rng_p,
      [&](int i) { return fabsf(sorted[i].w) * apref; }, &total);
  if (part * NW >= total) return;  // (uniform) no atom is this block's: nothing to add
  const float tscale = exp2f((float)shift);

  // per-lane (x, z) pair of each pass and its tile offset: the same for all atoms
  int poff[NPASS], psx[NPASS], psz[NPASS];
#pragma unroll
  for (int pass = 0; pass < NPASS; pass++) {
    const int p = pass * 32 + lane;
    const int pz = p < W * W ? p / W : 0, px = p < W * W ? p - (p / W) * W : 0;
    psx[pass] = px;
    psz[pass] = pz;
    poff[pass] = pz * G::PP + px;
  }

  for (int c0 = 0; c0 < total; c0 += kScatterList) {
    brick_atom_list<NT, kSB * kSB>(rng_a, rng_p, total, c0, kScatterList, alist);
    __syncthreads();
    const int nc = min(kScatterList, total - c0);
    for (int q = SPLIT ? warp + part * NW : warp; q < nc; q += SPLIT ? NW * nparts : NW) {
      const float4 a = sorted[alist[q]];
      const float pos3[3] = {a.x, a.y, a.z};
      const int org[3] = {x0, y0, z0};
      int loc[3];
      float wl[3];  // lane j < W: weight j along each axis
#pragma unroll
      for (int d = 0; d < 3; d++) {
        const int c = centre_cell(pos3[d], s.inv_h[d]);
        loc[d] = wrap1(c, s.M[d]) - org[d];  // window start in tile coordinates
        const float dd = sub_rn(mul_rn((float)(c - n + lane), s.h[d]), pos3[d]);
        wl[d] = (lane < W) ? wexp(mul_rn(mul_rn(-dd, dd), s.inv_2s2)) : 0.f;
      }
      // every lane needs all W y weights: stored once by the lanes that formed
      // them and read back by four 16-byte broadcast loads (13 shuffles took
      // the shared-memory pipe the reductions wait for; the x and z weights,
      // one each per pass, stay shuffles: per-lane loads of them were slower)
      float wy[W];
      {
        __syncwarp();  // the warp's previous atom has read its weights
        if (lane < 16) wys[warp][lane] = wl[1];
        __syncwarp();
        const float4* v = reinterpret_cast<const float4*>(wys[warp]);
#pragma unroll
        for (int q4 = 0; q4 < (W + 3) / 4; q4++) {
          const float4 t = v[q4];
          wy[4 * q4] = t.x;
          if (4 * q4 + 1 < W) wy[4 * q4 + 1] = t.y;
          if (4 * q4 + 2 < W) wy[4 * q4 + 2] = t.z;
          if (4 * q4 + 3 < W) wy[4 * q4 + 3] = t.w;
        }
      }
      // y weights in pairs for the packed fma (two points per instruction)
      unsigned long long wy2[W / 2];
#pragma unroll
      for (int k = 0; k + 1 < W; k += 2)
        asm("mov.b64 %0, {%1, %2};" : "=l"(wy2[k / 2]) : "f"(wy[k]), "f"(wy[k + 1]));
      unsigned long long magic2;
      asm("mov.b64 %0, {%1, %1};" : "=l"(magic2) : "f"(12582912.0f));
      const float qp = a.w * s.pref * tscale;
      int* base = tile + loc[2] * G::PP + loc[1] * G::RP + loc[0];
#pragma unroll
      for (int pass = 0; pass < NPASS; pass++) {
        const float wx = __shfl_sync(0xffffffffu, wl[0], psx[pass]);
        const float wz = __shfl_sync(0xffffffffu, wl[2], psz[pass]);
        if (pass * 32 + lane < W * W) {
          const float t = qp * wx * wz;
          int* cell = base + poff[pass];
          unsigned long long t2;
          asm("mov.b64 %0, {%1, %1};" : "=l"(t2) : "f"(t));
#pragma unroll
          for (int k = 0; k + 1 < W; k += 2) {
            // round(t wy) for two points: |t wy| < 2^22, so 1.5*2^23 + t wy has
            // unit spacing (each half rounded once, as fmaf does)
            unsigned long long r2;
            asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r2) : "l"(t2), "l"(wy2[k / 2]), "l"(magic2));
            unsigned lo, hi;
            asm("mov.b64 {%0, %1}, %2;" : "=r"(lo), "=r"(hi) : "l"(r2));
            atomicAdd(cell + k * G::RP, (int)lo - 0x4B400000);
            atomicAdd(cell + (k + 1) * G::RP, (int)hi - 0x4B400000);
          }
          {
            const int v = __float_as_int(fmaf(t, wy[W - 1], 12582912.0f)) - 0x4B400000;
            atomicAdd(cell + (W - 1) * G::RP, v);
          }
        }
      }
    }
    __syncthreads();
  }
  brick_flush<W, NT>(tile, b, x0, y0, z0, shift, grid64);
}

template <int W, bool SPLIT>
__global__ void __launch_bounds__(kScatterThreads)
    k_spread_scatter(const float4* __restrict__ sorted, const int* __restrict__ start,
                     BinLayout b, Stencil<float> s, int nparts,
                     long long* __restrict__ grid64) {
  pdl_trigger();
  pdl_wait();
  extern __shared__ int tile[];
  scatter_brick<W, SPLIT>(sorted, start, b, s, SPLIT ? blockIdx.x / nparts : blockIdx.x,
                          blockIdx.y, blockIdx.z, tile, grid64, SPLIT ? blockIdx.x % nparts : 0,
                          nparts);
}

// float grid from the int64 accumulation grid at 2^kFlushBits
__global__ void k_grid64_to_real(const long long* __restrict__ g64, long long size,
                                 float* __restrict__ out) {
  const double unscale = exp2(-(double)kFlushBits);
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < size;
       i += (long long)gridDim.x * blockDim.x)
    out[i] = (float)((double)g64[i] * unscale);
}

// ===========================================================================
// Gather
// ===========================================================================
// Sphere test of one stencil point.  FP64 form: the reference's own sum and
// order, (dx^2 + dy^2) + dz^2 < rcut^2 (CpuGaussCharge.cpp:157-158), so the
// point set is bit-identical.  Mixed form: dx^2 < rcut^2 - (dy^2 + dz^2).
template <typename CT>
__device__ __forceinline__ bool in_sphere(CT dx2, CT dy2, CT dz2, CT rem, CT rcut2);
template <>
__device__ __forceinline__ bool in_sphere<double>(double dx2, double dy2, double dz2, double,
                                                  double rcut2) {
  return add_rn(add_rn(dx2, dy2), dz2) < rcut2;
}
template <>
__device__ __forceinline__ bool in_sphere<float>(float dx2, float, float, float rem, float) {
  return dx2 < rem;
}

// s0 = sum_k m_k wx[k] row[k], s1 = sum_k m_k wx[k] dx[k] row[k] over the
// 2n+1 points of one stencil row, m_k the sphere test.  The test guards the
// two fmas (predicated, no select); a skipped point adds exactly nothing.
template <typename CT, int W, int K0 = 0, int K1 = W>
__device__ __forceinline__ void row_sums(const CT* row, const CT (&dx2)[W], const CT (&wx)[W],
                                         const CT (&wdx)[W], CT dy2, CT dz2, CT rem, CT rcut2,
                                         CT& s0, CT& s1) {
  CT a = (CT)0, c = (CT)0;
#pragma unroll
  for (int k = K0; k < K1; k++) {
    const CT ph = row[k];
    if (in_sphere<CT>(dx2[k], dy2, dz2, rem, rcut2)) {
      a = fma(wx[k], ph, a);
      c = fma(wdx[k], ph, c);
    }
  }
  s0 = a;
  s1 = c;
}

// Shared memory of the gather for calculation type CT and stencil width W:
// the potential tile [TZ][ZP] (rows of pitch TP), per-atom weight tables and
// the list of stencil rows.
template <typename CT, int W, int NT = kGatherThreads, int GL = kGatherLanes, int GY = kGY,
          int GZ = kGZ>
struct GatherGeom {
  static constexpr int n = (W - 1) / 2;
  static constexpr int TX = kGX + 2 * n, TY = GY + 2 * n, TZ = GZ + 2 * n;
  static constexpr int TP = TX | 1;  // odd row pitch
  // plane pitch = W*TP (mod 32): row (jy, jz) starts in bank TP*(jy + W*jz)
  // mod 32, distinct for 32 consecutive (jy, jz)
  static constexpr int ZP = TY * TP + ((W - TY) * TP % 32 + 32) % 32;
  static constexpr int NW = NT / 32;
  static constexpr int APW = 32 / GL;  // atoms per warp at a time
  static constexpr int NROW = (W * W + GL - 1) / GL * GL;  // rows, padded to whole steps
  static constexpr size_t bytes =
      sizeof(CT) * (TZ * ZP + NW * APW * 9 * kWPad) + sizeof(int) * NROW;
};

// The (2n+1)^2 stencil rows (jy, jz) in the order in which the gather's groups of GL
// lanes take them, the same for every atom: entries (tile offset << 8 | jz << 4 | jy),
// first the rows that an atom may have inside its sphere, in (jz, jy) order so that a
// step's rows start in different banks, of them the rarest last; then the rows out
// of reach.  A row's least distance from an atom is (|j - n| - 1/2) h per axis when
// the atom lies within half a cell of its stencil centre; 0.01 h of slack covers
// the rounding of the centre.  Returns through n_step[0] the steps every atom takes,
// [1] the steps that hold rows within reach.  One warp.
template <int W, int GL>
__device__ __forceinline__ void gather_rows(int TP, int ZP, float hy, float hz, float rcut2,
                                            int* __restrict__ rows, int* n_step) {
  constexpr int n = (W - 1) / 2, NP = (W * W + 31) / 32;
  constexpr int NROW = (W * W + GL - 1) / GL * GL;
  const int lane = threadIdx.x & 31;
  float m[NP];  // squared least distance
#pragma unroll
  for (int t = 0; t < NP; t++) {
    const int p = t * 32 + lane, jz = p / W, jy = p - jz * W;
    const float dy = fmaxf(0.f, fabsf((float)(jy - n)) - 0.51f) * hy,
                dz = fmaxf(0.f, fabsf((float)(jz - n)) - 0.51f) * hz;
    m[t] = p < W * W ? dy * dy + dz * dz : 3.0e38f;
  }
  auto count = [&](float lim) {
    int c = 0;
#pragma unroll
    for (int t = 0; t < NP; t++) c += __popc(__ballot_sync(0xffffffffu, m[t] < lim));
    return c;
  };
  const int nc = count(rcut2);
  // the farthest rows, which few atoms reach, go last: at least as many as fill the
  // last, incomplete step, which a vote then mostly skips
  float lim = rcut2;
  int ncommon = nc;
  for (int k = 1; k <= 16 && ncommon > nc / GL * GL; k++) {
    lim = rcut2 * (1.f - 0.02f * (float)k);
    ncommon = count(lim);
  }
  int at[3] = {0, ncommon, nc};
#pragma unroll
  for (int t = 0; t < NP; t++) {
    const int p = t * 32 + lane, jz = p / W, jy = p - jz * W;
    const int cls = m[t] < lim ? 0 : m[t] < rcut2 ? 1 : p < W * W ? 2 : 3;
#pragma unroll
    for (int c = 0; c < 3; c++) {
      const unsigned b = __ballot_sync(0xffffffffu, cls == c);
      if (cls == c)
        rows[at[c] + __popc(b & ((1u << lane) - 1u))] =
            ((jz * ZP + jy * TP) << 8) | (jz << 4) | jy;
      at[c] += __popc(b);
    }
  }
  // table entry 15 lies outside every sphere
  for (int i = W * W + lane; i < NROW; i += 32) rows[i] = 15;
  if (lane == 0) {
    n_step[0] = ncommon / GL;
    n_step[1] = (nc + GL - 1) / GL;
  }
}

// The gather of the atoms of one brick by a block of NT threads.  kGatherLanes
// lanes share one atom (two atoms per warp at 16): each group builds its
// atom's weight tables and sums the rows of the block's row list, one row per lane
// and step.  GL lanes per atom (16 by default; the batched launch may take 8).
// A list of the rows inside each atom's own sphere (96 to 101 of 169 at n = 6) saves
// no step over the 113 rows that any atom can reach, whose last step holds one rare
// row, and cost nine groups of dependent loads, votes and stores per atom pair: without
// it the mixed kernel takes 94 registers instead of 121 (80 under the bound, so that
// 24 warps fit an SM instead of 16) and 262,143 charges on 144^3 0.199 -> 0.165 ms;
// the FP64 one 0.395 -> 0.305 ms, of which the 12 warps instead of 8 are half.
template <typename CT, int W, int NT = kGatherThreads, int GL = kGatherLanes, int GY = kGY,
          int GZ = kGZ>
__device__ __forceinline__ void gather_brick(const typename Vec4<CT>::type* __restrict__ sorted,
                                             const int* __restrict__ perm,
                                             const int* __restrict__ start, const BinLayout& b,
                                             const Stencil<CT>& s, const CT* __restrict__ phi,
                                             double outscale, double* __restrict__ fx,
                                             double* __restrict__ fy, double* __restrict__ fz,
                                             int bxi, int byi, int bzi, unsigned char* gsm) {
  typedef GatherGeom<CT, W, NT, GL, GY, GZ> GG;
  constexpr int n = GG::n, TX = GG::TX, TY = GG::TY, TZ = GG::TZ, TP = GG::TP, ZP = GG::ZP;
  constexpr int NW = GG::NW, APW = GG::APW;
  constexpr int NR = GY * GZ;  // cell rows of the brick
  static_assert(W <= 15 && kWPad == 16, "table entry 15 is free");
  static_assert(TZ * ZP < (1 << 23), "tile offsets fit the row list entries");
  typedef typename Vec4<CT>::type V;
  CT* tile = (CT*)gsm;                                   // [TZ][ZP]
  CT* tabs = tile + TZ * ZP;                             // [NW][APW][axis][d, d^2, w][kWPad]
  int* rlist = (int*)(tabs + NW * APW * 9 * kWPad);      // [NROW]
  __shared__ int n_step[2];
  __shared__ int rng_a[NR], rng_p[NR + 1];
  __shared__ int alist[kGatherList];

  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int grp = lane / GL, gl = lane % GL;
  const int x0 = bxi * kGX, y0 = byi * GY, z0 = bzi * GZ;
  const int ex = min(kGX, b.M[0] - x0), ey = min(GY, b.M[1] - y0), ez = min(GZ, b.M[2] - z0);

  // atoms of the brick: one range per (y, z) cell row
  int cnt = 0;
  if (tid < NR) {
    const int yy = tid % GY, zz = tid / GY;
    int a0 = 0, a1 = 0;
    if (yy < ey && zz < ez) {
      const int rowkey = ((z0 + zz) * b.M[1] + (y0 + yy)) * b.nbx;
      a0 = start[rowkey + (x0 >> b.bxs)];
      a1 = start[rowkey + ((x0 + ex - 1) >> b.bxs) + 1];
    }
    rng_a[tid] = a0;
    cnt = a1 - a0;
  }
  int natoms;
  const int pos = block_exclusive_scan(cnt, &natoms);
  if (tid < NR) rng_p[tid] = pos;
  if (tid == 0) rng_p[NR] = natoms;
  if (natoms == 0) return;  // uniform: natoms is the same in every thread

  // potential of the brick plus halo, staged by asynchronous element copies
  // so that a warp keeps all of its rows in flight
  stage_tile_async<CT, TX, TY, TZ, TP, ZP, NW>(phi, b, x0, y0, z0, n, tile);
  if (warp == NW - 1)
    gather_rows<W, GL>(TP, ZP, (float)s.h[1], (float)s.h[2], (float)s.rcut2, rlist, n_step);
  CT* tb = tabs + (warp * APW + grp) * 9 * kWPad;  // [axis][d, d^2, w][j]
  if (gl < 9) tb[gl * kWPad + 15] = gl % 3 == 1 ? (CT)3.0e38 : (CT)0;
  if (GL < 9 && gl == 0) tb[8 * kWPad + 15] = (CT)0;
  asm volatile("cp.async.wait_all;" ::: "memory");
  __syncthreads();
  const int always = n_step[0], reach = n_step[1];
  for (int c0 = 0; c0 < natoms; c0 += kGatherList) {
    brick_atom_list<NT, NR>(rng_a, rng_p, natoms, c0, kGatherList, alist);
    __syncthreads();
    const int nc = min(kGatherList, natoms - c0);
    // the next atom's record and output slot are loaded one iteration ahead,
    // so their global-memory latency overlaps the current atom's work
    int ai_n = 0, o_n = 0;
    V a_n;
    auto fetch = [&](int qq0) {
      const int qq = qq0 + grp;
      ai_n = alist[qq < nc ? qq : qq0];
      a_n = sorted[ai_n];
      o_n = perm[ai_n];
    };
    if (APW * warp < nc) fetch(APW * warp);
    for (int q0 = APW * warp; q0 < nc; q0 += APW * NW) {
      const int q = q0 + grp;
      const bool valid = q < nc;  // the last group of a chunk may have no atom
      const V a = a_n;
      const int out_slot = o_n;
      if (q0 + APW * NW < nc) fetch(q0 + APW * NW);
      const CT pos3[3] = {a.x, a.y, a.z};
      const int org[3] = {x0, y0, z0};
      int loc[3];
      bool far = false;  // farther than half a cell (and rounding) from its centre
#pragma unroll
      for (int d = 0; d < 3; d++) {
        const int c = centre_cell(pos3[d], s.inv_h[d]);
        loc[d] = wrap1(c, s.M[d]) - org[d];  // first stencil cell in tile coordinates
        for (int j = gl; j < W; j += GL) {
          const CT dd = sub_rn(pos3[d], mul_rn((CT)(c - n + j), s.h[d]));
          if (d > 0 && j == n) far |= !(fabs(dd) <= (CT)0.505 * s.h[d]);
          const CT d2 = mul_rn(dd, dd);
          tb[(d * 3 + 0) * kWPad + j] = dd;
          tb[(d * 3 + 1) * kWPad + j] = d2;
          tb[(d * 3 + 2) * kWPad + j] = wexp(mul_rn(-d2, s.inv_2s2));
        }
      }
      __syncwarp();
      // coordinates so large that their rounding moves the centre: all rows
      const int steps = __any_sync(0xffffffffu, far) ? GG::NROW / GL : reach;
      CT dx2[W], wx[W], wdx[W];
#pragma unroll
      for (int k = 0; k < W; k++) {
        dx2[k] = tb[(0 * 3 + 1) * kWPad + k];
        wx[k] = tb[(0 * 3 + 2) * kWPad + k];
        wdx[k] = wx[k] * tb[(0 * 3 + 0) * kWPad + k];
      }
      // each row's 2n+1 terms and a lane's rows (seven at n = 6) in CT, the
      // lanes' sums in double (the reference's AT)
      CT lx = 0, ly = 0, lz = 0;
      const CT* abase = tile + loc[2] * ZP + loc[1] * TP + loc[0];  // the atom's first row
      // an end point of the rows lies outside the sphere for every row when
      // dx^2 >= rcut^2 there (rem <= rcut^2): the rows are then summed
      // without it, the same terms in the same order.  The first point is
      // outside for nearly every atom (n h >= rcut), the last for about half.
      const bool head = __any_sync(0xffffffffu, dx2[0] < s.rcut2);
      const bool tail = __any_sync(0xffffffffu, dx2[W - 1] < s.rcut2);
      auto rows = [&](auto k0, auto k1) {
        constexpr int K0 = decltype(k0)::value;
        constexpr int K1 = decltype(k1)::value;
        for (int i = 0; i < steps; i++) {
          const int r = rlist[i * GL + gl];
          const int jz = (r >> 4) & 15, jy = r & 15;
          const CT dy2 = tb[(1 * 3 + 1) * kWPad + jy], dz2 = tb[(2 * 3 + 1) * kWPad + jz];
          const CT rem = s.rcut2 - (dy2 + dz2);
          // adding dx^2 >= 0 cannot take the sum below dy^2 + dz^2
          if (i >= always && !__any_sync(0xffffffffu, add_rn(dy2, dz2) < s.rcut2)) continue;
          const CT* row = abase + (r >> 8);
          CT s0, s1;
          row_sums<CT, W, K0, K1>(row, dx2, wx, wdx, dy2, dz2, rem, s.rcut2, s0, s1);
          const CT wyz = tb[(1 * 3 + 2) * kWPad + jy] * tb[(2 * 3 + 2) * kWPad + jz];
          lx += wyz * s1;
          ly += wyz * tb[(1 * 3 + 0) * kWPad + jy] * s0;
          lz += wyz * tb[(2 * 3 + 0) * kWPad + jz] * s0;
        }
      };
      if (head)
        rows(std::integral_constant<int, 0>(), std::integral_constant<int, W>());
      else if (tail)
        rows(std::integral_constant<int, 1>(), std::integral_constant<int, W>());
      else
        rows(std::integral_constant<int, 1>(), std::integral_constant<int, W - 1>());
      double ax = (double)lx, ay = (double)ly, az = (double)lz;
#pragma unroll
      for (int o = GL / 2; o > 0; o >>= 1) {
        ax += __shfl_xor_sync(0xffffffffu, ax, o);
        ay += __shfl_xor_sync(0xffffffffu, ay, o);
        az += __shfl_xor_sync(0xffffffffu, az, o);
      }
      if (gl == 0 && valid) {
        const double f = outscale * (double)(a.w * s.pref);
        fx[out_slot] = f * ax;
        fy[out_slot] = f * ay;
        fz[out_slot] = f * az;
      }
      __syncwarp();
    }
    __syncthreads();
  }
}

template <typename CT, int W, int GY, int GZ>
__global__ void __launch_bounds__(kGatherThreads, sizeof(CT) == 4 ? 2 : 1)
    k_gather_tiled(const typename Vec4<CT>::type* __restrict__ sorted,
                   const int* __restrict__ perm, const int* __restrict__ start, BinLayout b,
                   Stencil<CT> s, const CT* __restrict__ phi, double outscale,
                   double* __restrict__ fx, double* __restrict__ fy, double* __restrict__ fz) {
  pdl_wait();
  extern __shared__ __align__(16) unsigned char gsm[];
  gather_brick<CT, W, kGatherThreads, kGatherLanes, GY, GZ>(sorted, perm, start, b, s, phi,
                                                            outscale, fx, fy, fz, blockIdx.x,
                                                            blockIdx.y, blockIdx.z, gsm);
}

// ===========================================================================
// Launchers
// ===========================================================================
template <typename CT>
cudaError_t launch_bin_sorted(const typename Vec4<CT>::type* xyzq, int n, const BinLayout& b,
                              CT inv_hx, CT inv_hy, CT inv_hz, BinScratch w,
                              typename Vec4<CT>::type* sorted, int* perm, cudaStream_t st) {
  const int nb = b.M[1] * b.M[2] * b.nbx;
  const int ntiles = (nb + kScanTile - 1) / kScanTile;
  if (ntiles > kScanTile) return cudaErrorInvalidValue;
  if (bin_small(sizeof(CT) == 8, n, nb)) {
    const int nclear =
        w.clear ? (int)std::min<long long>(sm_count(), (w.clear_n + kBinSmall - 1) / kBinSmall) : 0;
    k_bin_small<CT><<<1 + nclear, kBinSmall, sizeof(int) * nb, st>>>(
        xyzq, n, b, inv_hx, inv_hy, inv_hz, nb, sorted, perm, w.start, w.bad, w.clear, w.clear_n,
        w.basis);
    return cudaGetLastError();
  }
  cudaError_t e = cudaSuccess;
  // a grid to clear takes every SM; the atoms alone, one thread each up to that
  const int gb = w.clear ? sm_count() * 8
                         : (int)std::min<long long>(sm_count() * 8,
                                                    (n + 255) / 256 > 0 ? (n + 255) / 256 : 1);
  if (n > 0)
    k_bin_count<CT><<<gb, 256, 0, st>>>(xyzq, n, b, inv_hx, inv_hy, inv_hz, w.key, w.counts,
                                        w.bad, w.clear, w.clear_n, bin_rank<CT>(w, perm));
  else if (w.clear)
    e = cudaMemsetAsync(w.clear, 0, sizeof(long long) * w.clear_n, st);
  if (e != cudaSuccess) return e;
  const CT inv_h[3] = {inv_hx, inv_hy, inv_hz};
  return launch_bin_scan_place<CT>(xyzq, n, nb, w, sorted, perm, st, b, inv_h);
}

// counts (filled) and ranks -> start offsets -> placement of the atoms: stable (in
// the original order within a bin) for the FP64 form, whose output-stationary
// spread sums atoms in bin order; any order for the mixed form.  Each kernel is
// launched as the dependent of the one before (the counting, when there are atoms).
// Launches bound it: eight (two clears, count, three scans, two placements) for the
// FP64 form were 45.1 us of an energy-force call on two charges, these four 41.5.
template <typename CT>
cudaError_t launch_bin_scan_place(const typename Vec4<CT>::type* xyzq, int n, int nb,
                                  BinScratch w, typename Vec4<CT>::type* sorted, int* perm,
                                  cudaStream_t st, const BinLayout& b, const CT* inv_h) {
  const int ntiles = (nb + kScanTile - 1) / kScanTile;
  if (ntiles > kScanTile) return cudaErrorInvalidValue;
  const int gb = (int)std::min<long long>(sm_count() * 8, (n + 255) / 256 > 0 ? (n + 255) / 256 : 1);
  cudaError_t e = launch_dependent(n > 0, k_scan_tiles, dim3(ntiles), dim3(kScanThreads), 0, st,
                                   w.counts, nb, w.lstart, w.tile_sums);
  if (e != cudaSuccess) return e;
  const int* rank = bin_rank<CT>(w, perm);
  constexpr bool fp64 = sizeof(CT) == 8;
  // the placement also writes every bin: four bins a thread, or as many blocks as the SMs
  // hold.  Sized by the atoms alone it took, bins included, 263 us for 30 atoms on 144^3
  // in FP64 and 79 in mixed (126 and 26 for 1500), now 21 and 14 (23 and 14); one, two,
  // eight and sixteen bins a thread are within 2 us of four.
  const int gp = std::max(gb, std::min(sm_count() * 8, (nb + 1023) / 1024));
  e = launch_dependent(true, k_bin_place_final, dim3(gp), dim3(256), 0, st,
                       fp64 ? nullptr : (const float4*)xyzq, n, (const int*)w.key,
                       (const int*)w.lstart, (const int*)w.tile_sums, ntiles, w.counts,
                       fp64 ? nullptr : (float4*)sorted, fp64 ? w.tmp : perm, w.start, nb, rank);
  if (e != cudaSuccess) return e;
  if constexpr (fp64) {
    if (n > 0) {
      const double3 ih = inv_h ? make_double3(inv_h[0], inv_h[1], inv_h[2]) : double3{};
      e = launch_dependent(true, k_bin_place_stable, dim3(gb), dim3(256), 0, st, xyzq, n,
                           (const int*)w.key, (const int*)w.start, (const int*)w.tmp, sorted,
                           perm, b, ih, w.basis);
      if (e != cudaSuccess) return e;
    }
  }
  return cudaGetLastError();
}

template <typename CT>
bool spread_tiled_supported(const Stencil<CT>& s) {
  for (int d = 0; d < 3; d++)
    if (s.nst[d] != s.nst[0]) return false;
  const int W = 2 * s.nst[0] + 1;
  return W == 9 || W == 11 || W == 13 || W == 15;
}

template <typename CT, int W, int GY, int GZ>
static cudaError_t gather_shape(const typename Vec4<CT>::type* sorted, const int* perm,
                                const int* start, const BinLayout& b, const Stencil<CT>& s,
                                const CT* phi, double outscale, double* fx, double* fy,
                                double* fz, bool pdl, cudaStream_t st) {
  const size_t smem = GatherGeom<CT, W, kGatherThreads, kGatherLanes, GY, GZ>::bytes;
  static std::atomic<bool> attr[64];
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev < 0 || dev >= 64) return cudaErrorInvalidDevice;
  if (!attr[dev]) {
    const cudaError_t e = cudaFuncSetAttribute(
        k_gather_tiled<CT, W, GY, GZ>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
    attr[dev] = true;
  }
  dim3 grd((b.M[0] + kGX - 1) / kGX, (b.M[1] + GY - 1) / GY, (b.M[2] + GZ - 1) / GZ);
  const cudaError_t e = launch_dependent(pdl, k_gather_tiled<CT, W, GY, GZ>, grd,
                                         dim3(kGatherThreads), smem, st, sorted, perm, start, b,
                                         s, phi, outscale, fx, fy, fz);
  if (e != cudaSuccess) return e;
  return cudaGetLastError();
}

template <typename CT, int W>
static cudaError_t gather_w(const typename Vec4<CT>::type* sorted, const int* perm,
                            const int* start, const BinLayout& b, const Stencil<CT>& s,
                            const CT* phi, double outscale, double* fx, double* fy, double* fz,
                            bool pdl, cudaStream_t st) {
  // the smallest brick whose blocks all run at about once (two per SM in the mixed form,
  // one in FP64): a grid of few bricks is bound by one brick's time.  Gather stage in
  // us with 16 x 16 x 8, 16 x 8 x 8 and 16 x 8 x 4 cells: mixed 38^3 (45, 75, 150
  // bricks) 33, 23, 18; 64^3 (128, 256, 512) 35, 31, 32; 80^3 (250, 500, 1000) 47, 49,
  // 56; 144^3 169, 185, -; FP64 38^3 43, 29, 21; 64^3 45, 48, 54
  const int slots = (sizeof(CT) == 4 ? 2 : 1) * sm_count() * 9 / 8;
  auto bricks = [&](int gy, int gz) {
    return (long long)((b.M[0] + kGX - 1) / kGX) * ((b.M[1] + gy - 1) / gy) *
           ((b.M[2] + gz - 1) / gz);
  };
  if (bricks(8, 4) <= slots)
    return gather_shape<CT, W, 8, 4>(sorted, perm, start, b, s, phi, outscale, fx, fy, fz, pdl, st);
  if (bricks(8, 8) <= slots)
    return gather_shape<CT, W, 8, 8>(sorted, perm, start, b, s, phi, outscale, fx, fy, fz, pdl, st);
  return gather_shape<CT, W, kGY, kGZ>(sorted, perm, start, b, s, phi, outscale, fx, fy, fz, pdl,
                                       st);
}

template <typename CT>
cudaError_t launch_gather_tiled(const typename Vec4<CT>::type* sorted, const int* perm,
                                const int* start, const BinLayout& b, const Stencil<CT>& s,
                                const CT* phi, double outscale, double* fx, double* fy,
                                double* fz, bool pdl, cudaStream_t st) {
  switch (2 * s.nst[0] + 1) {
    case 9: return gather_w<CT, 9>(sorted, perm, start, b, s, phi, outscale, fx, fy, fz, pdl, st);
    case 11:
      return gather_w<CT, 11>(sorted, perm, start, b, s, phi, outscale, fx, fy, fz, pdl, st);
    case 13:
      return gather_w<CT, 13>(sorted, perm, start, b, s, phi, outscale, fx, fy, fz, pdl, st);
    case 15:
      return gather_w<CT, 15>(sorted, perm, start, b, s, phi, outscale, fx, fy, fz, pdl, st);
  }
  return cudaErrorInvalidValue;
}

cudaError_t launch_grid64_to_real(const long long* grid64, long long size, float* out,
                                  cudaStream_t st) {
  k_grid64_to_real<<<sm_count() * 8, 256, 0, st>>>(grid64, size, out);
  return cudaGetLastError();
}

template <int W, bool SPLIT>
static cudaError_t scatter_shape(const float4* sorted, const int* start, const BinLayout& b,
                                 const Stencil<float>& s, dim3 grid, int nparts,
                                 long long* grid64, float* rho, bool zeroed, cudaStream_t st) {
  typedef ScatterGeom<W> G;
  const size_t smem = sizeof(int) * G::words;
  static std::atomic<bool> attr[64];
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev < 0 || dev >= 64) return cudaErrorInvalidDevice;
  if (!attr[dev]) {
    const cudaError_t e = cudaFuncSetAttribute(
        k_spread_scatter<W, SPLIT>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
    attr[dev] = true;
  }
  const long long size = (long long)b.M[0] * b.M[1] * b.M[2];
  cudaError_t e = cudaSuccess;
  if (!zeroed) e = cudaMemsetAsync(grid64, 0, sizeof(long long) * size, st);
  if (e != cudaSuccess) return e;
  // with the grid cleared earlier the spread follows the binning's last kernel
  e = launch_dependent(zeroed, k_spread_scatter<W, SPLIT>, grid, dim3(kScatterThreads), smem, st,
                       sorted, start, b, s, nparts, grid64);
  if (e != cudaSuccess) return e;
  // rho == nullptr: the caller converts the int64 grid itself (the own FFT)
  if (rho) k_grid64_to_real<<<sm_count() * 8, 256, 0, st>>>(grid64, size, rho);
  return cudaGetLastError();
}

template <int W>
static cudaError_t scatter_w(const float4* sorted, const int* start, const BinLayout& b,
                             const Stencil<float>& s, long long* grid64, float* rho, bool zeroed,
                             cudaStream_t st) {
  dim3 grid((b.M[0] + kSB - 1) / kSB, (b.M[1] + kSB - 1) / kSB, (b.M[2] + kSB - 1) / kSB);
  const int nparts = scatter_parts((long long)grid.x * grid.y * grid.z, W);
  grid.x *= nparts;
  if (nparts > 1)
    return scatter_shape<W, true>(sorted, start, b, s, grid, nparts, grid64, rho, zeroed, st);
  return scatter_shape<W, false>(sorted, start, b, s, grid, 1, grid64, rho, zeroed, st);
}

cudaError_t launch_spread_scatter(const float4* sorted, const int* start, const BinLayout& b,
                                  const Stencil<float>& s, long long* grid64, float* rho,
                                  bool zeroed, cudaStream_t st) {
  switch (2 * s.nst[0] + 1) {
    case 9: return scatter_w<9>(sorted, start, b, s, grid64, rho, zeroed, st);
    case 11: return scatter_w<11>(sorted, start, b, s, grid64, rho, zeroed, st);
    case 13: return scatter_w<13>(sorted, start, b, s, grid64, rho, zeroed, st);
    case 15: return scatter_w<15>(sorted, start, b, s, grid64, rho, zeroed, st);
  }
  return cudaErrorInvalidValue;
}

// ===========================================================================
// Batched systems: persistent kernels over (system, brick) work items
// ===========================================================================
__global__ void k_batch_bin_count(const float4* __restrict__ xyzq, int ntot,
                                  const BatchSys* __restrict__ sys, const int* __restrict__ first,
                                  int nsys, int* __restrict__ key, int* __restrict__ counts,
                                  int* __restrict__ rank) {
  pdl_trigger();
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < ntot; i += gridDim.x * blockDim.x) {
    const float4 a = xyzq[i];
    const BatchSys& S = sys[batch_sys_of(first, nsys, i)];
    const int cx = wrap1(centre_cell(a.x, S.sp.inv_h[0]), S.b.M[0]);
    const int cy = wrap1(centre_cell(a.y, S.sp.inv_h[1]), S.b.M[1]);
    const int cz = wrap1(centre_cell(a.z, S.sp.inv_h[2]), S.b.M[2]);
    const int k = S.bin_off + (cz * S.b.M[1] + cy) * S.b.nbx + (cx >> S.b.bxs);
    key[i] = k;
    rank[i] = atomicAdd(&counts[k], 1);
  }
}

template <int W>
__global__ void __launch_bounds__(kScatterThreads)
    k_batch_scatter(const float4* __restrict__ sorted, const int* __restrict__ start,
                    const BatchSys* __restrict__ sys, const BatchItem* __restrict__ items,
                    int nitems, long long* __restrict__ grid64) {
  extern __shared__ int tile[];
  for (int it = blockIdx.x; it < nitems; it += gridDim.x) {
    const BatchItem item = items[it];
    const BatchSys& S = sys[item.sys];
    scatter_brick<W>(sorted, start + S.bin_off, S.b, S.sp, item.bx, item.by, item.bz, tile,
                     grid64 + S.grid_off);
    __syncthreads();
  }
}

// rhok *= G per bin; energy[s] += efac_s * sum_k G |rho(k)|^2 (full spectrum).
// kfirst: ascending first bins of the systems' spectra, ksys: the system of
// each of those slots (grids are grouped by size, not in system order).
// A block takes runs of kGreenRun bins, PER per thread with all loads in flight; the
// run's system is looked up once and followed from there, and a warp adds its energy
// once per run and once per 32 bins of a later system in it (such bins one by one cost
// more than everything else: their additions meet at one address).  A search, a
// division and an addition per warp and 32 bins were bound by the search's dependent
// loads: 256 systems of 16^3 to 40^3 took 47.8 us with energies and 36.5 without, now
// 25.7 and 16.5; the bytes (20 per bin) are the rest.
constexpr int kGreenPer = 8, kGreenThreads = 256, kGreenRun = kGreenPer * kGreenThreads;

template <bool ENERGY>
__global__ void __launch_bounds__(kGreenThreads)
    k_batch_green_apply(float2* __restrict__ rhok, const float* __restrict__ tab,
                        long long ktot, const BatchSys* __restrict__ sys,
                        const long long* __restrict__ kfirst, const int* __restrict__ ksys,
                        int nsys, double* __restrict__ energy) {
  const int lane = threadIdx.x & 31;
  for (long long base = (long long)blockIdx.x * kGreenRun; base < ktot;
       base += (long long)gridDim.x * kGreenRun) {
    float2 v[kGreenPer];
    float f[kGreenPer];
#pragma unroll
    for (int j = 0; j < kGreenPer; j++) {
      const long long idx = base + j * kGreenThreads + threadIdx.x;
      if (idx < ktot) {
        v[j] = rhok[idx];
        f[j] = tab[idx];
      }
    }
    if (ENERGY) {
      int lo = 0, hi = nsys - 1;
      while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (kfirst[mid] <= base) lo = mid; else hi = mid - 1;
      }
      const int s0 = ksys[lo], M0 = sys[s0].b.M[0];
      const double efac0 = sys[s0].efac;
      const long long k0 = kfirst[lo], k1 = lo + 1 < nsys ? kfirst[lo + 1] : ktot;
      auto weight = [](long long i, int Mx) {
        const unsigned ix = (unsigned)i % (unsigned)(Mx / 2 + 1);
        return ix == 0 || ((Mx & 1) == 0 && ix == Mx / 2) ? 1.0 : 2.0;
      };
      double e = 0.0;
#pragma unroll
      for (int j = 0; j < kGreenPer; j++) {
        const long long idx = base + j * kGreenThreads + threadIdx.x;
        const double g2 = (double)f[j] * ((double)v[j].x * v[j].x + (double)v[j].y * v[j].y);
        if (idx < k1) e += weight(idx - k0, M0) * g2;
        if (__any_sync(0xffffffffu, idx >= k1 && idx < ktot)) {  // a later system's bins
          int l = lo;
          double t = 0.0;
          if (idx >= k1 && idx < ktot) {
            for (l = lo + 1; l + 1 < nsys && kfirst[l + 1] <= idx;) l++;
            const BatchSys& S = sys[ksys[l]];
            t = S.efac * weight(idx - kfirst[l], S.b.M[0]) * g2;
          }
          const int l0 = __shfl_sync(0xffffffffu, l, 0);
          if (__all_sync(0xffffffffu, l == l0)) {
            t = warp_sum(t);
            if (lane == 0) atomicAdd(&energy[ksys[l0]], t);
          } else if (l > lo) {
            atomicAdd(&energy[ksys[l]], t);
          }
        }
      }
      e = efac0 * e;
      e = warp_sum(e);
      if (lane == 0) atomicAdd(&energy[s0], e);
    }
#pragma unroll
    for (int j = 0; j < kGreenPer; j++) {
      const long long idx = base + j * kGreenThreads + threadIdx.x;
      if (idx < ktot) rhok[idx] = make_float2(v[j].x * f[j], v[j].y * f[j]);
    }
  }
}

template <int W>
__global__ void __launch_bounds__(kGatherThreads, 2)
    k_batch_gather(const float4* __restrict__ sorted, const int* __restrict__ perm,
                   const int* __restrict__ start, const BatchSys* __restrict__ sys,
                   const BatchItem* __restrict__ items, int nitems, const float* __restrict__ phi,
                   double outscale, double* __restrict__ fx, double* __restrict__ fy,
                   double* __restrict__ fz) {
  extern __shared__ __align__(16) unsigned char gsm[];
  for (int it = blockIdx.x; it < nitems; it += gridDim.x) {
    const BatchItem item = items[it];
    const BatchSys& S = sys[item.sys];
    gather_brick<float, W>(sorted, perm, start + S.bin_off, S.b, S.sg, phi + S.grid_off, outscale,
                           fx, fy, fz, item.bx, item.by, item.bz, gsm);
    __syncthreads();
  }
}

template <class K>
static cudaError_t set_max_smem(K kernel, size_t bytes, std::atomic<bool>* done) {
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev < 0 || dev >= 64) return cudaErrorInvalidDevice;
  if (done[dev]) return cudaSuccess;
  const cudaError_t e =
      cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
  if (e == cudaSuccess) done[dev] = true;
  return e;
}

template <int W>
static cudaError_t batch_scatter_w(const float4* sorted, const int* start, const BatchSys* sys,
                                   const BatchItem* items, int nitems, int ctas,
                                   long long* grid64, cudaStream_t st) {
  static std::atomic<bool> done[64];
  const size_t smem = sizeof(int) * ScatterGeom<W>::words;
  const cudaError_t e = set_max_smem(k_batch_scatter<W>, smem, done);
  if (e != cudaSuccess) return e;
  k_batch_scatter<W><<<std::min(ctas, nitems), kScatterThreads, smem, st>>>(sorted, start, sys,
                                                                           items, nitems, grid64);
  return cudaGetLastError();
}

template <int W>
static cudaError_t batch_gather_w(const float4* sorted, const int* perm, const int* start,
                                  const BatchSys* sys, const BatchItem* items, int nitems,
                                  int ctas, const float* phi, double outscale, double* fx,
                                  double* fy, double* fz, cudaStream_t st) {
  static std::atomic<bool> done[64];
  const size_t smem = GatherGeom<float, W>::bytes;
  const cudaError_t e = set_max_smem(k_batch_gather<W>, smem, done);
  if (e != cudaSuccess) return e;
  k_batch_gather<W><<<std::min(ctas, nitems), kGatherThreads, smem, st>>>(
      sorted, perm, start, sys, items, nitems, phi, outscale, fx, fy, fz);
  return cudaGetLastError();
}

cudaError_t launch_batch_bin(const float4* xyzq, int ntot, const BatchSys* sys, const int* first,
                             int nsys, int nbins, BinScratch w, float4* sorted, int* perm,
                             cudaStream_t st) {
  const int gb = (int)std::min<long long>(sm_count() * 8, (ntot + 255) / 256 > 0 ? (ntot + 255) / 256 : 1);
  if (ntot > 0)
    k_batch_bin_count<<<gb, 256, 0, st>>>(xyzq, ntot, sys, first, nsys, w.key, w.counts, w.tmp);
  return launch_bin_scan_place<float>(xyzq, ntot, nbins, w, sorted, perm, st);
}

cudaError_t launch_batch_spread(const float4* sorted, const int* start, const BatchSys* sys,
                                const BatchItem* items, const BatchSeg* segs, int nseg, int ctas,
                                long long* grid64, long long gsize, float* rho, cudaStream_t st) {
  cudaError_t e = cudaMemsetAsync(grid64, 0, sizeof(long long) * gsize, st);
  if (e != cudaSuccess) return e;
  for (int k = 0; k < nseg; k++) {
    const BatchItem* it = items + segs[k].first;
    const int cnt = segs[k].count;
    if (cnt <= 0) continue;
    switch (segs[k].W) {
      case 9: e = batch_scatter_w<9>(sorted, start, sys, it, cnt, ctas, grid64, st); break;
      case 11: e = batch_scatter_w<11>(sorted, start, sys, it, cnt, ctas, grid64, st); break;
      case 13: e = batch_scatter_w<13>(sorted, start, sys, it, cnt, ctas, grid64, st); break;
      case 15: e = batch_scatter_w<15>(sorted, start, sys, it, cnt, ctas, grid64, st); break;
      default: e = cudaErrorInvalidValue;
    }
    if (e != cudaSuccess) return e;
  }
  k_grid64_to_real<<<sm_count() * 8, 256, 0, st>>>(grid64, gsize, rho);
  return cudaGetLastError();
}

cudaError_t launch_batch_green(float2* rhok, const float* tab, long long ktot, const BatchSys* sys,
                               const long long* kfirst, const int* ksys, int nsys, double* energy,
                               cudaStream_t st) {
  const int ctas = (int)std::min<long long>(sm_count() * 8, (ktot + kGreenRun - 1) / kGreenRun);
  if (energy)
    k_batch_green_apply<true><<<ctas, kGreenThreads, 0, st>>>(rhok, tab, ktot, sys, kfirst, ksys,
                                                              nsys, energy);
  else
    k_batch_green_apply<false><<<ctas, kGreenThreads, 0, st>>>(rhok, tab, ktot, sys, kfirst, ksys,
                                                               nsys, energy);
  return cudaGetLastError();
}

cudaError_t launch_batch_gather(const float4* sorted, const int* perm, const int* start,
                                const BatchSys* sys, const BatchItem* items, const BatchSeg* segs,
                                int nseg, int ctas, const float* phi, double outscale, double* fx,
                                double* fy, double* fz, cudaStream_t st) {
  for (int k = 0; k < nseg; k++) {
    const BatchItem* it = items + segs[k].first;
    const int cnt = segs[k].count;
    if (cnt <= 0) continue;
    cudaError_t e;
    switch (segs[k].W) {
      case 9: e = batch_gather_w<9>(sorted, perm, start, sys, it, cnt, ctas, phi, outscale, fx, fy, fz, st); break;
      case 11: e = batch_gather_w<11>(sorted, perm, start, sys, it, cnt, ctas, phi, outscale, fx, fy, fz, st); break;
      case 13: e = batch_gather_w<13>(sorted, perm, start, sys, it, cnt, ctas, phi, outscale, fx, fy, fz, st); break;
      case 15: e = batch_gather_w<15>(sorted, perm, start, sys, it, cnt, ctas, phi, outscale, fx, fy, fz, st); break;
      default: e = cudaErrorInvalidValue;
    }
    if (e != cudaSuccess) return e;
  }
  return cudaSuccess;
}


// ===========================================================================
// Batched systems in one persistent cooperative launch
// ===========================================================================
constexpr int kFusedThreads = 512;
static_assert(kFusedThreads == kScatterThreads, "the fused kernel runs the scatter bricks");
static_assert(kScanTile % kFusedThreads == 0, "scan tile per thread");

constexpr size_t cmax(size_t a, size_t b) { return a > b ? a : b; }

template <int GL>
constexpr size_t fused_fwd_smem() {
  return cmax(cmax(cmax(sizeof(int) * ScatterGeom<9>::words, sizeof(int) * ScatterGeom<11>::words),
                   cmax(sizeof(int) * ScatterGeom<13>::words, sizeof(int) * ScatterGeom<15>::words)),
              cmax(cmax(cmax(GatherGeom<float, 9, kFusedThreads, GL>::bytes,
                             GatherGeom<float, 11, kFusedThreads, GL>::bytes),
                        cmax(GatherGeom<float, 13, kFusedThreads, GL>::bytes,
                             GatherGeom<float, 15, kFusedThreads, GL>::bytes)),
                   sizeof(SmallFftTw) + sizeof(int) * 3 * (kSfSmemSystems + 1)));
}

bool batch_fused_supported(const BatchSys* sys, int nsys) {
  for (int s = 0; s < nsys; s++) {
    for (int d = 0; d < 3; d++)
      if (sys[s].b.M[d] % 8 != 0 || sys[s].b.M[d] > kSfMax) return false;
    if (sys[s].W != 9 && sys[s].W != 11 && sys[s].W != 13 && sys[s].W != 15) return false;
  }
  return nsys > 0;
}

// One tile of kScanTile bin counts: exclusive prefix into start, the tile's
// sum into tile_sums[t].  All threads of the block.
__device__ __forceinline__ int fused_scan_tile(const int* __restrict__ counts, int nb,
                                               int* __restrict__ start, int* __restrict__ sums,
                                               int t) {
  constexpr int PER = kScanTile / kFusedThreads;
  const int base = t * kScanTile + threadIdx.x * PER;
  int v[PER];
  int s = 0;
#pragma unroll
  for (int j = 0; j < PER; j++) {
    v[j] = (base + j < nb) ? counts[base + j] : 0;
    s += v[j];
  }
  int total;
  int run = block_exclusive_scan(s, &total);
#pragma unroll
  for (int j = 0; j < PER; j++) {
    if (base + j < nb) start[base + j] = run;
    run += v[j];
  }
  if (threadIdx.x == 0) sums[t] = total;
  return total;
}

template <int GL>
__global__ void __launch_bounds__(kFusedThreads, 1) k_batch_forward_fused(BatchFused a) {
  namespace cg = cooperative_groups;
  extern __shared__ __align__(16) unsigned char fsm[];
  const long long gtid = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  const long long gstride = (long long)gridDim.x * blockDim.x;
  // clear the bin counts and the int64 grid
  for (long long i = gtid; i < a.nbins; i += gstride) a.w.counts[i] = 0;
  for (long long i = gtid; i < a.gtot; i += gstride) a.g64[i] = 0;
  if (gtid < 2) a.qctr[gtid] = 0;
  cg::this_grid().sync();
  // bin keys and counts (the key of k_batch_bin_count)
  for (long long i = gtid; i < a.ntot; i += gstride) {
    const float4 p = a.xyzq[i];
    const BatchSys& S = a.sys[batch_sys_of(a.first, a.nsys, (int)i)];
    const int cx = wrap1(centre_cell(p.x, S.sp.inv_h[0]), S.b.M[0]);
    const int cy = wrap1(centre_cell(p.y, S.sp.inv_h[1]), S.b.M[1]);
    const int cz = wrap1(centre_cell(p.z, S.sp.inv_h[2]), S.b.M[2]);
    const int k = S.bin_off + (cz * S.b.M[1] + cy) * S.b.nbx + (cx >> S.b.bxs);
    a.w.key[i] = k;
    atomicAdd(&a.w.counts[k], 1);
  }
  cg::this_grid().sync();
  // exclusive scan of the counts: tiles, their sums, the offsets
  const int ntiles = (a.nbins + kScanTile - 1) / kScanTile;
  for (int t = blockIdx.x; t < ntiles; t += gridDim.x)
    fused_scan_tile(a.w.counts, a.nbins, a.w.start, a.w.tile_sums, t);
  cg::this_grid().sync();
  if (blockIdx.x == 0) {  // tile sums -> tile offsets, in place (ntiles <= kScanTile)
    const int total = fused_scan_tile(a.w.tile_sums, ntiles, a.w.tile_sums,
                                      a.w.tile_sums + ntiles, 0);
    if (threadIdx.x == 0) a.w.start[a.nbins] = total;
  }
  cg::this_grid().sync();
  for (long long i = gtid; i < a.nbins; i += gstride) a.w.start[i] += a.w.tile_sums[i / kScanTile];
  cg::this_grid().sync();
  // placement in any order within a bin (the counts return to zero)
  for (long long i = gtid; i < a.ntot; i += gstride) {
    const int k = a.w.key[i];
    const int slot = a.w.start[k] + atomicSub(&a.w.counts[k], 1) - 1;
    a.sorted[slot] = a.xyzq[i];
    a.perm[slot] = (int)i;
  }
  cg::this_grid().sync();
  // spread bricks
  for (int it = fused_next_item(&a.qctr[0]); it < a.nscat; it = fused_next_item(&a.qctr[0])) {
    const BatchItem item = a.scat[it];
    const BatchSys& S = a.sys[item.sys];
    const int* st = a.w.start + S.bin_off;
    long long* g = a.g64 + S.grid_off;
    int* tile = reinterpret_cast<int*>(fsm);
    switch (S.W) {
      case 9: scatter_brick<9>(a.sorted, st, S.b, S.sp, item.bx, item.by, item.bz, tile, g); break;
      case 11: scatter_brick<11>(a.sorted, st, S.b, S.sp, item.bx, item.by, item.bz, tile, g); break;
      case 13: scatter_brick<13>(a.sorted, st, S.b, S.sp, item.bx, item.by, item.bz, tile, g); break;
      default: scatter_brick<15>(a.sorted, st, S.b, S.sp, item.bx, item.by, item.bz, tile, g); break;
    }
    __syncthreads();
  }
  cg::this_grid().sync();
  fused_solve(a, a.phi, true, fsm);
  cg::this_grid().sync();
  // gather bricks
  for (int it = fused_next_item(&a.qctr[1]); it < a.ngath; it = fused_next_item(&a.qctr[1])) {
    const BatchItem item = a.gath[it];
    const BatchSys& S = a.sys[item.sys];
    const int* st = a.w.start + S.bin_off;
    const float* ph = a.phi + S.grid_off;
    switch (S.W) {
      case 9:
        gather_brick<float, 9, kFusedThreads, GL>(a.sorted, a.perm, st, S.b, S.sg, ph, a.ccelec,
                                                  a.fx, a.fy, a.fz, item.bx, item.by, item.bz, fsm);
        break;
      case 11:
        gather_brick<float, 11, kFusedThreads, GL>(a.sorted, a.perm, st, S.b, S.sg, ph, a.ccelec,
                                                   a.fx, a.fy, a.fz, item.bx, item.by, item.bz, fsm);
        break;
      case 13:
        gather_brick<float, 13, kFusedThreads, GL>(a.sorted, a.perm, st, S.b, S.sg, ph, a.ccelec,
                                                   a.fx, a.fy, a.fz, item.bx, item.by, item.bz, fsm);
        break;
      default:
        gather_brick<float, 15, kFusedThreads, GL>(a.sorted, a.perm, st, S.b, S.sg, ph, a.ccelec,
                                                   a.fx, a.fy, a.fz, item.bx, item.by, item.bz, fsm);
        break;
    }
    __syncthreads();
  }
}

template <int GL>
static int fused_fwd_ctas() {
  static std::atomic<int> cache[64];
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) {
    cudaGetLastError();
    return 0;
  }
  int v = cache[dev].load();
  if (v == 0) {
    const size_t smem = fused_fwd_smem<GL>();
    int nb = 0;
    if (cudaFuncSetAttribute(k_batch_forward_fused<GL>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             (int)smem) != cudaSuccess ||
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, k_batch_forward_fused<GL>,
                                                      kFusedThreads, smem) != cudaSuccess) {
      cudaGetLastError();
      nb = 0;
    }
    v = nb > 0 ? nb * sm_count() : -1;
    cache[dev].store(v);
  }
  return v > 0 ? v : 0;
}

int batch_fused_ctas(int gather_lanes) {
  return gather_lanes == 8 ? fused_fwd_ctas<8>() : fused_fwd_ctas<16>();
}

cudaError_t launch_batch_forward_fused(const BatchFused& a, int ctas, int gather_lanes,
                                       cudaStream_t st) {
  const int most = gather_lanes == 8 ? fused_fwd_ctas<8>() : fused_fwd_ctas<16>();
  if (most <= 0 || ctas < 1 || ctas > most) return cudaErrorCooperativeLaunchTooLarge;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(ctas);
  cfg.blockDim = dim3(kFusedThreads);
  cfg.dynamicSmemBytes = gather_lanes == 8 ? fused_fwd_smem<8>() : fused_fwd_smem<16>();
  cfg.stream = st;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeCooperative;
  attr[0].val.cooperative = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  if (gather_lanes == 8) return cudaLaunchKernelEx(&cfg, k_batch_forward_fused<8>, a);
  return cudaLaunchKernelEx(&cfg, k_batch_forward_fused<16>, a);
}

#define GSE_TILED_INST(CT)                                                                      \
  template cudaError_t launch_bin_sorted<CT>(const Vec4<CT>::type*, int, const BinLayout&, CT,  \
                                             CT, CT, BinScratch, Vec4<CT>::type*, int*,         \
                                             cudaStream_t);                                     \
  template cudaError_t launch_bin_scan_place<CT>(const Vec4<CT>::type*, int, int, BinScratch,   \
                                                 Vec4<CT>::type*, int*, cudaStream_t,           \
                                                 const BinLayout&, const CT*);                  \
  template bool spread_tiled_supported<CT>(const Stencil<CT>&);                                 \
  template cudaError_t launch_gather_tiled<CT>(const Vec4<CT>::type*, const int*, const int*,   \
                                               const BinLayout&, const Stencil<CT>&, const CT*, \
                                               double, double*, double*, double*, bool,         \
                                               cudaStream_t);

GSE_TILED_INST(double)
GSE_TILED_INST(float)

}  // namespace gse
