// gse_spread64.cu -- the FP64 form's tiled spread on the FP64 tensor pipe.
//
// CpuGaussCharge::spreadChargeToGrid (CpuGaussCharge.cpp:235-384),
// output-stationary: a CTA owns a block of the grid and every warp an 8 x 8 x 8
// patch of it, two accumulators per lane and z plane.  The atoms whose
// (2n+1)^3 cube reaches the block stream through shared memory in chunks as
// three rows of 1-D weights; each warp keeps the ones that reach its patch, in
// sorted order, four at a time.  For one z plane of the patch four atoms are
//   rho[x, y] += sum_i (q_i pref wx_i[x] wz_i[z]) wy_i[y],
// an 8 x 4 by 4 x 8 product: one mma.m8n8k4 in FP64 (products and sums rounded
// as fmas), with the plane factor folded into A by one multiply.  Planes that
// none of the four atoms reaches are skipped; the atoms come sorted by z cell,
// so the four mostly share their 2n+1 planes.  No atomics; every grid point is
// written once and the sums run in a fixed order.
//
// Bound: the FP64 pipe and the latency of a group's chain (list entry, weights,
// multiply, mma).  The pipe's mma rate is its fma rate (37 TFLOP/s measured for
// both on a B200), but one instruction holds 256 fmas, so the group of four
// atoms costs about 75 instructions where an fma per lane and column cost 25 per
// atom and patch besides the fmas.  A multiply between the mmas costs 4 pipe
// cycles, an mma 16.  Measured spread stage, before (fmas, 16 x 8 x 24 blocks,
// weights formed in every block) and after: 262,143 charges on 144^3 0.672 ->
// 0.275 ms, 48,192 on 80^3 0.330 -> 0.091, 23,559 on 64^3 0.307 -> 0.056, two
// charges on 20^3 0.016 -> 0.012.  Tried and slower at 144^3: producer warps
// behind named barriers (0.40: their multiplies queue behind the mmas),
// m16n8k8 with two planes and eight atoms (0.33), 16-plane patches (0.36),
// every plane tested by itself (0.31) or none (0.38).
#include "gse_internal.cuh"
#include "gse_tiled.cuh"
#include "gse_tiled_dev.cuh"

namespace gse {

constexpr int kS64Chunk = 64;    // atoms with weight rows in shared memory at a time
constexpr int kS64List = 2048;   // atoms listed at a time
constexpr int kS64Items = 1024;  // row segments scanned at a time

// Weight rows of one atom for stencil width W: a row has 7 zeros on either side, so
// that a patch that the cube overlaps reads its eight points without a test; record
// kS64Chunk is all zeros (pads a group of four).
template <int W>
struct Spread64Geom {
  static constexpr int RL = W + 14;
  static constexpr int RS = 3 * RL;  // 81 doubles at W = 13: successive atoms two banks apart
  static constexpr int SR = RS * (kS64Chunk + 1);
  static constexpr size_t rec_bytes = sizeof(double) * SR;
};

// Powers of exp(-2 h^2 / (2 sigma^2)) per axis: v[d][k] = its k(k+1)/2-th power, the
// factor of point k+1 from the centre beside the centre weight and the ratio's power.
struct Decay {
  double v[3][7];
};

// 1-D weights w[j] = exp(-(dc + (j - n) h)^2 / (2 sigma^2)), j < W = 2n+1, from
// the centre weight and the two ratios that the binning stored:
//   w[n +- k] = wc exp(-(k-1) k h^2 / (2 sigma^2)) r^k,  r = w[n +- 1] / w[n].
// The powers come by squaring (three products deep at k = 7).
template <int W>
__device__ __forceinline__ void gauss_row64(double wc, double ru, double rd,
                                            const double (&dec)[7], double* __restrict__ w) {
  constexpr int n = (W - 1) / 2;
  double pu[8], pd[8];
  pu[1] = ru;
  pd[1] = rd;
  w[n] = wc;
#pragma unroll
  for (int k = 1; k <= n; k++) {
    if (k > 1) {
      pu[k] = pu[k / 2] * pu[k - k / 2];
      pd[k] = pd[k / 2] * pd[k - k / 2];
    }
    const double f = k > 1 ? wc * dec[k - 1] : wc;
    w[n + k] = f * pu[k];
    w[n - k] = f * pd[k];
  }
}

// WX x WY x WZ patches of 8^3 points, S warps on each (every S-th group of four
// atoms).
template <int W, int WX, int WY, int WZ, int S>
__global__ void __launch_bounds__(32 * WX * WY * WZ * S)
    k_spread_mma64(const double* __restrict__ basis, const int* __restrict__ start, BinLayout b,
                   Decay dec, double* __restrict__ grid) {
  typedef Spread64Geom<W> G;
  constexpr int n = (W - 1) / 2, RL = G::RL, RS = G::RS;
  constexpr int NP = WX * WY * WZ, NW = NP * S, NT = 32 * NW;
  constexpr int PER = kS64Items / NT;
  constexpr int NU = (3 * kS64Chunk + NT - 1) / NT;  // weight rows per thread
  static_assert(kS64Items % NT == 0, "whole row segments per thread");
  static_assert(S == 1 || NP * 512 * (S / 2) <= G::SR, "partial sums fit");
  extern __shared__ __align__(16) double recs[];  // [kS64Chunk + 1][RS]
  __shared__ int win[kS64Chunk];  // window start per axis relative to the block, 8 bits each
  __shared__ int rng_a[kS64Items], rng_p[kS64Items + 1];
  __shared__ int list_atom[kS64List];
  __shared__ int list_win[kS64List];  // window start: y and z 8 bits each, segment above
  __shared__ int wlist[NW][kS64Chunk + 4];

  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int patch = warp % NP, split = warp / NP;
  const int x0 = blockIdx.x * 8 * WX, y0 = blockIdx.y * 8 * WY, z0 = blockIdx.z * 8 * WZ;
  const int ex = min(8 * WX, b.M[0] - x0), ey = min(8 * WY, b.M[1] - y0),
            ez = min(8 * WZ, b.M[2] - z0);
  const int px0 = 8 * (patch % WX), py0 = 8 * (patch / WX % WY), pz0 = 8 * (patch / (WX * WY));
  const int r8 = lane >> 2, k4 = lane & 3;  // fragment row (x of A, y of B) and atom
  const bool inside = px0 < ex && py0 < ey && pz0 < ez;  // the patch has points
  int* wl = wlist[warp];

  for (int i = tid; i < G::SR; i += NT) recs[i] = 0.0;

  double acc[8][2];
#pragma unroll
  for (int z = 0; z < 8; z++) acc[z][0] = acc[z][1] = 0.0;

  // row segments of the region that reaches the block, in unwrapped cells: rows
  // (uz, uy), each cut into nseg segments of one period in x
  const int ux_lo = x0 - n, ux_hi = x0 + ex + n;
  const int nry = ey + 2 * n, nrz = ez + 2 * n;
  int nseg = 0;
  for (int u = ux_lo; u < ux_hi; nseg++) u += b.M[0] - pmod(u, b.M[0]);
  const int nitems = nry * nrz * nseg;
  auto item_x = [&](int sg, int& cu, int& c1, int& sh) {  // segment sg: cells [cu, c1), shift
    int u = ux_lo;
    for (int i = 0; i < sg; i++) u += b.M[0] - pmod(u, b.M[0]);
    cu = pmod(u, b.M[0]);
    sh = u - cu;
    c1 = min(ux_hi - sh, b.M[0]);
  };

  for (int ibase = 0; ibase < nitems; ibase += kS64Items) {
    const int ni = min(kS64Items, nitems - ibase);
    int cnt[PER], sum = 0;
#pragma unroll
    for (int j = 0; j < PER; j++) {
      const int it = tid * PER + j;
      cnt[j] = 0;
      if (it < ni) {
        const int row = (ibase + it) / nseg;
        int cu, c1, sh;
        item_x(ibase + it - row * nseg, cu, c1, sh);
        const int ccy = pmod(y0 - n + row % nry, b.M[1]), ccz = pmod(z0 - n + row / nry, b.M[2]);
        const int rowkey = (ccz * b.M[1] + ccy) * b.nbx;
        const int a0 = start[rowkey + (cu >> b.bxs)];
        rng_a[it] = a0;
        cnt[j] = start[rowkey + ((c1 - 1) >> b.bxs) + 1] - a0;
        sum += cnt[j];
      }
    }
    int total;
    int run = block_exclusive_scan(sum, &total);
#pragma unroll
    for (int j = 0; j < PER; j++) {
      rng_p[tid * PER + j] = run;
      run += cnt[j];
    }
    if (tid == NT - 1) rng_p[kS64Items] = run;
    __syncthreads();
    for (int l0 = 0; l0 < total; l0 += kS64List) {
      const int nl = min(kS64List, total - l0);
      for (int r = tid; r < ni; r += NT) {
        const int p0 = rng_p[r], p1 = rng_p[r + 1], a0 = rng_a[r];
        const int q0 = max(p0, l0), q1 = min(p1, l0 + nl);
        if (q0 >= q1) continue;
        const int row = (ibase + r) / nseg, sg = ibase + r - row * nseg;
        const int wy = row % nry - 2 * n, wz = row / nry - 2 * n;
        for (int p = q0; p < q1; p++) {
          list_atom[p - l0] = a0 + (p - p0);
          list_win[p - l0] = (wy & 0xff) | ((wz & 0xff) << 8) | (sg << 16);
        }
      }
      __syncthreads();
      const int nchunks = (nl + kS64Chunk - 1) / kS64Chunk;
      // this thread's weight rows (atom u % kS64Chunk, axis u / kS64Chunk) of the next
      // chunk are fetched while the current one is summed
      double bw[NU][3];
      int bs[NU];  // the row's window start
      auto fetch = [&](int c) {
#pragma unroll
        for (int k = 0; k < NU; k++) {
          const int u = tid + k * NT, d = u / kS64Chunk, i = c * kS64Chunk + u % kS64Chunk;
          bs[k] = 64;  // reaches no patch
          if (d < 3 && i < nl) {
            const double* r = basis + (long long)list_atom[i] * kBasis64;
            const int lw = list_win[i];
            bw[k][0] = r[3 * d];
            bw[k][1] = r[3 * d + 1];
            bw[k][2] = r[3 * d + 2];
            if (d == 0) {
              int cu, c1, sh;
              item_x(lw >> 16, cu, c1, sh);
              bs[k] = (int)r[9] + sh - n - x0;
            } else {
              bs[k] = (signed char)(d == 1 ? lw : lw >> 8);
            }
          }
        }
      };
      fetch(0);
      for (int c = 0; c < nchunks; c++) {
#pragma unroll
        for (int k = 0; k < NU; k++) {
          const int u = tid + k * NT, i = u % kS64Chunk, d = u / kS64Chunk;
          if (d < 3) {
            reinterpret_cast<signed char*>(win + i)[d] = (signed char)bs[k];
            if (bs[k] < 64)
              gauss_row64<W>(bw[k][0], bw[k][1], bw[k][2],
                             d == 0 ? dec.v[0] : d == 1 ? dec.v[1] : dec.v[2],
                             recs + i * RS + d * RL + 7);
          }
        }
        __syncthreads();
        if (c + 1 < nchunks) fetch(c + 1);
        // --- each warp: the atoms that reach its patch, four at a time ---
        if (inside) {
          int m = 0;
#pragma unroll
          for (int base = 0; base < kS64Chunk; base += 32) {
            const int i = base + lane, h = win[i];
            const int tx = (signed char)h - px0, ty = (signed char)(h >> 8) - py0,
                      tz = (signed char)(h >> 16) - pz0;
            const bool rel = tx < 8 && tx > -W && ty < 8 && ty > -W && tz < 8 && tz > -W;
            const unsigned bal = __ballot_sync(0xffffffffu, rel);
            // the atom with its window start in patch coordinates (+ 16, 6 bits each)
            if (rel)
              wl[m + __popc(bal & ((1u << lane) - 1u))] =
                  (tx + 16) | ((ty + 16) << 6) | ((tz + 16) << 12) | (i << 18);
            m += __popc(bal);
          }
          // pad to whole groups with the zero record, its window beyond the patch in z
          if (lane < 4) wl[m + lane] = 16 | (16 << 6) | (24 << 12) | (kS64Chunk << 18);
          __syncwarp();
          // fragments of the group at g: A of every plane, B, and the planes of the
          // patch that any of the four windows covers
          auto load = [&](int g, double (&a)[8], double& by, unsigned& zm) {
            const int e = wl[g + k4];
            const int tz = ((e >> 12) & 63) - 16;
            const double* r = recs + (e >> 18) * RS + 7;
            const double ax = r[r8 + 16 - (e & 63)];
            by = r[RL + r8 + 16 - ((e >> 6) & 63)];
            const double* wz = r + 2 * RL - tz;
#pragma unroll
            for (int z = 0; z < 8; z++) a[z] = ax * wz[z];
            zm = __reduce_or_sync(0xffffffffu,
                                  tz >= 0 ? ((1u << W) - 1u) << tz : ((1u << W) - 1u) >> -tz);
          };
          // two planes at a time: a test of each plane costs more than the planes it saves
          auto mma = [&](const double (&a)[8], double by, unsigned zm) {
#pragma unroll
            for (int z = 0; z < 8; z++)
              if (zm & (3u << (z & 6)))
                asm("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};"
                    : "+d"(acc[z][0]), "+d"(acc[z][1])
                    : "d"(a[z]), "d"(by));
          };
          for (int g = 4 * split; g < m; g += 4 * S) {
            double a[8], by;
            unsigned zm;
            load(g, a, by, zm);
            mma(a, by, zm);
          }
        }
        __syncthreads();
      }
    }
  }
  // --- the splits' sums, pairwise in a fixed order, through the records' memory ---
#pragma unroll
  for (int h = S / 2; h > 0; h /= 2) {
    if (split >= h && split < 2 * h)
#pragma unroll
      for (int z = 0; z < 8; z++)
#pragma unroll
        for (int j = 0; j < 2; j++)
          recs[(((split - h) * NP + patch) * 16 + z * 2 + j) * 32 + lane] = acc[z][j];
    __syncthreads();
    if (split < h)
#pragma unroll
      for (int z = 0; z < 8; z++)
#pragma unroll
        for (int j = 0; j < 2; j++)
          acc[z][j] += recs[((split * NP + patch) * 16 + z * 2 + j) * 32 + lane];
    __syncthreads();
  }
  if (split > 0) return;
  // --- write the patch: every point exactly once ---
  const int gx = x0 + px0 + r8;
#pragma unroll
  for (int z = 0; z < 8; z++) {
#pragma unroll
    for (int j = 0; j < 2; j++) {
      const int gy = y0 + py0 + 2 * k4 + j, gz = z0 + pz0 + z;
      if (gx < b.M[0] && gy < b.M[1] && gz < b.M[2])
        grid[((long long)gz * b.M[1] + gy) * b.M[0] + gx] = acc[z][j];
    }
  }
}

template <int W, int WX, int WY, int WZ, int S>
static cudaError_t spread64_w(const double* basis, const int* start, const BinLayout& b,
                              const Stencil<double>& s, double* grid, cudaStream_t st) {
  const size_t smem = Spread64Geom<W>::rec_bytes;
  static std::atomic<bool> attr[64];
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev < 0 || dev >= 64) return cudaErrorInvalidDevice;
  if (!attr[dev]) {
    const cudaError_t e =
        cudaFuncSetAttribute(k_spread_mma64<W, WX, WY, WZ, S>,
                             cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
    attr[dev] = true;
  }
  const dim3 grd((b.M[0] + 8 * WX - 1) / (8 * WX), (b.M[1] + 8 * WY - 1) / (8 * WY),
                 (b.M[2] + 8 * WZ - 1) / (8 * WZ));
  Decay dec;
  for (int d = 0; d < 3; d++)
    for (int k = 0; k < 7; k++)
      dec.v[d][k] = std::exp(-(double)(k * (k + 1)) * s.h[d] * s.h[d] * s.inv_2s2);
  k_spread_mma64<W, WX, WY, WZ, S>
      <<<grd, 32 * WX * WY * WZ * S, smem, st>>>(basis, start, b, dec, grid);
  return cudaGetLastError();
}

template <int W>
static cudaError_t spread64_shape(const double* basis, const int* start, const BinLayout& b,
                                  const Stencil<double>& s, double* grid, cudaStream_t st) {
  // A block's atoms pass one chunk at a time (about 3 us each with one warp per patch),
  // so a grid of few blocks is bound by that chain: blocks as small, with as many
  // warps per patch, as two blocks per SM allow.  Spread stage in ms, shapes in this
  // order: 38^3 (125 patches) 0.028, 0.045, 0.064, 0.097; 64^3 (512) 0.060, 0.056,
  // 0.070, 0.102; 80^3 (1000) 0.113, 0.102, 0.092, 0.107; 100^3 (2197) 0.217, 0.164,
  // 0.182, 0.191; 144^3 (5832) 0.507, 0.355, 0.332, 0.275.
  const long long px = (b.M[0] + 7) / 8, py = (b.M[1] + 7) / 8, pz = (b.M[2] + 7) / 8;
  const long long two = 2 * sm_count();
  if (px * py * pz <= two) return spread64_w<W, 1, 1, 1, 8>(basis, start, b, s, grid, st);
  if (px * py * ((pz + 1) / 2) <= two)
    return spread64_w<W, 1, 1, 2, 4>(basis, start, b, s, grid, st);
  if (px * ((py + 1) / 2) * ((pz + 1) / 2) <= two)
    return spread64_w<W, 1, 2, 2, 2>(basis, start, b, s, grid, st);
  if (((px + 1) / 2) * ((py + 1) / 2) * ((pz + 1) / 2) <= 3 * sm_count())
    return spread64_w<W, 1, 1, 2, 4>(basis, start, b, s, grid, st);
  return spread64_w<W, 2, 2, 2, 1>(basis, start, b, s, grid, st);
}

cudaError_t launch_spread64(const double* basis, const int* start, const BinLayout& b,
                            const Stencil<double>& s, double* grid, cudaStream_t st) {
  switch (2 * s.nst[0] + 1) {
    case 9: return spread64_shape<9>(basis, start, b, s, grid, st);
    case 11: return spread64_shape<11>(basis, start, b, s, grid, st);
    case 13: return spread64_shape<13>(basis, start, b, s, grid, st);
    case 15: return spread64_shape<15>(basis, start, b, s, grid, st);
  }
  return cudaErrorInvalidValue;
}

}  // namespace gse
