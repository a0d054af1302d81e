// gse_ewald.cu -- FP64 Ewald reciprocal-space sum on the GPU.
//
// CpuEwaldRecip::calcForceEnergy (CpuEwaldRecip.cpp:87-147):
//   E   = sum_{k != 0, |k|_int^2 <= kcut^2} P(k) |S(k)|^2,
//   P   = (2 pi / V) ccelec exp(-sigma^2 k^2 / 2) / k^2,
//   S   = sum_i q_i exp(i k . r_i),
//   F_i = sum_k 2 P q_i k Im(conj(S) exp(i k . r_i))   (= -dE/dr_i).
// k and -k contribute equally; the sums run over the half space
// (kz > 0, or kz = 0 and ky > 0, or kz = ky = 0 and kx > 0) and are doubled.
//
// Rows of constant (ky, kz) with kx = 0..kxm, both signs of kx at once: with
// X_i(kx) = c + i s = exp(i kx 2 pi x_i / Lx) and R_i = q_i exp(i (ky.. + kz..)),
//   S(+-kx) = sum_i R_i c  +-  i sum_i R_i s,
// a real matrix product [Re R, Im R of every row] x [c, s of every kx] over the
// atoms.  With U+- = conj(P S(+-kx)) a row's part of the forces is
//   Im(R_i G0) (ky, kz) and Im(R_i G1) (kx), where
//   G0 = sum_kx (U+ + U-) c + i (U+ - U-) s,  G1 = sum_kx kx ((U+ - U-) c + i (U+ + U-) s),
// a product [c, s of every kx] x [four columns per row] for every atom.  Both run
// as mma.m8n8k4 in FP64 from shared memory; the phases come from one table per
// axis, sin and cos of k t with k t reduced to a period before the call.
//
// Bound: the FP64 pipe (37 TFLOP/s measured, fma and mma alike): 2 fmas per
// atom and k of the full sphere's half for S, 4 for the forces.  Rows are
// sorted by kxm so that a block's rows need about the same number of columns.
// At 23,559 charges and kcut 37: S 6.57 -> 0.60 ms (every row formed the phases of
// all atoms again before), forces 10.95 -> 1.03 ms (every atom stepped through every
// k by complex products); the pipe's floor is 0.27 and 0.54 ms.  What is left is the
// blocks' rounding to whole tiles and, in the force kernel, the phases of each step.
#include <cuda_runtime.h>
#include <math.h>

#include <algorithm>
#include <vector>

#include "gse_ewald.cuh"
#include "gse_internal.cuh"

namespace gse {

constexpr int kEwThreads = 256;
constexpr int kEwRows = 32;    // rows per block of the structure kernel (64 real rows)
constexpr int kEwCols = 80;    // its columns (c, s of 40 kx)
constexpr int kEwChunk = 32;   // its atoms per shared-memory chunk
constexpr int kEwPitch = 36;   // = 4 (mod 16): fragment loads hit 16 different banks
constexpr int kEwFRows = 16;   // rows per step of the force kernel (64 columns)
constexpr int kEwFK = 32;      // its kx table entries per shared-memory chunk
constexpr int kEwFPitch = 68;  // = 4 (mod 16)

__device__ __forceinline__ void mma884(double (&c)[2], double a, double b) {
  asm("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};"
      : "+d"(c[0]), "+d"(c[1])
      : "d"(a), "d"(b));
}

// T[axis][k][a] = exp(i k 2 pi x_a / L), k = 0..kmax, for the slab's atoms; the z
// axis carries the charge.  Atoms past the end get zero charge.
__global__ void __launch_bounds__(256)
    k_ewald_tables(const double4* __restrict__ xyzq, int na, int pitch, int kmax, EwGeom g,
                   double2* __restrict__ T) {
  const int a = blockIdx.x * 64 + (threadIdx.x & 63);
  const int axis = blockIdx.y;
  const double4 p = a < na ? xyzq[a] : make_double4(0.0, 0.0, 0.0, 0.0);
  double t = (axis == 0 ? p.x : axis == 1 ? p.y : p.z) * g.inv_box[axis];
  t -= rint(t);
  const double f = axis == 2 ? p.w : 1.0;
  for (int k = threadIdx.x >> 6; k <= kmax; k += 4) {
    const double h = (double)k * t, lo = fma((double)k, t, -h);  // k t = h + lo
    double s, c;
    sincospi(2.0 * ((h - rint(h)) + lo), &s, &c);
    T[((long long)axis * (kmax + 1) + k) * pitch + a] = make_double2(f * c, f * s);
  }
}

// R_i of a row from the tables.
__device__ __forceinline__ double2 ew_phase(double2 y, double2 z, int ky) {
  if (ky < 0) y.y = -y.y;
  return make_double2(y.x * z.x - y.y * z.y, y.x * z.y + y.y * z.x);
}

// part[split][row][Re, Im][column] (+)= the atoms of one split of the slab.  A block
// takes kEwRows rows and kEwCols columns; warp (wm, wn) a 16 x 40 tile.
__global__ void __launch_bounds__(kEwThreads, 2)
    k_ewald_structure(const double2* __restrict__ T, int pitch, int kmax,
                      const EwRow* __restrict__ rows, int nrows, int per_split, int ncols,
                      bool add, double* __restrict__ part) {
  __shared__ double As[2 * kEwRows][kEwPitch], Bs[kEwCols][kEwPitch];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int wm = warp >> 1, wn = warp & 1, r8 = lane >> 2, k4 = lane & 3;
  const int row0 = blockIdx.x * kEwRows, col0 = blockIdx.y * kEwCols;
  // columns of the block's rows (sorted: the first row has the most)
  const int bcols = 2 * (rows[row0].kxm + 1) - col0;
  if (bcols <= 0) return;
  const int strips = min(5, max(0, (bcols + 7) / 8 - 5 * wn));  // this warp's 8-column strips
  const int a0 = blockIdx.z * per_split, a1 = min(pitch, a0 + per_split);
  constexpr int NA = kEwRows / 8, NB = kEwCols / 2 / 8;  // rows and kx per warp
  const long long ax = (long long)(kmax + 1) * pitch;
  int kyv[NA], kzv[NA];
#pragma unroll
  for (int j = 0; j < NA; j++) {
    const int r = min(row0 + warp + 8 * j, nrows - 1);
    kyv[j] = rows[r].ky;
    kzv[j] = rows[r].kz;
  }
  double2 ra[NA], rb[NB];
  auto fetch = [&](int a) {  // the chunk's phases (rows) and x table, lane = atom
#pragma unroll
    for (int j = 0; j < NA; j++) {
      const int ky = kyv[j];
      ra[j] = ew_phase(T[ax + (long long)abs(ky) * pitch + a + lane],
                       T[2 * ax + (long long)kzv[j] * pitch + a + lane], ky);
    }
#pragma unroll
    for (int j = 0; j < NB; j++) {
      const int kx = col0 / 2 + warp + 8 * j;
      rb[j] = (2 * (warp + 8 * j) < bcols && kx <= kmax) ? T[(long long)kx * pitch + a + lane]
                                                         : make_double2(0.0, 0.0);
    }
  };
  double acc[2][5][2];
#pragma unroll
  for (int i = 0; i < 2; i++)
#pragma unroll
    for (int j = 0; j < 5; j++) acc[i][j][0] = acc[i][j][1] = 0.0;
  fetch(a0);
  for (int a = a0; a < a1; a += kEwChunk) {
#pragma unroll
    for (int j = 0; j < NA; j++) {
      As[2 * (warp + 8 * j)][lane] = ra[j].x;
      As[2 * (warp + 8 * j) + 1][lane] = ra[j].y;
    }
#pragma unroll
    for (int j = 0; j < NB; j++) {
      Bs[2 * (warp + 8 * j)][lane] = rb[j].x;
      Bs[2 * (warp + 8 * j) + 1][lane] = rb[j].y;
    }
    __syncthreads();
    if (a + kEwChunk < a1) fetch(a + kEwChunk);
    const double* pa = &As[16 * wm + r8][k4];
    const double* pb = &Bs[40 * wn + r8][k4];
    if (strips == 5) {
#pragma unroll
      for (int k = 0; k < kEwChunk; k += 4) {
        const double x0 = pa[k], x1 = pa[8 * kEwPitch + k];
#pragma unroll
        for (int j = 0; j < 5; j++) {
          const double y = pb[8 * j * kEwPitch + k];
          mma884(acc[0][j], x0, y);
          mma884(acc[1][j], x1, y);
        }
      }
    } else if (strips > 0) {
#pragma unroll
      for (int k = 0; k < kEwChunk; k += 4) {
        const double x0 = pa[k], x1 = pa[8 * kEwPitch + k];
#pragma unroll
        for (int j = 0; j < 4; j++) {
          if (j < strips) {
            const double y = pb[8 * j * kEwPitch + k];
            mma884(acc[0][j], x0, y);
            mma884(acc[1][j], x1, y);
          }
        }
      }
    }
    __syncthreads();
  }
#pragma unroll
  for (int i = 0; i < 2; i++)
#pragma unroll
    for (int j = 0; j < 5; j++) {
      const int m = 16 * wm + 8 * i + r8, row = row0 + (m >> 1);
      const int col = col0 + 40 * wn + 8 * j + 2 * k4;
      if (row < nrows && j < strips && col < ncols) {
        double2* o = reinterpret_cast<double2*>(
            part + (((long long)blockIdx.z * nrows + row) * 2 + (m & 1)) * ncols + col);
        double2 v = make_double2(acc[i][j][0], acc[i][j][1]);
        if (add) {
          v.x += o->x;
          v.y += o->y;
        }
        *o = v;
      }
    }
}

// A warp per row: S of every kx from the splits' sums, the row's energy, and the
// force kernel's four columns Wt[row][2 kx + {c, s}][G0 re, im, G1 re, im]
// (wpitch entries, zero past the row's kx).
__global__ void __launch_bounds__(256)
    k_ewald_finish(const double* __restrict__ part, int nsplit, int ncols,
                   const EwRow* __restrict__ rows, int nrows, EwGeom g, int wpitch,
                   double4* __restrict__ Wt, double* __restrict__ row_energy) {
  const int lane = threadIdx.x & 31;
  const int r = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  if (r >= nrows) return;
  const EwRow row = rows[r];
  const double kyv = 2.0 * kPi * row.ky * g.inv_box[1], kzv = 2.0 * kPi * row.kz * g.inv_box[2];
  double e = 0.0;
  for (int kx = lane; kx < wpitch / 2; kx += 32) {
    double4 wc = make_double4(0.0, 0.0, 0.0, 0.0), ws = wc;
    if (kx <= row.kxm && kx >= row.kx0) {
      double cr = 0.0, ci = 0.0, dr = 0.0, di = 0.0;  // sum R c, sum R s
      for (int s = 0; s < nsplit; s++) {
        const double* p = part + ((long long)s * nrows + r) * 2 * ncols + 2 * kx;
        cr += p[0];
        dr += p[1];
        ci += p[ncols];
        di += p[ncols + 1];
      }
      const double kxv = 2.0 * kPi * kx * g.inv_box[0];
      const double ksq = kxv * kxv + kyv * kyv + kzv * kzv;
      const double P = g.pref * exp(-ksq * g.half_sigmasq) / ksq;
      const bool both = kx > 0 && -kx >= row.kx0;  // the row has -kx too
      const double pr = cr - di, pi = ci + dr;     // S(+kx)
      const double mr = both ? cr + di : 0.0, mi = both ? ci - dr : 0.0;  // S(-kx)
      e += 2.0 * P * (pr * pr + pi * pi) + 2.0 * P * (mr * mr + mi * mi);
      const double sr = P * (pr + mr), si = -P * (pi + mi);  // U+ + U-
      const double tr = P * (pr - mr), ti = -P * (pi - mi);  // U+ - U-
      const double k = (double)kx;
      wc = make_double4(sr, si, k * tr, k * ti);
      ws = make_double4(-ti, tr, -k * si, k * sr);
    }
    if (Wt) {
      Wt[(long long)r * wpitch + 2 * kx] = wc;
      Wt[(long long)r * wpitch + 2 * kx + 1] = ws;
    }
  }
  e = warp_sum(e);
  if (lane == 0) row_energy[r] = e;
}

// fpart[split][d][a] = the rows of one split: sum of Im(R_a G1) (x), ky Im(R_a G0)
// (y), kz Im(R_a G0) (z).  A block takes 8 MI MW atoms (their x table stays in
// shared memory) and steps through its rows kEwFRows at a time; 8 warps, MW along
// the atoms and 8 / MW along the columns.
template <int MI, int MW>
__global__ void __launch_bounds__(kEwThreads)
    k_ewald_force(const double2* __restrict__ T, int pitch, int kmax,
                  const EwRow* __restrict__ rows, int nrows, int per_split, int wpitch,
                  const double4* __restrict__ Wt, double* __restrict__ fpart) {
  constexpr int MT = 8 * MI * MW, XP = MT + 4;  // XP = 4 (mod 16)
  constexpr int NWN = 8 / MW, NJ = 8 / NWN;     // column warps, 8-column strips per warp
  static_assert(XP % 16 == 4, "fragment loads hit 16 different banks");
  extern __shared__ __align__(16) double ew_sm[];
  double* Xs = ew_sm;               // [wpitch][XP]
  double* Bs = Xs + wpitch * XP;    // [2][kEwFK][kEwFPitch]
  __shared__ int rk[2][kEwFRows];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int wm = warp / NWN, wn = warp % NWN, r8 = lane >> 2, k4 = lane & 3;
  const int a0 = blockIdx.x * MT;
  const long long ax = (long long)(kmax + 1) * pitch;
  for (int i = tid; i < wpitch / 2 * MT; i += kEwThreads) {
    const int kx = i / MT, a = i % MT;
    const double2 v = kx <= kmax ? T[(long long)kx * pitch + a0 + a] : make_double2(0.0, 0.0);
    Xs[2 * kx * XP + a] = v.x;
    Xs[(2 * kx + 1) * XP + a] = v.y;
  }
  const int r0 = blockIdx.y * per_split, r1 = min(nrows, r0 + per_split);
  // chunk (row block, first k) into buffer b by asynchronous copies
  auto stage = [&](int row, int k0, int b) {
    for (int i = tid; i < kEwFRows * kEwFK * 2; i += kEwThreads) {
      const int half = i & 1, k = (i >> 1) % kEwFK, r = i / (2 * kEwFK);
      const bool in = row + r < r1;
      const double* src =
          reinterpret_cast<const double*>(Wt + (long long)(in ? row + r : r0) * wpitch + k0 + k) +
          2 * half;
      const unsigned dst = (unsigned)__cvta_generic_to_shared(
          Bs + (b * kEwFK + k) * kEwFPitch + 4 * r + 2 * half);
      asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src),
                   "r"(in ? 16 : 0)
                   : "memory");
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  double f[MI][2];  // G0 lanes: y, z; G1 lanes: x
#pragma unroll
  for (int i = 0; i < MI; i++) f[i][0] = f[i][1] = 0.0;
  double acc[MI][NJ][2];
#pragma unroll
  for (int i = 0; i < MI; i++)
#pragma unroll
    for (int j = 0; j < NJ; j++) acc[i][j][0] = acc[i][j][1] = 0.0;
  int row = r0, k0 = 0, buf = 0;
  int kend = r0 < r1 ? (2 * (rows[r0].kxm + 1) + 3) / 4 * 4 : 0;  // of the row block
  if (r0 < r1) stage(row, 0, 0);
  while (row < r1) {
    // the chunk after this one
    int nrow = row, nk0 = k0 + kEwFK;
    if (nk0 >= kend) {
      nrow = row + kEwFRows;
      nk0 = 0;
    }
    if (k0 == 0 && tid < kEwFRows) {
      const int r = min(row + tid, nrows - 1);
      rk[0][tid] = rows[r].ky;
      rk[1][tid] = rows[r].kz;
    }
    if (nrow < r1) {
      stage(nrow, nk0, buf ^ 1);
      asm volatile("cp.async.wait_group 1;" ::: "memory");
    } else {
      asm volatile("cp.async.wait_group 0;" ::: "memory");
    }
    __syncthreads();
    {
      const double* pa = Xs + (k0 + k4) * XP + 8 * MI * wm + r8;
      const double* pb = Bs + (buf * kEwFK + k4) * kEwFPitch + 8 * NJ * wn + r8;
      const int steps = min(kEwFK, kend - k0) / 4;
      auto step = [&](int k) {
        double x[MI];
#pragma unroll
        for (int i = 0; i < MI; i++) x[i] = pa[4 * k * XP + 8 * i];
#pragma unroll
        for (int j = 0; j < NJ; j++) {
          const double y = pb[4 * k * kEwFPitch + 8 * j];
#pragma unroll
          for (int i = 0; i < MI; i++) mma884(acc[i][j], x[i], y);
        }
      };
      if (steps == kEwFK / 4) {
#pragma unroll
        for (int k = 0; k < kEwFK / 4; k++) step(k);
      } else {
        for (int k = 0; k < steps; k++) step(k);
      }
    }
    if (nrow != row) {  // the row block's sums are complete
#pragma unroll
      for (int j = 0; j < NJ; j++) {
        const int r = 2 * (NJ * wn + j) + (k4 >> 1);
        const int ky = rk[0][r], kz = rk[1][r];
        const double2* ty = T + ax + (long long)abs(ky) * pitch + a0 + 8 * MI * wm + r8;
        const double2* tz = T + 2 * ax + (long long)kz * pitch + a0 + 8 * MI * wm + r8;
#pragma unroll
        for (int i = 0; i < MI; i++) {
          const double2 R = ew_phase(ty[8 * i], tz[8 * i], ky);
          const double im = R.x * acc[i][j][1] + R.y * acc[i][j][0];
          f[i][0] += ((k4 & 1) ? 1.0 : (double)ky) * im;
          f[i][1] += (double)kz * im;
          acc[i][j][0] = acc[i][j][1] = 0.0;
        }
      }
      kend = nrow < r1 ? (2 * (rows[nrow].kxm + 1) + 3) / 4 * 4 : 0;
    }
    __syncthreads();
    row = nrow;
    k0 = nk0;
    buf ^= 1;
  }
  // the four lanes of an atom (two rows x G0, G1), then the column warps in order
  double* red = Bs;  // [NWN][MT][3]
#pragma unroll
  for (int i = 0; i < MI; i++) {
    double u = f[i][0], v = f[i][1];
    u += __shfl_xor_sync(0xffffffffu, u, 2);
    v += __shfl_xor_sync(0xffffffffu, v, 2);
    const int a = 8 * (MI * wm + i) + r8;
    if (k4 == 0) {
      red[(wn * MT + a) * 3 + 1] = u;
      red[(wn * MT + a) * 3 + 2] = v;
    } else if (k4 == 1) {
      red[(wn * MT + a) * 3] = u;
    }
  }
  __syncthreads();
  for (int i = tid; i < 3 * MT; i += kEwThreads) {
    const int d = i / MT, a = i % MT;
    double s = 0.0;
#pragma unroll
    for (int w = 0; w < NWN; w++) s += red[(w * MT + a) * 3 + d];
    fpart[((long long)blockIdx.y * 3 + d) * pitch + a0 + a] = s;
  }
}

// Forces of the slab from the row splits, in split order (add: to the former blocks').
__global__ void k_ewald_force_sum(const double* __restrict__ fpart, int nsplit, int pitch, int na,
                                  EwGeom g, bool add, double* __restrict__ fx,
                                  double* __restrict__ fy, double* __restrict__ fz) {
  const int a = blockIdx.x * blockDim.x + threadIdx.x, d = blockIdx.y;
  if (a >= na) return;
  double s = 0.0;
  for (int w = 0; w < nsplit; w++) s += fpart[((long long)w * 3 + d) * pitch + a];
  s *= 4.0 * 2.0 * kPi * g.inv_box[d];
  double* f = (d == 0 ? fx : d == 1 ? fy : fz) + a;
  *f = add ? *f + s : s;
}

std::vector<EwRow> ewald_rows(int kcut) {
  std::vector<EwRow> rows;
  const int kc2 = kcut * kcut;
  for (int kz = 0; kz <= kcut; kz++)
    for (int ky = (kz == 0 ? 0 : -kcut); ky <= kcut; ky++) {
      const int rem = kc2 - ky * ky - kz * kz;
      if (rem < 0) continue;
      int kxm = (int)std::floor(std::sqrt((double)rem));
      while (kxm * kxm > rem) kxm--;
      while ((kxm + 1) * (kxm + 1) <= rem) kxm++;
      const int kx0 = (kz == 0 && ky == 0) ? 1 : -kxm;
      if (kxm < kx0) continue;
      rows.push_back({ky, kz, kx0, kxm});
    }
  std::stable_sort(rows.begin(), rows.end(),
                   [](const EwRow& a, const EwRow& b) { return a.kxm > b.kxm; });
  return rows;
}

// Force blocks of 64 atoms while their x table leaves room for two blocks per SM, 32
// beyond (the largest kcut's table fits no more).
constexpr int kEwWide = 128;  // of wpitch
static bool ew_wide(int wpitch) { return wpitch <= kEwWide; }

static size_t ew_force_smem(int wpitch, int mt) {
  return sizeof(double) * ((size_t)wpitch * (mt + 4) + 2 * kEwFK * kEwFPitch);
}

EwPlan ewald_plan(int n, const std::vector<EwRow>& rows, int kcut, bool forces, size_t budget) {
  EwPlan p;
  p.kmax = kcut;
  p.nrows = (int)rows.size();
  // atoms per slab: the phase tables (48 bytes per atom and k) within half the budget
  const long long half = (long long)(budget / 2), most = half / (48ll * (kcut + 1));
  p.slab = (int)std::min<long long>(n, std::max<long long>(64, most / 64 * 64));
  p.pitch = (p.slab + 63) / 64 * 64;
  const int sms = sm_count();
  auto block = [&](int row0, int nrows) {
    EwBlock b;
    b.row0 = row0;
    b.nrows = nrows;
    const int k2 = 2 * (rows[row0].kxm + 1);  // of its longest row
    b.ncols = (k2 + 7) / 8 * 8;
    b.wpitch = (k2 + kEwFK - 1) / kEwFK * kEwFK;
    // atom splits of the structure kernel: four blocks per SM slot pair, the splits'
    // sums within a quarter of the budget
    const int blocks = (nrows + kEwRows - 1) / kEwRows * ((b.ncols + kEwCols - 1) / kEwCols);
    int ks = std::max(1, std::min(16, 4 * sms / blocks));
    ks = std::min(ks, std::max(1, p.pitch / (4 * kEwChunk)));
    ks = (int)std::min<long long>(ks, std::max(1ll, half / 2 / (16ll * nrows * b.ncols)));
    b.per_split = ((p.pitch + ks - 1) / ks + kEwChunk - 1) / kEwChunk * kEwChunk;
    b.nsplit = (p.pitch + b.per_split - 1) / b.per_split;
    // row splits of the force kernel: at least twelve blocks per SM
    const int mt = ew_wide(b.wpitch) ? 64 : 32;
    const int fb = (p.pitch + mt - 1) / mt;
    const int rs = std::max(1, std::min(32, 12 * sms / fb));
    b.per_fsplit = ((nrows + rs - 1) / rs + kEwFRows - 1) / kEwFRows * kEwFRows;
    b.nfsplit = (nrows + b.per_fsplit - 1) / b.per_fsplit;
    return b;
  };
  auto part_bytes = [](const EwBlock& b) {
    return sizeof(double) * 2 * (size_t)b.nsplit * b.nrows * b.ncols;
  };
  auto w_bytes = [&](const EwBlock& b) {
    return forces ? sizeof(double4) * (size_t)b.nrows * b.wpitch : 0;
  };
  // rows per block: all of them unless their sums (32 bytes per kx and sign for the
  // forces, 16 per split for S) exceed half the budget, from about kcut 120 on; 2.4 GB
  // at kcut 255 in one block
  int per = p.nrows;
  while (per > kEwRows) {
    const EwBlock b = block(0, per);
    if (part_bytes(b) + w_bytes(b) <= (size_t)half) break;
    per = std::max(kEwRows, (per / 2 + kEwRows - 1) / kEwRows * kEwRows);
  }
  size_t part = 0, w = 0, f = 0;
  for (int r = 0; r < p.nrows; r += per) {
    const EwBlock b = block(r, std::min(per, p.nrows - r));
    part = std::max(part, part_bytes(b));
    w = std::max(w, w_bytes(b));
    if (forces) f = std::max(f, sizeof(double) * 3 * (size_t)b.nfsplit * p.pitch);
    p.blocks.push_back(b);
  }
  size_t off = 0;
  auto take = [&](size_t bytes) {
    const size_t o = off;
    off = (off + bytes + 255) / 256 * 256;
    return o;
  };
  p.off_rows = take(sizeof(EwRow) * p.nrows);
  p.off_energy = take(sizeof(double) * p.nrows);
  p.off_T = take(sizeof(double2) * 3 * (size_t)(kcut + 1) * p.pitch);
  p.off_part = take(part);
  p.off_W = take(w);
  p.off_f = take(f);
  p.bytes = off;
  return p;
}

cudaError_t launch_ewald(const double4* xyzq, int n, const std::vector<EwRow>& rows,
                         const EwGeom& g, const EwPlan& p, char* buf, double* fx, double* fy,
                         double* fz, cudaStream_t st) {
  EwRow* rows_d = (EwRow*)(buf + p.off_rows);
  double2* T = (double2*)(buf + p.off_T);
  double* part = (double*)(buf + p.off_part);
  double4* Wt = fx ? (double4*)(buf + p.off_W) : nullptr;
  double* fpart = (double*)(buf + p.off_f);
  cudaError_t e = cudaMemcpyAsync(rows_d, rows.data(), sizeof(EwRow) * p.nrows,
                                  cudaMemcpyHostToDevice, st);
  if (e != cudaSuccess) return e;
  // the tables of one slab stay for everything that follows when there is one only
  bool have = false;
  auto tables = [&](int a0) {
    const int na = std::min(p.slab, n - a0);
    if (!have)
      k_ewald_tables<<<dim3(p.pitch / 64, 3), 256, 0, st>>>(xyzq + a0, na, p.pitch, p.kmax, g, T);
    have = p.slab >= n;
    return na;
  };
  for (const EwBlock& b : p.blocks) {
    const EwRow* r = rows_d + b.row0;
    const dim3 sg((b.nrows + kEwRows - 1) / kEwRows, (b.ncols + kEwCols - 1) / kEwCols, b.nsplit);
    for (int a0 = 0; a0 < n; a0 += p.slab) {
      tables(a0);
      k_ewald_structure<<<sg, kEwThreads, 0, st>>>(T, p.pitch, p.kmax, r, b.nrows, b.per_split,
                                                   b.ncols, a0 > 0, part);
    }
    k_ewald_finish<<<(b.nrows + 7) / 8, 256, 0, st>>>(part, b.nsplit, b.ncols, r, b.nrows, g,
                                                      b.wpitch, Wt,
                                                      (double*)(buf + p.off_energy) + b.row0);
    if (!fx) continue;
    const bool wide = ew_wide(b.wpitch);
    const int mt = wide ? 64 : 32;
    const size_t smem = ew_force_smem(b.wpitch, mt);
    auto kernel = wide ? k_ewald_force<2, 4> : k_ewald_force<2, 2>;
    // the limit is the kernel's, not this call's: calls of other threads share it
    e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             (int)ew_force_smem(wide ? kEwWide : 2 * 256, mt));
    if (e != cudaSuccess) return e;
    for (int a0 = 0; a0 < n; a0 += p.slab) {
      const int na = tables(a0);
      kernel<<<dim3((p.pitch + mt - 1) / mt, b.nfsplit), kEwThreads, smem, st>>>(
          T, p.pitch, p.kmax, r, b.nrows, b.per_fsplit, b.wpitch, Wt, fpart);
      k_ewald_force_sum<<<dim3((na + 255) / 256, 3), 256, 0, st>>>(
          fpart, b.nfsplit, p.pitch, na, g, b.row0 > 0, fx + a0, fy + a0, fz + a0);
    }
  }
  return cudaGetLastError();
}

}  // namespace gse
