// gse_adjoint.cu -- reverse-mode derivatives of one GSE-k force evaluation.
//
// The forward pass (CpuGSEk::spreadCharge1 -> solvePoisson -> calculateEnergy
// -> interpolateForce, CpuGSEk.cpp:30-58, CpuGSE.cpp:70-103) is
//   rho(r) = sum_i q_i g(r - x_i)          over the (2n+1)^3 cube of atom i,
//            g = (2 pi s^2)^(-3/2) exp(-|r - x|^2 / (2 s^2)), s = sigma1
//   phi    = K rho                          K = c2r G(sigma2) r2c (symmetric)
//   E      = 1/2 c h^3 rho . phi            c = ccelec, h^3 = cell volume
//   F_i    = c q_i sum_{r in sphere_i} D_i(r) phi(r),
//            D_i(r) = A exp(-|u|^2 / (2 s^2)) u,  u = x_i - r,
//            A = (2 pi)^(-3/2) h^3 s^-5.
// Given dL/dE = gE and dL/dF_i = G_i, with
//   lambda(r) = c sum_i q_i G_i . D_i(r)     (the adjoint source, sphere)
//   Psi       = K lambda + gE c h^3 phi      (dL/drho)
// the derivatives are
//   dL/dq_j = sum_{cube} g(r - x_j) Psi(r) + c A sum_{sphere} e phi (G_j . u)
//   dL/dx_j = q_j sum_{cube} g (r - x_j) / s^2 Psi(r)
//           + c q_j A sum_{sphere} e phi [G_j - (G_j . u) u / s^2],
// e = exp(-|u|^2 / (2 s^2)).  The sphere's edge is not differentiated (its
// derivative is zero almost everywhere).
#include <atomic>
#include <type_traits>

#include "gse_adjoint.cuh"
#include "gse_internal.cuh"
#include "gse_tiled.cuh"
#include "gse_tiled_dev.cuh"

namespace gse {

// ---------------------------------------------------------------------------
// Atom-parallel kernels: the FP64 form, and the mixed form's shapes that the tiled
// kernels do not take.  A warp per atom, its two halves on every other z plane of the
// stencil, a lane on one x offset: the x factors stay in the lane's registers, the y
// and z factors come from tables of the warp, both grids are read along x, and what
// only depends on z is applied once per plane (five FP64 operations a point in the
// source, nine in the gather).  Every lane on a point of its own, with an exponential
// and four divisions each, took 0.31 ms for the source and 0.45 ms for the gather at
// 23,559 charges in FP64; now 0.071 and 0.162 ms, bound by the source's reductions at L2 and
// by the FP64 pipe and load latency at 16 warps per SM.
// ---------------------------------------------------------------------------
constexpr int kAdjWarps = 8;  // warps per block
constexpr int kAdjRows = 7;   // rows of a plane whose loads are in flight together

template <typename CT>
struct AdjRowTab {
  // y, z: u = x - r, u^2, e = exp(-u^2 / (2 s^2)), e u
  CT u[2][kMaxStencil], u2[2][kMaxStencil], e[2][kMaxStencil], eu[2][kMaxStencil];
  int off[2][kMaxStencil];  // wrapped index, along z times My
};

// Tables of one atom's y and z axes by its warp; returns its first x cell.
template <typename CT>
__device__ __forceinline__ int adj_tables(const CT (&pos)[3], const Stencil<CT>& s,
                                          AdjRowTab<CT>& t) {
  const int lane = threadIdx.x & 31;
  __syncwarp();  // the previous atom's tables are read
#pragma unroll
  for (int d = 1; d < 3; d++) {
    const int c0 = round_to_int(mul_rn(pos[d], s.inv_h[d])) - s.nst[d];
    for (int j = lane; j < 2 * s.nst[d] + 1; j += 32) {
      const CT u = sub_rn(pos[d], mul_rn((CT)(c0 + j), s.h[d])), u2 = mul_rn(u, u);
      const CT e = gexp(-u2 * s.inv_2s2);
      t.u[d - 1][j] = u;
      t.u2[d - 1][j] = u2;
      t.e[d - 1][j] = e;
      t.eu[d - 1][j] = e * u;
      t.off[d - 1][j] = pmod(c0 + j, s.M[d]) * (d == 1 ? 1 : s.M[1]);
    }
  }
  __syncwarp();
  return round_to_int(mul_rn(pos[0], s.inv_h[0])) - s.nst[0];
}

// The points of the cube by planes: for each run of 16 x offsets and each plane of
// this half-warp, plane(jz, e_x, u_x, u_x^2), then for its rows, up to kAdjRows at a
// time, load(k, grid index) of all of them and use(k, jy), then done(jz).
template <typename CT, class Plane, class Load, class Use, class Done>
__device__ __forceinline__ void adj_planes(const CT (&pos)[3], const Stencil<CT>& s,
                                           const AdjRowTab<CT>& t, int c0x, Plane plane,
                                           Load load, Use use, Done done) {
  const int lane = threadIdx.x & 31, xl = lane & 15, half = lane >> 4;
  const int W0 = 2 * s.nst[0] + 1, W1 = 2 * s.nst[1] + 1, W2 = 2 * s.nst[2] + 1;
  for (int xb = xl; xb < W0; xb += 16) {
    const CT u = sub_rn(pos[0], mul_rn((CT)(c0x + xb), s.h[0]));
    const CT u2 = mul_rn(u, u), e = gexp(-u2 * s.inv_2s2);
    const int x = pmod(c0x + xb, s.M[0]);
    for (int jz = half; jz < W2; jz += 2) {
      plane(jz, e, u, u2);
      const long long base = x + (long long)t.off[1][jz] * s.M[0];
      for (int j0 = 0; j0 < W1; j0 += kAdjRows) {
#pragma unroll
        for (int k = 0; k < kAdjRows; k++)
          if (j0 + k < W1) load(k, base + (long long)t.off[0][j0 + k] * s.M[0]);
#pragma unroll
        for (int k = 0; k < kAdjRows; k++)
          if (j0 + k < W1) use(k, j0 + k);
      }
      done(jz);
    }
  }
}

// lambda(r) += c q_i A e (G_i . u) over the sphere of atom i (global atomics).
template <typename CT>
__global__ void __launch_bounds__(32 * kAdjWarps)
    k_adj_source(const typename Vec4<CT>::type* __restrict__ xyzq, const int* __restrict__ perm,
                 int n, Stencil<CT> s, double c, const double* __restrict__ gfx,
                 const double* __restrict__ gfy, const double* __restrict__ gfz,
                 CT* __restrict__ lambda) {
  __shared__ AdjRowTab<CT> tabs[kAdjWarps];
  const int w = threadIdx.x >> 5;
  AdjRowTab<CT>& t = tabs[w];
  for (int ii = blockIdx.x * kAdjWarps + w; ii < n; ii += gridDim.x * kAdjWarps) {
    const auto a = xyzq[ii];
    const int i = perm[ii];
    const CT pos[3] = {a.x, a.y, a.z};
    const CT G[3] = {(CT)gfx[i], (CT)gfy[i], (CT)gfz[i]};
    const CT amp = (CT)(c * (double)a.w * (double)s.pref);
    const int c0x = adj_tables<CT>(pos, s, t);
    CT t1 = 0, t2 = 0, ux2 = 0, uz2 = 0;  // of the plane
    long long at[kAdjRows];
    adj_planes<CT>(
        pos, s, t, c0x,
        [&](int jz, CT e, CT u, CT u2) {
          const CT f = amp * e * t.e[1][jz];
          t1 = f * (G[0] * u + G[2] * t.u[1][jz]);
          t2 = f * G[1];
          ux2 = u2;
          uz2 = t.u2[1][jz];
        },
        [&](int k, long long idx) { at[k] = idx; },
        [&](int k, int jy) {
          if (add_rn(add_rn(ux2, t.u2[0][jy]), uz2) < s.rcut2)
            atomicAdd(lambda + at[k], t1 * t.e[0][jy] + t2 * t.eu[0][jy]);
        },
        [](int) {});
  }
}

// The lanes' sums of 16 values in FP64: at each step a lane keeps half of its values and
// hands the other half to its partner (the butterfly's sums, at a quarter of its
// shuffles).  v[0] of lanes 2 i and 2 i + 1 is the sum of value i.
__device__ __forceinline__ void warp_sum16(double (&v)[16]) {
  const int lane = threadIdx.x & 31;
#pragma unroll
  for (int h = 8; h > 0; h >>= 1) {
    const bool up = lane & (2 * h);
#pragma unroll
    for (int i = 0; i < h; i++) {
      const double give = up ? v[i] : v[i + h];
      v[i] = (up ? v[i + h] : v[i]) + __shfl_xor_sync(0xffffffffu, give, 2 * h);
    }
  }
  v[0] += __shfl_xor_sync(0xffffffffu, v[0], 1);
}

// One atom's outputs from its sums m = {P, V (3), T0, T1 (3), Mxx, Mxy, Mxz, Myy, Myz,
// Mzz} (the cube's over Psi without the spread's prefactor, the sphere's over phi), by
// lanes 0 to 3, which hold G: dL/dq and the three dL/dx.
__device__ __forceinline__ void adj_outputs(const double* m, const double (&G)[3], double q,
                                            double pref_sp, double inv_s2, double cA, int o,
                                            double* __restrict__ dq, double* __restrict__ dx,
                                            double* __restrict__ dy, double* __restrict__ dz) {
  const int lane = threadIdx.x & 31;
  // lane 0: T1 . G; lane 1 + d: row d of M times G
  const int i0 = lane == 0 ? 5 : 7 + lane, i1 = lane == 0 ? 6 : lane == 1 ? 9 : 9 + lane,
            i2 = lane == 0 ? 7 : lane == 1 ? 10 : 10 + lane;
  const double t = m[i0] * G[0] + m[i1] * G[1] + m[i2] * G[2];
  const double Gd = lane == 1 ? G[0] : lane == 2 ? G[1] : G[2];
  double* out = lane == 0 ? dq : lane == 1 ? dx : lane == 2 ? dy : dz;
  // (r - x) = -u
  out[o] = lane == 0 ? pref_sp * m[0] + cA * t
                     : -q * pref_sp * inv_s2 * m[lane] + cA * q * (Gd * m[4] - t * inv_s2);
}

// Per atom: the cube gather of Psi = psi + gE c h^3 phi and the sphere
// gather of phi, combined into dL/dq and dL/dx.
template <typename CT>
__global__ void __launch_bounds__(32 * kAdjWarps)
    k_adj_gather(const typename Vec4<CT>::type* __restrict__ xyzq, const int* __restrict__ perm,
                 int n, Stencil<CT> sp /*spread*/, Stencil<CT> sg /*gather*/, double c,
                 double gE_ch3, const CT* __restrict__ psi, const CT* __restrict__ phi,
                 const double* __restrict__ gfx, const double* __restrict__ gfy,
                 const double* __restrict__ gfz, double* __restrict__ dq,
                 double* __restrict__ dx, double* __restrict__ dy, double* __restrict__ dz) {
  __shared__ AdjRowTab<CT> tabs[kAdjWarps];
  __shared__ double sums[kAdjWarps][16];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  AdjRowTab<CT>& t = tabs[w];
  for (int ii = blockIdx.x * kAdjWarps + w; ii < n; ii += gridDim.x * kAdjWarps) {
    const auto a = xyzq[ii];
    const int i = perm[ii];
    const CT pos[3] = {a.x, a.y, a.z};
    double G[3] = {0.0, 0.0, 0.0};
    if (lane < 4 && gfx) {
      G[0] = gfx[i];
      G[1] = gfy[i];
      G[2] = gfz[i];
    }
    const int c0x = adj_tables<CT>(pos, sp, t);
    double v[16];
#pragma unroll
    for (int k = 0; k < 16; k++) v[k] = 0.0;
    // a plane's sums over y at this lane's x offset: C over Psi, D over phi in the sphere
    double C0 = 0, Cy = 0, D0 = 0, Dy = 0, Dyy = 0, ex = 0, ux = 0;
    CT ux2 = 0, uz2 = 0;
    CT lps[kAdjRows], lph[kAdjRows];
    adj_planes<CT>(
        pos, sp, t, c0x,
        [&](int jz, CT e, CT u, CT u2) {
          ex = (double)e;
          ux = (double)u;
          ux2 = u2;
          uz2 = t.u2[1][jz];
          C0 = Cy = D0 = Dy = Dyy = 0.0;
        },
        [&](int k, long long idx) {
          lph[k] = phi[idx];
          lps[k] = psi[idx];
        },
        [&](int k, int jy) {
          const double ey = (double)t.e[0][jy], eu = (double)t.eu[0][jy];
          const double ph = (double)lph[k], ps = fma(gE_ch3, ph, (double)lps[k]);
          C0 = fma(ey, ps, C0);
          Cy = fma(eu, ps, Cy);
          if (add_rn(add_rn(ux2, t.u2[0][jy]), uz2) < sg.rcut2) {
            D0 = fma(ey, ph, D0);
            Dy = fma(eu, ph, Dy);
            Dyy = fma(eu * (double)t.u[0][jy], ph, Dyy);
          }
        },
        [&](int jz) {
          const double f = ex * (double)t.e[1][jz], z = (double)t.u[1][jz];
          const double a0 = f * C0, b0 = f * D0, by = f * Dy;
          v[0] += a0;
          v[1] = fma(a0, ux, v[1]);
          v[2] = fma(f, Cy, v[2]);
          v[3] = fma(a0, z, v[3]);
          v[4] += b0;
          v[5] = fma(b0, ux, v[5]);
          v[6] += by;
          v[7] = fma(b0, z, v[7]);
          v[8] = fma(b0, ux * ux, v[8]);
          v[9] = fma(by, ux, v[9]);
          v[10] = fma(b0, ux * z, v[10]);
          v[11] = fma(f, Dyy, v[11]);
          v[12] = fma(by, z, v[12]);
          v[13] = fma(b0, z * z, v[13]);
        });
    warp_sum16(v);
    if (!(lane & 1)) sums[w][lane >> 1] = v[0];
    __syncwarp();
    if (lane < 4)
      adj_outputs(sums[w], G, (double)a.w, (double)sp.pref, 2.0 * (double)sp.inv_2s2,
                  c * (double)sg.pref, i, dq, dx, dy, dz);
  }
}

// ===========================================================================
// Tiled reverse pass (mixed form)
// ===========================================================================
// The same brick decomposition as the forward pass.  The adjoint source is
// scattered like the charge spread (one warp per atom, lanes over (x, z)
// pairs of the stencil plane, the y values in registers) into an int32 brick
// tile that is added into an int64 grid, so lambda is bit-identical from run
// to run.  The weight of a point is e (G . u) over the gather sphere:
// separable in its y factor, e_x e_z (Gx u_x + Gz u_z) e_y + e_x e_z Gy (e_y u_y).
// The sphere test here is u_y^2 < rcut^2 - (u_x^2 + u_z^2); it may differ
// from the forward gather's association of the same sum only for points
// whose distance equals the cut-off to rounding, whose weight is e^-9 of the
// centre's.
//
// Bound: issue and latency.  256 uneven systems, 678,657 charges, both before and
// after: source 1.19 -> 1.01 ms (the y tables left the registers, 112-126 -> 64, so
// two blocks fit an SM; a block of 384 threads that spilled took 1.33 ms, two blocks
// of 256 with the tables in registers 1.23; cotangents sorted once, 9 us; additions of
// zero instead of a branch around each reduction, 0.88 -> 0.70 at width 13), gather
// 1.73 -> 1.57 ms (two x offsets per packed fma in the cube rows, the 14 lane sums by
// halves instead of 14 full butterflies, the next atom fetched ahead).

constexpr int kFusedRevThreads = 512;   // the fused reverse kernel's block
constexpr int kAdjScatterThreads = 512;  // >= kSB * kSB; 64 registers at two blocks per SM

// Blocks per SM that the source and the gather are built for: two, but one at width 15,
// whose blocks (126 KB in the source, 141 KB in the gather) leave no room for a
// second.  Bounded for two all the same, width 15 had 64 and 128 registers instead of 80
// to 109 and 175 to 200: 128 systems, 407,193 charges, source 0.909 -> 0.741 ms, gather
// 1.887 -> 1.530; one system of 164,637 charges on 144^3 0.307 -> 0.288 and 0.743 -> 0.600.
// One block at the other widths: source 0.767 -> 0.853 ms at 13, 0.734 -> 0.779 at 11.
constexpr int adj_blocks(int W) { return W < 15 ? 2 : 1; }

// Per-warp slots for the y tables of the reverse-pass scatter, one array for
// every stencil width a kernel instantiates (a static array in the templated
// function would be one per width, too much static shared memory for the
// fused reverse kernel).  Two neighbouring y points share a slot: e, e u of
// both, and u^2 of both apart.
struct AdjYTab {
  float4 w[8];
  float2 u2[8];
};
__device__ __forceinline__ AdjYTab* adj_ytab() {
  __shared__ __align__(16) AdjYTab t[kScatterThreads / 32];
  return t;
}

// The force cotangents of the sorted atoms in FP32, {Gx, Gy, Gz, |G|}: read by the
// scatter twice per atom, in order instead of by the permutation.
__device__ __forceinline__ float4 adj_cotangent(int o, const double* __restrict__ gfx,
                                                const double* __restrict__ gfy,
                                                const double* __restrict__ gfz) {
  const float x = (float)gfx[o], y = (float)gfy[o], z = (float)gfz[o];
  return make_float4(x, y, z, sqrtf(x * x + y * y + z * z));
}

__global__ void k_adj_sort_g(const int* __restrict__ perm, int n, const double* __restrict__ gfx,
                             const double* __restrict__ gfy, const double* __restrict__ gfz,
                             float4* __restrict__ gs) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
    gs[i] = adj_cotangent(perm[i], gfx, gfy, gfz);
}

static cudaError_t launch_adj_sort_g(const int* perm, int n, const double* gfx, const double* gfy,
                                     const double* gfz, float4* gs, cudaStream_t st) {
  if (n <= 0) return cudaSuccess;
  k_adj_sort_g<<<std::min((n + 255) / 256, sm_count() * 8), 256, 0, st>>>(perm, n, gfx, gfy, gfz,
                                                                         gs);
  return cudaGetLastError();
}

template <int W, int NT>
__device__ __forceinline__ void adj_scatter_brick(
    const float4* __restrict__ sorted, const float4* __restrict__ gs,
    const int* __restrict__ start, const BinLayout& b, const Stencil<float>& s, float cA, int bxi,
    int byi, int bzi, int* __restrict__ tile, long long* __restrict__ grid64, int part = 0,
    int nparts = 1) {
  typedef ScatterGeom<W> G;
  constexpr int n = G::n;
  constexpr int NW = NT / 32;
  constexpr int NPASS = (W * W + 31) / 32;
  __shared__ int rng_a[kSB * kSB], rng_p[kSB * kSB];
  __shared__ int alist[kScatterList];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int x0 = bxi * kSB, y0 = byi * kSB, z0 = bzi * kSB;
  // |cA q e (G.u)| <= |cA q| |G| max_u |u| exp(-u^2/(2 s^2)) = |cA q| |G| s e^(-1/2)
  const float acA = fabsf(cA) * sqrtf(0.5f / s.inv_2s2) * 0.60653066f * 1.0001f;
  int total;
  const int shift = brick_prologue<W, NT>(
      start, b, x0, y0, z0, tile, rng_a, rng_p,
      [&](int i) { return fabsf(sorted[i].w) * acA * gs[i].w; }, &total);
  if (part * NW >= total) return;  // (uniform) as in scatter_brick
  const float tscale = exp2f((float)shift);
  // (x, z) pairs of the stencil plane each lane tests, the same for every atom
  int psxz[NPASS];  // x | z << 8
#pragma unroll
  for (int pass = 0; pass < NPASS; pass++) {
    const int p = pass * 32 + lane;
    psxz[pass] = p < W * W ? (p - (p / W) * W) | (p / W) << 8 : 0;
  }
  // per warp: the pairs whose column meets the sphere, packed x | z << 4
  __shared__ unsigned char plist_all[NW][W * W];
  AdjYTab& ytab = adj_ytab()[warp];
  unsigned char* plist = plist_all[warp];
  for (int c0 = 0; c0 < total; c0 += kScatterList) {
    brick_atom_list<NT, kSB * kSB>(rng_a, rng_p, total, c0, kScatterList, alist);
    __syncthreads();
    const int nc = min(kScatterList, total - c0);
    for (int q = warp + part * NW; q < nc; q += NW * nparts) {
      const int ai = alist[q];
      const float4 a = sorted[ai];
      const float4 gv = gs[ai];
      const float Gx = gv.x, Gy = gv.y, Gz = gv.z;
      const float pos3[3] = {a.x, a.y, a.z};
      const int org[3] = {x0, y0, z0};
      int loc[3];
      float ul[3], u2l[3], el[3];  // lane j < W: u = x - r_j, u^2 and e along each axis
#pragma unroll
      for (int d = 0; d < 3; d++) {
        const int cc = centre_cell(pos3[d], s.inv_h[d]);
        loc[d] = wrap1(cc, s.M[d]) - org[d];
        const float u = sub_rn(pos3[d], mul_rn((float)(cc - n + lane), s.h[d]));
        const float u2 = mul_rn(u, u);
        ul[d] = u;
        u2l[d] = u2;
        el[d] = (lane < W) ? expf(mul_rn(-u2, s.inv_2s2)) : 0.f;
      }
      // the y tables every lane needs, through the warp's shared slots; read again
      // for every pass by broadcast loads (in registers, 3 W of them, they cost half
      // of the warps an SM can hold)
      __syncwarp();  // the warp's previous atom has read its tables
      if (lane < 16) {
        float* w = reinterpret_cast<float*>(&ytab.w[lane >> 1]) + (lane & 1);
        w[0] = el[1];
        w[2] = el[1] * ul[1];
        reinterpret_cast<float*>(ytab.u2)[lane] = lane < W ? u2l[1] : __int_as_float(0x7f800000);
      }
      __syncwarp();
      unsigned long long magic2;
      asm("mov.b64 %0, {%1, %1};" : "=l"(magic2) : "f"(12582912.0f));
      // compact the (x, z) pairs with u_x^2 + u_z^2 < rcut^2: every point of
      // the other columns lies outside the sphere
      int npair = 0;
#pragma unroll
      for (int pass = 0; pass < NPASS; pass++) {
        const float ux2 = __shfl_sync(0xffffffffu, u2l[0], psxz[pass] & 15);
        const float uz2 = __shfl_sync(0xffffffffu, u2l[2], psxz[pass] >> 8);
        const bool ne = pass * 32 + lane < W * W && ux2 + uz2 < s.rcut2;
        const unsigned m = __ballot_sync(0xffffffffu, ne);
        if (ne) plist[npair + __popc(m & ((1u << lane) - 1u))] =
            (unsigned char)((psxz[pass] & 15) | (psxz[pass] >> 8 << 4));
        npair += __popc(m);
      }
      __syncwarp();
      const float amp = cA * a.w * tscale;
      int* base = tile + loc[2] * G::PP + loc[1] * G::RP + loc[0];
      for (int i0 = 0; i0 < npair; i0 += 32) {
        const bool live = i0 + lane < npair;
        const int pp = live ? plist[i0 + lane] : 0;
        const int px = pp & 15, pz = pp >> 4;
        const float ex = __shfl_sync(0xffffffffu, el[0], px);
        const float ux = __shfl_sync(0xffffffffu, ul[0], px);
        const float ux2 = __shfl_sync(0xffffffffu, u2l[0], px);
        const float ez = __shfl_sync(0xffffffffu, el[2], pz);
        const float uz = __shfl_sync(0xffffffffu, ul[2], pz);
        const float uz2 = __shfl_sync(0xffffffffu, u2l[2], pz);
        if (live) {
          const float w = amp * ex * ez;
          const float t1 = w * (Gx * ux + Gz * uz), t2 = w * Gy;
          const float rem = s.rcut2 - (ux2 + uz2);
          int* cell = base + pz * G::PP + px;
          unsigned long long t1p, t2p;
          asm("mov.b64 %0, {%1, %1};" : "=l"(t1p) : "f"(t1));
          asm("mov.b64 %0, {%1, %1};" : "=l"(t2p) : "f"(t2));
#pragma unroll
          for (int k = 0; k < (W + 1) / 2; k++) {
            // |t1 e_y + t2 e_y u_y| < 2^22: both roundings stay at unit spacing;
            // two y points per packed fma, each half rounded as fmaf rounds; the
            // point past the last fails its test
            const float4 w4 = ytab.w[k];
            const float2 v2 = ytab.u2[k];
            unsigned long long e2, eu2, r2;
            asm("mov.b64 %0, {%1, %2};" : "=l"(e2) : "f"(w4.x), "f"(w4.y));
            asm("mov.b64 %0, {%1, %2};" : "=l"(eu2) : "f"(w4.z), "f"(w4.w));
            asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r2) : "l"(t2p), "l"(eu2), "l"(magic2));
            asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(r2) : "l"(t1p), "l"(e2));
            unsigned lo, hi;
            asm("mov.b64 {%0, %1}, %2;" : "=r"(lo), "=r"(hi) : "l"(r2));
            // a point outside the sphere adds zero: a reduction costs the same for one
            // lane as for all, a branch around each costs more
            atomicAdd(cell + 2 * k * G::RP, v2.x < rem ? (int)lo - 0x4B400000 : 0);
            if (2 * k + 1 < W)
              atomicAdd(cell + (2 * k + 1) * G::RP, v2.y < rem ? (int)hi - 0x4B400000 : 0);
          }
        }
      }
      __syncwarp();
    }
    __syncthreads();
  }
  brick_flush<W, NT>(tile, b, x0, y0, z0, shift, grid64);
}

// Shared memory of the reverse-pass gather for stencil width W and a block of
// NT threads.
template <int W, int NT = kAdjThreads>
struct AdjGatherGeom {
  static constexpr int n = (W - 1) / 2;
  static constexpr int TX = kAX + 2 * n, TY = kAY + 2 * n, TZ = kAZ + 2 * n;
  static constexpr int TP = TX | 1;
  static constexpr int ZP = ((TY * TP + 31) / 32) * 32 + ((W * TP) % 32);
  static constexpr int NW = NT / 32;
  static constexpr size_t bytes =
      sizeof(float) * (2 * TZ * ZP + NW * 9 * kWPad) + sizeof(int) * NW * W * W;
};

// Reverse-pass gather of the atoms of one kAX x kAY x kAZ brick: Psi = psi +
// gE c h^3 phi and phi of the brick plus halo in shared memory; a whole warp
// per atom (two atoms would need more shared memory than two blocks per SM leave for
// their tables): the cube rows of Psi (moments e, e u_x) and the sphere rows
// of phi (moments e, e u_x, e u_x^2), combined into dL/dq and dL/dx.
template <int W, int NT = kAdjThreads>
__device__ __forceinline__ void adj_gather_brick(
    const float4* __restrict__ sorted, const int* __restrict__ perm, const int* __restrict__ start,
    const BinLayout& b, const Stencil<float>& sp, const Stencil<float>& sg, double c,
    double gE_ch3, const float* __restrict__ psi, const float* __restrict__ phi,
    const double* __restrict__ gfx, const double* __restrict__ gfy,
    const double* __restrict__ gfz, double* __restrict__ dq, double* __restrict__ dx,
    double* __restrict__ dy, double* __restrict__ dz, int bxi, int byi, int bzi,
    unsigned char* smem) {
  typedef AdjGatherGeom<W, NT> AG;
  constexpr int n = AG::n, TX = AG::TX, TY = AG::TY, TZ = AG::TZ, TP = AG::TP, ZP = AG::ZP;
  constexpr int NW = AG::NW;
  constexpr int NR = kAY * kAZ;
  constexpr int NG = (W * W + 31) / 32;
  float* tpsi = (float*)smem;                        // [TZ][ZP]
  float* tphi = tpsi + TZ * ZP;                      // [TZ][ZP]
  float* tabs = tphi + TZ * ZP;                      // [NW][axis][u, u^2, e][kWPad]
  int* rowl = (int*)(tabs + NW * 9 * kWPad);         // [NW][W*W]
  __shared__ int rng_a[NR], rng_p[NR + 1];
  __shared__ int alist[kGatherList];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int x0 = bxi * kAX, y0 = byi * kAY, z0 = bzi * kAZ;
  const int ex = min(kAX, b.M[0] - x0), ey = min(kAY, b.M[1] - y0), ez = min(kAZ, b.M[2] - z0);
  int cnt = 0;
  if (tid < NR) {
    const int yy = tid % kAY, zz = tid / kAY;
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
  if (natoms == 0) return;  // uniform
  stage_tile_async<float, TX, TY, TZ, TP, ZP, NW>(psi, b, x0, y0, z0, n, tpsi);
  stage_tile_async<float, TX, TY, TZ, TP, ZP, NW>(phi, b, x0, y0, z0, n, tphi);
  asm volatile("cp.async.wait_all;" ::: "memory");
  __syncthreads();
  {
    const float g = (float)gE_ch3;
    for (int i = tid; i < TZ * ZP; i += NT) tpsi[i] = fmaf(g, tphi[i], tpsi[i]);
  }
  __syncthreads();

  float* tb = tabs + warp * 9 * kWPad;
  int* rl = rowl + warp * W * W;
  int gjy[NG], gjz[NG];
#pragma unroll
  for (int g = 0; g < NG; g++) {
    const int r = g * 32 + lane;
    gjz[g] = r < W * W ? r / W : 0;
    gjy[g] = r < W * W ? r - (r / W) * W : 0;
  }
  const double pref_sp = (double)sp.pref, inv_s2 = 2.0 * (double)sp.inv_2s2;
  const double cA = c * (double)sg.pref;
  for (int c0 = 0; c0 < natoms; c0 += kGatherList) {
    brick_atom_list<NT, NR>(rng_a, rng_p, natoms, c0, kGatherList, alist);
    __syncthreads();
    const int nc = min(kGatherList, natoms - c0);
    // the next atom's record and output slot are loaded one iteration ahead, this
    // atom's cotangents (by the slot) ahead of its sums, which need them last
    float4 a_n;
    int o_n = 0;
    if (warp < nc) {
      a_n = sorted[alist[warp]];
      o_n = perm[alist[warp]];
    }
    for (int q = warp; q < nc; q += NW) {
      const float4 a = a_n;
      const int o = o_n;
      double G[3] = {0.0, 0.0, 0.0};
      if (lane < 4 && gfx) {
        G[0] = gfx[o];
        G[1] = gfy[o];
        G[2] = gfz[o];
      }
      if (q + NW < nc) {
        a_n = sorted[alist[q + NW]];
        o_n = perm[alist[q + NW]];
      }
      const float pos3[3] = {a.x, a.y, a.z};
      const int org[3] = {x0, y0, z0};
      int loc[3];
#pragma unroll
      for (int d = 0; d < 3; d++) {
        const int cc = centre_cell(pos3[d], sp.inv_h[d]);
        loc[d] = wrap1(cc, sp.M[d]) - org[d];
        for (int j = lane; j < W; j += 32) {
          const float u = sub_rn(pos3[d], mul_rn((float)(cc - n + j), sp.h[d]));
          const float u2 = mul_rn(u, u);
          tb[(d * 3 + 0) * kWPad + j] = u;
          tb[(d * 3 + 1) * kWPad + j] = u2;
          tb[(d * 3 + 2) * kWPad + j] = expf(mul_rn(-u2, sp.inv_2s2));
        }
      }
      __syncwarp();
      // (e_x, e_x u_x) per x offset, as scalars and in pairs of offsets
      float ex[W], eux[W];
      unsigned long long e2[W / 2], eu2p[W / 2];
#pragma unroll
      for (int k = 0; k < W; k++) {
        ex[k] = tb[(0 * 3 + 2) * kWPad + k];
        eux[k] = ex[k] * tb[(0 * 3 + 0) * kWPad + k];
      }
#pragma unroll
      for (int k = 0; k < W / 2; k++) {
        asm("mov.b64 %0, {%1, %2};" : "=l"(e2[k]) : "f"(ex[2 * k]), "f"(ex[2 * k + 1]));
        asm("mov.b64 %0, {%1, %2};" : "=l"(eu2p[k]) : "f"(eux[2 * k]), "f"(eux[2 * k + 1]));
      }
      // cube rows of Psi: P = sum e Psi, V = sum e Psi u, two offsets per packed fma
      // (a lane's rows summed in FP32, the lanes' sums in FP64 below)
      float P = 0.f, Vx = 0.f, Vy = 0.f, Vz = 0.f;
#pragma unroll
      for (int g = 0; g < NG; g++) {
        if (g * 32 + lane < W * W) {
          const int jy = gjy[g], jz = gjz[g];
          const float* row = tpsi + (loc[2] + jz) * ZP + (loc[1] + jy) * TP + loc[0];
          unsigned long long s0 = 0ull, s1 = 0ull;
#pragma unroll
          for (int k = 0; k < W / 2; k++) {
            unsigned long long p2;
            asm("mov.b64 %0, {%1, %2};" : "=l"(p2) : "f"(row[2 * k]), "f"(row[2 * k + 1]));
            asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(s0) : "l"(e2[k]), "l"(p2));
            asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(s1) : "l"(eu2p[k]), "l"(p2));
          }
          float r0, r0b, r1, r1b;
          asm("mov.b64 {%0, %1}, %2;" : "=f"(r0), "=f"(r0b) : "l"(s0));
          asm("mov.b64 {%0, %1}, %2;" : "=f"(r1), "=f"(r1b) : "l"(s1));
          r0 = fmaf(ex[W - 1], row[W - 1], r0 + r0b);
          r1 = fmaf(eux[W - 1], row[W - 1], r1 + r1b);
          const float w = tb[(1 * 3 + 2) * kWPad + jy] * tb[(2 * 3 + 2) * kWPad + jz];
          const float a0 = w * r0;
          P += a0;
          Vx += w * r1;
          Vy += a0 * tb[(1 * 3 + 0) * kWPad + jy];
          Vz += a0 * tb[(2 * 3 + 0) * kWPad + jz];
        }
      }
      // sphere rows of phi
      int nrow = 0;
#pragma unroll
      for (int g = 0; g < NG; g++) {
        const int r = g * 32 + lane;
        bool ne = false;
        if (r < W * W)
          ne = add_rn(tb[(1 * 3 + 1) * kWPad + gjy[g]], tb[(2 * 3 + 1) * kWPad + gjz[g]]) <
               sg.rcut2;
        const unsigned m = __ballot_sync(0xffffffffu, ne);
        if (ne) rl[nrow + __popc(m & ((1u << lane) - 1u))] = (gjz[g] << 8) | gjy[g];
        nrow += __popc(m);
      }
      __syncwarp();
      float dx2[W], eu2[W];
#pragma unroll
      for (int k = 0; k < W; k++) {
        dx2[k] = tb[(0 * 3 + 1) * kWPad + k];
        eu2[k] = ex[k] * dx2[k];
      }
      float T0 = 0, T1x = 0, T1y = 0, T1z = 0;
      float Mxx = 0, Mxy = 0, Mxz = 0, Myy = 0, Myz = 0, Mzz = 0;
      // the end points lie outside the sphere for every row when dx^2 >= rcut^2
      // there (rem <= rcut^2): the rows are then summed over the inner points
      const bool ends = dx2[0] < sg.rcut2 || dx2[W - 1] < sg.rcut2;
      const bool trim = !__any_sync(0xffffffffu, ends);
      for (int i = lane; i < nrow; i += 32) {
        const int r = rl[i];
        const int jz = r >> 8, jy = r & 255;
        const float uy2 = tb[(1 * 3 + 1) * kWPad + jy], uz2 = tb[(2 * 3 + 1) * kWPad + jz];
        const float rem = sg.rcut2 - (uy2 + uz2);
        const float* row = tphi + (loc[2] + jz) * ZP + (loc[1] + jy) * TP + loc[0];
        float s0 = 0.f, s1 = 0.f, s2 = 0.f;
        auto pts = [&](auto tr) {
          constexpr int K0 = decltype(tr)::value ? 1 : 0;
          constexpr int K1 = decltype(tr)::value ? W - 1 : W;
#pragma unroll
          for (int k = K0; k < K1; k++) {
            const float ph = row[k];
            if (dx2[k] < rem) {  // the test guards the fmas; a skipped point adds nothing
              s0 = fmaf(ex[k], ph, s0);
              s1 = fmaf(eux[k], ph, s1);
              s2 = fmaf(eu2[k], ph, s2);
            }
          }
        };
        if (trim)
          pts(std::true_type());
        else
          pts(std::false_type());
        const float w = tb[(1 * 3 + 2) * kWPad + jy] * tb[(2 * 3 + 2) * kWPad + jz];
        const float uy = tb[(1 * 3 + 0) * kWPad + jy], uz = tb[(2 * 3 + 0) * kWPad + jz];
        const float a0 = w * s0, a1 = w * s1;
        T0 += a0;
        T1x += a1;
        T1y += a0 * uy;
        T1z += a0 * uz;
        Mxx += w * s2;
        Mxy += a1 * uy;
        Mxz += a1 * uz;
        Myy += a0 * uy2;
        Myz += a0 * uy * uz;
        Mzz += a0 * uz2;
      }
      // lane 2 i then holds value i, and the first four lanes form one output each
      double v[16] = {P, Vx, Vy, Vz, T0, T1x, T1y, T1z, Mxx, Mxy, Mxz, Myy, Myz, Mzz, 0.0, 0.0};
      warp_sum16(v);
      double* m = reinterpret_cast<double*>(tb);  // the atom's tables are used up
      __syncwarp();
      if (!(lane & 1)) m[lane >> 1] = v[0];
      __syncwarp();
      if (lane < 4)
        adj_outputs(m, G, (double)a.w, pref_sp, inv_s2, cA, o, dq, dx, dy, dz);
      __syncwarp();
    }
    __syncthreads();
  }
}

template <int W>
__global__ void __launch_bounds__(kAdjScatterThreads, adj_blocks(W))
    k_adj_scatter(const float4* __restrict__ sorted, const float4* __restrict__ gs,
                  const int* __restrict__ start, BinLayout b, Stencil<float> s, float cA,
                  int nparts, long long* __restrict__ grid64) {
  extern __shared__ int atile[];
  adj_scatter_brick<W, kAdjScatterThreads>(sorted, gs, start, b, s, cA, blockIdx.x / nparts,
                                           blockIdx.y, blockIdx.z, atile, grid64,
                                           blockIdx.x % nparts, nparts);
}

template <int W>
__global__ void __launch_bounds__(kAdjThreads, adj_blocks(W))
    k_adj_gather_tiled(const float4* __restrict__ sorted, const int* __restrict__ perm,
                       const int* __restrict__ start, BinLayout b, Stencil<float> sp,
                       Stencil<float> sg, double c, double gE_ch3, const float* __restrict__ psi,
                       const float* __restrict__ phi, const double* __restrict__ gfx,
                       const double* __restrict__ gfy, const double* __restrict__ gfz,
                       double* __restrict__ dq, double* __restrict__ dx, double* __restrict__ dy,
                       double* __restrict__ dz) {
  extern __shared__ __align__(16) unsigned char asm_[];
  adj_gather_brick<W>(sorted, perm, start, b, sp, sg, c, gE_ch3, psi, phi, gfx, gfy, gfz, dq, dx,
                      dy, dz, blockIdx.x, blockIdx.y, blockIdx.z, asm_);
}

template <int W>
__global__ void __launch_bounds__(kAdjScatterThreads, adj_blocks(W))
    k_batch_adj_scatter(const float4* __restrict__ sorted, const float4* __restrict__ gs,
                        const int* __restrict__ start, const BatchSys* __restrict__ sys,
                        const BatchItem* __restrict__ items, int nitems, double c,
                        long long* __restrict__ grid64) {
  extern __shared__ int atile[];
  for (int it = blockIdx.x; it < nitems; it += gridDim.x) {
    const BatchItem item = items[it];
    const BatchSys& S = sys[item.sys];
    const float cA = (float)(c * (double)S.sg.pref);
    adj_scatter_brick<W, kAdjScatterThreads>(sorted, gs, start + S.bin_off, S.b, S.sg, cA, item.bx,
                                             item.by, item.bz, atile, grid64 + S.grid_off);
    __syncthreads();
  }
}

template <int W>
__global__ void __launch_bounds__(kAdjThreads, adj_blocks(W))
    k_batch_adj_gather_tiled(const float4* __restrict__ sorted, const int* __restrict__ perm,
                             const int* __restrict__ start, const BatchSys* __restrict__ sys,
                             const BatchItem* __restrict__ items, int nitems, double c,
                             const double* __restrict__ dLdE, const float* __restrict__ psi,
                             const float* __restrict__ phi, const double* __restrict__ gfx,
                             const double* __restrict__ gfy, const double* __restrict__ gfz,
                             double* __restrict__ dq, double* __restrict__ dx,
                             double* __restrict__ dy, double* __restrict__ dz) {
  extern __shared__ __align__(16) unsigned char asm_[];
  for (int it = blockIdx.x; it < nitems; it += gridDim.x) {
    const BatchItem item = items[it];
    const BatchSys& S = sys[item.sys];
    const double gE_ch3 = dLdE[item.sys] * c * S.h3;
    adj_gather_brick<W>(sorted, perm, start + S.bin_off, S.b, S.sp, S.sg, c, gE_ch3,
                        psi + S.grid_off, phi + S.grid_off, gfx, gfy, gfz, dq, dx, dy, dz, item.bx,
                        item.by, item.bz, asm_);
    __syncthreads();
  }
}

namespace {
template <class K>
cudaError_t set_smem_once(K kernel, size_t bytes, std::atomic<bool>* done) {
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
cudaError_t adj_scatter_w(const float4* sorted, const float4* gs, const int* start,
                          const BinLayout& b, const Stencil<float>& s, double c,
                          long long* grid64, float* lambda, cudaStream_t st) {
  static std::atomic<bool> done[64];
  const size_t smem = sizeof(int) * ScatterGeom<W>::words;
  cudaError_t e = set_smem_once(k_adj_scatter<W>, smem, done);
  if (e != cudaSuccess) return e;
  const long long size = (long long)b.M[0] * b.M[1] * b.M[2];
  e = cudaMemsetAsync(grid64, 0, sizeof(long long) * size, st);
  if (e != cudaSuccess) return e;
  dim3 grd((b.M[0] + kSB - 1) / kSB, (b.M[1] + kSB - 1) / kSB, (b.M[2] + kSB - 1) / kSB);
  const int nparts = scatter_parts((long long)grd.x * grd.y * grd.z, W);
  grd.x *= nparts;
  k_adj_scatter<W><<<grd, kAdjScatterThreads, smem, st>>>(
      sorted, gs, start, b, s, (float)(c * (double)s.pref), nparts, grid64);
  e = cudaGetLastError();
  if (e != cudaSuccess || !lambda) return e;
  return launch_grid64_to_real(grid64, size, lambda, st);
}

template <int W>
cudaError_t adj_gather_w(const float4* sorted, const int* perm, const int* start,
                         const BinLayout& b, const Stencil<float>& sp, const Stencil<float>& sg,
                         double c, double gE_ch3, const float* psi, const float* phi,
                         const double* gfx, const double* gfy, const double* gfz, double* dq,
                         double* dx, double* dy, double* dz, cudaStream_t st) {
  static std::atomic<bool> done[64];
  const size_t smem = AdjGatherGeom<W>::bytes;
  const cudaError_t e = set_smem_once(k_adj_gather_tiled<W>, smem, done);
  if (e != cudaSuccess) return e;
  const dim3 grd((b.M[0] + kAX - 1) / kAX, (b.M[1] + kAY - 1) / kAY, (b.M[2] + kAZ - 1) / kAZ);
  k_adj_gather_tiled<W><<<grd, kAdjThreads, smem, st>>>(sorted, perm, start, b, sp, sg, c, gE_ch3,
                                                        psi, phi, gfx, gfy, gfz, dq, dx, dy, dz);
  return cudaGetLastError();
}
}  // namespace

cudaError_t launch_adj_scatter(const float4* sorted, const int* perm, int n, const int* start,
                               const BinLayout& b, const Stencil<float>& sg, double c,
                               const double* gfx, const double* gfy, const double* gfz,
                               float4* gs, long long* grid64, float* lambda, cudaStream_t st) {
  const cudaError_t e = launch_adj_sort_g(perm, n, gfx, gfy, gfz, gs, st);
  if (e != cudaSuccess) return e;
  switch (2 * sg.nst[0] + 1) {
    case 9: return adj_scatter_w<9>(sorted, gs, start, b, sg, c, grid64, lambda, st);
    case 11: return adj_scatter_w<11>(sorted, gs, start, b, sg, c, grid64, lambda, st);
    case 13: return adj_scatter_w<13>(sorted, gs, start, b, sg, c, grid64, lambda, st);
    case 15: return adj_scatter_w<15>(sorted, gs, start, b, sg, c, grid64, lambda, st);
  }
  return cudaErrorInvalidValue;
}

cudaError_t launch_adj_gather_tiled(const float4* sorted, const int* perm, const int* start,
                                    const BinLayout& b, const Stencil<float>& sp,
                                    const Stencil<float>& sg, double c, double gE_ch3,
                                    const float* psi, const float* phi, const double* gfx,
                                    const double* gfy, const double* gfz, double* dq, double* dx,
                                    double* dy, double* dz, cudaStream_t st) {
  switch (2 * sp.nst[0] + 1) {
    case 9: return adj_gather_w<9>(sorted, perm, start, b, sp, sg, c, gE_ch3, psi, phi, gfx, gfy, gfz, dq, dx, dy, dz, st);
    case 11: return adj_gather_w<11>(sorted, perm, start, b, sp, sg, c, gE_ch3, psi, phi, gfx, gfy, gfz, dq, dx, dy, dz, st);
    case 13: return adj_gather_w<13>(sorted, perm, start, b, sp, sg, c, gE_ch3, psi, phi, gfx, gfy, gfz, dq, dx, dy, dz, st);
    case 15: return adj_gather_w<15>(sorted, perm, start, b, sp, sg, c, gE_ch3, psi, phi, gfx, gfy, gfz, dq, dx, dy, dz, st);
  }
  return cudaErrorInvalidValue;
}

cudaError_t launch_batch_adj_scatter(const float4* sorted, const int* perm, int ntot,
                                     const int* start, const BatchSys* sys,
                                     const BatchItem* items, const BatchSeg* segs, int nseg,
                                     int ctas, double c, const double* gfx, const double* gfy,
                                     const double* gfz, float4* gs, long long* grid64,
                                     long long gsize, float* lambda, cudaStream_t st) {
  cudaError_t e = launch_adj_sort_g(perm, ntot, gfx, gfy, gfz, gs, st);
  if (e != cudaSuccess) return e;
  e = cudaMemsetAsync(grid64, 0, sizeof(long long) * gsize, st);
  if (e != cudaSuccess) return e;
  for (int k = 0; k < nseg; k++) {
    const BatchItem* it = items + segs[k].first;
    const int cnt = std::min(ctas, segs[k].count), ni = segs[k].count;
    if (ni <= 0) continue;
#define GSE_BAS(WW)                                                                          \
  case WW: {                                                                                 \
    static std::atomic<bool> done[64];                                                               \
    const size_t smem = sizeof(int) * ScatterGeom<WW>::words;                                \
    e = set_smem_once(k_batch_adj_scatter<WW>, smem, done);                                  \
    if (e == cudaSuccess)                                                                    \
      k_batch_adj_scatter<WW><<<cnt, kAdjScatterThreads, smem, st>>>(                   \
          sorted, gs, start, sys, it, ni, c, grid64);                                        \
    break;                                                                                   \
  }
    switch (segs[k].W) {
      GSE_BAS(9)
      GSE_BAS(11)
      GSE_BAS(13)
      GSE_BAS(15)
      default: e = cudaErrorInvalidValue;
    }
#undef GSE_BAS
    if (e != cudaSuccess) return e;
    e = cudaGetLastError();
    if (e != cudaSuccess) return e;
  }
  return launch_grid64_to_real(grid64, gsize, lambda, st);
}

cudaError_t launch_batch_adj_gather_tiled(const float4* sorted, const int* perm, const int* start,
                                          const BatchSys* sys, const BatchItem* items,
                                          const BatchSeg* segs, int nseg, int ctas, double c,
                                          const double* dLdE, const float* psi, const float* phi,
                                          const double* gfx, const double* gfy, const double* gfz,
                                          double* dq, double* dx, double* dy, double* dz,
                                          cudaStream_t st) {
  for (int k = 0; k < nseg; k++) {
    const BatchItem* it = items + segs[k].first;
    const int cnt = std::min(ctas, segs[k].count), ni = segs[k].count;
    if (ni <= 0) continue;
    cudaError_t e;
#define GSE_BAG(WW)                                                                          \
  case WW: {                                                                                 \
    static std::atomic<bool> done[64];                                                               \
    const size_t smem = AdjGatherGeom<WW>::bytes;                                            \
    e = set_smem_once(k_batch_adj_gather_tiled<WW>, smem, done);                             \
    if (e == cudaSuccess)                                                                    \
      k_batch_adj_gather_tiled<WW><<<cnt, kAdjThreads, smem, st>>>(                          \
          sorted, perm, start, sys, it, ni, c, dLdE, psi, phi, gfx, gfy, gfz, dq, dx, dy, dz);   \
    break;                                                                                   \
  }
    switch (segs[k].W) {
      GSE_BAG(9)
      GSE_BAG(11)
      GSE_BAG(13)
      GSE_BAG(15)
      default: e = cudaErrorInvalidValue;
    }
#undef GSE_BAG
    if (e != cudaSuccess) return e;
    e = cudaGetLastError();
    if (e != cudaSuccess) return e;
  }
  return cudaSuccess;
}


// ---------------------------------------------------------------------------
// Reverse pass of a batch in one persistent cooperative launch (grids of at
// most 64 points, multiples of 8, per side): the adjoint source of every
// system into the int64 grid, its solve with the Green's function, and the
// reverse-pass gather.  Reads the forward pass's sorted atoms, bins and
// potential.
// ---------------------------------------------------------------------------
static_assert(kFusedRevThreads == kScatterThreads, "the fused kernel runs the scatter bricks");

constexpr size_t cmax_rev(size_t a, size_t b) { return a > b ? a : b; }
constexpr size_t fused_rev_smem() {
  return cmax_rev(
      cmax_rev(cmax_rev(sizeof(int) * ScatterGeom<9>::words, sizeof(int) * ScatterGeom<11>::words),
               cmax_rev(sizeof(int) * ScatterGeom<13>::words, sizeof(int) * ScatterGeom<15>::words)),
      cmax_rev(cmax_rev(cmax_rev(AdjGatherGeom<9, kFusedRevThreads>::bytes,
                                 AdjGatherGeom<11, kFusedRevThreads>::bytes),
                        cmax_rev(AdjGatherGeom<13, kFusedRevThreads>::bytes,
                                 AdjGatherGeom<15, kFusedRevThreads>::bytes)),
               sizeof(SmallFftTw) + sizeof(int) * 3 * (kSfSmemSystems + 1)));
}

__global__ void __launch_bounds__(kFusedRevThreads, 1) k_batch_reverse_fused(BatchFused a) {
  namespace cg = cooperative_groups;
  extern __shared__ __align__(16) unsigned char fsm[];
  const long long gtid = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  const long long gstride = (long long)gridDim.x * blockDim.x;
  for (long long i = gtid; i < a.gtot; i += gstride) a.g64[i] = 0;
  for (long long i = gtid; i < a.ntot; i += gstride)
    a.gs[i] = adj_cotangent(a.perm[i], a.gfx, a.gfy, a.gfz);
  if (gtid < 2) a.qctr[2 + gtid] = 0;
  cg::this_grid().sync();
  for (int it = fused_next_item(&a.qctr[2]); it < a.nscat; it = fused_next_item(&a.qctr[2])) {
    const BatchItem item = a.scat[it];
    const BatchSys& S = a.sys[item.sys];
    const int* st = a.w.start + S.bin_off;
    long long* g = a.g64 + S.grid_off;
    int* tile = reinterpret_cast<int*>(fsm);
    const float cA = (float)(a.ccelec * (double)S.sg.pref);
    switch (S.W) {
      case 9: adj_scatter_brick<9, kFusedRevThreads>(
          a.sorted, a.gs, st, S.b, S.sg, cA, item.bx, item.by, item.bz, tile, g); break;
      case 11: adj_scatter_brick<11, kFusedRevThreads>(
          a.sorted, a.gs, st, S.b, S.sg, cA, item.bx, item.by, item.bz, tile, g); break;
      case 13: adj_scatter_brick<13, kFusedRevThreads>(
          a.sorted, a.gs, st, S.b, S.sg, cA, item.bx, item.by, item.bz, tile, g); break;
      default: adj_scatter_brick<15, kFusedRevThreads>(
          a.sorted, a.gs, st, S.b, S.sg, cA, item.bx, item.by, item.bz, tile, g); break;
    }
    __syncthreads();
  }
  cg::this_grid().sync();
  fused_solve(a, a.psi, false, fsm);
  cg::this_grid().sync();
  for (int it = fused_next_item(&a.qctr[3]); it < a.nagath; it = fused_next_item(&a.qctr[3])) {
    const BatchItem item = a.agath[it];
    const BatchSys& S = a.sys[item.sys];
    const int* st = a.w.start + S.bin_off;
    const double gE_ch3 = a.dLdE[item.sys] * a.ccelec * S.h3;
    const float* ps = a.psi + S.grid_off;
    const float* ph = a.phi + S.grid_off;
    switch (S.W) {
#define GSE_FAG(WW)                                                                          \
  case WW:                                                                                   \
    adj_gather_brick<WW, kFusedRevThreads>(a.sorted, a.perm, st, S.b, S.sp, S.sg, a.ccelec,  \
                                           gE_ch3, ps, ph, a.gfx, a.gfy, a.gfz, a.dq, a.dx,  \
                                           a.dy, a.dz, item.bx, item.by, item.bz, fsm);      \
    break;
      GSE_FAG(9)
      GSE_FAG(11)
      GSE_FAG(13)
      default:
        adj_gather_brick<15, kFusedRevThreads>(a.sorted, a.perm, st, S.b, S.sp, S.sg, a.ccelec,
                                               gE_ch3, ps, ph, a.gfx, a.gfy, a.gfz, a.dq, a.dx,
                                               a.dy, a.dz, item.bx, item.by, item.bz, fsm);
        break;
#undef GSE_FAG
    }
    __syncthreads();
  }
}

int batch_fused_rev_ctas() {
  static std::atomic<int> cache[64];
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) {
    cudaGetLastError();
    return 0;
  }
  int v = cache[dev].load();
  if (v == 0) {
    const size_t smem = fused_rev_smem();
    int nb = 0;
    if (cudaFuncSetAttribute(k_batch_reverse_fused, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             (int)smem) != cudaSuccess ||
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, k_batch_reverse_fused,
                                                      kFusedRevThreads, smem) != cudaSuccess) {
      cudaGetLastError();
      nb = 0;
    }
    v = nb > 0 ? nb * sm_count() : -1;
    cache[dev].store(v);
  }
  return v > 0 ? v : 0;
}

cudaError_t launch_batch_reverse_fused(const BatchFused& a, int ctas, cudaStream_t st) {
  const int most = batch_fused_rev_ctas();
  if (most <= 0 || ctas < 1 || ctas > most) return cudaErrorCooperativeLaunchTooLarge;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(ctas);
  cfg.blockDim = dim3(kFusedRevThreads);
  cfg.dynamicSmemBytes = fused_rev_smem();
  cfg.stream = st;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeCooperative;
  attr[0].val.cooperative = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, k_batch_reverse_fused, a);
}

template <typename CT>
cudaError_t launch_adj_source(const typename Vec4<CT>::type* xyzq, const int* perm, int n,
                              const Stencil<CT>& s, double c, const double* gfx,
                              const double* gfy, const double* gfz, CT* lambda, cudaStream_t st) {
  if (n <= 0) return cudaSuccess;
  const int blocks = (int)std::min<long long>(sm_count() * 16, (n + 7) / 8);
  k_adj_source<CT><<<blocks, 32 * kAdjWarps, 0, st>>>(xyzq, perm, n, s, c, gfx, gfy, gfz, lambda);
  return cudaGetLastError();
}

template <typename CT>
cudaError_t launch_adj_gather(const typename Vec4<CT>::type* xyzq, const int* perm, int n,
                              const Stencil<CT>& sp, const Stencil<CT>& sg, double c,
                              double gE_ch3, const CT* psi, const CT* phi, const double* gfx,
                              const double* gfy, const double* gfz, double* dq, double* dx,
                              double* dy, double* dz, cudaStream_t st) {
  if (n <= 0) return cudaSuccess;
  const int blocks = (int)std::min<long long>(sm_count() * 16, (n + 7) / 8);
  k_adj_gather<CT><<<blocks, 32 * kAdjWarps, 0, st>>>(xyzq, perm, n, sp, sg, c, gE_ch3, psi, phi, gfx, gfy,
                                           gfz, dq, dx, dy, dz);
  return cudaGetLastError();
}

#define GSE_ADJ_INST(CT)                                                                        \
  template cudaError_t launch_adj_source<CT>(const Vec4<CT>::type*, const int*, int,           \
                                             const Stencil<CT>&, double, const double*,          \
                                             const double*, const double*, CT*, cudaStream_t);   \
  template cudaError_t launch_adj_gather<CT>(const Vec4<CT>::type*, const int*, int,           \
                                             const Stencil<CT>&, const Stencil<CT>&, double,     \
                                             double, const CT*, const CT*, const double*,        \
                                             const double*, const double*, double*, double*,     \
                                             double*, double*, cudaStream_t);

GSE_ADJ_INST(double)
GSE_ADJ_INST(float)

}  // namespace gse
