// gse_tiled.cuh -- tiled spread / gather kernels and the atom binning they use.
#pragma once

#include <cuda_runtime.h>

#include <vector>

#include "gse_internal.cuh"

namespace gse {

// x cells per bin (y and z bins are single cells): the FP64 spread reads atom
// ranges at 4-cell granularity; every mixed-form kernel reads whole 16-cell
// brick rows, so the mixed form bins 16 cells at a time (4x fewer bins to scan)
constexpr int kBinX64 = 4, kBinX32 = 16;
constexpr int kWPad = 16;           // padded stencil width (2n+1 <= 15 on the tiled path)
constexpr int kGX = 16, kGY = 16, kGZ = 8;  // gather brick (cells); kGX multiple of kBinX32
constexpr int kGatherThreads = 384;          // >= kGY * kGZ
constexpr int kGatherLanes = 16;             // lanes sharing one atom in the gather
constexpr int kMinTiledGrid = 10;   // smallest grid side on the tiled path
constexpr int kSB = 16;             // scatter-spread brick (cells per axis)
constexpr int kFlushBits = 40;  // scale of the int64 accumulation grids
constexpr int kScatterThreads = 512;  // >= kSB * kSB
constexpr int kScatterList = 1024;  // atoms per scatter round (per brick)
constexpr int kGatherList = 512;    // atoms per gather round (per brick)
constexpr int kAX = 16, kAY = 8, kAZ = 8;  // reverse-pass gather brick (two staged grids)
constexpr int kAdjThreads = 256;           // >= kAY * kAZ

// Atoms sorted by key (z cell, y cell, x bin); start[k] .. start[k+1] is bin k.
struct BinLayout {
  int M[3];
  int nbx;    // ceil(Mx / bin width)
  int bxs;    // log2 of the bin width in x cells
  // mixed-form scatter: set to kFlagRange when a brick's charge exceeds the
  // fixed-point range of its int32 tile (may be NULL: not reported)
  int* flags = nullptr;
};

// What the FP64 spread needs of an atom: per axis the weight of the stencil's
// centre point (x: times q pref) and the two ratios from which the axis' other
// weights follow, then the wrapped x cell.  Formed once per atom here instead of
// by every block that the atom's cube reaches (5.4 blocks of 16^3 points at n = 6).
constexpr int kBasis64 = 10;
struct SpreadBasis {
  double h[3], inv_2s2, pref;
  int nst;      // stencil half width n
  double* out;  // [n][kBasis64] in sorted order; NULL: not wanted
};

struct BinScratch {
  int* key;        // [n]
  int* counts;     // [nbins], zero on entry and again after the placement
  int* start;      // [nbins + 1]
  int* tile_sums;  // [ceil(nbins / 4096)]
  int* tmp;        // [n]: the mixed form's ranks in bin; the FP64 form's unordered placement
  int* lstart;     // [nbins]: the scan's tile-local prefix
  int* bad = nullptr;   // set to 1 when a position or charge is not finite (may be NULL)
  // an int64 array of clear_n elements (16-byte aligned) that the counting
  // kernel clears on the way (the mixed form's spread grid); NULL: none
  long long* clear = nullptr;
  long long clear_n = 0;
  // FP64 form: weights' basis of the sorted atoms, for the spread that follows
  SpreadBasis basis = {};
};

// Where the counting kernel leaves each atom's rank in its bin: the FP64 form's perm
// is written after the ranks are read, its tmp before.
template <typename CT>
inline int* bin_rank(const BinScratch& w, int* perm) {
  return sizeof(CT) == 8 ? perm : w.tmp;
}

// Few atoms in few bins are binned by one block in one launch: an atom per thread, the
// bins in shared memory within the 48 KB that need no opt-in.  Launches bound these
// calls; against the three or four launches of the general path an energy-force call
// takes (FP64) 37.0 instead of 41.1 us for 2 atoms on 20^3, 49.3 / 53.4 for 300 on 20^3;
// with 1000 atoms, past the FP64 limit, it took 65.7 / 66.7 on 24^3 and 58.8 / 57.6 on 32^3
// (the nine exponentials per atom then keep the one SM busy for longer than the launches
// saved), which set that limit; mixed 41.2 / 43.2 for 100 on 16^3, 55.4 / 57.5 for 1000
// on 24^3, 53.6 / 57.5 on 32^3.
constexpr int kBinSmall = 1024;
inline bool bin_small(bool fp64, int n, int nb) {
  return n <= (fp64 ? kBinSmall / 2 : kBinSmall) && nb <= 10240;
}

inline BinLayout make_bin_layout(const int M[3], int bin_width) {
  BinLayout b;
  for (int d = 0; d < 3; d++) b.M[d] = M[d];
  b.bxs = bin_width == 16 ? 4 : 2;
  b.nbx = (M[0] + (1 << b.bxs) - 1) >> b.bxs;
  return b;
}
static_assert(kGX % kBinX32 == 0 && kSB % kBinX32 == 0 && kAX % kBinX32 == 0,
              "mixed-form bricks start on bin boundaries");

inline int bin_count(const BinLayout& b) { return b.M[1] * b.M[2] * b.nbx; }

// One system of a batch (mixed form).  Atoms of all systems are binned with
// one global key: bin_off + the system's own (z cell, y cell, x bin) key.
struct BatchSys {
  BinLayout b;
  int bin_off;          // first bin of the system
  int atom_off, n;      // atom range in the caller's concatenated order
  int W;                // stencil width 2n+1
  long long grid_off;   // first point of the system's real grids
  long long kgrid_off;  // first bin of its half spectrum
  double efac;          // 1/2 ccelec hx hy hz
  double h3;            // hx hy hz
  Stencil<float> sp;    // spread stencil (sigma1, rcut1)
  Stencil<float> sg;    // gather stencil
};

struct BatchItem {
  int sys, bx, by, bz;  // brick of one system
};

// A run of work items whose systems share one stencil width W (the batched
// kernels are instantiated per width; one launch per run).
struct BatchSeg {
  int W, first, count;
};

// The batched evaluation in one persistent cooperative launch per direction:
// binning, spread, the small-grid FFT solve with the Green's multiply and
// energy, and gather (forward), or adjoint source, solve and reverse-pass
// gather (reverse), separated by grid-wide barriers.  Grids must be multiples
// of 8 and at most 64 points per side (batch_fused_supported).
struct BatchFused {
  const float4* xyzq;
  int ntot, nsys, nbins;
  const BatchSys* sys;
  const int* first;         // [nsys + 1] first atom of each system
  BinScratch w;
  float4* sorted;
  int* perm;
  const BatchItem* scat;    // spread / adjoint-source bricks
  int nscat;
  const BatchItem* gath;    // gather bricks
  int ngath;
  const BatchItem* agath;   // reverse-pass gather bricks
  int nagath;
  long long* g64;           // int64 accumulation grid (all systems)
  long long gtot;
  float2* rhok;             // half spectra
  const float* gtab;        // Green's tables (half-spectrum layout)
  float* phi;               // potential
  float* psi;               // reverse-pass potential of the adjoint source
  const int* xrow_first;    // [nsys + 1] prefix of the systems' x rows (My Mz)
  const int* ycol_first;    // [nsys + 1] prefix of their y columns (Mz (Mx/2+1))
  const int* zcol_first;    // [nsys + 1] prefix of their z columns (My (Mx/2+1))
  double* epart;            // [zcol_first[nsys]] k-space energy of each z column
  double* energy;           // [nsys]
  double ccelec;
  double *fx, *fy, *fz;     // forces [ntot]
  const double* dLdE;       // reverse pass inputs
  const double *gfx, *gfy, *gfz;
  float4* gs;               // [ntot] the sorted atoms' cotangents (scratch)
  double *dq, *dx, *dy, *dz;  // reverse pass outputs
  int* qctr;                // [4] work-item counters: spread, gather, adjoint source,
                            // reverse-pass gather (each kernel zeroes its own first)
};

bool batch_fused_supported(const BatchSys* sys, int nsys);
// Largest cooperative grid of the fused kernels on this device (0: cannot run).
int batch_fused_ctas(int gather_lanes);
int batch_fused_rev_ctas();
cudaError_t launch_batch_forward_fused(const BatchFused& a, int ctas, int gather_lanes,
                                       cudaStream_t st);
cudaError_t launch_batch_reverse_fused(const BatchFused& a, int ctas, cudaStream_t st);

cudaError_t launch_batch_bin(const float4* xyzq, int ntot, const BatchSys* sys, const int* first,
                             int nsys, int nbins, BinScratch w, float4* sorted, int* perm,
                             cudaStream_t st);
cudaError_t launch_batch_spread(const float4* sorted, const int* start, const BatchSys* sys,
                                const BatchItem* items, const BatchSeg* segs, int nseg, int ctas,
                                long long* grid64, long long gsize, float* rho, cudaStream_t st);
cudaError_t launch_batch_green(float2* rhok, const float* tab, long long ktot, const BatchSys* sys,
                               const long long* kfirst, const int* ksys, int nsys, double* energy,
                               cudaStream_t st);
cudaError_t launch_batch_gather(const float4* sorted, const int* perm, const int* start,
                                const BatchSys* sys, const BatchItem* items, const BatchSeg* segs,
                                int nseg, int ctas, const float* phi, double outscale, double* fx,
                                double* fy, double* fz, cudaStream_t st);

// float grid = int64 accumulation grid at 2^40 (the scatter kernels' output)
cudaError_t launch_grid64_to_real(const long long* grid64, long long size, float* out,
                                  cudaStream_t st);

// Mixed-form spread: brick tiles added into the int64 grid `grid64` at 2^40,
// then converted into the float grid `rho` (NULL: left to the caller).  The
// grid is cleared here unless `zeroed`: the caller cleared it before the
// binning, and the spread then launches as the dependent of the binning's
// last kernel, which directly precedes it on `st`.
cudaError_t launch_spread_scatter(const float4* sorted, const int* start, const BinLayout& b,
                                  const Stencil<float>& s, long long* grid64, float* rho,
                                  bool zeroed, cudaStream_t st);

template <typename CT>
cudaError_t launch_bin_sorted(const typename Vec4<CT>::type* xyzq, int n, const BinLayout& b,
                              CT inv_hx, CT inv_hy, CT inv_hz, BinScratch w,
                              typename Vec4<CT>::type* sorted, int* perm, cudaStream_t st);

template <typename CT>
cudaError_t launch_bin_scan_place(const typename Vec4<CT>::type* xyzq, int n, int nb,
                                  BinScratch w, typename Vec4<CT>::type* sorted, int* perm,
                                  cudaStream_t st, const BinLayout& b = BinLayout{},
                                  const CT* inv_h = nullptr);

template <typename CT>
bool spread_tiled_supported(const Stencil<CT>& s);

// FP64 form: the whole density grid from the sorted atoms (gse_spread64.cu).
// `basis` [n][kBasis64]: written by the binning (BinScratch::basis).
cudaError_t launch_spread64(const double* basis, const int* start, const BinLayout& b,
                            const Stencil<double>& s, double* grid, cudaStream_t st);

// pdl: the launch follows a kernel of this library directly on `st` and may
// overlap its end (programmatic dependent launch).
template <typename CT>
cudaError_t launch_gather_tiled(const typename Vec4<CT>::type* sorted, const int* perm,
                                const int* start, const BinLayout& b, const Stencil<CT>& s,
                                const CT* phi, double outscale, double* fx, double* fy,
                                double* fz, bool pdl, cudaStream_t st);

}  // namespace gse
