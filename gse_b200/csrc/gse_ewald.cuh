// gse_ewald.cuh -- FP64 Ewald reciprocal sum on the GPU (gse_ewald.cu).
#pragma once

#include <cuda_runtime.h>

#include <vector>

namespace gse {

struct EwGeom {
  double inv_box[3];
  double pref;          // 2 pi / V * ccelec
  double half_sigmasq;  // sigma^2 / 2
};

// One row of the half space: ky, kz, and kx = kx0 .. kxm (kx0 = -kxm, or 1 on the
// kx axis).
struct EwRow {
  int ky, kz, kx0, kxm;
};

// A run of rows whose sums are in the scratch at one time.
struct EwBlock {
  int row0, nrows;
  int ncols;   // columns of S: c, s of every kx, whole 8-column strips
  int wpitch;  // the same for the force kernel, whole chunks
  int per_split, nsplit;    // atoms per split of the structure sum
  int per_fsplit, nfsplit;  // rows per split of the force sum
};

// Sizes and scratch layout of one call (one allocation of `bytes`).
struct EwPlan {
  int kmax, nrows;
  int slab, pitch;  // atoms per pass, and rounded up to 64
  std::vector<EwBlock> blocks;
  size_t off_rows, off_energy, off_T, off_part, off_W, off_f, bytes;
};

// Rows of the half sphere |k| <= kcut, longest first.
std::vector<EwRow> ewald_rows(int kcut);
// `budget`: bytes of scratch to plan for, half of it for the phase tables (more atoms
// go in slabs) and half for the rows' sums (more rows go in blocks); at least 64 atoms
// and 32 rows at a time.  The rows themselves, 24 bytes each, and the forces' partial
// sums, a few MB, come on top.
constexpr size_t kEwBudget = 512ull << 20;
EwPlan ewald_plan(int n, const std::vector<EwRow>& rows, int kcut, bool forces, size_t budget);
// `buf`: p.bytes of device memory; the rows' energies are left at p.off_energy.
cudaError_t launch_ewald(const double4* xyzq, int n, const std::vector<EwRow>& rows,
                         const EwGeom& g, const EwPlan& p, char* buf, double* fx, double* fy,
                         double* fz, cudaStream_t st);

// ---- direct (real-space) sum, gse_ewald_direct.cu ----

constexpr int kEwdMaxCellsPerAxis = 128;

struct EwdGeom {
  double box[3], hbox[3], inv_box[3];
  int nc[3];  // cells per axis, each of side box / nc >= rcut
  int ncell;
  double rcut2, inv_sqrt2sigma, inv_2sigmasq, two_sqrtpi;
  double self;  // -ccelec / sqrt(2 pi sigma^2)
  double ccelec;
};

struct EwdScratch {
  int* key;         // [n] cell of each atom
  int* counts;      // [ncell]
  int* start;       // [ncell + 1]
  int* tile_sums;   // [ceil(ncell / 4096)]
  int* lstart;      // [ncell]
  int* tmp;         // [n]
  double4* sorted;  // [n] atoms in cell order
  int* perm;        // [n] original index of each sorted atom
  int* cells;       // [min(n, ncell)] cells that hold atoms
  double* partials; // [n] energies of the blocks
  unsigned* done;   // [2] counters of finished blocks and of such cells
};

EwdGeom ewald_direct_geom(double sigma, double rcut, const double box[3], double ccelec);
// ex_start[n + 1] / ex_idx: the excluded partners of every atom (both
// directions), or both NULL.  energy_out: one device double.  n > 0.
cudaError_t launch_ewald_direct(const double4* xyzq, int n, const EwdGeom& g, EwdScratch w,
                                const int* ex_start, const int* ex_idx, double* fx, double* fy,
                                double* fz, double* energy_out, cudaStream_t st);

}  // namespace gse
