// pcgr.cuh -- interface of the on-chip Jacobi-PCG (pcgr.cu).
#pragma once
#include <cstdint>

#include "grid_sync.cuh"

namespace bsp {

// First slot of the partial sums of each reduction of a solve, in both PCG kernels.  They
// follow each other with one grid barrier in between, after which every CTA reads what
// it published and may publish the next at once: a reduction has to keep off the
// slots of the one before, which a slow CTA may still be reading.
constexpr int PCG_SUM_INIT = 1;  // b.b, r.z
constexpr int PCG_SUM_A = 0;     // ps.Ap
constexpr int PCG_SUM_B = 1;     // r.z, r.r
constexpr int PCG_SUMS = 3;      // slots in all
static_assert(PCG_SUM_A < PCG_SUM_INIT && PCG_SUM_A < PCG_SUM_B, "INIT, A, B, A, B, ...");
static_assert(PCG_SUM_INIT + 2 <= PCG_SUMS && PCG_SUM_B + 2 <= PCG_SUMS, "slots");

constexpr int PR_AGAIN = -1;  // status: some block has more fluid than slots, nothing solved

struct PcgrArgs {
  float *p;
  const float *div;
  const int32_t *mat;
  float *z;          // exchange of the blocks' sides, by cell
  double *partials;  // PCG_SUMS * CTAs doubles
  GridCtl *ctl;
  float *outs[7];    // optional device floats: alpha beta rzold rznew bsq rsq pAp
  int nx, ny, nz, mf, ma, max_iter;
  int nbx, nby;      // blocks along i, j
  int cap;           // slots of a CTA
  int pad;           // floats of the largest padded block
  int cols;          // columns of the largest block
  float scale;       // -(rho dx dx)/dt as float
  double tol2;       // tol^2
};

struct PcgrPlan {
  int nbx, nby, cols, pad, cap, halo;
  size_t bytes;  // dynamic shared memory
};
bool pcg_resident_fits(int nx, int ny, int nz, int ctas, PcgrPlan &plan);
cudaError_t launch_pcg_resident(PcgrArgs &a, const PcgrPlan &plan, cudaStream_t s);

}  // namespace bsp
