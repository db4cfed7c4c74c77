// pcgr.cuh -- interface of the on-chip Jacobi-PCG (pcgr.cu).
#pragma once
#include <cstdint>

#include "grid_sync.cuh"

namespace bsp {

constexpr int PR_AGAIN = -1;  // status: some block has more fluid than slots, nothing solved

struct PcgrArgs {
  float *p;
  const float *div;
  const int32_t *mat;
  float *z;          // exchange of the blocks' sides, by cell
  double *partials;  // 3 * CTAs doubles
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
