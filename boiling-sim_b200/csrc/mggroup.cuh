// mggroup.cuh -- interface of the one-launch solve of small grids (mggroup.cu).
#pragma once
#include <cstddef>
#include <cstdint>

#include <cuda_runtime.h>

namespace bsp {
namespace grp {

constexpr int MAXL = 12;            // levels (solver.cuh: MAX_LEVELS)
constexpr int COARSEST = 256;       // cells of the coarsest level
constexpr int PSTRIDE = 8192;       // doubles per slot of sums (>= virtual warps)
constexpr int GROUP_MAX = 24;       // instances per launch
enum { SLOT_RR = 0, SLOT_RZ = 1, SLOT_PAP = 2, SLOT_MAX = 3 };

template <class T>
struct LevelP {
  int nx, ny, nz;
  const uint8_t *mask;
  T *r, *e;
};

// One instance: its workspace (offsets of solver.cu's layout) and arguments.
struct Inst {
  char *base;
  const uint8_t *mask;
  const float *div;
  float *p;
  const float *cinv;
  const int *cflag;
  double bscale;
  int nx, ny, nz, L;
  int cta0, ncta;  // first CTA of the group, CTAs
  size_t off_ctl, off_partials, off_result, off_x, off_e, off_z, off_r, off_r2, off_ps0, off_ps1,
      off_Ap;
  size_t off_lv[MAXL], off_lr[MAXL], off_le[MAXL];  // coarse masks, r, e
};

struct Params {
  int count, max_outer, max_inner, warm;
  float alpha;
  double tol, eta;
  Inst in[GROUP_MAX];
};

// Written at off_result by the group's first CTA.
struct Result {
  int status, outer_it, total_inner, pad;
  double rel;
};

}  // namespace grp

template <class T>
cudaError_t launch_group_solve(grp::Params &P, cudaStream_t s);

}  // namespace bsp
