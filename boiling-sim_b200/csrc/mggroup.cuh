// mggroup.cuh -- interface of the one-launch solve of small grids (mggroup.cu).
#pragma once
#include <cstddef>
#include <cstdint>

#include <cuda_runtime.h>

namespace bsp {
namespace grp {

constexpr int MAXL = 12;            // levels (solver.cuh: MAX_LEVELS)
constexpr int COARSEST = 256;       // cells of the coarsest level
constexpr int PSTRIDE = 256;       // doubles per slot of sums (>= virtual blocks)
constexpr int GROUP_MAX = 24;       // instances per launch
enum { SLOT_RR = 0, SLOT_RZ = 1, SLOT_PAP = 2, SLOT_MAX = 3 };

template <class T>
struct LevelP {
  int nx, ny, nz;
  const uint8_t *mask, *code;
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
  const uint32_t *units;  // level-0 units with fluid: their number, then their list
  double bscale;
  int nx, ny, nz, L;
  // which of the per-kernel path's orders of operations: level 0 on whole quads, its FP64
  // residual too, the coarse levels as the one-launch cycle
  bool paired0, quads, paired;
  int cta0, ncta;  // first CTA of the group, CTAs
  size_t off_ctl, off_partials, off_result, off_x, off_e, off_z, off_r, off_r2, off_ps0, off_ps1,
      off_Ap;
  size_t off_lv[MAXL], off_lr[MAXL], off_le[MAXL];  // coarse masks, r, e
  size_t off_code[MAXL];                            // code bytes
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

// Code bytes of a level (mggroup.cu) from its mask.
void launch_group_codes(uint8_t *code, const uint8_t *mask, int nx, int ny, int nz, cudaStream_t s);
// Work units of level 0, and the list of those with fluid (flag: scratch, one byte a unit).
size_t group_units(int nx, int ny, int nz);
void launch_group_units(uint32_t *list, uint8_t *flag, const uint8_t *mask, int nx, int ny, int nz,
                        cudaStream_t s);
// On at most `ctas` CTAs (at least one an instance).
template <class T>
cudaError_t launch_group_solve(grp::Params &P, int ctas, cudaStream_t s);

}  // namespace bsp
