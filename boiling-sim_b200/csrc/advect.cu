// advect.cu -- semi-Lagrangian advection of the MAC face velocities and the
// cell-centred temperature.
//
// Reference semantics:
//   _tri_sample, _sample_velocity_at     python/boilingsim/fluid.py:39-104
//   extend_temperature_into_solids       python/boilingsim/fluid.py:338-382
//   advect_temperature                   python/boilingsim/fluid.py:385-411
//   advect_ux / advect_uy / advect_uz    python/boilingsim/fluid.py:414-498
//   advect_all                           python/boilingsim/fluid.py:737-776
//
// Every operation is the reference expression as written, one IEEE single
// rounding each (__fadd_rn / __fmul_rn / __fdiv_rn, no contraction):
//   p      = origin + (idx + offset) * dx           per axis
//   p_back = p - u * dt                             u from three trilinear samples at p
//   f      = (p - origin) / dx - offset, clamped to [0, n - 1 - 1e-6] (float)
//   value  = ((c000 (1-tx) + c100 tx) (1-ty) + (c010 (1-tx) + c110 tx) ty) (1-tz) + ...
// (p - origin) / dx depends on the lattice index only and is computed once per
// CTA for its plane, rows and columns.  The clamp's upper bound rounds to
// n - 1 exactly for n above ~17; the +1 corner is then clamped to n - 1 (the
// reference would read one element past the array there).
//
// One thread per cell and plane, CTAs of 32 k x 8 j marching over consecutive i planes:
// the eight corners of each sample are read through the read-only cache, and a plane's
// samples reuse most of the lines fetched for the plane before.  A step of all four
// fields is one such march (advect_all_kernel).  The loads' latency and the
// instructions bound it, and warps in flight hide the former: forms that keep the
// corners of the plane before in registers, fetch planes ahead into L2 or take 64 registers
// were 3 to 18 % slower.  Measured, a kernel per field -> here, with the fields brought back:
// 384x384x256 1.94 -> 1.47 ms a step, 256x256x160 657 -> 502 us, 128x128x96 158 -> 92 us,
// 56x56x40 80 -> 24 us.
#include <cuda_runtime.h>

#include "../../include/bsproj.h"
#include "bsp_common.cuh"

namespace bsp {
namespace sl {

struct Geo {
  int nx, ny, nz;
  int planes;  // of a CTA, at most PL
  float ox, oy, oz, dx, dt, rdx, least;  // rdx, least: for div_by
};

constexpr int BK = 32, BJ = 8, PL = 8;  // CTA: 32 k x 8 j, marching up to 8 planes

// Planes a CTA marches.  Large grids: 8, whose samples reuse the lines of the plane before
// (384x384x256: 1464 us a step with 8 or more, 1483 us with 4); below 16 M cells
// the CTAs in flight count for more (256x256x160: 499 us with 2, 533 us with 1; 128x128x96:
// 94 us with 1, 139 us with 16; 56x56x40, when four copies brought the fields back: 34 us with 1,
// 36 us with 2).
inline int planes_of(int nx, int ny, int nz) {
  const int64_t n = (int64_t)nx * ny * nz;
  return n < (2 << 20) ? 1 : n < (16 << 20) ? 2 : PL;
}

// Trilinear sample of field f (shape fxn x fyn x fzn, lattice offset (sx, sy,
// sz)) at the point whose scaled coordinates (p - origin) / dx are (gx, gy, gz).
// Offsets are 32-bit (fields hold fewer than 2^31 elements).
__device__ __forceinline__ float tri(const float *__restrict__ f, int fxn, int fyn, int fzn,
                                     float gx, float gy, float gz, float sx, float sy, float sz) {
  float fx = __fsub_rn(gx, sx), fy = __fsub_rn(gy, sy), fz = __fsub_rn(gz, sz);
  fx = fminf(fmaxf(fx, 0.0f), __fsub_rn((float)(fxn - 1), 1.0e-6f));
  fy = fminf(fmaxf(fy, 0.0f), __fsub_rn((float)(fyn - 1), 1.0e-6f));
  fz = fminf(fmaxf(fz, 0.0f), __fsub_rn((float)(fzn - 1), 1.0e-6f));
  const int i0 = __float2int_rz(fx), j0 = __float2int_rz(fy), k0 = __float2int_rz(fz);
  const float tx = __fsub_rn(fx, (float)i0), ty = __fsub_rn(fy, (float)j0),
              tz = __fsub_rn(fz, (float)k0);
  const int pl = fyn * fzn;
  const int di = i0 + 1 < fxn ? pl : 0, dj = j0 + 1 < fyn ? fzn : 0, dk = k0 + 1 < fzn ? 1 : 0;
  const float *q = f + (i0 * pl + j0 * fzn + k0);
  const float c000 = __ldg(q), c001 = __ldg(q + dk);
  const float c010 = __ldg(q + dj), c011 = __ldg(q + dj + dk);
  const float c100 = __ldg(q + di), c101 = __ldg(q + di + dk);
  const float c110 = __ldg(q + di + dj), c111 = __ldg(q + di + dj + dk);
  const float ux = __fsub_rn(1.0f, tx), uy = __fsub_rn(1.0f, ty), uz = __fsub_rn(1.0f, tz);
  const float c00 = __fadd_rn(__fmul_rn(c000, ux), __fmul_rn(c100, tx));
  const float c10 = __fadd_rn(__fmul_rn(c010, ux), __fmul_rn(c110, tx));
  const float c01 = __fadd_rn(__fmul_rn(c001, ux), __fmul_rn(c101, tx));
  const float c11 = __fadd_rn(__fmul_rn(c011, ux), __fmul_rn(c111, tx));
  const float c0 = __fadd_rn(__fmul_rn(c00, uy), __fmul_rn(c10, ty));
  const float c1 = __fadd_rn(__fmul_rn(c01, uy), __fmul_rn(c11, ty));
  return __fadd_rn(__fmul_rn(c0, uz), __fmul_rn(c1, tz));
}

// One axis of a sample: the lower corner, the step to the upper one (0 at the array's
// end) and the weights; the same operations as tri's.
struct __align__(16) Axis {
  int lo, d;
  float t, u;
};
__device__ __forceinline__ Axis axis_of(float g, float s, int n) {
  const float f =
      fminf(fmaxf(__fsub_rn(g, s), 0.0f), __fsub_rn((float)(n - 1), 1.0e-6f));
  Axis a;
  a.lo = __float2int_rz(f);
  a.t = __fsub_rn(f, (float)a.lo);
  a.u = __fsub_rn(1.0f, a.t);
  a.d = a.lo + 1 < n ? 1 : 0;
  return a;
}

// What depends on a lattice index alone, computed once per CTA for its planes, rows
// and columns, for the lattices of offset 0 and 0.5: the world coordinate p = origin +
// (idx + s) dx, and from (p - origin) / dx the axes of samples of fields of offset 0
// and 0.5 there.
struct Coords {
  float px[2][PL], py[2][BJ], pz[2][BK];
  Axis x[2][2][PL], y[2][2][BJ], z[2][2][BK];  // [lattice][field]
};
__device__ __forceinline__ void coord(float &p, Axis &a0, Axis &a5, int idx, float s, float o,
                                      int n, const Geo &g) {
  p = __fadd_rn(o, __fmul_rn(__fadd_rn((float)idx, s), g.dx));
  const float q = __fdiv_rn(__fsub_rn(p, o), g.dx);
  a0 = axis_of(q, 0.0f, n + 1);
  a5 = axis_of(q, 0.5f, n);
}
__device__ __forceinline__ void coords(Coords &c, const Geo &g) {
  const int tx = threadIdx.x, ty = threadIdx.y, l = ty & 1;
  const float s = l ? 0.5f : 0.0f;
  if (ty < 2) {
    coord(c.pz[l][tx], c.z[l][0][tx], c.z[l][1][tx], blockIdx.x * BK + tx, s, g.oz, g.nz, g);
  } else if (ty < 4 && tx < BJ) {
    coord(c.py[l][tx], c.y[l][0][tx], c.y[l][1][tx], blockIdx.y * BJ + tx, s, g.oy, g.ny, g);
  } else if (ty >= 4 && ty < 6 && tx < PL) {
    const int q = tx;
    coord(c.px[l][q], c.x[l][0][q], c.x[l][1][q], blockIdx.z * g.planes + q, s, g.ox, g.nx, g);
  }
  __syncthreads();
}

// Trilinear sample at a lattice point, from its axes.
__device__ __forceinline__ float sample(const float *__restrict__ f, int fyn, int fzn,
                                        const Axis &x, const Axis &y, const Axis &z) {
  const int pl = fyn * fzn, di = x.d ? pl : 0, dj = y.d ? fzn : 0;
  const float *q = f + (x.lo * pl + y.lo * fzn + z.lo);
  const float c000 = __ldg(q), c001 = __ldg(q + z.d);
  const float c010 = __ldg(q + dj), c011 = __ldg(q + dj + z.d);
  const float c100 = __ldg(q + di), c101 = __ldg(q + di + z.d);
  const float c110 = __ldg(q + di + dj), c111 = __ldg(q + di + dj + z.d);
  const float c00 = __fadd_rn(__fmul_rn(c000, x.u), __fmul_rn(c100, x.t));
  const float c10 = __fadd_rn(__fmul_rn(c010, x.u), __fmul_rn(c110, x.t));
  const float c01 = __fadd_rn(__fmul_rn(c001, x.u), __fmul_rn(c101, x.t));
  const float c11 = __fadd_rn(__fmul_rn(c011, x.u), __fmul_rn(c111, x.t));
  const float c0 = __fadd_rn(__fmul_rn(c00, y.u), __fmul_rn(c10, y.t));
  const float c1 = __fadd_rn(__fmul_rn(c01, y.u), __fmul_rn(c11, y.t));
  return __fadd_rn(__fmul_rn(c0, z.u), __fmul_rn(c1, z.t));
}

// Field f (lattice AX: 0 ux, 1 uy, 2 uz, 3 cell centres) at the point backtraced from
// the thread's point of plane ii: the velocity there from three samples, then one
// at where it came from.
template <int AX>
__device__ __forceinline__ float advected(const float *__restrict__ f, const Coords &c, int ii,
                                          const float *__restrict__ ux,
                                          const float *__restrict__ uy,
                                          const float *__restrict__ uz, const Geo &g) {
  constexpr int LX = AX != 0, LY = AX != 1, LZ = AX != 2;
  const int ty = threadIdx.y, tx = threadIdx.x;
  const float u = sample(ux, g.ny, g.nz, c.x[LX][0][ii], c.y[LY][1][ty], c.z[LZ][1][tx]);
  const float v = sample(uy, g.ny + 1, g.nz, c.x[LX][1][ii], c.y[LY][0][ty], c.z[LZ][1][tx]);
  const float w = sample(uz, g.ny, g.nz + 1, c.x[LX][1][ii], c.y[LY][1][ty], c.z[LZ][0][tx]);
  const float qx = __fsub_rn(c.px[LX][ii], __fmul_rn(u, g.dt));
  const float qy = __fsub_rn(c.py[LY][ty], __fmul_rn(v, g.dt));
  const float qz = __fsub_rn(c.pz[LZ][tx], __fmul_rn(w, g.dt));
  const float bx = div_by(__fsub_rn(qx, g.ox), g.dx, g.rdx, g.least);
  const float by = div_by(__fsub_rn(qy, g.oy), g.dx, g.rdx, g.least);
  const float bz = div_by(__fsub_rn(qz, g.oz), g.dx, g.rdx, g.least);
  return tri(f, g.nx + !LX, g.ny + !LY, g.nz + !LZ, bx, by, bz, LX ? 0.5f : 0.0f,
             LY ? 0.5f : 0.0f, LZ ? 0.5f : 0.0f);
}

__device__ __forceinline__ bool fluid(const uint8_t *__restrict__ m, int64_t c) {
  return (__ldg(m + c) & BSP_MFLUID) != 0;
}

// A cell takes its temperature from itself if fluid, else from the first fluid neighbour
// in the order -x, +x, -y, +y, -z, +z (the six flags are loaded together), else itself.
// Single cells, in CTAs of 64 k x 4 j marching eight planes (200x200x130: 24 us; 32 us in the
// quads' shape).
constexpr int XK = 64, XJ = 4, XP = 8;
__global__ void __launch_bounds__(XK *XJ) extend_cells_kernel(float *__restrict__ T_ext,
                                                              const float *__restrict__ T,
                                                              const uint8_t *__restrict__ m, int nx,
                                                              int ny, int nz) {
  const int k = blockIdx.x * XK + threadIdx.x, j = blockIdx.y * XJ + threadIdx.y;
  if (k >= nz || j >= ny) return;
  const int64_t pl = (int64_t)ny * nz;
  for (int ii = 0; ii < XP; ++ii) {
    const int i = blockIdx.z * XP + ii;
    if (i >= nx) break;
    const int64_t c = i * pl + (int64_t)j * nz + k;
    int64_t s = c;
    if (!fluid(m, c)) {
      const bool f0 = i > 0 && fluid(m, c - pl), f1 = i < nx - 1 && fluid(m, c + pl);
      const bool f2 = j > 0 && fluid(m, c - nz), f3 = j < ny - 1 && fluid(m, c + nz);
      const bool f4 = k > 0 && fluid(m, c - 1), f5 = k < nz - 1 && fluid(m, c + 1);
      s = f0 ? c - pl : f1 ? c + pl : f2 ? c - nz : f3 ? c + nz : f4 ? c - 1 : f5 ? c + 1 : c;
    }
    T_ext[c] = __ldg(T + s);
  }
}

// Four cells a thread (rows of whole quads, aligned fields), copied as one where all are
// fluid.
__global__ void __launch_bounds__(BK *BJ) extend_quads_kernel(float *__restrict__ T_ext,
                                                              const float *__restrict__ T,
                                                              const uint8_t *__restrict__ m,
                                                              Geo g) {
  const int nz = g.nz, k = (blockIdx.x * BK + threadIdx.x) * 4;
  const int j = blockIdx.y * BJ + threadIdx.y;
  if (k >= nz || j >= g.ny) return;
  for (int ii = 0; ii < g.planes; ++ii) {
    const int i = blockIdx.z * g.planes + ii;
    if (i >= g.nx) break;
    const int64_t c = ((int64_t)i * g.ny + j) * nz + k;
    const uint32_t w = __ldg(reinterpret_cast<const uint32_t *>(m + c));
    float4 t = __ldg(reinterpret_cast<const float4 *>(T + c));
    constexpr uint32_t F = BSP_MFLUID;
    if ((w & F * 0x01010101u) != F * 0x01010101u) {
      const int64_t pl = (int64_t)g.ny * nz;
      auto word = [&](bool in, int64_t off) {
        return in ? __ldg(reinterpret_cast<const uint32_t *>(m + c + off)) : 0u;
      };
      const uint32_t w0 = word(i > 0, -pl), w1 = word(i < g.nx - 1, pl);
      const uint32_t w2 = word(j > 0, -nz), w3 = word(j < g.ny - 1, nz);
      const uint32_t km = k > 0 ? __ldg(m + c - 1) : 0u;
      const uint32_t kp = k + 4 < nz ? __ldg(m + c + 4) : 0u;
      const uint32_t w4 = w << 8 | km, w5 = w >> 8 | kp << 24;
      auto from = [&](int q, float own) {
        const uint32_t f = F << (8 * q);
        if (w & f) return own;
        const int64_t off = w0 & f   ? -pl
                            : w1 & f ? pl
                            : w2 & f ? -(int64_t)nz
                            : w3 & f ? nz
                            : w4 & f ? -1
                            : w5 & f ? 1
                                     : 0;
        return off ? __ldg(T + c + q + off) : own;
      };
      t = make_float4(from(0, t.x), from(1, t.y), from(2, t.z), from(3, t.w));
    }
    *reinterpret_cast<float4 *>(T_ext + c) = t;
  }
}

cudaError_t launch_extend(float *T_ext, const float *T, const uint8_t *m, const Geo &g,
                          cudaStream_t s) {
  const bool quad = g.nz % 4 == 0 && (((uintptr_t)T_ext | (uintptr_t)T) & 15u) == 0 &&
                    ((uintptr_t)m & 3u) == 0;
  if (quad)
    extend_quads_kernel<<<dim3((g.nz / 4 + BK - 1) / BK, (g.ny + BJ - 1) / BJ,
                               (g.nx + g.planes - 1) / g.planes),
                          dim3(BK, BJ), 0, s>>>(T_ext, T, m, g);
  else
    extend_cells_kernel<<<dim3((g.nz + XK - 1) / XK, (g.ny + XJ - 1) / XJ, (g.nx + XP - 1) / XP),
                          dim3(XK, XJ), 0, s>>>(T_ext, T, m, g.nx, g.ny, g.nz);
  return cudaGetLastError();
}

__global__ void __launch_bounds__(BK *BJ, 5) advect_T_kernel(
    float *__restrict__ T_new, const float *__restrict__ T_true, const float *__restrict__ T_ext,
    const float *__restrict__ ux, const float *__restrict__ uy, const float *__restrict__ uz,
    const uint8_t *__restrict__ m, Geo g) {
  __shared__ Coords cs;
  const int k = blockIdx.x * BK + threadIdx.x, j = blockIdx.y * BJ + threadIdx.y;
  coords(cs, g);
  if (k >= g.nz || j >= g.ny) return;
  for (int ii = 0; ii < g.planes; ++ii) {
    const int i = blockIdx.z * g.planes + ii;
    if (i >= g.nx) break;
    const int64_t c = ((int64_t)i * g.ny + j) * g.nz + k;
    T_new[c] = fluid(m, c) ? advected<3>(T_ext, cs, ii, ux, uy, uz, g) : __ldg(T_true + c);
  }
}

template <int AX>
__global__ void __launch_bounds__(BK *BJ, 5) advect_u_kernel(float *__restrict__ u_new,
                                                             const float *__restrict__ ux,
                                                             const float *__restrict__ uy,
                                                             const float *__restrict__ uz,
                                                             const uint8_t *__restrict__ m, Geo g) {
  __shared__ Coords cs;
  const int fxn = g.nx + (AX == 0), fyn = g.ny + (AX == 1), fzn = g.nz + (AX == 2);
  const int k = blockIdx.x * BK + threadIdx.x, j = blockIdx.y * BJ + threadIdx.y;
  coords(cs, g);
  if (k >= fzn || j >= fyn) return;
  const float *__restrict__ u = AX == 0 ? ux : (AX == 1 ? uy : uz);
  const int64_t pl = (int64_t)g.ny * g.nz;
  for (int ii = 0; ii < g.planes; ++ii) {
    const int i = blockIdx.z * g.planes + ii;
    if (i >= fxn) break;
    const int64_t f = ((int64_t)i * fyn + j) * fzn + k;
    const int a = AX == 0 ? i : (AX == 1 ? j : k);
    const int na = AX == 0 ? fxn : (AX == 1 ? fyn : fzn);
    if (a == 0 || a == na - 1) {
      u_new[f] = 0.0f;
      continue;
    }
    const int64_t c1 = i * pl + (int64_t)j * g.nz + k;
    const int64_t c0 = AX == 0 ? c1 - pl : (AX == 1 ? c1 - g.nz : c1 - 1);
    u_new[f] = fluid(m, c0) || fluid(m, c1) ? advected<AX>(u, cs, ii, ux, uy, uz, g)
                                            : __ldg(u + f);
  }
}

// ---- one field of a large grid ------------------------------------------------------
// From FIELD_CELLS cells: coordinates only from the tables, and the axes formed per thread, in
// CTAs of 64 k x 4 j marching eight planes.  One field's march reuses a line
// less often than four do, and shared axes then cost more than they save (single calls, axes per
// thread / shared, us: T at 384x384x256 362 / 421, 256x256x192 131 / 156, 192x192x128 55 / 65; uz at
// 256x256x192 142 / 165; below the line T at 150x150x100 34 / 32, 110x110x68 24 / 18).
constexpr int64_t FIELD_CELLS = 3 << 20;
namespace wide {

constexpr int BK = 64, BJ = 4, PL = 8;

// World and scaled coordinates of a CTA's lattice points, computed once per
// CTA: p = origin + (idx + s) dx and g = (p - origin) / dx per axis for its
// plane i, its BJ rows and its BK columns (they depend on the index only).
struct Coords {
  float px[PL], gx[PL], py[BJ], gy[BJ], pz[BK], gz[BK];
};

__device__ __forceinline__ void coords(Coords &c, float sx, float sy, float sz, const Geo &g) {
  const int tx = threadIdx.x, ty = threadIdx.y;
  if (ty == 0) {
    const int k = blockIdx.x * BK + tx;
    const float p = __fadd_rn(g.oz, __fmul_rn(__fadd_rn((float)k, sz), g.dx));
    c.pz[tx] = p;
    c.gz[tx] = __fdiv_rn(__fsub_rn(p, g.oz), g.dx);
  } else if (ty == 1 && tx < BJ) {
    const int j = blockIdx.y * BJ + tx;
    const float p = __fadd_rn(g.oy, __fmul_rn(__fadd_rn((float)j, sy), g.dx));
    c.py[tx] = p;
    c.gy[tx] = __fdiv_rn(__fsub_rn(p, g.oy), g.dx);
  } else if (ty == 2 && tx < PL) {
    const int i = blockIdx.z * PL + tx;
    const float p = __fadd_rn(g.ox, __fmul_rn(__fadd_rn((float)i, sx), g.dx));
    c.px[tx] = p;
    c.gx[tx] = __fdiv_rn(__fsub_rn(p, g.ox), g.dx);
  }
  __syncthreads();
}

// The velocity at the point (three samples at its scaled coordinates) and the
// backtraced point's scaled coordinates.
__device__ __forceinline__ void backtrace(float &bx, float &by, float &bz, const Coords &c,
                                          int ii, const float *__restrict__ ux,
                                          const float *__restrict__ uy,
                                          const float *__restrict__ uz, const Geo &g) {
  const float px = c.px[ii], gx = c.gx[ii];
  const float py = c.py[threadIdx.y], gy = c.gy[threadIdx.y];
  const float pz = c.pz[threadIdx.x], gz = c.gz[threadIdx.x];
  const float u = tri(ux, g.nx + 1, g.ny, g.nz, gx, gy, gz, 0.0f, 0.5f, 0.5f);
  const float v = tri(uy, g.nx, g.ny + 1, g.nz, gx, gy, gz, 0.5f, 0.0f, 0.5f);
  const float w = tri(uz, g.nx, g.ny, g.nz + 1, gx, gy, gz, 0.5f, 0.5f, 0.0f);
  const float qx = __fsub_rn(px, __fmul_rn(u, g.dt));
  const float qy = __fsub_rn(py, __fmul_rn(v, g.dt));
  const float qz = __fsub_rn(pz, __fmul_rn(w, g.dt));
  bx = __fdiv_rn(__fsub_rn(qx, g.ox), g.dx);
  by = __fdiv_rn(__fsub_rn(qy, g.oy), g.dx);
  bz = __fdiv_rn(__fsub_rn(qz, g.oz), g.dx);
}

__global__ void __launch_bounds__(BK *BJ) advect_T_kernel(
    float *__restrict__ T_new, const float *__restrict__ T_true, const float *__restrict__ T_ext,
    const float *__restrict__ ux, const float *__restrict__ uy, const float *__restrict__ uz,
    const uint8_t *__restrict__ m, Geo g) {
  __shared__ Coords cs;
  const int k = blockIdx.x * BK + threadIdx.x, j = blockIdx.y * BJ + threadIdx.y;
  coords(cs, 0.5f, 0.5f, 0.5f, g);
  if (k >= g.nz || j >= g.ny) return;
  for (int ii = 0; ii < PL; ++ii) {
    const int i = blockIdx.z * PL + ii;
    if (i >= g.nx) break;
    const int64_t c = ((int64_t)i * g.ny + j) * g.nz + k;
    if (!fluid(m, c)) {
      T_new[c] = __ldg(T_true + c);
      continue;
    }
    float bx, by, bz;
    backtrace(bx, by, bz, cs, ii, ux, uy, uz, g);
    T_new[c] = tri(T_ext, g.nx, g.ny, g.nz, bx, by, bz, 0.5f, 0.5f, 0.5f);
  }
}

template <int AX>
__global__ void __launch_bounds__(BK *BJ) advect_u_kernel(float *__restrict__ u_new,
                                                          const float *__restrict__ ux,
                                                          const float *__restrict__ uy,
                                                          const float *__restrict__ uz,
                                                          const uint8_t *__restrict__ m, Geo g) {
  __shared__ Coords cs;
  const int fxn = g.nx + (AX == 0), fyn = g.ny + (AX == 1), fzn = g.nz + (AX == 2);
  const int k = blockIdx.x * BK + threadIdx.x, j = blockIdx.y * BJ + threadIdx.y;
  const float sx = AX == 0 ? 0.0f : 0.5f, sy = AX == 1 ? 0.0f : 0.5f, sz = AX == 2 ? 0.0f : 0.5f;
  coords(cs, sx, sy, sz, g);
  if (k >= fzn || j >= fyn) return;
  const float *__restrict__ u = AX == 0 ? ux : (AX == 1 ? uy : uz);
  const int64_t pl = (int64_t)g.ny * g.nz;
  for (int ii = 0; ii < PL; ++ii) {
    const int i = blockIdx.z * PL + ii;
    if (i >= fxn) break;
    const int64_t f = ((int64_t)i * fyn + j) * fzn + k;
    const int a = AX == 0 ? i : (AX == 1 ? j : k);
    const int na = AX == 0 ? fxn : (AX == 1 ? fyn : fzn);
    if (a == 0 || a == na - 1) {
      u_new[f] = 0.0f;
      continue;
    }
    const int64_t c1 = i * pl + (int64_t)j * g.nz + k;
    const int64_t c0 = AX == 0 ? c1 - pl : (AX == 1 ? c1 - g.nz : c1 - 1);
    if (!fluid(m, c0) && !fluid(m, c1)) {
      u_new[f] = __ldg(u + f);
      continue;
    }
    float bx, by, bz;
    backtrace(bx, by, bz, cs, ii, ux, uy, uz, g);
    u_new[f] = tri(u, fxn, fyn, fzn, bx, by, bz, sx, sy, sz);
  }
}

// CTAs: 64 k x 4 j, PL planes each
inline dim3 grid_pl(int nx, int ny, int nz) {
  return dim3((unsigned)((nz + BK - 1) / BK), (unsigned)((ny + BJ - 1) / BJ),
              (unsigned)((nx + PL - 1) / PL));
}

}  // namespace wide

// All four fields in one march over the cells (the faces before them; the thread of
// the last cell also zeroes the face behind it): the twelve velocity samples and four
// backtraced ones of a cell read the same few lines, which four kernels
// fetch four times.
__global__ void __launch_bounds__(BK *BJ, 5) advect_all_kernel(
    float *__restrict__ ux_new, float *__restrict__ uy_new, float *__restrict__ uz_new,
    float *__restrict__ T_new, const float *__restrict__ ux, const float *__restrict__ uy,
    const float *__restrict__ uz, const float *__restrict__ T_true,
    const float *__restrict__ T_ext, const uint8_t *__restrict__ m, Geo g) {
  __shared__ Coords cs;
  const int k = blockIdx.x * BK + threadIdx.x, j = blockIdx.y * BJ + threadIdx.y;
  coords(cs, g);
  if (k >= g.nz || j >= g.ny) return;
  const int pl = g.ny * g.nz;
  int c = (int)(blockIdx.z * g.planes) * pl + j * g.nz + k;
  bool before = blockIdx.z > 0 && fluid(m, c - pl);
  for (int ii = 0; ii < g.planes; ++ii, c += pl) {
    const int i = blockIdx.z * g.planes + ii;
    if (i >= g.nx) break;
    const bool fl = fluid(m, c);
    {
      float v = 0.0f;
      if (i > 0) v = before || fl ? advected<0>(ux, cs, ii, ux, uy, uz, g) : __ldg(ux + c);
      ux_new[c] = v;
      if (i + 1 == g.nx) ux_new[c + pl] = 0.0f;
    }
    {
      const int f = c + i * g.nz;  // face (i, j, k) of an array of ny + 1 rows
      float v = 0.0f;
      if (j > 0)
        v = fl || fluid(m, c - g.nz) ? advected<1>(uy, cs, ii, ux, uy, uz, g) : __ldg(uy + f);
      uy_new[f] = v;
      if (j + 1 == g.ny) uy_new[f + g.nz] = 0.0f;
    }
    {
      const int f = c + i * g.ny + j;  // face (i, j, k) of an array of nz + 1 columns
      float v = 0.0f;
      if (k > 0) v = fl || fluid(m, c - 1) ? advected<2>(uz, cs, ii, ux, uy, uz, g) : __ldg(uz + f);
      uz_new[f] = v;
      if (k + 1 == g.nz) uz_new[f + 1] = 0.0f;
    }
    T_new[c] = fl ? advected<3>(T_ext, cs, ii, ux, uy, uz, g) : __ldg(T_true + c);
    before = fl;
  }
}

// The advected fields back into place where advect_all_kernel has changed them (a
// pot's air and walls are two fifths of its cells): one launch for small grids, where four
// copies take longer (56x56x40: 29 us a step, 36 us with the copies, both before the extension
// went by quads; 1.5 mm scene: 114 and 121 us); on large ones the copies' streams are the faster (200x193x130: 285 us
// both; 256x256x160: 527 and 499 us).
constexpr int64_t COPY_KERNEL_CELLS = 5 << 20;
__global__ void __launch_bounds__(BK *BJ) copy_back_kernel(
    float *__restrict__ ux, float *__restrict__ uy, float *__restrict__ uz, float *__restrict__ T,
    const float *__restrict__ ux_new, const float *__restrict__ uy_new,
    const float *__restrict__ uz_new, const float *__restrict__ T_new,
    const uint8_t *__restrict__ m, Geo g) {
  const int k = blockIdx.x * BK + threadIdx.x, j = blockIdx.y * BJ + threadIdx.y;
  if (k >= g.nz || j >= g.ny) return;
  const int pl = g.ny * g.nz;
  int c = (int)(blockIdx.z * g.planes) * pl + j * g.nz + k;
  bool before = blockIdx.z > 0 && fluid(m, c - pl);
  for (int ii = 0; ii < g.planes; ++ii, c += pl) {
    const int i = blockIdx.z * g.planes + ii, fy = c + i * g.nz, fz = c + i * g.ny + j;
    if (i >= g.nx) break;
    const bool fl = fluid(m, c);
    if (i == 0 || before || fl) ux[c] = __ldg(ux_new + c);
    if (i + 1 == g.nx) ux[c + pl] = 0.0f;
    if (j == 0 || fl || fluid(m, c - g.nz)) uy[fy] = __ldg(uy_new + fy);
    if (j + 1 == g.ny) uy[fy + g.nz] = 0.0f;
    if (k == 0 || fl || fluid(m, c - 1)) uz[fz] = __ldg(uz_new + fz);
    if (k + 1 == g.nz) uz[fz + 1] = 0.0f;
    if (fl) T[c] = __ldg(T_new + c);
    before = fl;
  }
}

// CTAs of the kernels: BK k x BJ j, g.planes planes each
inline dim3 grid_pl(int nx, int ny, int nz, int planes) {
  return dim3((unsigned)((nz + BK - 1) / BK), (unsigned)((ny + BJ - 1) / BJ),
              (unsigned)((nx + planes - 1) / planes));
}

cudaError_t launch_velocity(int axis, float *u_new, const float *ux, const float *uy,
                            const float *uz, const uint8_t *m, const Geo &g, cudaStream_t s) {
  if ((int64_t)g.nx * g.ny * g.nz >= FIELD_CELLS) {
    auto fn = axis == 0   ? wide::advect_u_kernel<0>
              : axis == 1 ? wide::advect_u_kernel<1>
                          : wide::advect_u_kernel<2>;
    fn<<<wide::grid_pl(g.nx + (axis == 0), g.ny + (axis == 1), g.nz + (axis == 2)),
         dim3(wide::BK, wide::BJ), 0, s>>>(u_new, ux, uy, uz, m, g);
    return cudaGetLastError();
  }
  const dim3 blk(BK, BJ);
  if (axis == 0)
    advect_u_kernel<0>
        <<<grid_pl(g.nx + 1, g.ny, g.nz, g.planes), blk, 0, s>>>(u_new, ux, uy, uz, m, g);
  else if (axis == 1)
    advect_u_kernel<1>
        <<<grid_pl(g.nx, g.ny + 1, g.nz, g.planes), blk, 0, s>>>(u_new, ux, uy, uz, m, g);
  else
    advect_u_kernel<2>
        <<<grid_pl(g.nx, g.ny, g.nz + 1, g.planes), blk, 0, s>>>(u_new, ux, uy, uz, m, g);
  return cudaGetLastError();
}

bool dims_ok(int nx, int ny, int nz) {
  // grid.z = nx + 1 planes and grid.y = ceil((ny + 1) / 4) rows (4: the fewest of a CTA) must
  // fit the launch limits; the samplers use 32-bit element offsets
  return nx + 1 <= 65535 && (ny + 1 + 3) / 4 <= 65535 &&
         (int64_t)(nx + 1) * (ny + 1) * (nz + 1) < (1LL << 31);
}

}  // namespace sl
}  // namespace bsp

using namespace bsp::sl;

extern "C" int bsp_extend_temperature(float *T_ext, const float *T, const uint8_t *mask, int nx,
                                      int ny, int nz, cudaStream_t s) {
  if (nx <= 0 || ny <= 0 || nz <= 0) return BSP_OK;
  if (!T_ext || !T || !mask) return BSP_ERR_NULL;
  if (T_ext == T) return BSP_ERR_ALIAS;
  if (!dims_ok(nx, ny, nz)) return BSP_ERR_SHAPE;
  const Geo g{nx, ny, nz, planes_of(nx, ny, nz), 0.0f, 0.0f, 0.0f, 1.0f, 0.0f, 1.0f, 1.0f};
  return (int)launch_extend(T_ext, T, mask, g, s);
}

extern "C" int bsp_advect_temperature(float *T_new, const float *T_true, const float *T_ext,
                                      const float *ux, const float *uy, const float *uz,
                                      const uint8_t *mask, int nx, int ny, int nz, float ox,
                                      float oy, float oz, float dx, float dt, cudaStream_t s) {
  if (nx <= 0 || ny <= 0 || nz <= 0) return BSP_OK;
  if (!T_new || !T_true || !T_ext || !ux || !uy || !uz || !mask) return BSP_ERR_NULL;
  if (T_new == T_true || T_new == T_ext) return BSP_ERR_ALIAS;
  if (!dims_ok(nx, ny, nz) || !(dx > 0.0f)) return BSP_ERR_SHAPE;
  const Geo g{nx, ny, nz, planes_of(nx, ny, nz), ox, oy, oz, dx, dt, bsp::rcp_of(dx),
              bsp::div_least(bsp::rcp_of(dx))};
  if ((int64_t)nx * ny * nz >= FIELD_CELLS)
    wide::advect_T_kernel<<<wide::grid_pl(nx, ny, nz), dim3(wide::BK, wide::BJ), 0, s>>>(
        T_new, T_true, T_ext, ux, uy, uz, mask, g);
  else
    advect_T_kernel<<<grid_pl(nx, ny, nz, g.planes), dim3(BK, BJ), 0, s>>>(T_new, T_true, T_ext,
                                                                           ux, uy, uz, mask, g);
  return (int)cudaGetLastError();
}

extern "C" int bsp_advect_velocity(int axis, float *u_new, const float *ux, const float *uy,
                                   const float *uz, const uint8_t *mask, int nx, int ny, int nz,
                                   float ox, float oy, float oz, float dx, float dt,
                                   cudaStream_t s) {
  if (nx <= 0 || ny <= 0 || nz <= 0) return BSP_OK;
  if (!u_new || !ux || !uy || !uz || !mask) return BSP_ERR_NULL;
  if (axis < 0 || axis > 2) return BSP_ERR_ARG;
  if (u_new == ux || u_new == uy || u_new == uz) return BSP_ERR_ALIAS;
  if (!dims_ok(nx, ny, nz) || !(dx > 0.0f)) return BSP_ERR_SHAPE;
  const Geo g{nx, ny, nz, planes_of(nx, ny, nz), ox, oy, oz, dx, dt, bsp::rcp_of(dx),
              bsp::div_least(bsp::rcp_of(dx))};
  return (int)launch_velocity(axis, u_new, ux, uy, uz, mask, g, s);
}

extern "C" int bsp_advect_all(float *ux, float *uy, float *uz, float *T, float *ux_tmp,
                              float *uy_tmp, float *uz_tmp, float *T_tmp, float *T_ext,
                              const uint8_t *mask, int nx, int ny, int nz, float ox, float oy,
                              float oz, float dx, float dt, int copy_back, cudaStream_t s) {
  if (nx <= 0 || ny <= 0 || nz <= 0) return BSP_OK;
  if (!ux || !uy || !uz || !T || !ux_tmp || !uy_tmp || !uz_tmp || !T_tmp || !T_ext || !mask)
    return BSP_ERR_NULL;
  const float *outs[] = {ux_tmp, uy_tmp, uz_tmp, T_tmp, T_ext};
  const float *ins[] = {ux, uy, uz, T};
  for (const float *o : outs)
    for (const float *in : ins)
      if (o == in) return BSP_ERR_ALIAS;
  // the five outputs are written by different kernels while T_ext is still
  // being sampled: no two may share a base, and none may be the mask
  for (int a = 0; a < 5; ++a) {
    if ((const void *)outs[a] == (const void *)mask) return BSP_ERR_ALIAS;
    for (int b = a + 1; b < 5; ++b)
      if (outs[a] == outs[b]) return BSP_ERR_ALIAS;
  }
  if (!dims_ok(nx, ny, nz) || !(dx > 0.0f)) return BSP_ERR_SHAPE;
  const Geo g{nx, ny, nz, planes_of(nx, ny, nz), ox, oy, oz, dx, dt, bsp::rcp_of(dx),
              bsp::div_least(bsp::rcp_of(dx))};
  cudaError_t e = cudaSuccess;
  e = launch_extend(T_ext, T, mask, g, s);
  if (e != cudaSuccess) return (int)e;
  advect_all_kernel<<<grid_pl(nx, ny, nz, g.planes), dim3(BK, BJ), 0, s>>>(
      ux_tmp, uy_tmp, uz_tmp, T_tmp, ux, uy, uz, T, T_ext, mask, g);
  e = cudaGetLastError();
  if (e != cudaSuccess || !copy_back) return (int)e;
  if ((int64_t)nx * ny * nz < COPY_KERNEL_CELLS) {
    copy_back_kernel<<<grid_pl(nx, ny, nz, g.planes), dim3(BK, BJ), 0, s>>>(
        ux, uy, uz, T, ux_tmp, uy_tmp, uz_tmp, T_tmp, mask, g);
    return (int)cudaGetLastError();
  }
  const size_t c = sizeof(float) * (size_t)nx * ny * nz;
  const size_t fx = sizeof(float) * (size_t)(nx + 1) * ny * nz;
  const size_t fy = sizeof(float) * (size_t)nx * (ny + 1) * nz;
  const size_t fz = sizeof(float) * (size_t)nx * ny * (nz + 1);
  e = cudaMemcpyAsync(ux, ux_tmp, fx, cudaMemcpyDeviceToDevice, s);
  if (e == cudaSuccess) e = cudaMemcpyAsync(uy, uy_tmp, fy, cudaMemcpyDeviceToDevice, s);
  if (e == cudaSuccess) e = cudaMemcpyAsync(uz, uz_tmp, fz, cudaMemcpyDeviceToDevice, s);
  if (e == cudaSuccess) e = cudaMemcpyAsync(T, T_tmp, c, cudaMemcpyDeviceToDevice, s);
  return (int)e;
}
