// mggroup.cu -- the to-tolerance solve (solver.cu) of small grids as one
// cooperative launch: FP64 refinement, conjugate gradient and V-cycle of one or
// many instances, each by a group of CTAs with a barrier of its own.
//
// On a grid of up to a few million cells an inner iteration's kernels take
// microseconds each, so its two dozen launches (and, in a batch, the WHILE nodes of
// a graph's branches, which hardly overlap) were the time: 83 us an iteration at
// 110x110x68, 2.7 ms an instance of a batch.  Here a group runs a phase and
// meets at a barrier on a counter in the instance's workspace (about 1.3 us over
// 148 CTAs, less over few); the SMs are shared out over the instances by their
// cells, so a batch's instances run side by side.
//
// The cycle, the smoother, the stopping tests and the storage are solver.cu's
// with one sweep a side on every level: the same expressions on the same stored
// values, sums in another order.  Every sum over cells is taken over a fixed
// number of virtual warps and then over those in a fixed order, so a result
// does not depend on how many CTAs its group has: single, batched, host-driven
// and device-driven solves agree bit for bit.
//
// Work unit of the level kernels: the 2 x 2 columns of one coarse column and 30
// k cells; a lane owns one k of the four columns (lanes 0 and 31 are the k halo),
// so 12 operand loads serve 4 cells' 7-point stencils, k neighbours come by
// shuffles, and a coarse cell's children are four sums and one shuffle.
#include <cuda_bf16.h>
#include <cuda_fp16.h>

#include <algorithm>
#include <cstring>
#include <vector>

#include "bsp_common.cuh"
#include "grid_sync.cuh"
#include "mggroup.cuh"
#include "profile.cuh"

namespace bsp {

int num_sms();

namespace grp {

constexpr int THREADS = 1024, WARPS = THREADS / 32;
constexpr int VW = 148 * WARPS;     // virtual warps of a sum
constexpr int KOUT = 30;            // k cells of a unit
constexpr float W = 6.0f / 7.0f;    // smoothing weight
constexpr int TAIL_CELLS = 2048;    // levels up to this size run in the group's first CTA
constexpr int SWEEPS = 64;          // coarsest level without an inverse

__device__ __forceinline__ float ld(const float *p, int64_t c) { return p[c]; }
__device__ __forceinline__ float ld(const __half *p, int64_t c) { return __half2float(p[c]); }
__device__ __forceinline__ float ld(const __nv_bfloat16 *p, int64_t c) {
  return __bfloat162float(p[c]);
}
__device__ __forceinline__ float rnd(float v, const float *) { return v; }
__device__ __forceinline__ float rnd(float v, const __half *) {
  return __half2float(__float2half_rn(v));
}
__device__ __forceinline__ float rnd(float v, const __nv_bfloat16 *) {
  return __bfloat162float(__float2bfloat16_rn(v));
}
__device__ __forceinline__ void stv(float *p, int64_t c, float v) { p[c] = v; }
__device__ __forceinline__ void stv(__half *p, int64_t c, float v) { p[c] = __float2half_rn(v); }
__device__ __forceinline__ void stv(__nv_bfloat16 *p, int64_t c, float v) {
  p[c] = __float2bfloat16_rn(v);
}

// What a CTA knows of its instance (shared memory).
template <class T>
struct Ctx {
  Inst in;
  int rank, size;                   // CTA in the group, CTAs of the group
  unsigned int epoch;               // barriers passed
  GridCtl *ctl;
  double *partials;                 // slot q: partials + q * PSTRIDE
  double red[32];
  double total;
  int ok;
  float wt[8];                      // W / (6 - n_solid), 0 where that vanishes
  float e0[COARSEST], e1[COARSEST], rr[COARSEST], part[THREADS];
};

// Group barrier: arrivals on a counter that only grows; bounded.
template <class T>
__device__ __forceinline__ bool barrier(Ctx<T> &g) {
  __syncthreads();
  if (threadIdx.x == 0) {
    const unsigned int target = ++g.epoch * (unsigned int)g.size;
    cuda::atomic_ref<unsigned int, cuda::thread_scope_device> cnt(g.ctl->bar_count);
    cuda::atomic_ref<int, cuda::thread_scope_device> err(g.ctl->err);
    asm volatile("fence.acq_rel.gpu;" ::: "memory");
    cnt.fetch_add(1u, cuda::memory_order_release);
    int ok = 1;
    unsigned int spins = 0;
    unsigned long long t0 = 0;
    while (cnt.load(cuda::memory_order_acquire) < target) {
      if ((++spins & 255u) == 0) {
        const unsigned long long now = gs_global_ns();
        if (t0 == 0) t0 = now;
        if (err.load(cuda::memory_order_relaxed) != 0) break;
        if (now - t0 > BAR_TIMEOUT_NS || spins > BAR_SPIN_LIMIT) {
          err.store(BSP_ERR_TIMEOUT, cuda::memory_order_relaxed);
          break;
        }
      }
    }
    asm volatile("fence.acq_rel.gpu;" ::: "memory");
    if (err.load(cuda::memory_order_relaxed) != 0) ok = 0;
    g.ok = ok;
  }
  __syncthreads();
  return g.ok != 0;
}

__device__ __forceinline__ double warp_sum(double v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}
__device__ __forceinline__ double warp_max(double v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v = fmax(v, __shfl_xor_sync(0xffffffffu, v, o));
  return v;
}
// Total over the n virtual warps of slot q (written before the last barrier),
// in a fixed order; every thread of the CTA gets it.
template <class T>
__device__ double total(Ctx<T> &g, int q, int n, bool is_max) {
  const double *p = g.partials + (size_t)q * PSTRIDE;
  double s = 0.0;
  for (int v = threadIdx.x; v < n; v += THREADS) {
    const double x = __ldcg(p + v);
    s = is_max ? fmax(s, x) : s + x;
  }
  s = is_max ? warp_max(s) : warp_sum(s);
  if ((threadIdx.x & 31) == 0) g.red[threadIdx.x >> 5] = s;
  __syncthreads();
  if (threadIdx.x < 32) {
    double t = g.red[threadIdx.x];
    t = is_max ? warp_max(t) : warp_sum(t);
    if (threadIdx.x == 0) g.total = t;
  }
  __syncthreads();
  return g.total;
}

// ---- 2 x 2 column blocks ------------------------------------------------------------
struct Dims {
  int nx, ny, nz, bj, ch;  // bj: blocks along j, ch: k chunks
  int units;
};
__device__ __forceinline__ Dims dims_of(int nx, int ny, int nz) {
  Dims d{nx, ny, nz, (ny + 1) / 2, (nz + KOUT - 1) / KOUT, 0};
  d.units = ((nx + 1) / 2) * d.bj * d.ch;
  return d;
}
// One lane's twelve positions of unit u: own columns (a, b) = (0,0), (0,1), (1,0),
// (1,1); outer ones L (i - 1) b = 0, 1; R (i + 2) b = 0, 1; D (j - 1) a = 0, 1;
// U (j + 2) a = 0, 1.
struct Block {
  int bi, bjx, i, j, k;
  bool out;          // the lane's k is one of the unit's outputs
  int64_t base;      // cell (i, j, k)
  uint32_t m[4], mo[8];
};
__device__ __forceinline__ void block_of(Block &b, const Dims &d, int u,
                                         const uint8_t *__restrict__ mask) {
  const int lane = threadIdx.x & 31;
  const int c = u % d.ch, r = u / d.ch;
  b.bjx = r % d.bj;
  b.bi = r / d.bj;
  b.i = b.bi * 2;
  b.j = b.bjx * 2;
  b.k = c * KOUT - 1 + lane;
  const bool kin = b.k >= 0 && b.k < d.nz;
  b.out = kin && lane >= 1 && lane <= KOUT;
  b.base = ((int64_t)b.i * d.ny + b.j) * d.nz + b.k;
  const int64_t pl = (int64_t)d.ny * d.nz;
  const bool i1 = b.i + 1 < d.nx, j1 = b.j + 1 < d.ny;
  const uint8_t *m = mask + b.base;
  b.m[0] = kin ? __ldg(m) : 0u;
  b.m[1] = kin && j1 ? __ldg(m + d.nz) : 0u;
  b.m[2] = kin && i1 ? __ldg(m + pl) : 0u;
  b.m[3] = kin && i1 && j1 ? __ldg(m + pl + d.nz) : 0u;
  const bool l = kin && b.i > 0, rr = kin && b.i + 2 < d.nx;
  const bool dn = kin && b.j > 0, up = kin && b.j + 2 < d.ny;
  b.mo[0] = l ? __ldg(m - pl) : 0u;
  b.mo[1] = l && j1 ? __ldg(m - pl + d.nz) : 0u;
  b.mo[2] = rr ? __ldg(m + 2 * pl) : 0u;
  b.mo[3] = rr && j1 ? __ldg(m + 2 * pl + d.nz) : 0u;
  b.mo[4] = dn ? __ldg(m - d.nz) : 0u;
  b.mo[5] = dn && i1 ? __ldg(m - d.nz + pl) : 0u;
  b.mo[6] = up ? __ldg(m + 2 * d.nz) : 0u;
  b.mo[7] = up && i1 ? __ldg(m + 2 * d.nz + pl) : 0u;
}
__device__ __forceinline__ int64_t own_off(const Dims &d, int q) {
  return (q & 2 ? (int64_t)d.ny * d.nz : 0) + (q & 1 ? d.nz : 0);
}
__device__ __forceinline__ int64_t outer_off(const Dims &d, int q) {
  const int64_t pl = (int64_t)d.ny * d.nz, nz = d.nz;
  switch (q) {
    case 0: return -pl;
    case 1: return -pl + nz;
    case 2: return 2 * pl;
    case 3: return 2 * pl + nz;
    case 4: return -nz;
    case 5: return -nz + pl;
    case 6: return 2 * nz;
    default: return 2 * nz + pl;
  }
}
// Neighbour value: fluid -> v, air -> 0, solid -> the cell's own (v is 0 there).
__device__ __forceinline__ float nb(uint32_t m, float v, float self) {
  return (m & BSP_MSOLID) ? self : v;
}
// Neighbour sums of the four own cells from the operand values (0 off fluid).
__device__ __forceinline__ void sums(const Block &b, const float (&c)[4], const float (&o)[8],
                                     float (&s)[4]) {
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    const float vb = __shfl_up_sync(0xffffffffu, c[q], 1);
    const float vf = __shfl_down_sync(0xffffffffu, c[q], 1);
    const uint32_t mb = __shfl_up_sync(0xffffffffu, b.m[q], 1);
    const uint32_t mf = __shfl_down_sync(0xffffffffu, b.m[q], 1);
    const int a = q >> 1, bb = q & 1;
    const float l = a ? nb(b.m[q - 2 < 0 ? 0 : q - 2], c[q - 2 < 0 ? 0 : q - 2], c[q])
                      : nb(b.mo[bb], o[bb], c[q]);
    const float r = a ? nb(b.mo[2 + bb], o[2 + bb], c[q])
                      : nb(b.m[q + 2 > 3 ? 3 : q + 2], c[q + 2 > 3 ? 3 : q + 2], c[q]);
    const float d = bb ? nb(b.m[q - 1 < 0 ? 0 : q - 1], c[q - 1 < 0 ? 0 : q - 1], c[q])
                       : nb(b.mo[4 + a], o[4 + a], c[q]);
    const float u = bb ? nb(b.mo[6 + a], o[6 + a], c[q])
                       : nb(b.m[q + 1 > 3 ? 3 : q + 1], c[q + 1 > 3 ? 3 : q + 1], c[q]);
    s[q] = l + r + d + u + nb(mb, vb, c[q]) + nb(mf, vf, c[q]);
  }
}
__device__ __forceinline__ bool any_fluid(const Block &b) {
  return ((b.m[0] | b.m[1] | b.m[2] | b.m[3]) & BSP_MFLUID) != 0;
}
// Value of virtual warp v's sum: one double per virtual warp of slot q.
template <class T>
__device__ __forceinline__ void put(Ctx<T> &g, int q, int v, double x) {
  x = warp_sum(x);
  if ((threadIdx.x & 31) == 0) __stcg(g.partials + (size_t)q * PSTRIDE + v, x);
}
template <class T>
__device__ __forceinline__ int vwarps(int units) {
  return units < VW ? units : VW;
}

// Restriction of the residual of e = w r on level f to level co's r.
// UPDATE (level 0): r = r_in - alpha Ap first (where a CG update is pending),
// stored to r_out, with e += alpha ps and the partial sum r.r.
template <class T, bool UPDATE>
__device__ void down(Ctx<T> &g, const LevelP<T> &f, const LevelP<T> &co, const T *r_in, T *r_out,
                     const T *Ap, const T *ps, float *e, float alpha, bool pending, int first,
                     int step) {
  const Dims d = dims_of(f.nx, f.ny, f.nz);
  const int nv = vwarps<T>(d.units);
  for (int v = first; v < nv; v += step) {
    double rr = 0.0;
    for (int u = v; u < d.units; u += VW) {
      Block b;
      block_of(b, d, u, f.mask);
      if (!__any_sync(0xffffffffu, any_fluid(b))) continue;
      auto res = [&](int64_t c) {
        const float r = ld(r_in, c);
        return UPDATE && pending ? rnd(fmaf(-alpha, ld(Ap, c), r), r_out) : r;
      };
      float r[4], c[4], o[8], s[4];
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const bool fl = (b.m[q] & BSP_MFLUID) != 0;
        r[q] = fl ? res(b.base + own_off(d, q)) : 0.0f;
        c[q] = r[q] * g.wt[b.m[q] & 7];
      }
#pragma unroll
      for (int q = 0; q < 8; ++q)
        o[q] = (b.mo[q] & BSP_MFLUID) ? res(b.base + outer_off(d, q)) * g.wt[b.mo[q] & 7] : 0.0f;
      sums(b, c, o, s);
      float acc = 0.0f;
#pragma unroll
      for (int q = 0; q < 4; ++q)
        if (b.m[q] & BSP_MFLUID) {
          if (b.out) acc += r[q] - (6.0f * c[q] - s[q]);
          if (UPDATE && b.out) {
            const int64_t x = b.base + own_off(d, q);
            stv(r_out, x, r[q]);
            if (pending) e[x] = fmaf(alpha, ld(ps, x), e[x]);
            rr += (double)r[q] * (double)r[q];
          }
        }
      // the coarse cell's other four children are the next lane's (k odd)
      const float next = __shfl_down_sync(0xffffffffu, acc, 1);
      if (b.out && !(b.k & 1)) {
        const int64_t C = ((int64_t)b.bi * co.ny + b.bjx) * co.nz + (b.k >> 1);
        if (__ldg(co.mask + C) & BSP_MFLUID) stv(co.r, C, 0.5f * (acc + next));
      }
    }
    if (UPDATE) put(g, SLOT_RR, v, rr);
  }
}

// Prolongation and post-smoothing: e^ = alpha e_coarse[parent] + w r,
// out = e^ + w (r - A e^).  FINE: partial sum r.out.
template <class T, bool FINE>
__device__ void up(Ctx<T> &g, const LevelP<T> &f, const LevelP<T> &co, const T *r, T *out,
                   float alpha, int first, int step) {
  const Dims d = dims_of(f.nx, f.ny, f.nz);
  const int nv = vwarps<T>(d.units);
  for (int v = first; v < nv; v += step) {
    double rz = 0.0;
    for (int u = v; u < d.units; u += VW) {
      Block b;
      block_of(b, d, u, f.mask);
      if (!__any_sync(0xffffffffu, any_fluid(b))) continue;
      // coarse corrections of the block and its four neighbours
      const int64_t P = ((int64_t)b.bi * co.ny + b.bjx) * co.nz + (b.k >> 1);
      const int64_t cp = (int64_t)co.ny * co.nz;
      const bool kin = b.k >= 0 && b.k < f.nz;
      const float p0 = kin ? ld(co.e, P) : 0.0f;
      const float pl = kin && b.bi > 0 ? ld(co.e, P - cp) : 0.0f;
      const float pr = kin && b.bi + 1 < co.nx ? ld(co.e, P + cp) : 0.0f;
      const float pd = kin && b.bjx > 0 ? ld(co.e, P - co.nz) : 0.0f;
      const float pu = kin && b.bjx + 1 < co.ny ? ld(co.e, P + co.nz) : 0.0f;
      float rc[4], c[4], o[8], s[4];
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const bool fl = (b.m[q] & BSP_MFLUID) != 0;
        rc[q] = fl ? ld(r, b.base + own_off(d, q)) : 0.0f;
        c[q] = fl ? fmaf(alpha, p0, rc[q] * g.wt[b.m[q] & 7]) : 0.0f;
      }
#pragma unroll
      for (int q = 0; q < 8; ++q) {
        const float pp = q < 2 ? pl : (q < 4 ? pr : (q < 6 ? pd : pu));
        o[q] = (b.mo[q] & BSP_MFLUID)
                   ? fmaf(alpha, pp, ld(r, b.base + outer_off(d, q)) * g.wt[b.mo[q] & 7])
                   : 0.0f;
      }
      sums(b, c, o, s);
#pragma unroll
      for (int q = 0; q < 4; ++q)
        if (b.out && (b.m[q] & BSP_MFLUID)) {
          const float x = fmaf(rc[q] - (6.0f * c[q] - s[q]), g.wt[b.m[q] & 7], c[q]);
          stv(out, b.base + own_off(d, q), x);
          if (FINE) rz += (double)rc[q] * (double)rnd(x, out);
        }
    }
    if (FINE) put(g, SLOT_RZ, v, rz);
  }
}

// ps = z + beta ps_prev (z on a pass's first iteration), Ap = A ps, partial ps.Ap.
template <class T>
__device__ void direction(Ctx<T> &g, const LevelP<T> &f, const T *z, const T *prev, T *cur, T *Ap,
                          float beta, bool first_it, int first, int step) {
  const Dims d = dims_of(f.nx, f.ny, f.nz);
  const int nv = vwarps<T>(d.units);
  for (int v = first; v < nv; v += step) {
    double pap = 0.0;
    for (int u = v; u < d.units; u += VW) {
      Block b;
      block_of(b, d, u, f.mask);
      if (!__any_sync(0xffffffffu, any_fluid(b))) continue;
      auto ps = [&](int64_t c) {
        const float x = ld(z, c);
        return first_it ? x : rnd(fmaf(beta, ld(prev, c), x), cur);
      };
      float c[4], o[8], s[4];
#pragma unroll
      for (int q = 0; q < 4; ++q)
        c[q] = (b.m[q] & BSP_MFLUID) ? ps(b.base + own_off(d, q)) : 0.0f;
#pragma unroll
      for (int q = 0; q < 8; ++q)
        o[q] = (b.mo[q] & BSP_MFLUID) ? ps(b.base + outer_off(d, q)) : 0.0f;
      sums(b, c, o, s);
#pragma unroll
      for (int q = 0; q < 4; ++q)
        if (b.out && (b.m[q] & BSP_MFLUID)) {
          const int64_t x = b.base + own_off(d, q);
          const float ap = rnd(6.0f * c[q] - s[q], Ap);
          stv(cur, x, c[q]);
          stv(Ap, x, ap);
          pap += (double)c[q] * (double)ap;
        }
    }
    put(g, SLOT_PAP, v, pap);
  }
}

// FP64 residual b - A x on level 0.  WRITE: rhat = scale r (stored as T), e = 0;
// else the partial sum of squares and the largest |r|.  ZERO: x is zero.
template <class T, bool WRITE>
__device__ void residual(Ctx<T> &g, const LevelP<T> &f, const double *x, T *rhat, float *e,
                         double scale, bool zero, int first, int step) {
  const int64_t n = (int64_t)f.nx * f.ny * f.nz, pl = (int64_t)f.ny * f.nz;
  const int nz = f.nz;
  const int64_t chunks = (n + 31) / 32;
  const int lane = threadIdx.x & 31;
  const int nv = (int)(chunks < VW ? chunks : VW);
  for (int v = first; v < nv; v += step) {
    double rr = 0.0, rm = 0.0;
    for (int64_t u = v; u < chunks; u += VW) {
      const int64_t c = u * 32 + lane;
      if (c >= n) continue;
      const uint32_t m = __ldg(f.mask + c);
      if (!(m & BSP_MFLUID)) continue;
      double r = g.in.bscale * (double)__ldg(g.in.div + c);
      if (!zero) {
        const int k = (int)(c % nz);
        const int64_t t = c / nz;
        const int j = (int)(t % f.ny), i = (int)(t / f.ny);
        const double xc = x[c];
        auto nbx = [&](bool in, int64_t off) {
          if (!in) return 0.0;
          const uint32_t mn = __ldg(f.mask + c + off);
          return (mn & BSP_MFLUID) ? x[c + off] : ((mn & BSP_MSOLID) ? xc : 0.0);
        };
        const double s = nbx(i > 0, -pl) + nbx(i + 1 < f.nx, pl) + nbx(j > 0, -nz) +
                         nbx(j + 1 < f.ny, nz) + nbx(k > 0, -1) + nbx(k + 1 < nz, 1);
        r -= 6.0 * xc - s;
      }
      if (WRITE) {
        stv(rhat, c, (float)(r * scale));
        e[c] = 0.0f;
      } else {
        rr += r * r;
        rm = fmax(rm, fabs(r));
      }
    }
    if (!WRITE) {
      put(g, SLOT_RR, v, rr);
      rm = warp_max(rm);
      if (lane == 0) __stcg(g.partials + (size_t)SLOT_MAX * PSTRIDE + v, rm);
    }
  }
}

// Coarsest level in one CTA: e = M r, or SWEEPS Jacobi sweeps from zero.
template <class T>
__device__ void coarsest(Ctx<T> &g, const LevelP<T> &L) {
  const int n = L.nx * L.ny * L.nz, t = threadIdx.x;
  if (t < n) {
    g.rr[t] = ld(L.r, t);
    g.e0[t] = 0.0f;
  }
  __syncthreads();
  if (*(volatile const int *)g.in.cflag) {
    const int parts = THREADS / n, col = t % n, pi = t / n;
    if (pi < parts) {
      const int j0 = n * pi / parts, j1 = n * (pi + 1) / parts;
      float acc = 0.0f;
      for (int j = j0; j < j1; ++j) acc = fmaf(__ldg(g.in.cinv + (int64_t)j * n + col), g.rr[j], acc);
      g.part[pi * n + col] = acc;
    }
    __syncthreads();
    if (t < n) {
      float acc = 0.0f;
      for (int q = 0; q < parts; ++q) acc += g.part[q * n + t];
      stv(L.e, t, (__ldg(L.mask + t) & BSP_MFLUID) ? acc : 0.0f);
    }
  } else {
    const int pl = L.ny * L.nz;
    float *a = g.e0, *b = g.e1;
    for (int s = 0; s < SWEEPS; ++s) {
      if (t < n) {
        const uint32_t m = __ldg(L.mask + t);
        float v = 0.0f;
        if (m & BSP_MFLUID) {
          const int k = t % L.nz, j = t / L.nz % L.ny, i = t / pl;
          const float ec = a[t];
          auto nbe = [&](bool in, int off) {
            if (!in) return 0.0f;
            const uint32_t mn = __ldg(L.mask + t + off);
            return (mn & BSP_MFLUID) ? a[t + off] : ((mn & BSP_MSOLID) ? ec : 0.0f);
          };
          const float sum = nbe(i > 0, -pl) + nbe(i + 1 < L.nx, pl) + nbe(j > 0, -L.nz) +
                            nbe(j + 1 < L.ny, L.nz) + nbe(k > 0, -1) + nbe(k + 1 < L.nz, 1);
          v = ec + (g.rr[t] - (6.0f * ec - sum)) / (6.0f - (float)(m & 7u));
        }
        b[t] = v;
      }
      __syncthreads();
      float *x = a;
      a = b;
      b = x;
    }
    if (t < n) stv(L.e, t, a[t]);
  }
  __syncthreads();
}

template <class T>
__global__ void __launch_bounds__(THREADS, 1) group_solve_kernel(const __grid_constant__ Params P) {
  __shared__ Ctx<T> g;
  __shared__ LevelP<T> lv[MAXL];
  int q = 0;
  while (q + 1 < P.count && (int)blockIdx.x >= P.in[q + 1].cta0) ++q;
  const int tid = threadIdx.x, warp = tid >> 5;
  if (tid == 0) {
    g.in = P.in[q];
    g.rank = (int)blockIdx.x - g.in.cta0;
    g.size = g.in.ncta;
    g.epoch = 0;
    g.ctl = reinterpret_cast<GridCtl *>(g.in.base + g.in.off_ctl);
    g.partials = reinterpret_cast<double *>(g.in.base + g.in.off_partials);
    for (int n = 0; n < 8; ++n) {
      const float d = 6.0f - (float)n;
      g.wt[n] = d > 0.0f ? __fdividef(W, d) : 0.0f;
    }
    int x = g.in.nx, y = g.in.ny, z = g.in.nz;
    for (int l = 0; l < g.in.L; ++l) {
      lv[l].nx = x;
      lv[l].ny = y;
      lv[l].nz = z;
      lv[l].mask = l == 0 ? g.in.mask : reinterpret_cast<const uint8_t *>(g.in.base + g.in.off_lv[l]);
      lv[l].r = reinterpret_cast<T *>(g.in.base + (l == 0 ? g.in.off_r : g.in.off_lr[l]));
      lv[l].e = reinterpret_cast<T *>(g.in.base + (l == 0 ? g.in.off_z : g.in.off_le[l]));
      x = (x + 1) / 2;
      y = (y + 1) / 2;
      z = (z + 1) / 2;
    }
  }
  __syncthreads();
  const int L = g.in.L;
  const int64_t n = (int64_t)g.in.nx * g.in.ny * g.in.nz;
  const int first = g.rank * WARPS + warp, step = g.size * WARPS;  // virtual warps of this warp
  const int64_t t0 = (int64_t)g.rank * THREADS + tid, tstep = (int64_t)g.size * THREADS;
  double *x = reinterpret_cast<double *>(g.in.base + g.in.off_x);
  float *e = reinterpret_cast<float *>(g.in.base + g.in.off_e);
  T *z = lv[0].e, *b0 = lv[0].r, *b1 = reinterpret_cast<T *>(g.in.base + g.in.off_r2);
  T *ps0 = reinterpret_cast<T *>(g.in.base + g.in.off_ps0);
  T *ps1 = reinterpret_cast<T *>(g.in.base + g.in.off_ps1);
  T *Ap = reinterpret_cast<T *>(g.in.base + g.in.off_Ap);
  const int nres = (int)((n + 31) / 32 < VW ? (n + 31) / 32 : VW);
  const Dims d0 = dims_of(g.in.nx, g.in.ny, g.in.nz);
  const int n0 = vwarps<T>(d0.units);
  // levels from `tail` on run in the group's first CTA
  int tail = 1;
  while (tail < L - 1 && (int64_t)lv[tail].nx * lv[tail].ny * lv[tail].nz > TAIL_CELLS) ++tail;

  int status = BSP_OK, outer_it = 0, total_inner = 0;
  double rel = 0.0;
  bool lost = false;  // a barrier gave up
  // ---- x from the guess, ||b|| ------------------------------------------------------
  residual<T, false>(g, lv[0], x, nullptr, nullptr, 1.0, true, first, step);
  for (int64_t c = t0; c < n; c += tstep)
    x[c] = P.warm && (__ldg(g.in.mask + c) & BSP_MFLUID) ? (double)g.in.p[c] : 0.0;
  lost = !barrier(g);
  double bb = 0.0, rr = 0.0, rmax = 0.0;
  if (!lost) {
    bb = total(g, SLOT_RR, nres, false);
    rr = bb;
    rmax = total(g, SLOT_MAX, nres, true);
  }
  bool xzero = !P.warm;
  for (int outer = 0; !lost; ++outer) {
    if (!xzero) {
      __syncthreads();
      if (outer == 0) {
        // the partials of ||b|| are read by every CTA before they are replaced
        if (!barrier(g)) { lost = true; break; }
      }
      residual<T, false>(g, lv[0], x, nullptr, nullptr, 1.0, false, first, step);
      if (!barrier(g)) { lost = true; break; }
      rr = total(g, SLOT_RR, nres, false);
      rmax = total(g, SLOT_MAX, nres, true);
    }
    // the outer check of solver.cu, the same in every CTA
    rel = bb > 0.0 ? sqrt(rr / bb) : 0.0;
    if (!(rr == rr) || rr > 1e300) {
      status = BSP_ERR_NONFINITE;
      break;
    }
    if (bb == 0.0 || rel <= P.tol) break;
    if (outer_it >= P.max_outer) {
      status = BSP_NOT_CONVERGED;
      break;
    }
    const double scale = rmax > 0.0 ? 1.0 / rmax : 1.0;
    const double rhat2 = rr * scale * scale;
    const double eta = fmax(P.eta, 0.5 * P.tol * sqrt(bb / rr));
    ++outer_it;
    residual<T, true>(g, lv[0], x, b1, e, scale, xzero, first, step);
    if (!barrier(g)) { lost = true; break; }
    // ---- conjugate gradient ---------------------------------------------------------
    double rz = 0.0, alpha = 0.0;
    bool pending = false;
    int it = 0;
    for (int s = 0;; ++s) {
      const T *rin = (s & 1) ? b0 : b1;
      T *r = (s & 1) ? b1 : b0;
      T *cur = (s & 1) ? ps1 : ps0;
      const T *prev = (s & 1) ? ps0 : ps1;
      down<T, true>(g, lv[0], lv[1], rin, r, Ap, prev, e, (float)alpha, pending, first, step);
      if (!barrier(g)) { lost = true; break; }
      if (pending) {
        const double r2 = total(g, SLOT_RR, n0, false);
        ++it;
        ++total_inner;
        if (!(r2 == r2) || r2 <= eta * eta * rhat2 || it >= P.max_inner || alpha == 0.0) break;
      }
      for (int l = 1; l < tail; ++l) {
        down<T, false>(g, lv[l], lv[l + 1], lv[l].r, nullptr, nullptr, nullptr, nullptr, 0.0f,
                       false, first, step);
        if (!barrier(g)) { lost = true; break; }
      }
      if (lost) break;
      if (g.rank == 0) {
        for (int l = tail; l < L - 1; ++l) {
          down<T, false>(g, lv[l], lv[l + 1], lv[l].r, nullptr, nullptr, nullptr, nullptr, 0.0f,
                         false, warp, WARPS);
          __syncthreads();
        }
        coarsest(g, lv[L - 1]);
        for (int l = L - 2; l >= tail; --l) {
          up<T, false>(g, lv[l], lv[l + 1], lv[l].r, lv[l].e, P.alpha, warp, WARPS);
          __syncthreads();
        }
      }
      if (!barrier(g)) { lost = true; break; }
      for (int l = tail - 1; l >= 1; --l) {
        up<T, false>(g, lv[l], lv[l + 1], lv[l].r, lv[l].e, P.alpha, first, step);
        if (!barrier(g)) { lost = true; break; }
      }
      if (lost) break;
      up<T, true>(g, lv[0], lv[1], r, z, P.alpha, first, step);
      if (!barrier(g)) { lost = true; break; }
      const double rzn = total(g, SLOT_RZ, n0, false);
      const double beta = (it == 0 || rz == 0.0) ? 0.0 : rzn / rz;
      rz = rzn;
      direction(g, lv[0], z, prev, cur, Ap, (float)beta, it == 0, first, step);
      if (!barrier(g)) { lost = true; break; }
      const double pap = total(g, SLOT_PAP, n0, false);
      alpha = pap > 0.0 ? rz / pap : 0.0;
      pending = true;
    }
    if (lost) break;
    const double inv = 1.0 / scale;
    for (int64_t c = t0; c < n; c += tstep)
      if (__ldg(g.in.mask + c) & BSP_MFLUID) x[c] += (double)e[c] * inv;
    xzero = false;
    if (!barrier(g)) { lost = true; break; }
  }
  if (lost) status = BSP_ERR_TIMEOUT;
  if (g.in.p && !lost)
    for (int64_t c = t0; c < n; c += tstep)
      g.in.p[c] = (__ldg(g.in.mask + c) & BSP_MFLUID) ? (float)x[c] : 0.0f;
  if (g.rank == 0 && tid == 0) {
    Result *o = reinterpret_cast<Result *>(g.in.base + g.in.off_result);
    o->status = status;
    o->outer_it = outer_it;
    o->total_inner = total_inner;
    o->rel = rel;
  }
}

template <class T>
cudaError_t launch(const Params &P, int ctas, cudaStream_t s) {
  void *args[] = {const_cast<Params *>(&P)};
  return cudaLaunchCooperativeKernel((const void *)group_solve_kernel<T>, dim3((unsigned)ctas),
                                     dim3(THREADS), args, 0, s);
}

}  // namespace grp

// Shares `sms` CTAs out over P's instances by their cells (at least one each) and
// launches.  P.count <= min(GROUP_MAX, sms).
template <class T>
cudaError_t launch_group_solve(grp::Params &P, cudaStream_t s) {
  const int sms = num_sms();
  double cells = 0.0;
  for (int q = 0; q < P.count; ++q) cells += (double)P.in[q].nx * P.in[q].ny * P.in[q].nz;
  int used = 0;
  std::vector<double> want(P.count);
  for (int q = 0; q < P.count; ++q) {
    want[q] = (double)P.in[q].nx * P.in[q].ny * P.in[q].nz / cells * sms;
    P.in[q].ncta = std::max(1, (int)want[q]);
    used += P.in[q].ncta;
  }
  // what the rounding left goes where the most cells wait per CTA
  for (; used < sms; ++used) {
    int at = 0;
    for (int q = 1; q < P.count; ++q)
      if (want[q] / P.in[q].ncta > want[at] / P.in[at].ncta) at = q;
    ++P.in[at].ncta;
  }
  for (; used > sms; --used) {
    int at = -1;
    for (int q = 0; q < P.count; ++q)
      if (P.in[q].ncta > 1 && (at < 0 || want[q] / P.in[q].ncta < want[at] / P.in[at].ncta)) at = q;
    --P.in[at].ncta;
  }
  int first = 0;
  for (int q = 0; q < P.count; ++q) {
    P.in[q].cta0 = first;
    first += P.in[q].ncta;
  }
  return grp::launch<T>(P, first, s);
}

template cudaError_t launch_group_solve<float>(grp::Params &, cudaStream_t);
template cudaError_t launch_group_solve<__half>(grp::Params &, cudaStream_t);
template cudaError_t launch_group_solve<__nv_bfloat16>(grp::Params &, cudaStream_t);

}  // namespace bsp
