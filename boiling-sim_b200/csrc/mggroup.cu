// mggroup.cu -- the to-tolerance solve (solver.cu) of small and ragged grids as one
// cooperative launch: FP64 refinement, conjugate gradient and V-cycle of one or
// many instances, each by a group of CTAs with a barrier of its own.
//
// On a grid of up to a few million cells an inner iteration's kernels take
// microseconds each, so its two dozen launches (and, in a batch, the WHILE nodes of
// a graph's branches, which hardly overlap) were the time: 83 us an iteration at
// 110x110x68, 2.7 ms an instance of a batch.  Here a group runs a phase and
// meets at a barrier on a counter in the instance's workspace (about 1.2 us over
// 148 CTAs, less over few), ten of them an iteration; the SMs are shared out over the
// instances by their cells, so a batch's instances run side by side.
//
// Measured, per-kernel path -> here: 110x110x68 FP16 2.00 -> 1.31 ms, 16 uneven pots
// FP32 12.7 -> 9.2 ms with their setups kept (39.9 ms instead of 47.0 with them made),
// 200x200x130 FP16 (rows of no whole quads, where the per-kernel path
// has no tiles) 10.3 -> 4.4 ms, 331x327x201 FP32 36.4 -> 13.5 ms, 384x384x120 BF16 10.7 ->
// 10.5 ms.  An iteration at 110x110x68 is 110 k cycles: 33 k on level 0, 40 k on the
// coarse levels (latency of one round each), 25 k of barriers; in a batch
// the level-0 phases' instructions bound it (54 % of the issue slots).
//
// The cycle, the smoother, the stopping tests, the storage and the order of the
// floating-point operations on every cell are the per-kernel path's with one sweep a
// side on every level, to the four-cell FP32 chains of its dots: 16-bit directions turn
// a last place of alpha or beta into another iterate within the tolerance.  Only the FP64 sums
// of those chains are taken in another order, far below a place of the FP32 scalars made
// from them, so the results are that path's bits.  Every such sum is taken over a fixed
// number of virtual warps and then over those in a fixed order, so a result does not depend on how
// many CTAs its group has: single, batched, host-driven and device-driven solves agree
// bit for bit.
#include <cuda_bf16.h>
#include <cuda_fp16.h>

#include <algorithm>
#include <cstring>

#include "bsp_common.cuh"
#include "grid_sync.cuh"
#include "mggroup.cuh"
#include "profile.cuh"

namespace bsp {

int num_sms();

namespace grp {

constexpr int THREADS = 1024, WARPS = THREADS / 32;
constexpr int VB = 148;             // virtual blocks of a sum
constexpr int KOUT = 30;            // k cells of a unit
constexpr int KQUADS = 28;          // of a level-0 unit on rows of whole quads: whole quads
constexpr float W = 6.0f / 7.0f;    // smoothing weight
constexpr float W_C = 1.0f - W;
constexpr int SEG = 4;              // j values of a level-0 unit
constexpr int SWEEPS = 64;          // coarsest level without an inverse
// code byte of a cell: bit 7 fluid, bits 0-5 solid neighbour (-i, +i, -j, +j, -k, +k)
constexpr uint32_t FLUID = 0x80u, SOLIDS = 0x3fu;

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
  int ok;
  double total;                     // of the last barrier's slot
  float wt[256], ns[64];            // by code: W / (6 - solid neighbours), 0 off fluid; the count
  union {                           // each between two barriers
    double sums[VB * WARPS];        // one per virtual warp of this CTA's virtual blocks
    float part[2 * THREADS];        // columns of a restriction
    struct {
      float e0[COARSEST], e1[COARSEST], rr[COARSEST], psum[512], M[32 * COARSEST];  // coarsest
    };
  };
};

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

// Group barrier: arrivals on a counter that only grows; bounded.  sum_of >= 0:
// g.total is then the sum over all blocks of that slot (publish), in one order
// everywhere.
template <class T>
__device__ __forceinline__ bool barrier(Ctx<T> &g, int sum_of = -1) {
  __syncthreads();
  if (threadIdx.x < 32) {
    const int lane = threadIdx.x;
    int ok = 1;
    if (lane == 0 && g.size > 1) {
      const unsigned int target = ++g.epoch * (unsigned int)g.size;
      cuda::atomic_ref<unsigned int, cuda::thread_scope_device> cnt(g.ctl->bar_count);
      cuda::atomic_ref<int, cuda::thread_scope_device> err(g.ctl->err);
      asm volatile("fence.acq_rel.gpu;" ::: "memory");
      cnt.fetch_add(1u, cuda::memory_order_relaxed);
      unsigned int spins = 0;
      unsigned long long t0 = 0;
      while (cnt.load(cuda::memory_order_acquire) < target) {
        if ((++spins & 255u) == 0) {
          const unsigned long long now = gs_global_ns();
          if (t0 == 0) t0 = now;
          if (err.load(cuda::memory_order_relaxed) != 0 || now - t0 > BAR_TIMEOUT_NS ||
              spins > BAR_SPIN_LIMIT) {
            err.store(BSP_ERR_TIMEOUT, cuda::memory_order_relaxed);
            ok = 0;
            break;
          }
        }
      }
      g.ok = ok;
    }
    __syncwarp();
    if (sum_of >= 0) {
      const double *p = g.partials + (size_t)sum_of * PSTRIDE;
      double v[(VB + 31) / 32], s = 0.0;
#pragma unroll
      for (int m = 0; m < (VB + 31) / 32; ++m)
        v[m] = m * 32 + lane < VB ? __ldcg(p + m * 32 + lane) : 0.0;
#pragma unroll
      for (int m = 0; m < (VB + 31) / 32; ++m) s += v[m];
      s = warp_sum(s);
      if (lane == 0) g.total = s;
    }
  }
  __syncthreads();
  return g.ok != 0;
}

// ---- sums over cells -------------------------------------------------------------------
// Work is dealt to VB virtual blocks of WARPS virtual warps, whatever the
// group's size: virtual block b is run by CTA b % size.  put() keeps a virtual
// warp's sum, publish() adds each of the CTA's blocks and stores it, and the
// next barrier adds the blocks.
template <class T>
__device__ __forceinline__ void put(Ctx<T> &g, int b, double x) {
  x = warp_sum(x);
  if ((threadIdx.x & 31) == 0) g.sums[(b / g.size) * WARPS + (threadIdx.x >> 5)] = x;
}
template <class T>
__device__ __forceinline__ void publish(Ctx<T> &g, int q) {
  __syncthreads();
  const int lane = threadIdx.x & 31;
  for (int m = threadIdx.x >> 5; g.rank + m * g.size < VB; m += WARPS) {
    const double x = warp_sum(g.sums[m * WARPS + lane]);
    if (lane == 0) g.partials[(size_t)q * PSTRIDE + g.rank + m * g.size] = x;
  }
}

// ---- level 0: pairs of columns marched along j -----------------------------------------
// Unit: the columns (i, i + 1) of SEG values of j and 30 of k; a lane owns one k
// (lanes 0 and 31 are the k halo).  A step forms the operand at (i, j + 1),
// (i + 1, j + 1), (i - 1, j) and (i + 2, j) and keeps the rest from the steps before,
// with the next step's loads in flight: two values formed a cell instead of the five of
// a cell by itself.  Only units with fluid are dealt out.
struct Fine {
  int nx, ny, nz, segs, ch, kout;
};
__host__ __device__ __forceinline__ Fine fine_of(int nx, int ny, int nz) {
  const int kout = nz % 4 == 0 ? KQUADS : KOUT;
  return Fine{nx, ny, nz, (ny + SEG - 1) / SEG, (nz + kout - 1) / kout, kout};
}
struct Seg {
  int i, j0, j1, k, c;      // c: cell (i, j0, k), k clamped into the grid
  int ob, ol, orr;          // offsets of the columns i + 1, i - 1, i + 2 (0 outside the grid)
  uint32_t ma, mb, ml, mr;  // code bits that count, column by column: 0 outside the grid
  bool out;                 // an output lane
};
__device__ __forceinline__ Seg seg_of(const Fine &d, uint32_t u) {
  const int lane = threadIdx.x & 31, pl = d.ny * d.nz;
  Seg t;
  const int r = (int)(u / (uint32_t)d.ch), c = (int)u - r * d.ch;
  const int bi = (int)((uint32_t)r / (uint32_t)d.segs);
  t.i = 2 * bi;
  t.j0 = (r - bi * d.segs) * SEG;
  t.j1 = min(t.j0 + SEG, d.ny);
  t.k = c * d.kout - 1 + lane;
  const bool in = t.k >= 0 && t.k < d.nz, b = t.i + 1 < d.nx, l = t.i > 0, rr = t.i + 2 < d.nx;
  t.c = (t.i * d.ny + t.j0) * d.nz + min(max(t.k, 0), d.nz - 1);
  t.ob = b ? pl : 0;
  t.ol = l ? -pl : 0;
  t.orr = rr ? 2 * pl : 0;
  t.ma = in ? 0xffu : 0u;
  t.mb = b ? t.ma : 0u;
  t.ml = l ? t.ma : 0u;
  t.mr = rr ? t.ma : 0u;
  t.out = in && lane >= 1 && lane <= d.kout;
  return t;
}
// Neighbour sum of the operand values (0 off fluid), a solid neighbour counting as
// the cell itself; the k neighbours are the lanes beside.  Two orders, the ones the
// per-kernel path sums in (in 16 bits a last place is 5e-4 of a value): paired with n_solid
// x centre added (rows of whole quads), or one after the other with the centre in a
// solid neighbour's place (code bits 0-5).
__device__ __forceinline__ float six(float l, float r, float d, float u, float b, float f) {
  return ((l + r) + (d + u)) + (b + f);
}
template <bool PAIRED>
__device__ __forceinline__ float nsum(const float *ns, uint32_t code, float c, float l, float r,
                                      float d, float u) {
  float b = __shfl_up_sync(0xffffffffu, c, 1), f = __shfl_down_sync(0xffffffffu, c, 1);
  if constexpr (PAIRED) return fmaf(ns[code & SOLIDS], c, six(l, r, d, u, b, f));
  if (__any_sync(0xffffffffu, (code & SOLIDS) != 0)) {
    l = code & 1u ? c : l;
    r = code & 2u ? c : r;
    d = code & 4u ? c : d;
    u = code & 8u ? c : u;
    b = code & 16u ? c : b;
    f = code & 32u ? c : f;
  }
  return l + r + d + u + b + f;
}
// A thread's products of a dot, for its FP64 sum.  PAIRED, as the per-kernel path's
// four-cell chains: the four cells of a quad in one chain of FP32 FMAs along k (each
// lane takes the chain over from the lane before; the quad's last cell adds it).
// Otherwise each product by itself in FP64.  x, y: 0 where the cell does not count.
template <bool PAIRED>
__device__ __forceinline__ double prod(float x, float y, int k) {
  if constexpr (!PAIRED) return (double)x * (double)y;
  float v = __fmul_rn(x, y);  // of the quad's first cell
#pragma unroll
  for (int q = 1; q < 4; ++q) v = fmaf(x, y, __shfl_up_sync(0xffffffffu, v, 1));
  return (k & 3) == 3 ? (double)v : 0.0;
}
// Sum of a coarse cell's children: columns (i, j), (i, j + 1), (i + 1, j),
// (i + 1, j + 1), each the lane's k and the next lane's; in the per-kernel path's order
// (level 0 by rows, or child after child).
template <bool PAIRED>
__device__ __forceinline__ float children(float a, float a1, float b, float b1) {
  const float an = __shfl_down_sync(0xffffffffu, a, 1), a1n = __shfl_down_sync(0xffffffffu, a1, 1);
  const float bn = __shfl_down_sync(0xffffffffu, b, 1), b1n = __shfl_down_sync(0xffffffffu, b1, 1);
  if constexpr (PAIRED) return ((a + an) + (b + bn)) + ((a1 + a1n) + (b1 + b1n));
  return a + an + a1 + a1n + b + bn + b1 + b1n;
}

// An operand that is a product is rounded by itself (__fmul_rn), as the per-kernel path
// stores it: contracted into the neighbour sum, it took the restricted residual, and
// with it z, off that path's by last places.

// The march's loads carry no predicates: addresses outside the grid are
// clamped to a cell of it, and what such a lane, column or row may not add is
// taken out by its code (0: weight 0) or by a select.  Before the first update alpha is 0
// and Ap any finite vector, so that r - alpha Ap = r.

// Restriction of the residual of e = w r, after the pending CG update:
// r = r_in - alpha Ap, stored to r_out, and the sum r.r.
template <class T, bool PAIRED>
__device__ __noinline__ void down0(Ctx<T> &g, const LevelP<T> &f, const LevelP<T> &co,
                                   const T *r_in, T *r_out, const T *Ap, float alpha) {
  const Fine d = fine_of(f.nx, f.ny, f.nz);
  const uint32_t units = g.in.units[0];
  const int nz = d.nz, warp = threadIdx.x >> 5;
  const uint8_t *code = f.code;
  struct Centre {
    uint32_t ka, kb;
    T ra, rb, pa, pb;
  };
  struct Outer {
    uint32_t kl, kr;
    T rl, rr, pl, pr;
  };
  for (int vb = g.rank; vb < VB; vb += g.size) {
    double rr = 0.0;
    for (uint32_t n = vb * WARPS + warp; n < units; n += VB * WARPS) {
      const Seg t = seg_of(d, __ldg(g.in.units + 1 + n));
      auto centre = [&](int c) {
        return Centre{__ldg(code + c), __ldg(code + c + t.ob), r_in[c], r_in[c + t.ob], Ap[c],
                      Ap[c + t.ob]};
      };
      auto outer = [&](int c) {
        return Outer{__ldg(code + c + t.ol), __ldg(code + c + t.orr), r_in[c + t.ol],
                     r_in[c + t.orr], Ap[c + t.ol], Ap[c + t.orr]};
      };
      auto res = [&](const T &a, const T &b) {
        return rnd(fmaf(-alpha, ld(&b, 0), ld(&a, 0)), r_out);
      };
      int c = t.c;
      const Centre m = centre(t.j0 > 0 ? c - nz : c), now = centre(c);
      Centre up = centre(t.j0 + 1 < d.ny ? c + nz : c);
      Outer side = outer(c);
      float am = t.j0 > 0 ? __fmul_rn(res(m.ra, m.pa), g.wt[m.ka & t.ma]) : 0.0f;
      float bm = t.j0 > 0 ? __fmul_rn(res(m.rb, m.pb), g.wt[m.kb & t.mb]) : 0.0f;
      float ra = res(now.ra, now.pa), rb = res(now.rb, now.pb);
      uint32_t ka = now.ka & t.ma, kb = now.kb & t.mb;
      float a = __fmul_rn(ra, g.wt[ka]), b = __fmul_rn(rb, g.wt[kb]), ya1 = 0.0f, yb1 = 0.0f;
#pragma unroll 1
      for (int j = t.j0; j < t.j1; ++j, c += nz) {
        Centre up2 = up;
        Outer side2 = side;
        if (j + 1 < t.j1) {
          up2 = centre(j + 2 < d.ny ? c + 2 * nz : c + nz);
          side2 = outer(c + nz);
        }
        const uint32_t row = j + 1 < d.ny ? 0xffu : 0u;
        const uint32_t kau = up.ka & t.ma & row, kbu = up.kb & t.mb & row;
        const float rau = res(up.ra, up.pa), rbu = res(up.rb, up.pb);
        const float au = __fmul_rn(rau, g.wt[kau]), bu = __fmul_rn(rbu, g.wt[kbu]);
        const float l = __fmul_rn(res(side.rl, side.pl), g.wt[side.kl & t.ml]);
        const float r = __fmul_rn(res(side.rr, side.pr), g.wt[side.kr & t.mr]);
        const bool oa = t.out && (ka & FLUID), ob = t.out && (kb & FLUID);
        const float sa = nsum<PAIRED>(g.ns, ka, a, l, b, am, au);
        const float sb = nsum<PAIRED>(g.ns, kb, b, a, r, bm, bu);
        const float ya = oa ? ra - fmaf(6.0f, a, -sa) : 0.0f, yb = ob ? rb - fmaf(6.0f, b, -sb) : 0.0f;
        if (oa) stv(r_out, c, ra);
        if (ob) stv(r_out, c + t.ob, rb);
        const float xa = oa ? ra : 0.0f, xb = ob ? rb : 0.0f;
        rr += prod<PAIRED>(xa, xa, t.k) + prod<PAIRED>(xb, xb, t.k);
        if ((j & 1) || j + 1 == d.ny) {
          const bool odd = j & 1;
          const float acc = children<PAIRED>(odd ? ya1 : ya, odd ? ya : 0.0f, odd ? yb1 : yb,
                                             odd ? yb : 0.0f);
          if (t.out && !(t.k & 1)) {
            const int C = ((t.i >> 1) * co.ny + (j >> 1)) * co.nz + (t.k >> 1);
            if (__ldg(co.code + C) & FLUID) stv(co.r, C, 0.5f * acc);
          }
        }
        ya1 = ya, yb1 = yb;
        am = a, bm = b, a = au, b = bu, ra = rau, rb = rbu, ka = kau, kb = kbu;
        up = up2;
        side = side2;
      }
    }
    put(g, vb, rr);
  }
  publish(g, SLOT_RR);
}

// Prolongation and post-smoothing: e^ = alpha e_coarse[parent] + w r,
// out = e^ + w (r - A e^), and the sum r.out.
template <class T, bool PAIRED>
__device__ __noinline__ void up0(Ctx<T> &g, const LevelP<T> &f, const LevelP<T> &co, const T *r,
                                 T *out, float alpha) {
  const Fine d = fine_of(f.nx, f.ny, f.nz);
  const uint32_t units = g.in.units[0];
  const int nz = d.nz, cp = co.ny * co.nz, warp = threadIdx.x >> 5;
  const uint8_t *code = f.code;
  const T *ce = co.e;
  struct Centre {
    uint32_t ka, kb;
    T ra, rb, p;
  };
  struct Outer {
    uint32_t kl, kr;
    T rl, rr, pl, pr;
  };
  for (int vb = g.rank; vb < VB; vb += g.size) {
    double rz = 0.0;
    for (uint32_t n = vb * WARPS + warp; n < units; n += VB * WARPS) {
      const Seg t = seg_of(d, __ldg(g.in.units + 1 + n));
      const int P0 = (t.i >> 1) * cp + (min(max(t.k, 0), nz - 1) >> 1);
      const int Pl = t.ol ? P0 - cp : P0, Pr = t.orr ? P0 + cp : P0;
      auto centre = [&](int c, int j) {
        return Centre{__ldg(code + c), __ldg(code + c + t.ob), r[c], r[c + t.ob],
                      ce[P0 + (j >> 1) * co.nz]};
      };
      auto outer = [&](int c, int j) {
        return Outer{__ldg(code + c + t.ol), __ldg(code + c + t.orr), r[c + t.ol], r[c + t.orr],
                     ce[Pl + (j >> 1) * co.nz], ce[Pr + (j >> 1) * co.nz]};
      };
      auto hat = [&](uint32_t k, const T &p, const T &y) {
        const float w = g.wt[k], q = ld(&p, 0), v = ld(&y, 0);
        return k & FLUID ? (PAIRED ? fmaf(v, w, alpha * q) : fmaf(alpha, q, v * w)) : 0.0f;
      };
      // z = e^ + w (r - A e^), or the same as (1 - W) e^ + w (r + sum of the six)
      auto smooth = [&](uint32_t k, float v, float e, float l, float r1, float dn, float u) {
        const float w = g.wt[k];
        if constexpr (PAIRED) {
          const float s6 = six(l, r1, dn, u, __shfl_up_sync(0xffffffffu, e, 1),
                               __shfl_down_sync(0xffffffffu, e, 1));
          return w > 0.0f ? fmaf(w, v + s6, W_C * e) : e;
        }
        return fmaf(v - fmaf(6.0f, e, -nsum<false>(g.ns, k, e, l, r1, dn, u)), w, e);
      };
      int c = t.c;
      const int jm = t.j0 > 0 ? -1 : 0, jp = t.j0 + 1 < d.ny ? 1 : 0;
      const Centre m = centre(c + jm * nz, t.j0 + jm), now = centre(c, t.j0);
      Centre up = centre(c + jp * nz, t.j0 + jp);
      Outer side = outer(c, t.j0);
      const uint32_t row0 = t.j0 > 0 ? 0xffu : 0u;
      float am = hat(m.ka & t.ma & row0, m.p, m.ra), bm = hat(m.kb & t.mb & row0, m.p, m.rb);
      uint32_t ka = now.ka & t.ma, kb = now.kb & t.mb;
      float a = hat(ka, now.p, now.ra), b = hat(kb, now.p, now.rb);
      float ra = ld(&now.ra, 0), rb = ld(&now.rb, 0);
#pragma unroll 1
      for (int j = t.j0; j < t.j1; ++j, c += nz) {
        Centre up2 = up;
        Outer side2 = side;
        if (j + 1 < t.j1) {
          const int q = j + 2 < d.ny ? 2 : 1;
          up2 = centre(c + q * nz, j + q);
          side2 = outer(c + nz, j + 1);
        }
        const uint32_t row = j + 1 < d.ny ? 0xffu : 0u;
        const uint32_t kau = up.ka & t.ma & row, kbu = up.kb & t.mb & row;
        const float au = hat(kau, up.p, up.ra), bu = hat(kbu, up.p, up.rb);
        const float l = hat(side.kl & t.ml, side.pl, side.rl);
        const float r1 = hat(side.kr & t.mr, side.pr, side.rr);
        const float ya = smooth(ka, ra, a, l, b, am, au);
        const float yb = smooth(kb, rb, b, a, r1, bm, bu);
        const bool oa = t.out && (ka & FLUID), ob = t.out && (kb & FLUID);
        if (oa) stv(out, c, ya);
        if (ob) stv(out, c + t.ob, yb);
        rz += prod<PAIRED>(oa ? ra : 0.0f, oa ? rnd(ya, out) : 0.0f, t.k) +
              prod<PAIRED>(ob ? rb : 0.0f, ob ? rnd(yb, out) : 0.0f, t.k);
        am = a, bm = b, a = au, b = bu, ka = kau, kb = kbu;
        ra = ld(&up.ra, 0), rb = ld(&up.rb, 0);
        up = up2;
        side = side2;
      }
    }
    put(g, vb, rz);
  }
  publish(g, SLOT_RZ);
}

// ps = z + beta ps_prev (on a pass's first iteration beta and alpha are 0 and
// ps_prev any finite vector), Ap = A ps, sum ps.Ap; and the update e += alpha ps_prev
// of the iteration before, whose ps_prev is at hand here.
template <class T, bool PAIRED>
__device__ __noinline__ void direction(Ctx<T> &g, const LevelP<T> &f, const T *z, const T *prev,
                                       T *cur, T *Ap, float *e, float alpha, float beta) {
  const Fine d = fine_of(f.nx, f.ny, f.nz);
  const uint32_t units = g.in.units[0];
  const int nz = d.nz, warp = threadIdx.x >> 5;
  const uint8_t *code = f.code;
  struct Centre {
    T za, zb, pa, pb;
  };
  struct Outer {
    uint32_t ka, kb;  // of the centre columns
    T zl, zr, pl, pr;
  };
  for (int vb = g.rank; vb < VB; vb += g.size) {
    double pap = 0.0;
    for (uint32_t n = vb * WARPS + warp; n < units; n += VB * WARPS) {
      const Seg t = seg_of(d, __ldg(g.in.units + 1 + n));
      auto centre = [&](int c) {
        return Centre{z[c], z[c + t.ob], prev[c], prev[c + t.ob]};
      };
      auto outer = [&](int c) {
        return Outer{__ldg(code + c), __ldg(code + c + t.ob), z[c + t.ol], z[c + t.orr],
                     prev[c + t.ol], prev[c + t.orr]};
      };
      auto dir = [&](bool in, const T &a, const T &b) {
        return in ? rnd(fmaf(beta, ld(&b, 0), ld(&a, 0)), cur) : 0.0f;
      };
      int c = t.c;
      const Centre m = centre(t.j0 > 0 ? c - nz : c), now = centre(c);
      Centre up = centre(t.j0 + 1 < d.ny ? c + nz : c);
      Outer side = outer(c);
      float am = dir(t.ma && t.j0 > 0, m.za, m.pa), bm = dir(t.mb && t.j0 > 0, m.zb, m.pb);
      float a = dir(t.ma, now.za, now.pa), b = dir(t.mb, now.zb, now.pb);
      T pa = now.pa, pb = now.pb;
#pragma unroll 1
      for (int j = t.j0; j < t.j1; ++j, c += nz) {
        const float ea = e[c], eb = e[c + t.ob];
        Centre up2 = up;
        Outer side2 = side;
        if (j + 1 < t.j1) {
          up2 = centre(j + 2 < d.ny ? c + 2 * nz : c + nz);
          side2 = outer(c + nz);
        }
        const bool row = j + 1 < d.ny;
        const float au = dir(t.ma && row, up.za, up.pa), bu = dir(t.mb && row, up.zb, up.pb);
        const float l = dir(t.ml, side.zl, side.pl), r = dir(t.mr, side.zr, side.pr);
        const float sa = nsum<PAIRED>(g.ns, side.ka, a, l, b, am, au);
        const float sb = nsum<PAIRED>(g.ns, side.kb, b, a, r, bm, bu);
        const bool oa = t.out && (side.ka & FLUID), ob = t.out && (side.kb & t.mb & FLUID);
        const float apa = oa ? rnd(fmaf(6.0f, a, -sa), Ap) : 0.0f;
        const float apb = ob ? rnd(fmaf(6.0f, b, -sb), Ap) : 0.0f;
        if (oa) {
          stv(cur, c, a);
          e[c] = fmaf(alpha, ld(&pa, 0), ea);
          stv(Ap, c, apa);
        }
        if (ob) {
          stv(cur, c + t.ob, b);
          e[c + t.ob] = fmaf(alpha, ld(&pb, 0), eb);
          stv(Ap, c + t.ob, apb);
        }
        pap += prod<PAIRED>(oa ? a : 0.0f, apa, t.k) + prod<PAIRED>(ob ? b : 0.0f, apb, t.k);
        am = a, bm = b, a = au, b = bu, pa = up.pa, pb = up.pb;
        up = up2;
        side = side2;
      }
    }
    put(g, vb, pap);
  }
  publish(g, SLOT_PAP);
}

// ---- coarse levels: one column and 30 k cells a warp ------------------------------------
// A level is a round or two over the group's warps, so its time is one chain of
// latency and the barrier: all loads of a column are issued together.
struct Col {
  int c, ol, orr, od, ou;          // the lane's cell (clamped into the grid), its lateral
                                   // neighbours' offsets (0 outside the grid)
  uint32_t m, ml, mr, md, mu;      // code bits that count: 0 outside the grid
  bool out;
};
__device__ __forceinline__ Col col_of(int nx, int ny, int nz, int i, int j, int k) {
  const int lane = threadIdx.x & 31;
  const bool in = i < nx && j < ny && k >= 0 && k < nz;
  Col x;
  x.c = (min(i, nx - 1) * ny + min(j, ny - 1)) * nz + min(max(k, 0), nz - 1);
  x.m = in ? 0xffu : 0u;
  x.ml = i > 0 ? x.m : 0u;
  x.mr = i + 1 < nx ? x.m : 0u;
  x.md = j > 0 ? x.m : 0u;
  x.mu = j + 1 < ny ? x.m : 0u;
  x.ol = x.ml ? -ny * nz : 0;
  x.orr = x.mr ? ny * nz : 0;
  x.od = x.md ? -nz : 0;
  x.ou = x.mu ? nz : 0;
  x.out = in && lane >= 1 && lane <= KOUT;
  return x;
}
template <class T>
struct Five {
  T c, l, r, d, u;
};
template <class T>
__device__ __forceinline__ Five<T> five(const T *a, const Col &x) {
  const T *p = a + x.c;
  return Five<T>{p[0], p[x.ol], p[x.orr], p[x.od], p[x.ou]};
}
__device__ __forceinline__ Five<uint32_t> codes(const uint8_t *a, const Col &x) {
  const uint8_t *p = a + x.c;
  return Five<uint32_t>{__ldg(p) & x.m, __ldg(p + x.ol) & x.ml, __ldg(p + x.orr) & x.mr,
                        __ldg(p + x.od) & x.md, __ldg(p + x.ou) & x.mu};
}

// Restriction of the residual of e = w r on level f to level co's r: the four
// columns of a coarse column are four warps', added in shared memory.
template <class T, bool PAIRED>
__device__ __noinline__ void down(Ctx<T> &g, const LevelP<T> &f, const LevelP<T> &co) {
  const int nz = f.nz, ch = (nz + KOUT - 1) / KOUT, units = co.nx * co.ny * ch;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, quad = warp >> 2, q = warp & 3;
  int flip = 0;
  for (int u = g.rank * (WARPS / 4) + quad; u < units; u += g.size * (WARPS / 4), flip ^= THREADS) {
    const int r = u / ch, I = r / co.ny, J = r - I * co.ny, k = (u - r * ch) * KOUT - 1 + lane;
    const Col x = col_of(f.nx, f.ny, nz, 2 * I + (q >> 1), 2 * J + (q & 1), k);
    const Five<uint32_t> m = codes(f.code, x);
    const Five<T> v = five(f.r, x);
    const int C = (I * co.ny + J) * co.nz + (k >> 1);
    const bool emit = q == 0 && !(k & 1) && k >= 0 && k < nz && lane >= 1 && lane <= KOUT;
    const uint32_t mc = emit ? (uint32_t)__ldg(co.code + C) : 0u;
    auto pre = [&](const T &r, uint32_t n) { return __fmul_rn(ld(&r, 0), g.wt[n]); };
    const float y = ld(&v.c, 0), c = pre(v.c, m.c);
    const float s = nsum<PAIRED>(g.ns, m.c, c, pre(v.l, m.l), pre(v.r, m.r), pre(v.d, m.d),
                                 pre(v.u, m.u));
    float *part = g.part + flip;
    part[threadIdx.x] = x.out && (m.c & FLUID) ? y - fmaf(6.0f, c, -s) : 0.0f;
    asm volatile("bar.sync %0, 128;" ::"r"(quad + 1) : "memory");
    if (q == 0) {
      const float *p = part + threadIdx.x;
      // child after child, or pair after pair of k
      float acc = 0.0f;
      for (int w = 0; w < 128; w += 32) {
        const float y0 = p[w], y1 = __shfl_down_sync(0xffffffffu, y0, 1);
        acc = PAIRED ? acc + (y0 + y1) : acc + y0 + y1;
      }
      if (mc & FLUID) stv(co.r, C, 0.5f * acc);
    }
  }
}

// Prolongation and post-smoothing of a coarse level (up0 without the sum).
template <class T, bool PAIRED>
__device__ __noinline__ void up(Ctx<T> &g, const LevelP<T> &f, const LevelP<T> &co, float alpha) {
  const int nz = f.nz, ch = (nz + KOUT - 1) / KOUT, units = f.nx * f.ny * ch;
  const int cp = co.ny * co.nz, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  for (int u = g.rank * WARPS + warp; u < units; u += g.size * WARPS) {
    const int t = u / ch, i = t / f.ny, j = t - i * f.ny, k = (u - t * ch) * KOUT - 1 + lane;
    const Col x = col_of(f.nx, f.ny, nz, i, j, k);
    const Five<uint32_t> m = codes(f.code, x);
    const Five<T> v = five(f.r, x);
    const T *ce = co.e;
    const int P = ((i >> 1) * co.ny + (j >> 1)) * co.nz + (min(max(k, 0), nz - 1) >> 1);
    // a neighbour's parent: the cell's own or the one beside it
    const Five<T> p{ce[P], ce[x.ml && !(i & 1) ? P - cp : P], ce[x.mr && (i & 1) ? P + cp : P],
                    ce[x.md && !(j & 1) ? P - co.nz : P], ce[x.mu && (j & 1) ? P + co.nz : P]};
    auto hat = [&](uint32_t n, const T &e, const T &y) {
      const float w = g.wt[n], q = ld(&e, 0), v1 = ld(&y, 0);
      return n & FLUID ? (PAIRED ? fmaf(v1, w, alpha * q) : fmaf(alpha, q, v1 * w)) : 0.0f;
    };
    const float y = ld(&v.c, 0), c = hat(m.c, p.c, v.c);
    const float s = nsum<PAIRED>(g.ns, m.c, c, hat(m.l, p.l, v.l),
                         hat(m.r, p.r, v.r), hat(m.d, p.d, v.d), hat(m.u, p.u, v.u));
    if (x.out && (m.c & FLUID)) stv(f.e, x.c, fmaf(y - fmaf(6.0f, c, -s), g.wt[m.c], c));
  }
}

// FP64 residual b - A x on level 0.  WRITE: rhat = scale r (stored as T), e = 0;
// else the sum of squares and the largest |r|.  zero: x is zero.  The neighbours are
// summed in the per-kernel path's orders, as in nsum (quads: paired).
template <class T, bool WRITE>
__device__ void residual(Ctx<T> &g, const LevelP<T> &f, const double *x, T *rhat, float *e,
                         double scale, bool zero) {
  const int ny = f.ny, nz = f.nz, pl = ny * nz, n = f.nx * pl;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  double rm = 0.0;
  for (int vb = g.rank; vb < VB; vb += g.size) {
    double rr = 0.0;
    for (int c = (vb * WARPS + warp) * 32 + lane; c < n; c += VB * THREADS) {
      const uint32_t m = __ldg(f.code + c);
      if (!(m & FLUID)) continue;
      const double b = (double)__ldg(g.in.div + c);
      double ax = 0.0;
      if (!zero) {
        const int t = c / nz, k = c - t * nz, i = t / ny, j = t - i * ny;
        const double xc = x[c];
        auto at = [&](bool in, int off) { return in ? x[c + off] : 0.0; };  // 0 off fluid
        const double l = at(i > 0, -pl), r1 = at(i + 1 < f.nx, pl), d = at(j > 0, -nz);
        const double u = at(j + 1 < ny, nz), k0 = at(k > 0, -1), k1 = at(k + 1 < nz, 1);
        double s;
        if (g.in.quads) {
          s = fma((double)__popc(m & SOLIDS), xc, ((l + r1) + (d + u)) + (k0 + k1));
        } else {  // a solid neighbour gives the cell's own value
          auto own = [&](uint32_t bit, double v) { return m & bit ? xc : v; };
          s = own(1u, l) + own(2u, r1) + own(4u, d) + own(8u, u) + own(16u, k0) + own(32u, k1);
        }
        ax = fma(6.0, xc, -s);
      }
      const double r = fma(g.in.bscale, b, -ax);
      if (WRITE) {
        stv(rhat, c, (float)(r * scale));
        e[c] = 0.0f;
      } else {
        rr += r * r;
        rm = fmax(rm, fabs(r));
      }
    }
    if (!WRITE) put(g, vb, rr);
  }
  if (!WRITE) {
    publish(g, SLOT_RR);
    __syncthreads();
    // the largest by CTA: exact in any order
    rm = warp_max(rm);
    if (lane == 0) g.sums[warp] = rm;
    __syncthreads();
    if (warp == 0) {
      rm = warp_max(g.sums[lane]);
      if (lane == 0) g.partials[(size_t)SLOT_MAX * PSTRIDE + g.rank] = rm;
    }
  }
}
template <class T>
__device__ double largest(const Ctx<T> &g) {
  const double *p = g.partials + (size_t)SLOT_MAX * PSTRIDE;
  double s = 0.0;
  for (int b = threadIdx.x & 31; b < g.size; b += 32) s = fmax(s, __ldcg(p + b));
  return warp_max(s);
}

// Coarsest level: e = M r, or, without an inverse, SWEEPS Jacobi sweeps from zero
// in the first CTA.  M is symmetric: a warp per row, or threads along a row of M
// with the sum of a column in parts (the per-kernel path's two orders).
template <class T>
__device__ void coarsest(Ctx<T> &g, const LevelP<T> &L) {
  const int n = L.nx * L.ny * L.nz, t = threadIdx.x;
  const bool direct = __ldg(g.in.cflag) != 0;
  if (direct && g.in.paired) {
    const int lane = t & 31;
    for (int row = g.rank * WARPS + (t >> 5); row < n; row += g.size * WARPS) {
      const float *M = g.in.cinv + row * n;
      float a[COARSEST / 32], y[COARSEST / 32];
#pragma unroll
      for (int m = 0; m < COARSEST / 32; ++m) {
        const int j = m * 32 + lane;
        a[m] = j < n ? __ldg(M + j) : 0.0f;
        y[m] = j < n ? ld(L.r, j) : 0.0f;
      }
      const uint32_t code = __ldg(L.code + row);
      float acc = 0.0f;
#pragma unroll
      for (int m = 0; m < COARSEST / 32; ++m) acc = fmaf(a[m], y[m], acc);
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
      if (lane == 0) stv(L.e, row, code & FLUID ? acc : 0.0f);
    }
  } else if (direct) {
    // 32 columns of M a CTA, staged so that all its loads are in flight together, their
    // parts side by side (512 / n parts: at most 512 threads)
    const int parts = 512 / n, cw = min(n, 32), pi = t / cw, lc = t - pi * cw;
    for (int c0 = g.rank * cw; c0 < n; c0 += g.size * cw) {
      const int col = min(c0 + (t & 31), n - 1);
#pragma unroll
      for (int q = 0; q < COARSEST / WARPS; ++q) {
        const int j = q * WARPS + (t >> 5);
        if (j < n) g.M[j * 32 + (t & 31)] = __ldg(g.in.cinv + j * n + col);
      }
      if (t < n) g.rr[t] = ld(L.r, t);
      __syncthreads();
      if (pi < parts) {
        const int j0 = n * pi / parts, j1 = n * (pi + 1) / parts;
        float acc = 0.0f;
#pragma unroll 8
        for (int j = j0; j < j1; ++j) acc = fmaf(g.M[j * 32 + lc], g.rr[j], acc);
        g.psum[t] = acc;
      }
      __syncthreads();
      if (t < cw && c0 + t < n) {
        float acc = 0.0f;
        for (int q = 0; q < parts; ++q) acc += g.psum[q * cw + t];
        stv(L.e, c0 + t, (__ldg(L.code + c0 + t) & FLUID) ? acc : 0.0f);
      }
    }
  } else if (g.rank == 0) {
    const int pl = L.ny * L.nz;
    float *a = g.e0, *b = g.e1;
    if (t < n) {
      g.rr[t] = ld(L.r, t);
      a[t] = 0.0f;
    }
    __syncthreads();
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
            return (mn & BSP_MFLUID) ? a[t + off] : ((mn & BSP_MSOLID) && !g.in.paired ? ec : 0.0f);
          };
          const float l = nbe(i > 0, -pl), r = nbe(i + 1 < L.nx, pl), d = nbe(j > 0, -L.nz);
          const float u = nbe(j + 1 < L.ny, L.nz), bk = nbe(k > 0, -1), f = nbe(k + 1 < L.nz, 1);
          if (g.in.paired) {  // damped; nbe of a solid is then 0 and the centre added after
            const float n = (float)(m & 7u), w = 6.0f - n;
            const float sum = fmaf(n, ec, six(l, r, d, u, bk, f));
            v = fmaf(g.rr[t] - fmaf(6.0f, ec, -sum), w > 0.0f ? __fdividef(W, w) : 0.0f, ec);
          } else {
            const float sum = l + r + d + u + bk + f;
            v = ec + (g.rr[t] - fmaf(6.0f, ec, -sum)) / (6.0f - (float)(m & 7u));
          }
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
}

template <class T>
__global__ void __launch_bounds__(THREADS, 1) group_solve_kernel(const __grid_constant__ Params P) {
  __shared__ Ctx<T> g;
  __shared__ LevelP<T> lv[MAXL];
  if (threadIdx.x < 256) {
    if (threadIdx.x < 64) g.ns[threadIdx.x] = (float)__popc(threadIdx.x);
    const float d = 6.0f - (float)__popc(threadIdx.x & SOLIDS);
    g.wt[threadIdx.x] = (threadIdx.x & FLUID) && d > 0.0f ? __fdividef(W, d) : 0.0f;
  }
  int q = 0;
  while (q + 1 < P.count && (int)blockIdx.x >= P.in[q + 1].cta0) ++q;
  const int tid = threadIdx.x;
  if (tid == 0) {
    g.in = P.in[q];
    g.rank = (int)blockIdx.x - g.in.cta0;
    g.size = g.in.ncta;
    g.epoch = 0;
    g.ok = 1;
    g.ctl = reinterpret_cast<GridCtl *>(g.in.base + g.in.off_ctl);
    g.partials = reinterpret_cast<double *>(g.in.base + g.in.off_partials);
    int x = g.in.nx, y = g.in.ny, z = g.in.nz;
    for (int l = 0; l < g.in.L; ++l) {
      lv[l].nx = x;
      lv[l].ny = y;
      lv[l].nz = z;
      lv[l].code = reinterpret_cast<const uint8_t *>(g.in.base + g.in.off_code[l]);
      lv[l].mask =
          l == 0 ? g.in.mask : reinterpret_cast<const uint8_t *>(g.in.base + g.in.off_lv[l]);
      lv[l].r = reinterpret_cast<T *>(g.in.base + (l == 0 ? g.in.off_r : g.in.off_lr[l]));
      lv[l].e = reinterpret_cast<T *>(g.in.base + (l == 0 ? g.in.off_z : g.in.off_le[l]));
      x = (x + 1) / 2;
      y = (y + 1) / 2;
      z = (z + 1) / 2;
    }
  }
  __syncthreads();
  const int L = g.in.L;
  const int n = g.in.nx * g.in.ny * g.in.nz;
  const int t0 = g.rank * THREADS + tid, tstep = g.size * THREADS;
  double *x = reinterpret_cast<double *>(g.in.base + g.in.off_x);
  float *e = reinterpret_cast<float *>(g.in.base + g.in.off_e);
  T *z = lv[0].e, *b0 = lv[0].r, *b1 = reinterpret_cast<T *>(g.in.base + g.in.off_r2);
  T *ps0 = reinterpret_cast<T *>(g.in.base + g.in.off_ps0);
  T *ps1 = reinterpret_cast<T *>(g.in.base + g.in.off_ps1);
  T *Ap = reinterpret_cast<T *>(g.in.base + g.in.off_Ap);
  int status = BSP_OK, outer_it = 0, total_inner = 0;
  double rel = 0.0;
  bool lost = false;  // a barrier gave up
  // ---- x from the guess, ||b|| ------------------------------------------------------
  residual<T, false>(g, lv[0], x, nullptr, nullptr, 1.0, true);
  for (int c = t0; c < n; c += tstep)
    x[c] = P.warm && (__ldg(lv[0].code + c) & FLUID) ? (double)g.in.p[c] : 0.0;
  lost = !barrier(g, SLOT_RR);
  double bb = 0.0, rr = 0.0, rmax = 0.0;
  if (!lost) {
    bb = g.total;
    rr = bb;
    rmax = largest(g);
  }
  bool xzero = !P.warm;
  for (int outer = 0; !lost; ++outer) {
    if (!xzero) {
      __syncthreads();
      if (outer == 0) {
        // the partials of ||b|| are read by every CTA before they are replaced
        if (!barrier(g)) { lost = true; break; }
      }
      residual<T, false>(g, lv[0], x, nullptr, nullptr, 1.0, false);
      if (!barrier(g, SLOT_RR)) { lost = true; break; }
      rr = g.total;
      rmax = largest(g);
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
    residual<T, true>(g, lv[0], x, b1, e, scale, xzero);
    if (!barrier(g)) { lost = true; break; }
    // ---- conjugate gradient ---------------------------------------------------------
    double rz = 0.0, alpha = 0.0;
    bool pending = false;
    int it = 0;
    const T *last = ps0;  // direction of the last update, not yet in e
    for (int s = 0;; ++s) {
      const T *rin = (s & 1) ? b0 : b1;
      T *r = (s & 1) ? b1 : b0;
      T *cur = (s & 1) ? ps1 : ps0;
      const T *prev = (s & 1) ? ps0 : ps1;
      const T *ap = pending ? Ap : rin;
      const float al = pending ? (float)alpha : 0.0f;
      if (g.in.paired0)
        down0<T, true>(g, lv[0], lv[1], rin, r, ap, al);
      else
        down0<T, false>(g, lv[0], lv[1], rin, r, ap, al);
      if (!barrier(g, SLOT_RR)) { lost = true; break; }
      if (pending) {
        const double r2 = g.total;
        ++it;
        ++total_inner;
        last = prev;
        if (!(r2 == r2) || r2 <= eta * eta * rhat2 || it >= P.max_inner || alpha == 0.0) break;
      }
      for (int l = 1; l < L - 1 && !lost; ++l) {
        if (g.in.paired)
          down<T, true>(g, lv[l], lv[l + 1]);
        else
          down<T, false>(g, lv[l], lv[l + 1]);
        lost = !barrier(g);
      }
      if (lost) break;
      coarsest(g, lv[L - 1]);
      if (!barrier(g)) { lost = true; break; }
      for (int l = L - 2; l >= 1 && !lost; --l) {
        if (g.in.paired)
          up<T, true>(g, lv[l], lv[l + 1], P.alpha);
        else
          up<T, false>(g, lv[l], lv[l + 1], P.alpha);
        lost = !barrier(g);
      }
      if (lost) break;
      if (g.in.paired0)
        up0<T, true>(g, lv[0], lv[1], r, z, P.alpha);
      else
        up0<T, false>(g, lv[0], lv[1], r, z, P.alpha);
      if (!barrier(g, SLOT_RZ)) { lost = true; break; }
      const double rzn = g.total;
      const double beta = (it == 0 || rz == 0.0) ? 0.0 : rzn / rz;
      rz = rzn;
      const T *dp = it == 0 ? z : prev;
      const float be = it == 0 ? 0.0f : (float)beta;
      if (g.in.paired0)
        direction<T, true>(g, lv[0], z, dp, cur, Ap, e, al, be);
      else
        direction<T, false>(g, lv[0], z, dp, cur, Ap, e, al, be);
      if (!barrier(g, SLOT_PAP)) { lost = true; break; }
      const double pap = g.total;
      alpha = pap > 0.0 ? rz / pap : 0.0;
      pending = true;
    }
    if (lost) break;
    const double inv = 1.0 / scale;
    for (int c = t0; c < n; c += tstep)
      if (__ldg(lv[0].code + c) & FLUID)
        x[c] += (double)fmaf((float)alpha, ld(last, c), e[c]) * inv;
    xzero = false;
    if (!barrier(g)) { lost = true; break; }
  }
  if (lost) status = BSP_ERR_TIMEOUT;
  if (g.in.p && !lost)
    for (int c = t0; c < n; c += tstep)
      g.in.p[c] = (__ldg(lv[0].code + c) & FLUID) ? (float)x[c] : 0.0f;
  if (g.rank == 0 && tid == 0) {
    Result *o = reinterpret_cast<Result *>(g.in.base + g.in.off_result);
    o->status = status;
    o->outer_it = outer_it;
    o->total_inner = total_inner;
    o->rel = rel;
  }
}

// Code bytes of a level from its mask (class and solid count).
__global__ void __launch_bounds__(256) code_kernel(uint8_t *__restrict__ code,
                                                   const uint8_t *__restrict__ mask, int nx, int ny,
                                                   int nz) {
  const int n = nx * ny * nz, pl = ny * nz;
  for (int c = blockIdx.x * 256 + threadIdx.x; c < n; c += gridDim.x * 256) {
    const uint32_t m = mask[c];
    uint32_t v = 0;
    if (m & BSP_MFLUID) {
      const int t = c / nz, k = c - t * nz, i = t / ny, j = t - i * ny;
      auto sol = [&](bool in, int off) { return in && (mask[c + off] & BSP_MSOLID) ? 1u : 0u; };
      v = FLUID;
      if (m & BSP_MASK_NSOLID)
        v |= sol(i > 0, -pl) | sol(i + 1 < nx, pl) << 1 | sol(j > 0, -nz) << 2 |
             sol(j + 1 < ny, nz) << 3 | sol(k > 0, -1) << 4 | sol(k + 1 < nz, 1) << 5;
    }
    code[c] = (uint8_t)v;
  }
}
// flag[u]: level-0 unit u has fluid (a warp each).
__global__ void __launch_bounds__(256) unit_flag_kernel(uint8_t *__restrict__ flag,
                                                        const uint8_t *__restrict__ mask, Fine d,
                                                        int units) {
  for (int u = blockIdx.x * 8 + (threadIdx.x >> 5); u < units; u += gridDim.x * 8) {
    const Seg t = seg_of(d, (uint32_t)u);
    uint32_t m = 0;
    for (int j = t.j0, c = t.c; j < t.j1; ++j, c += d.nz) {
      m |= mask[c] & t.ma;
      m |= mask[c + t.ob] & t.mb;
    }
    const bool any = __any_sync(0xffffffffu, t.out && (m & BSP_MFLUID));
    if ((threadIdx.x & 31) == 0) flag[u] = any;
  }
}
// list[0] = number of units with fluid, list[1..] = those units in order.  One CTA.
__global__ void __launch_bounds__(THREADS) unit_list_kernel(uint32_t *__restrict__ list,
                                                            const uint8_t *__restrict__ flag,
                                                            int units) {
  __shared__ uint32_t s[THREADS];
  const int t = threadIdx.x, per = (units + THREADS - 1) / THREADS;
  const int u0 = min(units, t * per), u1 = min(units, u0 + per);
  uint32_t n = 0;
  for (int u = u0; u < u1; ++u) n += flag[u];
  s[t] = n;
  __syncthreads();
  for (int o = 1; o < THREADS; o <<= 1) {
    const uint32_t v = t >= o ? s[t - o] : 0u;
    __syncthreads();
    s[t] += v;
    __syncthreads();
  }
  uint32_t at = 1 + s[t] - n;
  for (int u = u0; u < u1; ++u)
    if (flag[u]) list[at++] = (uint32_t)u;
  if (t == THREADS - 1) list[0] = s[t];
}

template <class T>
cudaError_t launch(const Params &P, int ctas, cudaStream_t s) {
  void *args[] = {const_cast<Params *>(&P)};
  return launch_coop((const void *)group_solve_kernel<T>, dim3((unsigned)ctas), dim3(THREADS), args,
                     0, s);
}

}  // namespace grp

void launch_group_codes(uint8_t *code, const uint8_t *mask, int nx, int ny, int nz,
                        cudaStream_t s) {
  const int n = nx * ny * nz;
  grp::code_kernel<<<std::max(1, std::min((n + 255) / 256, num_sms() * 8)), 256, 0, s>>>(
      code, mask, nx, ny, nz);
}
size_t group_units(int nx, int ny, int nz) {
  const grp::Fine d = grp::fine_of(nx, ny, nz);
  return (size_t)((nx + 1) / 2) * d.segs * d.ch;
}
void launch_group_units(uint32_t *list, uint8_t *flag, const uint8_t *mask, int nx, int ny, int nz,
                        cudaStream_t s) {
  const int n = (int)group_units(nx, ny, nz);
  grp::unit_flag_kernel<<<std::max(1, std::min((n + 7) / 8, num_sms() * 8)), 256, 0, s>>>(
      flag, mask, grp::fine_of(nx, ny, nz), n);
  grp::unit_list_kernel<<<1, grp::THREADS, 0, s>>>(list, flag, n);
}

// Shares the CTAs out over P's instances by their cells (at least one each) and
// launches.  P.count <= min(GROUP_MAX, the device's SMs).
template <class T>
cudaError_t launch_group_solve(grp::Params &P, int ctas, cudaStream_t s) {
  const int sms = std::min(std::max(ctas, P.count), num_sms());
  double cells = 0.0;
  for (int q = 0; q < P.count; ++q) cells += (double)P.in[q].nx * P.in[q].ny * P.in[q].nz;
  int used = 0;
  double want[grp::GROUP_MAX];
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

template cudaError_t launch_group_solve<float>(grp::Params &, int, cudaStream_t);
template cudaError_t launch_group_solve<__half>(grp::Params &, int, cudaStream_t);
template cudaError_t launch_group_solve<__nv_bfloat16>(grp::Params &, int, cudaStream_t);

}  // namespace bsp
