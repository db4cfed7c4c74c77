// pcgr.cu -- the reference-compatible Jacobi-PCG (pcg.cu) with every vector on chip.
//
// The two phases of an iteration move 10 floats a cell through L2 and classify the
// material ids of 7 cells in each: 22 us an iteration at 110x110x68, where the fluid
// is 5 k cells an SM.  Here a CTA owns a block of (i, j) columns for the whole solve:
// the search direction of the block and its halo and r lie in shared memory, p
// and z (A ps between the phases) in registers, and only fluid cells are worked
// on, from a list made once.  What crosses CTAs in an iteration is z of the cells at a
// block's sides, read after the barrier that the sum r.z needs anyway; the halo's
// search direction is formed from it on both sides of a border.
//
// An iteration is two barriers with their sums (2.9 k and 3.5 k cycles) and passes over
// four to six cells a thread (6.3 k cycles).  Measured, streaming form -> here: 110x110x68
// 6.25 -> 1.76 ms a solve, 56x56x40 4.14 -> 1.41 ms, 150x150x110 27.3 -> 7.7 ms.
//
// Per-cell arithmetic is pcg.cu's; the FP64 sums run in another order, fixed for a
// grid size.
#include <algorithm>

#include "blocks.cuh"
#include "grid_sync.cuh"
#include "pcgr.cuh"

namespace bsp {

int num_sms();

constexpr int PR_THREADS = 1024, PR_WARPS = PR_THREADS / 32;
constexpr int PR_SLOTS = 16;                  // fluid cells a thread, at most
constexpr int PR_COLS = 512;                  // columns of a block (list entry)
constexpr int PR_SMEM = 227 * 1024 - 4096;    // dynamic shared memory a CTA may take
// list entry: place in P | solid neighbours (-i, +i, -j, +j, -k, +k) << 16 | side << 22 |
// column << 23
constexpr uint32_t PR_SIDE = 1u << 22;

struct PrSync {
  double red[2][PR_WARPS];  // of the CTA's warps
  double tot[2];
  unsigned int epoch;       // barriers passed
  int ok;
  float2 dinv[64];          // by solid bits: D and 1 / D
};

__device__ __forceinline__ double pr_warp_sum(double v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// Grid barrier (arrivals on a counter that only grows; bounded) that adds up K sums:
// v[q] = the sum over the grid, in one order everywhere.  One thread polls and one
// warp reads the sums: with all CTAs polling all CTAs' sums themselves a
// barrier took 9 k to 20 k cycles instead of 4 k.
template <int K>
__device__ __forceinline__ bool pr_barrier(PrSync &s, const PcgrArgs &a, double (&v)[K],
                                           double *partials) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nb = gridDim.x;
#pragma unroll
  for (int q = 0; q < K; ++q) {
    v[q] = pr_warp_sum(v[q]);
    if (lane == 0) s.red[q][warp] = v[q];
  }
  __syncthreads();
  if (warp == 0) {
#pragma unroll
    for (int q = 0; q < K; ++q) v[q] = pr_warp_sum(s.red[q][lane]);
    if (lane == 0) {
#pragma unroll
      for (int q = 0; q < K; ++q) __stcg(partials + q * nb + blockIdx.x, v[q]);
      const unsigned int target = ++s.epoch * (unsigned int)nb;
      cuda::atomic_ref<unsigned int, cuda::thread_scope_device> cnt(a.ctl->bar_count);
      cuda::atomic_ref<int, cuda::thread_scope_device> err(a.ctl->err);
      asm volatile("fence.acq_rel.gpu;" ::: "memory");
      cnt.fetch_add(1u, cuda::memory_order_relaxed);
      int ok = 1;
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
      s.ok = ok;
    }
    __syncwarp();
    double t[K][5];
#pragma unroll
    for (int q = 0; q < K; ++q)
#pragma unroll
      for (int m = 0; m < 5; ++m) {  // at most 160 CTAs
        const int b = m * 32 + lane;
        t[q][m] = b < nb ? __ldcg(partials + q * nb + b) : 0.0;
      }
#pragma unroll
    for (int q = 0; q < K; ++q) {
      const double x = pr_warp_sum((((t[q][0] + t[q][1]) + t[q][2]) + t[q][3]) + t[q][4]);
      if (lane == 0) s.tot[q] = x;
    }
  }
  __syncthreads();
#pragma unroll
  for (int q = 0; q < K; ++q) v[q] = s.tot[q];
  return s.ok != 0;
}

// r / D, correctly rounded (D is 1 .. 6).  Its guard takes 1.6 % of a solve (1802 -> 1832 us at
// 110x110x68; with one guard for all of a thread's cells the registers spill, 2.4 %).
// A cell with no open neighbour keeps r.
__device__ __forceinline__ float pr_dinv(const PrSync &s, float r, uint32_t e) {
  const float2 d = s.dinv[(e >> 16) & 63u];
  return div_small(r, d.x, d.y);
}

__global__ void __launch_bounds__(PR_THREADS, 1)
    pcg_resident_kernel(const __grid_constant__ PcgrArgs a) {
  extern __shared__ float pr_smem[];
  __shared__ PrSync s;
  __shared__ int wcount[PR_WARPS + 1];
  float *P = pr_smem;                                      // ps of the block and its halo
  float *R = P + a.pad;                                    // r by slot
  uint32_t *E = reinterpret_cast<uint32_t *>(R + a.cap);   // the list
  int *gp = reinterpret_cast<int *>(E + a.cap);            // column -> cell - place in P
  int2 *H = reinterpret_cast<int2 *>(gp + (a.cols + 1) / 2 * 2);  // halo: 32 k cells each
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int nx = a.nx, ny = a.ny, nz = a.nz, plane = ny * nz;
  const int bi = blockIdx.x / a.nby, bj = blockIdx.x - bi * a.nby;
  const int i0 = (int)((int64_t)nx * bi / a.nbx), i1 = (int)((int64_t)nx * (bi + 1) / a.nbx);
  const int j0 = (int)((int64_t)ny * bj / a.nby), j1 = (int)((int64_t)ny * (bj + 1) / a.nby);
  const int w = i1 - i0, h = j1 - j0, ncol = w * h;
  const int dk = nz + 2, di = (h + 2) * dk;                // strides of P along j, i
  // halo columns (li, lj) of the four sides, 32 k cells at a time: cell and place in P |
  // cells << 16 (none outside the grid)
  const int hcols = 2 * (w + h), ch = (nz + 31) / 32, halo = hcols * ch;
  for (int n = tid; n < halo; n += PR_THREADS) {
    const int hc = n / ch, k = (n - hc * ch) * 32;
    int li, lj;
    if (hc < h) li = -1, lj = hc;
    else if (hc < 2 * h) li = w, lj = hc - h;
    else if (hc < 2 * h + w) li = hc - 2 * h, lj = -1;
    else li = hc - 2 * h - w, lj = h;
    const int i = i0 + li, j = j0 + lj;
    const bool in = i >= 0 && i < nx && j >= 0 && j < ny;
    H[n] = make_int2((i * ny + j) * nz + k,
                     ((li + 1) * di + (lj + 1) * dk + 1 + k) | (in ? min(nz - k, 32) << 16 : 0));
  }
  if (tid == 0) {
    s.ok = 1;
    s.epoch = 0;
  }
  if (tid < 64) {
    const float d = 6.0f - (float)__popc(tid);
    s.dinv[tid] = d > 0.0f ? make_float2(d, rcp_of(d)) : make_float2(1.0f, 1.0f);
  }
  for (int c = tid; c < ncol; c += PR_THREADS) {
    const int li = c / h, lj = c - li * h;
    gp[c] = ((i0 + li) * ny + j0 + lj) * nz - ((li + 1) * di + (lj + 1) * dk + 1);
  }
  for (int c = tid; c < (w + 2) * di; c += PR_THREADS) P[c] = 0.0f;
  __syncthreads();

  // ---- the list of fluid cells, b, and 0 where the solve writes nothing -------------
  int nf = 0;
  for (int base = 0; base < ncol * nz; base += PR_THREADS) {
    const int l = base + tid;
    bool fluid = false;
    uint32_t entry = 0;
    float b = 0.0f;
    if (l < ncol * nz) {
      const int col = l / nz, k = l - col * nz, li = col / h, lj = col - li * h;
      const int at = (li + 1) * di + (lj + 1) * dk + 1 + k, c = gp[col] + at;
      const int i = i0 + li, j = j0 + lj;
      const bool side = li == 0 || li + 1 == w || lj == 0 || lj + 1 == h;
      fluid = classify(__ldg(a.mat + c), a.mf, a.ma) == BSP_FLUID;
      if (fluid) {
        auto sol = [&](bool in, int off) {
          return in && classify(__ldg(a.mat + c + off), a.mf, a.ma) == BSP_SOLID ? 1u : 0u;
        };
        const uint32_t bits = sol(i > 0, -plane) | sol(i + 1 < nx, plane) << 1 |
                              sol(j > 0, -nz) << 2 | sol(j + 1 < ny, nz) << 3 |
                              sol(k > 0, -1) << 4 | sol(k + 1 < nz, 1) << 5;
        entry = (uint32_t)at | bits << 16 | (side ? PR_SIDE : 0u) | (uint32_t)col << 23;
        b = __fmul_rn(a.scale, __ldg(a.div + c));
      } else if (side) {
        a.z[c] = 0.0f;
      }
      a.p[c] = 0.0f;
    }
    const unsigned int vote = __ballot_sync(0xffffffffu, fluid);
    if (lane == 0) wcount[warp] = __popc(vote);
    __syncthreads();
    int before = 0, all = 0;
    {
      int n = wcount[lane], x = n;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= o) x += y;
      }
      all = __shfl_sync(0xffffffffu, x, 31);
      before = __shfl_sync(0xffffffffu, x - n, warp);
    }
    const int at = nf + before + __popc(vote & ((1u << lane) - 1u));
    if (fluid && at < a.cap) {
      E[at] = entry;
      R[at] = b;
    }
    nf += all;
    __syncthreads();
  }
  const bool over = nf > a.cap;
  nf = min(nf, a.cap);
  __syncthreads();

  // ---- z = D^-1 b, p = 0 -----------------------------------------------------------
  float X[PR_SLOTS], p[PR_SLOTS];  // X: z, and A ps between the phases
  double v[2] = {0.0, 0.0};
  // cleared by the host before the launch, read after the barrier
  if (over && tid == 0) __stcg(&a.ctl->status, PR_AGAIN);
#pragma unroll
  for (int q = 0; q < PR_SLOTS; ++q) {
    const int t = q * PR_THREADS + tid;
    X[q] = 0.0f;
    p[q] = 0.0f;
    if (t < nf) {
      const uint32_t e = E[t];
      const float b = R[t];
      X[q] = pr_dinv(s, b, e);
      if (e & PR_SIDE) __stcg(a.z + gp[e >> 23] + (int)(e & 0xffffu), X[q]);
      v[0] += (double)b * (double)b;
      v[1] += (double)b * (double)X[q];
    }
  }
  if (!pr_barrier<2>(s, a, v, a.partials + PCG_SUM_INIT * gridDim.x)) return;
  // the same in every CTA (nothing else that is ever written there is PR_AGAIN)
  if (__ldcg(&a.ctl->status) == PR_AGAIN) return;
  const double bsq = v[0];
  double rz = v[1];
  double alpha = 0.0, beta = 0.0, rz_new = 0.0, rsq = bsq, pAp = 0.0;
  int iters = 0, status = BSP_OK;
  if (!(bsq == bsq) || bsq > 1.0e300) status = BSP_ERR_NONFINITE;

  if (status == BSP_OK && bsq != 0.0) {
    const double tol_sq_bsq = a.tol2 * bsq;
    int it = 0;
    for (it = 0; it < a.max_iter; ++it) {
      const float bf = (float)beta;
      const bool first = it == 0;
      auto ps_of = [&](float z, float prev) { return first ? z : __fmaf_rn(bf, prev, z); };
      // ---- phase A: ps = z + beta ps on the block and its halo, A ps, ps.Ap ----------
      constexpr int HQ = 4;  // halo loads in flight under the block's own cells
      float hz[HQ];
      int hat[HQ];
#pragma unroll
      for (int m = 0; m < HQ; ++m) {
        const int n = warp + m * PR_WARPS;
        const int2 x = n < halo ? H[n] : make_int2(0, 0);
        const bool in = lane < x.y >> 16;
        hat[m] = in ? (x.y & 0xffff) + lane : -1;
        hz[m] = in ? __ldcg(a.z + x.x + lane) : 0.0f;
      }
#pragma unroll
      for (int q = 0; q < PR_SLOTS; ++q) {
        const int t = q * PR_THREADS + tid;
        if (q * PR_THREADS >= nf) break;
        if (t < nf) {
          const uint32_t e = E[t];
          float *ps = P + (e & 0xffffu);
          *ps = ps_of(X[q], *ps);
        }
      }
#pragma unroll
      for (int m = 0; m < HQ; ++m)
        if (hat[m] >= 0) P[hat[m]] = ps_of(hz[m], P[hat[m]]);
      for (int n = warp + HQ * PR_WARPS; n < halo; n += PR_WARPS) {
        const int2 x = H[n];
        float *ps = P + (x.y & 0xffff) + lane;
        if (lane < x.y >> 16) *ps = ps_of(__ldcg(a.z + x.x + lane), *ps);
      }
      __syncthreads();
      {
        double d[1] = {0.0};
#pragma unroll
        for (int q = 0; q < PR_SLOTS; ++q) {
          const int t = q * PR_THREADS + tid;
          if (q * PR_THREADS >= nf) break;
          if (t < nf) {
            const uint32_t e = E[t];
            const float *ps = P + (e & 0xffffu);
            // P is 0 on air and outside the grid; a solid neighbour gives the centre
            const float c = ps[0];
            float l = ps[-di], r = ps[di], dn = ps[-dk], up = ps[dk], bk = ps[-1], f = ps[1];
            const uint32_t m = e >> 16;
            if (m & 63u) {
              l = m & 1u ? c : l;
              r = m & 2u ? c : r;
              dn = m & 4u ? c : dn;
              up = m & 8u ? c : up;
              bk = m & 16u ? c : bk;
              f = m & 32u ? c : f;
            }
            X[q] = spmv_update(l, r, dn, up, bk, f, c);
            d[0] += (double)c * (double)X[q];
          }
        }
        if (!pr_barrier<1>(s, a, d, a.partials + PCG_SUM_A * gridDim.x)) return;
        pAp = d[0];
      }
      alpha = (pAp == 0.0) ? 0.0 : rz / pAp;
      const float af = (float)alpha;
      // ---- phase B: p += alpha ps, r -= alpha Ap, z = D^-1 r, r.z, r.r ---------------
      {
        double d[2] = {0.0, 0.0};
#pragma unroll
        for (int q = 0; q < PR_SLOTS; ++q) {
          const int t = q * PR_THREADS + tid;
          if (q * PR_THREADS >= nf) break;
          if (t < nf) {
            const uint32_t e = E[t];
            p[q] = __fmaf_rn(af, P[e & 0xffffu], p[q]);
            const float r = __fmaf_rn(-af, X[q], R[t]);
            R[t] = r;
            const float z = pr_dinv(s, r, e);
            X[q] = z;
            if (e & PR_SIDE) __stcg(a.z + gp[e >> 23] + (int)(e & 0xffffu), z);
            d[0] += (double)r * (double)z;
            d[1] += (double)r * (double)r;
          }
        }
        if (!pr_barrier<2>(s, a, d, a.partials + PCG_SUM_B * gridDim.x)) return;
        rz_new = d[0];
        rsq = d[1];
      }
      if (it >= 8 && (it % 5) == 0 && rsq < tol_sq_bsq) {
        ++it;
        break;
      }
      beta = (rz == 0.0) ? 0.0 : rz_new / rz;
      rz = rz_new;
    }
    iters = it;
#pragma unroll
    for (int q = 0; q < PR_SLOTS; ++q) {
      const int t = q * PR_THREADS + tid;
      if (t < nf) a.p[gp[E[t] >> 23] + (int)(E[t] & 0xffffu)] = p[q];
    }
  }
  if (blockIdx.x == 0 && tid == 0) {
    a.ctl->iters = iters;
    a.ctl->status = status;
    const double vals[7] = {alpha, beta, rz, rz_new, bsq, rsq, pAp};
#pragma unroll
    for (int q = 0; q < 7; ++q)
      if (a.outs[q]) *a.outs[q] = (float)vals[q];
  }
}

// Taken where the largest block's padded search direction leaves slots for 2/5 of
// its cells: the pots' fluid is half of their cells, and a block in the middle of one
// is nearly all fluid below the water line.  What does not fit is known only
// after the list is made (a few tens of microseconds of a solve of milliseconds)
// and solved by the streaming form.
bool pcg_resident_fits(int nx, int ny, int nz, int ctas, PcgrPlan &plan) {
  const int64_t n = (int64_t)nx * ny * nz;
  if (n > (1 << 28)) return false;
  ctas = std::min(ctas, 160);
  const BlockSplit b = split_blocks(nx, ny, ctas);
  plan.nbx = b.nbx;
  plan.nby = b.nby;
  const int w = b.w, h = b.h;
  const int64_t pad = (int64_t)(w + 2) * (h + 2) * (nz + 2);
  if ((int64_t)w * h > PR_COLS || pad > (1 << 16)) return false;
  plan.cols = w * h;
  plan.pad = (int)pad;
  plan.halo = 2 * (w + h) * ((nz + 31) / 32);
  const int cells = plan.cols * nz;
  const int64_t left = (int64_t)PR_SMEM - 4 * pad - 4 * (plan.cols + 2) - 8 * plan.halo;
  if (left <= 0) return false;
  plan.cap = (int)std::min<int64_t>({left / 8, (int64_t)cells, (int64_t)PR_SLOTS * PR_THREADS});
  plan.bytes = 4 * ((size_t)plan.pad + (plan.pad & 1) + 2 * (size_t)plan.cap +
                    (plan.cols + 1) / 2 * 2 + 2 * (size_t)plan.halo);
  return (int64_t)plan.cap * 5 >= (int64_t)cells * 2;
}

cudaError_t launch_pcg_resident(PcgrArgs &a, const PcgrPlan &plan, cudaStream_t s) {
  a.nbx = plan.nbx;
  a.nby = plan.nby;
  a.cap = plan.cap;
  a.pad = plan.pad + (plan.pad & 1);
  a.cols = plan.cols;
  const cudaError_t e = cudaFuncSetAttribute(
      pcg_resident_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, PR_SMEM);
  if (e != cudaSuccess) return e;
  void *args[] = {&a};
  return launch_coop((const void *)pcg_resident_kernel, dim3(a.nbx * a.nby), dim3(PR_THREADS), args,
                     plan.bytes, s);
}

}  // namespace bsp
