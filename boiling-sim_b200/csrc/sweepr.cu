// sweepr.cu -- the Jacobi sweeps of a projection with the pressure resident in
// shared memory: one cooperative launch runs all sweeps (jacobi.cu, from p = 0,
// rho dx^2 div / dt hoisted into rhs).
//
// A sweep of a small grid costs a launch and a chain of load latencies, and the
// instructions that form global addresses outnumber the arithmetic.  Taken for grids whose
// windows fit the SMs (make_plan: up to 2.1 M cells in rows of whole quads, 4.5 M in others): a
// CTA (one per SM) owns bi x bj columns of the grid and keeps them, with a halo
// of T columns, in shared memory over all sweeps.  A round is T sweeps (each
// valid one column less far into the halo), the store of the band of T columns
// along the tile's edge to global memory, a grid barrier and the load of the
// neighbours' bands.  The barrier's word is p_tmp's first element, which no neighbour's halo
// reaches (make_plan) and no band is stored to: memory of this call alone.  Only the last
// round stores whole tiles.  Bands alternate between p and p_tmp, so a CTA that runs ahead
// never overwrites a band that a neighbour still reads.  Every update is the reference's arithmetic in the
// reference's order: the result is bit-identical to single sweeps.
//
// A thread owns up to Q quads (four k cells) of the tile and its halo, keeps
// their new values in registers between the two CTA barriers of a sweep, and
// (RR) their rhs over the whole solve.  Quads without fluid are skipped.
#include <algorithm>

#include "bsp_common.cuh"
#include "f32x2.cuh"
#include "grid_sync.cuh"
#include "profile.cuh"
#include "waits.cuh"

namespace bsp {

int num_sms();
extern bool g_one_launch;      // BSP_TUNE_ONE_LAUNCH (stencil.cu)
extern int g_test_wait_error;  // BSP_TUNE_TEST_WAIT_ERROR (stencil.cu)

namespace swr {

constexpr int THREADS = 512;
constexpr int HQ = 2;  // halo quads a thread loads at once
// Sweeps from which one launch is taken: making the lists costs about five launches (a
// projection of 2 / 5 / 10 / 16 sweeps, single and in one launch, us: 58x58x38 34 / 42 / 48 / 62
// and 39 / 43 / 53 / 63; 110x110x68 52 / 71 / 88 / 115 and 61 / 73 / 90 / 111; 130x131x97 75 / 111 /
// 152 / 211 and 82 / 102 / 134 / 171).
constexpr int MIN_SWEEPS = 10;
constexpr int SMEM_MAX = 232448 - 1024;  // dynamic; the rest is static

struct Args {
  float *p, *p_tmp;
  const float *rhs;
  const uint8_t *mask;
  int *err;           // marked when the barrier gave up
  int nx, ny, nz;
  int bi, bj;
  int extra;      // arrivals beyond the CTAs that a barrier waits for (0, or the error test's 1)
  int n, rounds;  // sweeps, rounds (round r: n / rounds sweeps, one more while r < n % rounds)
};

// bits 0-3: bytes of w with bit 7 (fluid) / bit 6 (solid) set
__device__ __forceinline__ uint32_t bits4(uint32_t w, int bit) {
  const uint32_t b = (w >> bit) & 0x01010101u;
  return (b | (b >> 7) | (b >> 14) | (b >> 21)) & 15u;
}
template <bool AL>
__device__ __forceinline__ uint32_t mask4(const uint8_t *__restrict__ m, int64_t c, int k,
                                          int nz) {
  if (AL) return __ldg(reinterpret_cast<const uint32_t *>(m + c));
  uint32_t w = 0;
#pragma unroll
  for (int q = 0; q < 4; ++q)
    if (k + q < nz) w |= (uint32_t)__ldg(m + c + q) << (8 * q);
  return w;
}
// Four consecutive floats, +0 beyond the row's end.  Through L2 (the bands are
// written by other SMs in this launch).
template <bool AL>
__device__ __forceinline__ Quad load4(const float *m, int64_t c, int k, int nz) {
  if (AL) {
    const ulonglong2 t = __ldcg(reinterpret_cast<const ulonglong2 *>(m + c));
    return Quad{t.x, t.y};
  }
  float v[4];
#pragma unroll
  for (int q = 0; q < 4; ++q) v[q] = k + q < nz ? __ldcg(m + c + q) : 0.0f;
  return quad(v);
}
template <bool AL>
__device__ __forceinline__ void store4(float *m, int64_t c, int k, int nz, const Quad &v) {
  if (AL) {
    __stcg(reinterpret_cast<ulonglong2 *>(m + c), make_ulonglong2(v.a, v.b));
    return;
  }
  float x[4];
  cells(v, x);
#pragma unroll
  for (int q = 0; q < 4; ++q)
    if (k + q < nz) __stcg(m + c + q, x[q]);
}

__device__ __forceinline__ uint32_t smem_addr(const void *p) {
  return (uint32_t)__cvta_generic_to_shared(p);
}
__device__ __forceinline__ Quad lds4(uint32_t a) {
  Quad v;
  asm volatile("ld.shared.v2.b64 {%0, %1}, [%2];" : "=l"(v.a), "=l"(v.b) : "r"(a) : "memory");
  return v;
}
__device__ __forceinline__ float lds1(uint32_t a) {
  float v;
  asm volatile("ld.shared.f32 %0, [%1];" : "=f"(v) : "r"(a) : "memory");
  return v;
}
__device__ __forceinline__ void sts4(uint32_t a, const Quad &v) {
  asm volatile("st.shared.v2.b64 [%0], {%1, %2};" ::"r"(a), "l"(v.a), "l"(v.b) : "memory");
}
// rhs with 1 in the cells that are not fluid (their result is masked; a
// quotient away from 0 keeps them off the division's slow path)
__device__ __forceinline__ Quad off_fluid_one(const Quad &v, uint32_t f) {
  float c[4];
  cells(v, c);
#pragma unroll
  for (int e = 0; e < 4; ++e) c[e] = f >> e & 1u ? c[e] : 1.0f;
  return quad(c);
}

// A grid barrier by the whole CTA; false after one that gave up, whose result is lost.
__device__ __forceinline__ bool round_barrier(const Args &a, unsigned int target) {
  __shared__ int s_ok;
  __syncthreads();
  if (threadIdx.x == 0) {
    s_ok = counter_barrier(reinterpret_cast<unsigned int *>(a.p_tmp), target);
    if (!s_ok) wait_gave_up(a.err);
  }
  __syncthreads();
  return s_ok != 0;
}

// Flags of a quad: bits 0-3 fluid cells; bits 4 + 4 d + q: cell q's neighbour
// in direction d (-i, +i, -j, +j, -k, +k) is solid; bits 28-31: columns to the
// window's edge, at most 2 T.  0: no fluid.
template <int T, int Q, bool RR, bool AL>
__global__ void __launch_bounds__(THREADS, 1) resident_sweeps_kernel(const Args a) {
  extern __shared__ __align__(16) unsigned char smem[];
  const int nx = a.nx, ny = a.ny, nz = a.nz;
  const int WI = a.bi + 2 * T, WJ = a.bj + 2 * T, KQ = (nz + 3) / 4;
  // window quads, a zero quad before it and after each column: the k
  // neighbours beyond the grid
  const int CP = KQ + 1, sj = CP, si = WJ * CP, nq = WI * si + 1;
  Quad *W = reinterpret_cast<Quad *>(smem) + 1;
  uint32_t *flag = reinterpret_cast<uint32_t *>(smem + (size_t)nq * 16);
  const int tid = threadIdx.x;
  const int gj = (ny + a.bj - 1) / a.bj;
  const int i0 = (int)(blockIdx.x / gj) * a.bi - T, j0 = (int)(blockIdx.x % gj) * a.bj - T;
  const int64_t plane = (int64_t)ny * nz;
  for (int q = tid; q < nq; q += THREADS) W[q - 1] = Quad{0, 0};
  // ---- the fluid quads of the window less its outermost columns, in one list:
  // first those of four fluid cells without a solid neighbour, then (from a
  // warp of their own) the rest, which alone need the select and the mask; each
  // part from the columns farthest from the window's edge to
  // the nearest (the quads of a later sweep of a round are a front of it).
  // The order within a bin does not matter.
  uint16_t *list = reinterpret_cast<uint16_t *>(flag + Q * THREADS);
  uint16_t *halo = list + Q * THREADS;  // fluid quads of the halo
  __shared__ int s_bin[16], s_count, s_halo;
  if (tid == 0) s_halo = 0;
  if (tid < 16) s_bin[tid] = 0;
  __syncthreads();
  auto bin_of = [](uint32_t f) {
    return 2 * T - (int)(f >> 28) + ((f & 0x0fffffffu) == 15u ? 0 : 2 * T);
  };
  const int RJ = WJ - 2, region = (WI - 2) * RJ * KQ;
  uint32_t idx[Q], fl[Q];
#pragma unroll
  for (int q = 0; q < Q; ++q) {
    const int pos = tid + q * THREADS;
    uint32_t f = 0;
    idx[q] = 0;
    if (pos < region) {
      const int col = pos / KQ, wk = pos - col * KQ, wi = col / RJ + 1, wj = col % RJ + 1;
      const int i = i0 + wi, j = j0 + wj, k = wk * 4;
      idx[q] = (uint32_t)(wi * si + wj * sj + wk);
      if ((unsigned)i < (unsigned)nx && (unsigned)j < (unsigned)ny) {
        const int64_t c = (int64_t)i * plane + (int64_t)j * nz + k;
        const uint32_t m = mask4<AL>(a.mask, c, k, nz);
        f = bits4(m, 7);
        if (f) {
          // solid neighbours only where a fluid byte counts some (bits 0-2)
          if (m & (((m >> 7) & 0x01010101u) * 7u)) {
            if (i > 0) f |= bits4(mask4<AL>(a.mask, c - plane, k, nz), 6) << 4;
            if (i + 1 < nx) f |= bits4(mask4<AL>(a.mask, c + plane, k, nz), 6) << 8;
            if (j > 0) f |= bits4(mask4<AL>(a.mask, c - nz, k, nz), 6) << 12;
            if (j + 1 < ny) f |= bits4(mask4<AL>(a.mask, c + nz, k, nz), 6) << 16;
            const uint32_t s = bits4(m, 6);
            uint32_t km = s << 1, kp = s >> 1;
            if (k > 0 && (__ldg(a.mask + c - 1) & BSP_MSOLID)) km |= 1u;
            if (k + 4 < nz && (__ldg(a.mask + c + 4) & BSP_MSOLID)) kp |= 8u;
            f |= (km & 15u) << 20 | kp << 24;
          }
          f |= (uint32_t)min(min(min(wi, WI - 1 - wi), min(wj, WJ - 1 - wj)), 2 * T) << 28;
          atomicAdd(&s_bin[bin_of(f)], 1);
        }
      }
    }
    fl[q] = f;
  }
  __syncthreads();
  if (tid == 0) {
    int run = 0;
    for (int b = 0; b < 4 * T; ++b) {
      if (b == 2 * T) {  // the second part starts with a warp of its own
        for (; run & 31; ++run) {
          list[run] = (uint16_t)(si + sj);
          flag[run] = 0;
        }
      }
      const int n = s_bin[b];
      s_bin[b] = run;
      run += n;
    }
    s_count = run;
  }
  __syncthreads();
#pragma unroll
  for (int q = 0; q < Q; ++q)
    if (fl[q]) {
      const int pos = atomicAdd(&s_bin[bin_of(fl[q])], 1);
      list[pos] = (uint16_t)idx[q];
      flag[pos] = fl[q];
    }
  __syncthreads();
  const int count = s_count;
  const bool work = count != 0;  // else: only the barriers
  auto gofs = [&](uint32_t x, int &k) {
    const int col = (int)x / CP, wk = (int)x - col * CP, wi = col / WJ, wj = col - wi * WJ;
    k = wk * 4;
    return (int64_t)(i0 + wi) * plane + (int64_t)(j0 + wj) * nz + k;
  };
  const uint32_t wbase = smem_addr(W);
  const uint64_t ONE2 = pack2(1.0f, 1.0f);
  Quad rhs[RR ? Q : 1];
#pragma unroll
  for (int q = 0; q < Q; ++q) {
    const int pos = tid + q * THREADS;
    idx[q] = wbase + (uint32_t)(si + sj) * 16u;  // any quad whose neighbours are in the window
    if (RR) rhs[q] = Quad{ONE2, ONE2};
    if (pos < count) {
      const uint32_t x = list[pos], f = flag[pos];
      idx[q] = wbase + x * 16u;
      if (RR && f) {
        int k;
        const int64_t o = gofs(x, k);
        rhs[q] = off_fluid_one(load4<AL>(a.rhs, o, k, nz), f);
      }
    } else {
      flag[pos] = 0;
    }
  }
  __syncthreads();
  const uint32_t si16 = (uint32_t)si * 16u, sj16 = (uint32_t)sj * 16u;
  if (work) {
    // the fluid quads of the halo columns: T rows of columns before and after the
    // tile along i, then T columns on either side along j
    const int top = T * WJ, nh = (2 * top + 2 * T * a.bi) * KQ;
    for (int h = tid; h < nh; h += THREADS) {
      const int col = h / KQ, wk = h - col * KQ;
      int wi, wj;
      if (col < 2 * top) {
        wi = col / WJ;
        wj = col - wi * WJ;
        if (wi >= T) wi += a.bi;
      } else {
        const int c2 = col - 2 * top;
        wi = c2 / (2 * T);
        wj = c2 - wi * 2 * T;
        wi += T;
        if (wj >= T) wj += a.bj;
      }
      const int i = i0 + wi, j = j0 + wj;
      if ((unsigned)i < (unsigned)nx && (unsigned)j < (unsigned)ny &&
          bits4(mask4<AL>(a.mask, (int64_t)i * plane + (int64_t)j * nz + wk * 4, wk * 4, nz), 7))
        halo[atomicAdd(&s_halo, 1)] = (uint16_t)(wi * si + wj * sj + wk);
    }
  }
  __syncthreads();
  const int nhalo = s_halo;
  // this thread's first HQ halo quads
  uint32_t hx[HQ];
  int64_t hg[HQ];
#pragma unroll
  for (int q = 0; q < HQ; ++q) {
    const int h = tid + q * THREADS;
    int k;
    hx[q] = h < nhalo ? halo[h] : 0u;
    hg[q] = h < nhalo ? gofs(hx[q], k) : -1;
  }
  // bits 2 q, 2 q + 1: the neighbouring lane holds the quad before / after
  // along k (of the same column, so it is active in the same sweeps)
  uint32_t adj = 0;
#pragma unroll
  for (int q = 0; q < Q; ++q) {
    const uint32_t f = flag[tid + q * THREADS];
    const uint32_t x = f ? idx[q] : 0u;
    const uint32_t xm = __shfl_up_sync(0xffffffffu, x, 1);
    const uint32_t xp = __shfl_down_sync(0xffffffffu, x, 1);
    if (x && (tid & 31) != 0 && xm + 16u == x) adj |= 1u << (2 * q);
    if (x && (tid & 31) != 31 && xp == x + 16u) adj |= 2u << (2 * q);
  }
  // the quads' own values; those of the halo are read from the window
  Quad cen[Q];
#pragma unroll
  for (int q = 0; q < Q; ++q) cen[q] = Quad{0, 0};
  const int base = a.n / a.rounds, more = a.n % a.rounds;
  for (int rd = 0; rd < a.rounds; ++rd) {
    const int ns = base + (rd < more ? 1 : 0);
    const bool last = rd == a.rounds - 1;
    // the last round ends in p
    float *out = ((a.rounds - 1 - rd) & 1) ? a.p_tmp : a.p;
    if (work) {
      for (int s = 1; s <= ns; ++s) {
        const uint32_t need = (uint32_t)(T - ns + s);  // columns this sweep is valid from
#pragma unroll
        for (int q = 0; q < Q; ++q) {
          if (q * THREADS >= count) break;
          const uint32_t f = flag[tid + q * THREADS];
          const bool on = (f >> 28) >= need;
          if (!__any_sync(0xffffffffu, on)) continue;
          const uint32_t x = idx[q];
          Quad rh;
          if (RR) {
            rh = rhs[q];
          } else {
            rh = Quad{ONE2, ONE2};
            if (on) {
              int k;
              const int64_t o = gofs((x - wbase) >> 4, k);
              rh = load4<AL>(a.rhs, o, k, nz);
            }
          }
          const Quad l = lds4(x - si16), r = lds4(x + si16), d = lds4(x - sj16),
                     u = lds4(x + sj16);
          if (on && (f >> 28) < (uint32_t)T) cen[q] = lds4(x);
          float cc[4], t[4];
          cells(cen[q], cc);
          // the k neighbours: from the neighbouring lanes where those hold the
          // quads beside (every lane takes part in the shuffles)
          float km = __shfl_up_sync(0xffffffffu, cc[3], 1);
          float kp = __shfl_down_sync(0xffffffffu, cc[0], 1);
          if (!(adj >> (2 * q) & 1u)) km = lds1(x - 4);
          if (!(adj >> (2 * q + 1) & 1u)) kp = lds1(x + 16);
          const bool simple = (f & 0x0fffffffu) == 15u || f == 0u;
          if (__all_sync(0xffffffffu, simple)) {
            cells(Quad{add2(add2(add2(l.a, r.a), d.a), u.a), add2(add2(add2(l.b, r.b), d.b), u.b)},
                  t);
            t[0] = __fadd_rn(__fadd_rn(t[0], km), cc[1]);
            t[1] = __fadd_rn(__fadd_rn(t[1], cc[0]), cc[2]);
            t[2] = __fadd_rn(__fadd_rn(t[2], cc[1]), cc[3]);
            t[3] = __fadd_rn(__fadd_rn(t[3], cc[2]), kp);
            if (on) cen[q] = div6_quad(quad(t), rh);
          } else {
            // a solid neighbour's value is the cell's own (W is +0 off fluid)
            float v[6][4];
            cells(l, v[0]);
            cells(r, v[1]);
            cells(d, v[2]);
            cells(u, v[3]);
#pragma unroll
            for (int e = 0; e < 4; ++e) {
              v[4][e] = e == 0 ? km : cc[e > 0 ? e - 1 : 0];
              v[5][e] = e == 3 ? kp : cc[e < 3 ? e + 1 : 3];
#pragma unroll
              for (int dir = 0; dir < 6; ++dir)
                if (f >> (4 + 4 * dir + e) & 1u) v[dir][e] = cc[e];
              t[e] = __fadd_rn(__fadd_rn(__fadd_rn(__fadd_rn(__fadd_rn(v[0][e], v[1][e]), v[2][e]),
                                                   v[3][e]), v[4][e]), v[5][e]);
            }
            if (!RR) rh = off_fluid_one(rh, f);
            float y[4];
            cells(div6_quad(quad(t), rh), y);
#pragma unroll
            for (int e = 0; e < 4; ++e) y[e] = f >> e & 1u ? y[e] : 0.0f;
            if (on) cen[q] = quad(y);
          }
        }
        __syncthreads();
        const bool end = s == ns;
#pragma unroll
        for (int q = 0; q < Q; ++q) {
          if (q * THREADS >= count) break;
          const uint32_t f = flag[tid + q * THREADS];
          if ((f >> 28) < need) continue;
          sts4(idx[q], cen[q]);
          // the band along the tile's edge (T .. 2 T - 1 columns from the
          // window's), in the end the whole tile
          if (end && (last || (f >> 28) < 2u * T)) {
            int k;
            const int64_t g = gofs((idx[q] - wbase) >> 4, k);
            if (last || g != 0) store4<AL>(out, g, k, nz, cen[q]);  // 0: the barrier's word
          }
        }
        if (!end) __syncthreads();
      }
    }
    if (last) return;
    if (!round_barrier(a, (unsigned int)(rd + 1) * gridDim.x + a.extra)) return;
    if (work) {
      Quad hv[HQ];
#pragma unroll
      for (int q = 0; q < HQ; ++q)
        if (hg[q] >= 0) hv[q] = load4<AL>(out, hg[q], ((int)hx[q] % CP) * 4, nz);
      for (int h = tid + HQ * THREADS; h < nhalo; h += THREADS) {
        const uint32_t x = halo[h];
        int k;
        const int64_t g = gofs(x, k);
        sts4(wbase + x * 16u, load4<AL>(out, g, k, nz));
      }
#pragma unroll
      for (int q = 0; q < HQ; ++q)
        if (hg[q] >= 0) sts4(wbase + hx[q] * 16u, hv[q]);
      __syncthreads();
    }
  }
}

struct Plan {
  int T, Q, bi, bj, grid;
  size_t smem;
  double cost;
};

inline size_t smem_of(int T, int Q, int bi, int bj, int kq) {
  return ((size_t)(bi + 2 * T) * (bj + 2 * T) * (kq + 1) + 1) * 16 + (size_t)Q * THREADS * 6 +
         ((size_t)(bi + 2 * T) * (bj + 2 * T) - (size_t)bi * bj) * kq * 2;
}

// The tile and T of least estimated time per sweep, or grid = 0 when no tile
// fits (the grid is too large to be resident).
Plan make_plan(int nx, int ny, int nz, int sms, bool al) {
  const int kq = (nz + 3) / 4;
  Plan best{};
  best.cost = 1e30;
  for (int bi = 1; bi <= nx; ++bi) {
    const int gi = (nx + bi - 1) / bi;
    if (gi > sms) continue;
    const int bj0 = std::max(1, (ny + sms / gi - 1) / (sms / gi));
    for (int T = 1; T <= 4; ++T) {
      // bands reach one neighbour only, and the grid's first column none: a tile is wider
      // than a halo, or as wide as the grid
      const int bj = std::max(bj0, std::min(ny, T + 1));
      if (bi < T || bj < T || (bi == T && gi > 1)) continue;
      if (bi > 3 * bj || bj > 3 * bi) continue;
      const int64_t region = (int64_t)(bi + 2 * T - 2) * (bj + 2 * T - 2) * kq;
      const int q = (int)((region + 31 + THREADS - 1) / THREADS);
      const int Q = q <= 2 ? 2 : (q <= 4 ? 4 : (q <= 8 ? 8 : (q <= 16 ? 16 : 0)));
      // 16 quads a thread (rhs from L2 each sweep) only beats the point kernel
      // where that loads single cells (150x146x99: 10.4 against 16.9 us a sweep)
      if (!Q || (Q == 16 && al)) continue;
      const size_t sm = smem_of(T, Q, bi, bj, kq);
      if (sm > (size_t)SMEM_MAX) continue;
      // cycles, fitted to measured rounds: barrier, band and halo latency, halo
      // quads; per sweep two CTA barriers and the quads (half of them fluid)
      const double halo = (double)((bi + 2 * T) * (bj + 2 * T) - bi * bj) * kq / THREADS;
      double c = 3600 + halo * 150;
      for (int s = 1; s <= T; ++s) {
        const double quads = (double)(bi + 2 * T - 2 * s) * (bj + 2 * T - 2 * s) * kq;
        c += 600 + quads / THREADS * (Q == 16 ? 1700 : 900);
      }
      c /= T;
      if (c < best.cost) best = Plan{T, Q, bi, bj, gi * ((ny + bj - 1) / bj), sm, c};
    }
  }
  return best;
}

template <int T, int Q, bool RR>
cudaError_t launch(const Args &a, const Plan &p, bool al, cudaStream_t s) {
  const void *fn = al ? (const void *)resident_sweeps_kernel<T, Q, RR, true>
                      : (const void *)resident_sweeps_kernel<T, Q, RR, false>;
  if (!smem_opt_in(fn, SMEM_MAX)) return cudaErrorNotSupported;
  void *args[] = {const_cast<Args *>(&a)};
  return launch_coop(fn, dim3((unsigned)p.grid), dim3(THREADS), args, p.smem, s);
}

}  // namespace swr

// n sweeps from p = p_tmp = 0 with the result in p (p_tmp's first element is then a
// count).  False when the grid is too large to stay resident or the launch is refused:
// nothing runs then.
bool sweeps_resident(float *p, float *p_tmp, const float *rhs, const uint8_t *mask, int nx, int ny,
                     int nz, int n, cudaStream_t s, cudaError_t *e) {
  using namespace swr;
  if (!g_one_launch || n < MIN_SWEEPS || (int64_t)nx * ny * nz > (8LL << 20)) return false;
  const bool al = nz % 4 == 0 &&
                  (((uintptr_t)p | (uintptr_t)p_tmp | (uintptr_t)rhs) & 15u) == 0 &&
                  ((uintptr_t)mask & 3u) == 0;
  const Plan pl = make_plan(nx, ny, nz, num_sms(), al);
  if (!pl.grid) return false;
  const int rounds = (n + pl.T - 1) / pl.T;
  if ((int64_t)rounds * pl.grid + 1 >= COUNTER_LIMIT) return false;
  int *err = wait_word(WAIT_SWEEPS);
  if (!err) return false;
  Args a{p, p_tmp, rhs, mask, err, nx, ny, nz, pl.bi, pl.bj, 0, n, rounds};
  if (g_test_wait_error == 1) {
    a.extra = 1;
    g_test_wait_error = 0;
  }
  ProfScope ps(PROF_SWEEP, s);
#define R(T_, Q_, RR_) \
  if (pl.T == T_ && pl.Q == Q_) return *e = launch<T_, Q_, RR_>(a, pl, al, s), !coop_refused(*e)
  R(1, 2, true);
  R(1, 4, true);
  R(1, 8, true);
  R(1, 16, false);
  R(2, 2, true);
  R(2, 4, true);
  R(2, 8, true);
  R(2, 16, false);
  R(3, 2, true);
  R(3, 4, true);
  R(3, 8, true);
  R(3, 16, false);
  R(4, 2, true);
  R(4, 4, true);
  R(4, 8, true);
  R(4, 16, false);
#undef R
  return false;
}

}  // namespace bsp

