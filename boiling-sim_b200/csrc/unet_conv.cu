// unet_conv.cu -- the 3x3x3 convolutions of the warm-start network's training
// pass on the unpadded layout act[v][c], v = (i ny + j) nz + k, channels
// innermost (BF16), weights w[tap][co][ci] (tap = (di+1) 9 + (dj+1) 3 + (dk+1)):
// forward (and data gradient, the same kernel on flipped weights), weight and
// bias gradient.
//
// All three are mma.sync m16n8k16 (BF16 operands, FP32 accumulators).  The
// forward pass keeps one accumulation order per output -- taps ascending,
// 16-channel chunks ascending inside a tap -- because the ReLU gradient takes
// its mask from the sign of the rounded output: another order flips an output
// near zero once in a few million, and with it a term of the gradients.
// The data gradient, the same kernel, has no mask taken from it and could be summed in
// another order.  With both on tcgen05 (27 taps by moved descriptors; then the three di
// stacked along N) a layer's training pass of 32 -> 32 channels at 64x64x48 took 169 and 125 us,
// 154 us here; 16 -> 16 at 128x128x96 took 473 us with the first, 293 here.
//
// Forward.  A tile is 8 k x 16 j voxels; a CTA marches along i with the tile's
// input window (10 x 18 rows of all input channels) of each plane staged once by
// cp.async, zero-filled outside the grid.  A plane adds to three output planes
// (through di = +1, 0, -1), whose accumulators a warp keeps in registers, so an
// operand row read from shared memory feeds three taps, and a plane is read
// from L2 1.4 times; gathering the rows per tap read every voxel 27 times.
// Weights of the CTA's output channels stay in shared memory.
//
// Weight gradient.  dw[tap][co][ci] = sum_v g[v][co] in[v + d][ci]: the
// contraction runs over voxels, and M x N is a block of 16 or 32 channels a
// side (a fixed 64 x 64 tile did 4 to 16 times the work of these layers).  The
// nine warps of a CTA take the nine (dj, dk) taps; it marches along i with input
// and gradient planes in rings, all three di from the same staged planes.
// Chains of MMA accumulation are cut every 2048 voxels.  The bias gradient is
// summed from the staged gradient planes.  Partial sums per split are added
// in a fixed order (deterministic).
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include <algorithm>
#include <type_traits>

#include "bsp_common.cuh"

namespace bsp {
namespace uconv {

constexpr int TK = 8, TJ = 16;                 // voxels of a tile: 8 k x 16 j
constexpr int WK = TK + 2, WJ = TJ + 2;        // its input window
constexpr int WROWS = WK * WJ;                 // 180 rows
constexpr int HALF = WROWS * 16;               // bytes of one 8-channel group of a plane
constexpr int SMEM_MAX = 232448;

__device__ __forceinline__ uint32_t smem_u32(const void *p) {
  return (uint32_t)__cvta_generic_to_shared(p);
}
__device__ __forceinline__ void cp16(uint32_t dst, const void *src, bool valid) {
  // src-size 0 zero-fills the 16 destination bytes
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src),
               "r"(valid ? 16 : 0)
               : "memory");
}
__device__ __forceinline__ void cp_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_wait() {
  asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}
__device__ __forceinline__ void ldsm_x4(uint32_t &r0, uint32_t &r1, uint32_t &r2, uint32_t &r3,
                                        uint32_t addr) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];"
               : "=r"(r0), "=r"(r1), "=r"(r2), "=r"(r3)
               : "r"(addr)
               : "memory");
}
__device__ __forceinline__ void ldsm_x4_t(uint32_t &r0, uint32_t &r1, uint32_t &r2, uint32_t &r3,
                                          uint32_t addr) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];"
               : "=r"(r0), "=r"(r1), "=r"(r2), "=r"(r3)
               : "r"(addr)
               : "memory");
}
__device__ __forceinline__ void mma_bf16(float (&d)[4], const uint32_t (&a)[4], uint32_t b0,
                                         uint32_t b1) {
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, "
      "{%8,%9}, {%0,%1,%2,%3};"
      : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

struct FwdArgs {
  __nv_bfloat16 *out;
  const __nv_bfloat16 *in, *w;
  const float *bias;
  int nx, ny, nz, cout, relu;
  int nct;     // output-channel tiles
  int jt, kt;  // tiles per plane
  int len;     // output planes per CTA
};

// CIN input channels, NT output channels per CTA, MT 16-row blocks per warp
// (8 / MT warps of 16 MT voxels each), NS plane slots.
template <int CIN, int NT, int MT, int NS>
struct FwdShape {
  static constexpr int WARPS = 8 / MT, THREADS = WARPS * 32;
  static constexpr int PITCH = CIN * 2 + 16;  // bytes of a staged row
  static constexpr int W_BYTES = 27 * NT * PITCH, SLOT = WROWS * PITCH;
  static constexpr int SMEM = W_BYTES + NS * SLOT;
};

template <int CIN, int NT, int MT, int NS>
__global__ void __launch_bounds__(FwdShape<CIN, NT, MT, NS>::THREADS)
    conv_fwd_kernel(const FwdArgs a) {
  using S = FwdShape<CIN, NT, MT, NS>;
  extern __shared__ __align__(128) unsigned char smem[];
  constexpr int PITCH = S::PITCH, CG = CIN / 8, NK = CIN / 16, NG = NT / 16;
  constexpr int XQ = (WROWS * CG + S::THREADS - 1) / S::THREADS;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  int t = blockIdx.x;
  const int co0 = (t % a.nct) * NT;
  t /= a.nct;
  const int k0 = (t % a.kt) * TK;
  t /= a.kt;
  const int j0 = (t % a.jt) * TJ;
  const int i0 = (t / a.jt) * a.len;
  const int len = min(a.len, a.nx - i0);
  const uint32_t wsm = smem_u32(smem), slots = wsm + S::W_BYTES;
  // weights: [tap][n] rows of CIN channels
  for (int q = tid; q < 27 * NT * CG; q += S::THREADS) {
    const int row = q / CG, g8 = q % CG;
    const int tap = row / NT, n = row % NT;
    cp16(wsm + (uint32_t)(row * PITCH + g8 * 16),
         a.w + ((int64_t)tap * a.cout + co0 + n) * CIN + g8 * 8, true);
  }
  // this thread's pieces of an input window
  int xoff[XQ];
  uint32_t xok = 0;
#pragma unroll
  for (int q = 0; q < XQ; ++q) {
    const int p = tid + q * S::THREADS, row = p / CG;
    const int j = j0 - 1 + row / WK, k = k0 - 1 + row % WK;
    xoff[q] = (j * a.nz + k) * CIN + (p % CG) * 8;
    if (row < WROWS && (unsigned)j < (unsigned)a.ny && (unsigned)k < (unsigned)a.nz)
      xok |= 1u << q;
  }
  static_assert(XQ <= 32 && S::THREADS % CG == 0, "piece layout");
  const uint32_t xdst = (uint32_t)((tid / CG) * PITCH + (tid % CG) * 16);
  const int64_t plane = (int64_t)a.ny * a.nz * CIN;
  auto stage = [&](int pl, int s) {
    const int i = i0 - 1 + pl;
    const bool iok = (unsigned)i < (unsigned)a.nx;
    const __nv_bfloat16 *src = a.in + (iok ? i * plane : 0);
#pragma unroll
    for (int q = 0; q < XQ; ++q) {
      const bool v = iok && (xok >> q & 1);
      if (XQ * S::THREADS == WROWS * CG || tid + q * S::THREADS < WROWS * CG)
        cp16(slots + (uint32_t)(s * S::SLOT) + xdst +
                 (uint32_t)(q * (S::THREADS / CG) * PITCH),
             v ? src + xoff[q] : a.in, v);
    }
  };
  // operand addresses of this lane
  const int r = warp * 16 * MT + (lane & 15);  // voxel row of the first block
  const uint32_t xa = (uint32_t)(((r >> 3) * WK + (r & 7)) * PITCH + (lane >> 4) * 16);
  const uint32_t wa = wsm + (uint32_t)(((lane >> 4) * 8 + (lane & 7)) * PITCH +
                                       ((lane >> 3) & 1) * 16);
  // accumulators of outputs pl - 2, pl - 1, pl (through di = +1, 0, -1)
  float acc[3][MT][2 * NG][4];
#pragma unroll
  for (int d = 0; d < 3; ++d)
#pragma unroll
    for (int m = 0; m < MT; ++m)
#pragma unroll
      for (int n = 0; n < 2 * NG; ++n)
#pragma unroll
        for (int q = 0; q < 4; ++q) acc[d][m][n][q] = 0.0f;
#pragma unroll
  for (int s = 0; s < NS - 1; ++s) {
    if (s < len + 2) stage(s, s);
    cp_commit();
  }
  int slot = 0;
  for (int pl = 0; pl < len + 2; ++pl) {
    cp_wait<NS - 2>();
    __syncthreads();  // plane pl staged by every thread; plane pl - 1 no longer read
    if (pl + NS - 1 < len + 2) stage(pl + NS - 1, slot == 0 ? NS - 1 : slot - 1);
    cp_commit();
    const uint32_t xs = slots + (uint32_t)(slot * S::SLOT) + xa;
    const bool use[3] = {pl >= 2, pl >= 1 && pl <= len, pl < len};
#pragma unroll 1
    for (int dj = 0; dj < 3; ++dj) {
#pragma unroll
      for (int dk = 0; dk < 3; ++dk) {
#pragma unroll
        for (int kc = 0; kc < NK; ++kc) {
          uint32_t A[MT][4];
#pragma unroll
          for (int m = 0; m < MT; ++m)
            ldsm_x4(A[m][0], A[m][1], A[m][2], A[m][3],
                    xs + (uint32_t)((dj + 2 * m) * WK * PITCH + dk * PITCH + kc * 32));
#pragma unroll
          for (int d = 0; d < 3; ++d) {
            if (!use[d]) continue;
            const uint32_t wt = wa + (uint32_t)((((2 - d) * 9 + dk) * NT) * PITCH + kc * 32) +
                                (uint32_t)(dj * 3 * NT * PITCH);
#pragma unroll
            for (int n = 0; n < NG; ++n) {
              uint32_t b0, b1, b2, b3;
              ldsm_x4(b0, b1, b2, b3, wt + (uint32_t)(n * 16 * PITCH));
#pragma unroll
              for (int m = 0; m < MT; ++m) {
                mma_bf16(acc[d][m][2 * n], A[m], b0, b1);
                mma_bf16(acc[d][m][2 * n + 1], A[m], b2, b3);
              }
            }
          }
        }
      }
    }
    if (pl >= 2) {  // output pl - 2 is complete
      const int g = lane >> 2, t4 = lane & 3;
#pragma unroll
      for (int m = 0; m < MT; ++m)
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const int row = warp * 16 * MT + m * 16 + g + h * 8;
          const int j = j0 + (row >> 3), k = k0 + (row & 7);
          if (j >= a.ny || k >= a.nz) continue;
          const int64_t v = ((int64_t)(i0 + pl - 2) * a.ny + j) * a.nz + k;
#pragma unroll
          for (int n = 0; n < 2 * NG; ++n) {
            const int co = co0 + n * 8 + t4 * 2;
            float x0 = acc[0][m][n][2 * h], x1 = acc[0][m][n][2 * h + 1];
            if (a.bias) {
              x0 += a.bias[co];
              x1 += a.bias[co + 1];
            }
            if (a.relu) {
              x0 = fmaxf(x0, 0.0f);
              x1 = fmaxf(x1, 0.0f);
            }
            *reinterpret_cast<__nv_bfloat162 *>(a.out + v * a.cout + co) =
                __floats2bfloat162_rn(x0, x1);
          }
        }
    }
#pragma unroll
    for (int m = 0; m < MT; ++m)
#pragma unroll
      for (int n = 0; n < 2 * NG; ++n)
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          acc[0][m][n][q] = acc[1][m][n][q];
          acc[1][m][n][q] = acc[2][m][n][q];
          acc[2][m][n][q] = 0.0f;
        }
    slot = slot + 1 == NS ? 0 : slot + 1;
  }
}

// Any channel counts (multiples of 16): one tap and 16 channels per step,
// rows gathered per tap.  Serves the input-channel counts that have no staged
// kernel above (no layer of the network).  Its loads from shared memory are not fences to the
// compiler (the CTA barriers are), and a step's B rows come eight at a time: with fences and
// sixteen, 48 -> 48 channels at 32x32x24 took 69 us instead of 58.
constexpr int GM = 128, GROW = 48;  // voxels per CTA; bytes of a staged row
__device__ __forceinline__ void lds_x4(uint32_t (&r)[4], uint32_t addr) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
               : "r"(addr));
}
__device__ __forceinline__ void lds_x2(uint32_t &r0, uint32_t &r1, uint32_t addr) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x2.shared.b16 {%0,%1}, [%2];"
               : "=r"(r0), "=r"(r1)
               : "r"(addr));
}
template <int NT>
__global__ void __launch_bounds__(GM) conv_any_kernel(__nv_bfloat16 *__restrict__ out,
                                                      const __nv_bfloat16 *__restrict__ in,
                                                      const __nv_bfloat16 *__restrict__ w,
                                                      const float *__restrict__ bias, int nx,
                                                      int ny, int nz, int cin, int cout,
                                                      int relu) {
  __shared__ __align__(128) unsigned char sA[2][GM * GROW];
  __shared__ __align__(128) unsigned char sB[2][NT * GROW];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int64_t nvox = (int64_t)nx * ny * nz;
  const int64_t v0 = (int64_t)blockIdx.x * GM;
  const int co0 = blockIdx.y * NT;
  // this thread stages rows tid (A: one 32-byte row = 2 x 16 B per thread)
  const int64_t va = v0 + tid;
  const bool vin = va < nvox;
  int ia = 0, ja = 0, ka = 0;
  if (vin) {
    ka = (int)(va % nz);
    const int64_t rj = va / nz;
    ja = (int)(rj % ny);
    ia = (int)(rj / ny);
  }
  const int nchunk = cin >> 4;
  const int ksteps = 27 * nchunk;
  auto stage = [&](int s, int buf) {
    const int tap = s / nchunk, c0 = (s - tap * nchunk) << 4;
    const int di = tap / 9 - 1, dj = (tap / 3) % 3 - 1, dk = tap % 3 - 1;
    const int ii = ia + di, jj = ja + dj, kk = ka + dk;
    const bool ok = vin && ii >= 0 && ii < nx && jj >= 0 && jj < ny && kk >= 0 && kk < nz;
    const __nv_bfloat16 *src = ok ? in + (((int64_t)ii * ny + jj) * nz + kk) * cin + c0 : in;
    const uint32_t dst = smem_u32(sA[buf] + tid * GROW);
    cp16(dst, src, ok);
    cp16(dst + 16, ok ? src + 8 : src, ok);
    // weights: NT rows of 32 bytes
    for (int r = tid; r < NT * 2; r += GM) {
      const int row = r >> 1, half = r & 1;
      const __nv_bfloat16 *ws = w + ((int64_t)tap * cout + co0 + row) * cin + c0 + half * 8;
      cp16(smem_u32(sB[buf] + row * GROW + half * 16), ws, true);
    }
    cp_commit();
  };
  float acc[2][NT / 8][4];
#pragma unroll
  for (int m = 0; m < 2; ++m)
#pragma unroll
    for (int n = 0; n < NT / 8; ++n)
#pragma unroll
      for (int q = 0; q < 4; ++q) acc[m][n][q] = 0.0f;
  stage(0, 0);
  for (int s = 0; s < ksteps; ++s) {
    const int buf = s & 1;
    if (s + 1 < ksteps) {
      stage(s + 1, buf ^ 1);
      cp_wait<1>();
    } else {
      cp_wait<0>();
    }
    __syncthreads();
    uint32_t A[2][4];
#pragma unroll
    for (int m = 0; m < 2; ++m) {
      const int row = warp * 32 + m * 16 + (lane & 15);
      lds_x4(A[m], smem_u32(sA[buf] + row * GROW + (lane >> 4) * 16));
    }
#pragma unroll
    for (int n = 0; n < NT / 8; ++n) {
      uint32_t b0, b1;
      // rows n*8 + (lane & 7), k half (lane >> 3) & 1
      lds_x2(b0, b1, smem_u32(sB[buf] + (n * 8 + (lane & 7)) * GROW + ((lane >> 3) & 1) * 16));
#pragma unroll
      for (int m = 0; m < 2; ++m) mma_bf16(acc[m][n], A[m], b0, b1);
    }
    __syncthreads();
  }
  // epilogue: rows g and g + 8 of each m16 tile, columns 2t, 2t+1 of each n8 tile
  const int g = lane >> 2, t4 = lane & 3;
#pragma unroll
  for (int m = 0; m < 2; ++m)
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int64_t v = v0 + warp * 32 + m * 16 + g + h * 8;
      if (v >= nvox) continue;
#pragma unroll
      for (int n = 0; n < NT / 8; ++n) {
        const int co = co0 + n * 8 + t4 * 2;
        float x0 = acc[m][n][2 * h], x1 = acc[m][n][2 * h + 1];
        if (bias) {
          x0 += bias[co];
          x1 += bias[co + 1];
        }
        if (relu) {
          x0 = fmaxf(x0, 0.0f);
          x1 = fmaxf(x1, 0.0f);
        }
        *reinterpret_cast<__nv_bfloat162 *>(out + v * cout + co) = __floats2bfloat162_rn(x0, x1);
      }
    }
}

template <int CIN, int NT, int MT, int NS>
cudaError_t launch_fwd(FwdArgs a, cudaStream_t s) {
  using S = FwdShape<CIN, NT, MT, NS>;
  static_assert(S::SMEM <= SMEM_MAX, "shared memory");
  auto kern = conv_fwd_kernel<CIN, NT, MT, NS>;
  if (!smem_opt_in((const void *)kern, S::SMEM)) return cudaErrorNotSupported;
  a.nct = a.cout / NT;
  a.jt = (a.ny + TJ - 1) / TJ;
  a.kt = (a.nz + TK - 1) / TK;
  // Planes per CTA: waves x (planes + the two halo planes, which cost a third
  // of the MMAs each, + about two planes' time for loading the weights) least.
  const int occ = std::max(1, std::min(SMEM_MAX / (S::SMEM + 1024), MT == 2 ? 3 : 1));
  const int64_t cols = (int64_t)a.jt * a.kt * a.nct, slots = 148 * occ;
  int64_t best = INT64_MAX;
  for (int l = 1; l <= a.nx; ++l) {
    const int64_t items = cols * ((a.nx + l - 1) / l);
    const int64_t cost = ((items + slots - 1) / slots) * (l + 3);
    if (cost <= best) {
      best = cost;
      a.len = l;
    }
  }
  const int64_t items = cols * ((a.nx + a.len - 1) / a.len);
  if (items > 0x7fffffff) return cudaErrorInvalidValue;
  kern<<<(unsigned)items, S::THREADS, S::SMEM, s>>>(a);
  return cudaGetLastError();
}

// ---- weight and bias gradient -------------------------------------------------------------
constexpr int WG_VCH = 2048;      // voxels per partial-sum slot of the workspace
constexpr int WG_THREADS = 288;   // nine warps, one (dj, dk) tap each
constexpr int WG_FLUSH = 16;      // tiles (2048 voxels) per MMA accumulation chain

// Row pitches of C channels: C * 2 + 16 bytes put eight consecutive rows on
// distinct banks for ldmatrix (48 and 80 bytes).  ND: the di a CTA computes,
// all three (planes in a ring of 5 slots) or one.
template <int MC, int NC, int ND>
struct WgShape {
  static constexpr int GP = MC * 2 + 16, XP = NC * 2 + 16;
  static constexpr int GB = TK * TJ * GP, XB = WROWS * XP;
  static constexpr int GS = 3, XS = 2 + ND;  // slots: two steps ahead
  static constexpr int SMEM = GS * GB + XS * XB + 64;
};

struct WgArgs {
  float *dst;    // splits == 1: dw; else split s's [27][cout][cin] at s * 27 cout cin
  float *dbdst;  // NULL, or [split][cout] (splits == 1: db)
  const __nv_bfloat16 *g, *in;
  int nx, ny, nz, cin, cout;
  int jt, kt, nbi;  // tiles per plane, input-channel blocks
  int64_t tiles;    // (j, k) tiles x planes, plane index fastest
};

template <int MC, int NC, int ND>
__global__ void __launch_bounds__(WG_THREADS) conv_wgrad_kernel(const WgArgs a) {
  using S = WgShape<MC, NC, ND>;
  extern __shared__ __align__(128) unsigned char smem[];
  constexpr int GP = S::GP, XP = S::XP, GS = S::GS, XS = S::XS;
  constexpr int GC = MC / 8, XC = NC / 8;  // 16-byte pieces per row
  constexpr int GQ = (TK * TJ * GC + WG_THREADS - 1) / WG_THREADS;  // pieces per thread
  constexpr int XQ = (WROWS * XC + WG_THREADS - 1) / WG_THREADS;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  // grid.y: channel block, and the di with ND = 1
  const int blk = ND == 3 ? (int)blockIdx.y : (int)blockIdx.y / 3;
  const int di0 = ND == 3 ? -1 : (int)blockIdx.y % 3 - 1;  // first di
  const int co0 = (blk / a.nbi) * MC, ci0 = (blk % a.nbi) * NC;
  const int dj = warp / 3, dk = warp % 3;  // + 1
  int64_t t = a.tiles * blockIdx.x / gridDim.x;
  const int64_t t1 = a.tiles * (blockIdx.x + 1) / gridDim.x;
  const uint32_t gbase = smem_u32(smem), xbase = gbase + GS * S::GB, zrow = xbase + XS * S::XB;
  if (tid < 4)
    *reinterpret_cast<uint4 *>(smem + GS * S::GB + XS * S::XB + tid * 16) = make_uint4(0, 0, 0, 0);
  static_assert(WG_THREADS % GC == 0 && WG_THREADS % XC == 0, "pieces of a thread share a column");
  const uint32_t gdst = gbase + (uint32_t)((tid / GC) * GP + (tid % GC) * 16);
  const uint32_t xdst = xbase + (uint32_t)((tid / XC) * XP + (tid % XC) * 16);
  float acc[ND][MC / 16][NC / 8][4];
  auto clear = [&]() {
#pragma unroll
    for (int d = 0; d < ND; ++d)
#pragma unroll
      for (int m = 0; m < MC / 16; ++m)
#pragma unroll
        for (int n = 0; n < NC / 8; ++n)
#pragma unroll
          for (int q = 0; q < 4; ++q) acc[d][m][n][q] = 0.0f;
  };
  // adds the accumulators to this split's sums (each element belongs to one
  // thread of one CTA)
  bool stored = false;
  auto flush = [&]() {
    const int g4 = lane >> 2, t4 = lane & 3;
#pragma unroll
    for (int d = 0; d < ND; ++d) {
      float *dst = a.dst + ((int64_t)blockIdx.x * 27 + (di0 + d + 1) * 9 + warp) * a.cout * a.cin;
#pragma unroll
      for (int m = 0; m < MC / 16; ++m)
#pragma unroll
        for (int n = 0; n < NC / 8; ++n)
#pragma unroll
          for (int h = 0; h < 2; ++h) {
            const int co = co0 + m * 16 + g4 + h * 8, ci = ci0 + n * 8 + t4 * 2;
            float *p = dst + (int64_t)co * a.cin + ci;
            const float v0 = stored ? p[0] : 0.0f, v1 = stored ? p[1] : 0.0f;
            p[0] = v0 + acc[d][m][n][2 * h];
            p[1] = v1 + acc[d][m][n][2 * h + 1];
          }
    }
    stored = true;
    clear();
  };
  clear();
  const bool bias = a.dbdst != nullptr && (ND == 3 || di0 == 0) && ci0 == 0;
  constexpr int BG = WG_THREADS / MC;  // row groups of the bias sums
  float bsum = 0.0f;
  const int mat = lane >> 3, r = lane & 7;
  const uint32_t ga = gbase + (uint32_t)(((mat >> 1) * 8 + r) * GP + (mat & 1) * 16);
  const uint32_t xa =
      xbase + (uint32_t)((((mat & 1) + dj) * WK + r + dk) * XP + (mat >> 1) * 16);
  int chain = 0;
  // runs of planes ia .. ib - 1 of one (j, k) tile
  while (t < t1) {
    const int col = (int)(t / a.nx), ia = (int)(t - (int64_t)col * a.nx);
    const int ib = (int)(t1 - t < a.nx - ia ? ia + (t1 - t) : a.nx);
    t += ib - ia;
    const int k0 = col % a.kt * TK, j0 = col / a.kt * TJ;
    // this thread's pieces of the tile's planes
    int64_t goff[GQ], xoff[XQ];
    uint32_t ok = 0;
#pragma unroll
    for (int q = 0; q < GQ; ++q) {
      const int row = (tid + q * WG_THREADS) / GC, j = j0 + row / TK, k = k0 + row % TK;
      goff[q] = ((int64_t)j * a.nz + k) * a.cout + co0 + ((tid + q * WG_THREADS) % GC) * 8;
      if (row < TK * TJ && j < a.ny && k < a.nz) ok |= 1u << q;
    }
#pragma unroll
    for (int q = 0; q < XQ; ++q) {
      const int row = (tid + q * WG_THREADS) / XC, j = j0 - 1 + row / WK, k = k0 - 1 + row % WK;
      xoff[q] = ((int64_t)j * a.nz + k) * a.cin + ci0 + ((tid + q * WG_THREADS) % XC) * 8;
      if (row < WROWS && (unsigned)j < (unsigned)a.ny && (unsigned)k < (unsigned)a.nz)
        ok |= 1u << (8 + q);
    }
    const int64_t gplane = (int64_t)a.ny * a.nz * a.cout, xplane = (int64_t)a.ny * a.nz * a.cin;
    // step q stages input plane ia + di0 + q and gradient plane ia + q - (ND - 1),
    // and computes that gradient plane on input planes of steps q - (ND - 1) .. q
    const int nstep = ib - ia + ND - 1;
    auto stage = [&](int q, int xs, int gs) {
      const int i = ia + di0 + q;
      const bool iok = (unsigned)i < (unsigned)a.nx;
      const __nv_bfloat16 *x0 = a.in + (iok ? i * xplane : 0);
#pragma unroll
      for (int p = 0; p < XQ; ++p) {
        const bool v = iok && (ok >> (8 + p) & 1);
        if (XQ * WG_THREADS == WROWS * XC || tid + p * WG_THREADS < WROWS * XC)
          cp16(xdst + (uint32_t)(xs * S::XB + p * (WG_THREADS / XC) * XP), v ? x0 + xoff[p] : a.in,
               v);
      }
      if (q < ND - 1) return;
      const __nv_bfloat16 *g0 = a.g + (ia + q - (ND - 1)) * gplane;
#pragma unroll
      for (int p = 0; p < GQ; ++p) {
        const bool v = ok >> p & 1;
        if (GQ * WG_THREADS == TK * TJ * GC || tid + p * WG_THREADS < TK * TJ * GC)
          cp16(gdst + (uint32_t)(gs * S::GB + p * (WG_THREADS / GC) * GP), v ? g0 + goff[p] : a.g,
               v);
      }
    };
    const bool part = j0 + TJ > a.ny || k0 + TK > a.nz;
    const bool kok = k0 + r < a.nz;
    __syncthreads();  // the run before no longer reads its slots
    stage(0, 0, 0);
    cp_commit();
    if (1 < nstep) stage(1, 1, 1);
    cp_commit();
    int xs = 0, gs = 0;
    for (int q = 0; q < nstep; ++q) {
      cp_wait<1>();
      __syncthreads();  // step q staged by every thread; step q - 1 no longer reads
      const int xn = xs + 2 >= XS ? xs + 2 - XS : xs + 2, gn = gs + 2 >= GS ? gs + 2 - GS : gs + 2;
      if (q + 2 < nstep) stage(q + 2, xn, gn);
      cp_commit();
      if (q >= ND - 1) {
        const uint32_t gb = ga + (uint32_t)(gs * S::GB);
        uint32_t xb[ND];
#pragma unroll
        for (int d = 0; d < ND; ++d) {
          const int sl = xs - (ND - 1) + d;
          xb[d] = xa + (uint32_t)((sl < 0 ? sl + XS : sl) * S::XB);
        }
        // Voxels past the grid's end read a zero input row, so that their
        // zero gradient meets no value of a neighbour (only tiles that reach
        // past it pay for the select).
        auto plane_mma = [&](auto pt) {
          constexpr bool PART = decltype(pt)::value;
#pragma unroll
          for (int ks = 0; ks < TJ / 2; ++ks) {
            uint32_t A[MC / 16][4];
#pragma unroll
            for (int m = 0; m < MC / 16; ++m)
              // A = g^T (co x v): rows v, columns co, read transposed
              ldsm_x4_t(A[m][0], A[m][1], A[m][2], A[m][3],
                        gb + (uint32_t)(ks * 16 * GP + m * 32));
            const bool zr = PART && !(kok && j0 + ks * 2 + (mat & 1) < a.ny);
#pragma unroll
            for (int d = 0; d < ND; ++d) {
              const uint32_t xr = zr ? zrow : xb[d] + (uint32_t)(ks * 2 * WK * XP);
#pragma unroll
              for (int n = 0; n < NC / 8; n += 2) {
                uint32_t b0, b1, b2, b3;
                ldsm_x4_t(b0, b1, b2, b3, xr + (uint32_t)(n * 16));
#pragma unroll
                for (int m = 0; m < MC / 16; ++m) {
                  mma_bf16(acc[d][m][n], A[m], b0, b1);
                  mma_bf16(acc[d][m][n + 1], A[m], b2, b3);
                }
              }
            }
          }
        };
        if (part)
          plane_mma(std::true_type{});
        else
          plane_mma(std::false_type{});
        if (bias && tid < BG * MC) {
          const __nv_bfloat16 *gp =
              reinterpret_cast<const __nv_bfloat16 *>(smem + gs * S::GB) + tid % MC;
          for (int row = tid / MC; row < TK * TJ; row += BG)
            bsum += __bfloat162float(gp[row * (GP / 2)]);
        }
        if (++chain == WG_FLUSH) {
          chain = 0;
          flush();
        }
      }
      xs = xs + 1 == XS ? 0 : xs + 1;
      gs = gs + 1 == GS ? 0 : gs + 1;
    }
  }
  if (chain || !stored) flush();
  if (bias) {
    cp_wait<0>();
    __syncthreads();
    float *sh = reinterpret_cast<float *>(smem);
    if (tid < BG * MC) sh[tid] = bsum;
    __syncthreads();
    if (tid < MC) {
      float s = 0.0f;
      for (int q = 0; q < BG; ++q) s += sh[q * MC + tid];
      a.dbdst[(int64_t)blockIdx.x * a.cout + co0 + tid] = s;
    }
  }
}

// out[q] = sum over splits of part[s][q]: 8 groups of splits per output, then
// the groups, each in a fixed order.  Outputs n .. n + nb - 1 are the bias's.
__global__ void __launch_bounds__(256) sum_splits_kernel(float *__restrict__ out,
                                                         float *__restrict__ outb,
                                                         const float *__restrict__ part,
                                                         const float *__restrict__ partb,
                                                         int splits, int64_t n, int nb) {
  __shared__ float sh[8][33];
  const int x = threadIdx.x & 31, grp = threadIdx.x >> 5;
  const int64_t q = (int64_t)blockIdx.x * 32 + x;
  float s = 0.0f;
  if (q < n) {
    for (int c = grp; c < splits; c += 8) s += part[(int64_t)c * n + q];
  } else if (q < n + nb) {
    for (int c = grp; c < splits; c += 8) s += partb[(int64_t)c * nb + (q - n)];
  }
  sh[grp][x] = s;
  __syncthreads();
  if (grp == 0 && q < n + nb) {
    float t = sh[0][x];
#pragma unroll
    for (int g = 1; g < 8; ++g) t += sh[g][x];
    if (q < n)
      out[q] = t;
    else
      outb[q - n] = t;
  }
}

template <int MC, int NC, int ND>
cudaError_t launch_wgrad(WgArgs a, float *dw, float *db, float *ws, int64_t cap,
                         cudaStream_t s) {
  constexpr int SMEM = WgShape<MC, NC, ND>::SMEM;
  if (!smem_opt_in((const void *)conv_wgrad_kernel<MC, NC, ND>, SMEM))
    return cudaErrorNotSupported;
  a.nbi = a.cin / NC;
  const int blocks = a.nbi * (a.cout / MC) * (ND == 3 ? 1 : 3);
  // about three CTAs per SM where the workspace's slots allow as many splits
  const int64_t want = (148 * 3 + blocks - 1) / blocks;
  const int64_t splits = std::min<int64_t>({want, a.tiles, cap});
  const int64_t n = 27LL * a.cin * a.cout;
  float *partb = ws + splits * n;
  a.dst = splits > 1 ? ws : dw;
  a.dbdst = !db ? nullptr : (splits > 1 ? partb : db);
  conv_wgrad_kernel<MC, NC, ND><<<dim3((unsigned)splits, blocks), WG_THREADS, SMEM, s>>>(a);
  if (splits > 1) {
    const int nb = db ? a.cout : 0;
    sum_splits_kernel<<<(unsigned)((n + nb + 31) / 32), 256, 0, s>>>(dw, db, ws, partb,
                                                                     (int)splits, n, nb);
  }
  return cudaGetLastError();
}

}  // namespace uconv
}  // namespace bsp

using namespace bsp;
using namespace bsp::uconv;

extern "C" int bsp_unet_conv3_fwd(bsp_bf16_t *out_, const bsp_bf16_t *in_,
                                  const bsp_bf16_t *w_, const float *bias, int nx, int ny,
                                  int nz, int cin, int cout, int relu, cudaStream_t s) {
  if (nx <= 0 || ny <= 0 || nz <= 0) return BSP_OK;
  if (!out_ || !in_ || !w_) return BSP_ERR_NULL;
  if (cin <= 0 || cin % 16 || cout <= 0 || cout % 16) return BSP_ERR_SHAPE;
  if (((uintptr_t)in_ & 15u) || ((uintptr_t)w_ & 15u) || ((uintptr_t)out_ & 3u))
    return BSP_ERR_ALIGN;
  FwdArgs a{};
  a.out = reinterpret_cast<__nv_bfloat16 *>(out_);
  a.in = reinterpret_cast<const __nv_bfloat16 *>(in_);
  a.w = reinterpret_cast<const __nv_bfloat16 *>(w_);
  a.bias = bias;
  a.nx = nx;
  a.ny = ny;
  a.nz = nz;
  a.cout = cout;
  a.relu = relu;
  const int64_t nvox = (int64_t)nx * ny * nz;
  // Output channels per CTA: 32 where cout divides by it and 32-channel tiles
  // still give every SM a CTA, else 16 (at the deepest levels an SM's time is
  // its weights' load).  128 input channels leave room for 16.
  const int64_t cells = (int64_t)((ny + TJ - 1) / TJ) * ((nz + TK - 1) / TK) * nx;
  const bool n32 = cout % 32 == 0 && cells * (cout / 32) >= 148;
  if ((int64_t)ny * nz * cin < (1 << 30)) {  // offsets inside a plane are 32-bit
    switch (cin) {
      case 16: return (int)(n32 ? launch_fwd<16, 32, 2, 3>(a, s) : launch_fwd<16, 16, 2, 3>(a, s));
      case 32: return (int)(n32 ? launch_fwd<32, 32, 2, 3>(a, s) : launch_fwd<32, 16, 2, 3>(a, s));
      case 64: return (int)(n32 ? launch_fwd<64, 32, 1, 3>(a, s) : launch_fwd<64, 16, 1, 3>(a, s));
      case 128: return (int)launch_fwd<128, 16, 1, 2>(a, s);
      default: break;
    }
  }
  const int nt = cout % 64 == 0 ? 64 : (cout % 32 == 0 ? 32 : 16);
  const dim3 grid((unsigned)((nvox + GM - 1) / GM), cout / nt);
  if (nt == 64)
    conv_any_kernel<64><<<grid, GM, 0, s>>>(a.out, a.in, a.w, bias, nx, ny, nz, cin, cout, relu);
  else if (nt == 32)
    conv_any_kernel<32><<<grid, GM, 0, s>>>(a.out, a.in, a.w, bias, nx, ny, nz, cin, cout, relu);
  else
    conv_any_kernel<16><<<grid, GM, 0, s>>>(a.out, a.in, a.w, bias, nx, ny, nz, cin, cout, relu);
  return (int)cudaGetLastError();
}

extern "C" size_t bsp_unet_wgrad_workspace_bytes(int nx, int ny, int nz, int cin, int cout) {
  const int64_t nvox = (int64_t)nx * ny * nz;
  const int64_t nslots = (nvox + WG_VCH - 1) / WG_VCH;
  return (size_t)nslots * 27 * cin * cout * sizeof(float);
}

extern "C" int bsp_unet_conv3_wgrad(float *dw, float *db, const bsp_bf16_t *g_,
                                    const bsp_bf16_t *in_, int nx, int ny, int nz, int cin,
                                    int cout, float *workspace, size_t workspace_bytes,
                                    cudaStream_t s) {
  const __nv_bfloat16 *g = reinterpret_cast<const __nv_bfloat16 *>(g_);
  const __nv_bfloat16 *in = reinterpret_cast<const __nv_bfloat16 *>(in_);
  if (nx <= 0 || ny <= 0 || nz <= 0) return BSP_OK;
  if (!dw || !g || !in || !workspace) return BSP_ERR_NULL;
  if (cin <= 0 || cin % 16 || cout <= 0 || cout % 16) return BSP_ERR_SHAPE;
  if (workspace_bytes < bsp_unet_wgrad_workspace_bytes(nx, ny, nz, cin, cout))
    return BSP_ERR_WORKSPACE;
  if (((uintptr_t)in & 15u) || ((uintptr_t)g & 15u)) return BSP_ERR_ALIGN;
  const int64_t nvox = (int64_t)nx * ny * nz;
  WgArgs a{};
  a.g = g;
  a.in = in;
  a.nx = nx;
  a.ny = ny;
  a.nz = nz;
  a.cin = cin;
  a.cout = cout;
  a.jt = (ny + TJ - 1) / TJ;
  a.kt = (nz + TK - 1) / TK;
  a.tiles = (int64_t)nx * a.jt * a.kt;
  // Splits of the voxels: as many as the workspace's slots, less one that is
  // kept for the bias partials (they fit it up to 27 cin splits).
  const int64_t nslots = (nvox + WG_VCH - 1) / WG_VCH;
  const int64_t cap = std::min<int64_t>(std::max<int64_t>(nslots - 1, 1), 27 * 16);
  // Channel blocks of 32 where the channels divide by it and they still give
  // two CTAs per SM, else 16; below one CTA per SM each di gets its own.
  bool m32 = cout % 32 == 0, n32 = cin % 32 == 0;
  auto ctas = [&]() { return cap * (cout / (m32 ? 32 : 16)) * (cin / (n32 ? 32 : 16)); };
  if (n32 && ctas() < 2 * 148) n32 = false;
  if (m32 && ctas() < 2 * 148) m32 = false;
  if (ctas() < 148) return (int)launch_wgrad<16, 16, 1>(a, dw, db, workspace, cap, s);
  auto fn = m32 ? (n32 ? launch_wgrad<32, 32, 3> : launch_wgrad<32, 16, 3>)
                : (n32 ? launch_wgrad<16, 32, 3> : launch_wgrad<16, 16, 3>);
  return (int)fn(a, dw, db, workspace, cap, s);
}
