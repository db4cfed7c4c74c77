// unet_conv.cu -- the 3x3x3 convolutions of the warm-start network's training
// pass on the unpadded layout act[v][c], v = (i ny + j) nz + k, channels
// innermost (BF16), weights w[tap][co][ci] (tap = (di+1) 9 + (dj+1) 3 + (dk+1)):
// the forward pass (and the data gradient, the same kernel on flipped
// weights) on tcgen05 tensor cores, the weight and bias gradients on mma.sync.
//
// Forward.  A tile is 8 k x 16 j voxels of one i plane: the 128 rows (TMEM
// lanes) of D.  Its input window, 10 k x 18 j rows of one plane, is staged
// once per plane as [channel group of 8][j][k][16 bytes] -- exactly the
// K-major no-swizzle core matrix (8 rows of 16 bytes), so the operand of tap
// (dj, dk) is the same staged plane read through a descriptor whose start is
// moved by ((dj+1) 10 + (dk+1)) 16 bytes, with 8-row groups (one j line) 160
// bytes apart and the two 8-channel halves of a K step 2880 bytes apart.  A CTA
// marches along i with the planes i-1, i, i+1 in a ring, so a plane is read
// from L2 once per tile (1.4x its voxels) and feeds all 27 taps; gathering the
// rows per tap instead read every voxel 27 times and left the tensor cores
// waiting (143 us against 15 us here for 32 -> 32 channels at 64x64x48 on a
// B200; the bound is shared-memory operand reads, 32 cycles per M = 128,
// K = 16 MMA at these small N).  Rows outside the grid are zero-filled by the
// copy.  Weights stay in shared memory: at most 64 input channels x NT output
// channels with 64 NT <= 2048; more input channels run in passes that
// accumulate in tensor memory.
//
// Weight gradient.  dw[tap][co][ci] = sum_v g[v][co] in[v + d][ci]: the
// contraction runs over voxels and M x N is only 16 or 32 channels a side, so
// mma.sync m16n8k16 fits it without padding (a 64 x 64 tile did 4-16 times the
// work).  A CTA takes one di and a block of MC x NC channels; its nine warps
// take the nine (dj, dk) taps from the same staged 128-voxel g tile and
// 10 x 18 row input window: 358 us -> 22 us for the same layer.  Chains of MMA
// accumulation are cut every 2048 voxels into a second set of FP32 registers.
// The bias gradient is summed from the staged g tiles of di = 0.  Partial sums
// per split are added in a fixed order (deterministic).
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include <algorithm>

#include "bsp_common.cuh"
#include "tc5.cuh"

namespace bsp {
namespace uconv {

constexpr int TK = 8, TJ = 16;                 // voxels of a tile: 8 k x 16 j
constexpr int WK = TK + 2, WJ = TJ + 2;        // its input window
constexpr int WROWS = WK * WJ;                 // 180 rows
constexpr int HALF = WROWS * 16;               // bytes of one 8-channel group of a plane
constexpr int NPROD = 4;                       // producer warps
constexpr int FWD_THREADS = (4 + 1 + NPROD) * 32;
constexpr int MAXSLOT = 6, MAXACC = 8;
constexpr int CP_MAX = 64;                     // input channels per pass
constexpr int W_BYTES_MAX = 27 * 2048 * 2;     // weights of a pass: channels x NT <= 2048
constexpr int SMEM_MAX = 232448;

__device__ int g_conv_err;  // BSP_ERR_TIMEOUT once a bounded wait gave up

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

struct FwdArgs {
  __nv_bfloat16 *out;
  const __nv_bfloat16 *in, *w;
  const float *bias;
  int nx, ny, nz, cin, cout, relu;
  int nt, nct;      // output channels per CTA, channel tiles
  int jt, kt;       // tiles per plane
  int len, npass;   // planes per CTA, input-channel passes
  int cp;           // input channels of a full pass
  int nslot, nacc;  // plane ring, accumulators
  int wbytes, slot_bytes;
  int vec;          // out rows are 16-byte aligned
};

struct FwdCtl {
  uint64_t full[MAXSLOT], empty[MAXSLOT], acc_full[MAXACC], acc_empty[MAXACC], wfree, drain;
  uint32_t tmem_base;
  int abort;
};

__device__ __forceinline__ bool wait_ok(uint64_t *bar, uint32_t parity, FwdCtl *c) {
  if (mbar_wait(bar, parity)) return true;
  *(volatile int *)&c->abort = 1;
  atomicExch(&g_conv_err, BSP_ERR_TIMEOUT);
  return false;
}

// Warps 0-3: epilogue (TMEM lane quarter = warp), warp 4: TMEM allocation and
// MMA issue (one thread), warps 5-8: cp.async producers.
// Plane fills are numbered f = pass (len + 2) + pl, pl = 0 .. len + 1 for plane
// i0 - 1 + pl; fill f goes to slot f mod nslot.  Output o of a pass reads fills
// o, o + 1, o + 2 of it; fill o is free after output o (the last two after the
// last output).  A producer warp arrives for fill f only after its copies of
// f + la are issued, la = nslot - 3 (at most 2): waiting for the slot of f
// needs output f - nslot, i.e. fills up to f - nslot + 2 <= f - la - 1, which
// have been arrived for.  The pass's weights are copied before its first
// plane, so a full first plane implies them.
__global__ void __launch_bounds__(FWD_THREADS, 2) conv_fwd_kernel(const FwdArgs a) {
  extern __shared__ __align__(128) unsigned char smem[];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  unsigned char *wsm = smem;
  unsigned char *slots = smem + a.wbytes;
  FwdCtl *c = reinterpret_cast<FwdCtl *>(slots + (size_t)a.nslot * a.slot_bytes);
  int t = blockIdx.x;
  const int ct = t % a.nct;
  t /= a.nct;
  const int k0 = (t % a.kt) * TK;
  t /= a.kt;
  const int j0 = (t % a.jt) * TJ;
  const int i0 = (t / a.jt) * a.len;
  const int len = min(a.len, a.nx - i0);
  const int co0 = ct * a.nt;
  const int nt = a.nt, npass = a.npass;
  uint32_t tcols = 32;
  while (tcols < (uint32_t)(a.nacc * nt)) tcols <<= 1;

  if (threadIdx.x == 0) {
    for (int s = 0; s < a.nslot; ++s) {
      mbar_init(&c->full[s], NPROD);
      mbar_init(&c->empty[s], 1);
    }
    for (int b = 0; b < a.nacc; ++b) {
      mbar_init(&c->acc_full[b], 1);
      mbar_init(&c->acc_empty[b], 4);
    }
    mbar_init(&c->wfree, 1);
    mbar_init(&c->drain, 1);
    c->abort = 0;
    utc::fence_barrier_init();
  }
  if (warp == 4) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                     smem_u32(&c->tmem_base)),
                 "r"(tcols)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  utc::fence_async_shared();
  utc::tc_fence_before();
  __syncthreads();
  utc::tc_fence_after();
  const uint32_t tbase = c->tmem_base;

  if (warp >= 5) {
    // ---------------- producers ----------------
    const int pt = threadIdx.x - 160;  // 0 .. 127
    const uint32_t wsm_u = smem_u32(wsm), slots_u = smem_u32(slots);
    const int la = a.nslot >= 5 ? 2 : 1;
    const int64_t plane = (int64_t)a.ny * a.nz;
    int f = 0, arrived = 0;
    bool ok = true;
    auto arrive_next = [&]() {
      utc::fence_async_shared();
      __syncwarp();
      if (lane == 0) utc::mbar_arrive(&c->full[arrived % a.nslot]);
      ++arrived;
    };
    for (int ps = 0; ps < npass && ok; ++ps) {
      const int c0 = ps * a.cp, cp = min(a.cp, a.cin - c0), cg = cp >> 3;
      if (ps > 0) {
        // the weight buffer is read by the MMAs of the pass before
        cp_wait<0>();
        while (arrived < f) arrive_next();
        ok = __all_sync(0xffffffffu, wait_ok(&c->wfree, (uint32_t)((ps - 1) & 1), c));
        if (!ok) break;
      }
      // weights: [tap][channel group of 8][n][16 bytes]
      for (int q = pt; q < 27 * cg * nt; q += NPROD * 32) {
        const int g8 = q % cg, r = q / cg;
        const int n = r % nt, tap = r / nt;
        cp16(wsm_u + (uint32_t)(((tap * cg + g8) * nt + n) * 16),
             a.w + ((int64_t)tap * a.cout + co0 + n) * a.cin + c0 + g8 * 8, true);
      }
      for (int pl = 0; pl < len + 2; ++pl, ++f) {
        const int s = f % a.nslot;
        ok = __all_sync(0xffffffffu,
                        wait_ok(&c->empty[s], (uint32_t)(((f / a.nslot) & 1) ^ 1), c));
        if (!ok) break;
        const int i = i0 - 1 + pl;
        const bool iok = i >= 0 && i < a.nx;
        const uint32_t dst = slots_u + (uint32_t)(s * a.slot_bytes);
        for (int q = pt; q < WROWS * cg; q += NPROD * 32) {
          const int row = q / cg, g8 = q - row * cg;
          const int jj = row / WK, kk = row - jj * WK;
          const int j = j0 - 1 + jj, k = k0 - 1 + kk;
          const bool v = iok && j >= 0 && j < a.ny && k >= 0 && k < a.nz;
          const __nv_bfloat16 *src =
              v ? a.in + (i * plane + (int64_t)j * a.nz + k) * a.cin + c0 + g8 * 8 : a.in;
          cp16(dst + (uint32_t)(g8 * HALF + row * 16), src, v);
        }
        cp_commit();
        if (f - arrived >= la) {
          if (la == 2)
            cp_wait<2>();
          else
            cp_wait<1>();
          arrive_next();
        }
      }
    }
    cp_wait<0>();
    if (ok)
      while (arrived < f) arrive_next();
  } else if (warp == 4) {
    // ---------------- MMA issuer ----------------
    if (lane == 0) {
      const uint32_t idesc = utc::idesc_bf16(nt, 128);
      const uint32_t wsm_u = smem_u32(wsm), slots_u = smem_u32(slots);
      bool ok = true;
      for (int ps = 0; ps < npass && ok; ++ps) {
        const int cp = min(a.cp, a.cin - ps * a.cp), cg = cp >> 3;
        const int f0 = ps * (len + 2);
        const uint64_t bstep = (uint64_t)(cg * nt);  // 16-byte units per tap
        for (int o = 0; o < len && ok; ++o) {
          const int b = o % a.nacc;
          if (npass == 1) ok = wait_ok(&c->acc_empty[b], (uint32_t)(((o / a.nacc) & 1) ^ 1), c);
          for (int x = o == 0 ? 0 : 2; x < 3 && ok; ++x) {
            const int f = f0 + o + x;
            ok = wait_ok(&c->full[f % a.nslot], (uint32_t)((f / a.nslot) & 1), c);
          }
          if (!ok) break;
          utc::tc_fence_after();
          const uint32_t dt = tbase + (uint32_t)(b * nt);
          uint32_t acc = ps > 0 ? 1u : 0u;
          for (int di = 0; di < 3; ++di) {
            const uint32_t sl = slots_u + (uint32_t)(((f0 + o + di) % a.nslot) * a.slot_bytes);
            for (int kc = 0; kc < cg / 2; ++kc) {
              const uint64_t ad = utc::sdesc(sl + (uint32_t)(kc * 2 * HALF), HALF, WK * 16);
              const uint64_t bd = utc::sdesc(
                  wsm_u + (uint32_t)(((di * 9 * cg) + kc * 2) * nt * 16), nt * 16, 128);
#pragma unroll
              for (int s = 0; s < 9; ++s) {
                utc::tc_mma(dt, ad + (uint64_t)((s / 3) * WK + s % 3), bd + (uint64_t)s * bstep,
                            idesc, acc);
                acc = 1u;
              }
            }
          }
          utc::tc_commit(&c->empty[(f0 + o) % a.nslot]);
          if (o == len - 1) {
            utc::tc_commit(&c->empty[(f0 + len) % a.nslot]);
            utc::tc_commit(&c->empty[(f0 + len + 1) % a.nslot]);
          }
          if (ps == npass - 1) utc::tc_commit(&c->acc_full[b]);
        }
        if (ok && ps + 1 < npass) utc::tc_commit(&c->wfree);
      }
      // drain: every MMA issued has completed before TMEM is freed
      utc::tc_commit(&c->drain);
      mbar_wait(&c->drain, 0);
    }
  } else {
    // ---------------- epilogue ----------------
    const int row = warp * 32 + lane;
    const int j = j0 + (row >> 3), k = k0 + (row & 7);
    const bool valid = j < a.ny && k < a.nz;
    for (int o = 0; o < len; ++o) {
      const int b = o % a.nacc;
      if (!__all_sync(0xffffffffu,
                      wait_ok(&c->acc_full[b], (uint32_t)((o / a.nacc) & 1), c)))
        break;
      utc::tc_fence_after();
      const uint32_t trow = tbase + ((uint32_t)(warp * 32) << 16) + (uint32_t)(b * nt);
      const int64_t v = ((int64_t)(i0 + o) * a.ny + j) * a.nz + k;
      for (int cb = 0; cb < nt; cb += 16) {
        float x[16];
        utc::tmem_ld1x16(trow + (uint32_t)cb, x);
        if (!valid) continue;
        if (a.bias) {
#pragma unroll
          for (int e = 0; e < 16; ++e) x[e] += __ldg(a.bias + co0 + cb + e);
        }
        if (a.relu) {
#pragma unroll
          for (int e = 0; e < 16; ++e) x[e] = fmaxf(x[e], 0.0f);
        }
        uint32_t w[8];
#pragma unroll
        for (int e = 0; e < 8; ++e) w[e] = utc::pack_bf16x2(x[2 * e], x[2 * e + 1]);
        __nv_bfloat16 *dst = a.out + v * a.cout + co0 + cb;
        if (a.vec) {
          reinterpret_cast<uint4 *>(dst)[0] = make_uint4(w[0], w[1], w[2], w[3]);
          reinterpret_cast<uint4 *>(dst)[1] = make_uint4(w[4], w[5], w[6], w[7]);
        } else {
#pragma unroll
          for (int e = 0; e < 8; ++e) reinterpret_cast<uint32_t *>(dst)[e] = w[e];
        }
      }
      utc::tc_fence_before();
      __syncwarp();
      if (lane == 0) utc::mbar_arrive(&c->acc_empty[b]);
    }
  }
  utc::tc_fence_before();
  __syncthreads();
  utc::tc_fence_after();
  if (warp == 4)
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tbase),
                 "r"(tcols)
                 : "memory");
}

// ---- weight and bias gradient -------------------------------------------------------------
constexpr int WG_VCH = 2048;      // voxels per partial-sum slot of the workspace
constexpr int WG_THREADS = 288;   // nine warps, one (dj, dk) tap each
constexpr int WG_FLUSH = 16;      // tiles (2048 voxels) per MMA accumulation chain
constexpr int WG_STAGES = 3;

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

// Row pitches of C channels: C * 2 + 16 bytes put eight consecutive rows on
// distinct banks for ldmatrix (48 and 80 bytes).
template <int MC, int NC>
constexpr int wg_stage_bytes() {
  return TK * TJ * (MC * 2 + 16) + WROWS * (NC * 2 + 16);
}
template <int MC, int NC>
constexpr int wg_smem_bytes() {
  return WG_STAGES * wg_stage_bytes<MC, NC>() + 64;
}

struct WgArgs {
  float *dst;    // splits == 1: dw; else split s's [27][cout][cin] at s * 27 cout cin
  float *dbdst;  // NULL, or [split][cout] (splits == 1: db)
  const __nv_bfloat16 *g, *in;
  int nx, ny, nz, cin, cout;
  int jt, kt, nbi;  // tiles per plane, input-channel blocks
  int64_t tiles;
};

template <int MC, int NC>
__global__ void __launch_bounds__(WG_THREADS, 2) conv_wgrad_kernel(const WgArgs a) {
  extern __shared__ __align__(128) unsigned char smem[];
  constexpr int GP = MC * 2 + 16, XP = NC * 2 + 16;  // row pitches
  constexpr int GB = TK * TJ * GP, SB = wg_stage_bytes<MC, NC>();
  constexpr int GC = MC / 8, XC = NC / 8;            // 16-byte pieces per row
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int di = (int)blockIdx.y % 3 - 1, blk = (int)blockIdx.y / 3;
  const int co0 = (blk / a.nbi) * MC, ci0 = (blk % a.nbi) * NC;
  const int dj = warp / 3, dk = warp % 3;  // + 1
  const int64_t t0 = a.tiles * blockIdx.x / gridDim.x, t1 = a.tiles * (blockIdx.x + 1) / gridDim.x;
  const uint32_t base = smem_u32(smem), zrow = base + WG_STAGES * SB;
  if (tid < 4) *reinterpret_cast<uint4 *>(smem + WG_STAGES * SB + tid * 16) = make_uint4(0, 0, 0, 0);
  auto coords = [&](int64_t t, int &i, int &j0, int &k0) {
    k0 = (int)(t % a.kt) * TK;
    t /= a.kt;
    j0 = (int)(t % a.jt) * TJ;
    i = (int)(t / a.jt);
  };
  auto stage = [&](int64_t t, int s) {
    int i, j0, k0;
    coords(t, i, j0, k0);
    const uint32_t gs = base + s * SB, xs = gs + GB;
    for (int q = tid; q < TK * TJ * GC; q += WG_THREADS) {
      const int row = q / GC, p = q % GC;
      const int j = j0 + row / TK, k = k0 + row % TK;
      const bool v = j < a.ny && k < a.nz;
      cp16(gs + row * GP + p * 16,
           v ? a.g + (((int64_t)i * a.ny + j) * a.nz + k) * a.cout + co0 + p * 8 : a.g, v);
    }
    const int ii = i + di;
    const bool iok = ii >= 0 && ii < a.nx;
    for (int q = tid; q < WROWS * XC; q += WG_THREADS) {
      const int row = q / XC, p = q % XC;
      const int jj = row / WK, j = j0 - 1 + jj, k = k0 - 1 + row - jj * WK;
      const bool v = iok && j >= 0 && j < a.ny && k >= 0 && k < a.nz;
      cp16(xs + row * XP + p * 16,
           v ? a.in + (((int64_t)ii * a.ny + j) * a.nz + k) * a.cin + ci0 + p * 8 : a.in, v);
    }
  };
  float acc[MC / 16][NC / 8][4], sum[MC / 16][NC / 8][4];
#pragma unroll
  for (int m = 0; m < MC / 16; ++m)
#pragma unroll
    for (int n = 0; n < NC / 8; ++n)
#pragma unroll
      for (int q = 0; q < 4; ++q) acc[m][n][q] = sum[m][n][q] = 0.0f;
  const bool bias = a.dbdst != nullptr && di == 0 && ci0 == 0;
  constexpr int BG = WG_THREADS / MC;  // row groups of the bias sums
  float bsum = 0.0f;
  const int mat = lane >> 3, r = lane & 7;
#pragma unroll
  for (int s = 0; s < WG_STAGES - 1; ++s) {
    if (t0 + s < t1) stage(t0 + s, s);
    cp_commit();
  }
  int buf = 0, chain = 0;
  for (int64_t t = t0; t < t1; ++t) {
    cp_wait<WG_STAGES - 2>();
    __syncthreads();  // tile t staged by every thread; tile t - 1 no longer read
    if (t + WG_STAGES - 1 < t1) stage(t + WG_STAGES - 1, (buf + WG_STAGES - 1) % WG_STAGES);
    cp_commit();
    int i, j0, k0;
    coords(t, i, j0, k0);
    const uint32_t gs = base + buf * SB, xs = gs + GB;
    const bool kok = k0 + r < a.nz;
#pragma unroll
    for (int ks = 0; ks < TJ / 2; ++ks) {
      uint32_t A[MC / 16][4];
#pragma unroll
      for (int m = 0; m < MC / 16; ++m)
        // A = g^T (co x v): rows v, columns co, read transposed
        ldsm_x4_t(A[m][0], A[m][1], A[m][2], A[m][3],
                  gs + (ks * 16 + (mat >> 1) * 8 + r) * GP + (m * 16 + (mat & 1) * 8) * 2);
      const int jj = ks * 2 + (mat & 1);
      // voxels past the grid's end read a zero row, so that their zero
      // gradient meets no value of a neighbour
      const bool v = kok && j0 + jj < a.ny;
      const uint32_t xr = xs + ((jj + dj) * WK + r + dk) * XP;
#pragma unroll
      for (int n = 0; n < NC / 8; n += 2) {
        uint32_t b0, b1, b2, b3;
        const uint32_t off = (uint32_t)((n + (mat >> 1)) * 16);
        ldsm_x4_t(b0, b1, b2, b3, (v ? xr : zrow) + off);
#pragma unroll
        for (int m = 0; m < MC / 16; ++m) {
          mma_bf16(acc[m][n], A[m], b0, b1);
          mma_bf16(acc[m][n + 1], A[m], b2, b3);
        }
      }
    }
    if (bias && tid < BG * MC) {
      const __nv_bfloat16 *gp =
          reinterpret_cast<const __nv_bfloat16 *>(smem + buf * SB) + tid % MC;
      for (int row = tid / MC; row < TK * TJ; row += BG)
        bsum += __bfloat162float(gp[row * (GP / 2)]);
    }
    if (++chain == WG_FLUSH) {
      chain = 0;
#pragma unroll
      for (int m = 0; m < MC / 16; ++m)
#pragma unroll
        for (int n = 0; n < NC / 8; ++n)
#pragma unroll
          for (int q = 0; q < 4; ++q) {
            sum[m][n][q] += acc[m][n][q];
            acc[m][n][q] = 0.0f;
          }
    }
    buf = buf + 1 == WG_STAGES ? 0 : buf + 1;
  }
  const int g4 = lane >> 2, t4 = lane & 3;
  const int tap = (di + 1) * 9 + warp;
  float *dst = a.dst + ((int64_t)blockIdx.x * 27 + tap) * a.cout * a.cin;
#pragma unroll
  for (int m = 0; m < MC / 16; ++m)
#pragma unroll
    for (int n = 0; n < NC / 8; ++n)
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const int co = co0 + m * 16 + g4 + h * 8, ci = ci0 + n * 8 + t4 * 2;
        float *d = dst + (int64_t)co * a.cin + ci;
        d[0] = sum[m][n][2 * h] + acc[m][n][2 * h];
        d[1] = sum[m][n][2 * h + 1] + acc[m][n][2 * h + 1];
      }
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

template <int MC, int NC>
cudaError_t launch_wgrad(float *dw, float *db, const __nv_bfloat16 *g, const __nv_bfloat16 *in,
                         int nx, int ny, int nz, int cin, int cout, float *ws, int nslots,
                         cudaStream_t s) {
  constexpr int SMEM = wg_smem_bytes<MC, NC>();
  if (!smem_opt_in((const void *)conv_wgrad_kernel<MC, NC>, SMEM)) return cudaErrorNotSupported;
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
  a.nbi = cin / NC;
  const int blocks = 3 * a.nbi * (cout / MC);
  // Splits of the voxels: enough CTAs for about three per SM, as many as the
  // workspace's slots hold (one slot is kept for the bias partials, which fit
  // it up to 27 cin splits)
  const int64_t want = (148 * 3 + blocks - 1) / blocks;
  int64_t splits = std::min<int64_t>({want, a.tiles, nslots > 1 ? nslots - 1 : 1, 27 * 16});
  const int64_t n = 27LL * cin * cout;
  float *partb = ws + splits * n;
  a.dst = splits > 1 ? ws : dw;
  a.dbdst = !db ? nullptr : (splits > 1 ? partb : db);
  conv_wgrad_kernel<MC, NC><<<dim3((unsigned)splits, blocks), WG_THREADS, SMEM, s>>>(a);
  if (splits > 1) {
    const int nb = db ? cout : 0;
    sum_splits_kernel<<<(unsigned)((n + nb + 31) / 32), 256, 0, s>>>(dw, db, ws, partb,
                                                                     (int)splits, n, nb);
  }
  return cudaGetLastError();
}

}  // namespace uconv
}  // namespace bsp

using namespace bsp;
using namespace bsp::uconv;

namespace bsp {
// Reads and clears the convolution's give-up flag (bsp_unet_tc_error).
cudaError_t conv_error_take(int *flag) {
  cudaError_t e = cudaMemcpyFromSymbol(flag, uconv::g_conv_err, sizeof(int));
  if (e == cudaSuccess && *flag) {
    const int zero = 0;
    e = cudaMemcpyToSymbol(uconv::g_conv_err, &zero, sizeof(int));
  }
  return e;
}
}  // namespace bsp

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
  a.cin = cin;
  a.cout = cout;
  a.relu = relu;
  a.vec = ((uintptr_t)out_ & 15u) == 0;
  a.cp = cin < CP_MAX ? cin : CP_MAX;
  a.npass = (cin + CP_MAX - 1) / CP_MAX;
  // output channels per CTA: the largest tile that divides cout and whose
  // weights (27 x cp x nt) stay within W_BYTES_MAX
  a.nt = 64;
  while (cout % a.nt || a.cp * a.nt > 2048) a.nt >>= 1;
  a.nct = cout / a.nt;
  a.wbytes = (27 * a.cp * a.nt * 2 + 127) / 128 * 128;
  a.slot_bytes = a.cp / 8 * HALF;
  a.nslot = MAXSLOT;
  while (a.nslot > 4 && a.wbytes + a.nslot * a.slot_bytes + (int)sizeof(FwdCtl) > SMEM_MAX)
    --a.nslot;
  const int smem = a.wbytes + a.nslot * a.slot_bytes + (int)sizeof(FwdCtl);
  if (smem > SMEM_MAX) return BSP_ERR_SHAPE;
  a.jt = (ny + TJ - 1) / TJ;
  a.kt = (nz + TK - 1) / TK;
  const int64_t cols = (int64_t)a.jt * a.kt * a.nct;
  // planes per CTA: one wave of CTAs (two per SM when both fit), so that the
  // weights are loaded and the halo planes re-read as seldom as possible
  const int occ = smem <= SMEM_MAX / 2 - 1024 ? 2 : 1;
  int64_t len = (nx * cols + 148 * occ - 1) / (148 * occ);
  len = std::max<int64_t>(1, std::min<int64_t>(len, nx));
  a.nacc = 4;
  if (a.npass > 1) {  // every plane's accumulator stays until the last pass
    len = std::min<int64_t>(len, MAXACC);
    a.nacc = MAXACC;
  }
  a.len = (int)len;
  const int64_t items = cols * ((nx + len - 1) / len);
  if (items > 0x7fffffff) return BSP_ERR_SHAPE;
  if (!smem_opt_in((const void *)conv_fwd_kernel, SMEM_MAX)) return (int)cudaErrorNotSupported;
  conv_fwd_kernel<<<(unsigned)items, FWD_THREADS, smem, s>>>(a);
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
  const int nslots = (int)std::min<int64_t>((nvox + WG_VCH - 1) / WG_VCH, 1 << 30);
  // channel blocks of 32 where the channels divide by it, else 16
  const bool m32 = cout % 32 == 0, n32 = cin % 32 == 0;
  auto fn = m32 ? (n32 ? launch_wgrad<32, 32> : launch_wgrad<32, 16>)
                : (n32 ? launch_wgrad<16, 32> : launch_wgrad<16, 16>);
  return (int)fn(dw, db, g, in, nx, ny, nz, cin, cout, workspace, nslots, s);
}
