// unet.cu -- kernels of the learned warm start: a small 3-D U-Net over the
// pot grid, trained and run on the GPU by these kernels alone.
//
// Activations are channels-last BF16, act[v][c] with v = (i*ny + j)*nz + k;
// weights of a 3x3x3 convolution are BF16 w[tap][co][ci] (tap = (di+1)*9 +
// (dj+1)*3 + (dk+1)), with an FP32 master copy kept by the optimiser.  The
// convolutions and their gradients are in unet_conv.cu; here: weight flipping,
// ReLU gradient, pooling, upsampling, input packing, head, loss and Adam.
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include "bsproj.h"

namespace bsp {
namespace unet {

__global__ void sum_slots_kernel(float *__restrict__ out, const float *__restrict__ partials,
                                 int nblocks) {
  float acc = 0.0f;
  for (int b = 0; b < nblocks; ++b) acc += partials[(int64_t)threadIdx.x * nblocks + b];
  out[threadIdx.x] = acc;
}

// wt[tap'][ci][co] = w[26 - tap'][co][ci]: weights of the data-gradient convolution
__global__ void flip_weights_kernel(__nv_bfloat16 *__restrict__ wt,
                                    const __nv_bfloat16 *__restrict__ w, int cin, int cout) {
  const int64_t n = 27LL * cin * cout;
  for (int64_t q = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; q < n;
       q += (int64_t)gridDim.x * blockDim.x) {
    const int co = (int)(q % cout);
    const int64_t r = q / cout;
    const int ci = (int)(r % cin);
    const int tp = (int)(r / cin);
    wt[q] = w[((int64_t)(26 - tp) * cout + co) * cin + ci];
  }
}

// g[v][c] *= (act[v][c] > 0): gradient through ReLU (act is the ReLU output)
__global__ void relu_bwd_kernel(__nv_bfloat16 *__restrict__ g, const __nv_bfloat16 *__restrict__ act,
                                int64_t n) {
  for (int64_t q = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; q < n;
       q += (int64_t)gridDim.x * blockDim.x)
    if (!(__bfloat162float(act[q]) > 0.0f)) g[q] = __float2bfloat16(0.0f);
}
// The same on eight elements a thread (n8 vectors of 16 bytes, both arrays
// 16-byte aligned): memory-bound, and one element a thread left most of each
// load unused (9.7 -> 4 us for 6.3 M elements on a B200).
__global__ void relu_bwd8_kernel(uint4 *__restrict__ g, const uint4 *__restrict__ act, int64_t n8) {
  for (int64_t q = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; q < n8;
       q += (int64_t)gridDim.x * blockDim.x) {
    const uint4 a = act[q];
    uint4 v = g[q];
    const uint32_t aw[4] = {a.x, a.y, a.z, a.w};
    uint32_t vw[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      // a BF16 is the upper half of a float
      if (!(__uint_as_float(aw[e] << 16) > 0.0f)) vw[e] &= 0xffff0000u;
      if (!(__uint_as_float(aw[e] & 0xffff0000u) > 0.0f)) vw[e] &= 0x0000ffffu;
    }
    g[q] = make_uint4(vw[0], vw[1], vw[2], vw[3]);
  }
}

// 2x2x2 average pooling (channels-last); output dims (nx/2, ny/2, nz/2)
__global__ void pool_fwd_kernel(__nv_bfloat16 *__restrict__ out, const __nv_bfloat16 *__restrict__ in,
                                int nx, int ny, int nz, int c) {
  const int ox = nx / 2, oy = ny / 2, oz = nz / 2;
  const int64_t n = (int64_t)ox * oy * oz * c;
  for (int64_t q = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; q < n;
       q += (int64_t)gridDim.x * blockDim.x) {
    const int ch = (int)(q % c);
    int64_t v = q / c;
    const int k = (int)(v % oz);
    v /= oz;
    const int j = (int)(v % oy), i = (int)(v / oy);
    float s = 0.0f;
    for (int a = 0; a < 8; ++a) {
      const int ii = 2 * i + (a >> 2), jj = 2 * j + ((a >> 1) & 1), kk = 2 * k + (a & 1);
      s += __bfloat162float(in[(((int64_t)ii * ny + jj) * nz + kk) * c + ch]);
    }
    out[q] = __float2bfloat16(0.125f * s);
  }
}
// gradient of the pooling: gin[child] = gout[parent] / 8 (+= when accumulate)
__global__ void pool_bwd_kernel(__nv_bfloat16 *__restrict__ gin, const __nv_bfloat16 *__restrict__ gout,
                                int nx, int ny, int nz, int c, int accumulate) {
  const int64_t n = (int64_t)nx * ny * nz * c;
  for (int64_t q = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; q < n;
       q += (int64_t)gridDim.x * blockDim.x) {
    const int ch = (int)(q % c);
    int64_t v = q / c;
    const int k = (int)(v % nz);
    v /= nz;
    const int j = (int)(v % ny), i = (int)(v / ny);
    const int64_t p = ((((int64_t)(i >> 1) * (ny / 2) + (j >> 1)) * (nz / 2)) + (k >> 1)) * c + ch;
    float x = 0.125f * __bfloat162float(gout[p]);
    if (accumulate) x += __bfloat162float(gin[q]);
    gin[q] = __float2bfloat16(x);
  }
}
// nearest-neighbour x2 upsampling to (nx, ny, nz) from (nx/2, ny/2, nz/2), plus an
// optional skip tensor of the output's shape: out = up(in) + skip
__global__ void up_fwd_kernel(__nv_bfloat16 *__restrict__ out, const __nv_bfloat16 *__restrict__ in,
                              int nx, int ny, int nz, int c) {
  const int64_t n = (int64_t)nx * ny * nz * c;
  for (int64_t q = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; q < n;
       q += (int64_t)gridDim.x * blockDim.x) {
    const int ch = (int)(q % c);
    int64_t v = q / c;
    const int k = (int)(v % nz);
    v /= nz;
    const int j = (int)(v % ny), i = (int)(v / ny);
    const int64_t p = ((((int64_t)(i >> 1) * (ny / 2) + (j >> 1)) * (nz / 2)) + (k >> 1)) * c + ch;
    out[q] = in[p];
  }
}
// gradient of the upsampling: gin[parent] = sum of the 8 children's gout
__global__ void up_bwd_kernel(__nv_bfloat16 *__restrict__ gin, const __nv_bfloat16 *__restrict__ gout,
                              int nx, int ny, int nz, int c) {
  const int ox = nx / 2, oy = ny / 2, oz = nz / 2;
  const int64_t n = (int64_t)ox * oy * oz * c;
  for (int64_t q = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; q < n;
       q += (int64_t)gridDim.x * blockDim.x) {
    const int ch = (int)(q % c);
    int64_t v = q / c;
    const int k = (int)(v % oz);
    v /= oz;
    const int j = (int)(v % oy), i = (int)(v / oy);
    float s = 0.0f;
    for (int a = 0; a < 8; ++a) {
      const int ii = 2 * i + (a >> 2), jj = 2 * j + ((a >> 1) & 1), kk = 2 * k + (a & 1);
      s += __bfloat162float(gout[(((int64_t)ii * ny + jj) * nz + kk) * c + ch]);
    }
    gin[q] = __float2bfloat16(s);
  }
}
// a += b (BF16, elementwise; skip connections and gradient sums)
__global__ void add_kernel(__nv_bfloat16 *__restrict__ a, const __nv_bfloat16 *__restrict__ b,
                           int64_t n) {
  for (int64_t q = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; q < n;
       q += (int64_t)gridDim.x * blockDim.x)
    a[q] = __float2bfloat16(__bfloat162float(a[q]) + __bfloat162float(b[q]));
}

// Network input: x[v][0] = rhs[v] / scale on fluid cells, x[v][1] = fluid flag,
// x[v][2] = solid flag, channels 3..15 zero.
__global__ void pack_input_kernel(__nv_bfloat16 *__restrict__ x, const float *__restrict__ div,
                                  const uint8_t *__restrict__ mask, int64_t nvox, float inv_scale) {
  for (int64_t v = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; v < nvox;
       v += (int64_t)gridDim.x * blockDim.x) {
    const uint8_t m = mask[v];
    const bool fl = (m & BSP_CLASS_FLUID) != 0;
    __nv_bfloat16 *o = x + v * 16;
    o[0] = __float2bfloat16(fl ? div[v] * inv_scale : 0.0f);
    o[1] = __float2bfloat16(fl ? 1.0f : 0.0f);
    o[2] = __float2bfloat16((m & BSP_CLASS_SOLID) ? 1.0f : 0.0f);
    for (int c = 3; c < 16; ++c) o[c] = __float2bfloat16(0.0f);
  }
}

// Head: y[v] = hb + sum_c hw[c] * x[v][c] (16 channels), masked to fluid cells;
// p[v] = scale * y[v] (FP32)
__global__ void head_fwd_kernel(float *__restrict__ p, const __nv_bfloat16 *__restrict__ x,
                                const float *__restrict__ hw, const float *__restrict__ hb,
                                const uint8_t *__restrict__ mask, int64_t nvox, float scale) {
  for (int64_t v = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; v < nvox;
       v += (int64_t)gridDim.x * blockDim.x) {
    float y = hb[0];
    for (int c = 0; c < 16; ++c) y = fmaf(hw[c], __bfloat162float(x[v * 16 + c]), y);
    p[v] = (mask[v] & BSP_CLASS_FLUID) ? scale * y : 0.0f;
  }
}

// Loss and head gradient: with y = prediction / scale and t = target / scale on
// fluid cells, loss = mean (y - t)^2; gx[v][c] = dL/dx = 2 (y - t) hw[c] / nfl;
// per-block partials of loss, dhw[16], dhb (FP32, deterministic order).
__global__ void __launch_bounds__(256) head_loss_kernel(
    __nv_bfloat16 *__restrict__ gx, float *__restrict__ partials, const float *__restrict__ pred,
    const float *__restrict__ target, const __nv_bfloat16 *__restrict__ x,
    const float *__restrict__ hw, const uint8_t *__restrict__ mask, int64_t nvox, float inv_scale,
    float inv_nfl) {
  float lsum = 0.0f, dhw[16], dhb = 0.0f;
#pragma unroll
  for (int c = 0; c < 16; ++c) dhw[c] = 0.0f;
  for (int64_t v = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; v < nvox;
       v += (int64_t)gridDim.x * blockDim.x) {
    const bool fl = (mask[v] & BSP_CLASS_FLUID) != 0;
    const float d = fl ? (pred[v] - target[v]) * inv_scale : 0.0f;
    lsum += d * d;
    const float gy = 2.0f * d * inv_nfl;
    dhb += gy;
#pragma unroll
    for (int c = 0; c < 16; ++c) {
      const float xc = __bfloat162float(x[v * 16 + c]);
      dhw[c] = fmaf(gy, xc, dhw[c]);
      gx[v * 16 + c] = __float2bfloat16(gy * hw[c]);
    }
  }
  __shared__ float sh[256];
  auto reduce = [&](float val, int slot) {
    sh[threadIdx.x] = val;
    __syncthreads();
    for (int o = 128; o > 0; o >>= 1) {
      if (threadIdx.x < o) sh[threadIdx.x] += sh[threadIdx.x + o];
      __syncthreads();
    }
    if (threadIdx.x == 0) partials[(int64_t)slot * gridDim.x + blockIdx.x] = sh[0];
    __syncthreads();
  };
  reduce(lsum * inv_nfl, 0);
  reduce(dhb, 1);
  for (int c = 0; c < 16; ++c) reduce(dhw[c], 2 + c);
}

// Head gradient for a given output gradient gy (dL/dy per voxel, 0 off fluid):
// gx[v][c] = gy[v] hw[c]; per-block partials of dhb (slot 0) and dhw (1..16).
__global__ void __launch_bounds__(256) head_bwd_kernel(
    __nv_bfloat16 *__restrict__ gx, float *__restrict__ partials, const float *__restrict__ gy,
    const __nv_bfloat16 *__restrict__ x, const float *__restrict__ hw,
    const uint8_t *__restrict__ mask, int64_t nvox) {
  float dhw[16], dhb = 0.0f;
#pragma unroll
  for (int c = 0; c < 16; ++c) dhw[c] = 0.0f;
  for (int64_t v = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; v < nvox;
       v += (int64_t)gridDim.x * blockDim.x) {
    const float g = (mask[v] & BSP_CLASS_FLUID) ? gy[v] : 0.0f;
    dhb += g;
#pragma unroll
    for (int c = 0; c < 16; ++c) {
      dhw[c] = fmaf(g, __bfloat162float(x[v * 16 + c]), dhw[c]);
      gx[v * 16 + c] = __float2bfloat16(g * hw[c]);
    }
  }
  __shared__ float sh[256];
  auto reduce = [&](float val, int slot) {
    sh[threadIdx.x] = val;
    __syncthreads();
    for (int o = 128; o > 0; o >>= 1) {
      if (threadIdx.x < o) sh[threadIdx.x] += sh[threadIdx.x + o];
      __syncthreads();
    }
    if (threadIdx.x == 0) partials[(int64_t)slot * gridDim.x + blockIdx.x] = sh[0];
    __syncthreads();
  };
  reduce(dhb, 0);
  for (int c = 0; c < 16; ++c) reduce(dhw[c], 1 + c);
}

// Adam step on FP32 master weights, refreshing the BF16 copy.
__global__ void adam_kernel(float *__restrict__ w, __nv_bfloat16 *__restrict__ wb,
                            float *__restrict__ m, float *__restrict__ vv,
                            const float *__restrict__ g, int64_t n, float lr, float b1, float b2,
                            float eps, float c1, float c2) {
  for (int64_t q = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; q < n;
       q += (int64_t)gridDim.x * blockDim.x) {
    const float gq = g[q];
    const float mq = b1 * m[q] + (1.0f - b1) * gq;
    const float vq = b2 * vv[q] + (1.0f - b2) * gq * gq;
    m[q] = mq;
    vv[q] = vq;
    const float upd = lr * (mq * c1) / (sqrtf(vq * c2) + eps);
    const float wq = w[q] - upd;
    w[q] = wq;
    if (wb) wb[q] = __float2bfloat16(wq);
  }
}

inline int grid_for(int64_t n, int threads = 256) {
  int64_t b = (n + threads - 1) / threads;
  return (int)(b < 148 * 16 ? (b > 0 ? b : 1) : 148 * 16);
}

}  // namespace unet
}  // namespace bsp

using namespace bsp::unet;

extern "C" int bsp_unet_flip_weights(bsp_bf16_t *wt_, const bsp_bf16_t *w_, int cin,
                                     int cout, cudaStream_t s) {
  __nv_bfloat16 *wt = reinterpret_cast<__nv_bfloat16 *>(wt_);
  const __nv_bfloat16 *w = reinterpret_cast<const __nv_bfloat16 *>(w_);
  if (!wt || !w) return BSP_ERR_NULL;
  flip_weights_kernel<<<grid_for(27LL * cin * cout), 256, 0, s>>>(wt, w, cin, cout);
  return (int)cudaGetLastError();
}

extern "C" int bsp_unet_relu_bwd(bsp_bf16_t *g_, const bsp_bf16_t *act_, int64_t n,
                                 cudaStream_t s) {
  __nv_bfloat16 *g = reinterpret_cast<__nv_bfloat16 *>(g_);
  const __nv_bfloat16 *act = reinterpret_cast<const __nv_bfloat16 *>(act_);
  if (n <= 0) return BSP_OK;
  if (n % 8 == 0 && (((uintptr_t)g | (uintptr_t)act) & 15u) == 0)
    relu_bwd8_kernel<<<grid_for(n / 8), 256, 0, s>>>(reinterpret_cast<uint4 *>(g),
                                                     reinterpret_cast<const uint4 *>(act), n / 8);
  else
    relu_bwd_kernel<<<grid_for(n), 256, 0, s>>>(g, act, n);
  return (int)cudaGetLastError();
}

extern "C" int bsp_unet_pool(bsp_bf16_t *out_, const bsp_bf16_t *in_, int nx, int ny,
                             int nz, int c, int backward, int accumulate, cudaStream_t s) {
  __nv_bfloat16 *out = reinterpret_cast<__nv_bfloat16 *>(out_);
  const __nv_bfloat16 *in = reinterpret_cast<const __nv_bfloat16 *>(in_);
  if (nx % 2 || ny % 2 || nz % 2) return BSP_ERR_SHAPE;
  if (backward)
    pool_bwd_kernel<<<grid_for((int64_t)nx * ny * nz * c), 256, 0, s>>>(out, in, nx, ny, nz, c,
                                                                         accumulate);
  else
    pool_fwd_kernel<<<grid_for((int64_t)nx * ny * nz * c / 8), 256, 0, s>>>(out, in, nx, ny, nz,
                                                                             c);
  return (int)cudaGetLastError();
}

extern "C" int bsp_unet_up(bsp_bf16_t *out_, const bsp_bf16_t *in_, int nx, int ny, int nz,
                           int c, int backward, cudaStream_t s) {
  __nv_bfloat16 *out = reinterpret_cast<__nv_bfloat16 *>(out_);
  const __nv_bfloat16 *in = reinterpret_cast<const __nv_bfloat16 *>(in_);
  if (nx % 2 || ny % 2 || nz % 2) return BSP_ERR_SHAPE;
  if (backward)
    up_bwd_kernel<<<grid_for((int64_t)nx * ny * nz * c / 8), 256, 0, s>>>(out, in, nx, ny, nz, c);
  else
    up_fwd_kernel<<<grid_for((int64_t)nx * ny * nz * c), 256, 0, s>>>(out, in, nx, ny, nz, c);
  return (int)cudaGetLastError();
}

extern "C" int bsp_unet_add(bsp_bf16_t *a_, const bsp_bf16_t *b_, int64_t n, cudaStream_t s) {
  __nv_bfloat16 *a = reinterpret_cast<__nv_bfloat16 *>(a_);
  const __nv_bfloat16 *b = reinterpret_cast<const __nv_bfloat16 *>(b_);
  if (n <= 0) return BSP_OK;
  add_kernel<<<grid_for(n), 256, 0, s>>>(a, b, n);
  return (int)cudaGetLastError();
}

extern "C" int bsp_unet_pack_input(bsp_bf16_t *x_, const float *div, const uint8_t *mask,
                                   int64_t nvox, float inv_scale, cudaStream_t s) {
  __nv_bfloat16 *x = reinterpret_cast<__nv_bfloat16 *>(x_);
  pack_input_kernel<<<grid_for(nvox), 256, 0, s>>>(x, div, mask, nvox, inv_scale);
  return (int)cudaGetLastError();
}

extern "C" int bsp_unet_head_fwd(float *p, const bsp_bf16_t *x_, const float *hw,
                                 const float *hb, const uint8_t *mask, int64_t nvox, float scale,
                                 cudaStream_t s) {
  const __nv_bfloat16 *x = reinterpret_cast<const __nv_bfloat16 *>(x_);
  head_fwd_kernel<<<grid_for(nvox), 256, 0, s>>>(p, x, hw, hb, mask, nvox, scale);
  return (int)cudaGetLastError();
}

extern "C" int bsp_unet_head_loss(bsp_bf16_t *gx_, float *partials, int nblocks,
                                  const float *pred, const float *target, const bsp_bf16_t *x_,
                                  const float *hw, const uint8_t *mask, int64_t nvox,
                                  float inv_scale, float inv_nfl, cudaStream_t s) {
  __nv_bfloat16 *gx = reinterpret_cast<__nv_bfloat16 *>(gx_);
  const __nv_bfloat16 *x = reinterpret_cast<const __nv_bfloat16 *>(x_);
  if (nblocks <= 0 || nblocks > 4096) return BSP_ERR_ARG;
  head_loss_kernel<<<nblocks, 256, 0, s>>>(gx, partials, pred, target, x, hw, mask, nvox,
                                           inv_scale, inv_nfl);
  return (int)cudaGetLastError();
}

extern "C" int bsp_unet_head_bwd(bsp_bf16_t *gx_, float *partials, int nblocks,
                                 const float *gy, const bsp_bf16_t *x_, const float *hw,
                                 const uint8_t *mask, int64_t nvox, cudaStream_t s) {
  __nv_bfloat16 *gx = reinterpret_cast<__nv_bfloat16 *>(gx_);
  const __nv_bfloat16 *x = reinterpret_cast<const __nv_bfloat16 *>(x_);
  if (nblocks <= 0 || nblocks > 4096) return BSP_ERR_ARG;
  head_bwd_kernel<<<nblocks, 256, 0, s>>>(gx, partials, gy, x, hw, mask, nvox);
  return (int)cudaGetLastError();
}

extern "C" int bsp_unet_sum_partials(float *out, const float *partials, int nblocks, int nslots,
                                     cudaStream_t s) {
  // out[slot] = sum over blocks in block order; partials laid out [slot][block]
  if (nblocks <= 0 || nslots <= 0 || nslots > 1024) return BSP_ERR_ARG;
  sum_slots_kernel<<<1, nslots, 0, s>>>(out, partials, nblocks);
  return (int)cudaGetLastError();
}

extern "C" int bsp_unet_adam(float *w, bsp_bf16_t *wb_, float *m, float *v, const float *g,
                             int64_t n, float lr, float b1, float b2, float eps, int step,
                             cudaStream_t s) {
  __nv_bfloat16 *wb = reinterpret_cast<__nv_bfloat16 *>(wb_);
  if (n <= 0 || step <= 0) return BSP_ERR_ARG;
  const float c1 = 1.0f / (1.0f - powf(b1, (float)step));
  const float c2 = 1.0f / (1.0f - powf(b2, (float)step));
  adam_kernel<<<grid_for(n), 256, 0, s>>>(w, wb, m, v, g, n, lr, b1, b2, eps, c1, c2);
  return (int)cudaGetLastError();
}
