// f32x2.cuh -- packed pairs of FP32 (add / mul / fma.rn.f32x2, sm_100): each half
// is rounded on its own, to nearest even, so results equal the scalar
// instructions bit for bit at half the instruction count.
#pragma once
#include <cstdint>

#include "bsp_common.cuh"

namespace bsp {

__device__ __forceinline__ uint64_t add2(uint64_t a, uint64_t b) {
  uint64_t d;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
  return d;
}
__device__ __forceinline__ uint64_t mul2(uint64_t a, uint64_t b) {
  uint64_t d;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
  return d;
}
__device__ __forceinline__ uint64_t fma2(uint64_t a, uint64_t b, uint64_t c) {
  uint64_t d;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
  return d;
}
__device__ __forceinline__ uint64_t pack2(float lo, float hi) {
  uint64_t d;
  asm("mov.b64 %0, {%1, %2};" : "=l"(d) : "f"(lo), "f"(hi));
  return d;
}
__device__ __forceinline__ void unpack2(uint64_t a, float &lo, float &hi) {
  asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(a));
}
// Four consecutive cells.
struct Quad {
  uint64_t a, b;  // cells 0, 1 and 2, 3
};
__device__ __forceinline__ void cells(const Quad &v, float (&c)[4]) {
  unpack2(v.a, c[0], c[1]);
  unpack2(v.b, c[2], c[3]);
}
__device__ __forceinline__ Quad quad(const float (&c)[4]) {
  return Quad{pack2(c[0], c[1]), pack2(c[2], c[3])};
}

// (s - rhs) / 6 of four cells: s - rhs as fma(rhs, -1, s), the quotient as in
// div6 (bsp_common.cuh); where some |s - rhs| is 0, below 2^-119, huge, inf or
// NaN, the full div6.
__device__ __forceinline__ Quad div6_quad(const Quad &s, const Quad &rhs) {
  const uint64_t Z2 = pack2(0.16666667163372039795f, 0.16666667163372039795f);  // RN(1/6)
  const uint64_t N6 = pack2(-6.0f, -6.0f), N1 = pack2(-1.0f, -1.0f);
  const Quad y{fma2(rhs.a, N1, s.a), fma2(rhs.b, N1, s.b)};
  const Quad h{mul2(y.a, Z2), mul2(y.b, Z2)};
  Quad v{fma2(fma2(h.a, N6, y.a), Z2, h.a), fma2(fma2(h.b, N6, y.b), Z2, h.b)};
  float c[4];
  cells(y, c);
  uint32_t lo = 0xffffffffu, hi = 0u;  // top five exponent bits: none all zero or all one
#pragma unroll
  for (int e = 0; e < 4; ++e) {
    const uint32_t u = __float_as_uint(c[e]) & 0x7c000000u;
    lo = min(lo, u);
    hi = max(hi, u);
  }
  if (lo == 0u || hi == 0x7c000000u) {
#pragma unroll
    for (int e = 0; e < 4; ++e) c[e] = div6(c[e]);
    v = quad(c);
  }
  return v;
}

}  // namespace bsp
