// silu(gate) * up in fp32, the one function of every kernel that applies it: the stand-alone activation, the split-K sum and the
// GEMM epilogues.  A problem may take any of them by its shape, so the bits of the result must not depend on which.
#pragma once
#include <cstdint>

namespace oob {

__device__ __forceinline__ float swiglu_f32(float g, float u) { return g / (1.f + __expf(-g)) * u; }

// The same for N values held in registers, g[i] = silu(g[i]) * u[i] (bits of fp32).  The division operator branches for each value,
// which in a GEMM epilogue left one division at a time in flight: 300 x 57344 x 1024 took 201 us, 54 with this (51 with the
// approximate division, good to two units of the last place).  Here the quotient is Newton's reciprocal with Markstein's correction by the remainder (P. Markstein, Computation of
// elementary functions on the IBM RISC System/6000, 1990), straight-line code for all values at once.  Up to 80 in magnitude the
// denominator and its reciprocal are normal numbers and the quotient has the bits of the operator's (checked for every fp32
// gate); beyond, infinities and NaN included, the operator is used.
template <int N>
__device__ __forceinline__ void swiglu_n(uint32_t (&g)[N], const uint32_t (&u)[N]) {
  bool inside = true;
#pragma unroll
  for (int i = 0; i < N; ++i) inside = inside && fabsf(__uint_as_float(g[i])) < 80.f;
  if (inside) {
#pragma unroll
    for (int i = 0; i < N; ++i) {
      const float x = __uint_as_float(g[i]), d = 1.f + __expf(-x);
      float r;
      asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(d));
      r = fmaf(r, fmaf(-d, r, 1.f), r);
      float q = x * r;
      q = copysignf(fmaf(fmaf(-d, q, x), r, q), x);  // the sign of a zero
      g[i] = __float_as_uint(q * __uint_as_float(u[i]));
    }
  } else {
    // Rare: one copy of the operator's code, values through local memory.
    float x[N], y[N];
#pragma unroll
    for (int i = 0; i < N; ++i) {
      x[i] = __uint_as_float(g[i]);
      y[i] = __uint_as_float(u[i]);
    }
#pragma unroll 1
    for (int i = 0; i < N; ++i) x[i] = swiglu_f32(x[i], y[i]);
#pragma unroll
    for (int i = 0; i < N; ++i) g[i] = __float_as_uint(x[i]);
  }
}

}  // namespace oob
