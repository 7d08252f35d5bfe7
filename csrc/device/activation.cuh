// silu(gate) * up in fp32, the one formula of every kernel that applies it: the stand-alone activation, the split-K sum and the
// GEMM epilogues.  A problem may take any of them by its shape, so the rounding of the result must not depend on which.
// The division is the IEEE one: in the GEMM epilogues it hides behind the next tile's products or the weights' stream.
#pragma once

namespace oob {

__device__ __forceinline__ float swiglu_f32(float g, float u) { return g / (1.f + __expf(-g)) * u; }

}  // namespace oob
