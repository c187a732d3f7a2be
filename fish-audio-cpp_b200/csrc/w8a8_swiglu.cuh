// silu(gate) * up of the fused epilogues, with the roundings of the reference's GEMM, silu, GEMM, mul chain
// (ffn_activations.cu:12-17, :35-40): gate, up and silu(gate) are fp16 before they are used.
#pragma once

#include <cuda_fp16.h>

namespace w8a8 {

// x / (1 + exp(-x)) for an x that is an fp16 number. The quotient is an approximate reciprocal's, corrected once by its residual
// (Markstein, IBM J. Res. Dev. 34, 1990); rounded to fp16 it is the divide's for every one of the 65536 arguments (tested:
// test_fused_swiglu_of_every_gate, and for -0 test_fused_swiglu_of_gates_that_round_to_zero). Large denominators are cut off where the
// result has long been zero in fp16, so that nothing becomes infinite on the way; an infinite x gives what the divide gives.
// Why: with the divide it was the longest part of a tile's end. A 256 x 256 tile at g = 256 now ends in 3130 clocks, 1090 without the
// SwiGLU, after ten K-groups of 1451 (stamps of the clock). w1|w3 at g = 256, with all that changed since the divide, 150 tokens 30.0 ->
// 19.4 us and 8192 tokens 447 -> 393; rows without SwiGLU 7.2 -> 7.3 (6144, 150 tokens) and 126 -> 125 (8192).
// (The decode linears keep the divide: a launch there has one tile's worth per CTA, and ten fast-AR steps took 1553 us with the
// divide, 1559 without.)
__device__ __forceinline__ float silu_of_half(float x) {
    const float d = 1.0f + fminf(expf(-x), 0x1p100f);
    float r, n;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(d));
    asm("min.NaN.f32 %0, %1, %2;" : "=f"(n) : "f"(x), "f"(131072.0f));
    const float q = n * r;
    return fmaf(-fmaf(d, q, -n), r, q);  // (in these signs -0 stays -0)
}
// Two channels or tokens at once; the product of two fp16 numbers rounded once is the same in fp16 as by way of fp32.
__device__ __forceinline__ __half2 swiglu2(__half2 gate, __half2 up) {
    const float2 g = __half22float2(gate);
    return __hmul2_rn(__floats2half2_rn(silu_of_half(g.x), silu_of_half(g.y)), up);
}

}  // namespace w8a8
