// Arithmetic of SwiGLU, shared by the stand-alone kernels (elementwise.cu) and the GEMM epilogues
// (gemm_sm100.cu) so that both give bitwise the same result.
#pragma once

namespace ft {

// act = silu(g) * u;  d g = d * sig * (1 + g (1 - sig)) * u;  d u = d * g * sig
__device__ __forceinline__ void swiglu_bwd_elem(float d, float g, float u, float& dg, float& du) {
  const float sig = __fdividef(1.f, 1.f + __expf(-g));
  dg = d * sig * (1.f + g * (1.f - sig)) * u;
  du = d * g * sig;
}

// act = silu(g) * u
__device__ __forceinline__ float swiglu_fwd_elem(float g, float u) {
  const float sig = 1.f / (1.f + __expf(-g));
  return g * sig * u;
}

// Four activations, rounded to bf16 and packed: the bits of swiglu_fwd_elem, mostly without its
// division, whose range check is a branch per value: values one after the other, 150 cycles each,
// in an epilogue that has two warps per scheduler to hide them. The quick quotient is off by at most
// 2 ulp (CUDA's bound for denominators up to 2^126), the four products of the two variants by a
// rounding each, so the results differ by at most 4.5 * 2^-23 of the value, 9 ulp. Unless the quick
// one lies within 10 ulp of the middle between two bf16 values (one group of four in a warp out of
// 24), both round to the same bf16; otherwise, and for gates below -80 or NaN, the group is redone.
// FC1 + SwiGLU kernel, 0.5B: 256 / 2048 / 16384 tokens 17.8 -> 13.1, 43.4 -> 35.7, 255 -> 228 us.
__device__ __forceinline__ void swiglu_fwd_pack4(uint32_t g01, uint32_t g23, uint32_t u01,
                                                 uint32_t u23, uint32_t& a01, uint32_t& a23) {
  const float g[4] = {bf16_lo(g01), bf16_hi(g01), bf16_lo(g23), bf16_hi(g23)};
  const float u[4] = {bf16_lo(u01), bf16_hi(u01), bf16_lo(u23), bf16_hi(u23)};
  float a[4];
  bool redo = false;
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    a[i] = g[i] * __fdividef(1.f, 1.f + __expf(-g[i])) * u[i];
    redo |= ((__float_as_uint(a[i]) & 0xffffu) - (0x8000u - 10u) <= 20u) | !(g[i] > -80.f);
  }
  if (redo) {
#pragma unroll
    for (int i = 0; i < 4; ++i) a[i] = swiglu_fwd_elem(g[i], u[i]);
  }
  a01 = pack_bf16x2(a[0], a[1]);
  a23 = pack_bf16x2(a[2], a[3]);
}

}  // namespace ft
