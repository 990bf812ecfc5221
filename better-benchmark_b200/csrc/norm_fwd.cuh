// Pieces shared by the translation units of the LayerNorm / RMSNorm forward: the parameter block, the GELU prologue, the choice between
// the two forms of a residual sum, and the kernels for rows off the 16-byte grid (norm_fwd_span.cu).
#pragma once

#include "rowwise.cuh"

#include <type_traits>

namespace b200 {

struct NormFwdParams {
  const void* x;
  const void* w;  // may be null
  const void* b;  // may be null
  void* y;        // may be null
  float* mean_out;
  float* rstd_out;
  float* var_out;
  long long rows;
  int n;
  long long x_row_stride, y_row_stride;  // elements
  int w_dtype;
  float eps;
  float inv_n;      // 1 / n
  float inv_denom;  // 1 / (n - correction)
  int rms;
  int prologue;     // 0: none; 1: exact (erf) GELU of x, rounded to x's dtype, is what gets normalised
  // Residual prologue (the post-LayerNorm blocks, repros/canonical/var_mean_0ada225c0a04/repro.py:26-27):
  // what gets normalised is T(x + res); res has x's dtype and row stride. sum_out (may be null)
  // receives that rounded sum, rows of n elements, contiguous.
  const void* res;
  void* sum_out;
  // 1: the sum is rounded to x's dtype before it is normalised, as the eager graph materialises it;
  // 0: it stays in fp32, as in Inductor's fused kernel - the form the reference's fp64-anchored gate
  // accepts (the fp64 evaluation of the graph has no such rounding);
  // 2 (what the stubs use; LayerNorm of 16-bit tensors): both rows are normalised, each with its own
  // statistics, and every element takes the fp32 form where that form's rounded output exceeds 3 in
  // magnitude and the rounded form elsewhere - the rule of the reference's oracle for these regions
  // (repros/canonical/var_mean_45f7dfd4a983/oracle.py:96-107). Small outputs then equal the eager
  // module's (its element-wise check allows 1e-2 + 1e-2 |y|, less than two 16-bit steps between 1.3
  // and 2 and between 2.6 and 4), large ones, which decide the maximum error against the fp64 graph,
  // carry no intermediate rounding. The statistics that are returned are those of the fp32 sum.
  int res_round;
};

// Pointwise prologue of the LayerNorm regions that normalise an activation
// (repros/canonical/var_mean_af505388b035/repro.py:27-33): (x * 0.5) * (erf(x * 0.7071067811865476) + 1)
// in fp32, in that order, then rounded to the tensor dtype - the graph materialises the
// activation as a 16-bit tensor before the statistics are taken.
// (16-bit tensors: gelu_pair, whose fp32 result is as close to the fp64 one as that expression's.)
template <typename Tin>
__device__ __forceinline__ f32x2 gelu_erf_rounded2(f32x2 v) {
  if constexpr (sizeof(Tin) == 2) {
    return Pairs<Tin>::word(Pairs<Tin>::narrow(gelu_pair(v)));
  } else {
    float a, b;
    unpack2(v, a, b);
    return pack2((a * 0.5f) * (erff(a * 0.7071067811865476f) + 1.0f), (b * 0.5f) * (erff(b * 0.7071067811865476f) + 1.0f));
  }
}
template <typename Tin>
__device__ __forceinline__ float gelu_erf_rounded(float x) {
  float a, b;
  unpack2(gelu_erf_rounded2<Tin>(splat2(x)), a, b);
  return a;
}

// rsqrtf is the 2-ulp hardware approximation aten's CUDA rsqrt uses as well.
__device__ __forceinline__ float precise_rsqrt(float v) { return rsqrtf(v); }

// |a| > 3 per 16-bit half: all ones or zeros (zeros for NaN)
template <typename T>
__device__ __forceinline__ uint32_t beyond_three(uint32_t a) {
  if constexpr (std::is_same<T, __half>::value) {
    return __hgt2_mask(__habs2(*reinterpret_cast<const __half2*>(&a)), __float2half2_rn(3.0f));
  } else {
    return __hgt2_mask(__habs2(*reinterpret_cast<const __nv_bfloat162*>(&a)), __float2bfloat162_rn(3.0f));
  }
}

// Rows off the 16-byte grid whose results have their alignment (norm_fwd_span.cu). False: the caller takes another kernel.
template <typename T>
bool try_launch_norm_fwd_span(const NormFwdParams& p, cudaStream_t st);

}  // namespace b200
