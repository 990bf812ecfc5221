// Helpers shared by the row-wise families (row reductions, softmax, LayerNorm/RMSNorm forward).
//
// Work decomposition: a "group" of threads owns one row. The group is one warp (short rows,
// several rows per CTA, no block barrier) or the whole CTA (long rows). A row of n elements is
// nv = n / V sixteen-byte vectors; vector j belongs to group lane j % G and register slot j / G,
// so each slot is one fully coalesced G x 16-byte access and all of a thread's loads are issued
// before the first is consumed.
#pragma once

#include "common.cuh"

#include <cstdlib>

namespace b200 {

// Division by a run-time constant without a divide instruction: q = umulhi(n, mul) >> shr for
// 0 <= n < 2^31 (host side picks mul/shr for the divisor d >= 1).
struct FastDiv {
  unsigned int mul, shr, d;
};

inline FastDiv make_fast_div(long long d) {
  FastDiv f;
  f.d = (unsigned int)d;
  if (d <= 1) {
    f.mul = 0;
    f.shr = 0;
    return f;
  }
  unsigned int lg = 0;
  while ((1ull << lg) < (unsigned long long)d) ++lg;  // ceil(log2 d)
  const unsigned int p = 31 + lg;
  f.mul = (unsigned int)(((1ull << p) + (unsigned long long)d - 1) / (unsigned long long)d);
  f.shr = p - 32;
  return f;
}

__device__ __forceinline__ unsigned int fast_div(unsigned int n, const FastDiv& f) {
  return f.d == 1 ? n : (__umulhi(n, f.mul) >> f.shr);
}

// Maps a flat row index onto up to three outer dimensions with arbitrary element strides, so
// broadcast operands (stride 0) and non-contiguous views need no copy. row = (i0*d1 + i1)*d2 + i2.
// Rows are limited to 2^31 - 1 (checked by the host).
struct RowMap {
  long long s0, s1, s2;
  FastDiv d1, d2;
};

inline RowMap make_row_map_flat(long long row_stride) {
  RowMap m;
  m.s0 = row_stride;
  m.s1 = m.s2 = 0;
  m.d1 = make_fast_div(1);
  m.d2 = make_fast_div(1);
  return m;
}

// A tensor whose rows lie at one distance gets the flat map although the call has several outer dimensions (another
// operand, a broadcast mask, needs them): its loads then start without the divisions (softmax_resident_kernel).
inline RowMap make_row_map(const int64_t* strides, long long d1, long long d2) {
  if (d1 == 1 && d2 == 1) return make_row_map_flat(strides[0]);
  if (d2 == 1 && strides[0] == strides[1] * d1) return make_row_map_flat(strides[1]);
  if (d1 == 1 && strides[0] == strides[2] * d2) return make_row_map_flat(strides[2]);
  if (strides[1] == strides[2] * d2 && strides[0] == strides[1] * d1) return make_row_map_flat(strides[2]);
  RowMap m;
  m.s0 = strides[0];
  m.s1 = strides[1];
  m.s2 = strides[2];
  m.d1 = make_fast_div(d1);
  m.d2 = make_fast_div(d2);
  return m;
}

__device__ __forceinline__ long long row_offset(const RowMap& m, long long row) {
  if (m.d1.d == 1 && m.d2.d == 1) return row * m.s0;
  const unsigned int r = (unsigned int)row;
  const unsigned int t = fast_div(r, m.d2);
  const unsigned int i2 = r - t * m.d2.d;
  const unsigned int i0 = fast_div(t, m.d1);
  const unsigned int i1 = t - i0 * m.d1.d;
  return (long long)i0 * m.s0 + (long long)i1 * m.s1 + (long long)i2 * m.s2;
}

// ----------------------------------------------------------------------------------------------
// Packed fp32 pairs. sm_100 executes add/sub/mul/fma on two fp32 values held in one 64-bit
// register pair as ONE instruction (same per-lane arithmetic throughput, half the issue slots),
// with round-to-nearest on each half: numerically identical to the two scalar operations.
// ----------------------------------------------------------------------------------------------
typedef unsigned long long f32x2;

__device__ __forceinline__ f32x2 pack2(float a, float b) {
  f32x2 r;
  asm("mov.b64 %0, {%1,%2};" : "=l"(r) : "f"(a), "f"(b));
  return r;
}
__device__ __forceinline__ void unpack2(f32x2 v, float& a, float& b) {
  asm("mov.b64 {%0,%1}, %2;" : "=f"(a), "=f"(b) : "l"(v));
}
__device__ __forceinline__ f32x2 splat2(float a) { return pack2(a, a); }
__device__ __forceinline__ f32x2 add2(f32x2 a, f32x2 b) {
  f32x2 r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ f32x2 sub2(f32x2 a, f32x2 b) {
  f32x2 r;
  asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ f32x2 mul2(f32x2 a, f32x2 b) {
  f32x2 r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
// a*b+c with a single rounding per half: only where the evaluated graph has no separate
// multiply and add to mirror (polynomial/compensation steps, sums of squares for statistics).
__device__ __forceinline__ f32x2 fma2(f32x2 a, f32x2 b, f32x2 c) {
  f32x2 r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
  return r;
}

// 16-byte vector <-> packed fp32 pairs, converted word by word so that each pair is born in (and
// consumed from) an aligned register pair instead of being assembled from two scalars.
template <typename T>
struct Pairs;

template <>
struct Pairs<float> {
  static __device__ __forceinline__ void unpack(const uint4& r, f32x2 (&v)[2]) {
    asm("mov.b64 %0, {%1,%2};" : "=l"(v[0]) : "r"(r.x), "r"(r.y));
    asm("mov.b64 %0, {%1,%2};" : "=l"(v[1]) : "r"(r.z), "r"(r.w));
  }
  static __device__ __forceinline__ uint4 pack(const f32x2 (&v)[2]) {
    uint4 r;
    asm("mov.b64 {%0,%1}, %2;" : "=r"(r.x), "=r"(r.y) : "l"(v[0]));
    asm("mov.b64 {%0,%1}, %2;" : "=r"(r.z), "=r"(r.w) : "l"(v[1]));
    return r;
  }
};

template <>
struct Pairs<__nv_bfloat16> {
  static __device__ __forceinline__ f32x2 word(uint32_t w) {
    f32x2 r;  // bf16 -> fp32: the low element is a 16-bit shift, the high one a mask
    asm("{\n\t.reg .b32 lo, hi;\n\tshl.b32 lo, %1, 16;\n\tand.b32 hi, %1, 0xffff0000;\n\tmov.b64 %0, {lo,hi};\n\t}"
        : "=l"(r) : "r"(w));
    return r;
  }
  static __device__ __forceinline__ void unpack(const uint4& r, f32x2 (&v)[4]) {
    v[0] = word(r.x); v[1] = word(r.y); v[2] = word(r.z); v[3] = word(r.w);
  }
  static __device__ __forceinline__ uint32_t narrow(f32x2 v) {
    uint32_t r;
    asm("{\n\t.reg .b32 lo, hi;\n\tmov.b64 {lo,hi}, %1;\n\tcvt.rn.bf16x2.f32 %0, hi, lo;\n\t}" : "=r"(r) : "l"(v));
    return r;
  }
  static __device__ __forceinline__ uint4 pack(const f32x2 (&v)[4]) {
    return make_uint4(narrow(v[0]), narrow(v[1]), narrow(v[2]), narrow(v[3]));
  }
};

template <>
struct Pairs<__half> {
  static __device__ __forceinline__ f32x2 word(uint32_t w) {
    f32x2 r;
    asm("{\n\t.reg .b16 a, b;\n\t.reg .b32 lo, hi;\n\tmov.b32 {a,b}, %1;\n\tcvt.f32.f16 lo, a;\n\tcvt.f32.f16 hi, b;\n\t"
        "mov.b64 %0, {lo,hi};\n\t}"
        : "=l"(r) : "r"(w));
    return r;
  }
  static __device__ __forceinline__ void unpack(const uint4& r, f32x2 (&v)[4]) {
    v[0] = word(r.x); v[1] = word(r.y); v[2] = word(r.z); v[3] = word(r.w);
  }
  static __device__ __forceinline__ uint32_t narrow(f32x2 v) {
    uint32_t r;
    asm("{\n\t.reg .b32 lo, hi;\n\tmov.b64 {lo,hi}, %1;\n\tcvt.rn.f16x2.f32 %0, hi, lo;\n\t}" : "=r"(r) : "l"(v));
    return r;
  }
  static __device__ __forceinline__ uint4 pack(const f32x2 (&v)[4]) {
    return make_uint4(narrow(v[0]), narrow(v[1]), narrow(v[2]), narrow(v[3]));
  }
};

// Sum of the two halves of a pair.
__device__ __forceinline__ float hsum2(f32x2 v) {
  float a, b;
  unpack2(v, a, b);
  return a + b;
}

// Natural exponential of a pair for results that are rounded to a 16-bit type afterwards.
//
// exp_pair_compensated (the default): y = x * log2(e) is rounded to fp32 (yh); what that rounding
// and the rounding of the constant lost is recovered exactly as r = x - yh * ln 2 with one fused
// multiply-add (the product is exact inside the fma; r is the error of the exponent in natural
// units, |r| < 2^-20), 2^yh comes from the hardware approximation (relative error 2^-22) and the
// result is 2^yh * (1 + r). Relative error below 3.5e-7 for arguments down to -17 (below 6e-7 over
// the whole range): the accuracy class of expf (2 ulp), three orders of magnitude below half a
// bf16/fp16 ulp. x * log2(e) must not overflow, which it does below -2.36e38 and for -inf: inf - inf inside
// the fma then gives NaN where the exponential is 0. Callers clamp to a floor above that first, or look for the NaN and take the
// elements again with the floor (softmax_rows_kernel). NaN stays NaN.
// .ftz: results below 2^-126 become 0 instead of denormals; nothing a 16-bit output or the row sum
// can see.
__device__ __forceinline__ f32x2 exp_pair_compensated(f32x2 x) {
  const f32x2 yh = mul2(x, splat2(1.4426950216293335f));   // x * fl(log2 e), rounded
  const f32x2 r = fma2(yh, splat2(-0.6931471824645996f), x);  // x - yh * ln 2
  f32x2 p;
  asm("{\n\t.reg .f32 a, b, pa, pb;\n\tmov.b64 {a,b}, %1;\n\tex2.approx.ftz.f32 pa, a;\n\t"
      "ex2.approx.ftz.f32 pb, b;\n\tmov.b64 %0, {pa,pb};\n\t}"
      : "=l"(p) : "l"(yh));
  return fma2(p, r, p);
}

// exp_pair_fast (opt-in, -DB200_SOFTMAX_FAST_EXP): 2^(x * log2 e) with the hardware approximation
// alone, which is what Triton's tl.exp lowers to. Relative error <= 2^-22 + |x * log2 e| * 2^-24 * ln 2:
// below 1.3e-6 wherever an fp16 result is not zero (x > -17) and below 6e-6 over the whole bf16
// range. Not the natural-exponential accuracy the eager graphs have; kept for measurements.
__device__ __forceinline__ f32x2 exp_pair_fast(f32x2 x) {
  const f32x2 y = mul2(x, splat2(1.4426950216293335f));
  f32x2 r;
  asm("{\n\t.reg .f32 a, b, pa, pb;\n\tmov.b64 {a,b}, %1;\n\tex2.approx.ftz.f32 pa, a;\n\t"
      "ex2.approx.ftz.f32 pb, b;\n\tmov.b64 %0, {pa,pb};\n\t}"
      : "=l"(r) : "l"(y));
  return r;
}

// Exact (erf-form) GELU of a pair, x * Phi(x), for results that are rounded to a 16-bit type afterwards.
//
// With a = |x| and Q(a) = erfc(a / sqrt 2) / 2 the normal distribution is Phi(x) = Q(a) for x < 0 and
// 1 - Q(a) otherwise, and Q(a) = exp(-a^2 / 2) * P(t), t = 1 / (1 + 0.305 a), P a polynomial without a
// constant term: the form of Hastings' approximations (Abramowitz & Stegun 26.2.17), here of degree
// eight with coefficients fitted to erfcx by iteratively reweighted least squares (relative error of Q
// below 9.5e-8 for 0 <= a <= 14). Over 2^24 standard normal inputs the 2-norm of the error of the 16-bit results agrees
// in six digits with that of the (x / 2) * (erff(x / sqrt 2) + 1) it replaces, and fewer of them are not the nearest value
// (bf16 5.5e-5 -> 0, fp16 2.7e-4 -> 6.1e-5; of fp16 inputs around 0.1, none -> 4.0e-4, by a
// thousandth of half a step). For x < -3, where erff + 1 cancels, only this form keeps the value (within half a
// 16-bit step over every bf16 and normal fp16 input). Fewer than half the instructions of erff. Measured:
// GELU bf16 [32768, 1536] 69.6 -> 50.1 us, GELU -> LayerNorm bf16 [65536, 768] 81.2 -> 67.4 us.
// a is clamped to 64 for the exponential, which needs finite arguments (Q(64) = 0); the product takes x
// itself, so that inf, -inf (NaN, as -inf * 0) and NaN come out as the graph has them.
__device__ __forceinline__ f32x2 gelu_pair(f32x2 x) {
  float x0, x1, r0, r1, q0, q1, u0, u1;
  unpack2(x, x0, x1);
  const f32x2 a = pack2(fminf(fabsf(x0), 64.f), fminf(fabsf(x1), 64.f));
  const f32x2 e = exp_pair_compensated(mul2(mul2(a, a), splat2(-0.5f)));
  unpack2(fma2(a, splat2(0.305f), splat2(1.0f)), r0, r1);
  asm("rcp.approx.ftz.f32 %0, %0;" : "+f"(r0));
  asm("rcp.approx.ftz.f32 %0, %0;" : "+f"(r1));
  const f32x2 t = pack2(r0, r1);
  f32x2 h = fma2(splat2(0.03669983148574829f), t, splat2(-0.1529906988143921f));
  h = fma2(h, t, splat2(0.1857205182313919f));
  h = fma2(h, t, splat2(-0.037979673594236374f));
  h = fma2(h, t, splat2(0.12102290987968445f));
  h = fma2(h, t, splat2(0.10342058539390564f));
  h = fma2(h, t, splat2(0.12246684730052948f));
  h = fma2(h, t, splat2(0.12163973599672318f));
  const f32x2 q = mul2(e, mul2(h, t));
  unpack2(q, q0, q1);
  unpack2(sub2(splat2(1.0f), q), u0, u1);
  return mul2(x, pack2(x0 < 0.f ? q0 : u0, x1 < 0.f ? q1 : u1));
}

// SiLU of a pair, x / (exp(-x) + 1), for results that are rounded to a 16-bit type afterwards: the
// compensated pair exponential (the accuracy class of expf) and a hardware reciprocal refined by one Newton
// step (correctly rounded but for rare last-bit cases): 1.5 fp32 ulp, three orders of magnitude below half
// an ulp of the output (over 2^24 normal inputs as many results are not the nearest as with a correctly
// rounded reciprocal: none from 16-bit inputs, 7e-6 of f32 -> bf16, 5e-5 of f32 -> f16). The denominator is formed as (e + 1) / 8, which rounds like e + 1 and keeps
// its reciprocal a normal number up to the largest e. The exponential needs finite arguments: -x is clamped
// to [-87, 88.7228], where e + 1 is 1 on the left and e just below the largest float on the right. Beyond
// that, where expf overflows, the reciprocal is 0 as in the graph: a finite x gives -0, -inf gives NaN.
// The SFU pipe (two exponentials and two reciprocals a pair) is what bounds it. Measured on bf16
// [32768, 1536]: 63.5 us with the correctly rounded software reciprocal, 47.1 us with this one.
// ANY false: the caller knows that |x| <= 88 (or NaN), where neither the clamp nor the zero can matter; the
// bits are the same.
template <bool ANY = true>
__device__ __forceinline__ f32x2 silu_pair(f32x2 x) {
  float a, b, d0, d1, r0, r1;
  unpack2(x, a, b);
  f32x2 minus = pack2(-a, -b);
  if constexpr (ANY) minus = pack2(fminf(fmaxf(-a, -87.f), 88.7228f), fminf(fmaxf(-b, -87.f), 88.7228f));
  const f32x2 e = exp_pair_compensated(minus);
  unpack2(fma2(e, splat2(0.125f), splat2(0.125f)), d0, d1);
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r0) : "f"(d0));
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r1) : "f"(d1));
  f32x2 r = pack2(r0, r1);
  r = fma2(r, fma2(fma2(e, splat2(-0.125f), splat2(-0.125f)), r, splat2(1.0f)), r);
  if constexpr (ANY) {
    unpack2(r, r0, r1);
    r = pack2(a < -88.72284f ? 0.f : r0, b < -88.72284f ? 0.f : r1);
  }
  return mul2(mul2(x, splat2(0.125f)), r);
}

template <bool BLOCK>
__device__ __forceinline__ int group_lane() {
  return BLOCK ? (int)threadIdx.x : (int)(threadIdx.x & 31);
}
template <bool BLOCK>
__device__ __forceinline__ int group_size() {
  return BLOCK ? (int)blockDim.x : 32;
}
template <bool BLOCK>
__device__ __forceinline__ long long group_row() {
  return BLOCK ? (long long)blockIdx.x
               : (long long)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
}

// Store N fp32 values as N elements of Tout with the widest store the byte count allows
// (N * sizeof(Tout) is 8, 16 or 32 and `p` is aligned to min(16, that)).
template <typename Tout, int N>
__device__ __forceinline__ void store_converted(Tout* p, const float (&f)[N]) {
  if constexpr (sizeof(Tout) == 4) {
#pragma unroll
    for (int i = 0; i < N / 4; ++i) {
      uint4 o = make_uint4(__float_as_uint(f[4 * i]), __float_as_uint(f[4 * i + 1]),
                           __float_as_uint(f[4 * i + 2]), __float_as_uint(f[4 * i + 3]));
      st_stream(reinterpret_cast<float*>(p) + 4 * i, o);
    }
  } else if constexpr (N == 8) {
    st_stream(p, Elem<Tout>::pack(f));
  } else {
    static_assert(N == 4, "unexpected vector length");
    uint32_t w[2];
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      if constexpr (sizeof(Tout) == 2) {
        Tout a = Elem<Tout>::from_f32(f[2 * i]);
        Tout b = Elem<Tout>::from_f32(f[2 * i + 1]);
        w[i] = (uint32_t)(*reinterpret_cast<unsigned short*>(&a)) |
               ((uint32_t)(*reinterpret_cast<unsigned short*>(&b)) << 16);
      }
    }
    asm volatile("st.global.cs.v2.u32 [%0], {%1,%2};" ::"l"(p), "r"(w[0]), "r"(w[1]) : "memory");
  }
}

// store_converted for values held as packed pairs (N values = N/2 pairs).
template <typename Tout, int N>
__device__ __forceinline__ void store_pairs(Tout* p, const f32x2 (&v)[N / 2]) {
  if constexpr (sizeof(Tout) == 4) {
#pragma unroll
    for (int i = 0; i < N / 4; ++i) {
      const f32x2 two[2] = {v[2 * i], v[2 * i + 1]};
      st_stream(reinterpret_cast<float*>(p) + 4 * i, Pairs<float>::pack(two));
    }
  } else if constexpr (N == 8) {
    st_stream(p, Pairs<Tout>::pack(v));
  } else {
    static_assert(N == 4, "unexpected vector length");
    const uint32_t w0 = Pairs<Tout>::narrow(v[0]), w1 = Pairs<Tout>::narrow(v[1]);
    asm volatile("st.global.cs.v2.u32 [%0], {%1,%2};" ::"l"(p), "r"(w0), "r"(w1) : "memory");
  }
}

// Load N consecutive parameter values (weight, bias) whose dtype is only known at run time.
// These operands are tiny and shared by every row, so they come through L1 (ld_keep).
// `p` + idx must be aligned to min(16, N * element size).
template <int N>
__device__ __forceinline__ void load_param(const void* base, int dtype, long long idx,
                                           float (&f)[N]) {
  if (dtype == B200_F32) {
    const float* q = reinterpret_cast<const float*>(base) + idx;
#pragma unroll
    for (int i = 0; i < N / 4; ++i) {
      uint4 r = ld_keep(q + 4 * i);
      f[4 * i] = __uint_as_float(r.x);
      f[4 * i + 1] = __uint_as_float(r.y);
      f[4 * i + 2] = __uint_as_float(r.z);
      f[4 * i + 3] = __uint_as_float(r.w);
    }
  } else {
    const unsigned short* q = reinterpret_cast<const unsigned short*>(base) + idx;
    uint32_t w[N / 2];
    if constexpr (N == 8) {
      uint4 r = ld_keep(q);
      w[0] = r.x; w[1] = r.y; w[2] = r.z; w[3] = r.w;
    } else {
      uint2 r;
      asm volatile("ld.global.nc.v2.u32 {%0,%1}, [%2];" : "=r"(r.x), "=r"(r.y) : "l"(q));
      w[0] = r.x; w[1] = r.y;
    }
#pragma unroll
    for (int i = 0; i < N / 2; ++i) {
      if (dtype == B200_BF16) {
        f[2 * i] = __uint_as_float(w[i] << 16);
        f[2 * i + 1] = __uint_as_float(w[i] & 0xffff0000u);
      } else {
        float2 t = __half22float2(*reinterpret_cast<const __half2*>(&w[i]));
        f[2 * i] = t.x;
        f[2 * i + 1] = t.y;
      }
    }
  }
}

// Scalar parameter load with run-time dtype.
__device__ __forceinline__ float load_param1(const void* base, int dtype, long long idx) {
  if (dtype == B200_F32) return ld_here(reinterpret_cast<const float*>(base) + idx);
  if (dtype == B200_BF16)
    return __bfloat162float(ld_here(reinterpret_cast<const __nv_bfloat16*>(base) + idx));
  return __half2float(ld_here(reinterpret_cast<const __half*>(base) + idx));
}

// N parameters at a distance of `step`, those at n and beyond as 0: the type is asked for once, so that all loads are
// on their way together (with load_param1 in a loop each waits for the one before it).
template <int N>
__device__ __forceinline__ void load_params_strided(const void* base, int dtype, int first, int step, int n, float (&out)[N]) {
  auto load = [&](auto tag) {
    using P = decltype(tag);
    const P* p = reinterpret_cast<const P*>(base);
    P raw[N];
#pragma unroll
    for (int e = 0; e < N; ++e) raw[e] = first + e * step < n ? ld_here(p + first + e * step) : Elem<P>::from_f32(0.f);
#pragma unroll
    for (int e = 0; e < N; ++e) out[e] = Elem<P>::to_f32(raw[e]);
  };
  if (dtype == B200_F32) load(float{});
  else if (dtype == B200_BF16) load(__nv_bfloat16{});
  else load(__half{});
}

// Round an fp32 value to T and back: the rounding boundary a 16-bit intermediate tensor imposes.
template <typename T>
__device__ __forceinline__ float round_through(float v) {
  return Elem<T>::to_f32(Elem<T>::from_f32(v));
}

// ----------------------------------------------------------------------------------------------
// Register-resident rows: launch geometry and group helpers.
// A row of nv 16-byte vectors is owned by a group of G threads with CH register slots each
// (G * CH >= nv). Short rows use sub-warp groups of 8, 16 or 32 lanes with up to four slots, so
// that a thread still handles ~32 elements and the per-row bookkeeping (index arithmetic, two
// shuffle reductions, a reciprocal) is amortised; long rows use the whole CTA (G = 0).
//   nv <= 32   : G = 8,  CH = 1, 2 or 4      (256-thread CTA = 32 rows)
//   nv <= 64   : G = 16, CH = 4              (16 rows per CTA)
//   nv <= 128  : G = 32, CH = 4              (8 rows per CTA)
//   nv <= 4096 : G = 0 (CTA per row), CH = 2, 4 or 8, 96..512 threads
// ----------------------------------------------------------------------------------------------
struct RowGeometry {
  int g;        // lanes per row; 0 = the whole CTA
  int ch;       // register slots per thread
  int threads;  // CTA size
  bool block;   // g == 0
};

inline bool pick_row_geometry(long long nv, RowGeometry* g) {
  if (nv <= 0) return false;
  g->threads = 256;
  g->block = false;
  if (nv <= 32) {
    g->g = 8;
    g->ch = nv <= 8 ? 1 : (nv <= 16 ? 2 : 4);
    return true;
  }
  if (nv <= 64) {
    g->g = 16;
    g->ch = 4;
    return true;
  }
  if (nv <= 128) {
    g->g = 32;
    g->ch = 4;
    return true;
  }
  if (nv > 4096) return false;
  g->g = 0;
  g->block = true;
  // CTAs of about 128 threads for mid-size rows (measured on 4096 bf16 columns: 44.7 us with four
  // vectors per thread against 49.2 us with two), eight vectors per thread for the longest
  g->ch = nv <= 256 ? 2 : (nv <= 2048 ? 4 : 8);
  {
    static const int ch_env = [] { const char* e = getenv("B200_BLOCK_CH"); return e ? atoi(e) : 0; }();
    if (ch_env == 2 || ch_env == 4 || ch_env == 8) g->ch = ch_env;
  }
  long long t = (nv + g->ch - 1) / g->ch;
  t = (t + 31) / 32 * 32;
  g->threads = (int)t;
  return true;
}

// ----------------------------------------------------------------------------------------------
// Rows that start and end anywhere, as the 16-byte vectors of memory that they touch: vector j holds the row's elements
// j V - off .. j V - off + V - 1. Only the first and the last one may hold others beside them. Those two are written element by element, so
// that nothing outside the row changes; they are read whole wherever all of them lies between the first row's start and the last row's
// end (a neighbour's elements, or the gap of a padded tensor, which are masked out), and element by element elsewhere, so that nothing
// outside the tensor is read. Tensors with the same `off` in every row share the vectors.
// ----------------------------------------------------------------------------------------------
struct RowSpan {
  int off;   // elements between the 16-byte boundary and the row's first one
  int nv;    // vectors
  int last;  // elements of the last vector that lie in front of the row's end

  template <typename T>
  __device__ __forceinline__ static RowSpan of(const T* row, int n) {
    constexpr int V = Elem<T>::V;
    RowSpan s;
    s.off = (int)((reinterpret_cast<uintptr_t>(row) & 15u) / sizeof(T));
    s.nv = (n + s.off + V - 1) / V;
    s.last = n + s.off - (s.nv - 1) * V;
    return s;
  }
  // The elements of vector j that belong to the row: [lo(j), hi(j)).
  __device__ __forceinline__ int lo(int j) const { return j == 0 ? off : 0; }
  template <int V>
  __device__ __forceinline__ int hi(int j) const {
    return j == nv - 1 ? last : V;
  }
  template <int V>
  __device__ __forceinline__ bool whole(int j) const {
    return (j != 0 || off == 0) && (j != nv - 1 || last == V);
  }
};

// Turns of a CTA that takes `at_once` rows at a time, at most sixteen, so that the CTAs make whole waves of `resident` (rounded down, 24 rows
// per SM in CTAs that take 16 at a time an SM were two waves of one turn, 72 two waves of four).
inline int span_turns(long long rows, int at_once, long long resident) {
  const long long turns = (rows + at_once * resident - 1) / (at_once * resident);
  const long long waves = (turns + 15) / 16;
  return (int)((turns + waves - 1) / waves);
}

// Elements [lo, hi) of the vector at p, zeros beside them.
template <typename T>
__device__ __forceinline__ uint4 load_part(const T* p, int lo, int hi) {
  constexpr int V = Elem<T>::V;
  union {
    T e[V];
    uint4 raw;
  } u;
  u.raw = make_uint4(0u, 0u, 0u, 0u);
#pragma unroll
  for (int i = 0; i < V; ++i)
    if (i >= lo && i < hi) u.e[i] = ld_here(p + i);
  return u.raw;
}
template <typename T>
__device__ __forceinline__ void store_part(T* p, const uint4& raw, int lo, int hi) {
  constexpr int V = Elem<T>::V;
  union {
    T e[V];
    uint4 raw;
  } u;
  u.raw = raw;
#pragma unroll
  for (int i = 0; i < V; ++i)
    if (i >= lo && i < hi) p[i] = u.e[i];
}

// Which halves (fp32: words) of the first and the last vector belong to the row.
template <typename T>
__device__ __forceinline__ void span_edges(const RowSpan& span, uint32_t (&in_first)[4], uint32_t (&in_last)[4]) {
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    if constexpr (sizeof(T) == 2) {
      in_first[i] = (2 * i >= span.off ? 0xffffu : 0u) | (2 * i + 1 >= span.off ? 0xffff0000u : 0u);
      in_last[i] = (2 * i < span.last ? 0xffffu : 0u) | (2 * i + 1 < span.last ? 0xffff0000u : 0u);
    } else {
      in_first[i] = i >= span.off ? 0xffffffffu : 0u;
      in_last[i] = i < span.last ? 0xffffffffu : 0u;
    }
  }
}

// The vectors of row r, whole where all of them lies between the first row's start and the last row's end.
template <typename T, int K>
__device__ __forceinline__ void span_fetch(const void* base, long long pitch, long long rows, int n, long long r, bool there,
                                           const RowSpan& span, int lane, int gs, uint4 (&raw)[K]) {
  constexpr int V = Elem<T>::V;
  const T* x0 = reinterpret_cast<const T*>(base);
  const uintptr_t first = reinterpret_cast<uintptr_t>(x0), end = reinterpret_cast<uintptr_t>(x0 + (rows - 1) * pitch + n);
  const T* x = x0 + r * pitch - span.off + (long long)lane * V;
  const int nv = there ? span.nv : 0;
#pragma unroll
  for (int c = 0; c < K; ++c) raw[c] = make_uint4(0u, 0u, 0u, 0u);
  if (r > 0 && r + 1 < rows && pitch >= n) {  // rows on both sides
#pragma unroll
    for (int c = 0; c < K; ++c)
      if (c * gs + lane < nv) raw[c] = ld_stream(x + (long long)c * gs * V);
  } else {
#pragma unroll
    for (int c = 0; c < K; ++c) {
      const int j = c * gs + lane;
      const T* at = x + (long long)c * gs * V;
      if (j < nv) {
        const uintptr_t u = reinterpret_cast<uintptr_t>(at);
        if (u >= first && u + 16 <= end) raw[c] = ld_stream(at);
        else raw[c] = load_part(at, span.lo(j), span.hi<V>(j));
      }
    }
  }
}

template <int G>
__device__ __forceinline__ int glane() {
  return G == 0 ? (int)threadIdx.x : (int)(threadIdx.x & (G - 1));
}
template <int G>
__device__ __forceinline__ int gsize() {
  return G == 0 ? (int)blockDim.x : G;
}
template <int G>
__device__ __forceinline__ long long grow() {
  return G == 0 ? (long long)blockIdx.x
                : (long long)blockIdx.x * (blockDim.x / (G == 0 ? 1 : G)) + threadIdx.x / (G == 0 ? 1 : G);
}
// Reduction over the group; every lane of the warp must call it (sub-warp groups reduce side by
// side inside one shuffle).
template <typename Op, int G>
__device__ __forceinline__ float greduce(float v, float* scratch) {
  if constexpr (G == 0) {
    return block_reduce<Op>(v, scratch);
  } else {
#pragma unroll
    for (int o = G / 2; o > 0; o >>= 1) v = Op::apply(v, __shfl_xor_sync(0xffffffffu, v, o));
    return v;
  }
}

// Two sums over the group at once: the shuffle chains of the two values interleave, so the pair
// costs about one reduction's latency. `scratch` holds >= 64 floats.
template <int G>
__device__ __forceinline__ void greduce_sum2(float& a, float& b, float* scratch) {
  if constexpr (G == 0) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarps = (blockDim.x + 31) >> 5;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      a += __shfl_xor_sync(0xffffffffu, a, o);
      b += __shfl_xor_sync(0xffffffffu, b, o);
    }
    if (lane == 0) {
      scratch[warp] = a;
      scratch[32 + warp] = b;
    }
    __syncthreads();
    a = 0.f;
    b = 0.f;
    for (int w = 0; w < nwarps; ++w) {
      a += scratch[w];
      b += scratch[32 + w];
    }
    __syncthreads();
  } else {
#pragma unroll
    for (int o = G / 2; o > 0; o >>= 1) {
      a += __shfl_xor_sync(0xffffffffu, a, o);
      b += __shfl_xor_sync(0xffffffffu, b, o);
    }
  }
}

}  // namespace b200
