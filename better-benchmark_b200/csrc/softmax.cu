// Row softmax / log_softmax with optional fused scale and additive (broadcast) mask.
//
// Replaces the single-tile and online Triton softmax kernels of the amax_sum* repro family
// (repros/canonical/amax_sum_20ccc18dda60/oracle.py:11-58, amax_sum_d16035e7b826/oracle.py:14-33,
// amax_sum_7079889cfc04/oracle.py:10-36 in the reference).
//
// Evaluation order follows the decomposed aten graph:
//   t = x [* scale] [+ mask]
//   f = float(t); m = amax(f); e = exp(f - m); s = sum(e); y = e / s      (softmax)
//                                           y = (f - m) - log(s)          (log_softmax)
// Two prologue flavours exist, because graphs differ in where they convert to fp32:
//   fp32   : x and mask are converted first; multiply and add run in fp32, nothing is rounded.
//   packed : (16-bit inputs) multiply and add run in the input dtype and their results are
//            rounded to it, as a 16-bit aten graph materialises them. The kernel does this with
//            packed two-element arithmetic: the product of two 16-bit values is exact in fp32,
//            so a packed multiply by a scale that is representable in the input dtype is
//            bit-identical to "convert, multiply in fp32, round"; a scale that is not
//            representable takes exactly that longer route. The packed add rounds the exact sum
//            once, where aten rounds the fp32 sum; the two differ only when the fp32 sum lands
//            exactly on a 16-bit rounding tie, by one 16-bit ulp of a logit.
// fp32 outputs: expf / logf and the IEEE division. 16-bit outputs: the natural exponential is
// evaluated pairwise as a hardware 2^y with the rounding of y compensated (the accuracy class of
// expf, see exp_pair_compensated in rowwise.cuh) and e / s as e * (1 / s) with a correctly rounded
// reciprocal; both deviations are three orders of magnitude below half a 16-bit ulp. Building with
// -DB200_SOFTMAX_FAST_EXP drops the compensation (the bare ex2.approx that Triton's tl.exp emits);
// that build is for measurements only.
#include "rowwise.cuh"

#include <cooperative_groups.h>

#include <type_traits>

namespace b200 {

#define B200_SOFTMAX_LOG 1
#define B200_SOFTMAX_SCALE 2
#define B200_SOFTMAX_ROUND 4  // packed prologue semantics for 16-bit inputs

struct SoftmaxParams {
  const void* x;
  const void* mask;  // may be null; same dtype as x
  void* y;
  long long rows;
  int n;
  RowMap xmap, mmap, ymap;
  float scale;
  int has_scale;
  int scale_exact16;  // scale survives a round trip through the input dtype
  int log_mode;
};

// Maximum that ignores NaN operands. aten.amax keeps NaNs, but a NaN element makes the sum, and
// with it every output of the row, NaN either way.
struct FastMax {
  static __device__ __forceinline__ float identity() { return -INFINITY; }
  static __device__ __forceinline__ float apply(float a, float b) { return fmaxf(a, b); }
};

// Packed two-element views of the 16-bit types.
template <typename T>
struct Pair;
template <>
struct Pair<__half> {
  using type = __half2;
  static __device__ __forceinline__ __half2 splat(float v) { return __float2half2_rn(v); }
  static __device__ __forceinline__ float2 widen(__half2 v) { return __half22float2(v); }
  static __device__ __forceinline__ __half2 narrow(float a, float b) { return __floats2half2_rn(a, b); }
};
template <>
struct Pair<__nv_bfloat16> {
  using type = __nv_bfloat162;
  static __device__ __forceinline__ __nv_bfloat162 splat(float v) { return __float2bfloat162_rn(v); }
  static __device__ __forceinline__ float2 widen(__nv_bfloat162 v) {
    const uint32_t w = *reinterpret_cast<const uint32_t*>(&v);
    return make_float2(__uint_as_float(w << 16), __uint_as_float(w & 0xffff0000u));
  }
  static __device__ __forceinline__ __nv_bfloat162 narrow(float a, float b) {
    return __floats2bfloat162_rn(a, b);
  }
};
template <>
struct Pair<float> {  // never instantiated for arithmetic; keeps the packed branch well-formed
  using type = float2;
};

// Final phases shared by both prologues. v holds this thread's fp32 logits as packed pairs.
// FASTEXP (16-bit outputs) uses the compensated pair exponential (exp_pair_compensated, the
// accuracy class of expf); fp32 outputs use expf itself.
template <typename Tout, int CH, int V, int G, bool FASTEXP, bool EXACT = false>
__device__ __forceinline__ void softmax_finish(f32x2 (&v)[CH][V / 2], float mx, float mx_raw, Tout* y, int nv,
                                               int lane, int gs, bool log_mode, bool valid, float* red) {
  const f32x2 mx2 = splat2(mx);
  f32x2 s2 = splat2(0.f);
  auto exp_pair = [](f32x2 d) {
    if constexpr (FASTEXP) {
#ifdef B200_SOFTMAX_FAST_EXP
      return exp_pair_fast(d);
#else
      return exp_pair_compensated(d);
#endif
    } else {
      float a, b;
      unpack2(d, a, b);
      return pack2(expf(a), expf(b));
    }
  };
  if (log_mode) {  // keep x - max (it may be -inf); the exponentials only feed the sum
#pragma unroll
    for (int c = 0; c < CH; ++c) {
      if (EXACT || c * gs < nv) {  // group-uniform: skip slots no lane uses
#pragma unroll
        for (int i = 0; i < V / 2; ++i) {
          v[c][i] = sub2(v[c][i], mx2);
#ifndef B200_SOFTMAX_FAST_EXP
          if constexpr (FASTEXP) {
            float a, b;
            unpack2(v[c][i], a, b);
            a = a < -1e38f ? -1e38f : a;  // finite argument for the compensated exponential, NaN kept
            b = b < -1e38f ? -1e38f : b;
            s2 = add2(s2, exp_pair(pack2(a, b)));
          } else {
            s2 = add2(s2, exp_pair(v[c][i]));
          }
#else
          s2 = add2(s2, exp_pair(v[c][i]));
#endif
        }
      }
    }
  } else {
#pragma unroll
    for (int c = 0; c < CH; ++c) {
      if (EXACT || c * gs < nv) {
#pragma unroll
        for (int i = 0; i < V / 2; ++i) {
          v[c][i] = exp_pair(sub2(v[c][i], mx2));
          s2 = add2(s2, v[c][i]);
        }
      }
    }
  }
  float sa, sb;
  unpack2(s2, sa, sb);
  float s = greduce<SumOp, G>(sa + sb, red);
  if (mx_raw == -INFINITY) s = NAN;  // every logit -inf: aten's x - max is NaN for the whole row

  f32x2 k2;  // second operand of the last step
  if (log_mode) {
    k2 = splat2(logf(s));
  } else {
    k2 = splat2(__frcp_rn(s));
  }
  if (!valid) return;
  Tout* yl = y + (long long)lane * V;  // slot c of this lane starts c * gs vectors further on
#pragma unroll
  for (int c = 0; c < CH; ++c) {
    if (EXACT || c * gs + lane < nv) {
      f32x2 o[V / 2];
#pragma unroll
      for (int i = 0; i < V / 2; ++i) {
        if (log_mode) {
          o[i] = sub2(v[c][i], k2);
        } else if constexpr (sizeof(Tout) == 4) {
          float a, b;
          unpack2(v[c][i], a, b);
          o[i] = pack2(a / s, b / s);
        } else {
          o[i] = mul2(v[c][i], k2);
        }
      }
      store_pairs<Tout, V>(yl + (long long)c * gs * V, o);
    }
  }
}

template <typename Tin, typename Tout, int CH, int G, bool PACKED, bool EXACT = false>
__global__ void __launch_bounds__(G == 0 ? 512 : 256)
softmax_resident_kernel(const SoftmaxParams p) {
  wait_for_previous_kernel();
  constexpr int V = Elem<Tin>::V;
  constexpr bool FASTEXP = sizeof(Tout) == 2;
  __shared__ float red[32];
  const int lane = glane<G>();
  const int gs = gsize<G>();
  long long row = grow<G>();
  const bool valid = row < p.rows;  // lanes of a partly filled last CTA compute on the last row
  if (!valid) row = p.rows - 1;

  const Tin* x = reinterpret_cast<const Tin*>(p.x) + row_offset(p.xmap, row);
  const int nv = p.n / V;

  // slot c of this lane starts c * gs vectors after the lane's first one: one pointer per tensor,
  // constant offsets per slot (gs is a compile-time constant for sub-warp and warp groups)
  const Tin* xl = x + (long long)lane * V;
  uint4 raw[CH];
#pragma unroll
  for (int c = 0; c < CH; ++c) {
    if (EXACT || c * gs + lane < nv) raw[c] = ld_stream(xl + (long long)c * gs * V);
  }
  // Where the row's mask and result lie is worked out while the row is on its way: a mask that broadcasts over some of
  // the outer dimensions takes divisions, and in front of the loads they delayed every CTA (fp16 [16, 12, 512, 512] with
  // a [16, 1, 1, 512] mask: 38.6 us against 34.9 with a [1, 512] one; so, and with a flat map for x and y, 35.7 against 34.0).
  const Tin* m = p.mask ? reinterpret_cast<const Tin*>(p.mask) + row_offset(p.mmap, row) : nullptr;
  Tout* y = reinterpret_cast<Tout*>(p.y) + row_offset(p.ymap, row);
  const Tin* ml = m ? m + (long long)lane * V : nullptr;

  f32x2 v[CH][V / 2];
  float mx = -INFINITY;

  // The compensated pair exponential needs finite arguments (inf - inf inside its compensation step would
  // give NaN where exp(-inf) is 0): logits are clamped to a finite floor AFTER the row maximum was
  // taken from the unclamped values. A row whose maximum is -inf (fully masked with -inf) makes
  // aten return NaN for the whole row; the same happens here through the sum (see below).
  constexpr float kFloor = sizeof(Tin) == 2 && !std::is_same<Tin, __nv_bfloat16>::value ? -60000.f : -1e38f;
  // log_softmax returns x - max - log(sum) itself, which may legitimately be -inf: there only the
  // exponential's argument is clamped (in softmax_finish), not the stored value.
#ifdef B200_SOFTMAX_FAST_EXP
  const bool clamp_now = false;  // 2^(-inf) is 0 in the plain exponential: nothing to protect
#else
  const bool clamp_now = FASTEXP && !p.log_mode;
#endif
  if constexpr (PACKED && sizeof(Tin) == 2) {
    using P2 = typename Pair<Tin>::type;
    const P2 neg_inf = Pair<Tin>::splat(-INFINITY);
    const P2 floor2 = Pair<Tin>::splat(kFloor);
    P2 mx2 = neg_inf;
    // One copy of the slot loop per combination of the (warp-uniform) prologue switches, so that
    // they are tested once per row and not once per 16-byte slot.
    //   SK: 0 no scale, 1 packed multiply (scale representable in Tin), 2 fp32 multiply + rounding
    auto prologue = [&](auto sk_tag, auto hm_tag, auto clamp_tag) {
      constexpr int SK = decltype(sk_tag)::value;
      constexpr bool HM = decltype(hm_tag)::value;
      constexpr bool CLAMP = decltype(clamp_tag)::value;
      const P2 s2 = Pair<Tin>::splat(p.scale);
#pragma unroll
      for (int c = 0; c < CH; ++c) {
        P2 t[4];
        if (EXACT || c * gs + lane < nv) {
          const uint32_t w[4] = {raw[c].x, raw[c].y, raw[c].z, raw[c].w};
#pragma unroll
          for (int i = 0; i < 4; ++i) t[i] = *reinterpret_cast<const P2*>(&w[i]);
          if constexpr (SK == 1) {
#pragma unroll
            for (int i = 0; i < 4; ++i) t[i] = __hmul2(t[i], s2);
          } else if constexpr (SK == 2) {
#pragma unroll
            for (int i = 0; i < 4; ++i) {
              const float2 f = Pair<Tin>::widen(t[i]);
              t[i] = Pair<Tin>::narrow(f.x * p.scale, f.y * p.scale);
            }
          }
          if constexpr (HM) {
            const uint4 mr = ld_keep(ml + (long long)c * gs * V);
            const uint32_t mw[4] = {mr.x, mr.y, mr.z, mr.w};
#pragma unroll
            for (int i = 0; i < 4; ++i) t[i] = __hadd2(t[i], *reinterpret_cast<const P2*>(&mw[i]));
          }
#pragma unroll
          for (int i = 0; i < 4; ++i) mx2 = __hmax2(mx2, t[i]);
        } else {
#pragma unroll
          for (int i = 0; i < 4; ++i) t[i] = neg_inf;
        }
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const P2 u = CLAMP ? __hmax2_nan(t[i], floor2) : t[i];  // NaN stays NaN
          v[c][i] = Pairs<Tin>::word(*reinterpret_cast<const uint32_t*>(&u));
        }
      }
    };
    using I0 = std::integral_constant<int, 0>;
    using I1 = std::integral_constant<int, 1>;
    using I2 = std::integral_constant<int, 2>;
    auto with_mask_and_clamp = [&](auto sk_tag) {
      if (m != nullptr) {
        if (clamp_now) prologue(sk_tag, std::true_type{}, std::true_type{});
        else prologue(sk_tag, std::true_type{}, std::false_type{});
      } else {
        if (clamp_now) prologue(sk_tag, std::false_type{}, std::true_type{});
        else prologue(sk_tag, std::false_type{}, std::false_type{});
      }
    };
    if (!p.has_scale) with_mask_and_clamp(I0{});
    else if (p.scale_exact16) with_mask_and_clamp(I1{});
    else with_mask_and_clamp(I2{});
    const float2 mf = Pair<Tin>::widen(mx2);
    mx = greduce<FastMax, G>(fmaxf(mf.x, mf.y), red);
  } else {
#pragma unroll
    for (int c = 0; c < CH; ++c) {
      float f[V];
      if (EXACT || c * gs + lane < nv) {
        Elem<Tin>::unpack(raw[c], f);
        if (p.has_scale) {
#pragma unroll
          for (int i = 0; i < V; ++i) f[i] = f[i] * p.scale;
        }
        if (m != nullptr) {
          float mf[V];
          Elem<Tin>::unpack(ld_keep(ml + (long long)c * gs * V), mf);
#pragma unroll
          for (int i = 0; i < V; ++i) f[i] = f[i] + mf[i];
        }
#pragma unroll
        for (int i = 0; i < V; ++i) mx = fmaxf(mx, f[i]);
      } else {
#pragma unroll
        for (int i = 0; i < V; ++i) f[i] = -INFINITY;
      }
      if (clamp_now) {
#pragma unroll
        for (int i = 0; i < V; ++i) f[i] = f[i] < kFloor ? kFloor : f[i];  // a NaN logit stays NaN
      }
#pragma unroll
      for (int i = 0; i < V / 2; ++i) v[c][i] = pack2(f[2 * i], f[2 * i + 1]);
    }
    mx = greduce<FastMax, G>(mx, red);
  }

  // Subtract the maximum of the CLAMPED values (so every difference is <= 0 and finite); the
  // unclamped maximum still decides whether the whole row was -inf.
  const float mx_raw = mx;
  if (clamp_now) mx = fmaxf(mx, kFloor);
  softmax_finish<Tout, CH, V, G, FASTEXP, EXACT>(v, mx, mx_raw, y, nv, lane, gs, p.log_mode != 0, valid, red);
}

// Element-wise kernel for masked rows of more than 8192 elements that break the vector-path alignment
// rules: one CTA per row and three sweeps (max, sum of exp, write). Only the first sweep of a
// row comes from DRAM when the row fits in L2.
template <typename Tin, bool PACKED>
__device__ __forceinline__ float softmax_logit(const SoftmaxParams& p, const Tin* x, const Tin* m,
                                               long long i) {
  float t = Elem<Tin>::to_f32(x[i]);
  if (p.has_scale) {
    t = t * p.scale;
    if (PACKED) t = round_through<Tin>(t);
  }
  if (m != nullptr) {
    t = t + Elem<Tin>::to_f32(m[i]);
    if (PACKED) t = round_through<Tin>(t);
  }
  return t;
}

// Rows with a mask (or short ones) that neither the vector path nor softmax_span_kernel takes: a warp per row (n <= 512) or a
// CTA per row, E elements per thread at a distance of the group, held in registers: one read of the
// row and of its mask instead of the three sweeps below, every access of a warp one coalesced stretch
// whatever the alignment. Bound by the number of 2-byte accesses and the exponentials. Measured with a key mask: fp16
// [24576, 333] 203 us with the three sweeps, 25.4 us here; fp32 [24576, 5001] 915 -> 496 us.
// Few rows (up to four per SM of 65..512 elements, two per SM of up to 2048) take a CTA per row with two elements a
// thread: fp16 [384, 333] by warps 3.7 us, so 3.2; [8, 511] 3.8 and 2.5. fp32 rows of eight elements a thread keep to 32
// registers, two CTAs of 1024 threads per SM (50 registers: [24576, 5001] 1009 us).
template <typename Tin, typename Tout, bool PACKED, int E, int G>
__global__ void __launch_bounds__(G == 0 ? 1024 : 256, G == 0 && E == 8 ? 2 : 0) softmax_ragged_kernel(const SoftmaxParams p) {
  wait_for_previous_kernel();
  __shared__ float red[32];
  const int lane = glane<G>(), gs = gsize<G>();
  long long row = grow<G>();
  const bool valid = row < p.rows;  // warps of a partly filled last CTA compute on the last row
  if (!valid) row = p.rows - 1;
  const Tin* x = reinterpret_cast<const Tin*>(p.x) + row_offset(p.xmap, row);
  const Tin* m = p.mask ? reinterpret_cast<const Tin*>(p.mask) + row_offset(p.mmap, row) : nullptr;
  Tout* y = reinterpret_cast<Tout*>(p.y) + row_offset(p.ymap, row);
  float t[E];
  float mx = -INFINITY;
  {  // every load is on its way before the first value is looked at
    Tin xv[E], mv[E];
#pragma unroll
    for (int e = 0; e < E; ++e)
      if (e * gs + lane < p.n) xv[e] = ld_here(x + e * gs + lane);
    if (m) {
#pragma unroll
      for (int e = 0; e < E; ++e)
        if (e * gs + lane < p.n) mv[e] = ld_here(m + e * gs + lane);
    }
#pragma unroll
    for (int e = 0; e < E; ++e) {
      t[e] = -INFINITY;
      if (e * gs + lane < p.n) {
        t[e] = Elem<Tin>::to_f32(xv[e]);
        if (p.has_scale) t[e] = PACKED ? round_through<Tin>(t[e] * p.scale) : t[e] * p.scale;
        if (m) t[e] = PACKED ? round_through<Tin>(t[e] + Elem<Tin>::to_f32(mv[e])) : t[e] + Elem<Tin>::to_f32(mv[e]);
      }
    }
  }
#pragma unroll
  for (int e = 0; e < E; ++e) mx = fmaxf(mx, t[e]);
  mx = greduce<FastMax, G>(mx, red);
  float s = 0.f;
#pragma unroll
  for (int e = 0; e < E; ++e) {
    if (e * gs + lane < p.n) {
      t[e] = t[e] - mx;  // log_softmax keeps the difference, softmax the exponential
      const float v = expf(t[e]);
      s += v;
      if (!p.log_mode) t[e] = v;
    }
  }
  s = greduce<SumOp, G>(s, red);
  if (!valid) return;
  const float ls = logf(s), inv = __frcp_rn(s);
#pragma unroll
  for (int e = 0; e < E; ++e) {
    const int i = e * gs + lane;
    if (i < p.n) y[i] = Elem<Tout>::from_f32(p.log_mode ? t[e] - ls : (sizeof(Tout) == 4 ? t[e] / s : t[e] * inv));
  }
}

// 16-bit rows at one distance, off the 16-byte grid, whose result has their alignment (contiguous rows of an odd length, in the input's
// dtype): the row as the vectors it touches (RowSpan), in registers from the load to the store. A group of G lanes takes
// `reps` rows that are a multiple of eight apart and so have the same alignment: what belongs to a column, the mask, stays in its registers
// as long as the rows share it, and holds -inf where a vector reaches beyond the row, so that no other part of the loop asks what is
// inside. The next row is on its way meanwhile. Numerics as in softmax_ragged_kernel, expf included (the pair exponential, 5 to 15 % faster, is
// less exact and loses subnormal bf16 probabilities); the maximum keeps NaN. Bound by instructions (with every edge asked for
// in every row 709 a warp and row of 333 elements, 84 % of the issue slots), so the mask stays packed, four CTAs of 256 threads an SM up to two
// vectors a lane (three vectors: 8 bytes of spills at three CTAs, four: 24 at two). Key mask, fp16, against softmax_ragged_kernel: [60000, 333]
// 52.8 -> 35.2 us, [20000, 716] 38.5 -> 23.2, [60000, 1001] 141 -> 73, [60000, 114] 18.6 -> 14.3.
template <typename T, int K, int G>
__global__ void __launch_bounds__(256, K <= 2 ? 4 : K == 3 ? 3 : 2) softmax_span_kernel(const SoftmaxParams p, const int reps) {
  wait_for_previous_kernel();
  static_assert(sizeof(T) == 2, "pairs of 16-bit elements");
  constexpr int V = Elem<T>::V;
  constexpr int P = V / 2;
  const int lane = glane<G>();
  constexpr int gs = G, step = 256 / G;  // rows that the CTA takes at a time: a multiple of eight
  const int rows = (int)p.rows;
  int row = (int)blockIdx.x * reps * step + (int)threadIdx.x / G;
  const T* x0 = reinterpret_cast<const T*>(p.x);
  const long long pitch = p.xmap.s0;
  const RowSpan span = RowSpan::of(x0 + row * pitch, p.n);
  // whole vectors are read where all of them lies between the first row's start and the last row's end
  const uintptr_t x_first = reinterpret_cast<uintptr_t>(x0), x_end = reinterpret_cast<uintptr_t>(x0 + (rows - 1) * pitch + p.n);
  auto fetch = [&](int r, uint4 (&raw)[K]) {
    const T* x = x0 + r * pitch - span.off + (long long)lane * V;
#pragma unroll
    for (int c = 0; c < K; ++c) {
      const int j = c * gs + lane;
      const T* at = x + (long long)c * gs * V;
      raw[c] = make_uint4(0u, 0u, 0u, 0u);
      if (r < rows && j < span.nv) {
        const uintptr_t u = reinterpret_cast<uintptr_t>(at);
        if (u >= x_first && u + 16 <= x_end) raw[c] = ld_stream(at);
        else raw[c] = load_part(at, span.lo(j), span.hi<V>(j));
      }
    }
  };
  // which halves of the words of the first and the last vector belong to the row
  uint32_t in_first[P], in_last[P];
#pragma unroll
  for (int i = 0; i < P; ++i) {
    in_first[i] = (2 * i >= span.off ? 0xffffu : 0u) | (2 * i + 1 >= span.off ? 0xffff0000u : 0u);
    in_last[i] = (2 * i < span.last ? 0xffffu : 0u) | (2 * i + 1 < span.last ? 0xffff0000u : 0u);
  }
  uint4 m[K];
  auto set_mask = [&](const T* mask) {
#pragma unroll
    for (int c = 0; c < K; ++c) {
      const int j = c * gs + lane;
      const int lo = span.lo(j), hi = j < span.nv ? span.hi<V>(j) : 0;
      union {
        T e[V];
        uint4 raw;
      } u;
#pragma unroll
      for (int i = 0; i < V; ++i) {
        u.e[i] = Elem<T>::from_f32(-INFINITY);
        if (i >= lo && i < hi) u.e[i] = mask ? ld_here(mask - span.off + (long long)j * V + i) : Elem<T>::from_f32(0.f);
      }
      m[c] = u.raw;
    }
  };
  uint4 next[K];
  fetch(row, next);
  long long mask_at = -1;
  if (!p.mask) set_mask(nullptr);
  const f32x2 scale2 = splat2(p.has_scale ? p.scale : 1.f);

  for (int rep = 0; rep < reps; ++rep, row += step) {
    const bool valid = row < rows;
    if (!__any_sync(0xffffffffu, valid)) break;
    uint4 raw[K];
#pragma unroll
    for (int c = 0; c < K; ++c) raw[c] = next[c];
    if (rep + 1 < reps) fetch(row + step, next);
    if (p.mask && valid) {
      const long long at = row_offset(p.mmap, row);
      if (at != mask_at) {
        mask_at = at;
        set_mask(reinterpret_cast<const T*>(p.mask) + at);
      }
    }
    f32x2 t[K][P];
    float mx = -INFINITY;
#pragma unroll
    for (int c = 0; c < K; ++c) {
      uint32_t w[P] = {raw[c].x, raw[c].y, raw[c].z, raw[c].w};
      if (c == 0 && lane == 0) {
#pragma unroll
        for (int i = 0; i < P; ++i) w[i] &= in_first[i];
      }
      if (c * gs + lane == span.nv - 1) {
#pragma unroll
        for (int i = 0; i < P; ++i) w[i] &= in_last[i];
      }
      f32x2 mc[P];
      Pairs<T>::unpack(m[c], mc);
#pragma unroll
      for (int i = 0; i < P; ++i) {
        t[c][i] = add2(mul2(Pairs<T>::word(w[i]), scale2), mc[i]);
        float a, b;
        unpack2(t[c][i], a, b);
        mx = MaxOp::apply(mx, MaxOp::apply(a, b));
      }
    }
    mx = greduce<MaxOp, G>(mx, nullptr);

    auto finish = [&](auto log_tag) {
      constexpr bool LOG = decltype(log_tag)::value;
      const f32x2 mx2 = splat2(mx);
      f32x2 s2 = splat2(0.f);
#pragma unroll
      for (int c = 0; c < K; ++c) {
#pragma unroll
        for (int i = 0; i < P; ++i) {
          t[c][i] = sub2(t[c][i], mx2);
          float a, b;
          unpack2(t[c][i], a, b);
          const f32x2 e = pack2(expf(a), expf(b));
          s2 = add2(s2, e);
          if constexpr (!LOG) t[c][i] = e;
        }
      }
      float s = greduce<SumOp, G>(hsum2(s2), nullptr);
      if (!(fabsf(mx) < INFINITY)) s = NAN;  // aten's x - max is NaN for a row of -inf and where x is inf; a NaN poisons its row
      if (!valid) return;
      const f32x2 k2 = splat2(LOG ? logf(s) : __frcp_rn(s));
      T* y = reinterpret_cast<T*>(p.y) + row * p.ymap.s0 - span.off + (long long)lane * V;
#pragma unroll
      for (int c = 0; c < K; ++c) {
        const int j = c * gs + lane;
        if (j < span.nv) {
          f32x2 o[P];
#pragma unroll
          for (int i = 0; i < P; ++i) o[i] = LOG ? sub2(t[c][i], k2) : mul2(t[c][i], k2);
          const uint4 out = Pairs<T>::pack(o);
          if (span.whole<V>(j)) st_stream(y + (long long)c * gs * V, out);
          else store_part(y + (long long)c * gs * V, out, span.lo(j), span.hi<V>(j));
        }
      }
    };
    if (p.log_mode) finish(std::true_type{});
    else finish(std::false_type{});
  }
}

// The same for longer rows: a CTA per row, as many of them as the SM holds; the mask is read element by element through L1, where
// eight such loads a vector take as long as HBM takes for the vector and its result. (Eight rows per CTA in turn, as above, took 1.3 times
// as long.) fp16 with a key mask: [20000, 1241] 61.9 -> 40.3 us, [20000, 2047] 95.2 -> 63.9, [20000, 3001] 147 -> 80.
template <typename T, int K>
__global__ void __launch_bounds__(512) softmax_span_row_kernel(const SoftmaxParams p) {
  wait_for_previous_kernel();
  static_assert(sizeof(T) == 2, "pairs of 16-bit elements");
  constexpr int V = Elem<T>::V;
  constexpr int P = V / 2;
  __shared__ float red[32];
  const int lane = (int)threadIdx.x, gs = (int)blockDim.x;
  const long long row = blockIdx.x;
  const T* x = reinterpret_cast<const T*>(p.x) + row_offset(p.xmap, row);
  const RowSpan span = RowSpan::of(x, p.n);
  x -= span.off;
  uint4 raw[K];
#pragma unroll
  for (int c = 0; c < K; ++c) {
    const int j = c * gs + lane;
    raw[c] = make_uint4(0u, 0u, 0u, 0u);
    if (j < span.nv) {
      if (span.whole<V>(j)) raw[c] = ld_stream(x + (long long)j * V);
      else raw[c] = load_part(x + (long long)j * V, span.lo(j), span.hi<V>(j));
    }
  }
  const T* m = p.mask ? reinterpret_cast<const T*>(p.mask) + row_offset(p.mmap, row) - span.off : nullptr;
  T* y = reinterpret_cast<T*>(p.y) + row_offset(p.ymap, row) - span.off;

  f32x2 t[K][P];
  float mx = -INFINITY;
#pragma unroll
  for (int c = 0; c < K; ++c) {
    const int j = c * gs + lane;
    float f[V];
    Elem<T>::unpack(raw[c], f);
    if (p.has_scale) {
#pragma unroll
      for (int i = 0; i < V; ++i) f[i] = f[i] * p.scale;
    }
    if (j < span.nv) {
      const int lo = span.lo(j), hi = span.hi<V>(j);
      if (m) {
        const T* mj = m + (long long)j * V;
        T mv[V];
        if (span.whole<V>(j)) {
#pragma unroll
          for (int i = 0; i < V; ++i) mv[i] = ld_here(mj + i);
        } else {
#pragma unroll
          for (int i = 0; i < V; ++i) {
            mv[i] = Elem<T>::from_f32(0.f);
            if (i >= lo && i < hi) mv[i] = ld_here(mj + i);
          }
        }
#pragma unroll
        for (int i = 0; i < V; ++i) f[i] = f[i] + Elem<T>::to_f32(mv[i]);
      }
      if (!span.whole<V>(j)) {
#pragma unroll
        for (int i = 0; i < V; ++i)
          if (i < lo || i >= hi) f[i] = -INFINITY;
      }
#pragma unroll
      for (int i = 0; i < V; ++i) mx = MaxOp::apply(mx, f[i]);
    } else {
#pragma unroll
      for (int i = 0; i < V; ++i) f[i] = -INFINITY;
    }
#pragma unroll
    for (int i = 0; i < P; ++i) t[c][i] = pack2(f[2 * i], f[2 * i + 1]);
  }
  mx = block_reduce<MaxOp>(mx, red);

  auto finish = [&](auto log_tag) {
    constexpr bool LOG = decltype(log_tag)::value;
    const f32x2 mx2 = splat2(mx);
    f32x2 s2 = splat2(0.f);
#pragma unroll
    for (int c = 0; c < K; ++c) {
#pragma unroll
      for (int i = 0; i < P; ++i) {
        t[c][i] = sub2(t[c][i], mx2);
        float a, b;
        unpack2(t[c][i], a, b);
        const f32x2 e = pack2(expf(a), expf(b));
        s2 = add2(s2, e);
        if constexpr (!LOG) t[c][i] = e;
      }
    }
    float s = block_reduce<SumOp>(hsum2(s2), red);
    if (!(fabsf(mx) < INFINITY)) s = NAN;  // as above
    const f32x2 k2 = splat2(LOG ? logf(s) : __frcp_rn(s));
#pragma unroll
    for (int c = 0; c < K; ++c) {
      const int j = c * gs + lane;
      if (j < span.nv) {
        f32x2 o[P];
#pragma unroll
        for (int i = 0; i < P; ++i) o[i] = LOG ? sub2(t[c][i], k2) : mul2(t[c][i], k2);
        const uint4 out = Pairs<T>::pack(o);
        if (span.whole<V>(j)) st_stream(y + (long long)j * V, out);
        else store_part(y + (long long)j * V, out, span.lo(j), span.hi<V>(j));
      }
    }
  };
  if (p.log_mode) finish(std::true_type{});
  else finish(std::false_type{});
}

// Rows per SM from which on the two kernels above are ahead of softmax_ragged_kernel, or within 4 per cent, at every number of rows measured (0:
// never), for rows of n elements that touch nv vectors at most. A group reads its part of the mask once, 1 us; its slots are filled or not, as the
// other kernel's are. That kernel's time over this one's, fp16 with one mask for all rows, rows per SM in front:
//   n 57    32 0.99, 40 0.91, 48 1.00, 96 1.24        n 90    56 0.97, 64 1.05, 104 0.99, 128 1.13 (no mask 144 0.95, 160 1.03)
//   n 121   48 0.91, 56 1.01, 104 1.07, 250 1.41      n 150   48 0.93, 52 1.00, 104 1.10     n 201   160 1.01, 200 0.98, 250 1.19
//   n 249   80 1.01, 96 1.15, 200 1.04                n 257   22 0.88, 25 1.24, 36 1.16      n 378   22 0.96, 25 1.14, 36 1.00
//   n 420   3 0.95, 5 1.13, 22 1.02                   n 511   64 0.98, 72 1.05               n 601   8 0.99, 11 1.08, 18 1.15
//   n 900   8 1.01, 11 1.10, 64 1.90                  n 127   200 0.86, 405 1.01             n 255   144 0.97, 250 0.91
// The last two are of the rows that fill the other kernel's slots and have just left one of this one's. With a
// mask for so many rows as the CTA takes at two times the groups are still ahead ([20000, 1017] 50.6 / 41.3), with one for half as many no longer
// (50.6 / 53.3), with one for every row they are far behind (49.0 / 73.0, [60000, 249] 29.6 / 36.7).
static int softmax_span_rows_per_sm(int n, int nv, bool masked) {
  if (nv > 128) return 2;
  if ((n > 121 && n <= 128) || (n > 249 && n <= 256)) return 0;
  if (n <= 57) return 44;
  if (n <= 99) return masked ? (n <= 65 ? 80 : 64) : 160;
  if (n <= 249) return n <= 185 ? 52 : n <= 234 ? 250 : 96;
  return n <= 390 ? 25 : n <= 505 ? 5 : n <= 512 ? 72 : 11;
}

// How many rows that follow one another share their mask.
static long long softmax_rows_per_mask(const SoftmaxParams& p) {
  if (!p.mask) return p.rows;
  const RowMap& m = p.mmap;
  long long r = 1;
  if (m.d2.d > 1) {
    if (m.s2 != 0) return r;
    r *= m.d2.d;
  }
  if (m.d1.d > 1) {
    if (m.s1 != 0) return r;
    r *= m.d1.d;
  }
  return m.s0 != 0 ? r : p.rows;
}

// Whether the two kernels above take the rows: x and y have the same alignment in every row, and there are enough of them.
// Up to 1017 elements (four vectors a lane) groups, above that CTAs.
template <typename T>
static bool try_launch_softmax_span(const SoftmaxParams& p, cudaStream_t st) {
  constexpr int V = Elem<T>::V;
  const long long sms = device_info().sm_count;
  const int nv = (p.n + 2 * (V - 1)) / V;  // vectors that a row touches at most
  auto flat = [](const RowMap& m) { return m.d1.d == 1 && m.d2.d == 1 && m.s0 >= 0; };
  if (!flat(p.xmap) || !flat(p.ymap) || (reinterpret_cast<uintptr_t>(p.x) & 15u) != (reinterpret_cast<uintptr_t>(p.y) & 15u) ||
      (p.xmap.s0 - p.ymap.s0) % V != 0 || p.rows > 0x7fff0000LL)
    return false;
  if (nv <= 128 && softmax_rows_per_mask(p) < (nv <= 24 ? 64 : nv <= 48 ? 32 : 16)) return false;  // 2 * 256 / lanes of a group
  const int rows_per_sm = softmax_span_rows_per_sm(p.n, nv, p.mask != nullptr);
  if (rows_per_sm == 0 || p.rows < rows_per_sm * sms) return false;
  if (nv > 2048) return false;
  set_path_tag(nv > 128 ? "off-grid rows as vectors, CTA per row" : "off-grid rows as vectors, several rows in turn");
  if (nv > 128) {
    if (nv <= 512) launch_dependent(softmax_span_row_kernel<T, 2>, (unsigned)p.rows, (nv + 63) / 64 * 32, 0, st, p);
    else launch_dependent(softmax_span_row_kernel<T, 4>, (unsigned)p.rows, (nv + 127) / 128 * 32, 0, st, p);
    return true;
  }
  auto launch = [&](auto kernel, int lanes) {
    const int at_once = 256 / lanes;
    const long long resident = sms * cached_occupancy(reinterpret_cast<const void*>(kernel), 256);
    const int reps = span_turns(p.rows, at_once, resident);
    launch_dependent(kernel, (unsigned)((p.rows + (long long)at_once * reps - 1) / ((long long)at_once * reps)), 256, 0, st, p, reps);
    return true;
  };
  if (nv <= 8) return launch(softmax_span_kernel<T, 1, 8>, 8);
  if (nv <= 16) return launch(softmax_span_kernel<T, 2, 8>, 8);
  if (nv <= 24) return launch(softmax_span_kernel<T, 3, 8>, 8);
  if (nv <= 32) return launch(softmax_span_kernel<T, 2, 16>, 16);
  if (nv <= 48) return launch(softmax_span_kernel<T, 3, 16>, 16);
  if (nv <= 64) return launch(softmax_span_kernel<T, 2, 32>, 32);
  if (nv <= 96) return launch(softmax_span_kernel<T, 3, 32>, 32);
  return launch(softmax_span_kernel<T, 4, 32>, 32);
}

template <typename Tin, typename Tout, bool PACKED>
__global__ void __launch_bounds__(1024) softmax_streaming_kernel(const SoftmaxParams p) {
  wait_for_previous_kernel();
  __shared__ float red[32];
  const long long row = blockIdx.x;
  const Tin* x = reinterpret_cast<const Tin*>(p.x) + row_offset(p.xmap, row);
  const Tin* m = p.mask ? reinterpret_cast<const Tin*>(p.mask) + row_offset(p.mmap, row) : nullptr;
  Tout* y = reinterpret_cast<Tout*>(p.y) + row_offset(p.ymap, row);

  float mx = -INFINITY;
  for (long long i = threadIdx.x; i < p.n; i += blockDim.x)
    mx = fmaxf(mx, softmax_logit<Tin, PACKED>(p, x, m, i));
  mx = block_reduce<FastMax>(mx, red);

  float s = 0.f;
  for (long long i = threadIdx.x; i < p.n; i += blockDim.x)
    s += expf(softmax_logit<Tin, PACKED>(p, x, m, i) - mx);
  s = block_reduce<SumOp>(s, red);

  const float ls = logf(s);
  const float inv = __frcp_rn(s);
  for (long long i = threadIdx.x; i < p.n; i += blockDim.x) {
    const float d = softmax_logit<Tin, PACKED>(p, x, m, i) - mx;
    float o;
    if (p.log_mode) {
      o = d - ls;
    } else if (sizeof(Tout) == 4) {
      o = expf(d) / s;
    } else {
      o = expf(d) * inv;
    }
    y[i] = Elem<Tout>::from_f32(o);
  }
}

// ----------------------------------------------------------------------------------------------
// Rows that the register-resident kernel above does not take (longer than 4096 vectors, a length that
// is no whole number of vectors, or a start off the 16-byte grid; no mask): the row is held in
// registers as the raw 16-byte vectors that were loaded, so that it crosses HBM once whatever its
// alignment.
//   * A CTA of at most 512 threads holds up to CH = 8 vectors per thread (4096 vectors); longer rows,
//     and rows of a tensor with few of them, are split over a thread-block cluster of S <= 8 CTAs
//     that exchange one (maximum, sum) pair each through distributed shared memory.
//   * The body of the row is loaded from the first 16-byte boundary on; the at most V - 1 elements in
//     front of it and behind the last whole vector are held one per thread by the first CTA.
//   * The output row has an alignment of its own (fp32 rows of 20 005 elements start on any multiple
//     of four bytes). The outputs of a thread's vector are handed over by warp shuffles to where the
//     next aligned chunk of the output starts, so stores are whole chunks; only a warp's first and
//     last elements leave one by one.
// What bounds it: three CTAs per SM, as many as their registers allow, each of which loads its row, reduces it twice and stores it. Their
// phases cover one another in part: on the case below DRAM is 51 % busy, the issue slots 63 %, no pipe more than 42 %. Scale and log
// are template parameters, and nothing is clamped as long as the sum of a thread is a number (it is not when a difference lies
// below -2.36e38). Measured: bf16 [4096, 20005] (rows 20 008 apart) -> fp32 log_softmax 183.7 us with the two-sweep
// kernel below, 109 us with run-time switches and clamps, 104 here; bf16 [2000, 32001] softmax 192.6 -> 54.6 us.
// Not taken: the next row brought in by a bulk copy meanwhile (121 us: the loads are not what it waits for), stores
// whose shift is known at compile time (98.6 us where these take 95.8, rows 20 005 apart).
// ----------------------------------------------------------------------------------------------
// Stores a thread's V outputs, the first of which goes to `y`. `shift` (warp-uniform, below the chunk
// length VO) counts the elements from y to the next chunk boundary of the output; the lane above
// supplies what this lane's last chunk lacks, the lane below takes the first `shift` elements.
// Every lane of the warp calls it. has_next: the lane above holds the vector that follows this one.
template <typename Tout, int V>
__device__ __forceinline__ void store_shifted(Tout* y, const f32x2 (&o)[V / 2], int shift, int lane, bool valid,
                                              bool has_next) {
  constexpr int VO = V * (int)sizeof(Tout) <= 16 ? V : 16 / (int)sizeof(Tout);  // elements of a chunk
  if (shift == 0) {
    if (valid) store_pairs<Tout, V>(y, o);
    return;
  }
  if constexpr (sizeof(Tout) == 4) {
    float e[V + 3];
#pragma unroll
    for (int i = 0; i < V / 2; ++i) unpack2(o[i], e[2 * i], e[2 * i + 1]);
#pragma unroll
    for (int i = 0; i < 3; ++i) e[V + i] = __shfl_down_sync(0xffffffffu, e[i], 1);
    float* out = reinterpret_cast<float*>(y);
    if (lane == 0 && valid) {
      out[0] = e[0];
      if (shift > 1) out[1] = e[1];
      if (shift > 2) out[2] = e[2];
    }
    if (shift & 1) {
#pragma unroll
      for (int i = 0; i < V + 2; ++i) e[i] = e[i + 1];
    }
    if (shift & 2) {
#pragma unroll
      for (int i = 0; i < V + 1; ++i) e[i] = e[i + 2];
    }
    if (!valid) return;
    out += shift;
#pragma unroll
    for (int k = 0; k < V / VO; ++k) {
      if (k < V / VO - 1 || has_next) {
        st_stream(out + k * VO, make_uint4(__float_as_uint(e[k * VO]), __float_as_uint(e[k * VO + 1]),
                                           __float_as_uint(e[k * VO + 2]), __float_as_uint(e[k * VO + 3])));
      } else {
#pragma unroll
        for (int i = 0; i < VO - 1; ++i)
          if (i < VO - shift) out[k * VO + i] = e[k * VO + i];
      }
    }
  } else {
    constexpr int W = V / 2;  // 32-bit words of a thread's outputs
    uint32_t w[2 * W];
#pragma unroll
    for (int i = 0; i < W; ++i) w[i] = Pairs<Tout>::narrow(o[i]);
#pragma unroll
    for (int i = 0; i < W; ++i) w[W + i] = __shfl_down_sync(0xffffffffu, w[i], 1);
    unsigned short* out = reinterpret_cast<unsigned short*>(y);
    if (lane == 0 && valid) {
#pragma unroll
      for (int i = 0; i < V - 1; ++i)
        if (i < shift) out[i] = (unsigned short)(w[i / 2] >> (16 * (i & 1)));
    }
    if (W == 4 && (shift & 4)) {
#pragma unroll
      for (int i = 0; i + 2 < 2 * W; ++i) w[i] = w[i + 2];
    }
    if (shift & 2) {
#pragma unroll
      for (int i = 0; i + 1 < 2 * W; ++i) w[i] = w[i + 1];
    }
    if (shift & 1) {
#pragma unroll
      for (int i = 0; i < W; ++i) w[i] = __byte_perm(w[i], w[i + 1], 0x5432);
    }
    if (!valid) return;
    out += shift;
    if (has_next) {
      if constexpr (W == 4) st_stream(out, make_uint4(w[0], w[1], w[2], w[3]));
      else asm volatile("st.global.cs.v2.u32 [%0], {%1,%2};" ::"l"(out), "r"(w[0]), "r"(w[1]) : "memory");
    } else {
#pragma unroll
      for (int i = 0; i < V - 1; ++i)
        if (i < V - shift) out[i] = (unsigned short)(w[i / 2] >> (16 * (i & 1)));
    }
  }
}

template <typename Tin, typename Tout, int CH, bool CLUSTER, bool SCALED, bool LOG>
__global__ void __launch_bounds__(512, 2) softmax_rows_kernel(const SoftmaxParams p, const int S) {
  wait_for_previous_kernel();
  constexpr int V = Elem<Tin>::V;
  constexpr int P = V / 2;
  constexpr int VO = V * (int)sizeof(Tout) <= 16 ? V : 16 / (int)sizeof(Tout);
  constexpr float kFloor = -1e30f;  // where differences from the maximum are clamped for the pair exponential
  __shared__ float red[32];
  __shared__ float pairs[2][8];  // cluster: (maximum, sum) of every CTA of the row
  const int tid = threadIdx.x, lane = tid & 31, T_ = blockDim.x;
  // a CTA's shared memory may be written from another one only once it runs: arrive here, wait before the write
  if constexpr (CLUSTER) cooperative_groups::this_cluster().barrier_arrive();
  const int rank = CLUSTER ? (int)(blockIdx.x % (unsigned)S) : 0;
  const long long row = CLUSTER ? (long long)(blockIdx.x / (unsigned)S) : (long long)blockIdx.x;
  const Tin* x = reinterpret_cast<const Tin*>(p.x) + row_offset(p.xmap, row);

  // body: whole vectors from the first 16-byte boundary on; edge: what is in front of it and behind it
  int head = (int)(((16u - (unsigned)(reinterpret_cast<uintptr_t>(x) & 15u)) & 15u) / sizeof(Tin));
  if (head > p.n) head = p.n;
  const int nvec = (p.n - head) / V;
  const int tail0 = head + nvec * V;
  const int edges = head + (p.n - tail0);
  const int per = CLUSTER ? (nvec + S - 1) / S : nvec;
  const int v0 = CLUSTER ? rank * per : 0;
  const int cnt = nvec - v0 < per ? nvec - v0 : per;  // vectors of this CTA (may be negative: none)
  const Tin* xb = x + head + (long long)v0 * V;

  uint4 raw[CH];
#pragma unroll
  for (int c = 0; c < CH; ++c)
    if (c * T_ + tid < cnt) raw[c] = ld_stream(xb + (long long)(c * T_ + tid) * V);
  Tout* y = reinterpret_cast<Tout*>(p.y) + row_offset(p.ymap, row);
  Tout* yb = y + head + (long long)v0 * V;
  const bool has_edge = rank == 0 && tid < edges;
  const int edge_at = tid < head ? tid : tail0 + (tid - head);
  const f32x2 scale2 = splat2(p.scale);
  float edge = -INFINITY;
  if (has_edge) {
    edge = Elem<Tin>::to_f32(x[edge_at]);
    if constexpr (SCALED) edge = edge * p.scale;
  }
  auto logits = [&](int c, f32x2 (&t)[P]) {
    Pairs<Tin>::unpack(raw[c], t);
    if constexpr (SCALED) {
#pragma unroll
      for (int i = 0; i < P; ++i) t[i] = mul2(t[i], scale2);
    }
  };

  // ---- maximum (a NaN anywhere makes it NaN) ------------------------------------------------------
  float m = edge;
  if constexpr (sizeof(Tin) == 2 && !SCALED) {  // a maximum is exact in the input type: packed pairs, no conversion
    using P2 = typename Pair<Tin>::type;
    P2 m2 = Pair<Tin>::splat(-INFINITY);
#pragma unroll
    for (int c = 0; c < CH; ++c) {
      if (c * T_ + tid < cnt) {
        const uint32_t w[4] = {raw[c].x, raw[c].y, raw[c].z, raw[c].w};
#pragma unroll
        for (int i = 0; i < 4; ++i) m2 = MaxOp::apply2(m2, *reinterpret_cast<const P2*>(&w[i]));
      }
    }
    const float2 f = Pair<Tin>::widen(m2);
    m = MaxOp::apply(m, MaxOp::apply(f.x, f.y));
  } else {
#pragma unroll
    for (int c = 0; c < CH; ++c) {
      if (c * T_ + tid < cnt) {
        f32x2 t[P];
        logits(c, t);
#pragma unroll
        for (int i = 0; i < P; ++i) {
          float a, b;
          unpack2(t[i], a, b);
          m = MaxOp::apply(m, MaxOp::apply(a, b));
        }
      }
    }
  }
  float M = block_reduce<MaxOp>(m, red);

  // ---- sum of the exponentials --------------------------------------------------------------------
  auto clamped = [&](f32x2 d) {  // a NaN is lost here: the maximum has caught it
    float a, b;
    unpack2(d, a, b);
    return pack2(fmaxf(a, kFloor), fmaxf(b, kFloor));
  };
  auto exp_exact = [](f32x2 d) {
    float a, b;
    unpack2(d, a, b);
    return pack2(expf(a), expf(b));
  };
  // fp32 rows with 16-bit results keep their exponentials where the row was, and multiply them by the sum's inverse at the end (f32 -> bf16
  // [2000, 10698] 32.5 -> 29.3 us, [4000, 2909] 15.9 -> 14.7; with fp32 results, where the division takes as long as expf, they stand
  // in the way: 46.6 -> 50.5 us; and a cluster would have to agree on the maximum first: [1425, 29114] 72 -> 80).
  constexpr bool KEEP = sizeof(Tin) == 4 && sizeof(Tout) == 2 && !LOG && !CLUSTER;
  auto add_up = [&](auto exponential) {
    const f32x2 own = splat2(M);
    f32x2 sum = splat2(0.f);
#pragma unroll
    for (int c = 0; c < CH; ++c) {
      if (c * T_ + tid < cnt) {
        f32x2 t[P];
        logits(c, t);
        if constexpr (KEEP) {
          const f32x2 e0 = exponential(sub2(t[0], own)), e1 = exponential(sub2(t[1], own));
          sum = add2(sum, add2(e0, e1));
          float a, b, c2, d;
          unpack2(e0, a, b);
          unpack2(e1, c2, d);
          raw[c] = make_uint4(__float_as_uint(a), __float_as_uint(b), __float_as_uint(c2), __float_as_uint(d));
        } else {
          f32x2 part = exponential(sub2(t[0], own));
#pragma unroll
          for (int i = 1; i < P; ++i) part = add2(part, exponential(sub2(t[i], own)));
          sum = add2(sum, part);
        }
      }
    }
    return hsum2(sum);
  };
  // fp32 results sum expf, log_softmax too: the errors of the pair exponential have a mean of -4e-8, which the sum
  // keeps (mean error of the log-probabilities of 1003 standard normals times two +2.7e-8, against -1.3e-8; without that
  // mean it would take 4 % less, with errors up to 2 % larger in some cases and smaller in others). expf takes
  // differences of any size; the pair exponential none below -2.36e38: a thread whose sum is not a number takes its
  // elements again with a floor under them.
  float s;
  bool finite = true;
  if constexpr (sizeof(Tout) == 4) {
    s = add_up(exp_exact);
  } else if constexpr (KEEP) {  // no second try: the row is gone
    s = add_up([&](f32x2 d) { return exp_pair_compensated(clamped(d)); });
  } else {
    s = add_up([](f32x2 d) { return exp_pair_compensated(d); });
    finite = s == s;
    if (!finite) s = add_up([&](f32x2 d) { return exp_pair_compensated(clamped(d)); });
  }
  if (has_edge) s += expf(fmaxf(edge - M, kFloor));
  float sum = block_reduce<SumOp>(s, red);
  if constexpr (CLUSTER) {
    namespace cg = cooperative_groups;
    cg::cluster_group cluster = cg::this_cluster();
    cluster.barrier_wait();
    if (tid < S) {  // this CTA's pair into the table of CTA `tid`
      float* far = cluster.map_shared_rank(&pairs[0][0], tid);
      far[rank] = M;
      far[8 + rank] = sum;
    }
    cluster.sync();  // all pairs are in place; no CTA touches another's memory after this
    M = pairs[0][0];
    for (int r = 1; r < S; ++r) M = MaxOp::apply(M, pairs[0][r]);
    sum = 0.f;
    for (int r = 0; r < S; ++r) {
      // a CTA whose elements are all -inf (or that has none) adds nothing
      if (pairs[0][r] > -INFINITY) sum += pairs[1][r] * expf(fmaxf(pairs[0][r] - M, kFloor));
    }
  }
  // aten: x - max is NaN for a row of -inf and for +inf elements; a NaN logit poisons the row
  if (!(fabsf(M) < INFINITY)) sum = NAN;

  // ---- outputs ------------------------------------------------------------------------------------
  const float log_sum = logf(sum), inv = __frcp_rn(sum);
  const f32x2 M2 = splat2(M), log_sum2 = splat2(log_sum), inv2 = splat2(inv);
  const int shift = (int)(((0u - (unsigned)reinterpret_cast<uintptr_t>(yb)) & (VO * (unsigned)sizeof(Tout) - 1u)) /
                          sizeof(Tout));
  auto store_all = [&](auto plain_tag) {
#pragma unroll
    for (int c = 0; c < CH; ++c) {
      const int j = c * T_ + tid;
      if (j - lane >= cnt) break;  // warp-uniform: no lane of this warp has a vector here
      f32x2 t[P], o[P];
      const bool valid = j < cnt;
      if (!valid) raw[c] = make_uint4(0u, 0u, 0u, 0u);
      if constexpr (KEEP) Pairs<Tin>::unpack(raw[c], t);
      else logits(c, t);
      if constexpr (LOG) {
#pragma unroll
        for (int i = 0; i < P; ++i) o[i] = sub2(sub2(t[i], M2), log_sum2);
      } else if constexpr (KEEP) {
#pragma unroll
        for (int i = 0; i < P; ++i) o[i] = mul2(t[i], inv2);
      } else if constexpr (sizeof(Tout) == 4) {
#pragma unroll
        for (int i = 0; i < P; ++i) {
          float a, b;
          unpack2(exp_exact(sub2(t[i], M2)), a, b);
          o[i] = pack2(a / sum, b / sum);
        }
      } else {
#pragma unroll
        for (int i = 0; i < P; ++i) {
          const f32x2 d = sub2(t[i], M2);
          o[i] = mul2(exp_pair_compensated(decltype(plain_tag)::value ? d : clamped(d)), inv2);
        }
      }
      store_shifted<Tout, V>(yb + (long long)j * V, o, shift, lane, valid, lane < 31 && j + 1 < cnt);
    }
  };
  if constexpr (sizeof(Tout) == 2 && !LOG) {
    // the differences of the sum were in its range; in a cluster they were taken from another maximum
    if (!CLUSTER && __all_sync(0xffffffffu, finite)) store_all(std::true_type{});
    else store_all(std::false_type{});
  } else {
    store_all(std::true_type{});
  }
  if (has_edge) {
    float o;
    if constexpr (LOG) {
      o = (edge - M) - log_sum;
    } else {
      const float e = expf(fmaxf(edge - M, kFloor));
      o = sizeof(Tout) == 4 ? e / sum : e * inv;
    }
    y[edge_at] = Elem<Tout>::from_f32(o);
  }
}

// How many CTAs share a row of nvec whole vectors; 0: the two-sweep kernel below takes it. `aligned`: every row
// starts and ends on the 16-byte grid, on both sides.
//   * As few as hold the row: 64 registers a thread keep 8 vectors and what is computed from them, 512 threads 4096
//     vectors, and a cluster has at most 8 CTAs everywhere. fp32 log-probabilities of 16-bit rows go to two CTAs from 2560
//     vectors on, where only two CTAs fit an SM (bf16 [2000, 30001] 89.1 -> 79.6 us, [2000, 21001] 62.1 -> 59.1; probabilities
//     of the same rows 92.5 -> 98.5, 16-bit results 52.0 -> 59.0). From 8192 vectors on all 8, whose 256 threads fit an
//     SM four times (bf16 [1024, 131075]: 4 CTAs 193 us, 8 CTAs 182, two sweeps 317).
//   * No more than half as many rows as SMs: 8 CTAs once a row has 1024 vectors (bf16 [8, 131072] 7.4 us, two
//     sweeps 17.6; [64, 65536] 9.4 and 12.3; [16, 20005] 4.8, one CTA 5.7; f32 [16, 4099] 4.4 and 5.6).
//   * Up to one row per SM, aligned rows of more than 8192 vectors are read twice: the second sweep finds the row in L2, and a CTA per row
//     loads and stores at its own pace where a cluster waits for its slowest CTA twice a row (f32 [100, 98304] 31 us, clusters 35). So
//     are fp32 rows of more than 16384 vectors on any alignment.
//   * With more rows than SMs (the CTAs of a second wave, or the second row of some SMs, cost the sweeps a whole row's time), only aligned
//     ones of more than 16384 vectors (12288 of 16 bits with fp32 results) are: bf16 [682, 196608] two sweeps 132 us, clusters 171;
//     f32 [682, 98304] 148 and 182. Shorter ones: f32 [1500, 40000] 156 and 136, [195, 65536] 43 and 33; bf16 [300, 98304] 44 and 36; bf16 ->
//     f32 [2000, 67584] 266 and 254, but [1024, 131072] 216 and 219. fp32 rows with 16-bit results of any length: [195, 113832]
//     68 and 48, [682, 98304] 144 and 137. fp32 rows off the grid: [195, 113835] 98 and 64, -> bf16 96 and 48; [682, 98307] 207 and
//     183, -> bf16 198 and 138.
//     But where the sweeps' last row of an SM is there for nine SMs in ten, they are ahead of clusters for 16-bit rows of more than 10240 vectors
//     with 16-bit results: [296, 106000] 36.3 and 41.5, [1024, 106000] 116 and 127, [450, 106000] 66 and 59, [888, 80000] 81 and
//     78. (So they are in fp32, [592, 50000] 73 and 77, but with errors of 1.0e-7 instead of 8e-8.)
//   * fp32 log-probabilities of 16-bit rows are the exception, their sweeps being bound by expf (bf16 -> f32 log [1024, 131072]:
//     250 and 177 us, [682, 196608]: 246 and 237).
template <typename Tin, typename Tout>
static int softmax_ctas_per_row(long long nvec, long long rows, bool aligned, bool log_mode) {
  if (nvec > 8 * 4096) return 0;
  if (2 * rows <= device_info().sm_count && nvec >= 1024) return 8;
  if (nvec > 8192) {
    constexpr bool IN16 = sizeof(Tin) == 2, OUT16 = sizeof(Tout) == 2;
    const long long sms = device_info().sm_count;
    const bool many = rows > sms, full = rows * 10 >= (rows + sms - 1) / sms * sms * 9;
    if (aligned && many && full && IN16 && OUT16 && nvec > 10240) return 0;
    if (aligned && !(log_mode && IN16 && !OUT16) && !(many && ((!IN16 && OUT16) || nvec <= (IN16 && !OUT16 ? 12288 : 16384)))) return 0;
    if (!IN16 && nvec > 16384 && !many) return 0;
    return 8;
  }
  return nvec > (log_mode && sizeof(Tin) == 2 && sizeof(Tout) == 4 ? 2560 : 4096) ? 2 : 1;
}

// Returns false when the two-sweep kernel is to take the rows.
template <typename Tin, typename Tout>
static bool try_launch_softmax_rows(const SoftmaxParams& p, bool aligned, cudaStream_t st, int* rc) {
  const long long nvec = p.n / Elem<Tin>::V;  // no row has more whole vectors, whatever its alignment
  const int S = softmax_ctas_per_row<Tin, Tout>(nvec, p.rows, aligned, p.log_mode != 0);
  if (S == 0 || p.rows * S > 0x7fffffffLL) return false;
  const long long per = (nvec + S - 1) / S;
  const int ch = per > 512 ? 8 : (per > 128 || S > 1 ? 4 : 2);
  const int threads = (int)((per + ch - 1) / ch + 31) / 32 * 32;
  set_path_tag(S > 1 ? "row in the registers of a cluster, any alignment" : "row in the registers of a CTA, any alignment");
  const dim3 grid((unsigned)(p.rows * S)), block((unsigned)threads), cluster((unsigned)S);
  auto launch = [&](auto scaled_tag, auto log_tag) {
    constexpr bool SCALED = decltype(scaled_tag)::value, LOG = decltype(log_tag)::value;
    if (S > 1)
      return ch == 8 ? launch_clusters(cluster, softmax_rows_kernel<Tin, Tout, 8, true, SCALED, LOG>, grid, block, 0, st, p, S)
                     : launch_clusters(cluster, softmax_rows_kernel<Tin, Tout, 4, true, SCALED, LOG>, grid, block, 0, st, p, S);
    if (ch == 8) return launch_dependent(softmax_rows_kernel<Tin, Tout, 8, false, SCALED, LOG>, grid, block, 0, st, p, S);
    return ch == 4 ? launch_dependent(softmax_rows_kernel<Tin, Tout, 4, false, SCALED, LOG>, grid, block, 0, st, p, S)
                   : launch_dependent(softmax_rows_kernel<Tin, Tout, 2, false, SCALED, LOG>, grid, block, 0, st, p, S);
  };
  const std::true_type yes;
  const std::false_type no;
  const cudaError_t e = p.has_scale ? (p.log_mode ? launch(yes, yes) : launch(yes, no)) : (p.log_mode ? launch(no, yes) : launch(no, no));
  if (e != cudaSuccess) {
    cudaGetLastError();
    *rc = fail((int)e, "b200_softmax: launch failed: %s", cudaGetErrorString(e));
    return true;
  }
  *rc = launch_status("b200_softmax");
  return true;
}

// ----------------------------------------------------------------------------------------------
// Rows that softmax_ctas_per_row leaves (beyond 32768 vectors, that is 262 144 16-bit columns; long aligned ones, and fp32
// ones when there are few): one CTA per row, two sweeps.
//   sweep 1: every thread keeps a running maximum m and the sum of exp(t - m) of its elements,
//            rescaling the sum when the maximum grows; the CTA then combines the (m, s) pairs:
//            M = max m_i, S = sum s_i * exp(m_i - M)
//   sweep 2: the row is read again - it was just read by this CTA, so for rows up to a few hundred
//            KB it comes from L2 - and y = exp(t - M) / S (or t - M - log S) is written.
// Both sweeps use 16-byte loads when the row starts on a 16-byte boundary (the ragged tail is read
// element by element) and 16-byte stores when the output row does. No mask; the optional scale is
// applied in fp32.
// ----------------------------------------------------------------------------------------------
// d: differences from a maximum. -inf, and for the pair exponential all that is below its range, has the exponential 0; NaN may be lost.
template <typename Tout>
__device__ __forceinline__ f32x2 long_row_exp(f32x2 d) {
  float a, b;
  unpack2(d, a, b);
  if constexpr (sizeof(Tout) == 2) {
    constexpr float kFloor = -1e30f;
    return exp_pair_compensated(pack2(fmaxf(a, kFloor), fmaxf(b, kFloor)));
  } else {
    return pack2(expf(a), expf(b));
  }
}

template <typename Tin, typename Tout>
__global__ void __launch_bounds__(1024) softmax_long_kernel(const SoftmaxParams p) {
  wait_for_previous_kernel();
  constexpr int V = Elem<Tin>::V;
  constexpr int P = V / 2;
  constexpr int U = 4;  // vectors in flight per thread
  __shared__ float red[64];
  const long long row = blockIdx.x;
  const Tin* x = reinterpret_cast<const Tin*>(p.x) + row_offset(p.xmap, row);
  Tout* y = reinterpret_cast<Tout*>(p.y) + row_offset(p.ymap, row);
  const int tid = threadIdx.x, T_ = blockDim.x;
  const bool x_vec = (reinterpret_cast<uintptr_t>(x) & 15u) == 0;
  const int nvec = x_vec ? p.n / V : 0;
  const int body = nvec * V;  // elements covered by whole vectors
  const f32x2 scale2 = splat2(p.has_scale ? p.scale : 1.0f);
  const bool scaled = p.has_scale != 0;

  // ---- sweep 1 ----------------------------------------------------------------------------------
  float m = -INFINITY, s = 0.f;
  auto over_m = [&] { return m == -INFINITY ? 0.f : m; };  // nothing but -inf so far: their differences from any number are -inf
  auto absorb = [&](const f32x2 (&t)[P]) {  // one vector of logits into (m, s)
    float vm = -INFINITY;
#pragma unroll
    for (int i = 0; i < P; ++i) {
      float a, b;
      unpack2(t[i], a, b);
      vm = fmaxf(vm, fmaxf(a, b));
    }
    if (vm > m) {
      s = s * expf(m - vm);  // m = -inf the first time: the sum is still zero
      m = vm;
    }
    const f32x2 m2 = splat2(over_m());
    f32x2 acc = splat2(0.f);
#pragma unroll
    for (int i = 0; i < P; ++i) acc = add2(acc, long_row_exp<Tout>(sub2(t[i], m2)));
    s += hsum2(acc);
  };
  bool saw_nan = false;
  for (int j0 = tid; j0 < nvec; j0 += U * T_) {
    uint4 raw[U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int j = j0 + u * T_;
      if (j < nvec) raw[u] = ld_keep(x + (long long)j * V);  // read again in sweep 2: keep it cached
    }
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int j = j0 + u * T_;
      if (j < nvec) {
        f32x2 t[P];
        Pairs<Tin>::unpack(raw[u], t);
        if (scaled) {
#pragma unroll
          for (int i = 0; i < P; ++i) t[i] = mul2(t[i], scale2);
        }
#pragma unroll
        for (int i = 0; i < P; ++i) {
          float a, b;
          unpack2(t[i], a, b);
          saw_nan |= (a != a) | (b != b);
        }
        absorb(t);
      }
    }
  }
  for (int i = body + tid; i < p.n; i += T_) {  // ragged tail, or the whole row when it is unaligned
    float t = Elem<Tin>::to_f32(x[i]);
    if (scaled) t = t * p.scale;
    saw_nan |= t != t;
    if (t > m) {
      s = s * expf(m - t);
      m = t;
    }
    s += expf(t - over_m());
  }
  // CTA-wide (M, S)
  const float M = block_reduce<FastMax>(m, red);
  const float contrib = (m == -INFINITY) ? 0.f : s * expf(m - M);
  float S = block_reduce<SumOp>(contrib, red);
  const float nan_any = block_reduce<FastMax>(saw_nan ? 1.f : 0.f, red);
  if (!(fabsf(M) < INFINITY) || nan_any > 0.f) S = NAN;  // aten: x - max is NaN for a row of -inf and for inf; NaN logits poison the row

  // ---- sweep 2 ----------------------------------------------------------------------------------
  const float logS = logf(S);
  const float inv = __frcp_rn(S);
  const bool log_mode = p.log_mode != 0;
  auto finish = [&](float t) -> float {  // one logit -> one output value
    if (log_mode) return (t - M) - logS;
    const float e = expf(t - M);
    return sizeof(Tout) == 4 ? e / S : e * inv;
  };
  constexpr int VO = 16 / (int)sizeof(Tout);           // output elements per 16-byte store
  const bool y_vec = x_vec && (reinterpret_cast<uintptr_t>(y) & 15u) == 0 && V % VO == 0;
  const f32x2 M2 = splat2(M), inv2 = splat2(inv), logS2 = splat2(logS);
  if (!y_vec) {
    // The output row does not start on a 16-byte boundary where the input row does (a ragged row
    // length, another element size): vectors are formed on the OUTPUT side - up to the first
    // boundary element by element, then 16-byte stores whose inputs are read element by element
    // (they were read a moment ago and come from L1 / L2), then the rest.
    int ho = (int)(((16u - (unsigned)(reinterpret_cast<uintptr_t>(y) & 15u)) & 15u) / sizeof(Tout));
    if (ho > p.n) ho = p.n;
    const int nout = (p.n - ho) / VO;
    for (int i = tid; i < ho; i += T_) {
      float t = Elem<Tin>::to_f32(x[i]);
      if (scaled) t = t * p.scale;
      y[i] = Elem<Tout>::from_f32(finish(t));
    }
    for (int j = tid; j < nout; j += T_) {
      const int i0 = ho + j * VO;
      float o[VO];
#pragma unroll
      for (int k = 0; k < VO; ++k) o[k] = Elem<Tin>::to_f32(x[i0 + k]);
#pragma unroll
      for (int k = 0; k < VO; ++k) {
        if (scaled) o[k] = o[k] * p.scale;
        o[k] = finish(o[k]);
      }
      store_converted<Tout, VO>(y + i0, o);
    }
    for (int i = ho + nout * VO + tid; i < p.n; i += T_) {
      float t = Elem<Tin>::to_f32(x[i]);
      if (scaled) t = t * p.scale;
      y[i] = Elem<Tout>::from_f32(finish(t));
    }
    return;
  }
  for (int j0 = tid; j0 < nvec; j0 += U * T_) {
    uint4 raw[U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int j = j0 + u * T_;
      if (j < nvec) raw[u] = ld_stream(x + (long long)j * V);
    }
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int j = j0 + u * T_;
      if (j < nvec) {
        f32x2 t[P], o[P];
        Pairs<Tin>::unpack(raw[u], t);
#pragma unroll
        for (int i = 0; i < P; ++i) {
          if (scaled) t[i] = mul2(t[i], scale2);
          if (log_mode) {
            o[i] = sub2(sub2(t[i], M2), logS2);
          } else {
            const f32x2 e = long_row_exp<Tout>(sub2(t[i], M2));
            if constexpr (sizeof(Tout) == 4) {
              float ea, eb;
              unpack2(e, ea, eb);
              o[i] = pack2(ea / S, eb / S);
            } else {
              o[i] = mul2(e, inv2);
            }
          }
        }
        store_pairs<Tout, V>(y + (long long)j * V, o);
      }
    }
  }
  for (int i = body + tid; i < p.n; i += T_) {
    float t = Elem<Tin>::to_f32(x[i]);
    if (scaled) t = t * p.scale;
    y[i] = Elem<Tout>::from_f32(finish(t));
  }
}

template <typename Tin, typename Tout, bool PACKED>
static int launch_softmax(const SoftmaxParams& p, bool vector_ok, cudaStream_t st) {
  constexpr int V = Elem<Tin>::V;
  RowGeometry g;
  if (p.rows > 0x7fffffffLL) return fail(B200_ERR_UNSUPPORTED, "softmax: too many rows");
  if (vector_ok && p.n % V == 0 && pick_row_geometry(p.n / V, &g)) {
    set_path_tag(g.block ? "vector, row resident, CTA per row" : "vector, row resident, sub-warp rows");
    if (!g.block) {
      const int rows_per_cta = g.threads / g.g;
      const unsigned grid = (unsigned)((p.rows + rows_per_cta - 1) / rows_per_cta);
#define B200_SM_LAUNCH(GG, CC)                                                                   \
  do {                                                                                          \
    if (GG > 0 && p.n / V == (long long)GG * CC)                                                \
      launch_dependent(softmax_resident_kernel<Tin, Tout, CC, GG, PACKED, (GG > 0)>, grid, g.threads, 0, st, p); \
    else                                                                                        \
      launch_dependent(softmax_resident_kernel<Tin, Tout, CC, GG, PACKED, false>, grid, g.threads, 0, st, p);   \
  } while (0)
      if (g.g == 8) {
        if (g.ch == 1) B200_SM_LAUNCH(8, 1);
        else if (g.ch == 2) B200_SM_LAUNCH(8, 2);
        else B200_SM_LAUNCH(8, 4);
      } else if (g.g == 16) {
        B200_SM_LAUNCH(16, 4);
      } else {
        B200_SM_LAUNCH(32, 4);
      }
    } else {
      const unsigned grid = (unsigned)p.rows;
      if (g.ch == 2) B200_SM_LAUNCH(0, 2);
      else if (g.ch == 4) B200_SM_LAUNCH(0, 4);
      else B200_SM_LAUNCH(0, 8);
#undef B200_SM_LAUNCH
    }
  } else if (p.mask == nullptr && !PACKED && p.n >= 256) {
    int rc = B200_OK;
    if (try_launch_softmax_rows<Tin, Tout>(p, vector_ok && p.n % V == 0, st, &rc)) return rc;
    int threads = (int)((p.n / V + 3) / 4);
    threads = (threads + 31) / 32 * 32;
    threads = threads < 128 ? 128 : (threads > 1024 ? 1024 : threads);
    set_path_tag("two sweeps, CTA per row");
    launch_dependent(softmax_long_kernel<Tin, Tout>, (unsigned)p.rows, threads, 0, st, p);
  } else if (p.n <= 8192) {
    set_path_tag("elements in registers");
    if constexpr (std::is_same<Tin, Tout>::value && sizeof(Tin) == 2 && !PACKED) {
      if (try_launch_softmax_span<Tin>(p, st)) return launch_status("b200_softmax");
    }
    if (p.n > 64 && p.n <= 2048 && p.rows <= (p.n <= 512 ? 4LL : 2LL) * device_info().sm_count) {
      launch_dependent(softmax_ragged_kernel<Tin, Tout, PACKED, 2, 0>, (unsigned)p.rows, ((p.n + 1) / 2 + 31) / 32 * 32, 0, st, p);
    } else if (p.n <= 512) {
      const unsigned grid = (unsigned)((p.rows + 7) / 8);
      if (p.n <= 64) launch_dependent(softmax_ragged_kernel<Tin, Tout, PACKED, 2, 32>, grid, 256, 0, st, p);
      else if (p.n <= 128) launch_dependent(softmax_ragged_kernel<Tin, Tout, PACKED, 4, 32>, grid, 256, 0, st, p);
      else if (p.n <= 256) launch_dependent(softmax_ragged_kernel<Tin, Tout, PACKED, 8, 32>, grid, 256, 0, st, p);
      else launch_dependent(softmax_ragged_kernel<Tin, Tout, PACKED, 16, 32>, grid, 256, 0, st, p);
    } else {
      const int threads = ((p.n + 7) / 8 + 31) / 32 * 32;
      launch_dependent(softmax_ragged_kernel<Tin, Tout, PACKED, 8, 0>, (unsigned)p.rows, threads, 0, st, p);
    }
  } else {
    const int threads = 1024;
    set_path_tag("element-wise, three passes");
    launch_dependent(softmax_streaming_kernel<Tin, Tout, PACKED>, (unsigned)p.rows, threads, 0, st, p);
  }
  return launch_status("b200_softmax");
}

template <typename Tin, typename Tout>
static int launch_softmax_pro(const SoftmaxParams& p, bool packed, bool vector_ok, cudaStream_t st) {
  if constexpr (sizeof(Tin) == 2) {
    if (packed) return launch_softmax<Tin, Tout, true>(p, vector_ok, st);
  }
  return launch_softmax<Tin, Tout, false>(p, vector_ok, st);
}

}  // namespace b200

using namespace b200;

static bool map_vector_ok(const RowMap& m, int elem_bytes, int chunk) {
  // every row start stays `chunk`-byte aligned when all outer strides are multiples of it
  return (m.s0 * elem_bytes) % chunk == 0 && (m.s1 * elem_bytes) % chunk == 0 &&
         (m.s2 * elem_bytes) % chunk == 0;
}

static bool survives_round_trip(float v, int dtype) {
  if (dtype == B200_F16) return __half2float(__float2half_rn(v)) == v;
  if (dtype == B200_BF16) return __bfloat162float(__float2bfloat16_rn(v)) == v;
  return true;
}

extern "C" int b200_softmax(const void* x, const void* mask, void* y, int64_t rows, int64_t n,
                            int64_t d1, int64_t d2, const int64_t* x_strides,
                            const int64_t* mask_strides, const int64_t* y_strides, int32_t in_dtype,
                            int32_t out_dtype, double scale, int32_t flags, void* stream) {
  if (!x || !y || !x_strides || !y_strides) return fail(B200_ERR_INVALID, "b200_softmax: null argument");
  if (rows < 0 || n < 0 || d1 < 1 || d2 < 1 || n > 0x7fffffffLL)
    return fail(B200_ERR_INVALID, "b200_softmax: bad sizes rows=%lld n=%lld", (long long)rows, (long long)n);
  if (mask && !mask_strides) return fail(B200_ERR_INVALID, "b200_softmax: mask without strides");
  if (rows == 0 || n == 0) return B200_OK;
  if (rows % (d1 * d2) != 0) return fail(B200_ERR_INVALID, "b200_softmax: rows not divisible by d1*d2");

  SoftmaxParams p;
  p.x = x; p.mask = mask; p.y = y; p.rows = rows; p.n = (int)n;
  if (rows > 0x7fffffffLL) return fail(B200_ERR_UNSUPPORTED, "b200_softmax: more than 2^31-1 rows");
  p.xmap = make_row_map(x_strides, d1, d2);
  p.ymap = make_row_map(y_strides, d1, d2);
  p.mmap = mask ? make_row_map(mask_strides, d1, d2) : make_row_map_flat(0);
  p.scale = (float)scale;
  p.has_scale = (flags & B200_SOFTMAX_SCALE) ? 1 : 0;
  p.scale_exact16 = survives_round_trip(p.scale, in_dtype) ? 1 : 0;
  p.log_mode = (flags & B200_SOFTMAX_LOG) ? 1 : 0;
  const bool packed = (flags & B200_SOFTMAX_ROUND) != 0 && in_dtype != B200_F32 &&
                      (p.has_scale || mask != nullptr);

  const int ib = dtype_size(in_dtype), ob = dtype_size(out_dtype);
  const int v_in = 16 / ib;
  const int out_chunk = v_in * ob < 16 ? v_in * ob : 16;
  bool vec = aligned16(x) && map_vector_ok(p.xmap, ib, 16) &&
             (reinterpret_cast<uintptr_t>(y) % out_chunk == 0) && map_vector_ok(p.ymap, ob, out_chunk);
  if (mask) vec = vec && aligned16(mask) && map_vector_ok(p.mmap, ib, 16);
  cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);

#define B200_SOFTMAX_CASE(TI, TO, DI, DO) \
  if (in_dtype == DI && out_dtype == DO) return launch_softmax_pro<TI, TO>(p, packed, vec, st);
  B200_SOFTMAX_CASE(float, float, B200_F32, B200_F32)
  B200_SOFTMAX_CASE(__nv_bfloat16, __nv_bfloat16, B200_BF16, B200_BF16)
  B200_SOFTMAX_CASE(__half, __half, B200_F16, B200_F16)
  B200_SOFTMAX_CASE(__nv_bfloat16, float, B200_BF16, B200_F32)
  B200_SOFTMAX_CASE(__half, float, B200_F16, B200_F32)
  B200_SOFTMAX_CASE(float, __nv_bfloat16, B200_F32, B200_BF16)
  B200_SOFTMAX_CASE(float, __half, B200_F32, B200_F16)
#undef B200_SOFTMAX_CASE
  return fail(B200_ERR_UNSUPPORTED, "b200_softmax: dtype pair (%d -> %d) not built", in_dtype, out_dtype);
}
