// Row reductions over the last (contiguous) dimension: sum, mean, amax, amin.
//
// Replaces the row-form Triton kernels of the mean/sum/amax repros in the reference
// (repros/canonical/mean_c9e1a8113328/oracle.py:11-76 for the contiguous case,
// amax_sum_7079889cfc04/oracle.py:20-29 for the long-row loop).
//
// 4 to 32 lanes (rows of up to 256 vectors of 16 bytes), one warp (many longer rows) or one CTA (few or long rows) read a
// row once with four or eight 16-byte loads in flight per thread, accumulating in fp32 in V independent chains per
// thread, then a fixed-order shuffle/shared-memory tree. mean multiplies the sum by 1/n, as aten does.
// Rows may start and end anywhere: the body is loaded as whole vectors from the first 16-byte boundary on, the at
// most 2 (V - 1) elements beside it one per lane, asked for together with the vectors.
#include "rowwise.cuh"

#include <type_traits>

namespace b200 {

#define B200_REDUCE_SUM 0
#define B200_REDUCE_MEAN 1
#define B200_REDUCE_AMAX 2
#define B200_REDUCE_AMIN 3

struct RowReduceParams {
  const void* x;
  void* out;
  long long rows;
  long long n;
  RowMap xmap;
  long long out_stride;
  int out_dtype;
  float post_scale;  // 1/n for mean, 1 otherwise
};

__device__ __forceinline__ void store_scalar(void* out, int dtype, long long idx, float v) {
  if (dtype == B200_F32) {
    reinterpret_cast<float*>(out)[idx] = v;
  } else if (dtype == B200_BF16) {
    reinterpret_cast<__nv_bfloat16*>(out)[idx] = __float2bfloat16_rn(v);
  } else {
    reinterpret_cast<__half*>(out)[idx] = __float2half_rn(v);
  }
}

// The whole vectors of a row and the elements in front of and behind them.
template <typename I>
struct RowBody {
  int head;   // elements in front of the first 16-byte boundary
  int edges;  // those and the ones behind the last whole vector
  I nv;       // whole vectors
  I tail0;
};
template <typename I, typename T>
__device__ __forceinline__ RowBody<I> row_body(const T* x, I n) {
  constexpr int V = Elem<T>::V;
  RowBody<I> b;
  b.head = (int)(((16u - (unsigned)(reinterpret_cast<uintptr_t>(x) & 15u)) & 15u) / sizeof(T));
  if (b.head > n) b.head = (int)n;
  b.nv = (n - b.head) / V;
  b.tail0 = b.head + b.nv * V;
  b.edges = b.head + (int)(n - b.tail0);
  return b;
}

// s = a + b and what the addition rounded away (Knuth, TAOCP vol. 2, 4.2.2, theorem B): exact for finite s.
__device__ __forceinline__ f32x2 two_sum2(f32x2 a, f32x2 b, f32x2& rounded_away) {
  const f32x2 s = add2(a, b), bb = sub2(s, a);
  rounded_away = add2(sub2(a, sub2(s, bb)), sub2(b, bb));
  return s;
}

// What a thread holds of its row.
// Sums: V chains as pairs, joined without loss and only then converted: an addition takes part in the fp64 total with two
// conversions a thread, which run at 16 a clock and SM (fp32 [60000, 256] with every element converted 14.8 us, so 11.1).
//   kPlain   a chain is a chain of fp32 additions
//   kPairs   the vectors of a batch are added two by two; what the additions above round away is kept
//   kKept    what any addition rounds away is kept
// 16-bit elements are always kPlain: a short chain of values of 8 or 11 bits rarely rounds at all. fp32 rows are kKept up to
// 128 vectors and kPairs up to 256, where the CTA of 64 threads that took a row before had chains of one or two and of up to four
// additions (error of the sum of 333 / 946 standard normals, rows off the 16-byte grid, 5.3 / 7.8e-8 there, 2.5 / 3.6e-8 here;
// of 512 / 1024 3.7 / 4.8e-8 and 2.5 / 3.7e-8). [60000, 512] as plain chains 18.6 us, kept 19.9.
enum SumKind { kPlain, kPairs, kKept };
template <typename Tin, SumKind KIND>
struct SumChains {
  static constexpr int P = Elem<Tin>::V / 2;
  static constexpr SumKind kind = sizeof(Tin) == 4 ? KIND : kPlain;
  f32x2 hi[P], lo;
  __device__ __forceinline__ SumChains() {
#pragma unroll
    for (int i = 0; i < P; ++i) hi[i] = splat2(0.f);
    lo = splat2(0.f);
  }
  __device__ __forceinline__ void add_pair(f32x2& h, f32x2 v) {
    f32x2 e;
    h = two_sum2(h, v, e);
    lo = add2(lo, e);
  }
  static __device__ __forceinline__ uint4 nothing() { return make_uint4(0u, 0u, 0u, 0u); }
  // A batch of vectors, of which those with live(u) are there; the others are nothing().
  template <int U, typename Live>
  __device__ __forceinline__ void add(const uint4 (&raw)[U], Live&& live) {
#pragma unroll
    for (int u = 0; u < U; u += kind == kPairs ? 2 : 1) {
      f32x2 f[P], g[P];
      Pairs<Tin>::unpack(raw[u], f);
      if constexpr (kind == kPairs) {
        Pairs<Tin>::unpack(raw[u + 1], g);
#pragma unroll
        for (int i = 0; i < P; ++i) add_pair(hi[i], add2(f[i], g[i]));
      } else if constexpr (kind == kKept) {
        if (live(u)) {
#pragma unroll
          for (int i = 0; i < P; ++i) add_pair(hi[i], f[i]);
        }
      } else {
#pragma unroll
        for (int i = 0; i < P; ++i) hi[i] = add2(hi[i], f[i]);
      }
    }
  }
  __device__ __forceinline__ void add_one(float f) { add_pair(hi[0], pack2(f, 0.f)); }
  __device__ __forceinline__ double total() {
    f32x2 h[P];
#pragma unroll
    for (int i = 0; i < P; ++i) h[i] = hi[i];
#pragma unroll
    for (int w = P / 2; w > 0; w >>= 1) {
#pragma unroll
      for (int i = 0; i < w; ++i) add_pair(h[i], h[i + w]);
    }
    float a, b, la, lb;
    unpack2(h[0], a, b);
    add_pair(h[0], pack2(b, 0.f));  // its first half is a + b now
    unpack2(h[0], a, b);
    unpack2(lo, la, lb);
    double d = (double)a + (double)(la + lb);
    if (!(fabsf(a) < INFINITY)) {  // the chains may have a sum all the same; of infinities nothing is rounded away
      d = 0.0;
#pragma unroll
      for (int i = 0; i < P; ++i) {
        unpack2(hi[i], a, b);
        d += (double)a;
        d += (double)b;
      }
    }
    return d;
  }
};

// Extremes: fp32 in V chains, 16-bit elements, whose extremes are exact in the storage type, as packed pairs (one
// instruction per two elements, no conversion).
template <typename Tin, typename Op>
struct ExtremeChains {
  static constexpr int V = Elem<Tin>::V;
  static constexpr bool PACKED = sizeof(Tin) == 2;
  using P2 = typename std::conditional<std::is_same<Tin, __half>::value, __half2, __nv_bfloat162>::type;
  float acc[PACKED ? 1 : V];
  P2 m[PACKED ? 4 : 1];

  __device__ __forceinline__ ExtremeChains() {
#pragma unroll
    for (int i = 0; i < (PACKED ? 1 : V); ++i) acc[i] = Op::identity();
    if constexpr (PACKED) {
      const Tin id = Elem<Tin>::from_f32(Op::identity());
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        m[i].x = id;
        m[i].y = id;
      }
    }
  }
  static __device__ __forceinline__ uint4 nothing() {
    float f[V];
#pragma unroll
    for (int i = 0; i < V; ++i) f[i] = Op::identity();
    return Elem<Tin>::pack(f);
  }
  template <int U, typename Live>
  __device__ __forceinline__ void add(const uint4 (&raw)[U], Live&&) {
#pragma unroll
    for (int u = 0; u < U; ++u) {
      if constexpr (PACKED) {
        const uint32_t w[4] = {raw[u].x, raw[u].y, raw[u].z, raw[u].w};
#pragma unroll
        for (int i = 0; i < 4; ++i) m[i] = Op::apply2(m[i], *reinterpret_cast<const P2*>(&w[i]));
      } else {
        float f[V];
        Elem<Tin>::unpack(raw[u], f);
#pragma unroll
        for (int i = 0; i < V; ++i) acc[i] = Op::apply(acc[i], f[i]);
      }
    }
  }
  __device__ __forceinline__ void add_one(float f) { acc[0] = Op::apply(acc[0], f); }
  __device__ __forceinline__ float extreme() const {
    if constexpr (PACKED) {
      const P2 a = Op::apply2(Op::apply2(m[0], m[1]), Op::apply2(m[2], m[3]));
      return Op::apply(acc[0], Op::apply(Elem<Tin>::to_f32(a.x), Elem<Tin>::to_f32(a.y)));
    } else {
      float r = acc[0];
#pragma unroll
      for (int i = 1; i < V; ++i) r = Op::apply(r, acc[i]);
      return r;
    }
  }
};

template <typename Tin, typename Op, SumKind KIND>
using RowChains = typename std::conditional<Op::is_sum, SumChains<Tin, KIND>, ExtremeChains<Tin, Op>>::type;

// A warp per row that starts on a 16-byte boundary, four 16-byte loads in flight per lane and at most 32 registers, so that 64 warps fit
// on an SM. Bound by HBM: fp32 [8192, 4096] 21.5 us, 6.2 TB/s; with the head and the edges of the kernel below and its joins of the chains
// 21.8, and where the rows are in L2 up to twice as long (amax bf16 [2400, 8000] 5.9 and 12.1).
template <typename Tin, typename Op>
__global__ void __launch_bounds__(256, 8) row_reduce_grid_kernel(const RowReduceParams p) {
  wait_for_previous_kernel();
  constexpr int V = Elem<Tin>::V;
  constexpr int U = 4, G = 32;
  const int lane = group_lane<false>();
  const long long row = group_row<false>();
  if (row >= p.rows) return;
  const Tin* x = reinterpret_cast<const Tin*>(p.x) + row_offset(p.xmap, row);
  const long long nv = p.n / V;

  float acc[V];
#pragma unroll
  for (int i = 0; i < V; ++i) acc[i] = Op::identity();
  auto walk = [&](auto&& add) {
    for (long long j0 = lane; j0 < nv; j0 += (long long)G * U) {
      uint4 raw[U];
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const long long j = j0 + (long long)u * G;
        if (j < nv) raw[u] = ld_stream(x + j * V);
      }
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const long long j = j0 + (long long)u * G;
        if (j < nv) add(raw[u]);
      }
    }
  };
  if constexpr (!Op::is_sum && sizeof(Tin) == 2) {  // exact in the storage type: packed pairs, only the last of a thread is widened
    using P2 = typename std::conditional<std::is_same<Tin, __half>::value, __half2, __nv_bfloat162>::type;
    P2 m[4];
    {
      const Tin id = Elem<Tin>::from_f32(Op::identity());
      P2 idp;
      idp.x = id;
      idp.y = id;
#pragma unroll
      for (int i = 0; i < 4; ++i) m[i] = idp;
    }
    walk([&](const uint4& v) {
      const uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
      for (int i = 0; i < 4; ++i) m[i] = Op::apply2(m[i], *reinterpret_cast<const P2*>(&w[i]));
    });
    const P2 a = Op::apply2(Op::apply2(m[0], m[1]), Op::apply2(m[2], m[3]));
    acc[0] = Op::apply(Elem<Tin>::to_f32(a.x), Elem<Tin>::to_f32(a.y));
  } else {
    walk([&](const uint4& v) {
      float f[V];
      Elem<Tin>::unpack(v, f);
#pragma unroll
      for (int i = 0; i < V; ++i) acc[i] = Op::apply(acc[i], f[i]);
    });
  }
  for (long long i = nv * V + lane; i < p.n; i += G) acc[0] = Op::apply(acc[0], Elem<Tin>::to_f32(x[i]));

  float r;
  if constexpr (Op::is_sum) {
    // Chains are short (tens of elements); what is above them is combined in fp64, so that the result is the correctly rounded
    // sum of the chains.
    double d = 0.0;
#pragma unroll
    for (int i = 0; i < V; ++i) d += (double)acc[i];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) d += __shfl_xor_sync(0xffffffffu, d, o);
    r = (float)d;
  } else {
#pragma unroll
    for (int w = V / 2; w > 0; w >>= 1) {
#pragma unroll
      for (int i = 0; i < w; ++i) acc[i] = Op::apply(acc[i], acc[i + w]);
    }
    r = warp_reduce<Op>(acc[0]);
  }
  if (lane == 0) store_scalar(p.out, p.out_dtype, row * p.out_stride, r * p.post_scale);
}

// Rows that start and end anywhere. Warp mode: CTAS of 256 threads an SM. Six with U = 4, or four with U = 8, where all rows are then there at
// once: with the 32 registers of eight CTAs the loads and the edges spill (bf16 sum [5000, 5001] 9.2 us with eight, 7.7 with six). By the
// element [5000, 5001] takes 15.7, [8192, 1101] fp32 4.7 and 5.1 so, [5000, 2049] fp32 5.6 and 6.5: the two of some 200 shapes that lose.
// I: index type, long long for rows of 2^30 elements and more.
template <typename Tin, typename Op, bool BLOCK, typename I, int CTAS = 1>
__global__ void __launch_bounds__(BLOCK ? 1024 : 256, CTAS)
row_reduce_kernel(const RowReduceParams p) {
  wait_for_previous_kernel();
  constexpr int V = Elem<Tin>::V;
  constexpr int U = BLOCK || CTAS == 4 ? 8 : 4;
  __shared__ __align__(8) float red[64];
  const int lane = group_lane<BLOCK>();
  const int G = group_size<BLOCK>();
  const long long row = group_row<BLOCK>();
  if (row >= p.rows) return;
  const Tin* x = reinterpret_cast<const Tin*>(p.x) + row_offset(p.xmap, row);
  const RowBody<I> b = row_body<I>(x, (I)p.n);
  const Tin* xb = x + b.head;

  RowChains<Tin, Op, kPlain> chains;
  float edge = Op::identity();
  if (lane < b.edges) edge = Elem<Tin>::to_f32(ld_here(x + (lane < b.head ? lane : b.tail0 + (lane - b.head))));
  I j0 = lane;
  if constexpr (!BLOCK) {  // whole batches without a question asked
    for (; j0 + (U - 1) * G < b.nv; j0 += G * U) {
      uint4 raw[U];
#pragma unroll
      for (int u = 0; u < U; ++u) raw[u] = ld_stream(xb + (j0 + u * G) * V);
      chains.add(raw, [](int) { return true; });
    }
  }
  for (; j0 < b.nv; j0 += G * U) {
    uint4 raw[U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const I j = j0 + u * G;
      raw[u] = RowChains<Tin, Op, kPlain>::nothing();
      if (j < b.nv) raw[u] = ld_stream(xb + j * V);
    }
    chains.add(raw, [&](int u) { return j0 + u * G < b.nv; });
  }
  chains.add_one(edge);

  float r;
  if constexpr (Op::is_sum) {
    double d = chains.total();
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) d += __shfl_xor_sync(0xffffffffu, d, o);
    if constexpr (BLOCK) {
      double* dred = reinterpret_cast<double*>(red);
      const int warp = threadIdx.x >> 5, nwarps = (blockDim.x + 31) >> 5;
      if ((threadIdx.x & 31) == 0) dred[warp] = d;
      __syncthreads();
      d = 0.0;
      for (int w = 0; w < nwarps; ++w) d += dred[w];
    }
    r = (float)d;
  } else {
    r = group_reduce<Op, BLOCK>(chains.extreme(), red);
  }
  if (lane == 0) store_scalar(p.out, p.out_dtype, row * p.out_stride, r * p.post_scale);
}

// The row again, element by element in fp64, for the lanes of a row whose total is no finite number: infinities and NaN come
// out as they are, and a row whose chains left the range of fp32 although its sum is inside gets its sum, as it did when a
// thread held one element of such a row. (In the kernel above the mere call takes 0.5 of 21.1 us, fp32 [8192, 4096].)
template <typename Tin>
static __device__ __noinline__ double sum_in_fp64(const Tin* x, long long n, int lane, int lanes) {
  double d = 0.0;
  for (long long i = lane; i < n; i += lanes) d += (double)Elem<Tin>::to_f32(x[i]);
  return d;
}

// Rows of at most K L whole vectors: L lanes a row, 32 / L rows a warp, every load of a thread on its way at once. Bound by
// the warps' instructions where rows are very short (bf16 [60000, 64], 7.7 MB, 2.7 us) and by HBM above (fp32 [60000, 256]
// 10.0 us, 6.1 TB/s).
template <typename Tin, typename Op, int L, int K, SumKind KIND>
__global__ void __launch_bounds__(256, K == 4 ? 6 : 4) row_reduce_short_kernel(const RowReduceParams p) {
  wait_for_previous_kernel();
  constexpr int V = Elem<Tin>::V;
  constexpr int E = (2 * (V - 1) + L - 1) / L;  // elements beside the vectors, per lane
  const int lane = threadIdx.x & (L - 1);
  long long row = (long long)blockIdx.x * (256 / L) + threadIdx.x / L;
  const bool valid = row < p.rows;  // a partly filled last CTA takes the last row again
  if (!valid) row = p.rows - 1;
  const Tin* x = reinterpret_cast<const Tin*>(p.x) + row_offset(p.xmap, row);
  const RowBody<int> b = row_body<int>(x, (int)p.n);
  const Tin* xb = x + b.head;
  const int nv = b.nv;

  uint4 raw[K];
#pragma unroll
  for (int k = 0; k < K; ++k) {
    raw[k] = RowChains<Tin, Op, KIND>::nothing();
    if (k * L + lane < nv) raw[k] = ld_stream(xb + (k * L + lane) * V);
  }
  RowChains<Tin, Op, KIND> chains;
#pragma unroll
  for (int e = 0; e < E; ++e) {
    const int i = e * L + lane;
    if (i < b.edges) chains.add_one(Elem<Tin>::to_f32(ld_here(x + (i < b.head ? i : b.tail0 + (i - b.head)))));
  }
  chains.add(raw, [&](int k) { return k * L + lane < nv; });

  float r;
  if constexpr (Op::is_sum) {
    auto add_up = [](double d) {
#pragma unroll
      for (int o = L / 2; o > 0; o >>= 1) d += __shfl_xor_sync(0xffffffffu, d, o);
      return d;
    };
    double d = add_up(chains.total());
    if (__any_sync(0xffffffffu, !(fabs(d) < INFINITY))) d = add_up(sum_in_fp64<Tin>(x, p.n, lane, L));
    r = (float)d;
  } else {
    r = chains.extreme();
#pragma unroll
    for (int o = L / 2; o > 0; o >>= 1) r = Op::apply(r, __shfl_xor_sync(0xffffffffu, r, o));
  }
  if (lane == 0 && valid) store_scalar(p.out, p.out_dtype, row * p.out_stride, r * p.post_scale);
}

template <typename Tin, typename Op>
static int launch_row_reduce(const RowReduceParams& p, bool on_grid, cudaStream_t st) {
  constexpr int V = Elem<Tin>::V;
  const int sms = device_info().sm_count;
  if (p.rows > 0x7fffffffLL) return fail(B200_ERR_UNSUPPORTED, "row_reduce: too many rows");
  const long long nv = p.n / V;
  // CTA-per-row geometry: about eight vectors per thread.
  int threads = (int)((nv + 7) / 8);
  threads = (threads + 31) / 32 * 32;
  threads = threads < 64 ? 64 : (threads > 1024 ? 1024 : threads);
  // Tail model: work that needs more than one wave of resident CTAs loses the unfilled part of
  // its last wave. Warp-per-row (8 rows per 256-thread CTA, 8 CTAs per SM) needs enough rows to
  // fill the machine and rows short enough for one warp; otherwise one CTA per row.
  auto efficiency = [&](double units, double resident_per_sm) {
    const double waves = units / (sms * resident_per_sm);
    return waves <= 1.0 ? 1.0 : waves / (double)(long long)(waves + 0.999999);
  };
  const double eff_warp = efficiency((double)((p.rows + 7) / 8), 8.0);
  const double eff_block = efficiency((double)p.rows, (double)(2048 / threads > 32 ? 32 : 2048 / threads));
  // Rows of up to 128 vectors, whatever their number, and of up to 256 from four an SM on: all of a row's loads in one to 32
  // lanes at once. A CTA (of 64 threads) for each of many short rows costs its launch, 0.6 ns a row over the whole GPU: fp32
  // [60000, 64] 37.1 us as CTAs, 10.9 with a warp per row, 3.0 so, [64, 64] 1.9, 1.5 and 1.4; [60000, 640] 49.1, 24.0 (chains of fp32
  // additions) and 23.8, [2000, 946] 3.5, 2.2 and 2.2; bf16 [60000, 512] 46.9, 16.1 and 10.7, [10000, 2048] 11.0, 9.1 and 7.5,
  // [64, 1500] off the grid 3.3, 2.4 and 2.1.
  auto short_rows = [&](auto kernel, int lanes) {
    const int rows_per_cta = 256 / lanes;
    set_path_tag("several rows a warp");
    launch_dependent(kernel, (unsigned)((p.rows + rows_per_cta - 1) / rows_per_cta), 256, 0, st, p);
    return launch_status("b200_row_reduce");
  };
  // (fp32 sums of 64 to 256 vectors where a warp per row is one well filled wave, 2368 to some 9000 rows on 148 SMs, are bound by the additions that
  // keep what is rounded away: [8192, 512] 3.9 us, with plain chains of a warp per row 2.8. Those are off by 4.8e-8 instead of 2.5e-8.)
  if (nv <= 16) return short_rows(row_reduce_short_kernel<Tin, Op, 4, 4, kKept>, 4);
  if (nv <= 32) return short_rows(row_reduce_short_kernel<Tin, Op, 8, 4, kKept>, 8);
  if (nv <= 64) return short_rows(row_reduce_short_kernel<Tin, Op, 16, 4, kKept>, 16);
  if (nv <= 128) return short_rows(row_reduce_short_kernel<Tin, Op, 32, 4, kKept>, 32);
  if (nv <= 256 && p.rows >= 4LL * sms) return short_rows(row_reduce_short_kernel<Tin, Op, 32, 8, kPairs>, 32);
  const unsigned warp_ctas = (unsigned)((p.rows + 7) / 8);
  const bool warp_mode = nv > 256 && p.rows >= (long long)sms * 16 && p.n <= 16384 && eff_warp + 0.02 >= eff_block;
  // Where a warp takes a row of the grid: row_reduce_grid_kernel, but the other kernel for rows of 512 vectors and more that are all there at
  // once, with registers for more loads (f32 [2400, 8192] 13.2 and 12.3 us, bf16 [2400, 8192] 7.6 and 4.8, [5000, 4096] 6.1 and 5.1; shorter ones f32
  // [2400, 1500] 2.7 and 3.0, and above four CTAs an SM f32 and extremes [5000, 4000] 12.7 and 13.8), and for sums of 16 bits in whole
  // batches, whose loop spills in the former ([8192, 4096] 12.3 and 11.6). A CTA per row is faster so on the grid too (f32 [1200, 16384] amax
  // 14.1 and 12.6, a single row 2.2 and 2.0).
  const bool sum16 = Op::is_sum && sizeof(Tin) == 2;
  const bool at_once = nv >= 512 && warp_ctas <= (sum16 ? 6u : 4u) * sms;
  if (on_grid && warp_mode && !at_once && !(sum16 && nv % 128 == 0)) {
    set_path_tag("vector, warp per row");
    launch_dependent(row_reduce_grid_kernel<Tin, Op>, warp_ctas, 256, 0, st, p);
    return launch_status("b200_row_reduce");
  }
  set_path_tag(warp_mode ? "any alignment, warp per row" : "any alignment, CTA per row");
  if (warp_mode && warp_ctas <= 4u * sms) launch_dependent(row_reduce_kernel<Tin, Op, false, int, 4>, warp_ctas, 256, 0, st, p);
  else if (warp_mode && warp_ctas <= 6u * sms) launch_dependent(row_reduce_kernel<Tin, Op, false, int, 6>, warp_ctas, 256, 0, st, p);
  else if (warp_mode) launch_dependent(row_reduce_kernel<Tin, Op, false, int, 8>, warp_ctas, 256, 0, st, p);
  else if (p.n < (1 << 30)) launch_dependent(row_reduce_kernel<Tin, Op, true, int>, (unsigned)p.rows, threads, 0, st, p);
  else launch_dependent(row_reduce_kernel<Tin, Op, true, long long>, (unsigned)p.rows, threads, 0, st, p);
  return launch_status("b200_row_reduce");
}

template <typename Tin>
static int dispatch_row_reduce_op(const RowReduceParams& p, int op, bool on_grid, cudaStream_t st) {
  switch (op) {
    case B200_REDUCE_SUM:
    case B200_REDUCE_MEAN: return launch_row_reduce<Tin, SumOp>(p, on_grid, st);
    case B200_REDUCE_AMAX: return launch_row_reduce<Tin, MaxOp>(p, on_grid, st);
    case B200_REDUCE_AMIN: return launch_row_reduce<Tin, MinOp>(p, on_grid, st);
  }
  return fail(B200_ERR_INVALID, "b200_row_reduce: unknown op %d", op);
}

}  // namespace b200

using namespace b200;

extern "C" int b200_row_reduce(const void* x, void* out, int64_t rows, int64_t n, int64_t d1,
                               int64_t d2, const int64_t* x_strides, int64_t out_stride,
                               int32_t x_dtype, int32_t out_dtype, int32_t op, void* stream) {
  if (!x || !out || !x_strides) return fail(B200_ERR_INVALID, "b200_row_reduce: null argument");
  if (rows < 0 || n < 0 || d1 < 1 || d2 < 1)
    return fail(B200_ERR_INVALID, "b200_row_reduce: bad sizes rows=%lld n=%lld", (long long)rows, (long long)n);
  if (rows == 0) return B200_OK;
  if (rows % (d1 * d2) != 0) return fail(B200_ERR_INVALID, "b200_row_reduce: rows not divisible by d1*d2");
  if (n == 0 && (op == B200_REDUCE_AMAX || op == B200_REDUCE_AMIN))
    return fail(B200_ERR_INVALID, "b200_row_reduce: amax/amin of an empty row is undefined");

  RowReduceParams p;
  p.x = x; p.out = out; p.rows = rows; p.n = n;
  if (rows > 0x7fffffffLL) return fail(B200_ERR_UNSUPPORTED, "b200_row_reduce: more than 2^31-1 rows");
  p.xmap = make_row_map(x_strides, d1, d2);
  p.out_stride = out_stride; p.out_dtype = out_dtype;
  // mean of an empty row is 0 * (1/0) = NaN, as aten.mean returns
  p.post_scale = op == B200_REDUCE_MEAN ? 1.0f / (float)n : 1.0f;
  const int ib = dtype_size(x_dtype);
  const bool on_grid = aligned16(x) && (p.xmap.s0 * ib) % 16 == 0 && (p.xmap.s1 * ib) % 16 == 0 && (p.xmap.s2 * ib) % 16 == 0;
  cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
  switch (x_dtype) {
    case B200_F32: return dispatch_row_reduce_op<float>(p, op, on_grid, st);
    case B200_BF16: return dispatch_row_reduce_op<__nv_bfloat16>(p, op, on_grid, st);
    case B200_F16: return dispatch_row_reduce_op<__half>(p, op, on_grid, st);
  }
  return fail(B200_ERR_INVALID, "b200_row_reduce: unknown dtype %d", x_dtype);
}
