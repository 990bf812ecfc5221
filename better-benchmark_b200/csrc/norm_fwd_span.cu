// LayerNorm / RMSNorm forward, with or without a residual add or the GELU prologue, of rows that start and end off the 16-byte grid:
// as the vectors of memory that they touch instead of element by element.
#include "norm_fwd.cuh"

namespace b200 {

// ----------------------------------------------------------------------------------------------
// Rows off the 16-byte grid whose results have their alignment (contiguous rows of an odd length, in the input's dtype): the row as the
// 16-byte vectors that it touches (RowSpan). What lies beside the row in its first and last vector is zero from the load on,
// and stays out of the sum of squares.
//   KIND: 0 LayerNorm / RMSNorm, 1 the same behind the GELU prologue, 2 residual add in front (both forms of the sum at run time)
// The operations on an element and their roundings are those of norm_fwd_resident_kernel.
// param.weight(c, ..), .bias: those (weight: 1 where there is none) of the vector in slot c; any beside the row, which is not stored.
// ----------------------------------------------------------------------------------------------
template <typename T, int K, int G, int KIND, typename Param>
__device__ __forceinline__ void norm_span_row(const NormFwdParams& p, const RowSpan& span, uint4 (&raw)[K],
                                              const uint4 (&rraw)[KIND == 2 ? K : 1], const uint32_t (&in_first)[4],
                                              const uint32_t (&in_last)[4], long long row, bool valid, int lane, int gs, float* red,
                                              const Param& param) {
  constexpr int V = Elem<T>::V, P = V / 2;
  constexpr bool HALF = sizeof(T) == 2;
  const bool both = KIND == 2 && HALF && p.res_round == 2;
  auto is_last = [&](int c) { return c * gs + lane == span.nv - 1; };
  auto inside = [&](int c, uint4 w) {  // zeros beside the row
    if (c == 0 && lane == 0) w = make_uint4(w.x & in_first[0], w.y & in_first[1], w.z & in_first[2], w.w & in_first[3]);
    if (is_last(c)) w = make_uint4(w.x & in_last[0], w.y & in_last[1], w.z & in_last[2], w.w & in_last[3]);
    return w;
  };
  auto inside2 = [&](int c, f32x2 (&d)[P]) {
    auto keep = [&](const uint32_t (&in)[4]) {
#pragma unroll
      for (int i = 0; i < P; ++i) {
        float a, b;
        unpack2(d[i], a, b);
        if constexpr (HALF) d[i] = pack2((in[i] & 0xffffu) ? a : 0.f, (in[i] >> 16) ? b : 0.f);
        else d[i] = pack2(in[2 * i] ? a : 0.f, in[2 * i + 1] ? b : 0.f);
      }
    };
    if (c == 0 && lane == 0) keep(in_first);
    if (is_last(c)) keep(in_last);
  };
  // Whole vectors leave at once, a lane's first or last one of the row when the others have: the lanes that hold one do that together.
  struct Edge {
    uint4 packed;
    int j = -1;
  };
  auto store_edge = [&](T* first, const Edge& e) {  // first: the row's first vector in the result
    if (e.j >= 0) store_part(first + (long long)e.j * V, e.packed, span.lo(e.j), span.hi<V>(e.j));
  };
  auto store = [&](T* first, int c, const uint4& packed, Edge& e) {
    const int j = c * gs + lane;
    if (span.whole<V>(j)) {
      st_stream(first + (long long)j * V, packed);
    } else {
      store_edge(first, e);  // both in one lane
      e.packed = packed;
      e.j = j;
    }
  };

  // by the vector: one chain through all of a lane's elements loses more (rstd of 981 columns, RMSNorm: 5.0e-8 instead of 4.6e-8)
  auto total = [](const f32x2 (&d)[P]) {
    f32x2 t = d[0];
#pragma unroll
    for (int i = 1; i < P; ++i) t = add2(t, d[i]);
    return t;
  };
  auto squares = [](const f32x2 (&d)[P]) {
    f32x2 t = mul2(d[0], d[0]);
#pragma unroll
    for (int i = 1; i < P; ++i) t = fma2(d[i], d[i], t);
    return t;
  };

  f32x2 v[K][P], s2 = splat2(0.f), t2 = splat2(0.f);
  uint4 pr[KIND == 2 ? K : 1];
  Edge sum_edge;
  T* so = KIND == 2 && p.sum_out && valid ? reinterpret_cast<T*>(p.sum_out) + row * (long long)p.n - span.off : nullptr;
#pragma unroll
  for (int c = 0; c < K; ++c) {
    Pairs<T>::unpack(inside(c, raw[c]), v[c]);
    if constexpr (KIND == 2) {
      f32x2 r[P];
      Pairs<T>::unpack(inside(c, rraw[c]), r);
#pragma unroll
      for (int i = 0; i < P; ++i) v[c][i] = add2(v[c][i], r[i]);
      pr[c] = Pairs<T>::pack(v[c]);
      if (so && c * gs + lane < span.nv) store(so, c, pr[c], sum_edge);
      if (p.res_round == 1) Pairs<T>::unpack(pr[c], v[c]);
      if (both) {
        Pairs<T>::unpack(pr[c], r);
        t2 = add2(t2, total(r));
      }
    } else if constexpr (KIND == 1) {
#pragma unroll
      for (int i = 0; i < P; ++i) v[c][i] = gelu_erf_rounded2<T>(v[c][i]);  // gelu(0) = 0
    }
    s2 = add2(s2, KIND != 2 && p.rms ? squares(v[c]) : total(v[c]));
  }
  if (so) store_edge(so, sum_edge);
  float s = hsum2(s2), t = hsum2(t2);
  if (both) greduce_sum2<G>(s, t, red);
  else s = greduce<SumOp, G>(s, red);
  float mean = 0.f, var = s * p.inv_n, rstd_r = 0.f;
  const float mean_r = t * p.inv_n;
  if (KIND == 2 || !p.rms) {
    mean = s * p.inv_n;
    const f32x2 mean2 = splat2(mean), mean_r2 = splat2(mean_r);
    f32x2 q2 = splat2(0.f), u2 = splat2(0.f);
#pragma unroll
    for (int c = 0; c < K; ++c) {
      if (c * gs + lane < span.nv) {
#pragma unroll
        for (int i = 0; i < P; ++i) v[c][i] = sub2(v[c][i], mean2);  // kept: the output needs it again
        inside2(c, v[c]);
        q2 = add2(q2, squares(v[c]));
        if (both) {
          f32x2 r[P];
          Pairs<T>::unpack(pr[KIND == 2 ? c : 0], r);
#pragma unroll
          for (int i = 0; i < P; ++i) r[i] = sub2(r[i], mean_r2);
          inside2(c, r);
          u2 = add2(u2, squares(r));
        }
      }
    }
    float q = hsum2(q2), u = hsum2(u2);
    if (both) greduce_sum2<G>(q, u, red);
    else q = greduce<SumOp, G>(q, red);
    var = q * p.inv_denom;
    rstd_r = precise_rsqrt(u * p.inv_denom + p.eps);
  }
  const float rstd = precise_rsqrt(var + p.eps);
  if (!valid) return;
  if (lane == 0) {
    if (p.mean_out) p.mean_out[row] = mean;
    if (p.rstd_out) p.rstd_out[row] = rstd;
    if (p.var_out) p.var_out[row] = var;
  }
  const f32x2 rstd2 = splat2(rstd), rstd_r2 = splat2(rstd_r), mean_r2 = splat2(mean_r);
  T* y = reinterpret_cast<T*>(p.y) + row * p.y_row_stride - span.off;
  Edge edge;
  auto put_out = [&](auto bias_tag) {
    constexpr bool BIAS = decltype(bias_tag)::value;
#pragma unroll
    for (int c = 0; c < K; ++c) {
      if (c * gs + lane < span.nv) {
        f32x2 o[P], r[P], w[P], b[P];
        param.weight(c, w);
        if constexpr (BIAS) param.bias(c, b);
        if (both) Pairs<T>::unpack(pr[KIND == 2 ? c : 0], r);
#pragma unroll
        for (int i = 0; i < P; ++i) {
          o[i] = mul2(mul2(v[c][i], rstd2), w[i]);
          if constexpr (BIAS) o[i] = add2(o[i], b[i]);
          if (both) {
            r[i] = mul2(mul2(sub2(r[i], mean_r2), rstd_r2), w[i]);
            if constexpr (BIAS) r[i] = add2(r[i], b[i]);
          }
        }
        uint4 out = Pairs<T>::pack(o);
        if constexpr (KIND == 2 && HALF) {
          if (both) {
            const uint4 rounded = Pairs<T>::pack(r);
            auto pick = [&](uint32_t full, uint32_t round) {
              const uint32_t m = beyond_three<T>(full);
              return (full & m) | (round & ~m);
            };
            out = make_uint4(pick(out.x, rounded.x), pick(out.y, rounded.y), pick(out.z, rounded.z), pick(out.w, rounded.w));
          }
        }
        store(y, c, out, edge);
      }
    }
  };
  if (p.b) put_out(std::true_type{});
  else put_out(std::false_type{});
  store_edge(y, edge);
}

template <typename T>
struct GroupParams {
  static constexpr int P = Elem<T>::V / 2;
  const f32x2* const (&at)[P];  // weights of the pairs of the lane's first vector
  int step, to_bias;
  __device__ __forceinline__ void weight(int c, f32x2 (&out)[P]) const {
#pragma unroll
    for (int i = 0; i < P; ++i) out[i] = at[i][c * step];
  }
  __device__ __forceinline__ void bias(int c, f32x2 (&out)[P]) const {
#pragma unroll
    for (int i = 0; i < P; ++i) out[i] = at[i][c * step + to_bias];
  }
};

// A group of G lanes takes `reps` rows that are a multiple of eight apart and so have the same alignment; the next one is
// on its way meanwhile. Weight and bias lie in shared memory as fp32 pairs of neighbouring columns, one table for the pairs that begin at an
// even column and one for the others, column c of either at [c mod V / 2][c / V + 1]: for a pair of a vector's elements the lanes of
// a warp read consecutive pairs, whatever the alignment. (bf16 behind GELU spills 12 / 12 bytes at the CTAs per SM below.)
template <typename T, int K, int G, int KIND>
__global__ void __launch_bounds__(256, KIND == 2 ? 2 : K <= 2 ? 4 : K == 3 ? 3 : 2)
norm_fwd_span_kernel(const NormFwdParams p, const int reps) {
  wait_for_previous_kernel();
  constexpr int V = Elem<T>::V, P = V / 2;
  extern __shared__ __align__(16) unsigned char smem[];
  const int lane = glane<G>(), gs = gsize<G>();
  constexpr int step = 256 / G;
  const int S = p.n / V + 3;  // columns -V .. n + V - 1 may be asked for
  f32x2* wsm = reinterpret_cast<f32x2*>(smem);  // [2][P][S]
  f32x2* bsm = wsm + 2 * P * S;
  long long row = (long long)blockIdx.x * reps * step + (int)threadIdx.x / G;
  const RowSpan span = RowSpan::of(reinterpret_cast<const T*>(p.x) + row * p.x_row_stride, p.n);
  uint32_t in_first[4], in_last[4];
  span_edges<T>(span, in_first, in_last);
  uint4 next[K], rnext[KIND == 2 ? K : 1];
  auto fetch = [&](long long r, bool there) {
    span_fetch<T, K>(p.x, p.x_row_stride, p.rows, p.n, r, there, span, lane, gs, next);
    if constexpr (KIND == 2) span_fetch<T, K>(p.res, p.x_row_stride, p.rows, p.n, r, there, span, lane, gs, rnext);
  };
  for (int c = (int)threadIdx.x - V; c < p.n + V; c += blockDim.x) {
    float w = 1.f, b = 0.f;
    if (c >= 0 && c < p.n) {
      if (p.w) w = load_param1(p.w, p.w_dtype, c);
      if (p.b) b = load_param1(p.b, p.w_dtype, c);
    }
    // the first of one pair and the second of another; pairs are numbered by the column they begin at
    auto put = [&](int begin, int half) {
      if (begin < -V) return;
      const int at = ((begin & 1) * P + ((begin & (V - 1)) >> 1)) * S + (begin + V) / V;
      reinterpret_cast<float*>(wsm + at)[half] = w;
      reinterpret_cast<float*>(bsm + at)[half] = b;
    };
    put(c, 0);
    put(c - 1, 1);
  }
  fetch(row, row < p.rows);
  __syncthreads();
  const f32x2* at[P];
#pragma unroll
  for (int i = 0; i < P; ++i) {
    const int begin = lane * V - span.off + 2 * i;
    at[i] = wsm + ((begin & 1) * P + ((begin & (V - 1)) >> 1)) * S + (begin + V) / V;
  }
  for (int rep = 0; rep < reps; ++rep, row += step) {
    const bool valid = row < p.rows;
    if (!__any_sync(0xffffffffu, valid)) break;
    uint4 raw[K], rraw[KIND == 2 ? K : 1];
#pragma unroll
    for (int c = 0; c < K; ++c) raw[c] = next[c];
#pragma unroll
    for (int c = 0; c < (KIND == 2 ? K : 1); ++c) rraw[c] = rnext[c];
    if (rep + 1 < reps) fetch(row + step, row + step < p.rows);
    norm_span_row<T, K, G, KIND>(p, span, raw, rraw, in_first, in_last, row, valid, lane, gs, nullptr, GroupParams<T>{at, gs, 2 * P * S});
  }
}

// Elements j V - off .. j V - off + V - 1 of a parameter of the rows' type on the 16-byte grid, from the vectors j - 1 and j of it.
template <typename T>
__device__ __forceinline__ uint4 shifted_params(const void* base, int j, int off, int n) {
  constexpr int V = Elem<T>::V;
  const T* p = reinterpret_cast<const T*>(base);
  auto vec = [&](int k) {
    if (k < 0) return make_uint4(0u, 0u, 0u, 0u);
    if ((k + 1) * V <= n) return ld_keep(p + k * V);
    return load_part(p + k * V, 0, n - k * V);
  };
  const uint4 a = vec(j - 1), b = vec(j);
  uint32_t w[8] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
  const int by = V - off;  // elements: 1 .. V
  const int words = sizeof(T) == 2 ? by >> 1 : by;
  if (words & 4) {
#pragma unroll
    for (int i = 0; i < 4; ++i) w[i] = w[i + 4];
  }
  if (words & 2) {
#pragma unroll
    for (int i = 0; i < 6; ++i) w[i] = w[i + 2];
  }
  if (words & 1) {
#pragma unroll
    for (int i = 0; i < 5; ++i) w[i] = w[i + 1];
  }
  if (sizeof(T) == 2 && (by & 1)) {
#pragma unroll
    for (int i = 0; i < 4; ++i) w[i] = __funnelshift_r(w[i], w[i + 1], 16);
  }
  return make_uint4(w[0], w[1], w[2], w[3]);
}

template <typename T>
struct RowParams {
  static constexpr int V = Elem<T>::V, P = V / 2;
  const void *w, *b;
  int dtype, n, off, lane, gs;
  bool whole;  // the rows' type, on the 16-byte grid
  __device__ __forceinline__ void get(const void* base, int c, f32x2 (&out)[P]) const {
    const int j = c * gs + lane;
    if (whole) {
      Pairs<T>::unpack(shifted_params<T>(base, j, off, n), out);
    } else {
      float one[V];
#pragma unroll
      for (int i = 0; i < V; ++i) {
        const int col = j * V - off + i;
        one[i] = load_param1(base, dtype, col < 0 ? 0 : col >= n ? n - 1 : col);
      }
#pragma unroll
      for (int i = 0; i < P; ++i) out[i] = pack2(one[2 * i], one[2 * i + 1]);
    }
  }
  __device__ __forceinline__ void weight(int c, f32x2 (&out)[P]) const {
    if (w) {
      get(w, c, out);
    } else {
#pragma unroll
      for (int i = 0; i < P; ++i) out[i] = splat2(1.f);
    }
  }
  __device__ __forceinline__ void bias(int c, f32x2 (&out)[P]) const { get(b, c, out); }
};

// Longer rows: a CTA per row, as many of them as the SM holds (a table and rows in turn, as above: 20000 x 2661 140 us instead of 109).
// Weight and bias of the rows' own type through L1 by the vector, shifted to the row's alignment: 7081 columns 94 -> 65 us at 6000 rows
// against element by element, a residual add 184 -> 150; fp32, four loads instead of two: 48 instead of 55 us (4001 columns), so not there.
template <typename T, int K, int KIND>
__global__ void __launch_bounds__(512) norm_fwd_span_row_kernel(const NormFwdParams p, const bool whole_params) {
  wait_for_previous_kernel();
  constexpr int V = Elem<T>::V;
  __shared__ float red[64];
  const int lane = (int)threadIdx.x, gs = (int)blockDim.x;
  const long long row = blockIdx.x;
  const RowSpan span = RowSpan::of(reinterpret_cast<const T*>(p.x) + row * p.x_row_stride, p.n);
  uint32_t in_first[4], in_last[4];
  span_edges<T>(span, in_first, in_last);
  uint4 raw[K], rraw[KIND == 2 ? K : 1];
  span_fetch<T, K>(p.x, p.x_row_stride, p.rows, p.n, row, true, span, lane, gs, raw);
  if constexpr (KIND == 2) span_fetch<T, K>(p.res, p.x_row_stride, p.rows, p.n, row, true, span, lane, gs, rraw);
  norm_span_row<T, K, 0, KIND>(p, span, raw, rraw, in_first, in_last, row, true, lane, gs, red,
                               RowParams<T>{p.w, p.b, p.w_dtype, p.n, span.off, lane, gs, whole_params});
}

// The rows for which the two kernels above are faster than the one that goes element by element (norm_fwd_ragged_kernel), in rows per SM;
// fewer leave lanes of it idle that the other fills. One of the other kernel's times over one of theirs, us, bf16 LayerNorm with weight and bias
// (behind GELU a tenth less is won; floors are those of a copy):
//   columns       121          186          361          673          981          1317         2661         7081
//   600 rows      2.6 / 3.0    2.8 / 3.1    3.2 / 3.7    5.1 / 4.1    5.2 / 4.8    5.7 / 5.3    9.2 / 6.8    21.8 / 11.2
//   2000          2.8 / 3.0    3.4 / 3.1    4.6 / 3.8    7.4 / 4.8    8.8 / 5.6    12.2 / 10.3  21.9 / 14.6  59.3 / 24.8
//   6000          3.9 / 3.8    5.6 / 4.1    9.0 / 5.2    16.8 / 9.0   21.9 / 13.1  31.3 / 20.5  60.0 / 37.9  169 / 64.6
//   20000         8.6 / 6.3    12.1 / 9.2   23.8 / 12.0  50.4 / 21.0  66.9 / 31.3  98.3 / 59.9  193 / 109
//   60000 (floor) 22.6 / 12.3  34.5 / 21.9  69.7 / 30.0  146 / 56.7   195 / 66.7 (4.4, 6.8, 13.2, 24.7, 36.0)
// With a residual add, both forms of the sum: 186 columns, 20000 rows 17.6 / 19.3; 361: 2000 rows 5.5 / 5.1, 60000 92 / 73; 981: 600 rows
// 6.0 / 5.1, 20000 81 / 60; 2661: 600 rows 10.8 / 7.9, 20000 233 / 160; 7081: 2000 rows 72 / 53.
// fp32 (half as many elements a vector): 981 columns and below slower, 1317 equal at 2000 rows, 2049: 600 rows 4.6 / 5.0, 2661: 750 8.9 / 7.5, 6000 52 / 38.
// Bound by instructions (masks, edges, shifted parameters): 981 columns run at half the rate of a copy, a CTA per row at a third.
// The lines lie where this is ahead, or within 4 per cent, at every number of rows measured from there on. Rows that fill the other kernel's
// slots and have just left one of this one's (250..256, 506..512 and 1018..1024 columns) gain least: RMSNorm 255 at 26 rows per SM 3.4 / 3.6, GELU 255 at
// 40 6.3 / 6.9, residual add, both forms, 511 at 24 7.8 / 10.8 and at 160 41 / 41, 1019 at 12 9.3 / 10.2. Both forms of a residual add leave room for
// two CTAs an SM: 378 columns at 16, one wave, 6.0 / 5.5, at 24 6.9 / 8.2, at 28 10.5 / 8.3.
static bool norm_span_takes(const NormFwdParams& p, int nv, long long sms) {
  const bool both = p.res && p.res_round == 2;
  const bool edge = p.n > 128 && p.n <= 1024 && nv * 8 > (p.n + 255) / 256 * 256;
  if (edge && p.prologue && p.n <= 256) return false;
  int line;  // rows per SM
  if (nv > 128) line = both && edge ? 16 : 4;
  else if (p.n > 512) line = 8;
  else if (p.n > 256 && edge) line = both ? 64 : p.res ? 28 : p.rms ? 25 : 14;
  else if (p.n > 256) line = both && p.n > 377 && p.rows > 16 * sms ? 25 : 14;
  else if (p.n > 128) line = edge ? (p.rms ? 48 : 26) : p.rms ? 25 : 20;
  else line = 64;
  return p.rows >= line * sms;
}

template <typename T>
bool try_launch_norm_fwd_span(const NormFwdParams& p, cudaStream_t st) {
  constexpr int V = Elem<T>::V;
  constexpr bool HALF = sizeof(T) == 2;
  const long long sms = device_info().sm_count;
  const int nv = (p.n + 2 * (V - 1)) / V;  // vectors that a row touches at most
  auto off = [](const void* q) { return reinterpret_cast<uintptr_t>(q) & 15u; };
  if (!p.y || nv > 2048 || p.x_row_stride < p.n || off(p.x) != off(p.y) || (p.x_row_stride - p.y_row_stride) % V != 0) return false;
  if constexpr (HALF) {
    if (p.n <= (p.res ? 256 : 57)) return false;  // 57: two vectors a lane of eight
    if (!norm_span_takes(p, nv, sms)) return false;
    if (p.res && (p.rms || off(p.x) != off(p.res) ||
                  (p.sum_out && (off(p.x) != off(p.sum_out) || (p.x_row_stride - p.n) % V != 0)))) return false;
  } else {
    if (p.n <= 2048 || p.rows < 5 * sms || p.res || p.prologue) return false;
  }
  set_path_tag(p.res ? "residual add, off-grid rows as vectors" : "off-grid rows as vectors");
  auto go = [&](auto kind_tag) {
    constexpr int KIND = decltype(kind_tag)::value;
    const bool whole = HALF && p.w_dtype == (std::is_same<T, __half>::value ? B200_F16 : B200_BF16) && off(p.w) == 0 && off(p.b) == 0;
    if constexpr (HALF) {
      auto launch = [&](auto kernel, int lanes) {
        const size_t smem = (size_t)2 * V * (p.n / V + 3) * sizeof(f32x2);  // both tables of both: 16.5 KB at 1017 columns
        const int at_once = 256 / lanes;
        const long long resident = sms * cached_occupancy(reinterpret_cast<const void*>(kernel), 256, smem);
        // Behind GELU a row is bound by instructions: what counts is how many turns the SM with the most has, not whether its CTAs are there at
        // once ([23680, 249] 13.6 us with turns rounded down, 15.0 in whole waves).
        const long long whole = p.rows / (at_once * resident);
        const int reps = KIND != 1 ? span_turns(p.rows, at_once, resident) : whole < 1 ? 1 : whole > 16 ? 16 : (int)whole;
        launch_dependent(kernel, (unsigned)((p.rows + (long long)at_once * reps - 1) / ((long long)at_once * reps)), 256, smem, st, p, reps);
      };
      if (KIND != 2 && nv <= 16) { launch(norm_fwd_span_kernel<T, 2, 8, KIND == 2 ? 0 : KIND>, 8); return; }
      if (KIND != 2 && nv <= 24) { launch(norm_fwd_span_kernel<T, 3, 8, KIND == 2 ? 0 : KIND>, 8); return; }
      if (KIND != 2 && nv <= 32) { launch(norm_fwd_span_kernel<T, 2, 16, KIND == 2 ? 0 : KIND>, 16); return; }
      if (nv <= 48) { launch(norm_fwd_span_kernel<T, 3, 16, KIND>, 16); return; }
      if (nv <= 64) { launch(norm_fwd_span_kernel<T, 2, 32, KIND>, 32); return; }
      if (nv <= 96) { launch(norm_fwd_span_kernel<T, 3, 32, KIND>, 32); return; }
      // four vectors of two tensors a lane do not fit into the registers
      if (KIND != 2 && nv <= 128) { launch(norm_fwd_span_kernel<T, 4, 32, KIND == 2 ? 0 : KIND>, 32); return; }
      if (nv <= 512) { launch_dependent(norm_fwd_span_row_kernel<T, 2, KIND>, (unsigned)p.rows, (nv + 63) / 64 * 32, 0, st, p, whole); return; }
    }
    launch_dependent(norm_fwd_span_row_kernel<T, 4, KIND>, (unsigned)p.rows, (nv + 127) / 128 * 32, 0, st, p, whole);
  };
  if constexpr (HALF) {
    if (p.res) go(std::integral_constant<int, 2>{});
    else if (p.prologue) go(std::integral_constant<int, 1>{});
    else go(std::integral_constant<int, 0>{});
  } else {
    go(std::integral_constant<int, 0>{});
  }
  return true;
}

template bool try_launch_norm_fwd_span<float>(const NormFwdParams&, cudaStream_t);
template bool try_launch_norm_fwd_span<__nv_bfloat16>(const NormFwdParams&, cudaStream_t);
template bool try_launch_norm_fwd_span<__half>(const NormFwdParams&, cudaStream_t);

}  // namespace b200
