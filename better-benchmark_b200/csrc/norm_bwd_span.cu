// LayerNorm / RMSNorm backward of rows that start and end off the 16-byte grid, as the vectors of memory that they touch.
#include "norm_bwd.cuh"

namespace b200 {

// Rows off the 16-byte grid (RowSpan), x, dy and dx with the same alignment. A CTA takes rows that are a multiple of eight apart: their
// alignment is the same, so that a thread's KE columns are, and its weights and sums of dweight / dbias stay in registers.
// R rows at a time; the next ones are on their way meanwhile. What lies beside a row is zero from the load on.
// One partial row per CTA, added up by the launch that follows.
// Bound by the chain of a row (loads, two sums through the warps and a barrier) and the few CTAs that the registers leave to cover it: half
// the rate of a copy. Eight columns a thread with two rows per barrier up to some 1500 columns; from there on sixteen, with half
// as many warps to meet at the barrier (20 against 17 us at 4000 x 1317, 26 against 33 at 4000 x 2306, bf16).
template <typename T, bool LN, int KE, int R, int THREADS, int CTAS>
__global__ void __launch_bounds__(THREADS, CTAS) norm_bwd_span_kernel(const NormBwdParams p) {
  wait_for_previous_kernel();
  constexpr int V = Elem<T>::V, P = V / 2, K = KE / V;
  __shared__ float2 red[2][R][THREADS / 32];
  __shared__ uint4 edge[2];  // what belongs to the row of its first and its last vector
  const int tid = (int)threadIdx.x, gs = (int)blockDim.x, n = p.n;
  const int warp = tid >> 5, nwarps = gs >> 5;
  const long long first = blockIdx.x, stride = gridDim.x;
  const RowSpan span = RowSpan::of(reinterpret_cast<const T*>(p.x) + first * p.x_row_stride, n);
  if (tid == 0) {
    uint32_t in_first[4], in_last[4];
    span_edges<T>(span, in_first, in_last);
    edge[0] = make_uint4(in_first[0], in_first[1], in_first[2], in_first[3]);
    edge[1] = make_uint4(in_last[0], in_last[1], in_last[2], in_last[3]);
  }
  uint4 nx[R][K], ny[R][K];
  float nrstd[R], nmean[R];
  auto fetch = [&](long long row) {
#pragma unroll
    for (int r = 0; r < R; ++r) {
      const long long at = row + r * stride;
      const bool there = at < p.rows;
      nrstd[r] = there ? ld_here(p.rstd + at) : 0.f;
      nmean[r] = LN && there ? ld_here(p.mean + at) : 0.f;
      span_fetch<T, K>(p.x, p.x_row_stride, p.rows, n, at, there, span, tid, gs, nx[r]);
      span_fetch<T, K>(p.dy, p.dy_row_stride, p.rows, n, at, there, span, tid, gs, ny[r]);
    }
  };
  fetch(first);
  f32x2 w[K][P], acc_w[K][P], acc_b[LN ? K : 1][P];
#pragma unroll
  for (int c = 0; c < K; ++c) {
#pragma unroll
    for (int i = 0; i < P; ++i) {
      auto one = [&](int k) {
        const int col = (c * gs + tid) * V - span.off + k;
        return p.w && col >= 0 && col < n ? load_param1(p.w, p.w_dtype, col) : 1.f;
      };
      w[c][i] = pack2(one(2 * i), one(2 * i + 1));
      acc_w[c][i] = splat2(0.f);
      if constexpr (LN) acc_b[c][i] = splat2(0.f);
    }
  }
  __syncthreads();
  auto inside = [&](int c, uint4 v) {
    auto mask = [&](const uint4& m) { v = make_uint4(v.x & m.x, v.y & m.y, v.z & m.z, v.w & m.w); };
    if (c == 0 && tid == 0) mask(edge[0]);
    if (c * gs + tid == span.nv - 1) mask(edge[1]);
    return v;
  };
  int parity = 0;
  for (long long row = first; row < p.rows; row += R * stride) {  // the same rows for all threads
    f32x2 xv[R][K][P], gv[R][K][P];
    float rstd[R], mean[R], s1[R], s2[R];
#pragma unroll
    for (int r = 0; r < R; ++r) {
      rstd[r] = nrstd[r];
      mean[r] = nmean[r];
#pragma unroll
      for (int c = 0; c < K; ++c) {
        Pairs<T>::unpack(inside(c, nx[r][c]), xv[r][c]);
        Pairs<T>::unpack(inside(c, ny[r][c]), gv[r][c]);
      }
    }
    if (row + R * stride < p.rows) fetch(row + R * stride);
    f32x2 a1[R], a2[R];
#pragma unroll
    for (int r = 0; r < R; ++r) a1[r] = a2[r] = splat2(0.f);
#pragma unroll
    for (int c = 0; c < K; ++c) {
#pragma unroll
      for (int i = 0; i < P; ++i) {
        f32x2 dw, db;
#pragma unroll
        for (int r = 0; r < R; ++r) {
          const f32x2 d = gv[r][c][i], g = mul2(d, w[c][i]), rs = splat2(rstd[r]);
          f32x2 xhat;
          if constexpr (LN) {
            xhat = mul2(sub2(xv[r][c][i], splat2(mean[r])), rs);
            a1[r] = add2(a1[r], g);
            a2[r] = fma2(g, xhat, a2[r]);
            xv[r][c][i] = xhat;
          } else {
            a2[r] = fma2(g, xv[r][c][i], a2[r]);
            xhat = mul2(xv[r][c][i], rs);
          }
          gv[r][c][i] = g;
          // two rows are added to the sums as one: with fewer CTAs than the kernel by the element has, chains are no longer than its
          if (R == 1) dw = fma2(d, xhat, acc_w[c][i]);
          else dw = r == 0 ? mul2(d, xhat) : fma2(d, xhat, dw);
          if constexpr (LN) db = r == 0 ? d : add2(db, d);
        }
        acc_w[c][i] = R == 1 ? dw : add2(acc_w[c][i], dw);
        if constexpr (LN) acc_b[c][i] = add2(acc_b[c][i], db);
      }
    }
#pragma unroll
    for (int r = 0; r < R; ++r) {
      s1[r] = LN ? warp_reduce<SumOp>(hsum2(a1[r])) : 0.f;
      s2[r] = warp_reduce<SumOp>(hsum2(a2[r]));
      if ((tid & 31) == 0) red[parity][r][warp] = make_float2(s1[r], s2[r]);
    }
    __syncthreads();  // the only one: the other half of `red` is written next, and this one not before all have come here again
#pragma unroll
    for (int r = 0; r < R; ++r) {
      s1[r] = s2[r] = 0.f;
      for (int k = 0; k < nwarps; ++k) {
        const float2 t = red[parity][r][k];
        s1[r] += t.x;
        s2[r] += t.y;
      }
    }
    parity ^= 1;
#pragma unroll
    for (int r = 0; r < R; ++r) {
      const long long at = row + r * stride;
      if (at >= p.rows) break;
      const unsigned int bi = fast_div((unsigned int)at, p.seq_div);
      const unsigned int si = (unsigned int)at - bi * (unsigned int)p.seq;
      T* dx = reinterpret_cast<T*>(p.dx) + (long long)bi * p.dx_batch_stride + (long long)si * p.dx_seq_stride - span.off;
      const float k = LN ? rstd[r] / p.n_f : ((s2[r] * -0.5f) * (rstd[r] * rstd[r] * rstd[r])) / p.n_f;
      const f32x2 k2 = splat2(k), n2 = splat2(p.n_f), s12 = splat2(-s1[r]), s22 = splat2(-s2[r]), rs = splat2(rstd[r]), kk = splat2(k * 2.f);
#pragma unroll
      for (int c = 0; c < K; ++c) {
        const int j = c * gs + tid;
        if (j < span.nv) {
          f32x2 o[P];
#pragma unroll
          for (int i = 0; i < P; ++i) {
            const f32x2 g = gv[r][c][i];
            o[i] = LN ? mul2(k2, fma2(xv[r][c][i], s22, fma2(g, n2, s12))) : fma2(g, rs, mul2(kk, xv[r][c][i]));
          }
          const uint4 out = Pairs<T>::pack(o);
          if (span.whole<V>(j)) st_stream(dx + (long long)j * V, out);
          else store_part(dx + (long long)j * V, out, span.lo(j), span.hi<V>(j));
        }
      }
    }
  }
  if (!p.dw && !p.db) return;
  // By way of shared memory: a thread's columns are neighbours, and stored from here each store of a warp would touch 32 sectors.
  extern __shared__ float columns[];
  auto put = [&](const f32x2 (&acc)[K][P], float* out) {
#pragma unroll
    for (int c = 0; c < K; ++c) {
#pragma unroll
      for (int i = 0; i < V; ++i) {
        const int col = (c * gs + tid) * V - span.off + i;
        float a, b;
        unpack2(acc[c][i / 2], a, b);
        if (col >= 0 && col < n) columns[col] = i & 1 ? b : a;
      }
    }
    __syncthreads();
    for (int i = tid; i < n; i += gs) out[i] = columns[i];
  };
  put(acc_w, p.partials + (long long)blockIdx.x * n);
  if constexpr (LN) {
    __syncthreads();
    put(acc_b, p.partials + ((long long)p.groups + blockIdx.x) * n);
  }
}

// Whether the kernel above takes the rows; p.groups is then the number of partial rows.
template <typename T, bool LN>
bool try_launch_norm_bwd_span(NormBwdParams& p, size_t scratch_bytes, cudaStream_t st, int* rc) {
  constexpr int V = Elem<T>::V;
  const DeviceInfo& dev = device_info();
  auto off = [](const void* q) { return reinterpret_cast<uintptr_t>(q) & 15u; };
  if (p.dy_elem_stride != 1 || p.head_dim != p.n || p.n < 2 * V || p.x_row_stride < p.n || p.dy_row_stride < p.n) return false;
  if (off(p.x) != off(p.dy) || off(p.x) != off(p.dx) || (p.x_row_stride - p.dy_row_stride) % V != 0 ||
      (p.seq > 1 && (p.x_row_stride - p.dx_seq_stride) % V != 0) || (p.rows > p.seq && (p.dx_batch_stride - p.seq * p.x_row_stride) % V != 0)) return false;
  // The kernel that goes element by element (norm_bwd_ragged_kernel) / this one, us, LayerNorm with both gradients:
  //   columns    517          981          1317         2306         4001
  //   bf16 1200                                         19.6 / 14.9  24.4 / 17.5  rows
  //        4000                            28.3 / 17.2  52.3 / 26.3  65.1 / 31.4
  //        8000  25.9 / 20.1  31.5 / 23.4  50.6 / 27.8  98.6 / 42.5  122 / 51.0
  //       24000  63.4 / 42.0  81.7 / 52.7  139 / 67.6   283 / 110                 (floors 11.4, 21.6, 29.0, 50.7)
  //   f32  1200                                         18.6 / 15.9  23.3 / 21.0
  //        4000                            26.3 / 21.8  48.2 / 30.5  58.4 / 46.7
  constexpr bool HALF = sizeof(T) == 2;
  if (p.n <= (HALF ? 512 : 1024)) return false;
  // RMSNorm in fp32 has less to compute by the element: at these lines it is slower so ([2368, 1523] 15.7 / 16.6, [1200, 2305] 13.3 / 14.6;
  // from 24 and 14 rows per SM on it is not), but its errors are smaller, dweight's 6.5e-8 / 5.4e-8, dx' 4.4e-8 / 3.6e-8.
  // Fewer rows would gain up to a fifth, but with chains that are longer than before: RMSNorm's dweight, 1300 x 517, 5.7e-8 instead of 4.8e-8.
  if (p.rows < (HALF ? (p.n <= 1010 ? 32 : p.n <= 1522 ? 16 : 8) : p.n <= 2048 ? 16 : 8) * (long long)dev.sm_count) return false;
  const int nv = (p.n + 2 * (V - 1)) / V;  // vectors that a row touches at most
  const bool sums = p.dw || p.db;
  auto launch = [&](auto kernel, int threads) {
    const size_t smem = sums ? (size_t)p.n * sizeof(float) : 0;
    long long ctas = cached_occupancy(reinterpret_cast<const void*>(kernel), threads, smem);
    if (ctas > 8) ctas = 8;  // what b200_norm_bwd_scratch_bytes counts on
    long long grid = ctas * dev.sm_count;
    if (grid > p.rows / 4) grid = p.rows / 4;  // fewer rows than that do not pay for a partial row
    if (sums) {
      const long long max_groups = ((long long)scratch_bytes - 256) / (2 * (long long)p.n * (long long)sizeof(float));
      if (grid > max_groups) grid = max_groups;
    }
    grid &= ~7LL;  // a CTA's rows are a multiple of eight apart
    if (grid < 8) return false;
    p.groups = p.workers = (int)grid;
    launch_dependent(kernel, (unsigned)grid, threads, smem, st, p);
    *rc = launch_status("b200_norm_bwd [ragged rows, vectors in registers]");
    return true;
  };
  const int t8 = (nv * V + 255) / 256 * 32, t16 = (nv * V + 511) / 512 * 32;
  if constexpr (HALF) {
    if (t8 <= 128) return launch(norm_bwd_span_kernel<T, LN, 8, 2, 128, 4>, t8);
    if (t8 <= 192) return launch(norm_bwd_span_kernel<T, LN, 8, 2, 192, 2>, t8);
  }
  if (t16 <= 128) return launch(norm_bwd_span_kernel<T, LN, 16, 1, 128, 4>, t16);
  if (t16 <= 160) return launch(norm_bwd_span_kernel<T, LN, 16, 1, 160, 3>, t16);
  return t16 <= 256 && launch(norm_bwd_span_kernel<T, LN, 16, 1, 256, 2>, t16);
}

template bool try_launch_norm_bwd_span<float, true>(NormBwdParams&, size_t, cudaStream_t, int*);
template bool try_launch_norm_bwd_span<float, false>(NormBwdParams&, size_t, cudaStream_t, int*);
template bool try_launch_norm_bwd_span<__nv_bfloat16, true>(NormBwdParams&, size_t, cudaStream_t, int*);
template bool try_launch_norm_bwd_span<__nv_bfloat16, false>(NormBwdParams&, size_t, cudaStream_t, int*);
template bool try_launch_norm_bwd_span<__half, true>(NormBwdParams&, size_t, cudaStream_t, int*);
template bool try_launch_norm_bwd_span<__half, false>(NormBwdParams&, size_t, cudaStream_t, int*);

}  // namespace b200
