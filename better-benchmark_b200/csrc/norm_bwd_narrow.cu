// LayerNorm / RMSNorm backward of rows of at most 32 vectors: several rows per warp, and one partial row per CTA.
#include "norm_bwd.cuh"

namespace b200 {

constexpr int kNarrowThreads = 256;

// ----------------------------------------------------------------------------------------------
// One launch, two roles. The first `workers` CTAs that START are workers: they walk the rows, and the partial row that each
// leaves has the number of its ticket. The `finalizers` that start after them add the partial rows up once all workers have arrived.
// A worker waits for nobody, and a CTA that waits has started after every worker has: whatever else occupies the GPU, and however
// many waves of CTAs the workers are, the wait ends. Tickets decide who owns which rows, so the result does not
// depend on which CTA draws which.
// ----------------------------------------------------------------------------------------------
enum NarrowWords { kNarrowGone = 2, kNarrowTickets = 3 };  // beside kBwdArrived and kBwdError

// A CTA's number, among the workers or, from p.workers on, the finalizers: thread 0 draws it, the others know it after the CTA's next
// barrier. The shuffle tells the compiler that it is the same in a warp.
__device__ __forceinline__ void narrow_draw_ticket(const NormBwdParams& p, int* ticket) {
  if (threadIdx.x == 0) *ticket = p.finalizers > 0 ? (int)atomicAdd(&p.bar[kNarrowTickets], 1u) : (int)blockIdx.x;
}
__device__ __forceinline__ int narrow_cta(const int* ticket) { return __shfl_sync(0xffffffffu, *ticket, 0); }

// The last CTA puts the words back to zero (the error flag stays until the host has seen it).
__device__ __forceinline__ void narrow_depart(const NormBwdParams& p) {
  if (threadIdx.x == 0 && atomicAdd(&p.bar[kNarrowGone], 1u) == gridDim.x - 1) {
    atomicExch(&p.bar[kBwdArrived], 0u);
    atomicExch(&p.bar[kNarrowGone], 0u);
    atomicExch(&p.bar[kNarrowTickets], 0u);
    __threadfence();
  }
}

// A worker's partial row is written: every thread of the CTA calls this.
__device__ __forceinline__ void narrow_worker_done(const NormBwdParams& p) {
  if (p.finalizers == 0) return;
  __syncthreads();
  if (threadIdx.x == 0) {
    __threadfence();
    atomicAdd(&p.bar[kBwdArrived], 1u);
  }
  narrow_depart(p);
}

// Waits until all workers have arrived; false when an error is noted or the bound ran out (some seconds: with a scratch for few
// partial rows there are few workers, which may take long).
__device__ __forceinline__ bool narrow_wait_for_workers(const NormBwdParams& p, int* flag) {
  if (threadIdx.x == 0) {
    bool error = false;
    for (unsigned int polls = 0; bwd_arrived(p, error) < (unsigned int)p.workers; ++polls) {
      if (polls > (1u << 24)) {
        atomicExch(&p.bar[kBwdError], 1u);
        error = true;
        break;
      }
      __nanosleep(polls > 4096 ? 256 : 32);  // the workers' loads have the memory system
    }
    __threadfence();
    *flag = error ? 0 : 1;
  }
  __syncthreads();
  return *flag != 0;
}

// The finalize of this file's partial rows, which are fp64: the columns of dw and db in units of 8, a CTA each. n % 4 == 0.
__device__ __forceinline__ void finalize_units_f64(const double* partials, int groups, int n, float* dw, float* db, int first, int step,
                                                   double* smem /* [warps][8] */) {
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, nwarps = blockDim.x >> 5;
  const int units = (n + 7) / 8, total = units * ((dw ? 1 : 0) + (db ? 1 : 0));
  const int sub = tid & 3, rows_at_once = blockDim.x / 4;
  for (int s = first; s < total; s += step) {
    const bool is_db = !dw || s >= units;
    const int col = (dw && s >= units ? s - units : s) * 8;
    const int c = col + 2 * sub;
    const double* src = partials + (is_db ? (long long)groups * n : 0) + c;
    double a = 0.0, b = 0.0;
    if (c < n) {
#pragma unroll 1
      for (int g0 = tid / 4; g0 < groups; g0 += 4 * rows_at_once) {
        double2 v[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          const int g = g0 + u * rows_at_once;
          v[u] = g < groups ? __ldcg(reinterpret_cast<const double2*>(src + (long long)g * n)) : make_double2(0.0, 0.0);
        }
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          a += v[u].x;
          b += v[u].y;
        }
      }
    }
#pragma unroll
    for (int o = 16; o >= 4; o >>= 1) {
      a += __shfl_xor_sync(0xffffffffu, a, o);
      b += __shfl_xor_sync(0xffffffffu, b, o);
    }
    if (lane < 4) {
      smem[warp * 8 + lane * 2] = a;
      smem[warp * 8 + lane * 2 + 1] = b;
    }
    __syncthreads();
    if (tid < 8 && col + tid < n) {
      double t = 0.0;
      for (int w = 0; w < nwarps; ++w) t += smem[w * 8 + tid];
      (is_db ? db : dw)[col + tid] = (float)t;
    }
    __syncthreads();
  }
}

// A group of G lanes takes a row, a vector a lane, two rows on their way at once; a lane's columns are the same in every row, so its weights
// and sums stay in registers, and every few rows go to its own words of shared memory. At the end the CTA's groups are added up in
// fp64 into one partial row, and the partial rows by the launch's finalizers (the two roles above).
// A warp per row, as before, left up to 28 of its lanes idle and one partial row per warp: the finalizers' reads of up to 9472 of them took
// longer than the rows. LayerNorm bf16, us: [4000, 64] 13.8 -> 6.9, [24000, 64] 19.1 -> 9.3, [100000, 64] 46 -> 16.5, [100000, 128]
// 46 -> 25, [4000, 256] 14.7 -> 11.1, [100000, 256] 49 -> 42; RMSNorm [24000, 128] 21 -> 10.5; f32 [24000, 64] 20.0 -> 9.7. A few hundred rows
// stay at 6.0 to 6.6 (16-bit LayerNorm with 16 / 24 bytes of spills at three CTAs an SM): a ticket, a row, the partial rows and their sum, each a trip to memory that waits for the one before.
template <typename T, bool LN, int G>
__global__ void __launch_bounds__(kNarrowThreads, 3) norm_bwd_narrow_kernel(const NormBwdParams p) {
  wait_for_previous_kernel();
  constexpr int V = Elem<T>::V, P = V / 2, kGroups = kNarrowThreads / G, U = 2;
  __shared__ float fold[LN ? 2 : 1][kGroups][G * V];
  __shared__ double fin[8 * 8];
  __shared__ int bar_ok, ticket;
  narrow_draw_ticket(p, &ticket);
  const int lane = (int)threadIdx.x & (G - 1), group = (int)threadIdx.x / G, n = p.n;
  const bool live = lane * V < n;
  const int col = live ? lane * V : 0;
  f32x2 w[P], acc_w[P], acc_b[P];
  {  // while the ticket is on its way
    float wf[V];
    if (p.w && live) {
      load_param<V>(p.w, p.w_dtype, (long long)col, wf);
    } else {
#pragma unroll
      for (int i = 0; i < V; ++i) wf[i] = 1.f;
    }
#pragma unroll
    for (int i = 0; i < P; ++i) {
      w[i] = pack2(wf[2 * i], wf[2 * i + 1]);
      acc_w[i] = acc_b[i] = splat2(0.f);
    }
  }
  const long long dx_col = (long long)(col / p.head_dim) * p.dx_head_stride + (col % p.head_dim);
  __syncthreads();
  const int cta = narrow_cta(&ticket);
  double* partials = reinterpret_cast<double*>(p.partials);
  if (cta >= p.workers) {
    if (narrow_wait_for_workers(p, &bar_ok))
      finalize_units_f64(partials, p.groups, p.n, p.dw, LN ? p.db : nullptr, cta - p.workers, p.finalizers, fin);
    else
      bwd_no_sums(p.dw, LN ? p.db : nullptr, p.n, 8, cta - p.workers, p.finalizers);
    narrow_depart(p);
    return;
  }
  const T* x = reinterpret_cast<const T*>(p.x) + col;
  const T* dy = reinterpret_cast<const T*>(p.dy) + col;
  const long long stride = (long long)p.workers * kGroups;
  const long long first = (long long)cta * kGroups + group;
  // the same number of turns for all groups of a warp: they meet in its shuffles
  const long long turns = ((p.rows - (first & ~(long long)(32 / G - 1))) + U * stride - 1) / (U * stride);
  const long long block = turns > 8 ? 4 : 2;  // chains of eight rows, of four where there are few of those
  auto keep = [&](bool more) {  // the sums so far into the lane's own words of shared memory
#pragma unroll
    for (int i = 0; i < P; ++i) {
      f32x2* at_w = reinterpret_cast<f32x2*>(&fold[0][group][lane * V]) + i;
      *at_w = more ? add2(*at_w, acc_w[i]) : acc_w[i];
      acc_w[i] = splat2(0.f);
      if constexpr (LN) {
        f32x2* at_b = reinterpret_cast<f32x2*>(&fold[1][group][lane * V]) + i;
        *at_b = more ? add2(*at_b, acc_b[i]) : acc_b[i];
        acc_b[i] = splat2(0.f);
      }
    }
  };
  long long row0 = first;
  for (long long t = 0; t < turns; ++t, row0 += U * stride) {
    if ((t & (block - 1)) == 0 && t != 0) keep(t != block);
    uint4 xr[U], yr[U];
    float rstd[U], mean[U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const long long row = row0 + u * stride;
      xr[u] = yr[u] = make_uint4(0u, 0u, 0u, 0u);
      rstd[u] = mean[u] = 0.f;
      if (row < p.rows) {
        rstd[u] = ld_here(p.rstd + row);
        if constexpr (LN) mean[u] = ld_here(p.mean + row);
        if (live) {
          xr[u] = ld_stream(x + row * p.x_row_stride);
          yr[u] = ld_stream(dy + row * p.dy_row_stride);
        }
      }
    }
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const long long row = row0 + u * stride;
      f32x2 xv[P], gv[P], a1 = splat2(0.f), a2 = splat2(0.f);
      const f32x2 rs = splat2(rstd[u]), m2 = splat2(mean[u]);
      Pairs<T>::unpack(xr[u], xv);
      Pairs<T>::unpack(yr[u], gv);
#pragma unroll
      for (int i = 0; i < P; ++i) {
        const f32x2 d = gv[i], g = mul2(d, w[i]);
        if constexpr (LN) {
          const f32x2 xhat = mul2(sub2(xv[i], m2), rs);
          a1 = add2(a1, g);
          a2 = fma2(g, xhat, a2);
          acc_w[i] = fma2(d, xhat, acc_w[i]);
          acc_b[i] = add2(acc_b[i], d);
          xv[i] = xhat;
        } else {
          a2 = fma2(g, xv[i], a2);
          acc_w[i] = fma2(d, mul2(xv[i], rs), acc_w[i]);
        }
        gv[i] = g;
      }
      float s1 = hsum2(a1), s2 = hsum2(a2);
#pragma unroll
      for (int o = G / 2; o > 0; o >>= 1) {
        if constexpr (LN) s1 += __shfl_xor_sync(0xffffffffu, s1, o);
        s2 += __shfl_xor_sync(0xffffffffu, s2, o);
      }
      if (row < p.rows && live) {
        const unsigned int bi = fast_div((unsigned int)row, p.seq_div);
        const unsigned int si = (unsigned int)row - bi * (unsigned int)p.seq;
        T* dx = reinterpret_cast<T*>(p.dx) + (long long)bi * p.dx_batch_stride + (long long)si * p.dx_seq_stride + dx_col;
        const float k = LN ? rstd[u] / p.n_f : ((s2 * -0.5f) * (rstd[u] * rstd[u] * rstd[u])) / p.n_f;
        const f32x2 k2 = splat2(k), n2 = splat2(p.n_f), s12 = splat2(-s1), s22 = splat2(-s2), kk = splat2(k * 2.f);
        f32x2 o[P];
#pragma unroll
        for (int i = 0; i < P; ++i)
          o[i] = LN ? mul2(k2, fma2(xv[i], s22, fma2(gv[i], n2, s12))) : fma2(gv[i], rs, mul2(kk, xv[i]));
        st_stream(dx, Pairs<T>::pack(o));
      }
    }
  }
  if (p.dw || p.db) {
    keep(turns > block);
    __syncthreads();
    for (int c = threadIdx.x; c < (LN ? 2 : 1) * n; c += kNarrowThreads) {
      const int plane = c >= n ? 1 : 0;
      const float* src = &fold[plane][0][c - plane * n];
      double a[4] = {0.0, 0.0, 0.0, 0.0};
#pragma unroll
      for (int g = 0; g < kGroups; ++g) a[g & 3] += (double)src[g * G * V];
      partials[((long long)plane * p.groups + cta) * n + (c - plane * n)] = (a[0] + a[1]) + (a[2] + a[3]);
    }
  }
  narrow_worker_done(p);
}

__global__ void __launch_bounds__(kNarrowThreads) norm_bwd_narrow_finalize_kernel(const NormBwdParams p) {
  wait_for_previous_kernel();
  __shared__ double fin[8 * 8];
  finalize_units_f64(reinterpret_cast<const double*>(p.partials), p.groups, p.n, p.dw, p.db, blockIdx.x, gridDim.x, fin);
}

// Rows of at most 32 vectors on the 16-byte grid.
template <typename T, bool LN>
int launch_norm_bwd_narrow(NormBwdParams p, size_t scratch_bytes, bool fused, cudaStream_t st) {
  constexpr int V = Elem<T>::V;
  const int nv = p.n / V;
  auto launch = [&](auto kernel, int lanes) {
    // three CTAs an SM, as the kernel's launch bounds say and the advertised scratch counts on, also where a compiler leaves room for more
    const int resident = cached_occupancy(reinterpret_cast<const void*>(kernel), kNarrowThreads);
    const long long room = (long long)(resident < 3 ? resident : 3) * device_info().sm_count;
    const int at_once = kNarrowThreads / lanes;
    long long grid = (p.rows + at_once - 1) / at_once;
    // Rows of 17 vectors and more have a quarter of the groups that those of 8 have. As long as one wave of CTAs would leave a group at most 12
    // rows (42624 rows on 148 SMs) there are two waves, of chains half as long: without them errors of dweight and dbias are up to 15 % larger
    // than with a warp per row (LayerNorm bf16 [8000, 256] 10.8 us in one wave, 14.3 so; [20000, 256] 16.0 and 18.6). Longer chains are
    // cut into blocks of four rows and more, whose sums are added once each, so that the second wave gains nothing there.
    const long long most = lanes == 32 && p.rows <= 12 * room * at_once ? 2 * room : room;
    if (grid > most) grid = most;
    if (p.dw || p.db) {
      // in rows of floats, as callers count; a partial row here takes two of them
      const long long plane = (long long)p.n * sizeof(float), rows = ((long long)scratch_bytes - 256) / (2 * plane);
      if (rows < 8)
        return fail(B200_ERR_WORKSPACE, "b200_norm_bwd: scratch of %zu bytes is too small (need >= %lld)", scratch_bytes, 256 + 16 * plane);
      if (grid > rows / 2) grid = rows / 2;
    }
    p.groups = p.workers = (int)grid;
    const int units = (p.n + 7) / 8 * ((p.dw ? 1 : 0) + (p.db ? 1 : 0));
    if (fused) {
      p.finalizers = units;
      launch_dependent(kernel, (unsigned)(grid + units), kNarrowThreads, 0, st, p);
      return launch_status("b200_norm_bwd [several rows per warp, fused finalize]");
    }
    launch_dependent(kernel, (unsigned)grid, kNarrowThreads, 0, st, p);
    const int rc = launch_status("b200_norm_bwd [several rows per warp]");
    if (rc != B200_OK || !units) return rc;
    launch_dependent(norm_bwd_narrow_finalize_kernel, (unsigned)units, kNarrowThreads, 0, st, p);
    return launch_status("b200_norm_bwd finalize");
  };
  if (nv <= 8) return launch(norm_bwd_narrow_kernel<T, LN, 8>, 8);
  if (nv <= 16) return launch(norm_bwd_narrow_kernel<T, LN, 16>, 16);
  return launch(norm_bwd_narrow_kernel<T, LN, 32>, 32);
}

template int launch_norm_bwd_narrow<float, true>(NormBwdParams, size_t, bool, cudaStream_t);
template int launch_norm_bwd_narrow<float, false>(NormBwdParams, size_t, bool, cudaStream_t);
template int launch_norm_bwd_narrow<__nv_bfloat16, true>(NormBwdParams, size_t, bool, cudaStream_t);
template int launch_norm_bwd_narrow<__nv_bfloat16, false>(NormBwdParams, size_t, bool, cudaStream_t);
template int launch_norm_bwd_narrow<__half, true>(NormBwdParams, size_t, bool, cudaStream_t);
template int launch_norm_bwd_narrow<__half, false>(NormBwdParams, size_t, bool, cudaStream_t);

}  // namespace b200
