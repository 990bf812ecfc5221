// Pieces shared by the translation units of the LayerNorm / RMSNorm backward: the parameter block,
// the fp64 finalize of the per-group partial rows, and the launch-geometry helpers.
#pragma once

#include "rowwise.cuh"
#include "tile_stream.cuh"

namespace b200 {

struct NormBwdParams {
  const void* x;
  const void* dy;
  const void* w;      // may be null (treated as ones)
  const float* mean;  // LayerNorm only
  const float* rstd;
  void* dx;
  float* dw;  // may be null
  float* db;  // may be null
  long long rows;
  int n;
  long long x_row_stride, dy_row_stride;
  int dy_elem_stride;  // 1, or 0 when dy is one element broadcast over the whole tensor (dy_row_stride 0 too)
  int w_dtype;
  // dx element (r, c) lives at (r / seq) * dx_batch_stride + (r % seq) * dx_seq_stride
  //                            + (c / head_dim) * dx_head_stride + (c % head_dim)
  int seq, head_dim;
  FastDiv seq_div;  // rows < 2^31, so row / seq is a 32-bit fast division
  long long dx_batch_stride, dx_seq_stride, dx_head_stride;
  float n_f;
  float* partials;    // [groups][n] for dw, followed by [groups][n] for db
  unsigned int* bar;  // words that are zero between launches: [0] workers done, [1] error, [2] CTAs gone, [3] tickets
  int groups;
  int workers;  // CTAs that walk the rows
  int words_hold;  // the scratch has the zeroed words (all but the two-launch form, which reads none of them)
  // The finalize in the same launch (0: none, or a launch of its own): this many CTAs beside the workers, a unit of
  // `width` columns at a time.
  int finalizers;
  int width;
};

// ----------------------------------------------------------------------------------------------
// One launch, two roles. The first `workers` CTAs that START are workers: they walk the rows, and the partial row that each
// leaves has the number of its ticket. The CTAs that start after them add the partial rows up once all workers have arrived.
// A worker waits for nobody, and a CTA that waits has started after every worker has: whatever else occupies the GPU,
// the wait ends, so that the launch need not be cooperative. (Cooperative launches with a grid barrier took
// 2 to 3 us more back to back, 10.4 us for a few hundred rows whose kernel runs 7.7, and the CTAs that had finished
// early did nothing.) Tickets decide who owns which rows, so the result does not depend on which CTA draws which.
// ----------------------------------------------------------------------------------------------
// A CTA's number, among the workers or, from p.workers on, the finalizers: thread 0 draws it, the others know it after the CTA's next
// barrier. The shuffle tells the compiler that it is the same in a warp, so that what depends on it can live in uniform registers, as
// what depends on blockIdx does. (All the same the kernels of 64 registers spilled: RMSNorm backward bf16 [4, 4096, 32, 128] 70 ->
// 78 us. Those have a finalize of their own, chained to them.)
__device__ __forceinline__ void bwd_draw_ticket(const NormBwdParams& p, int* ticket) {
  if (threadIdx.x == 0) *ticket = p.finalizers > 0 ? (int)atomicAdd(&p.bar[3], 1u) : (int)blockIdx.x;
}
__device__ __forceinline__ int bwd_cta(const int* ticket) { return __shfl_sync(0xffffffffu, *ticket, 0); }

// The last CTA puts the words back to zero (the error flag stays until the host has seen it).
__device__ __forceinline__ void bwd_depart(const NormBwdParams& p) {
  if (threadIdx.x == 0 && atomicAdd(&p.bar[2], 1u) == gridDim.x - 1) {
    atomicExch(&p.bar[0], 0u);
    atomicExch(&p.bar[2], 0u);
    atomicExch(&p.bar[3], 0u);
    __threadfence();
  }
}

// A worker's partial row is written: every thread of the CTA calls this.
__device__ __forceinline__ void bwd_worker_done(const NormBwdParams& p) {
  if (p.finalizers == 0) return;
  __syncthreads();
  if (threadIdx.x == 0) {
    __threadfence();
    atomicAdd(&p.bar[0], 1u);
  }
  bwd_depart(p);
}

// Waits until all workers have arrived; false when one has given up or the bound ran out (some seconds: with a scratch for few
// partial rows there are few workers, which may take long).
__device__ __forceinline__ bool bwd_wait_for_workers(const NormBwdParams& p, int* flag) {
  if (threadIdx.x == 0) {
    int ok = 1;
    for (unsigned int spins = 0;; ++spins) {
      unsigned int seen, err;
      asm volatile("ld.global.acquire.gpu.u32 %0, [%1];" : "=r"(seen) : "l"(p.bar) : "memory");
      asm volatile("ld.global.relaxed.gpu.u32 %0, [%1];" : "=r"(err) : "l"(p.bar + 1) : "memory");
      if (err == 0u && seen >= (unsigned int)p.workers) break;
      if (err != 0u || spins > (1u << 24)) {
        atomicExch(&p.bar[1], 1u);
        ok = 0;
        break;
      }
      __nanosleep(spins > 4096 ? 256 : 32);  // the workers' copies have the memory system
    }
    __threadfence();
    *flag = ok;
  }
  __syncthreads();
  return *flag != 0;
}

template <int V>
__device__ __forceinline__ void zero(float (&a)[V]) {
#pragma unroll
  for (int i = 0; i < V; ++i) a[i] = 0.f;
}

// Sum `groups` partial rows into out[0..n): each CTA takes 64-column chunks, its warps split the
// partial rows, fp64 accumulation, fixed order.
__device__ __forceinline__ void finalize_columns(const float* partials, int groups, int n, float* out,
                                                 double* smem /* [warps][64] */) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarps = blockDim.x >> 5;
  const int chunks = (n + 63) / 64;
  for (int chunk = blockIdx.x; chunk < chunks; chunk += gridDim.x) {
    const int c0 = chunk * 64 + lane, c1 = c0 + 32;
    double a0 = 0.0, a1 = 0.0;
    for (int g0 = warp; g0 < groups; g0 += 4 * nwarps) {  // eight loads in flight, then added in order
      float v0[4], v1[4];
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const int g = g0 + u * nwarps;
        const float* row = partials + (long long)g * n;
        v0[u] = (g < groups && c0 < n) ? __ldcg(row + c0) : 0.f;
        v1[u] = (g < groups && c1 < n) ? __ldcg(row + c1) : 0.f;
      }
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        a0 += (double)v0[u];
        a1 += (double)v1[u];
      }
    }
    smem[warp * 64 + lane] = a0;
    smem[warp * 64 + 32 + lane] = a1;
    __syncthreads();
    if (warp == 0) {
      double s0 = 0.0, s1 = 0.0;
      for (int w = 0; w < nwarps; ++w) {
        s0 += smem[w * 64 + lane];
        s1 += smem[w * 64 + 32 + lane];
      }
      if (c0 < n) out[c0] = (float)s0;
      if (c1 < n) out[c1] = (float)s1;
    }
    __syncthreads();
  }
}

// The same by the finalizers of the launch, for rows of n % 4 == 0 columns: the
// columns of dw and db are dealt out in units of 8 (a 32-byte sector of a partial row), a finalizer each
// (192 CTAs for 768 columns of both). Where that makes more units than CTAs that fit, units of 16, 32 or 64
// columns: a unit is two barriers and a load latency, whatever its width (LayerNorm f32 [256, 8192]: 27.9 us with
// 2048 units of 8, 17.2 us with two times 128 of 64).
// width / 4 threads share a partial row's unit, the CTA's threads split the partial rows. fp64, fixed order.
// Four loads in flight per thread and no more: with the loop over the partial rows unrolled, this needed more
// registers than the kernels around it (the streaming kernel of fp32 RMSNorm 82 -> 120, so that one CTA of 288 threads
// fitted an SM instead of two: f32 [16352, 2052] 86 -> 112 us).
__device__ __forceinline__ void finalize_units(const float* partials, int groups, int n, float* dw, float* db,
                                               const int width, const int first, const int step,
                                               double* smem /* [warps][width] */) {
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, nwarps = blockDim.x >> 5;
  const int share = width / 4, units = (n + width - 1) / width, rows_at_once = blockDim.x / share;
  const int sub = tid & (share - 1);
  const int total = units * ((dw ? 1 : 0) + (db ? 1 : 0));
  for (int s = first; s < total; s += step) {
    const bool is_db = !dw || s >= units;
    const int col = (dw && s >= units ? s - units : s) * width;
    const int c = col + 4 * sub;
    const float* src = partials + (is_db ? (long long)groups * n : 0) + c;
    double acc[4] = {0.0, 0.0, 0.0, 0.0};
    if (c < n) {
#pragma unroll 1
      for (int g0 = tid / share; g0 < groups; g0 += 4 * rows_at_once) {
        float4 v[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          const int g = g0 + u * rows_at_once;
          v[u] = g < groups ? __ldcg(reinterpret_cast<const float4*>(src + (long long)g * n)) : make_float4(0.f, 0.f, 0.f, 0.f);
        }
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          acc[0] += (double)v[u].x;
          acc[1] += (double)v[u].y;
          acc[2] += (double)v[u].z;
          acc[3] += (double)v[u].w;
        }
      }
    }
#pragma unroll
    for (int o = 16; o >= 2; o >>= 1) {
      if (o < share) break;
#pragma unroll
      for (int i = 0; i < 4; ++i) acc[i] += __shfl_xor_sync(0xffffffffu, acc[i], o);
    }
    if (lane < share) {
#pragma unroll
      for (int i = 0; i < 4; ++i) smem[warp * width + lane * 4 + i] = acc[i];
    }
    __syncthreads();
    for (int k = tid; k < width && col + k < n; k += blockDim.x) {
      double t = 0.0;
      for (int w = 0; w < nwarps; ++w) t += smem[w * width + k];
      (is_db ? db : dw)[col + k] = (float)t;
    }
    __syncthreads();
  }
}

// What a CTA with a ticket beyond the workers' does: waits, adds up, leaves.
__device__ __forceinline__ void bwd_finalize(const NormBwdParams& p, int cta, float* db, double* smem, int* flag) {
  if (bwd_wait_for_workers(p, flag))
    finalize_units(p.partials, p.groups, p.n, p.dw, db, p.width, cta - p.workers, p.finalizers, smem);
  bwd_depart(p);
}

// Host: how many finalizers a launch of rows of n columns gets, and the width of their units. `room`: CTAs of the kernel that fit.
inline void bwd_plan_finalize(NormBwdParams& p, long long room) {
  const int planes = (p.dw ? 1 : 0) + (p.db ? 1 : 0);
  p.width = 8;
  while (p.width < 64 && (long long)(p.n + p.width - 1) / p.width * planes > room) p.width *= 2;
  const long long units = (long long)(p.n + p.width - 1) / p.width * planes;
  p.finalizers = (int)(units < room ? units : room);
}

// Warp reduction of N (2, 4 or 8) values per lane at once: in every step a lane keeps one half of
// its values and hands the other half to its partner, so N values need N - 1 + log2(32 / N)
// shuffles instead of 5 N.
template <int N>
__device__ __forceinline__ float warp_reduce_multi(float (&v)[N], int lane) {
  // After the call lane l holds the warp total of value l / (32 / N).
  int off = 16;
#pragma unroll
  for (int n = N; n > 1; n >>= 1) {
    const bool upper = (lane & off) != 0;
#pragma unroll
    for (int i = 0; i < n / 2; ++i) {
      const float send = upper ? v[i] : v[i + n / 2];
      const float keep = upper ? v[i + n / 2] : v[i];
      v[i] = keep + __shfl_xor_sync(0xffffffffu, send, off);
    }
    off >>= 1;
  }
#pragma unroll
  for (int k = 0; k < 5; ++k) {
    if (off >= 1) {
      v[0] += __shfl_xor_sync(0xffffffffu, v[0], off);
      off >>= 1;
    }
  }
  return v[0];
}

// Warp-per-row kernel with per-warp copy rings (norm_bwd_warp.cu): rows of 33..256 vectors.
// Returns false when the shape does not fit (the caller takes another kernel); otherwise *rc is
// the launch status.
template <typename T, bool LN>
bool try_launch_norm_bwd_warp(NormBwdParams p, size_t scratch_bytes, bool fused, cudaStream_t st, int* rc);

unsigned int norm_bwd_warp_wait_timeouts();  // bounded waits of that kernel that ran out

// Rows of at most 32 vectors (norm_bwd_narrow.cu).
template <typename T, bool LN>
int launch_norm_bwd_narrow(NormBwdParams p, size_t scratch_bytes, bool fused, cudaStream_t st);

// Rows off the 16-byte grid whose dy and dx have their alignment (norm_bwd_span.cu): the rows and p.groups partial rows. False: the caller
// takes another kernel.
template <typename T, bool LN>
bool try_launch_norm_bwd_span(NormBwdParams& p, size_t scratch_bytes, cudaStream_t st, int* rc);

}  // namespace b200
