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
  unsigned int* bar;  // words that are zero between launches (BwdWords)
  int groups;
  int workers;  // CTAs that walk the rows: the first of the grid
  int words_hold;  // the scratch has the zeroed words (all but the two-launch form, which reads none of them)
  // The partial rows are added up in the same launch, by all its CTAs (norm_bwd_narrow.cu: by so many beside the workers), a unit of
  // `width` columns at a time. 0: not at all, or by a launch of its own.
  int finalizers;
  int width;
};

// Words in front of the scratch, zero between launches. The two that CTAs ask for while others work lie in another sector than the rest.
enum BwdWords { kBwdArrived = 0, kBwdError = 1, kBwdLeft = 32, kBwdStarted = 48 };

__device__ __forceinline__ unsigned int bwd_peek(const unsigned int* word) {
  unsigned int v;
  asm volatile("ld.global.relaxed.gpu.u32 %0, [%1];" : "=r"(v) : "l"(word) : "memory");
  return v;
}
// Workers that have arrived, and with the same trip to memory whether an error is noted.
__device__ __forceinline__ unsigned int bwd_arrived(const NormBwdParams& p, bool& error) {
  static_assert(kBwdArrived == 0 && kBwdError == 1, "one aligned pair of words");
  unsigned long long v;
  asm volatile("ld.global.acquire.gpu.u64 %0, [%1];" : "=l"(v) : "l"(p.bar) : "memory");
  error = (v >> 32) != 0;
  return (unsigned int)v;
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

// The same for rows of n % 4 == 0 columns: the columns of dw and db are dealt out in units of 8 (a 32-byte sector of a partial
// row), a CTA each (192 CTAs for 768 columns of both). Where that makes more units than CTAs that fit, units of 16, 32 or 64
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

// ----------------------------------------------------------------------------------------------
// Rows and column sums in one launch that need not be cooperative. Every CTA, when its partial row is written, waits until all workers
// have arrived, and then adds its share of the columns up. The grid is no larger than what fits the GPU, so all of it is normally
// there; but nothing guarantees it (another stream's kernel may hold SMs), so a CTA that has seen all workers start waits for them,
// and one that has not leaves after a while, to make room; the CTA that leaves last then adds up all columns, whoever left early.
// Each wait ends: those it is for have started, and wait themselves for nothing but what has started.
// (A cooperative launch takes 2.5 us more when calls follow one another. With roles drawn as tickets, the first CTAs that start as
// workers and those behind them as finalizers, the draw came in front of the first copies and the finalizers' start behind
// the workers' end: in a graph LayerNorm bf16 [1000, 1024] 11.3 us, cooperative 9.2, so 9.2; [40000, 768] 39.8, 39.3 and 39.5; [40000, 1024] 49.3, 47.1 and 48.6.)
// ----------------------------------------------------------------------------------------------
// Asked of every CTA before its first row.
__device__ __forceinline__ void bwd_started(const NormBwdParams& p) {
  if (p.finalizers != 0 && threadIdx.x == 0 && (int)blockIdx.x < p.workers)
    asm volatile("red.global.relaxed.gpu.add.u32 [%0], 1;" ::"l"(p.bar + kBwdStarted) : "memory");
}

// A call, so that the widths that a few calls need stay out of the registers and the code of the kernels (with the width of 8 called
// too: LayerNorm bf16 [8000, 768] 15.0 -> 15.4 us).
static __device__ __noinline__ void finalize_any_units(const float* partials, int groups, int n, float* dw, float* db, int width, int first,
                                                       int step, double* smem) {
  finalize_units(partials, groups, n, dw, db, width, first, step, smem);
}

// Sums that cannot be formed are no numbers: the units first, first + step, ... of finalize_units.
__device__ __forceinline__ void bwd_no_sums(float* dw, float* db, int n, int width, int first, int step) {
  const int units = (n + width - 1) / width, total = units * ((dw ? 1 : 0) + (db ? 1 : 0));
  for (int s = first; s < total; s += step) {
    const bool is_db = !dw || s >= units;
    const int col = (dw && s >= units ? s - units : s) * width;
    for (int k = threadIdx.x; k < width && col + k < n; k += blockDim.x) (is_db ? db : dw)[col + k] = NAN;
  }
}

// Every thread of every CTA calls this when the CTA's partial row, if it has one, is written. flag: two words of shared memory.
__device__ __forceinline__ void bwd_combine(const NormBwdParams& p, float* db, double* smem /* [warps][64] */, int* flag) {
  if (p.finalizers == 0) return;
  enum { kAddUp, kLeave, kFailed };
  constexpr unsigned int kPatience = 64;  // polls, some 40 us
  __syncthreads();
  if (threadIdx.x == 0) {
    const unsigned int workers = (unsigned int)p.workers;
    if (blockIdx.x < workers) {
      __threadfence();
      atomicAdd(&p.bar[kBwdArrived], 1u);
    }
    int state = kAddUp;
    bool all_started = false, error = false;
    for (unsigned int polls = 0; bwd_arrived(p, error) < workers; ++polls) {
      if (polls >= kPatience && !all_started) {
        all_started = bwd_peek(p.bar + kBwdStarted) >= workers;
        if (!all_started) {
          state = kLeave;
          break;
        }
      }
      if (polls > (1u << 24)) {  // some seconds: with a scratch for few partial rows there are few workers, which may take long
        atomicExch(&p.bar[kBwdError], 1u);
        error = true;
        break;
      }
      if (polls > 4096) __nanosleep(64);
    }
    if (state == kAddUp && error) state = kFailed;
    __threadfence();
    flag[0] = state;
  }
  __syncthreads();
  const int state = flag[0];
  if (state == kAddUp && p.width == 8) finalize_units(p.partials, p.groups, p.n, p.dw, db, 8, (int)blockIdx.x, (int)gridDim.x, smem);
  else if (state == kAddUp) finalize_any_units(p.partials, p.groups, p.n, p.dw, db, p.width, (int)blockIdx.x, (int)gridDim.x, smem);
  else if (state == kFailed) bwd_no_sums(p.dw, db, p.n, p.width, (int)blockIdx.x, (int)gridDim.x);
  if (threadIdx.x == 0) {
    const unsigned int before = atomicAdd(&p.bar[kBwdLeft], state == kLeave ? 0x10001u : 1u);
    int missing = 0;
    if ((before & 0xffffu) == gridDim.x - 1) {  // the last one: no other CTA looks at the words any more
      missing = (before >> 16) != 0u || state == kLeave;
      if (missing && bwd_peek(p.bar + kBwdError) != 0u) missing = 2;
      atomicExch(&p.bar[kBwdArrived], 0u);
      atomicExch(&p.bar[kBwdStarted], 0u);
      atomicExch(&p.bar[kBwdLeft], 0u);
      __threadfence();
    }
    flag[1] = missing;
  }
  __syncthreads();
  if (flag[1] == 1) finalize_any_units(p.partials, p.groups, p.n, p.dw, db, p.width, 0, 1, smem);
  else if (flag[1] == 2) bwd_no_sums(p.dw, db, p.n, p.width, 0, 1);
}

// Host: the width of the units that rows of n columns are added up in, and how many there are, for `ctas` CTAs.
inline void bwd_plan_finalize(NormBwdParams& p, long long ctas) {
  const int planes = (p.dw ? 1 : 0) + (p.db ? 1 : 0);
  p.width = 8;
  while (p.width < 64 && (long long)(p.n + p.width - 1) / p.width * planes > ctas) p.width *= 2;
  p.finalizers = (p.n + p.width - 1) / p.width * planes;
}
// Host: the same for a launch whose CTAs add up themselves, and its grid: the workers where they get by with a unit each, more CTAs, up
// to what fits, where there are too few of them (LayerNorm f32 [64, 2048]: 6.9 us with 64 units for 64 workers, 7.4 with 256 for 256 CTAs).
inline unsigned bwd_plan_combined(NormBwdParams& p, long long room) {
  bwd_plan_finalize(p, p.workers);
  if (p.finalizers <= p.workers) return (unsigned)p.workers;
  bwd_plan_finalize(p, room);
  return (unsigned)(p.finalizers < room ? (p.finalizers > p.workers ? p.finalizers : p.workers) : room);
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
