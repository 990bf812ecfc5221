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
  unsigned int* bar;  // grid barrier words (cooperative variant)
  int groups;
  int fused;  // 1: barrier + finalize inside this launch
};

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

// The same inside a cooperative launch, after its grid barrier, for rows of n % 4 == 0 columns: the
// columns of dw and db are dealt out in units of 8 (a 32-byte sector of a partial row), so that the whole grid takes
// part (192 CTAs for 768 columns of both) and no second level, with a second grid barrier, is needed
// (LayerNorm backward bf16 [32768, 768], together with the copies that start before the weights are
// staged: 45.1 us with the two levels, 39.0 us so). Where that makes more units than CTAs, units of 16, 32 or 64
// columns: a unit is two barriers and a load latency, whatever its width (LayerNorm f32 [256, 8192]: 27.9 us with
// 2048 units of 8, 17.2 us with two times 128 of 64).
// width / 4 threads share a partial row's unit, the CTA's threads split the partial rows. fp64, fixed order.
// Four loads in flight per thread and no more: with the loop over the partial rows unrolled, this needed more
// registers than the kernels around it (the streaming kernel of fp32 RMSNorm 82 -> 120, so that one CTA of 288 threads
// fitted an SM instead of two: f32 [16352, 2052] 86 -> 112 us).
__device__ __forceinline__ void finalize_units(const float* partials, int groups, int n, float* dw, float* db,
                                               const int width, double* smem /* [warps][width] */) {
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, nwarps = blockDim.x >> 5;
  const int share = width / 4, units = (n + width - 1) / width, rows_at_once = blockDim.x / share;
  const int sub = tid & (share - 1);
  const int total = units * ((dw ? 1 : 0) + (db ? 1 : 0));
  for (int s = blockIdx.x; s < total; s += gridDim.x) {
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

// A call, so that the width that a few calls need stays out of the registers and the code of the kernels.
static __device__ __noinline__ void finalize_wide_units(const float* partials, int groups, int n, float* dw, float* db,
                                                        double* smem) {
  const int planes = (dw ? 1 : 0) + (db ? 1 : 0);
  int width = 16;
  while (width < 64 && (n + width - 1) / width * planes > (int)gridDim.x) width *= 2;
  finalize_units(partials, groups, n, dw, db, width, smem);
}

__device__ __forceinline__ void finalize_grid(const NormBwdParams& p, float* db, double* smem /* [warps][64] */) {
  if ((p.n + 7) / 8 * ((p.dw ? 1 : 0) + (db ? 1 : 0)) <= (int)gridDim.x)
    finalize_units(p.partials, p.groups, p.n, p.dw, db, 8, smem);
  else
    finalize_wide_units(p.partials, p.groups, p.n, p.dw, db, smem);
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
bool try_launch_norm_bwd_warp(NormBwdParams p, size_t scratch_bytes, bool cooperative, cudaStream_t st, int* rc);

unsigned int norm_bwd_warp_wait_timeouts();  // bounded waits of that kernel that ran out

}  // namespace b200
