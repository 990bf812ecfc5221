// Pieces shared by the translation units of the BatchNorm training forward: the parameter block and
// the step from the fp64 totals of a channel's shifted sums to its mean / invstd / running statistics.
#pragma once

#include "rowwise.cuh"

namespace b200 {

struct BatchNormParams {
  const void* x;
  void* y;
  const void* weight;  // may be null
  const void* bias;    // may be null
  float* running_mean;  // may be null (no update)
  float* running_var;
  float* save_mean;    // [C] fp32 out (may be null)
  float* save_invstd;  // [C] fp32 out (may be null)
  long long rows;      // N*H*W for channels-last; N for the general path
  int channels;
  long long spatial;   // general path: H*W
  long long sn, sc, ss;  // general path: element strides of (n, c, spatial)
  int w_dtype;
  float eps, momentum, one_minus_momentum, unbias;
  double count;  // elements per channel
  double inv_count;  // 1 / count (a multiplication by it replaces two fp64 divisions per channel)
  int relu;
  float* partials;  // [P][2][C]
  float* stats;     // [2][C] mean, invstd (scratch copy every CTA reads)
};

// The value every sum of a channel is shifted by. Any value works as long as all threads of all
// CTAs use the same one; the closer it is to the channel's mean, the less the variance
// (s2 - s1 * s1 / n) / n cancels, and the cancellation multiplies the rounding error of s2 by
// 1 + (shift - mean)^2 / var. The first element of the channel can sit three standard deviations
// away (a factor of ten); the mean of the channel's first sixteen rows (rows beyond the last one
// repeat it) rarely sits more than one.
constexpr int BN_SHIFT_ROWS = 16;

// The shift is cut to eight significant bits (a bf16 value). With 16-bit inputs x - shift then
// has so few bits that the sums of the differences are exact or nearly so; with a full fp32 shift
// every addition would drop the same low bits of the shift and the errors would add up instead
// of cancelling (measured: the mean of 6.4 M bf16 values off by 2e-6 instead of 1e-8).
__device__ __forceinline__ float bn_round_shift(float v) {
  return __uint_as_float((__float_as_uint(v) + 0x8000u) & 0xffff0000u);
}

// The shift from the sum of the sixteen rows; row 0 where that overflows although the values are finite (a channel of 3e37).
__device__ __forceinline__ float bn_shift_of_sum(float sum, float row0) {
  const float mean = bn_round_shift(__fmul_rn(sum, 1.0f / BN_SHIFT_ROWS));
  return fabsf(mean) < INFINITY ? mean : row0;
}

template <typename T>
__device__ __forceinline__ void bn_shift_load(const T* x, int c, int channels, long long rows, T (&v)[BN_SHIFT_ROWS]) {
#pragma unroll
  for (int r = 0; r < BN_SHIFT_ROWS; ++r) {
    const long long rr = r < rows ? r : rows - 1;
    v[r] = ld_here(x + rr * channels + c);
  }
}

template <typename T>
__device__ __forceinline__ float bn_shift_of(const T (&v)[BN_SHIFT_ROWS]) {
  float s = 0.f;
#pragma unroll
  for (int r = 0; r < BN_SHIFT_ROWS; ++r) s = __fadd_rn(s, Elem<T>::to_f32(v[r]));
  return bn_shift_of_sum(s, Elem<T>::to_f32(v[0]));
}

template <typename T>
__device__ __forceinline__ float bn_shift_scalar(const T* x, int c, int channels, long long rows) {
  T v[BN_SHIFT_ROWS];
  bn_shift_load<T>(x, c, channels, rows, v);
  return bn_shift_of<T>(v);
}

// Turns the fp64 totals of the shifted sums of one channel into mean / invstd and, for the one
// caller that owns the channel's global outputs, writes the saved and running statistics.
// old_mean, old_var: the channel's running statistics, which the caller fetched while the sums were being formed, so that
// their latency is not waited for here.
__device__ __forceinline__ void bn_channel_stats(const BatchNormParams& p, int c, double s1, double s2, float shift,
                                                 bool write_global, float* mean_out, float* invstd_out,
                                                 float old_mean, float old_var) {
  // On the critical path of every launch (one thread per channel computes this while the others
  // wait), so no fp64 division or square root: a product with 1/count and the fp64 rsqrt.
  const double mean_shifted = s1 * p.inv_count;
  double var = (s2 - s1 * mean_shifted) * p.inv_count;
  if (var < 0.0) var = 0.0;
  const float mean = (float)((double)shift + mean_shifted);
  const float varf = (float)var;
  // 1 / sqrt(var + eps) from the fp64 variance, rounded once: within an ulp or two of the graph's
  // rsqrt(fp32(var) + eps), and the closest fp32 value to what the graph gives in fp64
  const float invstd = (float)rsqrt(var + (double)p.eps);
  *mean_out = mean;
  *invstd_out = invstd;
  if (write_global) {
    if (p.save_mean) p.save_mean[c] = mean;
    if (p.save_invstd) p.save_invstd[c] = invstd;
    if (p.running_mean) {
      p.running_mean[c] = mean * p.momentum + old_mean * p.one_minus_momentum;
      p.running_var[c] = (varf * p.unbias) * p.momentum + old_var * p.one_minus_momentum;
    }
  }
}

// Adds up what the threads of a CTA hold: `one` and `two` are flat arrays of blockDim.x * V values each, of
// which value f belongs to channel f % channels (blockDim.x * V is a multiple of the channel count). fp64, fixed order.
// With at most a quarter as many channels as threads, as many threads share a channel as there are: one thread per channel is
// a chain of blockDim.x * V / channels additions there (forward, bf16 [N, 16, 7, 7] of 0.5 MB 10.8 us, so 7.4; 36 channels
// 8.5 and 7.4). With more channels the second step costs more than the chain (92 channels, 12 / 45 MB: bf16 14.2 / 28.0 us in one
// step, 14.4 / 28.6 in two, f32 12.4 / 23.6 and 13.1 / 24.4). `part`: 2 * blockDim.x doubles.
template <typename Out, int V>
__device__ __forceinline__ void bn_fold_channels(const float* one, const float* two, double* part, int channels,
                                                 Out* row_one, Out* row_two) {
  const int tid = threadIdx.x, threads = blockDim.x, values = threads * V;
  const int share = 4 * channels <= threads ? threads / channels : 1;  // threads per channel
  if (share == 1) {
    for (int c = tid; c < channels; c += threads) {
      double a = 0.0, b = 0.0;
      for (int f = c; f < values; f += channels) {
        a += (double)one[f];
        b += (double)two[f];
      }
      row_one[c] = (Out)a;
      row_two[c] = (Out)b;
    }
    return;
  }
  if (tid < share * channels) {
    double a = 0.0, b = 0.0;
    for (int f = tid; f < values; f += share * channels) {
      a += (double)one[f];
      b += (double)two[f];
    }
    part[tid] = a;
    part[threads + tid] = b;
  }
  __syncthreads();
  for (int i = tid; i < 2 * channels; i += threads) {  // both sums of a channel at the same time
    const int c = i < channels ? i : i - channels;
    const double* p = part + (i < channels ? 0 : threads) + c;
    double a = 0.0;
    for (int r = 0; r < share; ++r) a += p[r * channels];
    if (i < channels) row_one[c] = (Out)a;
    else row_two[c] = (Out)a;
  }
}

// A tensor whose elements are no whole number of vectors ends with fewer than V of them. The sums pass reads them
// one by one, in the thread whose next vector they would begin; the rest of that vector is zero.
template <typename T>
__device__ __forceinline__ uint4 load_first(const T* src, int count) {
  constexpr int V = Elem<T>::V;
  union {
    T e[V];
    uint4 raw;
  } u;
  u.raw = make_uint4(0u, 0u, 0u, 0u);
#pragma unroll
  for (int i = 0; i < V - 1; ++i)
    if (i < count) u.e[i] = ld_here(src + i);
  return u.raw;
}
// Contiguous NCHW tensors (batch_norm_nchw.cu): one launch, the CTAs that share a channel form a
// thread-block cluster. Returns false when the shape does not fit (the caller takes another path).
template <typename T>
bool try_launch_batch_norm_nchw(const BatchNormParams& p, cudaStream_t st, int* rc);

}  // namespace b200
