// BatchNorm2d training forward: per-channel var_mean over (N,H,W), normalise, affine, optional
// ReLU, running-statistics update.
//
// Replaces the three-kernel Triton plan of the BatchNorm repros in the reference
// (repros/canonical/var_mean_42fad1ece813/oracle.py:11-46 partial sums, :49-87 finalize and
// running stats, :90-119 normalise pass that re-reads x from DRAM).
//
// Evaluation order, as the decomposed aten graph has it (var_mean_42fad1ece813/repro.py:23-58):
//   var, mean = var_mean(float(x), correction 0);  invstd = rsqrt(var + eps)
//   y = relu(cast(((x - mean) * invstd) * w + b))           (ReLU after the cast)
//   running_mean = mean*m + running_mean*(1-m)
//   running_var  = (var*unbias)*m + running_var*(1-m),  unbias = n/(n-1)
//
// Channels-last tensors are flat arrays of 16-byte vectors for three launches (sums of shifted values,
// finalize, normalise), chained by programmatic dependent launch; the shift is a value of the channel itself or the
// mean of a few, so that S2 - S1^2/n does not cancel. Contiguous NCHW tensors take the single-launch cluster
// kernel of batch_norm_nchw.cu. Any other layout takes the three-launch general path: strided statistics,
// finalize, strided normalise.
#include "batch_norm.cuh"
#include "tile_stream.cuh"

#include <mutex>
#include <type_traits>

namespace b200 {

// ReLU of a packed vector after the cast, as the graph has it; NaN stays NaN.
template <typename T>
__device__ __forceinline__ uint4 relu_packed(uint4 packed) {
  if constexpr (std::is_same<T, __nv_bfloat16>::value) {
    const __nv_bfloat162 z = __float2bfloat162_rn(0.f);
    uint32_t* w = reinterpret_cast<uint32_t*>(&packed);
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      __nv_bfloat162 h = __hmax2_nan(*reinterpret_cast<__nv_bfloat162*>(&w[i]), z);
      w[i] = *reinterpret_cast<uint32_t*>(&h);
    }
  } else if constexpr (std::is_same<T, __half>::value) {
    const __half2 z = __float2half2_rn(0.f);
    uint32_t* w = reinterpret_cast<uint32_t*>(&packed);
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      __half2 h = __hmax2_nan(*reinterpret_cast<__half2*>(&w[i]), z);
      w[i] = *reinterpret_cast<uint32_t*>(&h);
    }
  } else {
    float* w = reinterpret_cast<float*>(&packed);
#pragma unroll
    for (int i = 0; i < 4; ++i) w[i] = w[i] < 0.f ? 0.f : w[i];  // NaN < 0 is false: NaN stays
  }
  return packed;
}

__device__ __forceinline__ void bn_finalize_channel(const BatchNormParams& p, int c, int num_partials, float shift) {
  // Called by one warp per channel: lanes split the partials, fp64 accumulation, fixed order.
  const int lane = threadIdx.x & 31;
  float old_mean = 0.f, old_var = 0.f;  // requested now, so that they do not cost a round trip after the sums
  if (lane == 0 && p.running_mean) {
    old_mean = __ldcg(p.running_mean + c);
    old_var = __ldcg(p.running_var + c);
  }
  double s1 = 0.0, s2 = 0.0;
  for (int g0 = lane; g0 < num_partials; g0 += 8 * 32) {  // eight pairs of loads in flight before any is used
    float a[8], b[8];
#pragma unroll
    for (int u = 0; u < 8; ++u) {
      const int g = g0 + u * 32;
      a[u] = g < num_partials ? __ldcg(p.partials + ((long long)g * 2) * p.channels + c) : 0.f;
      b[u] = g < num_partials ? __ldcg(p.partials + ((long long)g * 2 + 1) * p.channels + c) : 0.f;
    }
#pragma unroll
    for (int u = 0; u < 8; ++u) {
      s1 += (double)a[u];
      s2 += (double)b[u];
    }
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    s1 += __shfl_xor_sync(0xffffffffu, s1, o);
    s2 += __shfl_xor_sync(0xffffffffu, s2, o);
  }
  if (lane == 0) {
    float mean, invstd;
    bn_channel_stats(p, c, s1, s2, shift, true, &mean, &invstd, old_mean, old_var);
    p.stats[c] = mean;
    p.stats[p.channels + c] = invstd;
  }
}

// ----------------------------------------------------------------------------------------------
// General path: x addressed as (n, c, s) with arbitrary strides.
// ----------------------------------------------------------------------------------------------
template <typename T>
__global__ void __launch_bounds__(256) batch_norm_stats_general_kernel(const BatchNormParams p) {
  wait_for_previous_kernel();
  __shared__ float red[32];
  const int c = blockIdx.x;
  const int split = blockIdx.y, splits = gridDim.y;
  const T* x = reinterpret_cast<const T*>(p.x);
  const float shift = Elem<T>::to_f32(x[(long long)c * p.sc]);
  const long long total = p.rows * p.spatial;
  const long long per = (total + splits - 1) / splits;
  const long long e0 = (long long)split * per;
  const long long e1 = e0 + per < total ? e0 + per : total;
  float s1 = 0.f, s2 = 0.f;
  for (long long e = e0 + threadIdx.x; e < e1; e += blockDim.x) {
    const long long n = e / p.spatial, s = e % p.spatial;
    const float d = Elem<T>::to_f32(x[n * p.sn + (long long)c * p.sc + s * p.ss]) - shift;
    s1 += d;
    s2 += d * d;
  }
  s1 = block_reduce<SumOp>(s1, red);
  s2 = block_reduce<SumOp>(s2, red);
  if (threadIdx.x == 0) {
    p.partials[((long long)split * 2) * p.channels + c] = s1;
    p.partials[((long long)split * 2 + 1) * p.channels + c] = s2;
  }
}

// rows_shift: the sums were shifted by bn_shift_scalar (channels-last flat path, p.rows = N*H*W)
// instead of by the channel's first element.
template <typename T>
__global__ void __launch_bounds__(256) batch_norm_finalize_general_kernel(const BatchNormParams p,
                                                                          int num_partials, int rows_shift) {
  wait_for_previous_kernel();
  const int warps = blockDim.x >> 5;
  const int c = blockIdx.x * warps + (threadIdx.x >> 5);
  if (c >= p.channels) return;
  const T* x = reinterpret_cast<const T*>(p.x);
  const float shift = rows_shift ? bn_shift_scalar<T>(x, c, p.channels, p.rows) : Elem<T>::to_f32(x[(long long)c * p.sc]);
  bn_finalize_channel(p, c, num_partials, shift);
}

// One element of y, at `off` in both tensors.
template <typename T>
__device__ __forceinline__ void bn_apply_one(const BatchNormParams& p, long long off, int c) {
  const float w = p.weight ? load_param1(p.weight, p.w_dtype, c) : 1.f;
  const float b = p.bias ? load_param1(p.bias, p.w_dtype, c) : 0.f;
  float o = ((Elem<T>::to_f32(reinterpret_cast<const T*>(p.x)[off]) - p.stats[c]) * p.stats[p.channels + c]) * w + b;
  if (p.relu) o = o < 0.f ? 0.f : o;
  reinterpret_cast<T*>(p.y)[off] = Elem<T>::from_f32(o);
}

template <typename T>
__global__ void __launch_bounds__(256) batch_norm_apply_general_kernel(const BatchNormParams p) {
  wait_for_previous_kernel();
  const int c = blockIdx.x;
  const T* x = reinterpret_cast<const T*>(p.x);
  T* y = reinterpret_cast<T*>(p.y);
  const float mean = p.stats[c], invstd = p.stats[p.channels + c];
  const float w = p.weight ? load_param1(p.weight, p.w_dtype, c) : 1.f;
  const float b = p.bias ? load_param1(p.bias, p.w_dtype, c) : 0.f;
  const long long total = p.rows * p.spatial;
  const long long per = (total + gridDim.y - 1) / gridDim.y;
  const long long e0 = (long long)blockIdx.y * per;
  const long long e1 = e0 + per < total ? e0 + per : total;
  for (long long e = e0 + threadIdx.x; e < e1; e += blockDim.x) {
    const long long n = e / p.spatial, s = e % p.spatial;
    const long long off = n * p.sn + (long long)c * p.sc + s * p.ss;
    float o = ((Elem<T>::to_f32(x[off]) - mean) * invstd) * w + b;
    if (p.relu) o = o < 0.f ? 0.f : o;
    y[off] = Elem<T>::from_f32(o);
  }
}

// ----------------------------------------------------------------------------------------------
// Channels-last tensors whose channel pattern repeats within 512 vectors: three launches over the tensor as a flat
// array of 16-byte vectors, whatever the channel count (the corpus of the reference has channels-last BatchNorm points with 24, 36, 60,
// 92, 100, 480 ... channels; repros/canonical/var_mean_42fad1ece813/shapes.json).
//
// A vector holds V consecutive elements of the flat [rows * C] array, so it may straddle the end
// of a row. The pattern of channels under a vector repeats every PV = C / gcd(C, V) vectors
// (lcm(C, V) elements): vector i has phase i % PV and its element j belongs to channel
// (phase * V + j) % C. The CTA's vector range starts at a multiple of PV and blockDim.x is a
// multiple of PV, so a thread keeps its phase - its V channels - for the whole launch and its
// sums, and later its mean / invstd / weight / bias, stay in registers.
//   sums      CTA b takes vectors [b * per, (b + 1) * per): shifted sums per thread, the threads of
//             a phase folded in a fixed order (fp64), one fp32 partial row per CTA
//   finalize  a warp per channel (batch_norm_finalize_general_kernel)
//   apply     the same ranges walked from the end (what the sums pass read last is what L2 still
//             holds), y written with streaming stores
// ----------------------------------------------------------------------------------------------
// MAXT: 256 threads, or 512 for patterns of more than 256 vectors.
template <typename T, int MAXT>
__global__ void __launch_bounds__(MAXT, MAXT == 256 ? 3 : 1) batch_norm_sums_cl_flat_kernel(const BatchNormParams p, long long vecs_per_cta,
                                                                      int PV, int rows_shift) {
  wait_for_previous_kernel();
  constexpr int V = Elem<T>::V;
  __shared__ float red[2 * MAXT * V];  // [2][threads][V]
  const int tid = threadIdx.x, T_ = blockDim.x, C = p.channels;
  const int ph = tid % PV;
  const long long total = p.rows * C / V;
  const long long v0 = (long long)blockIdx.x * vecs_per_cta;
  long long v1 = v0 + vecs_per_cta;
  if (v1 > total) v1 = total;
  const T* xe = reinterpret_cast<const T*>(p.x);
  const uint4* x = reinterpret_cast<const uint4*>(p.x);
  // The shift of every channel (bn_shift_scalar: mean of its first sixteen rows, eight significant
  // bits; the finalize kernel forms the same value) is computed once per CTA into shared memory,
  // at most 2 * MAXT * V channels per round, and every thread picks up its V channels.
  f32x2 shift[V / 2], s1[V / 2], s2[V / 2];
  f32x2 upper[V / 2];  // a thread's sum of squares moves here every 16 vectors: two short chains instead of one long one
#pragma unroll
  for (int i = 0; i < V / 2; ++i) shift[i] = s1[i] = s2[i] = upper[i] = splat2(0.f);
  if (!rows_shift) {  // short chains (small tensors): the channel's element of row 0 will do
#pragma unroll
    for (int i = 0; i < V / 2; ++i)
      shift[i] = pack2(Elem<T>::to_f32(ld_here(xe + (ph * V + 2 * i) % C)), Elem<T>::to_f32(ld_here(xe + (ph * V + 2 * i + 1) % C)));
  }
  for (int c0 = 0; rows_shift && c0 < C; c0 += 2 * MAXT * V) {
    for (int c = c0 + tid; c < C && c < c0 + 2 * MAXT * V; c += T_) red[c - c0] = bn_shift_scalar<T>(xe, c, C, p.rows);
    __syncthreads();
#pragma unroll
    for (int i = 0; i < V / 2; ++i) {
      const int ca = (ph * V + 2 * i) % C, cb = (ph * V + 2 * i + 1) % C;
      float lo, hi;
      unpack2(shift[i], lo, hi);
      if (ca >= c0 && ca < c0 + 2 * MAXT * V) lo = red[ca - c0];
      if (cb >= c0 && cb < c0 + 2 * MAXT * V) hi = red[cb - c0];
      shift[i] = pack2(lo, hi);
    }
    __syncthreads();
  }
  constexpr int U = 4;  // vectors in flight per thread (three CTAs per SM)
  int round = 0;
  for (long long v = v0 + tid; v < v1; v += (long long)U * T_) {
    uint4 raw[U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const long long i = v + (long long)u * T_;
      if (i < v1) raw[u] = ld_stream(reinterpret_cast<const T*>(x + i));
    }
#pragma unroll
    for (int u = 0; u < U; ++u) {
      if (v + (long long)u * T_ < v1) {
        f32x2 f[V / 2];
        Pairs<T>::unpack(raw[u], f);
#pragma unroll
        for (int i = 0; i < V / 2; ++i) {
          const f32x2 d = sub2(f[i], shift[i]);
          s1[i] = add2(s1[i], d);
          s2[i] = fma2(d, d, s2[i]);
        }
      }
    }
    if ((++round & 3) == 0) {
#pragma unroll
      for (int i = 0; i < V / 2; ++i) {
        upper[i] = add2(upper[i], s2[i]);
        s2[i] = splat2(0.f);
      }
    }
  }
  float* r1 = red;
  float* r2 = red + MAXT * V;
#pragma unroll
  for (int i = 0; i < V / 2; ++i) {
    unpack2(s1[i], r1[tid * V + 2 * i], r1[tid * V + 2 * i + 1]);
    unpack2(add2(upper[i], s2[i]), r2[tid * V + 2 * i], r2[tid * V + 2 * i + 1]);
  }
  __syncthreads();
  const int period = PV * V;  // elements; a multiple of C
  for (int c = tid; c < C; c += T_) {
    double a = 0.0, b = 0.0;
    for (int idx = c; idx < period; idx += C) {  // every (phase, element) that lands on channel c
      const int col = idx / V, e = idx % V;
      for (int t = col; t < T_; t += PV) {
        a += (double)r1[t * V + e];
        b += (double)r2[t * V + e];
      }
    }
    p.partials[((long long)blockIdx.x * 2) * C + c] = (float)a;
    p.partials[((long long)blockIdx.x * 2 + 1) * C + c] = (float)b;
  }
}

template <typename T, int MAXT>
__global__ void __launch_bounds__(MAXT, MAXT == 256 ? 3 : 1) batch_norm_apply_cl_flat_kernel(const BatchNormParams p, long long vecs_per_cta,
                                                                       int PV) {
  wait_for_previous_kernel();
  constexpr int V = Elem<T>::V;
  const int tid = threadIdx.x, T_ = blockDim.x, C = p.channels;
  const int ph = PV - 1 - tid % PV;  // the range ends on a multiple of PV: its last vector has phase PV - 1
  const long long total = p.rows * C / V;
  const long long v0 = (long long)blockIdx.x * vecs_per_cta;
  long long v1 = v0 + vecs_per_cta;
  if (v1 > total) v1 = total;  // total is a multiple of PV as well (the launcher checks)
  const uint4* x = reinterpret_cast<const uint4*>(p.x);
  uint4* y = reinterpret_cast<uint4*>(p.y);
  f32x2 mean2[V / 2], inv2[V / 2], w2[V / 2], b2[V / 2];
#pragma unroll
  for (int i = 0; i < V / 2; ++i) {
    const int c0 = (ph * V + 2 * i) % C, c1 = (ph * V + 2 * i + 1) % C;
    mean2[i] = pack2(p.stats[c0], p.stats[c1]);
    inv2[i] = pack2(p.stats[C + c0], p.stats[C + c1]);
    w2[i] = p.weight ? pack2(load_param1(p.weight, p.w_dtype, c0), load_param1(p.weight, p.w_dtype, c1)) : splat2(1.f);
    b2[i] = p.bias ? pack2(load_param1(p.bias, p.w_dtype, c0), load_param1(p.bias, p.w_dtype, c1)) : splat2(0.f);
  }
  const bool relu = p.relu != 0;
  constexpr int U = 8;
  for (long long v = v1 - 1 - tid; v >= v0; v -= (long long)U * T_) {
    uint4 raw[U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const long long i = v - (long long)u * T_;
      if (i >= v0) raw[u] = ld_stream(reinterpret_cast<const T*>(x + i));
    }
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const long long i = v - (long long)u * T_;
      if (i >= v0) {
        f32x2 f[V / 2];
        Pairs<T>::unpack(raw[u], f);
#pragma unroll
        for (int k = 0; k < V / 2; ++k) {
          f[k] = add2(mul2(mul2(sub2(f[k], mean2[k]), inv2[k]), w2[k]), b2[k]);
          if (relu) {
            float lo, hi;
            unpack2(f[k], lo, hi);
            f[k] = pack2(lo < 0.f ? 0.f : lo, hi < 0.f ? 0.f : hi);
          }
        }
        st_stream(reinterpret_cast<T*>(y + i), Pairs<T>::pack(f));
      }
    }
  }
}

// Returns false when the shape does not fit (the caller takes the element-wise path).
template <typename T>
static bool try_launch_batch_norm_cl_flat(BatchNormParams p, size_t scratch_bytes, cudaStream_t st, int* rc) {
  constexpr int V = Elem<T>::V;
  const DeviceInfo& dev = device_info();
  const long long C = p.channels;
  long long g = C, h = V;  // gcd(C, V)
  while (h) { const long long t = g % h; g = h; h = t; }
  const long long PV = C / g;
  const long long elems = p.rows * C;
  if (PV > 512 || elems % (PV * V) != 0) return false;  // whole periods only: every range ends on a multiple of PV
  const long long total = elems / V;
  const int threads = (int)(PV <= 256 ? 256 / PV * PV : PV);
  const long long stats_floats = 2 * C;
  const long long room = ((long long)scratch_bytes - 256) / (long long)sizeof(float) - stats_floats;
  if (room < 2 * C) return false;
  long long splits = 8LL * dev.sm_count;
  if (splits > room / (2 * C)) splits = room / (2 * C);
  // at least one full round of loads (8 vectors) per thread: small tensors get few partial rows and a
  // short finalize
  if (splits * threads * 8 > total) splits = (total + threads * 8 - 1) / (threads * 8);
  if (splits < 1) splits = 1;
  long long per = (total + splits - 1) / splits;
  per = (per + PV - 1) / PV * PV;
  splits = (total + per - 1) / per;
  p.stats = p.partials + splits * 2 * C;
  const int rows_shift = per > 32LL * threads ? 1 : 0;  // more than 32 vectors per thread
  if (threads <= 256) launch_dependent(batch_norm_sums_cl_flat_kernel<T, 256>, (unsigned)splits, threads, 0, st, p, per, (int)PV, rows_shift);
  else launch_dependent(batch_norm_sums_cl_flat_kernel<T, 512>, (unsigned)splits, threads, 0, st, p, per, (int)PV, rows_shift);
  *rc = launch_status("b200_batch_norm_fwd sums [channels-last, flat vectors]");
  if (*rc != B200_OK) return true;
  launch_dependent(batch_norm_finalize_general_kernel<T>, (p.channels + 7) / 8, 256, 0, st, p, (int)splits, rows_shift);
  *rc = launch_status("b200_batch_norm_fwd finalize");
  if (*rc != B200_OK) return true;
  if (threads <= 256) launch_dependent(batch_norm_apply_cl_flat_kernel<T, 256>, (unsigned)splits, threads, 0, st, p, per, (int)PV);
  else launch_dependent(batch_norm_apply_cl_flat_kernel<T, 512>, (unsigned)splits, threads, 0, st, p, per, (int)PV);
  *rc = launch_status("b200_batch_norm_fwd apply [channels-last, flat vectors]");
  return true;
}

// ----------------------------------------------------------------------------------------------
// The same three steps as they are taken for most tensors. These kernels need no whole number of periods or vectors (odd channel
// counts whose rows are no multiple of 8: bf16 [39, 287, 7, 7] 18.6 us element by element, 8.1 so):
//   sums      all CTAs are resident and take chunks b, b + grid, ...: the launch moves through the tensor
//             from front to back as a whole, and what it leaves in L2 is the tensor's last part
//   finalize  a CTA per channel
//   apply     the chunks from the last to the first, so that it starts with what is in L2
// Both passes bring x in through a ring of each thread's own in shared memory (asynchronous 16-byte
// copies, read only by the thread that issued them: no barrier, no registers), which keeps about 160 KB
// per SM on the way whatever the arithmetic does. The three kernels are chained by programmatic
// dependent launch; apply fills its ring before the statistics are there.
// Measured against the kernels above: bf16 [672, 96, 28, 28] (101 MB) 86.7 -> 49.2 us, [1010, 92, 14, 14] (36 MB)
// 48.1 -> 24.0, [161, 96, 28, 28] (24 MB) 34.2 -> 19.2, [64, 120, 28, 28] (12 MB) 19.8 -> 13.7, [40, 480, 7, 7]
// (2 MB) 10.3 -> 8.6, [8, 24, 7, 7] (20 KB) 11.3 -> 7.3; f32 [1402, 92, 14, 14] (101 MB) 74.7 -> 51.6,
// [168, 92, 14, 14] (12 MB) 18.1 -> 12.5. Against one cooperative launch for power-of-two vector counts from 8 MB up
// (the tensor's end in shared memory between the passes, two grid barriers): bf16 64 channels 12 / 30 / 60 / 100 / 200 MB
// 20.9 / 27.3 / 37.7 / 56.0 / 107.5 -> 13.3 / 20.8 / 30.8 / 46.7 / 102.5, 256 channels 52.5 / 60.0 / 70.6 / 90.2 / 142.6 ->
// 14.6 / 22.4 / 32.8 / 51.3 / 104.5. The same with this file's copies in one cooperative launch: 18.6 / 26.2 / 35.6 / 49.4 / 103.0.
// What bounds it on 100 MB: the first pass reads x next to the write-back of the last y, the second finds 60 % of x in L2.
// apply reads x evict-first, as nothing reads it again: 53.2 -> 52.0 us (back to back) on bf16 [256, 64, 56, 56].
// With more than 1024 channels and less than 12 MB the CTAs of the finalize are the larger part of it, and the
// kernels above stay (bf16 [40, 2040, 7, 7] 19.0 us there, 20.9 here, [20, 4080, 7, 7] 19.9 and 23.9; 16 MB of 2040 channels 32.8 and 26.6;
// 1020 channels, 8 MB: 17.8 and 16.5; f32 1000 channels, 8 MB: 14.2 and 14.9). Just above 1024 channels the line could lie lower
// (1200 channels, 9.4 MB: 24.5 there, 20.4 here).
// ----------------------------------------------------------------------------------------------
static bool ring_is_slower(long long channels, long long bytes) { return channels > 1024 && bytes < 12000000; }

constexpr int kRingU = 4;  // vectors per thread in a stage
constexpr int kRingS = 6;  // stages
constexpr int kRingBytesPerThread = kRingS * kRingU * 16;  // 384

// Brings vectors v, v + T_, ... that lie in [0, total) into stage s; always one group. LAST: they are not read again.
template <bool LAST>
__device__ __forceinline__ void bn_ring_issue(const uint4* x, uint32_t mine, int s, long long v, long long total, int T_) {
  const uint64_t policy = LAST ? l2_policy_evict_first() : 0;
  const uint32_t dst = mine + (uint32_t)(s * kRingU * T_) * 16u;
#pragma unroll
  for (int u = 0; u < kRingU; ++u) {
    const long long i = v + (long long)u * T_;
    if (i >= 0 && i < total) {
      if constexpr (LAST) copy_async16_hint(dst + (uint32_t)(u * T_) * 16u, x + i, policy);
      else copy_async16(dst + (uint32_t)(u * T_) * 16u, x + i);
    }
  }
  copy_async_commit();
}

// MAXT: 256 threads, or 512 for patterns of more than 256 vectors.
// SHIFT: by what a channel's sums are shifted (batch_norm.cuh): kShiftRow0 by its element of row 0, asked for in front of the first
// copies; kShiftRows by the mean of its first sixteen rows, asked for behind them; kShiftRowsFirst by the same, in front of them.
// 85 registers: two CTAs of 256 threads then leave room on their SM for two CTAs of the finalize kernel (256 threads, 40 registers)
// while they drain; above 88 there is room for one, and 149 to 296 channels need two (bf16, 256 channels, 2 / 4 MB: 9.0 / 9.5 us
// with 102 registers, 8.0 / 8.7 so).
enum { kShiftRow0 = 0, kShiftRows = 1, kShiftRowsFirst = 2 };
// REST: there are elements behind the last whole vector.
template <typename T, int MAXT, int SHIFT, bool REST>
__global__ void __launch_bounds__(MAXT, 512 / MAXT)
batch_norm_sums_cl_ring_kernel(const BatchNormParams p, long long total, int PV, int tail) {
  wait_for_previous_kernel();
  constexpr int V = Elem<T>::V;
  extern __shared__ __align__(128) unsigned char smem[];
  float* red = reinterpret_cast<float*>(smem + (size_t)kRingBytesPerThread * MAXT);  // [MAXT * V]: the shifts
  const int tid = threadIdx.x, T_ = blockDim.x, C = p.channels;
  const int ph = tid % PV;
  const T* xe = reinterpret_cast<const T*>(p.x);
  const uint4* x = reinterpret_cast<const uint4*>(p.x);
  const uint32_t mine = smem_u32(smem) + (uint32_t)tid * 16u;
  const long long step = (long long)gridDim.x * kRingU * T_;
  long long v = (long long)blockIdx.x * kRingU * T_ + tid;
  T first[SHIFT == kShiftRowsFirst ? BN_SHIFT_ROWS : V];
  if constexpr (SHIFT == kShiftRowsFirst) {  // the launcher sees to C <= blockDim.x
    if (tid < C) bn_shift_load<T>(xe, tid, C, p.rows, first);
  } else if constexpr (SHIFT == kShiftRow0) {
    int c = ph * V % C;
#pragma unroll
    for (int i = 0; i < V; ++i) {
      first[i] = ld_here(xe + c);
      if (++c == C) c = 0;
    }
  }
#pragma unroll
  for (int s = 0; s < kRingS - 1; ++s) bn_ring_issue<false>(x, mine, s, v + s * step, total, T_);
  f32x2 shift[V / 2], s1[V / 2], s2[V / 2], t1[V / 2], t2[V / 2];
  f32x2 upper[V / 2];
#pragma unroll
  for (int i = 0; i < V / 2; ++i) shift[i] = s1[i] = s2[i] = t1[i] = t2[i] = upper[i] = splat2(0.f);
  if constexpr (SHIFT == kShiftRow0) {
#pragma unroll
    for (int i = 0; i < V / 2; ++i) shift[i] = pack2(Elem<T>::to_f32(first[2 * i]), Elem<T>::to_f32(first[2 * i + 1]));
  } else {
    // The shift of every channel (the finalize kernel forms the same value) is computed once per CTA into shared
    // memory, at most MAXT * V channels per round, and every thread picks up its V channels.
    for (int c0 = 0; c0 < C; c0 += MAXT * V) {
      if constexpr (SHIFT == kShiftRowsFirst) {
        if (tid < C) red[tid] = bn_shift_of<T>(first);
      } else {
        for (int c = c0 + tid; c < C && c < c0 + MAXT * V; c += T_) red[c - c0] = bn_shift_scalar<T>(xe, c, C, p.rows);
      }
      __syncthreads();
#pragma unroll
      for (int i = 0; i < V / 2; ++i) {
        const int ca = (ph * V + 2 * i) % C, cb = (ph * V + 2 * i + 1) % C;
        float lo, hi;
        unpack2(shift[i], lo, hi);
        if (ca >= c0 && ca < c0 + MAXT * V) lo = red[ca - c0];
        if (cb >= c0 && cb < c0 + MAXT * V) hi = red[cb - c0];
        shift[i] = pack2(lo, hi);
      }
      __syncthreads();
    }
  }
  // Additions of squares of 16-bit values are biased, in proportion to the length of the chain they
  // join: two stages' squares are summed by themselves, sixteen of those join one chain, the chains a third.
  int slot = 0, round = 0;
  for (; v < total; v += step) {
    bn_ring_issue<false>(x, mine, slot == 0 ? kRingS - 1 : slot - 1, v + (kRingS - 1) * step, total, T_);
    copy_async_wait<kRingS - 1>();
    const uint32_t src = mine + (uint32_t)(slot * kRingU * T_) * 16u;
#pragma unroll
    for (int u = 0; u < kRingU; ++u) {
      if (v + (long long)u * T_ < total) {
        f32x2 f[V / 2];
        Pairs<T>::unpack(lds128(src + (uint32_t)(u * T_) * 16u), f);
#pragma unroll
        for (int i = 0; i < V / 2; ++i) {
          const f32x2 d = sub2(f[i], shift[i]);
          t1[i] = add2(t1[i], d);
          t2[i] = fma2(d, d, t2[i]);
        }
      }
    }
    ++round;
    if ((round & 1) == 0) {
#pragma unroll
      for (int i = 0; i < V / 2; ++i) {
        s1[i] = add2(s1[i], t1[i]);
        s2[i] = add2(s2[i], t2[i]);
        t1[i] = t2[i] = splat2(0.f);
      }
    }
    if ((round & 31) == 0) {
#pragma unroll
      for (int i = 0; i < V / 2; ++i) {
        upper[i] = add2(upper[i], s2[i]);
        s2[i] = splat2(0.f);
      }
    }
    if (++slot == kRingS) slot = 0;
  }
  if (REST && blockIdx.x == 0 && tid == tail) {  // what is behind the last whole vector
    const int rest = (int)(p.rows * C - total * V);
    f32x2 f[V / 2];
    Pairs<T>::unpack(load_first<T>(xe + total * V, rest), f);
#pragma unroll
    for (int i = 0; i < V / 2; ++i) {
      float lo, hi;
      unpack2(sub2(f[i], shift[i]), lo, hi);
      const f32x2 d = pack2(2 * i < rest ? lo : 0.f, 2 * i + 1 < rest ? hi : 0.f);
      t1[i] = add2(t1[i], d);
      t2[i] = fma2(d, d, t2[i]);
    }
  }
  let_next_kernel_start();
  __syncthreads();  // every thread has read its ring: the memory is reused
  float* r1 = reinterpret_cast<float*>(smem);  // [2][MAXT][V], then [2][MAXT] fp64
  float* r2 = r1 + MAXT * V;
#pragma unroll
  for (int i = 0; i < V / 2; ++i) {
    unpack2(add2(s1[i], t1[i]), r1[tid * V + 2 * i], r1[tid * V + 2 * i + 1]);
    unpack2(add2(upper[i], add2(s2[i], t2[i])), r2[tid * V + 2 * i], r2[tid * V + 2 * i + 1]);
  }
  __syncthreads();
  float* row = p.partials + ((long long)blockIdx.x * 2) * C;
  bn_fold_channels<float, V>(r1, r2, reinterpret_cast<double*>(r2 + MAXT * V), C, row, row + C);
}

// Finalize: a CTA per channel, all partial rows of it in flight at once, fp64 in a fixed
// order. Everything but the partial rows (the shift) is requested before the sums are there. The sixteen
// values of the shift are added in the order of bn_shift_scalar: the same bits.
template <typename T>
__global__ void __launch_bounds__(256) batch_norm_finalize_ring_kernel(const BatchNormParams p, int splits, int rows_shift) {
  __shared__ double red[2][8];
  __shared__ float first_rows[BN_SHIFT_ROWS];
  const int c = blockIdx.x, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const T* x = reinterpret_cast<const T*>(p.x);
  if (tid < BN_SHIFT_ROWS) {
    const long long r = rows_shift ? (tid < p.rows ? tid : p.rows - 1) : 0;
    first_rows[tid] = Elem<T>::to_f32(ld_here(x + r * p.channels + c));
  }
  wait_for_previous_kernel();
  let_next_kernel_start();
  float old_mean = 0.f, old_var = 0.f;
  if (tid == 0 && p.running_mean) {
    old_mean = __ldcg(p.running_mean + c);
    old_var = __ldcg(p.running_var + c);
  }
  double s1 = 0.0, s2 = 0.0;
  for (int g0 = tid; g0 < splits; g0 += 4 * 256) {
    float a[4], b[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const int g = g0 + u * 256;
      a[u] = g < splits ? __ldcg(p.partials + ((long long)g * 2) * p.channels + c) : 0.f;
      b[u] = g < splits ? __ldcg(p.partials + ((long long)g * 2 + 1) * p.channels + c) : 0.f;
    }
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      s1 += (double)a[u];
      s2 += (double)b[u];
    }
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    s1 += __shfl_xor_sync(0xffffffffu, s1, o);
    s2 += __shfl_xor_sync(0xffffffffu, s2, o);
  }
  if (lane == 0) {
    red[0][warp] = s1;
    red[1][warp] = s2;
  }
  __syncthreads();
  if (tid == 0) {
    s1 = s2 = 0.0;
    for (int w = 0; w < 8; ++w) {
      s1 += red[0][w];
      s2 += red[1][w];
    }
    float shift = first_rows[0];
    if (rows_shift) {
      shift = 0.f;
      for (int r = 0; r < BN_SHIFT_ROWS; ++r) shift = __fadd_rn(shift, first_rows[r]);
      shift = bn_shift_of_sum(shift, first_rows[0]);
    }
    float mean, invstd;
    bn_channel_stats(p, c, s1, s2, shift, true, &mean, &invstd, old_mean, old_var);
    p.stats[c] = mean;
    p.stats[p.channels + c] = invstd;
  }
}

template <typename T, int MAXT, bool REST>
__global__ void __launch_bounds__(MAXT, 512 / MAXT) batch_norm_apply_cl_ring_kernel(const BatchNormParams p, long long total,
                                                                                    int PV, int rest) {
  constexpr int V = Elem<T>::V;
  extern __shared__ __align__(128) unsigned char smem[];
  const int tid = threadIdx.x, T_ = blockDim.x, C = p.channels;
  const int ph = tid % PV;
  const uint4* x = reinterpret_cast<const uint4*>(p.x);
  uint4* y = reinterpret_cast<uint4*>(p.y);
  const uint32_t mine = smem_u32(smem) + (uint32_t)tid * 16u;
  const long long chunk = (long long)kRingU * T_, step = (long long)gridDim.x * chunk;
  long long v = (total - 1) / chunk * chunk - (long long)blockIdx.x * chunk + tid;  // from the last chunk down
#pragma unroll
  for (int s = 0; s < kRingS - 1; ++s) bn_ring_issue<true>(x, mine, s, v - s * step, total, T_);
  f32x2 mean2[V / 2], inv2[V / 2], w2[V / 2], b2[V / 2];
#pragma unroll
  for (int i = 0; i < V / 2; ++i) {
    const int c0 = (ph * V + 2 * i) % C, c1 = (ph * V + 2 * i + 1) % C;
    w2[i] = p.weight ? pack2(load_param1(p.weight, p.w_dtype, c0), load_param1(p.weight, p.w_dtype, c1)) : splat2(1.f);
    b2[i] = p.bias ? pack2(load_param1(p.bias, p.w_dtype, c0), load_param1(p.bias, p.w_dtype, c1)) : splat2(0.f);
  }
  wait_for_previous_kernel();
  // through L1, as a CTA's threads read the same few lines 2 V times (past L1: bf16 [128, 96, 56, 56] 53.5 us,
  // so 42.3). They cannot be in L1 from before: the sums kernel started after their last use, the finalize
  // kernel only writes them.
#pragma unroll
  for (int i = 0; i < V / 2; ++i) {
    const int c0 = (ph * V + 2 * i) % C, c1 = (ph * V + 2 * i + 1) % C;
    mean2[i] = pack2(p.stats[c0], p.stats[c1]);
    inv2[i] = pack2(p.stats[C + c0], p.stats[C + c1]);
  }
  const bool relu = p.relu != 0;
  int slot = 0;
  for (; v >= 0; v -= step) {
    bn_ring_issue<true>(x, mine, slot == 0 ? kRingS - 1 : slot - 1, v - (kRingS - 1) * step, total, T_);
    copy_async_wait<kRingS - 1>();
    const uint32_t src = mine + (uint32_t)(slot * kRingU * T_) * 16u;
#pragma unroll
    for (int u = 0; u < kRingU; ++u) {
      const long long i = v + (long long)u * T_;
      if (i < total) {
        f32x2 f[V / 2];
        Pairs<T>::unpack(lds128(src + (uint32_t)(u * T_) * 16u), f);
#pragma unroll
        for (int k = 0; k < V / 2; ++k) f[k] = add2(mul2(mul2(sub2(f[k], mean2[k]), inv2[k]), w2[k]), b2[k]);
        uint4 packed = Pairs<T>::pack(f);
        if (relu) packed = relu_packed<T>(packed);
        st_stream(reinterpret_cast<T*>(y + i), packed);
      }
    }
    if (++slot == kRingS) slot = 0;
  }
  if (REST && blockIdx.x == 0 && tid < rest) bn_apply_one<T>(p, total * V + tid, (int)((total * V + tid) % C));
  copy_async_wait<0>();
}

// With row 0 alone the error of invstd depends on where that row lies: five standard deviations off the mean it is 1.5e-7
// instead of 2.9e-8 (rms, bf16), so row 0 is only for what cannot afford more. More than 32 vectors a thread (39 MB): the
// sixteen rows, asked for behind the copies (bf16 64 channels, 100 MB 46.9 us; in front of them 48.6). From 8 MB on, up to 256
// channels (at most one a thread): in front, where they cost nothing (64 channels, 12 / 18.5 / 30 MB: row 0 13.3 / 16.4 / 20.7, so
// 13.2 / 16.2 / 20.1, behind the copies 13.8 / 17.2 / 21.3; 256 channels 14.7 / 17.8 / 22.3 and 14.5 / 17.3 / 21.6). Below 8 MB they would
// cost 0.2 to 0.7 of 7 to 10 us, with 1024 channels of up to 39 MB 2.5 of 20.
static int bn_shift_kind(long long channels, long long vectors, long long all_threads) {
  if (vectors > 32 * all_threads) return kShiftRows;
  return channels <= 256 && vectors * 16 >= 8000000 ? kShiftRowsFirst : kShiftRow0;
}

// Returns false when the shape or the scratch does not fit (not one partial row), or the kernels above are faster (the
// caller takes them).
template <typename T>
static bool try_launch_batch_norm_cl_ring(BatchNormParams p, size_t scratch_bytes, cudaStream_t st, int* rc) {
  constexpr int V = Elem<T>::V;
  const DeviceInfo& dev = device_info();
  const long long C = p.channels;
  long long g = C, h = V;  // gcd(C, V)
  while (h) { const long long t = g % h; g = h; h = t; }
  const long long PV = C / g;
  const long long elems = p.rows * C;
  if (PV > 512 || elems < V) return false;
  // The flat kernels above need whole periods. (Where there are none, the strided kernels are faster for few rows, whose channels take a CTA
  // each and one load a thread: bf16, 401 channels, 147 rows 7.8 us strided, 10.2 so, 441 rows 9.9 and 9.9, 637 rows 11.3 and 10.2. But
  // their errors are up to six times as large, the mean's 8.3e-8 at 147 rows and 3.0e-8 so, 2.0e-7 and 4.8e-8 at 405 rows of 101 channels.)
  if (elems % (PV * V) == 0 && ring_is_slower(C, elems * (long long)sizeof(T))) return false;
  const long long total = elems / V;
  const long long stats_floats = 2 * C;
  const long long room = ((long long)scratch_bytes - 256) / (long long)sizeof(float) - stats_floats;
  if (room < 2 * C) return false;
  const long long most = room / (2 * C);  // partial rows that the scratch holds
  int threads = (int)(PV <= 256 ? 256 / PV * PV : PV);
  long long splits = (threads <= 256 ? 2LL : 1LL) * dev.sm_count;  // all CTAs resident
  // at least 8 vectors per thread: small tensors get few partial rows and a short finalize
  auto useful = [&](long long ctas) { return ctas * threads * 8 > total ? (total + threads * 8 - 1) / (threads * 8) : ctas; };
  splits = useful(splits);
  if (splits > most) {
    // No room for two partial rows per SM: one CTA per SM with the threads of both, and fewer of those when there is not even
    // room for that. bf16 64 channels, 148 rows, 10 / 30 / 100 MB: 12.3 / 19.9 / 48.6 us (CTAs of 256 threads 13.2 / 24.2 / 57.8, the flat
    // kernels on as few CTAs 19.5 / 39.6 / 109.6); 20 rows, 100 MB: 209 (288, 611).
    threads = (int)(512 / PV * PV);
    splits = useful(dev.sm_count);
    if (splits > most) splits = most;
  }
  p.stats = p.partials + splits * 2 * C;
  const int kind = bn_shift_kind(C, total, (long long)threads * splits);
  // The elements behind the last whole vector belong to the thread of CTA 0 that has the phase of the vector they begin.
  const int rest = (int)(elems % V), tail = rest ? (int)(total % threads) : -1;
  auto run = [&](auto maxt_tag, auto rest_tag) {
    constexpr int MAXT = decltype(maxt_tag)::value;
    constexpr bool REST = decltype(rest_tag)::value;
    auto sums = kind == kShiftRow0   ? batch_norm_sums_cl_ring_kernel<T, MAXT, kShiftRow0, REST>
                : kind == kShiftRows ? batch_norm_sums_cl_ring_kernel<T, MAXT, kShiftRows, REST>
                                     : batch_norm_sums_cl_ring_kernel<T, MAXT, kShiftRowsFirst, REST>;
    auto apply = batch_norm_apply_cl_ring_kernel<T, MAXT, REST>;
    const size_t ring = (size_t)kRingBytesPerThread * MAXT;  // 96 KB, or 192 KB: two CTAs, or one, per SM
    const size_t with_shifts = ring + (size_t)MAXT * V * sizeof(float);
    cudaError_t e = allow_dynamic_smem(reinterpret_cast<const void*>(sums), with_shifts);
    if (e == cudaSuccess)
      e = allow_dynamic_smem(reinterpret_cast<const void*>(apply), ring);
    // the finalize kernel uses next to no shared memory: asked to keep the split of its neighbours, it does
    // not make every SM drain and re-partition twice a call
    if (e == cudaSuccess)
      e = set_function_attribute_once(reinterpret_cast<const void*>(batch_norm_finalize_ring_kernel<T>),
                                      cudaFuncAttributePreferredSharedMemoryCarveout, cudaSharedmemCarveoutMaxShared);
    if (e != cudaSuccess) {
      cudaGetLastError();
      *rc = fail((int)e, "b200_batch_norm_fwd: cannot reserve %zu bytes of shared memory: %s", with_shifts, cudaGetErrorString(e));
      return;
    }
    launch_dependent(sums, (unsigned)splits, threads, with_shifts, st, p, total, (int)PV, tail);
    *rc = launch_status("b200_batch_norm_fwd sums [channels-last, flat vectors, copy rings]");
    if (*rc != B200_OK) return;
    launch_dependent(batch_norm_finalize_ring_kernel<T>, dim3((unsigned)p.channels), dim3(256), 0, st, p, (int)splits,
                     kind != kShiftRow0 ? 1 : 0);
    *rc = launch_status("b200_batch_norm_fwd finalize");
    if (*rc != B200_OK) return;
    launch_dependent(apply, dim3((unsigned)splits), dim3((unsigned)threads), ring, st, p, total, (int)PV, rest);
    *rc = launch_status("b200_batch_norm_fwd apply [channels-last, flat vectors, copy rings]");
  };
  using Narrow = std::integral_constant<int, 256>;
  using Wide = std::integral_constant<int, 512>;
  if (rest) threads <= 256 ? run(Narrow{}, std::true_type{}) : run(Wide{}, std::true_type{});
  else threads <= 256 ? run(Narrow{}, std::false_type{}) : run(Wide{}, std::false_type{});
  return true;
}

template <typename T>
static int launch_batch_norm(BatchNormParams p, bool channels_last, size_t scratch_bytes, cudaStream_t st) {
  const long long stats_floats = 2LL * p.channels;
  if (channels_last) {  // channel patterns of up to 512 vectors: the tensor as a flat array, three launches
    BatchNormParams q = p;
    q.rows = p.rows * p.spatial;
    int rc = B200_OK;
    if (try_launch_batch_norm_cl_ring<T>(q, scratch_bytes, st, &rc)) return rc;
    if (try_launch_batch_norm_cl_flat<T>(q, scratch_bytes, st, &rc)) return rc;
  }
  {  // contiguous NCHW: one launch, a cluster of CTAs per channel (batch_norm_nchw.cu)
    int rc = B200_OK;
    if (try_launch_batch_norm_nchw<T>(p, st, &rc)) return rc;
  }
  // general path
  const long long total = p.rows * p.spatial;
  long long splits = total / 16384;
  if (splits < 1) splits = 1;
  if (splits > 64) splits = 64;
  const long long need = 256 + (splits * 2 * p.channels + stats_floats) * (long long)sizeof(float);
  if ((long long)scratch_bytes < need)
    return fail(B200_ERR_WORKSPACE, "b200_batch_norm_fwd: scratch of %zu bytes, need %lld", scratch_bytes, need);
  p.stats = p.partials + splits * 2 * p.channels;
  launch_dependent(batch_norm_stats_general_kernel<T>, dim3(p.channels, (unsigned)splits), 256, 0, st, p);
  int rc = launch_status("b200_batch_norm_fwd stats [strided, element-wise]");
  if (rc != B200_OK) return rc;
  launch_dependent(batch_norm_finalize_general_kernel<T>, (p.channels + 7) / 8, 256, 0, st, p, (int)splits, 0);
  rc = launch_status("b200_batch_norm_fwd finalize");
  if (rc != B200_OK) return rc;
  launch_dependent(batch_norm_apply_general_kernel<T>, dim3(p.channels, (unsigned)splits), 256, 0, st, p);
  return launch_status("b200_batch_norm_fwd apply [strided, element-wise]");
}

}  // namespace b200

using namespace b200;

// Bounded waits that ran out since the library was loaded: none of these kernels has one.
extern "C" int64_t b200_batch_norm_wait_timeouts(void) { return 0; }

static int64_t batch_norm_scratch_for(int64_t rows, int64_t channels) {  // so many partial rows, and the statistics
  return 256 + (rows * 2 * channels + 2 * channels) * (int64_t)sizeof(float);
}

// What every path makes do with: a partial row per SM (or per split of the general path).
static int64_t batch_norm_least_scratch_bytes(int64_t channels) {
  const int sms = device_info().sm_count;
  return batch_norm_scratch_for(sms > 64 ? sms : 64, channels);
}

// What lets every path run its largest grid: the flat channels-last kernels take eight partial rows per SM
// (the copy rings two); their patterns of at most 512 vectors end at 4096 channels. With less scratch they
// run on fewer CTAs, which changes the order of the sums.
extern "C" int64_t b200_batch_norm_scratch_bytes(int64_t channels) {
  const int64_t rows = channels <= 4096 ? 8LL * device_info().sm_count : 0, least = batch_norm_least_scratch_bytes(channels);
  const int64_t largest = batch_norm_scratch_for(rows, channels);
  return largest > least ? largest : least;
}

// b200_batch_norm_fwd with the factor that turns the biased batch variance into the value blended
// into running_var given by the caller (unbiased_factor > 0) instead of n / (n - 1). A captured
// graph carries that factor as a literal of the shape it was captured at and applies it at every
// other shape point too; an oracle for such a graph has to do the same.
extern "C" int b200_batch_norm_fwd_ex(const void* x, void* y, const void* weight, const void* bias,
                                      float* running_mean, float* running_var, float* save_mean,
                                      float* save_invstd, int64_t batch, int64_t channels, int64_t spatial,
                                      int64_t stride_n, int64_t stride_c, int64_t stride_s,
                                      int32_t x_dtype, int32_t w_dtype, double eps, double momentum,
                                      double unbiased_factor, int32_t relu, void* scratch,
                                      int64_t scratch_bytes, void* stream) {
  if (!x || !y || !scratch) return fail(B200_ERR_INVALID, "b200_batch_norm_fwd: null argument");
  if (batch <= 0 || channels <= 0 || spatial <= 0 || channels > 0x7fffffffLL)
    return fail(B200_ERR_INVALID, "b200_batch_norm_fwd: bad sizes N=%lld C=%lld HW=%lld", (long long)batch,
                (long long)channels, (long long)spatial);
  if ((running_mean == nullptr) != (running_var == nullptr))
    return fail(B200_ERR_INVALID, "b200_batch_norm_fwd: running_mean and running_var come together");
  if (!aligned16(scratch)) return fail(B200_ERR_ALIGNMENT, "b200_batch_norm_fwd: scratch must be 16-byte aligned");

  BatchNormParams p;
  p.x = x; p.y = y; p.weight = weight; p.bias = bias;
  p.running_mean = running_mean; p.running_var = running_var;
  p.save_mean = save_mean; p.save_invstd = save_invstd;
  p.channels = (int)channels; p.spatial = spatial;
  p.sn = stride_n; p.sc = stride_c; p.ss = stride_s;
  p.w_dtype = w_dtype;
  p.eps = (float)eps; p.momentum = (float)momentum; p.one_minus_momentum = (float)(1.0 - momentum);
  const double count = (double)batch * (double)spatial;
  p.count = count;
  p.inv_count = 1.0 / count;
  p.unbias = unbiased_factor > 0.0 ? (float)unbiased_factor : (float)(count / (count - 1.0));
  p.relu = relu ? 1 : 0;
  p.partials = reinterpret_cast<float*>(reinterpret_cast<char*>(scratch) + 256);  // behind the words that the norm backward keeps at zero
  p.stats = nullptr;

  // channels-last: c is the unit-stride dimension, rows are (n, s) pairs with a uniform stride of C
  const bool cl = stride_c == 1 && stride_s == channels && stride_n == spatial * channels;
  const bool cl_vector = cl && aligned16(x) && aligned16(y);
  p.rows = batch;
  cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
  const LaunchesTogether together(st);
  switch (x_dtype) {
    case B200_F32: return launch_batch_norm<float>(p, cl_vector, (size_t)scratch_bytes, st);
    case B200_BF16: return launch_batch_norm<__nv_bfloat16>(p, cl_vector, (size_t)scratch_bytes, st);
    case B200_F16: return launch_batch_norm<__half>(p, cl_vector, (size_t)scratch_bytes, st);
  }
  return fail(B200_ERR_INVALID, "b200_batch_norm_fwd: unknown dtype %d", x_dtype);
}

extern "C" int b200_batch_norm_fwd(const void* x, void* y, const void* weight, const void* bias,
                                   float* running_mean, float* running_var, float* save_mean,
                                   float* save_invstd, int64_t batch, int64_t channels, int64_t spatial,
                                   int64_t stride_n, int64_t stride_c, int64_t stride_s,
                                   int32_t x_dtype, int32_t w_dtype, double eps, double momentum,
                                   int32_t relu, void* scratch, int64_t scratch_bytes, void* stream) {
  return b200_batch_norm_fwd_ex(x, y, weight, bias, running_mean, running_var, save_mean, save_invstd, batch,
                                channels, spatial, stride_n, stride_c, stride_s, x_dtype, w_dtype, eps, momentum,
                                0.0, relu, scratch, scratch_bytes, stream);
}

// ----------------------------------------------------------------------------------------------
// BatchNorm forward for callers that cannot hand over scratch memory.
//
// Some hosts of this library are not allowed to allocate device memory at all: a serving process
// whose framework carves one arena at start-up and forbids plug-ins to call cudaMalloc (the call
// would also synchronise the whole device in the middle of a request), or an embedding where the
// only device buffers the caller owns are the tensors it was given. b200_batch_norm_fwd needs a
// scratch buffer from its caller; this variant brings its own: a fixed array in the library's
// device image. Every GPU that loads the library holds those bytes until the process exits, which
// is why the size is capped (B200_BN_STATIC_MAX_CHANNELS channels, about 1.3 MB).
//
// The array's name is only meaningful in device code. On the host it is a stand-in symbol, not a
// device address, so the address is looked up once per device with cudaGetSymbolAddress - on the
// first call made while that device is current - and kept. That first call therefore does a little
// set-up work and should be made before any stream capture begins.
//
// All calls on a device share the one array and it keeps whatever the previous call left in it; partial
// sums and statistics are fully rewritten before they are read. Two calls that overlap on the GPU
// (different streams, no ordering between them) would race on the array: callers must order them.
// ----------------------------------------------------------------------------------------------
#define B200_BN_STATIC_MAX_CHANNELS 1024
#define B200_BN_STATIC_MAX_GROUPS 160  // partial rows at 1024 channels: one per CTA (<= SM count) or per split (<= 64)

namespace b200 {

constexpr size_t kBnStaticScratchBytes =
    256 + ((size_t)B200_BN_STATIC_MAX_GROUPS * 2 * B200_BN_STATIC_MAX_CHANNELS + 2 * B200_BN_STATIC_MAX_CHANNELS) *
              sizeof(float);

static __device__ __align__(256) unsigned char g_bn_static_scratch[kBnStaticScratchBytes];

// Device address of the array on the current device; looked up on first use per device.
static int bn_static_scratch_address(void** out) {
  static void* address[64] = {nullptr};
  static std::mutex mu;
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return fail((int)e, "b200_batch_norm_fwd_static_scratch: cudaGetDevice: %s", cudaGetErrorString(e));
  if (dev < 0 || dev >= 64) return fail(B200_ERR_UNSUPPORTED, "b200_batch_norm_fwd_static_scratch: device index %d", dev);
  std::lock_guard<std::mutex> lock(mu);
  if (address[dev] == nullptr) {
    void* ptr = nullptr;
    e = cudaGetSymbolAddress(&ptr, g_bn_static_scratch);  // `dev` is the current device
    if (e != cudaSuccess || ptr == nullptr) {
      cudaGetLastError();
      return fail(e != cudaSuccess ? (int)e : B200_ERR_INVALID,
                  "b200_batch_norm_fwd_static_scratch: cudaGetSymbolAddress failed: %s", cudaGetErrorString(e));
    }
    address[dev] = ptr;
  }
  *out = address[dev];
  return B200_OK;
}

}  // namespace b200

extern "C" int b200_batch_norm_fwd_static_scratch(const void* x, void* y, const void* weight, const void* bias,
                                                  float* running_mean, float* running_var, float* save_mean,
                                                  float* save_invstd, int64_t batch, int64_t channels,
                                                  int64_t spatial, int64_t stride_n, int64_t stride_c,
                                                  int64_t stride_s, int32_t x_dtype, int32_t w_dtype, double eps,
                                                  double momentum, int32_t relu, void* stream) {
  if (channels > B200_BN_STATIC_MAX_CHANNELS)
    return fail(B200_ERR_UNSUPPORTED,
                "b200_batch_norm_fwd_static_scratch: %lld channels exceed the built-in scratch (max %d); "
                "use b200_batch_norm_fwd with a caller-provided scratch buffer",
                (long long)channels, B200_BN_STATIC_MAX_CHANNELS);
  if (channels > 0 && batch_norm_least_scratch_bytes(channels) > (int64_t)kBnStaticScratchBytes)
    return fail(B200_ERR_UNSUPPORTED,
                "b200_batch_norm_fwd_static_scratch: this device needs %lld scratch bytes for %lld channels, "
                "the built-in array holds %zu",
                (long long)batch_norm_least_scratch_bytes(channels), (long long)channels, kBnStaticScratchBytes);
  void* scratch = nullptr;
  int rc = bn_static_scratch_address(&scratch);
  if (rc != B200_OK) return rc;
  return b200_batch_norm_fwd(x, y, weight, bias, running_mean, running_var, save_mean, save_invstd, batch,
                             channels, spatial, stride_n, stride_c, stride_s, x_dtype, w_dtype, eps, momentum,
                             relu, scratch, (int64_t)kBnStaticScratchBytes, stream);
}
