// LayerNorm / RMSNorm forward over the last dimension, and row-wise var_mean.
//
// Replaces the Triton kernels of the row-normalisation repros in the reference
// (repros/canonical/var_mean_f8ec553e339e/oracle.py:50-84, var_mean_af505388b035/oracle.py:11-40,
// var_mean_f7906a6c6957/oracle.py:14-50, mean_f667cd8901af/oracle.py:36-72).
//
// Evaluation order, as the decomposed aten graphs have it:
//   LayerNorm: mean = sum(x)/n; var = sum((x-mean)^2)/(n-correction); rstd = 1/sqrt(var+eps)
//              y = ((x - mean) * rstd) * w + b
//   RMSNorm  : ms = sum(x*x)/n; rstd = 1/sqrt(ms+eps); y = (x * rstd) * w
// The variance is the centred second pass over the row held in registers (squares accumulated with
// fused multiply-adds: aten's var_mean has no multiply/add sequence to mirror). Statistics are fp32.
// Any of y, mean, rstd, var may be null (var_mean alone = no y, no rstd).
#include "norm_fwd.cuh"
#include "tile_stream.cuh"

#include <cstdlib>
#include <type_traits>

namespace b200 {

template <typename Tin, typename Tout, int CH, int G, bool GELU, bool RES>
// Residual instantiations with sub-warp rows: three CTAs of 256 threads per SM (80 registers, a few
// spilled words) measured faster than two at 119 registers: 57.1 -> 45.8 us on [65536, 768] bf16
// under the reference's cold-L2 protocol.
// The GELU prologue is a template parameter: as a branch at run time its registers were the plain kernels'
// too (bf16, CTA per row of up to 1024 vectors 120, now 64; sub-warp rows of up to 128 vectors 138, now 54).
// RMSNorm bf16 [16384, 4096] 66.7 -> 44.2 us, [2048, 768] 5.0 -> 3.6; LayerNorm 83.5 -> 52.5 and 6.2 -> 4.5;
// GELU -> LayerNorm 112.5 -> 96.8 and 7.6 -> 5.6.
__global__ void __launch_bounds__(G == 0 ? 512 : 256, (RES && G != 0) ? 3 : 1)
norm_fwd_resident_kernel(const NormFwdParams p) {
  wait_for_previous_kernel();
  constexpr int V = Elem<Tin>::V;
  __shared__ float red[64];
  const int lane = glane<G>();
  const int gs = gsize<G>();
  long long row = grow<G>();
  const bool valid = row < p.rows;  // lanes of a partly filled last CTA recompute the last row
  if (!valid) row = p.rows - 1;

  const Tin* x = reinterpret_cast<const Tin*>(p.x) + row * p.x_row_stride;
  const int nv = p.n / V;

  uint4 raw[CH], rraw[RES ? CH : 1];
#pragma unroll
  for (int c = 0; c < CH; ++c) {
    const int j = c * gs + lane;
    if (j < nv) {
      raw[c] = ld_stream(x + (long long)j * V);
      if constexpr (RES)
        rraw[c] = ld_stream(reinterpret_cast<const Tin*>(p.res) + row * p.x_row_stride + (long long)j * V);
    }
  }
  // The row as packed fp32 pairs; slots past the end of the row hold zeros and add nothing.
  f32x2 v[CH][V / 2];
  constexpr bool DUAL = RES && sizeof(Tin) == 2;  // fp32 tensors: the rounded sum is the sum
  uint4 pr[DUAL ? CH : 1];                         // the rounded sums, packed, when both forms are asked for
  const bool both = DUAL && p.res_round == 2;
  f32x2 s2 = splat2(0.f);
#pragma unroll
  for (int c = 0; c < CH; ++c) {
    float f[V];
    if (c * gs + lane < nv) {
      Elem<Tin>::unpack(raw[c], f);
      if constexpr (RES) {  // x + res in fp32; sum_out receives it rounded to the tensor dtype
        float r[V];
        Elem<Tin>::unpack(rraw[c], r);
#pragma unroll
        for (int i = 0; i < V; ++i) f[i] = f[i] + r[i];
        const uint4 packed = Elem<Tin>::pack(f);
        if (p.sum_out && valid)
          st_stream(reinterpret_cast<Tin*>(p.sum_out) + row * (long long)p.n + (long long)(c * gs + lane) * V, packed);
        if constexpr (DUAL) pr[c] = packed;
        if (p.res_round == 1) {
#pragma unroll
          for (int i = 0; i < V; ++i) f[i] = round_through<Tin>(f[i]);
        }
      }
    } else {
#pragma unroll
      for (int i = 0; i < V; ++i) f[i] = 0.f;
      if constexpr (DUAL) pr[c] = make_uint4(0u, 0u, 0u, 0u);
    }
#pragma unroll
    for (int i = 0; i < V / 2; ++i) v[c][i] = pack2(f[2 * i], f[2 * i + 1]);
  }
  if constexpr (GELU) {  // gelu(0) = 0: the padding slots stay zero
#pragma unroll
    for (int c = 0; c < CH; ++c)
#pragma unroll
      for (int i = 0; i < V / 2; ++i) v[c][i] = gelu_erf_rounded2<Tin>(v[c][i]);
  }
  if (p.rms) {
#pragma unroll
    for (int c = 0; c < CH; ++c)
#pragma unroll
      for (int i = 0; i < V / 2; ++i) s2 = fma2(v[c][i], v[c][i], s2);
  } else {
#pragma unroll
    for (int c = 0; c < CH; ++c)
#pragma unroll
      for (int i = 0; i < V / 2; ++i) s2 = add2(s2, v[c][i]);
  }
  float sa, sb;
  unpack2(s2, sa, sb);
  float s = sa + sb, t = 0.f;  // t: the same sum over the rounded values (both forms)
  if constexpr (DUAL) {
    if (both) {
      f32x2 t2 = splat2(0.f);
#pragma unroll
      for (int c = 0; c < CH; ++c) {
        float fr[V];
        Elem<Tin>::unpack(pr[c], fr);  // zeros in the padding slots
#pragma unroll
        for (int i = 0; i < V / 2; ++i) t2 = add2(t2, pack2(fr[2 * i], fr[2 * i + 1]));
      }
      float ta, tb;
      unpack2(t2, ta, tb);
      t = ta + tb;
    }
  }
  if (both) greduce_sum2<G>(s, t, red);
  else s = greduce<SumOp, G>(s, red);
  const float mean_r = t * p.inv_n;

  float mean = 0.f, var, rstd, rstd_r = 0.f;
  if (p.rms) {
    var = s * p.inv_n;
    rstd = precise_rsqrt(var + p.eps);
  } else {
    mean = s * p.inv_n;
    const f32x2 mean2 = splat2(mean);
    f32x2 q2 = splat2(0.f);
#pragma unroll
    for (int c = 0; c < CH; ++c) {
      if (c * gs + lane < nv) {  // padding slots must not contribute (0 - mean)^2
#pragma unroll
        for (int i = 0; i < V / 2; ++i) {
          v[c][i] = sub2(v[c][i], mean2);  // keep the centred value: the output needs it again
          q2 = fma2(v[c][i], v[c][i], q2);
        }
      }
    }
    float qa, qb;
    unpack2(q2, qa, qb);
    float q = qa + qb, qr = 0.f;
    if constexpr (DUAL) {
      if (both) {
        const f32x2 mean_r2 = splat2(mean_r);
        f32x2 r2 = splat2(0.f);
#pragma unroll
        for (int c = 0; c < CH; ++c) {
          if (c * gs + lane < nv) {
            float fr[V];
            Elem<Tin>::unpack(pr[c], fr);
#pragma unroll
            for (int i = 0; i < V / 2; ++i) {
              const f32x2 d = sub2(pack2(fr[2 * i], fr[2 * i + 1]), mean_r2);
              r2 = fma2(d, d, r2);
            }
          }
        }
        float ra, rb;
        unpack2(r2, ra, rb);
        qr = ra + rb;
      }
    }
    if (both) greduce_sum2<G>(q, qr, red);
    else q = greduce<SumOp, G>(q, red);
    var = q * p.inv_denom;
    rstd = precise_rsqrt(var + p.eps);
    rstd_r = precise_rsqrt(qr * p.inv_denom + p.eps);  // LayerNorm only; the entry point rejects the rest
  }
  if (lane == 0 && valid) {
    if (p.mean_out) p.mean_out[row] = mean;
    if (p.rstd_out) p.rstd_out[row] = rstd;
    if (p.var_out) p.var_out[row] = var;
  }
  if (p.y == nullptr) return;

  Tout* y = reinterpret_cast<Tout*>(p.y) + row * p.y_row_stride;
  const f32x2 rstd2 = splat2(rstd);
  const f32x2 rstd_r2 = splat2(rstd_r), mean_r2 = splat2(mean_r);
#pragma unroll
  for (int c = 0; c < CH; ++c) {
    const int j = c * gs + lane;
    if (j < nv && valid) {
      f32x2 o[V / 2], orr[DUAL ? V / 2 : 1];
#pragma unroll
      for (int i = 0; i < V / 2; ++i) o[i] = mul2(v[c][i], rstd2);
      if constexpr (DUAL) {
        if (both) {
          float fr[V];
          Elem<Tin>::unpack(pr[c], fr);
#pragma unroll
          for (int i = 0; i < V / 2; ++i) orr[i] = mul2(sub2(pack2(fr[2 * i], fr[2 * i + 1]), mean_r2), rstd_r2);
        }
      }
      if (p.w) {
        float wf[V];
        load_param<V>(p.w, p.w_dtype, (long long)j * V, wf);
#pragma unroll
        for (int i = 0; i < V / 2; ++i) o[i] = mul2(o[i], pack2(wf[2 * i], wf[2 * i + 1]));
        if constexpr (DUAL) {
          if (both) {
#pragma unroll
            for (int i = 0; i < V / 2; ++i) orr[i] = mul2(orr[i], pack2(wf[2 * i], wf[2 * i + 1]));
          }
        }
      }
      if (p.b) {
        float bf[V];
        load_param<V>(p.b, p.w_dtype, (long long)j * V, bf);
#pragma unroll
        for (int i = 0; i < V / 2; ++i) o[i] = add2(o[i], pack2(bf[2 * i], bf[2 * i + 1]));
        if constexpr (DUAL) {
          if (both) {
#pragma unroll
            for (int i = 0; i < V / 2; ++i) orr[i] = add2(orr[i], pack2(bf[2 * i], bf[2 * i + 1]));
          }
        }
      }
      float of[V];
#pragma unroll
      for (int i = 0; i < V / 2; ++i) unpack2(o[i], of[2 * i], of[2 * i + 1]);
      if constexpr (DUAL) {
        if (both) {
#pragma unroll
          for (int i = 0; i < V / 2; ++i) {
            float ra, rb;
            unpack2(orr[i], ra, rb);
            if (!(fabsf(round_through<Tout>(of[2 * i])) > 3.0f)) of[2 * i] = ra;
            if (!(fabsf(round_through<Tout>(of[2 * i + 1])) > 3.0f)) of[2 * i + 1] = rb;
          }
        }
      }
      store_converted<Tout, V>(y + (long long)j * V, of);
    }
  }
}

// ----------------------------------------------------------------------------------------------
// Streaming variant for many short rows: a persistent CTA pulls tiles of R = blockDim/G rows into
// a ring of shared-memory stages with bulk asynchronous copies (S-1 tiles in flight per CTA,
// independent of register use), groups of G lanes normalise one row each from shared memory, and
// weight and bias are converted to fp32 once per CTA and kept in shared memory. One CTA barrier
// per tile: it makes the bounded-wait outcome CTA-uniform and, at the same time, proves that the
// previous tile's stage is free to be refilled.
// ----------------------------------------------------------------------------------------------
template <typename Tin, typename Tout, int CH, int G, bool EXACT, bool GELU>
__global__ void __launch_bounds__(256, 4)
norm_fwd_stream_kernel(const NormFwdParams p, const int stages, const int contiguous) {
  wait_for_previous_kernel();
  constexpr int V = Elem<Tin>::V;
  constexpr int PLANES = V / 4;  // fp32 copies of weight/bias are stored as planes of float4
  extern __shared__ __align__(128) unsigned char smem[];
  const int nv = p.n / V;
  const uint32_t row_bytes = (uint32_t)nv * 16u;
  const int R = blockDim.x / G;
  const uint32_t tile_bytes = (uint32_t)R * row_bytes;
  float* wsm = reinterpret_cast<float*>(smem + (size_t)stages * tile_bytes);
  float* bsm = wsm + (size_t)nv * V;
  uint64_t* full = reinterpret_cast<uint64_t*>(bsm + (size_t)nv * V);

  const int lane = threadIdx.x & (G - 1);
  const int grp = threadIdx.x / G;
  const long long num_tiles = (p.rows + R - 1) / R;
  const long long my_tiles =
      num_tiles > blockIdx.x ? (num_tiles - blockIdx.x + gridDim.x - 1) / gridDim.x : 0;
  const Tin* xg = reinterpret_cast<const Tin*>(p.x);

  // Thread 0 only: start the copy of this CTA's k-th tile into stage `slot` (= k mod stages,
  // tracked incrementally: a modulo per tile would cost more than the tile's arithmetic).
  const int rows_i = (int)p.rows;  // the launcher admits fewer than 2^31 rows
  const int num_tiles_i = (int)num_tiles, my_tiles_i = (int)my_tiles;
  auto issue = [&](int k, int slot) {
    const long long r0 = ((long long)blockIdx.x + (long long)k * gridDim.x) * R;
    const long long left = p.rows - r0;
    const uint32_t rows_here = (uint32_t)(left < R ? left : R);
    uint64_t* bar = &full[slot];
    unsigned char* dst = smem + (size_t)slot * tile_bytes;
    mbar_arrive_expect_tx(bar, rows_here * row_bytes);
    if (contiguous) {
      bulk_load(dst, xg + r0 * p.x_row_stride, rows_here * row_bytes, bar);
    } else {
      for (uint32_t r = 0; r < rows_here; ++r)
        bulk_load(dst + (size_t)r * row_bytes, xg + (r0 + r) * p.x_row_stride, row_bytes, bar);
    }
  };
  (void)num_tiles_i;
  // Thread 0 sets up the stage barriers and starts the first copies at once, before the CTA
  // converts weight and bias: HBM traffic begins with the CTA instead of after its prologue. (The
  // other threads first touch a barrier after the __syncthreads below.)
  float wf[V], bf[V];
  auto fetch_params = [&](int j) {
    if (p.w && j < nv) load_param<V>(p.w, p.w_dtype, (long long)j * V, wf);
    if (p.b && j < nv) load_param<V>(p.b, p.w_dtype, (long long)j * V, bf);
  };
  // Weight and bias are asked for first: behind the first copies of all CTAs (30 MB) they took 4 us to arrive, and no
  // row is worked on before they are there.
  fetch_params(threadIdx.x);
  // What has been issued follows from the tile at hand: max(k - 1, 0) + stages tiles before tile k. (Thread 0's counters of it cost every
  // thread eight registers: 32768 rows, LayerNorm bf16 640 columns 20.1 -> 19.3 us, behind GELU 768 32.6 -> 31.7 and f32 1024 57.5 -> 54.0;
  // slower only RMSNorm f32 640, 29.6 -> 30.1.)
  if (threadIdx.x == 0) {
    for (int s = 0; s < stages; ++s) mbar_init(&full[s], 1);
    mbar_init_fence();
    for (int k = 0; k < my_tiles_i && k < stages; ++k) issue(k, k);
  }

  for (int j = threadIdx.x; j < nv; j += blockDim.x) {
    if (j != threadIdx.x) fetch_params(j);
#pragma unroll
    for (int q = 0; q < PLANES; ++q) {
      const size_t at = ((size_t)q * nv + j) * 4;
      if (p.w) *reinterpret_cast<float4*>(wsm + at) = make_float4(wf[4 * q], wf[4 * q + 1], wf[4 * q + 2], wf[4 * q + 3]);
      if (p.b) *reinterpret_cast<float4*>(bsm + at) = make_float4(bf[4 * q], bf[4 * q + 1], bf[4 * q + 2], bf[4 * q + 3]);
    }
  }
  __syncthreads();

  // Everything a tile needs that does not change from tile to tile is set up here, as 32-bit
  // shared-memory addresses and one running output pointer: the per-tile code is then loads at
  // [register + constant], arithmetic and stores.
  const uint32_t x_lane = smem_u32(smem) + (uint32_t)grp * row_bytes + (uint32_t)lane * 16u;
  uint32_t w_lane[PLANES], b_lane[PLANES];
#pragma unroll
  for (int q = 0; q < PLANES; ++q) {
    w_lane[q] = smem_u32(wsm) + ((uint32_t)q * nv + lane) * 16u;
    b_lane[q] = smem_u32(bsm) + ((uint32_t)q * nv + lane) * 16u;
  }
  const bool has_w = p.w != nullptr, has_b = p.b != nullptr, has_y = p.y != nullptr, rms = p.rms != 0;
  const int row_step = (int)gridDim.x * R;
  int row = (int)blockIdx.x * R + grp;
  Tout* yrow = reinterpret_cast<Tout*>(p.y) + (long long)row * p.y_row_stride + (long long)lane * V;
  const long long y_step = (long long)row_step * p.y_row_stride;

  int st = 0;           // stage of tile k
  uint32_t phase = 0;   // parity of that stage's current use
  uint32_t x_stage = x_lane;
  for (int k = 0; k < my_tiles_i; ++k, row += row_step, yrow += y_step) {
    const bool arrived = mbar_wait(&full[st], phase);
    if (!__syncthreads_and(arrived)) {
      // A copy did not complete within the bound: stop streaming. Thread 0 waits (bounded) for
      // whatever it still has in flight so that nothing lands in shared memory after the exit.
      if (threadIdx.x == 0) {
        note_wait_timeout();
        int ds = st;
        uint32_t dp = phase;
        for (int d = k; d < my_tiles_i && d < (k > 0 ? k - 1 : 0) + stages; ++d) {
          mbar_wait(&full[ds], dp);
          if (++ds == stages) { ds = 0; dp ^= 1u; }
        }
      }
      return;
    }
    // Everyone has passed the barrier, so everyone is done with tile k-1: refill its stage.
    if (threadIdx.x == 0 && k >= 1 && k - 1 + stages < my_tiles_i) {
      fence_proxy_async_smem();
      issue(k - 1 + stages, st == 0 ? stages - 1 : st - 1);
    }
    const bool valid = row < rows_i;

    f32x2 v[CH][V / 2];
#pragma unroll
    for (int c = 0; c < CH; ++c) {
      if (EXACT || c * G + lane < nv) {
        Pairs<Tin>::unpack(lds128(x_stage + (uint32_t)(c * G * 16)), v[c]);
      } else {
#pragma unroll
        for (int i = 0; i < V / 2; ++i) v[c][i] = splat2(0.f);
      }
    }
    if constexpr (GELU) {  // gelu(0) = 0: the padding slots stay zero
#pragma unroll
      for (int c = 0; c < CH; ++c)
#pragma unroll
        for (int i = 0; i < V / 2; ++i) v[c][i] = gelu_erf_rounded2<Tin>(v[c][i]);
    }
    // one short chain per slot, combined afterwards: a single chain over the whole row would
    // serialise on the add latency
    f32x2 part[CH];
    if (rms) {
#pragma unroll
      for (int c = 0; c < CH; ++c) {
        part[c] = mul2(v[c][0], v[c][0]);
#pragma unroll
        for (int i = 1; i < V / 2; ++i) part[c] = fma2(v[c][i], v[c][i], part[c]);
      }
    } else {
#pragma unroll
      for (int c = 0; c < CH; ++c) {
        part[c] = v[c][0];
#pragma unroll
        for (int i = 1; i < V / 2; ++i) part[c] = add2(part[c], v[c][i]);
      }
    }
    f32x2 s2 = part[0];
#pragma unroll
    for (int c = 1; c < CH; ++c) s2 = add2(s2, part[c]);
    const float s = greduce<SumOp, G>(hsum2(s2), nullptr);

    float mean = 0.f, var, rstd;
    if (rms) {
      var = s * p.inv_n;
      rstd = precise_rsqrt(var + p.eps);
    } else {
      mean = s * p.inv_n;
      const f32x2 mean2 = splat2(mean);
#pragma unroll
      for (int c = 0; c < CH; ++c) {
        part[c] = splat2(0.f);
        if (EXACT || c * G + lane < nv) {
#pragma unroll
          for (int i = 0; i < V / 2; ++i) {
            v[c][i] = sub2(v[c][i], mean2);
            part[c] = fma2(v[c][i], v[c][i], part[c]);
          }
        }
      }
      f32x2 q2 = part[0];
#pragma unroll
      for (int c = 1; c < CH; ++c) q2 = add2(q2, part[c]);
      const float q = greduce<SumOp, G>(hsum2(q2), nullptr);
      var = q * p.inv_denom;
      rstd = precise_rsqrt(var + p.eps);
    }
    if (lane == 0 && valid) {
      if (p.mean_out) p.mean_out[row] = mean;
      if (p.rstd_out) p.rstd_out[row] = rstd;
      if (p.var_out) p.var_out[row] = var;
    }
    if (has_y && valid) {
      const f32x2 rstd2 = splat2(rstd);
#pragma unroll
      for (int c = 0; c < CH; ++c) {
        if (EXACT || c * G + lane < nv) {
          f32x2 o[V / 2];
#pragma unroll
          for (int i = 0; i < V / 2; ++i) o[i] = mul2(v[c][i], rstd2);
          if (has_w) {
#pragma unroll
            for (int q = 0; q < PLANES; ++q) {
              f32x2 w2[2];
              Pairs<float>::unpack(lds128(w_lane[q] + (uint32_t)(c * G * 16)), w2);
              o[2 * q] = mul2(o[2 * q], w2[0]);
              o[2 * q + 1] = mul2(o[2 * q + 1], w2[1]);
            }
          }
          if (has_b) {
#pragma unroll
            for (int q = 0; q < PLANES; ++q) {
              f32x2 b2[2];
              Pairs<float>::unpack(lds128(b_lane[q] + (uint32_t)(c * G * 16)), b2);
              o[2 * q] = add2(o[2 * q], b2[0]);
              o[2 * q + 1] = add2(o[2 * q + 1], b2[1]);
            }
          }
          store_pairs<Tout, V>(yrow + c * G * V, o);
        }
      }
    }
    x_stage += tile_bytes;
    if (++st == stages) {
      st = 0;
      phase ^= 1u;
      x_stage = x_lane;
    }
  }
}

// Geometry of the streaming kernel: lanes per row and register slots per lane for nv vectors.
// At most 32 elements per thread, so that the kernel fits in 64 registers and four 256-thread CTAs
// (32 warps) share an SM: with fewer warps the per-row dependency chains (two shuffle reductions)
// leave the schedulers idle.
// `wide` (fp32 inputs: two register pairs per vector instead of four) allows up to eight vectors per lane.
static bool pick_stream_geometry(long long nv, bool wide, int* g, int* ch) {
  if (nv <= 8) { *g = 8; *ch = 1; return true; }
  if (nv <= 16) { *g = 8; *ch = 2; return true; }
  if (nv <= 24) { *g = 8; *ch = 3; return true; }
  if (nv <= 32) { *g = 8; *ch = 4; return true; }
  if (nv <= 48) { *g = 16; *ch = 3; return true; }
  if (nv <= 64) { *g = 16; *ch = 4; return true; }
  if (nv <= 96) { *g = 32; *ch = 3; return true; }
  if (nv <= 128) { *g = 32; *ch = 4; return true; }
  if (wide && nv <= 192) { *g = 32; *ch = 6; return true; }
  if (wide && nv <= 256) { *g = 32; *ch = 8; return true; }
  return false;
}

static bool streaming_disabled() {
  static const bool off = [] {
    const char* e = getenv("B200_DISABLE_STREAMING");
    return e && e[0] == '1';
  }();
  return off;
}

template <typename Tin, typename Tout>
static bool try_launch_norm_fwd_stream(const NormFwdParams& p, cudaStream_t st, int* rc) {
  constexpr int V = Elem<Tin>::V;
  const long long nv = p.n / V;
  int g, ch;
  if (streaming_disabled() || !pick_stream_geometry(nv, V == 4, &g, &ch)) return false;
  if (p.rows > 0x7ffff000LL) return false;  // the kernel counts rows and tiles in 32 bits
  const long long total_bytes = p.rows * nv * 16;
  if (total_bytes < (8ll << 20)) return false;  // small problems: the resident kernel is fine
  const DeviceInfo& dev = device_info();
  static const int threads_env = [] { const char* e = getenv("B200_NF_THREADS"); return e ? atoi(e) : 0; }();
  // 128 threads: eight small CTAs per SM keep each other busy across the per-tile barrier better than
  // four of 256 (measured on the 32768 x 768 bf16 case: 18.3 us against 19.7 us)
  const int threads = threads_env ? threads_env : 128;
  const int R = threads / g;
  const size_t tile_bytes = (size_t)R * nv * 16;
  const size_t fixed = 2 * (size_t)nv * V * sizeof(float) + 8 * sizeof(uint64_t);
  // as many CTAs per SM as 1024 threads allow, fewer when two stages of long rows need the room
  int ctas_per_sm = 1024 / threads;
  const size_t usable = (size_t)dev.max_smem_optin;
  while (ctas_per_sm > 2 && (usable - 1024 * (size_t)ctas_per_sm) / (size_t)ctas_per_sm < fixed + 2 * tile_bytes)
    --ctas_per_sm;
  const size_t per_cta = (usable - 1024 * (size_t)ctas_per_sm) / (size_t)ctas_per_sm;
  if (fixed + 2 * tile_bytes > per_cta) return false;
  int stages = (int)((per_cta - fixed) / tile_bytes);
  if (stages > 8) stages = 8;
  const size_t smem = (size_t)stages * tile_bytes + fixed;
  const long long num_tiles = (p.rows + R - 1) / R;
  long long grid = (long long)ctas_per_sm * dev.sm_count;
  if (grid > num_tiles) grid = num_tiles;
  const int contiguous = p.x_row_stride == p.n ? 1 : 0;
  const bool exact = nv == (long long)g * ch;

  auto launch = [&](auto kernel) {
    cudaError_t e = allow_dynamic_smem(reinterpret_cast<const void*>(kernel), smem);
    if (e != cudaSuccess) {
      cudaGetLastError();
      *rc = fail((int)e, "b200_norm_fwd: cannot reserve %zu bytes of shared memory: %s", smem, cudaGetErrorString(e));
      return;
    }
    launch_dependent(kernel, (unsigned)grid, threads, smem, st, p, stages, contiguous);
    *rc = launch_status("b200_norm_fwd [streaming ring, sub-warp rows]");
  };
#define B200_NFS(GG, CC)                                                                  \
  if (g == GG && ch == CC) {                                                              \
    if (p.prologue) {                                                                     \
      if (exact) launch(norm_fwd_stream_kernel<Tin, Tout, CC, GG, true, true>);           \
      else launch(norm_fwd_stream_kernel<Tin, Tout, CC, GG, false, true>);                \
    } else {                                                                              \
      if (exact) launch(norm_fwd_stream_kernel<Tin, Tout, CC, GG, true, false>);          \
      else launch(norm_fwd_stream_kernel<Tin, Tout, CC, GG, false, false>);               \
    }                                                                                     \
    return true;                                                                          \
  }
  B200_NFS(8, 1) B200_NFS(8, 2) B200_NFS(8, 3) B200_NFS(8, 4) B200_NFS(16, 3) B200_NFS(16, 4) B200_NFS(32, 3) B200_NFS(32, 4)
  if constexpr (V == 4) {
    B200_NFS(32, 6) B200_NFS(32, 8)
  }
#undef B200_NFS
  return false;
}

// ----------------------------------------------------------------------------------------------
// Residual add -> LayerNorm, rows of 65..128 vectors: a warp per row, every warp with its own ring of
// copy stages (a row of x and a row of the residual, brought in by two bulk copies that lane 0 issues),
// no CTA barrier in the row loop. The stage is refilled as soon as the sums are in registers, so two
// stages keep a row in flight per warp. Weight and bias are converted to fp32 once per CTA, in a
// [slot][pair][lane] layout that a warp reads without bank conflicts. BOTH (res_round == 2): the choice
// between the two forms is made on the packed 16-bit results: round both, compare |full| > 3, select.
// Which rows take it does not depend on the form, so that an element of the both-forms result has the bits of the
// form it was taken from (residual_warp_rows below).
// What bounds it: HBM, with about 38 instructions per pair of elements (two complete normalisations and
// the roundings between them, 57 % of the issue slots) behind it. The resident kernel converts weight
// and bias in every row on top and overlaps its load and store phases less; it keeps the rows of up to
// 64 vectors, of which it puts two into a warp (f16 [46251, 448]: 34.9 us there, 36.9 us here). Measured on bf16
// [65536, 768] with the sum kept: 82.5 -> 76.8 us back to back (64 us, 6.25 TB/s, from a clean L2).
// ----------------------------------------------------------------------------------------------
constexpr int kResWarps = 8;  // warps per CTA

template <typename T, int CH, bool EXACT, bool BOTH>
__global__ void __launch_bounds__(kResWarps * 32, 3)
residual_norm_warp_kernel(const NormFwdParams p, const int stages) {
  wait_for_previous_kernel();
  constexpr int V = Elem<T>::V;
  constexpr int P = V / 2;
  extern __shared__ __align__(128) unsigned char smem[];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int nv = p.n / V;
  const uint32_t row_bytes = (uint32_t)nv * 16u, stage_bytes = 2u * row_bytes;
  // layout: [kResWarps][stages][x row | residual row] | mbarriers [kResWarps][4] | weight, bias [CH][P][32] fp32 pairs
  unsigned char* ring = smem + (size_t)warp * stages * stage_bytes;
  unsigned char* behind = smem + (size_t)kResWarps * stages * stage_bytes;
  uint64_t* full = reinterpret_cast<uint64_t*>(behind) + warp * 4;
  f32x2* wsm = reinterpret_cast<f32x2*>(behind + kResWarps * 4 * sizeof(uint64_t));
  f32x2* bsm = wsm + CH * P * 32;
  const int rows = (int)p.rows;  // the launcher admits fewer than 2^31 rows
  const int gwarp = (int)blockIdx.x * kResWarps + warp, gstep = (int)gridDim.x * kResWarps;
  const int my_rows = rows > gwarp ? (rows - gwarp + gstep - 1) / gstep : 0;
  const T* xg = reinterpret_cast<const T*>(p.x);
  const T* rg = reinterpret_cast<const T*>(p.res);
  auto issue = [&](int k, int slot) {  // lane 0 only
    const long long off = ((long long)gwarp + (long long)k * gstep) * p.x_row_stride;
    unsigned char* dst = ring + (size_t)slot * stage_bytes;
    mbar_arrive_expect_tx(&full[slot], stage_bytes);
    bulk_load(dst, xg + off, row_bytes, &full[slot]);
    bulk_load(dst + row_bytes, rg + off, row_bytes, &full[slot]);
  };
  if (lane == 0) {  // the first rows are on their way before the weights are staged
    for (int s = 0; s < stages; ++s) mbar_init(&full[s], 1);
    mbar_init_fence();
    for (int k = 0; k < my_rows && k < stages; ++k) issue(k, k);
  }
  for (int q = threadIdx.x; q < CH * 32; q += blockDim.x) {  // q = slot * 32 + lane: vector q of the row
    float wf[V], bf[V];
#pragma unroll
    for (int i = 0; i < V; ++i) {
      wf[i] = 1.f;
      bf[i] = 0.f;
    }
    if (q < nv && p.w) load_param<V>(p.w, p.w_dtype, (long long)q * V, wf);
    if (q < nv && p.b) load_param<V>(p.b, p.w_dtype, (long long)q * V, bf);
#pragma unroll
    for (int i = 0; i < P; ++i) {
      wsm[((q >> 5) * P + i) * 32 + (q & 31)] = pack2(wf[2 * i], wf[2 * i + 1]);
      bsm[((q >> 5) * P + i) * 32 + (q & 31)] = pack2(bf[2 * i], bf[2 * i + 1]);
    }
  }
  __syncthreads();  // barriers initialised (seen by every lane), weights in place

  const uint32_t ring_addr = smem_u32(ring) + (uint32_t)lane * 16u;
  const f32x2* w_lane = wsm + lane;
  const f32x2* b_lane = bsm + lane;
  int slot = 0;
  uint32_t phase = 0;
  long long row = gwarp;
  for (int k = 0; k < my_rows; ++k, row += gstep) {
    const bool arrived = __all_sync(0xffffffffu, mbar_wait(&full[slot], phase));
    if (!arrived) {  // stop; none of this warp's copies may be in flight at exit
      if (lane == 0) {
        note_wait_timeout();
        int ds = slot;
        uint32_t dp = phase;
        for (int d = k; d < my_rows && d < k + stages; ++d) {
          mbar_wait(&full[ds], dp);
          if (++ds == stages) { ds = 0; dp ^= 1u; }
        }
      }
      return;
    }
    const uint32_t sx = ring_addr + (uint32_t)slot * stage_bytes, sr = sx + row_bytes;
    f32x2 v[CH][P];
    uint4 pr[BOTH ? CH : 1];  // the rounded sums
    f32x2 s2 = splat2(0.f), t2 = splat2(0.f);
    T* so = p.sum_out ? reinterpret_cast<T*>(p.sum_out) + row * (long long)p.n + lane * V : nullptr;
#pragma unroll
    for (int c = 0; c < CH; ++c) {
      if (EXACT || c * 32 + lane < nv) {
        f32x2 r[P];
        Pairs<T>::unpack(lds128(sx + c * 512), v[c]);
        Pairs<T>::unpack(lds128(sr + c * 512), r);
#pragma unroll
        for (int i = 0; i < P; ++i) v[c][i] = add2(v[c][i], r[i]);
        const uint4 packed = Pairs<T>::pack(v[c]);
        if (so) st_stream(so + c * 32 * V, packed);
        if constexpr (BOTH) {
          pr[c] = packed;
          Pairs<T>::unpack(packed, r);
#pragma unroll
          for (int i = 0; i < P; ++i) t2 = add2(t2, r[i]);
        } else if (p.res_round == 1) {
          Pairs<T>::unpack(packed, v[c]);
        }
#pragma unroll
        for (int i = 0; i < P; ++i) s2 = add2(s2, v[c][i]);
      } else {
#pragma unroll
        for (int i = 0; i < P; ++i) v[c][i] = splat2(0.f);
        if constexpr (BOTH) pr[c] = make_uint4(0u, 0u, 0u, 0u);
      }
    }
    __syncwarp();  // every lane has read the stage
    if (lane == 0 && k + stages < my_rows) {
      fence_proxy_async_smem();
      issue(k + stages, slot);
    }
    if (++slot == stages) {
      slot = 0;
      phase ^= 1u;
    }
    float s = hsum2(s2), t = hsum2(t2);
    greduce_sum2<32>(s, t, nullptr);
    const float mean = s * p.inv_n, mean_r = t * p.inv_n;
    const f32x2 mean2 = splat2(mean), mean_r2 = splat2(mean_r);
    f32x2 q2 = splat2(0.f), u2 = splat2(0.f);
#pragma unroll
    for (int c = 0; c < CH; ++c) {
      if (EXACT || c * 32 + lane < nv) {
#pragma unroll
        for (int i = 0; i < P; ++i) {
          v[c][i] = sub2(v[c][i], mean2);  // the centred value: the output needs it again
          q2 = fma2(v[c][i], v[c][i], q2);
        }
        if constexpr (BOTH) {
          f32x2 r[P];
          Pairs<T>::unpack(pr[c], r);
#pragma unroll
          for (int i = 0; i < P; ++i) {
            r[i] = sub2(r[i], mean_r2);
            u2 = fma2(r[i], r[i], u2);
          }
        }
      }
    }
    float q = hsum2(q2), u = hsum2(u2);
    greduce_sum2<32>(q, u, nullptr);
    const float var = q * p.inv_denom;
    const float rstd = precise_rsqrt(var + p.eps), rstd_r = precise_rsqrt(u * p.inv_denom + p.eps);
    if (lane == 0) {
      if (p.mean_out) p.mean_out[row] = mean;
      if (p.rstd_out) p.rstd_out[row] = rstd;
      if (p.var_out) p.var_out[row] = var;
    }
    const f32x2 rstd2 = splat2(rstd), rstd_r2 = splat2(rstd_r);
    T* y = reinterpret_cast<T*>(p.y) + row * p.y_row_stride + lane * V;
#pragma unroll
    for (int c = 0; c < CH; ++c) {
      if (EXACT || c * 32 + lane < nv) {
        f32x2 o[P];
#pragma unroll
        for (int i = 0; i < P; ++i)
          o[i] = add2(mul2(mul2(v[c][i], rstd2), w_lane[(c * P + i) * 32]), b_lane[(c * P + i) * 32]);
        if constexpr (BOTH) {
          f32x2 r[P];
          uint32_t out[P];
          Pairs<T>::unpack(pr[c], r);
#pragma unroll
          for (int i = 0; i < P; ++i) {
            r[i] = add2(mul2(mul2(sub2(r[i], mean_r2), rstd_r2), w_lane[(c * P + i) * 32]), b_lane[(c * P + i) * 32]);
            const uint32_t full16 = Pairs<T>::narrow(o[i]), round16 = Pairs<T>::narrow(r[i]);
            const uint32_t pick = beyond_three<T>(full16);
            out[i] = (full16 & pick) | (round16 & ~pick);
          }
          st_stream(y + c * 32 * V, make_uint4(out[0], out[1], out[2], out[3]));
        } else {
          st_stream(y + c * 32 * V, Pairs<T>::pack(o));
        }
      }
    }
  }
}

// Measured against the resident kernel (sum kept; fp32-sum form / both forms). 16-bit rows of up to 112 vectors: ahead
// ([40000, 768] 44.7 / 51.6 -> 44.5 / 45.6 us, [2000, 520] 5.3 / 5.8 -> 5.1 / 5.7, [16000, 864] 23.8 / 27.1 -> 21.1 /
// 24.2), but for one form of the widest large ones ([40000, 896] 51.0 / 59.5 -> 53.0 / 52.5). 113..128 vectors: ahead up
// to 32 MB of x ([16000, 1024] 24.9 / 27.9 -> 24.4 / 25.9), behind from there ([40000, 1024] 53.5 / 60.8 -> 59.3 / 62.7).
// fp32 rows: ahead with no more than a row per warp of one CTA per SM ([1000, 512] 4.9 -> 4.4, [1500, 512] 5.3 -> 5.5,
// [40000, 512] 52.3 -> 58.1).
template <typename T>
static bool residual_warp_rows(long long rows, long long nv) {
  if (sizeof(T) == 4) return rows <= 8LL * device_info().sm_count;
  return nv <= 112 || rows * nv * 16 <= (32 << 20);
}

// Returns false when the shape does not fit (the caller takes the resident kernel).
template <typename T>
static bool try_launch_residual_norm_warp(const NormFwdParams& p, cudaStream_t st, int* rc) {
  constexpr int V = Elem<T>::V;
  const long long nv = p.n / V;
  if (streaming_disabled() || p.rms || p.prologue || !p.y || nv <= 64 || nv > 128 || p.rows >= 0x7fffffffLL ||
      !residual_warp_rows<T>(p.rows, nv)) return false;
  const DeviceInfo& dev = device_info();
  const int ch = (int)((nv + 31) / 32);
  const size_t stage_bytes = 2 * (size_t)nv * 16;
  const size_t fixed = kResWarps * 4 * sizeof(uint64_t) + 2 * (size_t)ch * (V / 2) * 32 * sizeof(f32x2);
  const size_t per_cta = ((size_t)dev.max_smem_optin - 1024 * 3) / 3;
  int stages = (int)((per_cta - fixed) / (kResWarps * stage_bytes));
  if (stages > 4) stages = 4;
  if (stages < 2) return false;
  const size_t smem = kResWarps * stages * stage_bytes + fixed;
  long long grid = 3LL * dev.sm_count;
  const long long useful = (p.rows + kResWarps - 1) / kResWarps;
  if (grid > useful) grid = useful;
  const bool exact = nv == 32LL * ch;
  auto launch = [&](auto kernel) {
    const cudaError_t e = allow_dynamic_smem(reinterpret_cast<const void*>(kernel), smem);
    if (e != cudaSuccess) {
      cudaGetLastError();
      *rc = fail((int)e, "b200_norm_fwd: cannot reserve %zu bytes of shared memory: %s", smem, cudaGetErrorString(e));
      return;
    }
    launch_dependent(kernel, (unsigned)grid, kResWarps * 32, smem, st, p, stages);
    *rc = launch_status("b200_norm_fwd [residual add, warp per row, warp rings]");
  };
  auto pick = [&](auto both_tag) {
    constexpr bool BOTH = decltype(both_tag)::value;
    if (ch == 3) {
      if (exact) launch(residual_norm_warp_kernel<T, 3, true, BOTH>);
      else launch(residual_norm_warp_kernel<T, 3, false, BOTH>);
    } else {
      if (exact) launch(residual_norm_warp_kernel<T, 4, true, BOTH>);
      else launch(residual_norm_warp_kernel<T, 4, false, BOTH>);
    }
  };
  if constexpr (sizeof(T) == 2) {
    if (p.res_round == 2) pick(std::true_type{});
    else pick(std::false_type{});
  } else {
    pick(std::false_type{});
  }
  return true;
}

// Element-wise kernel for ragged, unaligned or very long rows: one CTA per row, sweeps over
// global memory (the second and third sweep of a row that fits in L2 are served from there).
template <typename Tin, typename Tout>
__global__ void __launch_bounds__(1024) norm_fwd_streaming_kernel(const NormFwdParams p) {
  wait_for_previous_kernel();
  __shared__ float red[32];
  const long long row = blockIdx.x;
  const Tin* x = reinterpret_cast<const Tin*>(p.x) + row * p.x_row_stride;

  const Tin* res = p.res ? reinterpret_cast<const Tin*>(p.res) + row * p.x_row_stride : nullptr;
  auto value = [&](long long i) {
    float f = Elem<Tin>::to_f32(x[i]);
    if (res) {
      f = f + Elem<Tin>::to_f32(res[i]);
      if (p.res_round == 1) f = round_through<Tin>(f);
    }
    return p.prologue == 1 ? gelu_erf_rounded<Tin>(f) : f;
  };
  auto rounded_value = [&](long long i) {  // the other form of the residual sum (res_round == 2)
    return round_through<Tin>(Elem<Tin>::to_f32(x[i]) + Elem<Tin>::to_f32(res[i]));
  };
  if (res && p.sum_out) {
    Tin* so = reinterpret_cast<Tin*>(p.sum_out) + row * (long long)p.n;
    for (long long i = threadIdx.x; i < p.n; i += blockDim.x)
      so[i] = Elem<Tin>::from_f32(Elem<Tin>::to_f32(x[i]) + Elem<Tin>::to_f32(res[i]));
  }
  float s = 0.f;
  for (long long i = threadIdx.x; i < p.n; i += blockDim.x) {
    const float f = value(i);
    s += p.rms ? f * f : f;
  }
  s = block_reduce<SumOp>(s, red);
  float mean = 0.f, var, rstd;
  if (p.rms) {
    var = s * p.inv_n;
  } else {
    mean = s * p.inv_n;
    float q = 0.f;
    for (long long i = threadIdx.x; i < p.n; i += blockDim.x) {
      const float d = value(i) - mean;
      q += d * d;
    }
    q = block_reduce<SumOp>(q, red);
    var = q * p.inv_denom;
  }
  rstd = precise_rsqrt(var + p.eps);
  if (threadIdx.x == 0) {
    if (p.mean_out) p.mean_out[row] = mean;
    if (p.rstd_out) p.rstd_out[row] = rstd;
    if (p.var_out) p.var_out[row] = var;
  }
  if (p.y == nullptr) return;
  const bool both = res && p.res_round == 2;
  float mean_r = 0.f, rstd_r = 0.f;
  if (both) {
    float t = 0.f;
    for (long long i = threadIdx.x; i < p.n; i += blockDim.x) t += rounded_value(i);
    mean_r = block_reduce<SumOp>(t, red) * p.inv_n;
    float q = 0.f;
    for (long long i = threadIdx.x; i < p.n; i += blockDim.x) {
      const float d = rounded_value(i) - mean_r;
      q += d * d;
    }
    rstd_r = precise_rsqrt(block_reduce<SumOp>(q, red) * p.inv_denom + p.eps);
  }
  Tout* y = reinterpret_cast<Tout*>(p.y) + row * p.y_row_stride;
  for (long long i = threadIdx.x; i < p.n; i += blockDim.x) {
    float o = (value(i) - mean) * rstd;
    if (p.w) o = o * load_param1(p.w, p.w_dtype, i);
    if (p.b) o = o + load_param1(p.b, p.w_dtype, i);
    if (both && !(fabsf(round_through<Tout>(o)) > 3.0f)) {
      o = (rounded_value(i) - mean_r) * rstd_r;
      if (p.w) o = o * load_param1(p.w, p.w_dtype, i);
      if (p.b) o = o + load_param1(p.b, p.w_dtype, i);
    }
    y[i] = Elem<Tout>::from_f32(o);
  }
}

// Ragged or unaligned rows that fit in registers: a warp per row (n <= 512) or a CTA per row, E
// elements per thread at a distance of the group, so that every access of a warp is one coalesced
// stretch of 2- or 4-byte elements whatever the row's alignment. The row is read once; the element-wise
// sweeps below read it two to six times and are left with rows of more than 16 384 elements (16 a thread).
// Many rows of a 16-bit type, and long ones of fp32, go by the vector instead (norm_fwd_span.cu, with both sides' times).
// Bound by the number of those accesses: about 1.6 TB/s for 16-bit elements, 3.3 TB/s for fp32.
// Measured against the sweeps: LayerNorm bf16 [4800, 769] 114 -> 17.5 us, [4800, 8191] 246 -> 158, RMSNorm f32 [4800, 1001]
// 82 -> 14.6 us, residual LayerNorm (both forms) bf16 [18682, 449] 322 -> 52 us.
// Few rows (up to eight per SM of 129..512 elements, two per SM of up to 2048) take a CTA per row with two elements a
// thread, as the longer chains of a thread are not hidden then: LayerNorm bf16 [148, 449] by warps 4.8 us, so 3.0;
// [600, 257] 4.4 and 3.1 ([2400, 257] 4.8 by warps); [148, 769] with eight a thread 4.9, so 3.3.
// Weight and bias are asked for in groups before the stores: one by one they cost [148, 449] 9.9 us.
// G: 32 = a warp per row, 0 = the CTA.
template <typename Tin, typename Tout, int E, int G>
// (Two CTAs of 1024 threads per SM for 16-bit rows, 32 registers; otherwise no minimum, which is not the same as 1:
// that allows 64 registers, and fp32 rows of 5001 run one CTA per SM instead of two, [4800, 5001] 64.6 -> 101 us.)
__global__ void __launch_bounds__(G == 0 ? 1024 : 256, G == 0 && E == 8 && sizeof(Tin) == 2 ? 2 : 0)
norm_fwd_ragged_kernel(const NormFwdParams p) {
  wait_for_previous_kernel();
  __shared__ float red[64];
  constexpr bool DUAL = std::is_same<Tin, Tout>::value && sizeof(Tin) == 2;
  const int lane = glane<G>(), gs = gsize<G>();
  long long row = grow<G>();
  const bool valid = row < p.rows;  // warps of a partly filled last CTA recompute the last row
  if (!valid) row = p.rows - 1;
  const Tin* x = reinterpret_cast<const Tin*>(p.x) + row * p.x_row_stride;
  const Tin* res = p.res ? reinterpret_cast<const Tin*>(p.res) + row * p.x_row_stride : nullptr;
  const bool both = DUAL && res != nullptr && p.res_round == 2;
  const int n = p.n;
  float f[E];
#pragma unroll
  for (int e = 0; e < E; ++e) f[e] = e * gs + lane < n ? Elem<Tin>::to_f32(ld_here(x + e * gs + lane)) : 0.f;
  if (res) {
    float r[E];
#pragma unroll
    for (int e = 0; e < E; ++e) r[e] = e * gs + lane < n ? Elem<Tin>::to_f32(ld_here(res + e * gs + lane)) : 0.f;
    Tin* so = p.sum_out && valid ? reinterpret_cast<Tin*>(p.sum_out) + row * (long long)n : nullptr;
#pragma unroll
    for (int e = 0; e < E; ++e) {
      f[e] = f[e] + r[e];
      if (so && e * gs + lane < n) so[e * gs + lane] = Elem<Tin>::from_f32(f[e]);
      if (p.res_round == 1) f[e] = round_through<Tin>(f[e]);
    }
  }
  if (p.prologue == 1) {  // gelu(0) = 0: the padding stays zero
#pragma unroll
    for (int e = 0; e < E; e += 2) unpack2(gelu_erf_rounded2<Tin>(pack2(f[e], f[e + 1])), f[e], f[e + 1]);
  }
  float s = 0.f, t = 0.f;  // t: the sum over the rounded values (both forms)
#pragma unroll
  for (int e = 0; e < E; ++e) s += p.rms ? f[e] * f[e] : f[e];
  if constexpr (DUAL) {
    if (both) {
#pragma unroll
      for (int e = 0; e < E; ++e) t += round_through<Tin>(f[e]);
    }
  }
  greduce_sum2<G>(s, t, red);
  float mean = 0.f, var = s * p.inv_n, rstd_r = 0.f;
  const float mean_r = t * p.inv_n;
  if (!p.rms) {
    mean = s * p.inv_n;
    float q = 0.f, u = 0.f;
#pragma unroll
    for (int e = 0; e < E; ++e) {
      if (e * gs + lane < n) {
        const float d = f[e] - mean;
        q += d * d;
        if constexpr (DUAL) {
          if (both) {
            const float dr = round_through<Tin>(f[e]) - mean_r;
            u += dr * dr;
          }
        }
      }
    }
    greduce_sum2<G>(q, u, red);
    var = q * p.inv_denom;
    rstd_r = precise_rsqrt(u * p.inv_denom + p.eps);
  }
  const float rstd = precise_rsqrt(var + p.eps);
  if (lane == 0 && valid) {
    if (p.mean_out) p.mean_out[row] = mean;
    if (p.rstd_out) p.rstd_out[row] = rstd;
    if (p.var_out) p.var_out[row] = var;
  }
  if (p.y == nullptr || !valid) return;
  Tout* y = reinterpret_cast<Tout*>(p.y) + row * p.y_row_stride;
  // parameters in flight per thread: a CTA per row has other warps to hide them behind, and registers to save
  constexpr int AT_ONCE = E < 8 ? E : (G != 0 ? 8 : (E == 8 && sizeof(Tin) == 4 ? 4 : 2));
#pragma unroll
  for (int e0 = 0; e0 < E; e0 += AT_ONCE) {
    float w[AT_ONCE], b[AT_ONCE];
    if (p.w) load_params_strided(p.w, p.w_dtype, e0 * gs + lane, gs, n, w);
    if (p.b) load_params_strided(p.b, p.w_dtype, e0 * gs + lane, gs, n, b);
#pragma unroll
    for (int k = 0; k < AT_ONCE; ++k) {
      const int e = e0 + k, i = e * gs + lane;
      if (i < n) {
        float o = (f[e] - mean) * rstd;
        if (p.w) o = o * w[k];
        if (p.b) o = o + b[k];
        if constexpr (DUAL) {
          if (both && !(fabsf(round_through<Tout>(o)) > 3.0f)) {
            o = (round_through<Tin>(f[e]) - mean_r) * rstd_r;
            if (p.w) o = o * w[k];
            if (p.b) o = o + b[k];
          }
        }
        y[i] = Elem<Tout>::from_f32(o);
      }
    }
  }
}

template <typename Tin, typename Tout>
static int launch_norm_fwd(const NormFwdParams& p, bool vector_ok, cudaStream_t st) {
  constexpr int V = Elem<Tin>::V;
  if (p.rows > 0x7fffffffLL) return fail(B200_ERR_UNSUPPORTED, "norm_fwd: too many rows");
  RowGeometry g;
  constexpr bool kResBuilt = std::is_same<Tin, Tout>::value;  // the residual prologue: same-dtype pairs only
  if (p.res && !kResBuilt) return fail(B200_ERR_UNSUPPORTED, "norm_fwd: the residual prologue needs y in x's dtype");
  if (vector_ok && p.n % V == 0 && !p.res) {  // the ring kernel streams one tensor
    int rc = B200_OK;
    if (try_launch_norm_fwd_stream<Tin, Tout>(p, st, &rc)) return rc;
  }
  if constexpr (kResBuilt) {
    int rc = B200_OK;
    if (vector_ok && p.n % V == 0 && p.res && try_launch_residual_norm_warp<Tin>(p, st, &rc)) return rc;
  }
  if (vector_ok && p.n % V == 0 && pick_row_geometry(p.n / V, &g)) {
    set_path_tag(g.block ? (p.res ? "residual add, vector, row resident, CTA per row" : "vector, row resident, CTA per row")
                         : (p.res ? "residual add, vector, row resident, sub-warp rows" : "vector, row resident, sub-warp rows"));
#define B200_NF_LAUNCH(GG, CC)                                                                              \
  do {                                                                                                      \
    if constexpr (kResBuilt) {                                                                              \
      if (p.res) {                                                                                          \
        if (p.prologue) launch_dependent(norm_fwd_resident_kernel<Tin, Tout, CC, GG, true, true>, grid, g.threads, 0, st, p); \
        else launch_dependent(norm_fwd_resident_kernel<Tin, Tout, CC, GG, false, true>, grid, g.threads, 0, st, p);       \
        break;                                                                                              \
      }                                                                                                     \
    }                                                                                                       \
    if (p.prologue) launch_dependent(norm_fwd_resident_kernel<Tin, Tout, CC, GG, true, false>, grid, g.threads, 0, st, p); \
    else launch_dependent(norm_fwd_resident_kernel<Tin, Tout, CC, GG, false, false>, grid, g.threads, 0, st, p);          \
  } while (0)
    if (!g.block) {
      if (p.res) {  // CTAs of 128 threads for the residual kernels (measured: 45.8 -> 44.3 us on the case above)
        static const int t_env = [] { const char* e = getenv("B200_NF_RES_THREADS"); return e ? atoi(e) : 0; }();
        g.threads = (t_env == 64 || t_env == 128 || t_env == 256) ? t_env : 128;
      }
      const int rows_per_cta = g.threads / g.g;
      const unsigned grid = (unsigned)((p.rows + rows_per_cta - 1) / rows_per_cta);
      if (g.g == 8) {
        if (g.ch == 1) B200_NF_LAUNCH(8, 1);
        else if (g.ch == 2) B200_NF_LAUNCH(8, 2);
        else B200_NF_LAUNCH(8, 4);
      } else if (g.g == 16) {
        B200_NF_LAUNCH(16, 4);
      } else {
        B200_NF_LAUNCH(32, 4);
      }
    } else {
      const unsigned grid = (unsigned)p.rows;
      if (g.ch == 2) B200_NF_LAUNCH(0, 2);
      else if (g.ch == 4) B200_NF_LAUNCH(0, 4);
      else B200_NF_LAUNCH(0, 8);
    }
#undef B200_NF_LAUNCH
  } else if (p.n <= 16384) {
    set_path_tag(p.res ? "residual add, elements in registers" : "elements in registers");
    if constexpr (kResBuilt) {
      if (try_launch_norm_fwd_span<Tin>(p, st)) return launch_status("b200_norm_fwd");
    }
    if (p.n > 128 && p.n <= 2048 && p.rows <= (p.n <= 512 ? 8LL : 2LL) * device_info().sm_count) {
      launch_dependent(norm_fwd_ragged_kernel<Tin, Tout, 2, 0>, (unsigned)p.rows, ((p.n + 1) / 2 + 31) / 32 * 32, 0, st, p);
    } else if (p.n <= 512) {  // a warp per row
      const unsigned grid = (unsigned)((p.rows + 7) / 8);
      if (p.n <= 64) launch_dependent(norm_fwd_ragged_kernel<Tin, Tout, 2, 32>, grid, 256, 0, st, p);
      else if (p.n <= 128) launch_dependent(norm_fwd_ragged_kernel<Tin, Tout, 4, 32>, grid, 256, 0, st, p);
      else if (p.n <= 256) launch_dependent(norm_fwd_ragged_kernel<Tin, Tout, 8, 32>, grid, 256, 0, st, p);
      else launch_dependent(norm_fwd_ragged_kernel<Tin, Tout, 16, 32>, grid, 256, 0, st, p);
    } else if (p.n <= 8192) {
      const int threads = ((p.n + 7) / 8 + 31) / 32 * 32;
      launch_dependent(norm_fwd_ragged_kernel<Tin, Tout, 8, 0>, (unsigned)p.rows, threads, 0, st, p);
    } else {
      const int threads = ((p.n + 15) / 16 + 31) / 32 * 32;
      launch_dependent(norm_fwd_ragged_kernel<Tin, Tout, 16, 0>, (unsigned)p.rows, threads, 0, st, p);
    }
  } else {
    set_path_tag(p.res ? "residual add, element-wise, CTA per row" : "element-wise, CTA per row");
    launch_dependent(norm_fwd_streaming_kernel<Tin, Tout>, (unsigned)p.rows, 1024, 0, st, p);
  }
  return launch_status("b200_norm_fwd");
}

}  // namespace b200

using namespace b200;

// Bounded waits of the streaming kernel that ran out since the library was loaded (0 in normal
// operation). Synchronises the device.
extern "C" int64_t b200_norm_fwd_wait_timeouts(void) { return (int64_t)read_wait_timeouts(); }

extern "C" int b200_norm_fwd_residual(const void* x, const void* residual, void* sum_out, const void* weight,
                                      const void* bias, void* y, float* mean_out, float* rstd_out, float* var_out,
                                      int64_t rows, int64_t n, int64_t x_row_stride, int64_t y_row_stride,
                                      int32_t x_dtype, int32_t w_dtype, int32_t y_dtype, double eps,
                                      double correction, int32_t rms, void* stream) {
  if (!x) return fail(B200_ERR_INVALID, "b200_norm_fwd: null x");
  if (sum_out && !residual) return fail(B200_ERR_INVALID, "b200_norm_fwd_residual: sum_out without residual");
  if (rows < 0 || n < 0 || n > 0x7fffffffLL)
    return fail(B200_ERR_INVALID, "b200_norm_fwd: bad sizes rows=%lld n=%lld", (long long)rows, (long long)n);
  if (rows == 0) return B200_OK;
  if (n == 0) return fail(B200_ERR_INVALID, "b200_norm_fwd: empty rows have no statistics");
  if (w_dtype < 0 || w_dtype > 2) return fail(B200_ERR_INVALID, "b200_norm_fwd: bad weight dtype");

  NormFwdParams p;
  p.x = x; p.w = weight; p.b = bias; p.y = y;
  p.mean_out = mean_out; p.rstd_out = rstd_out; p.var_out = var_out;
  p.rows = rows; p.n = (int)n;
  p.x_row_stride = x_row_stride; p.y_row_stride = y_row_stride;
  p.w_dtype = w_dtype; p.eps = (float)eps; p.rms = (rms & 1) ? 1 : 0;
  p.prologue = (rms & 2) ? 1 : 0;  // bit 1 of the mode word: exact GELU of x, rounded to x's dtype, first
  p.res = residual; p.sum_out = sum_out;
  // bits 2 and 3 of the mode word: 4 rounds the residual sum to x's dtype first; 8 normalises both
  // forms and selects per element (LayerNorm without the GELU prologue; for fp32 tensors the two
  // forms are the same row, so 8 means 0 there)
  if ((rms & 12) == 12) return fail(B200_ERR_INVALID, "b200_norm_fwd_residual: mode bits 4 and 8 exclude each other");
  if ((rms & 12) && !residual) return fail(B200_ERR_INVALID, "b200_norm_fwd_residual: mode bits 4 and 8 need a residual");
  if ((rms & 8) && (rms & 3)) return fail(B200_ERR_UNSUPPORTED, "b200_norm_fwd_residual: both forms of the sum are built for plain LayerNorm only");
  p.res_round = (rms & 4) ? 1 : ((rms & 8) && x_dtype != B200_F32 ? 2 : 0);
  p.inv_n = (float)(1.0 / (double)n);
  p.inv_denom = (float)(1.0 / ((double)n - correction));  // inf/NaN for n <= correction, as aten

  const int ib = dtype_size(x_dtype), ob = dtype_size(y_dtype), wb = dtype_size(w_dtype);
  const int v_in = 16 / ib;
  const int out_chunk = v_in * ob < 16 ? v_in * ob : 16;
  const int w_chunk = v_in * wb < 16 ? v_in * wb : 16;
  bool vec = aligned16(x) && (x_row_stride * ib) % 16 == 0;
  if (residual) vec = vec && aligned16(residual) && (!sum_out || (aligned16(sum_out) && (n * ib) % 16 == 0));
  if (y) vec = vec && reinterpret_cast<uintptr_t>(y) % out_chunk == 0 && (y_row_stride * ob) % out_chunk == 0;
  if (weight) vec = vec && reinterpret_cast<uintptr_t>(weight) % w_chunk == 0;
  if (bias) vec = vec && reinterpret_cast<uintptr_t>(bias) % w_chunk == 0;
  cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);

#define B200_NORM_CASE(TI, TO, DI, DO) \
  if (x_dtype == DI && y_dtype == DO) return launch_norm_fwd<TI, TO>(p, vec, st);
  B200_NORM_CASE(float, float, B200_F32, B200_F32)
  B200_NORM_CASE(__nv_bfloat16, __nv_bfloat16, B200_BF16, B200_BF16)
  B200_NORM_CASE(__half, __half, B200_F16, B200_F16)
  B200_NORM_CASE(__nv_bfloat16, float, B200_BF16, B200_F32)
  B200_NORM_CASE(__half, float, B200_F16, B200_F32)
  B200_NORM_CASE(float, __nv_bfloat16, B200_F32, B200_BF16)
  B200_NORM_CASE(float, __half, B200_F32, B200_F16)
#undef B200_NORM_CASE
  return fail(B200_ERR_UNSUPPORTED, "b200_norm_fwd: dtype pair (%d -> %d) not built", x_dtype, y_dtype);
}

extern "C" int b200_norm_fwd(const void* x, const void* weight, const void* bias, void* y,
                             float* mean_out, float* rstd_out, float* var_out, int64_t rows,
                             int64_t n, int64_t x_row_stride, int64_t y_row_stride,
                             int32_t x_dtype, int32_t w_dtype, int32_t y_dtype, double eps,
                             double correction, int32_t rms, void* stream) {
  return b200_norm_fwd_residual(x, nullptr, nullptr, weight, bias, y, mean_out, rstd_out, var_out, rows, n,
                                x_row_stride, y_row_stride, x_dtype, w_dtype, y_dtype, eps, correction, rms, stream);
}
