// Layout-changing copies with a pointwise epilogue (optional scale, dtype conversion):
//   * general: up to four dimensions with arbitrary input strides into a contiguous output
//     (head split [B,S,H,D] -> [B,H,S,D], any permute + clone);
//   * transpose of the two innermost dimensions through a padded shared-memory tile, coalesced
//     row accesses on both sides;
//   * contiguous cast / scale (no layout change).
//
// Replaces the permuting pointwise Triton kernels of the reference:
// repros/canonical/pointwise_c0d19d490a2f/oracle.py:10-33 (head-split gather copy),
// pointwise_021e90d9c17d/oracle.py:10-51 (autotuned 2-D tile transpose),
// pointwise_8bb40810003c/oracle.py:11-15 and pointwise_95ed2ef35da9/oracle.py:10-44 (cast / scale).
//
// Pointwise semantics follow aten: the value is converted to fp32, multiplied by the scale (when
// given) and rounded once to the output dtype.
#include "rowwise.cuh"
#include "tile_stream.cuh"

#include <type_traits>
#include <cstdlib>

namespace b200 {

struct PermuteParams {
  const void* x;
  void* y;
  long long shape[4];      // OUTPUT shape, outermost first (unused leading dims are 1)
  long long in_stride[4];  // input stride of each OUTPUT dimension, in elements
  FastDiv d1, d2, d3;      // fast division by shape[1], shape[2], shape[3] (in units of the inner vector)
  long long total;         // output elements
  float scale;
  int has_scale;
};

// Activation bits of the mode word (after the optional scaling), each the fp32 expression of the
// decomposed aten graph: 2 ReLU (a NaN stays a NaN); 4 exact GELU, (x * 0.5) * (erf(x * 0.7071067811865476) + 1)
// (repros/canonical/pointwise_826ea0b5f6e4/repro.py:27-31); 8 SiLU, x / (exp(-x) + 1)
// (repros/canonical/pointwise_795cdbe23b17/repro.py:26-29).
// One activation per launch; ACT is its bit (0: none), so that each instantiation carries only the
// code it uses.
// For 16-bit results GELU and SiLU are evaluated by the pair forms of rowwise.cuh, in the vector loop and for
// single elements alike: a result does not depend on an element's position or on the tensor's alignment.
template <typename Tout, int ACT>
__device__ __forceinline__ f32x2 apply_activation2(f32x2 v) {
  if constexpr (ACT == 4 && sizeof(Tout) == 2) return gelu_pair(v);
  if constexpr (ACT == 8 && sizeof(Tout) == 2) return silu_pair(v);
  float a, b;
  unpack2(v, a, b);
  auto one = [](float f) {
    if constexpr (ACT == 2) f = f < 0.f ? 0.f : f;
    if constexpr (ACT == 4) f = (f * 0.5f) * (erff(f * 0.7071067811865476f) + 1.0f);
    if constexpr (ACT == 8) f = f / (expf(-f) + 1.0f);
    return f;
  };
  return pack2(one(a), one(b));
}

template <typename Tin, typename Tout, int ACT = 0>
__device__ __forceinline__ Tout convert_scaled(Tin v, float scale, int has_scale) {
  float f = Elem<Tin>::to_f32(v), unused;
  if (has_scale & 1) f = f * scale;
  unpack2(apply_activation2<Tout, ACT>(splat2(f)), f, unused);
  return Elem<Tout>::from_f32(f);
}

// General kernel. VEC: the innermost output dimension is also unit-stride in the input and both
// sides are 16-byte friendly, so a thread moves VIN = 16 / sizeof(Tin) elements at once.
template <typename Tin, typename Tout, bool VEC>
__global__ void __launch_bounds__(256) permute_general_kernel(const PermuteParams p) {
  wait_for_previous_kernel();
  constexpr int VIN = VEC ? Elem<Tin>::V : 1;
  constexpr int U = VEC ? 4 : 1;  // independent 16-byte loads in flight per thread
  const long long units = p.total / VIN;
  // input offset of unit u: decompose u over (shape[0], shape[1], shape[2], shape[3] / VIN)
  auto in_offset = [&](long long u) {
    long long i3, i2, i1, i0;
    if (u < 0x7fffffffLL) {
      unsigned int r = (unsigned int)u;
      unsigned int q = fast_div(r, p.d3);
      i3 = r - q * p.d3.d; r = q;
      q = fast_div(r, p.d2);
      i2 = r - q * p.d2.d; r = q;
      q = fast_div(r, p.d1);
      i1 = r - q * p.d1.d;
      i0 = q;
    } else {
      long long rest = u;
      const long long n3 = p.d3.d, n2 = p.d2.d, n1 = p.d1.d;
      i3 = rest % n3; rest /= n3;
      i2 = rest % n2; rest /= n2;
      i1 = rest % n1;
      i0 = rest / n1;
    }
    return i0 * p.in_stride[0] + i1 * p.in_stride[1] + i2 * p.in_stride[2] + i3 * VIN * p.in_stride[3];
  };
  // a CTA takes blocks of U * blockDim consecutive output units (block b, b + grid, ...), so that
  // its U stores (and, for most layouts, loads) in flight per thread fall into one stretch of memory
  const long long stride = blockDim.x;
  const long long block = (long long)U * blockDim.x;
  for (long long u0 = (long long)blockIdx.x * block + threadIdx.x; u0 < units; u0 += (long long)gridDim.x * block) {
    if constexpr (VEC) {
      uint4 raw[U];
#pragma unroll
      for (int k = 0; k < U; ++k) {
        const long long u = u0 + k * stride;
        if (u < units) raw[k] = ld_stream(reinterpret_cast<const Tin*>(p.x) + in_offset(u));
      }
#pragma unroll
      for (int k = 0; k < U; ++k) {
        const long long u = u0 + k * stride;
        if (u < units) {
          Tout* dst = reinterpret_cast<Tout*>(p.y) + u * VIN;
          if (std::is_same<Tin, Tout>::value && !p.has_scale) {
            st_stream(reinterpret_cast<Tin*>(dst), raw[k]);  // plain copy: no conversion at all
          } else {
            float f[VIN];
            Elem<Tin>::unpack(raw[k], f);
            if (p.has_scale) {
#pragma unroll
              for (int i = 0; i < VIN; ++i) f[i] = f[i] * p.scale;
            }
            store_converted<Tout, VIN>(dst, f);
          }
        }
      }
    } else {
      const Tin* src = reinterpret_cast<const Tin*>(p.x) + in_offset(u0);
      reinterpret_cast<Tout*>(p.y)[u0] = convert_scaled<Tin, Tout>(*src, p.scale, p.has_scale);
    }
  }
}

// Transpose of the two innermost dimensions: output [batch, C, P] from input [batch, P, C]
// (input row stride in_row_stride, batch stride in_batch_stride). 64 x 64 element tiles; a warp
// reads and writes whole tile rows (64 consecutive elements), the transposition happens in shared
// memory (row pitch padded by one 4-byte word to spread the column reads over the banks).
struct TransposeParams {
  const void* x;
  void* y;
  long long batch, P, C;
  long long in_batch_stride, in_row_stride;
  float scale;
  int has_scale;
};

template <typename Tin, typename Tout>
__global__ void __launch_bounds__(256) transpose_tile_kernel(const TransposeParams p) {
  wait_for_previous_kernel();
  constexpr int TILE = 64;
  __shared__ float tile[TILE][TILE + 1];
  const long long b = blockIdx.z;
  const long long p0 = (long long)blockIdx.y * TILE, c0 = (long long)blockIdx.x * TILE;
  const Tin* src = reinterpret_cast<const Tin*>(p.x) + b * p.in_batch_stride;
  Tout* dst = reinterpret_cast<Tout*>(p.y) + b * p.P * p.C;
  // load: thread (ty, tx) walks rows of the input tile, columns contiguous
  for (int r = threadIdx.x / TILE; r < TILE; r += 256 / TILE) {
    const int c = threadIdx.x % TILE;
    const long long pr = p0 + r, pc = c0 + c;
    float v = 0.f;
    if (pr < p.P && pc < p.C) {
      v = Elem<Tin>::to_f32(src[pr * p.in_row_stride + pc]);
      if (p.has_scale) v = v * p.scale;
    }
    tile[r][c] = v;
  }
  __syncthreads();
  // store: rows of the output tile are columns of the input tile
  for (int r = threadIdx.x / TILE; r < TILE; r += 256 / TILE) {
    const int c = threadIdx.x % TILE;
    const long long oc = c0 + r, op = p0 + c;  // output row index = input column
    if (oc < p.C && op < p.P) dst[oc * p.P + op] = Elem<Tout>::from_f32(tile[c][r]);
  }
}

// Transpose of 16-bit elements without conversion, whole 64 x 64 tiles only: 16-byte accesses on
// both sides. The tile lives in shared memory as 64 rows of 32 words (two elements per word), row r
// rotated by 4 * (r / 8) words. A thread then reads, for one pair of input columns and eight
// consecutive input rows, eight words that fall into eight different banks, and splits them into two
// output vectors with byte permutes: eight consecutive elements of output row 2c and of row 2c + 1.
__global__ void __launch_bounds__(256) transpose16_tile_kernel(const TransposeParams p) {
  wait_for_previous_kernel();
  __shared__ __align__(16) uint32_t tile[64][32];
  const long long b = blockIdx.z;
  const long long p0 = (long long)blockIdx.y * 64, c0 = (long long)blockIdx.x * 64;
  const unsigned short* src = reinterpret_cast<const unsigned short*>(p.x) + b * p.in_batch_stride;
  unsigned short* dst = reinterpret_cast<unsigned short*>(p.y) + b * p.P * p.C;
  const int tid = threadIdx.x;
#pragma unroll
  for (int k = 0; k < 2; ++k) {
    const int q = tid + k * 256;
    const int r = q >> 3, wv = q & 7;
    const uint4 v = ld_stream(reinterpret_cast<const __half*>(src + (p0 + r) * p.in_row_stride + c0 + wv * 8));
    *reinterpret_cast<uint4*>(&tile[r][(wv * 4 + 4 * (r >> 3)) & 31]) = v;
  }
  __syncthreads();
  const int ovc = tid & 7, cpair = tid >> 3;
  uint32_t w[8];
#pragma unroll
  for (int j = 0; j < 8; ++j) w[j] = tile[ovc * 8 + j][(cpair + 4 * ovc) & 31];
  uint4 lo, hi;
  lo.x = __byte_perm(w[0], w[1], 0x5410); hi.x = __byte_perm(w[0], w[1], 0x7632);
  lo.y = __byte_perm(w[2], w[3], 0x5410); hi.y = __byte_perm(w[2], w[3], 0x7632);
  lo.z = __byte_perm(w[4], w[5], 0x5410); hi.z = __byte_perm(w[4], w[5], 0x7632);
  lo.w = __byte_perm(w[6], w[7], 0x5410); hi.w = __byte_perm(w[6], w[7], 0x7632);
  unsigned short* o = dst + (c0 + 2 * cpair) * p.P + p0 + ovc * 8;
  st_stream(reinterpret_cast<__half*>(o), lo);
  st_stream(reinterpret_cast<__half*>(o + p.P), hi);
}

// Transpose of 16-bit elements without conversion for every shape that is not made of whole 64 x 64
// tiles: the tile is kept transposed in shared memory as words of two consecutive input rows, one
// word row per input column, so that an output row is written as 4-byte words whatever its parity
// (an output row of an odd length P starts on a 2-byte boundary: its first and last element then
// leave alone). A thread turns the words of rows 2r and 2r + 1 into the words of columns 2c and 2c + 1
// with two byte permutes; column c lives in row (c / 2) + 32 (c & 1), which keeps the writes of a warp
// in 32 different banks.
// pairs: rows start on 4-byte boundaries and C is even, so a warp reads a tile row as 32 words.
// Bound by HBM (half of the lines are touched by two CTAs). Measured against 2-byte accesses through a
// tile of floats: f16 [200, 501, 768] 173.6 -> 82.0 us, [300, 500, 333] 119.1 -> 56.3 us.
__global__ void __launch_bounds__(256) transpose16_ragged_kernel(const TransposeParams p, const int pairs) {
  wait_for_previous_kernel();
  __shared__ uint32_t tile[64 * 33];
  const long long b = blockIdx.z;
  const int p0 = (int)blockIdx.y * 64, c0 = (int)blockIdx.x * 64;
  const int np = p.P - p0 < 64 ? (int)(p.P - p0) : 64, nc = p.C - c0 < 64 ? (int)(p.C - c0) : 64;
  const unsigned short* src =
      reinterpret_cast<const unsigned short*>(p.x) + b * p.in_batch_stride + (long long)p0 * p.in_row_stride + c0;
  unsigned short* dst = reinterpret_cast<unsigned short*>(p.y) + b * p.P * p.C + (long long)c0 * p.P + p0;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if (pairs) {
    uint32_t w[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) {  // rows 2 (4 warp + i / 2) + (i & 1)
      const int r = warp * 8 + i;
      w[i] = r < np && 2 * lane < nc
                 ? ld_here(reinterpret_cast<const uint32_t*>(src + (long long)r * p.in_row_stride) + lane) : 0u;
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      tile[lane * 33 + warp * 4 + i] = __byte_perm(w[2 * i], w[2 * i + 1], 0x5410);
      tile[(lane + 32) * 33 + warp * 4 + i] = __byte_perm(w[2 * i], w[2 * i + 1], 0x7632);
    }
  } else {
    unsigned short e[2][8];
#pragma unroll
    for (int h = 0; h < 2; ++h)
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        const int r = warp * 8 + i, c = lane + 32 * h;
        e[h][i] = r < np && c < nc ? ld_here(src + (long long)r * p.in_row_stride + c) : (unsigned short)0;
      }
#pragma unroll
    for (int h = 0; h < 2; ++h)
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int c = lane + 32 * h;
        tile[((c >> 1) + 32 * (c & 1)) * 33 + warp * 4 + i] = (uint32_t)e[h][2 * i] | ((uint32_t)e[h][2 * i + 1] << 16);
      }
  }
  __syncthreads();
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const int c = warp * 8 + i;
    if (c >= nc) break;  // warp-uniform
    unsigned short* out = dst + (long long)c * p.P;
    const int odd = (int)((reinterpret_cast<uintptr_t>(out) >> 1) & 1u);
    const uint32_t* row = tile + ((c >> 1) + 32 * (c & 1)) * 33;
    uint32_t w = row[lane];
    const uint32_t next = __shfl_down_sync(0xffffffffu, w, 1);
    if (odd) {
      if (lane == 0) out[0] = (unsigned short)w;
      w = __byte_perm(w, next, 0x5432);  // elements 2 lane + 1 and 2 lane + 2; the second is missing in lane 31
    }
    const int at = 2 * lane + odd;
    if (at + 1 < np) *reinterpret_cast<uint32_t*>(out + at) = w;
    else if (at < np) out[at] = (unsigned short)w;
  }
}

// Batched transpose of SMALL 16-bit matrices without conversion (e.g. the [49, 128] and [196, 64]
// attention tiles of repros/canonical/pointwise_021e90d9c17d/shapes.json, whose 49 rows fill a 64 x 64
// tile only to three quarters and whose output rows of 49 elements start on 2-byte boundaries). One
// matrix, or a group of consecutive ones, is one contiguous block on both sides, so it crosses HBM as
// flat 16-byte vectors: asynchronous copies into a ring of `stages` shared-memory blocks, the
// transposition from shared memory to shared memory, one bulk store of the finished block.
//
// The transposition moves 4-byte words only. The output rows of columns 2c and 2c + 1 are 2 P
// consecutive elements, P whole words whether P is even or odd:
//   even P: word k of row 2c is (in[2k][2c], in[2k+1][2c]), the same for row 2c + 1
//   odd P : row 2c ends in the middle of a word, which row 2c + 1 completes; the latter's words pair
//           input rows (1, 2), (3, 4), ...
// so a thread that walks the words (2c, 2c + 1) of the input rows writes both. Neighbouring lanes take
// neighbouring column pairs: they read neighbouring words, and write words P apart - different banks
// when P is odd; for even P each lane starts its walk one word later than its neighbour, which makes
// the distance odd as well. Where P is a multiple of 8 that is not enough: 32 / gcd(P, 32) neighbours already
// meet every bank there is, so only the next such run of lanes starts a word later (bf16 [7324, 8, 512] 30.5 -> 28.2 us,
// [60000, 16, 32] 31.9 -> 29.4). P = 2 writes both words of a pair of columns at once ([14648, 2, 1024] 48.4 -> 25.0 us).
// What bounds it: HBM, with the shared-memory passes (copy in, read, write, copy out: about 390 cycles
// for a [49, 128] matrix, a third of the time its bytes take) behind it. Measured on bf16 [16384, 49, 128]:
// 139.5 us with two-byte gathers (four-way bank conflicts), 67.9 us (6.05 TB/s) here. The kernel divides by nothing but
// precomputed reciprocals: the divisions of its first form cost a tenth of that, and a fifth of a 2 us call.
template <int KIND>  // 0: P even, 1: P odd, 2: P = 2
__global__ void __launch_bounds__(256) transpose_pairs_kernel(const TransposeParams p, const int group, const long long groups,
                                                              const int stages, const int split, const FastDiv by_tasks,
                                                              const FastDiv by_pairs, const FastDiv by_split,
                                                              const FastDiv by_walk) {
  wait_for_previous_kernel();
  extern __shared__ __align__(128) unsigned char pairs_smem[];
  const int P = (int)p.P, C = (int)p.C, CW = C / 2;
  const int elems = P * C;
  const int span = group * elems * 2;  // bytes of a whole group, a multiple of 16
  const uint32_t ring = smem_u32(pairs_smem);
  unsigned char* const done = pairs_smem + (size_t)stages * span;  // the transposed group
  uint32_t* const out = reinterpret_cast<uint32_t*>(done);
  const int tid = threadIdx.x;
  // P a multiple of 8: rows of lanes whose words fall into the same banks start one word later than the row before
  const int stagger = P % 8 == 0 ? 5 - min(__ffs(P) - 1, 5) : 0;
  auto matrices_of = [&](long long g) {
    const long long left = p.batch - g * group;
    return (int)(left < group ? left : group);
  };
  auto load = [&](long long g, int slot) {
    if (g < groups) {
      const unsigned char* src = reinterpret_cast<const unsigned char*>(p.x) + g * group * p.in_batch_stride * 2;
      const int whole = matrices_of(g) * elems * 2 & ~15;
      for (int at = tid * 16; at < whole; at += 256 * 16) copy_async16(ring + (uint32_t)(slot * span + at), src + at);
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  long long g = blockIdx.x;
  for (int s = 0; s < stages - 1; ++s) load(g + (long long)s * gridDim.x, s);
  int slot = 0;
  for (; g < groups; g += gridDim.x) {
    const int ahead = slot == 0 ? stages - 1 : slot - 1;
    load(g + (long long)(stages - 1) * gridDim.x, ahead);  // its last reader passed the barrier below
    if (stages == 3) asm volatile("cp.async.wait_group 2;" ::: "memory");
    else asm volatile("cp.async.wait_group 1;" ::: "memory");
    const int here = matrices_of(g), bytes = here * elems * 2, whole = bytes & ~15;
    const unsigned char* block = pairs_smem + (size_t)slot * span;
    if (tid * 2 < bytes - whole)  // the last group may end between two 16-byte boundaries
      *reinterpret_cast<unsigned short*>(pairs_smem + (size_t)slot * span + whole + tid * 2) =
          ld_here(reinterpret_cast<const unsigned short*>(reinterpret_cast<const unsigned char*>(p.x) +
                                                        g * group * p.in_batch_stride * 2 + whole) + tid);
    if (tid == 0) asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");  // the block before has left
    __syncthreads();
    const uint32_t* in = reinterpret_cast<const uint32_t*>(block);
    const int tasks = group * CW, steps = P / 2;
    for (int t = tid; t < tasks * split; t += 256) {
      const int q = (int)fast_div((unsigned)t, by_tasks);
      const int u = t - q * tasks;
      const int m = (int)fast_div((unsigned)u, by_pairs);
      if (m >= here) continue;
      const int cp = u - m * CW;
      const int j0 = (int)fast_div((unsigned)(steps * q), by_split), j1 = (int)fast_div((unsigned)(steps * (q + 1)), by_split);
      const uint32_t* src = in + m * (elems / 2) + cp;
      uint32_t* dst = out + m * (elems / 2) + cp * P;
      if constexpr (KIND == 1) {
        uint32_t a = src[2 * j0 * CW];
#pragma unroll 4
        for (int j = j0; j < j1; ++j) {
          const uint32_t b = src[(2 * j + 1) * CW], n = src[(2 * j + 2) * CW];
          dst[j] = __byte_perm(a, b, 0x5410);
          dst[(P + 1) / 2 + j] = __byte_perm(b, n, 0x7632);
          a = n;
        }
        if (q == split - 1) dst[P / 2] = __byte_perm(src[(P - 1) * CW], src[0], 0x7610);
      } else if constexpr (KIND == 2) {  // P = 2: both words at once
        const uint32_t a = src[0], b = src[CW];
        *reinterpret_cast<uint2*>(dst) = make_uint2(__byte_perm(a, b, 0x5410), __byte_perm(a, b, 0x7632));
      } else {
        const int len = j1 - j0, x = cp >> stagger;
        int r = x - (int)fast_div((unsigned)x, by_walk) * (int)by_walk.d;  // below the shortest walk
#pragma unroll 4
        for (int j = 0; j < len; ++j) {
          const int k = j0 + r;
          const uint32_t a = src[2 * k * CW], b = src[(2 * k + 1) * CW];
          dst[k] = __byte_perm(a, b, 0x5410);
          dst[P / 2 + k] = __byte_perm(a, b, 0x7632);
          if (++r == len) r = 0;
        }
      }
    }
    fence_proxy_async_smem();  // the bulk store reads what the threads wrote
    __syncthreads();
    unsigned char* y = reinterpret_cast<unsigned char*>(p.y) + g * span;
    if (tid == 0 && whole > 0) {
      asm volatile("cp.async.bulk.global.shared::cta.bulk_group [%0], [%1], %2;" ::"l"(y), "r"(smem_u32(done)), "r"(whole)
                   : "memory");
      asm volatile("cp.async.bulk.commit_group;" ::: "memory");
    }
    if (tid * 2 < bytes - whole)
      reinterpret_cast<unsigned short*>(y + whole)[tid] = reinterpret_cast<const unsigned short*>(done + whole)[tid];
    if (++slot == stages) slot = 0;
  }
  asm volatile("cp.async.wait_all;" ::: "memory");
  if (tid == 0) asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");  // shared memory outlives the store
}

// Batched transpose of small 32-bit matrices (a [P, C] matrix fits in shared memory): both sides are
// moved with 16-byte accesses as flat arrays, the transposition is the shared-memory gather in
// between: output element o = c * P + p comes from [p][c]. A CTA takes matrices b, b + grid, ...
__global__ void __launch_bounds__(256) transpose_small_kernel(const TransposeParams p, const int pitch) {
  wait_for_previous_kernel();
  extern __shared__ __align__(16) unsigned char small_smem[];
  uint32_t* tile = reinterpret_cast<uint32_t*>(small_smem);  // [P][pitch]
  const int P = (int)p.P, C = (int)p.C;
  const int nvec = P * C / 4;
  for (long long b = blockIdx.x; b < p.batch; b += gridDim.x) {
    const uint32_t* src = reinterpret_cast<const uint32_t*>(p.x) + b * p.in_batch_stride;
    uint32_t* dst = reinterpret_cast<uint32_t*>(p.y) + b * (long long)P * C;
    for (int j0 = threadIdx.x; j0 < nvec; j0 += 4 * 256) {  // four loads in flight per thread
      uint4 raws[4];
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const int j = j0 + u * 256;
        if (j < nvec) raws[u] = ld_stream(src + (size_t)j * 4);
      }
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const int j = j0 + u * 256;
        if (j >= nvec) continue;
        const int r = j * 4 / C, c0 = j * 4 - r * C;  // C is a multiple of 4: the vector stays in one row
        uint32_t* t = tile + r * pitch + c0;
        t[0] = raws[u].x; t[1] = raws[u].y; t[2] = raws[u].z; t[3] = raws[u].w;
      }
    }
    __syncthreads();
    for (int j = threadIdx.x; j < nvec; j += 256) {
      int c = j * 4 / P, r = j * 4 - c * P;
      uint32_t w[4];
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        w[k] = tile[r * pitch + c];
        if (++r == P) { r = 0; ++c; }
      }
      st_stream(dst + (size_t)j * 4, make_uint4(w[0], w[1], w[2], w[3]));
    }
    __syncthreads();  // the tile is overwritten by the next matrix
  }
}

// Stores N values as Tout. WIDE: p lies on a 32-byte boundary, 32 bytes at a time where there are as many; otherwise p need
// only lie on min(16, N * sizeof(Tout)) bytes (8 values widened to fp32 are two stores of 16).
template <typename Tout, int N, bool WIDE>
__device__ __forceinline__ void store_unit(Tout* p, const f32x2 (&o)[N / 2]) {
  constexpr int BYTES = N * (int)sizeof(Tout);
  if constexpr (!WIDE || BYTES <= 16) {
    store_pairs<Tout, N>(p, o);
  } else {
    uint32_t w[BYTES / 4];
#pragma unroll
    for (int i = 0; i < N / 2; ++i) {
      if constexpr (sizeof(Tout) == 2) {
        w[i] = Pairs<Tout>::narrow(o[i]);
      } else {
        float a, b;
        unpack2(o[i], a, b);
        w[2 * i] = __float_as_uint(a);
        w[2 * i + 1] = __float_as_uint(b);
      }
    }
#pragma unroll
    for (int i = 0; i < BYTES / 32; ++i)
      st_stream32(reinterpret_cast<char*>(p) + 32 * i, make_uint4(w[8 * i], w[8 * i + 1], w[8 * i + 2], w[8 * i + 3]),
                  make_uint4(w[8 * i + 4], w[8 * i + 5], w[8 * i + 6], w[8 * i + 7]));
  }
}

// Contiguous cast / scale / activation (has_scale: bit 0 multiply by scale; bits 1..3 ReLU, exact GELU, SiLU after it).
// ACT: the activation bit of the mode word (0: none); the plain cast / scale instantiation carries none of
// the activations' code (the erf and exp sequences cost registers and instruction-cache lines that a 5 us
// parameter cast would pay for without using them).
// BYTES: what a thread loads at once (0: one element). Bound by HBM; SiLU by the SFU pipe (22 us of 35) next to it. Measured,
// 16 -> 32 bytes: SiLU bf16 [32768, 1536] 37.6 -> 35.0 us (5.75 TB/s), ReLU bf16 of 8 M elements 6.7 -> 6.4, f32 -> bf16 9.2 -> 8.6.
template <typename Tin, typename Tout, int BYTES, int ACT>
__global__ void __launch_bounds__(256, ACT >= 4 ? 5 : 4) cast_scale_kernel(const void* x, void* y, long long n, float scale,
                                                                            int mode_word) {
  wait_for_previous_kernel();
  const int has_scale = mode_word & 1;
  constexpr int NV = BYTES == 0 ? 1 : BYTES / 16;                // vectors of a unit
  constexpr int VIN = BYTES == 0 ? 1 : Elem<Tin>::V;             // elements of a vector
  const long long units = n / (NV * VIN);
  const Tin* src = reinterpret_cast<const Tin*>(x);
  Tout* dst = reinterpret_cast<Tout*>(y);
  if constexpr (BYTES != 0) {
    // A CTA takes blocks of U * blockDim consecutive units (block b, b + grid, ...): what its threads
    // have in flight falls into one contiguous stretch of memory.
    // GELU and SiLU: 32 bytes in flight and five CTAs per SM (48 registers) instead of 64 and three - their
    // arithmetic needs the warps more than the loads in flight (SiLU bf16 [32768, 1536] 47.1 -> 42.5 us).
    // They ask for their next block before they work on the one at hand (40.6 -> 37.6 us).
    constexpr int U = (ACT >= 4 ? 2 : 4) / NV;
    constexpr bool AHEAD = ACT >= 4;
    const long long stride = blockDim.x;
    const long long block = (long long)U * blockDim.x, step = (long long)gridDim.x * block;
    uint4 next[AHEAD ? U : 1][NV];
    auto fetch = [&](long long u0, auto& raw) {
#pragma unroll
      for (int k = 0; k < U; ++k) {
        const Tin* p = src + (u0 + k * stride) * (NV * VIN);
        if (u0 + k * stride < units) {
          if constexpr (NV == 2) ld_stream32(p, raw[k][0], raw[k][1]);
          else raw[k][0] = ld_stream(p);
        }
      }
    };
    const long long first = (long long)blockIdx.x * block + threadIdx.x;
    if constexpr (AHEAD) fetch(first, next);
    for (long long u0 = first; u0 < units; u0 += step) {
      uint4 raw[U][NV];
      if constexpr (AHEAD) {
#pragma unroll
        for (int k = 0; k < U; ++k)
#pragma unroll
          for (int v = 0; v < NV; ++v) raw[k][v] = next[k][v];
        fetch(u0 + step, next);
      } else {
        fetch(u0, raw);
      }
#pragma unroll
      for (int k = 0; k < U; ++k) {
        const long long u = u0 + k * stride;
        if (u < units) {
          f32x2 o[NV * VIN / 2];
#pragma unroll
          for (int v = 0; v < NV; ++v) {
            float f[VIN];
            Elem<Tin>::unpack(raw[k][v], f);
            if (has_scale & 1) {
#pragma unroll
              for (int i = 0; i < VIN; ++i) f[i] = f[i] * scale;
            }
            // SiLU: a vector without an element beyond 88 takes the form without clamps (bf16 [32768, 1536],
            // graph replay: 42.8 us with the clamps on every element, 40.8 us so)
            bool plain = false;
            if constexpr (ACT == 8 && sizeof(Tout) == 2) {
              float largest = fabsf(f[0]);
#pragma unroll
              for (int i = 1; i < VIN; ++i) largest = fmaxf(largest, fabsf(f[i]));
              plain = largest <= 88.f;
              if (plain) {
#pragma unroll
                for (int i = 0; i < VIN / 2; ++i)
                  o[v * (VIN / 2) + i] = silu_pair<false>(pack2(f[2 * i], f[2 * i + 1]));
              }
            }
            if (!plain) {
#pragma unroll
              for (int i = 0; i < VIN / 2; ++i)
                o[v * (VIN / 2) + i] = apply_activation2<Tout, ACT>(pack2(f[2 * i], f[2 * i + 1]));
            }
          }
          store_unit<Tout, NV * VIN, NV == 2>(dst + u * (NV * VIN), o);
        }
      }
    }
  } else {
    for (long long u = (long long)blockIdx.x * blockDim.x + threadIdx.x; u < units;
         u += (long long)gridDim.x * blockDim.x)
      dst[u] = convert_scaled<Tin, Tout, ACT>(src[u], scale, has_scale);
  }
  if constexpr (BYTES != 0) {  // ragged tail
    const long long done = units * (NV * VIN);
    const long long t = done + (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (t < n) dst[t] = convert_scaled<Tin, Tout, ACT>(src[t], scale, has_scale);
  }
}

// Grid of the flat streaming kernels: one CTA per 256 units (the caller counts a block of several per thread as 256) up to `per_sm` CTAs per SM, which then
// loop. Many small CTAs keep the window of addresses that are in flight at any moment narrow; for
// the cast kernel 128 per SM measured best on a 262 M-element bf16 -> f32 cast (8: 331 us, 16: 299,
// 32: 279, 64: 268, 128: 263, 256: 285, one CTA per block: 331). B200_STREAM_CTAS_PER_SM overrides both.
static unsigned streaming_grid(long long units, long long default_per_sm = 16) {
  const long long ctas = (units + 255) / 256;
  static const long long env_per_sm = [] { const char* e = getenv("B200_STREAM_CTAS_PER_SM"); return e ? atoll(e) : 0LL; }();
  const long long per_sm = env_per_sm > 0 ? env_per_sm : default_per_sm;
  const long long cap = (long long)device_info().sm_count * per_sm;
  return (unsigned)(ctas < 1 ? 1 : (ctas > cap ? cap : ctas));
}

template <typename Tin, typename Tout>
static int launch_permute(const PermuteParams& p, bool vec, cudaStream_t st) {
  const long long units = vec ? p.total / Elem<Tin>::V : p.total;
  set_path_tag(vec ? "vector gather" : "element-wise gather");
  if (vec) launch_dependent(permute_general_kernel<Tin, Tout, true>, streaming_grid(units), 256, 0, st, p);
  else launch_dependent(permute_general_kernel<Tin, Tout, false>, streaming_grid(units), 256, 0, st, p);
  return launch_status("b200_permute_copy");
}

// Groups of small 16-bit matrices through transpose_pairs_kernel; false when the shape does not fit.
static bool try_launch_transpose_pairs(const TransposeParams& p, cudaStream_t st, int* rc) {
  const long long elems = p.P * p.C;
  if (p.C % 2 != 0 || p.P < 2 || elems * 2 > 32 * 1024 || p.in_row_stride != p.C || !aligned16(p.x) || !aligned16(p.y))
    return false;
  const DeviceInfo& dev = device_info();
  int group = 1;  // the smallest group that is a whole number of 16-byte vectors
  while (group * elems % 8 != 0) group *= 2;
  if (group * elems * 2 > 32 * 1024) return false;
  if (p.in_batch_stride == elems || p.batch == 1) {
    // small matrices: larger groups (up to 12 KB a block), but no fewer than four blocks per SM
    while (2 * group * elems * 2 <= 12 * 1024 && p.batch / (2 * group) >= 4LL * dev.sm_count) group *= 2;
  } else if (group != 1 || p.in_batch_stride % 8 != 0) {
    return false;
  }
  const int span = (int)(group * elems * 2);
  // three stages while four CTAs fit an SM with them (bf16 [16384, 49, 128]: 67.9 us, 72.8 with two), two from there on
  // ([4185, 7, 1024] 21.1 us, 26.0 with three; [2441, 1024, 8] 20.8 and 23.4)
  const int stages = 4 * ((size_t)4 * span + 1024) <= (size_t)dev.max_smem_optin ? 3 : 2;
  const size_t smem = (size_t)(stages + 1) * span;
  const int tasks = (int)(group * (p.C / 2));
  int split = 256 / tasks;  // threads that share a pair of columns
  if (split > p.P / 2) split = (int)(p.P / 2);
  if (split < 1) split = 1;
  auto kernel = p.P % 2 ? transpose_pairs_kernel<1> : (p.P == 2 ? transpose_pairs_kernel<2> : transpose_pairs_kernel<0>);
  const cudaError_t e = allow_dynamic_smem(reinterpret_cast<const void*>(kernel), smem);
  if (e != cudaSuccess) {
    cudaGetLastError();
    return false;
  }
  int per_sm = (int)((size_t)dev.max_smem_optin / (smem + 1024));
  if (per_sm > 8) per_sm = 8;
  if (per_sm < 1) per_sm = 1;
  const long long groups = (p.batch + group - 1) / group;
  long long grid = groups;
  if (grid > (long long)dev.sm_count * per_sm) grid = (long long)dev.sm_count * per_sm;
  launch_dependent(kernel, (unsigned)grid, 256, smem, st, p, group, groups, stages, split, make_fast_div(tasks), make_fast_div(p.C / 2),
                                            make_fast_div(split), make_fast_div(p.P / 2 / split));
  *rc = launch_status("b200_transpose_copy [small matrices, word pairs]");
  return true;
}

template <typename Tin, typename Tout>
static int launch_transpose(const TransposeParams& p, cudaStream_t st) {
  dim3 grid((unsigned)((p.C + 63) / 64), (unsigned)((p.P + 63) / 64), (unsigned)p.batch);
  if constexpr (std::is_same<Tin, Tout>::value && sizeof(Tin) == 2) {
    if (!p.has_scale) {
      const bool whole = p.P % 64 == 0 && p.C % 64 == 0 && p.in_row_stride % 8 == 0 && p.in_batch_stride % 8 == 0 &&
                         aligned16(p.x) && aligned16(p.y);
      if (whole) {
        launch_dependent(transpose16_tile_kernel, grid, 256, 0, st, p);
        return launch_status("b200_transpose_copy [16-byte tiles]");
      }
      int rc = B200_OK;
      if (try_launch_transpose_pairs(p, st, &rc)) return rc;
      const bool words = p.C % 2 == 0 && p.in_row_stride % 2 == 0 && p.in_batch_stride % 2 == 0 &&
                         (reinterpret_cast<uintptr_t>(p.x) & 3u) == 0;
      if (p.P <= 0x7fffffffLL && p.C <= 0x7fffffffLL) {
        launch_dependent(transpose16_ragged_kernel, grid, 256, 0, st, p, words ? 1 : 0);
        return launch_status("b200_transpose_copy [ragged 16-bit tiles]");
      }
    }
  }
  if constexpr (std::is_same<Tin, Tout>::value && sizeof(Tin) == 4) {
    // small matrices: flat 16-byte copies around a shared-memory gather
    const long long elems = p.P * p.C;
    if (!p.has_scale && elems * 4 <= 32 * 1024 && p.C % 4 == 0 && p.in_row_stride == p.C && p.in_batch_stride % 4 == 0 &&
        aligned16(p.x) && aligned16(p.y) && p.batch >= 1) {
      const int pitch = (int)p.C + 1;
      const size_t smem = (size_t)p.P * pitch * sizeof(Tin);
      if (smem <= 48 * 1024) {
        long long ctas = p.batch;
        const long long cap = (long long)device_info().sm_count * 8;
        if (ctas > cap) ctas = cap;
        launch_dependent(transpose_small_kernel, (unsigned)ctas, 256, smem, st, p, pitch);
        return launch_status("b200_transpose_copy [small matrices, flat 16-byte copies]");
      }
    }
  }
  launch_dependent(transpose_tile_kernel<Tin, Tout>, grid, 256, 0, st, p);
  return launch_status("b200_transpose_copy [element tiles]");
}

template <typename Tin, typename Tout>
static int launch_cast(const void* x, void* y, long long n, float scale, int has_scale, bool vec, cudaStream_t st) {
  constexpr int V = Elem<Tin>::V;
  // 32 bytes a thread from 4096 units on, where that still makes 16 CTAs (SiLU bf16 of 1000 elements: 1.43 us, with
  // 32 bytes 1.84; of 65 536: 1.97 and 1.90)
  const bool wide = vec && aligned32(x) && aligned32(y) && n >= 4096 * 2 * V;
  const long long units = wide ? n / (2 * V) : (vec ? n / V : n);
  set_path_tag(wide ? "vector, 32 bytes" : (vec ? "vector" : "element-wise"));
  auto go = [&](auto act_tag) {
    constexpr int ACT = decltype(act_tag)::value;
    // GELU and SiLU: 20 CTAs per SM, four times what is resident (SiLU bf16 [32768, 1536]: 5 per SM 36.3 us, 10 35.6, 20 35.0)
    const long long per_cta = 256LL * (ACT >= 4 ? 2 : 4) / (wide ? 2 : 1);
    const long long blocks = vec ? (units + per_cta - 1) / per_cta : (units + 255) / 256;
    const unsigned grid = streaming_grid(256 * (blocks > 0 ? blocks : 1), ACT >= 4 && vec ? 20 : 128);
    if (wide) launch_dependent(cast_scale_kernel<Tin, Tout, 32, ACT>, grid, 256, 0, st, x, y, n, scale, has_scale);
    else if (vec) launch_dependent(cast_scale_kernel<Tin, Tout, 16, ACT>, grid, 256, 0, st, x, y, n, scale, has_scale);
    else launch_dependent(cast_scale_kernel<Tin, Tout, 0, ACT>, grid, 256, 0, st, x, y, n, scale, has_scale);
  };
  switch (has_scale & 14) {
    case 0: go(std::integral_constant<int, 0>{}); break;
    case 2: go(std::integral_constant<int, 2>{}); break;
    case 4: go(std::integral_constant<int, 4>{}); break;
    case 8: go(std::integral_constant<int, 8>{}); break;
    default: return fail(B200_ERR_INVALID, "b200_cast_scale: one activation at a time (mode %d)", has_scale);
  }
  return launch_status("b200_cast_scale");
}

}  // namespace b200

using namespace b200;

#define B200_DTYPE_PAIRS(MACRO)                                  \
  MACRO(float, float, B200_F32, B200_F32)                        \
  MACRO(__nv_bfloat16, __nv_bfloat16, B200_BF16, B200_BF16)      \
  MACRO(__half, __half, B200_F16, B200_F16)                      \
  MACRO(__nv_bfloat16, float, B200_BF16, B200_F32)               \
  MACRO(__half, float, B200_F16, B200_F32)                       \
  MACRO(float, __nv_bfloat16, B200_F32, B200_BF16)               \
  MACRO(float, __half, B200_F32, B200_F16)

extern "C" int b200_permute_copy(const void* x, void* y, const int64_t* out_shape, const int64_t* in_strides,
                                 int32_t in_dtype, int32_t out_dtype, double scale, int32_t has_scale,
                                 void* stream) {
  if (!x || !y || !out_shape || !in_strides) return fail(B200_ERR_INVALID, "b200_permute_copy: null argument");
  PermuteParams p;
  p.x = x; p.y = y; p.total = 1;
  for (int i = 0; i < 4; ++i) {
    if (out_shape[i] < 0) return fail(B200_ERR_INVALID, "b200_permute_copy: negative extent");
    p.shape[i] = out_shape[i];
    p.in_stride[i] = in_strides[i];
    p.total *= out_shape[i];
  }
  if (p.total == 0) return B200_OK;
  for (int i = 1; i < 4; ++i)
    if (out_shape[i] > 0x7fffffffLL) return fail(B200_ERR_UNSUPPORTED, "b200_permute_copy: extent beyond 2^31-1");
  p.scale = (float)scale; p.has_scale = has_scale ? 1 : 0;
  const int ib = dtype_size(in_dtype), ob = dtype_size(out_dtype);
  const int vin = 16 / ib;
  const int out_chunk = vin * ob < 16 ? vin * ob : 16;
  bool vec = in_strides[3] == 1 && out_shape[3] % vin == 0 && aligned16(x) &&
             reinterpret_cast<uintptr_t>(y) % out_chunk == 0;
  for (int i = 0; i < 3; ++i) vec = vec && (in_strides[i] * ib) % 16 == 0;
  p.d1 = make_fast_div(out_shape[1]);
  p.d2 = make_fast_div(out_shape[2]);
  p.d3 = make_fast_div(vec ? out_shape[3] / vin : out_shape[3]);
  cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
#define B200_CASE(TI, TO, DI, DO) if (in_dtype == DI && out_dtype == DO) return launch_permute<TI, TO>(p, vec, st);
  B200_DTYPE_PAIRS(B200_CASE)
#undef B200_CASE
  return fail(B200_ERR_UNSUPPORTED, "b200_permute_copy: dtype pair (%d -> %d) not built", in_dtype, out_dtype);
}

extern "C" int b200_transpose_copy(const void* x, void* y, int64_t batch, int64_t rows, int64_t cols,
                                   int64_t in_batch_stride, int64_t in_row_stride, int32_t in_dtype,
                                   int32_t out_dtype, double scale, int32_t has_scale, void* stream) {
  if (!x || !y) return fail(B200_ERR_INVALID, "b200_transpose_copy: null argument");
  if (batch < 0 || rows < 0 || cols < 0) return fail(B200_ERR_INVALID, "b200_transpose_copy: negative size");
  if (batch == 0 || rows == 0 || cols == 0) return B200_OK;
  if (batch > 65535 || (rows + 63) / 64 > 65535)
    return fail(B200_ERR_UNSUPPORTED, "b200_transpose_copy: grid too large (fold batch dimensions)");
  TransposeParams p;
  p.x = x; p.y = y; p.batch = batch; p.P = rows; p.C = cols;
  p.in_batch_stride = in_batch_stride; p.in_row_stride = in_row_stride;
  p.scale = (float)scale; p.has_scale = has_scale ? 1 : 0;
  cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
#define B200_CASE(TI, TO, DI, DO) if (in_dtype == DI && out_dtype == DO) return launch_transpose<TI, TO>(p, st);
  B200_DTYPE_PAIRS(B200_CASE)
#undef B200_CASE
  return fail(B200_ERR_UNSUPPORTED, "b200_transpose_copy: dtype pair (%d -> %d) not built", in_dtype, out_dtype);
}

extern "C" int b200_cast_scale(const void* x, void* y, int64_t n, int32_t in_dtype, int32_t out_dtype,
                               double scale, int32_t has_scale, void* stream) {
  if (n < 0) return fail(B200_ERR_INVALID, "b200_cast_scale: negative size");
  if (n == 0) return B200_OK;
  if (!x || !y) return fail(B200_ERR_INVALID, "b200_cast_scale: null argument");
  const int ib = dtype_size(in_dtype), ob = dtype_size(out_dtype);
  const int vin = 16 / ib;
  const int out_chunk = vin * ob < 16 ? vin * ob : 16;
  const bool vec = aligned16(x) && reinterpret_cast<uintptr_t>(y) % out_chunk == 0;
  cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
#define B200_CASE(TI, TO, DI, DO) \
  if (in_dtype == DI && out_dtype == DO) return launch_cast<TI, TO>(x, y, n, (float)scale, has_scale & 15, vec, st);
  B200_DTYPE_PAIRS(B200_CASE)
#undef B200_CASE
  return fail(B200_ERR_UNSUPPORTED, "b200_cast_scale: dtype pair (%d -> %d) not built", in_dtype, out_dtype);
}
