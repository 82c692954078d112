// One generation step of an attention decoder: a single new position for each of up to 16 rows.
//
// Such a step reads every weight once and does a handful of FLOPs per byte, so it is bounded by the weights' trip from HBM and,
// for small models, by launches.  The tile GEMMs do not fit: 128 rows of mostly padding per MMA, one block per 128 or 256 output
// columns (12 blocks for a 3072-wide projection).  Here a block owns 16 (or 64) output columns, weights go from global memory
// straight into the operand registers of mma.sync (every 16-byte load feeds two MMAs; the contraction index is permuted the same
// way on both sides, so no shuffling is needed) and the rows of x sit in shared memory.  Five kernels per decoder block:
//     norm + query/key/value projection;  rotary + cache append + attention;  output projection + residual;
//     norm + first MLP layer + activation;  second MLP layer + residual
// launched from one host call with programmatic stream serialization: a kernel's blocks start while the previous kernel drains,
// prefetch their first weights (which depend on nothing) and only then wait for its results.
#include "common.cuh"
#include "activations.cuh"
#include <cooperative_groups.h>

namespace {
using bf16 = __nv_bfloat16;
namespace cg = cooperative_groups;
constexpr int kWarps = 8, kThreads = 32 * kWarps;

__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void pdl_trigger() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ uint4 load_stream(const void* p) {
  uint4 v;
  asm volatile("ld.global.nc.L1::no_allocate.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p));
  return v;
}
__device__ __forceinline__ void mma16816(float* c, uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
  asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
               : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3]) : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
__device__ __forceinline__ const uint32_t* words(const uint4& v) { return reinterpret_cast<const uint32_t*>(&v); }

enum NormKind : int { kNormNone = 0, kNormRms = 1, kNormLayer = 2, kNormZeroCentered = 4 };

// ---- y = norm(x) W^T, W [N, K] -----------------------------------------------------------------------------------------
struct NkArgs {
  const bf16 *w, *bias, *x, *norm_w, *norm_b, *residual;
  void* out;
  int m, n, k, norm, act, out_f32;
  float eps;
};

// Rows of x into shared memory (row stride k + 32: 16-byte reads of eight rows without bank conflicts), normalised.  One to eight
// warps share a row.
__device__ void stage_rows(bf16* xs, const NkArgs& a) {
  __shared__ float part[16][8];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, stride = a.k + 32, vecs = a.k / 8;
  const int wpr = a.m == 1 ? 8 : a.m == 2 ? 4 : a.m <= 4 ? 2 : 1, piece = warp % wpr, kind = a.norm & 3;
  auto each = [&](auto&& fn) {
    for (int row = warp / wpr; row < a.m; row += kWarps / wpr)
      for (int v = piece * 32 + lane; v < vecs; v += wpr * 32) fn(row, v);
  };
  auto reduce = [&](auto&& value) {  // row sums of value(row, vector) into part[row][0..wpr)
    for (int row = warp / wpr; row < a.m; row += kWarps / wpr) {
      float s = 0.f;
      for (int v = piece * 32 + lane; v < vecs; v += wpr * 32) s += value(row, v);
      s = flb::warp_sum(s);
      if (lane == 0) part[row][piece] = s;
    }
  };
  auto total = [&](int row) {
    float s = 0.f;
    for (int i = 0; i < wpr; ++i) s += part[row][i];
    return s;
  };
  each([&](int row, int v) { *reinterpret_cast<uint4*>(xs + row * stride + v * 8) = *reinterpret_cast<const uint4*>(a.x + (long long)row * a.k + v * 8); });
  if (kind != kNormNone) {  // a thread only re-reads what it wrote itself
    float mean[16];
#pragma unroll
    for (int i = 0; i < 16; ++i) mean[i] = 0.f;
    if (kind == kNormLayer) {
      reduce([&](int row, int v) {
        float f[8], s = 0.f;
        flb::unpack8(*reinterpret_cast<const flb::bf16x8*>(xs + row * stride + v * 8), f);
#pragma unroll
        for (int i = 0; i < 8; ++i) s += f[i];
        return s;
      });
      __syncthreads();
#pragma unroll
      for (int i = 0; i < 16; ++i)
        if (i < a.m) mean[i] = total(i) / a.k;
      __syncthreads();
    }
    auto mean_of = [&](int row) {
      float r = 0.f;
#pragma unroll
      for (int i = 0; i < 16; ++i)
        if (i == row) r = mean[i];
      return r;
    };
    reduce([&](int row, int v) {
      float f[8], s = 0.f;
      const float mu = mean_of(row);
      flb::unpack8(*reinterpret_cast<const flb::bf16x8*>(xs + row * stride + v * 8), f);
#pragma unroll
      for (int i = 0; i < 8; ++i) s += (f[i] - mu) * (f[i] - mu);
      return s;
    });
    __syncthreads();
    const float shift = (a.norm & kNormZeroCentered) ? 1.f : 0.f;
    each([&](int row, int v) {
      float f[8], w[8];
      const float mu = mean_of(row), rstd = rsqrtf(total(row) / a.k + a.eps);
      bf16* at = xs + row * stride + v * 8;
      flb::unpack8(*reinterpret_cast<const flb::bf16x8*>(at), f);
#pragma unroll
      for (int i = 0; i < 8; ++i) f[i] = (f[i] - mu) * rstd;
      if (a.norm_w != nullptr) {
        flb::unpack8(*reinterpret_cast<const flb::bf16x8*>(a.norm_w + v * 8), w);
#pragma unroll
        for (int i = 0; i < 8; ++i) f[i] *= w[i] + shift;
      }
      if (a.norm_b != nullptr) {
        flb::unpack8(*reinterpret_cast<const flb::bf16x8*>(a.norm_b + v * 8), w);
#pragma unroll
        for (int i = 0; i < 8; ++i) f[i] += w[i];
      }
      *reinterpret_cast<flb::bf16x8*>(at) = flb::pack8(f);
    });
  }
  __syncthreads();
}

// TILES8: groups of eight rows of x (1 or 2).  GATED: W holds n gate rows, then n up rows; out = act(gate) * up.
// A warp takes every eighth 64-wide unit of K: 128-byte lines of 16 weight rows, `kUnits` units in flight.
template <int TILES8, bool GATED>
__global__ void __launch_bounds__(kThreads, 2) skinny_nk_kernel(const NkArgs a) {
  constexpr int H = GATED ? 2 : 1, kUnits = GATED ? 2 : 4, TOK = 8 * TILES8;
  extern __shared__ __align__(16) unsigned char raw[];
  bf16* xs = reinterpret_cast<bf16*>(raw);
  float* red = reinterpret_cast<float*>(raw + TOK * (a.k + 32) * 2);  // [warp][H][16][TOK]
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, g = lane >> 2, j = lane & 3, stride = a.k + 32;
  const int tiles = (a.n + 15) / 16, units = a.k / 64;
  uint4 w[H][kUnits][4];
  auto load = [&](int tile, int unit0) {
#pragma unroll
    for (int h = 0; h < H; ++h) {
      const int r0 = min(tile * 16 + g, a.n - 1) + h * a.n, r1 = min(tile * 16 + g + 8, a.n - 1) + h * a.n;
#pragma unroll
      for (int u = 0; u < kUnits; ++u) {
        const int unit = unit0 + u * kWarps;
        if (unit < units) {
          const bf16 *p0 = a.w + (long long)r0 * a.k + unit * 64 + j * 8, *p1 = a.w + (long long)r1 * a.k + unit * 64 + j * 8;
          w[h][u][0] = load_stream(p0);
          w[h][u][1] = load_stream(p1);
          w[h][u][2] = load_stream(p0 + 32);
          w[h][u][3] = load_stream(p1 + 32);
        }
      }
    }
  };
  if ((int)blockIdx.x < tiles) load(blockIdx.x, warp);
  pdl_wait();
  stage_rows(xs, a);
  for (int tile = blockIdx.x; tile < tiles; tile += gridDim.x) {
    float acc[H][TILES8][4];
#pragma unroll
    for (int h = 0; h < H; ++h)
#pragma unroll
      for (int t = 0; t < TILES8; ++t)
#pragma unroll
        for (int i = 0; i < 4; ++i) acc[h][t][i] = 0.f;
    for (int unit0 = warp; unit0 < units; unit0 += kUnits * kWarps) {
      if (unit0 != warp || tile != (int)blockIdx.x) load(tile, unit0);
#pragma unroll
      for (int u = 0; u < kUnits; ++u) {
        const int unit = unit0 + u * kWarps;
        if (unit >= units) break;
#pragma unroll
        for (int c = 0; c < 2; ++c)
#pragma unroll
          for (int t = 0; t < TILES8; ++t) {
            const uint4 x = *reinterpret_cast<const uint4*>(xs + (t * 8 + g) * stride + unit * 64 + c * 32 + j * 8);
#pragma unroll
            for (int h = 0; h < H; ++h) {
              const uint4 lo = w[h][u][2 * c], hi = w[h][u][2 * c + 1];
              mma16816(acc[h][t], lo.x, hi.x, lo.y, hi.y, x.x, x.y);
              mma16816(acc[h][t], lo.z, hi.z, lo.w, hi.w, x.z, x.w);
            }
          }
      }
    }
    if (tile + (int)gridDim.x >= tiles) pdl_trigger();
#pragma unroll
    for (int h = 0; h < H; ++h)
#pragma unroll
      for (int t = 0; t < TILES8; ++t) {
        float* r = red + ((warp * H + h) * 16 + g) * TOK + t * 8 + j * 2;
        *reinterpret_cast<float2*>(r) = make_float2(acc[h][t][0], acc[h][t][1]);
        *reinterpret_cast<float2*>(r + 8 * TOK) = make_float2(acc[h][t][2], acc[h][t][3]);
      }
    __syncthreads();
    for (int i = threadIdx.x; i < 16 * TOK; i += kThreads) {
      const int row = i & 15, token = i >> 4, col = tile * 16 + row;
      if (token < a.m && col < a.n) {
        float v[H];
#pragma unroll
        for (int h = 0; h < H; ++h) {
          v[h] = 0.f;
#pragma unroll
          for (int q = 0; q < kWarps; ++q) v[h] += red[((q * H + h) * 16 + row) * TOK + token];
          if (a.bias != nullptr) v[h] += __bfloat162float(a.bias[h * a.n + col]);
        }
        float y = GATED ? act_fwd(v[0], a.act) * v[H - 1] : act_fwd(v[0], a.act);
        const long long at = (long long)token * a.n + col;
        if (a.residual != nullptr) y += __bfloat162float(a.residual[at]);
        if (a.out_f32) reinterpret_cast<float*>(a.out)[at] = y;
        else reinterpret_cast<bf16*>(a.out)[at] = __float2bfloat16_rn(y);
      }
    }
    __syncthreads();
  }
}

// ---- y = x W + residual, W [K, N] --------------------------------------------------------------------------------------
// A block owns 64 output columns and a share of K; the blocks of a cluster share the columns and add up over distributed shared
// memory.  Two neighbouring weight rows are interleaved into operand registers with byte permutes: accumulator tile t of a lane
// group g holds output columns 8 g + 2 t and 8 g + 2 t + 1.
struct KnArgs {
  const bf16 *w, *bias, *x, *residual;
  bf16* out;
  int m, n, k;
};
template <int TILES8>
__global__ void __launch_bounds__(kThreads, 2) skinny_kn_kernel(const KnArgs a) {
  constexpr int TOK = 8 * TILES8, kBatch = 4;
  extern __shared__ __align__(16) unsigned char raw[];
  cg::cluster_group cluster = cg::this_cluster();
  const int ranks = cluster.num_blocks(), rank = cluster.block_rank();
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, g = lane >> 2, j = lane & 3, n0 = blockIdx.y * 64;
  const int steps = a.k / 16, begin = (int)((long long)steps * rank / ranks), end = (int)((long long)steps * (rank + 1) / ranks);
  const int slice = ((steps + ranks - 1) / ranks) * 16, stride = slice + 8;
  float* red = reinterpret_cast<float*>(raw);                 // [warp][64][TOK], then the block's sums [64][TOK]
  bf16* xs = reinterpret_cast<bf16*>(raw + kWarps * 64 * TOK * 4);
  uint4 w[kBatch][4];
  auto load = [&](int step0) {
#pragma unroll
    for (int b = 0; b < kBatch; ++b) {
      const int step = step0 + b * kWarps;
      if (step < end) {
        const bf16* p = a.w + (long long)(step * 16 + 2 * j) * a.n + n0 + g * 8;
        w[b][0] = load_stream(p);
        w[b][1] = load_stream(p + a.n);
        w[b][2] = load_stream(p + 8ll * a.n);
        w[b][3] = load_stream(p + 9ll * a.n);
      }
    }
  };
  load(begin + warp);
  pdl_wait();
  const int cols = (end - begin) * 16;
  for (int i = threadIdx.x; i < a.m * cols / 8; i += kThreads) {
    const int row = i / (cols / 8), c = (i % (cols / 8)) * 8;
    *reinterpret_cast<uint4*>(xs + row * stride + c) = *reinterpret_cast<const uint4*>(a.x + (long long)row * a.k + begin * 16 + c);
  }
  __syncthreads();
  float acc[4][TILES8][4];
#pragma unroll
  for (int t = 0; t < 4; ++t)
#pragma unroll
    for (int n = 0; n < TILES8; ++n)
#pragma unroll
      for (int i = 0; i < 4; ++i) acc[t][n][i] = 0.f;
  for (int step0 = begin + warp; step0 < end; step0 += kBatch * kWarps) {
    if (step0 != begin + warp) load(step0);
#pragma unroll
    for (int b = 0; b < kBatch; ++b) {
      const int step = step0 + b * kWarps;
      if (step >= end) break;
      uint32_t x0[TILES8], x1[TILES8];
#pragma unroll
      for (int n = 0; n < TILES8; ++n) {
        const uint32_t* p = reinterpret_cast<const uint32_t*>(xs + (n * 8 + g) * stride + (step - begin) * 16 + j * 2);
        x0[n] = p[0];
        x1[n] = p[4];
      }
#pragma unroll
      for (int t = 0; t < 4; ++t) {
        const uint32_t r0 = words(w[b][0])[t], r1 = words(w[b][1])[t], r2 = words(w[b][2])[t], r3 = words(w[b][3])[t];
        const uint32_t a0 = __byte_perm(r0, r1, 0x5410), a1 = __byte_perm(r0, r1, 0x7632), a2 = __byte_perm(r2, r3, 0x5410), a3 = __byte_perm(r2, r3, 0x7632);
#pragma unroll
        for (int n = 0; n < TILES8; ++n) mma16816(acc[t][n], a0, a1, a2, a3, x0[n], x1[n]);
      }
    }
  }
  pdl_trigger();
#pragma unroll
  for (int t = 0; t < 4; ++t)
#pragma unroll
    for (int n = 0; n < TILES8; ++n) {
      float* r = red + (warp * 64 + 8 * g + 2 * t) * TOK + n * 8 + j * 2;
      *reinterpret_cast<float2*>(r) = make_float2(acc[t][n][0], acc[t][n][1]);
      *reinterpret_cast<float2*>(r + TOK) = make_float2(acc[t][n][2], acc[t][n][3]);
    }
  __syncthreads();
  for (int i = threadIdx.x; i < 64 * TOK; i += kThreads) {
    float s = 0.f;
#pragma unroll
    for (int q = 0; q < kWarps; ++q) s += red[q * 64 * TOK + i];
    red[i] = s;  // only this thread reads or writes element i of warp 0's part
  }
  cluster.sync();
  for (int i = rank * kThreads + threadIdx.x; i < 64 * TOK; i += ranks * kThreads) {
    const int col = i & 63, token = i >> 6;
    if (token < a.m) {
      float y = 0.f;
      for (int r = 0; r < ranks; ++r) y += cluster.map_shared_rank(red, r)[col * TOK + token];
      if (a.bias != nullptr) y += __bfloat162float(a.bias[n0 + col]);
      const long long at = (long long)token * a.n + n0 + col;
      if (a.residual != nullptr) y += __bfloat162float(a.residual[at]);
      a.out[at] = __float2bfloat16_rn(y);
    }
  }
  cluster.sync();  // the peers may still be reading this block's sums
}
}  // namespace

// ---- rotary + cache append + attention of one position per row ----------------------------------------------------------
// Block = (share of the keys, key/value head, row); the blocks of a cluster split the cached keys between them (four warps each, 16
// keys at a time) and merge their softmax statistics and outputs over distributed shared memory.  The query heads of the group
// are the 16 MMA rows.  Bounded by the cache's bytes for long contexts, by the chain of latencies for short ones.
namespace {
struct AttentionArgs {
  const bf16* qkv;    // [rows][(heads + 2 kv_heads) * D], not yet rotated
  bf16* cache;        // this layer's [rows][capacity][2 kv_heads * D]: keys, then values
  const int* pads;    // left padding of every row
  const float* table; // rotary [position][rot_dim]: cosines, then sines
  bf16* out;          // [rows][heads * D]
  int length, capacity, heads, kv_heads, rot_dim, window;
  float scale_log2;
};
constexpr int kAttnWarps = 4;

template <int D>
struct DecodeAttnSmem {
  bf16 q[16][D + 8];
  bf16 knew[D], vnew[D];
  float m[kAttnWarps][16], l[kAttnWarps][16];
  float o[kAttnWarps][16][D + 4];
  float mc[16], lc[16];
};

template <int D>
__global__ void __launch_bounds__(kAttnWarps * 32) decode_attention_kernel(const AttentionArgs a) {
  extern __shared__ __align__(16) unsigned char raw[];
  DecodeAttnSmem<D>& s = *reinterpret_cast<DecodeAttnSmem<D>*>(raw);
  cg::cluster_group cluster = cg::this_cluster();
  const int ranks = cluster.num_blocks(), rank = cluster.block_rank(), kv = blockIdx.y, row = blockIdx.z;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, g = lane >> 2, j = lane & 3;
  const int group = a.heads / a.kv_heads, width = 2 * a.kv_heads * D;
  pdl_wait();
  const int pad = a.pads[row], position = a.length - pad, half = a.rot_dim / 2;
  const bf16* const qkv = a.qkv + (long long)row * (a.heads + 2 * a.kv_heads) * D;
  bf16* const cache = a.cache + (long long)row * a.capacity * width + kv * D;
  const float* const table = a.table + (long long)position * a.rot_dim;
  auto rotated = [&](const bf16* head, int d) {
    const float x = __bfloat162float(head[d]);
    if (d >= a.rot_dim) return x;
    const int i = d < half ? d : d - half;
    const float c = table[i], sn = table[half + i], other = __bfloat162float(head[d < half ? d + half : d - half]);
    return d < half ? x * c - other * sn : x * c + other * sn;
  };
  for (int i = threadIdx.x; i < 16 * D; i += kAttnWarps * 32) {
    const int h = i / D, d = i % D;
    s.q[h][d] = h < group ? __float2bfloat16_rn(rotated(qkv + (kv * group + h) * D, d)) : __float2bfloat16_rn(0.f);
  }
  for (int d = threadIdx.x; d < D; d += kAttnWarps * 32) {
    const bf16 k = __float2bfloat16_rn(rotated(qkv + (a.heads + kv) * D, d)), v = qkv[(a.heads + a.kv_heads + kv) * D + d];
    s.knew[d] = k;
    s.vnew[d] = v;
    if (rank == 0) {  // nobody reads this position from the cache in this launch
      cache[(long long)a.length * width + d] = k;
      cache[(long long)a.length * width + a.kv_heads * D + d] = v;
    }
  }
  __syncthreads();
  uint4 q[D / 32][2];
#pragma unroll
  for (int b = 0; b < D / 32; ++b) {
    q[b][0] = *reinterpret_cast<const uint4*>(&s.q[g][b * 32 + j * 8]);
    q[b][1] = *reinterpret_cast<const uint4*>(&s.q[g + 8][b * 32 + j * 8]);
  }
  float m[2] = {-INFINITY, -INFINITY}, l[2] = {0.f, 0.f}, o[D / 8][4];
#pragma unroll
  for (int n = 0; n < D / 8; ++n)
#pragma unroll
    for (int i = 0; i < 4; ++i) o[n][i] = 0.f;
  if (rank == 0 && warp == 0) {  // the new position itself
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      float dot = 0.f;  // the four lanes of row g (g + 8) share the head's dimensions
      for (int d = j; d < D; d += 4) dot += __bfloat162float(s.q[g + 8 * i][d]) * __bfloat162float(s.knew[d]);
      dot += __shfl_xor_sync(0xffffffffu, dot, 1);
      dot += __shfl_xor_sync(0xffffffffu, dot, 2);
      m[i] = dot * a.scale_log2;
      l[i] = 1.f;
    }
#pragma unroll
    for (int n = 0; n < D / 8; ++n) {
      const int d = (n / 8) * 64 + n % 8;  // accumulator column c of tile n is dimension d + 8 c
      o[n][0] = o[n][2] = __bfloat162float(s.vnew[d + 8 * (2 * j)]);
      o[n][1] = o[n][3] = __bfloat162float(s.vnew[d + 8 * (2 * j + 1)]);
    }
  }
  const int begin = a.window > 0 ? max(pad, a.length + 1 - a.window) : pad, end = a.length;
  const bf16* const keys = cache;
  const bf16* const values = cache + a.kv_heads * D;
  for (int base = begin + (rank * kAttnWarps + warp) * 16; base < end; base += ranks * kAttnWarps * 16) {
    float sc[2][4];
    uint4 kr[2][D / 32];
#pragma unroll
    for (int t = 0; t < 2; ++t) {
      const bf16* p = keys + (long long)min(base + t * 8 + g, end - 1) * width + j * 8;
#pragma unroll
      for (int b = 0; b < D / 32; ++b) kr[t][b] = *reinterpret_cast<const uint4*>(p + b * 32);
    }
    uint4 vr[D / 64][4];
#pragma unroll
    for (int r = 0; r < 4; ++r) {
      const bf16* p = values + (long long)min(base + 2 * j + (r & 1) + (r >> 1) * 8, end - 1) * width + g * 8;
#pragma unroll
      for (int nb = 0; nb < D / 64; ++nb) vr[nb][r] = *reinterpret_cast<const uint4*>(p + nb * 64);
    }
#pragma unroll
    for (int t = 0; t < 2; ++t) {
#pragma unroll
      for (int i = 0; i < 4; ++i) sc[t][i] = 0.f;
#pragma unroll
      for (int b = 0; b < D / 32; ++b) {
        mma16816(sc[t], q[b][0].x, q[b][1].x, q[b][0].y, q[b][1].y, kr[t][b].x, kr[t][b].y);
        mma16816(sc[t], q[b][0].z, q[b][1].z, q[b][0].w, q[b][1].w, kr[t][b].z, kr[t][b].w);
      }
#pragma unroll
      for (int i = 0; i < 4; ++i) sc[t][i] = base + t * 8 + 2 * j + (i & 1) < end ? sc[t][i] * a.scale_log2 : -INFINITY;
    }
    float alpha[2];
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      float top = fmaxf(fmaxf(sc[0][2 * i], sc[0][2 * i + 1]), fmaxf(sc[1][2 * i], sc[1][2 * i + 1]));
      top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, 1));
      top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, 2));
      const float next = fmaxf(m[i], top);  // finite: base < end
      alpha[i] = exp2f(m[i] - next);
      m[i] = next;
      float sum = 0.f;
#pragma unroll
      for (int t = 0; t < 2; ++t) {
        sc[t][2 * i] = exp2f(sc[t][2 * i] - next);
        sc[t][2 * i + 1] = exp2f(sc[t][2 * i + 1] - next);
        sum += sc[t][2 * i] + sc[t][2 * i + 1];
      }
      sum += __shfl_xor_sync(0xffffffffu, sum, 1);
      sum += __shfl_xor_sync(0xffffffffu, sum, 2);
      l[i] = l[i] * alpha[i] + sum;
    }
    auto pack = [](float x, float y) { __nv_bfloat162 v = __floats2bfloat162_rn(x, y); return *reinterpret_cast<uint32_t*>(&v); };
    const uint32_t p0 = pack(sc[0][0], sc[0][1]), p1 = pack(sc[0][2], sc[0][3]), p2 = pack(sc[1][0], sc[1][1]), p3 = pack(sc[1][2], sc[1][3]);
#pragma unroll
    for (int n = 0; n < D / 8; ++n) {
      o[n][0] *= alpha[0]; o[n][1] *= alpha[0]; o[n][2] *= alpha[1]; o[n][3] *= alpha[1];
      const int nb = n / 8, t = n % 8;
      const uint32_t sel = (t & 1) ? 0x7632 : 0x5410;
      const uint32_t b0 = __byte_perm(words(vr[nb][0])[t / 2], words(vr[nb][1])[t / 2], sel), b1 = __byte_perm(words(vr[nb][2])[t / 2], words(vr[nb][3])[t / 2], sel);
      mma16816(o[n], p0, p1, p2, p3, b0, b1);
    }
  }
  pdl_trigger();
  if (j == 0) {
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      s.m[warp][g + 8 * i] = m[i];
      s.l[warp][g + 8 * i] = l[i];
    }
  }
#pragma unroll
  for (int n = 0; n < D / 8; ++n) {
    const int d = (n / 8) * 64 + n % 8;
#pragma unroll
    for (int i = 0; i < 4; ++i) s.o[warp][g + 8 * (i >> 1)][d + 8 * (2 * j + (i & 1))] = o[n][i];
  }
  __syncthreads();
  if (threadIdx.x < 16) {
    const int h = threadIdx.x;
    float top = -INFINITY, sum = 0.f;
#pragma unroll
    for (int w = 0; w < kAttnWarps; ++w) top = fmaxf(top, s.m[w][h]);
#pragma unroll
    for (int w = 0; w < kAttnWarps; ++w) {
      const float f = s.m[w][h] == -INFINITY ? 0.f : exp2f(s.m[w][h] - top);
      s.m[w][h] = f;
      sum += f * s.l[w][h];
    }
    s.mc[h] = top;
    s.lc[h] = sum;
  }
  __syncthreads();
  for (int i = threadIdx.x; i < group * D; i += kAttnWarps * 32) {
    const int h = i / D, d = i % D;
    float v = 0.f;
#pragma unroll
    for (int w = 0; w < kAttnWarps; ++w) v += s.m[w][h] * s.o[w][h][d];
    s.o[0][h][d] = v;
  }
  cluster.sync();
  for (int i = rank * kAttnWarps * 32 + threadIdx.x; i < group * D; i += ranks * kAttnWarps * 32) {
    const int h = i / D, d = i % D;
    float top = -INFINITY, sum = 0.f, v = 0.f;
    for (int r = 0; r < ranks; ++r) top = fmaxf(top, cluster.map_shared_rank(s.mc, r)[h]);
    for (int r = 0; r < ranks; ++r) {
      const float mr = cluster.map_shared_rank(s.mc, r)[h];
      if (mr == -INFINITY) continue;
      const float f = exp2f(mr - top);
      sum += f * cluster.map_shared_rank(s.lc, r)[h];
      v += f * cluster.map_shared_rank(&s.o[0][0][0], r)[h * (D + 4) + d];
    }
    a.out[(long long)row * a.heads * D + (kv * group + h) * D + d] = __float2bfloat16_rn(v / sum);
  }
  cluster.sync();
}

__global__ void decode_embedding_kernel(const long long* __restrict__ ids, const bf16* __restrict__ table, bf16* __restrict__ out, int hidden, int vocab, float scale) {
  const long long id = ids[blockIdx.x];
  for (int v = threadIdx.x; v < hidden / 8; v += blockDim.x) {
    float f[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) f[i] = 0.f;
    if (id >= 0 && id < vocab) {
      flb::unpack8(*reinterpret_cast<const flb::bf16x8*>(table + id * hidden + v * 8), f);
#pragma unroll
      for (int i = 0; i < 8; ++i) f[i] *= scale;
    }
    *reinterpret_cast<flb::bf16x8*>(out + (long long)blockIdx.x * hidden + v * 8) = flb::pack8(f);
  }
}

// ---- host ----------------------------------------------------------------------------------------------------------
constexpr int kSmemLimit = 220 * 1024;

template <typename... Params, typename... Values>
cudaError_t launch(void (*kernel)(Params...), dim3 grid, int threads, int smem, int cluster, cudaStream_t stream, Values... values) {
  cudaLaunchConfig_t config{};
  config.gridDim = grid;
  config.blockDim = dim3(threads);
  config.dynamicSmemBytes = smem;
  config.stream = stream;
  cudaLaunchAttribute attributes[2];
  attributes[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attributes[0].val.programmaticStreamSerializationAllowed = 1;
  attributes[1].id = cudaLaunchAttributeClusterDimension;
  attributes[1].val.clusterDim.x = cluster;
  attributes[1].val.clusterDim.y = attributes[1].val.clusterDim.z = 1;
  config.attrs = attributes;
  config.numAttrs = 2;
  return cudaLaunchKernelEx(&config, kernel, values...);
}

int nk_smem(int tok, int k, bool gated) { return tok * (k + 32) * 2 + kWarps * (gated ? 2 : 1) * 16 * tok * 4; }
int kn_smem(int tok, int k, int ranks) { return kWarps * 64 * tok * 4 + tok * (((k / 16 + ranks - 1) / ranks) * 16 + 8) * 2; }
// Enough blocks for the chip (148 SMs, two each), at least two batches of loads per warp left for each.
int kn_ranks(int n, int k) {
  int ranks = 1;
  while (ranks < 8 && (n / 64) * ranks < 256 && k / 16 / (2 * ranks) >= 2 * kWarps) ranks *= 2;
  return ranks;
}

template <int TILES8, bool GATED>
cudaError_t run_nk(const NkArgs& a, cudaStream_t stream) {
  static const cudaError_t ready = cudaFuncSetAttribute(skinny_nk_kernel<TILES8, GATED>, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmemLimit);
  if (ready != cudaSuccess) return ready;
  const int smem = nk_smem(8 * TILES8, a.k, GATED), tiles = (a.n + 15) / 16, resident = smem <= 110 * 1024 ? 296 : 148;
  return launch(skinny_nk_kernel<TILES8, GATED>, dim3(tiles < resident ? tiles : resident), kThreads, smem, 1, stream, a);
}
cudaError_t run_nk(const NkArgs& a, bool gated, cudaStream_t stream) {
  if (a.m <= 8) return gated ? run_nk<1, true>(a, stream) : run_nk<1, false>(a, stream);
  return gated ? run_nk<2, true>(a, stream) : run_nk<2, false>(a, stream);
}
template <int TILES8>
cudaError_t run_kn(const KnArgs& a, cudaStream_t stream) {
  static const cudaError_t ready = cudaFuncSetAttribute(skinny_kn_kernel<TILES8>, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmemLimit);
  if (ready != cudaSuccess) return ready;
  const int ranks = kn_ranks(a.n, a.k);
  return launch(skinny_kn_kernel<TILES8>, dim3(ranks, a.n / 64), kThreads, kn_smem(8 * TILES8, a.k, ranks), ranks, stream, a);
}
template <int D>
cudaError_t run_attention(const AttentionArgs& a, int rows, cudaStream_t stream) {
  static const cudaError_t ready = cudaFuncSetAttribute(decode_attention_kernel<D>, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmemLimit);
  if (ready != cudaSuccess) return ready;
  // split the keys until the chip is full, but not below one 16-key step per warp
  const int keys = a.window > 0 && a.window < a.length ? a.window : a.length;
  int ranks = 1;
  while (ranks < 8 && rows * a.kv_heads * ranks < 256 && keys >= 2 * ranks * kAttnWarps * 16) ranks *= 2;
  return launch(decode_attention_kernel<D>, dim3(ranks, a.kv_heads, rows), kAttnWarps * 32, (int)sizeof(DecodeAttnSmem<D>), ranks, stream, a);
}
}  // namespace

// One decoder block as the host describes it (mirrored by a ctypes structure).
struct FlbDecodeLayer {
  const bf16 *norm1_w, *norm1_b, *qkv_w, *qkv_b, *dense_w, *dense_b, *norm2_w, *norm2_b, *w1, *b1, *w2, *b2;
  const float* table;
  int norm1, norm2, heads, kv_heads, head_dim, rot_dim, window, ffn, gated, act;
  float eps1, eps2, scale;
};

// Whether every kernel of a step fits: rows of x and of the MLP's inner activation in shared memory.
FLB_API int flb_decode_supported(const FlbDecodeLayer* layers, int count, int hidden, int rows) {
  if (rows < 1 || rows > 16 || hidden % 64) return 0;
  const int tok = rows <= 8 ? 8 : 16;
  for (int i = 0; i < count; ++i) {
    const FlbDecodeLayer& l = layers[i];
    const int width = l.heads * l.head_dim;
    if ((l.head_dim != 64 && l.head_dim != 128) || l.heads % l.kv_heads || l.heads / l.kv_heads > 16 || width % 64 || l.ffn % 16) return 0;
    if (nk_smem(tok, hidden, true) > kSmemLimit || nk_smem(tok, width, false) > kSmemLimit || kn_smem(tok, l.ffn, kn_ranks(hidden, l.ffn)) > kSmemLimit) return 0;
  }
  return 1;
}

// `ids` [rows]; `cache`: [layers][rows][capacity][2 kv_heads head_dim] with `cache_layer` elements between layers, the first `length`
// positions of every row filled, position `length` written here; `pads` [rows] on the device.  `x`, `x2` [rows, hidden], `qkv`, `attn`,
// `inner` hold the intermediates; `logits` [rows, vocab] fp32.
FLB_API int flb_decode_step(const FlbDecodeLayer* layers, int count, const long long* ids, int rows, const bf16* embedding, float embedding_scale,
                            int hidden, int vocab, const bf16* final_w, const bf16* final_b, int final_norm, float final_eps, const bf16* head_w,
                            bf16* cache, long long cache_layer, int capacity, int length, const int* pads, bf16* x, bf16* x2, bf16* qkv, bf16* attn,
                            bf16* inner, float* logits, cudaStream_t stream) {
  if (!flb_decode_supported(layers, count, hidden, rows) || length >= capacity) return FLB_ERR_SHAPE;
  decode_embedding_kernel<<<rows, 128, 0, stream>>>(ids, embedding, x, hidden, vocab, embedding_scale);
  cudaError_t e = cudaGetLastError();
  for (int i = 0; i < count && e == cudaSuccess; ++i) {
    const FlbDecodeLayer& l = layers[i];
    const int width = l.heads * l.head_dim;
    NkArgs p{l.qkv_w, l.qkv_b, x, l.norm1_w, l.norm1_b, nullptr, qkv, rows, width + 2 * l.kv_heads * l.head_dim, hidden, l.norm1, 0, 0, l.eps1};
    if ((e = run_nk(p, false, stream)) != cudaSuccess) break;
    AttentionArgs at{qkv, cache + i * cache_layer, pads, l.table, attn, length, capacity, l.heads, l.kv_heads, l.rot_dim, l.window, l.scale * 1.4426950408889634f};
    if ((e = l.head_dim == 64 ? run_attention<64>(at, rows, stream) : run_attention<128>(at, rows, stream)) != cudaSuccess) break;
    NkArgs d{l.dense_w, l.dense_b, attn, nullptr, nullptr, x, x2, rows, hidden, width, kNormNone, 0, 0, 0.f};
    if ((e = run_nk(d, false, stream)) != cudaSuccess) break;
    NkArgs u{l.w1, l.b1, x2, l.norm2_w, l.norm2_b, nullptr, inner, rows, l.ffn, hidden, l.norm2, l.act, 0, l.eps2};
    if ((e = run_nk(u, l.gated != 0, stream)) != cudaSuccess) break;
    KnArgs w{l.w2, l.b2, inner, x2, x, rows, hidden, l.ffn};
    e = rows <= 8 ? run_kn<1>(w, stream) : run_kn<2>(w, stream);
  }
  if (e == cudaSuccess) {
    NkArgs h{head_w, nullptr, x, final_w, final_b, nullptr, logits, rows, vocab, hidden, final_norm, 0, 1, final_eps};
    e = run_nk(h, false, stream);
  }
  if (e != cudaSuccess) return flb_record_cuda_error(e);
  return FLB_OK;
}
