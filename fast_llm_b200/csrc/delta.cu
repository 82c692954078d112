// Delta rule over packed documents: gated DeltaNet (one decay per token) and Kimi delta attention (one per key channel).
//
// Per head, with unit-scaled keys k^ and queries q^, decay sums c (from the start of the chunk), Gamma_t = exp(c_t) and
// pair(t, s) = exp(c_t - c_s) for s <= t (always <= 1), a chunk of 64 tokens entered with state S [dk, dv] is
//     N_ts = beta_s pair (k^_t . k^_s) for s < t,   P_ts = pair (q^_t . k^_s) for s <= t,   T = (I + N)^-1
//     U = T (V - Gamma K^ S)         O = Gamma Q^ S + P (beta U)         S' = Gamma_L S + K^T exp(c_L - c) (beta U)
// and its adjoint, entered with dS' from behind,
//     dU = beta (P^T dO + exp(c_L - c) K^ dS'),   dR = T^T dU (= dV),   dS = Gamma_L dS' + (Gamma Q^)^T dO - (Gamma K^)^T dR.
//
// Five kernels: `prepare` (all chunks at once: norms, decay sums, N, P, T), `scan_fwd` (chunk after chunk: U and the state
// entering every chunk), `output` (all chunks), `scan_bwd` (chunk after chunk, from the end: dR and dS'), `backward` (all
// chunks: dq, dk, dg, dbeta).  Only what hangs on the carried state is in the two sequential kernels.
//
// Precision is that of an fp32 product: an fp32 operand enters the tensor cores as the sum of three bf16 numbers (8 + 8 + 8
// mantissa bits) and the products down to 2^-24 are kept - three MMAs against an operand that is bf16 to begin with (q, k, v
// and dO are; the norm and, for one decay per token, the decay are row factors applied to the fp32 accumulators), six between
// two fp32 operands.  These are 64 x 64 x 128 pieces whose results feed the next piece from registers, in the transposed form
// [dv, ...] in which one MMA's accumulator layout is the next one's operand layout: warp-level mma.sync, a warp owning 16
// columns of dv, needs no exchange between warps at all.  What bounds the sequential kernels is that chain of dependent MMAs.
//
// Measured on a B200, 8192 tokens x 32 heads x 128, four documents: prepare 0.18, scan_fwd 0.28, output 0.16, scan_bwd 0.46, backward
// 0.98 ms (one document: the scans 0.68 and 0.93); the batched fp32 GEMM / triangular-solve formulation in PyTorch that this
// replaces took 8.3 ms forward and 12.2 backward.  One decay per channel, 4096 x 16 x 128, seven documents: 0.49 and 0.72 ms
// against 8.7 and about 14.
#include "common.cuh"
#include <cuda_bf16.h>

namespace {
using bf16 = __nv_bfloat16;
using bf162 = __nv_bfloat162;
constexpr int L = 64;                 // tokens per chunk
constexpr int TS = L + 8;             // shared-memory row stride (bf16) of a 64-wide tile: 16-byte rows, ldmatrix without bank conflicts
constexpr int kTri = 3 * L * L;       // one [3][64][64] set of planes
constexpr float kLog2e = 1.4426950408889634f;

__device__ __forceinline__ uint32_t smem_addr(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void cp16(void* dst, const void* src, bool valid) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(smem_addr(dst)), "l"(src), "r"(valid ? 16 : 0) : "memory");
}
__device__ __forceinline__ void cp4(void* dst, const void* src, bool valid) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(smem_addr(dst)), "l"(src), "r"(valid ? 4 : 0) : "memory");
}
__device__ __forceinline__ void cp_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

__device__ __forceinline__ void ldsm(uint32_t* r, uint32_t addr) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr) : "memory");
}
__device__ __forceinline__ void ldsm_t(uint32_t* r, uint32_t addr) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr) : "memory");
}
__device__ __forceinline__ void mma(float* c, const uint32_t* a, uint32_t b0, uint32_t b1) {
  asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
               : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3]) : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
// Four 8x8 blocks of a row-major tile X (row stride `rs` elements) at (r0, c0), in the order of the two MMA operand layouts.
//   load_nk  B operand, X[n][k]; also the A operand of X[m][k] transposed (X[k][m] with load_km below is its counterpart)
//   load_kn  B operand, X[k][n] (transposing)
//   load_mk  A operand, X[m][k]
//   load_km  A operand, X[k][m] (transposing); also two accumulator tiles [m 16][k 8] of X^T as packed bf16 pairs
__device__ __forceinline__ void load_nk(uint32_t* r, const bf16* x, int rs, int n0, int k0, int lane) {
  ldsm(r, smem_addr(x + (n0 + (lane >> 4) * 8 + (lane & 7)) * rs + k0 + ((lane >> 3) & 1) * 8));
}
__device__ __forceinline__ void load_kn(uint32_t* r, const bf16* x, int rs, int k0, int n0, int lane) {
  ldsm_t(r, smem_addr(x + (k0 + ((lane >> 3) & 1) * 8 + (lane & 7)) * rs + n0 + (lane >> 4) * 8));
}
__device__ __forceinline__ void load_mk(uint32_t* r, const bf16* x, int rs, int m0, int k0, int lane) {
  ldsm(r, smem_addr(x + (m0 + ((lane >> 3) & 1) * 8 + (lane & 7)) * rs + k0 + (lane >> 4) * 8));
}
__device__ __forceinline__ void load_km(uint32_t* r, const bf16* x, int rs, int k0, int m0, int lane) {
  ldsm_t(r, smem_addr(x + (k0 + (lane >> 4) * 8 + (lane & 7)) * rs + m0 + ((lane >> 3) & 1) * 8));
}

__device__ __forceinline__ uint32_t bits(bf162 v) { return *reinterpret_cast<uint32_t*>(&v); }
__device__ __forceinline__ float2 floats(uint32_t v) {
  return make_float2(__uint_as_float(v << 16), __uint_as_float(v & 0xffff0000u));
}
// The pair (a, b) as three packed bf16 pairs whose sum is (a, b) to 24 bits.
__device__ __forceinline__ void split(float a, float b, uint32_t& hi, uint32_t& mid, uint32_t& lo) {
  hi = bits(__floats2bfloat162_rn(a, b));
  float2 f = floats(hi);
  a -= f.x;
  b -= f.y;
  mid = bits(__floats2bfloat162_rn(a, b));
  f = floats(mid);
  lo = bits(__floats2bfloat162_rn(a - f.x, b - f.y));
}
// A operand (16 x 16) from two neighbouring accumulator tiles, in three planes.
__device__ __forceinline__ void split_a(const float* c0, const float* c1, uint32_t (*a)[4]) {
  split(c0[0], c0[1], a[0][0], a[1][0], a[2][0]);
  split(c0[2], c0[3], a[0][1], a[1][1], a[2][1]);
  split(c1[0], c1[1], a[0][2], a[1][2], a[2][2]);
  split(c1[2], c1[3], a[0][3], a[1][3], a[2][3]);
}
// c[tile] += a * b[tile] for `nt` tiles, a in three planes and b in one (exact bf16) or three, smallest products first.  The tiles
// take turns inside each product, so that consecutive MMAs do not wait for one another.
template <int NB>
__device__ __forceinline__ void mma_tiles(float (*c)[4], const uint32_t (*a)[4], const uint32_t (*b)[NB][2], int nt) {
  auto product = [&](int pa, int pb) {
#pragma unroll
    for (int t = 0; t < 4; ++t)
      if (t < nt) mma(c[t], a[pa], b[t][pb][0], b[t][pb][1]);
  };
  if constexpr (NB == 3) {
    product(0, 2);
    product(1, 1);
  }
  product(2, 0);
  if constexpr (NB == 3) product(0, 1);
  product(1, 0);
  product(0, 0);
}
// The same with a exact and b in three planes, or both exact.
template <int NB>
__device__ __forceinline__ void mma_tiles_exact(float (*c)[4], const uint32_t* a, const uint32_t (*b)[NB][2], int nt) {
#pragma unroll
  for (int pl = NB - 1; pl >= 0; --pl)
#pragma unroll
    for (int t = 0; t < 4; ++t)
      if (t < nt) mma(c[t], a, b[t][pl][0], b[t][pl][1]);
}
// B fragments of the 16 columns n0..n0 + 15 (two tiles) in NB planes, `plane` elements apart: X[n][k], or X[k][n] (TRANS).
template <int NB, bool TRANS>
__device__ __forceinline__ void load_b(uint32_t (*b)[NB][2], const bf16* x, int plane, int rs, int n0, int k0, int lane) {
#pragma unroll
  for (int pl = 0; pl < NB; ++pl) {
    uint32_t r[4];
    if constexpr (TRANS) load_kn(r, x + pl * plane, rs, k0, n0, lane);
    else load_nk(r, x + pl * plane, rs, n0, k0, lane);
    b[0][pl][0] = r[0]; b[0][pl][1] = r[1]; b[1][pl][0] = r[2]; b[1][pl][1] = r[3];
  }
}

struct DeltaArgs {
  const bf16 *q, *k, *v;        // rows of heads; row strides in elements
  long long q_row, k_row, v_row;
  int heads, repeat;            // value heads; value heads per key head
  int dv;
  const float* g;               // log decay [tokens, heads] or [tokens, heads, dk]
  const float* beta;            // [tokens, heads]
  const int2* chunk;            // (first token, tokens) of every chunk
  const int* doc_chunk;         // [documents + 1] first chunk of every document; the last entry is the number of chunks
  int docs;
  int normalize;
  float scale;
  // prepared
  float* decay;                 // c * log2(e): [chunk][head][64] or [chunk][head][64][dk]
  float* norm_q;                // [chunk][head][64] row factors (softmax-style scale and 1 / norm)
  float* norm_k;
  bf16 *tri_t, *tri_p;          // [chunk][head][3][64][64]
  float* tri_n;                 // [chunk][head][64][64] N without beta (only for the backward)
  bf16 *k_in, *k_out, *q_in;    // per-channel decay: planes [chunk][head][3][64][dk] of k^ exp(c), k^ exp(c_L - c), q^ exp(c)
  // scans
  float* u;                     // [chunk][head][64][dv]
  float* state;                 // [chunk][head][dv][dk] state entering the chunk
  bf16* out;                    // [tokens, heads, dv]
  const bf16* dout;
  float* dr;                    // [chunk][head][64][dv]
  float* dstate;                // [chunk][head][dv][dk] adjoint of the state leaving the chunk
  bf16 *dq, *dk, *dvalue;       // [tokens, heads, dk | dv]
  float *dg, *dbeta;
};

// ---- chunk table ---------------------------------------------------------------------------------------------------
// Documents [cu[i], cu[i + 1]) and, behind the last, the trailing padding, each cut into chunks of 64 tokens.
__global__ void delta_chunks_kernel(const int* __restrict__ cu, int docs, int total, int2* __restrict__ chunk, int* __restrict__ doc_chunk) {
  __shared__ int warp_total[32];
  __shared__ int base;
  if (threadIdx.x == 0) base = 0;
  __syncthreads();
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  for (int d0 = 0; d0 < docs; d0 += blockDim.x) {
    const int d = d0 + threadIdx.x;
    int begin = 0, end = 0;
    if (d < docs) {
      // the last entry of the list is the padding behind the last document (or everything, without a list)
      begin = cu == nullptr ? 0 : min(cu[d], total);
      end = (cu == nullptr || d == docs - 1) ? total : min(cu[d + 1], total);
    }
    const int count = end > begin ? (end - begin + L - 1) / L : 0;
    int sum = count;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int other = __shfl_up_sync(0xffffffffu, sum, o);
      if (lane >= o) sum += other;
    }
    if (lane == 31) warp_total[warp] = sum;
    __syncthreads();
    int before = base;
    for (int w = 0; w < warp; ++w) before += warp_total[w];
    int first = before + sum - count;
    if (d < docs) doc_chunk[d] = first;
    for (int i = 0; i < count; ++i) chunk[first + i] = make_int2(begin + i * L, min(L, end - begin - i * L));
    __syncthreads();
    if (threadIdx.x == blockDim.x - 1) base = before + sum;
    __syncthreads();
  }
  if (threadIdx.x == 0) doc_chunk[docs] = base;
}

// ---- prepare -------------------------------------------------------------------------------------------------------
// One block of four warps per chunk and head.  T = (I + N)^-1 by forward substitution, one thread per column with the column
// in registers: 2016 multiply-adds per column, all blocks of an SM together a few per cent of what the scans cost.
template <int DK, bool CHANNEL>
struct PrepareSmem {
  static constexpr int KS = DK + 8;
  bf16 q[L * KS], k[L * KS];
  float n[L * (L + 4)];
  float c[CHANNEL ? L * (DK + 4) : L];
  float nq[L], nk[L], beta[L];
};

template <int DK, bool CHANNEL>
__global__ void __launch_bounds__(128) delta_prepare_kernel(const DeltaArgs p) {
  extern __shared__ __align__(16) unsigned char raw[];
  using Smem = PrepareSmem<DK, CHANNEL>;
  Smem& s = *reinterpret_cast<Smem*>(raw);
  constexpr int KS = Smem::KS, CS = DK + 4, NS = L + 4;
  const int ch = blockIdx.x, head = blockIdx.y;
  if (ch >= p.doc_chunk[p.docs]) return;
  const int2 span = p.chunk[ch];
  const int len = span.y, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const long long slot = (long long)ch * p.heads + head;
  const int key_head = head / p.repeat;
  for (int i = tid; i < L * DK / 8; i += 128) {
    const int t = i / (DK / 8), d = (i % (DK / 8)) * 8;
    const bool ok = t < len;
    const long long row = span.x + (ok ? t : 0);
    cp16(s.q + t * KS + d, p.q + row * p.q_row + key_head * DK + d, ok);
    cp16(s.k + t * KS + d, p.k + row * p.k_row + key_head * DK + d, ok);
  }
  cp_commit();
  if (tid < L) s.beta[tid] = tid < len ? p.beta[(long long)(span.x + tid) * p.heads + head] : 0.f;
  if constexpr (CHANNEL) {
    if (tid < DK) {
      float c = 0.f;
      const float* g = p.g + ((long long)span.x * p.heads + head) * DK + tid;
#pragma unroll 8
      for (int t = 0; t < L; ++t) {
        if (t < len) c += g[(long long)t * p.heads * DK];
        s.c[t * CS + tid] = c * kLog2e;
      }
    }
  } else if (warp == 0) {
    float a = lane < len ? p.g[(long long)(span.x + lane) * p.heads + head] : 0.f;
    float b = lane + 32 < len ? p.g[(long long)(span.x + lane + 32) * p.heads + head] : 0.f;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const float x = __shfl_up_sync(0xffffffffu, a, o), y = __shfl_up_sync(0xffffffffu, b, o);
      if (lane >= o) { a += x; b += y; }
    }
    b += __shfl_sync(0xffffffffu, a, 31);
    s.c[lane] = a * kLog2e;
    s.c[lane + 32] = b * kLog2e;
  }
  cp_wait<0>();
  __syncthreads();
  for (int t = warp * 16; t < warp * 16 + 16; ++t) {
    float sq = 0.f, sk = 0.f;
#pragma unroll
    for (int d = lane * 2; d < DK; d += 64) {
      const float2 a = floats(*reinterpret_cast<const uint32_t*>(s.q + t * KS + d)), b = floats(*reinterpret_cast<const uint32_t*>(s.k + t * KS + d));
      sq += a.x * a.x + a.y * a.y;
      sk += b.x * b.x + b.y * b.y;
    }
    sq = flb::warp_sum(sq);
    sk = flb::warp_sum(sk);
    if (lane == 0) {
      s.nq[t] = p.scale * (p.normalize ? rsqrtf(sq + 1e-6f) : 1.f);
      s.nk[t] = p.normalize ? rsqrtf(sk + 1e-6f) : 1.f;
    }
  }
  __syncthreads();
  if (tid < L) {
    p.norm_q[slot * L + tid] = s.nq[tid];
    p.norm_k[slot * L + tid] = s.nk[tid];
    if constexpr (!CHANNEL) p.decay[slot * L + tid] = s.c[tid];
  }
  bf16* const tp = p.tri_p + slot * kTri;
  float* const tn = p.tri_n == nullptr ? nullptr : p.tri_n + slot * L * L;
  auto store_p = [&](int t, int c, float a, float b) {
    uint32_t h, m, l;
    split(a, b, h, m, l);
    uint32_t* dst = reinterpret_cast<uint32_t*>(tp + t * L + c);
    dst[0] = h;
    dst[L * L / 2] = m;
    dst[L * L] = l;
  };
  if constexpr (!CHANNEL) {
    // products of the raw bf16 rows are exact; norms and decay are factors of the result.  Warp w owns rows 16 w .. 16 w + 15.
    float kk[8][4], qk[8][4];
#pragma unroll
    for (int n = 0; n < 8; ++n)
#pragma unroll
      for (int i = 0; i < 4; ++i) kk[n][i] = qk[n][i] = 0.f;
#pragma unroll
    for (int d = 0; d < DK; d += 16) {
      uint32_t ak[4], aq[4];
      load_mk(ak, s.k, KS, warp * 16, d, lane);
      load_mk(aq, s.q, KS, warp * 16, d, lane);
#pragma unroll
      for (int n = 0; n < 4; ++n) {
        uint32_t b[4];
        load_nk(b, s.k, KS, n * 16, d, lane);
        mma(kk[2 * n], ak, b[0], b[1]);
        mma(kk[2 * n + 1], ak, b[2], b[3]);
        mma(qk[2 * n], aq, b[0], b[1]);
        mma(qk[2 * n + 1], aq, b[2], b[3]);
      }
    }
#pragma unroll
    for (int n = 0; n < 8; ++n)
#pragma unroll
      for (int half = 0; half < 2; ++half) {
        const int t = warp * 16 + (lane >> 2) + 8 * half, c = n * 8 + (lane & 3) * 2;
        float pv[2], nv[2];
#pragma unroll
        for (int i = 0; i < 2; ++i) {
          const float pair = c + i <= t ? exp2f(s.c[t] - s.c[c + i]) * s.nk[c + i] : 0.f;
          pv[i] = qk[n][2 * half + i] * pair * s.nq[t];
          nv[i] = c + i < t ? kk[n][2 * half + i] * pair * s.nk[t] : 0.f;
          s.n[t * NS + c + i] = nv[i] * s.beta[c + i];
        }
        store_p(t, c, pv[0], pv[1]);
        if (tn != nullptr) *reinterpret_cast<float2*>(tn + t * L + c) = make_float2(nv[0], nv[1]);
      }
  } else {
    // every (t, s, channel) has a decay of its own: fp32 multiply-adds, 2 x 2 tiles of (t, s) per thread; bounded by the
    // exponentials (64 * 65 / 2 * dk of them per chunk and head)
    for (int tile = tid; tile < 32 * 33 / 2; tile += 128) {
      int ti = (int)((sqrtf(8.f * tile + 1.f) - 1.f) * 0.5f);
      while ((ti + 1) * (ti + 2) / 2 <= tile) ++ti;
      while (ti * (ti + 1) / 2 > tile) --ti;
      const int t0 = 2 * ti, s0 = 2 * (tile - ti * (ti + 1) / 2);
      float kk[2][2] = {}, qk[2][2] = {};
#pragma unroll 4
      for (int d = 0; d < DK; d += 2) {
        float2 ct[2], cs[2], kt[2], ks[2], qt[2];
#pragma unroll
        for (int i = 0; i < 2; ++i) {
          ct[i] = *reinterpret_cast<const float2*>(s.c + (t0 + i) * CS + d);
          cs[i] = *reinterpret_cast<const float2*>(s.c + (s0 + i) * CS + d);
          kt[i] = floats(*reinterpret_cast<const uint32_t*>(s.k + (t0 + i) * KS + d));
          ks[i] = floats(*reinterpret_cast<const uint32_t*>(s.k + (s0 + i) * KS + d));
          qt[i] = floats(*reinterpret_cast<const uint32_t*>(s.q + (t0 + i) * KS + d));
        }
#pragma unroll
        for (int i = 0; i < 2; ++i)
#pragma unroll
          for (int j = 0; j < 2; ++j) {
            const float ex = exp2f(fminf(ct[i].x - cs[j].x, 0.f)) * ks[j].x, ey = exp2f(fminf(ct[i].y - cs[j].y, 0.f)) * ks[j].y;
            kk[i][j] = fmaf(kt[i].x, ex, fmaf(kt[i].y, ey, kk[i][j]));
            qk[i][j] = fmaf(qt[i].x, ex, fmaf(qt[i].y, ey, qk[i][j]));
          }
      }
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        const int t = t0 + i;
        float pv[2], nv[2];
#pragma unroll
        for (int j = 0; j < 2; ++j) {
          const int c = s0 + j;
          pv[j] = c <= t ? qk[i][j] * s.nq[t] * s.nk[c] : 0.f;
          nv[j] = c < t ? kk[i][j] * s.nk[t] * s.nk[c] : 0.f;
          s.n[t * NS + c] = nv[j] * s.beta[c];
        }
        store_p(t, s0, pv[0], pv[1]);
        if (tn != nullptr) *reinterpret_cast<float2*>(tn + t * L + s0) = make_float2(nv[0], nv[1]);
      }
    }
    for (int i = tid; i < 32 * 32; i += 128) {  // the tiles above the diagonal
      const int t0 = 2 * (i / 32), s0 = 2 * (i % 32);
      if (s0 <= t0) continue;
#pragma unroll
      for (int r = 0; r < 2; ++r) {
        store_p(t0 + r, s0, 0.f, 0.f);
        if (tn != nullptr) *reinterpret_cast<float2*>(tn + (t0 + r) * L + s0) = make_float2(0.f, 0.f);
      }
    }
    // operands of the scans, with their decays folded in
    for (int i = tid; i < L * DK / 2; i += 128) {
      const int t = i / (DK / 2), d = (i % (DK / 2)) * 2;
      const float2 c = *reinterpret_cast<const float2*>(s.c + t * CS + d), end = *reinterpret_cast<const float2*>(s.c + (L - 1) * CS + d);
      const float2 k = floats(*reinterpret_cast<const uint32_t*>(s.k + t * KS + d)), q = floats(*reinterpret_cast<const uint32_t*>(s.q + t * KS + d));
      *reinterpret_cast<float2*>(p.decay + (slot * L + t) * DK + d) = c;
      const float gx = exp2f(c.x), gy = exp2f(c.y);
      const long long at = (slot * 3 * L + t) * DK + d;
      auto store = [&](bf16* planes, float a, float b) {
        uint32_t h, m, l;
        split(a, b, h, m, l);
        uint32_t* dst = reinterpret_cast<uint32_t*>(planes + at);
        dst[0] = h;
        dst[L * DK / 2] = m;
        dst[L * DK] = l;
      };
      store(p.k_in, k.x * s.nk[t] * gx, k.y * s.nk[t] * gy);
      store(p.k_out, k.x * s.nk[t] * exp2f(end.x - c.x), k.y * s.nk[t] * exp2f(end.y - c.y));
      store(p.q_in, q.x * s.nq[t] * gx, q.y * s.nq[t] * gy);
    }
  }
  __syncthreads();
  if (tid < L) {
    float x[L];
#pragma unroll
    for (int t = 0; t < L; ++t) {
      float acc[4] = {t == tid ? 1.f : 0.f, 0.f, 0.f, 0.f};
#pragma unroll
      for (int c = 0; c + 4 <= t; c += 4) {
        const float4 n = *reinterpret_cast<const float4*>(s.n + t * NS + c);
        acc[0] = fmaf(-n.x, x[c], acc[0]);
        acc[1] = fmaf(-n.y, x[c + 1], acc[1]);
        acc[2] = fmaf(-n.z, x[c + 2], acc[2]);
        acc[3] = fmaf(-n.w, x[c + 3], acc[3]);
      }
#pragma unroll
      for (int c = t / 4 * 4; c < t; ++c) acc[c & 3] = fmaf(-s.n[t * NS + c], x[c], acc[c & 3]);
      x[t] = (acc[0] + acc[1]) + (acc[2] + acc[3]);
    }
    bf16* const tt = p.tri_t + slot * kTri + tid;
#pragma unroll
    for (int t = 0; t < L; ++t) {
      const bf16 h = __float2bfloat16_rn(x[t]);
      const float r = x[t] - __bfloat162float(h);
      const bf16 m = __float2bfloat16_rn(r);
      tt[t * L] = h;
      tt[L * L + t * L] = m;
      tt[2 * L * L + t * L] = __float2bfloat16_rn(r - __bfloat162float(m));
    }
  }
}
}  // namespace

// ---- operands of the sequential kernels --------------------------------------------------------------------------------
namespace {
constexpr int kScanWarps = 4;              // a block covers 64 columns of dv
constexpr int kScanCols = 16 * kScanWarps;
constexpr int kScanThreads = 32 * kScanWarps;

// Rows 0..63 of a [planes][64][DK] operand: raw rows of a token-major matrix (one plane; rows past the chunk are zero) or
// prepared planes.
template <int DK, int NP>
__device__ __forceinline__ void stage_operand(bf16* dst, const bf16* rows, long long row_stride, const bf16* planes, long long slot, int2 span, int col0,
                                              int threads) {
  constexpr int KS = DK + 8;
  for (int i = threadIdx.x; i < NP * L * DK / 8; i += threads) {
    const int row = i / (DK / 8), d = (i % (DK / 8)) * 8;  // row counts through the planes
    if constexpr (NP == 1) {
      const bool ok = row < span.y;
      cp16(dst + row * KS + d, rows + (long long)(span.x + (ok ? row : 0)) * row_stride + col0 + d, ok);
    } else {
      cp16(dst + row * KS + d, planes + (slot * NP * L + row) * DK + d, true);
    }
  }
}
__device__ __forceinline__ void stage_tri(bf16* dst, const bf16* src, int threads) {
  for (int i = threadIdx.x; i < kTri / 8; i += threads) {
    const int row = i / (L / 8), d = (i % (L / 8)) * 8;
    cp16(dst + row * TS + d, src + row * L + d, true);
  }
}
__device__ __forceinline__ void stage_rows(bf16* dst, const bf16* src, long long row_stride, int2 span, int threads) {  // [64][kScanCols] of v or dO
  for (int i = threadIdx.x; i < L * kScanCols / 8; i += threads) {
    const int t = i / (kScanCols / 8), d = (i % (kScanCols / 8)) * 8;
    const bool ok = t < span.y;
    cp16(dst + t * (kScanCols + 8) + d, src + (long long)(span.x + (ok ? t : 0)) * row_stride + d, ok);
  }
}
struct ScanScalars {  // per token of a chunk
  float decay[L], nq[L], nk[L], beta[L];
};
template <bool CHANNEL>
__device__ __forceinline__ void stage_scalars(ScanScalars& s, const DeltaArgs& p, long long slot, int2 span, int head) {
  const int t = threadIdx.x;
  if (t < L) {
    if constexpr (!CHANNEL) {
      cp4(&s.decay[t], p.decay + slot * L + t, true);
      cp4(&s.nq[t], p.norm_q + slot * L + t, true);
      cp4(&s.nk[t], p.norm_k + slot * L + t, true);
    }
    const bool ok = t < span.y;
    cp4(&s.beta[t], p.beta + (long long)(span.x + (ok ? t : 0)) * p.heads + head, ok);
  }
}

// ---- forward scan --------------------------------------------------------------------------------------------------
// Block = (document, head, 64 columns of dv), warp = 16 columns.  Per chunk: S^T K^T, then U^T = R^T T^T, then the state update;
// each operand has one buffer, refilled for the next chunk as soon as its product is done (three cp.async groups in flight).
template <int DK, bool CHANNEL>
struct ScanFwdSmem {
  static constexpr int NP = CHANNEL ? 3 : 1, KS = DK + 8;
  bf16 k_in[NP * L * KS], k_out[NP * L * KS], t[3 * L * TS], v[L * (kScanCols + 8)];
  ScanScalars scalar[2];
  float end[2][CHANNEL ? DK : 4];  // decay over the whole chunk
};

template <int DK, bool CHANNEL>
__global__ void __launch_bounds__(kScanThreads) delta_scan_fwd_kernel(const DeltaArgs p) {
  extern __shared__ __align__(16) unsigned char raw[];
  using Smem = ScanFwdSmem<DK, CHANNEL>;
  Smem& s = *reinterpret_cast<Smem*>(raw);
  constexpr int NP = Smem::NP, KS = Smem::KS;
  const int doc = blockIdx.x, head = blockIdx.y, col0 = blockIdx.z * kScanCols, key_head = head / p.repeat;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, j2 = (lane & 3) * 2, g8 = lane >> 2;
  const int first = p.doc_chunk[doc], last = p.doc_chunk[doc + 1];
  if (first >= last) return;
  float st[DK / 8][4];
#pragma unroll
  for (int n = 0; n < DK / 8; ++n)
#pragma unroll
    for (int i = 0; i < 4; ++i) st[n][i] = 0.f;

  auto stage_in = [&](int ch) {
    if (ch < last) {
      const int2 span = p.chunk[ch];
      const long long slot = (long long)ch * p.heads + head;
      stage_operand<DK, NP>(s.k_in, p.k, p.k_row, p.k_in, slot, span, key_head * DK, kScanThreads);
      stage_rows(s.v, p.v + head * p.dv + col0, p.v_row, span, kScanThreads);
      stage_scalars<CHANNEL>(s.scalar[ch & 1], p, slot, span, head);
      if constexpr (CHANNEL) {
        if (threadIdx.x < DK) cp4(&s.end[ch & 1][threadIdx.x], p.decay + (slot * L + L - 1) * DK + threadIdx.x, true);
      }
    }
    cp_commit();
  };
  auto stage_t = [&](int ch) {
    if (ch < last) stage_tri(s.t, p.tri_t + ((long long)ch * p.heads + head) * kTri, kScanThreads);
    cp_commit();
  };
  auto stage_out = [&](int ch) {
    if (ch < last) {
      const long long slot = (long long)ch * p.heads + head;
      stage_operand<DK, NP>(s.k_out, p.k, p.k_row, p.k_out, slot, p.chunk[ch], key_head * DK, kScanThreads);
    }
    cp_commit();
  };
  stage_in(first);
  stage_t(first);
  stage_out(first);
  for (int ch = first; ch < last; ++ch) {
    const long long slot = (long long)ch * p.heads + head;
    const ScanScalars& sc = s.scalar[ch & 1];
    // the state entering the chunk, transposed: [dv][dk]
    float* const state = p.state + (slot * p.dv + col0 + warp * 16 + g8) * DK + j2;
#pragma unroll
    for (int n = 0; n < DK / 8; ++n) {
      *reinterpret_cast<float2*>(state + n * 8) = make_float2(st[n][0], st[n][1]);
      *reinterpret_cast<float2*>(state + 8 * DK + n * 8) = make_float2(st[n][2], st[n][3]);
    }
    cp_wait<2>();
    __syncthreads();
    // R^T = V^T - (S^T K^T) Gamma
    float r[8][4];
#pragma unroll
    for (int n = 0; n < 8; ++n)
#pragma unroll
      for (int i = 0; i < 4; ++i) r[n][i] = 0.f;
    if (ch != first) {
#pragma unroll
      for (int kk = 0; kk < DK / 16; ++kk) {
        uint32_t a[3][4];
        split_a(st[2 * kk], st[2 * kk + 1], a);
#pragma unroll
        for (int n = 0; n < 4; n += 2) {
          uint32_t b[4][NP][2];
          load_b<NP, false>(b, s.k_in, L * KS, KS, n * 16, kk * 16, lane);
          load_b<NP, false>(b + 2, s.k_in, L * KS, KS, n * 16 + 16, kk * 16, lane);
          mma_tiles<NP>(r + 2 * n, a, b, 4);
        }
      }
    }
#pragma unroll
    for (int n = 0; n < 4; ++n) {
      uint32_t x[4];
      load_km(x, s.v, kScanCols + 8, n * 16, warp * 16, lane);
#pragma unroll
      for (int half = 0; half < 2; ++half) {
        const int t = n * 16 + half * 8 + j2;
        float f0 = 1.f, f1 = 1.f;
        if constexpr (!CHANNEL) {
          f0 = exp2f(sc.decay[t]) * sc.nk[t];
          f1 = exp2f(sc.decay[t + 1]) * sc.nk[t + 1];
        }
        const float2 lo = floats(x[2 * half]), hi = floats(x[2 * half + 1]);
        float* d = r[2 * n + half];
        d[0] = lo.x - d[0] * f0;
        d[1] = lo.y - d[1] * f1;
        d[2] = hi.x - d[2] * f0;
        d[3] = hi.y - d[3] * f1;
      }
    }
    cp_wait<1>();
    __syncthreads();
    stage_in(ch + 1);
    // U^T = R^T T^T, T lower triangular
    float u[8][4];
#pragma unroll
    for (int n = 0; n < 8; ++n)
#pragma unroll
      for (int i = 0; i < 4; ++i) u[n][i] = 0.f;
#pragma unroll
    for (int ks = 0; ks < 4; ++ks) {
      uint32_t a[3][4];
      split_a(r[2 * ks], r[2 * ks + 1], a);
#pragma unroll
      for (int n = ks; n < 4; n += 2) {
        uint32_t b[4][3][2];
        load_b<3, false>(b, s.t, L * TS, TS, n * 16, ks * 16, lane);
        if (n + 1 < 4) load_b<3, false>(b + 2, s.t, L * TS, TS, n * 16 + 16, ks * 16, lane);
        mma_tiles<3>(u + 2 * n, a, b, n + 1 < 4 ? 4 : 2);
      }
    }
    float* const up = p.u + slot * L * p.dv + col0 + warp * 16 + g8;
    const float end_decay = CHANNEL ? 0.f : sc.decay[L - 1];
#pragma unroll
    for (int n = 0; n < 8; ++n) {
      const int t = n * 8 + j2;
      up[(long long)t * p.dv] = u[n][0];
      up[(long long)(t + 1) * p.dv] = u[n][1];
      up[(long long)t * p.dv + 8] = u[n][2];
      up[(long long)(t + 1) * p.dv + 8] = u[n][3];
      float f0 = sc.beta[t], f1 = sc.beta[t + 1];
      if constexpr (!CHANNEL) {
        f0 *= exp2f(end_decay - sc.decay[t]) * sc.nk[t];
        f1 *= exp2f(end_decay - sc.decay[t + 1]) * sc.nk[t + 1];
      }
      u[n][0] *= f0;
      u[n][1] *= f1;
      u[n][2] *= f0;
      u[n][3] *= f1;
    }
    // S'^T = Gamma_L S^T + (beta U exp(c_L - c))^T K
    if constexpr (CHANNEL) {
#pragma unroll
      for (int n = 0; n < DK / 8; ++n) {
        const float f0 = exp2f(s.end[ch & 1][n * 8 + j2]), f1 = exp2f(s.end[ch & 1][n * 8 + j2 + 1]);
        st[n][0] *= f0; st[n][1] *= f1; st[n][2] *= f0; st[n][3] *= f1;
      }
    } else {
      const float f = exp2f(end_decay);
#pragma unroll
      for (int n = 0; n < DK / 8; ++n)
#pragma unroll
        for (int i = 0; i < 4; ++i) st[n][i] *= f;
    }
    cp_wait<1>();
    __syncthreads();
    stage_t(ch + 1);
#pragma unroll
    for (int ks = 0; ks < 4; ++ks) {
      uint32_t a[3][4];
      split_a(u[2 * ks], u[2 * ks + 1], a);
#pragma unroll
      for (int n = 0; n < DK / 16; n += 2) {
        uint32_t b[4][NP][2];
        load_b<NP, true>(b, s.k_out, L * KS, KS, n * 16, ks * 16, lane);
        load_b<NP, true>(b + 2, s.k_out, L * KS, KS, n * 16 + 16, ks * 16, lane);
        mma_tiles<NP>(st + 2 * n, a, b, 4);
      }
    }
    __syncthreads();
    stage_out(ch + 1);
  }
}
}  // namespace

// ---- output --------------------------------------------------------------------------------------------------------
// Block = (chunk, head), warp = 16 columns of dv: O = Gamma Q^ S + P (beta U).  S and U come from global memory straight in
// operand order (every element is read by one warp), Q and the planes of P through shared memory.
namespace {
template <int DK, bool CHANNEL>
struct OutputSmem {
  static constexpr int NP = CHANNEL ? 3 : 1, KS = DK + 8;
  bf16 q[NP * L * KS], p[3 * L * TS];
  float decay[L], nq[L], beta[L];
};

template <int DK, bool CHANNEL>
__global__ void __launch_bounds__(256) delta_output_kernel(const DeltaArgs p) {
  extern __shared__ __align__(16) unsigned char raw[];
  using Smem = OutputSmem<DK, CHANNEL>;
  Smem& s = *reinterpret_cast<Smem*>(raw);
  constexpr int NP = Smem::NP, KS = Smem::KS;
  const int ch = blockIdx.x, head = blockIdx.y;
  if (ch >= p.doc_chunk[p.docs]) return;
  const int2 span = p.chunk[ch];
  const long long slot = (long long)ch * p.heads + head;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, j2 = (lane & 3) * 2, g8 = lane >> 2;
  stage_operand<DK, NP>(s.q, p.q, p.q_row, p.q_in, slot, span, (head / p.repeat) * DK, blockDim.x);
  stage_tri(s.p, p.tri_p + slot * kTri, blockDim.x);
  cp_commit();
  if (threadIdx.x < L) {
    const int t = threadIdx.x;
    s.decay[t] = CHANNEL ? 0.f : p.decay[slot * L + t];
    s.nq[t] = CHANNEL ? 1.f : p.norm_q[slot * L + t];
    s.beta[t] = t < span.y ? p.beta[(long long)(span.x + t) * p.heads + head] : 0.f;
  }
  const int v0 = warp * 16;
  float acc[4][2][4];
#pragma unroll
  for (int m = 0; m < 4; ++m)
#pragma unroll
    for (int n = 0; n < 2; ++n)
#pragma unroll
      for (int i = 0; i < 4; ++i) acc[m][n][i] = 0.f;
  cp_wait<0>();
  __syncthreads();
  const float* const state = p.state + (slot * p.dv + v0 + g8) * DK + j2;
#pragma unroll 2
  for (int kk = 0; kk < DK; kk += 16) {
    uint32_t b[2][3][2];
#pragma unroll
    for (int n = 0; n < 2; ++n)
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const float2 x = __ldg(reinterpret_cast<const float2*>(state + n * 8 * DK + kk + h * 8));
        split(x.x, x.y, b[n][0][h], b[n][1][h], b[n][2][h]);
      }
#pragma unroll
    for (int m = 0; m < 4; ++m) {
      uint32_t a[NP][4];
#pragma unroll
      for (int pl = 0; pl < NP; ++pl) load_mk(a[pl], s.q + pl * L * KS, KS, m * 16, kk, lane);
      if constexpr (CHANNEL) mma_tiles<3>(acc[m], a, b, 2);
      else mma_tiles_exact<3>(acc[m], a[0], b, 2);
    }
  }
  if constexpr (!CHANNEL) {
#pragma unroll
    for (int m = 0; m < 4; ++m)
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const int t = m * 16 + g8 + h * 8;
        const float f = exp2f(s.decay[t]) * s.nq[t];
#pragma unroll
        for (int n = 0; n < 2; ++n) {
          acc[m][n][2 * h] *= f;
          acc[m][n][2 * h + 1] *= f;
        }
      }
  }
  const float* const u = p.u + slot * L * p.dv + v0 + g8;
#pragma unroll
  for (int ks = 0; ks < 4; ++ks) {
    uint32_t b[2][3][2];
#pragma unroll
    for (int n = 0; n < 2; ++n)
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const int t = ks * 16 + h * 8 + j2;
        split(__ldg(u + (long long)t * p.dv + n * 8) * s.beta[t], __ldg(u + (long long)(t + 1) * p.dv + n * 8) * s.beta[t + 1], b[n][0][h], b[n][1][h],
              b[n][2][h]);
      }
#pragma unroll
    for (int m = ks; m < 4; ++m) {
      uint32_t a[3][4];
#pragma unroll
      for (int pl = 0; pl < 3; ++pl) load_mk(a[pl], s.p + pl * L * TS, TS, m * 16, ks * 16, lane);
      mma_tiles<3>(acc[m], a, b, 2);
    }
  }
#pragma unroll
  for (int m = 0; m < 4; ++m)
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int t = m * 16 + g8 + h * 8;
      if (t >= span.y) continue;
      bf16* const out = p.out + ((long long)(span.x + t) * p.heads + head) * p.dv + v0 + j2;
#pragma unroll
      for (int n = 0; n < 2; ++n) *reinterpret_cast<bf162*>(out + n * 8) = __floats2bfloat162_rn(acc[m][n][2 * h], acc[m][n][2 * h + 1]);
    }
}

// ---- backward scan -------------------------------------------------------------------------------------------------
// The forward scan's layout, walking the chunks of a document from its end.
template <int DK, bool CHANNEL>
struct ScanBwdSmem {
  static constexpr int NP = CHANNEL ? 3 : 1, KS = DK + 8;
  bf16 k_in[NP * L * KS], k_out[NP * L * KS], q_in[NP * L * KS], t[3 * L * TS], p[3 * L * TS], dout[L * (kScanCols + 8)];
  ScanScalars scalar[2];
  float end[2][CHANNEL ? DK : 4];
};

template <int DK, bool CHANNEL>
__global__ void __launch_bounds__(kScanThreads) delta_scan_bwd_kernel(const DeltaArgs p) {
  extern __shared__ __align__(16) unsigned char raw[];
  using Smem = ScanBwdSmem<DK, CHANNEL>;
  Smem& s = *reinterpret_cast<Smem*>(raw);
  constexpr int NP = Smem::NP, KS = Smem::KS, VS = kScanCols + 8;
  const int doc = blockIdx.x, head = blockIdx.y, col0 = blockIdx.z * kScanCols, key_head = head / p.repeat;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, j2 = (lane & 3) * 2, g8 = lane >> 2;
  const int first = p.doc_chunk[doc], last = p.doc_chunk[doc + 1];
  if (first >= last) return;
  float ds[DK / 8][4];
#pragma unroll
  for (int n = 0; n < DK / 8; ++n)
#pragma unroll
    for (int i = 0; i < 4; ++i) ds[n][i] = 0.f;
  auto slot_of = [&](int ch) { return (long long)ch * p.heads + head; };
  auto stage_p = [&](int ch) {
    if (ch >= first) {
      const int2 span = p.chunk[ch];
      const long long slot = slot_of(ch);
      stage_tri(s.p, p.tri_p + slot * kTri, kScanThreads);
      stage_scalars<CHANNEL>(s.scalar[ch & 1], p, slot, span, head);
      if constexpr (CHANNEL) {
        if (threadIdx.x < DK) cp4(&s.end[ch & 1][threadIdx.x], p.decay + (slot * L + L - 1) * DK + threadIdx.x, true);
      }
    }
    cp_commit();
  };
  auto stage_out = [&](int ch) {
    if (ch >= first) stage_operand<DK, NP>(s.k_out, p.k, p.k_row, p.k_out, slot_of(ch), p.chunk[ch], key_head * DK, kScanThreads);
    cp_commit();
  };
  auto stage_t = [&](int ch) {
    if (ch >= first) stage_tri(s.t, p.tri_t + slot_of(ch) * kTri, kScanThreads);
    cp_commit();
  };
  auto stage_in = [&](int ch) {
    if (ch >= first) {
      const int2 span = p.chunk[ch];
      stage_operand<DK, NP>(s.q_in, p.q, p.q_row, p.q_in, slot_of(ch), span, key_head * DK, kScanThreads);
      stage_operand<DK, NP>(s.k_in, p.k, p.k_row, p.k_in, slot_of(ch), span, key_head * DK, kScanThreads);
    }
    cp_commit();
  };
  auto stage_dout = [&](int ch) {  // joins the group committed by the caller's next commit
    if (ch >= first) stage_rows(s.dout, p.dout + head * p.dv + col0, (long long)p.heads * p.dv, p.chunk[ch], kScanThreads);
  };
  stage_dout(last - 1);
  stage_p(last - 1);
  stage_out(last - 1);
  stage_t(last - 1);
  stage_in(last - 1);
  for (int ch = last - 1; ch >= first; --ch) {
    const long long slot = slot_of(ch);
    const ScanScalars& sc = s.scalar[ch & 1];
    float* const dstate = p.dstate + (slot * p.dv + col0 + warp * 16 + g8) * DK + j2;  // adjoint of the state leaving this chunk
#pragma unroll
    for (int n = 0; n < DK / 8; ++n) {
      *reinterpret_cast<float2*>(dstate + n * 8) = make_float2(ds[n][0], ds[n][1]);
      *reinterpret_cast<float2*>(dstate + 8 * DK + n * 8) = make_float2(ds[n][2], ds[n][3]);
    }
    cp_wait<2>();  // P, dO and K out (groups in flight: p, out, t, in)
    __syncthreads();
    // dS'^T K^T
    float d[8][4];
#pragma unroll
    for (int n = 0; n < 8; ++n)
#pragma unroll
      for (int i = 0; i < 4; ++i) d[n][i] = 0.f;
    if (ch != last - 1) {
#pragma unroll
      for (int kk = 0; kk < DK / 16; ++kk) {
        uint32_t a[3][4];
        split_a(ds[2 * kk], ds[2 * kk + 1], a);
#pragma unroll
        for (int n = 0; n < 4; n += 2) {
          uint32_t b[4][NP][2];
          load_b<NP, false>(b, s.k_out, L * KS, KS, n * 16, kk * 16, lane);
          load_b<NP, false>(b + 2, s.k_out, L * KS, KS, n * 16 + 16, kk * 16, lane);
          mma_tiles<NP>(d + 2 * n, a, b, 4);
        }
      }
    }
    const float end_decay = CHANNEL ? 0.f : sc.decay[L - 1];
    if constexpr (!CHANNEL) {
#pragma unroll
      for (int n = 0; n < 8; ++n) {
        const int t = n * 8 + j2;
        const float f0 = exp2f(end_decay - sc.decay[t]) * sc.nk[t], f1 = exp2f(end_decay - sc.decay[t + 1]) * sc.nk[t + 1];
        d[n][0] *= f0; d[n][1] *= f1; d[n][2] *= f0; d[n][3] *= f1;
      }
    }
    // + dO^T P, P lower triangular: token block n of P's columns meets rows t >= s
    uint32_t go[4][4];
#pragma unroll
    for (int ks = 0; ks < 4; ++ks) {
      load_km(go[ks], s.dout, VS, ks * 16, warp * 16, lane);
#pragma unroll
      for (int n = 0; n <= ks; n += 2) {
        uint32_t b[4][3][2];
        load_b<3, true>(b, s.p, L * TS, TS, n * 16, ks * 16, lane);
        if (n + 1 <= ks) load_b<3, true>(b + 2, s.p, L * TS, TS, n * 16 + 16, ks * 16, lane);
        mma_tiles_exact<3>(d + 2 * n, go[ks], b, n + 1 <= ks ? 4 : 2);
      }
    }
#pragma unroll
    for (int n = 0; n < 8; ++n) {
      const float f0 = sc.beta[n * 8 + j2], f1 = sc.beta[n * 8 + j2 + 1];
      d[n][0] *= f0; d[n][1] *= f1; d[n][2] *= f0; d[n][3] *= f1;
    }
    cp_wait<1>();  // T
    __syncthreads();
    stage_dout(ch - 1);
    stage_p(ch - 1);
    stage_out(ch - 1);
    // dR^T = dU^T T
    float r[8][4];
#pragma unroll
    for (int n = 0; n < 8; ++n)
#pragma unroll
      for (int i = 0; i < 4; ++i) r[n][i] = 0.f;
#pragma unroll
    for (int ks = 0; ks < 4; ++ks) {
      uint32_t a[3][4];
      split_a(d[2 * ks], d[2 * ks + 1], a);
#pragma unroll
      for (int n = 0; n <= ks; n += 2) {
        uint32_t b[4][3][2];
        load_b<3, true>(b, s.t, L * TS, TS, n * 16, ks * 16, lane);
        if (n + 1 <= ks) load_b<3, true>(b + 2, s.t, L * TS, TS, n * 16 + 16, ks * 16, lane);
        mma_tiles<3>(r + 2 * n, a, b, n + 1 <= ks ? 4 : 2);
      }
    }
    float* const rp = p.dr + slot * L * p.dv + col0 + warp * 16 + g8;
#pragma unroll
    for (int n = 0; n < 8; ++n) {
      const int t = n * 8 + j2;
      rp[(long long)t * p.dv] = r[n][0];
      rp[(long long)(t + 1) * p.dv] = r[n][1];
      rp[(long long)t * p.dv + 8] = r[n][2];
      rp[(long long)(t + 1) * p.dv + 8] = r[n][3];
      float f0 = -1.f, f1 = -1.f;
      if constexpr (!CHANNEL) {
        f0 = -exp2f(sc.decay[t]) * sc.nk[t];
        f1 = -exp2f(sc.decay[t + 1]) * sc.nk[t + 1];
      }
      r[n][0] *= f0; r[n][1] *= f1; r[n][2] *= f0; r[n][3] *= f1;
    }
    cp_wait<2>();  // q and k in (behind them: the next chunk's p and out)
    __syncthreads();
    stage_t(ch - 1);
    // dS^T = Gamma_L dS'^T + (Gamma dO)^T Q - (Gamma dR)^T K
    if constexpr (CHANNEL) {
#pragma unroll
      for (int n = 0; n < DK / 8; ++n) {
        const float f0 = exp2f(s.end[ch & 1][n * 8 + j2]), f1 = exp2f(s.end[ch & 1][n * 8 + j2 + 1]);
        ds[n][0] *= f0; ds[n][1] *= f1; ds[n][2] *= f0; ds[n][3] *= f1;
      }
    } else {
      const float f = exp2f(end_decay);
#pragma unroll
      for (int n = 0; n < DK / 8; ++n)
#pragma unroll
        for (int i = 0; i < 4; ++i) ds[n][i] *= f;
    }
#pragma unroll
    for (int ks = 0; ks < 4; ++ks) {
      uint32_t a[3][4], ao[3][4];
      split_a(r[2 * ks], r[2 * ks + 1], a);
      if constexpr (!CHANNEL) {
        // the row factors of q go on the dO side: [dv][t] pairs times the factors of their two tokens
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const int t = ks * 16 + (i >> 1) * 8 + j2;
          const float2 x = floats(go[ks][i]);
          split(x.x * exp2f(sc.decay[t]) * sc.nq[t], x.y * exp2f(sc.decay[t + 1]) * sc.nq[t + 1], ao[0][i], ao[1][i], ao[2][i]);
        }
      }
#pragma unroll
      for (int n = 0; n < DK / 16; n += 2) {
        uint32_t b[4][NP][2];
        load_b<NP, true>(b, s.q_in, L * KS, KS, n * 16, ks * 16, lane);
        load_b<NP, true>(b + 2, s.q_in, L * KS, KS, n * 16 + 16, ks * 16, lane);
        if constexpr (CHANNEL) mma_tiles_exact<NP>(ds + 2 * n, go[ks], b, 4);
        else mma_tiles<NP>(ds + 2 * n, ao, b, 4);
        load_b<NP, true>(b, s.k_in, L * KS, KS, n * 16, ks * 16, lane);
        load_b<NP, true>(b + 2, s.k_in, L * KS, KS, n * 16 + 16, ks * 16, lane);
        mma_tiles<NP>(ds + 2 * n, a, b, 4);
      }
    }
    __syncthreads();
    stage_in(ch - 1);
  }
}
}  // namespace

// ---- backward inside the chunks ----------------------------------------------------------------------------------------
// Block = (chunk, head), warp = 16 channels of dk.  With everything the scans left behind (S, dS', U, dR) all gradients are local
// to the chunk.  Gradients of the unit-scaled keys are kept apart by role - G_l where the token reads (the row of N and of
// Gamma K^ S), G_r where it is written (the columns, and the way into S') - because the decay gradient needs them apart:
//     dc_t = q.G_q + k.G_l - k.G_r  (+ what enters through c_L at the chunk's end),   dg = sum of dc from t to the chunk's end,
// per channel or summed over the channels.
namespace {
template <int DK, int DV, bool CHANNEL>
struct BackwardSmem {
  static constexpr int NW = DK / 16, KS = DK + 8, VS = DV + 8, GS = DK + 4;
  union {
    struct { bf16 u[3 * L * VS], r[3 * L * VS]; };
    struct { float gq[L * GS], gl[L * GS], gr[L * GS]; };
  };
  bf16 go[L * VS], k[L * KS], q[L * KS];
  union {
    struct { bf16 w1[3 * L * TS], w2[3 * L * TS]; } planes;
    struct { float w1[L * (L + 4)], w2[L * (L + 4)]; } full;
  };
  float decay[L], nq[L], nk[L], beta[L], dc[L];
  float dbeta[2 * NW][L];
  float end[DK];  // what enters the decay sum of the whole chunk, per channel
};

template <int DK, int DV, bool CHANNEL>
__global__ void __launch_bounds__(DK * 2, 1) delta_backward_kernel(const DeltaArgs p) {
  extern __shared__ __align__(16) unsigned char raw[];
  using Smem = BackwardSmem<DK, DV, CHANNEL>;
  Smem& s = *reinterpret_cast<Smem*>(raw);
  constexpr int NW = Smem::NW, KS = Smem::KS, VS = Smem::VS, GS = Smem::GS, NT = NW * 32, WS = L + 4;
  const int ch = blockIdx.x, head = blockIdx.y;
  if (ch >= p.doc_chunk[p.docs]) return;
  const int2 span = p.chunk[ch];
  const int len = span.y, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, j2 = (lane & 3) * 2, g8 = lane >> 2;
  const long long slot = (long long)ch * p.heads + head;
  const int key_head = head / p.repeat;
  stage_operand<DK, 1>(s.k, p.k, p.k_row, nullptr, slot, span, key_head * DK, NT);
  stage_operand<DK, 1>(s.q, p.q, p.q_row, nullptr, slot, span, key_head * DK, NT);
  for (int i = tid; i < L * DV / 8; i += NT) {
    const int t = i / (DV / 8), d = (i % (DV / 8)) * 8;
    const bool ok = t < len;
    cp16(s.go + t * VS + d, p.dout + ((long long)(span.x + (ok ? t : 0)) * p.heads + head) * DV + d, ok);
  }
  cp_commit();
  if (tid < L) {
    s.decay[tid] = CHANNEL ? 0.f : p.decay[slot * L + tid];
    s.nq[tid] = p.norm_q[slot * L + tid];
    s.nk[tid] = p.norm_k[slot * L + tid];
    s.beta[tid] = tid < len ? p.beta[(long long)(span.x + tid) * p.heads + head] : 0.f;
  }
  for (int i = tid; i < 2 * NW * L; i += NT) (&s.dbeta[0][0])[i] = 0.f;
  for (int i = tid; i < L * DV / 2; i += NT) {
    const int t = i / (DV / 2), d = (i % (DV / 2)) * 2;
    const float2 u = __ldg(reinterpret_cast<const float2*>(p.u + (slot * L + t) * DV + d)), r = __ldg(reinterpret_cast<const float2*>(p.dr + (slot * L + t) * DV + d));
    uint32_t h, m, l;
    split(u.x, u.y, h, m, l);
    uint32_t* dst = reinterpret_cast<uint32_t*>(s.u + t * VS + d);
    dst[0] = h; dst[L * VS / 2] = m; dst[L * VS] = l;
    split(r.x, r.y, h, m, l);
    dst = reinterpret_cast<uint32_t*>(s.r + t * VS + d);
    dst[0] = h; dst[L * VS / 2] = m; dst[L * VS] = l;
    if (t < len) *reinterpret_cast<uint32_t*>(p.dvalue + ((long long)(span.x + t) * p.heads + head) * DV + d) = h;
  }
  cp_wait<0>();
  __syncthreads();
  {
    // X = dO U^T and Y = -dR U^T: 16 columns per warp; with eight warps two share the columns and split the rows
    constexpr int MT = NW == 8 ? 2 : 4;
    const int n0 = (warp & 3) * 16, m_first = NW == 8 ? (warp >> 2) * 2 : 0;
    float x[MT][2][4], y[MT][2][4];
#pragma unroll
    for (int m = 0; m < MT; ++m)
#pragma unroll
      for (int n = 0; n < 2; ++n)
#pragma unroll
        for (int i = 0; i < 4; ++i) x[m][n][i] = y[m][n][i] = 0.f;
#pragma unroll 2
    for (int kk = 0; kk < DV; kk += 16) {
      uint32_t b[2][3][2];
      load_b<3, false>(b, s.u, L * VS, VS, n0, kk, lane);
#pragma unroll
      for (int m = 0; m < MT; ++m) {
        const int m0 = (m_first + m) * 16;
        if (m0 + 15 < n0) continue;
        uint32_t a[3][4], ao[4];
        load_mk(ao, s.go, VS, m0, kk, lane);
#pragma unroll
        for (int pl = 0; pl < 3; ++pl) load_mk(a[pl], s.r + pl * L * VS, VS, m0, kk, lane);
        mma_tiles_exact<3>(x[m], ao, b, 2);
        mma_tiles<3>(y[m], a, b, 2);
      }
    }
    const bf16* const tp = p.tri_p + slot * kTri;
    const float* const tn = p.tri_n + slot * L * L;
    float db[2][2] = {};
#pragma unroll
    for (int m = 0; m < MT; ++m)
#pragma unroll
      for (int n = 0; n < 2; ++n)
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const int t = (m_first + m) * 16 + g8 + 8 * h, c = n0 + n * 8 + j2;
          const uint32_t* pp = reinterpret_cast<const uint32_t*>(tp + t * L + c);
          const float2 p0 = floats(__ldg(pp)), p1 = floats(__ldg(pp + L * L / 2)), p2 = floats(__ldg(pp + L * L));
          const float2 nn = __ldg(reinterpret_cast<const float2*>(tn + t * L + c));
          float w1[2], w2[2];
#pragma unroll
          for (int i = 0; i < 2; ++i) {
            const float pv = i ? p1.y + p2.y + p0.y : p1.x + p2.x + p0.x, nv = i ? nn.y : nn.x;
            const float xv = x[m][n][2 * h + i], yv = -y[m][n][2 * h + i];
            db[n][i] += pv * xv + nv * yv;
            float f = c + i <= t ? s.beta[c + i] * s.nk[c + i] : 0.f;
            if constexpr (!CHANNEL) f *= exp2f(fminf(s.decay[t] - s.decay[c + i], 0.f));
            w1[i] = xv * f * s.nq[t];
            w2[i] = c + i < t ? yv * f * s.nk[t] : 0.f;
          }
          if constexpr (CHANNEL) {
            *reinterpret_cast<float2*>(s.full.w1 + t * WS + c) = make_float2(w1[0], w1[1]);
            *reinterpret_cast<float2*>(s.full.w2 + t * WS + c) = make_float2(w2[0], w2[1]);
          } else {
            uint32_t hi, mid, lo;
            split(w1[0], w1[1], hi, mid, lo);
            uint32_t* dst = reinterpret_cast<uint32_t*>(s.planes.w1 + t * TS + c);
            dst[0] = hi; dst[L * TS / 2] = mid; dst[L * TS] = lo;
            split(w2[0], w2[1], hi, mid, lo);
            dst = reinterpret_cast<uint32_t*>(s.planes.w2 + t * TS + c);
            dst[0] = hi; dst[L * TS / 2] = mid; dst[L * TS] = lo;
          }
        }
#pragma unroll
    for (int n = 0; n < 2; ++n)
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        float v = db[n][i];
#pragma unroll
        for (int o = 4; o < 32; o <<= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
        if (g8 == 0) s.dbeta[warp][n0 + n * 8 + j2 + i] = v;
      }
  }
  __syncthreads();
  // dO S^T, -dR S^T and U dS'^T for this warp's 16 channels
  const int d0 = warp * 16;
  float aq[4][2][4], al[4][2][4], ar[4][2][4], sdot[2] = {};
#pragma unroll
  for (int m = 0; m < 4; ++m)
#pragma unroll
    for (int n = 0; n < 2; ++n)
#pragma unroll
      for (int i = 0; i < 4; ++i) aq[m][n][i] = al[m][n][i] = ar[m][n][i] = 0.f;
  {
    const float* const state = p.state + (slot * DV + j2) * DK + d0 + g8;
    const float* const dstate = p.dstate + (slot * DV + j2) * DK + d0 + g8;
#pragma unroll 1
    for (int kk = 0; kk < DV; kk += 16) {
      uint32_t b[2][3][2], e[2][3][2];
#pragma unroll
      for (int n = 0; n < 2; ++n)
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const int at = (kk + h * 8) * DK + n * 8;
          const float x0 = __ldg(state + at), x1 = __ldg(state + at + DK), y0 = __ldg(dstate + at), y1 = __ldg(dstate + at + DK);
          sdot[n] = fmaf(x0, y0, fmaf(x1, y1, sdot[n]));
          split(x0, x1, b[n][0][h], b[n][1][h], b[n][2][h]);
          split(y0, y1, e[n][0][h], e[n][1][h], e[n][2][h]);
        }
#pragma unroll
      for (int m = 0; m < 4; ++m) {
        uint32_t a[3][4], ao[4];
        load_mk(ao, s.go, VS, m * 16, kk, lane);
        mma_tiles_exact<3>(aq[m], ao, b, 2);
#pragma unroll
        for (int pl = 0; pl < 3; ++pl) load_mk(a[pl], s.r + pl * L * VS, VS, m * 16, kk, lane);
        mma_tiles<3>(al[m], a, b, 2);
#pragma unroll
        for (int pl = 0; pl < 3; ++pl) load_mk(a[pl], s.u + pl * L * VS, VS, m * 16, kk, lane);
        mma_tiles<3>(ar[m], a, e, 2);
      }
    }
  }
  float zcol[2][2] = {};
#pragma unroll
  for (int m = 0; m < 4; ++m)
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int t = m * 16 + g8 + 8 * h;
      float fq, fl, fr, rowsum = 0.f;
      if constexpr (!CHANNEL) {
        const float grow = exp2f(s.decay[t]);
        fq = grow * s.nq[t];
        fl = -grow * s.nk[t];
        fr = exp2f(s.decay[L - 1] - s.decay[t]) * s.nk[t];
      }
#pragma unroll
      for (int n = 0; n < 2; ++n) {
        const int d = d0 + n * 8 + j2;
        const float2 kv = floats(*reinterpret_cast<const uint32_t*>(s.k + t * KS + d));
        float2 c, end;
        if constexpr (CHANNEL) {
          c = __ldg(reinterpret_cast<const float2*>(p.decay + (slot * L + t) * DK + d));
          end = __ldg(reinterpret_cast<const float2*>(p.decay + (slot * L + L - 1) * DK + d));
        }
#pragma unroll
        for (int i = 0; i < 2; ++i) {
          if constexpr (CHANNEL) {
            const float ci = i ? c.y : c.x, grow = exp2f(ci);
            fq = grow * s.nq[t];
            fl = -grow * s.nk[t];
            fr = exp2f((i ? end.y : end.x) - ci) * s.nk[t];
          }
          aq[m][n][2 * h + i] *= fq;
          al[m][n][2 * h + i] *= fl;
          const float v = ar[m][n][2 * h + i] * fr, kx = (i ? kv.y : kv.x) * v;
          rowsum += kx;
          zcol[n][i] = fmaf(s.beta[t], kx, zcol[n][i]);
          ar[m][n][2 * h + i] = v * s.beta[t];
        }
      }
      rowsum += __shfl_xor_sync(0xffffffffu, rowsum, 1);
      rowsum += __shfl_xor_sync(0xffffffffu, rowsum, 2);
      if ((lane & 3) == 0) s.dbeta[NW + warp][t] = rowsum;
    }
#pragma unroll
  for (int n = 0; n < 2; ++n) {
    sdot[n] += __shfl_xor_sync(0xffffffffu, sdot[n], 1);
    sdot[n] += __shfl_xor_sync(0xffffffffu, sdot[n], 2);  // channel d0 + n * 8 + g8
    const float grow_end = exp2f(CHANNEL ? __ldg(p.decay + (slot * L + L - 1) * DK + d0 + n * 8 + g8) : s.decay[L - 1]);
    const float value = sdot[n] * grow_end;
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      float z = zcol[n][i];
#pragma unroll
      for (int o = 4; o < 32; o <<= 1) z += __shfl_xor_sync(0xffffffffu, z, o);  // channel d0 + n * 8 + j2 + i
      const float other = __shfl_sync(0xffffffffu, value, (j2 + i) * 4);         // the lane whose g8 is this channel's
      if (g8 == 0) s.end[d0 + n * 8 + j2 + i] = z + other;
    }
  }
  if constexpr (!CHANNEL) {
    const bf16 *const w1 = s.planes.w1, *const w2 = s.planes.w2;
#pragma unroll
    for (int ks = 0; ks < 4; ++ks) {
      uint32_t bk[2][1][2], bq[2][1][2];
      load_b<1, true>(bk, s.k, 0, KS, d0, ks * 16, lane);
      load_b<1, true>(bq, s.q, 0, KS, d0, ks * 16, lane);
#pragma unroll
      for (int m = 0; m < 4; ++m) {
        uint32_t a[3][4];
        if (m >= ks) {  // rows t of block m, columns s of block ks
#pragma unroll
          for (int pl = 0; pl < 3; ++pl) load_mk(a[pl], w1 + pl * L * TS, TS, m * 16, ks * 16, lane);
          mma_tiles<1>(aq[m], a, bk, 2);
#pragma unroll
          for (int pl = 0; pl < 3; ++pl) load_mk(a[pl], w2 + pl * L * TS, TS, m * 16, ks * 16, lane);
          mma_tiles<1>(al[m], a, bk, 2);
        }
        if (m <= ks) {  // transposed: columns s of block m, rows t of block ks
#pragma unroll
          for (int pl = 0; pl < 3; ++pl) load_km(a[pl], w1 + pl * L * TS, TS, ks * 16, m * 16, lane);
          mma_tiles<1>(ar[m], a, bq, 2);
#pragma unroll
          for (int pl = 0; pl < 3; ++pl) load_km(a[pl], w2 + pl * L * TS, TS, ks * 16, m * 16, lane);
          mma_tiles<1>(ar[m], a, bk, 2);
        }
      }
    }
  }
  __syncthreads();  // every warp is done with the planes of U and dR: their space takes the gradients
#pragma unroll
  for (int m = 0; m < 4; ++m)
#pragma unroll
    for (int n = 0; n < 2; ++n)
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const int at = (m * 16 + g8 + 8 * h) * GS + d0 + n * 8 + j2;
        *reinterpret_cast<float2*>(s.gq + at) = make_float2(aq[m][n][2 * h], aq[m][n][2 * h + 1]);
        *reinterpret_cast<float2*>(s.gl + at) = make_float2(al[m][n][2 * h], al[m][n][2 * h + 1]);
        *reinterpret_cast<float2*>(s.gr + at) = make_float2(ar[m][n][2 * h], ar[m][n][2 * h + 1]);
      }
  __syncthreads();
  if constexpr (CHANNEL) {
    // The pairs inside the chunk: a thread per channel and parity of t, 16 columns s at a time with their decays, keys and
    // gradients in registers.  Bounded by the exponentials.
    const int d = tid % DK, parity = tid / DK;
    const float* const decay = p.decay + slot * L * DK + d;
#pragma unroll 1
    for (int sb = 0; sb < L; sb += 16) {
      float cs[16], ks[16], acc[16];
#pragma unroll
      for (int i = 0; i < 16; ++i) {
        cs[i] = __ldg(decay + (sb + i) * DK);
        ks[i] = __bfloat162float(s.k[(sb + i) * KS + d]);
        acc[i] = 0.f;
      }
#pragma unroll 1
      for (int t = sb + parity; t < L; t += 2) {
        const float ct = __ldg(decay + t * DK), kt = __bfloat162float(s.k[t * KS + d]), qt = __bfloat162float(s.q[t * KS + d]);
        float gq = 0.f, gl = 0.f;
#pragma unroll
        for (int i4 = 0; i4 < 16; i4 += 4) {
          const float4 a = *reinterpret_cast<const float4*>(s.full.w1 + t * WS + sb + i4), b = *reinterpret_cast<const float4*>(s.full.w2 + t * WS + sb + i4);
          const float av[4] = {a.x, a.y, a.z, a.w}, bv[4] = {b.x, b.y, b.z, b.w};
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            const float e = exp2f(fminf(ct - cs[i4 + i], 0.f)), ek = e * ks[i4 + i];
            gq = fmaf(av[i], ek, gq);
            gl = fmaf(bv[i], ek, gl);
            acc[i4 + i] = fmaf(e, fmaf(av[i], qt, bv[i] * kt), acc[i4 + i]);
          }
        }
        s.gq[t * GS + d] += gq;
        s.gl[t * GS + d] += gl;
      }
      if (parity == 0) {
#pragma unroll
        for (int i = 0; i < 16; ++i) s.gr[(sb + i) * GS + d] += acc[i];
      }
      __syncthreads();
      if (parity == 1) {
#pragma unroll
        for (int i = 0; i < 16; ++i) s.gr[(sb + i) * GS + d] += acc[i];
      }
    }
    __syncthreads();
    if (tid < DK) {
      float run = s.end[tid];
#pragma unroll 4
      for (int t = L - 1; t >= 0; --t) {
        const float kt = __bfloat162float(s.k[t * KS + tid]), qt = __bfloat162float(s.q[t * KS + tid]);
        run += qt * s.gq[t * GS + tid] + kt * (s.gl[t * GS + tid] - s.gr[t * GS + tid]);
        if (t < len) p.dg[((long long)(span.x + t) * p.heads + head) * DK + tid] = run;
      }
    }
  }
  // through the norms, and out: a warp per row
  for (int t = warp; t < len; t += NW) {
    constexpr int PER = DK / 32;
    float q[PER], k[PER], gq[PER], gk[PER], a = 0.f, bl = 0.f, br = 0.f;
#pragma unroll
    for (int i = 0; i < PER; i += 2) {
      const int d = lane * PER + i;
      const float2 qv = floats(*reinterpret_cast<const uint32_t*>(s.q + t * KS + d)), kv = floats(*reinterpret_cast<const uint32_t*>(s.k + t * KS + d));
      const float2 x = *reinterpret_cast<const float2*>(s.gq + t * GS + d), l = *reinterpret_cast<const float2*>(s.gl + t * GS + d),
                   r = *reinterpret_cast<const float2*>(s.gr + t * GS + d);
      q[i] = qv.x; q[i + 1] = qv.y; k[i] = kv.x; k[i + 1] = kv.y;
      gq[i] = x.x; gq[i + 1] = x.y; gk[i] = l.x + r.x; gk[i + 1] = l.y + r.y;
      a += qv.x * x.x + qv.y * x.y;
      bl += kv.x * l.x + kv.y * l.y;
      br += kv.x * r.x + kv.y * r.y;
    }
    a = flb::warp_sum(a);
    bl = flb::warp_sum(bl);
    br = flb::warp_sum(br);
    if (lane == 0) s.dc[t] = a + bl - br;
    float fq = 0.f, fk = 0.f;
    if (p.normalize) {
      const float rq = s.nq[t] / p.scale;
      fq = rq * rq * a;
      fk = s.nk[t] * s.nk[t] * (bl + br);
    }
    const long long at = ((long long)(span.x + t) * p.heads + head) * DK + lane * PER;
#pragma unroll
    for (int i = 0; i < PER; i += 2) {
      *reinterpret_cast<bf162*>(p.dq + at + i) = __floats2bfloat162_rn(gq[i] - fq * q[i], gq[i + 1] - fq * q[i + 1]);
      *reinterpret_cast<bf162*>(p.dk + at + i) = __floats2bfloat162_rn(gk[i] - fk * k[i], gk[i + 1] - fk * k[i + 1]);
    }
  }
  __syncthreads();
  if (tid < len) {
    float sum = 0.f;
#pragma unroll
    for (int w = 0; w < 2 * NW; ++w) sum += s.dbeta[w][tid];
    p.dbeta[(long long)(span.x + tid) * p.heads + head] = sum;
  }
  if (!CHANNEL && warp == 0) {
    float end = 0.f;
#pragma unroll
    for (int d = lane; d < DK; d += 32) end += s.end[d];
    end = flb::warp_sum(end);
    float hi = lane + 32 < len ? s.dc[lane + 32] : 0.f, lo = lane < len ? s.dc[lane] : 0.f;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {  // sums over the lanes behind
      const float x = __shfl_down_sync(0xffffffffu, hi, o), y = __shfl_down_sync(0xffffffffu, lo, o);
      if (lane + o < 32) { hi += x; lo += y; }
    }
    lo += __shfl_sync(0xffffffffu, hi, 0);
    if (lane + 32 < len) p.dg[(long long)(span.x + lane + 32) * p.heads + head] = hi + end;
    if (lane < len) p.dg[(long long)(span.x + lane) * p.heads + head] = lo + end;
  }
}

// ---- host ----------------------------------------------------------------------------------------------------------
template <typename F>
bool allow_smem(F kernel, int bytes) {
  return cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes) == cudaSuccess;
}

template <int DK, bool CHANNEL>
int launch_forward(const DeltaArgs& a, int max_chunks, cudaStream_t stream) {
  constexpr int kPrepare = sizeof(PrepareSmem<DK, CHANNEL>), kScan = sizeof(ScanFwdSmem<DK, CHANNEL>), kOut = sizeof(OutputSmem<DK, CHANNEL>);
  static const bool ready = allow_smem(delta_prepare_kernel<DK, CHANNEL>, kPrepare) && allow_smem(delta_scan_fwd_kernel<DK, CHANNEL>, kScan) &&
                            allow_smem(delta_output_kernel<DK, CHANNEL>, kOut);
  if (!ready) return FLB_ERR_CUDA;
  delta_prepare_kernel<DK, CHANNEL><<<dim3(max_chunks, a.heads), 128, kPrepare, stream>>>(a);
  delta_scan_fwd_kernel<DK, CHANNEL><<<dim3(a.docs, a.heads, a.dv / kScanCols), kScanThreads, kScan, stream>>>(a);
  delta_output_kernel<DK, CHANNEL><<<dim3(max_chunks, a.heads), a.dv * 2, kOut, stream>>>(a);
  FLB_CHECK_LAUNCH();
  return FLB_OK;
}
template <int DK, int DV, bool CHANNEL>
int launch_backward(const DeltaArgs& a, int max_chunks, cudaStream_t stream) {
  constexpr int kScan = sizeof(ScanBwdSmem<DK, CHANNEL>), kLocal = sizeof(BackwardSmem<DK, DV, CHANNEL>);
  static_assert(kScan <= 227 * 1024 && kLocal <= 227 * 1024, "shared memory");
  static const bool ready = allow_smem(delta_scan_bwd_kernel<DK, CHANNEL>, kScan) && allow_smem(delta_backward_kernel<DK, DV, CHANNEL>, kLocal);
  if (!ready) return FLB_ERR_CUDA;
  delta_scan_bwd_kernel<DK, CHANNEL><<<dim3(a.docs, a.heads, a.dv / kScanCols), kScanThreads, kScan, stream>>>(a);
  delta_backward_kernel<DK, DV, CHANNEL><<<dim3(max_chunks, a.heads), DK * 2, kLocal, stream>>>(a);
  FLB_CHECK_LAUNCH();
  return FLB_OK;
}
bool supported(int heads, int repeat, int dk, int dv) {
  return heads > 0 && repeat > 0 && heads % repeat == 0 && (dk == 64 || dk == 128) && (dv == 64 || dv == 128);
}
}  // namespace

// Chunks a batch can have at most: `docs` documents (the padding behind the last one counts) of `tokens` tokens together.
FLB_API int flb_delta_max_chunks(long long tokens, int docs) { return (int)(tokens / L) + docs; }
// cu: document boundaries [docs] on the device (the last entry ends the last document; behind it is padding), or null: one document.
FLB_API int flb_delta_chunks(const int* cu, int docs, int total, int2* chunk, int* doc_chunk, cudaStream_t stream) {
  if (docs <= 0 || total < 0) return FLB_ERR_SHAPE;
  delta_chunks_kernel<<<1, 256, 0, stream>>>(cu, docs, total, chunk, doc_chunk);
  FLB_CHECK_LAUNCH();
  return FLB_OK;
}
// q, k: bf16 [tokens, heads / repeat, dk] (row strides given, heads adjacent); v: bf16 [tokens, heads, dv]; g: fp32 log decay
// [tokens, heads] or, `channel`, [tokens, heads, dk]; beta: fp32 [tokens, heads].  Outputs and intermediates as in DeltaArgs
// (tri_n may be null when no backward follows; k_in, k_out, q_in are used with `channel` only).
FLB_API int flb_delta_fwd(const bf16* q, const bf16* k, const bf16* v, long long q_row, long long k_row, long long v_row, const float* g, const float* beta,
                          int heads, int repeat, int dk, int dv, int channel, int normalize, float scale, const int2* chunk, const int* doc_chunk, int docs,
                          int max_chunks, float* decay, float* norm_q, float* norm_k, bf16* tri_t, bf16* tri_p, float* tri_n, bf16* k_in, bf16* k_out,
                          bf16* q_in, float* u, float* state, bf16* out, cudaStream_t stream) {
  if (!supported(heads, repeat, dk, dv) || (q_row | k_row | v_row) % 8 || ((uintptr_t)q | (uintptr_t)k | (uintptr_t)v) % 16) return FLB_ERR_SHAPE;
  if (max_chunks == 0) return FLB_OK;
  DeltaArgs a{};
  a.q = q; a.k = k; a.v = v; a.q_row = q_row; a.k_row = k_row; a.v_row = v_row; a.heads = heads; a.repeat = repeat; a.dv = dv; a.g = g; a.beta = beta;
  a.chunk = chunk; a.doc_chunk = doc_chunk; a.docs = docs; a.normalize = normalize; a.scale = scale; a.decay = decay; a.norm_q = norm_q; a.norm_k = norm_k;
  a.tri_t = tri_t; a.tri_p = tri_p; a.tri_n = tri_n; a.k_in = k_in; a.k_out = k_out; a.q_in = q_in; a.u = u; a.state = state; a.out = out;
  if (channel) return dk == 64 ? launch_forward<64, true>(a, max_chunks, stream) : launch_forward<128, true>(a, max_chunks, stream);
  return dk == 64 ? launch_forward<64, false>(a, max_chunks, stream) : launch_forward<128, false>(a, max_chunks, stream);
}
// dout: bf16 [tokens, heads, dv] contiguous.  dq, dk: bf16 [tokens, heads, dk] per VALUE head; dvalue like v; dg like g; dbeta like beta.
FLB_API int flb_delta_bwd(const bf16* q, const bf16* k, long long q_row, long long k_row, const float* beta, int heads, int repeat, int dk, int dv,
                          int channel, int normalize, float scale, const int2* chunk, const int* doc_chunk, int docs, int max_chunks, const float* decay,
                          const float* norm_q, const float* norm_k, const bf16* tri_t, const bf16* tri_p, const float* tri_n, const bf16* k_in,
                          const bf16* k_out, const bf16* q_in, const float* u, const float* state, const bf16* dout, float* dr, float* dstate, bf16* dq,
                          bf16* dkey, bf16* dvalue, float* dg, float* dbeta, cudaStream_t stream) {
  if (!supported(heads, repeat, dk, dv) || (q_row | k_row) % 8 || ((uintptr_t)q | (uintptr_t)k | (uintptr_t)dout) % 16) return FLB_ERR_SHAPE;
  if (max_chunks == 0) return FLB_OK;
  DeltaArgs a{};
  a.q = q; a.k = k; a.q_row = q_row; a.k_row = k_row; a.heads = heads; a.repeat = repeat; a.dv = dv; a.beta = beta; a.chunk = chunk;
  a.doc_chunk = doc_chunk; a.docs = docs; a.normalize = normalize; a.scale = scale;
  a.decay = const_cast<float*>(decay); a.norm_q = const_cast<float*>(norm_q); a.norm_k = const_cast<float*>(norm_k);
  a.tri_t = const_cast<bf16*>(tri_t); a.tri_p = const_cast<bf16*>(tri_p); a.tri_n = const_cast<float*>(tri_n);
  a.k_in = const_cast<bf16*>(k_in); a.k_out = const_cast<bf16*>(k_out); a.q_in = const_cast<bf16*>(q_in);
  a.u = const_cast<float*>(u); a.state = const_cast<float*>(state); a.dout = dout; a.dr = dr; a.dstate = dstate;
  a.dq = dq; a.dk = dkey; a.dvalue = dvalue; a.dg = dg; a.dbeta = dbeta;
  if (dk == 64) {
    if (dv == 64) return channel ? launch_backward<64, 64, true>(a, max_chunks, stream) : launch_backward<64, 64, false>(a, max_chunks, stream);
    return channel ? launch_backward<64, 128, true>(a, max_chunks, stream) : launch_backward<64, 128, false>(a, max_chunks, stream);
  }
  if (dv == 64) return channel ? launch_backward<128, 64, true>(a, max_chunks, stream) : launch_backward<128, 64, false>(a, max_chunks, stream);
  return channel ? launch_backward<128, 128, true>(a, max_chunks, stream) : launch_backward<128, 128, false>(a, max_chunks, stream);
}
