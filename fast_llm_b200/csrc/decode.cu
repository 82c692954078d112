// One generation step of an attention decoder: a single new position for each of up to 32 rows, from one host call.
//
// A step does a handful of FLOPs per weight byte, so it is bounded by the weights' trip from HBM, then by launches and by the host:
// through the Python layers it took 3.6 ms for 8 blocks of 2048 where the weights take 0.17.  Here the kernels of a longer pass run
// one after another on the same numbers in the same order (the same logits, bit for bit), with three differences: the new keys and
// values are appended to one cache buffer instead of copying all earlier ones, the residual add after the MLP rides in the next
// block's norm, and the GEMMs (gemm_rows_kernel) start reading their weights while the kernel ahead of them runs.
// 8 blocks of 2048 / 8192, a prompt and 24 steps: one row after 100 positions 92 -> 18.5 ms, 8 rows after 512 95 -> 22 ms; a step is 0.6 ms
// of kernels one after another, half of it the GEMMs of the MLP.
#include "common.cuh"

FLB_API int flb_norm_fwd(const void* x, const void* delta, const void* w, const void* b, void* res_out, void* y, float* rstd, float* mean, int rows,
                         int cols, float eps, int zero_centered, int layer_norm, cudaStream_t stream);
FLB_API int flb_gemm_bf16_ex(const void* A, const void* B, void* C, int M, int N, int K, long long lda, long long ldb, long long ldc, int a_mn_major,
                             int b_mn_major, int epilogue, int block_n, int max_ctas, int flags, cudaStream_t stream);
FLB_API int flb_rope(void* x, const float* table, const int* positions, long long tokens, long long row_stride, int n_heads, int head_dim, int rot_dim,
                     int conj, cudaStream_t stream);
FLB_API int flb_attention_fwd(const void* q, long long q_stride, int q_col0, const void* kv, long long kv_stride, int k_col0, int v_col0, const int* cu_q,
                              const int* cu_k, int batch, int max_seqlen_q, long long total_q, long long total_k, int heads, int kv_heads, int head_dim,
                              void* out, float* lse, int causal, int window, float softmax_scale, cudaStream_t stream);
FLB_API int flb_act_fwd(const void* in, void* out, long long rows, int n, int gated, int type, cudaStream_t stream);
FLB_API int flb_embedding_fwd(const long long* ids, const void* w, void* out, long long tokens, int hidden, long long vocab_begin, long long vocab_end,
                              float scale, cudaStream_t stream);

namespace {
using bf16 = __nv_bfloat16;
constexpr int kMaxRows = 32;
enum NormKind : int { kNormLayer = 2, kNormZeroCentered = 4 };  // 1: RMS

// The packed documents of the attention kernel: a row of the cache is its left padding (no queries), the row's own positions with the
// new one as the only query, and the room behind it (no queries).
__global__ void decode_layout_kernel(const int* __restrict__ pads, int rows, int capacity, int length, int* __restrict__ positions, int* __restrict__ cu_q,
                                     int* __restrict__ cu_k) {
  const int r = threadIdx.x;
  if (r < rows) {
    positions[r] = length - pads[r];
    cu_q[3 * r] = cu_q[3 * r + 1] = r;
    cu_q[3 * r + 2] = r + 1;
    cu_k[3 * r] = r * capacity;
    cu_k[3 * r + 1] = r * capacity + pads[r];
    cu_k[3 * r + 2] = r * capacity + length + 1;
  }
  if (r == 0) {
    cu_q[3 * rows] = rows;
    cu_k[3 * rows] = rows * capacity;
  }
}

// Keys and values of the new position (columns from `offset` of the projection's rows) into the cache.
__global__ void decode_append_kernel(const bf16* __restrict__ qkv, int qkv_width, int offset, bf16* __restrict__ cache, long long row_stride, int width) {
  const uint4* src = reinterpret_cast<const uint4*>(qkv + (long long)blockIdx.x * qkv_width + offset);
  uint4* dst = reinterpret_cast<uint4*>(cache + blockIdx.x * row_stride);
  for (int i = threadIdx.x; i < width / 8; i += blockDim.x) dst[i] = src[i];
}

__global__ void decode_bias_kernel(bf16* __restrict__ x, const bf16* __restrict__ bias, int cols) {
  for (int i = threadIdx.x; i < cols; i += blockDim.x) {
    bf16* at = x + (long long)blockIdx.x * cols + i;
    *at = __float2bfloat16_rn(__bfloat162float(*at) + __bfloat162float(bias[i]));
  }
}
}  // namespace

// One decoder block as the host describes it (mirrored by a ctypes structure).
struct FlbDecodeLayer {
  const bf16 *norm1_w, *norm1_b, *qkv_w, *qkv_b, *dense_w, *dense_b, *norm2_w, *norm2_b, *w1, *b1, *w2, *b2;
  const float* table;
  int norm1, norm2, heads, kv_heads, head_dim, rot_dim, window, ffn, gated, act;
  float eps1, eps2, scale;
};

FLB_API int flb_decode_supported(const FlbDecodeLayer* layers, int count, int hidden, int rows) {
  if (rows < 1 || rows > kMaxRows || hidden % 8 || hidden > 16384) return 0;
  for (int i = 0; i < count; ++i) {
    const FlbDecodeLayer& l = layers[i];
    if (l.head_dim <= 0 || l.head_dim > 128 || l.head_dim % 8 || l.heads % l.kv_heads || l.rot_dim % 16 || l.rot_dim > l.head_dim || l.ffn % 16) return 0;
  }
  return 1;
}

namespace {
// Intermediates of a step in one buffer, every part on a 256-byte boundary.
struct Workspace {
  bf16 *x, *residual, *hidden, *delta, *qkv, *attn, *wide, *inner;
  float *rstd, *mean, *lse;
  int *positions, *cu_q, *cu_k;
  long long bytes = 0;
  Workspace(unsigned char* base, const FlbDecodeLayer* layers, int count, int hidden_size, int rows) {
    long long qkv_n = 0, attn_n = 0, wide_n = 0, inner_n = 0, heads = 0;
    for (int i = 0; i < count; ++i) {
      const FlbDecodeLayer& l = layers[i];
      auto most = [](long long& a, long long b) { a = a > b ? a : b; };
      most(qkv_n, (l.heads + 2ll * l.kv_heads) * l.head_dim);
      most(attn_n, (long long)l.heads * l.head_dim);
      most(wide_n, (l.gated ? 2ll : 1ll) * l.ffn);
      most(inner_n, l.ffn);
      most(heads, l.heads);
    }
    auto take = [&](long long size) {
      unsigned char* at = base + bytes;
      bytes += (size + 255) / 256 * 256;
      return at;
    };
    auto rows_of = [&](long long n) { return reinterpret_cast<bf16*>(take(2 * n * rows)); };
    x = rows_of(hidden_size); residual = rows_of(hidden_size); hidden = rows_of(hidden_size); delta = rows_of(hidden_size);
    qkv = rows_of(qkv_n); attn = rows_of(attn_n); wide = rows_of(wide_n); inner = rows_of(inner_n);
    rstd = reinterpret_cast<float*>(take(4 * rows)); mean = reinterpret_cast<float*>(take(4 * rows)); lse = reinterpret_cast<float*>(take(4 * heads * rows));
    positions = reinterpret_cast<int*>(take(4 * rows));
    cu_q = reinterpret_cast<int*>(take(4 * (3 * rows + 1))); cu_k = reinterpret_cast<int*>(take(4 * (3 * rows + 1)));
  }
};
}  // namespace

FLB_API long long flb_decode_workspace(const FlbDecodeLayer* layers, int count, int hidden, int rows) {
  return Workspace(nullptr, layers, count, hidden, rows).bytes;
}

// `ids` [rows]; `cache`: [layers][rows][capacity][2 kv_heads head_dim] with `cache_layer` elements between layers, the first `length`
// positions of every row filled, position `length` written here, everything behind it finite; `pads` [rows] on the device; `workspace`:
// flb_decode_workspace bytes on a 256-byte boundary; `logits` [rows, vocab] fp32.
FLB_API int flb_decode_step(const FlbDecodeLayer* layers, int count, const long long* ids, int rows, const bf16* embedding, float embedding_scale,
                            int hidden, int vocab, const bf16* final_w, const bf16* final_b, int final_norm, float final_eps, const bf16* head_w,
                            bf16* cache, long long cache_layer, int capacity, int length, const int* pads, void* workspace, float* logits,
                            cudaStream_t stream) {
  if (!flb_decode_supported(layers, count, hidden, rows) || length >= capacity) return FLB_ERR_SHAPE;
  Workspace w((unsigned char*)workspace, layers, count, hidden, rows);
  constexpr int kStoreBf16 = 0, kStoreF32 = 1, kOverlap = 2;
  int status = FLB_OK;
  bf16* delta = nullptr;  // what the next norm adds to x
  auto norm = [&](const bf16* weight, const bf16* bias, int kind, float eps) {
    status = flb_norm_fwd(w.x, delta, weight, bias, delta ? w.residual : nullptr, w.hidden, w.rstd, w.mean, rows, hidden, eps,
                          (kind & kNormZeroCentered) != 0, (kind & 3) == kNormLayer, stream);
    if (delta) { bf16* t = w.x; w.x = w.residual; w.residual = t; }
    return status == FLB_OK;
  };
  // a [rows, k] times [n, k] (or [k, n]) weights
  auto linear = [&](const bf16* a, const bf16* weight, const bf16* bias, void* out, int n, int k, bool transposed, int epilogue) {
    status = flb_gemm_bf16_ex(a, weight, out, rows, n, k, k, transposed ? n : k, n, 0, transposed, epilogue, 0, 0, kOverlap, stream);
    if (status == FLB_OK && bias != nullptr) decode_bias_kernel<<<rows, 256, 0, stream>>>((bf16*)out, bias, n);
    return status == FLB_OK;
  };
  decode_layout_kernel<<<1, 32, 0, stream>>>(pads, rows, capacity, length, w.positions, w.cu_q, w.cu_k);
  if ((status = flb_embedding_fwd(ids, embedding, w.x, rows, hidden, 0, vocab, embedding_scale, stream)) != FLB_OK) return status;
  for (int i = 0; i < count; ++i) {
    const FlbDecodeLayer& l = layers[i];
    const int attn = l.heads * l.head_dim, width = 2 * l.kv_heads * l.head_dim;
    bf16* const kv = cache + i * cache_layer;
    if (!norm(l.norm1_w, l.norm1_b, l.norm1, l.eps1) || !linear(w.hidden, l.qkv_w, l.qkv_b, w.qkv, attn + width, hidden, false, kStoreBf16)) return status;
    if (l.rot_dim && (status = flb_rope(w.qkv, l.table, w.positions, rows, attn + width, l.heads + l.kv_heads, l.head_dim, l.rot_dim, 0, stream)) != FLB_OK)
      return status;
    decode_append_kernel<<<rows, 128, 0, stream>>>(w.qkv, attn + width, attn, kv + (long long)length * width, (long long)capacity * width, width);
    status = flb_attention_fwd(w.qkv, attn + width, 0, kv, width, 0, width / 2, w.cu_q, w.cu_k, 3 * rows, 1, rows, (long long)rows * capacity, l.heads,
                               l.kv_heads, l.head_dim, w.attn, w.lse, 1, l.window, l.scale, stream);
    if (status != FLB_OK || !linear(w.attn, l.dense_w, l.dense_b, w.delta, hidden, attn, false, kStoreBf16)) return status;
    delta = w.delta;
    if (!norm(l.norm2_w, l.norm2_b, l.norm2, l.eps2) || !linear(w.hidden, l.w1, l.b1, w.wide, (l.gated ? 2 : 1) * l.ffn, hidden, false, kStoreBf16)) return status;
    if ((status = flb_act_fwd(w.wide, w.inner, rows, l.ffn, l.gated, l.act, stream)) != FLB_OK) return status;
    if (!linear(w.inner, l.w2, l.b2, w.delta, hidden, l.ffn, true, kStoreBf16)) return status;
  }
  if (!norm(final_w, final_b, final_norm, final_eps) || !linear(w.hidden, head_w, nullptr, logits, vocab, hidden, false, kStoreF32)) return status;
  FLB_CHECK_LAUNCH();
  return FLB_OK;
}
