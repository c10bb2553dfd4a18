// Encoder-only (BERT family) pieces that the decoder stack does not have:
//
//  * embedding: word + position + token-type rows summed and layer-normalised in one pass
//    (the three gathers never touch HBM as separate tensors);
//  * pooling: CLS row or mean over each sequence's rows, then optional L2 normalisation,
//    written as fp32 (what the embedding service returns).
//
// The reference obtains these from the vLLM pooling model that its embedding replica wraps
// (arctic_inference/embedding/replica.py:83-128).

#include <string.h>

#include "api.h"
#include "common/pdl.cuh"
#include "common/ptx.cuh"

namespace ab200 {

typedef __nv_bfloat16 bf16;

constexpr int kEncThreads = 128;
constexpr int kEncMaxVec = 8;  // hidden <= 128 * 8 * 8 = 8192

__device__ __forceinline__ void enc_unpack8(const uint4& q, float (&f)[8]) {
  const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&q);
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const float2 t = __bfloat1622float2(h[i]);
    f[2 * i] = t.x;
    f[2 * i + 1] = t.y;
  }
}

__device__ __forceinline__ float enc_block_sum(float v, float* red) {
  v = warp_sum(v);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  __syncthreads();
  if (lane == 0) red[warp] = v;
  __syncthreads();
  float t = (lane < (kEncThreads >> 5)) ? red[lane] : 0.f;
  return warp_sum(t);
}

__global__ void __launch_bounds__(kEncThreads)
bert_embed_ln_kernel(const long long* __restrict__ ids, const long long* __restrict__ positions,
                     const long long* __restrict__ type_ids, const bf16* __restrict__ word,
                     const bf16* __restrict__ pos, const bf16* __restrict__ type,
                     const bf16* __restrict__ gamma, const bf16* __restrict__ beta,
                     bf16* __restrict__ out, int hidden, long long vocab, long long max_pos,
                     long long n_types, float eps, int* status) {
  __shared__ float red[32];
  const long long t = blockIdx.x;
  long long id = ids[t], p = positions[t], ty = type_ids ? type_ids[t] : 0;
  if (id < 0 || id >= vocab || p < 0 || p >= max_pos || ty < 0 || ty >= n_types) {
    if (threadIdx.x == 0) report_error(status, kErrBounds, 4, (int)t);
    id = 0;
    p = 0;
    ty = 0;
  }
  const int nvec = hidden / 8;
  const uint4* wr = reinterpret_cast<const uint4*>(word + id * hidden);
  const uint4* pr = reinterpret_cast<const uint4*>(pos + p * hidden);
  const uint4* tr = reinterpret_cast<const uint4*>(type + ty * hidden);
  float vals[kEncMaxVec][8];
  float s = 0.f;
#pragma unroll
  for (int j = 0; j < kEncMaxVec; ++j) {
    const int i = threadIdx.x + j * kEncThreads;
    if (i < nvec) {
      float a[8], b[8], c[8];
      enc_unpack8(wr[i], a);
      enc_unpack8(pr[i], b);
      enc_unpack8(tr[i], c);
#pragma unroll
      for (int k = 0; k < 8; ++k) {
        vals[j][k] = a[k] + b[k] + c[k];
        s += vals[j][k];
      }
    }
  }
  const float mean = enc_block_sum(s, red) / (float)hidden;
  float v = 0.f;
#pragma unroll
  for (int j = 0; j < kEncMaxVec; ++j) {
    const int i = threadIdx.x + j * kEncThreads;
    if (i < nvec) {
#pragma unroll
      for (int k = 0; k < 8; ++k) {
        const float d = vals[j][k] - mean;
        v += d * d;
      }
    }
  }
  const float inv = rsqrtf(enc_block_sum(v, red) / (float)hidden + eps);
  const uint4* gr = reinterpret_cast<const uint4*>(gamma);
  const uint4* br = reinterpret_cast<const uint4*>(beta);
  uint4* yr = reinterpret_cast<uint4*>(out + t * hidden);
#pragma unroll
  for (int j = 0; j < kEncMaxVec; ++j) {
    const int i = threadIdx.x + j * kEncThreads;
    if (i < nvec) {
      float g[8], b[8];
      enc_unpack8(gr[i], g);
      enc_unpack8(br[i], b);
      uint4 q;
      uint32_t* qw = reinterpret_cast<uint32_t*>(&q);
#pragma unroll
      for (int k = 0; k < 4; ++k)
        qw[k] = pack_bf16x2((vals[j][2 * k] - mean) * inv * g[2 * k] + b[2 * k],
                            (vals[j][2 * k + 1] - mean) * inv * g[2 * k + 1] + b[2 * k + 1]);
      yr[i] = q;
    }
  }
}

// ------------------------- attention of short sequences -------------------------
// Sequences of at most 128 tokens, heads of 64, every token sees all of its sequence: one block of four
// warps per (sequence, head), a warp per 16 query rows, the whole row of scores in registers.
//
// Bound by memory (a text of 50 tokens moves 25 KB per head and multiplies 0.6 MFLOP), so what counts is
// how many sequences are in flight on an SM: blocks are small (3 x 128 bytes of shared memory per
// token) and a block needs no tensor memory, barriers or 128-row tiles. Hence the register form of
// the tensor core's product (mma.sync) here; the tcgen05 kernel holds one (sequence, head) per SM at
// a time and spends 5 us on each. 328 texts of 50 tokens, 12 heads: 179 -> 35 us; 128 of 128 tokens: 72 -> 41.
constexpr int kShortThreads = 128;
constexpr int kShortDim = 64;
constexpr int kShortLen = 128;

__device__ __forceinline__ void ldmatrix_x4(uint32_t (&r)[4], uint32_t addr) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0, %1, %2, %3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
               : "r"(addr)
               : "memory");
}
__device__ __forceinline__ void ldmatrix_x4_trans(uint32_t (&r)[4], uint32_t addr) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0, %1, %2, %3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
               : "r"(addr)
               : "memory");
}
__device__ __forceinline__ void mma_16816(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, "
      "{%0, %1, %2, %3};"
      : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

// KEYS: 16-key groups that the registers hold (the sequence's length, rounded up)
template <int KEYS>
__global__ void __launch_bounds__(kShortThreads)
attention_short_kernel(const bf16* __restrict__ q, const bf16* __restrict__ k, const bf16* __restrict__ v,
                       long long ldq, long long ld_kv, const int* __restrict__ work, int heads, float scale_log2,
                       bf16* __restrict__ out, long long ldo) {
  constexpr int kRows = KEYS * 16;
  constexpr int kTile = kRows * 128;   // bytes of Q, of K and of V
  extern __shared__ __align__(128) uint8_t short_smem[];
  pdl_wait();
  pdl_trigger();
  const int* wk = work + (long long)(blockIdx.x / heads) * 8;
  const int head = blockIdx.x % heads;
  const int nq = min(wk[2], kRows), n = min(wk[5] - wk[4], kRows);   // queries, keys
  if (nq <= 0) return;
  const long long row0 = wk[1], key0 = wk[0] + wk[4];
  const uint32_t sq = smem_u32(short_smem);
  // rows of 128 bytes, their eight 16-byte chunks XORed with the row; rows past the end are zero
  for (int i = threadIdx.x; i < 3 * kRows * 8; i += kShortThreads) {
    const int which = i / (kRows * 8), r = i / 8 % kRows, c = i & 7;
    const bool in = r < (which == 0 ? nq : n);
    const bf16* src = (which == 0 ? q + (row0 + r) * ldq : (which == 1 ? k : v) + (key0 + r) * ld_kv) +
                      head * kShortDim + 8 * c;
    const uint32_t dst = sq + which * kTile + r * 128 + ((c ^ (r & 7)) << 4);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(in ? src : q),
                 "r"(in ? 16 : 0)
                 : "memory");
  }
  asm volatile("cp.async.commit_group;\n\tcp.async.wait_group 0;" ::: "memory");
  __syncthreads();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  // row and 16-byte chunk that this lane names in an ldmatrix of 16 rows by 16 columns
  const int lm_row = lane & 15, lm_chunk = lane >> 4;
  auto at = [&](int tile, int r, int c) { return sq + tile * kTile + r * 128 + ((c ^ (r & 7)) << 4); };
  for (int m0 = warp * 16; m0 < nq; m0 += kShortThreads / 2) {
    uint32_t a[4][4];
#pragma unroll
    for (int d = 0; d < 4; ++d) ldmatrix_x4(a[d], at(0, m0 + lm_row, 2 * d + lm_chunk));
    float s[2 * KEYS][4];
#pragma unroll
    for (int g = 0; g < KEYS; ++g) {
#pragma unroll
      for (int t = 0; t < 4; ++t) s[2 * g][t] = s[2 * g + 1][t] = 0.f;
      if (16 * g < n) {
#pragma unroll
        for (int d = 0; d < 4; ++d) {
          uint32_t b[4];   // keys 16g .. +7 | +8 .. +15, for the lower and the upper eight columns
          ldmatrix_x4(b, at(1, 16 * g + lm_row, 2 * d + lm_chunk));
          mma_16816(s[2 * g], a[d], b[0], b[2]);
          mma_16816(s[2 * g + 1], a[d], b[1], b[3]);
        }
      }
    }
    // a thread holds columns 2 (lane % 4) + {0, 1} of rows lane / 4 and lane / 4 + 8
    float mx[2] = {-INFINITY, -INFINITY}, sum[2] = {0.f, 0.f};
#pragma unroll
    for (int j = 0; j < 2 * KEYS; ++j)
#pragma unroll
      for (int t = 0; t < 4; ++t) {
        if (8 * j + 2 * (lane & 3) + (t & 1) >= n) s[j][t] = -INFINITY;
        mx[t >> 1] = fmaxf(mx[t >> 1], s[j][t]);
      }
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      mx[h] = fmaxf(mx[h], __shfl_xor_sync(0xffffffffu, mx[h], 1));
      mx[h] = fmaxf(mx[h], __shfl_xor_sync(0xffffffffu, mx[h], 2));
      mx[h] = mx[h] == -INFINITY ? 0.f : -mx[h] * scale_log2;
    }
    float o[8][4];
#pragma unroll
    for (int j = 0; j < 8; ++j)
#pragma unroll
      for (int t = 0; t < 4; ++t) o[j][t] = 0.f;
#pragma unroll
    for (int g = 0; g < KEYS; ++g) {
      if (16 * g >= n) continue;
      uint32_t p[4];
#pragma unroll
      for (int h = 0; h < 2; ++h)
#pragma unroll
        for (int r = 0; r < 2; ++r) {
          const float e0 = ex2_approx(fmaf(s[2 * g + h][2 * r], scale_log2, mx[r]));
          const float e1 = ex2_approx(fmaf(s[2 * g + h][2 * r + 1], scale_log2, mx[r]));
          sum[r] += e0 + e1;
          p[2 * h + r] = pack_bf16x2(e0, e1);
        }
#pragma unroll
      for (int d = 0; d < 4; ++d) {
        uint32_t b[4];   // keys 16g .. +7 | +8 .. +15 of columns 16d .. +7, then of 16d + 8 .. +15
        ldmatrix_x4_trans(b, at(2, 16 * g + lm_row, 2 * d + lm_chunk));
        mma_16816(o[2 * d], p, b[0], b[1]);
        mma_16816(o[2 * d + 1], p, b[2], b[3]);
      }
    }
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      sum[h] += __shfl_xor_sync(0xffffffffu, sum[h], 1);
      sum[h] += __shfl_xor_sync(0xffffffffu, sum[h], 2);
      sum[h] = sum[h] > 0.f ? 1.f / sum[h] : 0.f;
    }
    // whole rows leave through this warp's rows of Q
    __syncwarp();
#pragma unroll
    for (int j = 0; j < 8; ++j)
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const int r = m0 + (lane >> 2) + 8 * h;
        *reinterpret_cast<uint32_t*>(short_smem + r * 128 + ((j ^ (r & 7)) << 4) + 4 * (lane & 3)) =
            pack_bf16x2(o[j][2 * h] * sum[h], o[j][2 * h + 1] * sum[h]);
      }
    __syncwarp();
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int r = m0 + 4 * i + (lane >> 3), c = lane & 7;
      if (r < nq)
        *reinterpret_cast<uint4*>(out + (row0 + r) * ldo + head * kShortDim + 8 * c) =
            *reinterpret_cast<const uint4*>(short_smem + r * 128 + ((c ^ (r & 7)) << 4));
    }
  }
}

// One block per sequence. mode 0: first row (CLS); 1: mean over the rows; 2: last row.
__global__ void __launch_bounds__(kEncThreads)
pool_normalize_kernel(const bf16* __restrict__ h, long long ld, const long long* __restrict__ starts,
                      float* __restrict__ out, int hidden, int mode, int normalize) {
  __shared__ float red[32];
  const int sidx = blockIdx.x;
  const long long r0 = starts[sidx], r1 = starts[sidx + 1];
  const int nvec = hidden / 8;
  float acc[kEncMaxVec][8];
  float ss = 0.f;
#pragma unroll
  for (int j = 0; j < kEncMaxVec; ++j) {
    const int i = threadIdx.x + j * kEncThreads;
#pragma unroll
    for (int k = 0; k < 8; ++k) acc[j][k] = 0.f;
    if (i < nvec && r1 > r0) {
      if (mode == 1) {
        for (long long r = r0; r < r1; ++r) {
          float f[8];
          enc_unpack8(reinterpret_cast<const uint4*>(h + r * ld)[i], f);
#pragma unroll
          for (int k = 0; k < 8; ++k) acc[j][k] += f[k];
        }
        const float invn = 1.f / (float)(r1 - r0);
#pragma unroll
        for (int k = 0; k < 8; ++k) acc[j][k] *= invn;
      } else {
        const long long r = mode == 0 ? r0 : r1 - 1;
        enc_unpack8(reinterpret_cast<const uint4*>(h + r * ld)[i], acc[j]);
      }
#pragma unroll
      for (int k = 0; k < 8; ++k) ss += acc[j][k] * acc[j][k];
    }
  }
  float scale = 1.f;
  if (normalize) {
    const float tot = enc_block_sum(ss, red);
    scale = rsqrtf(fmaxf(tot, 1e-24f));
  }
#pragma unroll
  for (int j = 0; j < kEncMaxVec; ++j) {
    const int i = threadIdx.x + j * kEncThreads;
    if (i < nvec) {
      float4* o = reinterpret_cast<float4*>(out + (long long)sidx * hidden + i * 8);
      o[0] = make_float4(acc[j][0] * scale, acc[j][1] * scale, acc[j][2] * scale, acc[j][3] * scale);
      o[1] = make_float4(acc[j][4] * scale, acc[j][5] * scale, acc[j][6] * scale, acc[j][7] * scale);
    }
  }
}

}  // namespace ab200

using namespace ab200;

extern "C" {

int ab200_bert_embed_ln(const void* ids, const void* positions, const void* type_ids,
                        const void* word, const void* pos, const void* type, const void* gamma,
                        const void* beta, void* out, long long T, int hidden, long long vocab,
                        long long max_pos, long long n_types, float eps, int* status,
                        cudaStream_t stream) {
  if (T <= 0) return 0;
  if ((hidden % 8) || hidden > kEncThreads * kEncMaxVec * 8) return -2;
  bert_embed_ln_kernel<<<(unsigned)T, kEncThreads, 0, stream>>>(
      reinterpret_cast<const long long*>(ids), reinterpret_cast<const long long*>(positions),
      reinterpret_cast<const long long*>(type_ids), reinterpret_cast<const bf16*>(word),
      reinterpret_cast<const bf16*>(pos), reinterpret_cast<const bf16*>(type),
      reinterpret_cast<const bf16*>(gamma), reinterpret_cast<const bf16*>(beta),
      reinterpret_cast<bf16*>(out), hidden, vocab, max_pos, n_types, eps, status);
  return cudaGetLastError() == cudaSuccess ? 0 : -5;
}

// Bidirectional attention over packed sequences of at most 128 tokens, heads of 64: q, k, v rows of strides
// ldq, ld_kv; `work` as ab200_attention's (contiguous keys), one item per sequence; max_len: the longest.
int ab200_attention_short(const void* q, long long ldq, const void* k, const void* v, long long ld_kv,
                          const void* work, int num_work, int heads, int max_len, float scale, void* out,
                          long long ldo, cudaStream_t stream) {
  if (num_work <= 0) return 0;
  const uintptr_t at = reinterpret_cast<uintptr_t>(q) | reinterpret_cast<uintptr_t>(k) |
                       reinterpret_cast<uintptr_t>(v) | reinterpret_cast<uintptr_t>(out);
  if ((ldq % 8) || (ld_kv % 8) || (ldo % 8) || (at & 15) || max_len < 1 || max_len > kShortLen) return -2;
  const int groups = (max_len + 15) / 16;
  auto kernel = groups <= 2   ? attention_short_kernel<2>
                : groups <= 4 ? attention_short_kernel<4>
                : groups <= 6 ? attention_short_kernel<6>
                              : attention_short_kernel<8>;
  const int held = groups <= 2 ? 2 : groups <= 4 ? 4 : groups <= 6 ? 6 : 8;
  return launch_pdl(kernel, dim3((unsigned)num_work * (unsigned)heads), dim3(kShortThreads),
                    (size_t)held * 3 * 16 * 128, stream, reinterpret_cast<const bf16*>(q),
                    reinterpret_cast<const bf16*>(k), reinterpret_cast<const bf16*>(v), ldq, ld_kv,
                    reinterpret_cast<const int*>(work), heads, scale * 1.4426950408889634f,
                    reinterpret_cast<bf16*>(out), ldo) == cudaSuccess
             ? 0
             : -5;
}

// All layers of an encoder over a packed batch: h [T, hidden] in and out; x [T, hidden], a [T, hidden]
// and wide [T, max(3 hidden, inter)] are scratch. One call enqueues the seven kernels of every layer:
// from Python each launch costs 17 us of the host, more than the kernel takes for a short text. max_len > 0: heads of 64
// take the kernel for short sequences, of which this is the longest.
int ab200_bert_layers(const Ab200BertLayer* layers, int n_layers, void* h, void* x, void* wide, void* a,
                      int T, int hidden, int inter, int heads, int D, float eps, const void* work,
                      int num_work, int tile_keys, int max_len, int* status, cudaStream_t stream) {
  if (T <= 0 || n_layers <= 0) return 0;
  if (layers == nullptr || heads * D != hidden) return -2;
  const float scale = 1.f / sqrtf((float)D);
  char* qkv = reinterpret_cast<char*>(wide);
  const size_t part = (size_t)hidden * 2;   // bytes
  auto linear = [&](const void* in, const void* w, const void* bias, void* out, int n, int k, int act,
                    const void* residual) -> int {
    Ab200LinearDesc d;
    memset(&d, 0, sizeof(d));
    d.x = in;
    d.ldx = k;
    d.w = w;
    d.ldw = k;
    d.out = out;
    d.ldo = n;
    d.M = T;
    d.N = n;
    d.K = k;
    d.bias = bias;
    d.residual = residual;
    d.ldr = residual != nullptr ? n : 0;
    d.act = act;
    d.status = status;
    d.w_static = 1;   // parameters: nothing enqueued here writes them
    return ab200_linear_desc(&d, stream);
  };
  for (int l = 0; l < n_layers; ++l) {
    const Ab200BertLayer& w = layers[l];
    int rc = linear(h, w.wqkv, w.bqkv, wide, 3 * hidden, hidden, 0, nullptr);
    if (rc != 0) return rc;
    rc = D == kShortDim && max_len > 0
             ? ab200_attention_short(qkv, 3 * hidden, qkv + part, qkv + 2 * part, 3 * hidden, work, num_work,
                                     heads, max_len, scale, a, hidden, stream)
             : ab200_attention(qkv, 3 * hidden, qkv + part, qkv + 2 * part, 3 * hidden, T, 0, nullptr, 0, work,
                               num_work, nullptr, 1, T, heads, heads, D, 0, scale, a, hidden, nullptr, nullptr,
                               nullptr, tile_keys, status, stream);
    if (rc == 0) rc = linear(a, w.wo, w.bo, x, hidden, hidden, 0, h);
    if (rc == 0) rc = ab200_layernorm(x, nullptr, w.ln1_g, w.ln1_b, h, T, hidden, eps, stream);
    if (rc == 0) rc = linear(h, w.wi, w.bi, wide, inter, hidden, 1, nullptr);
    if (rc == 0) rc = linear(wide, w.wd, w.bd, x, hidden, inter, 0, h);
    if (rc == 0) rc = ab200_layernorm(x, nullptr, w.ln2_g, w.ln2_b, h, T, hidden, eps, stream);
    if (rc != 0) return rc;
  }
  return 0;
}

int ab200_pool_normalize(const void* h, long long ld, const void* starts, void* out, int n_seqs,
                         int hidden, int mode, int normalize, cudaStream_t stream) {
  if (n_seqs <= 0) return 0;
  if ((hidden % 8) || (ld % 8) || hidden > kEncThreads * kEncMaxVec * 8 || mode < 0 || mode > 2)
    return -2;
  pool_normalize_kernel<<<(unsigned)n_seqs, kEncThreads, 0, stream>>>(
      reinterpret_cast<const bf16*>(h), ld, reinterpret_cast<const long long*>(starts),
      reinterpret_cast<float*>(out), hidden, mode, normalize);
  return cudaGetLastError() == cudaSuccess ? 0 : -5;
}

}  // extern "C"
