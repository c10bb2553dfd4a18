// bf16 linear layer  out[M,N] = x[M,K] * w[N,K]^T  (+bias)(+residual)(activation)
// for sm_100a, in three warp-specialised kernels: one warp feeds a ring of 128B-swizzled shared-memory
// stages with TMA, one walks the k-blocks with warp-uniform values while an elected lane issues tcgen05.mma
// (fp32 accumulators in tensor memory), and eight epilogue warps drain the accumulators with tcgen05.ld.
//   * gemm_few_kernel (common/gemm_few.cuh), M <= 256: the weights are streamed once, K is split over the
//     CTAs of a cluster;
//   * gemm_pair_kernel, M > 256: two CTAs on one tile of 256 rows (cta_group::2), persistent, accumulators
//     double-buffered, compiled once per kind of epilogue;
//   * gemm_bf16_kernel, what those two leave: outputs scattered to ranks, ordering between ranks, forced
//     splits, tiled fp8 weights of many rows, narrow or oddly aligned operands. Persistent single CTAs in two
//     orientations: token-major (A = 128 tokens, B = bn features), and for 129 .. 256 tokens feature-major
//     (A = 128 features, B = all tokens; the accumulator holds out^T and the epilogue stores it transposed).
//     Split-K partial sums go through a cluster's shared memory or to an fp32 scratch buffer supplied by the
//     caller, which a second kernel folds.
//
// The same kernels run W8A8 fp8 linears whose scales are one per token and one per output
// feature (ab200_linear_fp8_row): the operands are e4m3 bytes (a 128-byte swizzle atom is then
// 128 k-elements and one kind::f8f6f4 instruction covers 32 of them), the whole K loop
// accumulates in tensor memory with no rescaling on the way, and the epilogue multiplies each
// accumulator by scale_token * scale_feature. An instruction of either kind is accepted at
// the same interval, so the fp8 form does twice the work per unit time.
//
// The reference relies on library GEMMs for these layers (vLLM linear layers
// reached from arctic_inference/vllm/swiftkv/llama_swiftkv.py:165-202; fp8 with per-token and
// per-channel scales: arctic_inference/vllm/spec_dec/fp8.py:34-309).

#include <math.h>
#include <stdlib.h>
#include <mutex>
#include <unordered_map>

#include "api.h"
#include "common/pdl.cuh"
#include "common/peer.cuh"
#include "common/ptx.cuh"
#include "common/tensormap.h"

namespace ab200 {

constexpr int kBlockM = 128;
constexpr int kBlockK = 64;  // bf16 elements: one 128-byte swizzle atom per row
constexpr int kBlockKFp8 = 128;  // e4m3 elements in the same 128 bytes
constexpr int kBlockKBytes = 128;
constexpr int kUmmaK = 16;
// Warps: TMA, MMA, then eight for the epilogue, two per TMEM lane quadrant that take alternate
// 64-column groups.
constexpr int kEpilogueWarps = 8;
constexpr int kGemmThreads = (2 + kEpilogueWarps) * 32;
constexpr int kMaxStages = 8;
constexpr uint32_t kABytes = kBlockM * kBlockK * 2;
// Per-epilogue-warp staging tile for coalesced loads and stores: 32 rows x 64 bf16, the 16-byte
// chunks of a row XORed with the row so that eight lanes hit distinct banks both ways.
constexpr int kStoreStageBytes = 32 * 128;
constexpr int kColumnBytes = 64 * 4;   // a warp's column factors or biases
constexpr int kStoreBytes = kEpilogueWarps * (kStoreStageBytes + kColumnBytes);

struct GemmArgs {
  int rows_a, rows_b, K;
  int bn, stages, splits, kblocks_per_split, kblocks_total;
  int tiles_a, tiles_b;
  int transposed;  // 0: out[a_row*ldo + b_row], 1: out[b_row*ldo + a_row]
  int out_f32;     // 1: write fp32 partial sums (split-K), no bias/residual/activation
  int act;         // 0 none, 1 gelu (erf)
  int b_mn_major;  // 1: the B operand is given as [K, rows_b] (rows_b contiguous)
  int coalesce;    // 1: bf16 row-major output goes through a shared-memory transpose so that a
                   //    warp stores whole 128-byte lines (what NVLink and L2 both want)
  int a_tiled, b_tiled;  // the operand is an fp8 weight stored as [rows/16][K/128][16][128]
  int gate_rows;   // pair kernel: > 0: B is this many gate rows, then as many up rows, the output
                   // silu(gate) * up
  int fp8;         // 1: operands are e4m3 bytes (kind::f8f6f4), 128 k-elements per stage
  int kblock_elems;  // k-elements per stage: 64 (bf16) or 128 (fp8)
  int prefetch_w;    // 1: the weight operand is written by no kernel of the stream (a parameter)
  int b_parts;       // TMA boxes per B stage (1, or more boxes of bn / b_parts rows each)
  // Scatter epilogue: every rank walks the B tiles starting this many tiles in, i.e. at its own
  // share of the columns, so that at any moment the ranks store into different destination
  // ranks. With all ranks starting at tile 0 they all store into rank 0 first, then rank 1,
  // ...: one NVLink ingress carries everything while the others idle.
  int tile_b_rot;
  // > 1: the launch is made of clusters of this many CTAs. The CTAs of a cluster share one
  // output tile and split its K range; they exchange their fp32 partial sums through each
  // other's shared memory and each finishes and stores bn / cluster_splits columns (the
  // split-K of a one-row-of-tiles GEMM with no workspace traffic and no second kernel).
  int cluster_splits;
  const float* scale_a;  // fp8: one factor per A-operand row (null = 1)
  const float* scale_b;  // fp8: one factor per B-operand row
  uint32_t tmem_cols;
  long long ldo, ldr, partial_stride;
  void* out;
  const __nv_bfloat16* bias;
  const __nv_bfloat16* residual;
  int* status;
  // Peer scatter (Ulysses sequence->head exchange fused into the epilogue): when
  // peer_cols > 0, output feature f goes to buffer peer_out[f / peer_cols], column
  // f % peer_cols, row (token + peer_row_off). The buffers are the ranks' symmetric heaps,
  // reached with plain peer stores over NVLink.
  int peer_cols;
  long long peer_row_off;
  __nv_bfloat16* peer_out[16];
  // Cross-rank ordering without a barrier kernel (common/peer.cuh): `wait` holds back the
  // first operand load until every rank's producer of the A operand has signalled (the
  // head->sequence exchange lands in this rank's heap); `sig` tells every rank when the last
  // block of this kernel has finished storing (scatter epilogue, or a partial product that the
  // peers will reduce).
  PeerWait wait;
  TailSignal sig;
};

__device__ __forceinline__ uint32_t stage_chunk(int row, int chunk) {
  return (uint32_t)(row * 128 + ((chunk ^ (row & 7)) << 4));
}

// Adds eight bf16 values to eight floats.
__device__ __forceinline__ void add8(float (&v)[8], const uint4& q) {
  const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&q);
#pragma unroll
  for (int u = 0; u < 4; ++u) {
    const float2 f = __bfloat1622float2(h[u]);
    v[2 * u] += f.x;
    v[2 * u + 1] += f.y;
  }
}

// x * Phi(x), two values at a time for the packed fp32 instructions. From 1.25 on as max(x, 0) - |x| Phi(-|x|), with
// Phi(-a) = exp(-a^2 / 2) p(t), t = 1 / (1 + 0.4 a): the classic form of the error function's tail (Hastings;
// Abramowitz and Stegun 7.1.26), with a polynomial of degree seven fitted here to 3e-8 of the value over
// a = 1.2 .. 13.5. Below, where that form's t and exponential cost three to five times erff's error, as
// x (1/2 + x q(x^2)), q the Taylor-like polynomial of erf(x / sqrt 2) / 2x, fitted to 1e-8 of the result.
// Largest error over the value against 64 bits, in brackets 0.5 x (1 + erff(x / sqrt 2)): 0 .. 1.25 1.2e-7 (1.3e-7),
// above 1.1e-7 (1.2e-7), -1 .. 0 2.0e-7 (2.2e-7), -1.5 .. -1 4.7e-7 (6.3e-7), -3 .. -1.5 6.7e-7 (2.2e-5), -8 .. -3 2.8e-6
// (nothing left). 16384 x 3072 x 768 + bias takes 59 us without GELU, 83 with this and 94 with erff; 74 with
// the tail's form alone, whose error between -1 and 0.5 is 3.9e-7 to 6.7e-7.
__device__ __forceinline__ float2 gelu_x2(float2 x) {
  auto both = [](float c) { return make_float2(c, c); };
  const float2 a = make_float2(fminf(fabsf(x.x), 13.f), fminf(fabsf(x.y), 13.f));
  const float2 u = mul_x2(x, x);
  const float2 d = fma_x2(both(0.4f), a, both(1.f));
  const float2 t = make_float2(rcp_approx(d.x), rcp_approx(d.y));
  float2 p = both(7.106554484e-02f);
  p = fma_x2(p, t, both(-1.941660117e-01f));
  p = fma_x2(p, t, both(1.136968751e-01f));
  p = fma_x2(p, t, both(5.079642110e-02f));
  p = fma_x2(p, t, both(1.405362094e-01f));
  p = fma_x2(p, t, both(1.588197116e-01f));
  p = fma_x2(p, t, both(1.596224587e-01f));
  p = fma_x2(p, t, both(-1.015981127e-06f));
  // (a NaN stays one through the exponential, and -inf times its 0 is one, as -inf times 1 + erf is)
  const float2 e = mul_x2(u, both(-0.7213475204f));
  p = mul_x2(p, make_float2(ex2_approx(e.x), ex2_approx(e.y)));
  const float2 tail = fma_x2(make_float2(fminf(x.x, -a.x), fminf(x.y, -a.y)), p,
                             make_float2(fmaxf(x.x, 0.f), fmaxf(x.y, 0.f)));
  float2 q = both(-6.449855846e-06f);
  q = fma_x2(q, u, both(1.094731415e-04f));
  q = fma_x2(q, u, both(-1.181334374e-03f));
  q = fma_x2(q, u, both(9.970515966e-03f));
  q = fma_x2(q, u, both(-6.648968905e-02f));
  q = fma_x2(q, u, both(3.989422321e-01f));
  const float2 mid = mul_x2(x, fma_x2(x, q, both(0.5f)));
  return make_float2(fabsf(x.x) < 1.25f ? mid.x : tail.x, fabsf(x.y) < 1.25f ? mid.y : tail.y);
}
__device__ __forceinline__ float gelu_erf(float x) { return gelu_x2(make_float2(x, x)).x; }
__device__ __forceinline__ void gelu8(float (&v)[8]) {
#pragma unroll
  for (int t = 0; t < 8; t += 2) {
    const float2 y = gelu_x2(make_float2(v[t], v[t + 1]));
    v[t] = y.x;
    v[t + 1] = y.y;
  }
}

// The epilogue of a tile whose output leaves in whole lines, one of eight warps: 32 rows from
// warp_row0 on, alternate groups of 64 columns of the tile that starts at column b0.
// EPI: what the epilogue does, known when it is compiled (the code of all options together did not stay in
// the instruction cache), or kEpiAny: what the arguments say.
enum Epilogue : int { kEpiAny = -1, kEpiScaled = 1, kEpiBias = 2, kEpiGelu = 4, kEpiResidual = 8, kEpiGated = 16 };

template <int EPI>
struct CoalescedTile {
  static constexpr bool kAny = EPI < 0;
  __device__ __forceinline__ static bool scaled(const GemmArgs& p) {
    return kAny ? p.scale_a != nullptr : (EPI & kEpiScaled) != 0;
  }
  __device__ __forceinline__ static bool biased(const GemmArgs& p) {
    return kAny ? p.bias != nullptr : (EPI & kEpiBias) != 0;
  }
  __device__ __forceinline__ static bool summed(const GemmArgs& p) {
    return kAny ? p.residual != nullptr : (EPI & kEpiResidual) != 0;
  }

  uint4 rq[8];
  // This lane's two of the group's 64 column factors or biases; they reach the other lanes through shared
  // memory. A load per eight columns from global memory, behind stores that might alias it, took
  // longer than the products of a 768-deep tile: 16384 x 2304 x 768 + bias 65.7 -> 55.9 us, 8192 x 4096 x
  // 14336 fp8 366 -> 320.
  float cv[2];

  __device__ __forceinline__ void fetch_columns(const GemmArgs& p, long long b0, int c0, int lane) {
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const long long c = b0 + c0 + lane + 32 * h;
      cv[h] = 0.f;
      if (c < p.rows_b) {
        if (scaled(p)) cv[h] = p.scale_b[c];
        else if (biased(p)) cv[h] = __bfloat162float(p.bias[c]);
      }
    }
  }

  // residual rows of the 64 columns from c0 on, four whole 128-byte lines an instruction
  __device__ __forceinline__ void fetch_residual(const GemmArgs& p, long long warp_row0, long long b0,
                                                 int c0, int lane) {
#pragma unroll
    for (int it = 0; it < 8; ++it) {
      const long long grow = warp_row0 + it * 4 + (lane >> 3);
      const int c = c0 + 8 * (lane & 7);
      if (grow < p.rows_a && b0 + c + 8 <= p.rows_b && c + 8 <= p.bn)
        rq[it] = *reinterpret_cast<const uint4*>(p.residual + grow * p.ldr + b0 + c);
    }
  }

  // before the accumulator is complete
  __device__ __forceinline__ void prefetch(const GemmArgs& p, long long warp_row0, long long b0, int half,
                                           int lane) {
    fetch_columns(p, b0, half * 64, lane);
    if (summed(p) && half * 64 < p.bn) fetch_residual(p, warp_row0, b0, half * 64, lane);
  }

  // t_addr: the warp's lane quadrant of the accumulator; stg: its staging tile; cols: its 64 floats
  __device__ __forceinline__ void store(const GemmArgs& p, uint32_t t_addr, uint8_t* stg, float* cols,
                                        long long warp_row0, long long b0, int half, int lane, float sa) {
    const bool add_rows = summed(p);
    const bool row_ok = warp_row0 + lane < p.rows_a;
    // 64 output columns at a time: each thread converts its row, the warp transposes
    // through its private staging tile, and every store instruction then writes four
    // full 128-byte lines (rows) instead of 32 scattered 16-byte pieces. The residual comes
    // the same way in the other direction.
    for (int c0 = half * 64; c0 < p.bn; c0 += 128) {
      uint32_t r0[32], r1[32];
      __syncwarp();
      tmem_ld_x32(t_addr + (uint32_t)c0, r0);
      tmem_ld_x32(t_addr + (uint32_t)(c0 + 32), r1);
      cols[lane] = cv[0];
      cols[lane + 32] = cv[1];
      if (c0 + 128 < p.bn) fetch_columns(p, b0, c0 + 128, lane);
      if (add_rows) {
#pragma unroll
        for (int it = 0; it < 8; ++it)
          *reinterpret_cast<uint4*>(stg + stage_chunk(it * 4 + (lane >> 3), lane & 7)) = rq[it];
        if (c0 + 128 < p.bn) fetch_residual(p, warp_row0, b0, c0 + 128, lane);
      }
      __syncwarp();
      tmem_ld_wait_dep(r0);
      tmem_ld_wait_dep(r1);
      const long long col = b0 + c0;
      if (row_ok) {
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          float v[8];
#pragma unroll
          for (int t = 0; t < 8; ++t)
            v[t] = __uint_as_float(j < 4 ? r0[8 * j + t] : r1[8 * (j - 4) + t]);
          const long long cj = col + 8 * j;
          uint4* at = reinterpret_cast<uint4*>(stg + stage_chunk(lane, j));
          if (cj + 8 <= p.rows_b && c0 + 8 * j + 8 <= p.bn) {
            const float4 s0 = *reinterpret_cast<const float4*>(cols + 8 * j);
            const float4 s1 = *reinterpret_cast<const float4*>(cols + 8 * j + 4);
            if (scaled(p)) {
              v[0] *= sa * s0.x; v[1] *= sa * s0.y; v[2] *= sa * s0.z; v[3] *= sa * s0.w;
              v[4] *= sa * s1.x; v[5] *= sa * s1.y; v[6] *= sa * s1.z; v[7] *= sa * s1.w;
              if (biased(p)) add8(v, *reinterpret_cast<const uint4*>(p.bias + cj));
            } else if (biased(p)) {
              v[0] += s0.x; v[1] += s0.y; v[2] += s0.z; v[3] += s0.w;
              v[4] += s1.x; v[5] += s1.y; v[6] += s1.z; v[7] += s1.w;
            }
            if (kAny ? p.act == 1 : (EPI & kEpiGelu) != 0) gelu8(v);
            if (add_rows) add8(v, *at);
          }
          uint4 q;
          q.x = pack_bf16x2(v[0], v[1]);
          q.y = pack_bf16x2(v[2], v[3]);
          q.z = pack_bf16x2(v[4], v[5]);
          q.w = pack_bf16x2(v[6], v[7]);
          *at = q;
        }
      }
      __syncwarp();
      __nv_bfloat16* base = reinterpret_cast<__nv_bfloat16*>(p.out) + col;
      long long row_off = 0;
      if (kAny && p.peer_cols > 0) {  // a 64-column group never straddles a destination
        base = p.peer_out[col / p.peer_cols] + col % p.peer_cols;
        row_off = p.peer_row_off;
      }
      const int ch = lane & 7;
#pragma unroll
      for (int it = 0; it < 8; ++it) {
        const int rr = it * 4 + (lane >> 3);
        const long long grow = warp_row0 + rr;
        if (grow < p.rows_a && col + 8 * ch + 8 <= p.rows_b && c0 + 8 * ch + 8 <= p.bn) {
          const uint4 q = *reinterpret_cast<const uint4*>(stg + stage_chunk(rr, ch));
          *reinterpret_cast<uint4*>(base + (grow + row_off) * p.ldo + 8 * ch) = q;
        }
      }
    }
  }
};

// The epilogue of a gate / up tile: gate columns in the accumulator's first half, their up columns in the
// second; bf16 silu(gate) * up, 64 output columns at a time like CoalescedTile.
__device__ __forceinline__ void store_gated(const GemmArgs& p, uint32_t t_addr, uint8_t* stg,
                                            long long warp_row0, int tile_b, int half, int lane) {
  const int width = p.bn / 2;
  for (int c0 = half * 64; c0 < width; c0 += 128) {
    const long long col = (long long)tile_b * width + c0;
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      uint32_t g[32], u[32];
      __syncwarp();
      tmem_ld_x32(t_addr + (uint32_t)(c0 + 32 * h), g);
      tmem_ld_x32(t_addr + (uint32_t)(width + c0 + 32 * h), u);
      tmem_ld_wait_dep(g);
      tmem_ld_wait_dep(u);
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        float v[8];
#pragma unroll
        for (int t = 0; t < 8; ++t) {
          const float z = __uint_as_float(g[8 * j + t]);
          v[t] = __fdividef(z, 1.f + __expf(-z)) * __uint_as_float(u[8 * j + t]);
        }
        *reinterpret_cast<uint4*>(stg + stage_chunk(lane, 4 * h + j)) =
            make_uint4(pack_bf16x2(v[0], v[1]), pack_bf16x2(v[2], v[3]), pack_bf16x2(v[4], v[5]),
                       pack_bf16x2(v[6], v[7]));
      }
    }
    __syncwarp();
    const int ch = lane & 7;
#pragma unroll
    for (int it = 0; it < 8; ++it) {
      const int rr = it * 4 + (lane >> 3);
      if (warp_row0 + rr < p.rows_a && col + 8 * ch + 8 <= p.gate_rows && c0 + 8 * ch + 8 <= width)
        *reinterpret_cast<uint4*>(reinterpret_cast<__nv_bfloat16*>(p.out) + (warp_row0 + rr) * p.ldo + col +
                                  8 * ch) = *reinterpret_cast<const uint4*>(stg + stage_chunk(rr, ch));
    }
  }
}

__device__ __forceinline__ float* column_values(uint8_t* store_stage, int warp) {
  return reinterpret_cast<float*>(store_stage + (size_t)kEpilogueWarps * kStoreStageBytes) + (warp - 2) * 64;
}

// Work item -> (A tile, B tile, K split). Cluster launches hold one item per CTA, the K splits
// of a tile being the consecutive CTAs of one cluster.
__device__ __forceinline__ void decode_work(const GemmArgs& p, int w, int& tile_a, int& tile_b,
                                            int& split) {
  if (p.cluster_splits > 1) {
    tile_a = 0;
    split = w % p.cluster_splits;
    tile_b = w / p.cluster_splits + p.tile_b_rot;
    if (tile_b >= p.tiles_b) tile_b -= p.tiles_b;
    return;
  }
  tile_a = w % p.tiles_a;
  const int rest = w / p.tiles_a;
  tile_b = rest % p.tiles_b;
  split = rest / p.tiles_b;
  if (p.tile_b_rot) {
    tile_b += p.tile_b_rot;
    if (tile_b >= p.tiles_b) tile_b -= p.tiles_b;
  }
}

__global__ void __launch_bounds__(kGemmThreads, 1)
gemm_bf16_kernel(const __grid_constant__ CUtensorMap tmap_a,
                 const __grid_constant__ CUtensorMap tmap_b, const GemmArgs p) {
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  uint8_t* smem = smem_raw;
  if (smem_u32(smem) & 1023u) {  // swizzled tiles need 1024-byte alignment
    pdl_trigger();
    pdl_wait();
    if (threadIdx.x == 0) report_error(p.status, kErrBadArgument, 900, (int)(smem_u32(smem) & 1023u));
    return;
  }
  const uint32_t b_bytes = (uint32_t)p.bn * kBlockK * 2;
  const uint32_t stage_bytes = kABytes + b_bytes;
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + (size_t)p.stages * stage_bytes);
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 2 * kMaxStages + 4);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
  uint8_t* store_stage = reinterpret_cast<uint8_t*>(bars) + 256;
  const uint32_t smem_base = smem_u32(smem);
  const uint32_t bars_base = smem_u32(bars);
  auto full_bar = [&](int s) { return bars_base + 8u * s; };
  auto empty_bar = [&](int s) { return bars_base + 8u * (kMaxStages + s); };
  auto tfull_bar = [&](int a) { return bars_base + 8u * (2 * kMaxStages + a); };
  auto tempty_bar = [&](int a) { return bars_base + 8u * (2 * kMaxStages + 2 + a); };

  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;

  if (threadIdx.x == 0) {
    for (int s = 0; s < p.stages; ++s) {
      mbar_init(full_bar(s), 1);
      mbar_init(empty_bar(s), 1);
    }
    for (int a = 0; a < 2; ++a) {
      mbar_init(tfull_bar(a), 1);
      mbar_init(tempty_bar(a), kEpilogueWarps);
    }
    *abort_flag = 0;
    fence_barrier_init();
    prefetch_tensormap(&tmap_a);
    prefetch_tensormap(&tmap_b);
  }
  if (warp == 1) {
    tmem_alloc(smem_u32(tmem_slot), p.tmem_cols);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  // the next kernel of the stream may be placed as SMs free up; it waits for this one itself
  pdl_trigger();   // (tensor memory is owned)
  const uint32_t tmem_base = *tmem_slot;
  const uint32_t acc_stride = p.tmem_cols / 2;

  const int total_work = p.tiles_a * p.tiles_b * p.splits;
  bool cluster_acc_ok = false;   // epilogue threads of a cluster launch: the accumulator is complete

  if (warp == 0) {
    // ------------------------------ TMA producer ------------------------------
    // The weight operand is written by no kernel, so its first tiles are requested before
    // this kernel waits for the one before it in the stream: the stream of weights starts
    // while that kernel drains. Each of these stages has had its weight bytes announced to
    // its full barrier; the activation tile and the barrier's arrival follow after the wait.
    const bool w_is_b = !p.transposed;
    int pre = 0;
    if (lane == 0 && p.prefetch_w && blockIdx.x < total_work) {
      int tile_a0, tile_b0, split0;
      decode_work(p, blockIdx.x, tile_a0, tile_b0, split0);
      const int kb00 = split0 * p.kblocks_per_split;
      const int kb01 = min(kb00 + p.kblocks_per_split, p.kblocks_total);
      pre = min(p.stages, kb01 - kb00);
      for (int s = 0; s < pre; ++s) {
        const int kb = kb00 + s;
        const uint32_t dst = smem_base + (uint32_t)s * stage_bytes;
        if (w_is_b) {
          mbar_expect_tx(full_bar(s), b_bytes);
          const int pr = p.bn / p.b_parts;
          for (int h = 0; h < p.b_parts; ++h) {
            const uint32_t d2 = dst + kABytes + (uint32_t)(h * pr) * 128u;
            if (p.b_tiled)
              tma_load_4d(d2, &tmap_b, full_bar(s), 0, 0, kb, tile_b0 * (p.bn / 16) + h * (pr / 16));
            else
              tma_load_2d(d2, &tmap_b, full_bar(s), kb * p.kblock_elems, tile_b0 * p.bn + h * pr);
          }
        } else {
          mbar_expect_tx(full_bar(s), kABytes);
          if (p.a_tiled)
            tma_load_4d(dst, &tmap_a, full_bar(s), 0, 0, kb, tile_a0 * (kBlockM / 16));
          else
            tma_load_2d(dst, &tmap_a, full_bar(s), kb * p.kblock_elems, tile_a0 * kBlockM);
        }
      }
    }
    pdl_wait();
    bool peers_ok = true;
    if (p.wait.world > 0) {
      peers_ok = wait_peers(p.wait, p.status, kWaitLimitNs);
      fence_proxy_async_global();
      if (!peers_ok && lane == 0) *abort_flag = 1;
    }
    if (lane == 0) {
      int stage = 0;
      uint32_t phase = 0;
      long long issued = 0;
      bool ok = peers_ok;
      if (!ok) {
        // the prefetched weight tiles still land: let their barriers complete, then leave
        for (int s = 0; s < pre; ++s) {
          mbar_arrive(full_bar(s));
          mbar_drain(full_bar(s), 0);
        }
      }
      for (int w = blockIdx.x; w < total_work && ok; w += gridDim.x) {
        int tile_a, tile_b, split;
        decode_work(p, w, tile_a, tile_b, split);
        const int kb0 = split * p.kblocks_per_split;
        const int kb1 = min(kb0 + p.kblocks_per_split, p.kblocks_total);
        for (int kb = kb0; kb < kb1; ++kb) {
          if (!mbar_wait(empty_bar(stage), phase ^ 1u, abort_flag, p.status, 100 + stage, kb)) {
            ok = false;
            break;
          }
          const bool have_w = issued < pre;   // this stage's weight tile is already on its way
          const bool load_a = !(have_w && !w_is_b);
          const bool load_b = !(have_w && w_is_b);
          mbar_arrive_expect_tx(full_bar(stage),
                                have_w ? (w_is_b ? (uint32_t)kABytes : b_bytes) : stage_bytes);
          const uint32_t a_dst = smem_base + (uint32_t)stage * stage_bytes;
          if (load_a) {
            if (p.a_tiled)
              tma_load_4d(a_dst, &tmap_a, full_bar(stage), 0, 0, kb, tile_a * (kBlockM / 16));
            else
              tma_load_2d(a_dst, &tmap_a, full_bar(stage), kb * p.kblock_elems, tile_a * kBlockM);
          }
          if (!load_b) {
          } else if (!p.b_mn_major) {
            // tiled storage: 2 KB pieces (16 rows x 128 bytes) that are contiguous in memory
            const int pr = p.bn / p.b_parts;
            for (int h = 0; h < p.b_parts; ++h) {
              const uint32_t d2 = a_dst + kABytes + (uint32_t)(h * pr) * 128u;
              if (p.b_tiled)
                tma_load_4d(d2, &tmap_b, full_bar(stage), 0, 0, kb,
                            tile_b * (p.bn / 16) + h * (pr / 16));
              else
                tma_load_2d(d2, &tmap_b, full_bar(stage), kb * p.kblock_elems,
                            tile_b * p.bn + h * pr);
            }
          } else {
            // [64 k-rows][64 n] boxes, one per 64-wide atom along N
            for (int j = 0; j < p.bn / 64; ++j)
              tma_load_2d(a_dst + kABytes + (uint32_t)j * 8192u, &tmap_b, full_bar(stage),
                          tile_b * p.bn + j * 64, kb * kBlockK);
          }
          ++issued;
          if (++stage == p.stages) {
            stage = 0;
            phase ^= 1u;
          }
        }
      }
      if (!ok) {
        // Unwinding: give copies that were already issued a short time to land.
        const int pending = (int)min((long long)p.stages, issued);
        int s = stage;
        uint32_t ph = phase;
        for (int i = 0; i < pending; ++i) {
          if (--s < 0) {
            s = p.stages - 1;
            ph ^= 1u;
          }
          mbar_drain(full_bar(s), ph);
        }
      }
    }
  } else if (warp == 1) {
    // ------------------------------- MMA issuer -------------------------------
    // The whole warp walks the loop with warp-uniform values and one elected lane issues:
    // descriptors then live in uniform registers and an instruction goes out as fast as the
    // tensor core takes it (64 cycles at N = 128, 128 at N = 256; from a branch of one thread every
    // 186 cycles whatever its shape).
    const uint32_t idesc =
        p.fp8 ? make_idesc(kBlockM, (uint32_t)p.bn, 0, 0, 0, 0)
              : make_idesc(kBlockM, (uint32_t)p.bn, 1, 1, 0, p.b_mn_major ? 1u : 0u);
    const uint32_t tm = __shfl_sync(0xffffffffu, tmem_base, 0);
    const uint64_t a0 = make_desc_kmajor_sw128(smem_base);
    const uint64_t b0 = p.b_mn_major ? make_desc_mnmajor_sw128(smem_base + kABytes, 8192u)
                                     : make_desc_kmajor_sw128(smem_base + kABytes);
    const uint64_t stage_step = stage_bytes / 16;
    // K-major: 16 bf16 or 32 e4m3 (32 bytes) further inside the swizzle atom = +2 in the
    // encoded address; MN-major: 16 rows of 128 bytes further = +128.
    const uint64_t b_step = p.b_mn_major ? 128u : 2u;
    int stage = 0;
    uint32_t phase = 0;
    int acc = 0;
    uint32_t acc_phase = 0;
    bool ok = true;
    for (int w = blockIdx.x; w < total_work && ok; w += gridDim.x) {
      int tile_a, tile_b, split;
      decode_work(p, w, tile_a, tile_b, split);
      const int kb0 = split * p.kblocks_per_split;
      const int kb1 = min(kb0 + p.kblocks_per_split, p.kblocks_total);
      if (!__all_sync(0xffffffffu, mbar_wait(tempty_bar(acc), acc_phase ^ 1u, abort_flag, p.status,
                                             200 + acc, w)))
        break;
      tc_fence_after();
      const uint32_t d_tmem = tm + (uint32_t)acc * acc_stride;
      for (int kb = kb0; kb < kb1; ++kb) {
        if (!__all_sync(0xffffffffu, mbar_wait(full_bar(stage), phase, abort_flag, p.status,
                                               300 + stage, kb))) {
          ok = false;
          break;
        }
        tc_fence_after();
        const uint64_t a_desc = a0 + (uint64_t)stage * stage_step;
        const uint64_t b_desc = b0 + (uint64_t)stage * stage_step;
        if (elect_one()) {
          if (p.fp8) {
#pragma unroll
            for (int k = 0; k < kBlockKBytes / 32; ++k)
              umma_f8_ss(d_tmem, a_desc + (uint64_t)(2 * k), b_desc + (uint64_t)(2 * k), idesc,
                         (kb > kb0 || k > 0) ? 1u : 0u);
          } else {
#pragma unroll
            for (int k = 0; k < kBlockK / kUmmaK; ++k)
              umma_f16_ss(d_tmem, a_desc + (uint64_t)(2 * k), b_desc + b_step * (uint64_t)k, idesc,
                          (kb > kb0 || k > 0) ? 1u : 0u);
          }
          tc_commit(empty_bar(stage));
          if (kb == kb1 - 1) tc_commit(tfull_bar(acc));
        }
        __syncwarp();
        if (++stage == p.stages) {
          stage = 0;
          phase ^= 1u;
        }
      }
      acc ^= 1;
      if (acc == 0) acc_phase ^= 1u;
    }
  } else {
    // --------------------------------- epilogue --------------------------------
    pdl_wait();  // scales, bias and residual come from earlier kernels; the output may still be read by one
    const int quad = warp & 3;  // TMEM lane quadrant this warp may read
    const int half = (warp - 2) >> 2;  // which of the quadrant's two warps this is
    const int row = quad * 32 + lane;
    int acc = 0;
    uint32_t acc_phase = 0;
    const bool scaled = p.scale_a != nullptr && !p.out_f32;
    if (p.cluster_splits > 1) {
      // one work item per CTA; what follows the accumulator is the cluster exchange below
      cluster_acc_ok = mbar_wait(tfull_bar(0), 0, abort_flag, p.status, 400, (int)blockIdx.x);
      tc_fence_after();
    } else
    for (int w = blockIdx.x; w < total_work; w += gridDim.x) {
      int tile_a, tile_b, split;
      decode_work(p, w, tile_a, tile_b, split);
      const long long a_row = (long long)tile_a * kBlockM + row;
      const bool row_ok = a_row < p.rows_a;
      const long long b0 = (long long)tile_b * p.bn;
      const float sa = (scaled && row_ok) ? p.scale_a[a_row] : 1.f;
      // The tile's column values and the residual's first columns are requested while the k-loop
      // runs: a lone tile per CTA pays for every load that waits for its accumulator.
      const long long warp_row0 = (long long)tile_a * kBlockM + quad * 32;
      CoalescedTile<kEpiAny> ct;
      if (p.coalesce) ct.prefetch(p, warp_row0, b0, half, lane);
      if (!mbar_wait(tfull_bar(acc), acc_phase, abort_flag, p.status, 400 + acc, w)) break;
      tc_fence_after();
      const uint32_t t_addr =
          tmem_base + (uint32_t)acc * acc_stride + ((uint32_t)(quad * 32) << 16);

      if (p.coalesce) {
        ct.store(p, t_addr, store_stage + (size_t)(warp - 2) * kStoreStageBytes,
                 column_values(store_stage, warp), warp_row0, b0, half, lane, sa);
      } else
      for (int c0 = half * 16; c0 < p.bn; c0 += 32) {
        uint32_t r[16];
        __syncwarp();
        tmem_ld_x16(t_addr + (uint32_t)c0, r);
        tmem_ld_wait();
        float v[16];
#pragma unroll
        for (int t = 0; t < 16; ++t) v[t] = __uint_as_float(r[t]);
        if (!row_ok) continue;
        if (p.out_f32) {
          float* o = reinterpret_cast<float*>(p.out) + (long long)split * p.partial_stride;
          if (!p.transposed) {
            float* dst = o + a_row * p.ldo + b0 + c0;
#pragma unroll
            for (int t = 0; t < 16; t += 4) {
              if (b0 + c0 + t + 4 <= p.rows_b)
                *reinterpret_cast<float4*>(dst + t) = make_float4(v[t], v[t + 1], v[t + 2], v[t + 3]);
            }
          } else {
#pragma unroll
            for (int t = 0; t < 16; ++t) {
              const long long b_row = b0 + c0 + t;
              if (b_row < p.rows_b) o[b_row * p.ldo + a_row] = v[t];
            }
          }
          continue;
        }
        if (scaled) {
#pragma unroll
          for (int t = 0; t < 16; ++t)
            v[t] *= sa * (b0 + c0 + t < p.rows_b ? p.scale_b[b0 + c0 + t] : 0.f);
        }
        if (!p.transposed) {
          const long long col = b0 + c0;
          if (p.bias != nullptr) {
#pragma unroll
            for (int t = 0; t < 16; ++t)
              if (col + t < p.rows_b) v[t] += __bfloat162float(p.bias[col + t]);
          }
          if (p.act == 1) {
#pragma unroll
            for (int t = 0; t < 16; ++t) v[t] = gelu_erf(v[t]);
          }
          if (p.residual != nullptr) {
            const __nv_bfloat16* rs = p.residual + a_row * p.ldr + col;
#pragma unroll
            for (int t = 0; t < 16; t += 8) {
              if (col + t + 8 <= p.rows_b) {
                const uint4 q = *reinterpret_cast<const uint4*>(rs + t);
                const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&q);
#pragma unroll
                for (int u = 0; u < 4; ++u) {
                  const float2 f = __bfloat1622float2(h[u]);
                  v[t + 2 * u] += f.x;
                  v[t + 2 * u + 1] += f.y;
                }
              }
            }
          }
          __nv_bfloat16* dst = reinterpret_cast<__nv_bfloat16*>(p.out) + a_row * p.ldo + col;
          if (p.peer_cols > 0)  // a 16-column chunk never straddles a destination (peer_cols % 16 == 0)
            dst = p.peer_out[col / p.peer_cols] + (a_row + p.peer_row_off) * p.ldo +
                  col % p.peer_cols;
#pragma unroll
          for (int t = 0; t < 16; t += 8) {
            if (col + t + 8 <= p.rows_b) {
              uint4 q;
              q.x = pack_bf16x2(v[t], v[t + 1]);
              q.y = pack_bf16x2(v[t + 2], v[t + 3]);
              q.z = pack_bf16x2(v[t + 4], v[t + 5]);
              q.w = pack_bf16x2(v[t + 6], v[t + 7]);
              *reinterpret_cast<uint4*>(dst + t) = q;
            }
          }
        } else {
          // accumulator holds out^T: this thread owns output feature a_row
          const float bias = (p.bias != nullptr) ? __bfloat162float(p.bias[a_row]) : 0.f;
          __nv_bfloat16* o = reinterpret_cast<__nv_bfloat16*>(p.out);
          long long o_col = a_row, o_row_off = 0;
          if (p.peer_cols > 0) {
            o = p.peer_out[a_row / p.peer_cols];
            o_col = a_row % p.peer_cols;
            o_row_off = p.peer_row_off;
          }
#pragma unroll
          for (int t = 0; t < 16; ++t) {
            const long long b_row = b0 + c0 + t;
            if (b_row < p.rows_b) {
              float x = v[t] + bias;
              if (p.act == 1) x = gelu_erf(x);
              if (p.residual != nullptr) x += __bfloat162float(p.residual[b_row * p.ldr + a_row]);
              o[(b_row + o_row_off) * p.ldo + o_col] = __float2bfloat16(x);
            }
          }
        }
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(tempty_bar(acc));
      acc ^= 1;
      if (acc == 0) acc_phase ^= 1u;

    }
  }

  if (p.cluster_splits > 1) {
    // ---- split-K inside a cluster: partial sums cross through shared memory ----
    // CTA r of the cluster owns columns [r * cw, (r + 1) * cw) of the tile. Every CTA writes,
    // for each owner, its fp32 partial sums of the owner's columns into the owner's shared
    // memory (the pipeline stages, idle by now), slot [source CTA][row][cw + 4 pad]; the
    // owner adds the slots in source order, so the result does not depend on timing.
    const int ns = p.cluster_splits;
    const int cw = p.bn / ns;
    const int pitch = cw + 4;   // words; 16 B of padding keeps 16-byte row accesses of a warp
                                // on distinct banks
    const uint32_t my = cluster_ctarank();
    const int quad = warp & 3;
    const int half = (warp - 2) >> 2;
    const int row = quad * 32 + lane;
    // first barrier: every CTA of the cluster has consumed its last pipeline stage (its
    // epilogue warps arrive only after their accumulator is complete)
    cluster_sync();
    if (warp >= 2 && cluster_acc_ok) {
      const uint32_t t_addr = tmem_base + ((uint32_t)(quad * 32) << 16);
      for (int c0 = half * 16; c0 < p.bn; c0 += 32) {
        uint32_t r[16];
        __syncwarp();
        tmem_ld_x16(t_addr + (uint32_t)c0, r);
        tmem_ld_wait();
        const uint32_t owner = (uint32_t)(c0 / cw);
        const uint32_t local =
            smem_base + (uint32_t)(((int)my * kBlockM + row) * pitch + (c0 % cw)) * 4u;
        const uint32_t remote = map_to_cta(local, owner);
#pragma unroll
        for (int t = 0; t < 16; t += 4)
          st_cluster_v4(remote + 4u * t, r[t], r[t + 1], r[t + 2], r[t + 3]);
      }
    }
    // second barrier: all partial sums have landed (release / acquire at cluster scope)
    cluster_sync();
    if (warp >= 2 && cluster_acc_ok && !*abort_flag) {
      int tile_a, tile_b, split;
      decode_work(p, (int)blockIdx.x, tile_a, tile_b, split);
      const long long a_row = row;
      const bool row_ok = a_row < p.rows_a;
      const long long col0 = (long long)tile_b * p.bn + (long long)my * cw;
      const float sa = (p.scale_a != nullptr && row_ok) ? p.scale_a[a_row] : 1.f;
      const float* slots = reinterpret_cast<const float*>(smem);
      for (int j = half * 8; j < cw; j += 16) {
        float v[8];
#pragma unroll
        for (int t = 0; t < 8; ++t) v[t] = 0.f;
        for (int src = 0; src < ns; ++src) {
          const float* q = slots + ((size_t)src * kBlockM + row) * pitch + j;
          const float4 x0 = *reinterpret_cast<const float4*>(q);
          const float4 x1 = *reinterpret_cast<const float4*>(q + 4);
          v[0] += x0.x; v[1] += x0.y; v[2] += x0.z; v[3] += x0.w;
          v[4] += x1.x; v[5] += x1.y; v[6] += x1.z; v[7] += x1.w;
        }
        const long long col = col0 + j;
        if (!row_ok || col + 8 > p.rows_b) continue;
        if (p.scale_a != nullptr) {
          const float4 s0 = *reinterpret_cast<const float4*>(p.scale_b + col);
          const float4 s1 = *reinterpret_cast<const float4*>(p.scale_b + col + 4);
          v[0] *= sa * s0.x; v[1] *= sa * s0.y; v[2] *= sa * s0.z; v[3] *= sa * s0.w;
          v[4] *= sa * s1.x; v[5] *= sa * s1.y; v[6] *= sa * s1.z; v[7] *= sa * s1.w;
        }
        if (p.bias != nullptr) {
          const uint4 q = *reinterpret_cast<const uint4*>(p.bias + col);
          const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&q);
#pragma unroll
          for (int u = 0; u < 4; ++u) {
            const float2 f = __bfloat1622float2(h[u]);
            v[2 * u] += f.x;
            v[2 * u + 1] += f.y;
          }
        }
        if (p.act == 1) {
#pragma unroll
          for (int t = 0; t < 8; ++t) v[t] = gelu_erf(v[t]);
        }
        if (p.residual != nullptr) {
          const uint4 q = *reinterpret_cast<const uint4*>(p.residual + a_row * p.ldr + col);
          const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&q);
#pragma unroll
          for (int u = 0; u < 4; ++u) {
            const float2 f = __bfloat1622float2(h[u]);
            v[2 * u] += f.x;
            v[2 * u + 1] += f.y;
          }
        }
        __nv_bfloat16* dst = reinterpret_cast<__nv_bfloat16*>(p.out) + a_row * p.ldo + col;
        if (p.peer_cols > 0)  // eight columns never straddle a destination (peer_cols % 8 == 0)
          dst = p.peer_out[col / p.peer_cols] + (a_row + p.peer_row_off) * p.ldo +
                col % p.peer_cols;
        uint4 q;
        q.x = pack_bf16x2(v[0], v[1]);
        q.y = pack_bf16x2(v[2], v[3]);
        q.z = pack_bf16x2(v[4], v[5]);
        q.w = pack_bf16x2(v[6], v[7]);
        *reinterpret_cast<uint4*>(dst) = q;
      }
    }
  }

  tail_signal(p.sig, gridDim.x);
  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem_base, p.tmem_cols);
  }
}

// Two CTAs of a cluster on one tile of 256 rows by bn columns (cta_group::2), for products with more
// rows than a few tiles: each CTA stages 128 rows of A and bn / 2 rows of B per k-block, the even
// one issues the products for both, and each drains the 128 rows that its own TMEM holds.
//
// Why: one CTA with a 128 x 256 tile stages 48 KB per k-block of 512 tensor-core cycles and reads as
// much again from shared memory for its operands, more than the 128 bytes a cycle that an SM's
// shared memory moves. A pair needs 32 KB per CTA for the same work. 8192 x 28672 x 4096 bf16 went from
// 1757 to 1219 us (1095 to 1578 TFLOP/s), fp8 from 866 to 678 us (2221 to 2837), 2048 x 28672 x 4096 from
// 401 to 315 us, 16384 x 768 x 3072 + residual from 86 to 64 us. Tiles are walked in groups of eight rows of tiles, so
// that the operands that the resident pairs share stay in L2.
constexpr int kPairGroup = 8;

__device__ __forceinline__ void decode_pair(const GemmArgs& p, int w, int& tile_a, int& tile_b) {
  const int per_group = kPairGroup * p.tiles_b;
  const int first = w / per_group * kPairGroup;
  const int rows = min(kPairGroup, p.tiles_a - first);
  const int r = w % per_group;
  tile_a = first + r % rows;
  tile_b = r / rows;
}

template <int EPI>
__global__ void __launch_bounds__(kGemmThreads, 1)
gemm_pair_kernel(const __grid_constant__ CUtensorMap tmap_a,
                 const __grid_constant__ CUtensorMap tmap_b, const GemmArgs p) {
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  uint8_t* smem = smem_raw;
  if (smem_u32(smem) & 1023u) {  // swizzled tiles need 1024-byte alignment
    pdl_trigger();
    pdl_wait();
    if (threadIdx.x == 0) report_error(p.status, kErrBadArgument, 900, (int)(smem_u32(smem) & 1023u));
    return;
  }
  const uint32_t half_b = (uint32_t)p.bn / 2;
  const uint32_t stage_bytes = kABytes + half_b * kBlockKBytes;
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + (size_t)p.stages * stage_bytes);
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 2 * kMaxStages + 4);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
  uint8_t* store_stage = reinterpret_cast<uint8_t*>(bars) + 256;
  const uint32_t smem_base = smem_u32(smem);
  const uint32_t bars_base = smem_u32(bars);
  auto full_bar = [&](int s) { return bars_base + 8u * s; };
  auto empty_bar = [&](int s) { return bars_base + 8u * (kMaxStages + s); };
  auto tfull_bar = [&](int a) { return bars_base + 8u * (2 * kMaxStages + a); };
  auto tempty_bar = [&](int a) { return bars_base + 8u * (2 * kMaxStages + 2 + a); };

  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  const int rank = (int)cluster_ctarank();

  if (threadIdx.x == 0) {
    for (int s = 0; s < p.stages; ++s) {
      mbar_init(full_bar(s), 1);
      mbar_init(empty_bar(s), 1);
    }
    for (int a = 0; a < 2; ++a) {
      mbar_init(tfull_bar(a), 1);
      mbar_init(tempty_bar(a), 2 * kEpilogueWarps);   // (the even CTA's: both CTAs drain)
    }
    *abort_flag = 0;
    fence_barrier_init();
    prefetch_tensormap(&tmap_a);
    prefetch_tensormap(&tmap_b);
  }
  if (warp == 1) {
    tmem_alloc_pair(smem_u32(tmem_slot), 512);
    tmem_relinquish_pair();
  }
  tc_fence_before();
  __syncthreads();
  cluster_sync();   // the other CTA's barriers are ready for this one's copies and arrivals
  tc_fence_after();
  pdl_trigger();   // (tensor memory is owned)
  const uint32_t tmem_base = *tmem_slot;

  const int total_work = p.tiles_a * p.tiles_b;
  const int first_work = (int)blockIdx.x / 2, work_step = (int)gridDim.x / 2;

  if (warp == 0) {
    pdl_wait();
    if (lane == 0) {
      int stage = 0;
      uint32_t phase = 0;
      bool ok = true;
      for (int w = first_work; w < total_work && ok; w += work_step) {
        int tile_a, tile_b;
        decode_pair(p, w, tile_a, tile_b);
        const int row_a = (2 * tile_a + rank) * kBlockM;
        // (gate / up: the even CTA stages gate rows, the odd one the same columns' up rows)
        const int row_b = EPI == kEpiGated ? tile_b * (int)half_b + rank * p.gate_rows
                                          : tile_b * p.bn + rank * (int)half_b;
        for (int kb = 0; kb < p.kblocks_total; ++kb) {
          if (!mbar_wait(empty_bar(stage), phase ^ 1u, abort_flag, p.status, 100 + stage, kb)) {
            ok = false;
            break;
          }
          // one barrier, the even CTA's, collects the four boxes of both CTAs
          if (rank == 0) mbar_arrive_expect_tx(full_bar(stage), 2 * stage_bytes);
          const uint32_t full = map_to_cta(full_bar(stage), 0);
          const uint32_t dst = smem_base + (uint32_t)stage * stage_bytes;
          tma_load_2d_pair(dst, &tmap_a, full, kb * p.kblock_elems, row_a);
          tma_load_2d_pair(dst + kABytes, &tmap_b, full, kb * p.kblock_elems, row_b);
          if (++stage == p.stages) {
            stage = 0;
            phase ^= 1u;
          }
        }
      }
      if (!ok) {
        // Unwinding: copies already issued, by either CTA, get a short time to land.
        const unsigned long long t0 = globaltimer_ns();
        while (globaltimer_ns() - t0 < 20000000ull) {
        }
      }
    }
  } else if (warp == 1) {
    if (rank == 0) {
      const uint32_t idesc = p.fp8 ? make_idesc(2 * kBlockM, (uint32_t)p.bn, 0, 0, 0, 0)
                                   : make_idesc(2 * kBlockM, (uint32_t)p.bn, 1, 1, 0, 0);
      const uint32_t tm = __shfl_sync(0xffffffffu, tmem_base, 0);
      const uint64_t a0 = make_desc_kmajor_sw128(smem_base);
      const uint64_t b0 = make_desc_kmajor_sw128(smem_base + kABytes);
      const uint64_t stage_step = stage_bytes / 16;
      int stage = 0;
      uint32_t phase = 0;
      int acc = 0;
      uint32_t acc_phase = 0;
      bool ok = true;
      for (int w = first_work; w < total_work && ok; w += work_step) {
        if (!__all_sync(0xffffffffu, mbar_wait(tempty_bar(acc), acc_phase ^ 1u, abort_flag, p.status,
                                               200 + acc, w)))
          break;
        tc_fence_after();
        const uint32_t d_tmem = tm + (uint32_t)acc * 256u;
        for (int kb = 0; kb < p.kblocks_total; ++kb) {
          if (!__all_sync(0xffffffffu, mbar_wait(full_bar(stage), phase, abort_flag, p.status,
                                                 300 + stage, kb))) {
            ok = false;
            break;
          }
          tc_fence_after();
          const uint64_t a_desc = a0 + (uint64_t)stage * stage_step;
          const uint64_t b_desc = b0 + (uint64_t)stage * stage_step;
          if (elect_one()) {
            if (p.fp8) {
#pragma unroll
              for (int k = 0; k < kBlockKBytes / 32; ++k)
                umma_f8_ss_pair(d_tmem, a_desc + (uint64_t)(2 * k), b_desc + (uint64_t)(2 * k), idesc,
                                (kb > 0 || k > 0) ? 1u : 0u);
            } else {
#pragma unroll
              for (int k = 0; k < kBlockK / kUmmaK; ++k)
                umma_f16_ss_pair(d_tmem, a_desc + (uint64_t)(2 * k), b_desc + (uint64_t)(2 * k), idesc,
                                 (kb > 0 || k > 0) ? 1u : 0u);
            }
            tc_commit_pair(empty_bar(stage));
            if (kb == p.kblocks_total - 1) tc_commit_pair(tfull_bar(acc));
          }
          __syncwarp();
          if (++stage == p.stages) {
            stage = 0;
            phase ^= 1u;
          }
        }
        acc ^= 1;
        if (acc == 0) acc_phase ^= 1u;
      }
    }
  } else {
    pdl_wait();
    const int quad = warp & 3;
    const int half = (warp - 2) >> 2;
    int acc = 0;
    uint32_t acc_phase = 0;
    for (int w = first_work; w < total_work; w += work_step) {
      int tile_a, tile_b;
      decode_pair(p, w, tile_a, tile_b);
      const long long warp_row0 = (long long)(2 * tile_a + rank) * kBlockM + quad * 32;
      const long long col0 = (long long)tile_b * p.bn;
      const float sa =
          (p.scale_a != nullptr && warp_row0 + lane < p.rows_a) ? p.scale_a[warp_row0 + lane] : 1.f;
      CoalescedTile<EPI> ct;
      if (EPI != kEpiGated) ct.prefetch(p, warp_row0, col0, half, lane);
      if (!__all_sync(0xffffffffu, mbar_wait(tfull_bar(acc), acc_phase, abort_flag, p.status, 400 + acc, w)))
        break;
      tc_fence_after();
      const uint32_t t_addr = tmem_base + ((uint32_t)(quad * 32) << 16) + (uint32_t)acc * 256u;
      uint8_t* stg = store_stage + (size_t)(warp - 2) * kStoreStageBytes;
      if (EPI == kEpiGated)
        store_gated(p, t_addr, stg, warp_row0, tile_b, half, lane);
      else
        ct.store(p, t_addr, stg, column_values(store_stage, warp), warp_row0, col0, half, lane, sa);
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive_cluster(map_to_cta(tempty_bar(acc), 0));
      acc ^= 1;
      if (acc == 0) acc_phase ^= 1u;
    }
  }

  tc_fence_before();
  __syncthreads();
  cluster_sync();   // neither CTA leaves while the other may still signal it
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc_pair(tmem_base, 512);
  }
}

}  // namespace ab200

#include "common/gemm_few.cuh"

namespace ab200 {

// out[m,n] = sum_s partial[s][m,n] (+bias[n]) -> activation -> (+residual[m,n])
__global__ void splitk_reduce_kernel(const float* __restrict__ partial, int splits,
                                     long long partial_stride, int M, int N,
                                     __nv_bfloat16* __restrict__ out, long long ldo,
                                     const __nv_bfloat16* __restrict__ bias,
                                     const __nv_bfloat16* __restrict__ residual, long long ldr,
                                     int act, const float* __restrict__ scale_m,
                                     const float* __restrict__ scale_n, const TailSignal sig) {
  pdl_wait();
  pdl_trigger();
  const long long n4 = N / 4;
  const long long total = (long long)M * n4;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < total;
       i += (long long)gridDim.x * blockDim.x) {
    const long long m = i / n4;
    const long long n = (i % n4) * 4;
    float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
    for (int s = 0; s < splits; ++s) {
      const float4 v =
          *reinterpret_cast<const float4*>(partial + s * partial_stride + m * (long long)N + n);
      acc.x += v.x;
      acc.y += v.y;
      acc.z += v.z;
      acc.w += v.w;
    }
    float v[4] = {acc.x, acc.y, acc.z, acc.w};
    if (scale_m != nullptr) {
      const float sm = scale_m[m];
#pragma unroll
      for (int t = 0; t < 4; ++t) v[t] *= sm * scale_n[n + t];
    }
#pragma unroll
    for (int t = 0; t < 4; ++t) {
      if (bias != nullptr) v[t] += __bfloat162float(bias[n + t]);
      if (act == 1) v[t] = gelu_erf(v[t]);
      if (residual != nullptr) v[t] += __bfloat162float(residual[m * ldr + n + t]);
    }
    uint2 q;
    q.x = pack_bf16x2(v[0], v[1]);
    q.y = pack_bf16x2(v[2], v[3]);
    *reinterpret_cast<uint2*>(out + m * ldo + n) = q;
  }
  tail_signal(sig, gridDim.x);
}

// ------------------------------- host side ---------------------------------
struct TmapKey {
  const void* ptr;
  uint64_t rows, cols, ld;
  uint32_t box_rows;  // bit 31 set: e4m3 bytes instead of bf16
  uint64_t tile_stride_n = 0;  // tiled fp8 weights: bytes between 16-row tiles (0: row-major)
  uint32_t group = 0;  // k-blocks per box of a map [K / block][rows][block] (0: two dimensions)
  bool operator==(const TmapKey& o) const {
    return ptr == o.ptr && rows == o.rows && cols == o.cols && ld == o.ld &&
           box_rows == o.box_rows && tile_stride_n == o.tile_stride_n && group == o.group;
  }
};
struct TmapKeyHash {
  size_t operator()(const TmapKey& k) const {
    size_t h = reinterpret_cast<size_t>(k.ptr);
    h ^= k.rows * 0x9E3779B97F4A7C15ull + (h << 6) + (h >> 2);
    h ^= k.cols * 0xC2B2AE3D27D4EB4Full + (h << 6) + (h >> 2);
    h ^= k.ld * 0x165667B19E3779F9ull + (h << 6) + (h >> 2);
    h ^= k.box_rows * 0x27D4EB2F165667C5ull + (h << 6) + (h >> 2);
    h ^= k.tile_stride_n * 0x9FB21C651E98DF25ull + (h << 6) + (h >> 2);
    h ^= k.group * 0xD6E8FEB86659FD93ull + (h << 6) + (h >> 2);
    return h;
  }
};

static int get_tmap(CUtensorMap* out, const void* ptr, uint64_t rows, uint64_t cols, uint64_t ld,
                    uint32_t box_rows, bool fp8, uint64_t tile_stride_n = 0, uint32_t group = 0);
static int get_tmap_bf16(CUtensorMap* out, const void* ptr, uint64_t rows, uint64_t cols,
                         uint64_t ld, uint32_t box_rows) {
  return get_tmap(out, ptr, rows, cols, ld, box_rows, false);
}
// tile_stride_n > 0: the matrix is an fp8 weight stored as [rows/16][K/128][16][128] bytes;
// `ld` is then the byte distance between consecutive k-tiles of one 16-row tile and
// tile_stride_n the distance between 16-row tiles (views of a larger tiled matrix keep their
// parent's strides). A box of box_rows rows is box_rows/16 contiguous 2 KB pieces.
static int get_tmap(CUtensorMap* out, const void* ptr, uint64_t rows, uint64_t cols, uint64_t ld,
                    uint32_t box_rows, bool fp8, uint64_t tile_stride_n, uint32_t group) {
  static std::mutex mu;
  static std::unordered_map<TmapKey, CUtensorMap, TmapKeyHash> cache;
  TmapKey key{ptr, rows, cols, ld, box_rows | (fp8 ? 0x80000000u : 0u), tile_stride_n, group};
  std::lock_guard<std::mutex> lock(mu);
  auto it = cache.find(key);
  if (it != cache.end()) {
    *out = it->second;
    return 0;
  }
  CUtensorMap m;
  int rc;
  if (group > 0) {
    const uint64_t elems = fp8 ? kBlockKFp8 : kBlockK, bytes = fp8 ? 1 : 2;
    const uint64_t dims[3] = {elems, rows, cols / elems};
    const uint64_t strides[2] = {ld * bytes, 128};
    const uint32_t box[3] = {(uint32_t)elems, box_rows, group};
    rc = make_tmap_nd(&m, ptr, fp8 ? CU_TENSOR_MAP_DATA_TYPE_UINT8 : CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, dims,
                      strides, box);
  } else if (tile_stride_n > 0) {
    const uint64_t dims[4] = {128, 16, cols / 128, (rows + 15) / 16};
    const uint64_t strides[3] = {128, ld, tile_stride_n};
    const uint32_t box[4] = {128, 16, 1, box_rows / 16};
    rc = make_tmap_nd(&m, ptr, CU_TENSOR_MAP_DATA_TYPE_UINT8, 4, dims, strides, box);
  } else
  rc = fp8 ? make_tmap_2d(&m, ptr, CU_TENSOR_MAP_DATA_TYPE_UINT8, rows, cols, ld, box_rows,
                              kBlockKFp8)
               : make_tmap_2d(&m, ptr, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, rows, cols, ld * 2,
                              box_rows, kBlockK);
  if (rc != 0) return rc;
  if (cache.size() > 8192) cache.clear();
  cache.emplace(key, m);
  *out = m;
  return 0;
}

static int g_num_sms = 0;
static int num_sms() {
  if (g_num_sms == 0) {
    int dev = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&g_num_sms, cudaDevAttrMultiProcessorCount, dev);
    if (g_num_sms <= 0) g_num_sms = 148;
  }
  return g_num_sms;
}

static int pick_stages(int bn) {
  const int stage_bytes = (int)kABytes + bn * kBlockK * 2;
  int s = (227 * 1024 - 256 - kStoreBytes) / stage_bytes;
  if (s > kMaxStages) s = kMaxStages;
  return s;
}

static bool cluster_splits_off() {
  static const bool off = [] {
    const char* e = getenv("AB200_GEMM_CLUSTER");
    return e != nullptr && e[0] == '0';
  }();
  return off;
}

// How many clusters of `cs` CTAs (one CTA per SM: the kernel takes an SM's shared memory) the
// device can hold at once; 0 when such a cluster cannot be placed.
static int cluster_capacity(int cs, size_t smem) {
  static int cache[64][4];   // [device][log2 cs]: 0 unknown, -1 none, else capacity
  int dev = 0;
  cudaGetDevice(&dev);
  int lg = cs == 2 ? 1 : cs == 4 ? 2 : cs == 8 ? 3 : -1;
  if (dev < 0 || dev >= 64 || lg < 0) return 0;
  if (cache[dev][lg] == 0) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)cs * 16);
    cfg.blockDim = dim3(kGemmThreads);
    cfg.dynamicSmemBytes = smem;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = (unsigned)cs;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    int n = 0;
    if (cudaOccupancyMaxActiveClusters(&n, gemm_bf16_kernel, &cfg) != cudaSuccess) {
      cudaGetLastError();
      n = 0;
    }
    cache[dev][lg] = n > 0 ? n : -1;
  }
  return cache[dev][lg] > 0 ? cache[dev][lg] : 0;
}

// Rough time (us) of a one-row-of-tiles GEMM plan: every wave pays its k-loop (four MMA
// instructions per k-block at the measured issue interval, ~0.45 us per k-block with its
// stage turnaround) plus a fixed ramp; split-K through the workspace pays the fp32 partials'
// round trip and a second kernel, split-K inside a cluster a shared-memory exchange.
static double plan_cost_us(int tiles, int splits, int kblocks, int capacity, bool cluster, int M,
                           int N) {
  const int ctas = tiles * splits;
  const int waves = (ctas + capacity - 1) / capacity;
  const int per = (kblocks + splits - 1) / splits;
  double t = waves * (per * 0.45 + 2.0);
  if (splits > 1)
    t += cluster ? 1.0 : 3.0 + 2.0 * splits * (double)M * N * 4.0 / 3.0e6;
  return t;
}

// Cycles that a CTA of a pair spends on one k-block of a 256 x bn tile: the tensor core's (2 per column), or
// what its shared memory takes to receive and to read the operands (128 bytes a cycle).
static double pair_kblock_cycles(int bn) {
  const double mma = 2.0 * bn, smem = 2.0 * (kABytes + 64.0 * bn) / 128.0;
  return mma > smem ? mma : smem;
}

// Width of the tiles that a product on `pairs` pairs of CTAs is cut into: the one with the least time in whole waves.
static int pick_pair_width(int tiles_a, int N, int kblocks, int pairs) {
  int best = 0;
  double cycles = 0;
  for (int bn = 256; bn >= 128; bn -= 64) {
    if (bn > 128 && bn > ((N + 63) / 64) * 64) continue;
    const long long tiles = (long long)tiles_a * ((N + bn - 1) / bn);
    const double t = (double)((tiles + pairs - 1) / pairs) * (kblocks * pair_kblock_cycles(bn) + 1000.0);
    if (best == 0 || t < cycles) {
      best = bn;
      cycles = t;
    }
  }
  return best;
}

// The plan of a size, made once (a hundred candidates cost the host 2 us, as much as the launch).
// Token counts are planned in classes, so that a step and the same step padded to a captured one's size
// sum in the same order.
static FewPlan few_plan_of(int tokens, int N, int kblocks, int group_max, int sms) {
  int M = 8;
  while (M < tokens) M += M < 128 ? M : 64;
  static std::mutex mu;
  static std::unordered_map<uint64_t, FewPlan> plans;
  const uint64_t key = ((uint64_t)M << 54) ^ ((uint64_t)group_max << 50) ^ ((uint64_t)N << 20) ^ (uint64_t)kblocks;
  std::lock_guard<std::mutex> lock(mu);
  auto it = plans.find(key);
  if (it != plans.end()) return it->second;
  const FewPlan plan = plan_few(M, N, kblocks, group_max, sms, cluster_capacity);
  if (plans.size() > 8192) plans.clear();
  plans.emplace(key, plan);
  return plan;
}

// The pair kernel's forms with an epilogue of their own, and the one for any other.
struct PairForm {
  int epi;
  void (*kernel)(CUtensorMap, CUtensorMap, GemmArgs);
};
static const PairForm pair_forms[] = {
    {0, gemm_pair_kernel<0>},
    {kEpiScaled, gemm_pair_kernel<kEpiScaled>},
    {kEpiBias, gemm_pair_kernel<kEpiBias>},
    {kEpiBias | kEpiGelu, gemm_pair_kernel<kEpiBias | kEpiGelu>},
    {kEpiBias | kEpiResidual, gemm_pair_kernel<kEpiBias | kEpiResidual>},
    {kEpiGated, gemm_pair_kernel<kEpiGated>},
    {kEpiAny, gemm_pair_kernel<kEpiAny>},
};
constexpr int kPairForms = sizeof(pair_forms) / sizeof(pair_forms[0]);

static uint32_t pow2_at_least(uint32_t v) {
  uint32_t p = 32;
  while (p < v) p <<= 1;
  return p;
}

}  // namespace ab200

using namespace ab200;

extern "C" {

// Number of fp32 scratch bytes ab200_linear_bf16 may need for (M, N, K).
size_t ab200_linear_bf16_workspace_bytes(int M, int N, int K) {
  if (M > 256) return 0;
  return (size_t)(M <= 128 ? 16 : 8) * (size_t)M * (size_t)N * sizeof(float);
}

// For the calls with few tokens that the general kernel still serves (scattered outputs, ordering between
// ranks): the weights go on the N side, 256 features per instruction, the tokens on the (padded) M side, and
// split-K spreads the instructions over all SMs. The interval is that of instructions issued from a branch of one
// thread; the warp-uniform loop takes 64 to 128 cycles, so these plans err towards more splits.
constexpr double kMmaIssueCycles = 186.0;

// Split-K factor for a one-row-of-tiles (M <= 128) token-major GEMM: the smallest estimate of
// max(instruction-issue time, HBM time incl. fp32 partials) plus a reduce-launch penalty.
static int pick_token_major_splits(int tiles_b, int kblocks, int M, int N, int K, int sms,
                                   size_t workspace_bytes, int elem_bytes) {
  int best = 1;
  double best_t = 1e30;
  for (int s = 1; s <= 16; s *= 2) {
    if (s > 1 && (kblocks / s < 4 || (size_t)s * M * N * sizeof(float) > workspace_bytes)) break;
    const int per_split = (kblocks + s - 1) / s;
    const int waves = (tiles_b * s + sms - 1) / sms;
    const double issue_us = waves * per_split * (kBlockK / kUmmaK) * kMmaIssueCycles / 1.9e3;
    const double bytes = (double)elem_bytes * N * K + (s > 1 ? 2.0 * s * M * (double)N * 4.0 : 0.0);
    const double hbm_us = bytes / 6.5e6;
    const double t = (issue_us > hbm_us ? issue_us : hbm_us) + (s > 1 ? 4.0 : 0.0);
    if (t < best_t - 0.25) {
      best_t = t;
      best = s;
    }
  }
  return best;
}

static int launch_linear(const void* x, long long ldx, const void* w, long long ldw, void* out,
                         long long ldo, int M, int N, int K, const void* bias,
                         const void* residual, long long ldr, int act, void* workspace,
                         size_t workspace_bytes, int force_splits, int* status,
                         cudaStream_t stream, const void* const* peer_ptrs, int world,
                         int peer_cols, long long peer_row_off, const float* scale_x = nullptr,
                         const float* scale_w = nullptr, const Ab200PeerSync* sync = nullptr,
                         long long w_tile_stride_n = 0, long long w_tile_stride_k = 0,
                         int w_static = 0, int gate_rows = 0) {
  if (M <= 0 || N <= 0 || K <= 0) return 0;
  const bool fp8 = scale_x != nullptr;  // e4m3 operands with per-token / per-feature scales
  const int opa = fp8 ? 16 : 8;         // operand rows must start on 16-byte boundaries
  if ((K % opa) || (N % 8) || (ldx % opa) || (ldw % opa) || (ldo % 8) ||
      (reinterpret_cast<uintptr_t>(x) & 15) || (reinterpret_cast<uintptr_t>(w) & 15) ||
      (reinterpret_cast<uintptr_t>(out) & 15))
    return -2;
  if (fp8 && (scale_w == nullptr || (reinterpret_cast<uintptr_t>(scale_w) & 15))) return -2;
  const bool w_tiled = w_tile_stride_n > 0;
  if (w_tiled && (!fp8 || (K % 128) || (N % 16) || (w_tile_stride_n % 16) ||
                  (w_tile_stride_k % 16) || w_tile_stride_k < 2048))
    return -2;
  if (residual != nullptr && ((ldr % 8) || (reinterpret_cast<uintptr_t>(residual) & 15))) return -2;

  static bool attr_set[64] = {false};
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev < 0 || dev >= 64) return -3;
  if (!attr_set[dev]) {
    cudaError_t e = cudaFuncSetAttribute(gemm_bf16_kernel,
                                         cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024);
    for (int i = 0; i < kPairForms && e == cudaSuccess; ++i)
      e = cudaFuncSetAttribute(pair_forms[i].kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024);
    if (e == cudaSuccess)
      e = cudaFuncSetAttribute(gemm_few_kernel<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024);
    if (e == cudaSuccess)
      e = cudaFuncSetAttribute(gemm_few_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024);
    if (e != cudaSuccess) return -3;
    attr_set[dev] = true;
  }

  const bool alone = sync == nullptr || (sync->wait_world == 0 && sync->sig_world == 0);
  // (that kernel splits K in clusters alone; without them the general one does, through the workspace)
  if (M <= 256 && peer_cols == 0 && alone && force_splits == 0 && !cluster_splits_off() &&
      (reinterpret_cast<uintptr_t>(bias) & 15) == 0) {
    const int elems = fp8 ? kBlockKFp8 : kBlockK;
    const int kblocks = (K + elems - 1) / elems;
    const FewPlan plan = few_plan_of(M, N, kblocks, K % elems == 0 ? 4 : 1, num_sms());
    if (plan.bn > 0) {
      FewArgs f;
      f.scale_x = scale_x;
      f.scale_w = scale_w;
      f.bias = reinterpret_cast<const __nv_bfloat16*>(bias);
      f.residual = reinterpret_cast<const __nv_bfloat16*>(residual);
      f.out = reinterpret_cast<__nv_bfloat16*>(out);
      f.status = status;
      f.ldo = ldo;
      f.ldr = ldr;
      f.M = M;
      f.N = N;
      f.x_rows = (M + 7) / 8 * 8;
      f.bn = plan.bn;
      f.stages = plan.stages;
      f.group = plan.group;
      f.groups = (kblocks + plan.group - 1) / plan.group;
      f.groups_per_split = (f.groups + plan.splits - 1) / plan.splits;
      f.splits = plan.splits;
      f.act = act;
      f.w_tiled = w_tiled ? 1 : 0;
      // (without programmatic launches no kernel runs beside this one)
      f.w_static = (w_static || !pdl_enabled()) ? 1 : 0;
      f.tmem_cols = pow2_at_least((uint32_t)plan.bn * (M > 128 ? 2u : 1u));
      f.ragged = K % elems != 0 ? 1 : 0;
      const uint32_t group = f.ragged ? 0 : (uint32_t)plan.group;
      CUtensorMap tx, tw;
      if (get_tmap(&tx, x, (uint64_t)M, (uint64_t)K, (uint64_t)ldx, (uint32_t)f.x_rows, fp8, 0, group) != 0 ||
          get_tmap(&tw, w, (uint64_t)N, (uint64_t)K, (uint64_t)(w_tiled ? w_tile_stride_k : ldw),
                   (uint32_t)plan.bn, fp8, w_tiled ? (uint64_t)w_tile_stride_n : 0, w_tiled ? 0 : group) != 0)
        return -4;
      const unsigned ctas = (unsigned)((N + plan.bn - 1) / plan.bn * plan.splits);
      return launch_pdl_cluster(fp8 ? gemm_few_kernel<true> : gemm_few_kernel<false>, dim3(ctas),
                                dim3(kFewThreads), plan.smem, stream, (unsigned)plan.splits, tx, tw,
                                f) == cudaSuccess
                 ? 0
                 : -5;
    }
  }

  GemmArgs a;
  memset(&a, 0, sizeof(a));
  if (peer_cols > 0) {
    if (world < 1 || world > 16 || (peer_cols % 16) || N != world * peer_cols) return -2;
    a.peer_cols = peer_cols;
    a.peer_row_off = peer_row_off;
    for (int i = 0; i < world; ++i)
      a.peer_out[i] = reinterpret_cast<__nv_bfloat16*>(const_cast<void*>(peer_ptrs[i]));
    force_splits = 1;  // partial sums would need the scatter in the reduce kernel as well
  }
  a.K = K;
  a.fp8 = fp8 ? 1 : 0;
  a.kblock_elems = fp8 ? kBlockKFp8 : kBlockK;
  a.kblocks_total = (K + a.kblock_elems - 1) / a.kblock_elems;
  a.status = status;
  a.act = act;
  a.bias = reinterpret_cast<const __nv_bfloat16*>(bias);
  a.residual = reinterpret_cast<const __nv_bfloat16*>(residual);
  a.ldr = ldr;
  a.ldo = ldo;
  a.out = out;
  a.splits = 1;

  const void* pa;
  const void* pb;
  long long lda, ldb;
  const int sms = num_sms();
  if (M > kBlockM && M <= 256) {
    // feature-major: weights are the 128-row operand, all tokens form the N side
    a.transposed = 1;
    a.rows_a = N;
    a.rows_b = M;
    a.bn = ((M + 15) / 16) * 16;
    pa = w;
    lda = ldw;
    pb = x;
    ldb = ldx;
    a.tiles_a = (N + kBlockM - 1) / kBlockM;
    a.tiles_b = 1;
    a.scale_a = scale_w;
    a.scale_b = scale_x;
    int splits = force_splits;
    if (splits <= 0) {
      splits = 1;
      while (a.tiles_a * splits * 2 <= sms + sms / 4 && splits < 8 &&
             a.kblocks_total / (splits * 2) >= 8)
        splits *= 2;
    }
    if (splits > 8) splits = 8;
    if (splits > a.kblocks_total) splits = a.kblocks_total;
    if (splits > 1 &&
        (workspace == nullptr || workspace_bytes < (size_t)splits * M * N * sizeof(float)))
      splits = 1;
    a.splits = splits;
  } else {
    a.transposed = 0;
    a.rows_a = M;
    a.rows_b = N;
    pa = x;
    lda = ldx;
    pb = w;
    ldb = ldw;
    a.tiles_a = (M + kBlockM - 1) / kBlockM;
    a.scale_a = scale_x;
    a.scale_b = scale_w;
    const int tiles256 = a.tiles_a * ((N + 255) / 256);
    a.bn = ((tiles256 >= sms || a.tiles_a == 1) && N >= 256) ? 256 : 128;
    if (N < 128) a.bn = ((N + 15) / 16) * 16;
    if (a.tiles_a == 1 && peer_cols == 0 && a.bn == 256) {
      // One row of tiles that streams the whole weight matrix (decode): when 256-wide tiles
      // leave a good part of the SMs without one (gate/up of an 8B model: 112 tiles on 148
      // SMs), narrow them to the widest size that still fits one wave. A narrower tile is also
      // a smaller pipeline stage, i.e. one more stage of loads in flight per SM.
      const int t256 = (N + 255) / 256;
      if (t256 * 4 > sms * 2 && t256 * 8 < sms * 7) {
        int bn = 256;
        while (bn > 128 && (N + (bn - 16) - 1) / (bn - 16) <= sms) bn -= 16;
        a.bn = bn;
      }
    }
    if (a.tiles_a == 1 && peer_cols > 0 && N >= 256) {
      // One row of tiles and no split-K (the scatter epilogue writes final values): a CTA
      // streams its weight tile at a fraction of an SM's share of HBM bandwidth, so narrow the
      // tiles until most SMs hold one.
      while (a.bn > 64 && (N + a.bn - 1) / a.bn < (sms * 3) / 5) a.bn /= 2;
    }
    a.tiles_b = (N + a.bn - 1) / a.bn;
    if (a.tiles_a == 1) {
      int splits = force_splits;
      if (splits <= 0)
        splits = (N % 4 == 0 && workspace != nullptr)
                     ? pick_token_major_splits(a.tiles_b, a.kblocks_total, M, N, K, sms,
                                               workspace_bytes, fp8 ? 1 : 2)
                     : 1;
      if (splits > 16) splits = 16;
      if (splits > a.kblocks_total) splits = a.kblocks_total;
      if (splits > 1 && (workspace == nullptr || (N % 4) ||
                         workspace_bytes < (size_t)splits * M * N * sizeof(float)))
        splits = 1;
      a.splits = splits;
    }
  }
  // One row of tiles (at most 128 tokens): consider splitting K inside thread-block clusters
  // instead of through the workspace. The scatter epilogue qualifies too: the CTA that
  // finishes a column range stores it to the rank that owns it.
  if (!a.transposed && a.tiles_a == 1 && !cluster_splits_off() && (force_splits == 0 || peer_cols > 0) &&
      N % 8 == 0 && ldo % 8 == 0 && (peer_cols == 0 || peer_cols % 8 == 0) &&
      (reinterpret_cast<uintptr_t>(bias) % 16) == 0 && (residual == nullptr || ldr % 8 == 0)) {
    double best = plan_cost_us(a.tiles_b, a.splits, a.kblocks_total, sms, false, M, N);
    int best_bn = 0, best_s = 0, best_ctas = 0;
    const size_t smem_full = 227 * 1024 - 1024;
    for (int bn = 256; bn >= 64; bn -= 64) {
      if (bn > ((N + 63) / 64) * 64) continue;
      const int tiles = (N + bn - 1) / bn;
      for (int cs = 2; cs <= 8; cs *= 2) {
        // (each CTA keeps at least 8 k-blocks: with fewer, the cluster's placement and its two
        // barriers cost more than the shorter loop saves; measured on the 4096 x 4096 o_proj)
        if (bn % (16 * cs) != 0 || a.kblocks_total < 8 * cs) continue;
        const int per = (a.kblocks_total + cs - 1) / cs;
        if ((a.kblocks_total + per - 1) / per != cs) continue;   // every CTA of a cluster has work
        const int cap = cluster_capacity(cs, smem_full) * cs;
        if (cap <= 0 || tiles * cs > 4 * cap) continue;
        const double c = plan_cost_us(tiles, cs, a.kblocks_total, cap, true, M, N);
        if (c < best - 0.25 || (c < best + 0.25 && best_s > 0 && tiles * cs > best_ctas)) {
          best = c < best ? c : best;
          best_bn = bn;
          best_s = cs;
          best_ctas = tiles * cs;
        }
      }
    }
    if (best_s > 0) {
      a.bn = best_bn;
      a.tiles_b = (N + a.bn - 1) / a.bn;
      a.splits = best_s;
      a.cluster_splits = best_s;
    }
  }
  a.kblocks_per_split = (a.kblocks_total + a.splits - 1) / a.splits;
  a.splits = (a.kblocks_total + a.kblocks_per_split - 1) / a.kblocks_per_split;
  a.stages = pick_stages(a.bn);
  a.tmem_cols = pow2_at_least(2u * (uint32_t)(a.bn < 64 ? 64 : a.bn));  // (groups of 64 are read)
  if (a.cluster_splits > 1 &&
      (size_t)a.stages * (kABytes + (size_t)a.bn * kBlockK * 2) <
          (size_t)kBlockM * (a.bn + 4 * a.cluster_splits) * sizeof(float)) {
    return -2;   // cannot happen for the tile sizes above: the exchange slots fit the pipeline
  }

  a.coalesce = !a.transposed && a.splits == 1 && a.bn % 8 == 0 &&
               N % 8 == 0 && ldo % 8 == 0 &&
               (peer_cols == 0 || (peer_cols % 64 == 0 && a.bn % 64 == 0)) &&
               (reinterpret_cast<uintptr_t>(bias) % 16) == 0 &&
               (residual == nullptr || ldr % 8 == 0);

  // More than one row of tiles: CTA pairs. Also where tiles of single CTAs would come in one wave and those of pairs
  // in two: 6272 x 768 x 3072 28.7 us on pairs, 33.3 on single CTAs with tiles of 256 columns, 53 of 128; 1100 x 4096
  // x 4096 35.6, 40.2 and 67; 1152 x 4096 x 14336 119, 121 and 210.
  if (!a.transposed && a.tiles_a > 1 && M > 256 && N >= 128 && peer_cols == 0 && alone && !w_tiled &&
      a.coalesce) {
    const int tiles_pair = (M + 2 * kBlockM - 1) / (2 * kBlockM);
    const int bn = pick_pair_width(tiles_pair, N, a.kblocks_total, sms / 2);
    if (cluster_capacity(2, 227 * 1024 - 1024) > 0) {
      a.gate_rows = gate_rows;
      a.bn = bn;
      a.tiles_a = tiles_pair;
      a.tiles_b = gate_rows > 0 ? (gate_rows + bn / 2 - 1) / (bn / 2) : (N + bn - 1) / bn;
      const int stage_bytes = (int)kABytes + bn / 2 * kBlockKBytes;
      a.stages = (227 * 1024 - 256 - kStoreBytes) / stage_bytes;
      if (a.stages > kMaxStages) a.stages = kMaxStages;
      CUtensorMap ta, tb;
      if (get_tmap(&ta, pa, (uint64_t)M, (uint64_t)K, (uint64_t)lda, kBlockM, fp8) != 0 ||
          get_tmap(&tb, pb, (uint64_t)N, (uint64_t)K, (uint64_t)ldb, (uint32_t)(bn / 2), fp8) != 0)
        return -4;
      const long long tiles = (long long)a.tiles_a * a.tiles_b;
      const unsigned pairs = (unsigned)(tiles < sms / 2 ? tiles : sms / 2);
      const size_t smem = (size_t)a.stages * stage_bytes + 256 + kStoreBytes;
      const int epi = gate_rows > 0 ? kEpiGated
                                    : (fp8 ? kEpiScaled : 0) | (bias != nullptr ? kEpiBias : 0) |
                                          (act == 1 ? kEpiGelu : 0) | (residual != nullptr ? kEpiResidual : 0);
      auto kernel = gemm_pair_kernel<kEpiAny>;
      for (int i = 0; i < kPairForms; ++i)
        if (pair_forms[i].epi == epi) kernel = pair_forms[i].kernel;
      return launch_pdl_cluster(kernel, dim3(2 * pairs), dim3(kGemmThreads), smem, stream, 2u,
                                ta, tb, a) == cudaSuccess
                 ? 0
                 : -5;
    }
  }

  if (gate_rows > 0) return -6;   // only the pairs above have that epilogue
  TailSignal sig;
  memset(&sig, 0, sizeof(sig));
  if (sync != nullptr) {
    if (sync->wait_world < 0 || sync->wait_world > kMaxPeers || sync->sig_world < 0 ||
        sync->sig_world > kMaxPeers)
      return -2;
    a.wait.flags = reinterpret_cast<const unsigned int*>(sync->wait_flags);
    a.wait.epoch_ctr = reinterpret_cast<const unsigned int*>(sync->wait_epoch_ctr);
    a.wait.world = sync->wait_world;
    if (sync->sig_world > 0) {
      for (int i = 0; i < sync->sig_world; ++i)
        sig.flags[i] = reinterpret_cast<unsigned int*>(const_cast<void*>(sync->sig_flag_ptrs[i]));
      sig.done_ctr = reinterpret_cast<unsigned int*>(sync->sig_done_ctr);
      sig.epoch_ctr = reinterpret_cast<unsigned int*>(sync->sig_epoch_ctr);
      sig.my_rank = sync->sig_rank;
      sig.world = sync->sig_world;
    }
  }
  if (peer_cols > 0 && sig.world > 1)
    a.tile_b_rot = (int)(((long long)sig.my_rank * a.tiles_b) / sig.world);
  void* final_out = out;
  const bool ws_split = a.splits > 1 && a.cluster_splits <= 1;
  if (!ws_split) a.sig = sig;   // with split-K through the workspace the reduce kernel writes the output
  if (ws_split) {
    a.out_f32 = 1;
    a.out = workspace;
    a.ldo = N;  // partials are stored as [split][M][N] regardless of orientation
    a.partial_stride = (long long)M * N;
  }

  CUtensorMap ta, tb;
  a.a_tiled = (w_tiled && a.transposed) ? 1 : 0;
  a.b_tiled = (w_tiled && !a.transposed) ? 1 : 0;
  a.prefetch_w = w_static ? 1 : 0;
  // One row of tiles over a row-major weight: two half-height boxes per stage instead of one
  // (the same bytes in flight as twice as many TMA operations: 35.6 -> 33.8 us on the 128-token
  // gate/up projection; thirteen 16-row boxes, in contrast, took 54 us).
  a.b_parts = (a.tiles_a == 1 && !a.transposed && !a.b_tiled && a.bn % 16 == 0) ? 2 : 1;
  if (get_tmap(&ta, pa, (uint64_t)a.rows_a, (uint64_t)K,
               a.a_tiled ? (uint64_t)w_tile_stride_k : (uint64_t)lda, kBlockM, fp8,
               a.a_tiled ? (uint64_t)w_tile_stride_n : 0) != 0)
    return -4;
  if (get_tmap(&tb, pb, (uint64_t)a.rows_b, (uint64_t)K,
               a.b_tiled ? (uint64_t)w_tile_stride_k : (uint64_t)ldb,
               (uint32_t)(a.bn / a.b_parts), fp8,
               a.b_tiled ? (uint64_t)w_tile_stride_n : 0) != 0)
    return -4;

  const int total = a.tiles_a * a.tiles_b * a.splits;
  const int grid = (a.cluster_splits > 1 || total < sms) ? total : sms;
  const size_t smem =
      (size_t)a.stages * (kABytes + (size_t)a.bn * kBlockK * 2) + 256 + kStoreBytes;
  if (launch_pdl_cluster(gemm_bf16_kernel, dim3(grid), dim3(kGemmThreads), smem, stream,
                         a.cluster_splits > 1 ? (unsigned)a.cluster_splits : 1u, ta, tb,
                         a) != cudaSuccess)
    return -5;

  if (ws_split) {
    const long long total4 = (long long)M * (N / 4);
    int blocks = (int)((total4 + 255) / 256);
    if (blocks > sms * 8) blocks = sms * 8;
    if (launch_pdl(splitk_reduce_kernel, dim3(blocks), dim3(256), 0, stream,
                   reinterpret_cast<const float*>(workspace), a.splits, a.partial_stride, M, N,
                   reinterpret_cast<__nv_bfloat16*>(final_out), ldo,
                   reinterpret_cast<const __nv_bfloat16*>(bias),
                   reinterpret_cast<const __nv_bfloat16*>(residual), ldr, act, scale_x, scale_w,
                   sig) != cudaSuccess)
      return -5;
  }
  return 0;
}


// force_splits: 0 = heuristic, >0 = use exactly this split-K factor (feature-major only).
int ab200_linear_bf16(const void* x, long long ldx, const void* w, long long ldw, void* out,
                      long long ldo, int M, int N, int K, const void* bias, const void* residual,
                      long long ldr, int act, void* workspace, size_t workspace_bytes,
                      int force_splits, int* status, cudaStream_t stream) {
  return launch_linear(x, ldx, w, ldw, out, ldo, M, N, K, bias, residual, ldr, act, workspace,
                       workspace_bytes, force_splits, status, stream, nullptr, 0, 0, 0);
}

// out[m, n] = silu(x[m] . w[n]) * (x[m] . w[inter + n]) for w [2 inter, K] (gate rows, then up rows), without
// a pass over the gate / up rows in between (8192 x 28672 x 4096: 1325 us in two kernels, 1174 in one; 512 tokens 110 -> 98).
// More than 256 tokens; -6 for what the callers leave to the two separate kernels.
int ab200_linear_silu(const void* x, long long ldx, const void* w, long long ldw, void* out, long long ldo, int M,
                      int inter, int K, int* status, cudaStream_t stream) {
  if (M <= 256 || (inter % 8) || inter < 128) return -6;
  return launch_linear(x, ldx, w, ldw, out, ldo, M, 2 * inter, K, nullptr, nullptr, 0, 0, nullptr, 0, 0, status,
                       stream, nullptr, 0, 0, 0, nullptr, nullptr, nullptr, 0, 0, 0, inter);
}

// Linear layer whose output columns are scattered to `world` peer buffers: feature f of
// token m lands in peer_ptrs[f / peer_cols] at row (m + peer_row_off), column f % peer_cols
// (row stride ldo). N must equal world * peer_cols. The caller synchronises the ranks
// (ab200_barrier) before the destination buffers are read.
int ab200_linear_bf16_scatter(const void* x, long long ldx, const void* w, long long ldw,
                              const void* const* peer_ptrs, int world, int peer_cols,
                              long long peer_row_off, long long ldo, int M, int N, int K,
                              int* status, cudaStream_t stream) {
  if (peer_cols <= 0 || world <= 0) return -2;
  return launch_linear(x, ldx, w, ldw, const_cast<void*>(peer_ptrs[0]), ldo, M, N, K, nullptr,
                       nullptr, 0, 0, nullptr, 0, 1, status, stream, peer_ptrs, world, peer_cols,
                       peer_row_off);
}

// W8A8 fp8 linear with one scale per token and one per output feature:
//   out[m,n] = sx[m] * sw[n] * sum_k xq[m,k] * wq[n,k]   (+bias)(activation)(+residual)
// xq [M,K] and wq [N,K] are e4m3 bytes (row strides in elements, multiples of 16), sx fp32 [M],
// sw fp32 [N] (16-byte aligned). With peer_ptrs the output columns are scattered to the ranks'
// buffers as in ab200_linear_bf16_scatter (pass world = 0 for a plain output).
int ab200_linear_fp8_row(const void* xq, long long ldx, const void* sx, const void* wq,
                         long long ldw, const void* sw, void* out, long long ldo, int M, int N,
                         int K, const void* bias, const void* residual, long long ldr, int act,
                         void* workspace, size_t workspace_bytes, int force_splits,
                         const void* const* peer_ptrs, int world, int peer_cols,
                         long long peer_row_off, int* status, cudaStream_t stream) {
  if (sx == nullptr || sw == nullptr) return -2;
  if (world > 0 && peer_cols > 0) {
    return launch_linear(xq, ldx, wq, ldw, const_cast<void*>(peer_ptrs[0]), ldo, M, N, K, nullptr,
                         nullptr, 0, 0, nullptr, 0, 1, status, stream, peer_ptrs, world, peer_cols,
                         peer_row_off, reinterpret_cast<const float*>(sx),
                         reinterpret_cast<const float*>(sw));
  }
  return launch_linear(xq, ldx, wq, ldw, out, ldo, M, N, K, bias, residual, ldr, act, workspace,
                       workspace_bytes, force_splits, status, stream, nullptr, 0, 0, 0,
                       reinterpret_cast<const float*>(sx), reinterpret_cast<const float*>(sw));
}

// One entry point for every form of the linear layer, described by a struct: bf16 operands
// (sx == null) or e4m3 operands with per-token / per-feature scales, plain or peer-scattered
// output, and optional cross-rank ordering (wait for the producers of x, signal completion).
int ab200_linear_desc(const Ab200LinearDesc* d, cudaStream_t stream) {
  if (d == nullptr) return -2;
  const bool scatter = d->world > 0 && d->peer_cols > 0;
  if (scatter && d->peer_ptrs == nullptr) return -2;
  if ((d->sx == nullptr) != (d->sw == nullptr)) return -2;
  return launch_linear(d->x, d->ldx, d->w, d->ldw,
                       scatter ? const_cast<void*>(d->peer_ptrs[0]) : d->out, d->ldo, d->M, d->N,
                       d->K, scatter ? nullptr : d->bias, scatter ? nullptr : d->residual,
                       scatter ? 0 : d->ldr, scatter ? 0 : d->act, scatter ? nullptr : d->workspace,
                       scatter ? 0 : d->workspace_bytes, scatter ? 1 : d->force_splits, d->status,
                       stream, scatter ? d->peer_ptrs : nullptr, scatter ? d->world : 0,
                       scatter ? d->peer_cols : 0, scatter ? d->peer_row_off : 0,
                       reinterpret_cast<const float*>(d->sx), reinterpret_cast<const float*>(d->sw),
                       &d->sync, d->w_tile_stride_n, d->w_tile_stride_k, d->w_static);
}

// out[M,N] = x[M,K] * wt[K,N] with wt row-major (N contiguous): exercises the
// MN-major shared-memory descriptor for the B operand. N must be a multiple of 64.
int ab200_gemm_bf16_nn(const void* x, long long ldx, const void* wt, long long ldw, void* out,
                       long long ldo, int M, int N, int K, int* status, cudaStream_t stream) {
  if (M <= 0 || N <= 0 || K <= 0) return 0;
  if ((K % 8) || (N % 64) || (ldx % 8) || (ldw % 8) || (ldo % 8)) return -2;
  if (cudaFuncSetAttribute(gemm_bf16_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                           227 * 1024) != cudaSuccess)
    return -3;
  GemmArgs a;
  memset(&a, 0, sizeof(a));
  a.K = K;
  a.kblock_elems = kBlockK;
  a.kblocks_total = (K + kBlockK - 1) / kBlockK;
  a.kblocks_per_split = a.kblocks_total;
  a.splits = 1;
  a.status = status;
  a.ldo = ldo;
  a.out = out;
  a.rows_a = M;
  a.rows_b = N;
  a.b_mn_major = 1;
  a.b_parts = 1;
  a.bn = (N % 128 == 0) ? 128 : 64;
  a.tiles_a = (M + kBlockM - 1) / kBlockM;
  a.tiles_b = N / a.bn;
  a.stages = pick_stages(a.bn);
  a.tmem_cols = pow2_at_least(2u * (uint32_t)(a.bn < 64 ? 64 : a.bn));  // (groups of 64 are read)
  CUtensorMap ta, tb;
  if (get_tmap_bf16(&ta, x, (uint64_t)M, (uint64_t)K, (uint64_t)ldx, kBlockM) != 0) return -4;
  if (make_tmap_2d(&tb, wt, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, (uint64_t)K, (uint64_t)N,
                   (uint64_t)ldw * 2, 64, 64) != 0)
    return -4;
  const int total = a.tiles_a * a.tiles_b;
  const int sms = num_sms();
  const int grid = total < sms ? total : sms;
  const size_t smem =
      (size_t)a.stages * (kABytes + (size_t)a.bn * kBlockK * 2) + 256 + kStoreBytes;
  gemm_bf16_kernel<<<grid, kGemmThreads, smem, stream>>>(ta, tb, a);
  return cudaGetLastError() == cudaSuccess ? 0 : -5;
}

}  // extern "C"
