// GEMM for few tokens (at most 256): the weights are streamed once, which bounds it. One work item
// per CTA: a tile of bn output features, or the part of its K range that this CTA of a cluster
// takes (the CTAs of a cluster exchange their fp32 sums through shared memory and each finishes
// bn / splits of the columns).
//
// Tokens are the 128 rows of the tensor core's M side, padded by nothing: a stage holds M rounded up to
// eight rows of x, and the products of the rows above them read whatever lies there, which only
// reaches accumulator rows that nobody reads. A stage is then little more than its weights, and the
// ring keeps up to 200 KB of them in flight per SM. Two accumulators for more than 128 tokens. A stage
// holds up to four k-blocks, each operand's fetched by one copy: a stage's wait, copies and commit
// cost 0.25 us whatever its size, which with one block per stage was more than the block itself.
//
// Why a kernel of its own: the general one (gemm_bf16_kernel) stages 128 rows of tokens, and its long
// code runs cold in a kernel of a few microseconds. 50 tokens, 768 x 768: 15.3 -> 4.7 us; 1 token,
// 28672 x 4096 bf16 59.1 -> 41.6 us (5.6 of 6.46 TB/s), 4096 x 4096 14.1 -> 12.0; 128 tokens, 4096 x 14336
// 38.9 -> 30.0; 128 tokens fp8, 4096 x 14336 26.0 -> 18.2; 256 tokens, 28672 x 4096 88.9 -> 58.9. With
// programmatic launches 4.0, 40.3, 10.3, 28.7, 16.6 and 57.5.
#pragma once

namespace ab200 {

constexpr int kFewEpilogueWarps = 8;
constexpr int kFewThreads = (2 + kFewEpilogueWarps) * 32;
constexpr int kFewMaxStages = 32;
constexpr int kFewHeader = 3072;   // barriers and the tile's column factors and biases, in front of the stages

struct FewArgs {
  const float* scale_x;   // e4m3 operands: one factor per token and per feature
  const float* scale_w;
  const __nv_bfloat16* bias;
  const __nv_bfloat16* residual;
  __nv_bfloat16* out;
  int* status;
  long long ldo, ldr;
  int M, N, x_rows, bn, stages, group, groups, groups_per_split, splits, act, w_static;
  int ragged;    // K ends inside a k-block: plain two-dimensional maps, one block per stage
  int w_tiled;   // the weight is stored as [N / 16][K / 128][16][128] bytes
  uint32_t tmem_cols;
};

// Eight finished columns from c on of a token's row; `at`: the first one's place among `cols`, the factors
// and, 256 floats on, the biases of the columns that this CTA finishes.
__device__ __forceinline__ void few_store8(const FewArgs& p, int m, int c, const float* cols, int at, float sx,
                                           float (&v)[8]) {
  const float4* f = reinterpret_cast<const float4*>(cols + at);
  if (p.scale_x != nullptr) {
    const float4 s0 = f[0], s1 = f[1];
    v[0] *= sx * s0.x; v[1] *= sx * s0.y; v[2] *= sx * s0.z; v[3] *= sx * s0.w;
    v[4] *= sx * s1.x; v[5] *= sx * s1.y; v[6] *= sx * s1.z; v[7] *= sx * s1.w;
  }
  if (p.bias != nullptr) {
    const float4 b0 = f[64], b1 = f[65];
    v[0] += b0.x; v[1] += b0.y; v[2] += b0.z; v[3] += b0.w;
    v[4] += b1.x; v[5] += b1.y; v[6] += b1.z; v[7] += b1.w;
  }
  if (p.act == 1) gelu8(v);
  if (p.residual != nullptr) add8(v, *reinterpret_cast<const uint4*>(p.residual + m * p.ldr + c));
  uint4 q;
  q.x = pack_bf16x2(v[0], v[1]);
  q.y = pack_bf16x2(v[2], v[3]);
  q.z = pack_bf16x2(v[4], v[5]);
  q.w = pack_bf16x2(v[6], v[7]);
  *reinterpret_cast<uint4*>(p.out + m * p.ldo + c) = q;
}

// Group g of k-blocks: [block][row][128 bytes] in shared memory.
__device__ __forceinline__ void few_load_w(const FewArgs& p, uint32_t dst, const void* tmap, uint32_t bar, int g,
                                           int tile, int elems) {
  if (p.w_tiled) {
    for (int j = 0; j < p.group; ++j)
      tma_load_4d(dst + (uint32_t)(j * p.bn) * 128u, tmap, bar, 0, 0, g * p.group + j, tile * (p.bn / 16));
  } else if (p.ragged) {
    tma_load_2d(dst, tmap, bar, g * elems, tile * p.bn);
  } else {
    tma_load_3d(dst, tmap, bar, 0, tile * p.bn, g * p.group);
  }
}

template <bool FP8>
__global__ void __launch_bounds__(kFewThreads, 1)
gemm_few_kernel(const __grid_constant__ CUtensorMap tmap_x, const __grid_constant__ CUtensorMap tmap_w,
                const FewArgs p) {
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  const uint32_t raw = smem_u32(smem_raw);
  const uint32_t base = (raw + 1023u) & ~1023u;
  const uint32_t w_bytes = (uint32_t)(p.group * p.bn) * 128u, x_bytes = (uint32_t)(p.group * p.x_rows) * 128u;
  const uint32_t stage_bytes = w_bytes + x_bytes;
  const uint32_t stages0 = base + kFewHeader;
  auto full_bar = [&](int s) { return base + 8u * s; };
  auto empty_bar = [&](int s) { return base + 8u * (kFewMaxStages + s); };
  const uint32_t done_bar = base + 8u * (2 * kFewMaxStages);
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(smem_raw + (base - raw) + 8 * (2 * kFewMaxStages + 1));
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

  float* cols = reinterpret_cast<float*>(smem_raw + (base - raw) + 1024);

  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  const int tile = (int)blockIdx.x / p.splits, split = (int)blockIdx.x % p.splits;
  constexpr int kElems = FP8 ? kBlockKFp8 : kBlockK;
  const int g0 = split * p.groups_per_split;
  const int n = min(p.groups_per_split, p.groups - g0);
  if (warp == 0 && lane == 0) {
    for (int s = 0; s < p.stages; ++s) {
      mbar_init(full_bar(s), 1);
      mbar_init(empty_bar(s), 1);
    }
    mbar_init(done_bar, 1);
    *abort_flag = 0;
    fence_barrier_init();
    // The weights are written by no kernel of the stream: their first tiles are requested before
    // anything else, the tokens' once the kernel before this one has finished.
    const int pre = min(p.stages, n);
    if (p.w_static)
      for (int i = 0; i < pre; ++i) {
        mbar_expect_tx(full_bar(i), w_bytes);
        few_load_w(p, stages0 + (uint32_t)i * stage_bytes, &tmap_w, full_bar(i), g0 + i, tile, kElems);
      }
  }
  if (warp == 1) {
    tmem_alloc(smem_u32(tmem_slot), p.tmem_cols);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  pdl_trigger();   // (tensor memory is owned)
  const uint32_t tmem_base = *tmem_slot;
  bool ok = true;

  if (warp == 0) {
    if (lane == 0) {
      pdl_wait();
      const int pre = p.w_static ? min(p.stages, n) : 0;
      int s = 0;
      uint32_t phase = 1;
      for (int i = 0; i < n; ++i) {
        const uint32_t dst = stages0 + (uint32_t)s * stage_bytes;
        if (!mbar_wait(empty_bar(s), phase, abort_flag, p.status, 100 + s, i)) {
          ok = false;
          break;
        }
        mbar_arrive_expect_tx(full_bar(s), i < pre ? x_bytes : stage_bytes);
        if (i >= pre) few_load_w(p, dst, &tmap_w, full_bar(s), g0 + i, tile, kElems);
        if (p.ragged)
          tma_load_2d(dst + w_bytes, &tmap_x, full_bar(s), (g0 + i) * kElems, 0);
        else
          tma_load_3d(dst + w_bytes, &tmap_x, full_bar(s), 0, 0, (g0 + i) * p.group);
        if (++s == p.stages) {
          s = 0;
          phase ^= 1u;
        }
      }
      if (!ok) {   // copies already issued get a short time to land
        const unsigned long long t0 = globaltimer_ns();
        while (globaltimer_ns() - t0 < 20000000ull) {
        }
      }
    }
    __syncwarp();
  } else if (warp == 1) {
    const uint32_t idesc = FP8 ? make_idesc(128, (uint32_t)p.bn, 0, 0, 0, 0)
                               : make_idesc(128, (uint32_t)p.bn, 1, 1, 0, 0);
    const uint32_t tm = __shfl_sync(0xffffffffu, tmem_base, 0);
    const uint64_t w0 = make_desc_kmajor_sw128(stages0), x0 = make_desc_kmajor_sw128(stages0 + w_bytes);
    const uint64_t stage_step = stage_bytes / 16;
    int s = 0;
    uint32_t phase = 0;
    for (int i = 0; i < n; ++i) {
      if (!__all_sync(0xffffffffu, mbar_wait(full_bar(s), phase, abort_flag, p.status, 300 + s, i))) break;
      tc_fence_after();
      const uint64_t wd = w0 + (uint64_t)s * stage_step, xd = x0 + (uint64_t)s * stage_step;
      if (elect_one()) {
        for (int half = 0; half < (p.M > 128 ? 2 : 1); ++half) {
          const uint32_t d = tm + (uint32_t)(half * p.bn);
#pragma unroll 1
          for (int j = 0; j < p.group; ++j) {
            const uint64_t a = xd + (uint64_t)(half * 1024 + j * p.x_rows * 8);
            const uint64_t b = wd + (uint64_t)(j * p.bn * 8);
#pragma unroll
            for (int k = 0; k < 4; ++k) {
              if (FP8)
                umma_f8_ss(d, a + (uint64_t)(2 * k), b + (uint64_t)(2 * k), idesc, (i + j + k > 0) ? 1u : 0u);
              else
                umma_f16_ss(d, a + (uint64_t)(2 * k), b + (uint64_t)(2 * k), idesc, (i + j + k > 0) ? 1u : 0u);
            }
          }
        }
        tc_commit(empty_bar(s));
        if (i == n - 1) tc_commit(done_bar);
      }
      __syncwarp();
      if (++s == p.stages) {
        s = 0;
        phase ^= 1u;
      }
    }
  } else {
    pdl_wait();
    // Factors and biases of the columns come from memory while the products run: a load per eight columns
    // after them cost an epilogue several trips to memory, one after the other.
    const int t = (int)threadIdx.x - 64, width = p.bn / p.splits;
    const int c = tile * p.bn + split * width + t;
    if (t < width && c < p.N) {
      if (p.scale_x != nullptr) cols[t] = p.scale_w[c];
      if (p.bias != nullptr) cols[256 + t] = __bfloat162float(p.bias[c]);
    }
    asm volatile("bar.sync 1, %0;" ::"n"(kFewEpilogueWarps * 32) : "memory");
    ok = __all_sync(0xffffffffu, mbar_wait(done_bar, 0, abort_flag, p.status, 400, n));
    tc_fence_after();
  }
  const int quad = warp & 3;             // TMEM lane quadrant that this warp may read
  const int part = (warp - 2) >> 2;      // which of the quadrant's two warps this is
  if (p.splits == 1) {
    if (warp >= 2 && ok) {
      for (int m0 = quad * 32; m0 < p.M; m0 += 128) {
        const uint32_t t_addr = tmem_base + ((uint32_t)(quad * 32) << 16) + (m0 >= 128 ? (uint32_t)p.bn : 0u);
        const float sx = p.scale_x != nullptr && m0 + lane < p.M ? p.scale_x[m0 + lane] : 1.f;
#pragma unroll 1
        for (int c0 = part * 16; c0 < p.bn; c0 += 32) {
          uint32_t r[16];
          tmem_ld_x16(t_addr + (uint32_t)c0, r);
          tmem_ld_wait_dep(r);
#pragma unroll
          for (int g = 0; g < 2; ++g) {
            const int c = tile * p.bn + c0 + 8 * g;
            float v[8];
#pragma unroll
            for (int t = 0; t < 8; ++t) v[t] = __uint_as_float(r[8 * g + t]);
            if (m0 + lane < p.M && c < p.N) few_store8(p, m0 + lane, c, cols, c0 + 8 * g, sx, v);
          }
          __syncwarp();
        }
      }
    }
  } else {
    // [source][token][cw] floats where the stages were, rows padded by 16 bytes
    const int cw = p.bn / p.splits, pitch = cw + 4;
    const uint32_t slot = (uint32_t)(p.M * pitch) * 4u;
    const uint32_t my = cluster_ctarank();
    cluster_sync();   // every CTA of the cluster has read its last stage
    if (warp >= 2 && ok) {
      for (int m0 = quad * 32; m0 < p.M; m0 += 128) {
        const uint32_t t_addr = tmem_base + ((uint32_t)(quad * 32) << 16) + (m0 >= 128 ? (uint32_t)p.bn : 0u);
#pragma unroll 1
        for (int c0 = part * 8; c0 < p.bn; c0 += 16) {
          uint32_t r[8];
          tmem_ld_x8(t_addr + (uint32_t)c0, r);
          tmem_ld_wait_dep(r);
          if (m0 + lane < p.M) {
            const uint32_t to = map_to_cta(stages0 + my * slot + (uint32_t)((m0 + lane) * pitch + c0 % cw) * 4u,
                                           (uint32_t)(c0 / cw));
            st_cluster_v4(to, r[0], r[1], r[2], r[3]);
            st_cluster_v4(to + 16u, r[4], r[5], r[6], r[7]);
          }
          __syncwarp();
        }
      }
    }
    cluster_sync();
    if (warp >= 2 && ok) {
      const uint8_t* sums = smem_raw + (stages0 - raw);
      const int vecs = cw / 8;
#pragma unroll 1
      for (int i = (int)threadIdx.x - 64; i < p.M * vecs; i += kFewEpilogueWarps * 32) {
        const int m = i / vecs, c8 = i % vecs * 8;
        const int c = tile * p.bn + (int)my * cw + c8;
        if (c >= p.N) continue;
        float v[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
#pragma unroll 1
        for (int src = 0; src < p.splits; ++src) {
          const float4* a =
              reinterpret_cast<const float4*>(sums + src * slot + (size_t)(m * pitch + c8) * 4);
          const float4 lo = a[0], hi = a[1];
          v[0] += lo.x; v[1] += lo.y; v[2] += lo.z; v[3] += lo.w;
          v[4] += hi.x; v[5] += hi.y; v[6] += hi.z; v[7] += hi.w;
        }
        few_store8(p, m, c, cols, c8, p.scale_x != nullptr ? p.scale_x[m] : 1.f, v);
      }
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem_base, p.tmem_cols);
  }
}

struct FewPlan {
  int bn, splits, group, stages;
  size_t smem;
};

// Stages of `group` blocks that fit, and the shared memory they take: the products of the last stage's last
// block read 128 rows of x (256 for two accumulators) from where its rows begin, and the exchange takes
// the place of the stages.
static int few_stages(int M, int x_rows, int bn, int splits, int group, int most, size_t* smem) {
  const size_t limit = 227 * 1024 - kFewHeader - 1024;
  const size_t stage = (size_t)(bn + x_rows) * group * 128, tail = (size_t)((M > 128 ? 256 : 128) - x_rows) * 128;
  const size_t exchange = splits > 1 ? (size_t)splits * M * (bn / splits + 4) * sizeof(float) : 0;
  if (exchange > limit || stage + tail > limit) return 0;
  size_t n = (limit - tail) / stage;
  if (n > (size_t)most) n = most;
  const size_t ring = n * stage + tail;
  *smem = (ring > exchange ? ring : exchange) + kFewHeader + 1024;
  return (int)n;
}

// Width of the tiles, K splits and k-blocks per stage: few enough to try them all. Times in us, fitted to a
// sweep over all plans of the projections of 768- and 4096-wide models with 1 - 256 tokens: weights come
// from HBM at 6.4 MB/us in all; an SM takes in weights and tokens at 0.2 MB/us; a stage costs its
// wait, copies and commit (0.25), a block its four instructions (44 cycles or half a cycle per
// feature each); a cluster's exchange 1.5 and 0.09 per KB of a CTA's sums. `group_max` is 1 where K
// ends inside a block.
static FewPlan plan_few(int M, int N, int kblocks, int group_max, int sms, int (*capacity)(int, size_t)) {
  FewPlan best = {0, 0, 0, 0, 0};
  double best_t = 1e30;
  const int x_rows = (M + 7) / 8 * 8;
  const int halves = M > 128 ? 2 : 1;
  for (int splits = 1; splits <= 8; splits *= 2)
    for (int group = group_max; group >= 1; group /= 2) {
      const int groups = (kblocks + group - 1) / group;
      const int per = (groups + splits - 1) / splits;
      if ((groups + per - 1) / per != splits) continue;   // every CTA of a cluster has work
      for (int bn = 256; bn >= 16; bn -= 16) {
        if (bn % (8 * splits) || (bn > 16 && bn - 16 >= N)) continue;
        size_t smem = 0;
        const int stages =
            few_stages(M, x_rows, bn, splits, group, per < kFewMaxStages ? per : kFewMaxStages, &smem);
        if (stages == 0 || (stages < 3 && stages < per)) continue;
        const int tiles = (N + bn - 1) / bn;
        const int cap = splits > 1 ? capacity(splits, 226 * 1024) * splits : sms;
        if (cap <= 0) continue;
        const double waves = (double)((tiles * splits + cap - 1) / cap);
        const double sm_us = (bn + x_rows) * group * 128.0 / 0.2e6;
        const double mma_us = 0.25 + group * 4.0 * halves * (bn > 88 ? bn / 2.0 : 44.0) / 1.9e3;
        const double hbm_us = (double)N * kblocks * 128.0 / 6.4e6;
        double t = waves * (per * (sm_us > mma_us ? sm_us : mma_us) + 0.05 * halves * bn / 16 / splits);
        if (t < hbm_us) t = hbm_us + 0.1 * t;
        t += 4.0 * (waves - 1.0);
        if (splits > 1) t += 1.5 + 0.09 * M * bn * 4.0 / 1024.0;
        if (t < best_t - 0.05) {
          best_t = t;
          best = {bn, splits, group, stages, smem};
        }
      }
    }
  return best;
}

}  // namespace ab200
