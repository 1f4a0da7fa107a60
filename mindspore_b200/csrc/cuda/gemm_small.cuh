// 16-bit GEMM for problems with too few output tiles to fill the machine: 128 x 64 tiles, the k-loop of a tile split
// over the CTAs of a thread-block cluster, partial sums exchanged through distributed shared memory.
//
//   C[b][m][n] (+)= alpha * sum_k A[b][m][k] * B[b][n][k] (+ bias[n])     (operand storage flags as in gemm_sm100.cu)
//
// Such a problem - a projection of a few tokens, a small layer - is bound by reading its weights: 24 x 4096 x 4096 is
// 34 MB of B, 5 us at HBM's rate, but 32 tiles of 128 x 128 put it on 32 of 148 SMs, each of which streams a megabyte
// through one pipeline (32 us).  Here CTA r of a cluster of `split` multiplies k-blocks [r, r + 1) * num_kb / split of
// its tile, leaves the fp32 accumulator in its shared memory, and after a cluster barrier every CTA adds up its share of
// the tile's rows over the cluster, always in rank order (deterministic), and stores them row by row.  Two CTAs fit an SM.
// Measured: 24 x 4096 x 4096 bf16 32 -> 13 us; the 27 products of a two-layer decoder of width 512 (512 tokens) 249 ->
// 228 us.
//
// Roles per CTA: warp 0 TMA, warp 1 MMA issue, warps 2-5 epilogue.  Every wait is bounded; a CTA that gave up still takes
// part in both cluster barriers.
#pragma once
#include "host_common.h"
#include "ptx.cuh"

namespace msb {

constexpr int kGsBM = 128, kGsBN = 64, kGsBK = 64, kGsThreads = 192, kGsStages = 4;
constexpr int kGsABytes = kGsBM * kGsBK * 2;
constexpr int kGsBBytes = kGsBN * kGsBK * 2;
constexpr int kGsStageBytes = kGsABytes + kGsBBytes;
constexpr int kGsPitch = kGsBN + 4;              // floats per row of the exchanged accumulator: conflict-free 16-byte rows
constexpr int kGsBarOffset = kGsStages * kGsStageBytes;
constexpr int kGsSmemBytes = kGsBarOffset + 256 + 1024;
constexpr int kGsMaxSplit = 8;
static_assert(kGsBM * kGsPitch * 4 <= kGsBarOffset, "the accumulator takes the place of the stage ring");

struct GemmSmallParams {
  void* C;
  const void* bias;
  int* status;
  long long c_batch_stride, ldc;
  int M, N, K, tiles_m, tiles_n, split;
  int out_fp32, accumulate, fp16, vec_ok;
  float alpha;
};

__device__ __forceinline__ void gs_cluster_sync() {
  asm volatile("barrier.cluster.arrive.release.aligned;\nbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ float4 gs_ld_cluster(uint32_t local, uint32_t rank) {
  uint32_t a;
  float4 v;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"(local), "r"(rank));
  asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];"
               : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w)
               : "r"(a)
               : "memory");
  return v;
}

template <bool A_MN, bool B_MN>
__global__ void __launch_bounds__(kGsThreads, 2)
gemm_small_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB,
                  const GemmSmallParams p) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* smem_a = smem;
  uint8_t* smem_b = smem + kGsStages * kGsABytes;
  uint64_t* full_bar = reinterpret_cast<uint64_t*>(smem + kGsBarOffset);
  uint64_t* empty_bar = full_bar + kGsStages;
  uint64_t* done_bar = empty_bar + kGsStages;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(done_bar + 1);
  volatile int* cta_abort = reinterpret_cast<volatile int*>(tmem_slot + 1);

  const int warp = uniform_warp(), lane = threadIdx.x & 31;
  const AbortCtx ab{cta_abort, p.status};
  const int rank = blockIdx.x % p.split;          // clusters are consecutive blocks: the rank inside the cluster
  int tile = blockIdx.x / p.split;
  const int b = tile / (p.tiles_m * p.tiles_n);
  tile -= b * p.tiles_m * p.tiles_n;
  const int m0 = (tile % p.tiles_m) * kGsBM, n0 = (tile / p.tiles_m) * kGsBN;
  const int num_kb = (p.K + kGsBK - 1) / kGsBK;
  const int kb0 = static_cast<int>(static_cast<long long>(rank) * num_kb / p.split);
  const int kb1 = static_cast<int>(static_cast<long long>(rank + 1) * num_kb / p.split);

  if (threadIdx.x == 0) {
    for (int s = 0; s < kGsStages; ++s) {
      mbar_init(&full_bar[s], 1);
      mbar_init(&empty_bar[s], 1);
    }
    mbar_init(done_bar, 1);
    *cta_abort = 0;
    fence_mbar_init();
    tma_prefetch_desc(&tmA);
    tma_prefetch_desc(&tmB);
  }
  if (warp == 1) {
    tmem_alloc(tmem_slot, kGsBN);
    tmem_relinquish();
  }
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tmem_base = __shfl_sync(0xffffffffu, *tmem_slot, 0);

  float* acc_s = reinterpret_cast<float*>(smem);   // [128][kGsPitch] once the stage ring is idle
  if (warp == 0) {
    if (lane == 0) {
      int s = 0;
      uint32_t ph = 0;
      for (int kb = kb0; kb < kb1; ++kb) {
        if (!mbar_wait(&empty_bar[s], ph ^ 1, ab)) break;
        mbar_expect_tx(&full_bar[s], kGsStageBytes);
        uint8_t* a_dst = smem_a + s * kGsABytes;
        uint8_t* b_dst = smem_b + s * kGsBBytes;
        const int k0 = kb * kGsBK;
        if (B_MN) tma_load_3d(b_dst, &tmB, &full_bar[s], n0, k0, b);
        else tma_load_3d(b_dst, &tmB, &full_bar[s], k0, n0, b);
        if (A_MN) {
          tma_load_3d(a_dst, &tmA, &full_bar[s], m0, k0, b);
          tma_load_3d(a_dst + 8192, &tmA, &full_bar[s], m0 + 64, k0, b);
        } else {
          tma_load_3d(a_dst, &tmA, &full_bar[s], k0, m0, b);
        }
        if (++s == kGsStages) { s = 0; ph ^= 1; }
      }
    }
    __syncwarp();
  } else if (warp == 1) {
    // the whole warp, one elected lane's instructions take effect
    const uint32_t idesc = p.fp16 ? umma_idesc_f16(kGsBM, kGsBN, A_MN, B_MN) : umma_idesc_bf16(kGsBM, kGsBN, A_MN, B_MN);
    const uint32_t lead = elect_one();
    const uint64_t a_desc = umma_smem_desc(smem_u32(smem_a), A_MN ? 8192 : 16, 1024);
    const uint64_t b_desc = umma_smem_desc(smem_u32(smem_b), B_MN ? 8192 : 16, 1024);
    int s = 0;
    uint32_t ph = 0;
    bool ok = true;
    for (int kb = kb0; kb < kb1; ++kb) {
      if (!(ok = mbar_wait_warp(&full_bar[s], ph, ab))) break;
      tc_fence_after_sync();
      const uint64_t ad = a_desc + s * (kGsABytes >> 4), bd = b_desc + s * (kGsBBytes >> 4);
      if (lead) {
#pragma unroll
        for (int kk = 0; kk < kGsBK / 16; ++kk)
          umma_bf16(tmem_base, ad + kk * (A_MN ? 128 : 2), bd + kk * (B_MN ? 128 : 2), idesc, (kb != kb0) || (kk != 0));
        umma_commit(&empty_bar[s]);
      }
      __syncwarp();
      if (++s == kGsStages) { s = 0; ph ^= 1; }
    }
    if (ok && lead) umma_commit(done_bar);
    __syncwarp();
  } else {
    // the accumulator into shared memory: the last product has read the stage ring
    const int q = warp & 3, row = q * 32 + lane;
    if (mbar_wait(done_bar, 0, ab)) {
      __syncwarp();
      tc_fence_after_sync();
      uint32_t r[2][32];
      const uint32_t t_row = tmem_base + (static_cast<uint32_t>(q * 32) << 16);
      tmem_ld_32x32(t_row, r[0]);
      tmem_ld_32x32(t_row + 32, r[1]);
      tmem_ld_wait();
#pragma unroll
      for (int j = 0; j < 16; ++j)
        *reinterpret_cast<uint4*>(acc_s + row * kGsPitch + j * 4) =
            make_uint4(r[j >> 3][(j & 7) * 4], r[j >> 3][(j & 7) * 4 + 1], r[j >> 3][(j & 7) * 4 + 2],
                       r[j >> 3][(j & 7) * 4 + 3]);
    }
    __syncwarp();
  }
  tc_fence_before_sync();
  if (p.split > 1) gs_cluster_sync();
  else __syncthreads();
  if (warp >= 2 && !*cta_abort) {
    // rows [lo, hi) of the tile are this CTA's to finish; 16 consecutive threads take the 64 columns of a row
    const int rows = min(kGsBM, p.M - m0);
    const int lo = rank * rows / p.split, hi = (rank + 1) * rows / p.split;
    const int t = threadIdx.x - 64, c = (t & 15) * 4, col = n0 + c;
    float bv[4] = {0.f, 0.f, 0.f, 0.f};
    if (p.bias) {
#pragma unroll
      for (int j = 0; j < 4; ++j)
        if (col + j < p.N) bv[j] = load_16(p.bias, col + j, p.fp16);
    }
    for (int row = lo + (t >> 4); row < hi; row += 8) {
      const uint32_t at = smem_u32(acc_s + row * kGsPitch + c);
      float v[4] = {0.f, 0.f, 0.f, 0.f};
      if (p.split > 1) {
        for (int k = 0; k < p.split; ++k) {
          const float4 x = gs_ld_cluster(at, k);
          v[0] += x.x; v[1] += x.y; v[2] += x.z; v[3] += x.w;
        }
      } else {
        *reinterpret_cast<float4*>(v) = *reinterpret_cast<const float4*>(acc_s + row * kGsPitch + c);
      }
#pragma unroll
      for (int j = 0; j < 4; ++j) v[j] = v[j] * p.alpha + bv[j];
      const long long off = b * p.c_batch_stride + static_cast<long long>(m0 + row) * p.ldc + col;
      if (p.out_fp32) {
        float* dst = static_cast<float*>(p.C) + off;
        if (p.vec_ok && col + 4 <= p.N) {
          float4 o = make_float4(v[0], v[1], v[2], v[3]);
          if (p.accumulate) {
            const float4 old = *reinterpret_cast<const float4*>(dst);
            o.x += old.x; o.y += old.y; o.z += old.z; o.w += old.w;
          }
          *reinterpret_cast<float4*>(dst) = o;
        } else {
          for (int j = 0; j < 4; ++j)
            if (col + j < p.N) dst[j] = p.accumulate ? dst[j] + v[j] : v[j];
        }
      } else if (p.vec_ok && col + 4 <= p.N) {
        *reinterpret_cast<uint2*>(static_cast<uint16_t*>(p.C) + off) =
            make_uint2(pack_16x2(v[0], v[1], p.fp16), pack_16x2(v[2], v[3], p.fp16));
      } else {
        for (int j = 0; j < 4; ++j)
          if (col + j < p.N) store_16(p.C, off + j, v[j], p.fp16);
      }
    }
  }
  // ---- teardown: no CTA leaves while another may read its accumulator
  __syncthreads();
  if (*cta_abort && threadIdx.x == 0) {
    // a wait was abandoned: give bulk copies that may still be in flight a bounded time to land
    const unsigned long long t0 = globaltimer_ns();
    while (globaltimer_ns() - t0 < 100000000ull) {
    }
  }
  __syncthreads();
  if (p.split > 1) gs_cluster_sync();
  if (warp == 1) {
    tc_fence_after_sync();
    tmem_dealloc(tmem_base, kGsBN);
  }
}

// How many CTAs share a tile's k-loop, or 0 when the problem is not small: fewer than half as many 128 x 128 tiles as
// SMs.  A larger split streams the operands through more SMs (two CTAs each) but leaves every CTA at least four k-blocks,
// the depth of its pipeline.
static inline int gemm_small_split(int M, int N, int K, int batch) {
  const long long t128 = static_cast<long long>((M + 127) / 128) * ((N + 127) / 128) * batch;
  if (2 * t128 > sm_count()) return 0;
  const long long tiles = static_cast<long long>((M + kGsBM - 1) / kGsBM) * ((N + kGsBN - 1) / kGsBN) * batch;
  const int num_kb = (K + kGsBK - 1) / kGsBK;
  int split = 1;
  while (split < kGsMaxSplit && tiles * split * 2 <= 2LL * sm_count() && num_kb / (split * 2) >= kGsStages) split *= 2;
  return split;
}

template <bool A_MN, bool B_MN>
static int launch_gemm_small(const CUtensorMap& tmA, const CUtensorMap& tmB, const GemmSmallParams& p, int batch,
                             cudaStream_t stream) {
  auto kern = gemm_small_kernel<A_MN, B_MN>;
  static bool configured = false;
  if (!configured) {
    MSB_CUDA_CHECK(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, kGsSmemBytes));
    configured = true;
  }
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(static_cast<unsigned>(p.tiles_m) * p.tiles_n * batch * p.split, 1, 1);
  cfg.blockDim = dim3(kGsThreads, 1, 1);
  cfg.dynamicSmemBytes = kGsSmemBytes;
  cfg.stream = stream;
  cudaLaunchAttribute attr;
  attr.id = cudaLaunchAttributeClusterDimension;
  attr.val.clusterDim.x = p.split;
  attr.val.clusterDim.y = 1;
  attr.val.clusterDim.z = 1;
  cfg.attrs = &attr;
  cfg.numAttrs = 1;
  MSB_CUDA_CHECK(cudaLaunchKernelEx(&cfg, kern, tmA, tmB, p));
  return kOk;
}

}  // namespace msb
