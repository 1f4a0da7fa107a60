// FlashAttention backward for sm_100a (head_dim 128, bf16; several query heads may share one k / v head), tcgen05 +
// TMEM + TMA.
//
// Three launches, all deterministic (no atomics):
//   1. row statistics: per 128-row block of a (batch, head), -lse * log2(e) and -scale * sum_d O * dO of its rows;
//      rows beyond the sequence get -inf and 0, so that their probabilities vanish
//   2. dK/dV kernel: one work item = (batch, k/v head, 128 keys); loops over the group's query heads and their 128-row
//      query blocks.  With keys as the M dimension, TMEM lane t belongs to key row t:
//         S^T  = K Q^T                          (TMEM, 128 columns)
//         P^T  = exp2(S^T * c - lse)            -> 16 bit, back into the columns it came from
//         dV  += P^T dO                         (A operand P^T from TMEM; accumulator 128 columns)
//         dP^T = V dO^T                         (TMEM, 128 columns)
//         dS^T = P^T o (dP^T - delta) * scale   -> 16 bit, back into dP^T's columns
//         dK  += dS^T Q                         (A operand dS^T from TMEM; accumulator 128 columns)
//      The Q and dO tiles are read both K-major (as B of S^T / dP^T) and MN-major (as B of dK / dV) from the
//      same shared-memory bytes.
//   3. dQ kernel: one work item = (batch, head, 128 queries); loops over 128-key blocks, TMEM lane t is query row t:
//         S = Q K^T (two buffers), dP = dO V^T, dS = P o (dP - delta) * scale -> S's columns, dQ += dS K.
// Warp roles: warp 0 TMA, warp 1 MMA issue, warps 2-5 / 6-9 compute and epilogue: both groups of four own all 128 rows,
// the first the left 64 columns of a tile, the second the right 64.
//
// What bounds them.  Per 128 x 128 tile the tensor core needs 4 x 512 cycles (dK/dV) or 3 x 512 (dQ), the exponentials
// 1024 (16 per cycle per SM).  The products of a tile are ordered so that one pair of them always runs beside the
// elementwise work: dK(i), dP(i+1) while P(i+1) is computed, dV(i+1), S(i+2) while dS(i+1) is.  Keeping P and dS in
// tensor memory takes their shared-memory round trip, its proxy fence and half of the operand reads away.
// Measured, 1 x 4096 x 32 heads causal, bf16: dK/dV 646 -> 262 us, dQ 299 -> 198 us, statistics 26 -> 18 us, against one
// warpgroup with P and dS in shared memory.  Groups that take whole 64-wide blocks in turn, each with buffers of its own,
// measured 305 us (dK/dV) and 253 us (dQ): a 64-column product reads as much of its A operand for half of the work.
//
// This text is compiled twice: for bf16 tensors (flash_attn_bwd_sm100.cu), and with MSB_ELEM_FP16 defined for fp16 tensors
// (flash_attn_bwd_sm100_fp16.cu), where every entry point carries the suffix _fp16 and "bf16" in a comment reads "fp16".
#include "fa_common.cuh"

namespace msb {
namespace MSB_ELEM_NS {

constexpr int kBwdThreads = 320;

struct FaBwdParams {
  const float* stats;   // [B][H][ceil(S / 128)][2][128]
  elem_t* dq;
  elem_t* dk;
  elem_t* dv;
  int* status;
  long long dq_pitch, dkv_pitch;
  int B, H, Hk, S;
  int causal;
  float scale, scale_log2;
};

// ------------------------------------------------------------------------------------------------ row statistics
// Sixteen lanes per row, 16 bytes each.
__global__ void __launch_bounds__(256)
fa_stats_kernel(const elem_t* __restrict__ o, const elem_t* __restrict__ dout, const float* __restrict__ lse,
                float* __restrict__ stats, int B, int S, int H, long long o_pitch, long long do_pitch, float scale) {
  const int nb = (S + 127) / 128;
  const long long g = (blockIdx.x * 256ll + threadIdx.x) >> 4;       // row index over (batch, padded token, head)
  const int part = threadIdx.x & 15;
  if (g >= (long long)B * nb * 128 * H) return;
  const int h = static_cast<int>(g % H);
  const long long t = g / H;
  const int s = static_cast<int>(t % (nb * 128)), b = static_cast<int>(t / (nb * 128));
  float d = 0.f, l = -INFINITY;
  if (s < S) {
    const long long tok = (long long)b * S + s;
    const uint4 x = *reinterpret_cast<const uint4*>(o + tok * o_pitch + (long long)h * kFaD + part * 8);
    const uint4 y = *reinterpret_cast<const uint4*>(dout + tok * do_pitch + (long long)h * kFaD + part * 8);
    const elem2_t* xe = reinterpret_cast<const elem2_t*>(&x);
    const elem2_t* ye = reinterpret_cast<const elem2_t*>(&y);
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const float2 u = e2_to_f2(xe[i]), v = e2_to_f2(ye[i]);
      d += u.x * v.x + u.y * v.y;
    }
    l = lse[((long long)b * H + h) * S + s] * -1.4426950408889634f;
  }
#pragma unroll
  for (int off = 8; off > 0; off >>= 1) d += __shfl_xor_sync(0xffffffffu, d, off);
  if (part == 0) {
    float* out = stats + (((long long)b * H + h) * nb + (s >> 7)) * 256 + (s & 127);
    out[0] = l;
    out[128] = -d * scale;
  }
}

// 1 KB of row statistics into shared memory, counted on `bar`.
__device__ __forceinline__ void fa_load_stats(void* dst, const float* src, uint64_t* bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                   smem_u32(dst)),
               "l"(src), "r"(1024), "r"(smem_u32(bar))
               : "memory");
}

// One 128-column accumulator row (this thread's TMEM lane) as 16-bit values to global memory.
__device__ __forceinline__ void fa_store_row(uint32_t tm, elem_t* dst, bool live) {
#pragma unroll
  for (int c = 0; c < 4; ++c) {
    uint32_t r[32];
    tmem_ld_32x32(tm + c * 32, r);
    tmem_ld_wait();
    if (live) {
#pragma unroll
      for (int t = 0; t < 32; t += 8) {
        uint4 v;
        v.x = pack_e2(__uint_as_float(r[t + 0]), __uint_as_float(r[t + 1]));
        v.y = pack_e2(__uint_as_float(r[t + 2]), __uint_as_float(r[t + 3]));
        v.z = pack_e2(__uint_as_float(r[t + 4]), __uint_as_float(r[t + 5]));
        v.w = pack_e2(__uint_as_float(r[t + 6]), __uint_as_float(r[t + 7]));
        *reinterpret_cast<uint4*>(dst + c * 32 + t) = v;
      }
    }
  }
}

// TMEM column of k-step kk (16 values, 8 columns) of a 16-bit A operand whose two 64-wide halves lie in the first 32 of
// the 64 columns that each compute group owns.
__device__ __forceinline__ uint32_t fa_half_col(int kk) { return (kk >> 2) * 64 + (kk & 3) * 8; }

// ------------------------------------------------------------------------------------------------ dK / dV
struct KvSmem {
  static constexpr int kK = 0;                 // 32 KB
  static constexpr int kV = 32768;             // 32 KB
  static constexpr int kQ = 65536;             // 2 x 32 KB
  static constexpr int kDO = 131072;           // 2 x 32 KB
  static constexpr int kStats = 196608;        // 2 x 1 KB
  static constexpr int kBar = 198656;
  static constexpr int kBytes = kBar + 256 + 1024;
};

__global__ void __launch_bounds__(kBwdThreads, 1)
fa_bwd_dkdv_kernel(const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ CUtensorMap tmK,
                   const __grid_constant__ CUtensorMap tmV, const __grid_constant__ CUtensorMap tmDO,
                   const FaBwdParams p) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + KvSmem::kBar);
  uint64_t* kv_full = bars + 0;
  uint64_t* kv_empty = bars + 1;
  uint64_t* q_full = bars + 2;     // [2]  Q tile and row statistics
  uint64_t* q_empty = bars + 4;    // [2]
  uint64_t* do_full = bars + 6;    // [2]
  uint64_t* do_empty = bars + 8;   // [2]
  uint64_t* s_full = bars + 10;
  uint64_t* dp_full = bars + 11;
  uint64_t* p_ready = bars + 12;
  uint64_t* ds_ready = bars + 13;
  uint64_t* acc_done = bars + 14;
  uint64_t* acc_empty = bars + 15;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 16);
  volatile int* cta_abort = reinterpret_cast<volatile int*>(tmem_slot + 1);

  const int warp = uniform_warp(), lane = threadIdx.x & 31;
  const AbortCtx ab{cta_abort, p.status};
  const int nb = (p.S + 127) / 128;
  const int total = p.B * p.Hk * nb;
  const int group = p.H / p.Hk;

  if (threadIdx.x == 0) {
    mbar_init(kv_full, 1);
    mbar_init(kv_empty, 1);
    for (int i = 0; i < 2; ++i) {
      mbar_init(&q_full[i], 1);
      mbar_init(&q_empty[i], 1);
      mbar_init(&do_full[i], 1);
      mbar_init(&do_empty[i], 1);
    }
    mbar_init(s_full, 1);
    mbar_init(dp_full, 1);
    mbar_init(p_ready, 8);
    mbar_init(ds_ready, 8);
    mbar_init(acc_done, 1);
    mbar_init(acc_empty, 8);
    *cta_abort = 0;
    fence_mbar_init();
    tma_prefetch_desc(&tmQ);
    tma_prefetch_desc(&tmK);
    tma_prefetch_desc(&tmV);
    tma_prefetch_desc(&tmDO);
  }
  if (warp == 1) {
    tmem_alloc(tmem_slot, 512);
    tmem_relinquish();
  }
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tmem_base = __shfl_sync(0xffffffffu, *tmem_slot, 0);
  const uint32_t tm_s = tmem_base, tm_dp = tmem_base + 128, tm_dv = tmem_base + 256, tm_dk = tmem_base + 384;

  // item w -> (b, hk, key block jb); causal: the long items (small jb) first
  auto item = [&](int w, int& b, int& hk, int& jb) {
    const int bh = p.B * p.Hk;
    jb = w / bh;
    const int r = w % bh;
    b = r / p.Hk;
    hk = r % p.Hk;
  };

  if (warp == 0) {
    if (lane == 0) {
      uint32_t items = 0, qc = 0;
      bool ok = true;
      for (int round = 0, w; ok && (w = fa_snake(round)) < total; ++round, ++items) {
        int b, hk, jb;
        item(w, b, hk, jb);
        const int i0 = p.causal ? jb : 0;
        if (!mbar_wait(kv_empty, (items & 1) ^ 1, ab)) { ok = false; break; }
        mbar_expect_tx(kv_full, 65536);
        fa_load_tile(smem + KvSmem::kK, &tmK, kv_full, 128, hk, jb * 128, b);
        fa_load_tile(smem + KvSmem::kV, &tmV, kv_full, 128, hk, jb * 128, b);
        for (int g = 0; g < group && ok; ++g) {
          const int h = hk * group + g;
          for (int i = i0; i < nb; ++i, ++qc) {
            const int st = qc & 1;
            const uint32_t ph = (qc >> 1) & 1;
            if (!mbar_wait(&q_empty[st], ph ^ 1, ab)) { ok = false; break; }
            mbar_expect_tx(&q_full[st], 32768 + 1024);
            fa_load_tile(smem + KvSmem::kQ + st * 32768, &tmQ, &q_full[st], 128, h, i * 128, b);
            fa_load_stats(smem + KvSmem::kStats + st * 1024,
                          p.stats + ((static_cast<long long>(b) * p.H + h) * nb + i) * 256, &q_full[st]);
            if (!mbar_wait(&do_empty[st], ph ^ 1, ab)) { ok = false; break; }
            mbar_expect_tx(&do_full[st], 32768);
            fa_load_tile(smem + KvSmem::kDO + st * 32768, &tmDO, &do_full[st], 128, h, i * 128, b);
          }
        }
      }
    }
    __syncwarp();
  } else if (warp == 1) {
    // the whole warp, one elected lane's instructions take effect
    constexpr uint32_t idesc_st = umma_idesc_elem(128, 128, false, false);   // [keys x queries], K = d
    constexpr uint32_t idesc_acc = umma_idesc_elem(128, 128, false, true);   // [keys x d], K = queries, B MN-major
    const uint32_t lead = elect_one();
    const uint64_t k_desc = umma_smem_desc(smem_u32(smem + KvSmem::kK), 16, 1024);
    const uint64_t v_desc = umma_smem_desc(smem_u32(smem + KvSmem::kV), 16, 1024);
    // Q and dO tiles: K-major for S^T / dP^T, MN-major for dK / dV; the two buffers are 32 KB apart
    const uint64_t q_desc = umma_smem_desc(smem_u32(smem + KvSmem::kQ), 16, 1024);
    const uint64_t do_desc = umma_smem_desc(smem_u32(smem + KvSmem::kDO), 16, 1024);
    const uint64_t q_mn_desc = umma_smem_desc(smem_u32(smem + KvSmem::kQ), 16384, 1024);
    const uint64_t do_mn_desc = umma_smem_desc(smem_u32(smem + KvSmem::kDO), 16384, 1024);
    constexpr uint64_t kBuf = 32768 >> 4;
    uint32_t items = 0, qc = 0;
    bool ok = true;
    auto commit = [&](uint64_t* bar) {
      if (lead) umma_commit(bar);
      __syncwarp();
    };
    auto issue_front = [&](uint32_t tm, uint64_t ad, uint64_t bd, uint64_t* done) {
      if (lead) {
#pragma unroll
        for (int kk = 0; kk < 8; ++kk) {
          const uint32_t off = ((kk >> 2) * 16384 + (kk & 3) * 32) >> 4;
          umma_bf16(tm, ad + off, bd + off, idesc_st, kk != 0);
        }
        umma_commit(done);
      }
      __syncwarp();
    };
    auto issue_acc = [&](uint32_t tm_acc, uint32_t tm_a, uint64_t bd, bool first, uint64_t* done) {
      if (lead) {
#pragma unroll
        for (int kk = 0; kk < 8; ++kk)
          umma_ts(tm_acc, tm_a + fa_half_col(kk), bd + ((kk * 2048) >> 4), idesc_acc, !(first && kk == 0));
        umma_commit(done);
      }
      __syncwarp();
    };
    auto issue_s = [&](uint32_t c) -> bool {
      const int st = c & 1;
      if (!mbar_wait_warp(&q_full[st], (c >> 1) & 1, ab)) return false;
      tc_fence_after_sync();
      issue_front(tm_s, k_desc, q_desc + st * kBuf, s_full);
      return true;
    };
    auto issue_dp = [&](uint32_t c) -> bool {
      const int st = c & 1;
      if (!mbar_wait_warp(&do_full[st], (c >> 1) & 1, ab)) return false;
      tc_fence_after_sync();
      issue_front(tm_dp, v_desc, do_desc + st * kBuf, dp_full);
      return true;
    };
    for (int round = 0, w; ok && (w = fa_snake(round)) < total; ++round, ++items) {
      int b, hk, jb;
      item(w, b, hk, jb);
      const int nblk = group * (nb - (p.causal ? jb : 0));
      if (!mbar_wait_warp(kv_full, items & 1, ab)) { ok = false; break; }
      if (!issue_s(qc) || !issue_dp(qc)) { ok = false; break; }
      if (nblk == 1) commit(kv_empty);
      for (int i = 0; i < nblk; ++i) {
        const uint32_t c = qc + i;
        const int st = c & 1;
        if (i == 0 && !mbar_wait_warp(acc_empty, (items & 1) ^ 1, ab)) { ok = false; break; }
        if (!mbar_wait_warp(p_ready, c & 1, ab)) { ok = false; break; }
        tc_fence_after_sync();
        issue_acc(tm_dv, tm_s, do_mn_desc + st * kBuf, i == 0, &do_empty[st]);
        // S of the next block goes over P^T: it executes behind the product that reads P^T
        if (i + 1 < nblk && !issue_s(c + 1)) { ok = false; break; }
        if (!mbar_wait_warp(ds_ready, c & 1, ab)) { ok = false; break; }
        tc_fence_after_sync();
        issue_acc(tm_dk, tm_dp, q_mn_desc + st * kBuf, i == 0, &q_empty[st]);
        if (i + 1 < nblk && !issue_dp(c + 1)) { ok = false; break; }
        if (i + 2 == nblk) commit(kv_empty);      // the last products with K and V are in flight
      }
      if (!ok) break;
      commit(acc_done);
      qc += nblk;
    }
    __syncwarp();
  } else {
    const int half = (warp - 2) >> 2;  // which 64 query columns
    const int q4 = warp & 3;
    const int row = q4 * 32 + lane;    // key row inside the 128-key block == TMEM lane
    const uint32_t sel = (static_cast<uint32_t>(q4 * 32) << 16) + half * 64;
    uint32_t items = 0, qc = 0;
    bool ok = true;
    const uint64_t slog2 = f32x2(p.scale_log2, p.scale_log2), scale2 = f32x2(p.scale, p.scale);
    for (int round = 0, w; ok && (w = fa_snake(round)) < total; ++round, ++items) {
      int b, hk, jb;
      item(w, b, hk, jb);
      const int per = nb - (p.causal ? jb : 0);
      const int nblk = group * per;
      int in_head = 0;                 // query block counted from the head's first one
      for (int i = 0; i < nblk; ++i, ++qc) {
        const int st = qc & 1;
        const float* stats = reinterpret_cast<const float*>(smem + KvSmem::kStats + st * 1024) + half * 64;
        float pv[64];
        if (!mbar_wait(&q_full[st], (qc >> 1) & 1, ab)) { ok = false; break; }     // the row statistics
        if (!mbar_wait(s_full, qc & 1, ab)) { ok = false; break; }
        tc_fence_after_sync();
        {
          uint32_t r[2][32];
          tmem_ld_32x32(tm_s + sel, r[0]);
          tmem_ld_32x32(tm_s + sel + 32, r[1]);
          tmem_ld_wait();
          uint32_t pk[32];
#pragma unroll
          for (int c4 = 0; c4 < 16; ++c4) {
            const ulonglong2 nl = *reinterpret_cast<const ulonglong2*>(stats + c4 * 4);
#pragma unroll
            for (int u = 0; u < 2; ++u) {
              const int c = c4 * 4 + u * 2;
              f32x2_split(fma2(f32x2(__uint_as_float(r[c >> 5][c & 31]), __uint_as_float(r[c >> 5][(c & 31) + 1])),
                               slog2, u ? nl.y : nl.x),
                          pv[c], pv[c + 1]);
              pv[c] = ex2(pv[c]);
              pv[c + 1] = ex2(pv[c + 1]);
            }
          }
          if (p.causal && in_head == 0) {       // diagonal block: query c sees keys up to its own
#pragma unroll
            for (int c = 0; c < 64; ++c)
              if (half * 64 + c < row) pv[c] = 0.f;
          }
#pragma unroll
          for (int c = 0; c < 32; ++c) pk[c] = pack_e2(pv[2 * c], pv[2 * c + 1]);
          tmem_st_32x32(tm_s + sel, pk);
        }
        tmem_st_wait();
        tc_fence_before_sync();
        warp_arrive(p_ready, lane);
        // ---- dS^T
        if (!mbar_wait(dp_full, qc & 1, ab)) { ok = false; break; }
        tc_fence_after_sync();
        {
          uint32_t r[2][32];
          tmem_ld_32x32(tm_dp + sel, r[0]);
          tmem_ld_32x32(tm_dp + sel + 32, r[1]);
          tmem_ld_wait();
          uint32_t pk[32];
#pragma unroll
          for (int c4 = 0; c4 < 16; ++c4) {
            const ulonglong2 nd = *reinterpret_cast<const ulonglong2*>(stats + 128 + c4 * 4);
#pragma unroll
            for (int u = 0; u < 2; ++u) {
              const int c = c4 * 4 + u * 2;
              const uint64_t d = fma2(f32x2(__uint_as_float(r[c >> 5][c & 31]), __uint_as_float(r[c >> 5][(c & 31) + 1])),
                                      scale2, u ? nd.y : nd.x);
              float x, y;
              f32x2_split(mul2(f32x2(pv[c], pv[c + 1]), d), x, y);
              pk[c >> 1] = pack_e2(x, y);
            }
          }
          tmem_st_32x32(tm_dp + sel, pk);
        }
        tmem_st_wait();
        tc_fence_before_sync();
        warp_arrive(ds_ready, lane);
        if (++in_head == per) in_head = 0;
      }
      if (!ok) break;
      // ---- epilogue: the first group stores the dV rows, the second the dK rows
      if (!mbar_wait(acc_done, items & 1, ab)) { ok = false; break; }
      tc_fence_after_sync();
      const int key = jb * 128 + row;
      elem_t* orow = (half == 0 ? p.dv : p.dk) + (static_cast<long long>(b) * p.S + key) * p.dkv_pitch +
                     static_cast<long long>(hk) * kFaD;
      fa_store_row((half == 0 ? tm_dv : tm_dk) + (static_cast<uint32_t>(q4 * 32) << 16), orow, key < p.S);
      tc_fence_before_sync();
      warp_arrive(acc_empty, lane);
    }
  }

  tc_fence_before_sync();
  __syncthreads();
  if (*cta_abort && threadIdx.x == 0) {
    // a wait was abandoned: give bulk copies that may still be in flight a bounded time to land
    const unsigned long long t0 = globaltimer_ns();
    while (globaltimer_ns() - t0 < 100000000ull) {
    }
  }
  __syncthreads();
  if (warp == 1) {
    tc_fence_after_sync();
    tmem_dealloc(tmem_base, 512);
  }
}

// ------------------------------------------------------------------------------------------------ dQ
struct DqSmem {
  static constexpr int kQ = 0;          // 32 KB
  static constexpr int kDO = 32768;     // 32 KB
  static constexpr int kK = 65536;      // 2 x 32 KB
  static constexpr int kV = 131072;     // 2 x 32 KB
  static constexpr int kBar = 196608;
  static constexpr int kBytes = kBar + 256 + 1024;
};

__global__ void __launch_bounds__(kBwdThreads, 1)
fa_bwd_dq_kernel(const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ CUtensorMap tmK,
                 const __grid_constant__ CUtensorMap tmV, const __grid_constant__ CUtensorMap tmDO,
                 const FaBwdParams p) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + DqSmem::kBar);
  uint64_t* qdo_full = bars + 0;
  uint64_t* qdo_empty = bars + 1;
  uint64_t* k_full = bars + 2;    // [2]
  uint64_t* k_empty = bars + 4;   // [2]
  uint64_t* v_full = bars + 6;    // [2]
  uint64_t* v_empty = bars + 8;   // [2]
  uint64_t* s_full = bars + 10;   // [2]
  uint64_t* dp_full = bars + 12;
  uint64_t* ds_ready = bars + 13;
  uint64_t* dq_done = bars + 14;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 15);
  volatile int* cta_abort = reinterpret_cast<volatile int*>(tmem_slot + 1);

  const int warp = uniform_warp(), lane = threadIdx.x & 31;
  const AbortCtx ab{cta_abort, p.status};
  const int nb = (p.S + 127) / 128;
  const int total = p.B * p.H * nb;
  const int group = p.H / p.Hk;

  if (threadIdx.x == 0) {
    mbar_init(qdo_full, 1);
    mbar_init(qdo_empty, 1);
    for (int i = 0; i < 2; ++i) {
      mbar_init(&k_full[i], 1);
      mbar_init(&k_empty[i], 1);
      mbar_init(&v_full[i], 1);
      mbar_init(&v_empty[i], 1);
      mbar_init(&s_full[i], 1);
    }
    mbar_init(dp_full, 1);
    mbar_init(ds_ready, 8);
    mbar_init(dq_done, 1);
    *cta_abort = 0;
    fence_mbar_init();
    tma_prefetch_desc(&tmQ);
    tma_prefetch_desc(&tmK);
    tma_prefetch_desc(&tmV);
    tma_prefetch_desc(&tmDO);
  }
  if (warp == 1) {
    tmem_alloc(tmem_slot, 512);
    tmem_relinquish();
  }
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tmem_base = __shfl_sync(0xffffffffu, *tmem_slot, 0);
  const uint32_t tm_s = tmem_base, tm_dp = tmem_base + 256, tm_dq = tmem_base + 384;

  auto item = [&](int w, int& b, int& h, int& qb) {
    const int bh = p.B * p.H;
    qb = nb - 1 - w / bh;
    const int r = w % bh;
    b = r / p.H;
    h = r % p.H;
  };

  if (warp == 0) {
    if (lane == 0) {
      uint32_t items = 0, kvc = 0;
      bool ok = true;
      for (int round = 0, w; ok && (w = fa_snake(round)) < total; ++round, ++items) {
        int b, h, qb;
        item(w, b, h, qb);
        const int nblk = p.causal ? qb + 1 : nb, hk = h / group;
        if (!mbar_wait(qdo_empty, (items & 1) ^ 1, ab)) { ok = false; break; }
        mbar_expect_tx(qdo_full, 65536);
        fa_load_tile(smem + DqSmem::kQ, &tmQ, qdo_full, 128, h, qb * 128, b);
        fa_load_tile(smem + DqSmem::kDO, &tmDO, qdo_full, 128, h, qb * 128, b);
        for (int j = 0; j < nblk; ++j, ++kvc) {
          const int st = kvc & 1;
          const uint32_t ph = (kvc >> 1) & 1;
          if (!mbar_wait(&k_empty[st], ph ^ 1, ab)) { ok = false; break; }
          mbar_expect_tx(&k_full[st], 32768);
          fa_load_tile(smem + DqSmem::kK + st * 32768, &tmK, &k_full[st], 128, hk, j * 128, b);
          if (!mbar_wait(&v_empty[st], ph ^ 1, ab)) { ok = false; break; }
          mbar_expect_tx(&v_full[st], 32768);
          fa_load_tile(smem + DqSmem::kV + st * 32768, &tmV, &v_full[st], 128, hk, j * 128, b);
        }
      }
    }
    __syncwarp();
  } else if (warp == 1) {
    // the whole warp, one elected lane's instructions take effect
    constexpr uint32_t idesc_kk = umma_idesc_elem(128, 128, false, false);
    constexpr uint32_t idesc_mn = umma_idesc_elem(128, 128, false, true);
    const uint32_t lead = elect_one();
    const uint64_t q_desc = umma_smem_desc(smem_u32(smem + DqSmem::kQ), 16, 1024);
    const uint64_t do_desc = umma_smem_desc(smem_u32(smem + DqSmem::kDO), 16, 1024);
    const uint64_t k_desc = umma_smem_desc(smem_u32(smem + DqSmem::kK), 16, 1024);
    const uint64_t v_desc = umma_smem_desc(smem_u32(smem + DqSmem::kV), 16, 1024);
    const uint64_t k_mn_desc = umma_smem_desc(smem_u32(smem + DqSmem::kK), 16384, 1024);
    constexpr uint64_t kBuf = 32768 >> 4;
    uint32_t items = 0, kvc = 0;
    bool ok = true;
    auto commit = [&](uint64_t* bar) {
      if (lead) umma_commit(bar);
      __syncwarp();
    };
    auto issue_front = [&](uint32_t tm, uint64_t ad, uint64_t bd, uint64_t* done) {
      if (lead) {
#pragma unroll
        for (int kk = 0; kk < 8; ++kk) {
          const uint32_t off = ((kk >> 2) * 16384 + (kk & 3) * 32) >> 4;
          umma_bf16(tm, ad + off, bd + off, idesc_kk, kk != 0);
        }
        umma_commit(done);
      }
      __syncwarp();
    };
    auto issue_s = [&](uint32_t c) -> bool {
      const int st = c & 1;
      if (!mbar_wait_warp(&k_full[st], (c >> 1) & 1, ab)) return false;
      tc_fence_after_sync();
      issue_front(tm_s + st * 128, q_desc, k_desc + st * kBuf, &s_full[st]);
      return true;
    };
    auto issue_dp = [&](uint32_t c) -> bool {
      const int st = c & 1;
      if (!mbar_wait_warp(&v_full[st], (c >> 1) & 1, ab)) return false;
      tc_fence_after_sync();
      issue_front(tm_dp, do_desc, v_desc + st * kBuf, dp_full);
      commit(&v_empty[st]);
      return true;
    };
    for (int round = 0, w; ok && (w = fa_snake(round)) < total; ++round, ++items) {
      int b, h, qb;
      item(w, b, h, qb);
      const int nblk = p.causal ? qb + 1 : nb;
      if (!mbar_wait_warp(qdo_full, items & 1, ab)) { ok = false; break; }
      if (!issue_s(kvc) || !issue_dp(kvc)) { ok = false; break; }
      if (nblk == 1) commit(qdo_empty);
      for (int j = 0; j < nblk; ++j) {
        const uint32_t c = kvc + j;
        const int st = c & 1;
        // S of the next block goes into the buffer whose dS the previous block's product has read
        if (j + 1 < nblk && !issue_s(c + 1)) { ok = false; break; }
        if (!mbar_wait_warp(ds_ready, c & 1, ab)) { ok = false; break; }
        tc_fence_after_sync();
        if (lead) {
#pragma unroll
          for (int kk = 0; kk < 8; ++kk)
            umma_ts(tm_dq, tm_s + st * 128 + fa_half_col(kk), k_mn_desc + st * kBuf + ((kk * 2048) >> 4), idesc_mn,
                    (j | kk) != 0);
          umma_commit(&k_empty[st]);
        }
        __syncwarp();
        if (j + 1 < nblk && !issue_dp(c + 1)) { ok = false; break; }
        if (j + 2 == nblk) commit(qdo_empty);     // the last products with Q and dO are in flight
      }
      if (!ok) break;
      commit(dq_done);
      kvc += nblk;
    }
    __syncwarp();
  } else {
    const int half = (warp - 2) >> 2;  // which 64 key columns
    const int q4 = warp & 3;
    const int row = q4 * 32 + lane;
    const uint32_t lane_sel = static_cast<uint32_t>(q4 * 32) << 16;
    const uint32_t sel = lane_sel + half * 64;
    uint32_t items = 0, kvc = 0;
    bool ok = true;
    const uint64_t slog2 = f32x2(p.scale_log2, p.scale_log2), scale2 = f32x2(p.scale, p.scale);
    for (int round = 0, w; ok && (w = fa_snake(round)) < total; ++round, ++items) {
      int b, h, qb;
      item(w, b, h, qb);
      const int nblk = p.causal ? qb + 1 : nb;
      const float* stats = p.stats + ((static_cast<long long>(b) * p.H + h) * nb + qb) * 256 + row;
      const float nl = stats[0], nd = stats[128];
      const uint64_t nl2 = f32x2(nl, nl), nd2 = f32x2(nd, nd);
      for (int j = 0; j < nblk; ++j, ++kvc) {
        const int st = kvc & 1;
        float pv[64];
        if (!mbar_wait(&s_full[st], (kvc >> 1) & 1, ab)) { ok = false; break; }
        tc_fence_after_sync();
        {
          uint32_t r[2][32];
          tmem_ld_32x32(tm_s + st * 128 + sel, r[0]);
          tmem_ld_32x32(tm_s + st * 128 + sel + 32, r[1]);
          tmem_ld_wait();
#pragma unroll
          for (int c = 0; c < 64; c += 2) {
            f32x2_split(fma2(f32x2(__uint_as_float(r[c >> 5][c & 31]), __uint_as_float(r[c >> 5][(c & 31) + 1])), slog2,
                             nl2),
                        pv[c], pv[c + 1]);
            pv[c] = ex2(pv[c]);
            pv[c + 1] = ex2(pv[c + 1]);
          }
        }
        const bool diag = p.causal && j == qb, tail = (j + 1) * 128 > p.S;
        if (diag || tail) {
          int limit = p.S - j * 128;
          if (diag) limit = min(limit, row + 1);
#pragma unroll
          for (int c = 0; c < 64; ++c)
            if (half * 64 + c >= limit) pv[c] = 0.f;
        }
        if (!mbar_wait(dp_full, kvc & 1, ab)) { ok = false; break; }
        tc_fence_after_sync();
        {
          uint32_t r[2][32];
          tmem_ld_32x32(tm_dp + sel, r[0]);
          tmem_ld_32x32(tm_dp + sel + 32, r[1]);
          tmem_ld_wait();
          uint32_t pk[32];
#pragma unroll
          for (int c = 0; c < 64; c += 2) {
            const uint64_t d = fma2(f32x2(__uint_as_float(r[c >> 5][c & 31]), __uint_as_float(r[c >> 5][(c & 31) + 1])),
                                    scale2, nd2);
            float x, y;
            f32x2_split(mul2(f32x2(pv[c], pv[c + 1]), d), x, y);
            pk[c >> 1] = pack_e2(x, y);
          }
          tmem_st_32x32(tm_s + st * 128 + sel, pk);
        }
        tmem_st_wait();
        tc_fence_before_sync();
        warp_arrive(ds_ready, lane);
      }
      if (!ok) break;
      if (!mbar_wait(dq_done, items & 1, ab)) { ok = false; break; }
      tc_fence_after_sync();
      // epilogue: each group stores the left or the right half of the rows.  The next write to dQ comes behind these
      // threads' next ds_ready.
      const int qrow = qb * 128 + row;
      elem_t* orow = p.dq + (static_cast<long long>(b) * p.S + qrow) * p.dq_pitch + static_cast<long long>(h) * kFaD +
                     half * 64;
#pragma unroll
      for (int c = 0; c < 2; ++c) {
        uint32_t r[32];
        tmem_ld_32x32(tm_dq + sel + c * 32, r);
        tmem_ld_wait();
        if (qrow < p.S) {
#pragma unroll
          for (int t = 0; t < 32; t += 8) {
            uint4 v;
            v.x = pack_e2(__uint_as_float(r[t + 0]), __uint_as_float(r[t + 1]));
            v.y = pack_e2(__uint_as_float(r[t + 2]), __uint_as_float(r[t + 3]));
            v.z = pack_e2(__uint_as_float(r[t + 4]), __uint_as_float(r[t + 5]));
            v.w = pack_e2(__uint_as_float(r[t + 6]), __uint_as_float(r[t + 7]));
            *reinterpret_cast<uint4*>(orow + c * 32 + t) = v;
          }
        }
      }
      tc_fence_before_sync();
    }
  }

  tc_fence_before_sync();
  __syncthreads();
  if (*cta_abort && threadIdx.x == 0) {
    const unsigned long long t0 = globaltimer_ns();
    while (globaltimer_ns() - t0 < 100000000ull) {
    }
  }
  __syncthreads();
  if (warp == 1) {
    tc_fence_after_sync();
    tmem_dealloc(tmem_base, 512);
  }
}

}  // namespace MSB_ELEM_NS
}  // namespace msb

using namespace msb;
using namespace msb::MSB_ELEM_NS;

static int fa_bwd_impl(const void* q, const void* k, const void* v, const void* o, const void* dout, const float* lse,
                       float* stats, void* dq, void* dk, void* dv, int B, int S, int H, int Hk, int D,
                       long long q_pitch, long long k_pitch, long long v_pitch, long long o_pitch, long long do_pitch,
                       long long dq_pitch, long long dkv_pitch, int causal, float scale, void* stream_) {
  if ((dq_pitch % 8) || (dkv_pitch % 8) || (reinterpret_cast<uintptr_t>(dq) & 15) ||
      (reinterpret_cast<uintptr_t>(dk) & 15) || (reinterpret_cast<uintptr_t>(dv) & 15)) {
    set_last_error("flash_attn_bwd: gradient pitches must be multiples of 8 elements and pointers 16-byte aligned");
    return kBadArg;
  }
  if (D != kFaD || S <= 0 || Hk <= 0 || H % Hk != 0 || B <= 0) {
    set_last_error("flash_attn_bwd: needs head_dim 128 and H a multiple of Hk "
                   "(got D=%d S=%d H=%d Hk=%d)", D, S, H, Hk);
    return kBadArg;
  }
  if (o_pitch % 8 || do_pitch % 8 || (reinterpret_cast<uintptr_t>(o) & 15) || (reinterpret_cast<uintptr_t>(stats) & 15)) {
    set_last_error("flash_attn_bwd: o/do pitches must be multiples of 8 elements and o, stats 16-byte aligned");
    return kBadArg;
  }
  int* status = status_ptr();
  if (!status) { set_last_error("flash_attn_bwd: no status word"); return kCudaError; }
  cudaStream_t stream = static_cast<cudaStream_t>(stream_);
  const int nb = (S + 127) / 128;
  const long long rows = (long long)B * nb * 128 * H;
  fa_stats_kernel<<<(unsigned)((rows * 16 + 255) / 256), 256, 0, stream>>>(
      static_cast<const elem_t*>(o), static_cast<const elem_t*>(dout), lse, stats, B, S, H, o_pitch, do_pitch, scale);
  MSB_CUDA_CHECK(cudaGetLastError());

  CUtensorMap tq, tdo, tk, tv;
  int rc;
  if ((rc = fa_encode_map(&tq, q, B, S, H, q_pitch, 128)) != kOk) return rc;
  if ((rc = fa_encode_map(&tdo, dout, B, S, H, do_pitch, 128)) != kOk) return rc;
  if ((rc = fa_encode_map(&tk, k, B, S, Hk, k_pitch, 128)) != kOk) return rc;
  if ((rc = fa_encode_map(&tv, v, B, S, Hk, v_pitch, 128)) != kOk) return rc;
  static bool configured = false;
  if (!configured) {
    MSB_CUDA_CHECK(cudaFuncSetAttribute(fa_bwd_dkdv_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                        KvSmem::kBytes));
    MSB_CUDA_CHECK(cudaFuncSetAttribute(fa_bwd_dq_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                        DqSmem::kBytes));
    configured = true;
  }
  FaBwdParams p;
  p.stats = stats;
  p.dq = static_cast<elem_t*>(dq);
  p.dk = static_cast<elem_t*>(dk);
  p.dv = static_cast<elem_t*>(dv);
  p.status = status;
  p.dq_pitch = dq_pitch;
  p.dkv_pitch = dkv_pitch;
  p.B = B; p.H = H; p.Hk = Hk; p.S = S; p.causal = causal;
  p.scale = scale;
  p.scale_log2 = scale * 1.4426950408889634f;
  const int kv_items = B * Hk * nb, q_items = B * H * nb;
  fa_bwd_dkdv_kernel<<<kv_items < sm_count() ? kv_items : sm_count(), kBwdThreads, KvSmem::kBytes, stream>>>(tq, tk, tv, tdo,
                                                                                                         p);
  MSB_CUDA_CHECK(cudaGetLastError());
  fa_bwd_dq_kernel<<<q_items < sm_count() ? q_items : sm_count(), kBwdThreads, DqSmem::kBytes, stream>>>(tq, tk, tv, tdo, p);
  MSB_CUDA_CHECK(cudaGetLastError());
  return kOk;
}

// All tensors token-major [B,S,H,128] with the given token pitches (elements).  stats: fp32 scratch of
// 2 * B * H * (S rounded up to 128) floats that this call fills.  dq / dk / dv are written densely ([B,S,H,128]).
MSB_EXPORT int MSB_FN(msb_flash_attn_bwd)(const void* q, const void* k, const void* v, const void* o, const void* dout,
                                  const float* lse, float* stats, void* dq, void* dk, void* dv, int B, int S, int H,
                                  int Hk, int D, long long q_pitch, long long k_pitch, long long v_pitch,
                                  long long o_pitch, long long do_pitch, int causal, float scale, void* stream) {
  return fa_bwd_impl(q, k, v, o, dout, lse, stats, dq, dk, dv, B, S, H, Hk, D, q_pitch, k_pitch, v_pitch, o_pitch,
                     do_pitch, (long long)H * kFaD, (long long)Hk * kFaD, causal, scale, stream);
}

// Same, with the token pitches of the gradient outputs given: lets dq, dk, dv be column blocks of one packed
// [tokens, (H + 2 Hk) * 128] gradient of a fused QKV projection.
MSB_EXPORT int MSB_FN(msb_flash_attn_bwd_strided)(const void* q, const void* k, const void* v, const void* o,
                                          const void* dout, const float* lse, float* stats, void* dq, void* dk,
                                          void* dv, int B, int S, int H, int Hk, int D, long long q_pitch,
                                          long long k_pitch, long long v_pitch, long long o_pitch, long long do_pitch,
                                          long long dq_pitch, long long dkv_pitch, int causal, float scale,
                                          void* stream) {
  return fa_bwd_impl(q, k, v, o, dout, lse, stats, dq, dk, dv, B, S, H, Hk, D, q_pitch, k_pitch, v_pitch, o_pitch,
                     do_pitch, dq_pitch, dkv_pitch, causal, scale, stream);
}
