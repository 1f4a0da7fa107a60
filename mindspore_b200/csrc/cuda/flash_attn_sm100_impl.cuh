// FlashAttention forward for sm_100a (head_dim 128, bf16, causal or full), tcgen05 + TMEM + TMA.
//
// Tensors are token-major: q[b][s][h][d], k/v[b][s][hk][d], o[b][s][h][d]; row pitches are parameters so
// q/k/v may be column slices of one fused QKV GEMM output.  One work item = (batch, head, 256 query rows): two
// tiles of 128 rows that share every K and V tile.
//
// Persistent CTA, 384 threads (three warpgroups; the first gives most of its registers to the other two):
//   warp 0    : TMA producer  (both Q tiles once per item; K and V tiles of 128 keys through one ring of four)
//   warp 1    : MMA issuer    per key block and tile: O_t += P_t V, then S_t = Q_t K^T of the next block
//   warps 2-3 : idle
//   warps 4-7 : softmax of tile 0, warps 8-11 : softmax of tile 1.  Thread t owns query row t of its tile: reads its S
//                             row from TMEM (no shuffles), keeps the running max / sum, writes P (16-bit) back into
//                             the first 64 columns of the S row it came from, where the P V product reads it as its
//                             TMEM operand; rescales O in TMEM only when the row max grew by more than 2^8
//                             (warp-uniform decision), and finally normalises and stores O and LSE.
// TMEM: S0 / P0 [0,128)  S1 / P1 [128,256)  O0 [256,384)  O1 [384,512).
//
// Why this split.  The exponentials (16 per cycle per SM: 1024 cycles per 128 x 128 tile) and the two products of a
// tile (1024 cycles) take equally long, so they have to run at the same time: while one tile's softmax runs, the
// tensor core works for the other tile.  One tile per CTA with P going through shared memory (the earlier form of this
// kernel) left the tensor pipe idle for two thirds of the time.  All products of a CTA are issued by one thread and
// execute in issue order, which is what orders "S_t of the next block overwrites P_t" behind "P_t V has read it".
//
// Measured, 2 x 4096 tokens x 32 heads, bf16: causal 0.41 -> 0.27 ms (1030 TFLOP/s), full 0.74 -> 0.49 ms (1124); 0.35 and
// 0.58 ms while a lone lane issued the products (see elect_one).  What bounds it now are the products: with the softmax's
// arithmetic left out the full case still takes 0.43 ms.  Q K^T reads 8 KB of shared memory per 64 cycles, all that an SM
// can, and the TMA's writes come on top.  Moving a quarter to a half of the exponentials to the FMA pipe (degree-5
// polynomial) cost 5 to 11 %, handing the first half of P to the tensor core early 7 %.
//
// The reference defines FlashAttentionScore (core/ops/ops_def/flash_attention_score_op.yaml) but ships no GPU
// kernel for it; its GPU path would be BatchMatMul + Softmax + BatchMatMul through cuBLAS/cuDNN.
//
// This text is compiled twice: for bf16 tensors (flash_attn_sm100.cu), and with MSB_ELEM_FP16 defined for fp16 tensors
// (flash_attn_sm100_fp16.cu), where every entry point carries the suffix _fp16 and "bf16" in a comment reads "fp16".
#include "fa_common.cuh"

namespace msb {
namespace MSB_ELEM_NS {

constexpr int kFaBM = 128;       // query rows per tile
constexpr int kFaBN = 128;       // keys per block
constexpr int kFaThreads = 384;
constexpr int kFaRing = 4;       // K / V tiles in flight
constexpr int kTileBytes = 128 * 128 * 2;  // 32 KB: one 128x128 bf16 tile (two 128B-swizzled halves)

struct FaParams {
  elem_t* o;
  float* lse;          // [B][H][S] natural-log sum-exp of scaled scores
  int* status;
  long long o_pitch;   // elements between consecutive tokens of o
  int B, H, Hk, S;
  int causal;
  float scale_log2;    // softmax scale * log2(e)
  float scale;
};

// shared memory map (1024B aligned): Q0 32K | Q1 32K | ring of four 32K tiles | barriers
struct FaSmem {
  static constexpr int kQ = 0;
  static constexpr int kRing = 2 * kTileBytes;
  static constexpr int kBar = (2 + kFaRing) * kTileBytes;
  static constexpr int kBytes = kBar + 256 + 1024;
};

// Work item -> (batch, head, pair of query tiles, key blocks of each tile).  n1 is 0 when the second tile lies beyond
// the sequence.
struct FaItem {
  int b, h, qb, n0, n1;
};
__device__ __forceinline__ FaItem fa_item(int w, const FaParams& p, int nq2, int nk) {
  FaItem it;
  const int bh = p.B * p.H;
  it.qb = nq2 - 1 - w / bh;     // longest (latest) query blocks first
  const int r = w % bh;
  it.b = r / p.H;
  it.h = r % p.H;
  const bool second = it.qb * 256 + 128 < p.S;
  it.n0 = p.causal ? 2 * it.qb + 1 : nk;
  it.n1 = second ? (p.causal ? 2 * it.qb + 2 : nk) : 0;
  return it;
}

__global__ void __launch_bounds__(kFaThreads, 1)
flash_fwd_kernel(const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ CUtensorMap tmK,
                 const __grid_constant__ CUtensorMap tmV, const FaParams p) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + FaSmem::kBar);
  uint64_t* q_full = bars + 0;    // [2]
  uint64_t* q_empty = bars + 2;   // [2]
  uint64_t* r_full = bars + 4;    // [kFaRing]
  uint64_t* r_empty = bars + 8;   // [kFaRing]
  uint64_t* s_full = bars + 12;   // [2]
  uint64_t* p_ready = bars + 14;  // [2]
  uint64_t* o_full = bars + 16;   // [2]
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 18);
  volatile int* cta_abort = reinterpret_cast<volatile int*>(tmem_slot + 1);

  const int warp = uniform_warp(), lane = threadIdx.x & 31;
  const AbortCtx ab{cta_abort, p.status};
  const int nq2 = (p.S + 2 * kFaBM - 1) / (2 * kFaBM);
  const int nk = (p.S + kFaBN - 1) / kFaBN;
  const int total = p.B * p.H * nq2;
  const int group = p.H / p.Hk;

  if (threadIdx.x == 0) {
    for (int i = 0; i < 2; ++i) {
      mbar_init(&q_full[i], 1);
      mbar_init(&q_empty[i], 1);
      mbar_init(&s_full[i], 1);
      mbar_init(&p_ready[i], 4);
      mbar_init(&o_full[i], 1);
    }
    for (int i = 0; i < kFaRing; ++i) {
      mbar_init(&r_full[i], 1);
      mbar_init(&r_empty[i], 1);
    }
    *cta_abort = 0;
    fence_mbar_init();
    tma_prefetch_desc(&tmQ);
    tma_prefetch_desc(&tmK);
    tma_prefetch_desc(&tmV);
  }
  if (warp == 1) {
    tmem_alloc(tmem_slot, 512);
    tmem_relinquish();
  }
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tmem_base = __shfl_sync(0xffffffffu, *tmem_slot, 0);

  // registers: 384 threads x 168 at launch = 128 x 88 + 256 x 208 (the MMA thread spills below 88)
  if (warp < 4) {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 88;");
    if (warp == 0 && lane == 0) {
      // ------------------------------------------------------------------ TMA producer
      uint32_t qc[2] = {0, 0}, rc = 0;
      bool ok = true;
      auto load_q = [&](const FaItem& it, int t) -> bool {
        if (!mbar_wait(&q_empty[t], (qc[t] & 1) ^ 1, ab)) return false;
        ++qc[t];
        mbar_expect_tx(&q_full[t], kTileBytes);
        fa_load_tile(smem + FaSmem::kQ + t * kTileBytes, &tmQ, &q_full[t], 128, it.h, it.qb * 256 + t * 128, it.b);
        return true;
      };
      auto load_kv = [&](const CUtensorMap* tm, int hk, int j, int b) -> bool {
        const int st = rc & (kFaRing - 1);
        if (!mbar_wait(&r_empty[st], ((rc / kFaRing) & 1) ^ 1, ab)) return false;
        mbar_expect_tx(&r_full[st], kTileBytes);
        fa_load_tile(smem + FaSmem::kRing + st * kTileBytes, tm, &r_full[st], 128, hk, j * kFaBN, b);
        ++rc;
        return true;
      };
      for (int round = 0, w; ok && (w = fa_snake(round)) < total; ++round) {
        const FaItem it = fa_item(w, p, nq2, nk);
        const int hk = it.h / group, n = it.n1 > it.n0 ? it.n1 : it.n0;
        ok = load_q(it, 0) && load_kv(&tmK, hk, 0, it.b) && (it.n1 == 0 || load_q(it, 1)) &&
             load_kv(&tmV, hk, 0, it.b);
        for (int j = 1; j < n && ok; ++j) ok = load_kv(&tmK, hk, j, it.b) && load_kv(&tmV, hk, j, it.b);
      }
    } else if (warp == 1) {
      // ------------------------------------------------------------------ MMA issuer (the whole warp, one elected lane)
      constexpr uint32_t idesc_qk = umma_idesc_elem(128, 128, false, false);
      constexpr uint32_t idesc_pv = umma_idesc_elem(128, 128, false, true);   // V is MN-major (d contiguous)
      const uint32_t lead = elect_one();
      uint32_t base = 0;              // ring index of K of block 0 of the item; K_j at base + 2j, V_j at base + 2j + 1
      uint32_t qc[2] = {0, 0}, pc[2] = {0, 0};
      const uint64_t q_desc = umma_smem_desc(smem_u32(smem + FaSmem::kQ), 16, 1024);
      const uint64_t k_desc = umma_smem_desc(smem_u32(smem + FaSmem::kRing), 16, 1024);
      const uint64_t v_desc = umma_smem_desc(smem_u32(smem + FaSmem::kRing), 16384, 1024);
      auto wait_ring = [&](uint32_t i) -> bool {
        const bool r = mbar_wait_warp(&r_full[i & (kFaRing - 1)], (i / kFaRing) & 1, ab);
        tc_fence_after_sync();
        return r;
      };
      auto issue_qk = [&](int t, uint32_t ki) {
        const uint64_t qd = q_desc + t * (kTileBytes >> 4), kd = k_desc + (ki & (kFaRing - 1)) * (kTileBytes >> 4);
        if (lead) {
#pragma unroll
          for (int kk = 0; kk < kFaD / 16; ++kk) {
            const uint32_t off = ((kk >> 2) * 16384 + (kk & 3) * 32) >> 4;
            umma_bf16(tmem_base + t * 128, qd + off, kd + off, idesc_qk, kk != 0);
          }
          umma_commit(&s_full[t]);
        }
        __syncwarp();
      };
      auto issue_pv = [&](int t, uint32_t vi, bool first) {
        const uint64_t vd = v_desc + (vi & (kFaRing - 1)) * (kTileBytes >> 4);
        if (lead) {
#pragma unroll
          for (int kk = 0; kk < kFaBN / 16; ++kk)
            umma_ts(tmem_base + 256 + t * 128, tmem_base + t * 128 + kk * 8, vd + ((kk * 2048) >> 4), idesc_pv,
                    !(first && kk == 0));
        }
        __syncwarp();
      };
      auto commit = [&](uint64_t* bar) {
        if (lead) umma_commit(bar);
        __syncwarp();
      };
      bool ok = true;
      for (int round = 0, w; ok && (w = fa_snake(round)) < total; ++round) {
        const FaItem it = fa_item(w, p, nq2, nk);
        const int n = it.n1 > it.n0 ? it.n1 : it.n0;
        const int cnt[2] = {it.n0, it.n1};
        ok = wait_ring(base);
#pragma unroll
        for (int t = 0; t < 2; ++t) {
          if (!ok || cnt[t] == 0) continue;
          if (!(ok = mbar_wait_warp(&q_full[t], qc[t] & 1, ab))) break;
          ++qc[t];
          tc_fence_after_sync();
          issue_qk(t, base);
          if (cnt[t] == 1) commit(&q_empty[t]);
        }
        if (ok) commit(&r_empty[base & (kFaRing - 1)]);
        for (int j = 0; j < n && ok; ++j) {
          const uint32_t vi = base + 2 * j + 1, ki = base + 2 * j + 2;
          const int last = j < it.n1 ? 1 : 0;          // the last tile that reads V_j
#pragma unroll
          for (int t = 0; t < 2; ++t) {
            if (!ok || j >= cnt[t]) continue;
            if (!(ok = wait_ring(vi))) break;
            if (!(ok = mbar_wait_warp(&p_ready[t], pc[t] & 1, ab))) break;
            ++pc[t];
            tc_fence_after_sync();
            issue_pv(t, vi, j == 0);
            if (t == last) commit(&r_empty[vi & (kFaRing - 1)]);
            if (j + 1 == cnt[t]) commit(&o_full[t]);
            if (j + 1 < cnt[t]) {
              if (!(ok = wait_ring(ki))) break;
              issue_qk(t, ki);
              // the last tile that reads K_{j+1} releases it; the last product with Q_t releases Q_t
              if (t == (j + 1 < it.n1 ? 1 : 0)) commit(&r_empty[ki & (kFaRing - 1)]);
              if (j + 2 == cnt[t]) commit(&q_empty[t]);
            }
          }
        }
        base += 2 * n;
      }
    }
    __syncwarp();
  } else {
    asm volatile("setmaxnreg.inc.sync.aligned.u32 208;");
    // -------------------------------------------------------------------- softmax / correction / epilogue
    const int t = (warp >> 2) - 1;                 // tile
    const int q = warp & 3;
    const int row = q * 32 + lane;                 // row inside the 128-row tile == TMEM lane
    const uint32_t lane_sel = static_cast<uint32_t>(q * 32) << 16;
    const uint32_t tm_s = tmem_base + t * 128 + lane_sel;
    const uint32_t tm_o = tmem_base + 256 + t * 128 + lane_sel;
    uint32_t sc = 0, oc = 0;
    bool ok = true;
    for (int round = 0, w; ok && (w = fa_snake(round)) < total; ++round) {
      const FaItem it = fa_item(w, p, nq2, nk);
      const int nblk = t == 0 ? it.n0 : it.n1;
      if (nblk == 0) continue;
      const int tile = it.qb * 2 + t;
      float m_used = -INFINITY;   // max the stored probabilities are relative to (log2 domain)
      float l = 0.f;
      for (int j = 0; j < nblk; ++j, ++sc) {
        if (!mbar_wait(&s_full[t], sc & 1, ab)) { ok = false; break; }
        tc_fence_after_sync();
        // raw scores; the softmax scale is folded into the exponent below (one FFMA per element)
        uint32_t s[4][32];
#pragma unroll
        for (int c = 0; c < 4; ++c) tmem_ld_32x32(tm_s + c * 32, s[c]);
        tmem_ld_wait();
        // keys this row may see in this block: the diagonal block is cut after the row's own key, the last block of a
        // ragged sequence after the sequence's last key
        int limit = p.S - j * kFaBN;
        if (p.causal && j == tile) limit = min(limit, row + 1);
        if ((p.causal && j == tile) || (j + 1) * kFaBN > p.S) {
#pragma unroll
          for (int i = 0; i < 128; ++i)
            if (i >= limit) s[i >> 5][i & 31] = __float_as_uint(-INFINITY);
        }
        float mx4[4];
#pragma unroll
        for (int c = 0; c < 4; ++c) {
          mx4[c] = fmaxf(__uint_as_float(s[c][0]), __uint_as_float(s[c][1]));
#pragma unroll
          for (int i = 2; i < 32; i += 2)
            mx4[c] = fmaxf(fmaxf(mx4[c], __uint_as_float(s[c][i])), __uint_as_float(s[c][i + 1]));
        }
        const float mx = fmaxf(fmaxf(mx4[0], mx4[1]), fmaxf(mx4[2], mx4[3])) * p.scale_log2;   // scale > 0
        // rescale only when some row of this warp grew its max by more than 8 (in log2 units)
        const bool grow = mx > m_used + 8.f;
        if (__any_sync(0xffffffffu, grow)) {
          const float m_new = fmaxf(m_used, mx);
          const float alpha = (m_used == -INFINITY) ? 0.f : ex2(m_used - m_new);
          m_used = m_new;
          l *= alpha;
          // S of this block was issued behind P V of the previous one: O is complete and nobody else touches it
          if (j > 0) {
#pragma unroll 1
            for (int c = 0; c < 4; ++c) {
              uint32_t r[32];
              tmem_ld_32x32(tm_o + c * 32, r);
              tmem_ld_wait();
#pragma unroll
              for (int i = 0; i < 32; ++i) r[i] = __float_as_uint(__uint_as_float(r[i]) * alpha);
              tmem_st_32x32(tm_o + c * 32, r);
            }
          }
        }
        const uint64_t scale2 = f32x2(p.scale_log2, p.scale_log2), neg_m2 = f32x2(-m_used, -m_used);
        uint64_t rs[4] = {0, 0, 0, 0};
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          // pairs 2i, 2i + 1 become word i of the same register array: nothing else is needed to hold P
#pragma unroll
          for (int i = h * 32; i < h * 32 + 32; ++i) {
            const uint32_t* e = &s[i >> 4][(2 * i) & 31];
            float a, b;
            f32x2_split(fma2(f32x2(__uint_as_float(e[0]), __uint_as_float(e[1])), scale2, neg_m2), a, b);
            a = ex2(a);
            b = ex2(b);
            rs[i & 3] = add2(rs[i & 3], f32x2(a, b));
            s[h][i & 31] = pack_e2(a, b);
          }
          tmem_st_32x32(tm_s + h * 32, s[h]);
        }
        tmem_st_wait();
        tc_fence_before_sync();
        warp_arrive(&p_ready[t], lane);
        float a, b;
        f32x2_split(add2(add2(rs[0], rs[1]), add2(rs[2], rs[3])), a, b);
        l += a + b;
      }
      if (!ok) break;
      // ---- epilogue: O / l -> global, LSE.  The next write to O comes behind this thread's next p_ready.
      if (!mbar_wait(&o_full[t], oc & 1, ab)) { ok = false; break; }
      ++oc;
      tc_fence_after_sync();
      const float inv_l = 1.f / l;
      const int qrow = tile * kFaBM + row;
      const bool live = qrow < p.S;
      elem_t* orow = p.o + (static_cast<long long>(it.b) * p.S + qrow) * p.o_pitch + static_cast<long long>(it.h) * kFaD;
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        uint32_t r[32];
        tmem_ld_32x32(tm_o + c * 32, r);
        tmem_ld_wait();
        if (live) {
#pragma unroll
          for (int i = 0; i < 32; i += 8) {
            uint4 v;
            v.x = pack_e2(__uint_as_float(r[i + 0]) * inv_l, __uint_as_float(r[i + 1]) * inv_l);
            v.y = pack_e2(__uint_as_float(r[i + 2]) * inv_l, __uint_as_float(r[i + 3]) * inv_l);
            v.z = pack_e2(__uint_as_float(r[i + 4]) * inv_l, __uint_as_float(r[i + 5]) * inv_l);
            v.w = pack_e2(__uint_as_float(r[i + 6]) * inv_l, __uint_as_float(r[i + 7]) * inv_l);
            *reinterpret_cast<uint4*>(orow + c * 32 + i) = v;
          }
        }
      }
      tc_fence_before_sync();
      if (p.lse && live) {
        p.lse[(static_cast<long long>(it.b) * p.H + it.h) * p.S + qrow] =
            (m_used + log2f(l)) * 0.6931471805599453f;
      }
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

}  // namespace MSB_ELEM_NS
}  // namespace msb

using namespace msb;
using namespace msb::MSB_ELEM_NS;

// q [B,S,H,128], k/v [B,S,Hk,128] with token pitches (elements) q_pitch / k_pitch / v_pitch; o [B,S,H,128] with o_pitch.
// lse (fp32 [B,H,S]) may be null.
MSB_EXPORT int MSB_FN(msb_flash_attn_fwd)(const void* q, const void* k, const void* v, void* o, float* lse, int B, int S,
                                  int H, int Hk, int D, long long q_pitch, long long k_pitch, long long v_pitch,
                                  long long o_pitch,
                                  int causal, float scale, void* stream_) {
  if (D != kFaD || S <= 0 || Hk <= 0 || H % Hk != 0 || B <= 0) {
    set_last_error("flash_attn_fwd: needs head_dim 128 and H a multiple of Hk "
                   "(got D=%d S=%d H=%d Hk=%d)", D, S, H, Hk);
    return kBadArg;
  }
  if (o_pitch % 8) {
    set_last_error("flash_attn_fwd: o_pitch must be a multiple of 8");
    return kBadArg;
  }
  int* status = status_ptr();
  if (!status) { set_last_error("flash_attn_fwd: no status word"); return kCudaError; }
  CUtensorMap tq, tk, tv;
  int rc;
  if ((rc = fa_encode_map(&tq, q, B, S, H, q_pitch, 128)) != kOk) return rc;
  if ((rc = fa_encode_map(&tk, k, B, S, Hk, k_pitch, 128)) != kOk) return rc;
  if ((rc = fa_encode_map(&tv, v, B, S, Hk, v_pitch, 128)) != kOk) return rc;
  static bool configured = false;
  if (!configured) {
    MSB_CUDA_CHECK(cudaFuncSetAttribute(flash_fwd_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                        FaSmem::kBytes));
    configured = true;
  }
  FaParams p;
  p.o = static_cast<elem_t*>(o);
  p.lse = lse;
  p.status = status;
  p.o_pitch = o_pitch;
  p.B = B; p.H = H; p.Hk = Hk; p.S = S;
  p.causal = causal;
  p.scale = scale;
  p.scale_log2 = scale * 1.4426950408889634f;
  const int total = B * H * ((S + 255) / 256);
  const int grid = total < sm_count() ? total : sm_count();
  flash_fwd_kernel<<<grid, kFaThreads, FaSmem::kBytes, static_cast<cudaStream_t>(stream_)>>>(tq, tk, tv, p);
  MSB_CUDA_CHECK(cudaGetLastError());
  return kOk;
}
