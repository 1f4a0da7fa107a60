// NHWC bf16 convolution as an implicit GEMM on tcgen05: no im2col matrix is ever written.
//
// Forward / data gradient (WGRAD = false):  Y[pix, co] = sum_{tap, ci} X[pix + offset(tap), ci] * W[co, tap, ci]
//   GEMM M = output pixels, N = output channels, K = taps * Cin.  A tile of 128 output pixels is a box
//   (tw x th x tn) of the output grid; for filter tap t and channel block c the A operand of that k-block is one
//   4-D TMA load of the input at (c, w0 + dw[t], h0 + dh[t], n0): 128 rows of 64 channels, 128-byte swizzled, i.e.
//   exactly the K-major tile the MMA wants.  Padding is the TMA's out-of-bounds zero fill.  Strided convolutions
//   read one of up to four "parity planes" of the input (views with doubled W/H strides), chosen per tap, so the
//   same box load applies.  The epilogue writes bf16 NHWC rows and can accumulate the per-channel sum and sum of
//   squares of the output in shared memory (flushed once per CTA) - the BatchNorm statistics come for free.
// Weight gradient (WGRAD = true):  dW[co, tap, ci] = sum_pix dY[pix, co] * X[pix + offset(tap), ci]
//   GEMM M = Cout, N = Cin, K = pixels; both operands are MN-major 4-D box loads (64 pixels x 64 channels), the
//   k-loop runs over pixel tiles and is split across CTAs (fp32 atomic accumulation into dW).  Whole blocks of 64 input
//   channels make N run over (tap, ci) together - the order of a row of dW -, so a tile of several narrow taps reads dY once.
//
// The reference calls cudnnConvolutionForward / BackwardData / BackwardFilter
// (plugin/device/gpu/kernel/nn/conv2d_gpu_kernel.h, conv2d_grad_input_gpu_kernel.h, conv2d_grad_filter_gpu_kernel.h)
// followed by a separate cuDNN BatchNorm pass over the output.
//
// This text is compiled twice: for bf16 tensors (conv_sm100.cu), and with MSB_ELEM_FP16 defined for fp16 tensors
// (conv_sm100_fp16.cu), where every entry point carries the suffix _fp16 and "bf16" in a comment reads "fp16".
#include "host_common.h"
#include "elem.cuh"

namespace msb {
namespace MSB_ELEM_NS {

constexpr int kConvBM = 128;
constexpr int kConvBK = 64;
constexpr int kConvThreads = 320;      // TMA warp, MMA warp, two epilogue groups of four warps
constexpr int kMaxTaps = 49;
constexpr int kMaxStatChannels = 2048;

struct ConvParams {
  void* C;
  float* stats;          // fwd: [2 * Cout] running sum / sum of squares of the bf16 output, or nullptr
  int* status;
  int N, Ho, Wo;         // pixel grid that the boxes tile (fwd: output pixels; wgrad: dY pixels)
  int tw, th, tn;        // box extents (product 128 fwd, 64 wgrad)
  int tiles_w, tiles_h, tiles_n;
  int cin_blocks;        // fwd: Cin / 64
  int taps;
  int Cout, Cin;
  long long ldc;         // fwd: elements between output pixels; wgrad: elements between rows of dW
  int out_fp32, accumulate, ksplit;
  int flat;              // wgrad: the columns of the GEMM run over (tap, ci); 0: over ci, one tap per tile
  // 1: output tiles go through swizzled shared memory and leave as TMA stores (wgrad: TMA reduce-adds); 0: per-thread
  // stores / atomics, for fp32 forward outputs, channel counts and pitches that the tensor map cannot describe
  int tma_out;
  short tap_map[kMaxTaps], tap_dh[kMaxTaps], tap_dw[kMaxTaps];
};

__device__ __forceinline__ void tma_load_4d(void* smem_dst, const CUtensorMap* tmap, uint64_t* bar, int c, int w,
                                            int h, int n) {
  asm volatile(
      "cp.async.bulk.tensor.4d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5, %6}], [%2];"
      ::"r"(smem_u32(smem_dst)), "l"(reinterpret_cast<uint64_t>(tmap)), "r"(smem_u32(bar)), "r"(c), "r"(w), "r"(h),
      "r"(n)
      : "memory");
}

template <int BN>
struct ConvCfg {
  static constexpr int kStages = (BN == 256) ? 3 : (BN == 192) ? 4 : (BN == 128) ? 5 : 7;
  static constexpr int kTmemCols = (BN == 192) ? 512 : 2 * BN;      // a power of two
  static constexpr int kABytes = kConvBM * kConvBK * 2;
  static constexpr int kBBytes = BN * kConvBK * 2;
  static constexpr int kStageBytes = kABytes + kBBytes;
  // epilogue staging: 8 warps x (32 rows x 128 B), 1024-byte aligned behind the stage ring
  static constexpr int kStagingOffset = kStages * kStageBytes;
  static constexpr int kBarOffset = kStagingOffset + 8 * 4096;
  static constexpr int kStatOffset = kBarOffset + 256;
  static constexpr int kSmemBytes = kStatOffset + 2 * kMaxStatChannels * 4 + 1024;
};

__device__ __forceinline__ void tma_store_4d(const CUtensorMap* tmap, const void* smem_src, int c, int w, int h, int n) {
  asm volatile("cp.async.bulk.tensor.4d.global.shared::cta.bulk_group [%0, {%2, %3, %4, %5}], [%1];" ::"l"(
                   reinterpret_cast<uint64_t>(tmap)),
               "r"(smem_u32(smem_src)), "r"(c), "r"(w), "r"(h), "r"(n)
               : "memory");
}
__device__ __forceinline__ void tma_reduce_add_3d(const CUtensorMap* tmap, const void* smem_src, int x, int y, int z) {
  asm volatile("cp.reduce.async.bulk.tensor.3d.global.shared::cta.add.tile.bulk_group [%0, {%2, %3, %4}], [%1];" ::"l"(
                   reinterpret_cast<uint64_t>(tmap)),
               "r"(smem_u32(smem_src)), "r"(x), "r"(y), "r"(z)
               : "memory");
}

// B_MN: B is read MN-major (always in the weight gradient; in the data gradient, whose weights are [k, tap, n]).
template <int BN, bool WGRAD, bool B_MN>
__global__ void __launch_bounds__(kConvThreads, 1)
conv_igemm_kernel(const __grid_constant__ CUtensorMap tmX0, const __grid_constant__ CUtensorMap tmX1,
                  const __grid_constant__ CUtensorMap tmX2, const __grid_constant__ CUtensorMap tmX3,
                  const __grid_constant__ CUtensorMap tmO, const __grid_constant__ CUtensorMap tmY, const ConvParams p) {
  // tmX*: input activations (parity planes).  tmO: fwd = weights [Cout, taps*Cin] (3-D map, K-major);
  // wgrad = dY (4-D map).  tmY: the output (fwd 4-D, boxes of 64 channels x 32 pixels; wgrad dW as a matrix, boxes of
  // 32 x 32), valid when p.tma_out.
  using Cfg = ConvCfg<BN>;
  constexpr int kStages = Cfg::kStages;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* smem_a = smem;
  uint8_t* smem_b = smem + kStages * Cfg::kABytes;
  uint64_t* full_bar = reinterpret_cast<uint64_t*>(smem + Cfg::kBarOffset);
  uint64_t* empty_bar = full_bar + kStages;
  uint64_t* tfull_bar = empty_bar + kStages;
  uint64_t* tempty_bar = tfull_bar + 2;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(tempty_bar + 2);
  volatile int* cta_abort = reinterpret_cast<volatile int*>(tmem_slot + 1);
  volatile int* issued_cnt = cta_abort + 1;
  volatile int* consumed_cnt = cta_abort + 2;
  float* s_stats = reinterpret_cast<float*>(smem + Cfg::kStatOffset);

  const int warp = uniform_warp();
  const int lane = threadIdx.x & 31;
  const AbortCtx ab{cta_abort, p.status};
  const CUtensorMap* maps[4] = {&tmX0, &tmX1, &tmX2, &tmX3};

  const int pix_tiles = p.tiles_w * p.tiles_h * p.tiles_n;
  // GEMM tiling
  const int gemm_m = WGRAD ? p.Cout : 0;
  const int tiles_m = WGRAD ? (gemm_m + kConvBM - 1) / kConvBM : pix_tiles;
  const int gemm_n = WGRAD ? (p.flat ? p.taps * p.Cin : p.Cin) : p.Cout;
  const int tiles_n = (gemm_n + BN - 1) / BN;
  const int outer = WGRAD ? (p.flat ? 1 : p.taps) * p.ksplit : 1;
  const int total_tiles = tiles_m * tiles_n * outer;
  const int kb_total = WGRAD ? pix_tiles : p.taps * p.cin_blocks;
  const int kb_per = WGRAD ? (kb_total + p.ksplit - 1) / p.ksplit : kb_total;
  const bool want_stats = !WGRAD && p.stats != nullptr;

  if (threadIdx.x == 0) {
    for (int s = 0; s < kStages; ++s) {
      mbar_init(&full_bar[s], 1);
      mbar_init(&empty_bar[s], 1);
    }
    mbar_init(&tfull_bar[0], 1);
    mbar_init(&tfull_bar[1], 1);
    mbar_init(&tempty_bar[0], 128);
    mbar_init(&tempty_bar[1], 128);
    *cta_abort = 0;
    *issued_cnt = 0;
    *consumed_cnt = 0;
    fence_mbar_init();
    tma_prefetch_desc(&tmX0);
    tma_prefetch_desc(&tmO);
  }
  if (want_stats)
    for (int i = threadIdx.x; i < 2 * p.Cout; i += kConvThreads) s_stats[i] = 0.f;
  if (warp == 1) {
    tmem_alloc(tmem_slot, Cfg::kTmemCols);
    tmem_relinquish();
  }
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tmem_base = __shfl_sync(0xffffffffu, *tmem_slot, 0);

  // tile -> (outer index, m block, n block); m fastest so that CTAs running together share the weight tile
  auto tile_coords = [&](int tile, int& o, int& m_blk, int& n_blk) {
    o = tile / (tiles_m * tiles_n);
    const int t = tile - o * tiles_m * tiles_n;
    m_blk = t % tiles_m;
    n_blk = t / tiles_m;
  };
  auto pixel_origin = [&](int pt, int& n0, int& h0, int& w0) {
    const int iw = pt % p.tiles_w;
    const int ih = (pt / p.tiles_w) % p.tiles_h;
    const int in_ = pt / (p.tiles_w * p.tiles_h);
    n0 = in_ * p.tn;
    h0 = ih * p.th;
    w0 = iw * p.tw;
  };
  auto k_range = [&](int o, int& kb_lo, int& kb_hi) {
    if (WGRAD) {
      const int split = o % p.ksplit;
      kb_lo = split * kb_per;
      kb_hi = min(kb_lo + kb_per, kb_total);
    } else {
      kb_lo = 0;
      kb_hi = kb_total;
    }
  };

  if (warp == 0) {
    if (lane == 0) {
      // ------------------------------------------------------------------ TMA producer
      int s = 0;
      uint32_t ph = 0;
      int issued = 0;
      bool ok = true;
      for (int tile = blockIdx.x; tile < total_tiles && ok; tile += gridDim.x) {
        int o, m_blk, n_blk, kb_lo, kb_hi;
        tile_coords(tile, o, m_blk, n_blk);
        k_range(o, kb_lo, kb_hi);
        const int nc0 = n_blk * BN;
        int n0 = 0, h0 = 0, w0 = 0;
        if (!WGRAD) pixel_origin(m_blk, n0, h0, w0);
        // wgrad: where each 64-column block of B comes from, and how many blocks there are; what lies beyond the matrix is
        // not loaded (its rows and columns of the product are not stored either)
        const CUtensorMap* bx[BN / 64];
        int bc[BN / 64], bh[BN / 64], bw[BN / 64], a_blocks = 2, b_blocks = BN / 64;
        if (B_MN) b_blocks = min(BN / 64, (gemm_n - nc0 + 63) / 64);
        if (WGRAD) {
          a_blocks = min(2, (p.Cout - m_blk * kConvBM + 63) / 64);
#pragma unroll
          for (int j = 0; j < BN / 64; ++j) {
            const int col = min(nc0 + 64 * j, gemm_n - 1);
            const int tap = p.flat ? col / p.Cin : o / p.ksplit;
            bx[j] = maps[p.tap_map[tap]];
            bc[j] = p.flat ? col - tap * p.Cin : col;
            bh[j] = p.tap_dh[tap];
            bw[j] = p.tap_dw[tap];
          }
        }
        const int stage_bytes = (a_blocks + b_blocks) * 8192;
        for (int kb = kb_lo; kb < kb_hi; ++kb) {
          if (!mbar_wait(&empty_bar[s], ph ^ 1, ab)) { ok = false; break; }
          mbar_expect_tx(&full_bar[s], stage_bytes);
          uint8_t* a_dst = smem_a + s * Cfg::kABytes;
          uint8_t* b_dst = smem_b + s * Cfg::kBBytes;
          if (WGRAD) {
            pixel_origin(kb, n0, h0, w0);
            const int m0 = m_blk * kConvBM;
#pragma unroll
            for (int j = 0; j < kConvBM / 64; ++j)
              if (j < a_blocks) tma_load_4d(a_dst + j * 8192, &tmO, &full_bar[s], m0 + 64 * j, w0, h0, n0);
#pragma unroll
            for (int j = 0; j < BN / 64; ++j)
              if (j < b_blocks) tma_load_4d(b_dst + j * 8192, bx[j], &full_bar[s], bc[j], w0 + bw[j], h0 + bh[j], n0);
          } else {
            const int tap = kb / p.cin_blocks;
            const int cb = kb - tap * p.cin_blocks;
            tma_load_4d(a_dst, maps[p.tap_map[tap]], &full_bar[s], cb * 64, w0 + p.tap_dw[tap], h0 + p.tap_dh[tap],
                        n0);
            if (B_MN) {
#pragma unroll
              for (int j = 0; j < BN / 64; ++j)
                if (j < b_blocks)
                  tma_load_3d(b_dst + j * 8192, &tmO, &full_bar[s], tap * p.Cout + nc0 + 64 * j, cb * 64, 0);
            } else {
              tma_load_3d(b_dst, &tmO, &full_bar[s], kb * kConvBK, nc0, 0);
            }
          }
          ++issued;
          *issued_cnt = issued;
          if (++s == kStages) { s = 0; ph ^= 1; }
        }
      }
    }
    __syncwarp();
  } else if (warp == 1) {
    // -------------------------------------------------------------------- MMA issuer (whole warp, one elected lane)
    constexpr uint32_t idesc = umma_idesc_elem(kConvBM, BN, WGRAD, B_MN);
    const uint32_t lead = elect_one();
    const uint64_t a_desc = umma_smem_desc(smem_u32(smem_a), WGRAD ? 8192 : 16, 1024);
    const uint64_t b_desc = umma_smem_desc(smem_u32(smem_b), B_MN ? 8192 : 16, 1024);
    int s = 0;
    uint32_t ph = 0;
    int it = 0;
    int consumed = 0;
    bool ok = true;
    for (int tile = blockIdx.x; tile < total_tiles && ok; tile += gridDim.x, ++it) {
      int o, m_blk, n_blk, kb_lo, kb_hi;
      tile_coords(tile, o, m_blk, n_blk);
      k_range(o, kb_lo, kb_hi);
      const int acc = it & 1;
      const uint32_t acc_ph = (it >> 1) & 1;
      if (!mbar_wait_warp(&tempty_bar[acc], acc_ph ^ 1, ab)) { ok = false; break; }
      tc_fence_after_sync();
      const uint32_t d_tmem = tmem_base + acc * BN;
      for (int kb = kb_lo; kb < kb_hi; ++kb) {
        if (!mbar_wait_warp(&full_bar[s], ph, ab)) { ok = false; break; }
        ++consumed;
        tc_fence_after_sync();
        const uint64_t ad = a_desc + s * (Cfg::kABytes >> 4), bd = b_desc + s * (Cfg::kBBytes >> 4);
        if (lead) {
          *consumed_cnt = consumed;
#pragma unroll
          for (int kk = 0; kk < kConvBK / 16; ++kk)
            umma_bf16(d_tmem, ad + kk * (WGRAD ? 128 : 2), bd + kk * (B_MN ? 128 : 2), idesc, (kb != kb_lo) || (kk != 0));
          umma_commit(&empty_bar[s]);
        }
        __syncwarp();
        if (++s == kStages) { s = 0; ph ^= 1; }
      }
      if (ok && lead) umma_commit(&tfull_bar[acc]);
      __syncwarp();
    }
    __syncwarp();
  } else {
    // -------------------------------------------------------------------- epilogue
    // Two groups of four warps take the tiles in turn, each on its own accumulator.  A 1x1 convolution of 256 channels
    // has about 2700 cycles per tile from HBM's side; one group with per-thread row stores needed four times that.
    // 64 x 56 x 56 pixels, 64 -> 256 and back: 64 -> 31 us each; weight gradients, whose tiles left as fp32 atomics of
    // single elements: 88 -> 29 us (1x1, 256 columns).
    const int q = warp & 3, grp = (warp - 2) >> 2;
    int it = grp;
    bool ok = true;
    uint8_t* staging = smem + Cfg::kStagingOffset + (warp - 2) * 4096;
    const int sw = lane & 7;
    uint8_t* rowp = staging + lane * 128;
    bool pending = false;
    auto staging_free = [&]() {           // the store that reads the staging buffer has read it
      if (pending) {
        if (lane == 0) tma_store_wait_read<0>();
        __syncwarp();
      }
      pending = true;
    };
    // statistics of this lane's two columns of every 64-column chunk, flushed when the column block changes
    float st[BN / 64][4];
#pragma unroll
    for (int c = 0; c < BN / 64; ++c)
#pragma unroll
      for (int j = 0; j < 4; ++j) st[c][j] = 0.f;
    int st_n0 = -1;
    auto flush_stats = [&]() {
#pragma unroll
      for (int c = 0; c < BN / 64; ++c) {
        const int col = st_n0 + c * 64 + lane * 2;
#pragma unroll
        for (int j = 0; j < 2; ++j) {
          if (col + j < p.Cout) {
            atomicAdd(&s_stats[col + j], st[c][j]);
            atomicAdd(&s_stats[p.Cout + col + j], st[c][2 + j]);
          }
          st[c][j] = st[c][2 + j] = 0.f;
        }
      }
    };
    for (int tile = blockIdx.x + grp * gridDim.x; tile < total_tiles && ok; tile += 2 * gridDim.x, it += 2) {
      int o, m_blk, n_blk, kb_lo, kb_hi;
      tile_coords(tile, o, m_blk, n_blk);
      k_range(o, kb_lo, kb_hi);
      const int acc = it & 1;
      const uint32_t acc_ph = (it >> 1) & 1;
      if (!mbar_wait(&tfull_bar[acc], acc_ph, ab)) { ok = false; break; }
      tc_fence_after_sync();
      const int r = q * 32 + lane;
      const int nc0 = n_blk * BN;
      const uint32_t t_row = tmem_base + acc * BN + (static_cast<uint32_t>(q * 32) << 16);
      bool row_ok;
      long long c_off;
      int bw0 = 0, bh0 = 0, bn0 = 0;       // origin of this warp's 32 pixels
      if (WGRAD) {
        const int co = m_blk * kConvBM + r;
        row_ok = co < p.Cout && kb_lo < kb_hi;
        c_off = static_cast<long long>(co) * p.ldc + static_cast<long long>(o / p.ksplit) * p.Cin;
      } else {
        int n0, h0, w0;
        pixel_origin(m_blk, n0, h0, w0);
        const int n = n0 + r / (p.tw * p.th), h = h0 + (r / p.tw) % p.th, w = w0 + r % p.tw;
        row_ok = n < p.N && h < p.Ho && w < p.Wo;
        c_off = ((static_cast<long long>(n) * p.Ho + h) * p.Wo + w) * p.ldc;
        const int r0 = q * 32;
        bn0 = n0 + r0 / (p.tw * p.th);
        bh0 = h0 + (r0 / p.tw) % p.th;
        bw0 = w0 + r0 % p.tw;
      }
      if (!WGRAD && p.tma_out) {
        if (want_stats && st_n0 != nc0) {
          if (st_n0 >= 0) flush_stats();
          st_n0 = nc0;
        }
        const bool box_ok = bn0 < p.N && bh0 < p.Ho && bw0 < p.Wo;
#pragma unroll
        for (int c = 0; c < BN / 64; ++c) {
          const int col0 = nc0 + c * 64;
          if (col0 >= gemm_n) break;       // warp-uniform
          uint32_t rr[2][32];
          tmem_ld_32x32(t_row + c * 64, rr[0]);
          tmem_ld_32x32(t_row + c * 64 + 32, rr[1]);
          tmem_ld_wait();
          staging_free();
#pragma unroll
          for (int j = 0; j < 8; ++j) {
            const uint32_t* e = &rr[j >> 2][(j & 3) * 8];
            uint4 ov;
            ov.x = pack_e2(__uint_as_float(e[0]), __uint_as_float(e[1]));
            ov.y = pack_e2(__uint_as_float(e[2]), __uint_as_float(e[3]));
            ov.z = pack_e2(__uint_as_float(e[4]), __uint_as_float(e[5]));
            ov.w = pack_e2(__uint_as_float(e[6]), __uint_as_float(e[7]));
            if (!row_ok) ov = make_uint4(0, 0, 0, 0);
            *reinterpret_cast<uint4*>(rowp + ((j ^ sw) << 4)) = ov;
          }
          fence_proxy_async_smem();
          __syncwarp();
          if (lane == 0 && box_ok) {
            tma_store_4d(&tmY, staging, col0, bw0, bh0, bn0);
            tma_store_commit();
          }
          if (want_stats) {
            // of what was stored (the rounded values); rows outside the image contribute zero.  Lane l sums columns 2l and
            // 2l + 1 down the 32 staged rows: 32 conflict-free loads instead of 124 shuffles.
#pragma unroll 8
            for (int rw = 0; rw < 32; ++rw) {
              const float2 v = e2_to_f2(*reinterpret_cast<const elem2_t*>(staging + rw * 128 + (((lane >> 2) ^ (rw & 7)) << 4) +
                                                                         (lane & 3) * 4));
              st[c][0] += v.x;
              st[c][1] += v.y;
              st[c][2] += v.x * v.x;
              st[c][3] += v.y * v.y;
            }
            __syncwarp();
          }
        }
      } else if (WGRAD && p.tma_out) {
        const int row0 = m_blk * kConvBM + q * 32, x0 = (o / p.ksplit) * p.Cin;
        const bool box_ok = row0 < p.Cout && kb_lo < kb_hi;
#pragma unroll 1
        for (int c = 0; c < BN; c += 32) {
          if (nc0 + c >= gemm_n || !box_ok) break;     // warp-uniform
          uint32_t rr[32];
          tmem_ld_32x32(t_row + c, rr);
          tmem_ld_wait();
          staging_free();
#pragma unroll
          for (int j = 0; j < 8; ++j)
            *reinterpret_cast<uint4*>(rowp + ((j ^ sw) << 4)) = make_uint4(rr[4 * j], rr[4 * j + 1], rr[4 * j + 2],
                                                                           rr[4 * j + 3]);
          fence_proxy_async_smem();
          __syncwarp();
          if (lane == 0) {
            tma_reduce_add_3d(&tmY, staging, x0 + nc0 + c, row0, 0);
            tma_store_commit();
          }
        }
      } else {
#pragma unroll 1
        for (int c = 0; c < BN; c += 32) {
          if (nc0 + c >= gemm_n) break;  // warp-uniform
          uint32_t rr[32];
          tmem_ld_32x32(t_row + c, rr);
          tmem_ld_wait();
          const int col0 = nc0 + c;
          if (row_ok && (WGRAD || p.out_fp32)) {
            float* dst = static_cast<float*>(p.C) + c_off + col0;
            if (WGRAD && (p.ksplit > 1 || p.accumulate)) {
              for (int j = 0; j < 32; ++j)
                if (col0 + j < gemm_n) atomicAdd(dst + j, __uint_as_float(rr[j]));
            } else {
              for (int j = 0; j < 32; ++j)
                if (col0 + j < gemm_n) dst[j] = __uint_as_float(rr[j]);
            }
          } else if (row_ok) {
            elem_t* dst = static_cast<elem_t*>(p.C) + c_off + col0;
            for (int j = 0; j < 32; ++j) {
              if (col0 + j < gemm_n) {
                const elem_t e = f_to_e(__uint_as_float(rr[j]));
                dst[j] = e;
                if (want_stats) {
                  const float v = e_to_f(e);
                  atomicAdd(&s_stats[col0 + j], v);
                  atomicAdd(&s_stats[p.Cout + col0 + j], v * v);
                }
              }
            }
          }
          __syncwarp();
        }
      }
      tc_fence_before_sync();
      mbar_arrive(&tempty_bar[acc]);
    }
    if (want_stats && st_n0 >= 0) flush_stats();
    if (lane == 0) asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");
  }

  // ---------------------------------------------------------------------- teardown
  tc_fence_before_sync();
  __syncthreads();
  if (want_stats)
    for (int i = threadIdx.x; i < 2 * p.Cout; i += kConvThreads)
      if (s_stats[i] != 0.f) atomicAdd(p.stats + i, s_stats[i]);
  if (*cta_abort && threadIdx.x == 0) {
    const int issued = *issued_cnt, consumed = *consumed_cnt;
    for (int i = consumed; i < issued; ++i) {
      const int s = i % kStages;
      const uint32_t ph = (i / kStages) & 1;
      const unsigned long long t0 = globaltimer_ns();
      while (!mbar_try_wait(&full_bar[s], ph)) {
        if (globaltimer_ns() - t0 > 200000000ull) break;
      }
    }
  }
  __syncthreads();
  if (warp == 1) {
    tc_fence_after_sync();
    tmem_dealloc(tmem_base, Cfg::kTmemCols);
  }
}

}  // namespace MSB_ELEM_NS
}  // namespace msb

using namespace msb;
using namespace msb::MSB_ELEM_NS;

namespace {

// Box (tw, th, tn) with tw*th*tn == pixels_per_tile (all powers of two) that covers the N x H x W grid with the
// fewest tiles; ties go to the widest box.
void pick_box(int N, int H, int W, int pixels_per_tile, int* tw, int* th, int* tn) {
  long long best = -1;
  for (int a = 1; a <= pixels_per_tile; a <<= 1) {
    for (int b = 1; a * b <= pixels_per_tile; b <<= 1) {
      const int c = pixels_per_tile / (a * b);
      if (a > 256 || b > 256 || c > 256) continue;
      const long long tiles = static_cast<long long>((W + a - 1) / a) * ((H + b - 1) / b) * ((N + c - 1) / c);
      if (best < 0 || tiles < best || (tiles == best && a > *tw)) {
        best = tiles;
        *tw = a; *th = b; *tn = c;
      }
    }
  }
}

// Tensor maps of the (parity planes of the) NHWC input and the tap table.
int setup_input(CUtensorMap maps[4], ConvParams* p, const void* x, int N, int H, int W, int C, long long ldx, int R,
                int S, int stride, int pad_h, int pad_w, int flip) {
  if (stride != 1 && stride != 2) { set_last_error("conv: stride %d is not supported (1 or 2)", stride); return kBadArg; }
  if (R * S > kMaxTaps) { set_last_error("conv: %dx%d filter has more than %d taps", R, S, kMaxTaps); return kBadArg; }
  if (ldx % 8) { set_last_error("conv: pixel pitch %lld must be a multiple of 8 elements", ldx); return kBadArg; }
  const uint32_t box[4] = {64u, (uint32_t)p->tw, (uint32_t)p->th, (uint32_t)p->tn};
  const int planes = stride == 1 ? 1 : 4;
  for (int pl = 0; pl < 4; ++pl) {
    const int ph = stride == 1 ? 0 : (pl >> 1), pw = stride == 1 ? 0 : (pl & 1);
    if (pl >= planes || ph >= H || pw >= W) { maps[pl] = maps[0]; continue; }
    const elem_t* base = static_cast<const elem_t*>(x) + (static_cast<long long>(ph) * W + pw) * ldx;
    const uint64_t dims[4] = {(uint64_t)C, (uint64_t)((W - pw + stride - 1) / stride),
                              (uint64_t)((H - ph + stride - 1) / stride), (uint64_t)N};
    const uint64_t st[3] = {(uint64_t)(stride * ldx * 2), (uint64_t)(stride * W * ldx * 2),
                            (uint64_t)((long long)H * W * ldx * 2)};
    if (int rc = encode_tmap_4d(&maps[pl], base, dims, st, box)) return rc;
  }
  p->taps = R * S;
  for (int r = 0; r < R; ++r) {
    for (int s = 0; s < S; ++s) {
      const int oh = flip ? pad_h - r : r - pad_h, ow = flip ? pad_w - s : s - pad_w;
      const int ph = stride == 1 ? 0 : (oh & 1), pw = stride == 1 ? 0 : (ow & 1);
      const int t = r * S + s;
      p->tap_map[t] = static_cast<short>(stride == 1 ? 0 : ph * 2 + pw);
      p->tap_dh[t] = static_cast<short>(stride == 1 ? oh : (oh - ph) / 2);
      p->tap_dw[t] = static_cast<short>(stride == 1 ? ow : (ow - pw) / 2);
    }
  }
  return kOk;
}

template <int BN, bool WGRAD, bool B_MN = WGRAD>
int launch_conv(const CUtensorMap maps[4], const CUtensorMap& tmO, const CUtensorMap& tmY, const ConvParams& p, int tiles,
                cudaStream_t stream) {
  using Cfg = ConvCfg<BN>;
  auto kern = conv_igemm_kernel<BN, WGRAD, B_MN>;
  static bool configured = false;
  if (!configured) {
    MSB_CUDA_CHECK(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, Cfg::kSmemBytes));
    configured = true;
  }
  const int grid = tiles < sm_count() ? tiles : sm_count();
  kern<<<grid, kConvThreads, Cfg::kSmemBytes, stream>>>(maps[0], maps[1], maps[2], maps[3], tmO, tmY, p);
  MSB_CUDA_CHECK(cudaGetLastError());
  return kOk;
}

}  // namespace

// y[N, Ho, Wo, Cout] = conv(x[N, H, W, Cin], w[Cout, R, S, Cin]); bf16 NHWC; ldx / ldy = elements between pixels.
// flip = 0: y[ho, wo] += x[ho*stride + r - pad_h, wo*stride + s - pad_w] * w[r, s]      (forward)
// flip = 1: y[ho, wo] += x[ho + pad_h - r, wo + pad_w - s] * w[r, s]  (stride 1 only)   (data gradient, with
//           x = dY, w = weights permuted to [Cin, R, S, Cout])
// flip = 2: as 1 with w as the forward pass holds it, which is [Cin, R, S, Cout] in the terms of this call: no permuted copy
//           of the weights, one launch less per layer (Cout a multiple of 8)
// stats (optional): fp32 [2 * Cout], += per-channel sum and sum of squares of y (caller zeroes it).
// Cin must be a multiple of 64.
MSB_EXPORT int MSB_FN(msb_conv_fwd)(const void* x, const void* w, void* y, float* stats, int N, int H, int W, int Cin,
                            int Cout, int R, int S, int stride, int pad_h, int pad_w, int flip, int Ho, int Wo,
                            long long ldx, long long ldy, int out_fp32, void* stream_) {
  if (N <= 0 || H <= 0 || W <= 0 || Ho <= 0 || Wo <= 0 || Cin <= 0 || Cout <= 0 || (Cin % 64)) {
    set_last_error("conv_fwd: bad shape N=%d H=%d W=%d Cin=%d (multiple of 64) Cout=%d Ho=%d Wo=%d", N, H, W, Cin,
                   Cout, Ho, Wo);
    return kBadArg;
  }
  if (flip && stride != 1) { set_last_error("conv_fwd: the data-gradient form needs stride 1"); return kBadArg; }
  if (flip == 2 && (Cout % 8)) { set_last_error("conv_fwd: data gradient of %d channels (multiple of 8)", Cout); return kBadArg; }
  if (stats && (Cout > kMaxStatChannels || out_fp32)) {
    set_last_error("conv_fwd: fused statistics need bf16 output and at most %d channels", kMaxStatChannels);
    return kBadArg;
  }
  ConvParams p = {};
  p.C = y; p.stats = stats; p.status = status_ptr();
  if (!p.status) { set_last_error("conv_fwd: no status word"); return kCudaError; }
  p.N = N; p.Ho = Ho; p.Wo = Wo; p.Cin = Cin; p.Cout = Cout; p.ldc = ldy; p.out_fp32 = out_fp32; p.ksplit = 1;
  pick_box(N, Ho, Wo, kConvBM, &p.tw, &p.th, &p.tn);
  p.tiles_w = (Wo + p.tw - 1) / p.tw; p.tiles_h = (Ho + p.th - 1) / p.th; p.tiles_n = (N + p.tn - 1) / p.tn;
  p.cin_blocks = Cin / 64;
  CUtensorMap maps[4], tmW;
  if (int rc = setup_input(maps, &p, x, N, H, W, Cin, ldx, R, S, stride, pad_h, pad_w, flip)) return rc;
  const long long pix_tiles = static_cast<long long>(p.tiles_w) * p.tiles_h * p.tiles_n;
  // Up to 64 channels: half of a 128-column tile's weight rows, products and shared memory would be padding (64 x 56 x 56,
  // 1x1 256 -> 64 and 3x3 64 -> 64, forward and data gradient: 172 -> 139 us).
  const int bn = Cout <= 64 ? 64 : (Cout <= 128 || pix_tiles * ((Cout + 255) / 256) < sm_count()) ? 128 : 256;
  const long long K = static_cast<long long>(R) * S * Cin;
  const bool b_mn = flip == 2;
  if (b_mn) {
    const long long row = static_cast<long long>(R) * S * Cout;
    if (int rc = encode_tmap_3d(&tmW, w, 2, row, Cin, 1, row * 2, row * 2 * Cin, 64, 64, 1)) return rc;
  } else {
    if (int rc = encode_tmap_3d(&tmW, w, 2, K, Cout, 1, K * 2, K * 2 * Cout, 64, bn, 1)) return rc;
  }
  // the output as TMA sees it: a warp's 32 rows are a sub-box of the tile's (all extents are powers of two)
  CUtensorMap tmY = tmW;
  if (!out_fp32 && (reinterpret_cast<uintptr_t>(y) & 15) == 0 && ldy % 8 == 0) {
    const uint32_t bw = p.tw < 32 ? p.tw : 32, bh = p.th < 32 / (int)bw ? p.th : 32 / bw;
    const uint32_t ybox[4] = {64u, bw, bh, 32u / (bw * bh)};
    const uint64_t ydims[4] = {(uint64_t)Cout, (uint64_t)Wo, (uint64_t)Ho, (uint64_t)N};
    const uint64_t yst[3] = {(uint64_t)(ldy * 2), (uint64_t)(Wo * ldy * 2), (uint64_t)((long long)Ho * Wo * ldy * 2)};
    if (int rc = encode_tmap_4d(&tmY, y, ydims, yst, ybox)) return rc;
    p.tma_out = 1;
  }
  const long long tiles = pix_tiles * ((Cout + bn - 1) / bn);
  if (tiles > 0x7fffffffLL) { set_last_error("conv_fwd: too many tiles"); return kTooLarge; }
  cudaStream_t stream = static_cast<cudaStream_t>(stream_);
  if (b_mn) {
    if (bn == 256) return launch_conv<256, false, true>(maps, tmW, tmY, p, (int)tiles, stream);
    if (bn == 64) return launch_conv<64, false, true>(maps, tmW, tmY, p, (int)tiles, stream);
    return launch_conv<128, false, true>(maps, tmW, tmY, p, (int)tiles, stream);
  }
  if (bn == 256) return launch_conv<256, false>(maps, tmW, tmY, p, (int)tiles, stream);
  if (bn == 64) return launch_conv<64, false>(maps, tmW, tmY, p, (int)tiles, stream);
  return launch_conv<128, false>(maps, tmW, tmY, p, (int)tiles, stream);
}

// dw[Cout, R, S, Cin] (fp32) (+)= sum over pixels of dy[N, Ho, Wo, Cout] x shifted x[N, H, W, Cin].
MSB_EXPORT int MSB_FN(msb_conv_wgrad)(const void* x, const void* dy, float* dw, int N, int H, int W, int Cin, int Cout,
                              int R, int S, int stride, int pad_h, int pad_w, int Ho, int Wo, long long ldx,
                              long long ldy, int accumulate, void* stream_) {
  if (N <= 0 || H <= 0 || W <= 0 || Ho <= 0 || Wo <= 0 || Cin <= 0 || Cout <= 0 || (Cin % 8) || (Cout % 8) ||
      (ldy % 8)) {
    set_last_error("conv_wgrad: bad shape N=%d H=%d W=%d Cin=%d Cout=%d Ho=%d Wo=%d (channels multiples of 8)", N, H,
                   W, Cin, Cout, Ho, Wo);
    return kBadArg;
  }
  ConvParams p = {};
  p.C = dw; p.status = status_ptr();
  if (!p.status) { set_last_error("conv_wgrad: no status word"); return kCudaError; }
  p.N = N; p.Ho = Ho; p.Wo = Wo; p.Cin = Cin; p.Cout = Cout; p.out_fp32 = 1; p.accumulate = 1;
  p.ldc = static_cast<long long>(R) * S * Cin;
  pick_box(N, Ho, Wo, kConvBK, &p.tw, &p.th, &p.tn);
  p.tiles_w = (Wo + p.tw - 1) / p.tw; p.tiles_h = (Ho + p.th - 1) / p.th; p.tiles_n = (N + p.tn - 1) / p.tn;
  CUtensorMap maps[4], tmDY;
  if (int rc = setup_input(maps, &p, x, N, H, W, Cin, ldx, R, S, stride, pad_h, pad_w, 0)) return rc;
  const uint32_t box[4] = {64u, (uint32_t)p.tw, (uint32_t)p.th, (uint32_t)p.tn};
  const uint64_t dims[4] = {(uint64_t)Cout, (uint64_t)Wo, (uint64_t)Ho, (uint64_t)N};
  const uint64_t st[3] = {(uint64_t)(ldy * 2), (uint64_t)(Wo * ldy * 2), (uint64_t)((long long)Ho * Wo * ldy * 2)};
  if (int rc = encode_tmap_4d(&tmDY, dy, dims, st, box)) return rc;
  // The feed of shared memory bounds a tile (an A block of 128 rows costs as much as 128 columns of B), so: the fewest
  // tiles, and of the widths that give that count the narrowest.  64 x 56 x 56, 3x3 64 -> 64 and 1x1 64 -> 256 together, one
  // tap per tile of 128 columns 122 us, this way 39 + 28.
  p.flat = Cin % 64 == 0;
  int bn = Cin <= 128 ? 128 : 256;
  if (p.flat) {
    const int blocks = p.taps * (Cin / 64), fewest = (blocks + 3) / 4;
    bn = 64;
    while ((blocks + bn / 64 - 1) / (bn / 64) > fewest) bn += 64;
  }
  const int cols = p.flat ? p.taps * Cin : Cin;
  const long long base_tiles =
      static_cast<long long>((Cout + kConvBM - 1) / kConvBM) * ((cols + bn - 1) / bn) * (p.flat ? 1 : p.taps);
  const long long pix_tiles = static_cast<long long>(p.tiles_w) * p.tiles_h * p.tiles_n;
  // Split of the pixel loop with the fewest k-blocks on the longest CTA: rounds of one tile per SM, each as long as its
  // k-blocks plus about eight for filling the pipeline and adding the tile into dW.
  long long split = 1, best = -1;
  for (long long t = 1; t <= pix_tiles && (t == 1 || base_tiles * (t - 1) < 2LL * sm_count()); ++t) {
    const long long rounds = (base_tiles * t + sm_count() - 1) / sm_count(), cost = rounds * ((pix_tiles + t - 1) / t + 8);
    if (best < 0 || cost < best) { best = cost; split = t; }
  }
  p.ksplit = static_cast<int>(split);
  CUtensorMap tmY = tmDY;
  if (Cin % 32 == 0 && (reinterpret_cast<uintptr_t>(dw) & 15) == 0) {
    if (int rc = encode_tmap_3d(&tmY, dw, 4, (uint64_t)p.ldc, Cout, 1, p.ldc * 4, (uint64_t)p.ldc * 4 * Cout, 32, 32, 1))
      return rc;
    p.tma_out = 1;
  }
  cudaStream_t stream = static_cast<cudaStream_t>(stream_);
  if (!accumulate)
    MSB_CUDA_CHECK(cudaMemsetAsync(dw, 0, sizeof(float) * static_cast<size_t>(Cout) * R * S * Cin, stream));
  const long long tiles = base_tiles * split;
  if (bn == 256) return launch_conv<256, true>(maps, tmDY, tmY, p, (int)tiles, stream);
  if (bn == 192) return launch_conv<192, true>(maps, tmDY, tmY, p, (int)tiles, stream);
  if (bn == 64) return launch_conv<64, true>(maps, tmDY, tmY, p, (int)tiles, stream);
  return launch_conv<128, true>(maps, tmDY, tmY, p, (int)tiles, stream);
}

namespace msb {
namespace MSB_ELEM_NS {
// Patch matrix for convolutions whose input has too few channels for the 64-channel box loads (the first layer of
// image networks): out[pix, (r*S + s)*Cin + c] = x[n, ho*stride + r - pad, wo*stride + s - pad, c], zero outside the
// image and in the padding columns k >= R*S*Cin.
__global__ void __launch_bounds__(256)
im2col_nhwc_kernel(const elem_t* __restrict__ x, elem_t* __restrict__ out, int N, int H, int W, int Cin,
                   int R, int S, int stride, int pad_h, int pad_w, int Ho, int Wo, int Kpad) {
  // One thread per 16-byte chunk (8 columns) of a patch row, so stores are coalesced; where column k comes from
  // (filter row, offset inside the contiguous S*Cin input segment) is looked up in a table built once per block.
  extern __shared__ short tab[];          // [Kpad][2]: filter row (or -1 for padding columns), segment offset
  const int K = R * S * Cin, seg = S * Cin;
  for (int k = threadIdx.x; k < Kpad; k += blockDim.x) {
    tab[2 * k] = k < K ? (short)(k / seg) : (short)-1;
    tab[2 * k + 1] = (short)(k % seg);
  }
  __syncthreads();
  const int chunks = Kpad / 8;
  const long long total = (long long)N * Ho * Wo * chunks;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < total;
       i += (long long)gridDim.x * blockDim.x) {
    const int ch = (int)(i % chunks);
    const long long pix = i / chunks;
    const int wo = (int)(pix % Wo);
    const int ho = (int)((pix / Wo) % Ho);
    const int n = (int)(pix / ((long long)Wo * Ho));
    const int h0 = ho * stride - pad_h, w0 = wo * stride - pad_w;
    const elem_t* img = x + (long long)n * H * W * Cin;
    __align__(16) elem_t v[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      const int k = ch * 8 + j;
      const int r = tab[2 * k], off = tab[2 * k + 1];
      const int h = h0 + r, w = w0 + off / Cin;
      const bool in = r >= 0 && h >= 0 && h < H && w >= 0 && w < W;
      v[j] = in ? img[((long long)h * W + w0) * Cin + off] : f_to_e(0.f);
    }
    reinterpret_cast<uint4*>(out)[i] = *reinterpret_cast<const uint4*>(v);
  }
}
}  // namespace MSB_ELEM_NS
}  // namespace msb

MSB_EXPORT int MSB_FN(msb_im2col_nhwc)(const void* x, void* out, int N, int H, int W, int Cin, int R, int S, int stride,
                               int pad_h, int pad_w, int Ho, int Wo, int Kpad, void* stream) {
  if (Kpad < R * S * Cin || (Kpad % 8)) {
    set_last_error("im2col: padded width %d must be a multiple of 8 and at least %d", Kpad, R * S * Cin);
    return kBadArg;
  }
  const long long total = (long long)N * Ho * Wo * (Kpad / 8);
  if (total <= 0) return kOk;
  long long blocks = (total + 255) / 256;
  const long long cap = (long long)sm_count() * 16;
  blocks = blocks > cap ? cap : blocks;
  im2col_nhwc_kernel<<<(unsigned)blocks, 256, Kpad * 4, (cudaStream_t)stream>>>(
      (const elem_t*)x, (elem_t*)out, N, H, W, Cin, R, S, stride, pad_h, pad_w, Ho, Wo, Kpad);
  MSB_CUDA_CHECK(cudaGetLastError());
  return kOk;
}
