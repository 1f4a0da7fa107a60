// Memory-bound transformer kernels for sm_100a: RMSNorm / LayerNorm (forward, backward, fused
// residual add), RoPE, SwiGLU, GELU.  All move 16 bytes per thread per access and make one pass
// over HBM per tensor; reductions stay in registers / shared memory.
//
// The reference has a block-per-row Welford LayerNorm for GPU
// (plugin/device/gpu/kernel/cuda_impl/cuda_ops/layer_norm_impl.cu:218) and a half2 GELU
// (gelu_impl.cu:56); RmsNorm, ApplyRotaryPosEmb and SwiGLU have op definitions
// (core/ops/ops_def/rms_norm_op.yaml, apply_rotary_pos_emb_op.yaml) but no GPU kernel.
//
// This text is compiled twice: for bf16 tensors (norm_act.cu), and with MSB_ELEM_FP16 defined for fp16 tensors
// (norm_act_fp16.cu), where every entry point carries the suffix _fp16 and "bf16" in a comment reads "fp16".
#include "host_common.h"
#include "elem.cuh"

namespace msb {
namespace MSB_ELEM_NS {

struct alignas(16) bf16x8 {
  elem2_t v[4];
};

__device__ __forceinline__ void load8(const elem_t* p, float (&f)[8]) {
  const bf16x8 raw = *reinterpret_cast<const bf16x8*>(p);
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const float2 t = e2_to_f2(raw.v[i]);
    f[2 * i] = t.x;
    f[2 * i + 1] = t.y;
  }
}
__device__ __forceinline__ void store8(elem_t* p, const float (&f)[8]) {
  bf16x8 raw;
#pragma unroll
  for (int i = 0; i < 4; ++i) raw.v[i] = f2_to_e2(f[2 * i], f[2 * i + 1]);
  *reinterpret_cast<bf16x8*>(p) = raw;
}

// ------------------------------------------------------------------------------------ norms: threads and rows
// A row of H elements is H / 8 vectors of 16 bytes.  T threads (a multiple of 32) share a row, V vectors each, and a block
// holds R such groups, each with a row of its own.  The bound is HBM; what costs time beside it is a row's chain of load,
// reduction and store, so an SM needs many rows in flight and no thread without a vector.  One row per block of 256
// threads, as before, idled three quarters of the second round of vectors at H = 2560 and held two rows per SM in the
// backward kernels, whose loads of the residual gradient moreover waited for the reduction.  Measured, bf16: RMSNorm
// backward of 4096 x 4096 with residual 52 -> 38 us, LayerNorm backward of 8191 x 2560 68 -> 43 us, forward 35 -> 31 us.
// A forward kernel that prefetches the next row measured no better than one block per row.
struct NormShape {
  int T, R, V;
};
constexpr int kNormMaxV = 4;
constexpr int kNormMaxThreads = 512;      // H = 16384
constexpr int kNormBwdPerSm = 4;          // most blocks per SM of a backward kernel

// Of the shapes with at most max_v vectors per thread the one with the fewest idle slots, the most vectors per thread
// among those.
static inline NormShape norm_shape(int H, int max_v) {
  const int vecs = H / 8;
  NormShape best = {0, 1, 0};
  int waste = 1 << 30;
  for (int v = max_v; v >= 1; --v) {
    const int t = (vecs + 32 * v - 1) / (32 * v) * 32;
    if (t <= kNormMaxThreads && t * v - vecs < waste) {
      waste = t * v - vecs;
      best.T = t;
      best.V = v;
    }
  }
  return best;
}
// Forward: a warp per row needs no barrier, eight of them make a block; longer rows have the block to themselves.
static inline NormShape norm_fwd_shape(int H) {
  NormShape n = norm_shape(H, H <= 16 * kNormMaxThreads ? 2 : kNormMaxV);
  if (n.T == 32) n.R = 8;
  return n;
}
// Backward: the accumulators of the weight gradients take 8 registers per vector, so two vectors per thread as far as
// 512 threads reach, and groups of a block share one row of partial sums.
static inline NormShape norm_bwd_shape(int H) {
  NormShape n = norm_shape(H, H <= 16 * kNormMaxThreads ? 2 : kNormMaxV);
  n.R = n.T >= 256 ? 1 : 256 / n.T;
  return n;
}

// Reductions over the T threads of a row.  MULTI: several groups per block, each with a named barrier of its own (1 +
// group); otherwise the group is one warp or the whole block.
template <bool MULTI>
struct NormGroup {
  int T, tid, group, warps, buf;
  float2* red;                            // [2][16] of this group
  __device__ __forceinline__ NormGroup(int T_, float2* smem) : T(T_), buf(0) {
    group = threadIdx.x / T_;
    tid = threadIdx.x - group * T_;
    warps = T_ >> 5;
    red = smem + (MULTI ? group * 32 : 0);
  }
  // At most four groups are wider than a warp (T >= 64).  Barrier numbers are constants: a number in a register makes the
  // compiler reserve all sixteen barriers for every block.
  __device__ __forceinline__ void barrier() {
    if (!MULTI) { __syncthreads(); return; }
    if (group == 0) asm volatile("bar.sync 1, %0;" ::"r"(T) : "memory");
    else if (group == 1) asm volatile("bar.sync 2, %0;" ::"r"(T) : "memory");
    else if (group == 2) asm volatile("bar.sync 3, %0;" ::"r"(T) : "memory");
    else asm volatile("bar.sync 4, %0;" ::"r"(T) : "memory");
  }
  // Sums of a and b over the group, in every thread.  The scratch alternates between two halves: a warp can be at most one
  // sum ahead of the others of its group.
  __device__ __forceinline__ float2 sum2(float a, float b) {
    a = warp_sum(a);
    b = warp_sum(b);
    if (warps == 1) return make_float2(a, b);
    const int lane = tid & 31;
    float2* half = red + buf * 16;
    buf ^= 1;
    if (lane == 0) half[tid >> 5] = make_float2(a, b);
    barrier();
    const float2 t = lane < warps ? half[lane] : make_float2(0.f, 0.f);
    return make_float2(warp_sum(t.x), warp_sum(t.y));
  }
  __device__ __forceinline__ float sum(float a) {
    a = warp_sum(a);
    if (warps == 1) return a;
    const int lane = tid & 31;
    float2* half = red + buf * 16;
    buf ^= 1;
    if (lane == 0) half[tid >> 5].x = a;
    barrier();
    return warp_sum(lane < warps ? half[lane].x : 0.f);
  }
};
constexpr int kNormRed = 32, kNormRedMulti = 8 * 32;    // float2 scratch of a block (8 groups at most)

__device__ __forceinline__ void unpack8(const bf16x8& raw, float (&f)[8]) {
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const float2 t = e2_to_f2(raw.v[i]);
    f[2 * i] = t.x;
    f[2 * i + 1] = t.y;
  }
}
__device__ __forceinline__ bf16x8 load_raw(const elem_t* p) { return *reinterpret_cast<const bf16x8*>(p); }

// ------------------------------------------------------------------------------------ RMSNorm
// y = (x [+ res]) * rstd * w ; optionally writes the summed residual stream to `xsum`.
// H must be a multiple of 8 and at most 8 * kNormMaxV * kNormMaxThreads.
template <int V>
__global__ void __launch_bounds__(kNormMaxThreads)
rmsnorm_fwd_kernel(const elem_t* __restrict__ x, const elem_t* __restrict__ res,
                   const elem_t* __restrict__ w, elem_t* __restrict__ y,
                   elem_t* __restrict__ xsum, float* __restrict__ rstd_out, long long rows, int H, float eps, int T, int R) {
  __shared__ float2 red[kNormRed];
  NormGroup<false> g(T, red);
  const long long row = blockIdx.x * static_cast<long long>(R) + g.group;
  if (row >= rows) return;
  float v[V][8];
  {
    bf16x8 rx[V], rr[V];
#pragma unroll
    for (int it = 0; it < V; ++it) {
      const int c = (it * T + g.tid) * 8;
      if (c < H) {
        rx[it] = load_raw(x + row * H + c);
        if (res) rr[it] = load_raw(res + row * H + c);
      }
    }
#pragma unroll
    for (int it = 0; it < V; ++it) {
      const int c = (it * T + g.tid) * 8;
      if (c < H) {
        unpack8(rx[it], v[it]);
        if (res) {
          float r[8];
          unpack8(rr[it], r);
#pragma unroll
          for (int j = 0; j < 8; ++j) v[it][j] += r[j];
          if (xsum) {
            // round once so that the normalised value matches what the backward pass re-reads
            store8(xsum + row * H + c, v[it]);
#pragma unroll
            for (int j = 0; j < 8; ++j) v[it][j] = e_to_f(f_to_e(v[it][j]));
          }
        }
      }
    }
  }
  float ss = 0.f;
#pragma unroll
  for (int it = 0; it < V; ++it) {
    if ((it * T + g.tid) * 8 < H) {
#pragma unroll
      for (int j = 0; j < 8; ++j) ss += v[it][j] * v[it][j];
    }
  }
  const float rstd = rsqrtf(g.sum(ss) / H + eps);
  if (g.tid == 0 && rstd_out) rstd_out[row] = rstd;
#pragma unroll
  for (int it = 0; it < V; ++it) {
    const int c = (it * T + g.tid) * 8;
    if (c < H) {
      float gm[8], o[8];
      load8(w + c, gm);
#pragma unroll
      for (int j = 0; j < 8; ++j) o[j] = v[it][j] * rstd * gm[j];
      store8(y + row * H + c, o);
    }
  }
}

// Adds the groups' partial sums of a block (registers `mine`, element c of the row at (it * T + tid) * 8) in group order
// through shared memory and stores the total as row blockIdx.x of dst[gridDim.x][H].
template <int V>
__device__ __forceinline__ void store_partials(const float (&mine)[V][8], float* dst, float* acc, const NormGroup<true>& g,
                                               int R, int H) {
  dst += static_cast<long long>(blockIdx.x) * H;
#pragma unroll 1
  for (int k = 0; k < R; ++k) {
    if (g.group == k) {
#pragma unroll
      for (int it = 0; it < V; ++it) {
        const int c = (it * g.T + g.tid) * 8;
        if (c < H) {
          float4 lo = make_float4(mine[it][0], mine[it][1], mine[it][2], mine[it][3]);
          float4 hi = make_float4(mine[it][4], mine[it][5], mine[it][6], mine[it][7]);
          if (k > 0) {
            const float4 a = *reinterpret_cast<const float4*>(acc + c), b = *reinterpret_cast<const float4*>(acc + c + 4);
            lo.x += a.x; lo.y += a.y; lo.z += a.z; lo.w += a.w;
            hi.x += b.x; hi.y += b.y; hi.z += b.z; hi.w += b.w;
          }
          float* out = k == R - 1 ? dst : acc;
          *reinterpret_cast<float4*>(out + c) = lo;
          *reinterpret_cast<float4*>(out + c + 4) = hi;
        }
      }
    }
    if (R > 1) __syncthreads();
  }
}

// dx = rstd * (dy*w - xhat * mean(dy*w*xhat)) (+ dres_in) ; dw = sum_rows dy * xhat.
// Persistent over rows; per-group partial dw kept in registers.  Two-stage reduction (ATOMIC = false): CTA b stores the sum
// of its groups as row b of dw_acc[gridDim.x][H] and reduce_partials_kernel sums the rows in a fixed order
// (deterministic).  ATOMIC = true adds into a single dw_acc[H] instead (the allocation-free entry point, whose
// scratch is one row).  All loads of a row, the residual gradient's too, are issued before its reduction.
template <int V, bool ATOMIC>
__global__ void __maxnreg__(V <= 2 ? 64 : 128)
rmsnorm_bwd_kernel(const elem_t* __restrict__ dy, const elem_t* __restrict__ x,
                   const elem_t* __restrict__ w, const float* __restrict__ rstd,
                   const elem_t* __restrict__ dres, elem_t* __restrict__ dx,
                   float* __restrict__ dw_acc, long long rows, int H, int T, int R) {
  extern __shared__ float part[];          // [H] when R > 1
  __shared__ float2 red[kNormRedMulti];
  NormGroup<true> g(T, red);
  float dwreg[V][8];
#pragma unroll
  for (int it = 0; it < V; ++it)
#pragma unroll
    for (int j = 0; j < 8; ++j) dwreg[it][j] = 0.f;
#pragma unroll 1
  for (long long row = blockIdx.x * static_cast<long long>(R) + g.group; row < rows;
       row += static_cast<long long>(gridDim.x) * R) {
    const float rs = rstd[row];
    const elem_t* wp = w;                  // opaque: w comes from the L1 cache instead of filling registers
    asm volatile("" : "+l"(wp));
    bf16x8 rg[V], rx[V], rd[V];            // kept as loaded and unpacked twice: half the registers of fp32 values
    float dot = 0.f;
#pragma unroll
    for (int it = 0; it < V; ++it) {
      const int c = (it * T + g.tid) * 8;
      if (c < H) {
        rg[it] = load_raw(dy + row * H + c);
        rx[it] = load_raw(x + row * H + c);
        if (dres) rd[it] = load_raw(dres + row * H + c);
      }
    }
#pragma unroll
    for (int it = 0; it < V; ++it) {
      const int c = (it * T + g.tid) * 8;
      if (c < H) {
        float wv[8], gv[8], xh[8];
        load8(wp + c, wv);
        unpack8(rg[it], gv);
        unpack8(rx[it], xh);
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          xh[j] *= rs;
          dwreg[it][j] += gv[j] * xh[j];
          dot += (gv[j] * wv[j]) * xh[j];
        }
      }
    }
    dot = g.sum(dot) / H;
#pragma unroll
    for (int it = 0; it < V; ++it) {
      const int c = (it * T + g.tid) * 8;
      if (c < H) {
        float wv[8], gv[8], xh[8], o[8];
        load8(wp + c, wv);
        unpack8(rg[it], gv);
        unpack8(rx[it], xh);
#pragma unroll
        for (int j = 0; j < 8; ++j) o[j] = rs * (gv[j] * wv[j] - xh[j] * rs * dot);
        if (dres) {
          float r[8];
          unpack8(rd[it], r);
#pragma unroll
          for (int j = 0; j < 8; ++j) o[j] += r[j];
        }
        store8(dx + row * H + c, o);
      }
    }
  }
  if (ATOMIC) {
#pragma unroll
    for (int it = 0; it < V; ++it) {
      const int c = (it * T + g.tid) * 8;
      if (c < H) {
#pragma unroll
        for (int j = 0; j < 8; ++j) atomicAdd(dw_acc + c + j, dwreg[it][j]);
      }
    }
  } else {
    store_partials<V>(dwreg, dw_acc, part, g, R, H);
  }
}

// Second stage of the weight-gradient reduction: out[c] (+)= sum_b partial[b][c] for b = 0..parts-1, rows visited
// in a fixed order.  Block = 32 columns x 8 row lanes; lane r sums rows r, r+8, ... and the 8 lanes are combined
// through shared memory, always in the same order.  blockIdx.y chooses between two such reductions (dw, db).
struct PartialsOut {
  const float* partial;
  elem_t* out_bf16;
  float* out_f32;
};
__global__ void __launch_bounds__(256)
reduce_partials_kernel(const PartialsOut first, const PartialsOut second, int parts, int H, int accumulate) {
  __shared__ float sm[8][33];
  const PartialsOut o = blockIdx.y == 0 ? first : second;
  const int cx = threadIdx.x & 31, ry = threadIdx.x >> 5;
  const int c = blockIdx.x * 32 + cx;
  float s = 0.f;
  if (c < H) {
#pragma unroll 8
    for (int b = ry; b < parts; b += 8) s += o.partial[static_cast<long long>(b) * H + c];
  }
  sm[ry][cx] = s;
  __syncthreads();
  if (ry == 0 && c < H) {
    float v = sm[0][cx];
#pragma unroll
    for (int r = 1; r < 8; ++r) v += sm[r][cx];
    if (o.out_f32) o.out_f32[c] = accumulate ? o.out_f32[c] + v : v;
    if (o.out_bf16) o.out_bf16[c] = f_to_e(accumulate ? e_to_f(o.out_bf16[c]) + v : v);
  }
}

// ------------------------------------------------------------------------------------ LayerNorm
template <int V>
__global__ void __launch_bounds__(kNormMaxThreads)
layernorm_fwd_kernel(const elem_t* __restrict__ x, const elem_t* __restrict__ w,
                     const elem_t* __restrict__ b, elem_t* __restrict__ y,
                     float* __restrict__ mean_out, float* __restrict__ rstd_out, long long rows, int H, float eps, int T,
                     int R) {
  __shared__ float2 red[kNormRed];
  NormGroup<false> g(T, red);
  const long long row = blockIdx.x * static_cast<long long>(R) + g.group;
  if (row >= rows) return;
  float v[V][8];
  {
    bf16x8 rx[V];
#pragma unroll
    for (int it = 0; it < V; ++it) {
      const int c = (it * T + g.tid) * 8;
      if (c < H) rx[it] = load_raw(x + row * H + c);
    }
#pragma unroll
    for (int it = 0; it < V; ++it)
      if ((it * T + g.tid) * 8 < H) unpack8(rx[it], v[it]);
  }
  float s = 0.f;
#pragma unroll
  for (int it = 0; it < V; ++it) {
    if ((it * T + g.tid) * 8 < H) {
#pragma unroll
      for (int j = 0; j < 8; ++j) s += v[it][j];
    }
  }
  const float mean = g.sum(s) / H;
  float ss = 0.f;
#pragma unroll
  for (int it = 0; it < V; ++it) {
    if ((it * T + g.tid) * 8 < H) {
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        const float d = v[it][j] - mean;
        ss += d * d;
      }
    }
  }
  const float rstd = rsqrtf(g.sum(ss) / H + eps);
  if (g.tid == 0) {
    if (mean_out) mean_out[row] = mean;
    if (rstd_out) rstd_out[row] = rstd;
  }
#pragma unroll
  for (int it = 0; it < V; ++it) {
    const int c = (it * T + g.tid) * 8;
    if (c < H) {
      float gm[8], bb[8], o[8];
      load8(w + c, gm);
      if (b) load8(b + c, bb);
#pragma unroll
      for (int j = 0; j < 8; ++j) o[j] = (v[it][j] - mean) * rstd * gm[j] + (b ? bb[j] : 0.f);
      store8(y + row * H + c, o);
    }
  }
}

template <int V>
__global__ void __maxnreg__(V <= 2 ? 80 : 128)
layernorm_bwd_kernel(const elem_t* __restrict__ dy, const elem_t* __restrict__ x,
                     const elem_t* __restrict__ w, const float* __restrict__ mean,
                     const float* __restrict__ rstd, elem_t* __restrict__ dx, float* __restrict__ dw_acc,
                     float* __restrict__ db_acc, long long rows, int H, int T, int R) {
  extern __shared__ float part[];          // [H] when R > 1
  __shared__ float2 red[kNormRedMulti];
  NormGroup<true> g(T, red);
  float dwreg[V][8], dbreg[V][8];
#pragma unroll
  for (int it = 0; it < V; ++it)
#pragma unroll
    for (int j = 0; j < 8; ++j) dwreg[it][j] = dbreg[it][j] = 0.f;
#pragma unroll 1
  for (long long row = blockIdx.x * static_cast<long long>(R) + g.group; row < rows;
       row += static_cast<long long>(gridDim.x) * R) {
    const float mu = mean[row], rs = rstd[row];
    const elem_t* wp = w;
    asm volatile("" : "+l"(wp));
    bf16x8 rg[V], rx[V];
    float s1 = 0.f, s2 = 0.f;
#pragma unroll
    for (int it = 0; it < V; ++it) {
      const int c = (it * T + g.tid) * 8;
      if (c < H) {
        rg[it] = load_raw(dy + row * H + c);
        rx[it] = load_raw(x + row * H + c);
      }
    }
#pragma unroll
    for (int it = 0; it < V; ++it) {
      const int c = (it * T + g.tid) * 8;
      if (c < H) {
        float wv[8], gv[8], xh[8];
        load8(wp + c, wv);
        unpack8(rg[it], gv);
        unpack8(rx[it], xh);
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          xh[j] = (xh[j] - mu) * rs;
          dwreg[it][j] += gv[j] * xh[j];
          dbreg[it][j] += gv[j];
          gv[j] *= wv[j];
          s1 += gv[j];
          s2 += gv[j] * xh[j];
        }
      }
    }
    const float2 t = g.sum2(s1, s2);
    s1 = t.x / H;
    s2 = t.y / H;
#pragma unroll
    for (int it = 0; it < V; ++it) {
      const int c = (it * T + g.tid) * 8;
      if (c < H) {
        float wv[8], gv[8], xh[8], o[8];
        load8(wp + c, wv);
        unpack8(rg[it], gv);
        unpack8(rx[it], xh);
#pragma unroll
        for (int j = 0; j < 8; ++j) o[j] = rs * (gv[j] * wv[j] - s1 - (xh[j] - mu) * rs * s2);
        store8(dx + row * H + c, o);
      }
    }
  }
  // two-stage reduction: this CTA's partial sums are row blockIdx.x of dw_acc / db_acc ([gridDim.x][H] each)
  store_partials<V>(dwreg, dw_acc, part, g, R, H);
  if (db_acc) store_partials<V>(dbreg, db_acc, part, g, R, H);
}

// fp32 accumulator -> bf16 parameter gradient (optionally accumulating into an existing bf16/fp32 grad)
__global__ void finalize_acc_kernel(const float* __restrict__ acc, elem_t* __restrict__ out_bf16,
                                    float* __restrict__ out_f32, int n, int accumulate) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  float v = acc[i];
  if (out_f32) out_f32[i] = accumulate ? out_f32[i] + v : v;
  if (out_bf16) out_bf16[i] = f_to_e(accumulate ? e_to_f(out_bf16[i]) + v : v);
}

// ------------------------------------------------------------------------------------ RoPE
// src, dst: [tokens, heads, D] (row pitches in elements per token; they may be the same memory), rotate-half convention:
//   out[..., i]       = x[i]*cos[i] - x[i+D/2]*sin[i]
//   out[..., i+D/2]   = x[i+D/2]*cos[i] + x[i]*sin[i]
// cos/sin: fp32 [seq, D/2]; position of token t is pos[t] if given, else (t % seq).
// sign = -1 gives the backward (inverse) rotation.
// A block rotates one token: a thread keeps the eight angles of its vector pair in registers and walks over the heads, two
// of them in flight.  Bound by reading and writing x; the angles used to be looked up again for every vector (16 scalar
// loads and three 64-bit divisions per 32 bytes).  4096 tokens x 64 heads of 128, bf16: 33 -> 29 us.
constexpr int kRopeThreads = 256;
__global__ void __launch_bounds__(kRopeThreads)
rope_kernel(const elem_t* src, elem_t* dst, const float* __restrict__ cosb,
            const float* __restrict__ sinb, const int* __restrict__ pos, int heads, int D, long long src_pitch,
            long long dst_pitch, int seq, float sign, int lanes, int hstep, int aligned) {
  const int half = D / 2, vph = half / 8;
  if (threadIdx.x >= lanes * hstep) return;
  const long long t = blockIdx.x;
  const long long p = pos ? pos[t] : t % seq;
  const int h0 = threadIdx.x / lanes;
  for (int vi = threadIdx.x % lanes; vi < vph; vi += lanes) {
    float c[8], sn[8];
    const float* cp = cosb + p * half + vi * 8;
    const float* sp = sinb + p * half + vi * 8;
    if (aligned) {
#pragma unroll
      for (int j = 0; j < 8; j += 4) {
        *reinterpret_cast<float4*>(c + j) = *reinterpret_cast<const float4*>(cp + j);
        *reinterpret_cast<float4*>(sn + j) = *reinterpret_cast<const float4*>(sp + j);
      }
    } else {
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        c[j] = cp[j];
        sn[j] = sp[j];
      }
    }
#pragma unroll
    for (int j = 0; j < 8; ++j) sn[j] *= sign;
    auto rotate = [&](const bf16x8& ra, const bf16x8& rb, int h) {
      float a[8], b[8], oa[8], ob[8];
      unpack8(ra, a);
      unpack8(rb, b);
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        oa[j] = a[j] * c[j] - b[j] * sn[j];
        ob[j] = b[j] * c[j] + a[j] * sn[j];
      }
      elem_t* q = dst + t * dst_pitch + (long long)h * D + vi * 8;
      store8(q, oa);
      store8(q + half, ob);
    };
    const elem_t* x = src + t * src_pitch + vi * 8;
    int h = h0;
    for (; h + hstep < heads; h += 2 * hstep) {
      const elem_t* x0 = x + (long long)h * D;
      const elem_t* x1 = x + (long long)(h + hstep) * D;
      const bf16x8 a0 = load_raw(x0), b0 = load_raw(x0 + half), a1 = load_raw(x1), b1 = load_raw(x1 + half);
      rotate(a0, b0, h);
      rotate(a1, b1, h + hstep);
    }
    if (h < heads) {
      const elem_t* x0 = x + (long long)h * D;
      const bf16x8 a0 = load_raw(x0), b0 = load_raw(x0 + half);
      rotate(a0, b0, h);
    }
  }
}

// ------------------------------------------------------------------------------------ SwiGLU / GELU
__device__ __forceinline__ float sigmoidf_(float x) { return 1.f / (1.f + __expf(-x)); }

// Quotients by a divisor that is the same for the whole launch: a multiplication and a shift for the vector indices of a
// tensor of fewer than 2^31 vectors (exact: m = ceil(2^(32 + s) / d) with 2^s >= d, and n < 2^31), a division beyond.
struct FastDiv {
  unsigned d, m, s, small;
  __device__ __forceinline__ void operator()(long long n, long long& q, int& r) const {
    if (small) {
      const unsigned u = static_cast<unsigned>(n);
      const unsigned long long w = static_cast<unsigned long long>(u) * m;
      const unsigned k = static_cast<unsigned>((w + (static_cast<unsigned long long>(u) << 32)) >> (32 + s));
      q = k;
      r = static_cast<int>(u - k * d);
    } else {
      q = n / d;
      r = static_cast<int>(n - q * d);
    }
  }
};
static inline FastDiv fast_div(int d, long long total) {
  FastDiv f;
  f.d = static_cast<unsigned>(d);
  f.s = 0;
  while ((1ull << f.s) < f.d) ++f.s;
  // ceil(2^(32 + s) / d) lies in [2^32, 2^33): its low 32 bits are kept, the top one is added back above
  f.m = static_cast<unsigned>(((1ull << (32 + f.s)) + f.d - 1) / f.d);
  f.small = total < (1ll << 31);
  return f;
}

// gu: [rows, 2F] with gate in [:, :F], up in [:, F:]; out [rows, F] = silu(gate) * up
// Bound by its loads and stores; two vector positions (64 bytes of loads) are in flight per thread, and the row of a vector
// comes from a multiplication instead of a 64-bit division per 16 bytes (4096 x 11008 bf16: 72 -> 65 us).
__global__ void __launch_bounds__(256)
swiglu_fwd_kernel(const elem_t* __restrict__ gu, elem_t* __restrict__ out, long long total, int F, const FastDiv div) {
  const long long step = (long long)gridDim.x * 256;
  for (long long i = blockIdx.x * 256ll + threadIdx.x; i < total; i += 2 * step) {
    bf16x8 rg[2], ru[2];
#pragma unroll
    for (int u = 0; u < 2; ++u) {
      if (i + u * step < total) {
        long long r;
        int c;
        div(i + u * step, r, c);
        const elem_t* p = gu + r * 2 * F + c * 8;
        rg[u] = load_raw(p);
        ru[u] = load_raw(p + F);
      }
    }
#pragma unroll
    for (int u = 0; u < 2; ++u) {
      if (i + u * step < total) {
        float g[8], v[8], o[8];
        unpack8(rg[u], g);
        unpack8(ru[u], v);
#pragma unroll
        for (int j = 0; j < 8; ++j) o[j] = g[j] * sigmoidf_(g[j]) * v[j];
        store8(out + (i + u * step) * 8, o);
      }
    }
  }
}
// dgu[:, :F] = dout * up * (s + g*s*(1-s)) ; dgu[:, F:] = dout * g*s
// One position per thread: three loads and two stores keep enough bytes in flight, and a second position halves the
// resident threads (4096 x 11008 bf16: 92 -> 87 us, 102 with two).
__global__ void __launch_bounds__(256, 5)
swiglu_bwd_kernel(const elem_t* __restrict__ gu, const elem_t* __restrict__ dout, elem_t* __restrict__ dgu,
                  long long total, int F, const FastDiv div) {
  const long long step = (long long)gridDim.x * 256;
  for (long long i = blockIdx.x * 256ll + threadIdx.x; i < total; i += step) {
    long long r;
    int c;
    div(i, r, c);
    const long long at = r * 2 * F + c * 8;
    const bf16x8 rg = load_raw(gu + at), ru = load_raw(gu + at + F), rd = load_raw(dout + i * 8);
    float g[8], v[8], d[8], dg[8], du[8];
    unpack8(rg, g);
    unpack8(ru, v);
    unpack8(rd, d);
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      const float s = sigmoidf_(g[j]);
      dg[j] = d[j] * v[j] * (s + g[j] * s * (1.f - s));
      du[j] = d[j] * g[j] * s;
    }
    store8(dgu + at, dg);
    store8(dgu + at + F, du);
  }
}

// tanh-approximated GELU on x (+ bias[n]) ; mode 0 fwd: y = gelu(x+b); mode 1 bwd: y = dy * gelu'(x+b)
__global__ void gelu_kernel(const elem_t* __restrict__ x, const elem_t* __restrict__ bias,
                            const elem_t* __restrict__ dy, elem_t* __restrict__ y, long long rows,
                            int N, int mode) {
  const int vecs = N / 8;
  const long long total = rows * vecs;
  constexpr float k0 = 0.7978845608028654f, k1 = 0.044715f;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < total;
       i += (long long)gridDim.x * blockDim.x) {
    const int c = (i % vecs) * 8;
    float v[8], o[8], b[8], d[8];
    load8(x + i * 8, v);
    if (bias) {
      load8(bias + c, b);
#pragma unroll
      for (int j = 0; j < 8; ++j) v[j] += b[j];
    }
    if (mode == 1) load8(dy + i * 8, d);
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      const float t = tanhf(k0 * (v[j] + k1 * v[j] * v[j] * v[j]));
      if (mode == 0) {
        o[j] = 0.5f * v[j] * (1.f + t);
      } else {
        const float dt = (1.f - t * t) * k0 * (1.f + 3.f * k1 * v[j] * v[j]);
        o[j] = d[j] * (0.5f * (1.f + t) + 0.5f * v[j] * dt);
      }
    }
    store8(y + i * 8, o);
  }
}

static inline int ew_grid(long long work_items, int threads) {
  long long b = (work_items + threads - 1) / threads;
  const long long cap = static_cast<long long>(sm_count()) * 8;
  return static_cast<int>(b < 1 ? 1 : (b > cap ? cap : b));
}

}  // namespace MSB_ELEM_NS
}  // namespace msb

using namespace msb;
using namespace msb::MSB_ELEM_NS;

#define MSB_NORM_DISPATCH(V, CALL) \
  do {                             \
    if ((V) == 1) { CALL(1); }     \
    else if ((V) == 2) { CALL(2); } \
    else if ((V) == 3) { CALL(3); } \
    else { CALL(4); }              \
  } while (0)

static int check_h(const char* what, int H) {
  if (H <= 0 || (H % 8) != 0 || H > 8 * kNormMaxV * kNormMaxThreads) {
    set_last_error("%s: hidden size %d must be a positive multiple of 8 and <= %d", what, H,
                   8 * kNormMaxV * kNormMaxThreads);
    return kBadArg;
  }
  return kOk;
}

// Blocks of a backward kernel: as many as are resident (`threads` per SM at the kernel's registers), fewer where the rows
// run out.  The scratch holds a partial row for each.
static int norm_bwd_grid(long long rows, const NormShape& n, int threads) {
  int per = threads / (n.T * n.R);
  per = per < 1 ? 1 : (per > kNormBwdPerSm ? kNormBwdPerSm : per);
  const long long need = (rows + n.R - 1) / n.R, cap = (long long)per * sm_count();
  return (int)(need < cap ? need : cap);
}
constexpr int kRmsBwdThreads = 1024, kLnBwdThreads = 768;

MSB_EXPORT int MSB_FN(msb_rmsnorm_fwd)(const void* x, const void* res, const void* w, void* y, void* xsum, float* rstd,
                               long long rows, int H, float eps, void* stream) {
  if (int rc = check_h("rmsnorm_fwd", H)) return rc;
  if (rows <= 0) return kOk;
  const NormShape n = norm_fwd_shape(H);
#define CALL(V_)                                                                                         \
  rmsnorm_fwd_kernel<V_><<<(unsigned)((rows + n.R - 1) / n.R), n.T * n.R, 0, (cudaStream_t)stream>>>(      \
      (const elem_t*)x, (const elem_t*)res, (const elem_t*)w, (elem_t*)y,    \
      (elem_t*)xsum, rstd, rows, H, eps, n.T, n.R)
  MSB_NORM_DISPATCH(n.V, CALL);
#undef CALL
  MSB_CUDA_CHECK(cudaGetLastError());
  return kOk;
}

// dw_out (bf16 or fp32 by dw_fp32) receives (accumulate ? dw_out + dw : dw), dw = sum_rows dy * xhat.
// Floats of scratch the norm backward launchers need for hidden size H: one partial row per CTA.
#ifndef MSB_ELEM_FP16
MSB_EXPORT long long msb_norm_bwd_scratch_elems(int H, int with_bias) {
  return (long long)kNormBwdPerSm * sm_count() * H * (with_bias ? 2 : 1);
}
#endif

// dw_acc: fp32 scratch of msb_norm_bwd_scratch_elems(H, 0) floats (per-CTA partial rows; nothing needs clearing).
MSB_EXPORT int MSB_FN(msb_rmsnorm_bwd)(const void* dy, const void* x, const void* w, const float* rstd, const void* dres,
                               void* dx, float* dw_acc, void* dw_out, int dw_fp32, int accumulate, long long rows,
                               int H, void* stream_) {
  if (int rc = check_h("rmsnorm_bwd", H)) return rc;
  cudaStream_t stream = (cudaStream_t)stream_;
  int grid = 0;
  if (rows > 0) {
    const NormShape n = norm_bwd_shape(H);
    grid = norm_bwd_grid(rows, n, kRmsBwdThreads);
#define CALL(V_)                                                                                     \
  rmsnorm_bwd_kernel<V_, false><<<grid, n.T * n.R, n.R > 1 ? H * 4 : 0, stream>>>(                    \
      (const elem_t*)dy, (const elem_t*)x, (const elem_t*)w, rstd,              \
      (const elem_t*)dres, (elem_t*)dx, dw_acc, rows, H, n.T, n.R)
    MSB_NORM_DISPATCH(n.V, CALL);
#undef CALL
  }
  if (dw_out) {
    const PartialsOut dw = {dw_acc, dw_fp32 ? nullptr : (elem_t*)dw_out, dw_fp32 ? (float*)dw_out : nullptr};
    reduce_partials_kernel<<<(H + 31) / 32, 256, 0, stream>>>(dw, dw, grid, H, accumulate);
  }
  MSB_CUDA_CHECK(cudaGetLastError());
  return kOk;
}

MSB_EXPORT int MSB_FN(msb_layernorm_fwd)(const void* x, const void* w, const void* b, void* y, float* mean, float* rstd,
                                 long long rows, int H, float eps, void* stream) {
  if (int rc = check_h("layernorm_fwd", H)) return rc;
  if (rows <= 0) return kOk;
  const NormShape n = norm_fwd_shape(H);
#define CALL(V_)                                                                                         \
  layernorm_fwd_kernel<V_><<<(unsigned)((rows + n.R - 1) / n.R), n.T * n.R, 0, (cudaStream_t)stream>>>(    \
      (const elem_t*)x, (const elem_t*)w, (const elem_t*)b, (elem_t*)y, mean, rstd, rows, H, eps, n.T, n.R)
  MSB_NORM_DISPATCH(n.V, CALL);
#undef CALL
  MSB_CUDA_CHECK(cudaGetLastError());
  return kOk;
}

// acc: fp32 scratch of msb_norm_bwd_scratch_elems(H, 1) floats: per-CTA partial rows of dw, then those of db.
MSB_EXPORT int MSB_FN(msb_layernorm_bwd)(const void* dy, const void* x, const void* w, const float* mean, const float* rstd,
                                 void* dx, float* acc, void* dw_out, void* db_out, int out_fp32, int accumulate,
                                 long long rows, int H, void* stream_) {
  if (int rc = check_h("layernorm_bwd", H)) return rc;
  cudaStream_t stream = (cudaStream_t)stream_;
  int grid = 0;
  float* db_part = acc + (long long)kNormBwdPerSm * sm_count() * H;
  if (rows > 0) {
    const NormShape n = norm_bwd_shape(H);
    grid = norm_bwd_grid(rows, n, kLnBwdThreads);
#define CALL(V_)                                                                                  \
  layernorm_bwd_kernel<V_><<<grid, n.T * n.R, n.R > 1 ? H * 4 : 0, stream>>>(                      \
      (const elem_t*)dy, (const elem_t*)x, (const elem_t*)w, mean, rstd,     \
      (elem_t*)dx, acc, db_out ? db_part : nullptr, rows, H, n.T, n.R)
    MSB_NORM_DISPATCH(n.V, CALL);
#undef CALL
  }
  const PartialsOut dw = {acc, out_fp32 ? nullptr : (elem_t*)dw_out, out_fp32 ? (float*)dw_out : nullptr};
  const PartialsOut db = {db_part, out_fp32 ? nullptr : (elem_t*)db_out, out_fp32 ? (float*)db_out : nullptr};
  if (dw_out && db_out)
    reduce_partials_kernel<<<dim3((H + 31) / 32, 2), 256, 0, stream>>>(dw, db, grid, H, accumulate);
  else if (dw_out || db_out)
    reduce_partials_kernel<<<(H + 31) / 32, 256, 0, stream>>>(dw_out ? dw : db, db, grid, H, accumulate);
  MSB_CUDA_CHECK(cudaGetLastError());
  return kOk;
}

// Rotates src into dst; the two may be the same tensor.
MSB_EXPORT int MSB_FN(msb_rope_to)(const void* src, void* dst, const float* cosb, const float* sinb, const int* pos,
                        long long tokens, int heads, int D, long long src_pitch, long long dst_pitch, int seq,
                        int backward, void* stream) {
  if (D % 16 != 0 || src_pitch % 8 != 0 || dst_pitch % 8 != 0) {
    set_last_error("rope: head dim %d must be a multiple of 16 and pitches %lld, %lld multiples of 8", D, src_pitch,
                   dst_pitch);
    return kBadArg;
  }
  if (tokens * heads * (D / 16) <= 0) return kOk;
  const int vph = D / 16, lanes = vph < kRopeThreads ? vph : kRopeThreads;
  int hstep = kRopeThreads / lanes;
  if (hstep > heads) hstep = heads;
  const int threads = (lanes * hstep + 31) / 32 * 32;
  const int aligned = ((reinterpret_cast<uintptr_t>(cosb) | reinterpret_cast<uintptr_t>(sinb)) & 15) == 0;
  rope_kernel<<<(unsigned)tokens, threads, 0, (cudaStream_t)stream>>>((const elem_t*)src, (elem_t*)dst, cosb, sinb, pos,
                                                                      heads, D, src_pitch, dst_pitch, seq,
                                                                      backward ? -1.f : 1.f, lanes, hstep, aligned);
  MSB_CUDA_CHECK(cudaGetLastError());
  return kOk;
}
MSB_EXPORT int MSB_FN(msb_rope)(void* x, const float* cosb, const float* sinb, const int* pos, long long tokens, int heads,
                        int D, long long pitch, int seq, int backward, void* stream) {
  return MSB_FN(msb_rope_to)(x, x, cosb, sinb, pos, tokens, heads, D, pitch, pitch, seq, backward, stream);
}

MSB_EXPORT int MSB_FN(msb_swiglu_fwd)(const void* gu, void* out, long long rows, int F, void* stream) {
  if (F % 8 != 0) { set_last_error("swiglu: F=%d must be a multiple of 8", F); return kBadArg; }
  if (rows <= 0 || F <= 0) return kOk;
  const long long total = rows * (F / 8);
  swiglu_fwd_kernel<<<ew_grid((total + 1) / 2, 256), 256, 0, (cudaStream_t)stream>>>(
      (const elem_t*)gu, (elem_t*)out, total, F, fast_div(F / 8, total));
  MSB_CUDA_CHECK(cudaGetLastError());
  return kOk;
}
MSB_EXPORT int MSB_FN(msb_swiglu_bwd)(const void* gu, const void* dout, void* dgu, long long rows, int F, void* stream) {
  if (F % 8 != 0) { set_last_error("swiglu: F=%d must be a multiple of 8", F); return kBadArg; }
  if (rows <= 0 || F <= 0) return kOk;
  const long long total = rows * (F / 8);
  swiglu_bwd_kernel<<<ew_grid(total, 256), 256, 0, (cudaStream_t)stream>>>(
      (const elem_t*)gu, (const elem_t*)dout, (elem_t*)dgu, total, F, fast_div(F / 8, total));
  MSB_CUDA_CHECK(cudaGetLastError());
  return kOk;
}
MSB_EXPORT int MSB_FN(msb_gelu)(const void* x, const void* bias, const void* dy, void* y, long long rows, int N, int backward,
                        void* stream) {
  if (N % 8 != 0) { set_last_error("gelu: N=%d must be a multiple of 8", N); return kBadArg; }
  if (rows <= 0) return kOk;
  gelu_kernel<<<ew_grid(rows * (N / 8), 256), 256, 0, (cudaStream_t)stream>>>(
      (const elem_t*)x, (const elem_t*)bias, (const elem_t*)dy, (elem_t*)y, rows, N,
      backward);
  MSB_CUDA_CHECK(cudaGetLastError());
  return kOk;
}

#ifndef MSB_ELEM_FP16
// ----------------------------------------------------------------------------------------------------------------
// RMSNorm backward without any allocation (declared in no_alloc.h): the [H] fp32 weight-gradient accumulator is the
// static device array below.  One array per device (each device holds its own instance of a __device__ variable).
#include "no_alloc.h"

#include <atomic>

static __device__ __align__(256) float g_rmsnorm_bwd_static_acc[MSB_RMSNORM_BWD_STATIC_MAX_H];

namespace {
constexpr int kMaxDevices = 64;
std::atomic<float*> g_static_acc_ptr[kMaxDevices];

// Device address of this device's instance of the array; looked up on the first call per device and kept.
int static_acc_ptr(float** out) {
  int dev = 0;
  MSB_CUDA_CHECK(cudaGetDevice(&dev));
  if (dev < 0 || dev >= kMaxDevices) {
    set_last_error("rmsnorm_bwd_static: device ordinal %d is beyond %d", dev, kMaxDevices - 1);
    return kTooLarge;
  }
  float* p = g_static_acc_ptr[dev].load(std::memory_order_acquire);
  if (p == nullptr) {
    MSB_CUDA_CHECK(cudaGetSymbolAddress((void**)&p, g_rmsnorm_bwd_static_acc));
    if (p == nullptr) {
      set_last_error("rmsnorm_bwd_static: cudaGetSymbolAddress returned a null address");
      return kCudaError;
    }
    g_static_acc_ptr[dev].store(p, std::memory_order_release);
  }
  *out = p;
  return kOk;
}
}  // namespace

MSB_EXPORT int msb_rmsnorm_bwd_static(const void* dy, const void* x, const void* w, const float* rstd,
                                      const void* dres, void* dx, void* dw_out, int dw_fp32, int accumulate,
                                      long long rows, int H, void* stream_) {
  if (H > MSB_RMSNORM_BWD_STATIC_MAX_H) {
    set_last_error("rmsnorm_bwd_static: hidden size %d exceeds the static scratch of %d floats", H,
                   MSB_RMSNORM_BWD_STATIC_MAX_H);
    return kTooLarge;
  }
  if (int rc = check_h("rmsnorm_bwd_static", H)) return rc;
  float* acc = nullptr;
  if (int rc = static_acc_ptr(&acc)) return rc;
  cudaStream_t stream = (cudaStream_t)stream_;
  MSB_CUDA_CHECK(cudaMemsetAsync(acc, 0, sizeof(float) * H, stream));
  if (rows > 0) {
    const NormShape n = norm_bwd_shape(H);
    const int grid = norm_bwd_grid(rows, n, kRmsBwdThreads);
#define CALL(V_)                                                                                     \
  rmsnorm_bwd_kernel<V_, true><<<grid, n.T * n.R, 0, stream>>>(                                       \
      (const elem_t*)dy, (const elem_t*)x, (const elem_t*)w, rstd,              \
      (const elem_t*)dres, (elem_t*)dx, acc, rows, H, n.T, n.R)
    MSB_NORM_DISPATCH(n.V, CALL);
#undef CALL
  }
  if (dw_out) {
    finalize_acc_kernel<<<(H + 255) / 256, 256, 0, stream>>>(acc, dw_fp32 ? nullptr : (elem_t*)dw_out,
                                                             dw_fp32 ? (float*)dw_out : nullptr, H, accumulate);
  }
  MSB_CUDA_CHECK(cudaGetLastError());
  return kOk;
}
#endif  // MSB_ELEM_FP16
