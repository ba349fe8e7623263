// Fused kernels for the decode step (a handful of tokens per launch), where launch count and
// round trips through HBM dominate the time outside the weight-streaming GEMMs:
//   * gdn_decode_fused   - everything between the qkv|z projection and the output projection of a
//                          Gated DeltaNet layer in one launch: the a/b head projections, the gates
//                          g = -exp(A_log) softplus(a + dt_bias) and beta = sigmoid(b), the causal
//                          depth-wise conv step with its tail update, SiLU, L2-normalised q/k, the
//                          gated delta-rule state update and read-out, and the per-head gated RMSNorm;
//   * rmsnorm_split      - residual add + RMSNorm that also emits the activation as E4M3 terms for
//                          the weight-streaming GEMM (gemm_w8a8s.cu), saving the separate split launch;
//   * silu_mul_split     - SwiGLU activation that emits E4M3 terms directly.
// Reference counterparts are separate kernels per step
// (cpp_engine/backends/cuda/kernels/qwen_half_ops.cu: conv_silu_f16_batched :2233, linear_gates_f16 :2265,
//  gated_delta_step_batched_f16 :2350, gated_rmsnorm_f16 :2163, residual_add_rmsnorm_f16 :2072, silu_mul_f16 :2741).
#include <cuda_bf16.h>
#include <cuda_fp8.h>
#include <stdint.h>
#include "fp8_terms.cuh"
#include "ops.h"
#include "launch.h"
#include "per_device.h"
#include "tma_host.h"

namespace {

constexpr int DK = 128, DV = 128;

__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}
__device__ __forceinline__ float warp_max(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
  return v;
}
__device__ __forceinline__ float silu_f(float x) { return x / (1.f + __expf(-x)); }
__device__ __forceinline__ float sigmoid_f(float x) { return 1.f / (1.f + __expf(-x)); }
__device__ __forceinline__ float bf16_round(float x) { return __bfloat162float(__float2bfloat16(x)); }

struct GdnDecodeParams {
  const __nv_bfloat16* proj;   // [B, ldp]: q | k | v | z  (q at 0, k at kd, v at 2kd, z at 2kd + vd)
  int ldp;
  const __nv_bfloat16* x;      // [B, hidden] normed layer input (for the a/b projections)
  int hidden;
  const __nv_bfloat16* w_ab;   // [2*Hv, hidden]: rows 0..Hv-1 = a, Hv..2Hv-1 = b
  const float* a_log;          // [Hv]
  const float* dt_bias;        // [Hv]
  const __nv_bfloat16* conv_w; // [C, KW], C = 2kd + vd
  __nv_bfloat16* tails;        // [slots, KW-1, C]
  size_t tail_stride;
  float* states;               // [slots, Hv, 128, 128] at slot_stride
  size_t state_stride;
  const int* slot_ids;         // [B] or null
  const __nv_bfloat16* gamma;  // [128] gated-norm weight
  __nv_bfloat16* out;          // [B, Hv*128]
  int Hv, Hk;
  float eps, q_scale;
  bool vec;                    // rows, tails and the small weights lie on 16-byte boundaries
  int B;
  bool ahead;                  // several rows a block: dynamic shared memory for the next state, and for the a / b weights if `keep_w`
  bool keep_w;
  b200::f8t::TermsOut terms;   // where the result goes as FP8 terms (xq set) instead of `out`: a head is one block of 128
};

// 128 bf16 values on their way to shared memory, 8 a thread; `vec`: 16 bytes at a time (cp.async), else one by one.
__device__ __forceinline__ void copy8(__nv_bfloat16* dst, const __nv_bfloat16* src, bool vec) {
  if (vec) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src) : "memory");
  } else {
#pragma unroll
    for (int i = 0; i < 8; ++i) dst[i] = src[i];
  }
}

// grid (Hv, row groups), clusters of the R = Hv / Hk value heads that share a key head; block = 128 * RG threads.  Thread (rg, j) owns
// rows [rg*128/RG, (rg+1)*128/RG) of column j of the head's state; the row groups cut the serial length of the recurrence per
// thread, their partial dot products meet in shared memory.
//
// What a step costs beside the state's 64 KB in and out per head is a chain of loads and barriers, so everything small - the
// projection's row, the convolution's tails and weights, the norm's weight - is asked for at once, straight to shared memory.  Two blocks
// fit an SM; with more rows than these hold a block walks several rows of its head, the constants stay, and the next row's state
// and small inputs are on their way while one is computed.  A few rows ask L2 for the a / b weights even before the previous kernel has
// ended.  us a layer of 32 heads: 1 row 10.7, 16 rows 17, 32 rows 29, 64 rows 53.5 (the state's bytes take 0.7, 10, 21, 42); with each
// input loaded where it is used and a row per block 1 row took 13.7, 32 rows 43, 64 rows 85.  (A cluster arrival with release, which waits
// for the row before's state to reach memory: 34.5 and 68 for 32 and 64 rows.)
// Every block convolves the q and k channels of its key head itself; the first of the cluster moves their tail on when all of
// them have read it.
template <int KW, int R, int RG>
__global__ void __launch_bounds__(128 * RG, 2)
gdn_decode_fused_kernel(GdnDecodeParams p) {
  static_assert(KW == 4 && RG == 4, "three rows of tail; row groups for q, k, v and the gates");
  constexpr int ROWS = DK / RG;
  constexpr int WARPS = 4 * RG;
  __shared__ __align__(16) float sq[DK], sk[DK], s_v[DV];
  __shared__ __align__(16) float s_part[2][RG][DV];
  __shared__ float red_ab[WARPS][2];
  __shared__ float red_qk[8];
  __shared__ float red_o[4];
  __shared__ float s_gate[2];
  __shared__ __align__(16) __nv_bfloat16 s_rows[2][4][128], s_tails[2][3][KW - 1][128], s_cw[3][128 * KW], s_gamma[128];   // q, k, v (, z)
  __shared__ uint64_t s_bar;
  extern __shared__ __align__(128) uint8_t dyn[];
  float* s_state = reinterpret_cast<float*>(dyn);
  __nv_bfloat16* s_w = reinterpret_cast<__nv_bfloat16*>(dyn + DK * DV * 4);
  const int h = blockIdx.x, kh = h / R, tid = threadIdx.x;
  const int j = tid & 127, rg = tid >> 7;
  const int kd = p.Hk * DK, vd = p.Hv * DV, C = 2 * kd + vd;
  auto chan = [&](int c) { return c == 0 ? kh * DK : c == 1 ? kd + kh * DK : 2 * kd + h * DV; };
  b200::pdl_grid_trigger();
  // constants do not wait for the previous kernel
  if (tid < 3 * 64) copy8(s_cw[tid >> 6] + (tid & 63) * 8, p.conv_w + (size_t)chan(tid >> 6) * KW + (tid & 63) * 8, p.vec);
  else if (tid < 3 * 64 + 16) copy8(s_gamma + (tid - 3 * 64) * 8, p.gamma + (tid - 3 * 64) * 8, p.vec);
  float a_log = 0.f, dt_bias = 0.f;
  if (tid == 3 * 128) {
    a_log = p.a_log[h];
    dt_bias = p.dt_bias[h];
  }
  const __nv_bfloat16* wa = p.w_ab + (size_t)h * p.hidden;
  const __nv_bfloat16* wb = p.w_ab + (size_t)(p.Hv + h) * p.hidden;
  if (p.keep_w) {
    for (int i = tid * 8; i < p.hidden; i += 128 * RG * 8) {
      copy8(s_w + i, wa + i, true);
      copy8(s_w + p.hidden + i, wb + i, true);
    }
    wa = s_w;
    wb = s_w + p.hidden;
  } else if (gridDim.y <= 4) {
    for (int i = tid * 64; i < p.hidden; i += 128 * RG * 64) {
      asm volatile("prefetch.global.L2 [%0];" ::"l"(wa + i));
      asm volatile("prefetch.global.L2 [%0];" ::"l"(wb + i));
    }
  }
  if (p.ahead && tid == 0) {
    b200::mbar_init(&s_bar, 1);
    b200::mbar_fence_init();
  }
  b200::pdl_grid_wait();
  p.terms.zero_counters(blockIdx.x == 0 && blockIdx.y == 0);
  auto slot_of = [&](int b) { return p.slot_ids ? p.slot_ids[b] : b; };
  auto ask = [&](int b, int slot, int buf) {                // 13 pieces of 128 values: the row's four, the tails' nine
    const __nv_bfloat16* row = p.proj + (size_t)b * p.ldp;
    const __nv_bfloat16* tail = p.tails + (size_t)slot * p.tail_stride;
    const int part = tid >> 4, i = (tid & 15) * 8;
    if (part < 4) {
      copy8(s_rows[buf][part] + i, row + (part < 3 ? chan(part) : C + h * DV) + i, p.vec);
    } else if (part < 13) {
      const int c = (part - 4) / 3, k = (part - 4) % 3;
      copy8(s_tails[buf][c][k] + i, tail + (size_t)k * C + chan(c) + i, p.vec);
    }
  };
  int slot = slot_of(blockIdx.y);
  ask(blockIdx.y, slot, 0);
  for (int b = blockIdx.y, round = 0; b < p.B; b += gridDim.y, ++round) {
  const int buf = round & 1, nb = b + gridDim.y;
  const int next_slot = nb < p.B ? slot_of(nb) : 0;
  __nv_bfloat16* tail = p.tails + (size_t)slot * p.tail_stride;
  const auto& s_row = s_rows[buf];
  const auto& s_tail = s_tails[buf];
  float* S = p.states + (size_t)slot * p.state_stride + (size_t)h * DK * DV + (size_t)rg * ROWS * DV;
  const __nv_bfloat16* xr = p.x + (size_t)b * p.hidden;
  uint4 xv = make_uint4(0, 0, 0, 0), xw = xv;              // the first two pieces of the row, asked for before the state is waited for
  if (tid * 8 < p.hidden) xv = *reinterpret_cast<const uint4*>(xr + tid * 8);
  if (tid * 8 + 128 * RG * 8 < p.hidden) xw = *reinterpret_cast<const uint4*>(xr + tid * 8 + 128 * RG * 8);
  float col[ROWS];
  if (round > 0 && b200::mbar_wait(&s_bar, (round - 1) & 1)) {
#pragma unroll
    for (int i = 0; i < ROWS; ++i) col[i] = s_state[(rg * ROWS + i) * DV + j];
  } else {
#pragma unroll
    for (int i = 0; i < ROWS; ++i) col[i] = S[(size_t)i * DV + j];
  }
  if (round == 0 && p.keep_w) {          // the a / b weights are read before the first barrier below
    asm volatile("cp.async.wait_all;" ::: "memory");
    __syncthreads();
  }

  // ---- a/b projections of this value head: two dot products of length hidden
  {
    float da = 0.f, db = 0.f;
    for (int i = tid * 8; i < p.hidden; i += 128 * RG * 8) {
      if (i >= 2 * 128 * RG * 8) xv = *reinterpret_cast<const uint4*>(xr + i);
      const uint4 av = *reinterpret_cast<const uint4*>(wa + i);
      const uint4 bv = *reinterpret_cast<const uint4*>(wb + i);
      const __nv_bfloat162* xh = reinterpret_cast<const __nv_bfloat162*>(&xv);
      const __nv_bfloat162* ah = reinterpret_cast<const __nv_bfloat162*>(&av);
      const __nv_bfloat162* bh = reinterpret_cast<const __nv_bfloat162*>(&bv);
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const float2 xf = __bfloat1622float2(xh[e]), af = __bfloat1622float2(ah[e]), bf = __bfloat1622float2(bh[e]);
        da += xf.x * af.x + xf.y * af.y;
        db += xf.x * bf.x + xf.y * bf.y;
      }
      xv = xw;
    }
    da = warp_sum(da);
    db = warp_sum(db);
    if ((j & 31) == 0) {
      red_ab[tid >> 5][0] = da;
      red_ab[tid >> 5][1] = db;
    }
  }
  if (p.vec) asm volatile("cp.async.wait_all;" ::: "memory");
  __syncthreads();
  if (nb < p.B) {
    if (tid == 0) {
      b200::fence_proxy_async_smem();    // every thread has its share of this state
      b200::mbar_expect_tx(&s_bar, DK * DV * 4);
      b200::bulk_load(s_state, p.states + (size_t)next_slot * p.state_stride + (size_t)h * DK * DV, DK * DV * 4, &s_bar);
    }
    ask(nb, next_slot, buf ^ 1);
  }
  // This block has read its tails: they are in shared memory.  Nothing else is published, and a release would wait for the previous row's
  // state to reach memory.
  if constexpr (R > 1) asm volatile("barrier.cluster.arrive.relaxed.aligned;" ::: "memory");
  if (rg < 3) {                            // a row group each for q, k and v
    // y = silu(sum_k w[c][k] * v[k]), rounded as the unfused path stores it
    auto conv = [&](int c) {
      float acc = __bfloat162float(s_row[c][j]) * __bfloat162float(s_cw[c][j * KW + KW - 1]);
#pragma unroll
      for (int k = 0; k < KW - 1; ++k) acc += __bfloat162float(s_tail[c][k][j]) * __bfloat162float(s_cw[c][j * KW + k]);
      return bf16_round(silu_f(acc));
    };
    const float y = conv(rg);
    if (rg == 2) {
      s_v[j] = y;
    } else {
      const float ss = warp_sum(y * y);
      if ((j & 31) == 0) red_qk[tid >> 5] = ss;
      asm volatile("bar.sync %0, 128;" ::"r"(1 + rg) : "memory");
      const float* red = red_qk + 4 * rg;
      const float n = rsqrtf(red[0] + red[1] + red[2] + red[3] + 1e-6f);
      if (rg == 0) sq[j] = y * n * p.q_scale;
      else sk[j] = y * n;
    }
  } else if (tid == 3 * 128) {
    float a = 0.f, bb = 0.f;
#pragma unroll
    for (int w = 0; w < WARPS; ++w) {
      a += red_ab[w][0];
      bb += red_ab[w][1];
    }
    // the unfused path rounds the a/b projection outputs to bf16 before the gate math
    a = bf16_round(a);
    bb = bf16_round(bb);
    const float av = a + dt_bias;
    const float sp = av > 20.f ? av : log1pf(expf(av));
    s_gate[0] = __expf(-expf(a_log) * sp);   // decay = exp(g)
    s_gate[1] = sigmoid_f(bb);
  }
  if (rg == 3 && tid >= 3 * 128 + 32) {
    // the value channels' tail, this block's own, moves on
    for (int c = j - 32; c < DV; c += 96)
#pragma unroll
      for (int k = 0; k < KW - 1; ++k) tail[(size_t)k * C + chan(2) + c] = k + 1 < KW - 1 ? s_tail[2][k + 1][c] : s_row[2][c];
  }
  __syncthreads();
  // ---- gated delta rule on rows [rg*ROWS, (rg+1)*ROWS) of state column j
  const float decay = s_gate[0], bt = s_gate[1];
  float part = 0.f;
#pragma unroll
  for (int i = 0; i < ROWS; i += 4) {      // four keys a read: one at a time, the reads are half of what shared memory has to do
    const float4 k4 = *reinterpret_cast<const float4*>(sk + rg * ROWS + i);
    const float kk[4] = {k4.x, k4.y, k4.z, k4.w};
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      col[i + e] *= decay;
      part += col[i + e] * kk[e];
    }
  }
  s_part[0][rg][j] = part;
  __syncthreads();
  float kv_mem = 0.f;
#pragma unroll
  for (int g2 = 0; g2 < RG; ++g2) kv_mem += s_part[0][g2][j];
  const float delta = (s_v[j] - kv_mem) * bt;
  part = 0.f;
#pragma unroll
  for (int i = 0; i < ROWS; i += 4) {
    const float4 k4 = *reinterpret_cast<const float4*>(sk + rg * ROWS + i), q4 = *reinterpret_cast<const float4*>(sq + rg * ROWS + i);
    const float kk[4] = {k4.x, k4.y, k4.z, k4.w}, qq[4] = {q4.x, q4.y, q4.z, q4.w};
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      col[i + e] += kk[e] * delta;
      S[(size_t)(i + e) * DV + j] = col[i + e];
      part += col[i + e] * qq[e];
    }
  }
  s_part[1][rg][j] = part;
  if constexpr (R > 1) asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");   // every head has read the q and k tails
  if (rg == RG - 1 && h % R == 0) {
#pragma unroll
    for (int c = 0; c < 2; ++c)
#pragma unroll
      for (int k = 0; k < KW - 1; ++k) tail[(size_t)k * C + chan(c) + j] = k + 1 < KW - 1 ? s_tail[c][k + 1][j] : s_row[c][j];
  }
  __syncthreads();
  slot = next_slot;
  if (rg != 0) continue;
  // ---- per-head gated RMSNorm by row group 0 (the unfused path stores o as bf16 first)
  float o = 0.f;
#pragma unroll
  for (int g2 = 0; g2 < RG; ++g2) o += s_part[1][g2][j];
  o = bf16_round(o);
  const float ss = warp_sum(o * o);
  if ((j & 31) == 0) red_o[j >> 5] = ss;
  asm volatile("bar.sync 1, 128;" ::: "memory");
  const float inv = rsqrtf((red_o[0] + red_o[1] + red_o[2] + red_o[3]) / (float)DV + p.eps);
  const float z = __bfloat162float(s_row[3][j]);
  const float y = bf16_round(o * inv * __bfloat162float(s_gamma[j]) * silu_f(z));
  if (!p.terms.xq) {
    p.out[((size_t)b * p.Hv + h) * DV + j] = __float2bfloat16(y);
    continue;
  }
  s_part[0][0][j] = y;
  asm volatile("bar.sync 1, 128;" ::: "memory");
  if (j < 32) {
    const float4 f = *reinterpret_cast<const float4*>(&s_part[0][0][j * 4]);
    const float v[4] = {f.x, f.y, f.z, f.w};
    b200::f8t::put_terms(p.terms, b, h * DV + j * 4, v, true);
  }
  }
}

template <int R>
static int launch_gdn(GdnDecodeParams p, int B, cudaStream_t stream) {
  // rows a block walks: as few as two blocks per SM allow, shared evenly
  const bool walk = (reinterpret_cast<uintptr_t>(p.states) & 15) == 0 && p.state_stride % 4 == 0;
  const int groups = 2 * b200::sm_count() / p.Hv, rounds = !walk || groups < 1 ? 1 : (B + groups - 1) / groups;
  p.B = B;
  p.ahead = rounds > 1;
  p.keep_w = p.ahead && p.vec && p.hidden <= 6144;         // 2 x 12 KB beside the state, twice an SM
  const int smem = p.ahead ? DK * DV * 4 + (p.keep_w ? p.hidden * 4 : 0) : 0;
  if (p.ahead) {
    static b200::PerDeviceOnce once_;
    bool& configured = once_.slot();
    if (!configured) {
      const cudaError_t e = cudaFuncSetAttribute(gdn_decode_fused_kernel<4, R, 4>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                                 DK * DV * 4 + 6144 * 4);
      if (e != cudaSuccess) return (int)e;
      configured = true;
    }
  }
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(p.Hv, (B + rounds - 1) / rounds);
  cfg.dynamicSmemBytes = smem;
  cfg.blockDim = dim3(512);
  cfg.stream = stream;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  attr[1].id = cudaLaunchAttributeClusterDimension;
  attr[1].val.clusterDim.x = R;
  attr[1].val.clusterDim.y = 1;
  attr[1].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = R > 1 ? 2 : 1;
  return (int)cudaLaunchKernelEx(&cfg, gdn_decode_fused_kernel<4, R, 4>, p);
}

// ------------------------------------------------------------------------------------------------
// E4M3 term split of one value already scaled by the row scale; byte order (x0,x2,x1,x3) per 4 values.
template <int TERMS>
__device__ __forceinline__ void split4_store(float (&v)[4], uint8_t* xq_row0, size_t term_stride, int i) {
#pragma unroll
  for (int t = 0; t < TERMS; ++t) {
    uint8_t q[4];
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const __nv_fp8_e4m3 f8(v[e]);
      q[e] = f8.__x;
      v[e] = (v[e] - float(f8)) * 16.f;
    }
    *reinterpret_cast<uint32_t*>(xq_row0 + t * term_stride + i) =
        (uint32_t)q[0] | ((uint32_t)q[2] << 8) | ((uint32_t)q[1] << 16) | ((uint32_t)q[3] << 24);
  }
}

__device__ __forceinline__ float block_max(float v, float* red) {
  v = warp_max(v);
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  __syncthreads();
  if (lane == 0) red[w] = v;
  __syncthreads();
  const int nw = (blockDim.x + 31) >> 5;
  float t = (threadIdx.x < nw) ? red[threadIdx.x] : 0.f;
  if (w == 0) {
    t = warp_max(t);
    if (lane == 0) red[0] = t;
  }
  __syncthreads();
  t = red[0];
  __syncthreads();
  return t;
}
__device__ __forceinline__ float block_sum2(float v, float* red) {
  v = warp_sum(v);
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  __syncthreads();
  if (lane == 0) red[w] = v;
  __syncthreads();
  const int nw = (blockDim.x + 31) >> 5;
  float t = (threadIdx.x < nw) ? red[threadIdx.x] : 0.f;
  if (w == 0) {
    t = warp_sum(t);
    if (lane == 0) red[0] = t;
  }
  __syncthreads();
  t = red[0];
  __syncthreads();
  return t;
}

// One block per row, 4 values per thread per step; cols % 4 == 0, cols <= 4 * MAXV * blockDim.
template <int MAXV, int TERMS>
__global__ void rmsnorm_split_kernel(__nv_bfloat16* __restrict__ x, const __nv_bfloat16* __restrict__ delta,
                                     const __nv_bfloat16* __restrict__ gamma, __nv_bfloat16* __restrict__ out,
                                     uint8_t* __restrict__ xq, float* __restrict__ inv_c, int cols, float eps,
                                     int unit_offset) {
  __shared__ float red[32];
  b200::pdl_grid_trigger();   // the GEMM that follows may start streaming its weights now
  b200::pdl_grid_wait();
  const size_t row = blockIdx.x;
  float cache[MAXV][4];
  float ss = 0.f;
#pragma unroll
  for (int it = 0; it < MAXV; ++it) {
    const int i = (threadIdx.x + it * blockDim.x) * 4;
    if (i < cols) {
      const uint2 u = *reinterpret_cast<const uint2*>(x + row * cols + i);
      const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&u);
      float2 a = __bfloat1622float2(h[0]), b = __bfloat1622float2(h[1]);
      if (delta) {
        const uint2 d = *reinterpret_cast<const uint2*>(delta + row * cols + i);
        const __nv_bfloat162* dh = reinterpret_cast<const __nv_bfloat162*>(&d);
        const float2 da = __bfloat1622float2(dh[0]), db = __bfloat1622float2(dh[1]);
        // the residual stream is bf16: round first so the norm input equals the stored residual
        uint2 r;
        __nv_bfloat162* rh = reinterpret_cast<__nv_bfloat162*>(&r);
        rh[0] = __floats2bfloat162_rn(a.x + da.x, a.y + da.y);
        rh[1] = __floats2bfloat162_rn(b.x + db.x, b.y + db.y);
        *reinterpret_cast<uint2*>(x + row * cols + i) = r;
        a = __bfloat1622float2(rh[0]);
        b = __bfloat1622float2(rh[1]);
      }
      cache[it][0] = a.x; cache[it][1] = a.y; cache[it][2] = b.x; cache[it][3] = b.y;
      ss += a.x * a.x + a.y * a.y + b.x * b.x + b.y * b.y;
    }
  }
  const float inv = rsqrtf(block_sum2(ss, red) / (float)cols + eps);
  float m = 0.f;
#pragma unroll
  for (int it = 0; it < MAXV; ++it) {
    const int i = (threadIdx.x + it * blockDim.x) * 4;
    if (i < cols) {
      const uint2 g = *reinterpret_cast<const uint2*>(gamma + i);
      const __nv_bfloat162* gh = reinterpret_cast<const __nv_bfloat162*>(&g);
      const float2 g0 = __bfloat1622float2(gh[0]), g1 = __bfloat1622float2(gh[1]);
      const float gf[4] = {g0.x, g0.y, g1.x, g1.y};
      uint2 r;
      __nv_bfloat162* rh = reinterpret_cast<__nv_bfloat162*>(&r);
      float o[4];
#pragma unroll
      for (int e = 0; e < 4; ++e) o[e] = cache[it][e] * inv * (unit_offset ? 1.f + gf[e] : gf[e]);
      rh[0] = __floats2bfloat162_rn(o[0], o[1]);
      rh[1] = __floats2bfloat162_rn(o[2], o[3]);
      if (out) *reinterpret_cast<uint2*>(out + row * cols + i) = r;
      const float2 q0 = __bfloat1622float2(rh[0]), q1 = __bfloat1622float2(rh[1]);
      cache[it][0] = q0.x; cache[it][1] = q0.y; cache[it][2] = q1.x; cache[it][3] = q1.y;
      m = fmaxf(m, fmaxf(fmaxf(fabsf(q0.x), fabsf(q0.y)), fmaxf(fabsf(q1.x), fabsf(q1.y))));
    }
  }
  m = block_max(m, red);
  const float c = m > 0.f ? 224.f / m : 1.f;
  if (threadIdx.x == 0) inv_c[row] = 1.f / c;
#pragma unroll
  for (int it = 0; it < MAXV; ++it) {
    const int i = (threadIdx.x + it * blockDim.x) * 4;
    if (i < cols) {
      float v[4] = {cache[it][0] * c, cache[it][1] * c, cache[it][2] * c, cache[it][3] * c};
      split4_store<TERMS>(v, xq + row * TERMS * (size_t)cols, (size_t)cols, i);
    }
  }
}

// act[t, i] = silu(gu[t, i]) * gu[t, inter + i]; one block per row; inter % 4 == 0, inter <= 4 * MAXV * blockDim.
template <int MAXV, int TERMS>
__global__ void silu_mul_split_kernel(const __nv_bfloat16* __restrict__ gu, int inter, uint8_t* __restrict__ xq,
                                      float* __restrict__ inv_c) {
  __shared__ float red[32];
  b200::pdl_grid_trigger();   // the GEMM that follows may start streaming its weights now
  b200::pdl_grid_wait();
  const size_t row = blockIdx.x;
  const __nv_bfloat16* g = gu + row * 2 * (size_t)inter;
  const __nv_bfloat16* u = g + inter;
  float cache[MAXV][4];
  float m = 0.f;
#pragma unroll
  for (int it = 0; it < MAXV; ++it) {
    const int i = (threadIdx.x + it * blockDim.x) * 4;
    if (i < inter) {
      const uint2 gv = *reinterpret_cast<const uint2*>(g + i);
      const uint2 uv = *reinterpret_cast<const uint2*>(u + i);
      const __nv_bfloat162* gh = reinterpret_cast<const __nv_bfloat162*>(&gv);
      const __nv_bfloat162* uh = reinterpret_cast<const __nv_bfloat162*>(&uv);
      const float2 g0 = __bfloat1622float2(gh[0]), g1 = __bfloat1622float2(gh[1]);
      const float2 u0 = __bfloat1622float2(uh[0]), u1 = __bfloat1622float2(uh[1]);
      cache[it][0] = bf16_round(silu_f(g0.x) * u0.x);
      cache[it][1] = bf16_round(silu_f(g0.y) * u0.y);
      cache[it][2] = bf16_round(silu_f(g1.x) * u1.x);
      cache[it][3] = bf16_round(silu_f(g1.y) * u1.y);
#pragma unroll
      for (int e = 0; e < 4; ++e) m = fmaxf(m, fabsf(cache[it][e]));
    }
  }
  m = block_max(m, red);
  const float c = m > 0.f ? 224.f / m : 1.f;
  if (threadIdx.x == 0) inv_c[row] = 1.f / c;
#pragma unroll
  for (int it = 0; it < MAXV; ++it) {
    const int i = (threadIdx.x + it * blockDim.x) * 4;
    if (i < inter) {
      float v[4] = {cache[it][0] * c, cache[it][1] * c, cache[it][2] * c, cache[it][3] * c};
      split4_store<TERMS>(v, xq + row * TERMS * (size_t)inter, (size_t)inter, i);
    }
  }
}

}  // namespace

extern "C" {

// proj: [B, ldp] bf16 holding q | k | v | z at offsets 0, kd, 2kd, 2kd+vd (kd = Hk*128, vd = Hv*128);
// x: [B, hidden] bf16; w_ab: [2*Hv, hidden] bf16; conv_w: [2kd+vd, kw] bf16; tails: [slots, kw-1, 2kd+vd] bf16
// (tail_stride elements per slot); states: fp32 [slots, Hv, 128, 128] (state_stride floats per slot);
// out: [B, Hv*128] bf16, or null with the terms_ pointers (gemm.Terms): the result as FP8 terms (gemm_fp8_terms.cu,
// tok tokens per tile, no pair).  Hv / Hk must be 1, 2 or 4 and kw == 4.
int b200_gdn_decode_fused(const void* proj, int ldp, const void* x, int hidden, const void* w_ab, const float* a_log,
                          const float* dt_bias, const void* conv_w, int kw, void* tails, long long tail_stride,
                          float* states, long long state_stride, const int* slot_ids, const void* gamma, void* out,
                          int B, int Hv, int Hk, float eps, void* terms_xq, float* terms_sx, void* terms_rest,
                          int* terms_counters, int tok, cudaStream_t stream) {
  if ((!out && (!terms_xq || !terms_sx || !terms_rest || !terms_counters || tok < B || tok > b200::f8t::MAX_SINGLE)) || B <= 0 || Hv <= 0 || Hk <= 0 || Hv % Hk != 0 || kw != 4 || hidden % 8 != 0) return -6;
  GdnDecodeParams p;
  p.proj = reinterpret_cast<const __nv_bfloat16*>(proj);
  p.ldp = ldp;
  p.x = reinterpret_cast<const __nv_bfloat16*>(x);
  p.hidden = hidden;
  p.w_ab = reinterpret_cast<const __nv_bfloat16*>(w_ab);
  p.a_log = a_log;
  p.dt_bias = dt_bias;
  p.conv_w = reinterpret_cast<const __nv_bfloat16*>(conv_w);
  p.tails = reinterpret_cast<__nv_bfloat16*>(tails);
  p.tail_stride = (size_t)tail_stride;
  p.states = states;
  p.state_stride = (size_t)state_stride;
  p.slot_ids = slot_ids;
  p.gamma = reinterpret_cast<const __nv_bfloat16*>(gamma);
  p.out = reinterpret_cast<__nv_bfloat16*>(out);
  p.Hv = Hv;
  p.Hk = Hk;
  p.eps = eps;
  p.q_scale = rsqrtf((float)DK);
  const uintptr_t all = reinterpret_cast<uintptr_t>(proj) | reinterpret_cast<uintptr_t>(conv_w) | reinterpret_cast<uintptr_t>(tails) |
                        reinterpret_cast<uintptr_t>(gamma);
  p.vec = all % 16 == 0 && ldp % 8 == 0 && tail_stride % 8 == 0;
  p.terms.xq = out ? nullptr : reinterpret_cast<uint8_t*>(terms_xq);
  p.terms.sx = terms_sx;
  p.terms.rest = reinterpret_cast<__nv_bfloat16*>(terms_rest);
  p.terms.counters = terms_counters;
  p.terms.n_counters = out ? 0 : b200::sm_count();
  p.terms.tok = p.terms.cap = tok;
  p.terms.kb = Hv;
  switch (Hv / Hk) {
    case 1: return launch_gdn<1>(p, B, stream);
    case 2: return launch_gdn<2>(p, B, stream);
    case 4: return launch_gdn<4>(p, B, stream);
    default: return -6;
  }
}

// x[T, cols] (+= delta, written back when delta is given) -> out = rmsnorm(x) * gamma (bf16, optional) and the
// E4M3 terms of that bf16 result: xq [T*terms, cols], inv_c [T].  cols % 4 == 0, cols <= 16384.
int b200_rmsnorm_split(void* x, const void* delta, const void* gamma, void* out, void* xq, float* inv_c, int T,
                       int cols, float eps, int unit_offset, int terms, cudaStream_t stream) {
  if (T <= 0 || cols <= 0 || cols % 4 != 0 || cols > 16384 || (terms != 2 && terms != 3)) return -6;
  auto* xp = reinterpret_cast<__nv_bfloat16*>(x);
  auto* dp = reinterpret_cast<const __nv_bfloat16*>(delta);
  auto* gp = reinterpret_cast<const __nv_bfloat16*>(gamma);
  auto* op = reinterpret_cast<__nv_bfloat16*>(out);
  auto* qp = reinterpret_cast<uint8_t*>(xq);
  const int threads = cols <= 4096 ? 256 : 512;
  if (terms == 3)
    return (int)b200::launch_pdl(rmsnorm_split_kernel<8, 3>, dim3(T), dim3(threads), 0, stream, xp, dp, gp, op, qp, inv_c,
                                 cols, eps, unit_offset);
  return (int)b200::launch_pdl(rmsnorm_split_kernel<8, 2>, dim3(T), dim3(threads), 0, stream, xp, dp, gp, op, qp, inv_c,
                               cols, eps, unit_offset);
}

// gu[T, 2*inter] (gate | up) -> E4M3 terms of bf16(silu(gate) * up): xq [T*terms, inter], inv_c [T].
int b200_silu_mul_split(const void* gu, void* xq, float* inv_c, int T, int inter, int terms, cudaStream_t stream) {
  if (T <= 0 || inter <= 0 || inter % 4 != 0 || inter > 4 * 8 * 1024 || (terms != 2 && terms != 3)) return -6;
  auto* gp = reinterpret_cast<const __nv_bfloat16*>(gu);
  auto* qp = reinterpret_cast<uint8_t*>(xq);
  if (terms == 3) return (int)b200::launch_pdl(silu_mul_split_kernel<8, 3>, dim3(T), dim3(1024), 0, stream, gp, inter, qp, inv_c);
  return (int)b200::launch_pdl(silu_mul_split_kernel<8, 2>, dim3(T), dim3(1024), 0, stream, gp, inter, qp, inv_c);
}

}  // extern "C"
