// The a / b projections of a Gated DeltaNet layer and the gates made of them, for prompt portions:
//   a = x Wa^T, b = x Wb^T (rounded to bf16),  g = -exp(A_log) softplus(a + dt_bias),  beta = sigmoid(b).
//
// 64 features for 16 tokens are too little for a tensor-core tile of 128 features, which left one SM per 64 tokens walking all of K
// (20 us at 5120 inputs, then 2 us and a gap for the gates; here 11).  Here a cluster of four CTAs, 32 warps, shares the inputs of 16 tokens
// chunk by chunk of 32, straight from L2 to mma.sync fragments (16 bytes a load: the eight inputs a thread holds serve as its columns
// of two products, for both operands alike), and the partial sums meet in shared memory, then across the cluster, in a fixed order.
// Every cluster reads all weights, 0.65 MB from L2 per 16 tokens, so long portions (2048 tokens and more) stay with the tiled product.
#include <cuda_bf16.h>
#include <stdint.h>
#include "launch.h"
#include "ops.h"

namespace {

constexpr int ROWS = 16, CT = 4, WARPS = 8, MAX_N = 64;

__device__ __forceinline__ void mma_bf16(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
      : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
      : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

__global__ void __cluster_dims__(1, CT, 1) __launch_bounds__(WARPS * 32)
gdn_ab_gates_kernel(const __nv_bfloat16* __restrict__ x, int H, const __nv_bfloat16* __restrict__ w, const float* __restrict__ a_log,
                    const float* __restrict__ dt_bias, float* __restrict__ gate, float* __restrict__ beta, int T, int Hv) {
  __shared__ float part[WARPS][ROWS][MAX_N + 2];     // rows two banks apart: the eight rows of a store do not meet
  __shared__ float sum[ROWS][MAX_N];
  b200::pdl_grid_trigger();
  b200::pdl_grid_wait();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, q = lane & 3;
  const int rank = blockIdx.y, t0 = blockIdx.x * ROWS, N = 2 * Hv;
  float acc[MAX_N / 8][4] = {};
  const uint4 zero = make_uint4(0, 0, 0, 0);
  const __nv_bfloat16* xr = x + (size_t)(t0 + g) * H + 8 * q;
  const __nv_bfloat16* wr = w + (size_t)g * H + 8 * q;
#pragma unroll 2
  for (int c = rank * WARPS + warp; c < H / 32; c += CT * WARPS) {
    const uint4 a = t0 + g < T ? *reinterpret_cast<const uint4*>(xr + c * 32) : zero;
    const uint4 b = t0 + g + 8 < T ? *reinterpret_cast<const uint4*>(xr + (size_t)8 * H + c * 32) : zero;
    uint4 v[MAX_N / 8];
#pragma unroll
    for (int n = 0; n < MAX_N / 8; ++n)
      v[n] = n * 8 + g < N ? __ldg(reinterpret_cast<const uint4*>(wr + (size_t)n * 8 * H + c * 32)) : zero;
#pragma unroll
    for (int n = 0; n < MAX_N / 8; ++n) {
      mma_bf16(acc[n], a.x, b.x, a.y, b.y, v[n].x, v[n].y);
      mma_bf16(acc[n], a.z, b.z, a.w, b.w, v[n].z, v[n].w);
    }
  }
#pragma unroll
  for (int n = 0; n < MAX_N / 8; ++n)
#pragma unroll
    for (int e = 0; e < 4; ++e) part[warp][g + (e >> 1) * 8][n * 8 + 2 * q + (e & 1)] = acc[n][e];
  __syncthreads();
  for (int i = threadIdx.x; i < ROWS * MAX_N; i += WARPS * 32) {
    float s = 0.f;
#pragma unroll
    for (int k = 0; k < WARPS; ++k) s += part[k][i / MAX_N][i % MAX_N];
    sum[i / MAX_N][i % MAX_N] = s;
  }
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
  // each CTA finishes a quarter of the tokens
  static_assert(ROWS / CT * MAX_N == WARPS * 32, "a value per thread");
  const int row = rank * (ROWS / CT) + threadIdx.x / MAX_N, n = threadIdx.x % MAX_N, t = t0 + row;
  const uint32_t local = (uint32_t)__cvta_generic_to_shared(&sum[row][n]);
  float s = 0.f;
#pragma unroll
  for (int r = 0; r < CT; ++r) {
    uint32_t remote;
    float v;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(remote) : "r"(local), "r"(r));
    asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(remote) : "memory");
    s += v;
  }
  if (t < T && n < N) {
    s = __bfloat162float(__float2bfloat16(s));
    if (n < Hv) {
      const float av = s + dt_bias[n];
      const float sp = av > 20.f ? av : log1pf(expf(av));
      gate[(size_t)t * Hv + n] = -expf(a_log[n]) * sp;
    } else {
      beta[(size_t)t * Hv + n - Hv] = 1.f / (1.f + __expf(-s));
    }
  }
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");   // sums are still being read
}

}  // namespace

// x [T, H] bf16, w [2 Hv, H] (a rows, then b rows); g, beta fp32 [T, Hv].  H % 32 == 0, Hv <= 32, all 16-byte aligned.
extern "C" int b200_gdn_ab_gates(const void* x, int H, const void* w, const float* a_log, const float* dt_bias, float* g, float* beta, int T,
                                 int Hv, cudaStream_t stream) {
  if (!x || !w || !a_log || !dt_bias || !g || !beta || T <= 0 || H <= 0 || H % 32 || Hv <= 0 || Hv > MAX_N / 2 ||
      (reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(w)) % 16)
    return -6;
  return (int)b200::launch_pdl(gdn_ab_gates_kernel, dim3((T + ROWS - 1) / ROWS, CT), dim3(WARPS * 32), 0, stream,
                               reinterpret_cast<const __nv_bfloat16*>(x), H, reinterpret_cast<const __nv_bfloat16*>(w), a_log, dt_bias, g,
                               beta, T, Hv);
}
