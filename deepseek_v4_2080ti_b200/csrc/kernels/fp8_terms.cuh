// What the FP8 term kernels share (gemm_fp8_terms.cu, gemm_fp8_pair.cu): packed fp32 arithmetic, products issued by a whole
// warp, and the cut of the work list.
#pragma once
#include <cuda_bf16.h>
#include <cuda_fp8.h>
#include "../ptx/sm100.cuh"

namespace b200 {
namespace f8t {

constexpr int BM = 128;             // features of a weight block
constexpr int W_BYTES = BM * 128;   // one 128 x 128 block: two 64-byte-swizzled halves of 8 KB
constexpr int RUN = 256;            // weight scales of a run of K blocks kept in shared memory
constexpr int MAX_SINGLE = 64;      // tokens up to which one CTA per worker is used
constexpr int PAIR_TOK = 256;       // tokens of a pair's tile

struct Params {
  int T, N, m_tiles, n_tiles, kb;   // kb: 128-wide K blocks; m_tiles: 128-feature tiles; n_tiles: token tiles
  int units, workers;               // units = tiles x kb (a pair's tile covers two m tiles)
  const uint8_t* w;                 // [m_tiles][kb][16 KB]
  const float* scales;              // [m_tiles][kb]
  const uint8_t* xq;                // [n_tiles][kb][CTA of the worker][hi, mid][tokens of a CTA][128 bytes]
  const float* sx;                  // [n_tiles][kb][tokens of a tile]
  __nv_bfloat16* out;               // [T, N]
  const __nv_bfloat16* residual;
  float* partial;                   // [workers][2][CTAs][tokens of a CTA's tile x its features]
  int* counters;                    // [tiles x CTAs], zero, left zero
  int* status;
  int vec;                          // rows of `out` (and `residual`) are whole, aligned 16-byte groups
  // first unit of a worker
  __device__ __forceinline__ int first(int worker) const { return (int)((long long)units * worker / workers); }
  // worker of a unit: the largest i with units * i / workers <= u
  __device__ __forceinline__ int owner(int u) const { return (int)((((long long)u + 1) * workers - 1) / units); }
  // where worker i leaves its share of a cut tile: its first tile in place 0, its last in place 1
  __device__ __forceinline__ int place(int i, int tile) const { return first(i) / kb == tile ? 0 : 1; }
};

// ---- activations as terms.  Where the terms of a [T, K] matrix go: tiles of `tok` tokens, each CTA of a worker staging `cap`.
struct TermsOut {
  uint8_t* xq;
  float* sx;
  int tok, cap, kb;
  // first byte of token t's hi row in block c; its mid row is `cap` rows further
  __device__ __forceinline__ uint8_t* hi_row(int t, int c, int& row) const {
    const int n = t / tok, tt = t - n * tok, r = tt / cap;
    row = tt - r * cap;
    return xq + ((size_t)n * kb + c) * (tok * 256) + r * (cap * 256) + row * 128;
  }
  __device__ __forceinline__ float* scale(int t, int c) const { return sx + ((size_t)(t / tok) * kb + c) * tok + t % tok; }
};
// The scale of a block whose largest bf16 magnitude has the bits m (magnitudes of bf16 order like integers, infinity and NaN
// above all): a power of two that puts it in [128, 256).  `inv` undoes it.  An infinity gives an infinite scale with terms of
// +-1 at its places (the product keeps the sign the plain sum has), a NaN a NaN scale.
struct TermScale {
  float scale, inv;
  bool special;
  __device__ __forceinline__ explicit TermScale(uint32_t m) {
    const int sh = max(min(7 - (max((int)(m >> 7), 1) - 127), 120), -126);
    scale = __uint_as_float((uint32_t)(127 + sh) << 23);
    inv = __uint_as_float((uint32_t)(127 - sh) << 23);
    special = m >= 0x7f80u;
    if (special) inv = __uint_as_float(m > 0x7f80u ? 0x7fc00000u : 0x7f800000u);
  }
  // terms of a bf16 value given as fp32
  __device__ __forceinline__ void split(float x, uint32_t& hi, uint32_t& mid) const {
    if (special) {
      const uint32_t b = __float_as_uint(x);
      hi = (b & 0x7f800000u) == 0x7f800000u ? 0x38u | (b >> 31) << 7 : 0u;
      mid = 0;
      return;
    }
    const float v = x * scale;
    const __nv_fp8_e4m3 q(v);
    const __nv_fp8_e4m3 r(v - float(q));
    hi = q.__x;
    mid = r.__x;
  }
  // four neighbours; bytes of a group are stored as (x0, x2, x1, x3), the order the packed weights use
  __device__ __forceinline__ void split4(const float* x, uint32_t& hi, uint32_t& mid) const {
    hi = mid = 0;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      uint32_t a, b;
      split(x[i], a, b);
      const int at = i == 1 ? 16 : i == 2 ? 8 : i * 8;
      hi |= a << at;
      mid |= b << at;
    }
  }
};
// Byte offset of 4-byte group g (0 .. 31) in a row of 128 bytes with the 128-byte swizzle.
__device__ __forceinline__ int term_offset(int row, int g) { return (((g >> 2) ^ (row & 7)) << 4) + (g & 3) * 4; }
__device__ __forceinline__ uint32_t bf16_magnitude(float x) { return __float_as_uint(x) >> 16 & 0x7fffu; }

// K-major operand with the 64-byte swizzle: rows of 64 bytes, 8-row groups 512 bytes apart.
__device__ __forceinline__ uint64_t desc_sw64(const void* smem_tile) {
  uint64_t d = 0;
  d |= (uint64_t)((smem_u32(smem_tile) & 0x3FFFF) >> 4);
  d |= (uint64_t)(512 >> 4) << 32;
  d |= (uint64_t)1 << 46;
  d |= (uint64_t)4 << 61;   // SWIZZLE_64B
  return d;
}
// Descriptor offset of 32-byte K step k (0 .. 3) of a weight block.
__device__ __forceinline__ uint64_t w_step(int k) { return (uint64_t)((k >> 1) * (W_BYTES / 2 / 16) + 2 * (k & 1)); }

typedef unsigned long long f2;      // two packed floats
__device__ __forceinline__ f2 pack2(uint32_t a, uint32_t b) {
  f2 d;
  asm("mov.b64 %0, {%1, %2};" : "=l"(d) : "r"(a), "r"(b));
  return d;
}
__device__ __forceinline__ f2 pack2f(float a, float b) { return pack2(__float_as_uint(a), __float_as_uint(b)); }
__device__ __forceinline__ f2 fma2(f2 a, f2 b, f2 c) {
  f2 d;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
  return d;
}
__device__ __forceinline__ f2 add2(f2 a, f2 b) {
  f2 d;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
  return d;
}
__device__ __forceinline__ float at(const f2* v, int i) { return __uint_as_float((uint32_t)(v[i / 2] >> (32 * (i & 1)))); }

// Products are issued by the elected lane of a converged warp (`on`): the operands then sit in uniform registers.  From a
// lane that branched off alone each instruction costs some 120 cycles.
__device__ __forceinline__ void umma_f8_warp(uint32_t on, uint32_t tmem_d, uint64_t da, uint64_t db, uint32_t idesc, uint32_t acc) {
  asm volatile(
      "{\n\t.reg .pred p, e;\n\t"
      "setp.ne.b32 e, %5, 0;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "@e tcgen05.mma.cta_group::1.kind::f8f6f4 [%0], %1, %2, %3, p;\n\t}\n"
      :
      : "r"(tmem_d), "l"(da), "l"(db), "r"(idesc), "r"(acc), "r"(on)
      : "memory");
}
__device__ __forceinline__ void umma_f8_pair_warp(uint32_t on, uint32_t tmem_d, uint64_t da, uint64_t db, uint32_t idesc, uint32_t acc) {
  const uint32_t z = 0;
  asm volatile(
      "{\n\t.reg .pred p, e;\n\t"
      "setp.ne.b32 e, %6, 0;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "@e tcgen05.mma.cta_group::2.kind::f8f6f4 [%0], %1, %2, %3, {%5, %5, %5, %5, %5, %5, %5, %5}, p;\n\t}\n"
      :
      : "r"(tmem_d), "l"(da), "l"(db), "r"(idesc), "r"(acc), "r"(z), "r"(on)
      : "memory");
}
__device__ __forceinline__ void commit_pair_warp(uint32_t on, uint64_t* bar) {
  const uint16_t both = 3;
  asm volatile(
      "{\n\t.reg .pred e;\n\t"
      "setp.ne.b32 e, %2, 0;\n\t"
      "@e tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;\n\t}\n" ::"r"(
          smem_u32(bar)),
      "h"(both), "r"(on)
      : "memory");
}

}  // namespace f8t

int gemm_fp8_pair_launch(const f8t::Params& p, cudaStream_t stream);

}  // namespace b200
