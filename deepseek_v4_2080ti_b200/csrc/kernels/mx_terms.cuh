// Rows of bf16 activations as pairs of E4M3 terms for block-scaled tensor products (gemm_fp4_terms.cu).
//
// A value x of a block of 32 is  x = 2^s (hi + 2^-5 mid),  hi and mid in E4M3, 4 significant bits each of the 8 that bf16 has.  The
// scale 2^s puts the block's largest value in [2^7, 2^8): hi is x rounded to 4 bits, what is left is at most 8 units of the last of
// bf16's places, which 4 bits hold.  So the pair is exact down to 2^-14 of the largest value (where the last place of mid, 2^-9, is
// bf16's), and below off by at most 2^-15, 2^-22 of the largest.  Blocks where more than a quarter of the nonzero values lie below, or
// that hold infinities or NaNs, get a smaller top: the values past it stay as they are in `rest`, and the product adds them in fp32
// (the rule of term_scale in fp8_terms.cuh).
#pragma once
#include "fp8_terms.cuh"

namespace b200 {
namespace mx {

constexpr int DEPTH = 14, TOP = 7;

struct Rows {
  uint8_t* xq;                 // [2][R][K] larger terms, then the smaller ones; of eight neighbours the even ones first
  uint8_t* sf;                 // [K / 128][R][4] UE8M0 scales of the larger terms; the smaller ones' are 2^-5 of them
  int* outside;                // [R] the row has values outside its terms
  __nv_bfloat16* rest;         // [R][K]: those among zeros; rows without any are undefined
  int R, K;

  // Stores values i0 .. i0 + 7 of a row as terms, for threads that are `on`; four neighbouring lanes hold a block, and the whole warp
  // takes part.  Returns the block's scale.
  __device__ __forceinline__ f8t::TermScale put(int row, int i0, const float (&v)[8], bool on) const {
    const f8t::TermScale ts = f8t::term_scale<8, 4, DEPTH, TOP>(v);
    if (!on) return ts;
    uint32_t hi[4], mid[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {              // values 0 2, 4 6, 1 3, 5 7: the order the product has the weights of eight inputs in
      const int j = (i & 1) * 4 + (i >> 1);
      const float a = f8t::bf16_magnitude(v[j]) < ts.top ? v[j] * ts.scale : 0.f;
      const float b = f8t::bf16_magnitude(v[j + 2]) < ts.top ? v[j + 2] * ts.scale : 0.f;
      hi[i] = __nv_cvt_float2_to_fp8x2(make_float2(a, b), __NV_SATFINITE, __NV_E4M3);
      const float2 q = f8t::e4m3x2_to_float2(hi[i]);
      mid[i] = __nv_cvt_float2_to_fp8x2(make_float2((a - q.x) * 32.f, (b - q.y) * 32.f), __NV_SATFINITE, __NV_E4M3);
    }
    uint8_t* dst = xq + (size_t)row * K + i0;
    *reinterpret_cast<uint2*>(dst) = make_uint2(hi[0] | hi[1] << 16, hi[2] | hi[3] << 16);
    *reinterpret_cast<uint2*>(dst + (size_t)R * K) = make_uint2(mid[0] | mid[1] << 16, mid[2] | mid[3] << 16);
    if ((i0 & 31) == 0) sf[((size_t)(i0 >> 7) * R + row) * 4 + (i0 >> 5 & 3)] = (uint8_t)(__float_as_uint(ts.inv) >> 23);
    return ts;
  }
  // A whole row by the block: values(i, v) gives values i .. i + 7, rounded to bf16, and may be asked twice.
  template <class F>
  __device__ __forceinline__ void put_row(int row, F values) const {
    bool any = false;
#pragma unroll 2
    for (int i0 = 0; i0 < K; i0 += blockDim.x * 8) {
      const int i = i0 + threadIdx.x * 8;
      float v[8] = {};
      if (i < K) values(i, v);
      any |= put(row, i, v, i < K).outside;
    }
    any = __syncthreads_or(any);
    if (threadIdx.x == 0) outside[row] = any;
    if (!any) return;                          // as a rule
    for (int i0 = 0; i0 < K; i0 += blockDim.x * 8) {
      const int i = i0 + threadIdx.x * 8;
      float v[8] = {};
      if (i < K) values(i, v);
      const uint32_t top = f8t::term_scale<8, 4, DEPTH, TOP>(v).top;
      if (i < K) {
#pragma unroll
        for (int j = 0; j < 8; ++j) rest[(size_t)row * K + i + j] = __float2bfloat16(f8t::bf16_magnitude(v[j]) < top ? 0.f : v[j]);
      }
    }
  }
};

}  // namespace mx
}  // namespace b200
