// What the FP8 term kernels share (gemm_fp8_terms.cu, gemm_fp8_pair.cu): activations as terms, packed fp32 arithmetic, products
// issued by a whole warp, and the cut of the work list.
#pragma once
#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cuda_fp8.h>
#include "../ptx/sm100.cuh"

namespace b200 {
namespace f8t {

constexpr int BM = 128;             // features of a weight block
constexpr int W_BYTES = BM * 128;   // one 128 x 128 block: two 64-byte-swizzled halves of 8 KB
constexpr int RUN = 256;            // weight scales of a run of K blocks kept in shared memory
constexpr int MAX_SINGLE = 128;      // tokens up to which one CTA per worker is used
constexpr int PAIR_TOK = 256;       // tokens of a pair's tile

struct Params {
  int T, N, m_tiles, n_tiles, kb;   // kb: 128-wide K blocks; m_tiles: 128-feature tiles; n_tiles: token tiles
  int workers;                      // CTAs or pairs; a pair's tile covers two m tiles
  int waves;                        // whole tiles that every worker takes, one of each run of `workers` tiles,
  int units;                        // and (tile, K block) pairs of the tiles after those, shared in equal contiguous runs
  const uint8_t* w;                 // [m_tiles][kb][16 KB]
  const float* scales;              // [m_tiles][kb]
  const uint8_t* xq;                // [n_tiles][kb][CTA of the worker][hi, mid][tokens of a CTA][128 bytes]
  const float* sx;                  // [n_tiles][kb][tokens of a tile]; negative: the block has values outside its terms
  const __nv_bfloat16* rest;        // [T][kb][128]: those values among zeros; other blocks undefined
  __nv_bfloat16* out;               // [T, N]
  const __nv_bfloat16* residual;
  float* partial;                   // [workers][2][CTAs][tokens of a CTA's tile x its features]
  int* counters;                    // [workers x CTAs], zero, left zero; a cut tile uses those of its first contributor
  int* status;
  int vec;                          // rows of `out` (and `residual`) are whole, aligned 16-byte groups
  // first unit of a worker
  __device__ __forceinline__ int first(int worker) const { return (int)((long long)units * worker / workers); }
  __device__ __forceinline__ int tail() const { return waves * workers; }
  // worker of a unit: the largest i with units * i / workers <= u
  __device__ __forceinline__ int owner(int u) const { return (int)((((long long)u + 1) * workers - 1) / units); }
  // where worker i leaves its share of a cut tile (counted from the tail): its first tile in place 0, its last in place 1
  __device__ __forceinline__ int place(int i, int tile) const { return first(i) / kb == tile ? 0 : 1; }
};

// The pieces of tiles that a worker computes, in order.
struct Pieces {
  const Params& p;
  int worker, wave, u, u1;
  int tile, c0, len;                // the piece: K blocks c0 .. c0 + len - 1 of a tile
  __device__ __forceinline__ Pieces(const Params& p, int worker) : p(p), worker(worker), wave(0), u(p.first(worker)), u1(p.first(worker + 1)) {}
  __device__ __forceinline__ bool next() {
    if (wave < p.waves) {
      tile = wave++ * p.workers + worker;
      c0 = 0;
      len = p.kb;
      return true;
    }
    if (u >= u1) return false;
    const int t = u / p.kb;
    tile = p.tail() + t;
    c0 = u - t * p.kb;
    len = min(p.kb - c0, u1 - u);
    u += len;
    return true;
  }
};

// ---- activations as terms.  Where the terms of a [T, K] matrix go: tiles of `tok` tokens, each CTA of a worker staging `cap`.
struct TermsOut {
  uint8_t* xq;
  float* sx;
  __nv_bfloat16* rest;                // [T, K]; written only in blocks that have values outside their terms
  int* counters;                      // [n_counters], zeroed by the kernel that makes the terms for the products that take them
  int tok, cap, kb, n_counters;
  __device__ __forceinline__ void zero_counters(bool first_block) const {
    if (first_block)
      for (int i = threadIdx.x; i < n_counters; i += blockDim.x) counters[i] = 0;
  }
  // first byte of token t's hi row in block c; its mid row is `cap` rows further
  __device__ __forceinline__ uint8_t* hi_row(int t, int c, int& row) const {
    const int n = t / tok, tt = t - n * tok, r = tt / cap;
    row = tt - r * cap;
    return xq + ((size_t)n * kb + c) * (tok * 256) + r * (cap * 256) + row * 128;
  }
  __device__ __forceinline__ float* scale(int t, int c) const { return sx + ((size_t)(t / tok) * kb + c) * tok + t % tok; }
};
// Byte offset of 4-byte group g (0 .. 31) in a row of 128 bytes with the 128-byte swizzle.
__device__ __forceinline__ int term_offset(int row, int g) { return (((g >> 2) ^ (row & 7)) << 4) + (g & 3) * 4; }
// A bf16 value's bits without the sign: they order like integers, infinity and NaN above all.
__device__ __forceinline__ uint32_t bf16_magnitude(float x) { return __float_as_uint(x) >> 16 & 0x7fffu; }

// Terms of one bf16 value x, scaled by a power of two c of its block: x c = hi + mid, hi in E5M2 (3 significant bits), mid in
// E4M3 (4).  Rounding to hi leaves at most 16 units of the last of a bf16 number's 8 places, which 4 bits hold, so the pair is
// exact while that last place is a multiple of 2^-9, E4M3's smallest step; below, it is off by at most 2^-10.  With hi < 2^12 (mid
// stays under 448) the exact values reach down to 2^-2, 2^-13 of the largest.  (hi in E4M3 too: 2^-9 of the largest.)
//
// The scale of a block puts its largest value in [2^11, 2^12), unless more than a quarter of its nonzero values would fall below
// 2^-2: then it is the largest scale that leaves them a quarter, and the values past the top - infinities and NaNs always - are not
// terms but stay as they are, in `rest`; the block's scale is stored negative and the product adds them in fp32.  So every value
// is exact, or among the smallest quarter of its block and off by at most 2^-8 of the value at the quarter.
constexpr uint32_t BF16_INF = 0x7f80u;
constexpr int MIN_TOP = 18;            // exponent field of the smallest top: its scale 2^120 has a normal inverse
struct TermScale {
  uint32_t top;                        // magnitudes from here on are outside the terms
  float scale, inv;
  bool outside;                        // the block has such values
};
template <int LANES>
__device__ __forceinline__ uint32_t block_max(uint32_t v) {
#pragma unroll
  for (int d = LANES / 2; d > 0; d >>= 1) v = max(v, __shfl_xor_sync(0xffffffffu, v, d));
  return v;
}
template <int LANES>
__device__ __forceinline__ uint32_t block_sum(uint32_t v) {
#pragma unroll
  for (int d = LANES / 2; d > 0; d >>= 1) v += __shfl_xor_sync(0xffffffffu, v, d);
  return v;
}
// The scale of a block of V values on each of LANES neighbouring lanes; the whole warp takes part.  It puts the top at 2^TOP;
// values are exact terms down to DEPTH exponents below it.
template <int V, int LANES = 128 / V, int DEPTH = 13, int TOP = 11>
__device__ __forceinline__ TermScale term_scale(const float (&x)[V]) {
  uint32_t m = 0;
#pragma unroll
  for (int i = 0; i < V; ++i) m = max(m, bf16_magnitude(x[i]));
  m = block_max<LANES>(m);
  // values more than DEPTH below a top exponent e, and nonzero ones, in the halves of a word
  auto counts = [&](int e) {
    uint32_t n = 0;
#pragma unroll
    for (int i = 0; i < V; ++i) {
      const uint32_t b = bf16_magnitude(x[i]);
      n += b ? (b >> 7 < (uint32_t)(e - DEPTH) ? 0x10001u : 1u) : 0u;
    }
    return block_sum<LANES>(n);
  };
  auto fits = [&](uint32_t n) { return 4 * (n >> 16) <= (n & 0xffffu); };
  int e = max((int)(m >> 7), MIN_TOP);
  TermScale r;
  r.outside = m >= BF16_INF;
  const uint32_t n = counts(e);
  const bool wide = r.outside || (e > MIN_TOP && !fits(n));
  if (__any_sync(0xffffffffu, wide)) {           // rare
    uint32_t f = 0;                              // the largest finite magnitude
#pragma unroll
    for (int i = 0; i < V; ++i) f = max(f, bf16_magnitude(x[i]) < BF16_INF ? bf16_magnitude(x[i]) : 0u);
    const int last = max((int)(block_max<LANES>(f) >> 7), MIN_TOP);
    // the largest exponent up to `last` under which at most a quarter falls below
    int lo = MIN_TOP, hi = last + 1;
    while (__any_sync(0xffffffffu, hi - lo > 1)) {
      const int mid = hi - lo > 1 ? (hi + lo) >> 1 : lo;
      const bool ok = fits(counts(mid));
      if (hi - lo > 1) (ok ? lo : hi) = mid;
    }
    e = lo;
    r.outside |= lo < last;
  }
  r.top = (uint32_t)(e + 1) << 7;
  r.scale = __uint_as_float((uint32_t)(254 + TOP - e) << 23);       // x < 2^(e - 126) -> x scale < 2^(TOP + 1)
  r.inv = __uint_as_float((uint32_t)(e - TOP) << 23);
  return r;
}
// Two values (as fp32) -> their terms, a byte each.
__device__ __forceinline__ void split2(const TermScale& ts, float a, float b, uint32_t& hi, uint32_t& mid) {
  a = bf16_magnitude(a) < ts.top ? a * ts.scale : 0.f;
  b = bf16_magnitude(b) < ts.top ? b * ts.scale : 0.f;
  hi = __nv_cvt_float2_to_fp8x2(make_float2(a, b), __NV_SATFINITE, __NV_E5M2);
  const float2 q = __half22float2(__half2(__nv_cvt_fp8x2_to_halfraw2((__nv_fp8x2_storage_t)hi, __NV_E5M2)));
  mid = __nv_cvt_float2_to_fp8x2(make_float2(a - q.x, b - q.y), __NV_SATFINITE, __NV_E4M3);
}
// Stores values i0 .. i0 + V - 1 of token t as terms, for threads that are `on`; the whole warp takes part.  V = 4 or 8, i0 a
// multiple of V, the 128 / V lanes of a block next to each other.
template <int V>
__device__ __forceinline__ void put_terms(const TermsOut& o, int t, int i0, const float (&v)[V], bool on) {
  const TermScale ts = term_scale(v);
  if (!on) return;
  const int c = i0 >> 7;
  int row;
  uint8_t* dst = o.hi_row(t, c, row);
  dst += term_offset(row, (i0 & 127) >> 2);
  uint32_t hi[V / 4], mid[V / 4];
#pragma unroll
  for (int g = 0; g < V / 4; ++g) {      // bytes of a group are stored as (x0, x2, x1, x3), the order the packed weights use
    uint32_t h0, m0, h1, m1;
    split2(ts, v[4 * g], v[4 * g + 2], h0, m0);
    split2(ts, v[4 * g + 1], v[4 * g + 3], h1, m1);
    hi[g] = h0 | h1 << 16;
    mid[g] = m0 | m1 << 16;
  }
  if constexpr (V == 8) {
    *reinterpret_cast<uint2*>(dst) = make_uint2(hi[0], hi[1]);
    *reinterpret_cast<uint2*>(dst + o.cap * 128) = make_uint2(mid[0], mid[1]);
  } else {
    *reinterpret_cast<uint32_t*>(dst) = hi[0];
    *reinterpret_cast<uint32_t*>(dst + o.cap * 128) = mid[0];
  }
  if (ts.outside) {
    __nv_bfloat16* rest = o.rest + (size_t)t * o.kb * 128 + i0;
#pragma unroll
    for (int i = 0; i < V; ++i) rest[i] = bf16_magnitude(v[i]) < ts.top ? __float2bfloat16(0.f) : __float2bfloat16(v[i]);
  }
  if ((i0 & 127) == 0) *o.scale(t, c) = ts.outside ? -ts.inv : ts.inv;
}

// Byte of input k in feature r's row of a packed 128 x 128 weight block: two halves of 64 inputs, four-byte groups as
// (w0, w2, w1, w3), 16-byte chunks under the 64-byte swizzle.
__device__ __forceinline__ int w_offset(int r, int k) {
  return (k >> 6) * (W_BYTES / 2) + r * 64 + ((((k >> 4) & 3) ^ ((r >> 1) & 3)) << 4) + (k & 12) + ((k & 1) << 1) + ((k >> 1) & 1);
}
__device__ __forceinline__ float2 e4m3x2_to_float2(uint32_t two) {
  return __half22float2(__half2(__nv_cvt_fp8x2_to_halfraw2((__nv_fp8x2_storage_t)two, __NV_E4M3)));
}
// Calls f(k, value) for the values that token t has outside its terms in block c; the whole warp calls it together.
template <class F>
__device__ __forceinline__ void for_each_outside(const __nv_bfloat16* rest, int kb, int t, int c, F f) {
  const int lane = threadIdx.x & 31;
  const uint2 u = __ldcg(reinterpret_cast<const uint2*>(rest + ((size_t)t * kb + c) * 128 + lane * 4));
#pragma unroll
  for (int e = 0; e < 4; ++e) {
    const uint32_t h = ((e & 2 ? u.y : u.x) >> (16 * (e & 1))) << 16;
    for (uint32_t on = __ballot_sync(0xffffffffu, (h & 0x7fffffffu) != 0); on; on &= on - 1) {
      const int src = __ffs(on) - 1;
      f(src * 4 + e, __uint_as_float(__shfl_sync(0xffffffffu, h, src)));
    }
  }
}

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
