// FP8 block-128 weights times bf16 activations on the FP8 tensor pipe, for token counts below the bf16 prefill kernel's:
//   Y[T, N] = X[T, K] * W[N, K]^T,  W = E4M3 with one scale per 128 x 128 block.
//
// Weights go from HBM to the tensor core untouched; the activations are adapted.  A bf16 number has 8 significant bits, an
// E5M2 number 3, an E4M3 number 4, so with a power-of-two scale c per (token, 128 inputs) an activation is
//   x c = hi + mid,   hi in E5M2, mid in E4M3
// exactly where it is above 2^-13 of the block's largest (fp8_terms.cuh has what lies below, and what happens to blocks where
// that is much).  Both terms have the same scale, so the tensor core adds them: two products per K block into one accumulator, at
// twice the bf16 rate - the tensor time of bf16, half the weight bytes, no decode warps, and no rounding of the scaled weights to
// bf16, which the decode-warp kernel (gemm_wdec_kernel.cuh) needs and which costs 1.6e-3 of a result.  The scales are applied
// outside the tensor core: each 128-wide K block is accumulated into its own TMEM buffer; one warp multiplies the weight scale
// into the block's activation scales, and the epilogue warps add scale x block into fp32 registers, two tokens per instruction,
// while the tensor core is on the next blocks.
//
// This file: up to 128 tokens, one CTA per worker, weights as the MMA's M operand; bound by the weight stream, 160 KB of it in flight
// per SM at 16 tokens, 144 at 32, 96 at 64, 64 at 128.  More tokens: gemm_fp8_pair.cu.
//
// Work: the (tile, K block) pairs are one list, cut into equal contiguous runs, one per worker, so no wave is partly empty
// whatever N and K are.  A tile that is cut is finished by whichever contributor arrives last, which adds the fp32 partial
// sums in K order (the result does not depend on who is last).
//
// Roles: warps 0-7 epilogue, warp 8 weight copies, warp 9 MMA issuer, warp 10 activation copies, warp 11 scales.  All waits
// are bounded.  The two epilogue groups of four share the work of a block by tokens (32 tokens and more) or take every other
// block.
//
// Measured, us per product in a graph of 16, the split not counted (weights 63, 21, 178, 89 MB: 12288 x 5120, 5120 x 4096,
// 34816 x 5120, 5120 x 17408; a plain read of as many bytes takes 9.7, 3.7, 25.3, 13.2):
//   1 token 14.8, 9.4, 31, 19.4;  32 tokens 16.6, 10.6, 33.9, 20.5;  64 tokens 20.8, 13.5, 42.2, 26.0;
// with the split: 65 tokens 31.5, 19.6, 63, 42;  100 tokens 35, 21.8, 70.5, 48;  128 tokens 37, 22.8, 74, 50.7.  (On pairs, half of whose 256
// tokens are padding then: 65 tokens 44, 28.5, 81.6, 57;  128 tokens 47.6, 31, 88, 60.)
// Of these, about 6.5 us a product are fixed at 1 token and 8 at 64: filling the pipeline and the sums of cut tiles; above them a
// block takes 0.354 us at 1 token, 6.85 TB/s, and 0.467 at 64.  Tried at 64 tokens and slower: more weight slots beside fewer activation
// slots (47.8 to 50 for 45.8), slots given back by the commit and accumulators read a block ahead (54.5), two feature blocks per
// activation block (47.0, and 21.5 for 15.3 where every tile is cut), the next blocks prefetched to L2 (1 to 8 % more).
// The kernels this one took over from, in a chain: gemm_w8a8s.cu at 1 token 20.6, 12.0, 38.7, 29.8, at 32 tokens 47.6, 52.6,
// 45.9, 71.8; the decode-warp kernel at 64 tokens 77.9, 83.1, 188, 111 (with the converged issue it has now 38, 41, 193, 57).
//
// Reference behaviour covered: the FP8 block-128 projections of the Qwen path
// (cpp_engine/backends/cuda/kernels/qwen_half_ops.cu:130-535, 988-1199).
#include <cuda_bf16.h>
#include <cuda_fp8.h>
#include <string.h>
#include <initializer_list>
#include "../ptx/sm100.cuh"
#include "fp8_terms.cuh"
#include "launch.h"
#include "ops.h"
#include "per_device.h"
#include "tma_host.h"

namespace b200 {
namespace f8t {

constexpr int EPI_WARPS = 8;
constexpr int EPI_THREADS = EPI_WARPS * 32;
constexpr int WARP_W = EPI_WARPS, WARP_MMA = EPI_WARPS + 1, WARP_X = EPI_WARPS + 2, WARP_S = EPI_WARPS + 3;
constexpr int THREADS = (EPI_WARPS + 4) * 32;

template <int TOK>
struct Cfg {
  static constexpr int X_BYTES = 2 * TOK * 128;
  static constexpr int SLOT = W_BYTES + X_BYTES;
  static constexpr int SX_BYTES = TOK * 4;
  static constexpr bool BY_TOKENS = TOK >= 32;            // how the epilogue groups share the work
  static constexpr int WT = BY_TOKENS ? TOK / 2 : TOK;    // tokens of a thread
  static constexpr int SUM_BYTES = BY_TOKENS ? 0 : TOK * BM * 4;
  static constexpr int BUDGET = 232448 - 1024 - 1024 - SUM_BYTES - RUN * 4;
  static constexpr int S_FIT = BUDGET / (SLOT + SX_BYTES);
  static constexpr int S = S_FIT > 12 ? 12 : S_FIT;
  static constexpr int A = 512 / TOK < S ? 512 / TOK : S; // accumulator buffers
  static constexpr uint32_t TMEM_COLS = A * TOK <= 128 ? 128 : A * TOK <= 256 ? 256 : 512;
  static constexpr int TOTAL = S * (SLOT + SX_BYTES) + SUM_BYTES + RUN * 4 + 2048;
};
__host__ __device__ constexpr int round16(int v) { return (v + 15) / 16 * 16; }

// acc[i] += sc[i] v[i] for 16 tokens; sc: 16-byte-aligned shared memory.
__device__ __forceinline__ void add_scaled(f2* acc, const uint32_t* v, const float* sc) {
#pragma unroll
  for (int i = 0; i < 16; i += 4) {
    const ulonglong2 s = *reinterpret_cast<const ulonglong2*>(sc + i);
    acc[i / 2] = fma2(pack2(v[i], v[i + 1]), s.x, acc[i / 2]);
    acc[i / 2 + 1] = fma2(pack2(v[i + 2], v[i + 3]), s.y, acc[i / 2 + 1]);
  }
}

__device__ __forceinline__ void epi_sync() { asm volatile("bar.sync 1, %0;" ::"n"(EPI_THREADS) : "memory"); }

template <int TOK>
__global__ void __launch_bounds__(THREADS, 1)
gemm_fp8_terms_kernel(Params p) {
  using L = Cfg<TOK>;
  constexpr int S = L::S, A = L::A, WT = L::WT;
  constexpr int READERS = L::BY_TOKENS ? EPI_WARPS : EPI_WARPS / 2;   // epilogue warps that read a block
  extern __shared__ uint8_t smem_raw_base[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw_base) + 1023) & ~uintptr_t(1023));
  uint8_t* sW = smem;
  uint8_t* sX = sW + S * W_BYTES;
  float* sSx = reinterpret_cast<float*>(sX + S * L::X_BYTES);
  float* sSum = sSx + S * TOK;           // [TOK][BM] sums of the second group, where the groups share blocks
  float* sRun = sSum + L::SUM_BYTES / 4;
  uint64_t* bars = reinterpret_cast<uint64_t*>(sRun + RUN);
  uint64_t* full = bars;                 // [S] operands landed
  uint64_t* sx_full = bars + S;          // [S] activation scales landed
  uint64_t* sc_full = bars + 4 * S + A;  // [S] scales of the block's products ready
  uint64_t* done = bars + 2 * S;         // [S] the block's MMAs are finished: accumulator readable
  uint64_t* slot_free = bars + 3 * S;    // [S] the epilogue is through with the block: slot reusable
  uint64_t* acc_free = bars + 4 * S;     // [A] accumulator reusable
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 5 * S + A);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
  volatile int* epi_abort = abort_flag + 1;     // written by epilogue threads only, always before a barrier
  int* fix_last = const_cast<int*>(abort_flag) + 2;
  volatile int* last_outside = abort_flag + 3;  // the last block so far in which a token has values outside its terms

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (threadIdx.x == 0) {
    for (int s = 0; s < S; ++s) {
      mbar_init(&full[s], 2);             // weights and activations announce their bytes
      mbar_init(&sx_full[s], 1);
      mbar_init(&sc_full[s], 1);
      mbar_init(&done[s], 1);
      mbar_init(&slot_free[s], READERS);
    }
    for (int a = 0; a < A; ++a) mbar_init(&acc_free[a], READERS);
    *abort_flag = 0;
    *epi_abort = 0;
    *last_outside = -1;
    mbar_fence_init();
  }
  if (warp == WARP_MMA) {
    tmem_alloc(tmem_slot, L::TMEM_COLS);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  pdl_launch_dependents();   // the next kernel may be scheduled; it waits for this grid before touching memory

  const int worker = blockIdx.x;
  const int u0 = p.first(worker), u1 = p.first(worker + 1);

  if (warp == WARP_W) {
    // ------------------------------------------------------------ weight copies
    // The weights do not depend on the previous kernel of the stream: as a programmatic dependent this warp fills the ring
    // while the predecessor still runs.
    if (lane == 0) {
      for (int blk = 0; blk < u1 - u0 && !*abort_flag; ++blk) {
        const int b = blk % S;
        if (blk >= S && !mbar_wait(&slot_free[b], ((blk / S) & 1) ^ 1)) {
          atomicExch(p.status, ERR_WAIT_STAGE);
          *abort_flag = 1;
          break;
        }
        mbar_expect_tx(&full[b], W_BYTES);
        bulk_load(sW + b * W_BYTES, p.w + (size_t)(u0 + blk) * W_BYTES, W_BYTES, &full[b]);
      }
    }
  } else if (warp == WARP_X) {
    // ------------------------------------------------------------ activation copies
    if (lane == 0) {
      pdl_wait();
      int c = u0 % p.kb;
      for (int blk = 0; blk < u1 - u0 && !*abort_flag; ++blk) {
        const int b = blk % S;
        if (blk >= S && !mbar_wait(&slot_free[b], ((blk / S) & 1) ^ 1)) {
          atomicExch(p.status, ERR_WAIT_STAGE);
          *abort_flag = 1;
          break;
        }
        mbar_expect_tx(&full[b], L::X_BYTES);
        bulk_load(sX + b * L::X_BYTES, p.xq + (size_t)c * L::X_BYTES, L::X_BYTES, &full[b]);
        mbar_expect_tx(&sx_full[b], L::SX_BYTES);
        bulk_load(sSx + b * TOK, p.sx + (size_t)c * TOK, L::SX_BYTES, &sx_full[b]);
        if (++c == p.kb) c = 0;
      }
    }
  } else if (warp == WARP_MMA) {
    // -------------------------------------------------------------- MMA issuer
    {
      const uint32_t on = elect_one();
      // as many columns as there are tokens
      const uint32_t idesc_hi = umma_idesc_f8(BM, round16(p.T), false, true), idesc_mid = umma_idesc_f8(BM, round16(p.T));
      for (int blk = 0; blk < u1 - u0; ++blk) {
        const int b = blk % S, a = blk % A;
        int err = 0;
        if (!mbar_wait(&acc_free[a], ((blk / A) & 1) ^ 1)) err = ERR_WAIT_ACC;
        else if (!mbar_wait(&full[b], (blk / S) & 1)) err = ERR_WAIT_TMA;
        if (__any_sync(0xffffffffu, err != 0 || *abort_flag != 0)) {
          err = (int)__reduce_max_sync(0xffffffffu, (unsigned)err);
          if (err && lane == 0) atomicExch(p.status, err);
          *abort_flag = 1;
          break;
        }
        tc_fence_after();
        const uint32_t d = tmem_base + a * TOK;
        const uint64_t da = desc_sw64(sW + b * W_BYTES), db = umma_desc_sw128(sX + b * L::X_BYTES);
        // one instruction covers 32 K bytes: +32 bytes = +2 in 16-byte units
#pragma unroll
        for (int k = 0; k < 8; ++k) {
          const uint64_t dbk = db + (k >> 2) * (L::X_BYTES / 2 / 16) + 2 * (k & 3);
          umma_f8_warp(on, d, da + w_step(k & 3), dbk, k < 4 ? idesc_hi : idesc_mid, k > 0);
        }
        umma_commit_warp(on, &done[b]);
      }
    }
  } else if (warp == WARP_S) {
    // ------------------------------------------------------------ weight scale into the activation scales, in place
    // The weight scales of a run of blocks are fetched a run ahead: a load per block would wait behind the weight stream on
    // every eighth block.
    auto fetch = [&](int u, float (&v)[RUN / 32]) {
      const int len = u < u1 ? min(p.kb - u % p.kb, u1 - u) : 0;
#pragma unroll
      for (int j = 0; j < RUN / 32; ++j) v[j] = j * 32 + lane < len ? __ldg(p.scales + u + j * 32 + lane) : 0.f;
    };
    float next[RUN / 32];
    fetch(u0, next);
    bool ok = true;
    for (int u = u0; u < u1 && ok;) {
      const int len = min(p.kb - u % p.kb, u1 - u);
      __syncwarp();
#pragma unroll
      for (int j = 0; j < RUN / 32; ++j) sRun[j * 32 + lane] = next[j];
      __syncwarp();
      fetch(u + len, next);
      for (int c = 0; c < len; ++c) {
        const int blk = u - u0 + c, b = blk % S;
        const float sc = c < RUN ? sRun[c] : __ldg(p.scales + u + c);
        ok = __all_sync(0xffffffffu, mbar_wait(&sx_full[b], (blk / S) & 1));
        if (!ok) break;
        float* sx = sSx + b * TOK;
        bool outside = false;
        for (int i = lane; i < TOK; i += 32) {
          const float v = sx[i];
          outside |= i < p.T && v < 0.f;
          sx[i] = fabsf(v) * sc;
        }
        if (__any_sync(0xffffffffu, outside) && lane == 0) *last_outside = blk;
        fence_proxy_async_smem();          // the next copy into this slot comes after these writes
        __syncwarp();
        if (lane == 0) mbar_arrive(&sc_full[b]);
      }
      u += len;
    }
    if (!ok) {
      if (lane == 0) atomicExch(p.status, ERR_WAIT_TMA);
      *abort_flag = 1;
    }
  } else {
    // ---------------------------------------------------------------- epilogue
    const int row = (warp & 3) * 32 + lane;             // TMEM lane = feature within the CTA's tile
    const int group = warp >> 2;
    pdl_wait();   // everything this role reads, or writes, belongs after the previous kernel
    for (int u = u0; u < u1;) {
      const int tile = u / p.kb, c0 = u - tile * p.kb;
      const int len = min(p.kb - c0, u1 - u);
      // tokens [w0, w1) belong to this thread
      const int share = L::BY_TOKENS ? round16(round16(p.T) / 2) : TOK;
      const int w0 = L::BY_TOKENS ? group * share : 0, w1 = L::BY_TOKENS && group == 0 ? min(p.T, share) : p.T;
      f2 acc[WT / 2];
#pragma unroll
      for (int i = 0; i < WT / 2; ++i) acc[i] = 0;
      bool ok = true;
      for (int c = L::BY_TOKENS ? 0 : (group ^ ((u - u0) & 1)); c < len; c += L::BY_TOKENS ? 1 : 2) {
        const int blk = u - u0 + c, b = blk % S, a = blk % A;
        ok = mbar_wait(&sc_full[b], (blk / S) & 1) && mbar_wait(&done[b], (blk / S) & 1);
        ok = __all_sync(0xffffffffu, ok);
        if (!ok) break;
        tc_fence_after();
        const uint32_t taddr = tmem_base + (uint32_t((warp & 3) * 32) << 16) + a * TOK + w0;
        const float* sc = sSx + b * TOK + w0;
        // the read of the next 16 tokens is in flight while this one's sums are taken
        uint32_t v[2][16];
        auto give_back = [&] {        // the accumulator, once its last values are in registers
          tc_fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive(&acc_free[a]);
        };
        if (w0 < w1) tmem_ld_32x16(taddr, v[0]);
        else give_back();
#pragma unroll
        for (int q = 0; q < WT / 16; ++q) {
          if (w0 + q * 16 < w1) {
            tmem_ld_wait();
            if (q + 1 < WT / 16 && w0 + (q + 1) * 16 < w1) tmem_ld_32x16(taddr + (q + 1) * 16, v[(q + 1) & 1]);
            else give_back();
            add_scaled(acc + q * 8, v[q & 1], sc + q * 16);
          }
        }
        __syncwarp();
        if (lane == 0) mbar_arrive(&slot_free[b]);
      }
      if (!ok) {
        if (lane == 0) atomicExch(p.status, ERR_WAIT_ACC);
        *abort_flag = 1;
        *epi_abort = 1;
      } else if (*last_outside >= u - u0) {
        // values outside the terms, on the CUDA cores: as a rule there are none, and in a block that has them a few
        for (int c = L::BY_TOKENS ? 0 : (group ^ ((u - u0) & 1)); c < len; c += L::BY_TOKENS ? 1 : 2) {
          const uint8_t* wb = p.w + (size_t)(u + c) * W_BYTES;
          const float sc = __ldg(p.scales + u + c);
#pragma unroll 1
          for (int t0 = 0; t0 < WT; t0 += 32) {
            const float* sx = p.sx + (size_t)(c0 + c) * TOK + w0 + t0;
            uint32_t tokens = __ballot_sync(0xffffffffu, t0 + lane < WT && w0 + t0 + lane < w1 && __ldcg(sx + lane) < 0.f);
            for (; tokens; tokens &= tokens - 1) {
              const int t = t0 + __ffs(tokens) - 1;
              float sum = 0.f;
              for_each_outside(p.rest, p.kb, w0 + t, c0 + c,
                               [&](int k, float x) { sum += x * (e4m3x2_to_float2(wb[w_offset(row, k)]).x * sc); });
#pragma unroll
              for (int i = 0; i < WT / 2; ++i) acc[i] = add2(acc[i], pack2f(t == 2 * i ? sum : 0.f, t == 2 * i + 1 ? sum : 0.f));
            }
          }
        }
      }
      if constexpr (!L::BY_TOKENS) {
        if (group == 1) {
#pragma unroll
          for (int t = 0; t < TOK; ++t) sSum[t * BM + row] = at(acc, t);
        }
      }
      epi_sync();
      if (*epi_abort) break;
      if constexpr (!L::BY_TOKENS) {
        if (group == 0) {
#pragma unroll
          for (int i = 0; i < WT / 2; ++i)
            acc[i] = pack2(__float_as_uint(at(acc, 2 * i) + sSum[2 * i * BM + row]),
                           __float_as_uint(at(acc, 2 * i + 1) + sSum[(2 * i + 1) * BM + row]));
        }
      }
      if constexpr (!L::BY_TOKENS) epi_sync();                 // the second group may write its next sums
      const bool holds = L::BY_TOKENS || group == 0;           // this thread holds finished sums of tokens w0 ..
      const int f = tile * BM + row;
      if (len == p.kb) {
        if (holds) {
          if (p.vec) {
            // neighbouring lanes trade halves of a token pair: each stores two features of one token
            const int odd = lane & 1;
#pragma unroll
            for (int t = 0; t < WT; t += 2) {
              const float v0 = at(acc, t), v1 = at(acc, t + 1);
              const float other = __shfl_xor_sync(0xffffffffu, odd ? v0 : v1, 1);
              float a = odd ? other : v0, b = odd ? v1 : other;
              if (w0 + t + odd < w1 && f < p.N) {
                const size_t off = (size_t)(w0 + t + odd) * p.N + f - odd;
                if (p.residual) {
                  const float2 r = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(p.residual + off));
                  a += r.x;
                  b += r.y;
                }
                *reinterpret_cast<__nv_bfloat162*>(p.out + off) = __floats2bfloat162_rn(a, b);
              }
            }
          } else if (f < p.N) {
#pragma unroll
            for (int t = 0; t < WT; ++t)
              if (w0 + t < w1) {
                const size_t off = (size_t)(w0 + t) * p.N + f;
                p.out[off] = __float2bfloat16(at(acc, t) + (p.residual ? __bfloat162float(p.residual[off]) : 0.f));
              }
          }
        }
      } else {
        // ---- a cut tile: leave the partial sums; the last contributor adds them in K order
        const int i0 = p.owner(tile * p.kb), i1 = p.owner(tile * p.kb + p.kb - 1);
        // (a tile is the first of all its contributors but the first of them, and place() divides)
        const int first_place = p.place(i0, tile);
        auto part = [&](int i) { return p.partial + ((size_t)i * 2 + (i == i0 ? first_place : 0)) * (TOK * BM); };
        if (holds) {
          float* mine = part(worker) + w0 * BM + row;
#pragma unroll
          for (int t = 0; t < WT; ++t)
            if (w0 + t < w1) mine[t * BM] = at(acc, t);
          __threadfence();
        }
        epi_sync();
        if (threadIdx.x == 0) {
          int* cnt = p.counters + i0;
          const int prev = atomicAdd(cnt, 1);
          *fix_last = prev == i1 - i0;
          if (prev == i1 - i0) *cnt = 0;
        }
        epi_sync();
        if (*fix_last) {
          __threadfence();
          constexpr int U = TOK >= 64 ? 8 : TOK / 8;   // tokens of a thread in flight; warps take every eighth
          const int fc = tile * BM + lane * 4;
          for (int tb = warp; tb < p.T; tb += EPI_WARPS * U) {
            float4 s[U];
#pragma unroll
            for (int j = 0; j < U; ++j) s[j] = make_float4(0.f, 0.f, 0.f, 0.f);
            if constexpr (TOK < 64) {
              // eight values of a thread in flight, from several contributors: one after the other, each is a round trip to L2
              constexpr int B = 8 / U;
              for (int i = i0; i <= i1; i += B) {
                float4 v[B][U];
#pragma unroll
                for (int e = 0; e < B; ++e) {
                  const float* src = part(i + e) + tb * BM + lane * 4;
#pragma unroll
                  for (int j = 0; j < U; ++j)
                    if (i + e <= i1 && tb + EPI_WARPS * j < p.T)
                      v[e][j] = __ldcg(reinterpret_cast<const float4*>(src + EPI_WARPS * j * BM));
                }
#pragma unroll
                for (int e = 0; e < B; ++e)
#pragma unroll
                  for (int j = 0; j < U; ++j)
                    if (i + e <= i1 && tb + EPI_WARPS * j < p.T) {
                      s[j].x += v[e][j].x; s[j].y += v[e][j].y; s[j].z += v[e][j].z; s[j].w += v[e][j].w;
                    }
              }
            } else {
#pragma unroll 2
              for (int i = i0; i <= i1; ++i) {
                const float* src = part(i) + lane * 4;
#pragma unroll
                for (int j = 0; j < U; ++j)
                  if (tb + EPI_WARPS * j < p.T) {
                    const float4 v = __ldcg(reinterpret_cast<const float4*>(src + (tb + EPI_WARPS * j) * BM));
                    s[j].x += v.x; s[j].y += v.y; s[j].z += v.z; s[j].w += v.w;
                  }
              }
            }
#pragma unroll
            for (int j = 0; j < U; ++j) {
              if (tb + EPI_WARPS * j >= p.T) continue;
              const size_t off = (size_t)(tb + EPI_WARPS * j) * p.N + fc;
              float v[4] = {s[j].x, s[j].y, s[j].z, s[j].w};
              if (p.vec) {                       // four whole features
                if (fc >= p.N) continue;
                if (p.residual) {
                  const uint2 r = *reinterpret_cast<const uint2*>(p.residual + off);
                  const float2 a = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&r.x));
                  const float2 bq = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&r.y));
                  v[0] += a.x; v[1] += a.y; v[2] += bq.x; v[3] += bq.y;
                }
                uint2 o;
                *reinterpret_cast<__nv_bfloat162*>(&o.x) = __floats2bfloat162_rn(v[0], v[1]);
                *reinterpret_cast<__nv_bfloat162*>(&o.y) = __floats2bfloat162_rn(v[2], v[3]);
                *reinterpret_cast<uint2*>(p.out + off) = o;
              } else {
#pragma unroll
                for (int e = 0; e < 4; ++e)
                  if (fc + e < p.N) p.out[off + e] = __float2bfloat16(v[e] + (p.residual ? __bfloat162float(p.residual[off + e]) : 0.f));
              }
            }
          }
        }
      }
      u += len;
    }
  }

  tc_fence_before();
  __syncthreads();
  if (*abort_flag) {
    // let copies that may still be in flight land before shared memory is released
    const uint64_t t0 = globaltimer_ns();
    while (globaltimer_ns() - t0 < 200000ull) __nanosleep(1000);
    __syncthreads();
  }
  if (warp == WARP_MMA) {
    tc_fence_after();
    tmem_dealloc(tmem_base, L::TMEM_COLS);
  }
}

// Row kernels that leave their result as terms.  Eight neighbouring values per thread, sixteen threads per K block.
struct Eight {
  float v[8];
  // HALVES: `p` is aligned to 8 bytes only
  template <bool HALVES = false>
  __device__ __forceinline__ void load(const __nv_bfloat16* p) {
    uint4 u;
    if constexpr (HALVES) {
      const uint2 a = *reinterpret_cast<const uint2*>(p), b = *reinterpret_cast<const uint2*>(p + 4);
      u = make_uint4(a.x, a.y, b.x, b.y);
    } else {
      u = *reinterpret_cast<const uint4*>(p);
    }
    const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&u);
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const float2 f = __bfloat1622float2(h[i]);
      v[2 * i] = f.x;
      v[2 * i + 1] = f.y;
    }
  }
  // rounds the values to bf16 and stores them
  __device__ __forceinline__ uint4 round() {
    uint4 u;
    __nv_bfloat162* h = reinterpret_cast<__nv_bfloat162*>(&u);
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      h[i] = __floats2bfloat162_rn(v[2 * i], v[2 * i + 1]);
      const float2 f = __bfloat1622float2(h[i]);
      v[2 * i] = f.x;
      v[2 * i + 1] = f.y;
    }
    return u;
  }
};

template <bool HALVES>
__global__ void __launch_bounds__(256) split_terms_kernel(const __nv_bfloat16* __restrict__ x, int K, TermsOut o) {
  pdl_launch_dependents();
  pdl_wait();
  o.zero_counters(blockIdx.x == 0 && blockIdx.y == 0);
  const int i = (blockIdx.x * 256 + threadIdx.x) * 8, t = blockIdx.y;
  Eight e = {};
  if (i < K) e.load<HALVES>(x + (size_t)t * K + i);
  put_terms(o, t, i, e.v, i < K);
}

// silu(gate) up of rows [gate | up], rounded to bf16, as terms.
__global__ void __launch_bounds__(256) silu_mul_terms_kernel(const __nv_bfloat16* __restrict__ gu, int I, TermsOut o) {
  pdl_launch_dependents();
  pdl_wait();
  o.zero_counters(blockIdx.x == 0 && blockIdx.y == 0);
  const int i = (blockIdx.x * 256 + threadIdx.x) * 8, t = blockIdx.y;
  Eight g = {}, u = {};
  if (i < I) {
    g.load(gu + (size_t)t * 2 * I + i);
    u.load(gu + (size_t)t * 2 * I + I + i);
#pragma unroll
    for (int k = 0; k < 8; ++k) g.v[k] = g.v[k] / (1.f + __expf(-g.v[k])) * u.v[k];
    g.round();
  }
  put_terms(o, t, i, g.v, i < I);
}

// x (+= delta, written back) -> rmsnorm(x) (1 +) gamma in bf16: stored (out, optional) and as terms.  One block per row, V
// groups of eight values per thread, one pass over memory.
template <int V>
__global__ void __launch_bounds__(1024) rmsnorm_terms_kernel(__nv_bfloat16* __restrict__ x, const __nv_bfloat16* __restrict__ delta,
                                                             const __nv_bfloat16* __restrict__ gamma, __nv_bfloat16* __restrict__ out,
                                                             int cols, float eps, float one, TermsOut o) {
  __shared__ float part[32];
  pdl_launch_dependents();
  Eight g[V];                                  // constants: before the wait
#pragma unroll
  for (int j = 0; j < V; ++j) {
    const int i = (j * blockDim.x + threadIdx.x) * 8;
    if (i < cols) g[j].load(gamma + i);
  }
  pdl_wait();
  o.zero_counters(blockIdx.x == 0);
  const int t = blockIdx.x;
  Eight e[V];
  float ss = 0.f;
#pragma unroll
  for (int j = 0; j < V; ++j) {
    const int i = (j * blockDim.x + threadIdx.x) * 8;
    e[j] = {};
    if (i < cols) {
      const size_t at = (size_t)t * cols + i;
      e[j].load(x + at);
      if (delta) {
        Eight d;
        d.load(delta + at);
#pragma unroll
        for (int k = 0; k < 8; ++k) e[j].v[k] += d.v[k];
        *reinterpret_cast<uint4*>(x + at) = e[j].round();     // the norm takes the residual as it is stored
      }
#pragma unroll
      for (int k = 0; k < 8; ++k) ss += e[j].v[k] * e[j].v[k];
    }
  }
#pragma unroll
  for (int d = 16; d > 0; d >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, d);
  if ((threadIdx.x & 31) == 0) part[threadIdx.x >> 5] = ss;
  __syncthreads();
  ss = (threadIdx.x & 31) < blockDim.x / 32 ? part[threadIdx.x & 31] : 0.f;
#pragma unroll
  for (int d = 16; d > 0; d >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, d);
  const float inv = rsqrtf(ss / (float)cols + eps);
#pragma unroll
  for (int j = 0; j < V; ++j) {
    const int i = (j * blockDim.x + threadIdx.x) * 8;
    if (i < cols) {
#pragma unroll
      for (int k = 0; k < 8; ++k) e[j].v[k] *= inv * (one + g[j].v[k]);
      const uint4 r = e[j].round();
      if (out) *reinterpret_cast<uint4*>(out + (size_t)t * cols + i) = r;
    }
    put_terms(o, t, i, e[j].v, i < cols);
  }
}

template <int TOK>
static int launch(const Params& p, cudaStream_t stream) {
  using L = Cfg<TOK>;
  static b200::PerDeviceOnce once_;
  bool& configured = once_.slot();
  if (!configured) {
    cudaError_t e = cudaFuncSetAttribute(gemm_fp8_terms_kernel<TOK>, cudaFuncAttributeMaxDynamicSharedMemorySize, L::TOTAL);
    if (e != cudaSuccess) return (int)e;
    configured = true;
  }
  return (int)launch_pdl(gemm_fp8_terms_kernel<TOK>, dim3(p.workers), dim3(THREADS), L::TOTAL, stream, p);
}

// CTAs (pairs) that share `tiles` tiles of `kb` blocks.  Enough tiles: all of them, in equal runs.  Where every tile is cut more
// than once, each contributor costs the last one a read of its partial sums, about as long as two blocks of one CTA or four of a
// pair, so a tile takes some sqrt(kb / 2) (kb / 4) contributors at most; and a whole number of them, so that none works on two cut
// tiles.  us with its split, against all SMs: 576 x 7168 9.4 for 11.2 at 1 token, 14.5 for 25 at 64, 20 for 43 at 65, 36 for 63 on pairs
// at 129; 2048 x 5120 at 1, 64, 129 tokens 8.9 for 11, 14.8 for 18, 29 for 42; 5120 x 4096 9.7 for 11.9, 15.6 for 18, 30 for 36.
static int workers(int tiles, int kb, int cg) {
  const int all = sm_count() / cg;
  if (2 * tiles > all) return all < tiles * kb ? all : tiles * kb;
  int most = 1;
  while ((most + 1) * (most + 1) * 2 * cg <= kb) ++most;
  const int each = all / tiles < most + 1 ? all / tiles : most + 1;
  return tiles * (each < kb ? each : kb);
}

// Tokens of a tile for T tokens.
static int tile_tokens(int T) { return T <= 16 ? 16 : T <= 32 ? 32 : T <= 64 ? 64 : T <= MAX_SINGLE ? MAX_SINGLE : PAIR_TOK; }

}  // namespace f8t
}  // namespace b200

using namespace b200;

extern "C" {

// Tokens per tile of T-token terms, the counters that go with them, and the floats of partial sums of a product that takes them.
int b200_fp8_terms_plan(int T, int* tok, long long* partial_floats, int* counters) {
  if (T <= 0) return -ERR_BAD_ARG;
  const int tk = f8t::tile_tokens(T), cg = tk == f8t::PAIR_TOK ? 2 : 1;
  *tok = tk;
  *partial_floats = (long long)(sm_count() / cg) * 2 * tk * 128 * cg;
  *counters = sm_count();
  return 0;
}

static bool aligned(std::initializer_list<const void*> ptrs, int bytes) {
  uintptr_t all = 0;
  for (const void* p : ptrs) all |= reinterpret_cast<uintptr_t>(p);
  return all % bytes == 0;
}

static bool terms_out(f8t::TermsOut* o, int T, int K, int tok, void* xq, float* sx, void* rest, int* counters) {
  if (!xq || !sx || !rest || !counters || !aligned({xq, sx, rest}, 16)) return false;
  if (T <= 0 || T > 65535 || K <= 0 || (K % 128) != 0 || tok != f8t::tile_tokens(T)) return false;
  o->xq = reinterpret_cast<uint8_t*>(xq);
  o->sx = sx;
  o->rest = reinterpret_cast<__nv_bfloat16*>(rest);
  o->counters = counters;
  o->n_counters = sm_count();
  o->tok = tok;
  o->cap = tok == f8t::PAIR_TOK ? tok / 2 : tok;
  o->kb = K / 128;
  return true;
}

// x [T, K] bf16 -> xq: ceil(T / tok) * (K / 128) blocks of 256 tok bytes, sx: as many blocks of tok floats, rest: [T, K] bf16,
// counters: as many as b200_fp8_terms_plan says (zeroed).
int b200_split_terms(const void* x_bf16, int T, int K, int tok, void* xq, float* sx, void* rest, int* counters, cudaStream_t stream) {
  f8t::TermsOut o;
  // up to 32 rows need to be aligned to 8 bytes only, as they do for the weight-streaming kernel
  const bool halves = !aligned({x_bf16}, 16);
  if (!x_bf16 || (halves && (T > 32 || !aligned({x_bf16}, 8)))) return -ERR_BAD_ARG;
  if (!terms_out(&o, T, K, tok, xq, sx, rest, counters)) return -ERR_BAD_ARG;
  return (int)launch_pdl(halves ? f8t::split_terms_kernel<true> : f8t::split_terms_kernel<false>, dim3((K / 8 + 255) / 256, T), dim3(256),
                         0, stream, reinterpret_cast<const __nv_bfloat16*>(x_bf16), K, o);
}

// gu [T, 2 I] (gate | up) -> terms of bf16(silu(gate) up).
int b200_silu_mul_terms(const void* gu, int T, int I, int tok, void* xq, float* sx, void* rest, int* counters, cudaStream_t stream) {
  f8t::TermsOut o;
  if (!gu || !aligned({gu}, 16) || !terms_out(&o, T, I, tok, xq, sx, rest, counters)) return -ERR_BAD_ARG;
  return (int)launch_pdl(f8t::silu_mul_terms_kernel, dim3((I / 8 + 255) / 256, T), dim3(256), 0, stream,
                         reinterpret_cast<const __nv_bfloat16*>(gu), I, o);
}

// x [T, cols] (+= delta, written back when delta is given) -> out = rmsnorm(x) gamma (bf16, optional) and its terms.
int b200_rmsnorm_terms(void* x, const void* delta, const void* gamma, void* out, int T, int cols, float eps, int unit_offset, int tok,
                       void* xq, float* sx, void* rest, int* counters, cudaStream_t stream) {
  f8t::TermsOut o;
  if (!x || !gamma || !aligned({x, delta, gamma, out}, 16) || cols > 4 * 8192) return -ERR_BAD_ARG;
  if (!terms_out(&o, T, cols, tok, xq, sx, rest, counters)) return -ERR_BAD_ARG;
  auto* xp = reinterpret_cast<__nv_bfloat16*>(x);
  auto* dp = reinterpret_cast<const __nv_bfloat16*>(delta);
  auto* gp = reinterpret_cast<const __nv_bfloat16*>(gamma);
  auto* op = reinterpret_cast<__nv_bfloat16*>(out);
  const float one = unit_offset ? 1.f : 0.f;
  const int v = cols <= 8192 ? 1 : cols <= 16384 ? 2 : 4;
  const dim3 threads((cols / 8 / v + 31) / 32 * 32);
  if (v == 1) return (int)launch_pdl(f8t::rmsnorm_terms_kernel<1>, dim3(T), threads, 0, stream, xp, dp, gp, op, cols, eps, one, o);
  if (v == 2) return (int)launch_pdl(f8t::rmsnorm_terms_kernel<2>, dim3(T), threads, 0, stream, xp, dp, gp, op, cols, eps, one, o);
  return (int)launch_pdl(f8t::rmsnorm_terms_kernel<4>, dim3(T), threads, 0, stream, xp, dp, gp, op, cols, eps, one, o);
}

// Y = X W^T (+ residual) from the terms of X.  W: packed FP8 tiles (b200_gemm_wdec, wfmt 1), scales [ceil(N/128), K/128].
int b200_gemm_fp8_terms(const void* W, const float* scales, const void* xq, const float* sx, const void* rest, void* out_bf16,
                        const void* residual, int T, int N, int K, float* partial, int* counters, int* status, cudaStream_t stream) {
  if (!W || !scales || !xq || !sx || !rest || !out_bf16 || !partial || !counters || !aligned({W, xq, sx, rest, partial}, 16) ||
      T <= 0 || N <= 0 || K <= 0 || K % 128)
    return -ERR_BAD_ARG;
  const int tok = f8t::tile_tokens(T), cg = tok == f8t::PAIR_TOK ? 2 : 1;
  f8t::Params p;
  memset(&p, 0, sizeof(p));
  p.T = T; p.N = N; p.kb = K / 128;
  p.m_tiles = (N + 127) / 128;
  p.n_tiles = (T + tok - 1) / tok;
  const long long units = (long long)((p.m_tiles + cg - 1) / cg) * p.n_tiles * p.kb;
  if (units > 0x7fffffff) return -ERR_BAD_ARG;
  const int tiles = (int)(units / p.kb);
  p.workers = f8t::workers(tiles, p.kb, cg);
  // one CTA: one token tile, so tiles share nothing but the rows
  p.waves = cg == 1 || tiles <= p.workers ? 0 : tiles % p.workers ? tiles / p.workers - 1 : tiles / p.workers;
  p.units = (tiles - p.waves * p.workers) * p.kb;
  p.w = reinterpret_cast<const uint8_t*>(W);
  p.scales = scales;
  p.xq = reinterpret_cast<const uint8_t*>(xq);
  p.sx = sx;
  p.rest = reinterpret_cast<const __nv_bfloat16*>(rest);
  p.out = reinterpret_cast<__nv_bfloat16*>(out_bf16);
  p.residual = reinterpret_cast<const __nv_bfloat16*>(residual);
  p.partial = partial;
  p.counters = counters;
  p.status = status;
  p.vec = N % 8 == 0 && ((reinterpret_cast<uintptr_t>(out_bf16) | reinterpret_cast<uintptr_t>(residual)) & 15) == 0;
  if (cg == 2) return gemm_fp8_pair_launch(p, stream);
  if (tok == 16) return f8t::launch<16>(p, stream);
  if (tok == 32) return f8t::launch<32>(p, stream);
  if (tok == 64) return f8t::launch<64>(p, stream);
  return f8t::launch<f8t::MAX_SINGLE>(p, stream);
}

}  // extern "C"
