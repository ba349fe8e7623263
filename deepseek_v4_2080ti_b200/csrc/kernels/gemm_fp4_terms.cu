// Grouped products of routed experts with FP4 matrices on the block-scaled tensor pipe:
//   Y[row, N] = X[row, K] * W_e[N, K]^T,  W_e = E2M1 with one power-of-two scale (UE8M0) per 32 inputs.
//
// The weights keep their codes up to the tensor core: kind::mxf8f6f4 takes E2M1 operands and a UE8M0 scale per 32 inputs for either
// side, which tcgen05.cp brings to tensor memory as they are stored.  The activations, 8 significant bits in bf16, come as two E4M3
// terms of 4 bits under scales of their own, one per 32 inputs and term (mx_terms.cuh), stored as two rows each: a tile of t tokens is
// an operand of 2 t rows, so the weights are read once for both terms, and the epilogue adds the two accumulator columns of a token.
// Nothing is rounded on the way, all scales are applied by the tensor core, and a K block costs the epilogue nothing.
//
// The codes are the operand in tensor memory: warps put each in a byte of its own (two shifts and two ands for eight).  From shared
// memory a product of 128 features x 32 inputs takes 32 cycles to read the features alone, and shared memory has to take the codes
// in 8 of 16 bytes besides - by TMA (CU_TENSOR_MAP_DATA_TYPE_16U4_ALIGN16B) or by warps, both 1040 cycles for 256 x 128 weights at
// 16 rows, where HBM brings them in 740.  Cycles of a product of 128 features by N columns, features in shared memory / in tensor
// memory: N 32 40 / 16, 64 48 / 32, 128 64 / 64.
//
// Work: a tile is two blocks of 128 features and up to TOK rows of one expert.  Whole waves of tiles are dealt one per CTA, so that at
// any time the chip works on neighbouring tiles, which share rows (all features of an expert) or weights (its token tiles): of 2000
// tokens, the rows of the 148 experts that contiguous runs walk at once and the weights that pass between two uses of them do not fit
// L2.  The tiles that are left are cut into (tile, K block) runs of equal length, and a cut tile is finished by the contributor that
// arrives last, in K order.
//
// Roles: warps 0-7 epilogue, 8 weight copies, 9 MMA issuer, 10 activation copies and weight scales, 11 activation scales, 12-27 codes
// to tensor memory, two groups by turns (one group: 200 tokens 486 us for 444, 2000 tokens 779 for 738).  All waits are bounded.
//
// Measured, us for [gate | up] 4096 x 4096 and down 4096 x 2048 of 256 experts, top 6 (reading the experts that get a token once takes,
// at 6.43 TB/s, 8 and 4 for one token, 355 and 178 from 200 tokens on): 1 token 25, 17; 200 tokens 433, 230; 2000 tokens 670, 381.
// gemm_wdec_kernel.cuh, which turns every weight into bf16 on the CUDA cores: 1 token 47, 47; 2000 tokens 2218 together.
// What bounds it: one token, the fixed part of a launch and the sums of cut tiles; 200 tokens, the weight stream (5.3 TB/s) and the chain
// copy - spread - product of a stage; 2000 tokens, the same chain, with rows of 13 KB beside 17 KB of weights per stage.
#include <cuda_bf16.h>
#include <string.h>
#include "../ptx/sm100.cuh"
#include "launch.h"
#include "ops.h"
#include "per_device.h"
#include "tma_host.h"

namespace b200 {
namespace f4t {

constexpr int BM = 128;
constexpr int MT = 2, TOK = 64;              // feature blocks and rows of a tile
constexpr int EPI_WARPS = 8, EPI_THREADS = EPI_WARPS * 32;
constexpr int WARP_W = 8, WARP_MMA = 9, WARP_X = 10, WARP_S = 11, WARP_U = 12, U_WARPS = 4 * MT, U_GROUPS = 2;
constexpr int THREADS = (WARP_U + U_GROUPS * U_WARPS) * 32;
constexpr int CODE_BYTES = BM * 64;          // stored block: 128 rows x 128 inputs, codes as [32 inputs][row][16 bytes]
constexpr int SF_BYTES = BM * 4;             // and their scales, row r at 16 (r % 32) + 4 (r / 32), as tcgen05.cp takes them
constexpr int BLOCK_BYTES = CODE_BYTES + SF_BYTES;
constexpr int A_COLS = 32;                   // tensor memory columns of a block's codes, a byte each

struct Params {
  int R, N, kb, m_tiles, workers;
  int most;                         // contributors of a tile that is cut, at most
  const int4* work;                 // {expert, pair of feature blocks, first row, rows}
  const int* num_work;
  const uint8_t* w;                 // [expert][m_tile][kb][BLOCK_BYTES]
  const uint32_t* sf;               // [kb][R] scales of the larger terms, four of 32 inputs each
  const int* row_outside;           // [R] the row has values that are not in its terms,
  const __nv_bfloat16* rest;        // [R][K] which are here among zeros (other rows undefined)
  __nv_bfloat16* out;               // [R, N]
  float* partial;                   // [workers][2][MT][part_rows / 4][128][4]
  int part_rows;                    // rows of a tile in `partial`: partial_rows(R)
  int* counters;                    // [workers], zero, left zero
  int* status;
  int vec;                          // even rows of `out`
};

constexpr int X_BYTES = 2 * TOK * 128;
constexpr int X_STAGE = X_BYTES + (MT + 1) * SF_BYTES;
constexpr int D_COLS = MT * 2 * TOK;         // accumulators of a tile
constexpr int SA = 3;                        // code buffers in tensor memory
constexpr int SX = 7;                        // stages of terms and scales
constexpr int SR = (232448 - 2048 - SX * X_STAGE) / (MT * CODE_BYTES);     // stages of codes as they are stored
constexpr int A_COL = D_COLS, SF_COL = A_COL + SA * MT * A_COLS;
constexpr uint32_t TMEM_COLS = 512;
constexpr int SMEM = SX * X_STAGE + SR * MT * CODE_BYTES + 2048;
// rows of a tile that partial sums are kept for: with fewer than TOK in all, none has more
__host__ __device__ constexpr int partial_rows(int R) { return R < TOK ? (R + 3) / 4 * 4 : TOK; }
static_assert(SF_COL + (MT + 1) * 4 <= 512 && SX > SA && SR >= 4 && SMEM <= 232448, "tensor and shared memory");

__device__ __forceinline__ void epi_sync() { asm volatile("bar.sync 1, %0;" ::"n"(EPI_THREADS) : "memory"); }

// Scales of 128 rows x 4 in shared memory, row r at 16 (r % 32) + 4 (r / 32): eight-row groups of 16-byte rows, no swizzle.
__device__ __forceinline__ uint64_t desc_sf(const void* smem) {
  uint64_t d = 0;
  d |= (uint64_t)((smem_u32(smem) & 0x3FFFF) >> 4);
  d |= (uint64_t)(128 >> 4) << 32;
  d |= (uint64_t)1 << 46;
  return d;
}
// kind::mxf8f6f4 with E2M1 features, E4M3 tokens, UE8M0 scales; `k`: which of the four scales of a word.
__device__ __forceinline__ uint32_t idesc_mx(int n, int k) {
  return ((uint32_t)k << 4) | (5u << 7) | (0u << 10) | ((uint32_t)(n >> 3) << 17) | (1u << 23) | ((uint32_t)(BM >> 4) << 24) |
         ((uint32_t)k << 29);
}
__device__ __forceinline__ void umma_mx_warp(uint32_t on, uint32_t tmem_d, uint32_t tmem_a, uint64_t db, uint32_t idesc, uint32_t sfa,
                                             uint32_t sfb, uint32_t acc) {
  asm volatile(
      "{\n\t.reg .pred p, e;\n\t"
      "setp.ne.b32 e, %7, 0;\n\t"
      "setp.ne.b32 p, %6, 0;\n\t"
      "@e tcgen05.mma.cta_group::1.kind::mxf8f6f4.block_scale.scale_vec::1X [%0], [%1], %2, %3, [%4], [%5], p;\n\t}\n"
      :
      : "r"(tmem_d), "r"(tmem_a), "l"(db), "r"(idesc), "r"(sfa), "r"(sfb), "r"(acc), "r"(on)
      : "memory");
}
__device__ __forceinline__ void copy_sf_warp(uint32_t on, uint32_t tmem, uint64_t desc) {
  asm volatile(
      "{\n\t.reg .pred e;\n\t"
      "setp.ne.b32 e, %2, 0;\n\t"
      "@e tcgen05.cp.cta_group::1.32x128b.warpx4 [%0], %1;\n\t}\n"
      :
      : "r"(tmem), "l"(desc), "r"(on)
      : "memory");
}
__device__ __forceinline__ void tma_load_3d_warp(uint32_t on, void* smem_dst, const CUtensorMap* tmap, uint64_t* bar, int x, int y, int z) {
  asm volatile(
      "{\n\t.reg .pred e;\n\t"
      "setp.ne.b32 e, %6, 0;\n\t"
      "@e cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes"
      " [%0], [%1, {%3, %4, %5}], [%2];\n\t}\n"
      :
      : "r"(smem_u32(smem_dst)), "l"(tmap), "r"(smem_u32(bar)), "r"(x), "r"(y), "r"(z), "r"(on)
      : "memory");
}
// Weight of input k (of 128) in feature r of a stored block.
__device__ __forceinline__ float weight_at(const uint8_t* block, int r, int k) {
  const uint32_t code = __ldg(block + (k >> 5) * (BM * 16) + r * 16 + ((k & 31) >> 1)) >> (4 * (k & 1)) & 15u;
  const uint32_t e = __ldg(block + CODE_BYTES + (r & 31) * 16 + (r >> 5) * 4 + (k >> 5));
  const uint32_t m = code & 1u, x = code >> 1 & 3u;
  const float v = x ? __uint_as_float((126 + x) << 23 | m << 22) : 0.5f * m;
  const float s = e ? __uint_as_float(e << 23) : 0x1p-126f * 0.5f;
  return (code & 8u ? -v : v) * s;
}

__global__ void __launch_bounds__(THREADS, 1)
gemm_fp4_terms_kernel(const __grid_constant__ CUtensorMap tmX, Params p) {
  extern __shared__ uint8_t smem_raw_base[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw_base) + 1023) & ~uintptr_t(1023));
  uint8_t* sX = smem;                                  // [SX] terms: the larger ones, then the others
  uint8_t* sRaw = sX + SX * X_BYTES;                // [SR][MT] codes
  uint8_t* sSf = sRaw + SR * MT * CODE_BYTES;          // [SX][MT + 1] scales of the weights, scales of the terms
  uint64_t* bars = reinterpret_cast<uint64_t*>(sSf + SX * (MT + 1) * SF_BYTES);
  uint64_t* raw_full = bars;                  // [SR] codes landed
  uint64_t* raw_empty = raw_full + SR;        // [SR] codes read
  uint64_t* x_full = raw_empty + SR;          // [SX] terms and scales ready
  uint64_t* done = x_full + SX;               // [SX] products of the stage finished
  uint64_t* a_full = done + SX;               // [SA] codes in tensor memory
  uint64_t* acc_full = a_full + SA;           // accumulators readable
  uint64_t* acc_empty = acc_full + 1;         // and read
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(acc_empty + 1);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
  volatile int* epi_abort = abort_flag + 1;
  int* fix_last = const_cast<int*>(abort_flag) + 2;

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (threadIdx.x == 0) {
    for (int s = 0; s < SR; ++s) {
      mbar_init(&raw_full[s], 1);
      mbar_init(&raw_empty[s], U_WARPS);
    }
    for (int s = 0; s < SX; ++s) {
      mbar_init(&x_full[s], 2);                // the copies announce their bytes, the scales of the terms are written
      mbar_init(&done[s], 1);
    }
    for (int s = 0; s < SA; ++s) mbar_init(&a_full[s], U_WARPS);
    mbar_init(acc_full, 1);
    mbar_init(acc_empty, EPI_WARPS);
    *abort_flag = 0;
    *epi_abort = 0;
    mbar_fence_init();
  }
  if (warp == WARP_MMA) {
    tmem_alloc(tmem_slot, TMEM_COLS);
    tmem_relinquish();
  }
  if (warp == WARP_X && lane == 0) tma_prefetch_desc(&tmX);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  pdl_launch_dependents();
  pdl_wait();                                 // the work list, the terms and the counters are the previous kernels'

  const int tiles = *p.num_work, worker = blockIdx.x, waves = tiles / p.workers, tail = waves * p.workers;
  const int units = (tiles - tail) * p.kb;                    // of the tiles that are left, the first of them `tail`
  const size_t part_size = (size_t)MT * BM * p.part_rows;
  const int workers = max(min(p.workers, min(units, (tiles - tail) * p.most)), 1);          // those that have some of them
  auto first = [&](int i) { return (int)((long long)units * i / workers); };
  const int u0 = worker < workers ? first(worker) : 0, u1 = worker < workers ? first(worker + 1) : 0;
  // The pieces of tiles that this worker computes: f(tile, first K block, K blocks), until it returns false.
  auto for_pieces = [&](auto f) {
    for (int i = 0; i < waves; ++i)
      if (!f(i * p.workers + worker, 0, p.kb)) return;
    for (int u = u0; u < u1;) {
      const int t = u / p.kb, c0 = u - t * p.kb, len = min(p.kb - c0, u1 - u);
      if (!f(tail + t, c0, len)) return;
      u += len;
    }
  };
  auto blocks_of = [&](int tile, int4& e) {   // a tile's entry and how many feature blocks it has
    e = __ldg(p.work + tile);
    return min(MT, p.m_tiles - e.y * MT);
  };
  auto block_at = [&](const int4& e, int c) { return p.w + ((size_t)(e.x * p.m_tiles + e.y * MT) * p.kb + c) * BLOCK_BYTES; };
  auto fail = [&](int err) {
    if (lane == 0) atomicExch(p.status, err);
    *abort_flag = 1;
  };

  if (warp == WARP_W) {
    // ------------------------------------------------------------ weight copies
    const uint32_t on = elect_one();
    int it = 0;
    for_pieces([&](int tile, int c0, int len) {
      int4 e;
      const int n = blocks_of(tile, e);
      const uint8_t* src = block_at(e, c0);
      for (int c = 0; c < len; ++c, ++it, src += BLOCK_BYTES) {
        const int s = it % SR;
        const bool got = mbar_wait(&raw_empty[s], ((it / SR) & 1) ^ 1);
        if (!__all_sync(0xffffffffu, got && *abort_flag == 0)) {
          if (!got) fail(ERR_WAIT_STAGE);
          return false;
        }
        mbar_expect_tx_warp(on, &raw_full[s], n * CODE_BYTES);
        for (int m = 0; m < n; ++m)
          bulk_load_warp(on, sRaw + (s * MT + m) * CODE_BYTES, src + (size_t)m * p.kb * BLOCK_BYTES, CODE_BYTES, &raw_full[s]);
      }
      return true;
    });
  } else if (warp == WARP_X) {
    // ------------------------------------------------------------ activation copies, sixteen tokens at a time, and weight scales
    const uint32_t on = elect_one();
    int it = 0;
    for_pieces([&](int tile, int c0, int len) {
      int4 e;
      const int n = blocks_of(tile, e), nb = (e.w + 15) >> 4;
      const uint8_t* src = block_at(e, c0) + CODE_BYTES;
      for (int c = c0; c < c0 + len; ++c, ++it, src += BLOCK_BYTES) {
        const int s = it % SX;
        const bool got = mbar_wait(&done[s], ((it / SX) & 1) ^ 1);
        if (!__all_sync(0xffffffffu, got && *abort_flag == 0)) {
          if (!got) fail(ERR_WAIT_STAGE);
          return false;
        }
        mbar_expect_tx_warp(on, &x_full[s], nb * 2 * 2048 + n * SF_BYTES);
        for (int m = 0; m < n; ++m)
          bulk_load_warp(on, sSf + (s * (MT + 1) + m) * SF_BYTES, src + (size_t)m * p.kb * BLOCK_BYTES, SF_BYTES, &x_full[s]);
        for (int i = 0; i < nb; ++i) {
          tma_load_3d_warp(on, sX + s * X_BYTES + i * 2048, &tmX, &x_full[s], c * 128, e.z + i * 16, 0);
          tma_load_3d_warp(on, sX + s * X_BYTES + (nb + i) * 2048, &tmX, &x_full[s], c * 128, e.z + i * 16, 1);
        }
      }
      return true;
    });
  } else if (warp == WARP_S) {
    // ------------------------------------------------------------ activation scales, fetched PF blocks at a time, ahead of their use
    constexpr int PF = 4, WD = TOK / 32;
    int it = 0;
    for_pieces([&](int tile, int c0, int len) {
      int4 e;
      blocks_of(tile, e);
      const int nb = (e.w + 15) >> 4;
      uint32_t v[PF][WD], next[PF][WD];
      auto fetch = [&](int c, uint32_t (&d)[PF][WD]) {
#pragma unroll
        for (int j = 0; j < PF; ++j)
#pragma unroll
          for (int i = 0; i < WD; ++i) {
            const int t = i * 32 + lane, row = e.z + t;
            d[j][i] = c + j < len && row < p.R ? __ldg(p.sf + (size_t)(c0 + c + j) * p.R + row) : 0;
          }
      };
      fetch(0, next);
      for (int cb = 0; cb < len; cb += PF) {
#pragma unroll
        for (int j = 0; j < PF; ++j)
#pragma unroll
          for (int i = 0; i < WD; ++i) v[j][i] = next[j][i];
        fetch(cb + PF, next);
#pragma unroll
        for (int j = 0; j < PF; ++j) {
          if (cb + j >= len) break;
          const int s = it % SX;
          const bool got = mbar_wait(&done[s], ((it / SX) & 1) ^ 1);
          if (!__all_sync(0xffffffffu, got && *abort_flag == 0)) {
            if (!got) fail(ERR_WAIT_STAGE);
            return false;
          }
          uint32_t* dst = reinterpret_cast<uint32_t*>(sSf + (s * (MT + 1) + MT) * SF_BYTES);
          auto put = [&](int r, uint32_t word) { dst[(r & 31) * 4 + (r >> 5)] = word; };
#pragma unroll
          for (int i = 0; i < WD; ++i) {
            const int t = i * 32 + lane;
            if (t < nb * 16) {
              put(t, v[j][i]);
              put(nb * 16 + t, __vsubus4(v[j][i], 0x05050505u));     // the smaller terms: 2^-5
            }
          }
          fence_proxy_async_smem();
          __syncwarp();
          if (lane == 0) mbar_arrive(&x_full[s]);
          ++it;
        }
      }
      return true;
    });
  } else if (warp >= WARP_U) {
    // ------------------------------------------------------------ codes to tensor memory: a thread is a row of one feature block
    const int group = (warp - WARP_U) / U_WARPS, m = (warp - WARP_U) / 4 % MT, r = (warp & 3) * 32 + lane;
    int it = 0;
    for_pieces([&](int tile, int c0, int len) {
      int4 e;
      const bool busy = m < blocks_of(tile, e);
      for (int c = 0; c < len; ++c, ++it) {
        if (it % U_GROUPS != group) continue;
        const int sr = it % SR, sa = it % SA;
        bool got = true;
        if (it >= SA) got = mbar_wait(&done[(it - SA) % SX], ((it - SA) / SX) & 1);
        got = got && mbar_wait(&raw_full[sr], (it / SR) & 1);
        if (!__all_sync(0xffffffffu, got && *abort_flag == 0)) {
          if (!got) fail(ERR_WAIT_DEQUANT);
          return false;
        }
        if (busy) {
          const uint8_t* raw = sRaw + (sr * MT + m) * CODE_BYTES + r * 16;
          uint32_t v[32];
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            const uint4 q = *reinterpret_cast<const uint4*>(raw + j * (BM * 16));
            const uint32_t w[4] = {q.x, q.y, q.z, q.w};
#pragma unroll
            for (int i = 0; i < 4; ++i) {                // eight codes: the even ones, then the odd ones, in bits 2 to 5 of a byte
              v[j * 8 + i * 2] = w[i] << 2 & 0x3C3C3C3Cu;
              v[j * 8 + i * 2 + 1] = w[i] >> 2 & 0x3C3C3C3Cu;
            }
          }
          __syncwarp();
          if (lane == 0) mbar_arrive(&raw_empty[sr]);
          tc_fence_after();
          tmem_st_32x32(tmem_base + (uint32_t((warp & 3) * 32) << 16) + A_COL + (sa * MT + m) * A_COLS, v);
          tmem_st_wait();
          tc_fence_before();
        } else if (lane == 0) {
          mbar_arrive(&raw_empty[sr]);
        }
        __syncwarp();
        if (lane == 0) mbar_arrive(&a_full[sa]);
      }
      return true;
    });
  } else if (warp == WARP_MMA) {
    // -------------------------------------------------------------- MMA issuer
    const uint32_t on = elect_one();
    int it = 0, piece = 0, err = 0;
    for_pieces([&](int tile, int c0, int len) {
      int4 e;
      const int n = blocks_of(tile, e), cols = 2 * ((e.w + 15) >> 4) * 16;
      if (!mbar_wait(acc_empty, (piece & 1) ^ 1)) err = ERR_WAIT_ACC;
      for (int c = 0; c < len; ++c, ++it) {
        const int s = it % SX, sa = it % SA;
        if (!err && !mbar_wait(&x_full[s], (it / SX) & 1)) err = ERR_WAIT_TMA;
        if (!err && !mbar_wait(&a_full[sa], (it / SA) & 1)) err = ERR_WAIT_DEQUANT;
        if (__any_sync(0xffffffffu, err != 0 || *abort_flag != 0)) {
          err = (int)__reduce_max_sync(0xffffffffu, (unsigned)err);
          if (err) fail(err);
          *abort_flag = 1;
          return false;
        }
        tc_fence_after();
        const uint8_t* sf = sSf + s * (MT + 1) * SF_BYTES;
        const uint32_t sf_col = tmem_base + SF_COL;
#pragma unroll
        for (int m = 0; m < MT; ++m)
          if (m < n) copy_sf_warp(on, sf_col + 4 * m, desc_sf(sf + m * SF_BYTES));
        copy_sf_warp(on, sf_col + 4 * MT, desc_sf(sf + MT * SF_BYTES));
        const uint64_t db = umma_desc_sw128(sX + s * X_BYTES);
        // (inputs outside, feature blocks inside: 14 % slower)
#pragma unroll
        for (int m = 0; m < MT; ++m)
          if (m < n) {
#pragma unroll
            for (int k = 0; k < 4; ++k)
              umma_mx_warp(on, tmem_base + m * 2 * TOK, tmem_base + A_COL + (sa * MT + m) * A_COLS + 8 * k, db + 2 * k,
                           idesc_mx(cols, k), sf_col + 4 * m, sf_col + 4 * MT, c > 0 || k > 0);
          }
        umma_commit_warp(on, &done[s]);
      }
      umma_commit_warp(on, acc_full);
      ++piece;
      return true;
    });
  } else {
    // ---------------------------------------------------------------- epilogue: a thread is a feature of one of the tile's blocks
    const int row = (warp & 3) * 32 + lane, m = warp >> 2;
    int piece = 0;
    for_pieces([&](int tile, int c0, int len) {
      int4 e;
      const bool busy = m < blocks_of(tile, e);
      const int rows = e.w, nb = (rows + 15) >> 4;
      const int f = (e.y * MT + m) * BM + row;
      // tokens t, t + 1 of this thread's feature
      auto store2 = [&](int t, float v0, float v1) {
        if (p.vec) {                 // neighbouring lanes trade halves: each stores two features of one token
          const int odd = lane & 1;
          const float other = __shfl_xor_sync(0xffffffffu, odd ? v0 : v1, 1);
          if (t + odd < rows && f < p.N)
            *reinterpret_cast<__nv_bfloat162*>(p.out + (size_t)(e.z + t + odd) * p.N + f - odd) =
                __floats2bfloat162_rn(odd ? other : v0, odd ? v1 : other);
        } else if (f < p.N) {
          if (t < rows) p.out[(size_t)(e.z + t) * p.N + f] = __float2bfloat16(v0);
          if (t + 1 < rows) p.out[(size_t)(e.z + t + 1) * p.N + f] = __float2bfloat16(v1);
        }
      };
      int outside = 0;
      for (int t = lane; t < rows; t += 32) outside |= __ldg(p.row_outside + e.z + t);
      outside = __any_sync(0xffffffffu, outside != 0);
      const bool whole = len == p.kb && !outside;
      float* mine = p.partial + ((size_t)worker * 2 + (u0 / p.kb == tile - tail ? 0 : 1)) * part_size + m * p.part_rows * BM + row * 4;
      const bool ok = __all_sync(0xffffffffu, mbar_wait(acc_full, piece & 1));
      tc_fence_after();
      if (!ok) {
        fail(ERR_WAIT_ACC);
        *epi_abort = 1;
      } else {
        const uint32_t taddr = tmem_base + (uint32_t((warp & 3) * 32) << 16) + m * 2 * TOK;
        if (busy)
          for (int q = 0; q < nb; ++q) {
            uint32_t hi[16], mid[16];
            tmem_ld_32x16(taddr + q * 16, hi);
            tmem_ld_32x16(taddr + (nb + q) * 16, mid);
            tmem_ld_wait();
            if (whole) {
#pragma unroll
              for (int t = 0; t < 16; t += 2)
                store2(q * 16 + t, __uint_as_float(hi[t]) + __uint_as_float(mid[t]),
                       __uint_as_float(hi[t + 1]) + __uint_as_float(mid[t + 1]));
            } else {
              auto sum = [&](int t) { return __uint_as_float(hi[t]) + __uint_as_float(mid[t]); };
#pragma unroll
              for (int t = 0; t < 16; t += 4)
                if (q * 16 + t < rows)
                  *reinterpret_cast<float4*>(mine + (q * 16 + t) * BM) = make_float4(sum(t), sum(t + 1), sum(t + 2), sum(t + 3));
            }
          }
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(acc_empty);
      }
      epi_sync();
      if (*epi_abort) return false;
      if (!whole) {
        if (outside && busy) {
          // values outside the terms, on the CUDA cores: as a rule there are none
          const uint8_t* wb = block_at(e, c0) + (size_t)m * p.kb * BLOCK_BYTES;
          for (int t = 0; t < rows; ++t) {
            if (!__ldg(p.row_outside + e.z + t)) continue;
            const __nv_bfloat16* rest = p.rest + ((size_t)(e.z + t) * p.kb + c0) * 128;
            float sum = 0.f;
            for (int k = 0; k < len * 128; k += 8) {
              const uint4 q = __ldg(reinterpret_cast<const uint4*>(rest + k));
              if (!((q.x | q.y | q.z | q.w) & 0x7fff7fffu)) continue;
#pragma unroll
              for (int j = 0; j < 8; ++j) {
                const uint32_t word = j < 2 ? q.x : j < 4 ? q.y : j < 6 ? q.z : q.w;
                const uint32_t x = (j & 1 ? word >> 16 : word & 0xffffu) << 16;
                if (x & 0x7fffffffu) sum += __uint_as_float(x) * weight_at(wb + (size_t)(k >> 7) * BLOCK_BYTES, row, (k & 127) + j);
              }
            }
            mine[(t & ~3) * BM + (t & 3)] += sum;
          }
        }
        // ---- the last contributor of a cut tile adds the partial sums in K order
        const int a = (tile - tail) * p.kb, z = a + p.kb - 1;
        const bool cut = len != p.kb;
        const int i0 = cut ? (int)((((long long)a + 1) * workers - 1) / units) : worker;
        const int i1 = cut ? (int)((((long long)z + 1) * workers - 1) / units) : worker;
        __threadfence();
        epi_sync();
        if (threadIdx.x == 0) {
          const int prev = cut ? atomicAdd(p.counters + i0, 1) : 0;
          *fix_last = prev == i1 - i0;
          if (cut && prev == i1 - i0) p.counters[i0] = 0;
        }
        epi_sync();
        if (*fix_last && busy) {
          __threadfence();
          // contributors after the first one begin within the tile
          const int place = first(i0) / p.kb == tile - tail ? 0 : 1;
          const float* part = p.partial + m * p.part_rows * BM + row * 4;
          for (int t0 = 0; t0 < rows; t0 += 8) {
            float4 a = make_float4(0.f, 0.f, 0.f, 0.f), b = a;
#pragma unroll 4
            for (int i = i0; i <= i1; ++i) {
              const float* src = part + ((size_t)i * 2 + (i == i0 ? place : 0)) * part_size;
              const float4 c = __ldcg(reinterpret_cast<const float4*>(src + t0 * BM));
              const float4 d = t0 + 4 < rows ? __ldcg(reinterpret_cast<const float4*>(src + (t0 + 4) * BM)) : make_float4(0.f, 0.f, 0.f, 0.f);
              a.x += c.x; a.y += c.y; a.z += c.z; a.w += c.w;
              b.x += d.x; b.y += d.y; b.z += d.z; b.w += d.w;
            }
            store2(t0, a.x, a.y);
            store2(t0 + 2, a.z, a.w);
            store2(t0 + 4, b.x, b.y);
            store2(t0 + 6, b.z, b.w);
          }
        }
      }
      ++piece;
      return true;
    });
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
    tmem_dealloc(tmem_base, TMEM_COLS);
  }
}

}  // namespace f4t
}  // namespace b200

using namespace b200;

extern "C" {

// Rows of a tile of a grouped product, floats of the partial sums of one with R rows in all, tile counters.
int b200_fp4_terms_plan(int R, int* tok, long long* partial_floats, int* counters) {
  if (R <= 0) return -ERR_BAD_ARG;
  *tok = f4t::TOK;
  *partial_floats = (long long)sm_count() * 2 * f4t::MT * f4t::BM * f4t::partial_rows(R);
  *counters = sm_count();
  return 0;
}

// out [R, N] = rows times the FP4 matrices of their experts.  W: [groups][ceil(N/128)][K/128] blocks of 4 x 128 x 16 code bytes
// (low nibble first; 32 inputs of 128 features) and 512 scale bytes in the order of tcgen05.cp; work / num_work:
// b200_moe_plan_ordered (rows first) with ceil(N/256) tiles of as many rows as b200_fp4_terms_plan says; xq [2][R][K],
// sf [K/128][R][4], outside [R], rest [R][K]: b200_moe_gather_terms / b200_moe_glu_terms.  K % 128 == 0.
int b200_gemm_fp4_terms(const void* W, const void* xq, const void* sf, const int* outside, const void* rest, void* out_bf16, int R, int N,
                        int K, int groups, const void* work, const int* num_work, int max_work, float* partial, int* counters,
                        int* status, cudaStream_t stream) {
  const uintptr_t all = reinterpret_cast<uintptr_t>(W) | reinterpret_cast<uintptr_t>(xq) | reinterpret_cast<uintptr_t>(work) |
                        reinterpret_cast<uintptr_t>(rest) | reinterpret_cast<uintptr_t>(out_bf16) | reinterpret_cast<uintptr_t>(partial);
  if (!W || !xq || !sf || !outside || !rest || !out_bf16 || !work || !num_work || !partial || !counters || all % 16 || R <= 0 || N <= 0 ||
      K <= 0 || K % 128 || groups <= 0 || max_work <= 0 || (long long)max_work * (K / 128) > 0x7fffffff ||
      (long long)groups * ((N + 127) / 128) > 0x7fffffff)
    return -ERR_BAD_ARG;
  f4t::Params p;
  memset(&p, 0, sizeof(p));
  p.R = R; p.N = N; p.kb = K / 128;
  p.m_tiles = (N + 127) / 128;
  p.workers = sm_count();
  // A K block takes some 0.45 us, a contributor's sums of 16 rows 0.35 us to read: of the tiles that are left after whole waves, too
  // few for all SMs, each is shared by as many as make the sum of both least (8 experts of 4096 x 2048, 192 rows each: 170 us for 422
  // with all SMs on the last four tiles, 32 contributors each).
  const int rows = (R + groups - 1) / groups, sets = rows >= f4t::TOK ? f4t::TOK / 16 : (rows + 15) / 16;
  for (p.most = 1; (p.most + 1) * (p.most + 1) * 7 * sets <= 9 * p.kb;) ++p.most;
  p.work = reinterpret_cast<const int4*>(work);
  p.num_work = num_work;
  p.w = reinterpret_cast<const uint8_t*>(W);
  p.sf = reinterpret_cast<const uint32_t*>(sf);
  p.row_outside = outside;
  p.rest = reinterpret_cast<const __nv_bfloat16*>(rest);
  p.out = reinterpret_cast<__nv_bfloat16*>(out_bf16);
  p.partial = partial;
  p.part_rows = f4t::partial_rows(R);
  p.counters = counters;
  p.status = status;
  p.vec = N % 2 == 0;
  CUtensorMap tmX;
  if (!make_tmap_3d(&tmX, CU_TENSOR_MAP_DATA_TYPE_UINT8, xq, K, R, 2, K, (uint64_t)R * K, 128, 16, 1, CU_TENSOR_MAP_SWIZZLE_128B))
    return -ERR_BAD_ARG;
  static PerDeviceOnce once_;
  bool& configured = once_.slot();
  if (!configured) {
    cudaError_t e = cudaFuncSetAttribute(f4t::gemm_fp4_terms_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, f4t::SMEM);
    if (e != cudaSuccess) return (int)e;
    configured = true;
  }
  return (int)launch_pdl(f4t::gemm_fp4_terms_kernel, dim3(p.workers), dim3(f4t::THREADS), f4t::SMEM, stream, tmX, p);
}

}  // extern "C"
