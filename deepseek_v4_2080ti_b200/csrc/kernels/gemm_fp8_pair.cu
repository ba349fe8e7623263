// The products of gemm_fp8_terms.cu for more than 128 tokens, on CTA pairs (tcgen05.mma.cta_group::2):
//   Y[T, N] = X[T, K] * W[N, K]^T,  W = E4M3 with one scale per 128 x 128 block, X as two FP8 terms.
//
// Here the tokens are the MMA's M dimension: a pair computes 256 tokens x 256 features, each CTA its own 128 tokens, and a
// TMEM lane is a token.  The scale of a K block is then one number per thread (activation scale of its token x weight scale
// of its 128 features).  With the features as lanes, as in the one-CTA kernel, every thread needs the scales of all tokens:
// 32 shared-memory reads of 16 bytes per block and thread, beside operand traffic that already fills shared memory (112 KB
// per 1024 tensor cycles), doubled the time (978 against 670 us for 1920 x 34816 x 5120).
//
// Measured, us per product in a graph of 16 (12288 x 5120, 5120 x 4096, 34816 x 5120, 5120 x 17408): 333
// tokens 65, 35.5, 155, 79; 1901 tokens 205 to 260, 83 to 100, 553 to 643, 295 to 310 (the larger ones go with the power limit).  The split of
// the activations, 5 us at 333 tokens and 13 to 55 at 1901, is not counted.  The decode-warp kernel, which needs none, as it is
// now: 333 tokens 82, 40, 188, 138; 1901 tokens 266, 96, 790, 468.  Where it is the faster one with the split counted, `linear` takes it
// (terms_pay in ops/gemm.py).
//
// What bounds it: with two accumulators of 256 columns (all of tensor memory) the products of a block wait for the epilogue to have
// read the block before last; the tensor pipe is busy for 66 % of the cycles at 1901 tokens.  The epilogue's 216 registers are all
// in use and 52 bytes are spilled.
//
// Work: as long as there are more tiles than workers, every worker takes a whole tile of each run of as many tiles, so that at any time the
// chip works on neighbouring tiles, which share weights (all token tiles of a pair of weight tiles follow each other) and rows.  (With
// contiguous runs 74 workers hold the weights of 74 places and all rows live, 116 MB at 1901 x 34816 x 5120: L2 gave back 59 % of the
// operands, and without the products and the epilogue's reads of tensor memory it took 468 of 640 us.)  What is left, between one and
// two tiles a worker, is cut as in the one-CTA kernel.  The tokens past the last one of a tile are not staged when
// they fill a CTA, and not read back.  Roles: warps 0-7 epilogue (group of four: one weight tile of the pair), warp 8 weight
// copies, warp 9 MMA issuer (first CTA), warp 10 activation copies.  All waits are bounded.
#include <cuda_bf16.h>
#include <string.h>
#include "../ptx/sm100.cuh"
#include "fp8_terms.cuh"
#include "ops.h"
#include "per_device.h"
#include "tma_host.h"

namespace b200 {
namespace f8t {
namespace {

constexpr int EPI_WARPS = 8, EPI_THREADS = EPI_WARPS * 32;
constexpr int WARP_W = 8, WARP_MMA = 9, WARP_X = 10;
constexpr int PAIR_THREADS = 12 * 32;
constexpr int ROWS = PAIR_TOK / 2;                 // tokens of a CTA
constexpr int X_BYTES = 2 * ROWS * 128;
constexpr int S = 4, A = 2;
constexpr int SX_BYTES = ROWS * 4;
constexpr int SMEM = S * (W_BYTES + X_BYTES + SX_BYTES) + 2 * 2 * RUN * 4 + 2048;
constexpr int PART = ROWS * 2 * BM;                // floats of a CTA's share of a cut tile
static_assert(SMEM <= 232448, "shared memory");

__device__ __forceinline__ uint32_t ctarank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ uint32_t on_leader(const void* p) {
  uint32_t r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, 0;" : "=r"(r) : "r"(smem_u32(p)));
  return r;
}
__device__ __forceinline__ void cluster_sync_all() {
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// Arrival on the leader's barrier.  It orders tensor memory reads only (tcgen05 fence before it), no generic writes, so the
// default CTA-scope release is enough; a cluster-scope release per K block waits for the warp's outstanding memory traffic
// (152 instead of 87 us for 100 x 34816 x 5120, with the kernel otherwise as it then was).
__device__ __forceinline__ void remote_arrive(uint32_t cluster_bar_addr) {
  asm volatile("mbarrier.arrive.shared::cluster.b64 _, [%0];" ::"r"(cluster_bar_addr) : "memory");
}
// Load into this CTA's shared memory whose bytes are counted on a barrier of the pair's leader.
__device__ __forceinline__ void tma_load_pair(void* smem_dst, const CUtensorMap* tmap, uint32_t leader_bar, int x, int y) {
  asm volatile(
      "cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes"
      " [%0], [%1, {%3, %4}], [%2];"
      :
      : "r"(smem_u32(smem_dst)), "l"(tmap), "r"(leader_bar), "r"(x), "r"(y)
      : "memory");
}
__device__ __forceinline__ void epi_sync() { asm volatile("bar.sync 1, %0;" ::"n"(EPI_THREADS) : "memory"); }

// Adds to a thread's partial sums ([4 features][token]) what its token has outside its terms in K blocks c0 .. c0 + len - 1.  The
// warp calls it together; `rows`: how many of its tokens there are.  It works on memory because the sums' registers are few enough
// as it is (in registers: up to 1 % more for products that have no such values).
__device__ __forceinline__ void add_outside(const Params& p, float* sums, int m, int n, int c0, int len, int t0, int rows) {
  const int lane = threadIdx.x & 31;
#pragma unroll 1
  for (int c = c0; c < c0 + len; ++c) {
    const float* sx = p.sx + ((size_t)n * p.kb + c) * PAIR_TOK + t0;
    uint32_t tokens = __ballot_sync(0xffffffffu, lane < rows && __ldcg(sx + lane) < 0.f);
    const uint8_t* wb = p.w + ((size_t)m * p.kb + c) * W_BYTES;
    const float sw = __ldg(p.scales + (size_t)m * p.kb + c);
#pragma unroll 1
    for (; tokens; tokens &= tokens - 1) {
      const int src = __ffs(tokens) - 1;
      for_each_outside(p.rest, p.kb, n * PAIR_TOK + t0 + src, c, [&](int k, float x) {
        // the token's sums, four features a lane
        float* at = sums + (src - lane) * 4 + lane * (ROWS * 4);
        float4 v = *reinterpret_cast<float4*>(at);
        const float2 a = e4m3x2_to_float2(wb[w_offset(4 * lane, k)] | wb[w_offset(4 * lane + 1, k)] << 8);
        const float2 b = e4m3x2_to_float2(wb[w_offset(4 * lane + 2, k)] | wb[w_offset(4 * lane + 3, k)] << 8);
        v.x += x * (a.x * sw); v.y += x * (a.y * sw); v.z += x * (b.x * sw); v.w += x * (b.y * sw);
        *reinterpret_cast<float4*>(at) = v;
      });
    }
  }
}

__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(PAIR_THREADS, 1)
gemm_fp8_pair_kernel(const __grid_constant__ CUtensorMap tmW, const __grid_constant__ CUtensorMap tmX, Params p) {
  extern __shared__ uint8_t smem_raw_base[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw_base) + 1023) & ~uintptr_t(1023));
  uint8_t* sW = smem;
  uint8_t* sX = sW + S * W_BYTES;
  float* sSx = reinterpret_cast<float*>(sX + S * X_BYTES);
  float* sRun = sSx + S * ROWS;          // [2][2 weight tiles][RUN]
  uint64_t* bars = reinterpret_cast<uint64_t*>(sRun + 2 * 2 * RUN);
  uint64_t* full = bars;                 // [S] leader: both CTAs' operands landed
  uint64_t* sx_full = bars + S;          // [S] activation scales landed
  uint64_t* done = bars + 2 * S;         // [S] the block's MMAs are finished: accumulator readable
  uint64_t* slot_free = bars + 3 * S;    // [S] the epilogue is through with the block: slot reusable
  uint64_t* acc_free = bars + 4 * S;     // [A] leader: both CTAs' accumulators reusable
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 4 * S + A);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
  volatile int* epi_abort = abort_flag + 1;     // written by epilogue threads only, always before a barrier
  int* fix_last = const_cast<int*>(abort_flag) + 2;
  volatile int* last_outside = abort_flag + 3;  // the last block so far in which a token of this CTA has values outside its terms

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int rank = (int)ctarank();
  if (threadIdx.x == 0) {
    for (int s = 0; s < S; ++s) {
      mbar_init(&full[s], 2);             // weights and activations announce their bytes
      mbar_init(&sx_full[s], 1);
      mbar_init(&done[s], 1);
      mbar_init(&slot_free[s], EPI_WARPS);
    }
    for (int a = 0; a < A; ++a) mbar_init(&acc_free[a], 2 * EPI_WARPS);
    *abort_flag = 0;
    *epi_abort = 0;
    *last_outside = -1;
    mbar_fence_init();
  }
  if (warp == WARP_MMA) {
    asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], 512;" ::"r"(smem_u32(tmem_slot)) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
  }
  if (warp == WARP_W && lane == 0) {
    tma_prefetch_desc(&tmW);
    tma_prefetch_desc(&tmX);
  }
  tc_fence_before();
  __syncthreads();
  cluster_sync_all();        // the peer's barriers exist before anything is signalled across the pair
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");

  const int worker = blockIdx.x >> 1;
  Pieces piece(p, worker);

  // A thread of the epilogue holds 128 sums: its warps take registers from the others
  // (12 warps x 168 at launch; 8 x 32 x 216 + 4 x 32 x 64 = 63,488 of 64,512).
  if (warp >= EPI_WARPS) {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 64;");
    if (warp == WARP_W) {
      // ---------------------------------------------------------- weight copies, ahead of the previous kernel's end
      if (lane == 0) {
        bool ok = true;
        for (int blk = 0; ok && piece.next();) {
          // an odd last weight tile: its partner lies past the map and reads zeros
          const int m = (piece.tile / p.n_tiles) * 2 + rank;
          int row = (m * p.kb + piece.c0) * (W_BYTES / 256);
          for (int c = 0; c < piece.len; ++c, ++blk, row += W_BYTES / 256) {
            const int b = blk % S;
            ok = blk < S || mbar_wait(&slot_free[b], ((blk / S) & 1) ^ 1);
            if (!ok) atomicExch(p.status, ERR_WAIT_STAGE);
            if (!ok || *abort_flag) {
              ok = false;
              *abort_flag = 1;
              break;
            }
            if (rank == 0) mbar_expect_tx(&full[b], 2 * W_BYTES);
            tma_load_pair(sW + b * W_BYTES, &tmW, on_leader(&full[b]), 0, row);
          }
        }
      }
    } else if (warp == WARP_X) {
      // ---------------------------------------------------------- activation copies
      if (lane == 0) {
        pdl_wait();
        bool ok = true;
        for (int blk = 0; ok && piece.next();) {
          const int n = piece.tile % p.n_tiles;
          const bool both = p.T - n * PAIR_TOK > ROWS;       // else the second CTA has no tokens
          size_t xb = (size_t)n * p.kb + piece.c0;
          for (int c = 0; c < piece.len; ++c, ++blk, ++xb) {
            const int b = blk % S;
            ok = blk < S || mbar_wait(&slot_free[b], ((blk / S) & 1) ^ 1);
            if (!ok) atomicExch(p.status, ERR_WAIT_STAGE);
            if (!ok || *abort_flag) {
              ok = false;
              *abort_flag = 1;
              break;
            }
            if (rank == 0) mbar_expect_tx(&full[b], both ? 2 * X_BYTES : X_BYTES);
            if (rank == 0 || both)
              tma_load_pair(sX + b * X_BYTES, &tmX, on_leader(&full[b]), 0, (int)(xb * 2 + rank) * (X_BYTES / 256));
            mbar_expect_tx(&sx_full[b], SX_BYTES);
            bulk_load(sSx + b * ROWS, p.sx + xb * PAIR_TOK + rank * ROWS, SX_BYTES, &sx_full[b]);
          }
        }
      }
    } else if (warp == WARP_MMA && rank == 0) {
      // ---------------------------------------------------------- MMA issuer
      const uint32_t on = elect_one();
      constexpr uint32_t idesc_hi = umma_idesc_f8(2 * ROWS, 2 * BM, true), idesc_mid = umma_idesc_f8(2 * ROWS, 2 * BM);
      const int blocks = p.waves * p.kb + piece.u1 - piece.u;
      for (int blk = 0; blk < blocks; ++blk) {
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
        const uint64_t da = umma_desc_sw128(sX + b * X_BYTES), db = desc_sw64(sW + b * W_BYTES);
        // one instruction covers 32 K bytes: +32 bytes = +2 in 16-byte units
#pragma unroll
        for (int k = 0; k < 8; ++k)
          umma_f8_pair_warp(on, tmem_base + a * 2 * BM, da + (k >> 2) * (X_BYTES / 2 / 16) + 2 * (k & 3), db + w_step(k & 3),
                            k < 4 ? idesc_hi : idesc_mid, k > 0);
        commit_pair_warp(on, &done[b]);
      }
    }
  } else {
    asm volatile("setmaxnreg.inc.sync.aligned.u32 216;");
    // ------------------------------------------------------------ epilogue: one token, the 128 features of one weight tile
    const int group = warp >> 2, row = (warp & 3) * 32 + lane;
    float sc_a = 0.f, sc_b = 0.f;
    bool more = piece.next();
    auto fetch_scales = [&] {              // of the next piece, a piece ahead
      if (!more) return;
      const int m = min((piece.tile / p.n_tiles) * 2 + group, p.m_tiles - 1);
      const float* srow = p.scales + (size_t)m * p.kb + piece.c0;
      if (row < piece.len) sc_a = __ldg(srow + row);
      if (128 + row < piece.len) sc_b = __ldg(srow + 128 + row);
    };
    fetch_scales();
    pdl_wait();   // everything else this role reads, or writes, belongs after the previous kernel
    int run = 0, blk0 = 0;
    for (; more; ++run) {
      const int tile = piece.tile, c0 = piece.c0, len = piece.len;
      const int m = (tile / p.n_tiles) * 2 + group, n = tile % p.n_tiles;
      const int rows = min(PAIR_TOK, p.T - n * PAIR_TOK) - rank * ROWS;       // tokens of this CTA (0 and less: none)
      const bool busy = (warp & 3) * 32 < rows && m < p.m_tiles;
      const float* srow = p.scales + (size_t)min(m, p.m_tiles - 1) * p.kb + c0;
      float* sc_run = sRun + ((run & 1) * 2 + group) * RUN;
      sc_run[row] = sc_a;
      sc_run[128 + row] = sc_b;
      epi_sync();
      more = piece.next();
      fetch_scales();
      f2 acc[BM / 2];
#pragma unroll
      for (int i = 0; i < BM / 2; ++i) acc[i] = 0;
      bool ok = true;
      const float lim = row < rows ? 0.f : -INFINITY;      // scales of tokens past the last one are undefined
      for (int c = 0; c < len; ++c) {
        const int blk = blk0 + c, b = blk % S, a = blk % A;
        const float sw = c < RUN ? sc_run[c] : __ldg(srow + c);
        ok = mbar_wait(&sx_full[b], (blk / S) & 1) && mbar_wait(&done[b], (blk / S) & 1);
        ok = __all_sync(0xffffffffu, ok);
        if (!ok) break;
        tc_fence_after();
        // With two accumulators the tensor core waits for this chain, so it is kept short: half of the columns per read, and
        // the accumulator is given back when its last values are in registers, before they are used.
        auto give_back = [&] {
          tc_fence_before();
          __syncwarp();
          if (lane == 0) {
            mbar_arrive(&slot_free[b]);
            remote_arrive(on_leader(&acc_free[a]));
          }
        };
        if (busy) {
          const float sr = sSx[b * ROWS + row], sv = fabsf(sr) * sw;
          if (sr < lim) *last_outside = blk;
          const f2 s = pack2f(sv, sv);
          const uint32_t taddr = tmem_base + (uint32_t((warp & 3) * 32) << 16) + a * 2 * BM + group * BM;
#pragma unroll
          for (int half = 0; half < 2; ++half) {
            uint32_t v[2][32];
            tmem_ld_32x32(taddr + half * 64, v[0]);
            tmem_ld_32x32(taddr + half * 64 + 32, v[1]);
            tmem_ld_wait();
            if (half == 1) give_back();
#pragma unroll
            for (int i = 0; i < 32; ++i)
              acc[half * 32 + i] = fma2(pack2(v[i >> 4][2 * (i & 15)], v[i >> 4][2 * (i & 15) + 1]), s, acc[half * 32 + i]);
          }
        } else {
          give_back();
        }
      }
      if (!ok) {
        if (lane == 0) atomicExch(p.status, ERR_WAIT_ACC);
        *abort_flag = 1;
        *epi_abort = 1;
      }
      epi_sync();
      if (*epi_abort) break;
      const bool mine = busy && row < rows;
      // values outside the terms are added to the partial sums, so a tile that has some goes that way even if it is whole
      const bool outside = *last_outside >= blk0;
      bool store = len == p.kb && !outside;
      if (!store) {
        // ---- a cut tile: leave the partial sums; the last contributor adds them in K order
        const int tt = tile - p.tail();
        const bool cut = len != p.kb;
        const int i0 = cut ? p.owner(tt * p.kb) : worker, i1 = cut ? p.owner(tt * p.kb + p.kb - 1) : worker;
        auto part = [&](int i) {     // [4 features][token]; contributors after the first one begin within the tile
          return p.partial + (((size_t)i * 2 + (i > i0 ? 0 : p.place(i, tt))) * 2 + rank) * PART + (size_t)group * (ROWS * BM) + row * 4;
        };
        if (mine) {
          float* dst = part(worker);
#pragma unroll
          for (int j = 0; j < BM / 4; ++j)
            *reinterpret_cast<float4*>(dst + j * (ROWS * 4)) = make_float4(at(acc, 4 * j), at(acc, 4 * j + 1), at(acc, 4 * j + 2), at(acc, 4 * j + 3));
        }
        if (outside && busy) {
          __syncwarp();
          add_outside(p, part(worker), m, n, c0, len, rank * ROWS + (warp & 3) * 32, rows - (warp & 3) * 32);
        }
        if (busy) __threadfence();
        epi_sync();
        if (threadIdx.x == 0) {
          int* cnt = p.counters + i0 * 2 + rank;
          const int prev = cut ? atomicAdd(cnt, 1) : 0;
          *fix_last = prev == i1 - i0;
          if (cut && prev == i1 - i0) *cnt = 0;
        }
        epi_sync();
        store = *fix_last != 0;
        if (store && mine) {
          __threadfence();
#pragma unroll
          for (int j = 0; j < BM / 4; j += 8) {
            f2 sum[16];
#pragma unroll
            for (int e = 0; e < 16; ++e) sum[e] = 0;
#pragma unroll 1
            for (int i = i0; i <= i1; ++i) {
              const float* src = part(i) + j * (ROWS * 4);
              float4 v[8];
#pragma unroll
              for (int e = 0; e < 8; ++e) v[e] = __ldcg(reinterpret_cast<const float4*>(src + e * (ROWS * 4)));
#pragma unroll
              for (int e = 0; e < 8; ++e) {
                sum[2 * e] = add2(sum[2 * e], pack2f(v[e].x, v[e].y));
                sum[2 * e + 1] = add2(sum[2 * e + 1], pack2f(v[e].z, v[e].w));
              }
            }
#pragma unroll
            for (int e = 0; e < 16; ++e) acc[2 * j + e] = sum[e];
          }
        }
      }
      if (store && mine) {
        const size_t off = (size_t)(n * PAIR_TOK + rank * ROWS + row) * p.N + (size_t)m * BM;
        const int left = min(BM, p.N - m * BM);
        if (p.vec) {                     // rows of whole, aligned 16-byte groups
#pragma unroll
          for (int j = 0; j < BM; j += 8)
            if (j < left) {
              float v[8];
#pragma unroll
              for (int e = 0; e < 8; ++e) v[e] = at(acc, j + e);
              if (p.residual) {
                const uint4 r = *reinterpret_cast<const uint4*>(p.residual + off + j);
                const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&r);
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                  const float2 x = __bfloat1622float2(h[e]);
                  v[2 * e] += x.x;
                  v[2 * e + 1] += x.y;
                }
              }
              uint4 o;
              __nv_bfloat162* oh = reinterpret_cast<__nv_bfloat162*>(&o);
#pragma unroll
              for (int e = 0; e < 4; ++e) oh[e] = __floats2bfloat162_rn(v[2 * e], v[2 * e + 1]);
              *reinterpret_cast<uint4*>(p.out + off + j) = o;
            }
        } else {
#pragma unroll
          for (int j = 0; j < BM; ++j)
            if (j < left) p.out[off + j] = __float2bfloat16(at(acc, j) + (p.residual ? __bfloat162float(p.residual[off + j]) : 0.f));
        }
      }
      blk0 += len;
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
  cluster_sync_all();        // the peer may still signal, or read through the tensor core, until here
  if (warp == WARP_MMA) {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, 512;" ::"r"(tmem_base) : "memory");
  }
}

}  // namespace
}  // namespace f8t

// p.n_tiles counts tiles of PAIR_TOK tokens, p.units pairs of weight tiles.
int gemm_fp8_pair_launch(const f8t::Params& p, cudaStream_t stream) {
  using namespace f8t;
  static PerDeviceOnce once_;
  bool& configured = once_.slot();
  if (!configured) {
    cudaError_t e = cudaFuncSetAttribute(gemm_fp8_pair_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM);
    if (e != cudaSuccess) return (int)e;
    configured = true;
  }
  // both operands are stored in the order shared memory wants them: maps over rows of 256 bytes copy them as they lie
  CUtensorMap tmW, tmX;
  const uint64_t wr = (uint64_t)p.m_tiles * p.kb * (W_BYTES / 256), xr = (uint64_t)p.n_tiles * p.kb * PAIR_TOK;
  if (!make_tmap_2d(&tmW, CU_TENSOR_MAP_DATA_TYPE_UINT8, 1, p.w, wr, 256, 256, W_BYTES / 256, 256, CU_TENSOR_MAP_SWIZZLE_NONE) ||
      !make_tmap_2d(&tmX, CU_TENSOR_MAP_DATA_TYPE_UINT8, 1, p.xq, xr, 256, 256, X_BYTES / 256, 256, CU_TENSOR_MAP_SWIZZLE_NONE))
    return -ERR_BAD_ARG;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(p.workers * 2);
  cfg.blockDim = dim3(PAIR_THREADS);
  cfg.dynamicSmemBytes = SMEM;
  cfg.stream = stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  return (int)cudaLaunchKernelEx(&cfg, gemm_fp8_pair_kernel, tmW, tmX, p);
}

}  // namespace b200
