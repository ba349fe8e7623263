// One prompt portion of a sequence through the layers of the hybrid decoder (models/qwen_hybrid.py), issued from native code: the
// launches of `_forward` for portions whose FP8 products take their activations as terms, on one rank, over a bf16 cache.  A layer is
// 13 launches; issued one by one from Python they take 1.8 ms for eight layers, longer than a portion of up to 300 tokens needs
// on the GPU.  Scratch comes from the caller, and no pointer is kept.
#include <stdint.h>
#include <string.h>
#include "launch.h"
#include "ops.h"

namespace {

// Positions, cache rows and lengths of a portion of T tokens after `past` others.
__global__ void portion_meta_kernel(const int* __restrict__ block_row, int past, int T, int block_size, int* __restrict__ pos,
                                    int* __restrict__ kv_slots, int* __restrict__ meta, long long* __restrict__ last_row) {
  b200::pdl_grid_trigger();
  b200::pdl_grid_wait();
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i == 0) {
    meta[0] = 0;
    meta[1] = T;
    meta[2] = past + T;
    *last_row = T - 1;
  }
  if (i >= T) return;
  const int p = past + i;
  pos[i] = p;
  kv_slots[i] = block_row[p / block_size] * block_size + p % block_size;
}

// What a decode step reads of its batch, row by row: {position, length with the new token, state slot, cache row}.  The values come as
// kernel arguments: an upload of a few hundred bytes, five copies and an indexing of the block table were 36 us before each step.
constexpr int META_ROWS = 128;
struct StepRows {
  int v[META_ROWS][4];
};
__global__ void step_meta_kernel(const __grid_constant__ StepRows rows, int row0, const int* __restrict__ ids, const int* __restrict__ tables,
                                 int max_blocks, int* __restrict__ o_ids, int* __restrict__ pos, int* __restrict__ kv_len,
                                 int* __restrict__ slots, int* __restrict__ kv_slots, int* __restrict__ bt) {
  b200::pdl_grid_trigger();
  b200::pdl_grid_wait();
  const int i = blockIdx.x, b = row0 + i;
  const int slot = rows.v[i][2];
  if (threadIdx.x == 0) {
    o_ids[b] = ids[b];
    pos[b] = rows.v[i][0];
    kv_len[b] = rows.v[i][1];
    slots[b] = slot;
    kv_slots[b] = rows.v[i][3];
  }
  for (int j = threadIdx.x; j < max_blocks; j += blockDim.x) bt[(size_t)b * max_blocks + j] = tables[(size_t)slot * max_blocks + j];
}

struct Arena {
  uint8_t* base;
  size_t used;
  void* take(size_t bytes) {
    void* at = base + used;
    used += (bytes + 255) / 256 * 256;
    return base ? at : nullptr;
  }
};

// A matrix of terms: activations and the counters of the products that take them (gemm_fp8_terms.cu).
struct Terms {
  int K;
  void *xq, *rest;
  float* sx;
  int* counters;
  void place(Arena& a, int T, int k, int tok, int n_counters) {
    const size_t blocks = (size_t)((T + tok - 1) / tok * (k / 128));
    K = k;
    xq = a.take(blocks * tok * 256);
    sx = reinterpret_cast<float*>(a.take(blocks * tok * 4));
    rest = a.take((size_t)T * k * 2);
    counters = reinterpret_cast<int*>(a.take((size_t)n_counters * 4));
  }
};

}  // namespace

extern "C" {

// All fields are 64 bits: models/qwen_hybrid.py fills them as arrays of integers, in this order.
struct B200QwenRowsLayer {
  long long linear;                                     // Gated DeltaNet layer, else attention
  const void *in_ln, *post_ln;
  const void* proj_w; const float* proj_s; long long proj_n;
  const void* out_w; const float* out_s; long long out_k, out_terms;      // out_terms: the output projection takes terms too
  const void* gate_up_w; const float* gate_up_s;
  const void* down_w; const float* down_s;
  const void* ab_w; const float *a_log, *dt_bias; const void *conv_w, *gdn_norm;
  void* tail; float* state;                             // of this sequence
  const void *q_norm, *k_norm; void *k_cache, *v_cache;
};
struct B200QwenRows {
  long long T, H, I, hq, hkv, hk, hv, output_gate, rot, block_size, max_blocks, num_blocks, window, sinks;
  const float* inv_freq;
  const int *positions, *kv_slots, *block_table, *q_start, *q_len, *kv_len;
  void *h, *delta;                                      // [T, H]: embedding in, residual out; what is still to be added to it
  uint8_t* scratch; long long scratch_bytes;
  int* status;
  long long launches;                                   // out
};

int b200_portion_meta(const int* block_row, int past, int T, int block_size, int* pos, int* kv_slots, int* meta, long long* last_row,
                      cudaStream_t stream) {
  if (!block_row || past < 0 || T <= 0 || block_size <= 0) return -6;
  return (int)b200::launch_pdl(portion_meta_kernel, dim3((T + 255) / 256), dim3(256), 0, stream, block_row, past, T, block_size, pos, kv_slots,
                               meta, last_row);
}

// rows: host array [B][4] as in StepRows; ids [B], tables [slots][max_blocks] on the device.
int b200_step_meta(const int* rows, int B, const int* ids, const int* tables, int max_blocks, int* o_ids, int* pos, int* kv_len, int* slots,
                   int* kv_slots, int* bt, cudaStream_t stream) {
  if (!rows || B <= 0 || max_blocks <= 0) return -6;
  for (int b = 0; b < B; b += META_ROWS) {
    StepRows part = {};
    const int n = B - b < META_ROWS ? B - b : META_ROWS;
    memcpy(part.v, rows + (size_t)b * 4, (size_t)n * 16);
    const cudaError_t e = b200::launch_pdl(step_meta_kernel, dim3(n), dim3(128), 0, stream, part, b, ids, tables, max_blocks, o_ids, pos, kv_len,
                                           slots, kv_slots, bt);
    if (e != cudaSuccess) return (int)e;
  }
  return 0;
}

// scratch == null: scratch_bytes is set to what a call needs, and nothing runs.  layer_words, row_words: 64-bit words of a layer and of
// `r` as the caller has them.
int b200_qwen_rows(const B200QwenRowsLayer* layers, int n_layers, int layer_words, B200QwenRows* r, int row_words, float eps,
                   float softmax_scale, cudaStream_t stream) {
  if (!layers || !r || layer_words * 8 != (int)sizeof(B200QwenRowsLayer) || row_words * 8 != (int)sizeof(B200QwenRows)) return -6;
  const int T = (int)r->T, H = (int)r->H, I = (int)r->I, hq = (int)r->hq, hkv = (int)r->hkv, hk = (int)r->hk, hv = (int)r->hv;
  const int kd = hk * 128, vd = hv * 128, cw = 2 * kd + vd, qd = hq * 128;
  int tok, counters;
  long long partial_floats;
  if (T <= 0 || b200_fp8_terms_plan(T, &tok, &partial_floats, &counters)) return -6;
  int widest = 0, deepest = I;
  bool any_linear = false, any_full = false;
  for (int i = 0; i < n_layers; ++i) {
    widest = layers[i].proj_n > widest ? (int)layers[i].proj_n : widest;
    deepest = layers[i].out_k > deepest ? (int)layers[i].out_k : deepest;
    (layers[i].linear ? any_linear : any_full) = true;
  }
  Arena a = {r->scratch, 0};
  const size_t t = T;
  Terms norm, act;
  norm.place(a, T, H, tok, counters);
  act.place(a, T, deepest, tok, counters);
  float* partial = reinterpret_cast<float*>(a.take((size_t)partial_floats * 4));
  void *x = a.take(t * H * 2), *d_attn = a.take(t * H * 2), *proj = a.take(t * widest * 2), *gu = a.take(t * 2 * I * 2);
  const size_t mixers = a.used;                     // a layer has one of the two
  float *g = nullptr, *beta = nullptr, *gdn_ws = nullptr;
  void *mixed = nullptr, *core = nullptr, *y = nullptr, *q = nullptr, *gate = nullptr, *attn = nullptr;
  if (any_linear) {
    g = reinterpret_cast<float*>(a.take(t * hv * 4));
    beta = reinterpret_cast<float*>(a.take(t * hv * 4));
    mixed = a.take(t * cw * 2);
    gdn_ws = reinterpret_cast<float*>(a.take((size_t)b200_gdn_workspace_floats(T, hv) * 4));
    core = a.take(t * vd * 2);
    y = a.take(t * vd * 2);
  }
  const size_t after_linear = a.used;
  if (any_full) {
    a.used = mixers;
    q = a.take(t * qd * 2);
    gate = r->output_gate ? a.take(t * qd * 2) : nullptr;
    attn = a.take(t * qd * 2);
    if (a.used < after_linear) a.used = after_linear;
  }
  if (!r->scratch) {
    r->scratch_bytes = (long long)a.used;
    return 0;
  }
  if ((long long)a.used > r->scratch_bytes) return -6;

  long long launches = 0;
  int rc = 0;
  auto ok = [&](int code, int n = 1) {
    if (!rc) rc = code;
    launches += n;
    return rc == 0;
  };
  auto product = [&](const Terms& m, const void* w, const float* s, void* out, int n) {
    return ok(b200_gemm_fp8_terms(w, s, m.xq, m.sx, m.rest, out, nullptr, T, n, m.K, partial, m.counters, r->status, stream));
  };
  auto normed = [&](const void* delta, const void* gamma, void* out) {
    return ok(b200_rmsnorm_terms(r->h, const_cast<void*>(delta), gamma, out, T, H, eps, 1, tok, norm.xq, norm.sx, norm.rest, norm.counters, stream));
  };
  const void* delta = nullptr;
  for (int i = 0; i < n_layers; ++i) {
    const B200QwenRowsLayer& L = layers[i];
    const int ldp = (int)L.proj_n;
    if (!normed(delta, L.in_ln, L.linear ? x : nullptr) || !product(norm, L.proj_w, L.proj_s, proj, ldp)) return rc;
    const void* mix;
    if (L.linear) {
      ok(b200_gdn_ab_gates(x, H, L.ab_w, L.a_log, L.dt_bias, g, beta, T, hv, stream));
      ok(b200_conv_silu(proj, ldp, L.conv_w, L.tail, mixed, cw, T, cw, 4, 1, stream));
      ok(b200_gdn_chunked(mixed, cw, 0, kd, 2 * kd, g, beta, L.state, core, gdn_ws, T, hv, hk, stream), 2);
      ok(b200_gated_rmsnorm(core, static_cast<uint8_t*>(proj) + (size_t)cw * 2, L.gdn_norm, y, (long long)T * hv, 128, eps, hv, ldp, stream));
      mix = y;
    } else {
      const int gate_mul = r->output_gate ? 2 : 1, qw = qd * gate_mul;
      ok(b200_qk_norm_rope_append(proj, ldp, 0, 128 * gate_mul, (int)r->output_gate, proj, ldp, qw, proj, ldp, qw + hkv * 128, L.q_norm, L.k_norm,
                                  1, eps, r->inv_freq, (int)r->rot, 1.0f, r->positions, r->kv_slots, q, gate, L.k_cache, L.v_cache,
                                  (int)r->block_size, T, hq, hkv, stream));
      ok(b200_gqa_prefill_ex(q, L.k_cache, L.v_cache, attn, gate, r->block_table, r->q_start, r->q_len, r->kv_len, 1, T, T, (int)r->max_blocks,
                             (int)r->num_blocks, (int)r->block_size, hq, hkv, softmax_scale, (int)r->window, (int)r->sinks, r->status, stream));
      mix = attn;
    }
    if (rc) return rc;
    if (L.out_terms) {
      act.K = (int)L.out_k;
      ok(b200_split_terms(mix, T, act.K, tok, act.xq, act.sx, act.rest, act.counters, stream));
      product(act, L.out_w, L.out_s, d_attn, H);
    } else {
      ok(b200_gemm_wdec(1, L.out_w, L.out_s, mix, d_attn, nullptr, nullptr, T, H, (int)L.out_k, 1, r->status, stream));
    }
    if (rc || !normed(d_attn, L.post_ln, nullptr) || !product(norm, L.gate_up_w, L.gate_up_s, gu, 2 * I)) return rc;
    act.K = I;
    ok(b200_silu_mul_terms(gu, T, I, tok, act.xq, act.sx, act.rest, act.counters, stream));
    if (rc || !product(act, L.down_w, L.down_s, r->delta, H)) return rc;
    delta = r->delta;
  }
  r->launches = launches;
  return rc;
}

}  // extern "C"
