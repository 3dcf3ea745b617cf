// MoE grouped expert matmul for trellis 3INST experts:
//     out[t] = sum_j w[t,j] * W2_e( act( W13_e x_t ) ),   e = topk_ids[t,j]
// (reference: glq_fused_moe_trellis_3inst_cuda, glq/csrc/glq_cuda.cu:5042; eager loop
// glq_vllm/fused_moe_method.py:393-440; storage glq_vllm/moe_shapes.py:56-72).
//
// Six launches (eight kernels and a memset from 65536 routings, see moe_launch_group), fixed grids, no host
// synchronisation (capture-safe):
//   1 moe_group_kernel     count tokens per expert, prefix sums, place every (token, j) routing in a slot
//                          (tensor-core form: also the per-expert layer entries and the GEMM work lists)
//   2 moe_rht_in_kernel    input transform of every TOKEN once (all experts share SV of w13)
//   3 trellis_moe_mv_kernel  w13: experts' weights decoded once per 8*NB routed tokens, partial sums per slot
//   4 moe_mid_kernel       a few slots per CTA: sum partials, Wscale, output transform, SU, gated activation,
//                          then the w2 input transform (SV, Hadamard) — three reference launches in one
//                          (moe_mid_warp_kernel with enough routings, where no block is longer than 1024 values)
//   5 trellis_moe_mv_kernel  w2
//   6 moe_out_kernel       per token: its routings are the rows of one tile transform; then, for j in fixed
//                          order, acc += w * SU * H(Wscale * partials)
// Work units of the two matmuls are (expert, 32-row strip, K chunk) and are handed out by an atomic
// counter, so skewed routing (a few hot experts) does not idle the warps that drew empty experts; the
// partial-sum slot of a unit is its K-chunk number, so results do not depend on which warp ran it.
// Integer atomics decide only WHERE a routing is stored, never a numeric value: outputs are
// bit-identical run to run.
//
// Steps with enough routed tokens per expert (moe_gemm_min_avg) take the tensor-core form instead, E8 experts always:
// launches 3 and 5 become trellis_gemm_kernel (E8: glq_gemm_kernel) over a work list that the grouping kernel builds
// on the device from the expert counts — every expert is a "layer" whose token count, activation tiles and
// partial-sum rows are patched in each run; an expert's routings are split evenly over tiles of at most 160 (E8: 192), each
// padded to a multiple of 16.  The transforms write the activations straight into the swizzled tile images the GEMM's
// bulk copies fetch.
#include <algorithm>
#include <climits>
#include <cstdarg>
#include <cstdio>
#include <cstring>
#include <vector>

#include "glqb_kernels.cuh"
#include "glqb_gemm.cuh"
#include "glqb_tgemm.cuh"
#include "glqb_launch.h"

namespace glqb {

struct MoeDev {
  // weights, expert-stacked
  const uint8_t* w13[2];
  const uint8_t* w2[2];
  long long w13_stride[2], w2_stride[2];   // bytes between experts
  const __half* w13_su; const __half* w13_sv; const float* w13_wscale; const float* w13_inv2;
  const __half* w2_su; const __half* w2_sv; const float* w2_wscale; const float* w2_inv2;
  int E, hidden, inter, w13_out, top_k, max_tokens, act, gated;
  int ids_i64, x_dtype, y_dtype;
  int wide_m13;                        // some block of the w13 output is longer than a chunk of 1024
  // Hadamard blocks: n13 (hidden), m13 (w13_out), n2 (inter), m2 (hidden)
  int nb_n13, nb_m13, nb_n2, nb_m2;
  int off_n13[GLQB_MAX_BLOCKS], log_n13[GLQB_MAX_BLOCKS];
  int off_m13[GLQB_MAX_BLOCKS], log_m13[GLQB_MAX_BLOCKS];
  int off_n2[GLQB_MAX_BLOCKS], log_n2[GLQB_MAX_BLOCKS];
  int off_m2[GLQB_MAX_BLOCKS], log_m2[GLQB_MAX_BLOCKS];
  // K chunking of the two matmuls
  int kch13, gpc13, kch2, gpc2;
  // workspace offsets (bytes)
  long long o_count, o_base, o_cursor, o_work, o_route_tok, o_route_exp, o_slot_of, o_xr1, o_part1, o_xr2, o_part2;
  // tensor-core form (gemm != 0): tile rows, device-built layer tables and work lists
  int gemm, tile_tn, k13a, k13b, k2a, k2b, max_items13, max_items2;
  long long o_trow, o_row0, o_layers13, o_layers2, o_items13, o_items2, o_nitems, o_status;
  // E8 shell experts (format == GLQB_FMT_E8_SHELL; tensor-core form only): index matrices per stage,
  // expert-stacked, the packed tables, and the per-expert cumulative inverse residual scales of stages 2, 3
  int format, e8_ns;
  const uint8_t* e8_w13[3];
  const uint8_t* e8_w2[3];
  const uint32_t* e8_tab[3];
  int e8_ent[3];
  const float* e8_w13_inv[2];
  const float* e8_w2_inv[2];
};

// Routed tokens per GEMM tile: an expert's tokens are split evenly over ceil(count / tn) tiles, each padded to 16.  Trellis
// experts: 160, of which an item takes two, so that 320 tokens are one pass over the weights and tensor memory has a third
// stage of weights; E8 experts: 192.
constexpr int MOE_TN = 160, MOE_TN_E8 = 192;
__device__ __forceinline__ int moe_tile_tokens(int cnt, int tn) {           // tokens of an expert's tiles but the last
  const int n = max(1, (cnt + tn - 1) / tn);
  return max(16, ((cnt + n - 1) / n + 15) & ~15);
}
__device__ __forceinline__ int moe_tile_count(int cnt, int tn) {
  const int tt = moe_tile_tokens(cnt, tn);
  return (cnt + tt - 1) / tt;
}
__device__ __forceinline__ int moe_tile_rows(int cnt, int tn) {             // 128-byte activation rows of an expert's tiles, per chunk
  const int n = moe_tile_count(cnt, tn), tt = moe_tile_tokens(cnt, tn);
  return n ? (n - 1) * tt + ((cnt - (n - 1) * tt + 15) & ~15) : 0;
}
// where routing number i of an expert (activation rows from `row0` on) has its row: rows in front of its tile, and
// rows of the tile << 16 | row inside it
__device__ __forceinline__ int2 moe_tile_place(int cnt, int tn, int row0, int i) {
  const int tt = moe_tile_tokens(cnt, tn), j = i / tt, left = cnt - j * tt;
  return make_int2(row0 + j * tt, (left >= tt ? tt : (left + 15) & ~15) << 16 | (i - j * tt));
}

__device__ __forceinline__ float moe_act(float g, int act) {
  if (act == GLQB_ACT_SILU || act == 3) return g / (1.0f + __expf(-g));
  if (act == GLQB_ACT_GELU_TANH) {
    // (2-norm of the error over N(0, 1): 3.8e-8 of the result's; g / (1 + __expf(-2u)) is 0.5 % of a step faster at 4.9e-8)
    const float u = 0.7978845608028654f * (g + 0.044715f * g * g * g);
    return 0.5f * g * (1.0f + tanhf(u));
  }
  if (act == 4) return 0.5f * g * (1.0f + erff(g * 0.7071067811865476f));     // gelu (exact), not gated
  const float r = fmaxf(g, 0.f);                                                 // relu^2 (codes 2 and 5)
  return r * r;
}

// ---- 1: grouping ------------------------------------------------------------------------------------
// phase 0: one launch of up to 32 CTAs.  Every CTA counts all routings (their ids come from L2), so that each knows the
// counts, the prefix sums and how many routings of an expert lie in front of its own share; tables and placements are
// shared out, and nothing has to be cleared first.  phase 1: the counts were made by moe_count_kernel and the
// routings are placed by moe_place_kernel (many CTAs each); this kernel only does the prefix sums and tables.
constexpr int MOE_GROUP_CHUNK = 8192;          // routings per CTA of the count / place kernels
constexpr int MOE_GROUP_SPLIT_MIN = 65536;     // routings from which the three-kernel form is used
constexpr int MOE_GROUP_SHARE = 256, MOE_GROUP_CTAS = 32;      // routings per CTA of the one-launch form, most CTAs

__device__ __forceinline__ int moe_expert_of(const MoeDev& M, const void* ids, int i) {
  const long long v = M.ids_i64 ? reinterpret_cast<const long long*>(ids)[i] : (long long)reinterpret_cast<const int*>(ids)[i];
  return (v < 0 || v >= M.E) ? -1 : (int)v;
}

__global__ void __launch_bounds__(1024) moe_count_kernel(const __grid_constant__ MoeDev M, const void* __restrict__ ids,
                                                         int T, uint8_t* __restrict__ ws) {
  extern __shared__ int sh[];            // counts[E] of this CTA's chunk
  const int R = T * M.top_k;
  for (int e = threadIdx.x; e < M.E; e += blockDim.x) sh[e] = 0;
  __syncthreads();
  const int i0 = blockIdx.x * MOE_GROUP_CHUNK + threadIdx.x;
  int ev[8];
#pragma unroll
  for (int u = 0; u < 8; ++u) { const int i = i0 + u * 1024; ev[u] = i < R ? moe_expert_of(M, ids, i) : -1; }
#pragma unroll
  for (int u = 0; u < 8; ++u) if (ev[u] >= 0) atomicAdd(&sh[ev[u]], 1);
  __syncthreads();
  int* g_count = reinterpret_cast<int*>(ws + M.o_count);
  for (int e = threadIdx.x; e < M.E; e += blockDim.x) if (sh[e]) atomicAdd(&g_count[e], sh[e]);
}

// Each CTA reserves, per expert, a contiguous run of slots for its chunk's routings (one global atomic per
// expert and CTA) and places them with shared-memory atomics.
__global__ void __launch_bounds__(1024) moe_place_kernel(const __grid_constant__ MoeDev M, const void* __restrict__ ids,
                                                         int T, uint8_t* __restrict__ ws) {
  extern __shared__ int sh[];            // counts[E], then cursor[E]
  int* cnt = sh;
  int* cur = sh + M.E;
  const int R = T * M.top_k;
  for (int e = threadIdx.x; e < M.E; e += blockDim.x) cnt[e] = 0;
  __syncthreads();
  const int i0 = blockIdx.x * MOE_GROUP_CHUNK + threadIdx.x;
  int ev[8];
#pragma unroll
  for (int u = 0; u < 8; ++u) { const int i = i0 + u * 1024; ev[u] = i < R ? moe_expert_of(M, ids, i) : -1; }
#pragma unroll
  for (int u = 0; u < 8; ++u) if (ev[u] >= 0) atomicAdd(&cnt[ev[u]], 1);
  __syncthreads();
  int* g_cursor = reinterpret_cast<int*>(ws + M.o_cursor);
  for (int e = threadIdx.x; e < M.E; e += blockDim.x) cur[e] = cnt[e] ? atomicAdd(&g_cursor[e], cnt[e]) : 0;
  __syncthreads();
  const int* g_base = reinterpret_cast<const int*>(ws + M.o_base);
  const int* g_row0 = reinterpret_cast<const int*>(ws + M.o_row0);
  const int* g_count = reinterpret_cast<const int*>(ws + M.o_count);
  int* route_tok = reinterpret_cast<int*>(ws + M.o_route_tok);
  int* route_exp = reinterpret_cast<int*>(ws + M.o_route_exp);
  int* slot_of = reinterpret_cast<int*>(ws + M.o_slot_of);
  int2* trow = reinterpret_cast<int2*>(ws + M.o_trow);
#pragma unroll
  for (int u = 0; u < 8; ++u) {
    const int i = i0 + u * 1024;
    if (i < R) {
      int slot = -1;
      if (ev[u] >= 0) {
        slot = atomicAdd(&cur[ev[u]], 1);
        route_tok[slot] = i / M.top_k;
        route_exp[slot] = ev[u];
        if (M.gemm) trow[slot] = moe_tile_place(g_count[ev[u]], M.tile_tn, g_row0[ev[u]], slot - g_base[ev[u]]);
      }
      slot_of[i] = slot;
    }
  }
}

__global__ void __launch_bounds__(1024) moe_group_kernel(const __grid_constant__ MoeDev M, const void* __restrict__ ids,
                                                         int T, uint8_t* __restrict__ ws, int phase) {
  extern __shared__ int sh[];            // counts[E], cursor[E], first slot[E], first token tile[E + 1], first row[E], in front[E]
  pdl_trigger();
  int* cnt = sh;
  int* cur = sh + M.E;
  int* base_s = sh + 2 * M.E;
  int* tile0 = sh + 3 * M.E;
  int* row0 = sh + 4 * M.E + 1;
  int* front = sh + 5 * M.E + 1;         // routings of the expert in front of this CTA's share
  int* g_count = reinterpret_cast<int*>(ws + M.o_count);
  int* g_base = reinterpret_cast<int*>(ws + M.o_base);
  int* g_work = reinterpret_cast<int*>(ws + M.o_work);
  int* route_tok = reinterpret_cast<int*>(ws + M.o_route_tok);
  int* route_exp = reinterpret_cast<int*>(ws + M.o_route_exp);
  int* slot_of = reinterpret_cast<int*>(ws + M.o_slot_of);
  const int R = T * M.top_k;
  const int per_item = M.format == GLQB_FMT_E8_SHELL ? 1 : 2;        // token tiles of a work item
  const int share = (R + (int)gridDim.x - 1) / (int)gridDim.x, lo = (int)blockIdx.x * share, hi = min(R, lo + share);
  const int tid = (int)(blockIdx.x * blockDim.x + threadIdx.x), step = (int)(gridDim.x * blockDim.x);
  for (int e = threadIdx.x; e < M.E; e += blockDim.x) cnt[e] = front[e] = 0;
  if (tid < 2) g_work[tid] = 0;
  __syncthreads();
  auto expert_of = [&](int i) -> int { return moe_expert_of(M, ids, i); };
  if (phase == 0) {
    // 8 routings per thread and round: the id loads of a round are issued together
    for (int i0 = threadIdx.x; i0 < R; i0 += 8 * blockDim.x) {
      int ev[8];
#pragma unroll
      for (int u = 0; u < 8; ++u) { const int i = i0 + u * blockDim.x; ev[u] = i < R ? expert_of(i) : -1; }
#pragma unroll
      for (int u = 0; u < 8; ++u)
        if (ev[u] >= 0) {
          atomicAdd(&cnt[ev[u]], 1);
          if (i0 + u * (int)blockDim.x < lo) atomicAdd(&front[ev[u]], 1);
        }
    }
  } else {
    __syncthreads();
    for (int e = threadIdx.x; e < M.E; e += blockDim.x) cnt[e] = g_count[e];
  }
  __syncthreads();
  if (threadIdx.x < 32) {
    // running sums over the experts: slots, token tiles, activation rows
    int run = 0, tiles = 0, rows = 0;
    for (int e0 = 0; e0 < M.E; e0 += 32) {
      const int e = e0 + threadIdx.x, c = e < M.E ? cnt[e] : 0;
      const int nt = (moe_tile_count(c, M.tile_tn) + per_item - 1) / per_item, nr = moe_tile_rows(c, M.tile_tn);
      int a = c, b = nt, d = nr;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int pa = __shfl_up_sync(0xffffffffu, a, o), pb = __shfl_up_sync(0xffffffffu, b, o), pd = __shfl_up_sync(0xffffffffu, d, o);
        if ((int)threadIdx.x >= o) { a += pa; b += pb; d += pd; }
      }
      if (e < M.E) { base_s[e] = run + a - c; cur[e] = base_s[e] + front[e]; tile0[e] = tiles + b - nt; row0[e] = rows + d - nr; }
      run += __shfl_sync(0xffffffffu, a, 31);
      tiles += __shfl_sync(0xffffffffu, b, 31);
      rows += __shfl_sync(0xffffffffu, d, 31);
    }
    if (threadIdx.x == 0) tile0[M.E] = tiles;
  }
  __syncthreads();
  if (blockIdx.x == 0) {
    int* g_cursor = reinterpret_cast<int*>(ws + M.o_cursor);
    int* g_row0 = reinterpret_cast<int*>(ws + M.o_row0);
    for (int e = threadIdx.x; e < M.E; e += blockDim.x) {
      g_base[e] = base_s[e]; g_count[e] = cnt[e]; g_cursor[e] = base_s[e]; g_row0[e] = row0[e];
    }
  }
  int2* trow = reinterpret_cast<int2*>(ws + M.o_trow);
  if (M.gemm) {
    // Tensor-core form.  Expert e with c routings owns moe_tile_count(c) token tiles; routing number i of the expert
    // sits where moe_tile_place says.  Every expert becomes a "layer" of the GEMM kernel (token count, activations and
    // partial-sum rows of this step), and the work list is ordered (token tile, row tile) so that the CTAs working at
    // one moment share an activation tile in L2.
    const int kc13 = M.hidden / GM_TILE_K, kc2 = M.inter / GM_TILE_K;
    const int mt13 = (M.w13_out + GM_TILE_M - 1) / GM_TILE_M, mt2 = (M.hidden + GM_TILE_M - 1) / GM_TILE_M;
    const int tiles = tile0[M.E];
    if (tid == 0) {
      int* nitems = reinterpret_cast<int*>(ws + M.o_nitems);
      nitems[0] = min(tiles * mt13, M.max_items13);
      nitems[1] = min(tiles * mt2, M.max_items2);
      reinterpret_cast<int*>(ws + M.o_status)[0] = 0;
    }
    DevLinear* L13 = reinterpret_cast<DevLinear*>(ws + M.o_layers13);
    DevLinear* L2 = reinterpret_cast<DevLinear*>(ws + M.o_layers2);
    // (field by field: only what the GEMM kernel reads; thread 2e writes expert e's w13 entry, 2e + 1 its w2 entry)
    for (int i = tid; i < 2 * M.E; i += step) {
      const int e = i >> 1;
      const bool second = i & 1;
      DevLinear& a = (second ? L2 : L13)[e];
      a.batch = cnt[e];
      a.m = second ? M.hidden : M.w13_out;
      a.n = second ? M.inter : M.hidden;
      a.strips = a.m / 32;
      a.groups_per_strip = a.n / 32;
      a.xr_off = (second ? M.o_xr2 : M.o_xr1) + (long long)row0[e] * (second ? kc2 : kc13) * 128;
      a.part_off = (second ? M.o_part2 : M.o_part1) + (long long)base_s[e] * (second ? M.hidden : M.w13_out) * 4;
      a.stage_scale[0] = 1.f;
      if (M.format == GLQB_FMT_E8_SHELL) {
        for (int s = 0; s < M.e8_ns; ++s) {
          a.codes[s] = (second ? M.e8_w2[s] : M.e8_w13[s]) + (long long)e * (second ? M.w2_stride[0] : M.w13_stride[0]);
          a.table[s] = M.e8_tab[s];
          a.table_entries[s] = M.e8_ent[s];
          if (s) a.stage_scale[s] = (second ? M.e8_w2_inv : M.e8_w13_inv)[s - 1][e];
        }
      } else {
        const uint8_t* const* w = second ? M.w2 : M.w13;
        const long long* st = second ? M.w2_stride : M.w13_stride;
        const float* inv = second ? M.w2_inv2 : M.w13_inv2;
        a.codes[0] = w[0] + (long long)e * st[0];
        a.codes[1] = w[1] ? w[1] + (long long)e * st[1] : nullptr;
        a.stage_scale[1] = inv ? inv[e] : 0.f;
      }
    }
    auto expert_of_tile = [&](int tile) -> int {       // last e with tile0[e] <= tile
      int lo = 0, hi = M.E - 1;
      while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (tile0[mid] <= tile) lo = mid; else hi = mid - 1;
      }
      return lo;
    };
    GemmItem* I13 = reinterpret_cast<GemmItem*>(ws + M.o_items13);
    GemmItem* I2 = reinterpret_cast<GemmItem*>(ws + M.o_items2);
    auto item = [&](int tile, int mt, int kc) -> GemmItem {
      const int e = expert_of_tile(tile), j = (tile - tile0[e]) * per_item, tt = moe_tile_tokens(cnt[e], M.tile_tn), left = cnt[e] - j * tt;
      return GemmItem{e, mt, j, 0, kc, 0, j * tt, min(tt, left), j * tt, per_item > 1 ? max(0, min(tt, left - tt)) : 0};
    };
    for (int idx = tid; idx < min(tiles * mt13, M.max_items13); idx += step) I13[idx] = item(idx / mt13, idx % mt13, kc13);
    for (int idx = tid; idx < min(tiles * mt2, M.max_items2); idx += step) I2[idx] = item(idx / mt2, idx % mt2, kc2);
  }
  if (phase != 0) return;
  for (int i0 = lo + (int)threadIdx.x; i0 < hi; i0 += 8 * blockDim.x) {
    int ev[8];
#pragma unroll
    for (int u = 0; u < 8; ++u) { const int i = i0 + u * blockDim.x; ev[u] = i < hi ? expert_of(i) : -1; }
#pragma unroll
    for (int u = 0; u < 8; ++u) {
      const int i = i0 + u * blockDim.x;
      if (i < hi) {
        int slot = -1;
        if (ev[u] >= 0) {
          slot = atomicAdd(&cur[ev[u]], 1);
          route_tok[slot] = i / M.top_k;
          route_exp[slot] = ev[u];
          if (M.gemm) trow[slot] = moe_tile_place(cnt[ev[u]], M.tile_tn, row0[ev[u]], slot - base_s[ev[u]]);
        }
        slot_of[i] = slot;
      }
    }
  }
}

// Columns c .. c + 3 (c % 4 == 0) of a token's activations in the streaming kernels' fragment order.
__device__ __forceinline__ void moe_store_xr4(__half2* row, int c, const f2 (&q)[2]) {
  float r[4];
  f2_unpack(q[0], r[0], r[1]);
  f2_unpack(q[1], r[2], r[3]);
  // (xr_pos_trellis: columns c, c + 1 share a lane's 16 halfs, c + 2 and c + 3 sit 16 halfs on)
  __half2* p = row + (((c & ~31) * XR_TRELLIS_EXPAND + xr_pos_trellis(c & 31)) >> 1);
  const __half z = __float2half_rn(0.f);
  p[0] = __halves2half2(__float2half_rn(r[0]), z);
  p[2] = __halves2half2(__float2half_rn(r[1]), z);
  p[8] = __halves2half2(__float2half_rn(r[2]), z);
  p[10] = __halves2half2(__float2half_rn(r[3]), z);
}

// ---- 2: input transform per token (w13 side) -----------------------------------------------------------
constexpr int MOE_XF_THREADS = FHT_THREADS;
// One CTA takes `tt` consecutive tokens; store(t, c, logbs, n, v) gets a thread's finished groups of four: group k < n holds
// columns c + fht_col(k, 128, logbs) .. + 3 of token t + fht_row(k, 128, logbs).
template <class Store>
__device__ __forceinline__ void moe_rht_in_body(const MoeDev& M, int T, int tt, const uint8_t* __restrict__ x, float* fb, Store store) {
  const int t0 = blockIdx.x * tt, nt = min(tt, T - t0);
  const bool vec = act_rows_aligned4(x, 0, M.hidden, M.x_dtype);
  const int hidden = M.hidden;
  for (int b = 0; b < M.nb_n13; ++b) {
    const int logbs = M.log_n13[b], off = M.off_n13[b], mask = (1 << logbs) - 1;
    const float rs = rsqrtf((float)(1 << logbs));
    const f2 rs2 = f2_pack(rs, rs);
    const int step = min(nt, 8192 >> logbs);               // tokens per tile
    for (int r0 = 0; r0 < nt; r0 += step) {
      const int total = min(step, nt - r0) << logbs;
      auto load = [&](int e0, f2 (&v)[8][2]) {
        const int i0 = off + (e0 & mask);
        const long long o0 = (long long)(t0 + r0 + (e0 >> logbs)) * hidden + i0;
        const __half* sv = M.w13_sv + i0;
        with_dtype(M.x_dtype, [&](auto dt) {
#pragma unroll
          for (int k = 0; k < 8; ++k) {
            v[k][0] = v[k][1] = 0;
            if (e0 + (k << 10) < total) {
              const long long o = o0 + fht_row(k, 1024, logbs) * hidden + fht_col(k, 1024, logbs);
              float q[4];
              if (vec) load_act4(x, o, decltype(dt)::value, q);
              else {
#pragma unroll
                for (int j = 0; j < 4; ++j) q[j] = load_act(x, o + j, decltype(dt)::value);
              }
              f2 s[2];
              load_sign4(sv + fht_col(k, 1024, logbs), s);
              v[k][0] = f2_mul(f2_pack(q[0], q[1]), s[0]);
              v[k][1] = f2_mul(f2_pack(q[2], q[3]), s[1]);
            }
          }
        });
      };
      auto store_all = [&](int e1, const f2 (&v)[8][2]) {
        f2 r[8][2];
#pragma unroll
        for (int k = 0; k < 8; ++k) { r[k][0] = f2_mul(v[k][0], rs2); r[k][1] = f2_mul(v[k][1], rs2); }
        if (e1 < total) store(t0 + r0 + (e1 >> logbs), off + (e1 & mask), logbs, min(8, (total - e1 + 127) >> 7), r);
      };
      fht_block_all(fb, logbs, total, load, store_all);
      __syncthreads();
    }
  }
}

__global__ void __launch_bounds__(MOE_XF_THREADS, 3) moe_rht_in_kernel(const __grid_constant__ MoeDev M, int T, int tt,
                                                                       const uint8_t* __restrict__ x, uint8_t* __restrict__ ws) {
  extern __shared__ __align__(16) float fb[];
  const int hidden = M.hidden;
  pdl_trigger();
  __half2* xr = reinterpret_cast<__half2*>(ws + M.o_xr1);
  moe_rht_in_body(M, T, tt, x, fb, [&](int t, int c, int logbs, int n, const f2 (&v)[8][2]) {
#pragma unroll
    for (int k = 0; k < 8; ++k)
      if (k < n) moe_store_xr4(xr + (long long)(t + fht_row(k, 128, logbs)) * hidden, c + fht_col(k, 128, logbs), v[k]);
  });
}

__device__ __forceinline__ uint2 pack4_half(const f2 (&q)[2]) {
  float r[4];
  f2_unpack(q[0], r[0], r[1]);
  f2_unpack(q[1], r[2], r[3]);
  const __half2 a = __floats2half2_rn(r[0], r[1]), b = __floats2half2_rn(r[2], r[3]);
  return make_uint2(*reinterpret_cast<const uint32_t*>(&a), *reinterpret_cast<const uint32_t*>(&b));
}
// place of columns col .. col + 3 of the activation row `t` (moe_tile_place)
__device__ __forceinline__ uint8_t* moe_tile_at(uint8_t* base, int2 t, int kchunks, int col) {
  return base + ((size_t)t.x * kchunks + (size_t)(col >> 6) * (t.y >> 16)) * 128 + sw128_offset(t.y & 0xFFFF, col & 63);
}

// Input transform of one token, stored once per routing into the token tiles of the routed experts.
__global__ void __launch_bounds__(MOE_XF_THREADS, 3) moe_rht_in_gemm_kernel(const __grid_constant__ MoeDev M, int T, int tt,
                                                                            const uint8_t* __restrict__ x, uint8_t* __restrict__ ws) {
  extern __shared__ __align__(16) float fb[];
  pdl_trigger();
  pdl_wait();
  const int* slot_of = reinterpret_cast<const int*>(ws + M.o_slot_of);
  const int2* trow = reinterpret_cast<const int2*>(ws + M.o_trow);
  const int kchunks = M.hidden / GM_TILE_K;
  int2* rows = reinterpret_cast<int2*>(fb + fht_words(8192));        // activation row of every routing of the CTA's tokens
  const int t0 = blockIdx.x * tt, nr = min(tt, T - t0) * M.top_k;
  for (int i = threadIdx.x; i < nr; i += blockDim.x) {
    const int slot = slot_of[t0 * M.top_k + i];
    rows[i] = slot >= 0 ? trow[slot] : make_int2(-1, 0);
  }
  __syncthreads();
  const int top_k = M.top_k;
  uint8_t* xr = ws + M.o_xr1;
  moe_rht_in_body(M, T, tt, x, fb, [&](int t, int c, int logbs, int n, const f2 (&v)[8][2]) {
    uint2 h[8];
#pragma unroll
    for (int k = 0; k < 8; ++k) h[k] = pack4_half(v[k]);
    if (logbs >= 10) {               // a thread's groups are columns 128 apart of one token
      for (int j = 0; j < top_k; ++j) {
        const int2 r = rows[(t - t0) * top_k + j];
        if (r.x < 0) continue;
        const int step = (r.y >> 16) * 256;                          // two chunks
        uint8_t* p = moe_tile_at(xr, r, kchunks, c);
#pragma unroll
        for (int k = 0; k < 8; ++k)
          if (k < n) *reinterpret_cast<uint2*>(p + k * step) = h[k];
      }
    } else {
#pragma unroll
      for (int k = 0; k < 8; ++k)
        if (k < n)
          for (int j = 0; j < top_k; ++j) {
            const int2 r = rows[(t + fht_row(k, 128, logbs) - t0) * top_k + j];
            if (r.x >= 0) *reinterpret_cast<uint2*>(moe_tile_at(xr, r, kchunks, c + fht_col(k, 128, logbs))) = h[k];
          }
    }
  });
}

// ---- 3 / 5: grouped decode + mma ------------------------------------------------------------------------
struct MoeMvArgs {
  const uint8_t* codes[2];
  long long stride[2];
  const float* inv2;       // (E,) cumulative inverse residual scale of stage 2, or null
  const int* count;        // (E,)
  const int* base;         // (E,)
  const int* row_map;      // slot -> activation row, or null (identity)
  const __half* xr;        // activation rows, 2*n halfs each
  float* part;             // [kchunks][R][m]
  int* work;               // atomic unit counter
  int E, m, n, gps, strips, kchunks, gpc, R;
};

// One pass of a unit: the unit's groups are decoded once and multiplied with up to 8*NB routed tokens
// starting at t0.  Codes of MOE_PF groups are in flight per lane.
constexpr int MOE_PF = 4;

template <int K1, int K2, int NB>
__device__ __forceinline__ void moe_unit_pass(const MoeMvArgs& A, const uint8_t* p1, const uint8_t* p2, float s2, int ng,
                                              int c0, int strip, int kc, int base, int cnt, int t0, int lane) {
  const int gq = lane >> 2, tq = lane & 3;
  float acc[NB][2][4];
  float acc2[K2 ? NB : 1][2][4];
#pragma unroll
  for (int nb = 0; nb < NB; ++nb)
#pragma unroll
    for (int mi = 0; mi < 2; ++mi)
#pragma unroll
      for (int i = 0; i < 4; ++i) { acc[nb][mi][i] = 0.f; if constexpr (K2 > 0) acc2[nb][mi][i] = 0.f; }
  const uint4* xq[NB];
#pragma unroll
  for (int nb = 0; nb < NB; ++nb) {
    const int local = min(t0 + nb * 8 + gq, cnt - 1);     // columns past the count repeat the last token
    const int row = A.row_map ? A.row_map[base + local] : base + local;
    xq[nb] = reinterpret_cast<const uint4*>(A.xr + ((long long)row * A.n + c0 * 32) * XR_TRELLIS_EXPAND + tq * 16);
  }
  Words<K1> cur[MOE_PF];
  Words<(K2 > 0 ? K2 : 1)> cur2[MOE_PF];
#pragma unroll
  for (int i = 0; i < MOE_PF; ++i)
    if (i < ng) {
      cur[i] = load_words<K1>(p1 + i * (128 * K1));
      if constexpr (K2 > 0) cur2[i] = load_words<K2>(p2 + i * (128 * K2));
    }
  for (int c = 0; c < ng; c += MOE_PF) {
#pragma unroll
    for (int i = 0; i < MOE_PF; ++i) {
      if (c + i < ng) {
        const Words<K1> v = cur[i];
        Words<(K2 > 0 ? K2 : 1)> v2;
        if constexpr (K2 > 0) v2 = cur2[i];
        if (c + i + MOE_PF < ng) {
          cur[i] = load_words<K1>(p1 + (long long)(c + i + MOE_PF) * (128 * K1));
          if constexpr (K2 > 0) cur2[i] = load_words<K2>(p2 + (long long)(c + i + MOE_PF) * (128 * K2));
        }
        uint4 xb[NB][2];
#pragma unroll
        for (int nb = 0; nb < NB; ++nb) {
          xb[nb][0] = __ldg(xq[nb] + (c + i) * 8);
          xb[nb][1] = __ldg(xq[nb] + (c + i) * 8 + 1);
        }
        group_mma<K1, NB>(v, lane, xb, acc);
        if constexpr (K2 > 0) group_mma<K2, NB>(v2, lane, xb, acc2);
      }
    }
  }
  float* part = A.part + (long long)kc * A.R * A.m;
#pragma unroll
  for (int nb = 0; nb < NB; ++nb)
#pragma unroll
    for (int mi = 0; mi < 2; ++mi)
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int local = t0 + nb * 8 + tq * 2 + (i & 1);
        const int row = strip * 32 + mi * 16 + gq + ((i >> 1) ? 8 : 0);
        if (local < cnt) {
          float v = acc[nb][mi][i];
          if constexpr (K2 > 0) v = __fadd_rn(v, __fmul_rn(s2, acc2[nb][mi][i]));
          part[(long long)(base + local) * A.m + row] = v;
        }
      }
}

// NBMAX = largest number of token-column blocks per pass (4 = 32 tokens; 2 with a second stage).  Every unit
// picks the smallest block count that covers its expert's tokens, so lightly loaded experts do not pay
// for MMAs on empty columns and heavily loaded ones are decoded once per 8*NBMAX tokens.
template <int K1, int K2, int NBMAX>
__global__ void __launch_bounds__(MV_THREADS, 2) trellis_moe_mv_kernel(const __grid_constant__ MoeMvArgs A) {
  pdl_trigger();
  pdl_wait();
  const int lane = threadIdx.x & 31;
  const int units_per_expert = A.strips * A.kchunks;
  const int total_units = A.E * units_per_expert;
  // Every warp draws one unit at a time from an atomic counter (units of experts without tokens are
  // skipped at once, so skewed routing does not idle warps).
  for (;;) {
    int u = 0;
    if (lane == 0) u = atomicAdd(A.work, 1);
    u = __shfl_sync(0xffffffffu, u, 0);
    if (u >= total_units) break;
    const int e = u / units_per_expert;
    const int cnt = A.count[e];
    if (cnt == 0) continue;
    const int rem = u - e * units_per_expert;
    const int kc = rem / A.strips, strip = rem - kc * A.strips;
    const int c0 = kc * A.gpc, c1 = min(A.gps, c0 + A.gpc);
    const int base = A.base[e];
    const uint8_t* p1 = A.codes[0] + (long long)e * A.stride[0] + ((long long)strip * A.gps + c0) * (128 * K1) + lane * (4 * K1);
    const uint8_t* p2 = nullptr;
    float s2 = 0.f;
    if constexpr (K2 > 0) {
      p2 = A.codes[1] + (long long)e * A.stride[1] + ((long long)strip * A.gps + c0) * (128 * K2) + lane * (4 * K2);
      s2 = A.inv2[e];
    }
    const int ng = c1 - c0;
    int t0 = 0;
    for (; cnt - t0 > 8 * (NBMAX / 2); t0 += 8 * NBMAX)
      moe_unit_pass<K1, K2, NBMAX>(A, p1, p2, s2, ng, c0, strip, kc, base, cnt, t0, lane);
    if (cnt - t0 > 0) {
      if (NBMAX >= 4 && cnt - t0 > 8) moe_unit_pass<K1, K2, (NBMAX >= 4 ? 2 : 1)>(A, p1, p2, s2, ng, c0, strip, kc, base, cnt, t0, lane);
      else moe_unit_pass<K1, K2, 1>(A, p1, p2, s2, ng, c0, strip, kc, base, cnt, t0, lane);
    }
  }
}

// The transforms of the mid and combine kernels work on 1024-value chunks, one warp each (fht_warp).  `rows` arrays of a
// block of 2^log values take moe_chunks(rows, log) chunks: value i of row r is value (r << log | i) & 1023 of chunk
// (r << log | i) >> 10.  Blocks of more than 1024 values span chunks; what reads their results does the last stages.
__host__ __device__ __forceinline__ int moe_chunks(int rows, int lg) { return ((rows << lg) + 1023) >> 10; }
__host__ __device__ __forceinline__ int moe_chunks_all(int rows, int nb, const int* lg) {
  int c = 0;
  for (int b = 0; b < nb; ++b) c += moe_chunks(rows, lg[b]);
  return c;
}
// block of chunk `ch`; `base` receives the block's first chunk
__device__ __forceinline__ int moe_chunk_block(int ch, int rows, int nb, const int* lg, int& base) {
  int b = 0;
  base = 0;
  for (; b + 1 < nb; ++b) {
    const int n = moe_chunks(rows, lg[b]);
    if (ch < base + n) break;
    base += n;
  }
  return b;
}
// 16 bytes from global to shared memory, past the registers (complete after cp.async.wait_group, for the issuing thread)
__device__ __forceinline__ void cp_async16(float* dst, const float* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_u32(dst)), "l"(src) : "memory");
}
// A chunk's values: sums of `cnt` partial sums `kstride` floats apart.  row_off(r): first value of row r (floats from
// `src`, which points at the block's first column), negative for a row of zeros; rows from `nrow` on are zero.
template <class RowOff>
__device__ __forceinline__ void moe_load_chunk(f2 (&v)[8][2], int c, int logbs, int nrow, const float* __restrict__ src, int cnt,
                                               long long kstride, RowOff row_off) {
  const int e = (c << 10) | ((threadIdx.x & 31) << 2), i0 = e & ((1 << logbs) - 1);
  const float* p[8];
#pragma unroll
  for (int k = 0; k < 8; ++k) {
    const int r = (e >> logbs) + fht_row(k, 128, logbs);
    const long long o = r < nrow ? row_off(r) : -1;
    p[k] = o >= 0 ? src + o + i0 + fht_col(k, 128, logbs) : nullptr;
    v[k][0] = v[k][1] = 0;
    if (p[k]) {
      const ulonglong2 t = __ldcg(reinterpret_cast<const ulonglong2*>(p[k]));
      v[k][0] = t.x; v[k][1] = t.y;
    }
  }
  for (int s = 1; s < cnt; ++s) {
#pragma unroll
    for (int k = 0; k < 8; ++k)
      if (p[k]) {
        const ulonglong2 t = __ldcg(reinterpret_cast<const ulonglong2*>(p[k] + s * kstride));
        v[k][0] = f2_add(v[k][0], t.x);
        v[k][1] = f2_add(v[k][1], t.y);
      }
  }
}
// The stages beyond the chunks of a block of 2^logbs values, 2^TOP chunks a row, for the first `nrow` rows from `area` on:
// put(row, i, v) takes values i .. i + 3 of a row.  Every value is read once, by all threads of the CTA (leaving
// the stages to the mid kernel's loads, 2^TOP reads per value in the few warps that have a chunk, made a step of two
// tokens, top 2, hidden 4096, inter 2048 take 92 us instead of 84).
template <int TOP, class Put>
__device__ __forceinline__ void moe_finish_top(const float* area, int logbs, int nrow, Put put) {
  constexpr int N = 1 << TOP;
  for (int o = threadIdx.x * 4; o < nrow << 10; o += MOE_XF_THREADS * 4) {
    const int row = o >> 10, i = o & 1023;
    f2 v[N][2];
#pragma unroll
    for (int t = 0; t < N; ++t) fht_ld4(area + fht_pos((row << logbs) | (t << 10) | i), v[t]);
#pragma unroll
    for (int s = 0; s < TOP; ++s)
#pragma unroll
      for (int t = 0; t < N; ++t)
        if (!(t & (1 << s))) { f2_butterfly(v[t][0], v[t | (1 << s)][0]); f2_butterfly(v[t][1], v[t | (1 << s)][1]); }
#pragma unroll
    for (int t = 0; t < N; ++t) put(row, (t << 10) | i, v[t]);
  }
}
template <class Put>
__device__ __forceinline__ void moe_finish(const float* area, int logbs, int nrow, Put put) {
  if (logbs == 11) moe_finish_top<1>(area, logbs, nrow, put);
  else if (logbs == 12) moe_finish_top<2>(area, logbs, nrow, put);
  else if (logbs == 13) moe_finish_top<3>(area, logbs, nrow, put);
}

__device__ __forceinline__ float round_half(float v) { return __half2float(__float2half_rn(v)); }

// ---- 4: per slot  h = act(gate) * up  from w13 partials, then the w2 input transform ---------------------
// One CTA handles `sg` consecutive slots.  Bound by memory (it reads a slot's w13 outputs as fp32 and writes its w2
// inputs as fp16); chunk by chunk in one warp each, the gated activation is evaluated where the second transform
// loads its values, so nothing but the two transforms' chunks passes through shared memory.  4096 tokens, top 8, 1536
// and 768 columns: 243 -> 219 us (slots per CTA from 5 to 7 make no difference: latency and the one barrier are the
// rest); the combine below 212 -> 116 us, the input transform 60 -> 45 us.
__global__ void __launch_bounds__(MOE_XF_THREADS, 3) moe_mid_kernel(const __grid_constant__ MoeDev M, int T, int sg,
                                                                    uint8_t* __restrict__ ws) {
  extern __shared__ __align__(16) float fb[];   // chunks of sg w13 rows, then of sg w2 rows
  pdl_trigger();
  pdl_wait();
  const int R = T * M.top_k;
  const int* g_count = reinterpret_cast<const int*>(ws + M.o_count);
  const int* g_base = reinterpret_cast<const int*>(ws + M.o_base);
  const int used = g_base[M.E - 1] + g_count[M.E - 1];
  const int slot0 = blockIdx.x * sg;
  if (slot0 >= used) return;
  const int nrow = min(sg, used - slot0);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  __shared__ int row_e[8];                   // expert of each row (sg <= 8)
  __shared__ float row_wsc[8];
  __shared__ int2 row_t[8];
  if (threadIdx.x < nrow) {
    const int e = reinterpret_cast<const int*>(ws + M.o_route_exp)[slot0 + threadIdx.x];
    row_e[threadIdx.x] = e;
    row_wsc[threadIdx.x] = M.w13_wscale[e];
    row_t[threadIdx.x] = M.gemm ? reinterpret_cast<const int2*>(ws + M.o_trow)[slot0 + threadIdx.x] : make_int2(0, 0);
  }
  const int inter = M.inter, w13_out = M.w13_out, kch = M.kch13;
  const int n13 = moe_chunks_all(sg, M.nb_m13, M.log_m13), n2 = moe_chunks_all(sg, M.nb_n2, M.log_n2);
  const long long kstride = (long long)R * w13_out;
  const float* part1 = reinterpret_cast<const float*>(ws + M.o_part1) + (long long)slot0 * w13_out;

  // -- output transform of w13; results stay in shared memory
  for (int ch = warp; ch < n13; ch += MOE_XF_THREADS / 32) {
    int base;
    const int b = moe_chunk_block(ch, sg, M.nb_m13, M.log_m13, base);
    f2 v[8][2];
    moe_load_chunk(v, ch - base, M.log_m13[b], nrow, part1 + M.off_m13[b], kch, kstride,
                   [&](int r) -> long long { return r * w13_out; });
    fht_warp(fb + ch * FHT_CHUNK_WORDS, v, M.log_m13[b]);
  }
  __syncthreads();
  if (M.wide_m13) {                          // blocks of more than one chunk, in place
    int base = 0;
    for (int b = 0; b < M.nb_m13; ++b) {
      float* area = fb + base * FHT_CHUNK_WORDS;
      const int logbs = M.log_m13[b];
      moe_finish(area, logbs, nrow, [&](int row, int i, const f2 (&v)[2]) { fht_st4(area + fht_pos((row << logbs) | i), v); });
      base += moe_chunks(sg, logbs);
    }
    __syncthreads();
  }
  // -- columns c .. c + 3 of the w13 output: Wscale, 1/sqrt(bs) and SU, fp16 rounding (the reference's w13 op returns
  //    fp16: glq_vllm/fused_moe_method.py:412-421)
  auto y13_4 = [&](int row, int c, float (&f)[4]) {
    int base = 0, b = 0;
    while (b + 1 < M.nb_m13 && c >= M.off_m13[b + 1]) { base += moe_chunks(sg, M.log_m13[b]); ++b; }
    const float sc = rsqrtf((float)(1 << M.log_m13[b])) * row_wsc[row];
    f2 p[2], s[2];
    fht_ld4(fb + base * FHT_CHUNK_WORDS + fht_pos((row << M.log_m13[b]) | (c - M.off_m13[b])), p);
    load_sign4(M.w13_su + (long long)row_e[row] * w13_out + c, s);
    const f2 sc2 = f2_pack(sc, sc);
    f2_unpack(f2_mul(f2_mul(p[0], sc2), s[0]), f[0], f[1]);
    f2_unpack(f2_mul(f2_mul(p[1], sc2), s[1]), f[2], f[3]);
#pragma unroll
    for (int k = 0; k < 4; ++k) f[k] = round_half(f[k]);
  };
  // -- input transform of w2 on act(gate) * up (fp16) times SV, stored from its chunks
  float* area2 = fb + n13 * FHT_CHUNK_WORDS;
  const int kchunks = inter / GM_TILE_K;
  uint8_t* xr2 = ws + M.o_xr2;
  __half2* xs2 = reinterpret_cast<__half2*>(xr2) + (long long)slot0 * inter;
  const bool gemm = M.gemm != 0;
  auto put = [&](int row, int c, const f2 (&v)[2], f2 rs2) {
    const f2 r[2] = {f2_mul(v[0], rs2), f2_mul(v[1], rs2)};
    if (gemm) *reinterpret_cast<uint2*>(moe_tile_at(xr2, row_t[row], kchunks, c)) = pack4_half(r);
    else moe_store_xr4(xs2 + row * inter, c, r);
  };
  bool spans = false;                        // blocks of more than one chunk are finished when all chunks are done
  for (int ch = warp; ch < n2; ch += MOE_XF_THREADS / 32) {
    int base;
    const int b = moe_chunk_block(ch, sg, M.nb_n2, M.log_n2, base);
    const int logbs = M.log_n2[b], off = M.off_n2[b];
    const int e = ((ch - base) << 10) | (lane << 2), row0 = e >> logbs, c0 = off + (e & ((1 << logbs) - 1));
    f2 v[8][2];
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      const int row = row0 + fht_row(k, 128, logbs), c = c0 + fht_col(k, 128, logbs);
      v[k][0] = v[k][1] = 0;
      if (row < nrow) {
        float g[4], u[4];
        f2 sv[2];
        y13_4(row, c, g);
        load_sign4(M.w2_sv + c, sv);
        if (M.gated) y13_4(row, inter + c, u);
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const float a = moe_act(g[j], M.act);
          g[j] = round_half(M.gated ? a * u[j] : a);
        }
        v[k][0] = f2_mul(f2_pack(g[0], g[1]), sv[0]);
        v[k][1] = f2_mul(f2_pack(g[2], g[3]), sv[1]);
      }
    }
    float* sm = area2 + ch * FHT_CHUNK_WORDS;
    fht_warp(sm, v, logbs);
    if (logbs > 10) { spans = true; continue; }
    const float rs = rsqrtf((float)(1 << logbs));
    const f2 rs2 = f2_pack(rs, rs);
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      const int row = row0 + fht_row(k, 128, logbs);
      if (row < nrow) {
        fht_ld4(sm + (lane << 2) + k * 132, v[k]);
        put(row, c0 + fht_col(k, 128, logbs), v[k], rs2);
      }
    }
  }
  if (!__syncthreads_or(spans)) return;
  int base = 0;
  for (int b = 0; b < M.nb_n2; ++b) {
    const int logbs = M.log_n2[b];
    const float rs = rsqrtf((float)(1 << logbs));
    const f2 rs2 = f2_pack(rs, rs);
    moe_finish(area2 + base * FHT_CHUNK_WORDS, logbs, nrow,
               [&](int row, int i, const f2 (&v)[2]) { put(row, M.off_n2[b] + i, v, rs2); });
    base += moe_chunks(sg, logbs);
  }
}

// The same for blocks of up to 1024 values on both sides: a warp takes two consecutive slots by itself, no block barrier.
// The w13 outputs of its slots pass through shared memory as the fp16 values they are rounded to, in column order, so
// Wscale, SU and the rounding are done once per value and gate and up are one 8-byte load each; the partial sums of the
// next chunk are in flight while one is transformed.  4096 tokens, top 8, 1536 and 768 columns: 190 us by
// the kernel above, 175 us by this (104 and 91 M warp instructions; tanhf and the roundings are a third of them).
constexpr int MIDW_ROWS = 2, MIDW_WARPS = 4;
__host__ __device__ __forceinline__ size_t moe_midw_warp_bytes(int w13_out) { return FHT_CHUNK_WORDS * 4 + (size_t)MIDW_ROWS * w13_out * 2; }
template <class F>
__device__ __forceinline__ void with_act(int act, F f) {
  switch (act) {
    case 0: f(IntC<0>()); break;
    case 1: f(IntC<1>()); break;
    case 2: f(IntC<2>()); break;
    case 3: f(IntC<3>()); break;
    case 4: f(IntC<4>()); break;
    default: f(IntC<5>()); break;
  }
}
__global__ void __launch_bounds__(MIDW_WARPS * 32, 4) moe_mid_warp_kernel(const __grid_constant__ MoeDev M, int T,
                                                                          uint8_t* __restrict__ ws) {
  extern __shared__ __align__(16) uint8_t fb8[];
  pdl_trigger();
  pdl_wait();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int R = T * M.top_k;
  const int used = reinterpret_cast<const int*>(ws + M.o_base)[M.E - 1] + reinterpret_cast<const int*>(ws + M.o_count)[M.E - 1];
  const int slot0 = (blockIdx.x * MIDW_WARPS + warp) * MIDW_ROWS;
  if (slot0 >= used) return;
  const int nrow = min(MIDW_ROWS, used - slot0);
  const int inter = M.inter, w13_out = M.w13_out, kch = M.kch13;
  float* sm = reinterpret_cast<float*>(fb8 + warp * moe_midw_warp_bytes(w13_out));
  __half* h13 = reinterpret_cast<__half*>(sm + FHT_CHUNK_WORDS);          // [row][w13_out]
  int ex[MIDW_ROWS];
  float wsc[MIDW_ROWS];
  int2 tr[MIDW_ROWS];
#pragma unroll
  for (int r = 0; r < MIDW_ROWS; ++r) {
    const int slot = slot0 + min(r, nrow - 1);
    ex[r] = reinterpret_cast<const int*>(ws + M.o_route_exp)[slot];
    wsc[r] = M.w13_wscale[ex[r]];
    tr[r] = M.gemm ? reinterpret_cast<const int2*>(ws + M.o_trow)[slot] : make_int2(0, 0);
  }
  const long long kstride = (long long)R * w13_out;
  const float* part1 = reinterpret_cast<const float*>(ws + M.o_part1) + (long long)slot0 * w13_out + (lane << 2);
  // -- output transform of w13, chunk by chunk (chunk c of block b holds values c << 10 .. of the block's rows)
  auto load = [&](int b, int c, f2 (&v)[8][2]) {
    const int logbs = M.log_m13[b], mask = (1 << logbs) - 1;
    const float* src = part1 + M.off_m13[b];
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      const int e = (c << 10) | (k << 7), r = (e | (lane << 2)) >> logbs;
      v[k][0] = v[k][1] = 0;
      if (r < nrow) {
        // (a block of less than 128 values: the row changes within the warp's 128 values)
        const float* p = src + (logbs >= 7 ? r * w13_out + (e & mask) : r * w13_out + ((e | (lane << 2)) & mask) - (lane << 2));
        ulonglong2 t = __ldcg(reinterpret_cast<const ulonglong2*>(p));
        v[k][0] = t.x; v[k][1] = t.y;
        for (int s = 1; s < kch; ++s) {
          t = __ldcg(reinterpret_cast<const ulonglong2*>(p + s * kstride));
          v[k][0] = f2_add(v[k][0], t.x);
          v[k][1] = f2_add(v[k][1], t.y);
        }
      }
    }
  };
  int b = 0, c = 0;
  f2 nxt[8][2];
  load(0, 0, nxt);
  while (b < M.nb_m13) {
    const int logbs = M.log_m13[b], off = M.off_m13[b], mask = (1 << logbs) - 1, base = c << 10;
    f2 v[8][2];
#pragma unroll
    for (int k = 0; k < 8; ++k) { v[k][0] = nxt[k][0]; v[k][1] = nxt[k][1]; }
    if (++c >= moe_chunks(MIDW_ROWS, logbs)) { c = 0; ++b; }
    if (b < M.nb_m13) load(b, c, nxt);
    fht_warp(sm, v, logbs);
    const float rs = rsqrtf((float)(1 << logbs));
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      const int e = base | (k << 7) | (lane << 2), r = e >> logbs, col = off + (e & mask);
      if (r < nrow) {
        f2 p[2], sg[2];
        float f[4];
        fht_ld4(sm + (lane << 2) + k * 132, p);
        load_sign4(M.w13_su + (long long)(r ? ex[1] : ex[0]) * w13_out + col, sg);
        const float sc = rs * (r ? wsc[1] : wsc[0]);
        const f2 sc2 = f2_pack(sc, sc);
        f2_unpack(f2_mul(f2_mul(p[0], sc2), sg[0]), f[0], f[1]);
        f2_unpack(f2_mul(f2_mul(p[1], sc2), sg[1]), f[2], f[3]);
        const __half2 lo = __floats2half2_rn(f[0], f[1]), hi = __floats2half2_rn(f[2], f[3]);
        *reinterpret_cast<uint2*>(h13 + r * w13_out + col) =
            make_uint2(*reinterpret_cast<const uint32_t*>(&lo), *reinterpret_cast<const uint32_t*>(&hi));
      }
    }
    __syncwarp();
  }
  // -- gated activation (fp16), SV and the input transform of w2
  const int kchunks = inter / GM_TILE_K;
  uint8_t* xr2 = ws + M.o_xr2;
  __half2* xs2 = reinterpret_cast<__half2*>(xr2) + (long long)slot0 * inter;
  const bool gated = M.gated != 0, gemm = M.gemm != 0;
  auto unpack4 = [](const __half* p, float (&f)[4]) {
    const uint2 t = *reinterpret_cast<const uint2*>(p);
    const float2 a = __half22float2(*reinterpret_cast<const __half2*>(&t.x)), d = __half22float2(*reinterpret_cast<const __half2*>(&t.y));
    f[0] = a.x; f[1] = a.y; f[2] = d.x; f[3] = d.y;
  };
  for (int b2 = 0; b2 < M.nb_n2; ++b2) {
    const int logbs = M.log_n2[b2], off = M.off_n2[b2], mask = (1 << logbs) - 1;
    const float rs = rsqrtf((float)(1 << logbs));
    const f2 rs2 = f2_pack(rs, rs);
    for (int c2 = 0; c2 < moe_chunks(MIDW_ROWS, logbs); ++c2) {
      f2 v[8][2];
      with_act(M.act, [&](auto act) {
#pragma unroll
        for (int k = 0; k < 8; ++k) {
          const int e = (c2 << 10) | (k << 7) | (lane << 2), r = e >> logbs, col = off + (e & mask);
          v[k][0] = v[k][1] = 0;
          if (r < nrow) {
            float g[4], u[4] = {1.f, 1.f, 1.f, 1.f};
            f2 sv[2];
            unpack4(h13 + r * w13_out + col, g);
            if (gated) unpack4(h13 + r * w13_out + inter + col, u);
            load_sign4(M.w2_sv + col, sv);
#pragma unroll
            for (int j = 0; j < 4; ++j) g[j] = round_half(moe_act(g[j], decltype(act)::value) * u[j]);
            v[k][0] = f2_mul(f2_pack(g[0], g[1]), sv[0]);
            v[k][1] = f2_mul(f2_pack(g[2], g[3]), sv[1]);
          }
        }
      });
      fht_warp(sm, v, logbs);
#pragma unroll
      for (int k = 0; k < 8; ++k) {
        const int e = (c2 << 10) | (k << 7) | (lane << 2), r = e >> logbs, col = off + (e & mask);
        if (r < nrow) {
          f2 q[2];
          fht_ld4(sm + (lane << 2) + k * 132, q);
          const f2 o[2] = {f2_mul(q[0], rs2), f2_mul(q[1], rs2)};
          if (gemm) *reinterpret_cast<uint2*>(moe_tile_at(xr2, r ? tr[1] : tr[0], kchunks, col)) = pack4_half(o);
          else moe_store_xr4(xs2 + r * inter, col, o);
        }
      }
      __syncwarp();
    }
  }
}

// ---- 6: per token weighted combine ------------------------------------------------------------------------
// The routings of a token are the rows of the transform (`rg` at a time), 1024 values per warp; a thread then owns groups
// of four output columns, 1024 apart within a block, does the stages beyond the chunks and adds the routings' results
// in fixed j order.
template <int TOP>
__device__ __forceinline__ void moe_combine_block(const MoeDev& M, const float* area, int logbs, int off, int nrow, bool first, bool last,
                                                  const long long* row_off, const int* row_e, const float* row_wsc, const float* row_w,
                                                  float* accs, uint8_t* y, long long y_row, bool y_vec) {
  constexpr int N = 1 << TOP;
  const float rs = rsqrtf((float)(1 << logbs));
  const int span = 1 << (logbs - TOP);
  for (int i = threadIdx.x * 4; i < span; i += MOE_XF_THREADS * 4) {
    float a[N][4];
#pragma unroll
    for (int t = 0; t < N; ++t)
#pragma unroll
      for (int j = 0; j < 4; ++j) a[t][j] = first ? 0.f : accs[off + (t << 10) + i + j];
    for (int row = 0; row < nrow; ++row) {
      if (row_off[row] < 0) continue;
      const float w = row_w[row], sc = rs * row_wsc[row];
      const f2 sc2 = f2_pack(sc, sc);
      f2 v[N][2];
#pragma unroll
      for (int t = 0; t < N; ++t) fht_ld4(area + fht_pos((row << logbs) | (t << 10) | i), v[t]);
#pragma unroll
      for (int s = 0; s < TOP; ++s)
#pragma unroll
        for (int t = 0; t < N; ++t)
          if (!(t & (1 << s))) { f2_butterfly(v[t][0], v[t | (1 << s)][0]); f2_butterfly(v[t][1], v[t | (1 << s)][1]); }
      const __half* su = M.w2_su + (long long)row_e[row] * M.hidden + off + i;
#pragma unroll
      for (int t = 0; t < N; ++t) {
        f2 s[2];
        float r[4];
        load_sign4(su + (t << 10), s);
        f2_unpack(f2_mul(f2_mul(v[t][0], sc2), s[0]), r[0], r[1]);
        f2_unpack(f2_mul(f2_mul(v[t][1], sc2), s[1]), r[2], r[3]);
        // the reference's w2 op returns fp16 before the weighted sum
#pragma unroll
        for (int j = 0; j < 4; ++j) a[t][j] += w * round_half(r[j]);
      }
    }
#pragma unroll
    for (int t = 0; t < N; ++t) {
      const int c = off + (t << 10) + i;
      if (!last) {
#pragma unroll
        for (int j = 0; j < 4; ++j) accs[c + j] = a[t][j];
      } else if (y_vec) {
        store_act4(y, y_row + c, M.y_dtype, a[t]);
      } else {
#pragma unroll
        for (int j = 0; j < 4; ++j) store_act(y, y_row + c + j, M.y_dtype, a[t][j]);
      }
    }
  }
}

__global__ void __launch_bounds__(MOE_XF_THREADS, 3) moe_out_kernel(const __grid_constant__ MoeDev M, int T, int rg,
                                                                    const float* __restrict__ topk_w,
                                                                    const uint8_t* __restrict__ ws, uint8_t* __restrict__ y) {
  extern __shared__ __align__(16) float fb[];   // chunks of rg rows of hidden (+ hidden floats when several passes are needed)
  pdl_wait();
  const int t = blockIdx.x, lane = threadIdx.x & 31;
  const int R = T * M.top_k;
  const int* slot_of = reinterpret_cast<const int*>(ws + M.o_slot_of);
  const int* route_exp = reinterpret_cast<const int*>(ws + M.o_route_exp);
  const float* part2 = reinterpret_cast<const float*>(ws + M.o_part2);
  __shared__ long long row_off[64];          // per routing j of this token (top_k <= 64): its partial sums, or -1
  __shared__ int row_e[64];
  __shared__ float row_wsc[64], row_w[64];
  if (threadIdx.x < M.top_k) {
    const int slot = slot_of[t * M.top_k + threadIdx.x];
    const int e = slot >= 0 ? route_exp[slot] : 0;
    row_off[threadIdx.x] = slot >= 0 ? (long long)slot * M.hidden : -1;
    row_e[threadIdx.x] = e;
    row_wsc[threadIdx.x] = M.w2_wscale[e];
    row_w[threadIdx.x] = topk_w[t * M.top_k + threadIdx.x];
  }
  __syncthreads();
  const int hidden = M.hidden, kch = M.kch2, n2 = moe_chunks_all(rg, M.nb_m2, M.log_m2);
  float* accs = fb + n2 * FHT_CHUNK_WORDS;   // running sums over the passes, hidden floats
  const long long kstride = (long long)R * hidden;
  const bool y_vec = act_rows_aligned4(y, 0, hidden, M.y_dtype);
  for (int j0 = 0; j0 < M.top_k; j0 += rg) {
    const int nrow = min(rg, M.top_k - j0);
    if (kch == 1) {
      // one partial sum per value: all chunks of a warp travel at once, each lane to where it will read them
      for (int ch = threadIdx.x >> 5; ch < n2; ch += MOE_XF_THREADS / 32) {
        int base;
        const int b = moe_chunk_block(ch, rg, M.nb_m2, M.log_m2, base), logbs = M.log_m2[b];
        const int e = ((ch - base) << 10) | (lane << 2), i0 = M.off_m2[b] + (e & ((1 << logbs) - 1));
        float* dst = fb + ch * FHT_CHUNK_WORDS + (lane << 2);
#pragma unroll
        for (int k = 0; k < 8; ++k) {
          const int r = (e >> logbs) + fht_row(k, 128, logbs);
          const long long o = r < nrow ? row_off[j0 + r] : -1;
          if (o >= 0) cp_async16(dst + k * 132, part2 + o + i0 + fht_col(k, 128, logbs));
          else *reinterpret_cast<float4*>(dst + k * 132) = make_float4(0.f, 0.f, 0.f, 0.f);
        }
      }
      asm volatile("cp.async.commit_group;\n\tcp.async.wait_group 0;" ::: "memory");
    }
    for (int ch = threadIdx.x >> 5; ch < n2; ch += MOE_XF_THREADS / 32) {
      int base;
      const int b = moe_chunk_block(ch, rg, M.nb_m2, M.log_m2, base);
      f2 v[8][2];
      if (kch == 1) {
#pragma unroll
        for (int k = 0; k < 8; ++k) fht_ld4(fb + ch * FHT_CHUNK_WORDS + (lane << 2) + k * 132, v[k]);
      } else moe_load_chunk(v, ch - base, M.log_m2[b], nrow, part2 + M.off_m2[b], kch, kstride,
                     [&](int r) -> long long { return row_off[j0 + r]; });
      fht_warp(fb + ch * FHT_CHUNK_WORDS, v, M.log_m2[b]);
    }
    __syncthreads();
    const bool first = j0 == 0, last = j0 + rg >= M.top_k;
    int base = 0;
    for (int b = 0; b < M.nb_m2; ++b) {
      const int logbs = M.log_m2[b], off = M.off_m2[b];
      const float* area = fb + base * FHT_CHUNK_WORDS;
      auto go = [&](auto top) {
        moe_combine_block<decltype(top)::value>(M, area, logbs, off, nrow, first, last, row_off + j0, row_e + j0, row_wsc + j0,
                                                row_w + j0, accs, y, (long long)t * hidden, y_vec);
      };
      if (logbs <= 10) go(IntC<0>());
      else if (logbs == 11) go(IntC<1>());
      else if (logbs == 12) go(IntC<2>());
      else go(IntC<3>());
      base += moe_chunks(rg, logbs);
    }
    __syncthreads();
  }
}

typedef void (*MoeMvKernel)(const MoeMvArgs);

template <int NB>
static MoeMvKernel moe_mv_pick(int k1, int k2) {
#define M_CASE(A, B) if (k1 == A && k2 == B) return trellis_moe_mv_kernel<A, B, NB>;
  M_CASE(2, 0) M_CASE(3, 0) M_CASE(4, 0) M_CASE(4, 1) M_CASE(4, 2) M_CASE(4, 3) M_CASE(4, 4)
#undef M_CASE
  return nullptr;
}

typedef void (*MoeGemmKernel)(const DevLinear*, const GemmItem*, int, uint8_t*, int*, const int*, int);
// E8 experts: three stages of 40 KiB leave the codebook gathers of the producers as much L1 as 128-token tiles with four
// did.  8 experts, top 2, 4096 x 2048, two stages, four / three: 8 tokens 318 / 281 us, 1024 tokens 672 / 618.
constexpr int MOE_GEMM_STAGES = 3;
static MoeGemmKernel moe_gemm_pick(int k1, int k2) {
#define M_CASE(A, B) if (k1 == A && k2 == B) return trellis_gemm_kernel<A, B, MOE_TN>;
  M_CASE(2, 0) M_CASE(3, 0) M_CASE(4, 0) M_CASE(4, 1) M_CASE(4, 2) M_CASE(4, 3) M_CASE(4, 4)
#undef M_CASE
  return nullptr;
}
static MoeGemmKernel moe_gemm_pick_e8(int ns) {
  switch (ns) {
    case 1: return glq_gemm_kernel<1, 1, 0, MOE_TN_E8, MOE_GEMM_STAGES>;
    case 2: return glq_gemm_kernel<1, 2, 0, MOE_TN_E8, MOE_GEMM_STAGES>;
    case 3: return glq_gemm_kernel<1, 3, 0, MOE_TN_E8, MOE_GEMM_STAGES>;
  }
  return nullptr;
}
static size_t moe_gemm_smem_bytes(bool e8) {
  if (!e8) return TgShape<MOE_TN>::SMEM_BYTES;
  return (size_t)MOE_GEMM_STAGES * (GM_A_BYTES + (size_t)MOE_TN_E8 * 128) + (3 * MOE_GEMM_STAGES + 5) * 8 + 16 + 1024;
}
// routed tokens per expert (average) from which the tensor-core form is used (measured, 128 experts, top 8, streaming /
// tensor-core: 64 tokens 260 / 263 us, 128 tokens 283 / 264, 256 tokens 333 / 271, 512 tokens 518 / 325; at an average of 8:
// 64 experts, 1024 x 512, 3 bits 84 / 85; 32 experts, 2048 x 768, 2 bits 113 / 98, 2048 x 1536, 4 bits 167 / 150; 8 experts,
// 4096 x 2048 120 / 115).  With two stages the GEMM multiplies fp16(w1 + s * w2), where the streaming kernel keeps exact weights and an fp32 sum per stage:
// steps below 64 routed tokens per expert keep that precision.
static int moe_gemm_min_avg(bool two_stages) {
  const char* e = getenv("GLQB_MOE_GEMM_MIN_AVG");
  return e ? atoi(e) : (two_stages ? 64 : 6);
}

}  // namespace glqb

using namespace glqb;

struct GlqbMoePlan {
  GlqbMoeDesc desc;
  MoeDev dev;
  size_t ws_bytes = 0;
  int sm_count = 0;
  int nb = 2;              // token-column blocks per pass (8*nb routed tokens share one decode)
  MoeMvKernel k13 = nullptr, k2 = nullptr;
  int grid13 = 0, grid2 = 0;
  int mid_sg = 1, out_rg = 1;          // slots per CTA of the mid kernel, routings per pass of the combine
  // routings from which moe_mid_warp_kernel is used, streaming and tensor-core form (moe_mid_warp_min; INT_MAX: not for these blocks)
  int mid_warp_min = INT_MAX, mid_warp_min_gemm = INT_MAX;
  size_t mid_smem = 0, out_smem = 0;
  // tensor-core form
  bool gemm_ok = false, two_stages = false;
  MoeDev devg;             // same weights, workspace laid out for the GEMM kernels
  MoeGemmKernel g13 = nullptr, g2 = nullptr;
  // optional timing of the two expert matmuls (event pairs around each, on the launching stream)
  bool timing = false;
  std::vector<cudaEvent_t> ev;
  size_t ev_used = 0;
};

// brackets one matmul launch with an event pair when timing is on
struct MoeTimer {
  GlqbMoePlan* P;
  cudaStream_t st;
  bool on;
  MoeTimer(GlqbMoePlan* p, cudaStream_t s) : P(p), st(s), on(p->timing) {
    if (!on) return;
    while (P->ev.size() < P->ev_used + 2) {
      cudaEvent_t e;
      if (cudaEventCreate(&e) != cudaSuccess) { on = false; return; }
      P->ev.push_back(e);
    }
    cudaEventRecord(P->ev[P->ev_used], st);
  }
  ~MoeTimer() {
    if (!on) return;
    cudaEventRecord(P->ev[P->ev_used + 1], st);
    P->ev_used += 2;
  }
};

static int moe_fail(int code, const char* fmt, ...) {
  char buf[512];
  va_list ap;
  va_start(ap, fmt);
  vsnprintf(buf, sizeof buf, fmt, ap);
  va_end(ap);
  set_error_message(buf);
  return code;
}

static size_t al(size_t v) { return (v + 255) / 256 * 256; }

static int fill_blocks(const int32_t* blocks, int nb, int total, int* off, int* lg, const char* what) {
  if (nb < 1 || nb > GLQB_MAX_BLOCKS) return moe_fail(GLQB_E_INVALID, "moe: %s block count %d", what, nb);
  int o = 0;
  for (int i = 0; i < nb; ++i) {
    const int b = blocks[i];
    if (b < 32 || (b & (b - 1))) return moe_fail(GLQB_E_INVALID, "moe: %s block %d", what, b);
    off[i] = o;
    lg[i] = 31 - __builtin_clz((unsigned)b);
    o += b;
  }
  if (o != total) return moe_fail(GLQB_E_INVALID, "moe: %s blocks sum to %d, expected %d", what, o, total);
  return GLQB_OK;
}

// Steps of fewer routings through trellis experts are chained (launch_chained): every launch of the tensor-core form, whose GEMMs let
// what follows them start when they end, the two matmuls of the streaming form.  Its other launches, started early, take
// registers and shared memory from the matmul that they wait for; E8 experts, whose shared memory is the L1 that their gathers
// live in, are not chained at all.  Eager calls of 128 experts, top 8, of 2048 x 768, 512 tokens, matmuls / every launch 290.8 / 286.0 us, of
// 64 experts, top 2, of 1024 x 512, 97.4 / 91.5.  In a graph, none / the matmuls / every launch with triggers in all of them: 32 experts,
// top 2, of 1024 x 512, 32 tokens (streaming) 58.2 / 57.6 / 67.6; E8, 32 experts, top 4, of 2048 x 768, 256 tokens 236.5 / 306.9 / 396.1.
constexpr long long MOE_CHAIN_MAX = 8192;

// grouping: one launch; count / tables / place kernels (many CTAs) for steps in which counting all routings in every CTA
// would take longer than three launches.  128 experts, top 8, one CTA or three launches / one launch of many: 256 tokens
// 24 / 19 us, 4096 tokens 56 / 25 us (cold, by ncu).
static void moe_launch_group(const MoeDev& M, const void* ids, int tokens, uint8_t* ws, cudaStream_t st) {
  const int R = tokens * M.top_k;
  const size_t sh = (6 * (size_t)M.E + 1) * sizeof(int);
  if (R < MOE_GROUP_SPLIT_MIN) {
    const int ctas = std::max(1, std::min(MOE_GROUP_CTAS, (R + MOE_GROUP_SHARE - 1) / MOE_GROUP_SHARE));
    moe_group_kernel<<<ctas, 1024, sh, st>>>(M, ids, tokens, ws, 0);
    return;
  }
  const int nb = (R + MOE_GROUP_CHUNK - 1) / MOE_GROUP_CHUNK;
  cudaMemsetAsync(ws + M.o_count, 0, sizeof(int) * M.E, st);
  moe_count_kernel<<<nb, 1024, M.E * sizeof(int), st>>>(M, ids, tokens, ws);
  moe_group_kernel<<<1, 1024, sh, st>>>(M, ids, tokens, ws, 1);
  moe_place_kernel<<<nb, 1024, 2 * M.E * sizeof(int), st>>>(M, ids, tokens, ws);
}

// moe_mid_warp_kernel works through the chunks of a pair of slots in one warp, moe_mid_kernel spreads those of some slots over
// eight: the longer that chain, the more routings it takes to fill the SMs in spite of it.  `steps`: chunks that a pair loads.
// By CTAs / by warps, in a graph.  128 experts, top 8, of 2048 x 768: eight steps (streaming form), 1 token 88.7 / 102.8 us, 64 tokens
// 243 / 255; five, 256 tokens 239.7 / 243.1, 512 tokens 286.6 / 281.7, 2048 tokens 432 / 418.  Three (32 experts, top 2, of 1024 x 512): 1 token 51.2 /
// 53.8, 4 tokens 56.1 / 55.2, 64 tokens 59.0 / 57.8; 64 experts, 1024 tokens 94.0 / 92.7.  Five, of which four are partial sums (8
// experts, top 2, of 2048 x 512): 8 tokens 60.3 / 63.6.
static int moe_mid_warp_min(int steps) {
  const char* e = getenv("GLQB_MOE_MID_WARP_MIN");
  return e ? atoi(e) : steps <= 3 ? 8 : 4096;
}
static void moe_launch_mid(const GlqbMoePlan* P, const MoeDev& M, int tokens, uint8_t* ws, bool chain, cudaStream_t st) {
  const int R = tokens * M.top_k;
  const bool by_warps = R >= (M.gemm ? P->mid_warp_min_gemm : P->mid_warp_min);
  const int per = by_warps ? MIDW_ROWS * MIDW_WARPS : P->mid_sg;
  if (by_warps) launch_chained(chain, moe_mid_warp_kernel, (R + per - 1) / per, MIDW_WARPS * 32, MIDW_WARPS * moe_midw_warp_bytes(M.w13_out), st, M, tokens, ws);
  else launch_chained(chain, moe_mid_kernel, (R + per - 1) / per, MOE_XF_THREADS, P->mid_smem, st, M, tokens, per, ws);
}

// tokens per CTA of the input transform: one tile of 8192 values, fewer when that would leave SMs without work
static int moe_in_tokens(const MoeDev& M, int tokens) {
  int tt = std::max(1, std::min(8, 8192 / M.hidden));
  while (tt > 1 && (tokens + tt - 1) / tt < 296) --tt;
  return tt;
}

extern "C" {

int glqb_moe_plan_create(const GlqbMoeDesc* d, GlqbMoePlan** out) {
  if (!d || !out) return moe_fail(GLQB_E_INVALID, "moe_plan_create: null argument");
  if (d->num_experts < 1 || d->num_experts > 4096 || d->top_k < 1 || d->top_k > 64 || d->max_tokens < 1)
    return moe_fail(GLQB_E_INVALID, "moe_plan_create: experts=%d top_k=%d max_tokens=%d", d->num_experts, d->top_k,
                    d->max_tokens);
  const bool gated = d->activation >= 0 && d->activation <= 2;
  if (d->activation < 0 || d->activation > 5) return moe_fail(GLQB_E_INVALID, "moe_plan_create: activation %d", d->activation);
  const bool e8 = d->format == GLQB_FMT_E8_SHELL;
  if (d->format != GLQB_FMT_TRELLIS_3INST && !e8) return moe_fail(GLQB_E_INVALID, "moe_plan_create: format %d", d->format);
  if (d->hidden % 32 || d->inter % 32 || d->w13_out % 32)
    return moe_fail(GLQB_E_INVALID, "moe_plan_create: hidden/inter/w13_out must be multiples of 32");
  if (e8) {
    if (d->hidden % GM_TILE_K || d->inter % GM_TILE_K)
      return moe_fail(GLQB_E_INVALID, "moe_plan_create: E8 experts need hidden and inter to be multiples of 64");
    if (d->e8_stages < 1 || d->e8_stages > 3) return moe_fail(GLQB_E_INVALID, "moe_plan_create: E8 stages %d (1..3)", d->e8_stages);
    for (int s = 0; s < d->e8_stages; ++s) {
      const int en = d->e8_table_entries[s];
      if (!d->w13_qidxs[s] || !d->w2_qidxs[s] || !d->e8_table[s] || en < 1 || en > 65536 || (en & (en - 1)))
        return moe_fail(GLQB_E_INVALID, "moe_plan_create: E8 stage %d: null index matrix / table, or %d table entries", s, en);
      if (s && (!d->w13_inv_rs[s - 1] || !d->w2_inv_rs[s - 1]))
        return moe_fail(GLQB_E_INVALID, "moe_plan_create: E8 stage %d without its inverse residual scales", s);
    }
  }
  if (d->w13_out != (gated ? 2 : 1) * d->inter)
    return moe_fail(GLQB_E_INVALID, "moe_plan_create: w13_out=%d does not match inter=%d for activation %d", d->w13_out,
                    d->inter, d->activation);
  if (d->hidden > 8 * 1024 || d->inter > 4 * 1024 || d->w13_out > 16384)
    return moe_fail(GLQB_E_INVALID, "moe_plan_create: hidden <= 8192, inter <= 4096 supported");
  if ((!e8 && (!d->w13_packed || !d->w2_packed)) || !d->w13_su || !d->w13_sv || !d->w2_su || !d->w2_sv || !d->w13_wscale ||
      !d->w2_wscale)
    return moe_fail(GLQB_E_INVALID, "moe_plan_create: null weight pointer");
  if ((reinterpret_cast<uintptr_t>(d->w13_su) | reinterpret_cast<uintptr_t>(d->w13_sv) | reinterpret_cast<uintptr_t>(d->w2_su) |
       reinterpret_cast<uintptr_t>(d->w2_sv)) & 15)
    return moe_fail(GLQB_E_INVALID, "moe_plan_create: SU/SV tensors must be 16-byte aligned");
  GlqbMoePlan* P = new GlqbMoePlan();
  P->desc = *d;
  MoeDev& M = P->dev;
  memset(&M, 0, sizeof M);
  int rc;
  if ((rc = fill_blocks(d->blocks_n_w13, d->n_blocks_n_w13, d->hidden, M.off_n13, M.log_n13, "n_w13")) ||
      (rc = fill_blocks(d->blocks_m_w13, d->n_blocks_m_w13, d->w13_out, M.off_m13, M.log_m13, "m_w13")) ||
      (rc = fill_blocks(d->blocks_n_w2, d->n_blocks_n_w2, d->inter, M.off_n2, M.log_n2, "n_w2")) ||
      (rc = fill_blocks(d->blocks_m_w2, d->n_blocks_m_w2, d->hidden, M.off_m2, M.log_m2, "m_w2"))) {
    delete P;
    return rc;
  }
  for (int b = 0; b < d->n_blocks_m_w13; ++b) M.wide_m13 |= M.log_m13[b] > 10;
  M.nb_n13 = d->n_blocks_n_w13; M.nb_m13 = d->n_blocks_m_w13; M.nb_n2 = d->n_blocks_n_w2; M.nb_m2 = d->n_blocks_m_w2;
  // E8 experts run the tensor-core form at every token count; the streaming kernels below are picked with
  // placeholder rates and never launched for them
  const int k13a = e8 ? 4 : d->w13_bits, k13b = (!e8 && d->w13_packed2) ? d->w13_bits2 : 0;
  const int k2a = e8 ? 4 : d->w2_bits, k2b = (!e8 && d->w2_packed2) ? d->w2_bits2 : 0;
  // tokens per decode pass: 16 for small steps, 32 when experts see many tokens
  const double avg = (double)d->max_tokens * d->top_k / d->num_experts;
  (void)avg;
  P->nb = (k13b || k2b) ? 2 : 4;
  P->k13 = P->nb == 4 ? moe_mv_pick<4>(k13a, k13b) : moe_mv_pick<2>(k13a, k13b);
  P->k2 = P->nb == 4 ? moe_mv_pick<4>(k2a, k2b) : moe_mv_pick<2>(k2a, k2b);
  if (!P->k13 || !P->k2) {
    delete P;
    return moe_fail(GLQB_E_INVALID, "moe_plan_create: no kernel for trellis rates w13 K=%d+%d, w2 K=%d+%d", k13a, k13b, k2a,
                    k2b);
  }
  M.w13[0] = (const uint8_t*)d->w13_packed; M.w13[1] = (const uint8_t*)d->w13_packed2;
  M.w2[0] = (const uint8_t*)d->w2_packed; M.w2[1] = (const uint8_t*)d->w2_packed2;
  M.w13_stride[0] = (long long)d->w13_out * d->hidden * k13a / 8;
  M.w13_stride[1] = (long long)d->w13_out * d->hidden * k13b / 8;
  M.w2_stride[0] = (long long)d->hidden * d->inter * k2a / 8;
  M.w2_stride[1] = (long long)d->hidden * d->inter * k2b / 8;
  M.format = d->format;
  if (e8) {
    M.e8_ns = d->e8_stages;
    M.w13_stride[0] = (long long)d->w13_out * (d->hidden / 8) * 2;     // int16 per 8 weights, every stage
    M.w2_stride[0] = (long long)d->hidden * (d->inter / 8) * 2;
    M.w13_stride[1] = M.w2_stride[1] = 0;
    for (int s = 0; s < d->e8_stages; ++s) {
      M.e8_w13[s] = (const uint8_t*)d->w13_qidxs[s];
      M.e8_w2[s] = (const uint8_t*)d->w2_qidxs[s];
      M.e8_tab[s] = d->e8_table[s];
      M.e8_ent[s] = d->e8_table_entries[s];
      if (s) { M.e8_w13_inv[s - 1] = d->w13_inv_rs[s - 1]; M.e8_w2_inv[s - 1] = d->w2_inv_rs[s - 1]; }
    }
  }
  M.w13_su = (const __half*)d->w13_su; M.w13_sv = (const __half*)d->w13_sv;
  M.w13_wscale = d->w13_wscale; M.w13_inv2 = d->w13_inv_resid_scale2;
  M.w2_su = (const __half*)d->w2_su; M.w2_sv = (const __half*)d->w2_sv;
  M.w2_wscale = d->w2_wscale; M.w2_inv2 = d->w2_inv_resid_scale2;
  if ((k13b && !M.w13_inv2) || (k2b && !M.w2_inv2)) {
    delete P;
    return moe_fail(GLQB_E_INVALID, "moe_plan_create: second stage without its inverse residual scales");
  }
  M.E = d->num_experts; M.hidden = d->hidden; M.inter = d->inter; M.w13_out = d->w13_out; M.top_k = d->top_k;
  M.max_tokens = d->max_tokens; M.act = d->activation; M.gated = gated ? 1 : 0;
  M.ids_i64 = d->ids_are_int64; M.x_dtype = d->x_dtype; M.y_dtype = d->y_dtype;
  // K chunking: 32 groups (1024 columns) per unit
  const int gps13 = d->hidden / 32, gps2 = d->inter / 32;
  M.gpc13 = std::min(gps13, 32); M.kch13 = (gps13 + M.gpc13 - 1) / M.gpc13;
  M.gpc2 = std::min(gps2, 32); M.kch2 = (gps2 + M.gpc2 - 1) / M.gpc2;
  // workspace
  const size_t R = (size_t)d->max_tokens * d->top_k;
  size_t o = 0;
  M.o_count = o; o = al(o + 4 * (size_t)M.E);
  M.o_base = o; o = al(o + 4 * (size_t)M.E);
  M.o_cursor = o; o = al(o + 4 * (size_t)M.E);
  M.o_row0 = o; o = al(o + 4 * (size_t)M.E);
  M.o_work = o; o = al(o + 16);
  M.o_route_tok = o; o = al(o + 4 * R);
  M.o_route_exp = o; o = al(o + 4 * R);
  M.o_slot_of = o; o = al(o + 4 * R);
  M.o_xr1 = o; o = al(o + (size_t)d->max_tokens * d->hidden * 2 * XR_TRELLIS_EXPAND);
  M.o_part1 = o; o = al(o + (size_t)M.kch13 * R * d->w13_out * 4);
  M.o_xr2 = o; o = al(o + R * d->inter * 2 * XR_TRELLIS_EXPAND);
  M.o_part2 = o; o = al(o + (size_t)M.kch2 * R * d->hidden * 4);
  P->ws_bytes = o;
  P->two_stages = k13b || k2b;
  // tensor-core form: its buffers overlay the decode form's (a step runs one or the other)
  P->g13 = e8 ? moe_gemm_pick_e8(d->e8_stages) : moe_gemm_pick(k13a, k13b);
  P->g2 = e8 ? moe_gemm_pick_e8(d->e8_stages) : moe_gemm_pick(k2a, k2b);
  P->gemm_ok = P->g13 && P->g2 && d->hidden % GM_TILE_K == 0 && d->inter % GM_TILE_K == 0 && M.E <= 4096 &&
               (e8 || R >= (size_t)M.E * moe_gemm_min_avg(P->two_stages));
  if (P->gemm_ok) {
    MoeDev& G = P->devg;
    G = M;
    G.gemm = 1; G.kch13 = 1; G.kch2 = 1;
    G.tile_tn = e8 ? MOE_TN_E8 : MOE_TN;
    G.k13a = k13a; G.k13b = k13b; G.k2a = k2a; G.k2b = k2b;
    const size_t tiles = R / G.tile_tn + M.E;
    const size_t mt13 = (d->w13_out + GM_TILE_M - 1) / GM_TILE_M, mt2 = (d->hidden + GM_TILE_M - 1) / GM_TILE_M;
    G.max_items13 = (int)(tiles * mt13);
    G.max_items2 = (int)(tiles * mt2);
    auto al1k = [](size_t v) { return (v + 1023) / 1024 * 1024; };
    size_t g = al1k((size_t)M.o_xr1);
    const size_t rows = R + 16 * tiles;                        // every tile rounds its tokens up to 16
    G.o_xr1 = g; g = al1k(g + rows * (d->hidden / GM_TILE_K) * 128);
    G.o_part1 = g; g = al1k(g + R * d->w13_out * 4);
    G.o_xr2 = g; g = al1k(g + rows * (d->inter / GM_TILE_K) * 128);
    G.o_part2 = g; g = al1k(g + R * d->hidden * 4);
    G.o_trow = g; g = al1k(g + 8 * R);
    G.o_layers13 = g; g = al1k(g + sizeof(DevLinear) * M.E);
    G.o_layers2 = g; g = al1k(g + sizeof(DevLinear) * M.E);
    G.o_items13 = g; g = al1k(g + sizeof(GemmItem) * G.max_items13);
    G.o_items2 = g; g = al1k(g + sizeof(GemmItem) * G.max_items2);
    G.o_nitems = g; g = al1k(g + 16);
    G.o_status = g; g = al1k(g + 16);
    P->ws_bytes = std::max(P->ws_bytes, g);
    if (cudaFuncSetAttribute(P->g13, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)moe_gemm_smem_bytes(e8)) != cudaSuccess ||
        cudaFuncSetAttribute(P->g2, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)moe_gemm_smem_bytes(e8)) != cudaSuccess) {
      cudaGetLastError();
      P->gemm_ok = false;
    }
  }
  {
    // Slots per CTA and routings per pass are chosen for three CTAs per SM; one row may need more: a block shorter than
    // 1024 values takes a whole chunk, and 16 blocks per side at the largest served sizes come to 156,288 bytes (mid kernel).  The limit is a
    // property of the kernels, not of a plan, so every plan sets the same one.
    const size_t budget = 74 * 1024, limit = 200 * 1024;
    auto mid_bytes = [&](int sg) { return (size_t)4 * FHT_CHUNK_WORDS * (moe_chunks_all(sg, M.nb_m13, M.log_m13) + moe_chunks_all(sg, M.nb_n2, M.log_n2)); };
    auto out_bytes = [&](int rg) { return 4 * ((size_t)FHT_CHUNK_WORDS * moe_chunks_all(rg, M.nb_m2, M.log_m2) + (rg < d->top_k ? (size_t)d->hidden : 0)); };
    P->mid_sg = 8;
    while (P->mid_sg > 1 && mid_bytes(P->mid_sg) > budget) --P->mid_sg;
    P->out_rg = std::min(8, d->top_k);
    // (running sums between passes are only needed when one pass cannot hold all routings of a token)
    while (P->out_rg > 1 && out_bytes(P->out_rg) > budget) --P->out_rg;
    P->mid_smem = mid_bytes(P->mid_sg);
    bool by_warps = !M.wide_m13 && MIDW_WARPS * moe_midw_warp_bytes(d->w13_out) <= budget;
    for (int b = 0; b < M.nb_n2; ++b) by_warps = by_warps && M.log_n2[b] <= 10;
    if (by_warps) {
      const int c13 = moe_chunks_all(MIDW_ROWS, M.nb_m13, M.log_m13), c2 = moe_chunks_all(MIDW_ROWS, M.nb_n2, M.log_n2);
      P->mid_warp_min = moe_mid_warp_min(c13 * M.kch13 + c2);
      P->mid_warp_min_gemm = moe_mid_warp_min(c13 + c2);
    }
    P->out_smem = out_bytes(P->out_rg);
    if (P->mid_smem > limit || P->out_smem > limit) {
      delete P;
      return moe_fail(GLQB_E_INVALID, "moe_plan_create: one row of the expert transforms needs more than %zu bytes of shared memory", limit);
    }
    if (cudaFuncSetAttribute(moe_group_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             (int)((6 * 4096 + 1) * sizeof(int))) != cudaSuccess ||
        cudaFuncSetAttribute(moe_mid_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)limit) != cudaSuccess ||
        cudaFuncSetAttribute(moe_mid_warp_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)limit) != cudaSuccess ||
        cudaFuncSetAttribute(moe_out_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)limit) != cudaSuccess) {
      delete P;
      return moe_fail(GLQB_E_CUDA, "moe_plan_create: %s", cudaGetErrorString(cudaGetLastError()));
    }
  }
  if (e8 && !P->gemm_ok) {
    delete P;
    return moe_fail(GLQB_E_INVALID, "moe_plan_create: the tensor-core form is unavailable for these E8 experts");
  }
  int dev_id = 0;
  if (cudaGetDevice(&dev_id) != cudaSuccess ||
      cudaDeviceGetAttribute(&P->sm_count, cudaDevAttrMultiProcessorCount, dev_id) != cudaSuccess) {
    delete P;
    return moe_fail(GLQB_E_CUDA, "moe_plan_create: no CUDA device");
  }
  const int units13 = M.E * (d->w13_out / 32) * M.kch13, units2 = M.E * (d->hidden / 32) * M.kch2;
  const int ctas = P->sm_count * 2;
  P->grid13 = std::max(1, std::min(ctas, (units13 + MV_WARPS - 1) / MV_WARPS));
  P->grid2 = std::max(1, std::min(ctas, (units2 + MV_WARPS - 1) / MV_WARPS));
  *out = P;
  return GLQB_OK;
}

size_t glqb_moe_plan_workspace_bytes(const GlqbMoePlan* p) { return p ? p->ws_bytes : 0; }

int64_t glqb_moe_plan_code_bytes(const GlqbMoePlan* p) {
  if (!p) return 0;
  const MoeDev& M = p->dev;
  if (M.format == GLQB_FMT_E8_SHELL) return (int64_t)M.E * M.e8_ns * (M.w13_stride[0] + M.w2_stride[0]);
  return (int64_t)M.E * (M.w13_stride[0] + M.w13_stride[1] + M.w2_stride[0] + M.w2_stride[1]);
}

int glqb_moe_plan_run(GlqbMoePlan* P, const void* x, const void* topk_ids, const float* topk_weights, void* y,
                      int32_t tokens, void* workspace, size_t workspace_bytes, void* stream_) {
  if (!P || !x || !topk_ids || !topk_weights || !y) return moe_fail(GLQB_E_INVALID, "moe_plan_run: null argument");
  if (tokens < 1 || tokens > P->desc.max_tokens)
    return moe_fail(GLQB_E_INVALID, "moe_plan_run: %d tokens, plan was built for at most %d", tokens, P->desc.max_tokens);
  if (!workspace || workspace_bytes < P->ws_bytes)
    return moe_fail(GLQB_E_WORKSPACE, "moe_plan_run: workspace of %zu bytes needed, %zu given", P->ws_bytes, workspace_bytes);
  if (reinterpret_cast<uintptr_t>(workspace) & 255) return moe_fail(GLQB_E_WORKSPACE, "workspace must be 256-byte aligned");
  cudaStream_t st = reinterpret_cast<cudaStream_t>(stream_);
  uint8_t* ws = reinterpret_cast<uint8_t*>(workspace);
  const bool chain = P->dev.format != GLQB_FMT_E8_SHELL && (long long)tokens * P->dev.top_k < MOE_CHAIN_MAX;
  if (P->gemm_ok && (P->dev.format == GLQB_FMT_E8_SHELL ||
                     (long long)tokens * P->dev.top_k >= (long long)P->dev.E * moe_gemm_min_avg(P->two_stages))) {
    const MoeDev& G = P->devg;
    const int R = tokens * G.top_k;
    moe_launch_group(G, topk_ids, tokens, ws, st);
    const int tt = moe_in_tokens(G, tokens);
    launch_chained(chain, moe_rht_in_gemm_kernel, (tokens + tt - 1) / tt, MOE_XF_THREADS, (fht_words(8192) + 2 * tt * G.top_k) * 4, st, G, tokens,
                   tt, reinterpret_cast<const uint8_t*>(x), ws);
    const bool g_e8 = G.format == GLQB_FMT_E8_SHELL;
    const int g_threads = g_e8 ? GM_THREADS : TG_THREADS;
    int* status = reinterpret_cast<int*>(ws + G.o_status);
    const int* nitems = reinterpret_cast<const int*>(ws + G.o_nitems);
    {
      MoeTimer t(P, st);
      launch_chained(chain, P->g13, std::min(P->sm_count, G.max_items13), g_threads, moe_gemm_smem_bytes(g_e8), st,
                     reinterpret_cast<const DevLinear*>(ws + G.o_layers13), reinterpret_cast<const GemmItem*>(ws + G.o_items13),
                     G.max_items13, ws, status, nitems, tokens);
    }
    moe_launch_mid(P, G, tokens, ws, chain, st);
    {
      MoeTimer t(P, st);
      launch_chained(chain, P->g2, std::min(P->sm_count, G.max_items2), g_threads, moe_gemm_smem_bytes(g_e8), st,
                     reinterpret_cast<const DevLinear*>(ws + G.o_layers2), reinterpret_cast<const GemmItem*>(ws + G.o_items2),
                     G.max_items2, ws, status, nitems + 1, tokens);
    }
    launch_chained(chain, moe_out_kernel, tokens, MOE_XF_THREADS, P->out_smem, st, G, tokens, P->out_rg, topk_weights, ws,
                   reinterpret_cast<uint8_t*>(y));
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return moe_fail(GLQB_E_CUDA, "moe_plan_run: %s", cudaGetErrorString(e));
    return GLQB_OK;
  }
  const MoeDev& M = P->dev;
  const int R = tokens * M.top_k;
  moe_launch_group(M, topk_ids, tokens, ws, st);
  const int tt = moe_in_tokens(M, tokens);
  moe_rht_in_kernel<<<(tokens + tt - 1) / tt, MOE_XF_THREADS, fht_words(8192) * 4, st>>>(M, tokens, tt, reinterpret_cast<const uint8_t*>(x), ws);
  MoeMvArgs A;
  memset(&A, 0, sizeof A);
  A.codes[0] = M.w13[0]; A.codes[1] = M.w13[1]; A.stride[0] = M.w13_stride[0]; A.stride[1] = M.w13_stride[1];
  A.inv2 = M.w13_inv2;
  A.count = reinterpret_cast<const int*>(ws + M.o_count);
  A.base = reinterpret_cast<const int*>(ws + M.o_base);
  A.row_map = reinterpret_cast<const int*>(ws + M.o_route_tok);
  A.xr = reinterpret_cast<const __half*>(ws + M.o_xr1);
  A.part = reinterpret_cast<float*>(ws + M.o_part1);
  A.work = reinterpret_cast<int*>(ws + M.o_work);
  A.E = M.E; A.m = M.w13_out; A.n = M.hidden; A.gps = M.hidden / 32; A.strips = M.w13_out / 32;
  A.kchunks = M.kch13; A.gpc = M.gpc13; A.R = R;
  {
    MoeTimer t(P, st);
    launch_chained(chain, P->k13, P->grid13, MV_THREADS, 0, st, A);
  }
  moe_launch_mid(P, M, tokens, ws, false, st);
  A.codes[0] = M.w2[0]; A.codes[1] = M.w2[1]; A.stride[0] = M.w2_stride[0]; A.stride[1] = M.w2_stride[1];
  A.inv2 = M.w2_inv2;
  A.row_map = nullptr;
  A.xr = reinterpret_cast<const __half*>(ws + M.o_xr2);
  A.part = reinterpret_cast<float*>(ws + M.o_part2);
  A.work = reinterpret_cast<int*>(ws + M.o_work) + 1;
  A.m = M.hidden; A.n = M.inter; A.gps = M.inter / 32; A.strips = M.hidden / 32;
  A.kchunks = M.kch2; A.gpc = M.gpc2;
  {
    MoeTimer t(P, st);
    launch_chained(chain, P->k2, P->grid2, MV_THREADS, 0, st, A);
  }
  moe_out_kernel<<<tokens, MOE_XF_THREADS, P->out_smem, st>>>(M, tokens, P->out_rg, topk_weights, ws, reinterpret_cast<uint8_t*>(y));
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return moe_fail(GLQB_E_CUDA, "moe_plan_run: %s", cudaGetErrorString(e));
  return GLQB_OK;
}

int glqb_moe_plan_status(const GlqbMoePlan* P, const void* workspace, void* stream_) {
  if (!P || !workspace) return moe_fail(GLQB_E_INVALID, "moe_plan_status: null argument");
  if (!P->gemm_ok) return GLQB_OK;
  int st = 0;
  cudaStream_t s = reinterpret_cast<cudaStream_t>(stream_);
  if (cudaMemcpyAsync(&st, reinterpret_cast<const uint8_t*>(workspace) + P->devg.o_status, sizeof st, cudaMemcpyDeviceToHost, s) !=
          cudaSuccess ||
      cudaStreamSynchronize(s) != cudaSuccess)
    return moe_fail(GLQB_E_CUDA, "moe_plan_status: %s", cudaGetErrorString(cudaGetLastError()));
  // (a workspace in which no tensor-core step has run yet, only been captured, holds anything)
  if (st >= ST_GAVE_UP_PRODUCER && st <= ST_GAVE_UP_PEER)
    return moe_fail(GLQB_E_DEVICE, "moe: a bounded wait inside the GEMM kernel gave up (role %d); results are invalid", st);
  return GLQB_OK;
}

int glqb_moe_plan_set_timing(GlqbMoePlan* P, int32_t enable) {
  if (!P) return moe_fail(GLQB_E_INVALID, "moe_plan_set_timing: null plan");
  P->timing = enable != 0;
  P->ev_used = 0;
  return GLQB_OK;
}

int glqb_moe_plan_kernel_ms(GlqbMoePlan* P, double* total_ms_out, int32_t* runs_out) {
  if (!P || !total_ms_out || !runs_out) return moe_fail(GLQB_E_INVALID, "moe_plan_kernel_ms: null argument");
  double total = 0.0;
  for (size_t i = 0; i + 1 < P->ev_used; i += 2) {
    float ms = 0.f;
    if (cudaEventSynchronize(P->ev[i + 1]) != cudaSuccess || cudaEventElapsedTime(&ms, P->ev[i], P->ev[i + 1]) != cudaSuccess)
      return moe_fail(GLQB_E_CUDA, "moe_plan_kernel_ms: %s", cudaGetErrorString(cudaGetLastError()));
    total += ms;
  }
  *total_ms_out = total;
  *runs_out = (int32_t)(P->ev_used / 4);        // two matmuls per run
  return GLQB_OK;
}

void glqb_moe_plan_destroy(GlqbMoePlan* p) {
  if (!p) return;
  for (cudaEvent_t e : p->ev) cudaEventDestroy(e);
  delete p;
}

}  // extern "C"
