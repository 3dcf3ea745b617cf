// Single-launch decode kernels: input transform, decode + mma and output transform of a few tokens in one kernel.
#pragma once
#include "glqb_kernels.cuh"
#include "glqb_fht_fast.cuh"

namespace glqb {

// ---------------------------------------------------------------------------------------------
// One launch per decode linear (up to 8 tokens): input transform, 3INST decode + mma, output transform.
//
// Used for plans whose layers all read the same input (one layer, or the q/k/v / gate/up shards of a fused
// projection).  The reference's counterpart is its FUSE_IN matvec (glq/csrc/glq_trellis.cu:315-370, chosen at
// :1290-1295), which still needs a second launch for the output transform.
//   phase 1  every CTA recomputes the (cheap) input transform of the shared input into its own shared memory,
//            in the B-fragment layout of the MMAs (fht_fast);
//   phase 2  work unit = (layer, 32-row strip, chunk of 64 column groups): warp w of the CTA decodes groups
//            [8w, 8w + 8) of the chunk; the eight warps' partial sums are added in warp order through shared
//            memory and written as partial sum number `chunk` of the strip (a strip of up to 2048 columns has
//            exactly one);
//   phase 3  a CTA that finishes the last unit of a Hadamard block of the output (integer ticket per block,
//            released and acquired by one atomic, see fused_ticket; nobody ever waits) runs that block's output transform.  The
//            result does not depend on which CTA that is.  Tickets are returned to zero by the CTA that completes them.
// ---------------------------------------------------------------------------------------------
constexpr int FUSED_MAX_LAYERS = 8;
constexpr int FUSED_MAX_TODO = FUSED_MAX_LAYERS * GLQB_MAX_BLOCKS;       // one CTA may complete every output block of a launch
constexpr int FUSED_CHUNK_GROUPS = 64;          // column groups per work unit: 8 warps x 8 groups
constexpr int FUSED_MAX_TOKENS = FUSED_MAX_TOKENS_C;

__device__ __forceinline__ uint4 lds_v4(uint32_t addr) {
  uint4 v;
  asm volatile("ld.shared.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(addr));
  return v;
}

// bytes of shared memory the transformed activations of a single-launch call take: trellis keeps (x, 0) half pairs
// in fragment order; E8 keeps fp16 in the order of xr_index_e8 (several tokens: interleaved in groups of eight)
template <bool E8FMT>
__host__ __device__ __forceinline__ size_t fused_xs_bytes(int n, int batch) {
  if (E8FMT) return (size_t)(batch == 1 ? 1 : 8) * n * 2;
  return (size_t)batch * n * 4;
}

// shared-memory bytes of the fused kernel: activations (2 halfs per column and token), transform scratch
// (the largest input block, or output tile, padded by one word per 32), the warps' partial sums
__host__ __device__ __forceinline__ size_t fused_smem_bytes(int n, int batch, int scratch_elems, bool e8 = false) {
  const size_t xs = e8 ? ((fused_xs_bytes<true>(n, batch) + 15) & ~(size_t)15) : fused_xs_bytes<false>(n, batch);
  return xs + ((size_t)scratch_elems + scratch_elems / 32) * 4 + 8 * 256 * 4 + 64;
}

// longest input block of the in-kernel shuffle transform (8192; E8, whose prefetched indices leave fewer registers, 4096)
__host__ __device__ constexpr int fused_in_max_log(bool e8) { return e8 ? 12 : 13; }
constexpr int FUSED_OUT_MAX_LOG = 13;            // longest output block the kernel can transform itself: 8192 (see out_split_log)

// Output transform of one (layer, Hadamard block, token) by the CTA that completed the block, with the
// low-latency transform.  Blocks of up to 8192 rows (longer ones are left to rht_out_kernel).
// `C` (tensor-parallel ranks, row-parallel layer): instead of being written to y, the block's transformed values are
// stored into every rank's receive area at float offset `piece` (this rank's source slot of epoch `comm_e`); the
// caller exchanges flags and adds the ranks' blocks afterwards.
// Registers are short here (128 per thread, two CTAs per SM, the next unit's codes may be in flight): one offset instead
// of a pointer per rank, signs packed (E8) and requested late by threads with LATE values or more (fht_fast_e).  E8 kernels
// without that spilled 51 words instead of 22 and took 17.5 us for two stages of 2048 x 2048 (one token, in a graph) instead
// of 16.8, 14.2 instead of 12.6 for 4096 x 512.
template <bool E8FMT, int LATE>
__device__ __forceinline__ void fused_out_block(const DevLinear& L, int b, int tok, float in_scale,
                                                const uint8_t* __restrict__ ws, uint8_t* __restrict__ y_base, float* fbuf,
                                                const CommDev* C = nullptr, int comm_e = 0, long long piece = 0) {
  const int logbs = L.bm_log[b], off = L.bm_off[b];
  const int m = L.m, cnt = L.fixed_slots, out_f = L.out_f, y_dtype = L.y_dtype;
  const long long slot_stride = (long long)L.batch * m;
  const float wscale = L.wscale * in_scale;                  // in_scale: 1 / rms of the token (fused RMSNorm), else 1
  const float* row_scale = L.row_scale;
  const float* part = reinterpret_cast<const float*>(ws + L.part_off) + (long long)tok * m + off;
  // the sums of a thread's values, slot by slot in ascending order; the loads of a few slots are in flight together (a value's
  // slots one after the other, value after value, made the block wait for E / 4 * slots round trips to L2; with that, loads of
  // a thread's inputs together and one ticket per block and CTA four decoder layers take 333 us instead of 344.5)
  auto load = [&](int i0, auto& v) {
    constexpr int E = sizeof(v) / sizeof(float), V = E >= 4 ? 4 : 1, UNROLL = E >= 32 ? 1 : E >= 16 ? 2 : 4;
#pragma unroll
    for (int j = 0; j < E; ++j) v[j] = 0.f;
#pragma unroll UNROLL
    for (int k = 0; k < cnt; ++k) {
      const float* p = part + i0 + k * slot_stride;
#pragma unroll
      for (int j = 0; j < E; j += V) {
        if constexpr (V == 4) {
          const float4 t = __ldcg(reinterpret_cast<const float4*>(p + j));
          v[j] += t.x; v[j + 1] += t.y; v[j + 2] += t.z; v[j + 3] += t.w;
        } else {
          v[j] += __ldcg(p + j);
        }
      }
    }
#pragma unroll
    for (int j = 0; j < E; ++j) {
      v[j] *= wscale;
      if (row_scale) v[j] *= row_scale[off + i0 + j];
    }
  };
  const long long yo = L.y_off + (long long)tok * L.y_stride + off;
  if (L.stop_at_yrht) {            // rotated-domain result wanted: reduce and scale only
    for (int i = threadIdx.x; i < (1 << logbs); i += blockDim.x) {
      float v[1];
      load(i, v);
      reinterpret_cast<float*>(y_base)[yo + i] = v[0];
    }
    return;
  }
  const float rs = rsqrtf((float)(1 << logbs));
  const __half* su = L.su + off;
  const bool accumulate = L.y_accumulate != 0;
  auto pre = [&](int i) {                                              // the sign, requested before the partial sums
    if constexpr (E8FMT) return su[i]; else return __half2float(su[i]);
  };
  auto store = [&](int i, float val, float sign) {
    if (off + i < out_f) {
      float r = val * rs * sign;
      if (accumulate) r += load_act(y_base, yo + i, y_dtype);          // residual add
      store_act(y_base, yo + i, y_dtype, r);
    }
  };
  if (C) {
    const int world = C->world;
    const size_t at = (size_t)(comm_slot(*C, 0, comm_e, C->rank) - C->data[0]) + (size_t)piece;      // the same in every area
    auto push = [&](int i, float val, float sign) {                    // consecutive threads, consecutive i
      const float r = val * rs * sign;
#pragma unroll
      for (int k = 0; k < COMM_MAX_RANKS; ++k)
        if (k < world) C->data[k][at + i] = r;
    };
    fht_fast<FUSED_OUT_MAX_LOG, LATE, E8FMT>(fbuf, logbs, load, pre, push);
    return;
  }
  fht_fast<FUSED_OUT_MAX_LOG, LATE, E8FMT>(fbuf, logbs, load, pre, store);
}

// Phase 1 of the single-launch decode kernels: the transformed activations of the shared input, in shared memory
// (every CTA computes them itself; wide inputs are copied from the workspace, where rht_in_kernel left them).
// Fused RMSNorm: rstd_s[token] receives 1 / rms, which the callers apply to the OUTPUT.
template <bool E8FMT>
__device__ __forceinline__ void fused_phase1(const DevLinear& L0, int batch, const uint8_t* __restrict__ x_base,
                                             const uint8_t* __restrict__ ws, __half2* xs, float* fbuf, float* red,
                                             float* rstd_s) {
  const int n = L0.n;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (L0.xr_global) {
    // wide inputs: rht_in_kernel transformed them once, just before this kernel; every CTA copies the result
    const uint4* src = reinterpret_cast<const uint4*>(ws + L0.xr_off);
    uint4* dst = reinterpret_cast<uint4*>(xs);
    const int n16 = (int)(fused_xs_bytes<E8FMT>(n, batch) >> 4);
    for (int i = threadIdx.x; i < n16; i += blockDim.x) dst[i] = __ldcg(src + i);
    __syncthreads();
  } else {
    const int x_dtype = L0.x_dtype;
    const void* nw = L0.in_norm_w;
    const int nw_dtype = L0.in_norm_dtype;
    const bool gated = L0.in_gated_act != 0;
    const bool vec_ok = !gated && act_rows_aligned4(x_base, L0.x_off, L0.x_stride, x_dtype) &&
                        (nw == nullptr || (reinterpret_cast<uintptr_t>(nw) & 15) == 0);
    const __half* sv = L0.sv;
    for (int tok = 0; tok < batch; ++tok) {
      const long long xt0 = L0.x_off + (long long)tok * L0.x_stride;
      float ss = 0.f;                                        // this thread's share of sum(x^2) (fused RMSNorm)
      // value of column i_abs fed to the transform: x (or act(gate) * up), times the norm weight, times the sign.
      // The 1 / rms factor of the norm is a scalar per token and is applied to the output instead.
      auto load1 = [&](int i_abs) -> float {
        if (E8FMT && i_abs >= L0.in_f) return 0.f;           // padded E8 layers (trellis layers are never padded)
        float v = input_value(L0, x_base, xt0, i_abs);
        ss += v * v;
        if (nw) v *= load_act(nw, i_abs, nw_dtype);
        return v * __half2float(sv[i_abs]);
      };
      for (int b = 0; b < L0.nbn; ++b) {
        const int off = L0.bn_off[b], logbs = L0.bn_log[b];
        const float rs = rsqrtf((float)(1 << logbs));
        const bool vok = vec_ok && (off & 3) == 0;
        __half2* xt = xs + (size_t)tok * n;                  // trellis: n half2 per token, (x, 0) pairs in fragment order
        auto put = [&](int i, float val) {
          const int col = off + i;
          if constexpr (E8FMT) {
            reinterpret_cast<__half*>(xs)[xr_index_e8(tok, col, n, batch)] = __float2half_rn(val * rs);
          } else {
            xt[((col & ~31) * XR_TRELLIS_EXPAND + xr_pos_trellis(col & 31)) >> 1] =
                __halves2half2(__float2half_rn(val * rs), __float2half_rn(0.f));
          }
        };
        auto none = [](int) -> float { return 0.f; };
        auto put3 = [&](int i, float val, float) { put(i, val); };
        auto load = [&](int i0, auto& v) {
          constexpr int E = sizeof(v) / sizeof(float);
          if constexpr (E >= 4) {
            if (vok && (!E8FMT || off + i0 + E - 1 < L0.in_f)) {   // (padded E8 layers: columns past in_features read as zero)
              // signs, norm weights and activations are all requested before the first is used
              uint2 s4[E / 4];
#pragma unroll
              for (int j = 0; j < E / 4; ++j) s4[j] = *reinterpret_cast<const uint2*>(sv + off + i0 + 4 * j);
              float q[E / 4][4];
              with_dtype(x_dtype, [&](auto dt) {
#pragma unroll
                for (int j = 0; j < E / 4; ++j) load_act4(x_base, xt0 + off + i0 + 4 * j, decltype(dt)::value, q[j]);
              });
              if (nw) {
                with_dtype(nw_dtype, [&](auto dt) {
                  float w4[E / 4][4];
#pragma unroll
                  for (int j = 0; j < E / 4; ++j) load_act4(nw, off + i0 + 4 * j, decltype(dt)::value, w4[j]);
#pragma unroll
                  for (int j = 0; j < E / 4; ++j) {
                    ss += q[j][0] * q[j][0] + q[j][1] * q[j][1] + q[j][2] * q[j][2] + q[j][3] * q[j][3];
#pragma unroll
                    for (int c = 0; c < 4; ++c) q[j][c] *= w4[j][c];
                  }
                });
              }
#pragma unroll
              for (int j = 0; j < E / 4; ++j) {
                const float2 a = __half22float2(*reinterpret_cast<const __half2*>(&s4[j].x));
                const float2 c = __half22float2(*reinterpret_cast<const __half2*>(&s4[j].y));
                v[4 * j] = q[j][0] * a.x; v[4 * j + 1] = q[j][1] * a.y; v[4 * j + 2] = q[j][2] * c.x; v[4 * j + 3] = q[j][3] * c.y;
              }
              return;
            }
          }
          if constexpr (E8FMT && E >= 4) {
            // padded layers: the thread in whose values the columns end takes the groups of four before the end in one load each
            // (8 tokens of 3640 columns, padded to 4096, two stages of 1024 rows, value by value / this: 57 / 51 us)
            if (vok) {
#pragma unroll
              for (int j = 0; j < E; j += 4) {
                float q[4] = {0.f, 0.f, 0.f, 0.f};
                if (off + i0 + j + 3 < L0.in_f) {
                  load_act4(x_base, xt0 + off + i0 + j, x_dtype, q);
                  float w[4] = {1.f, 1.f, 1.f, 1.f};
                  if (nw) load_act4(nw, off + i0 + j, nw_dtype, w);
                  ss += q[0] * q[0] + q[1] * q[1] + q[2] * q[2] + q[3] * q[3];
                  const uint2 s4 = *reinterpret_cast<const uint2*>(sv + off + i0 + j);
                  const float2 a = __half22float2(*reinterpret_cast<const __half2*>(&s4.x));
                  const float2 c = __half22float2(*reinterpret_cast<const __half2*>(&s4.y));
                  q[0] = q[0] * w[0] * a.x; q[1] = q[1] * w[1] * a.y; q[2] = q[2] * w[2] * c.x; q[3] = q[3] * w[3] * c.y;
                } else if (off + i0 + j < L0.in_f) {
#pragma unroll 1
                  for (int c = 0; c < 3; ++c) {
                    const float t = load1(off + i0 + j + c);
                    q[0] = c == 0 ? t : q[0]; q[1] = c == 1 ? t : q[1]; q[2] = c == 2 ? t : q[2];
                  }
                }
                v[j] = q[0]; v[j + 1] = q[1]; v[j + 2] = q[2]; v[j + 3] = q[3];
              }
              return;
            }
          }
#pragma unroll
          for (int j = 0; j < E; ++j) v[j] = load1(off + i0 + j);
        };
        fht_fast<fused_in_max_log(E8FMT), 64, false>(fbuf, logbs, load, none, put3);
        __syncthreads();
      }
      if (nw) {                                              // every value of the token was loaded exactly once
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
        if (lane == 0) red[warp] = ss;
        __syncthreads();
        if (threadIdx.x == 0) {
          float tot = 0.f;
          for (int w = 0; w < MV_WARPS; ++w) tot += red[w];
          rstd_s[tok] = rsqrtf(tot / (float)L0.in_f + L0.in_norm_eps);
        }
        __syncthreads();
      }
    }
  }

}

// First work unit of CTA b: consecutive ones, the CTAs with one more than the others in front, so that with two CTAs per SM no SM
// has two of those while another has none.  Spread evenly over the grid / this, one token of 11008 x 2048 (4 + 2 bits, 344 units
// for 296 CTAs): 30.7 / 27.2 us.
__device__ __forceinline__ int fused_first_unit(int b, int total_units) {
  const int each = total_units / (int)gridDim.x, more = total_units - each * (int)gridDim.x;
  return b * each + min(b, more);
}

// `done` more units of an output block are finished: whoever completes it (`need` units) transforms it.  Release (the CTA's
// stores, ordered before this by a barrier) and acquire (the other CTAs' stores, released before their increments) in one
// device-scope atomic; nobody ever waits on a ticket.
__device__ __forceinline__ void fused_ticket(int* __restrict__ tickets, int ticket, int done, int need, int code, int* todo, int* n_todo) {
  int old;
  asm volatile("atom.acq_rel.gpu.global.add.s32 %0, [%1], %2;" : "=r"(old) : "l"(tickets + ticket), "r"(done) : "memory");
  if (old + done == need) {
    tickets[ticket] = 0;                                      // ready for the next run
    todo[(*n_todo)++] = code;
  }
}

// Phase 3 of the single-launch decode kernels: output transforms of the blocks this CTA completed (`todo` entries
// are (layer << 8) | block), with the sum over tensor-parallel ranks when the layer asks for it.
template <bool E8FMT, int LATE>
__device__ __forceinline__ void fused_phase3(const DevLinear* layers, const int* todo, int nt, int batch, const float* rstd_s,
                                             const uint8_t* __restrict__ ws, uint8_t* __restrict__ y_base, float* fbuf,
                                             int scratch_elems, const CommDev& C, int comm_e) {
  for (int k = 0; k < nt; ++k) {
    const int li = todo[k] >> 8, b = todo[k] & 255;
    const DevLinear& L = layers[li];
    // (blocks longer than the split threshold take no ticket: rht_out_kernel transforms them)
    if (C.world > 1 && L.reduce) {
      // Row-parallel layer: every rank transforms its own partial result (its own signs), stores the block into
      // all ranks' receive areas, and after the flag exchange adds the ranks' blocks in rank order: the same bits
      // on every rank, residual add included.
      const int logbs = L.bm_log[b], bs = 1 << logbs, off = L.bm_off[b];
      const long long piece = (long long)L.comm_off + (long long)off * batch;            // floats; a multiple of 32
      for (int tok = 0; tok < batch; ++tok) {
        fused_out_block<E8FMT, LATE>(L, b, tok, rstd_s[tok], ws, y_base, fbuf, &C, comm_e, piece + ((long long)tok << logbs));
        __syncthreads();
      }
      comm_signal_and_wait(C, comm_e, L.comm_unit_base + b);
      const float* src = comm_slot(C, C.rank, comm_e, 0) + piece;
      const bool accumulate = L.y_accumulate != 0;
      for (int i = threadIdx.x * 4; i < bs * batch; i += blockDim.x * 4) {
        float4 a4 = make_float4(0.f, 0.f, 0.f, 0.f);
        for (int r = 0; r < C.world; ++r) {
          const float4 t = __ldcg(reinterpret_cast<const float4*>(src + (size_t)r * C.max_floats + i));
          a4.x += t.x; a4.y += t.y; a4.z += t.z; a4.w += t.w;
        }
        const float o[4] = {a4.x, a4.y, a4.z, a4.w};
        const int tok = i >> logbs, j = i & (bs - 1);
        const long long yo = L.y_off + (long long)tok * L.y_stride + off + j;
#pragma unroll
        for (int c = 0; c < 4; ++c)
          if (off + j + c < L.out_f) {
            float r = o[c];
            if (accumulate) r += load_act(y_base, yo + c, L.y_dtype);
            store_act(y_base, yo + c, L.y_dtype, r);
          }
      }
      __syncthreads();
    } else {
      for (int tok = 0; tok < batch; ++tok) {
        fused_out_block<E8FMT, LATE>(L, b, tok, rstd_s[tok], ws, y_base, fbuf);
        __syncthreads();
      }
    }
  }
}

#ifndef GLQB_FUSED_MINB
#define GLQB_FUSED_MINB 2
#endif
// The layers of a single-launch call travel in kernel-parameter space (constant bank): reading the plan's table
// from global memory would put several dependent L2 round trips at the head of a few-microsecond kernel.
struct FusedLayers {
  DevLinear L[FUSED_MAX_LAYERS];
};

template <int K1, int K2>
__global__ void __launch_bounds__(MV_THREADS, GLQB_FUSED_MINB)
trellis_fused_kernel(const __grid_constant__ FusedLayers T, int n_layers, int total_units, int scratch_elems,
                     const uint8_t* __restrict__ x_base, uint8_t* __restrict__ y_base, uint8_t* __restrict__ ws,
                     int* __restrict__ tickets, const __grid_constant__ CommDev C) {
  extern __shared__ __align__(16) uint8_t fsm[];
  const DevLinear* layers = T.L;
  const DevLinear& L0 = layers[0];
  const int n = L0.n, batch = L0.batch;
  __half2* xs = reinterpret_cast<__half2*>(fsm);                              // [batch][n] (x, 0) pairs, fragment order
  float* fbuf = reinterpret_cast<float*>(fsm + (size_t)batch * n * 4);
  float* red = fbuf + scratch_elems + scratch_elems / 32;                       // [8 warps][8 values][32 lanes]
  __shared__ int todo[FUSED_MAX_TODO];
  __shared__ int n_todo;
  if (threadIdx.x == 0) n_todo = 0;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int gq = lane >> 2, tq = lane & 3;

  // position of work unit u: layer, strip, chunk, this warp's first group and group count
  struct Unit { int li, strip, chunk, c0, ng; };
  auto locate = [&](int u) -> Unit {
    int li = 0;
    while (li + 1 < n_layers && layers[li + 1].group_base <= u) ++li;
    const DevLinear& L = layers[li];
    const int kch = L.fixed_slots;                          // chunks (= partial sums) per strip
    const int local = u - (int)L.group_base;
    const int strip = local / kch, chunk = local - strip * kch;
    const int gpw = L.per_warp;                             // column groups per warp and unit: 2, 4 or 8
    const int c0 = (chunk * MV_WARPS + warp) * gpw;
    return Unit{li, strip, chunk, c0, max(0, min(gpw, L.groups_per_strip - c0))};
  };
  // the stage-1 codes of a unit: all of a warp's (up to eight) groups in flight at once
  auto fetch = [&](const Unit& U, Words<K1> (&w1)[8]) {
    const DevLinear& L = layers[U.li];
    const uint8_t* p1 = L.codes[0] + ((long long)U.strip * L.groups_per_strip + U.c0) * (128 * K1) + lane * (4 * K1);
#pragma unroll
    for (int i = 0; i < 8; ++i)
      if (i < U.ng) w1[i] = load_words<K1>(p1 + i * (128 * K1));
  };

  // The codes do not depend on the activations: request the first unit's before the input transform, so the
  // trip to HBM overlaps it.
  int u = fused_first_unit(blockIdx.x, total_units);
  const int u_end = fused_first_unit(blockIdx.x + 1, total_units);
  Unit U = locate(min(u, total_units - 1));
  Words<K1> w1[8];
  if (u < u_end) fetch(U, w1);
  // Programmatic dependent launch: let the next kernel of the stream start its own prologue, and wait here for
  // the previous kernel (which may have produced x) to finish.  Everything above reads only weights and the
  // plan's table.  Both are no-ops when the launch did not ask for the overlap.
  asm volatile("griddepcontrol.launch_dependents;");
  asm volatile("griddepcontrol.wait;" ::: "memory");
  // tensor-parallel ranks (C.world > 1): the outputs are summed over the ranks inside this kernel (phase 3)
  const int comm_e = C.world > 1 ? comm_epoch(C) : 0;

  // ---- phase 1: the transformed activations of the shared input, in shared memory
  __shared__ float rstd_s[FUSED_MAX_TOKENS];                 // fused RMSNorm: 1 / rms per token, applied to the OUTPUT
  if (threadIdx.x < FUSED_MAX_TOKENS) rstd_s[threadIdx.x] = 1.f;
  fused_phase1<false>(L0, batch, x_base, ws, xs, fbuf, red, rstd_s);
  if (blockIdx.x == 0 && threadIdx.x < batch && L0.in_norm_w && !L0.xr_global)      // for rht_out_kernel (long blocks)
    for (int li = 0; li < n_layers; ++li) reinterpret_cast<float*>(ws + layers[li].rstd_off)[threadIdx.x] = rstd_s[threadIdx.x];

  // ---- phase 2: work units
  const uint32_t xs_addr = (uint32_t)__cvta_generic_to_shared(xs);
  int ticket = -1, done = 0, need = 0, code = 0;              // (thread 0) the output block of the units so far, see below
  while (u < u_end) {
    const DevLinear& L = layers[U.li];
    const int kch = L.fixed_slots, strip = U.strip, chunk = U.chunk, ng = U.ng, c0 = U.c0;
    const int gps = L.groups_per_strip;
    float acc[1][2][4], acc2[1][2][4];
#pragma unroll
    for (int mi = 0; mi < 2; ++mi)
#pragma unroll
      for (int i = 0; i < 4; ++i) { acc[0][mi][i] = 0.f; acc2[0][mi][i] = 0.f; }
    if (ng > 0) {
      Words<(K2 > 0 ? K2 : 1)> w2[8];
      if constexpr (K2 > 0) {
        const uint8_t* p2 = L.codes[1] + ((long long)strip * gps + c0) * (128 * K2) + lane * (4 * K2);
#pragma unroll
        for (int i = 0; i < 8; ++i)
          if (i < ng) w2[i] = load_words<K2>(p2 + i * (128 * K2));
      }
      const int token = min(gq, batch - 1);                 // columns past the batch repeat the last token
      const uint32_t xa = xs_addr + (uint32_t)((((size_t)token * n + (size_t)c0 * 32) * XR_TRELLIS_EXPAND + tq * 16) * 2);
#pragma unroll
      for (int i = 0; i < 8; ++i)
        if (i < ng) {                                       // uniform per warp: the shuffles inside see all lanes
          uint4 xb[1][2];
          xb[0][0] = lds_v4(xa + i * 128);                  // 64 halfs = 128 bytes per group
          xb[0][1] = lds_v4(xa + i * 128 + 16);
          group_mma<K1, 1>(w1[i], lane, xb, acc);
          if constexpr (K2 > 0) group_mma<K2, 1>(w2[i], lane, xb, acc2);
        }
    }
    // next unit of this CTA: its codes travel while this one is reduced
    const int li_now = U.li;
    ++u;
    if (u < u_end) { U = locate(u); fetch(U, w1); }
    {
      const float s2 = L.stage_scale[1];
#pragma unroll
      for (int mi = 0; mi < 2; ++mi)
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          float v = acc[0][mi][i];
          if constexpr (K2 > 0) v = __fadd_rn(v, __fmul_rn(s2, acc2[0][mi][i]));
          red[(warp * 8 + mi * 4 + i) * 32 + lane] = v;
        }
    }
    __syncthreads();
    {
      // thread (f, ln): fragment value f = mi * 4 + i of lane ln, summed over the warps in warp order
      const int f = threadIdx.x >> 5, ln = threadIdx.x & 31;
      float s = 0.f;
#pragma unroll
      for (int w = 0; w < MV_WARPS; ++w) s += red[(w * 8 + f) * 32 + ln];
      const int mi = f >> 2, i = f & 3;
      const int row = strip * 32 + mi * 16 + (ln >> 2) + ((i >> 1) ? 8 : 0);
      const int token = (ln & 3) * 2 + (i & 1);
      if (token < batch) reinterpret_cast<float*>(ws + L.part_off)[((long long)chunk * batch + token) * L.m + row] = s;
    }
    __syncthreads();                                        // the partial sums of the unit are written (and `red` is free)
    if (threadIdx.x == 0) {
      // Which Hadamard block of the output holds this strip, and how many units make it complete.  The units of a CTA follow
      // one another, so it takes a ticket per block that it has worked on, not per unit (an atomic with its fences is a trip
      // to L2 that the first warp's next unit would wait for).
      int b = 0;
      while (b + 1 < L.nbm && strip * 32 >= L.bm_off[b + 1]) ++b;
      // long output blocks are left to rht_out_kernel, launched right behind this kernel: S CTAs share one there
      const int mine = L.bm_log[b] < L.out_split_log || L.stop_at_yrht ? L.ticket_base + b : -1;
      if (mine != ticket) {
        if (ticket >= 0) fused_ticket(tickets, ticket, done, need, code, todo, &n_todo);
        ticket = mine;
        done = 0;
      }
      need = ((1 << L.bm_log[b]) >> 5) * kch;              // (output blocks hold whole strips)
      code = (li_now << 8) | b;
      ++done;
    }
  }
  if (threadIdx.x == 0 && ticket >= 0) fused_ticket(tickets, ticket, done, need, code, todo, &n_todo);
  __syncthreads();

  // ---- phase 3: output transforms of the blocks this CTA completed
  fused_phase3<false, 32>(layers, todo, n_todo, batch, rstd_s, ws, y_base, fbuf, scratch_elems, C, comm_e);
  if (C.world > 1) comm_cta_done(C, comm_e);
}

// ---------------------------------------------------------------------------------------------
// Single-launch decode linear for E8-shell layers (at most 8 tokens, up to FUSED_MAX_LAYERS layers that read the
// same input): the same three phases as trellis_fused_kernel with the E8 streaming arithmetic in the middle.
// A work unit is (layer, 16-row strip, chunk of 8 warps x `per_warp` column groups of 256 columns); a lane (g, t)
// holds 8 consecutive indices of rows g and g + 8 per group and stage, gathers their packed table entries from
// global memory (L1 / L2: these launches are far too small to pay for a resident table), expands them with
// e8_entry_to_half2 and multiplies against the activations kept in shared memory in the order of xr_index_e8.
// Residual stages keep separate accumulators and are combined with fp32 multiply and add when the unit ends, as
// in e8_mv_body.  Replaces the three launches (input transform, matvec, output transform) of the reference's E8
// decode path (glq/csrc/glq_cuda.cu:2533, 3038) by one.
// ---------------------------------------------------------------------------------------------
constexpr int E8F_MAX_GPW = 4;                  // column groups per warp and unit (index registers: 8 per group)

// RES: the first `res_entries` entries of the 65,536-entry table (and a small second-stage table) are copied into
// shared memory at the start of the kernel — before the wait for the previous kernel, so the copy overlaps its tail
// — and one CTA runs per SM.  Used for launches of a few MB and more, where every SM would otherwise pull most of
// the table through L2 one 32-byte sector per gather (the launch's shared memory leaves too little L1 to hold it).
template <int NS, bool RES>
__global__ void __launch_bounds__(MV_THREADS, RES ? 1 : GLQB_FUSED_MINB)
e8_fused_kernel(const __grid_constant__ FusedLayers T, int n_layers, int total_units, int scratch_elems,
                const uint8_t* __restrict__ x_base, uint8_t* __restrict__ y_base, uint8_t* __restrict__ ws,
                int* __restrict__ tickets, const __grid_constant__ CommDev C, const uint32_t* __restrict__ big_table,
                int res_entries, const uint32_t* __restrict__ small_table, int small_entries) {
  extern __shared__ __align__(16) uint8_t fsm_all[];
  uint8_t* fsm = fsm_all + (RES ? (size_t)res_entries * 4 + 1024 : 0);
  const uint32_t table_smem = (uint32_t)__cvta_generic_to_shared(fsm_all);
  const uint32_t small_smem = table_smem + (uint32_t)res_entries * 4u;
  if constexpr (RES) {
    const uint4* src = reinterpret_cast<const uint4*>(big_table);
    uint4* dst = reinterpret_cast<uint4*>(fsm_all);
    for (int i = threadIdx.x; i < res_entries / 4; i += blockDim.x) dst[i] = __ldg(src + i);
    uint32_t* sm = reinterpret_cast<uint32_t*>(fsm_all + (size_t)res_entries * 4);
    for (int i = threadIdx.x; i < small_entries && i < 256; i += blockDim.x) sm[i] = __ldg(small_table + i);
  }
  const DevLinear* layers = T.L;
  const DevLinear& L0 = layers[0];
  const int n = L0.n, batch = L0.batch;
  __half2* xs = reinterpret_cast<__half2*>(fsm);
  float* fbuf = reinterpret_cast<float*>(fsm + ((fused_xs_bytes<true>(n, batch) + 15) & ~(size_t)15));
  float* red = fbuf + scratch_elems + scratch_elems / 32;                       // [8 warps][4 values][32 lanes]
  __shared__ int todo[FUSED_MAX_TODO];
  __shared__ int n_todo;
  if (threadIdx.x == 0) n_todo = 0;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int gq = lane >> 2, tq = lane & 3;

  struct Unit { int li, strip, chunk, c0, ng; };
  auto locate = [&](int u) -> Unit {
    int li = 0;
    while (li + 1 < n_layers && layers[li + 1].group_base <= u) ++li;
    const DevLinear& L = layers[li];
    const int kch = L.fixed_slots;
    const int local = u - (int)L.group_base;
    const int strip = local / kch, chunk = local - strip * kch;
    const int gpw = L.per_warp;
    const int c0 = (chunk * MV_WARPS + warp) * gpw;
    return Unit{li, strip, chunk, c0, max(0, min(gpw, L.groups_per_strip - c0))};
  };
  // the indices of one stage of a unit: per group 8 of row g (qa) and 8 of row g + 8 (qb), 16 bytes each
  auto fetch = [&](const Unit& U, int stage, uint4 (&qa)[E8F_MAX_GPW], uint4 (&qb)[E8F_MAX_GPW]) {
    const DevLinear& L = layers[U.li];
    const int nidx = L.n >> 3;
    const uint16_t* q = reinterpret_cast<const uint16_t*>(L.codes[stage]);
    const int rowA = U.strip * 16 + gq, rowB = rowA + 8;
    const bool vec_ok = (nidx & 7) == 0 && (reinterpret_cast<uintptr_t>(q) & 15) == 0;
#pragma unroll
    for (int i = 0; i < E8F_MAX_GPW; ++i) {
      qa[i] = make_uint4(0u, 0u, 0u, 0u);
      qb[i] = make_uint4(0u, 0u, 0u, 0u);
      if (i < U.ng) {
        const int i0 = (U.c0 + i) * 32 + tq * 8;
        const uint16_t* pa = q + (long long)rowA * nidx + i0;
        const uint16_t* pb = q + (long long)rowB * nidx + i0;
        if (vec_ok && i0 + 8 <= nidx) {
          if (rowA < L.m) qa[i] = ld_stream_v4(pa);
          if (rowB < L.m) qb[i] = ld_stream_v4(pb);
        } else {
          uint32_t wa[4] = {0u, 0u, 0u, 0u}, wb[4] = {0u, 0u, 0u, 0u};
#pragma unroll
          for (int k = 0; k < 8; ++k)
            if (i0 + k < nidx) {
              if (rowA < L.m) wa[k >> 1] |= (uint32_t)pa[k] << ((k & 1) * 16);
              if (rowB < L.m) wb[k >> 1] |= (uint32_t)pb[k] << ((k & 1) * 16);
            }
          qa[i] = make_uint4(wa[0], wa[1], wa[2], wa[3]);
          qb[i] = make_uint4(wb[0], wb[1], wb[2], wb[3]);
        }
      }
    }
  };

  // The indices do not depend on the activations: request the first unit's before the input transform.
  int u = fused_first_unit(blockIdx.x, total_units);
  const int u_end = fused_first_unit(blockIdx.x + 1, total_units);
  Unit U = locate(min(u, total_units - 1));
  uint4 qa0[E8F_MAX_GPW], qb0[E8F_MAX_GPW];
  if (u < u_end) fetch(U, 0, qa0, qb0);
  asm volatile("griddepcontrol.launch_dependents;");
  asm volatile("griddepcontrol.wait;" ::: "memory");
  const int comm_e = C.world > 1 ? comm_epoch(C) : 0;

  // ---- phase 1: the transformed activations of the shared input, in shared memory
  __shared__ float rstd_s[FUSED_MAX_TOKENS];
  if (threadIdx.x < FUSED_MAX_TOKENS) rstd_s[threadIdx.x] = 1.f;
  fused_phase1<true>(L0, batch, x_base, ws, xs, fbuf, red, rstd_s);
  if (blockIdx.x == 0 && threadIdx.x < batch && L0.in_norm_w && !L0.xr_global)
    for (int li = 0; li < n_layers; ++li) reinterpret_cast<float*>(ws + layers[li].rstd_off)[threadIdx.x] = rstd_s[threadIdx.x];

  // ---- phase 2: work units
  const uint32_t xs_addr = (uint32_t)__cvta_generic_to_shared(xs);
  const int nidx = n >> 3;
  // B fragments of one index (8-column block) for this lane's token: 16 bytes at block * xstep
  const int token = min(gq, batch - 1);                     // columns past the batch repeat the last token
  const uint32_t xa = xs_addr + (uint32_t)(batch == 1 ? 0 : (token & 7) * 16);
  const uint32_t xstep = batch == 1 ? 16u : 128u;
  int ticket = -1, done = 0, need = 0, code = 0;              // (thread 0) the output block of the units so far, see below
  while (u < u_end) {
    const DevLinear& L = layers[U.li];
    const int kch = L.fixed_slots, strip = U.strip, chunk = U.chunk, ng = U.ng, c0 = U.c0;
    float acc[NS][4];
#pragma unroll
    for (int st = 0; st < NS; ++st)
#pragma unroll
      for (int i = 0; i < 4; ++i) acc[st][i] = 0.f;
    if (ng > 0) {
#pragma unroll
      for (int st = 0; st < NS; ++st) {
        uint4 qa[E8F_MAX_GPW], qb[E8F_MAX_GPW];
        if (st > 0) fetch(U, st, qa, qb);
        const uint32_t* table = L.table[st];
        const uint32_t mask = (uint32_t)L.table_entries[st] - 1u;
        // resident form: big-table entries below res_entries and every small-table entry come from shared memory
        const bool is_big = L.table_entries[st] == 65536;
        const uint32_t sbase = is_big ? table_smem : small_smem;
        const uint32_t slimit = is_big ? (uint32_t)res_entries : 256u;
        auto gather = [&](uint32_t idx) -> uint32_t {
          if constexpr (RES) {
            uint32_t v;
            asm volatile("{\n\t.reg .pred p;\n\t"
                         "setp.ge.u32 p, %1, %2;\n\t"
                         "@!p ld.shared.u32 %0, [%3];\n\t"
                         "@p ld.global.nc.u32 %0, [%4];\n\t}"
                         : "=r"(v)
                         : "r"(idx), "r"(slimit), "r"(sbase + (idx << 2)), "l"(table + idx));
            return v;
          } else {
            return __ldg(table + idx);
          }
        };
#pragma unroll
        for (int i = 0; i < E8F_MAX_GPW; ++i) {
          if (i < ng) {
            const uint4 a4 = st == 0 ? qa0[i] : qa[i], b4 = st == 0 ? qb0[i] : qb[i];
            const uint32_t wa[4] = {a4.x, a4.y, a4.z, a4.w}, wb[4] = {b4.x, b4.y, b4.z, b4.w};
            uint32_t ea[8], eb[8];
#pragma unroll
            for (int k = 0; k < 8; ++k) {                   // all sixteen gathers of the group in flight
              ea[k] = gather((wa[k >> 1] >> ((k & 1) * 16)) & mask);
              eb[k] = gather((wb[k >> 1] >> ((k & 1) * 16)) & mask);
            }
            const int i0 = (c0 + i) * 32 + tq * 8;
#pragma unroll
            for (int k = 0; k < 8; ++k) {
              const int blk = min(i0 + k, nidx - 1);
              uint4 xb = lds_v4(xa + (uint32_t)blk * xstep);
              if (i0 + k >= nidx) xb = make_uint4(0u, 0u, 0u, 0u);     // past the row end: contributes nothing
              uint32_t ha[4], hb[4];
              e8_entry_to_half2(ea[k], ha);
              e8_entry_to_half2(eb[k], hb);
              const uint32_t a1[4] = {ha[0], hb[0], ha[1], hb[1]};
              const uint32_t a2[4] = {ha[2], hb[2], ha[3], hb[3]};
              mma16816(acc[st], a1, xb.x, xb.y);
              mma16816(acc[st], a2, xb.z, xb.w);
            }
          }
        }
      }
    }
    // next unit of this CTA: its first-stage indices travel while this one is reduced
    const int li_now = U.li;
    ++u;
    if (u < u_end) { U = locate(u); fetch(U, 0, qa0, qb0); }
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      float v = acc[0][i];
#pragma unroll
      for (int st = 1; st < NS; ++st) v = __fadd_rn(v, __fmul_rn(L.stage_scale[st], acc[st][i]));
      red[(warp * 4 + i) * 32 + lane] = v;
    }
    __syncthreads();
    if (threadIdx.x < 128) {
      // thread (f, ln): fragment value f of lane ln, summed over the warps in warp order
      const int f = threadIdx.x >> 5, ln = threadIdx.x & 31;
      float sum = 0.f;
#pragma unroll
      for (int w = 0; w < MV_WARPS; ++w) sum += red[(w * 4 + f) * 32 + ln];
      const int row = strip * 16 + (ln >> 2) + ((f >> 1) ? 8 : 0);
      const int tk = (ln & 3) * 2 + (f & 1);
      if (tk < batch && row < L.m) reinterpret_cast<float*>(ws + L.part_off)[((long long)chunk * batch + tk) * L.m + row] = sum;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
      // Which Hadamard block of the output holds this strip, and how many units make it complete.  The units of a CTA follow
      // one another, so it takes a ticket per block that it has worked on, not per unit (an atomic with its fences is a trip
      // to L2 that the first warp's next unit would wait for).
      int b = 0;
      while (b + 1 < L.nbm && strip * 16 >= L.bm_off[b + 1]) ++b;
      // long output blocks are left to rht_out_kernel, launched right behind this kernel: S CTAs share one there
      const int mine = L.bm_log[b] < L.out_split_log || L.stop_at_yrht ? L.ticket_base + b : -1;
      if (mine != ticket) {
        if (ticket >= 0) fused_ticket(tickets, ticket, done, need, code, todo, &n_todo);
        ticket = mine;
        done = 0;
      }
      need = ((1 << L.bm_log[b]) >> 4) * kch;              // (output blocks hold whole strips)
      code = (li_now << 8) | b;
      ++done;
    }
  }
  if (threadIdx.x == 0 && ticket >= 0) fused_ticket(tickets, ticket, done, need, code, todo, &n_todo);
  __syncthreads();

  // ---- phase 3: output transforms of the blocks this CTA completed
  fused_phase3<true, RES ? 64 : 16>(layers, todo, n_todo, batch, rstd_s, ws, y_base, fbuf, scratch_elems, C, comm_e);
  if (C.world > 1) comm_cta_done(C, comm_e);
}

}  // namespace glqb
