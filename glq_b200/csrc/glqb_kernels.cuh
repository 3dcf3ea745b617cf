// Kernels of the decode (small-batch) path: streaming decode + mma, and the dump kernels used by the bit-exact gate.
#pragma once
#include "glqb_internal.h"
#include "glqb_decode.cuh"
#include "glqb_comm.cuh"

namespace glqb {

#ifndef GLQB_LUT_THREADS
#define GLQB_LUT_THREADS 768
#endif
constexpr int MV_THREADS = 256;               // 8 warps per CTA in the streaming kernels
constexpr int MV_WARPS = MV_THREADS / 32;

// ---------------------------------------------------------------------------------------------
// small helpers
// ---------------------------------------------------------------------------------------------
__device__ __forceinline__ float load_act(const void* base, long long idx, int dtype) {
  if (dtype == GLQB_DT_F16) return __half2float(reinterpret_cast<const __half*>(base)[idx]);
  if (dtype == GLQB_DT_BF16) return __bfloat162float(reinterpret_cast<const __nv_bfloat16*>(base)[idx]);
  return reinterpret_cast<const float*>(base)[idx];
}

__device__ __forceinline__ void store_act(void* base, long long idx, int dtype, float v) {
  if (dtype == GLQB_DT_F16) reinterpret_cast<__half*>(base)[idx] = __float2half_rn(v);
  else if (dtype == GLQB_DT_BF16) reinterpret_cast<__nv_bfloat16*>(base)[idx] = __float2bfloat16_rn(v);
  else reinterpret_cast<float*>(base)[idx] = v;
}

// four consecutive activations; idx must be a multiple of 4 and the row 8/16-byte aligned (the callers
// check) — one 8- or 16-byte access instead of four
__device__ __forceinline__ void load_act4(const void* base, long long idx, int dtype, float (&v)[4]) {
  if (dtype == GLQB_DT_F32) {
    const float4 t = *reinterpret_cast<const float4*>(reinterpret_cast<const float*>(base) + idx);
    v[0] = t.x; v[1] = t.y; v[2] = t.z; v[3] = t.w;
  } else {
    const uint2 t = *reinterpret_cast<const uint2*>(reinterpret_cast<const uint16_t*>(base) + idx);
    if (dtype == GLQB_DT_F16) {
      const float2 a = __half22float2(*reinterpret_cast<const __half2*>(&t.x));
      const float2 b = __half22float2(*reinterpret_cast<const __half2*>(&t.y));
      v[0] = a.x; v[1] = a.y; v[2] = b.x; v[3] = b.y;
    } else {
      v[0] = __uint_as_float(t.x << 16); v[1] = __uint_as_float(t.x & 0xFFFF0000u);
      v[2] = __uint_as_float(t.y << 16); v[3] = __uint_as_float(t.y & 0xFFFF0000u);
    }
  }
}
__device__ __forceinline__ void store_act4(void* base, long long idx, int dtype, const float (&v)[4]) {
  if (dtype == GLQB_DT_F32) {
    *reinterpret_cast<float4*>(reinterpret_cast<float*>(base) + idx) = make_float4(v[0], v[1], v[2], v[3]);
  } else if (dtype == GLQB_DT_F16) {
    const __half2 a = __floats2half2_rn(v[0], v[1]), b = __floats2half2_rn(v[2], v[3]);
    *reinterpret_cast<uint2*>(reinterpret_cast<uint16_t*>(base) + idx) =
        make_uint2(*reinterpret_cast<const uint32_t*>(&a), *reinterpret_cast<const uint32_t*>(&b));
  } else {
    const __nv_bfloat162 a = __floats2bfloat162_rn(v[0], v[1]), b = __floats2bfloat162_rn(v[2], v[3]);
    *reinterpret_cast<uint2*>(reinterpret_cast<uint16_t*>(base) + idx) =
        make_uint2(*reinterpret_cast<const uint32_t*>(&a), *reinterpret_cast<const uint32_t*>(&b));
  }
}
// calls f(integral constant) for the dtype code, so that loops over a thread's values carry no branch on it
template <int V> struct IntC { static constexpr int value = V; };
template <class F>
__device__ __forceinline__ void with_dtype(int dtype, F f) {
  if (dtype == GLQB_DT_F32) f(IntC<GLQB_DT_F32>());
  else if (dtype == GLQB_DT_BF16) f(IntC<GLQB_DT_BF16>());
  else f(IntC<GLQB_DT_F16>());
}
__device__ __forceinline__ bool act_rows_aligned4(const void* base, long long off, long long stride, int dtype) {
  const int es = dtype == GLQB_DT_F32 ? 4 : 2;
  return ((off | stride) & 3) == 0 && (reinterpret_cast<uintptr_t>(base) & (4 * es - 1)) == 0;
}

// value after a round trip through the activation dtype (what a separate kernel would have stored)
__device__ __forceinline__ float round_act(float v, int dtype) {
  if (dtype == GLQB_DT_F16) return __half2float(__float2half_rn(v));
  if (dtype == GLQB_DT_BF16) return __bfloat162float(__float2bfloat16_rn(v));
  return v;
}
// gated / plain activations of the MoE ops and of the fused decode input (GLQB_ACT_*)
__device__ __forceinline__ float act_fn(float g, int act) {
  if (act == GLQB_ACT_SILU) return g / (1.0f + __expf(-g));
  if (act == GLQB_ACT_GELU_TANH) {
    const float u = 0.7978845608028654f * (g + 0.044715f * g * g * g);
    return 0.5f * g * (1.0f + tanhf(u));
  }
  const float r = fmaxf(g, 0.f);
  return r * r;
}

// streaming 128/64/32-bit loads of weight codes: read once, keep out of L1
__device__ __forceinline__ uint4 ld_stream_v4(const void* p) {
  uint4 v;
  asm volatile("ld.global.nc.L1::no_allocate.v4.u32 {%0,%1,%2,%3}, [%4];"
               : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p));
  return v;
}
__device__ __forceinline__ uint2 ld_stream_v2(const void* p) {
  uint2 v;
  asm volatile("ld.global.nc.L1::no_allocate.v2.u32 {%0,%1}, [%2];" : "=r"(v.x), "=r"(v.y) : "l"(p));
  return v;
}
__device__ __forceinline__ uint32_t ld_stream_u32(const void* p) {
  uint32_t v;
  asm volatile("ld.global.nc.L1::no_allocate.u32 %0, [%1];" : "=r"(v) : "l"(p));
  return v;
}

// D(16x8, f32) += A(16x16, f16, row) * B(16x8, f16, col)
__device__ __forceinline__ void mma16816(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
      : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

// Trellis activations are stored per 32-column group as 64 halfs: column c = 16ni + 8h + 2t + e sits at
// half index t*16 + ni*8 + e*4 + h*2 and is followed by a zero, i.e. every B-fragment register of
// the MMA is (x, 0).  Lane t fetches its 32 bytes of a group with two 16-byte loads (one per ni).
constexpr int XR_TRELLIS_EXPAND = 2;   // halfs stored per activation
__device__ __forceinline__ int xr_pos_trellis(int c) {
  int ni = c >> 4, h = (c >> 3) & 1, t = (c >> 1) & 3, e = c & 1;
  return t * 16 + ni * 8 + e * 4 + h * 2;
}
// position of column i (0..7) of an E8 block: (x0,x4,x1,x5,x2,x6,x3,x7)
__device__ __forceinline__ int xr_pos_e8(int i) { return (i & 3) * 2 + (i >> 2); }
// E8 activations for the streaming kernel.  One token: 8-column blocks in order.  Several tokens: the
// blocks of 8 consecutive tokens are interleaved (token group, block, token in group, 8 halfs), so that
// the 8 tokens a warp multiplies against one block sit in one 128-byte line instead of eight.
__device__ __forceinline__ long long xr_index_e8(long long token, int col, int n, int batch) {
  const int j = xr_pos_e8(col & 7);
  if (batch == 1) return (col & ~7) + j;
  return ((((token >> 3) * (n >> 3) + (col >> 3)) << 3) + (token & 7)) * 8 + j;
}

constexpr int FUSED_MAX_TOKENS_C = 8;     // tokens served by the single-launch decode form and its fused steps

// Input value of column `col` of token row starting at element `xt0`, before the sign vector: x itself, or
// act(gate) * up for a [gate | up] row (both factors and the product rounded to the activation dtype, as
// separate kernels would store them).
__device__ __forceinline__ float input_value(const DevLinear& L, const uint8_t* x_base, long long xt0, int col) {
  float v = load_act(x_base, xt0 + col, L.x_dtype);
  if (L.in_gated_act)
    v = round_act(round_act(act_fn(v, L.in_gated_act - 1), L.x_dtype) * load_act(x_base, xt0 + L.in_f + col, L.x_dtype), L.x_dtype);
  return v;
}
// ---------------------------------------------------------------------------------------------
// Trellis 3INST streaming decode + mma (batch <= 8*NB tokens ride the MMA columns).
//
// Work is the flattened list of 32x32 groups of every layer of the launch; warp w owns the
// contiguous range [w*per_warp, (w+1)*per_warp).  Inside a strip of 32 rows the warp accumulates in
// registers; at a strip boundary (or the end of its range) it writes one partial sum per
// (token, row) to slot (w - first warp touching the strip).  No atomics: the output transform adds
// the slots in ascending order, so results do not depend on scheduling.
//
// Per group and lane: one 4K-byte load of codes, K shuffles to fetch the next lane's chunks (the
// 16 bits that follow a lane's chunk in the tile's cyclic stream), one 16-byte load of rotated
// activations per 8 tokens, 32 state decodes, 4 MMAs per 8 tokens (two with a second stage).
// ---------------------------------------------------------------------------------------------
template <int K>
__device__ __forceinline__ Words<K> load_words(const uint8_t* p) {
  Words<K> v;
  if constexpr (K == 4) {
    uint4 t = ld_stream_v4(p); v.w[0] = t.x; v.w[1] = t.y; v.w[2] = t.z; v.w[3] = t.w;
  } else if constexpr (K == 2) {
    uint2 t = ld_stream_v2(p); v.w[0] = t.x; v.w[1] = t.y;
  } else if constexpr (K == 1) {
    v.w[0] = ld_stream_u32(p);
  } else {
    v.w[0] = ld_stream_u32(p); v.w[1] = ld_stream_u32(p + 4); v.w[2] = ld_stream_u32(p + 8);
  }
  return v;
}

template <int K>
__device__ __forceinline__ Words<K> shfl_words(const Words<K>& v, int src) {
  Words<K> r;
#pragma unroll
  for (int i = 0; i < K; ++i) r.w[i] = __shfl_sync(0xffffffffu, v.w[i], src);
  return r;
}

// decode the four tiles of a group and issue their MMAs against the B fragments xb[nb][ni]
// (xb[nb][ni] = {e0:(x,0) k-lo, e0 k-hi, e1 k-lo, e1 k-hi})
template <int K, int NB, int LUT = 0>
__device__ __forceinline__ void group_mma(const Words<K>& v, int lane, const uint4 (&xb)[NB][2],
                                          float (&acc)[NB][2][4], uint32_t lut_base = 0u) {
  const Words<K> vn = shfl_words<K>(v, (lane + 1) & 31);
  Words<K> vn2 = vn;
  if constexpr (K == 1) vn2 = shfl_words<K>(v, (lane + 2) & 31);
#pragma unroll
  for (int ni = 0; ni < 2; ++ni) {
#pragma unroll
    for (int mi = 0; mi < 2; ++mi) {
      const int q = ni * 2 + mi;
      uint32_t a[8];
      decode_tile<K, LUT>(chunk_of<K>(v, q), chunk_of<K>(vn, q), chunk_of<K>(vn2, q), a, lut_base);
      const uint32_t a_even[4] = {a[0], a[2], a[4], a[6]};   // columns 2t   / 8+2t   of the tile
      const uint32_t a_odd[4] = {a[1], a[3], a[5], a[7]};    // columns 2t+1 / 8+2t+1
#pragma unroll
      for (int nb = 0; nb < NB; ++nb) {
        mma16816(acc[nb][mi], a_even, xb[nb][ni].x, xb[nb][ni].y);
        mma16816(acc[nb][mi], a_odd, xb[nb][ni].z, xb[nb][ni].w);
      }
    }
  }
}

#ifndef GLQB_MINB
#define GLQB_MINB 3
#endif
// LUT > 0: the table form for large launches — one CTA of MV_LUT_THREADS per SM next to the 128 KiB table of the
// code's 65,536 fp16 values, which the CTA fills with the arithmetic decode when it starts (see decode_tile).
constexpr int MV_LUT_STATES = 2;
constexpr int MV_LUT_THREADS = GLQB_LUT_THREADS;
constexpr int MV_LUT_SMEM_BYTES = 65536 * 2;
template <int K1, int K2, int NB, int LUT = 0>
__global__ void __launch_bounds__(LUT ? MV_LUT_THREADS : MV_THREADS, LUT ? 1 : ((NB == 1 && K2 == 0) ? GLQB_MINB : 1))
trellis_mv_kernel(const DevLinear* __restrict__ layers, int n_layers, long long total_groups,
                  int per_warp, uint8_t* __restrict__ ws, int tokens) {
  uint32_t lut_base = 0u;
  if constexpr (LUT > 0) {
    extern __shared__ __align__(16) unsigned short lut3[];
    for (int st = threadIdx.x; st < 65536; st += blockDim.x) lut3[st] = (unsigned short)(sum_dup3(hash3((uint32_t)st)) & 0xFFFFu);
    __syncthreads();
    lut_base = (uint32_t)__cvta_generic_to_shared(lut3);
  }
#ifndef GLQB_PF
#define GLQB_PF 4
#endif
  constexpr int PF = GLQB_PF;   // codes of PF groups in flight per lane
  const int lane = threadIdx.x & 31;
  const long long w = (long long)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  long long g = w * per_warp;
  const long long gend = min(g + per_warp, total_groups);
  if (g >= gend) return;
  // locate the layer holding group g (layers are sorted by group_base)
  int lo = 0, hi = n_layers - 1;
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (layers[mid].group_base <= g) lo = mid; else hi = mid - 1;
  }
  int li = lo;
  const int gq = lane >> 2, tq = lane & 3;

  while (g < gend) {
    const DevLinear& L = layers[li];
    const long long local = g - L.group_base;
    const int gps = L.groups_per_strip;
    const int strip = (int)(local / gps);
    const int c0 = (int)(local - (long long)strip * gps);
    const int c1 = (int)min((long long)gps, c0 + (gend - g));
    const int batch = L.batch, used = min(batch, tokens);    // rows of the buffers; rows of this run

    float acc[NB][2][4];
    float acc2[K2 ? NB : 1][2][4];
#pragma unroll
    for (int nb = 0; nb < NB; ++nb)
#pragma unroll
      for (int mi = 0; mi < 2; ++mi)
#pragma unroll
        for (int i = 0; i < 4; ++i) { acc[nb][mi][i] = 0.f; if constexpr (K2 > 0) acc2[nb][mi][i] = 0.f; }

    const uint8_t* p1 = L.codes[0] + ((long long)strip * gps + c0) * (128 * K1) + lane * (4 * K1);
    const uint8_t* p2 = nullptr;
    if constexpr (K2 > 0) p2 = L.codes[1] + ((long long)strip * gps + c0) * (128 * K2) + lane * (4 * K2);
    const __half* xr = reinterpret_cast<const __half*>(ws + L.xr_off);
    // MMA column gq of block nb carries token 8*nb + gq.  Columns past the tokens of the run read the last
    // token again: their products land in accumulator columns that are never stored, which saves the
    // predicate and the zero fill on every group.
    const uint4* xq[NB];
#pragma unroll
    for (int nb = 0; nb < NB; ++nb) {
      const int token = min(nb * 8 + gq, used - 1);
      xq[nb] = reinterpret_cast<const uint4*>(xr + ((long long)token * L.n + c0 * 32) * XR_TRELLIS_EXPAND + tq * 16);
    }

    const int ng = c1 - c0;
    // One group step: codes of this group are in v/v2; the codes of the group PF ahead are requested
    // before the decode starts so that PF groups per lane are always in flight.
    Words<K1> cur[PF];
    Words<(K2 > 0 ? K2 : 1)> cur2[PF];
#pragma unroll
    for (int i = 0; i < PF; ++i) {
      if (i < ng) {
        cur[i] = load_words<K1>(p1 + i * (128 * K1));
        if constexpr (K2 > 0) cur2[i] = load_words<K2>(p2 + i * (128 * K2));
      }
    }
    const uint8_t* q1 = p1 + PF * (128 * K1);     // next codes to request
    const uint8_t* q2 = p2 + PF * (128 * K2);
    int c = 0;
    // full chunks with every prefetch in range: no per-group bounds checks
    for (; c + 2 * PF <= ng; c += PF) {
#pragma unroll
      for (int i = 0; i < PF; ++i) {
        const Words<K1> v = cur[i];
        Words<(K2 > 0 ? K2 : 1)> v2;
        if constexpr (K2 > 0) v2 = cur2[i];
        cur[i] = load_words<K1>(q1 + i * (128 * K1));
        if constexpr (K2 > 0) cur2[i] = load_words<K2>(q2 + i * (128 * K2));
        uint4 xb[NB][2];
#pragma unroll
        for (int nb = 0; nb < NB; ++nb) {
          xb[nb][0] = __ldg(xq[nb] + i * 8);               // 64 halfs = 8 uint4 per group
          xb[nb][1] = __ldg(xq[nb] + i * 8 + 1);
        }
        group_mma<K1, NB, LUT>(v, lane, xb, acc, lut_base);
        if constexpr (K2 > 0) group_mma<K2, NB, LUT>(v2, lane, xb, acc2, lut_base);
      }
      q1 += PF * (128 * K1);
      q2 += PF * (128 * K2);
#pragma unroll
      for (int nb = 0; nb < NB; ++nb) xq[nb] += PF * 8;
    }
    // tail: up to 2*PF - 1 groups, bounds checked
    for (; c < ng; c += PF) {
#pragma unroll
      for (int i = 0; i < PF; ++i) {
        if (c + i < ng) {
          const Words<K1> v = cur[i];
          Words<(K2 > 0 ? K2 : 1)> v2;
          if constexpr (K2 > 0) v2 = cur2[i];
          if (c + i + PF < ng) {
            cur[i] = load_words<K1>(q1 + i * (128 * K1));
            if constexpr (K2 > 0) cur2[i] = load_words<K2>(q2 + i * (128 * K2));
          }
          uint4 xb[NB][2];
#pragma unroll
          for (int nb = 0; nb < NB; ++nb) {
            xb[nb][0] = __ldg(xq[nb] + i * 8);
            xb[nb][1] = __ldg(xq[nb] + i * 8 + 1);
          }
          group_mma<K1, NB, LUT>(v, lane, xb, acc, lut_base);
          if constexpr (K2 > 0) group_mma<K2, NB, LUT>(v2, lane, xb, acc2, lut_base);
        }
      }
      q1 += PF * (128 * K1);
      q2 += PF * (128 * K2);
#pragma unroll
      for (int nb = 0; nb < NB; ++nb) xq[nb] += PF * 8;
    }

    // flush: C fragment (row gq / gq+8, tokens 2tq, 2tq+1 of each column block)
    {
      const long long g0 = L.group_base + (long long)strip * gps;
      const int slot = (int)(w - g0 / per_warp);
      float* part = reinterpret_cast<float*>(ws + L.part_off) + (long long)slot * batch * L.m;
      const float s2 = L.stage_scale[1];
#pragma unroll
      for (int nb = 0; nb < NB; ++nb) {
#pragma unroll
        for (int mi = 0; mi < 2; ++mi) {
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            const int token = nb * 8 + tq * 2 + (i & 1);
            const int row = strip * 32 + mi * 16 + gq + ((i >> 1) ? 8 : 0);
            if (token < used) {
              float v = acc[nb][mi][i];
              if constexpr (K2 > 0) v = __fadd_rn(v, __fmul_rn(s2, acc2[nb][mi][i]));
              part[(long long)token * L.m + row] = v;
            }
          }
        }
      }
    }
    g += ng;
    if (c1 == gps && strip == L.strips - 1) ++li;
  }
}

// ---------------------------------------------------------------------------------------------
// E8 shell streaming gather + mma.
//
// Work group = 16 rows x 256 columns (32 indices per row).  Lane (g, t) loads 8 consecutive indices
// of row g and of row g+8 (columns 256*G + 64*t ...), gathers their nibble-packed codebook entries,
// expands each to 8 exact fp16 values and feeds two MMAs per index pair.  The MMA's k index is a
// dummy summation index, so a lane's 8 weights of one index may sit in any k slots as long as the
// activations are permuted the same way: the rotated activations are stored per 8-column block in
// the order (x0,x4,x1,x5,x2,x6,x3,x7), which lets a lane fetch the B fragments of both MMAs with
// one 16-byte load.  Every residual stage has its own accumulator (all stage values are exact in
// fp16); stages are combined in fp32 when a strip is flushed.
// ---------------------------------------------------------------------------------------------
// Where the codebook entries come from.  TM = 0: the packed tables stay in global memory (L1/L2
// gathers).  TM = 1: the first E8S_RESIDENT entries of the 65,536-entry table live in the CTA's shared
// memory (one CTA per SM) and are fetched with plain shared loads, bank conflicts and all; the few
// indices past the resident part still go to global memory.  Tables of up to 256 entries (the small
// second-stage codebook) are fully resident.
constexpr int E8S_RESIDENT = 56 * 1024;
struct E8Tables {
  uint32_t table_base;     // shared-window address of the resident part of the big table
  uint32_t small_base;     // shared-window address of the small table
};

// One stage's gather parameters, fixed per layer.
struct E8Stage {
  const uint32_t* table;   // global table
  uint32_t mask;           // entries - 1
  uint32_t base;           // TM = 1: shared-window address of the resident copy this stage indexes
};

// The gathers are volatile so that they keep their place ahead of the (volatile) MMAs of the chunk being
// consumed: that ordering is what keeps a whole chunk of gathers in flight.
template <int TM, int RESIDENT = E8S_RESIDENT>
__device__ __forceinline__ uint32_t e8_gather(const E8Stage& S, uint32_t idx) {
  uint32_t v;
  const uint32_t* gp = S.table + idx;
  if constexpr (TM == 0) {
    asm volatile("ld.global.nc.u32 %0, [%1];" : "=r"(v) : "l"(gp));
  } else {
    // branch-free: lanes whose index is resident read shared memory, the others global memory
    asm volatile("{\n\t.reg .pred p;\n\t"
                 "setp.ge.u32 p, %1, %2;\n\t"
                 "@!p ld.shared.u32 %0, [%3];\n\t"
                 "@p ld.global.nc.u32 %0, [%4];\n\t}"
                 : "=r"(v)
                 : "r"(idx), "r"((uint32_t)RESIDENT), "r"(S.base + (idx << 2)), "l"(gp));
  }
  return v;
}

#ifndef GLQB_E8_KC
#define GLQB_E8_KC 8
#endif
#ifndef GLQB_E8_MINB
#define GLQB_E8_MINB 2
#endif
template <int NS, int NB, int TM>
__device__ __forceinline__ void e8_mv_body(const DevLinear* __restrict__ layers, int n_layers, long long total_groups,
                                           int per_warp, uint8_t* __restrict__ ws, const E8Tables& T,
                                           int warps_per_cta, int tokens) {
  const int lane = threadIdx.x & 31;
  const long long w = (long long)blockIdx.x * warps_per_cta + (threadIdx.x >> 5);
  long long g = w * per_warp;
  const long long gend = min(g + per_warp, total_groups);
  if (g >= gend) return;
  int lo = 0, hi = n_layers - 1;
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (layers[mid].group_base <= g) lo = mid; else hi = mid - 1;
  }
  int li = lo;
  const int gq = lane >> 2, tq = lane & 3;

  while (g < gend) {
    const DevLinear& L = layers[li];
    const long long local = g - L.group_base;
    const int gps = L.groups_per_strip;
    const int strip = (int)(local / gps);
    const int c0 = (int)(local - (long long)strip * gps);
    const int c1 = (int)min((long long)gps, c0 + (gend - g));
    const int batch = L.batch, used = min(batch, tokens);    // rows of the buffers; rows of this run
    const int nidx = L.n >> 3;                 // indices per row
    bool vec_ok = (nidx & 7) == 0;             // rows (and the matrices themselves) start 16-byte aligned
#pragma unroll
    for (int s = 0; s < NS; ++s) vec_ok = vec_ok && (reinterpret_cast<uintptr_t>(L.codes[s]) & 15) == 0;
    const int rowA = strip * 16 + gq, rowB = rowA + 8;
    const bool okA = rowA < L.m, okB = rowB < L.m;

    float acc[NS][NB][4];
#pragma unroll
    for (int s = 0; s < NS; ++s)
#pragma unroll
      for (int nb = 0; nb < NB; ++nb)
#pragma unroll
        for (int i = 0; i < 4; ++i) acc[s][nb][i] = 0.f;

    const __half* xr = reinterpret_cast<const __half*>(ws + L.xr_off);

    // Software pipeline over chunks of KC index pairs (a group is 8 / KC chunks).  As soon as pair k of a chunk has been
    // expanded and multiplied, the entries of pair k of the next chunk are requested into the registers it leaves, so that
    // gathers and arithmetic alternate instruction by instruction (a chunk of gathers, then a chunk of arithmetic, kept the
    // load pipe and the issue slots busy in turn); the index words of the chunk after that are on their way from HBM.
    // Whole calls, a chunk at a time / this: one token of 14336 x 4096 56.1 / 52.1 us, 16 tokens of 4096 x 14336 69.2 / 67.9.
    // (512 threads with 128 registers instead of 384 with 168: 55.3 and 71.0.)
    constexpr int KC = (NS <= 2 && NB <= 2) ? GLQB_E8_KC : 4;
    constexpr int CPG = 8 / KC;
    constexpr int W = KC / 2;
    auto load_indices = [&](int cc, uint32_t (&qa)[NS][W], uint32_t (&qb)[NS][W]) {
      const int i0 = (cc / CPG) * 32 + tq * 8 + (cc % CPG) * KC;
#pragma unroll
      for (int s = 0; s < NS; ++s) {
        const uint16_t* q = reinterpret_cast<const uint16_t*>(L.codes[s]);
        const uint16_t* pa = q + (long long)rowA * nidx + i0;
        const uint16_t* pb = q + (long long)rowB * nidx + i0;
        if (vec_ok && i0 + KC <= nidx) {
          if constexpr (KC == 8) {
            uint4 va = make_uint4(0, 0, 0, 0), vb = make_uint4(0, 0, 0, 0);
            if (okA) va = ld_stream_v4(pa);
            if (okB) vb = ld_stream_v4(pb);
            qa[s][0] = va.x; qa[s][1] = va.y; qa[s][2] = va.z; qa[s][3] = va.w;
            qb[s][0] = vb.x; qb[s][1] = vb.y; qb[s][2] = vb.z; qb[s][3] = vb.w;
          } else {
            uint2 va = make_uint2(0, 0), vb = make_uint2(0, 0);
            if (okA) va = ld_stream_v2(pa);
            if (okB) vb = ld_stream_v2(pb);
            qa[s][0] = va.x; qa[s][1] = va.y;
            qb[s][0] = vb.x; qb[s][1] = vb.y;
          }
        } else {
#pragma unroll
          for (int k = 0; k < W; ++k) {
            uint32_t a0 = 0, a1 = 0, b0 = 0, b1 = 0;
            if (i0 + 2 * k < nidx) { if (okA) a0 = pa[2 * k]; if (okB) b0 = pb[2 * k]; }
            if (i0 + 2 * k + 1 < nidx) { if (okA) a1 = pa[2 * k + 1]; if (okB) b1 = pb[2 * k + 1]; }
            qa[s][k] = a0 | (a1 << 16);
            qb[s][k] = b0 | (b1 << 16);
          }
        }
      }
    };
    E8Stage stg[NS];
#pragma unroll
    for (int s = 0; s < NS; ++s) {
      stg[s].table = L.table[s];
      stg[s].mask = (uint32_t)L.table_entries[s] - 1u;
      stg[s].base = L.table_entries[s] == 65536 ? T.table_base : T.small_base;
    }
    auto gather = [&](const uint32_t (&qa)[NS][W], const uint32_t (&qb)[NS][W], int k, uint32_t (&ea)[NS][KC], uint32_t (&eb)[NS][KC]) {
#pragma unroll
      for (int s = 0; s < NS; ++s) {
        ea[s][k] = e8_gather<TM>(stg[s], (qa[s][k >> 1] >> ((k & 1) * 16)) & stg[s].mask);
        eb[s][k] = e8_gather<TM>(stg[s], (qb[s][k >> 1] >> ((k & 1) * 16)) & stg[s].mask);
      }
    };
    // columns past the tokens of the run read the last token again (their accumulator columns are never stored)
    const uint4* xrow[NB];
    const int xstep = batch == 1 ? 1 : 8;      // 16-byte units between consecutive 8-column blocks
#pragma unroll
    for (int nb = 0; nb < NB; ++nb) {
      const int tok = min(nb * 8 + gq, used - 1);
      xrow[nb] = reinterpret_cast<const uint4*>(xr) + (batch == 1 ? 0 : (long long)(tok >> 3) * nidx * 8 + (tok & 7));
    }
    auto consume = [&](int i0, int k, const uint32_t (&ea)[NS][KC], const uint32_t (&eb)[NS][KC]) {
      const int blk = min(i0 + k, nidx - 1);
      uint4 xb[NB];
#pragma unroll
      for (int nb = 0; nb < NB; ++nb) {
        xb[nb] = __ldg(xrow[nb] + blk * xstep);
        if (i0 + k >= nidx) xb[nb] = make_uint4(0u, 0u, 0u, 0u);   // past the row end: contributes nothing
      }
#pragma unroll
      for (int s = 0; s < NS; ++s) {
        uint32_t ha[4], hb[4];
        e8_entry_to_half2(ea[s][k], ha);
        e8_entry_to_half2(eb[s][k], hb);
        const uint32_t a1[4] = {ha[0], hb[0], ha[1], hb[1]};
        const uint32_t a2[4] = {ha[2], hb[2], ha[3], hb[3]};
#pragma unroll
        for (int nb = 0; nb < NB; ++nb) {
          mma16816(acc[s][nb], a1, xb[nb].x, xb[nb].y);
          mma16816(acc[s][nb], a2, xb[nb].z, xb[nb].w);
        }
      }
    };

    const int cc0 = c0 * CPG, cc1 = c1 * CPG;
    uint32_t qa[NS][W], qb[NS][W], na[NS][W], nb2[NS][W];
    uint32_t eA[NS][KC], eB[NS][KC];
    load_indices(cc0, qa, qb);
#pragma unroll
    for (int k = 0; k < KC; ++k) gather(qa, qb, k, eA, eB);
    if (cc0 + 1 < cc1) load_indices(cc0 + 1, qa, qb);
#pragma unroll 1
    for (int cc = cc0; cc < cc1; ++cc) {
      const int i0 = (cc / CPG) * 32 + tq * 8 + (cc % CPG) * KC;   // first index (8-column block) of this lane
      if (cc + 2 < cc1) load_indices(cc + 2, na, nb2);
      if (cc + 1 < cc1) {
#pragma unroll
        for (int k = 0; k < KC; ++k) {
          consume(i0, k, eA, eB);
          gather(qa, qb, k, eA, eB);
        }
      } else {
#pragma unroll
        for (int k = 0; k < KC; ++k) consume(i0, k, eA, eB);
      }
#pragma unroll
      for (int s = 0; s < NS; ++s)
#pragma unroll
        for (int i = 0; i < W; ++i) { qa[s][i] = na[s][i]; qb[s][i] = nb2[s][i]; }
    }

    {
      const long long g0 = L.group_base + (long long)strip * gps;
      const int slot = (int)(w - g0 / per_warp);
      float* part = reinterpret_cast<float*>(ws + L.part_off) + (long long)slot * batch * L.m;
#pragma unroll
      for (int nb = 0; nb < NB; ++nb) {
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const int token = nb * 8 + tq * 2 + (i & 1);
          const int row = (i >> 1) ? rowB : rowA;
          if (token < used && row < L.m) {
            float v = acc[0][nb][i];
#pragma unroll
            for (int s = 1; s < NS; ++s) v = __fadd_rn(v, __fmul_rn(L.stage_scale[s], acc[s][nb][i]));
            part[(long long)token * L.m + row] = v;
          }
        }
      }
    }
    g += c1 - c0;
    if (c1 == gps && strip == L.strips - 1) ++li;
  }
}

template <int NS, int NB>
__global__ void __launch_bounds__(MV_THREADS, (NB <= 2 ? GLQB_E8_MINB : 1))
e8_mv_kernel(const DevLinear* __restrict__ layers, int n_layers, long long total_groups,
             int per_warp, uint8_t* __restrict__ ws, int tokens) {
  const E8Tables T = {0u, 0u};
  e8_mv_body<NS, NB, 0>(layers, n_layers, total_groups, per_warp, ws, T, MV_WARPS, tokens);
}

// Resident-table form: one CTA per SM keeps most of the 65,536-entry table in shared memory.
#ifndef GLQB_E8S_THREADS
#define GLQB_E8S_THREADS 384
#endif
constexpr int E8S_THREADS = GLQB_E8S_THREADS;
constexpr int E8S_SMEM_BYTES = E8S_RESIDENT * 4 + 256 * 4;

template <int NS, int NB>
__global__ void __launch_bounds__(E8S_THREADS, 1)
e8_mv_smem_kernel(const DevLinear* __restrict__ layers, int n_layers, long long total_groups, int per_warp,
                  uint8_t* __restrict__ ws, const uint32_t* __restrict__ big_table,
                  const uint32_t* __restrict__ small_table, int small_entries, int tokens) {
  extern __shared__ __align__(16) uint32_t e8_smem[];
  pdl_trigger();
  const uint4* src = reinterpret_cast<const uint4*>(big_table);
  uint4* dst = reinterpret_cast<uint4*>(e8_smem);
  for (int i = threadIdx.x; i < E8S_RESIDENT / 4; i += blockDim.x) dst[i] = __ldg(src + i);
  for (int i = threadIdx.x; i < small_entries && i < 256; i += blockDim.x) e8_smem[E8S_RESIDENT + i] = __ldg(small_table + i);
  E8Tables T;
  const uint32_t local = (uint32_t)__cvta_generic_to_shared(e8_smem);
  T.table_base = local;
  T.small_base = local + E8S_RESIDENT * 4;
  __syncthreads();
  pdl_wait();                                    // (the table fill overlaps the input transform)
  e8_mv_body<NS, NB, 1>(layers, n_layers, total_groups, per_warp, ws, T, E8S_THREADS / 32, tokens);
}

// ---------------------------------------------------------------------------------------------
// Dump kernels (bit-exact gate).  They call the same decode_tile / table expansion as the compute
// kernels and write the reconstructed rotated-domain weights in natural (row, col) order.
// ---------------------------------------------------------------------------------------------
template <int K1, int K2>
__global__ void __launch_bounds__(MV_THREADS)
trellis_dump_kernel(const uint8_t* __restrict__ p1, const uint8_t* __restrict__ p2, float s2,
                    int m, int n, void* __restrict__ out, int out_f32) {
  const int lane = threadIdx.x & 31;
  const int gps = n >> 5;
  const long long total = (long long)(m >> 5) * gps;
  for (long long g = (long long)blockIdx.x * MV_WARPS + (threadIdx.x >> 5); g < total;
       g += (long long)gridDim.x * MV_WARPS) {
    const int strip = (int)(g / gps), cp = (int)(g % gps);
    const Words<K1> v = load_words<K1>(p1 + g * (128 * K1) + lane * (4 * K1));
    const Words<K1> vn = shfl_words<K1>(v, (lane + 1) & 31);
    Words<K1> vn2 = vn;
    if constexpr (K1 == 1) vn2 = shfl_words<K1>(v, (lane + 2) & 31);
    Words<(K2 > 0 ? K2 : 1)> u, un, un2;
    if constexpr (K2 > 0) {
      u = load_words<K2>(p2 + g * (128 * K2) + lane * (4 * K2));
      un = shfl_words<K2>(u, (lane + 1) & 31);
      un2 = un;
      if constexpr (K2 == 1) un2 = shfl_words<K2>(u, (lane + 2) & 31);
    }
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const int ni = q >> 1, mi = q & 1;
      uint32_t a[8], b[8];
      decode_tile<K1>(chunk_of<K1>(v, q), chunk_of<K1>(vn, q), chunk_of<K1>(vn2, q), a);
      if constexpr (K2 > 0) decode_tile<K2>(chunk_of<K2>(u, q), chunk_of<K2>(un, q), chunk_of<K2>(un2, q), b);
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        const int row = strip * 32 + mi * 16 + tile_row(lane, j);
        const int col = cp * 32 + ni * 16 + tile_col(lane, j);
        const __half h = __ushort_as_half((unsigned short)(a[j] & 0xFFFFu));
        if (out_f32) {
          float f = __half2float(h);
          if constexpr (K2 > 0) {
            const __half h2 = __ushort_as_half((unsigned short)(b[j] & 0xFFFFu));
            f = __fadd_rn(f, __fmul_rn(__half2float(h2), s2));
          }
          reinterpret_cast<float*>(out)[(long long)row * n + col] = f;
        } else {
          reinterpret_cast<__half*>(out)[(long long)row * n + col] = h;
        }
      }
    }
  }
}

struct E8DumpArgs {
  const uint16_t* q[GLQB_MAX_STAGES];
  const uint32_t* table[GLQB_MAX_STAGES];
  int entries[GLQB_MAX_STAGES];
  float scale[GLQB_MAX_STAGES];
  int n_stages, m, n;
};

static __global__ void __launch_bounds__(256) e8_dump_kernel(E8DumpArgs A, float* __restrict__ out) {
  const int nidx = A.n >> 3;
  const long long total = (long long)A.m * nidx;
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < total;
       i += (long long)gridDim.x * blockDim.x) {
    float v[8];
    {
      const uint32_t e = A.table[0][A.q[0][i] & (uint32_t)(A.entries[0] - 1)];
      uint32_t h[4];
      e8_entry_to_half2(e, h);     // same expansion the matvec uses; unpack (c_k, c_{k+4})
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        v[k] = __half2float(__ushort_as_half((unsigned short)(h[k] & 0xFFFFu)));
        v[k + 4] = __half2float(__ushort_as_half((unsigned short)(h[k] >> 16)));
      }
    }
    for (int s = 1; s < A.n_stages; ++s) {
      const uint32_t e = A.table[s][A.q[s][i] & (uint32_t)(A.entries[s] - 1)];
      uint32_t h[4];
      e8_entry_to_half2(e, h);
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        const float lo = __half2float(__ushort_as_half((unsigned short)(h[k] & 0xFFFFu)));
        const float hi = __half2float(__ushort_as_half((unsigned short)(h[k] >> 16)));
        v[k] = __fadd_rn(v[k], __fmul_rn(lo, A.scale[s]));
        v[k + 4] = __fadd_rn(v[k + 4], __fmul_rn(hi, A.scale[s]));
      }
    }
    float* o = out + i * 8;
#pragma unroll
    for (int k = 0; k < 8; ++k) o[k] = v[k];
  }
}

static __global__ void e8_pack_table_kernel(const __half* __restrict__ cb, int entries, uint32_t* __restrict__ out) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= entries) return;
  uint32_t p = 0;
#pragma unroll
  for (int k = 0; k < 8; ++k) {
    const int code = __float2int_rn(__half2float(cb[i * 8 + k]) * 2.0f) + 6;
    p |= (uint32_t)(code & 0xF) << (4 * k);
  }
  out[i] = p;
}

}  // namespace glqb
