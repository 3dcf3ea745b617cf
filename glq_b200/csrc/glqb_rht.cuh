// Transform kernels: rotated activations of a layer, results from its partial sums, and the unfused transform ops.
#pragma once
#include "glqb_kernels.cuh"
#include "glqb_fht.cuh"
#include "glqb_fht_fast.cuh"

namespace glqb {

// ---------------------------------------------------------------------------------------------
// Input transform:  xr = fp16( H_blocks( SV * pad(x) ) / sqrt(bs) ), written in the layout the
// decode kernel of the layer's format reads (reference: glq_input_rht_multiblock_kernel,
// glq/csrc/glq_cuda.cu:2092; rounding to fp16 as glq/csrc/glq_cuda.cu:2625).
// One CTA per (layer, Hadamard block, tile of tokens); the transform itself is fht_block (first pass
// fused with the global loads, last pass with the stores).
// PLAIN_F32: write fp32 in natural order instead (the unfused input_rht op).
// ---------------------------------------------------------------------------------------------
constexpr int RHT_THREADS = FHT_THREADS;
constexpr int RHT_MINB = 3;                      // 85 registers: the eight 16-byte loads of a thread stay in flight

// 1 / rms of a token's input values (fused RMSNorm), by all threads of the CTA; `red` holds >= 32 floats
__device__ __forceinline__ float token_rstd(const DevLinear& L, const uint8_t* x_base, long long xt0, float* red) {
  float ss = 0.f;
  for (int i = threadIdx.x; i < L.in_f; i += blockDim.x) { const float v = input_value(L, x_base, xt0, i); ss += v * v; }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
  __syncthreads();
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = ss;
  __syncthreads();
  float tot = 0.f;
  for (int w = 0; w < (int)(blockDim.x >> 5); ++w) tot += red[w];
  return rsqrtf(tot / (float)L.in_f + L.in_norm_eps);
}

// four fp16 signs (8-byte aligned) as two packed pairs
__device__ __forceinline__ void load_sign4(const __half* p, f2 (&s)[2]) {
  const uint2 t = *reinterpret_cast<const uint2*>(p);
  const float2 a = __half22float2(*reinterpret_cast<const __half2*>(&t.x));
  const float2 b = __half22float2(*reinterpret_cast<const __half2*>(&t.y));
  s[0] = f2_pack(a.x, a.y);
  s[1] = f2_pack(b.x, b.y);
}

// The load pass of an input tile (fht_block's `load`): x * SV, zero past in_features.  `log_t`: log2 of the arrays of
// the tile, whose first column is `col0` (the tile's rows are tokens it.tok0 ..).  A block longer than a tile comes
// as S = 2 or 4 runs (RhtItem::sub): run k of the result is the transform of sum_kk H_S[k][kk] * (run kk of x).
// `one(row, i)`: the value of column col0 + i alone, for everything the vector path does not take.
template <class One>
__device__ __forceinline__ void rht_load_x(const DevLinear& L, const RhtItem& it, const uint8_t* __restrict__ x_base, int col0,
                                           int log_t, int total, int S, bool vec, One one, int e0, f2 (&v)[8][2]) {
#pragma unroll
  for (int k = 0; k < 8; ++k) v[k][0] = v[k][1] = 0;
  for (int kk = 0; kk < S; ++kk) {
    const float sg = (__popc(max(it.sub, 0) & kk) & 1) ? -1.f : 1.f;
    const f2 sg2 = f2_pack(sg, sg);
    const int c0 = col0 + (kk << FHT_LOG);
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      const int e = e0 + (k << 10);
      if (e < total) {
        const int row = e >> log_t, i = e & ((1 << log_t) - 1);
        if (vec && c0 + i + 3 < L.in_f) {
          float t[4];
          f2 s[2];
          load_act4(x_base, L.x_off + (long long)(it.tok0 + row) * L.x_stride + c0 + i, L.x_dtype, t);
          load_sign4(L.sv + c0 + i, s);
          v[k][0] = f2_fma(f2_mul(f2_pack(t[0], t[1]), s[0]), sg2, v[k][0]);
          v[k][1] = f2_fma(f2_mul(f2_pack(t[2], t[3]), s[1]), sg2, v[k][1]);
        } else {
          float t[4];
#pragma unroll
          for (int j = 0; j < 4; ++j)
            t[j] = e + j < total ? one((e + j) >> log_t, (kk << FHT_LOG) + ((e + j) & ((1 << log_t) - 1))) : 0.f;
          v[k][0] = f2_fma(f2_pack(t[0], t[1]), sg2, v[k][0]);
          v[k][1] = f2_fma(f2_pack(t[2], t[3]), sg2, v[k][1]);
        }
      }
    }
  }
}

// The same for what the plain kernels serve: aligned rows, no fused step, every column below in_features.
__device__ __forceinline__ void rht_load_x_plain(const DevLinear& L, const RhtItem& it, const uint8_t* __restrict__ x_base, int col0,
                                                 int log_t, int total, int S, int e0, f2 (&v)[8][2]) {
  const int i0 = col0 + (e0 & ((1 << log_t) - 1));
  const long long o = L.x_off + (long long)(it.tok0 + (e0 >> log_t)) * L.x_stride + i0;
  const long long stride = L.x_stride;
  const __half* sv = L.sv + i0;
  with_dtype(L.x_dtype, [&](auto dt) {
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      v[k][0] = v[k][1] = 0;
      if (e0 + (k << 10) < total) {
        float t[4];
        f2 s[2];
        load_act4(x_base, o + fht_row(k, 1024, log_t) * stride + fht_col(k, 1024, log_t), decltype(dt)::value, t);
        load_sign4(sv + fht_col(k, 1024, log_t), s);
        v[k][0] = f2_mul(f2_pack(t[0], t[1]), s[0]);
        v[k][1] = f2_mul(f2_pack(t[2], t[3]), s[1]);
      }
    }
    for (int kk = 1; kk < S; ++kk) {                       // (blocks longer than a tile: one token, full tile)
      const f2 sg2 = (__popc(it.sub & kk) & 1) ? F2_MINUS1 : F2_ONE;
#pragma unroll
      for (int k = 0; k < 8; ++k) {
        float t[4];
        f2 s[2];
        load_act4(x_base, o + (kk << FHT_LOG) + (k << 10), decltype(dt)::value, t);
        load_sign4(sv + (kk << FHT_LOG) + (k << 10), s);
        v[k][0] = f2_fma(f2_mul(f2_pack(t[0], t[1]), s[0]), sg2, v[k][0]);
        v[k][1] = f2_fma(f2_mul(f2_pack(t[2], t[3]), s[1]), sg2, v[k][1]);
      }
    }
  });
}

// Input of a decode step with the fused steps (RMSNorm weight, act(gate) * up), aligned rows, whole blocks, one run.
__device__ __forceinline__ void rht_load_x_fused(const DevLinear& L, const RhtItem& it, const uint8_t* __restrict__ x_base, int col0,
                                                 int log_t, int total, int e0, f2 (&v)[8][2]) {
  const int i0 = col0 + (e0 & ((1 << log_t) - 1));
  const long long o = L.x_off + (long long)(it.tok0 + (e0 >> log_t)) * L.x_stride + i0;
  const long long stride = L.x_stride;
  const int act = L.in_gated_act;
  with_dtype(L.x_dtype, [&](auto dt) {
    constexpr int DT = decltype(dt)::value;
    float q[8][4];
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      q[k][0] = q[k][1] = q[k][2] = q[k][3] = 0.f;
      if (e0 + (k << 10) < total) load_act4(x_base, o + fht_row(k, 1024, log_t) * stride + fht_col(k, 1024, log_t), DT, q[k]);
    }
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      v[k][0] = v[k][1] = 0;
      if (e0 + (k << 10) < total) {
        const int i = fht_col(k, 1024, log_t);
        if (act) {
          float u[4];
          load_act4(x_base, o + fht_row(k, 1024, log_t) * stride + i + L.in_f, DT, u);
#pragma unroll
          for (int j = 0; j < 4; ++j) q[k][j] = round_act(round_act(act_fn(q[k][j], act - 1), DT) * u[j], DT);
        }
        if (L.in_norm_w) {
#pragma unroll
          for (int j = 0; j < 4; ++j) q[k][j] *= load_act(L.in_norm_w, i0 + i + j, L.in_norm_dtype);
        }
        f2 s[2];
        load_sign4(L.sv + i0 + i, s);
        v[k][0] = f2_mul(f2_pack(q[k][0], q[k][1]), s[0]);
        v[k][1] = f2_mul(f2_pack(q[k][2], q[k][3]), s[1]);
      }
    }
  });
}

// A thread's finished groups of four as rotated activations of the streaming kernels (fragment order of the format);
// `sc`: scale per token of the tile, 1 / sqrt(bs) included.  Tiles of arrays of 128 values or more (a warp's 32 groups
// are then all valid or all not).
template <class Scale>
__device__ __forceinline__ void rht_store_xr(const DevLinear& L, const RhtItem& it, uint8_t* __restrict__ ws, int col0, int log_t,
                                             int total, int e1, const f2 (&v)[8][2], Scale sc) {
  const int c0 = col0 + (e1 & ((1 << log_t) - 1)), r0 = e1 >> log_t;
  const bool odd = threadIdx.x & 1;
#pragma unroll
  for (int k = 0; k < 8; ++k)
    if (e1 + (k << 7) < total) {
      const int row = r0 + fht_row(k, 128, log_t), c = c0 + fht_col(k, 128, log_t);
      const float w = sc(row);
      const f2 w2 = f2_pack(w, w);
      float r[4];
      f2_unpack(f2_mul(v[k][0], w2), r[0], r[1]);
      f2_unpack(f2_mul(v[k][1], w2), r[2], r[3]);
      const long long token = it.tok0 + row;
      if (L.format == GLQB_FMT_TRELLIS_3INST) {
        // (xr_pos_trellis: columns c, c + 1 share a lane's 16 halfs, c + 2 and c + 3 sit 16 halfs on)
        __half2* p = reinterpret_cast<__half2*>(ws + L.xr_off) + token * L.n +
                     (((c & ~31) * XR_TRELLIS_EXPAND + xr_pos_trellis(c & 31)) >> 1);
        const __half z = __float2half_rn(0.f);
        p[0] = __halves2half2(__float2half_rn(r[0]), z);
        p[2] = __halves2half2(__float2half_rn(r[1]), z);
        p[8] = __halves2half2(__float2half_rn(r[2]), z);
        p[10] = __halves2half2(__float2half_rn(r[3]), z);
      } else {
        // a block of 8 columns is held by two lanes and stored as (x0,x4,x1,x5 | x2,x6,x3,x7)
        const __half2 lo2 = __floats2half2_rn(r[0], r[1]), hi2 = __floats2half2_rn(r[2], r[3]);
        const uint32_t lo = *reinterpret_cast<const uint32_t*>(&lo2), hi = *reinterpret_cast<const uint32_t*>(&hi2);
        const uint32_t got = __shfl_xor_sync(0xffffffffu, odd ? lo : hi, 1);
        const uint32_t a = odd ? got : lo, b = odd ? hi : got;          // first and second of each stored pair
        const long long base = xr_index_e8(token, c & ~7, L.n, L.batch) + (odd ? 4 : 0);
        *reinterpret_cast<uint2*>(reinterpret_cast<__half*>(ws + L.xr_off) + base) =
            make_uint2(__byte_perm(a, b, 0x5410), __byte_perm(a, b, 0x7632));
      }
    }
}

template <bool PLAIN_F32>
__device__ __forceinline__ void rht_in_body(const DevLinear& L, const RhtItem it, const uint8_t* __restrict__ x_base,
                                            uint8_t* __restrict__ ws, float* fbuf) {
  __shared__ float rstd_s[FUSED_MAX_TOKENS_C];
  const int off = L.bn_off[it.block];
  const int logbs = L.bn_log[it.block];
  const int bs = 1 << logbs;
  const bool trellis = (L.format == GLQB_FMT_TRELLIS_3INST);
  const float rs = L.x_is_rotated ? 1.0f : rsqrtf((float)bs);
  auto store1 = [&](int row, int i, float v) {
    const int col = off + i;
    const long long token = it.tok0 + row;
    if constexpr (PLAIN_F32) {
      reinterpret_cast<float*>(ws + L.xr_off)[token * L.n + col] = v;
    } else if (trellis) {
      const int pos = (col & ~31) * XR_TRELLIS_EXPAND + xr_pos_trellis(col & 31);   // half index, even
      (reinterpret_cast<__half2*>(ws + L.xr_off) + token * L.n)[pos >> 1] =
          __halves2half2(__float2half_rn(v), __float2half_rn(0.f));
    } else {
      reinterpret_cast<__half*>(ws + L.xr_off)[xr_index_e8(token, col, L.n, L.batch)] = __float2half_rn(v);
    }
  };
  const bool fusions = L.in_gated_act != 0 || L.in_norm_w != nullptr;
  auto load1 = [&](int row, int i) -> float {
    const int col = off + i;
    if (col >= L.in_f) return 0.f;
    const long long xt0 = L.x_off + (long long)(it.tok0 + row) * L.x_stride;
    float v = fusions ? input_value(L, x_base, xt0, col) : load_act(x_base, xt0 + col, L.x_dtype);
    if (L.in_norm_w) v *= load_act(L.in_norm_w, col, L.in_norm_dtype);
    if (!L.x_is_rotated) v *= __half2float(L.sv[col]);
    return v;
  };
  const int S = it.sub >= 0 ? bs >> FHT_LOG : 1, log_t = min(logbs, FHT_LOG), run0 = max(it.sub, 0) << FHT_LOG;
  const int total = it.ntok << log_t;
  if (L.x_is_rotated) {            // already transformed by the caller: convert and lay out only
    for (int o = threadIdx.x; o < total; o += blockDim.x) {
      const int row = o >> log_t, i = run0 + (o & ((1 << log_t) - 1));
      store1(row, i, load1(row, i));
    }
    return;
  }
  // fused RMSNorm (at most 8 tokens): 1 / rms of the token is folded into the stored values
  if (L.in_norm_w)
    for (int r = 0; r < it.ntok; ++r) {
      const float v = token_rstd(L, x_base, L.x_off + (long long)(it.tok0 + r) * L.x_stride, fbuf);
      if (threadIdx.x == 0) rstd_s[r] = v;
      __syncthreads();
    }
  const bool normed = L.in_norm_w != nullptr;
  const bool rows_ok = (off & 7) == 0 && act_rows_aligned4(x_base, L.x_off, L.x_stride, L.x_dtype) && off + bs <= L.in_f &&
                       (!L.in_gated_act || (L.in_f & 3) == 0);
  if (!PLAIN_F32 && rows_ok && log_t >= 7 && !(fusions && S > 1)) {
    auto load = [&](int e0, f2 (&v)[8][2]) {
      if (fusions) rht_load_x_fused(L, it, x_base, off, log_t, total, e0, v);
      else rht_load_x_plain(L, it, x_base, off, log_t, total, S, e0, v);
    };
    auto store = [&](int e1, const f2 (&v)[8][2]) {
      rht_store_xr(L, it, ws, off + run0, log_t, total, e1, v, [&](int row) { return normed ? rs * rstd_s[row] : rs; });
    };
    fht_block_all(fbuf, log_t, total, load, store);
    return;
  }
  const bool out_vec = PLAIN_F32 && ((L.n | off) & 3) == 0 && log_t >= 2 && (reinterpret_cast<uintptr_t>(ws + L.xr_off) & 15) == 0;
  if constexpr (PLAIN_F32) {
    // aligned rows, whole blocks: block lengths known at compile time (one token of 8192 columns 7.0 us with the general
    // body below, 2048 tokens of 32768 399 us; 3.7 and 156 here)
    if (rows_ok && out_vec) {
      auto load = [&](int e0, f2 (&v)[8][2]) { rht_load_x_plain(L, it, x_base, off, log_t, total, S, e0, v); };
      auto store = [&](int e1, const f2 (&v)[8][2]) {
        const f2 rs2 = f2_pack(rs, rs);
        float* p = reinterpret_cast<float*>(ws + L.xr_off) + (long long)(it.tok0 + (e1 >> log_t)) * L.n + off + run0 +
                   (e1 & ((1 << log_t) - 1));
#pragma unroll
        for (int k = 0; k < 8; ++k)
          if (e1 + (k << 7) < total) {
            const f2 r[2] = {f2_mul(v[k][0], rs2), f2_mul(v[k][1], rs2)};
            fht_st4(p + (long long)fht_row(k, 128, log_t) * L.n + fht_col(k, 128, log_t), r);
          }
      };
      fht_block_all(fbuf, log_t, total, load, store);
      return;
    }
  }
  const bool vec = !fusions && (off & 3) == 0 && log_t >= 2 && act_rows_aligned4(x_base, L.x_off, L.x_stride, L.x_dtype);
  auto load = [&](int e0, f2 (&v)[8][2]) { rht_load_x(L, it, x_base, off, log_t, total, S, vec, load1, e0, v); };
  auto store = [&](int e, const f2 (&q)[2]) {
    float r[4];
    f2_unpack(q[0], r[0], r[1]);
    f2_unpack(q[1], r[2], r[3]);
    if (out_vec) {
      const int row = e >> log_t, i = run0 + (e & ((1 << log_t) - 1));
      *reinterpret_cast<float4*>(reinterpret_cast<float*>(ws + L.xr_off) + (long long)(it.tok0 + row) * L.n + off + i) =
          make_float4(r[0] * rs, r[1] * rs, r[2] * rs, r[3] * rs);
      return;
    }
#pragma unroll
    for (int j = 0; j < 4; ++j)
      if (e + j < total) {
        const int row = (e + j) >> log_t;
        const float v = r[j] * rs;
        store1(row, run0 + ((e + j) & ((1 << log_t) - 1)), normed ? v * rstd_s[row] : v);
      }
  };
  fht_block(fbuf, log_t, total, load, store);
}

// the tile of an item that lies below `tokens`, the tokens of this run; false: none of it does
__device__ __forceinline__ bool rht_item_trim(RhtItem& it, int tokens) {
  it.ntok = min(it.ntok, tokens - it.tok0);
  return it.ntok > 0;
}

template <bool PLAIN_F32>
__global__ void __launch_bounds__(RHT_THREADS, RHT_MINB) rht_in_kernel(const DevLinear* __restrict__ layers,
                                                             const RhtItem* __restrict__ items,
                                                             const uint8_t* __restrict__ x_base,
                                                             uint8_t* __restrict__ ws, int tokens) {
  extern __shared__ __align__(16) float fbuf[];
  pdl_wait();
  pdl_trigger();
  RhtItem it = items[blockIdx.x];
  if (rht_item_trim(it, tokens)) rht_in_body<PLAIN_F32>(layers[it.layer], it, x_base, ws, fbuf);
}

// The same for launches of few tiles whose inputs come with fused steps (the [gate | up] rows of a down projection in a decode
// step).  Four decoder layers, one token 333.5 / 328.6 us.
static __global__ void __launch_bounds__(FHT_WIDE_THREADS, 1) rht_in_wide_kernel(const DevLinear* __restrict__ layers,
                                                              const RhtItem* __restrict__ items,
                                                              const uint8_t* __restrict__ x_base,
                                                              uint8_t* __restrict__ ws, int tokens) {
  extern __shared__ __align__(16) float fbuf[];
  __shared__ float rstd_s[FUSED_MAX_TOKENS_C];
  pdl_wait();
  pdl_trigger();
  RhtItem it = items[blockIdx.x];
  if (!rht_item_trim(it, tokens)) return;
  const DevLinear& L = layers[it.layer];
  const int off = L.bn_off[it.block], logbs = L.bn_log[it.block], bs = 1 << logbs;
  const bool trellis = L.format == GLQB_FMT_TRELLIS_3INST, fusions = L.in_gated_act != 0 || L.in_norm_w != nullptr;
  const bool normed = L.in_norm_w != nullptr, rotated = L.x_is_rotated != 0;
  const float rs = rotated ? 1.0f : rsqrtf((float)bs);
  const int S = it.sub >= 0 ? bs >> FHT_LOG : 1, log_t = min(logbs, FHT_LOG), run0 = max(it.sub, 0) << FHT_LOG;
  const int total = it.ntok << log_t;
  if (normed)                                              // (at most 8 tokens)
    for (int r = 0; r < it.ntok; ++r) {
      const float v = token_rstd(L, x_base, L.x_off + (long long)(it.tok0 + r) * L.x_stride, fbuf);
      if (threadIdx.x == 0) rstd_s[r] = v;
      __syncthreads();
    }
  auto load = [&](int e0, float (&v)[8]) {
#pragma unroll
    for (int k = 0; k < 8; ++k) v[k] = 0.f;
    for (int kk = 0; kk < S; ++kk) {
      if (rotated && kk != max(it.sub, 0)) continue;
      const float sg = !rotated && (__popc(max(it.sub, 0) & kk) & 1) ? -1.f : 1.f;
      float t[8];
#pragma unroll
      for (int k = 0; k < 8; ++k) {
        const int e = e0 + (k << 10), col = off + (kk << FHT_LOG) + (e & ((1 << log_t) - 1));
        t[k] = 0.f;
        if (e < total && col < L.in_f) {
          const long long xt0 = L.x_off + (long long)(it.tok0 + (e >> log_t)) * L.x_stride;
          t[k] = fusions ? input_value(L, x_base, xt0, col) : load_act(x_base, xt0 + col, L.x_dtype);
          if (normed) t[k] *= load_act(L.in_norm_w, col, L.in_norm_dtype);
          if (!rotated) t[k] *= __half2float(L.sv[col]);
        }
      }
#pragma unroll
      for (int k = 0; k < 8; ++k) v[k] = fmaf(t[k], sg, v[k]);
    }
  };
  auto store = [&](int e, float v) {
    const int row = e >> log_t, col = off + run0 + (e & ((1 << log_t) - 1));
    const long long token = it.tok0 + row;
    v *= normed ? rs * rstd_s[row] : rs;
    if (trellis) {
      const int pos = (col & ~31) * XR_TRELLIS_EXPAND + xr_pos_trellis(col & 31);   // half index, even
      (reinterpret_cast<__half2*>(ws + L.xr_off) + token * L.n)[pos >> 1] = __halves2half2(__float2half_rn(v), __float2half_rn(0.f));
    } else {
      reinterpret_cast<__half*>(ws + L.xr_off)[xr_index_e8(token, col, L.n, L.batch)] = __float2half_rn(v);
    }
  };
  fht_wide(fbuf, rotated ? 0 : log_t, total, load, store);
}

// One layer described entirely in kernel-parameter space (no device table, nothing to allocate or copy):
// the unfused input_rht / output_rht ops.  CTA b of Hadamard block k handles the token tile
// b - first_cta[k]; tile_tokens[k] tokens per tile (blocks longer than a tile: one token and one run per CTA).
struct RhtSingle {
  int first_cta[GLQB_MAX_BLOCKS + 1];
  int tile_tokens[GLQB_MAX_BLOCKS];
  int runs[GLQB_MAX_BLOCKS];
  int n_blocks;
};
__device__ __forceinline__ RhtItem rht_single_item(const RhtSingle& S, int batch) {
  int k = 0;
  while (k + 1 < S.n_blocks && (int)blockIdx.x >= S.first_cta[k + 1]) ++k;
  const int c = (int)blockIdx.x - S.first_cta[k];
  if (S.runs[k] > 1) return RhtItem{0, k, c / S.runs[k], 1, c % S.runs[k]};
  const int tok0 = c * S.tile_tokens[k];
  return RhtItem{0, k, tok0, min(S.tile_tokens[k], batch - tok0), -1};
}
static __global__ void __launch_bounds__(RHT_THREADS, RHT_MINB) rht_in_single_kernel(const __grid_constant__ DevLinear L,
                                                                    const __grid_constant__ RhtSingle S,
                                                                    const uint8_t* __restrict__ x_base,
                                                                    uint8_t* __restrict__ out) {
  extern __shared__ __align__(16) float fbuf[];
  rht_in_body<true>(L, rht_single_item(S, L.batch), x_base, out, fbuf);
}

// ---------------------------------------------------------------------------------------------
// Output transform: sums the partial sums of every strip in fixed (ascending slot) order, applies
// wscale (and the optional per-row scale), the block Hadamard, 1/sqrt(bs) and SU, and writes
// y[:, :out_features] (reference: glq_output_rht_multiblock_kernel, glq/csrc/glq_cuda.cu:2151).
// FROM_F32: input is a plain fp32 (batch, m) matrix (the unfused output_rht op).
// WIDE: batch * m may be 2^32 or more.  The tile's first token is then part of the pointer; elsewhere it is part of the
// 32-bit offsets, which is 3 % faster where there are many slots (16 tokens of 2048 x 2048: 37.4 / 39.0 us).
// ---------------------------------------------------------------------------------------------
template <bool FROM_F32, bool WIDE>
__device__ __forceinline__ void rht_out_body(const DevLinear& L, const RhtItem it, const uint8_t* __restrict__ ws,
                                             uint8_t* __restrict__ y_base, const float* __restrict__ yrht_in,
                                             float* fbuf) {
  const int off = L.bm_off[it.block];
  const int logbs = L.bm_log[it.block];
  const int bs = 1 << logbs;
  const int strip_log = (L.format == GLQB_FMT_TRELLIS_3INST) ? 5 : 4;
  const int m = L.m, gps = L.groups_per_strip;
  const unsigned per_warp = (unsigned)L.per_warp;
  const int fixed_slots = FROM_F32 ? 1 : L.fixed_slots;
  const long long slot_stride = (long long)L.batch * m;
  const float wscale = L.wscale;
  const float* row_scale = L.row_scale;
  const float* src = FROM_F32 ? yrht_in : reinterpret_cast<const float*>(ws + L.part_off);
  if constexpr (WIDE) src += (long long)it.tok0 * m;
  const int tok0 = WIDE ? 0 : it.tok0;             // first token of the tile, counted from `src`
  // partial sums of a row: a property of its strip (the warps whose group ranges touch the strip)
  auto slots_of = [&](int row) -> int {
    if (fixed_slots > 0) return fixed_slots;
    const long long g0 = L.group_base + (long long)(row >> strip_log) * gps;
    if (g0 + gps <= 0xFFFFFFFFll) return (int)(((unsigned)g0 + gps - 1) / per_warp - (unsigned)g0 / per_warp) + 1;
    return (int)((g0 + gps - 1) / per_warp - g0 / per_warp) + 1;
  };
  auto load1 = [&](int trow, int i) -> float {
    const int row = off + i;
    const float* p = src + (long long)(tok0 + trow) * m + row;
    if constexpr (FROM_F32) return *p;
    if (row >= m) return 0.f;
    const int cnt = slots_of(row);
    float s = 0.f;
    for (int k = 0; k < cnt; ++k) s += __ldcg(p + k * slot_stride);
    s *= wscale;
    if (row_scale) s *= row_scale[row];
    return s;
  };
  const int S = it.sub >= 0 ? bs >> FHT_LOG : 1, log_t = min(logbs, FHT_LOG), run0 = max(it.sub, 0) << FHT_LOG;
  const int total = it.ntok << log_t;
  if (L.stop_at_yrht) {            // rotated-domain result wanted: reduce and scale only
    for (int o = threadIdx.x; o < total; o += blockDim.x) {
      const int tk = o >> log_t, i = run0 + (o & ((1 << log_t) - 1));
      if (off + i < m) reinterpret_cast<float*>(y_base)[L.y_off + (long long)(it.tok0 + tk) * L.y_stride + off + i] = load1(tk, i);
    }
    return;
  }
  const bool vec = ((m | off) & 3) == 0 && log_t >= 2 && (!FROM_F32 || (reinterpret_cast<uintptr_t>(src) & 15) == 0);
  auto load = [&](int e0, f2 (&v)[8][2]) {
#pragma unroll
    for (int k = 0; k < 8; ++k) v[k][0] = v[k][1] = 0;
    if (!vec) {
      for (int kk = 0; kk < S; ++kk) {
        const float sg = (__popc(max(it.sub, 0) & kk) & 1) ? -1.f : 1.f;
#pragma unroll
        for (int k = 0; k < 8; ++k) {
          const int e = e0 + (k << 10);
          float t[4];
#pragma unroll
          for (int j = 0; j < 4; ++j)
            t[j] = e + j < total ? sg * load1((e + j) >> log_t, (kk << FHT_LOG) + ((e + j) & ((1 << log_t) - 1))) : 0.f;
          v[k][0] = f2_add(f2_pack(t[0], t[1]), v[k][0]);
          v[k][1] = f2_add(f2_pack(t[2], t[3]), v[k][1]);
        }
      }
      return;
    }
    // all eight loads of a slot are issued together; element offsets fit 32 bits (a tile: at most 64 tokens x 524288 rows)
    for (int kk = 0; kk < S; ++kk) {
      unsigned idx[8];
      int cnt[8];
      int most = 0;
#pragma unroll
      for (int k = 0; k < 8; ++k) {
        const int e = e0 + (k << 10);
        const int row = off + (kk << FHT_LOG) + (e & ((1 << log_t) - 1));
        idx[k] = (unsigned)(tok0 + (e >> log_t)) * (unsigned)m + (unsigned)row;
        cnt[k] = e < total ? (fixed_slots > 0 ? fixed_slots : slots_of(row)) : 0;
        most = max(most, cnt[k]);
      }
      const f2 sg2 = (__popc(max(it.sub, 0) & kk) & 1) ? F2_MINUS1 : F2_ONE;
      for (int s = 0; s < most; ++s) {
        const float* p = src + s * slot_stride;
        ulonglong2 t[8];
#pragma unroll
        for (int k = 0; k < 8; ++k)
          t[k] = s < cnt[k] ? __ldcg(reinterpret_cast<const ulonglong2*>(p + idx[k])) : make_ulonglong2(0, 0);
#pragma unroll
        for (int k = 0; k < 8; ++k) {
          f2 c0 = sg2, c1 = sg2;
          if (row_scale && s < cnt[k]) {
            const float* r = row_scale + off + (kk << FHT_LOG) + ((e0 + (k << 10)) & ((1 << log_t) - 1));
            c0 = f2_mul(c0, f2_pack(r[0], r[1]));
            c1 = f2_mul(c1, f2_pack(r[2], r[3]));
          }
          v[k][0] = f2_fma(t[k].x, c0, v[k][0]);
          v[k][1] = f2_fma(t[k].y, c1, v[k][1]);
        }
      }
    }
    if constexpr (!FROM_F32) {
      const f2 w2 = f2_pack(wscale, wscale);
#pragma unroll
      for (int k = 0; k < 8; ++k) { v[k][0] = f2_mul(v[k][0], w2); v[k][1] = f2_mul(v[k][1], w2); }
    }
  };
  const float rs = rsqrtf((float)bs);
  const int out_f = L.out_f, y_dtype = L.y_dtype;
  const long long y_off = L.y_off, y_stride = L.y_stride;
  const __half* su = L.su;
  const bool accumulate = L.y_accumulate != 0;
  // a fused RMSNorm of the single-launch kernel scales the output: its 1 / rms sits in the workspace
  const float* rstd = (L.in_norm_w && !L.xr_global) ? reinterpret_cast<const float*>(ws + L.rstd_off) : nullptr;
  // four outputs per call: one 8-byte SU load and one 8-byte (16-byte for fp32) store when aligned
  const bool out_vec = (off & 3) == 0 && log_t >= 2 && !accumulate && (reinterpret_cast<uintptr_t>(su) & 7) == 0 &&
                       act_rows_aligned4(y_base, y_off, y_stride, y_dtype);
  auto store = [&](int e, const f2 (&q)[2]) {
    float r[4];
    f2_unpack(q[0], r[0], r[1]);
    f2_unpack(q[1], r[2], r[3]);
    const int trow = e >> log_t, row0 = off + run0 + (e & ((1 << log_t) - 1));
    if (out_vec && row0 + 4 <= out_f) {
      const float sc = rstd ? rs * rstd[it.tok0 + trow] : rs;
      f2 s[2];
      load_sign4(su + row0, s);
      const f2 sc2 = f2_pack(sc, sc);
      f2_unpack(f2_mul(f2_mul(q[0], sc2), s[0]), r[0], r[1]);
      f2_unpack(f2_mul(f2_mul(q[1], sc2), s[1]), r[2], r[3]);
      store_act4(y_base, y_off + (long long)(it.tok0 + trow) * y_stride + row0, y_dtype, r);
      return;
    }
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int t = (e + j) >> log_t, row = off + run0 + ((e + j) & ((1 << log_t) - 1));
      if (e + j < total && row < out_f) {
        const float sc = rstd ? rs * rstd[it.tok0 + t] : rs;
        const long long o = y_off + (long long)(it.tok0 + t) * y_stride + row;
        float v = r[j] * sc * __half2float(su[row]);
        if (accumulate) v += load_act(y_base, o, y_dtype);          // residual add
        store_act(y_base, o, y_dtype, v);
      }
    }
  };
  fht_block(fbuf, log_t, total, load, store);
}

// The same for launches of few tiles (decode steps) without per-row scales.  Whole calls, 256 threads a tile / this: 16 tokens of 4096 x 14336 70.6 /
// 67.3 us, 27 tokens of 11008 x 2048 (4 + 2 bits) 55.0 / 54.2, one token of 14336 x 4096 49.4 / 49.2.
static __global__ void __launch_bounds__(FHT_WIDE_THREADS, 1) rht_out_wide_kernel(const DevLinear* __restrict__ layers,
                                                              const RhtItem* __restrict__ items,
                                                              const uint8_t* __restrict__ ws,
                                                              uint8_t* __restrict__ y_base, int tokens) {
  extern __shared__ __align__(16) float fbuf[];
  pdl_trigger();
  RhtItem it = items[blockIdx.x];
  if (!rht_item_trim(it, tokens)) return;
  const DevLinear& L = layers[it.layer];
  const int off = L.bm_off[it.block], logbs = L.bm_log[it.block], bs = 1 << logbs;
  const int strip_log = (L.format == GLQB_FMT_TRELLIS_3INST) ? 5 : 4;
  const int m = L.m, gps = L.groups_per_strip, fixed_slots = L.fixed_slots;
  const unsigned per_warp = (unsigned)L.per_warp;
  const long long slot_stride = (long long)L.batch * m;
  const float* src = reinterpret_cast<const float*>(ws + L.part_off);
  const int S = it.sub >= 0 ? bs >> FHT_LOG : 1, log_t = min(logbs, FHT_LOG), run0 = max(it.sub, 0) << FHT_LOG;
  const int total = it.ntok << log_t;
  auto slots_of = [&](int row) -> int {                    // (rht_out_body)
    if (fixed_slots > 0) return fixed_slots;
    const long long g0 = L.group_base + (long long)(row >> strip_log) * gps;
    if (g0 + gps <= 0xFFFFFFFFll) return (int)(((unsigned)g0 + gps - 1) / per_warp - (unsigned)g0 / per_warp) + 1;
    return (int)((g0 + gps - 1) / per_warp - g0 / per_warp) + 1;
  };
  const float rs = rsqrtf((float)bs), wscale = L.wscale;
  const float* rstd = (L.in_norm_w && !L.xr_global) ? reinterpret_cast<const float*>(ws + L.rstd_off) : nullptr;
  const bool stop = L.stop_at_yrht != 0, accumulate = L.y_accumulate != 0;
  // (the sums in rht_out_body's order, which is another one where it loads groups of four: the same bits)
  auto load = [&](auto in_fours, int e0, float (&v)[8]) {
    constexpr bool fours = decltype(in_fours)::value;
#pragma unroll
    for (int k = 0; k < 8; ++k) v[k] = 0.f;
    for (int kk = 0; kk < S; ++kk) {
      if (stop && kk != max(it.sub, 0)) continue;
      const float sg = !stop && (__popc(max(it.sub, 0) & kk) & 1) ? -1.f : 1.f;
      float t[8];
      int cnt[8], most = 0;
#pragma unroll
      for (int k = 0; k < 8; ++k) {
        const int e = e0 + (k << 10), row = off + (kk << FHT_LOG) + (e & ((1 << log_t) - 1));
        cnt[k] = e < total && row < m ? slots_of(row) : 0;
        most = max(most, cnt[k]);
        t[k] = fours ? v[k] : 0.f;
      }
      for (int s = 0; s < most; ++s) {
        float q[8];
#pragma unroll
        for (int k = 0; k < 8; ++k) {
          const int e = e0 + (k << 10), row = off + (kk << FHT_LOG) + (e & ((1 << log_t) - 1));
          q[k] = s < cnt[k] ? __ldcg(src + s * slot_stride + (long long)(it.tok0 + (e >> log_t)) * m + row) : 0.f;
        }
#pragma unroll
        for (int k = 0; k < 8; ++k) t[k] = fours ? fmaf(q[k], sg, t[k]) : t[k] + q[k];
      }
#pragma unroll
      for (int k = 0; k < 8; ++k) v[k] = fours ? t[k] : fmaf(t[k] * wscale, sg, v[k]);
    }
    if (fours)
#pragma unroll
      for (int k = 0; k < 8; ++k) v[k] *= wscale;
  };
  auto store = [&](int e, float v) {
    const int token = it.tok0 + (e >> log_t), row = off + run0 + (e & ((1 << log_t) - 1));
    const long long o = L.y_off + (long long)token * L.y_stride + row;
    if (stop) {
      if (row < m) reinterpret_cast<float*>(y_base)[o] = v;
    } else if (row < L.out_f) {
      float r = v * (rstd ? rs * rstd[token] : rs) * __half2float(L.su[row]);
      if (accumulate) r += load_act(y_base, o, L.y_dtype);            // residual add
      store_act(y_base, o, L.y_dtype, r);
    }
  };
  pdl_wait();
  if (!stop && ((m | off) & 3) == 0 && log_t >= 2)
    fht_wide(fbuf, log_t, total, [&](int e0, float (&v)[8]) { load(IntC<1>(), e0, v); }, store);
  else
    fht_wide(fbuf, stop ? 0 : log_t, total, [&](int e0, float (&v)[8]) { load(IntC<0>(), e0, v); }, store);
}

// The prefill case: partial sums in a fixed number of slots, whole blocks, aligned rows, no per-row scales or residual.
// Addresses are one base per thread plus offsets all threads share, the scales are folded into one.
template <bool FROM_F32>
__device__ __forceinline__ bool rht_out_is_plain(const DevLinear& L, const RhtItem& it, const uint8_t* y_base, const float* src) {
  const int off = L.bm_off[it.block], bs = 1 << L.bm_log[it.block];
  return !L.stop_at_yrht && ((L.m | off) & 3) == 0 && bs >= 4 && (FROM_F32 || L.fixed_slots > 0) && it.sub < 0 && !L.row_scale &&
         !L.y_accumulate && !(L.in_norm_w && !L.xr_global) && off + bs <= L.out_f && (reinterpret_cast<uintptr_t>(L.su) & 7) == 0 &&
         (reinterpret_cast<uintptr_t>(src) & 15) == 0 && act_rows_aligned4(y_base, L.y_off, L.y_stride, L.y_dtype);
}
template <bool FROM_F32>
__device__ __forceinline__ void rht_out_plain(const DevLinear& L, const RhtItem it, const float* __restrict__ src,
                                              uint8_t* __restrict__ y_base, float* fbuf) {
  const int off = L.bm_off[it.block], log_t = L.bm_log[it.block], m = L.m;
  const int total = it.ntok << log_t, slots = FROM_F32 ? 1 : L.fixed_slots;
  const long long slot_stride = (long long)L.batch * m;
  auto load = [&](int e0, f2 (&v)[8][2]) {
    const float* p = src + (long long)(it.tok0 + (e0 >> log_t)) * m + off + (e0 & ((1 << log_t) - 1));
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      v[k][0] = v[k][1] = 0;
      if (e0 + (k << 10) < total) {
        const ulonglong2 t = __ldcg(reinterpret_cast<const ulonglong2*>(p + fht_row(k, 1024, log_t) * m + fht_col(k, 1024, log_t)));
        v[k][0] = t.x; v[k][1] = t.y;
      }
    }
    for (int s = 1; s < slots; ++s) {
      p += slot_stride;
#pragma unroll
      for (int k = 0; k < 8; ++k)
        if (e0 + (k << 10) < total) {
          const ulonglong2 t = __ldcg(reinterpret_cast<const ulonglong2*>(p + fht_row(k, 1024, log_t) * m + fht_col(k, 1024, log_t)));
          v[k][0] = f2_add(v[k][0], t.x); v[k][1] = f2_add(v[k][1], t.y);
        }
    }
  };
  auto store = [&](int e1, const f2 (&v)[8][2]) {
    const float sc = FROM_F32 ? rsqrtf((float)(1 << log_t)) : rsqrtf((float)(1 << log_t)) * L.wscale;
    const int i0 = off + (e1 & ((1 << log_t) - 1));
    const long long y_stride = L.y_stride, o = L.y_off + (long long)(it.tok0 + (e1 >> log_t)) * y_stride + i0;
    const __half* sp = L.su + i0;
    const f2 sc2 = f2_pack(sc, sc);
    with_dtype(L.y_dtype, [&](auto dt) {
#pragma unroll
      for (int k = 0; k < 8; ++k)
        if (e1 + (k << 7) < total) {
          f2 s[2];
          float r[4];
          load_sign4(sp + fht_col(k, 128, log_t), s);
          f2_unpack(f2_mul(f2_mul(v[k][0], sc2), s[0]), r[0], r[1]);
          f2_unpack(f2_mul(f2_mul(v[k][1], sc2), s[1]), r[2], r[3]);
          store_act4(y_base, o + fht_row(k, 128, log_t) * y_stride + fht_col(k, 128, log_t), decltype(dt)::value, r);
        }
    });
  };
  fht_block_all(fbuf, log_t, total, load, store);
}
// 64 registers: four CTAs per SM, which the latency of a tile (load, two exchanges, store) needs more than registers
static __global__ void __launch_bounds__(RHT_THREADS, 4) rht_out_plain_kernel(const DevLinear* __restrict__ layers,
                                                              const RhtItem* __restrict__ items,
                                                              const uint8_t* __restrict__ ws,
                                                              uint8_t* __restrict__ y_base, int tokens) {
  extern __shared__ __align__(16) float fbuf[];
  pdl_trigger();
  pdl_wait();
  RhtItem it = items[blockIdx.x];
  if (!rht_item_trim(it, tokens)) return;
  const DevLinear& L = layers[it.layer];
  rht_out_plain<false>(L, it, reinterpret_cast<const float*>(ws + L.part_off), y_base, fbuf);
}

template <bool WIDE>
__global__ void __launch_bounds__(RHT_THREADS, RHT_MINB) rht_out_kernel(const DevLinear* __restrict__ layers,
                                                              const RhtItem* __restrict__ items,
                                                              const uint8_t* __restrict__ ws,
                                                              uint8_t* __restrict__ y_base,
                                                              const float* __restrict__ yrht_in, int tokens) {
  extern __shared__ __align__(16) float fbuf[];
  pdl_trigger();
  pdl_wait();
  RhtItem it = items[blockIdx.x];
  if (rht_item_trim(it, tokens)) rht_out_body<false, WIDE>(layers[it.layer], it, ws, y_base, yrht_in, fbuf);
}

// One array of 32 to 1024 values of the unfused op: the shuffle transform (one token of 1024 values 2.3 us; fht_block, whose
// second pass is one warp's at that size, 3.7; 64 tokens, a CTA each, 2.4 and 4.0).
__device__ __forceinline__ void rht_out_short(const DevLinear& L, const RhtItem it, const float* __restrict__ src,
                                              uint8_t* __restrict__ y_base, float* fbuf) {
  const int off = L.bm_off[it.block], logbs = L.bm_log[it.block];
  const float* p = src + (long long)it.tok0 * L.m + off;
  const __half* su = L.su + off;
  const long long o = L.y_off + (long long)it.tok0 * L.y_stride + off;
  const float rs = rsqrtf((float)(1 << logbs));
  auto load = [&](int i, auto& v) {
    constexpr int E = sizeof(v) / sizeof(float);
    if constexpr (E >= 4) {
#pragma unroll
      for (int q = 0; q < E; q += 4) {
        const float4 t = __ldcg(reinterpret_cast<const float4*>(p + i + q));
        v[q] = t.x; v[q + 1] = t.y; v[q + 2] = t.z; v[q + 3] = t.w;
      }
    } else {
#pragma unroll
      for (int q = 0; q < E; ++q) v[q] = __ldcg(p + i + q);
    }
  };
  fht_fast<10, 64, false>(fbuf, logbs, load, [&](int i) { return __half2float(su[i]); },
                          [&](int i, float v, float sign) { store_act(y_base, o + i, L.y_dtype, v * rs * sign); });
}

static __global__ void __launch_bounds__(RHT_THREADS, RHT_MINB) rht_out_single_kernel(const __grid_constant__ DevLinear L,
                                                                     const __grid_constant__ RhtSingle S,
                                                                     uint8_t* __restrict__ y_base,
                                                                     const float* __restrict__ yrht_in) {
  extern __shared__ __align__(16) float fbuf[];
  const RhtItem it = rht_single_item(S, L.batch);
  const int logbs = L.bm_log[it.block];
  if (rht_out_is_plain<true>(L, it, y_base, yrht_in)) {
    if (it.ntok == 1 && logbs >= 5 && logbs <= 10) rht_out_short(L, it, yrht_in, y_base, fbuf);
    else rht_out_plain<true>(L, it, yrht_in, y_base, fbuf);
  } else rht_out_body<true, true>(L, it, nullptr, y_base, yrht_in, fbuf);
}

}  // namespace glqb
