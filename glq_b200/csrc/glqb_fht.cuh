// In-CTA Walsh-Hadamard transform on a shared-memory buffer.
// Butterfly order follows the reference (glq/hadamard.py:18-26, glq/csrc/glq_fht.cuh:14-21):
// stages in ascending distance 1,2,4,...; the lower index of a pair receives a+b, the upper a-b.
// The caller applies the 1/sqrt(bs) normalisation.
#pragma once
#include "glqb_internal.h"

namespace glqb {

template <int R>   // R = number of stages done in registers this pass (1..3)
__device__ __forceinline__ void fht_pass(float* buf, int bs, int done) {
  constexpr int N = 1 << R;
  const int stride = 1 << done;
  const int ngroups = bs >> R;
  for (int o = threadIdx.x; o < ngroups; o += blockDim.x) {
    const int low = o & (stride - 1);
    const int high = o >> done;
    const int base = (high << (done + R)) | low;
    float v[N];
#pragma unroll
    for (int k = 0; k < N; ++k) v[k] = buf[base + k * stride];
#pragma unroll
    for (int s = 0; s < R; ++s) {
#pragma unroll
      for (int k = 0; k < N; ++k) {
        if (!(k & (1 << s))) {
          float a = v[k], b = v[k | (1 << s)];
          v[k] = a + b;
          v[k | (1 << s)] = a - b;
        }
      }
    }
#pragma unroll
    for (int k = 0; k < N; ++k) buf[base + k * stride] = v[k];
  }
}

// All threads of the CTA must call this; buf holds bs = 2^logbs floats and is fully written.
__device__ __forceinline__ void fht_smem(float* buf, int logbs) {
  const int bs = 1 << logbs;
  int done = 0;
  __syncthreads();
  while (done < logbs) {
    const int r = min(3, logbs - done);
    if (r == 3) fht_pass<3>(buf, bs, done);
    else if (r == 2) fht_pass<2>(buf, bs, done);
    else fht_pass<1>(buf, bs, done);
    __syncthreads();
    done += r;
  }
}

}  // namespace glqb

// ---------------------------------------------------------------------------------------------------
// Tile transform of the transform kernels, the grouped-expert kernels and the single-launch decode kernels.
//
// A tile is up to 8192 values held by 256 threads, 32 per thread: `total` = rows << logbs values, value e being
// element e & (bs - 1) of row e >> logbs, each row of bs = 2^logbs (1 .. 8192) values transformed by itself.
// The 13 bits of e are taken in three register passes:
//   1  e = k << 10 | warp << 7 | lane << 2 | j     bits 0, 1 and 10 .. 12, straight from the caller's loads
//   2  e = warp << 10 | (lane >> 2) << 7 | r << 2 | (lane & 3)                    bits 2 .. 6
//   3  e = warp << 10 | k << 7 | lane << 2 | j                                    bits 7 .. 9, handed to the stores
// so every global access is four consecutive values per thread and 128 per warp (the earlier form loaded 32
// consecutive values per thread: 32 half-used sectors per warp instruction), pass 2 -> 3 stays inside a warp and
// one block barrier remains.  Shared memory is padded by four words per 128 values, which makes the 16-byte
// accesses of passes 1 and 3 and the stride-4 accesses of pass 2 conflict-free.  Butterflies run on packed fp32
// pairs (add / fma .f32x2, the same roundings as the scalar forms).  Bound by the latency of a tile (long-scoreboard
// stalls; issue slots 33 % busy where the earlier form had 51 instructions per value and 50 %).  Measured, warm caches:
// output transform 2048 x 11008 70 -> 43 us, 21504 columns x 700 tokens of input 57 -> 37 us, one token of 14336 outputs
// 49 -> 14 us.
// ---------------------------------------------------------------------------------------------------
namespace glqb {

typedef unsigned long long f2;                   // two packed fp32
__device__ __forceinline__ f2 f2_pack(float lo, float hi) {
  f2 r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
  return r;
}
__device__ __forceinline__ void f2_unpack(f2 v, float& lo, float& hi) { asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v)); }
__device__ __forceinline__ f2 f2_add(f2 a, f2 b) {
  f2 r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ f2 f2_mul(f2 a, f2 b) {
  f2 r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ f2 f2_fma(f2 a, f2 b, f2 c) {
  f2 r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
  return r;
}
constexpr f2 F2_MINUS1 = 0xBF800000BF800000ull, F2_ONE = 0x3F8000003F800000ull;
// (a, b) <- (a + b, a - b), both pairs at once; a - b as fma(b, -1, a): one rounding, the same value
__device__ __forceinline__ void f2_butterfly(f2& a, f2& b) {
  const f2 s = f2_add(a, b);
  b = f2_fma(b, F2_MINUS1, a);
  a = s;
}
// the butterfly inside one pair
__device__ __forceinline__ void f2_cross(f2& v) {
  float lo, hi;
  f2_unpack(v, lo, hi);
  v = f2_pack(lo + hi, lo - hi);
}

constexpr int FHT_LOG = 13;                      // largest array of a tile; longer blocks: RhtItem::sub
constexpr int FHT_THREADS = 256;
__host__ __device__ __forceinline__ int fht_pos(int e) { return e + ((e >> 7) << 2); }
__host__ __device__ __forceinline__ int fht_words(int total) { return ((total + 127) >> 7) * 132; }

__device__ __forceinline__ void fht_ld4(const float* p, f2 (&v)[2]) {
  const ulonglong2 t = *reinterpret_cast<const ulonglong2*>(p);
  v[0] = t.x; v[1] = t.y;
}
__device__ __forceinline__ void fht_st4(float* p, const f2 (&v)[2]) { *reinterpret_cast<ulonglong2*>(p) = make_ulonglong2(v[0], v[1]); }

// Element offset of a thread's k-th group of four from its first one, in a matrix of `stride` elements per row; `step`
// is 1024 when loading and 128 when storing.  (The bits of k * step and of the first group's index are disjoint, so
// row and column add up; the offsets are the same for all threads.)
__device__ __forceinline__ int fht_row(int k, int step, int logbs) { return (k * step) >> logbs; }
__device__ __forceinline__ int fht_col(int k, int step, int logbs) { return (k * step) & ((1 << logbs) - 1); }

// load(e0, v): v[k] <- values e0 + 1024 k .. + 3 of the tile (zero past `total`); store(e1, v): takes the finished values
// e1 + 128 k .. + 3 (those below `total`).  `sm`: fht_words(total) floats, 16-byte aligned.  All 256 threads call; a
// caller that reuses `sm` puts a barrier in between.
// LOG >= 0: logbs known at compile time (stages behind a runtime test cost a select per value and stage: 2 x the
// instructions of the whole transform).
template <int LOG, class Load, class Store>
__device__ __forceinline__ void fht_block_t(float* sm, int logbs_, int total, Load load, Store store) {
  const int logbs = LOG >= 0 ? LOG : logbs_;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  f2 v[8][2];
  const int e0 = (warp << 7) | (lane << 2);
  load(e0, v);
  if (logbs > 0) {
#pragma unroll
    for (int k = 0; k < 8; ++k) { f2_cross(v[k][0]); f2_cross(v[k][1]); }
  }
  if (logbs > 1) {
#pragma unroll
    for (int k = 0; k < 8; ++k) f2_butterfly(v[k][0], v[k][1]);
  }
#pragma unroll
  for (int s = 0; s < 3; ++s)
    if (logbs > 10 + s) {
#pragma unroll
      for (int k = 0; k < 8; ++k)
        if (!(k & (1 << s))) { f2_butterfly(v[k][0], v[k | (1 << s)][0]); f2_butterfly(v[k][1], v[k | (1 << s)][1]); }
    }
#pragma unroll
  for (int k = 0; k < 8; ++k)
    if (e0 + (k << 10) < total) fht_st4(sm + fht_pos(e0) + k * (1024 + 32), v[k]);
  __syncthreads();
  if ((warp << 10) >= total) return;
  if (logbs > 2) {
    float* p = sm + fht_pos((warp << 10) | ((lane >> 2) << 7)) + (lane & 3);
    if (((warp << 10) | ((lane >> 2) << 7)) < total) {
      f2 w[16];                                  // pair i = (r = 2 i, 2 i + 1)
#pragma unroll
      for (int i = 0; i < 16; ++i) w[i] = f2_pack(p[8 * i], p[8 * i + 4]);
#pragma unroll
      for (int i = 0; i < 16; ++i) f2_cross(w[i]);
#pragma unroll
      for (int s = 0; s < 4; ++s)
        if (logbs > 3 + s) {
#pragma unroll
          for (int i = 0; i < 16; ++i)
            if (!(i & (1 << s))) f2_butterfly(w[i], w[i | (1 << s)]);
        }
#pragma unroll
      for (int i = 0; i < 16; ++i) {
        float lo, hi;
        f2_unpack(w[i], lo, hi);
        p[8 * i] = lo;
        p[8 * i + 4] = hi;
      }
    }
    __syncwarp();
  }
  const int e1 = (warp << 10) | (lane << 2);
#pragma unroll
  for (int k = 0; k < 8; ++k)
    if (e1 + (k << 7) < total) fht_ld4(sm + fht_pos(e1) + k * 132, v[k]);
    else { v[k][0] = 0; v[k][1] = 0; }
#pragma unroll
  for (int s = 0; s < 3; ++s)
    if (logbs > 7 + s) {
#pragma unroll
      for (int k = 0; k < 8; ++k)
        if (!(k & (1 << s))) { f2_butterfly(v[k][0], v[k | (1 << s)][0]); f2_butterfly(v[k][1], v[k | (1 << s)][1]); }
    }
  store(e1, v);
}

template <class Load, class Store>
__device__ __forceinline__ void fht_block_all(float* sm, int logbs, int total, Load load, Store store) {
  switch (logbs) {
    case 13: fht_block_t<13>(sm, logbs, total, load, store); break;
    case 12: fht_block_t<12>(sm, logbs, total, load, store); break;
    case 11: fht_block_t<11>(sm, logbs, total, load, store); break;
    case 10: fht_block_t<10>(sm, logbs, total, load, store); break;
    case 9: fht_block_t<9>(sm, logbs, total, load, store); break;
    case 8: fht_block_t<8>(sm, logbs, total, load, store); break;
    default: fht_block_t<-1>(sm, logbs, total, load, store); break;
  }
}

// the same with a store(e, q) per group of four and one body for all lengths
template <class Load, class Store>
__device__ __forceinline__ void fht_block(float* sm, int logbs, int total, Load load, Store store) {
  fht_block_t<-1>(sm, logbs, total, load, [&](int e1, const f2 (&v)[8][2]) {
#pragma unroll
    for (int k = 0; k < 8; ++k)
      if (e1 + (k << 7) < total) store(e1 + (k << 7), v[k]);
  });
}

// The tile transform for launches of few tiles, where the latency of one tile is the launch's: 1024 threads with eight values
// each instead of 256 with 32, single values instead of groups of four (no alignment to ask for).  Passes:
//   1  e = k << 10 | warp << 5 | lane     bits 10 .. 12 in registers, 0 .. 4 across the lanes
//   2  e = warp << 8 | k << 5 | lane      bits 5 .. 7
//   3  e = (warp >> 3) << 11 | k << 8 | (warp & 7) << 5 | lane      bits 8 and 9
// so every access, global or shared, is 32 consecutive values per warp.  The stages come in fht_block's order (0, 1, 10 .. 12,
// 2 .. 9), so that a value has the same bits whichever of the two computed it.  `sm`: `total` floats; load(e0, v) fills all
// eight values, those past `total` with zeros; all 1024 threads call.
constexpr int FHT_WIDE_THREADS = 1024;
template <class Load, class Store>
__device__ __forceinline__ void fht_wide(float* sm, int logbs, int total, Load load, Store store) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  float v[8];
  const int e0 = (warp << 5) | lane;
  auto stage = [&](int s) {
#pragma unroll
    for (int k = 0; k < 8; ++k)
      if (!(k & (1 << s))) {
        const float a = v[k], b = v[k | (1 << s)];
        v[k] = a + b;
        v[k | (1 << s)] = a - b;
      }
  };
  auto lanes = [&](int s) {                                // (uniform per warp)
    if (logbs > s && (e0 & ~31) < total) {
      const float sg = (lane >> s) & 1 ? -1.f : 1.f;
#pragma unroll
      for (int k = 0; k < 8; ++k) v[k] = fmaf(v[k], sg, __shfl_xor_sync(0xffffffffu, v[k], 1 << s));
    }
  };
  load(e0, v);
  lanes(0);
  lanes(1);
#pragma unroll
  for (int s = 0; s < 3; ++s)
    if (logbs > 10 + s) stage(s);
#pragma unroll
  for (int s = 2; s < 5; ++s) lanes(s);
  if (logbs <= 5) {                                        // (no stage crosses a warp)
#pragma unroll
    for (int k = 0; k < 8; ++k)
      if (e0 + (k << 10) < total) store(e0 + (k << 10), v[k]);
    return;
  }
#pragma unroll
  for (int k = 0; k < 8; ++k)
    if (e0 + (k << 10) < total) sm[e0 + (k << 10)] = v[k];
  __syncthreads();
  const int e1 = (warp << 8) | lane;
#pragma unroll
  for (int k = 0; k < 8; ++k) v[k] = e1 + (k << 5) < total ? sm[e1 + (k << 5)] : 0.f;
#pragma unroll
  for (int s = 0; s < 3; ++s)
    if (logbs > 5 + s) stage(s);
  if (logbs <= 8) {
#pragma unroll
    for (int k = 0; k < 8; ++k)
      if (e1 + (k << 5) < total) store(e1 + (k << 5), v[k]);
    return;
  }
#pragma unroll
  for (int k = 0; k < 8; ++k)
    if (e1 + (k << 5) < total) sm[e1 + (k << 5)] = v[k];
  __syncthreads();
  const int e2 = ((warp >> 3) << 11) | ((warp & 7) << 5) | lane;
#pragma unroll
  for (int k = 0; k < 8; ++k) v[k] = e2 + (k << 8) < total ? sm[e2 + (k << 8)] : 0.f;
  stage(0);
  if (logbs > 9) stage(1);
#pragma unroll
  for (int k = 0; k < 8; ++k)
    if (e2 + (k << 8) < total) store(e2 + (k << 8), v[k]);
}

// One warp, 1024 values, two register passes and no block barrier: v[k] holds values k << 7 | lane << 2 | j (bits 0, 1
// and 7 .. 9), the second pass bits 2 .. 6; arrays of 2^logbs <= 1024 values side by side (logbs >= 5).  Blocks longer
// than 1024 are 1024-value chunks whose remaining bits the consumer of the results combines.  Results: value e at
// sm[fht_pos(e)] (FHT_CHUNK_WORDS floats), visible to the warp.
constexpr int FHT_CHUNK_WORDS = 1056;
template <int LOG>
__device__ __forceinline__ void fht_warp_t(float* sm, f2 (&v)[8][2], int logbs_) {
  const int logbs = LOG >= 0 ? LOG : logbs_;
  const int lane = threadIdx.x & 31;
#pragma unroll
  for (int k = 0; k < 8; ++k) { f2_cross(v[k][0]); f2_cross(v[k][1]); f2_butterfly(v[k][0], v[k][1]); }
#pragma unroll
  for (int s = 0; s < 3; ++s)
    if (logbs > 7 + s) {
#pragma unroll
      for (int k = 0; k < 8; ++k)
        if (!(k & (1 << s))) { f2_butterfly(v[k][0], v[k | (1 << s)][0]); f2_butterfly(v[k][1], v[k | (1 << s)][1]); }
    }
#pragma unroll
  for (int k = 0; k < 8; ++k) fht_st4(sm + (lane << 2) + k * 132, v[k]);
  __syncwarp();
  float* p = sm + (lane >> 2) * 132 + (lane & 3);
  f2 w[16];
#pragma unroll
  for (int i = 0; i < 16; ++i) w[i] = f2_pack(p[8 * i], p[8 * i + 4]);
#pragma unroll
  for (int i = 0; i < 16; ++i) f2_cross(w[i]);
#pragma unroll
  for (int s = 0; s < 4; ++s)
    if (s < 2 || logbs > 3 + s) {
#pragma unroll
      for (int i = 0; i < 16; ++i)
        if (!(i & (1 << s))) f2_butterfly(w[i], w[i | (1 << s)]);
    }
#pragma unroll
  for (int i = 0; i < 16; ++i) {
    float lo, hi;
    f2_unpack(w[i], lo, hi);
    p[8 * i] = lo;
    p[8 * i + 4] = hi;
  }
  __syncwarp();
}
__device__ __forceinline__ void fht_warp(float* sm, f2 (&v)[8][2], int logbs) {
  if (logbs >= 10) fht_warp_t<10>(sm, v, logbs);
  else if (logbs == 9) fht_warp_t<9>(sm, v, logbs);
  else if (logbs == 8) fht_warp_t<8>(sm, v, logbs);
  else fht_warp_t<-1>(sm, v, logbs);
}

}  // namespace glqb
