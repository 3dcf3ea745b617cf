// Walsh-Hadamard transform of one array by one CTA with shuffles, for the single-launch decode kernels.
#pragma once
#include "glqb_internal.h"

namespace glqb {

__device__ __forceinline__ int fht_pad(int i) { return i + (i >> 5); }
template <int R>
__device__ __forceinline__ void fht_regs(float (&v)[1 << R]) {
#pragma unroll
  for (int s = 0; s < R; ++s) {
#pragma unroll
    for (int k = 0; k < (1 << R); ++k) {
      if (!(k & (1 << s))) {
        const float a = v[k], b = v[k | (1 << s)];
        v[k] = a + b;
        v[k | (1 << s)] = a - b;
      }
    }
  }
}

// ---------------------------------------------------------------------------------------------------
// Low-latency transform of ONE array of 32 .. 8192 values by a 256-thread CTA, for the single-launch decode
// kernel where the transform sits on the critical path of a few-microsecond kernel: one round of global
// loads, one shared-memory exchange, one __syncthreads.
//   thread t holds E = max(1, bs / 256) consecutive values (index t * E + j): stages 0 .. log2(E) - 1 run in
//   registers, the next five across the lanes of a warp with shuffles, the last log2(W) (W = warps holding the
//   array, at most 8) after an exchange through shared memory, where a thread gathers the W values that differ
//   in the warp bits, finishes the butterflies and hands every finished value to `store(i, value)`; for a fixed
//   call of `store` the lanes of a warp hold consecutive i.
// `smem` needs bs + bs / 32 floats (index i lives at i + i / 32).  All 256 threads must call; `load(i0, v)` fills v[0..E) with values
// i0 .. i0 + E - 1.
// What `store` needs besides the transformed value (a sign) is requested by `pre(i)` for exactly the indices the thread
// will store: up front, so that it arrives while the transform runs, or, with LATE values per thread and more, once the
// values sit in shared memory and have left their registers free.  PACK: `pre` gives fp16 and two are kept per register,
// else fp32.  (Both kinds of register cost spills in kernels that hold prefetched codes, see fused_out_block.)
// ---------------------------------------------------------------------------------------------------
template <int E, int LATE, bool PACK, class Load, class Pre, class Store>
__device__ __forceinline__ void fht_fast_e(float* smem, int logbs, Load& load, Pre& pre, Store& store) {
  constexpr int LOGE = E == 1 ? 0 : E == 2 ? 1 : E == 4 ? 2 : E == 8 ? 3 : E == 16 ? 4 : 5;
  constexpr int QMAX = E >= 8 ? E / 8 : 1;         // rounds of the final loop (values per warp / 256)
  const int bs = 1 << logbs;
  const int t = threadIdx.x, lane = t & 31;
  const int nthreads = bs >> LOGE;                 // threads that hold values (32 .. 256)
  const int W = nthreads >> 5;                     // warps that hold values (1 .. 8)
  const bool active = t < nthreads;
  const int span = 32 << LOGE;                     // values per warp = distance between the W partners
  uint32_t aux[QMAX][PACK ? 4 : 8];
  auto aux_of = [](const uint32_t (&a)[PACK ? 4 : 8], int w) -> float {
    if constexpr (PACK) return __half2float(__ushort_as_half((unsigned short)(a[w >> 1] >> ((w & 1) * 16))));
    else return __uint_as_float(a[w]);
  };
  auto request = [&]() {
    if (W == 1) {
      if (active) {
#pragma unroll
        for (int j = 0; j < E; ++j) {                                  // E <= 1 here (32 values, one warp)
          if constexpr (PACK) aux[0][0] = __half_as_ushort(pre(t * E + j));
          else aux[0][j & 7] = __float_as_uint(pre(t * E + j));
        }
      }
      return;
    }
#pragma unroll
    for (int q = 0; q < QMAX; ++q) {
      const int r = t + 256 * q;
#pragma unroll
      for (int w = 0; w < 8; ++w) {
        if constexpr (PACK) {
          if (w & 1) continue;
          const __half z = __ushort_as_half(0), lo = (r < span && w < W) ? pre(w * span + r) : z;
          const __half hi = (r < span && w + 1 < W) ? pre((w + 1) * span + r) : z;
          aux[q][w >> 1] = (uint32_t)__half_as_ushort(lo) | ((uint32_t)__half_as_ushort(hi) << 16);
        } else {
          aux[q][w] = __float_as_uint((r < span && w < W) ? pre(w * span + r) : 0.f);
        }
      }
    }
  };
  if constexpr (E < LATE) request();
  float v[E];
  if (active) {
    load(t * E, v);
    fht_regs<LOGE>(v);
#pragma unroll
    for (int k = 0; k < 5; ++k) {
      const bool upper = (lane >> k) & 1;
#pragma unroll
      for (int j = 0; j < E; ++j) {
        const float p = __shfl_xor_sync(0xffffffffu, v[j], 1 << k);
        v[j] = upper ? (p - v[j]) : (v[j] + p);    // lower index: a + b, upper index: a - b (a = lower element)
      }
    }
  }
  if (W == 1) {
    if (active) {
#pragma unroll
      for (int j = 0; j < E; ++j) store(t * E + j, v[j], aux_of(aux[0], j & 7));
    }
    return;
  }
  if (active) {
#pragma unroll
    for (int j = 0; j < E; ++j) smem[fht_pad(t * E + j)] = v[j];
  }
  if constexpr (E >= LATE) request();
  __syncthreads();
  const int logw = W == 2 ? 1 : W == 4 ? 2 : 3;
#pragma unroll
  for (int q = 0; q < QMAX; ++q) {
    const int r = t + 256 * q;
    if (r < span) {
      float u[8];
#pragma unroll
      for (int w = 0; w < 8; ++w) u[w] = w < W ? smem[fht_pad(w * span + r)] : 0.f;
      if (logw == 1) {
        const float a = u[0], b = u[1];
        u[0] = a + b; u[1] = a - b;
      } else if (logw == 2) {
        float h[4] = {u[0], u[1], u[2], u[3]};
        fht_regs<2>(h);
        u[0] = h[0]; u[1] = h[1]; u[2] = h[2]; u[3] = h[3];
      } else {
        fht_regs<3>(u);
      }
#pragma unroll
      for (int w = 0; w < 8; ++w)
        if (w < W) store(w * span + r, u[w], aux_of(aux[q], w));
    }
  }
}

// dispatch on the array length (2^logbs, 32 .. 8192)
// load(i0, float (&v)[E]) -> values i0 .. i0 + E - 1 (i0 a multiple of E): a thread's values in one call, so that their loads
// can all be in flight;  pre(i) -> what store(i, value, x) gets as x (fp32; PACK: given as fp16)
template <int MAXLOG, int LATE, bool PACK, class Load, class Pre, class Store>
__device__ __forceinline__ void fht_fast(float* smem, int logbs, Load load, Pre pre, Store store) {
  // arrays longer than 2^MAXLOG never reach this instantiation (their cases are not compiled)
  if (logbs == 9) { fht_fast_e<2, LATE, PACK>(smem, logbs, load, pre, store); return; }
  if (logbs == 10) { fht_fast_e<4, LATE, PACK>(smem, logbs, load, pre, store); return; }
  if constexpr (MAXLOG >= 11) if (logbs == 11) { fht_fast_e<8, LATE, PACK>(smem, logbs, load, pre, store); return; }
  if constexpr (MAXLOG >= 12) if (logbs == 12) { fht_fast_e<16, LATE, PACK>(smem, logbs, load, pre, store); return; }
  if constexpr (MAXLOG >= 13) if (logbs == 13) { fht_fast_e<32, LATE, PACK>(smem, logbs, load, pre, store); return; }
  fht_fast_e<1, LATE, PACK>(smem, logbs, load, pre, store);                       // 32 .. 256 values
}
constexpr int FHT_FAST_MAX_LOG = 13;

}  // namespace glqb
