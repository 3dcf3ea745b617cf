// Prefill and grouped experts on trellis weights: states decoded straight into tensor memory as the A operand of
// tcgen05.mma, activations streamed through shared memory.
//
// Why A goes to tensor memory: a lane of a decoding warp holds exactly the fragment layout of tcgen05.st.16x128b (row g
// and g + 8, columns 2t and 2t + 1 of every 16 x 8 block), so two stores replace sixteen and a 128 x 64 x 256 chunk leaves
// 64 KiB of shared-memory traffic instead of 96 (768 clocks at 128 bytes, where the tensor pipe needs 512).  That alone
// changed nothing (1010 -> 1045 clocks per chunk): the limit was the issuing thread's own loop, see the MMA issuer below,
// and with that loop warp-uniform a chunk took 742.
//
// One CTA computes 128 weight rows x one or two tiles of up to TN tokens: an accumulator of TN columns per tile; the other
// 512 - 2 TN columns of tensor memory are stages of A (two 64-column chunks of 32 columns each).  An item of two tiles decodes
// their weights once, both accumulators are then its own; items of one tile alternate.  Warp roles: warp 0 issues MMAs, warp 1
// the bulk copies (TMA without multicast) of the activation tiles, warp 2 joins the activations of a pair to its weights, warps
// 4-7 drain accumulators, 16 producer warps in two groups of eight
// (group p % 2 decodes pair p; warp w of a group rows 32 (w % 4) and chunk w / 4 of the pair: two 32 x 32 trellis groups).
// Experts of 4096 tokens, top 8 of 128 (256 tokens each on average), a tile of up to 192 tokens / two of up to 160 per item:
// 788 / 717 us.
// Bound by the instructions of the state decode (issue slots 76 and 73 % busy in the two matmuls with 16 routed tokens per expert, 55
// and 51 % with 256, where the tensor pipe is 56 and 43 % busy): with a loop
// turn per pair instead of per chunk a trellis group takes 229 instructions instead of 263, and 80 registers hold both
// decoded groups until the stage is free.  24 producer warps, a chunk per turn / this: experts of 256 tokens 273 / 257 us,
// 333 tokens of 2048 x 11008 80 / 76 us.
// Stages hand over through mbarriers; every wait is bounded as in glq_gemm_kernel.
#pragma once
#include "glqb_gemm.cuh"

namespace glqb {

// Buffers by the most tokens TN of a tile.  A stage is a pair of 64-column chunks: 64 columns of tensor memory; a unit of B
// is the two chunks' activations of one tile.
constexpr int TG_A_COLS = 32;                    // columns per chunk
template <int TN>
struct TgShape {
  static constexpr int A_STAGES = (512 - 2 * TN) / (2 * TG_A_COLS);       // what the two accumulators leave
  static constexpr int B_BYTES = 2 * TN * 128;
  static constexpr int B_STAGES = 220 * 1024 / B_BYTES;
  static constexpr int SMEM_BYTES = B_STAGES * B_BYTES + (2 * A_STAGES + 2 * B_STAGES + 5) * 8 + 16 + 1024;
};
constexpr int TG_GROUPS = 2;                     // producer groups
constexpr int TG_MMA_WARP = 0, TG_LOAD_WARP = 1, TG_GATE_WARP = 2, TG_EPI_WARP0 = 4, TG_PROD_WARP0 = 8;   // (3 only keeps warp % 4 aligned)
constexpr int TG_THREADS = (TG_PROD_WARP0 + TG_GROUPS * 8) * 32;

__device__ __forceinline__ void tmem_st_16x128b_x4(uint32_t taddr, const uint32_t (&r)[8]) {
  asm volatile("tcgen05.st.sync.aligned.16x128b.x4.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};" ::"r"(taddr), "r"(r[0]), "r"(r[1]),
               "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7])
               : "memory");
}
__device__ __forceinline__ void tmem_st_wait() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }
// A from tensor memory, B from shared memory
__device__ __forceinline__ void umma_f16_ta(uint32_t d_tmem, uint32_t a_tmem, uint64_t b_desc, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{ .reg .pred p; setp.ne.b32 p, %4, 0; tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p; }" ::"r"(d_tmem),
      "r"(a_tmem), "l"(b_desc), "r"(idesc), "r"(accumulate)
      : "memory");
}

// One trellis group -> the A fragments of its two 16-row halves: r[mi][(ni * 2 + c) * 2 + a] = weights (2t, 2t + 1) of
// row g + 8 a in the 16 x 8 block (ni, c).
template <int K1, int K2>
__device__ __forceinline__ void tg_decode_group(int lane, const Words<K1>& v, const Words<(K2 > 0 ? K2 : 1)>& v2, __half2 s2,
                                                uint32_t (&r)[2][8]) {
  const Words<K1> vn = shfl_words<K1>(v, (lane + 1) & 31);
  Words<K1> vn2 = vn;
  if constexpr (K1 == 1) vn2 = shfl_words<K1>(v, (lane + 2) & 31);
  Words<(K2 > 0 ? K2 : 1)> un, un2;
  if constexpr (K2 > 0) {
    un = shfl_words<K2>(v2, (lane + 1) & 31);
    un2 = un;
    if constexpr (K2 == 1) un2 = shfl_words<K2>(v2, (lane + 2) & 31);
  }
#pragma unroll
  for (int q = 0; q < 4; ++q) {                  // q = ni * 2 + mi
    uint32_t a[8], b[8];
    decode_tile<K1>(chunk_of<K1>(v, q), chunk_of<K1>(vn, q), chunk_of<K1>(vn2, q), a);
    if constexpr (K2 > 0) decode_tile<K2>(chunk_of<K2>(v2, q), chunk_of<K2>(un, q), chunk_of<K2>(un2, q), b);
#pragma unroll
    for (int p = 0; p < 4; ++p) {                // p = c * 2 + a
      uint32_t w = __byte_perm(a[2 * p], a[2 * p + 1], 0x5410);
      if constexpr (K2 > 0) {
        // second stage folded into the fp16 operand: w = fp16(w1 + s2 * w2), one rounding
        const uint32_t w2 = __byte_perm(b[2 * p], b[2 * p + 1], 0x5410);
        const __half2 z = __hfma2(*reinterpret_cast<const __half2*>(&w2), s2, *reinterpret_cast<const __half2*>(&w));
        w = *reinterpret_cast<const uint32_t*>(&z);
      }
      r[q & 1][(q >> 1) * 4 + p] = w;
    }
  }
}

// Activations of a tile: ntok rounded up to 16 rows of 128 bytes per 64-column chunk, [k chunk][row], behind the row0
// rows of the tiles before it.  An item multiplies exactly the columns it has.
template <int K1, int K2, int TN>
__global__ void __launch_bounds__(TG_THREADS, 1)
trellis_gemm_kernel(const DevLinear* __restrict__ layers, const GemmItem* __restrict__ items, int n_items,
                    uint8_t* __restrict__ ws, int* __restrict__ status, const int* __restrict__ n_items_dev, int tokens) {
  // (as in glq_gemm_kernel: no trigger; of a plan's layers the producers decode before the kernel in front of this one has completed)
  if (n_items_dev) { pdl_wait(); n_items = min(n_items, *n_items_dev); }
  // first token and tokens of an item's tile (none: every role skips the item), the activation rows in front of it, and the
  // tokens of its second tile, which lies right behind (whole tiles are multiples of 16)
  struct Tile { int tok0, ntok, row0, ntok2; };
  auto tile_of = [&](const GemmItem& it, const DevLinear& L) -> Tile {
    if (n_items_dev) return Tile{it.tok0, it.ntok, it.row0, it.ntok2};
    const int used = min(L.batch, tokens), tt = tile_tokens(used), tok0 = it.n_tile * tt;
    return Tile{tok0, min(tt, used - tok0), tok0, it.ntok2 ? max(0, min(tt, used - tok0 - tt)) : 0};
  };
  constexpr int MMA_WARP = TG_MMA_WARP, LOAD_WARP = TG_LOAD_WARP;
  constexpr int A_STAGES = TgShape<TN>::A_STAGES, B_STAGES = TgShape<TN>::B_STAGES, B_BYTES = TgShape<TN>::B_BYTES;
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  uint8_t* b_base = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
  uint64_t* bars = reinterpret_cast<uint64_t*>(b_base + B_STAGES * B_BYTES);
  uint64_t* full_a = bars;
  uint64_t* empty_a = full_a + A_STAGES;
  uint64_t* full_b = empty_a + A_STAGES;
  uint64_t* empty_b = full_b + B_STAGES;
  uint64_t* acc_full = empty_b + B_STAGES;      // [2]
  uint64_t* acc_empty = acc_full + 2;              // [2]
  uint64_t* drain = acc_empty + 2;                 // give-up path only: completion of the MMAs issued so far
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(drain + 1);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (threadIdx.x == 0) {
    for (int s = 0; s < A_STAGES; ++s) { mbar_init(&full_a[s], 9); mbar_init(&empty_a[s], 1); }
    for (int s = 0; s < B_STAGES; ++s) { mbar_init(&full_b[s], 1); mbar_init(&empty_b[s], 1); }
    for (int a = 0; a < 2; ++a) { mbar_init(&acc_full[a], 1); mbar_init(&acc_empty[a], 4); }
    mbar_init(drain, 1);
    *abort_flag = 0;
    fence_mbar_init();
  }
  if (warp == MMA_WARP) {
    tmem_alloc(tmem_slot, 512);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *tmem_slot, tmem_a = tmem + 2 * TN;
  uint32_t loads_issued = 0;                       // loader thread: stages armed so far

  if (warp == MMA_WARP) {
    // ------------------------------------------------------------------ MMA issuer
    // The whole warp walks the chunks and one elected lane issues: with warp-uniform control flow descriptors and
    // addresses stay in uniform registers, and one wait per pair is left (a producer warp hands A over only after it
    // has seen B arrive).  This loop, not the operands, was the limit: 1040 clocks per chunk with two waits per chunk
    // under a lane == 0 branch, whatever the number of tokens, 740 in this form chunk by chunk; hence pairs.
    const uint32_t d0 = __shfl_sync(0xffffffffu, tmem, 0);
    const uint32_t b0 = smem_u32(b_base);
    uint32_t q = 0, u = 0, seq = 0;                // pairs of chunks, units of B, accumulators so far
    bool ok = true;
    for (int item = blockIdx.x; item < n_items && ok; item += gridDim.x) {
      const int chunks = __shfl_sync(0xffffffffu, items[item].k_end - items[item].k_begin, 0);
      const Tile t = tile_of(items[item], layers[items[item].layer]);
      const int cols = (__shfl_sync(0xffffffffu, t.ntok, 0) + 15) & ~15, cols2 = (__shfl_sync(0xffffffffu, t.ntok2, 0) + 15) & ~15;
      if (cols <= 0) continue;
      const uint32_t idesc = umma_idesc_f16(cols), step = (uint32_t)cols * 8u, idesc2 = umma_idesc_f16(cols2), step2 = (uint32_t)cols2 * 8u;
      if (!mbar_wait(&acc_empty[seq & 1u], ((seq >> 1) & 1u) ^ 1u, abort_flag)) { ok = false; break; }
      tc_fence_after();
      for (int c = 0; c < chunks; c += 2, ++q) {
        const uint32_t sa = q % A_STAGES;
        if (!mbar_wait(&full_a[sa], (q / A_STAGES) & 1u, abort_flag)) { ok = false; break; }
        tc_fence_after();
        const uint32_t ta = d0 + 2 * TN + sa * (2 * TG_A_COLS);
        // one tile's columns: accumulator `s`, the activations of unit u, 16-byte units of a chunk's activations
        auto issue = [&](uint32_t s, uint32_t idesc, uint32_t step, bool last) {
          const uint32_t d_tmem = d0 + (s & 1u) * TN, sb = u % B_STAGES;
          const uint64_t db = umma_desc_sw128(b0 + sb * B_BYTES);
          if (elect_one()) {
#pragma unroll
            for (int k = 0; k < GM_TILE_K / 16; ++k)        // K step of 16: 8 columns of A, 32 bytes of B
              umma_f16_ta(d_tmem, ta + (uint32_t)(8 * k), db + (uint64_t)(2 * k), idesc, (c > 0 || k > 0) ? 1u : 0u);
            if (c + 1 < chunks) {
#pragma unroll
              for (int k = 0; k < GM_TILE_K / 16; ++k)
                umma_f16_ta(d_tmem, ta + (uint32_t)(TG_A_COLS + 8 * k), db + (uint64_t)(step + 2 * k), idesc, 1u);
            }
            umma_commit(&empty_b[sb]);                     // stages reusable once these MMAs have read them
            if (last) umma_commit(&empty_a[sa]);
          }
          __syncwarp();
          ++u;
        };
        issue(seq, idesc, step, cols2 <= 0);
        if (cols2 > 0) {
          if (c == 0) {
            if (!mbar_wait(&acc_empty[(seq + 1) & 1u], (((seq + 1) >> 1) & 1u) ^ 1u, abort_flag)) { ok = false; break; }
            tc_fence_after();
          }
          issue(seq + 1, idesc2, step2, true);
        }
      }
      if (!ok) break;
      if (elect_one()) {
        umma_commit(&acc_full[seq & 1u]);
        if (cols2 > 0) umma_commit(&acc_full[(seq + 1) & 1u]);
      }
      __syncwarp();
      seq += cols2 > 0 ? 2u : 1u;
    }
    if (!ok) { *abort_flag = 1; if (lane == 0) atomicCAS(status, 0, (int)ST_GAVE_UP_MMA); }
  } else if (warp == LOAD_WARP) {
    // ------------------------------------------------------------------ activation loader
    if (lane == 0) {
      pdl_wait();
      uint32_t q = 0;
      bool ok = true;
      for (int item = blockIdx.x; item < n_items && ok; item += gridDim.x) {
        const GemmItem it = items[item];
        const DevLinear& L = layers[it.layer];
        const int kchunks = (L.n + GM_TILE_K - 1) / GM_TILE_K;
        const Tile t = tile_of(it, L);
        if (t.ntok <= 0) continue;
        const uint8_t* src = ws + L.xr_off + (size_t)t.row0 * kchunks * 128;
        const uint8_t* src2 = src + (size_t)t.ntok * kchunks * 128;
        auto load = [&](const uint8_t* p, int ntok, int kc) -> bool {
          const uint32_t bytes = (uint32_t)((ntok + 15) & ~15) * 128u, n = kc + 1 < it.k_end ? 2u * bytes : bytes, sb = q % B_STAGES;
          if (!mbar_wait(&empty_b[sb], ((q / B_STAGES) & 1u) ^ 1u, abort_flag)) return false;
          mbar_expect_tx(&full_b[sb], n);
          bulk_g2s(b_base + sb * B_BYTES, p + (size_t)kc * bytes, n, &full_b[sb]);
          ++loads_issued;
          ++q;
          return true;
        };
        for (int kc = it.k_begin; kc < it.k_end && ok; kc += 2)
          ok = load(src, t.ntok, kc) && (t.ntok2 <= 0 || load(src2, t.ntok2, kc));
      }
      if (!ok) { *abort_flag = 1; atomicCAS(status, 0, (int)ST_GAVE_UP_LOADER); }
    }
  } else if (warp == TG_GATE_WARP) {
    // ------------------------------------------------------------------ gate
    // The ninth arrival at a stage of A: the pair's activations are there.  So the MMA warp waits once per pair, and the
    // producers, who hand over the rest, do not wait for activations.
    if (lane == 0) {
      uint32_t p = 0, u = 0;
      bool ok = true;
      for (int item = blockIdx.x; item < n_items && ok; item += gridDim.x) {
        const GemmItem it = items[item];
        const Tile t = tile_of(it, layers[it.layer]);
        if (t.ntok <= 0) continue;
        const int units = t.ntok2 > 0 ? 2 : 1;
        for (int kc = it.k_begin; kc < it.k_end && ok; kc += 2, ++p) {
          const uint32_t stage = p % A_STAGES;
          ok = mbar_wait(&empty_a[stage], ((p / A_STAGES) & 1u) ^ 1u, abort_flag);
          for (int i = 0; i < units && ok; ++i, ++u) ok = mbar_wait(&full_b[u % B_STAGES], (u / B_STAGES) & 1u, abort_flag);
          if (ok) mbar_arrive(&full_a[stage]);
        }
      }
      if (!ok) { *abort_flag = 1; atomicCAS(status, 0, (int)ST_GAVE_UP_LOADER); }
    }
  } else if (warp >= TG_PROD_WARP0) {
    // ------------------------------------------------------------------ producers
    // Group g takes pairs g, g + 2, ... of this CTA (counted over all its items).  A warp
    // decodes both 32 x 32 groups of one chunk of the pair before it asks for the stage, so that a stage is held for
    // the stores alone.
    const int grp = (warp - TG_PROD_WARP0) >> 3, strip = warp & 3, half = (warp >> 2) & 1;
    const uint32_t dst0 = tmem_a + ((uint32_t)(strip * 32) << 16) + (uint32_t)(half * TG_A_COLS);
    uint32_t p0 = 0;                               // pairs of the items before
    bool ok = true;
    for (int item = blockIdx.x; item < n_items && ok; item += gridDim.x) {
      const GemmItem it = items[item];
      const DevLinear& L = layers[it.layer];
      if (tile_of(it, L).ntok <= 0) continue;
      const int rp = it.m_tile * 4 + strip, gps = L.groups_per_strip, k_end = it.k_end;
      const bool row_ok = rp < L.strips;
      // chunks below k_both have two groups, chunk k_both may have one (columns past the matrix are zeros)
      const int k_both = row_ok ? min(k_end, gps >> 1) : 0, k_any = row_ok ? k_end : 0;
      int kc = it.k_begin + 2 * (int)((grp ^ p0) & 1u) + half;
      const uint8_t* p1 = L.codes[0] + ((long long)rp * gps + 2 * kc) * (128 * K1) + lane * (4 * K1);
      const uint8_t* p2 = nullptr;
      if constexpr (K2 > 0) p2 = L.codes[1] + ((long long)rp * gps + 2 * kc) * (128 * K2) + lane * (4 * K2);
      const __half2 s2 = __float2half2_rn(L.stage_scale[1]);
      Words<K1> v[2];
      Words<(K2 > 0 ? K2 : 1)> v2[2];
      auto fetch = [&](int g) {
        v[g] = load_words<K1>(p1 + g * (128 * K1));
        if constexpr (K2 > 0) v2[g] = load_words<K2>(p2 + g * (128 * K2));
      };
      if (kc < k_any) fetch(0);
      if (kc < k_both) fetch(1);
      const int pairs = (k_end - it.k_begin + 1) >> 1;
      for (int pair = (int)((grp ^ p0) & 1u); pair < pairs; pair += 2, kc += 4) {
        const uint32_t q = p0 + (uint32_t)pair, stage = q % A_STAGES, dst = dst0 + stage * (2 * TG_A_COLS);
        p1 += 8 * (128 * K1);                      // the codes of this warp's next chunk
        if constexpr (K2 > 0) p2 += 8 * (128 * K2);
        auto decode = [&](int g, int k_lim, uint32_t (&r)[2][8]) {
          if (kc < k_lim) {                        // (uniform per warp: the shuffles inside see all lanes)
            tg_decode_group<K1, K2>(lane, v[g], v2[g], s2, r);
            if (kc + 4 < k_lim) fetch(g);
          } else {                                 // rows or columns past the matrix: zeros
#pragma unroll
            for (int i = 0; i < 16; ++i) r[i >> 3][i & 7] = 0u;
          }
        };
        auto wait = [&]() -> bool {
          if (!mbar_wait(&empty_a[stage], ((q / A_STAGES) & 1u) ^ 1u, abort_flag)) return false;
          __syncwarp();
          tc_fence_after();
          return true;
        };
        auto put = [&](int g, const uint32_t (&r)[2][8]) {
          tmem_st_16x128b_x4(dst + (uint32_t)(g * 16), r[0]);
          tmem_st_16x128b_x4(dst + (16u << 16) + (uint32_t)(g * 16), r[1]);
        };
        if constexpr (K2 == 0) {
          uint32_t r[2][2][8];
          decode(0, k_any, r[0]);
          decode(1, k_both, r[1]);
          if (!wait()) { ok = false; break; }
          put(0, r[0]);
          put(1, r[1]);
        } else {                                   // (two stages: no registers for both groups)
          uint32_t r[2][8];
          decode(0, k_any, r);
          if (!wait()) { ok = false; break; }
          put(0, r);
          decode(1, k_both, r);
          put(1, r);
        }
        tmem_st_wait();
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(&full_a[stage]);
      }
      p0 += (uint32_t)pairs;
    }
    if (!ok) { *abort_flag = 1; if (lane == 0) atomicCAS(status, 0, (int)ST_GAVE_UP_PRODUCER); }
  } else if (warp >= TG_EPI_WARP0) {
    // ------------------------------------------------------------------ epilogue warps
    pdl_wait();
    const int quarter = warp & 3;                          // TMEM lanes 32*quarter .. 32*quarter + 31
    uint32_t seq = 0;
    bool ok = true;
    for (int item = blockIdx.x; item < n_items && ok; item += gridDim.x) {
      const GemmItem it = items[item];
      const DevLinear& L = layers[it.layer];
      const Tile t = tile_of(it, L);
      if (t.ntok <= 0) continue;
      const int row = it.m_tile * GM_TILE_M + quarter * 32 + lane, m = L.m;
      for (int h = 0; h < (t.ntok2 > 0 ? 2 : 1); ++h, ++seq) {
        const uint32_t a = seq & 1u;
        if (!mbar_wait(&acc_full[a], (seq >> 1) & 1u, abort_flag)) { ok = false; break; }
        __syncwarp();
        tc_fence_after();
        const int cols = h ? t.ntok2 : t.ntok;
        float* part = reinterpret_cast<float*>(ws + L.part_off) + ((long long)it.slot * L.batch + t.tok0 + (h ? t.ntok : 0)) * m + row;
#pragma unroll 1
        for (int c0 = 0; c0 < cols; c0 += 32) {
          uint32_t r[32];
          tmem_ld32(tmem + ((uint32_t)(quarter * 32) << 16) + a * TN + (uint32_t)c0, r);
          tmem_ld_wait();
          if (row < m) {
            float* p = part + (long long)c0 * m;
            if (c0 + 32 <= cols) {
#pragma unroll
              for (int i = 0; i < 32; ++i) p[(long long)i * m] = __uint_as_float(r[i]);
            } else {
#pragma unroll
              for (int i = 0; i < 32; ++i)
                if (c0 + i < cols) p[(long long)i * m] = __uint_as_float(r[i]);
            }
          }
          __syncwarp();
        }
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(&acc_empty[a]);
      }
    }
    if (!ok) { *abort_flag = 1; if (lane == 0) atomicCAS(status, 0, (int)ST_GAVE_UP_EPILOGUE); }
  }
  // ---- teardown: every thread arrives here (also after a wait gave up)
  tc_fence_before();
  __syncthreads();
  if (*abort_flag) {
    // A role gave up.  Before shared memory and tensor memory are released, wait (bounded again) for what may still be
    // in flight: the bulk copies into the stages armed last, and the MMAs issued so far.
    if (warp == LOAD_WARP && lane == 0) {
      const uint32_t n = loads_issued < (uint32_t)B_STAGES ? loads_issued : (uint32_t)B_STAGES;
      for (uint32_t i = 0; i < n; ++i) {
        const uint32_t q = loads_issued - 1 - i;
        mbar_wait(&full_b[q % B_STAGES], (q / B_STAGES) & 1u);
      }
    }
    // (commit tracks the MMAs of the issuing thread: the lane elect.sync picks)
    if (warp == MMA_WARP && elect_one()) {
      umma_commit(drain);
      mbar_wait(drain, 0);
    }
    tc_fence_before();
    __syncthreads();
  }
  if (warp == MMA_WARP) {
    tc_fence_after();
    tmem_dealloc(tmem, 512);
  }
}

}  // namespace glqb
