// Prefill path with both operands in swizzled shared memory (E8 layers, weight tiles decoded beforehand, two-stage trellis
// codes; the other trellis layers: glqb_tgemm.cuh) -> tcgen05.mma with fp32 accumulators in tensor memory (TMEM).  One CTA computes D[128 weight rows x TN tokens] = W~[128 x K] * X~[TN x K]^T.
//
// Warp roles (GM_THREADS = 704):
//   warps 0-15 decode producers in two groups of eight; group 0 produces the even 128x64 weight chunks,
//              group 1 the odd ones (two stages are always being filled).  Inside a group every warp
//              decodes 16 rows x 64 columns of E8 indices, or a 32 x 32 trellis group, into the stage's A tile,
//              K-major with the 128-byte swizzle the tensor core expects
//   warps 18-21 epilogue: tcgen05.ld of the finished accumulator (two accumulators alternate, so the
//              next tile's MMAs run while these warps write the previous tile's partial sums)
//   warp  16   one thread issues tcgen05.mma (4 per chunk: K = 16 each) and tcgen05.commit
//   warp  17   one thread fetches the activation tile of the chunk with a bulk async copy (TMA, no
//              multicast); the input-transform kernel has already written the activations in the
//              exact shared-memory image (swizzled), so one contiguous copy per chunk suffices
// Stages hand over through mbarriers.  Every wait is bounded: on expiry the kernel records a status
// word, stops issuing work, frees its TMEM columns and returns.
#pragma once
#include "glqb_rht.cuh"

namespace glqb {

constexpr int GM_THREADS = 704;
constexpr int GM_PRODUCER_WARPS = 16;     // two groups of 8
constexpr int GM_GROUP_WARPS = 8;
constexpr int GM_MMA_WARP = 16;
constexpr int GM_LOAD_WARP = 17;
constexpr int GM_EPI_WARP0 = 18;          // warps 18..21 drain the accumulators (TMEM lane quarter = warp % 4)
constexpr int GM_TILE_M = 128;
constexpr int GM_TILE_K = 64;                      // fp16 elements = 128 bytes = one swizzle row
constexpr int GM_A_BYTES = GM_TILE_M * GM_TILE_K * 2;   // 16 KiB
constexpr uint32_t GM_SPIN_LIMIT = 1u << 22;       // try_wait attempts before a wait gives up

struct GemmItem {
  int layer;       // index into the device table
  int m_tile;      // 128-row tile
  int n_tile;      // TN-token tile
  int k_begin;     // first 64-column chunk
  int k_end;       // one past the last chunk
  int slot;        // partial-sum slot this item writes
  int tok0, ntok;  // lists built on the device (grouped experts): first token and tokens of the tile inside its layer,
  int row0;        // and the 128-byte rows of activations in front of it; other lists: see tile_tokens and glq_gemm_kernel
  int ntok2;       // trellis_gemm_kernel: tokens of the tile behind it, which the item takes as well (other lists: 1), or 0
};

// Token tiles of the layers whose codes are decoded in the GEMM (trellis_gemm_kernel): as few as possible of at most 192
// tokens, the tokens split evenly in steps of 16.
constexpr int TG_TN = 192;
__host__ __device__ __forceinline__ int tile_tokens(int tokens) {
  const int tiles = (tokens + TG_TN - 1) / TG_TN;
  return ((tokens + tiles - 1) / tiles + 15) & ~15;
}

// ---- PTX wrappers ---------------------------------------------------------------------------------
__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

__device__ __forceinline__ void mbar_init(uint64_t* bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count));
}
__device__ __forceinline__ void mbar_arrive(uint64_t* bar) {
  asm volatile("{ .reg .b64 st; mbarrier.arrive.shared::cta.b64 st, [%0]; }" ::"r"(smem_u32(bar)) : "memory");
}
__device__ __forceinline__ void mbar_expect_tx(uint64_t* bar, uint32_t bytes) {
  asm volatile("{ .reg .b64 st; mbarrier.arrive.expect_tx.shared::cta.b64 st, [%0], %1; }" ::"r"(smem_u32(bar)),
               "r"(bytes)
               : "memory");
}
// bounded wait; false = gave up.  `abort_flag` (shared memory, optional) is set by any role of the CTA whose
// own wait ran out: the others then stop waiting at once instead of each running down its own limit.
__device__ __forceinline__ bool mbar_wait(uint64_t* bar, uint32_t parity, const volatile int* abort_flag = nullptr) {
  const uint32_t addr = smem_u32(bar);
  for (uint32_t it = 0; it < GM_SPIN_LIMIT; ++it) {
    uint32_t ok;
    asm volatile(
        "{ .reg .pred p; mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2; selp.u32 %0, 1, 0, p; }"
        : "=r"(ok)
        : "r"(addr), "r"(parity)
        : "memory");
    if (ok) return true;
    if (abort_flag && (it & 63u) == 63u && *abort_flag) return false;
  }
  return false;
}
__device__ __forceinline__ void fence_async_smem() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }
__device__ __forceinline__ void fence_mbar_init() { asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }

__device__ __forceinline__ void bulk_g2s(void* dst, const void* src, uint32_t bytes, uint64_t* bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                   smem_u32(dst)),
               "l"(src), "r"(bytes), "r"(smem_u32(bar))
               : "memory");
}

__device__ __forceinline__ void tmem_alloc(uint32_t* dst_smem, uint32_t cols) {
  asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(dst_smem)), "r"(cols)
               : "memory");
}
__device__ __forceinline__ void tmem_relinquish() {
  asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_dealloc(uint32_t taddr, uint32_t cols) {
  asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(cols) : "memory");
}
__device__ __forceinline__ void umma_f16(uint32_t d_tmem, uint64_t a_desc, uint64_t b_desc, uint32_t idesc,
                                         uint32_t accumulate) {
  asm volatile(
      "{ .reg .pred p; setp.ne.b32 p, %4, 0; tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p; }" ::"r"(d_tmem),
      "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(accumulate)
      : "memory");
}
__device__ __forceinline__ void umma_commit(uint64_t* bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(bar))
               : "memory");
}
__device__ __forceinline__ void tmem_ld32(uint32_t taddr, uint32_t (&r)[32]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
      "{%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,"
      "%29,%30,%31}, [%32];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
        "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]), "=r"(r[16]),
        "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]),
        "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
      : "r"(taddr)
      : "memory");
}
// one lane of the (converged) warp
__device__ __forceinline__ bool elect_one() {
  uint32_t ok;
  asm volatile("{ .reg .pred p; elect.sync _|p, 0xffffffff; selp.u32 %0, 1, 0, p; }" : "=r"(ok));
  return ok != 0;
}
__device__ __forceinline__ void tmem_ld_wait() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }

// K-major operand tile with 128-byte swizzle: rows of 128 bytes, 8-row atoms of 1024 bytes stacked along
// M/N (stride byte offset 1024), descriptor version 1 (Blackwell), layout type 2 (SWIZZLE_128B).
__device__ __forceinline__ uint64_t umma_desc_sw128(uint32_t smem_addr) {
  uint64_t d = 0;
  d |= (uint64_t)((smem_addr >> 4) & 0x3FFF);
  d |= (uint64_t)1 << 16;                 // leading byte offset (unused for swizzled K-major) = 1
  d |= (uint64_t)(1024 >> 4) << 32;       // stride byte offset
  d |= (uint64_t)1 << 46;                 // descriptor version
  d |= (uint64_t)2 << 61;                 // SWIZZLE_128B
  return d;
}
// instruction descriptor: D fp32, A and B fp16, both K-major, M = 128, N = tn
__device__ __forceinline__ uint32_t umma_idesc_f16(int tn) {
  return (1u << 4) | ((uint32_t)(tn >> 3) << 17) | ((uint32_t)(GM_TILE_M >> 4) << 24);
}
// byte offset of element (row r, fp16 column e) inside a swizzled K-major tile
__device__ __forceinline__ uint32_t sw128_offset(int r, int e) {
  return (uint32_t)((r >> 3) * 1024 + (r & 7) * 128 + ((((e >> 3) ^ (r & 7)) & 7) << 4) + (e & 7) * 2);
}

// ---- input transform for the GEMM path: activations written as swizzled TN x 64 tiles ---------------
// One CTA per (layer, Hadamard block, tile of tokens); tiles ordered [n_tile][k_chunk], each TN*128
// bytes.  Columns past n (the last chunk of a layer whose n is not a multiple of 64) are written as
// zeros by the CTAs of the last block.
static __global__ void __launch_bounds__(RHT_THREADS, RHT_MINB) rht_in_gemm_kernel(const DevLinear* __restrict__ layers,
                                                                  const RhtItem* __restrict__ items,
                                                                  const uint8_t* __restrict__ x_base,
                                                                  uint8_t* __restrict__ ws, int tokens) {
  extern __shared__ __align__(16) float fbuf[];
  pdl_wait();
  pdl_trigger();
  RhtItem it = items[blockIdx.x];
  if (!rht_item_trim(it, tokens)) return;
  const DevLinear& L = layers[it.layer];
  const bool steps = L.gemm_even != 0;             // tiles of the tokens of this run, the last one ends on 16 rows
  const int used = min(L.batch, tokens), tn = steps ? tile_tokens(used) : L.gemm_tn;
  const int off = L.bn_off[it.block];
  const int logbs = L.bn_log[it.block];
  const int bs = 1 << logbs;
  const int kchunks = (L.n + GM_TILE_K - 1) / GM_TILE_K;
  const float rs = L.x_is_rotated ? 1.0f : rsqrtf((float)bs);
  uint8_t* xr = ws + L.xr_off;
  auto tile_rows = [&](int tile) -> int { return steps ? min(tn, (used - tile * tn + 15) & ~15) : tn; };
  auto place = [&](int token, int col) -> uint8_t* {
    const int tile = token / tn;
    return xr + ((size_t)tile * tn * kchunks + (size_t)(col >> 6) * tile_rows(tile)) * 128 + sw128_offset(token - tile * tn, col & 63);
  };
  auto store1 = [&](int row, int i, float v) { *reinterpret_cast<__half*>(place(it.tok0 + row, off + i)) = __float2half_rn(v); };
  auto load1 = [&](int row, int i) -> float {
    const int col = off + i;
    if (col >= L.in_f) return 0.f;
    float v = load_act(x_base, L.x_off + (long long)(it.tok0 + row) * L.x_stride + col, L.x_dtype);
    if (!L.x_is_rotated) v *= __half2float(L.sv[col]);
    return v;
  };
  const int S = it.sub >= 0 ? bs >> FHT_LOG : 1, log_t = min(logbs, FHT_LOG), run0 = max(it.sub, 0) << FHT_LOG;
  const int total = it.ntok << log_t;
  if (L.x_is_rotated) {
    for (int o = threadIdx.x; o < total; o += blockDim.x) {
      const int row = o >> log_t, i = run0 + (o & ((1 << log_t) - 1));
      store1(row, i, load1(row, i));
    }
  } else {
    const bool vec = (off & 3) == 0 && log_t >= 2 && act_rows_aligned4(x_base, L.x_off, L.x_stride, L.x_dtype);
    if (vec && off + bs <= L.in_f && logbs >= 10) {
      // whole blocks of 1024 columns and more: a warp's stores stay in one token, two 64-column chunks apart each
      auto load_plain = [&](int e0, f2 (&v)[8][2]) { rht_load_x_plain(L, it, x_base, off, log_t, total, S, e0, v); };
      auto store_plain = [&](int e1, const f2 (&v)[8][2]) {
        const f2 rs2 = f2_pack(rs, rs);
        const int token = it.tok0 + (e1 >> log_t);
        const size_t step = (size_t)tile_rows(token / tn) * 256;
        uint8_t* p = place(token, off + run0 + (e1 & ((1 << log_t) - 1)));
#pragma unroll
        for (int k = 0; k < 8; ++k)
          if (e1 + (k << 7) < total) {
            float r[4];
            f2_unpack(f2_mul(v[k][0], rs2), r[0], r[1]);
            f2_unpack(f2_mul(v[k][1], rs2), r[2], r[3]);
            const __half2 a = __floats2half2_rn(r[0], r[1]), b = __floats2half2_rn(r[2], r[3]);
            *reinterpret_cast<uint2*>(p + k * step) =
                make_uint2(*reinterpret_cast<const uint32_t*>(&a), *reinterpret_cast<const uint32_t*>(&b));
          }
      };
      fht_block_all(fbuf, log_t, total, load_plain, store_plain);
    } else {
      auto load = [&](int e0, f2 (&v)[8][2]) { rht_load_x(L, it, x_base, off, log_t, total, S, vec, load1, e0, v); };
      const bool out_vec = (off & 3) == 0 && log_t >= 2;
      auto store = [&](int e, const f2 (&q)[2]) {
        float r[4];
        f2_unpack(q[0], r[0], r[1]);
        f2_unpack(q[1], r[2], r[3]);
        if (out_vec) {         // four columns are 8 bytes of a swizzled 128-byte row, a warp writes 256 bytes
          const __half2 a = __floats2half2_rn(r[0] * rs, r[1] * rs), b = __floats2half2_rn(r[2] * rs, r[3] * rs);
          *reinterpret_cast<uint2*>(place(it.tok0 + (e >> log_t), off + run0 + (e & ((1 << log_t) - 1)))) =
              make_uint2(*reinterpret_cast<const uint32_t*>(&a), *reinterpret_cast<const uint32_t*>(&b));
        } else {
  #pragma unroll
          for (int j = 0; j < 4; ++j)
            if (e + j < total) store1((e + j) >> log_t, run0 + ((e + j) & ((1 << log_t) - 1)), r[j] * rs);
        }
      };
      fht_block(fbuf, log_t, total, load, store);
    }
  }
  if (it.block == L.nbn - 1 && it.sub <= 0) {
    const int padc = kchunks * GM_TILE_K - L.n;
    for (int o = threadIdx.x; o < it.ntok * padc; o += blockDim.x) {
      const int tk = o / padc;
      *reinterpret_cast<__half*>(place(it.tok0 + tk, L.n + (o - tk * padc))) = __float2half_rn(0.f);
    }
  }
}

// ---- weight producers ------------------------------------------------------------------------------
__device__ __forceinline__ void st_shared_v4(uint32_t addr, uint4 v) {
  asm volatile("st.shared.v4.u32 [%0], {%1,%2,%3,%4};" ::"r"(addr), "r"(v.x), "r"(v.y), "r"(v.z), "r"(v.w) : "memory");
}

// Where a lane's 16 register pairs of a 32 x 32 group go inside the 32-row slice of a swizzled 128 x 64 tile: pair
// (ni, c, mi, a) at addr[ni * 2 + c] + mi * 2048 + a * 1024.  Only the 16-byte unit is swizzled, so four addresses and
// immediate offsets cover all sixteen.
__device__ __forceinline__ void gemm_lane_addrs(uint32_t slice, int cg, int lane, uint32_t (&addr)[4]) {
  const int g = lane >> 2, t = lane & 3;
#pragma unroll
  for (int u = 0; u < 4; ++u) addr[u] = slice + (uint32_t)(g * 128 + (((cg * 4 + u) ^ g) << 4) + t * 4);
}
template <int OFF>
__device__ __forceinline__ void st_shared_u32_at(uint32_t addr, uint32_t v) {
  asm volatile("st.shared.u32 [%0 + %2], %1;" ::"r"(addr), "r"(v), "n"(OFF) : "memory");
}
__device__ __forceinline__ void gemm_store_quad(const uint32_t (&addr)[4], int q, const uint32_t (&w)[4]) {
  // q = ni * 2 + mi; w[p], p = c * 2 + a
  const uint32_t a0 = addr[(q >> 1) * 2], a1 = addr[(q >> 1) * 2 + 1];
  if (q & 1) {
    st_shared_u32_at<2048>(a0, w[0]); st_shared_u32_at<3072>(a0, w[1]);
    st_shared_u32_at<2048>(a1, w[2]); st_shared_u32_at<3072>(a1, w[3]);
  } else {
    st_shared_u32_at<0>(a0, w[0]); st_shared_u32_at<1024>(a0, w[1]);
    st_shared_u32_at<0>(a1, w[2]); st_shared_u32_at<1024>(a1, w[3]);
  }
}

template <int K1, int K2>
__device__ __forceinline__ void gemm_store_group(const uint32_t (&addr)[4], int lane, const Words<K1>& v,
                                                 const Words<(K2 > 0 ? K2 : 1)>& v2, __half2 s2) {
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
  for (int q = 0; q < 4; ++q) {
    uint32_t a[8], b[8], w[4];
    decode_tile<K1>(chunk_of<K1>(v, q), chunk_of<K1>(vn, q), chunk_of<K1>(vn2, q), a);
    if constexpr (K2 > 0) decode_tile<K2>(chunk_of<K2>(v2, q), chunk_of<K2>(un, q), chunk_of<K2>(un2, q), b);
#pragma unroll
    for (int p = 0; p < 4; ++p) {
      w[p] = __byte_perm(a[2 * p], a[2 * p + 1], 0x5410);        // (w_{2p}, w_{2p+1})
      if constexpr (K2 > 0) {
        // second stage folded into the fp16 operand: w = fp16(w1 + s2 * w2), one rounding
        const uint32_t w2 = __byte_perm(b[2 * p], b[2 * p + 1], 0x5410);
        const __half2 r = __hfma2(*reinterpret_cast<const __half2*>(&w2), s2, *reinterpret_cast<const __half2*>(&w[p]));
        w[p] = *reinterpret_cast<const uint32_t*>(&r);
      }
    }
    gemm_store_quad(addr, q, w);
  }
}

// ---- the GEMM kernel -------------------------------------------------------------------------------
// FORMAT 0: two-stage trellis codes (K1, K2 bits), 256 tokens per tile; FORMAT 1: E8 (K1 = number of stages); FORMAT 2: the weight tiles were decoded beforehand (e8_tiles_kernel,
//           trellis_tiles_kernel) and are fetched like the activation tiles, one bulk copy per stage; the producer warps
//           have nothing to do.  (Other trellis layers are decoded by trellis_gemm_kernel.)
// TN = 192: variable token tiles, for grouped experts.  A tile's activations are rows of ntok rounded up to 16, [k chunk]
// [row] behind the row0 rows of the tiles before it; an item multiplies exactly that many columns.
template <int FORMAT, int K1, int K2, int TN, int STAGES>
__global__ void __launch_bounds__(GM_THREADS, 1)
glq_gemm_kernel(const DevLinear* __restrict__ layers, const GemmItem* __restrict__ items, int n_items,
                uint8_t* __restrict__ ws, int* __restrict__ status, const int* __restrict__ n_items_dev, int tokens) {
  // No trigger, except in the form that gathers: CTAs of the output transform that start early go where the GEMM leaves room, which
  // is a few SMs, and these then do all of it.  In a graph, trigger / none: trellis, 256 tokens of 1024 x 4096 22.5 / 20.1 us, of 5376 x
  // 4096 31.5 / 30.3, 2048 tokens of 11008 x 2048 131.4 / 129.0.  E8, 128 tokens of 11008 x 2048 54.3 / 61.3, of 5376 x 4096 45.8 / 50.1,
  // of 2048 x 11008 49.9 / 47.9.
  if constexpr (FORMAT == 1) pdl_trigger();
  // work lists built on the device (grouped expert matmul) pass their length through memory; other lists and the weights are
  // there before: then only the loader and the epilogue wait for the kernel before this one
  if (n_items_dev) { pdl_wait(); n_items = min(n_items, *n_items_dev); }
  constexpr int B_BYTES = TN * 128;
  constexpr bool VAR = TN == 192;
  constexpr int TMEM_COLS = VAR ? 512 : 2 * TN;
  // tokens of an item's tile (none: every role skips the item); an MMA takes them rounded up to 16
  auto cols_of = [&](const GemmItem& it, const DevLinear& L) -> int {
    return VAR ? it.ntok : min(TN, min(L.batch, tokens) - it.n_tile * TN);
  };
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
  uint8_t* a_base = smem;                                   // STAGES x 16 KiB
  uint8_t* b_base = smem + STAGES * GM_A_BYTES;             // STAGES x TN*128
  uint64_t* bars = reinterpret_cast<uint64_t*>(b_base + STAGES * B_BYTES);
  uint64_t* full_a = bars;
  uint64_t* full_b = bars + STAGES;
  uint64_t* empty = bars + 2 * STAGES;
  uint64_t* acc_full = bars + 3 * STAGES;          // [2]
  uint64_t* acc_empty = acc_full + 2;              // [2]
  uint64_t* drain = acc_empty + 2;                 // give-up path only: completion of the MMAs issued so far
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(drain + 1);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (threadIdx.x == 0) {
    for (int s = 0; s < STAGES; ++s) {
      mbar_init(&full_a[s], GM_GROUP_WARPS);
      mbar_init(&full_b[s], 1);
      mbar_init(&empty[s], 1);
    }
    for (int a = 0; a < 2; ++a) {
      mbar_init(&acc_full[a], 1);
      mbar_init(&acc_empty[a], 4);
    }
    mbar_init(drain, 1);
    *abort_flag = 0;
    fence_mbar_init();
  }
  if (warp == GM_MMA_WARP) {
    tmem_alloc(tmem_slot, TMEM_COLS);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_acc = *tmem_slot;
  uint32_t loads_issued = 0;                       // activation-loader thread: stages armed so far

  if (warp < GM_PRODUCER_WARPS) {
    // ------------------------------------------------------------------ producers (+ epilogue)
    // q numbers the chunks of this CTA over all its items; chunk q lives in stage q % STAGES and is
    // produced by group (q & 1).  Every role derives stage and phase from q in the same way.
    const int grp = warp >> 3, wl = warp & 7;
    uint32_t q0 = 0;
    bool ok = true;
    for (int item = blockIdx.x; item < n_items && ok; item += gridDim.x) {
      const GemmItem it = items[item];
      const DevLinear& L = layers[it.layer];
      if (cols_of(it, L) <= 0) continue;
      const int first = it.k_begin + (int)((grp - q0) & 1u);       // this group's first chunk of the item
      if constexpr (FORMAT == 2) {
        (void)first; (void)wl; (void)L;
      } else if constexpr (FORMAT == 0) {
        // warp wl of a group decodes the 32 x 32 trellis group at rows 32 (wl >> 1), columns 32 (wl & 1) of the chunk
        const int strip = wl >> 1, cg = wl & 1;
        const int rp = it.m_tile * 4 + strip, gps = L.groups_per_strip;
        const bool row_ok = rp < L.strips;
        const uint8_t* p1 = L.codes[0] + (long long)rp * gps * (128 * K1) + lane * (4 * K1);
        const uint8_t* p2 = L.codes[1] + (long long)rp * gps * (128 * K2) + lane * (4 * K2);
        const __half2 s2 = __float2half2_rn(L.stage_scale[1]);
        Words<K1> nxt;
        Words<K2> nxt2;
        auto fetch = [&](int kc) {
          const int cp = kc * 2 + cg;
          if (row_ok && cp < gps) {
            nxt = load_words<K1>(p1 + (long long)cp * (128 * K1));
            nxt2 = load_words<K2>(p2 + (long long)cp * (128 * K2));
          }
        };
        if (first < it.k_end) fetch(first);
        for (int kc = first; kc < it.k_end; kc += 2) {
          const uint32_t q = q0 + (uint32_t)(kc - it.k_begin);
          const int stage = (int)(q % STAGES);
          const Words<K1> v = nxt;
          const Words<K2> v2 = nxt2;
          if (kc + 2 < it.k_end) fetch(kc + 2);
          if (!mbar_wait(&empty[stage], ((q / STAGES) & 1u) ^ 1u, abort_flag)) { ok = false; break; }
          __syncwarp();
          uint32_t addr[4];
          gemm_lane_addrs(smem_u32(a_base) + stage * GM_A_BYTES + strip * 4096, cg, lane, addr);
          if (row_ok && kc * 2 + cg < gps) {                 // (uniform per warp: the shuffles inside see all lanes)
            gemm_store_group<K1, K2>(addr, lane, v, v2, s2);
          } else {                                           // rows or columns past the matrix: zeros
            const uint32_t zero[4] = {0u, 0u, 0u, 0u};
#pragma unroll
            for (int p = 0; p < 4; ++p) gemm_store_quad(addr, p, zero);
          }
          fence_async_smem();
          __syncwarp();
          if (lane == 0) mbar_arrive(&full_a[stage]);
        }
      } else {
        // E8: 128 rows x 8 indices per chunk; thread (row = tid >> 1, half = tid & 1) expands 4 indices
        const int tid = threadIdx.x & 255;                // thread inside the producer group
        const int row_l = tid >> 1, hf = tid & 1;
        const int row = it.m_tile * GM_TILE_M + row_l;
        const int nidx = L.n >> 3;
        const bool row_ok = row < L.m;
        // 8-byte loads need every row (and the matrix itself) to start on an 8-byte boundary
        bool vec_ok = (nidx & 3) == 0;
#pragma unroll
        for (int s = 0; s < K1; ++s) vec_ok = vec_ok && (reinterpret_cast<uintptr_t>(L.codes[s]) & 7) == 0;
        uint2 nq[K1];                                     // 4 indices (8 bytes) per stage
        auto fetch = [&](int kc) {
          const int i0 = kc * 8 + hf * 4;
#pragma unroll
          for (int s = 0; s < K1; ++s) {
            nq[s] = make_uint2(0u, 0u);
            if (row_ok && vec_ok && i0 + 4 <= nidx) {
              nq[s] = ld_stream_v2(reinterpret_cast<const uint16_t*>(L.codes[s]) + (long long)row * nidx + i0);
            } else if (row_ok) {
              const uint16_t* qd = reinterpret_cast<const uint16_t*>(L.codes[s]) + (long long)row * nidx;
              uint32_t v[4] = {0, 0, 0, 0};
              for (int k = 0; k < 4; ++k) if (i0 + k < nidx) v[k] = qd[i0 + k];
              nq[s] = make_uint2(v[0] | (v[1] << 16), v[2] | (v[3] << 16));
            }
          }
        };
        if (first < it.k_end) fetch(first);
        for (int kc = first; kc < it.k_end; kc += 2) {
          const uint32_t q = q0 + (uint32_t)(kc - it.k_begin);
          const int stage = (int)(q % STAGES);
          const uint32_t phase = (q / STAGES) & 1u;
          uint2 cq[K1];
#pragma unroll
          for (int s = 0; s < K1; ++s) cq[s] = nq[s];
          if (kc + 2 < it.k_end) fetch(kc + 2);
          // gather before waiting for the stage: the table reads overlap the wait
          uint32_t ent[K1][4];
          const int i0 = kc * 8 + hf * 4;
#pragma unroll
          for (int s = 0; s < K1; ++s) {
            const uint32_t mask = (uint32_t)L.table_entries[s] - 1u;
#pragma unroll
            for (int k = 0; k < 4; ++k) {
              const uint32_t idx = ((k < 2 ? cq[s].x : cq[s].y) >> ((k & 1) * 16)) & 0xFFFFu;
              ent[s][k] = __ldg(L.table[s] + (idx & mask));
            }
          }
          if (!mbar_wait(&empty[stage], phase ^ 1, abort_flag)) { ok = false; break; }
          const uint32_t a_tile = smem_u32(a_base) + stage * GM_A_BYTES;
#pragma unroll
          for (int k = 0; k < 4; ++k) {
            uint4 out = make_uint4(0u, 0u, 0u, 0u);
            if (row_ok && i0 + k < nidx) {
              uint32_t h[4];
              e8_entry_to_half2(ent[0][k], h);               // (c0,c4),(c1,c5),(c2,c6),(c3,c7)
#pragma unroll
              for (int s = 1; s < K1; ++s) {
                uint32_t h2[4];
                e8_entry_to_half2(ent[s][k], h2);
                const __half2 sc = __float2half2_rn(L.stage_scale[s]);
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                  const __half2 r = __hfma2(*reinterpret_cast<const __half2*>(&h2[j]), sc,
                                            *reinterpret_cast<const __half2*>(&h[j]));
                  h[j] = *reinterpret_cast<const uint32_t*>(&r);
                }
              }
              // natural column order inside the 16-byte chunk: (c0,c1),(c2,c3),(c4,c5),(c6,c7)
              out.x = __byte_perm(h[0], h[1], 0x5410);
              out.y = __byte_perm(h[2], h[3], 0x5410);
              out.z = __byte_perm(h[0], h[1], 0x7632);
              out.w = __byte_perm(h[2], h[3], 0x7632);
            }
            st_shared_v4(a_tile + sw128_offset(row_l, (hf * 4 + k) * 8), out);
          }
          fence_async_smem();
          __syncwarp();
          if (lane == 0) mbar_arrive(&full_a[stage]);
        }
      }
      q0 += (uint32_t)(it.k_end - it.k_begin);
      if (!ok) break;
    }
    if (!ok) { *abort_flag = 1; if (lane == 0) atomicCAS(status, 0, (int)ST_GAVE_UP_PRODUCER); }
  } else if (warp == GM_MMA_WARP) {
    // ------------------------------------------------------------------ MMA issuer
    // The whole warp walks the chunks and one elected lane issues: warp-uniform control flow keeps descriptors and
    // addresses in uniform registers (under a lane == 0 branch this loop itself took longer than the MMAs).
    const uint32_t d0 = __shfl_sync(0xffffffffu, tmem_acc, 0);
    const uint32_t a0 = smem_u32(a_base), b0 = smem_u32(b_base);
    int stage = 0;
    uint32_t phase = 0, seq = 0;
    bool ok = true;
    for (int item = blockIdx.x; item < n_items && ok; item += gridDim.x) {
      const int chunks = __shfl_sync(0xffffffffu, items[item].k_end - items[item].k_begin, 0);
      const int cols = __shfl_sync(0xffffffffu, cols_of(items[item], layers[items[item].layer]), 0);
      if (cols <= 0) continue;
      const uint32_t idesc = umma_idesc_f16((cols + 15) & ~15);
      const uint32_t a = seq & 1u, a_phase = (seq >> 1) & 1u;     // accumulator and its use count parity
      const uint32_t d_tmem = d0 + a * TN;
      if (!mbar_wait(&acc_empty[a], a_phase ^ 1, abort_flag)) { ok = false; break; }
      tc_fence_after();
      for (int c = 0; c < chunks; ++c) {
        if ((FORMAT != 2 && !mbar_wait(&full_a[stage], phase, abort_flag)) || !mbar_wait(&full_b[stage], phase, abort_flag)) { ok = false; break; }
        tc_fence_after();
        const uint64_t da = umma_desc_sw128(a0 + stage * GM_A_BYTES);
        const uint64_t db = umma_desc_sw128(b0 + stage * B_BYTES);
        if (elect_one()) {
#pragma unroll
          for (int k = 0; k < GM_TILE_K / 16; ++k)      // +32 bytes (2 x 16-byte units) per K step of 16
            umma_f16(d_tmem, da + (uint64_t)(2 * k), db + (uint64_t)(2 * k), idesc, (c > 0 || k > 0) ? 1u : 0u);
          umma_commit(&empty[stage]);                    // stage reusable once these MMAs have read it
        }
        __syncwarp();
        if (++stage == STAGES) { stage = 0; phase ^= 1; }
      }
      if (!ok) break;
      if (elect_one()) umma_commit(&acc_full[a]);
      __syncwarp();
      ++seq;
    }
    if (!ok) { *abort_flag = 1; if (lane == 0) atomicCAS(status, 0, (int)ST_GAVE_UP_MMA); }
  } else if (warp == GM_LOAD_WARP) {
    // ------------------------------------------------------------------ activation loader
    if (lane == 0) {
      pdl_wait();
      int stage = 0;
      uint32_t phase = 0;
      bool ok = true;
      for (int item = blockIdx.x; item < n_items && ok; item += gridDim.x) {
        const GemmItem it = items[item];
        const DevLinear& L = layers[it.layer];
        const int kchunks = (L.n + GM_TILE_K - 1) / GM_TILE_K;
        const int cols = cols_of(it, L);
        if (cols <= 0) continue;
        // (tiles of VAR hold just these rows, the others TN)
        const uint32_t b_bytes = (uint32_t)((cols + 15) & ~15) * 128u, b_step = VAR ? b_bytes : (uint32_t)B_BYTES;
        const uint8_t* src = ws + L.xr_off + (VAR ? (size_t)it.row0 * kchunks * 128 : (size_t)it.n_tile * kchunks * B_BYTES);
        for (int kc = it.k_begin; kc < it.k_end; ++kc) {
          if (!mbar_wait(&empty[stage], phase ^ 1, abort_flag)) { ok = false; break; }
          if constexpr (FORMAT == 2) {
            mbar_expect_tx(&full_b[stage], b_bytes + GM_A_BYTES);
            bulk_g2s(a_base + stage * GM_A_BYTES,
                     ws + L.atile_off + ((size_t)it.m_tile * kchunks + kc) * GM_A_BYTES, GM_A_BYTES, &full_b[stage]);
          } else {
            mbar_expect_tx(&full_b[stage], b_bytes);
          }
          bulk_g2s(b_base + stage * B_BYTES, src + (size_t)kc * b_step, b_bytes, &full_b[stage]);
          ++loads_issued;
          if (++stage == STAGES) { stage = 0; phase ^= 1; }
        }
      }
      if (!ok) { *abort_flag = 1; atomicCAS(status, 0, (int)ST_GAVE_UP_LOADER); }
    }
  }
  else {
    // ------------------------------------------------------------------ epilogue warps
    pdl_wait();
    const int quarter = warp & 3;                          // TMEM lanes 32*quarter .. 32*quarter + 31
    uint32_t seq = 0;
    bool ok = true;
    for (int item = blockIdx.x; item < n_items && ok; item += gridDim.x) {
      const GemmItem it = items[item];
      const DevLinear& L = layers[it.layer];
      const int cols = cols_of(it, L);                                  // columns that are tokens
      if (cols <= 0) continue;
      const uint32_t a = seq & 1u, a_phase = (seq >> 1) & 1u;
      if (!mbar_wait(&acc_full[a], a_phase, abort_flag)) { ok = false; break; }
      tc_fence_after();
      const int row = it.m_tile * GM_TILE_M + quarter * 32 + lane;
      const int m = L.m, first = VAR ? it.tok0 : it.n_tile * TN;
      float* part = reinterpret_cast<float*>(ws + L.part_off) + ((long long)it.slot * L.batch + first) * m + row;
#pragma unroll 1
      for (int c0 = 0; c0 < cols; c0 += 32) {
        uint32_t r[32];
        tmem_ld32(tmem_acc + ((uint32_t)(quarter * 32) << 16) + a * TN + (uint32_t)c0, r);
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
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&acc_empty[a]);
      ++seq;
    }
    if (!ok) { *abort_flag = 1; if (lane == 0) atomicCAS(status, 0, (int)ST_GAVE_UP_EPILOGUE); }
  }
  // ---- teardown: every thread arrives here (also after a wait gave up)
  tc_fence_before();
  __syncthreads();
  if (*abort_flag) {
    // A role gave up.  Before shared memory and tensor memory are released, wait (bounded again) for what
    // may still be in flight: the bulk copies into the stages armed last, and the MMAs issued so far.
    if (warp == GM_LOAD_WARP && lane == 0) {
      const uint32_t n = loads_issued < (uint32_t)STAGES ? loads_issued : (uint32_t)STAGES;
      for (uint32_t i = 0; i < n; ++i) {
        const uint32_t q = loads_issued - 1 - i;
        mbar_wait(&full_b[q % STAGES], (q / STAGES) & 1u);
      }
    }
    // (commit tracks the MMAs of the issuing thread: the lane elect.sync picks)
    if (warp == GM_MMA_WARP && elect_one()) {
      umma_commit(drain);
      mbar_wait(drain, 0);
    }
    tc_fence_before();
    __syncthreads();
  }
  if (warp == GM_MMA_WARP) tmem_dealloc(tmem_acc, TMEM_COLS);
}

// ---- decode once: E8 indices -> swizzled fp16 weight tiles in global memory ----------------------------
// For large token counts the fused kernel would decode every weight tile once per token tile; this
// kernel decodes each 128 x 64 tile ONCE into the exact shared-memory image (K-major, 128-byte swizzle),
// [m_tile][k_chunk] x 16 KiB, which glq_gemm_kernel<2,...> then fetches with one bulk copy per stage.
// A warp takes 8 rows x 4 consecutive chunks.  Indices: one 16-byte load per lane and stage, requested a unit ahead, turned
// through 512 bytes of shared memory so that lane (c, k) gets index k of chunk c, row after row: a row's four decoded
// 128-byte tile rows are then one store of whole lines (a thread per row, 16 bytes of 32 different lines per store
// instruction, spent more of the L1 pipe on stores than on the gathers).  8 x NS gathers are in flight per lane.
// Bound by the gathers and the expansion, which alternate row by row: the entries of a unit are requested while the unit
// before it is expanded.  All of a unit's gathers first / this: whole calls of 2048 tokens of 14336 x 4096 346 / 336 us, of
// 700 tokens of 5376 x 21504 (three stages, resident) 313 / 301 us.
// TM = 0: table gathers from global memory.  TM = 1: most of the table resident in shared memory (see e8_gather), one
// CTA per SM.
constexpr int E8T_ROWS = 8;
constexpr int E8T_RESIDENT = 54 * 1024;          // leaves 512 bytes per warp for the indices
template <int NS, int TM>
__device__ __forceinline__ void e8_tiles_body(const DevLinear* __restrict__ layers, int first, int count,
                                              uint8_t* __restrict__ ws, const E8Tables& T, int warp0, int warps, uint4* buf) {
  const int lane = threadIdx.x & 31, c = lane >> 3, k = lane & 7;
  const uint16_t* mine = reinterpret_cast<const uint16_t*>(buf) + c * 8 + k;       // + 32 per row
  for (int li = first; li < first + count; ++li) {
    const DevLinear& L = layers[li];
    const int kchunks = (L.n + GM_TILE_K - 1) / GM_TILE_K;
    const int m_tiles = (L.m + GM_TILE_M - 1) / GM_TILE_M;
    const int kgroups = (kchunks + 3) >> 2;
    const int nidx = L.n >> 3, m = L.m;
    bool vec_ok = (nidx & 7) == 0;                       // every row starts 16-byte aligned
    const uint16_t* codes[NS];
    E8Stage stg[NS];
    __half2 sc[NS];
#pragma unroll
    for (int s = 0; s < NS; ++s) {
      codes[s] = reinterpret_cast<const uint16_t*>(L.codes[s]);
      vec_ok = vec_ok && (reinterpret_cast<uintptr_t>(L.codes[s]) & 15) == 0;
      stg[s].table = L.table[s];
      stg[s].mask = (uint32_t)L.table_entries[s] - 1u;
      stg[s].base = L.table_entries[s] == 65536 ? T.table_base : T.small_base;
      sc[s] = __float2half2_rn(L.stage_scale[s]);
    }
    uint8_t* tiles = ws + L.atile_off;
    const int units = m_tiles * kgroups * (GM_TILE_M / E8T_ROWS);
    uint4 nxt[NS];
    auto fetch = [&](int u) {
      const int t = u / (GM_TILE_M / E8T_ROWS), mt = t / kgroups;
      const int row = mt * GM_TILE_M + (u % (GM_TILE_M / E8T_ROWS)) * E8T_ROWS + (lane >> 2);
      const int i0 = ((t - mt * kgroups) * 4 + (lane & 3)) * 8;
#pragma unroll
      for (int s = 0; s < NS; ++s) {
        nxt[s] = make_uint4(0u, 0u, 0u, 0u);
        const uint16_t* q = codes[s] + (long long)row * nidx + i0;
        if (row < m && vec_ok && i0 + 8 <= nidx) {
          nxt[s] = ld_stream_v4(q);
        } else if (row < m) {
          uint32_t w[4] = {0u, 0u, 0u, 0u};
#pragma unroll
          for (int z = 0; z < 8; ++z)
            if (i0 + z < nidx) w[z >> 1] |= (uint32_t)q[z] << ((z & 1) * 16);
          nxt[s] = make_uint4(w[0], w[1], w[2], w[3]);
        }
      }
    };
    // the indices in `nxt`, two rows per register, for lane (c, k)
    uint32_t ix[NS][E8T_ROWS / 2], ent[NS][E8T_ROWS];
    auto turn = [&]() {
#pragma unroll
      for (int s = 0; s < NS; ++s) {
        buf[lane] = nxt[s];
        __syncwarp();
#pragma unroll
        for (int r = 0; r < E8T_ROWS; r += 2) ix[s][r >> 1] = (uint32_t)mine[r * 32] | ((uint32_t)mine[r * 32 + 32] << 16);
        __syncwarp();
      }
    };
    auto gather = [&](int r) {
#pragma unroll
      for (int s = 0; s < NS; ++s) ent[s][r] = e8_gather<TM, E8T_RESIDENT>(stg[s], (ix[s][r >> 1] >> ((r & 1) * 16)) & stg[s].mask);
    };
    if (warp0 < units) {
      fetch(warp0);
      turn();
      if (warp0 + warps < units) fetch(warp0 + warps);
#pragma unroll
      for (int r = 0; r < E8T_ROWS; ++r) gather(r);
    }
    for (int u = warp0; u < units; u += warps) {
      // (the entries of row r of the next unit are requested as soon as row r of this one is expanded: gathers and arithmetic
      // alternate, and a unit's gathers have the arithmetic of another one to arrive)
      const bool more = u + warps < units;
      if (more) {
        turn();
        if (u + 2 * warps < units) fetch(u + 2 * warps);
      }
      const int r8 = u % (GM_TILE_M / E8T_ROWS), t = u / (GM_TILE_M / E8T_ROWS);
      const int mt = t / kgroups, kc = (t - mt * kgroups) * 4 + c;
      const int row0 = r8 * E8T_ROWS;                             // first row inside the tile
      const bool col_ok = kc * 8 + k < nidx;
      uint8_t* tile = tiles + ((size_t)mt * kchunks + kc) * GM_A_BYTES + row0 * 128;
#pragma unroll
      for (int r = 0; r < E8T_ROWS; ++r) {
        uint4 out = make_uint4(0u, 0u, 0u, 0u);
        if (col_ok && mt * GM_TILE_M + row0 + r < m) {
          uint32_t h[4];
          e8_entry_to_half2(ent[0][r], h);
#pragma unroll
          for (int s = 1; s < NS; ++s) {
            uint32_t h2[4];
            e8_entry_to_half2(ent[s][r], h2);
#pragma unroll
            for (int j = 0; j < 4; ++j) {
              const __half2 z = __hfma2(*reinterpret_cast<const __half2*>(&h2[j]), sc[s], *reinterpret_cast<const __half2*>(&h[j]));
              h[j] = *reinterpret_cast<const uint32_t*>(&z);
            }
          }
          // natural column order inside the 16-byte chunk: (c0,c1),(c2,c3),(c4,c5),(c6,c7)
          out.x = __byte_perm(h[0], h[1], 0x5410);
          out.y = __byte_perm(h[2], h[3], 0x5410);
          out.z = __byte_perm(h[0], h[1], 0x7632);
          out.w = __byte_perm(h[2], h[3], 0x7632);
        }
        if (kc < kchunks) *reinterpret_cast<uint4*>(tile + r * 128 + ((k ^ r) << 4)) = out;  // (sw128_offset; row0 is a multiple of 8)
        if (more) gather(r);
      }
    }
  }
}

template <int NS>
__global__ void __launch_bounds__(256) e8_tiles_kernel(const DevLinear* __restrict__ layers, int first, int count,
                                                       uint8_t* __restrict__ ws) {
  __shared__ uint4 idx[8][32];
  const E8Tables T = {0u, 0u};
  e8_tiles_body<NS, 0>(layers, first, count, ws, T, blockIdx.x * 8 + (threadIdx.x >> 5), gridDim.x * 8, idx[threadIdx.x >> 5]);
}

constexpr int E8TS_THREADS = 512;
constexpr int E8TS_SMEM_BYTES = E8T_RESIDENT * 4 + 256 * 4 + E8TS_THREADS / 32 * 512;
template <int NS>
__global__ void __launch_bounds__(E8TS_THREADS, 1)
e8_tiles_smem_kernel(const DevLinear* __restrict__ layers, int first, int count, uint8_t* __restrict__ ws,
                     const uint32_t* __restrict__ big_table, const uint32_t* __restrict__ small_table, int small_entries) {
  extern __shared__ __align__(16) uint32_t e8t_smem[];    // table, small table, 512 bytes of indices per warp
  pdl_trigger();
  const uint4* src = reinterpret_cast<const uint4*>(big_table);
  uint4* dst = reinterpret_cast<uint4*>(e8t_smem);
  for (int i = threadIdx.x; i < E8T_RESIDENT / 4; i += blockDim.x) dst[i] = __ldg(src + i);
  for (int i = threadIdx.x; i < small_entries && i < 256; i += blockDim.x) e8t_smem[E8T_RESIDENT + i] = __ldg(small_table + i);
  E8Tables T;
  const uint32_t local = (uint32_t)__cvta_generic_to_shared(e8t_smem);
  T.table_base = local;
  T.small_base = local + E8T_RESIDENT * 4;
  __syncthreads();
  const int warp = threadIdx.x >> 5;
  e8_tiles_body<NS, 1>(layers, first, count, ws, T, blockIdx.x * (E8TS_THREADS / 32) + warp, gridDim.x * (E8TS_THREADS / 32),
                       reinterpret_cast<uint4*>(e8t_smem + E8T_RESIDENT + 256) + warp * 32);
  pdl_wait();
}

// ---- decode once: trellis bit-streams -> swizzled fp16 weight tiles ------------------------------------------
// The counterpart of e8_tiles_kernel: a warp decodes a 32-row x 64-column slice (two 32 x 32 groups) into its own 4 KiB of
// shared memory with the stores the GEMM's producers use — the slice is 4 KiB of the tile image in one piece — and
// copies it out with whole-line 16-byte stores.  The codes of the next slice are in flight meanwhile.  Bound by the
// state decode: 11008 x 2048 in 13 us.  Whole linears of 2048 tokens with the copy-fed GEMM behind it / with
// trellis_gemm_kernel: 11008 x 2048 138 / 146 us, 14336 x 4096 272 / 288, two stages (4 + 2 bits) 142 / 207, 279 / 438.
constexpr int TT_THREADS = 256;
template <int K1, int K2>
__global__ void __launch_bounds__(TT_THREADS, 3)
trellis_tiles_kernel(const DevLinear* __restrict__ layers, int first, int count, uint8_t* __restrict__ ws) {
  __shared__ __align__(1024) uint8_t slices[TT_THREADS / 32][4096];
  pdl_trigger();
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int warp0 = blockIdx.x * (TT_THREADS / 32) + warp, warps = gridDim.x * (TT_THREADS / 32);
  const uint32_t slice = smem_u32(slices[warp]);
  uint32_t addr[2][4];
  gemm_lane_addrs(slice, 0, lane, addr[0]);
  gemm_lane_addrs(slice, 1, lane, addr[1]);
  for (int li = first; li < first + count; ++li) {
    const DevLinear& L = layers[li];
    const int kchunks = (L.n + GM_TILE_K - 1) / GM_TILE_K, gps = L.groups_per_strip, strips = L.strips;
    const int units = ((L.m + GM_TILE_M - 1) / GM_TILE_M) * 4 * kchunks;      // 32-row slices of whole tiles
    const __half2 s2 = __float2half2_rn(L.stage_scale[1]);
    uint8_t* tiles = ws + L.atile_off;
    const uint8_t* p1 = L.codes[0] + lane * (4 * K1);
    const uint8_t* p2 = K2 > 0 ? L.codes[1] + lane * (4 * K2) : nullptr;
    Words<K1> v[2];
    Words<(K2 > 0 ? K2 : 1)> v2[2];
    auto fetch = [&](int u) {
      const int strip = u / kchunks, kc = u - strip * kchunks;
#pragma unroll
      for (int cg = 0; cg < 2; ++cg)
        if (strip < strips && kc * 2 + cg < gps) {
          const long long g = (long long)strip * gps + kc * 2 + cg;
          v[cg] = load_words<K1>(p1 + g * (128 * K1));
          if constexpr (K2 > 0) v2[cg] = load_words<K2>(p2 + g * (128 * K2));
        }
    };
    if (warp0 < units) fetch(warp0);
    for (int u = warp0; u < units; u += warps) {
      const int strip = u / kchunks, kc = u - strip * kchunks;
      const Words<K1> cur[2] = {v[0], v[1]};
      const Words<(K2 > 0 ? K2 : 1)> cur2[2] = {v2[0], v2[1]};
      if (u + warps < units) fetch(u + warps);
#pragma unroll
      for (int cg = 0; cg < 2; ++cg) {
        if (strip < strips && kc * 2 + cg < gps) {
          gemm_store_group<K1, K2>(addr[cg], lane, cur[cg], cur2[cg], s2);
        } else {                                             // rows or columns past the matrix: zeros
          const uint32_t zero[4] = {0u, 0u, 0u, 0u};
#pragma unroll
          for (int q = 0; q < 4; ++q) gemm_store_quad(addr[cg], q, zero);
        }
      }
      __syncwarp();
      uint4* dst = reinterpret_cast<uint4*>(tiles + ((size_t)(strip >> 2) * kchunks + kc) * GM_A_BYTES + (strip & 3) * 4096) + lane;
      const uint4* src = reinterpret_cast<const uint4*>(slices[warp]) + lane;
#pragma unroll
      for (int i = 0; i < 8; ++i) dst[i * 32] = src[i * 32];
      __syncwarp();
    }
  }
  pdl_wait();                                    // (the decode itself needs nothing of the kernel before: the GEMM behind does)
}

}  // namespace glqb
