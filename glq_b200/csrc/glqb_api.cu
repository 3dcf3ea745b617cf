// C ABI of libglq_b200: plan builder, launch sequencing, stateless wrappers.
#include <algorithm>
#include <cmath>
#include <cstdarg>
#include <cstdio>
#include <cstring>
#include <map>
#include <mutex>
#include <string>
#include <tuple>
#include <vector>

#include "glqb_kernels.cuh"
#include "glqb_fused.cuh"
#include "glqb_gemm.cuh"
#include "glqb_tgemm.cuh"
#include "glqb_launch.h"

namespace glqb {

static thread_local std::string g_err;

void set_error_message(const char* msg) { g_err = msg ? msg : ""; }

static int fail(int code, const char* fmt, ...) {
  char buf[512];
  va_list ap;
  va_start(ap, fmt);
  vsnprintf(buf, sizeof buf, fmt, ap);
  va_end(ap);
  g_err = buf;
  return code;
}

#define CUDA_TRY(expr)                                                                   \
  do {                                                                                   \
    cudaError_t _e = (expr);                                                             \
    if (_e != cudaSuccess) return fail(GLQB_E_CUDA, "%s: %s", #expr, cudaGetErrorString(_e)); \
  } while (0)

static inline size_t align_up(size_t v, size_t a) { return (v + a - 1) / a * a; }
static inline int ilog2(int v) { int l = 0; while ((1 << l) < v) ++l; return l; }

constexpr int DECODE_MAX_BATCH = 64;   // above this the GEMM path is used

}  // namespace glqb

using namespace glqb;

struct GlqbPlan {
  std::vector<GlqbLinearDesc> descs;   // in caller order
  std::vector<int> order;              // device-table position -> caller index
  std::vector<DevLinear> dev;          // host copy of the device table
  std::vector<Segment> segs;
  std::vector<RhtItem> items_in, items_out;
  std::vector<RhtItem> items_in_gemm;
  std::vector<GemmItem> gemm_items;
  DevLinear* d_layers = nullptr;
  RhtItem* d_items_in = nullptr;
  RhtItem* d_items_in_gemm = nullptr;
  RhtItem* d_items_out = nullptr;
  GemmItem* d_gemm_items = nullptr;
  // A run of at most `few_tokens` tokens needs one token tile fewer than the plan's bucket (trellis_gemm_kernel): work list,
  // K splits and the layer table that names them are kept for both.  0: there is one schedule only.
  int few_tokens = 0;
  std::vector<Segment> few_segs;
  DevLinear* d_few_layers = nullptr;
  GemmItem* d_few_items = nullptr;
  int* d_status = nullptr;
  // Completion tickets of the single-launch form, all zero between runs.  A set belongs to a workspace: runs on one workspace
  // follow one another, runs that may overlap (other streams, a graph beside eager calls) have a workspace each.
  struct TicketSet { const void* workspace; int* tickets; bool captured; };     // captured: a graph may replay on it at any time
  std::mutex ticket_mutex;
  std::vector<TicketSet> ticket_sets;
  std::vector<int*> free_tickets, ticket_chunks;
  const GlqbComm* comm = nullptr;  // tensor-parallel ranks whose outputs the single-launch kernel sums (glqb_plan_set_comm)
  int n_tickets = 0;
  int max_batch_gemm = 1;
  size_t ws_bytes = 0;
  int max_batch = 1;
  bool out_plain_static = false; // every output item takes the plain transform when the output is aligned
  bool in_few = false, out_few = false;          // few tiles: the transforms with 1024 threads per tile
  bool out_wide = false;         // some layer has 2^32 partial sums per slot or more
  int max_elems_in = 32, max_elems_out = 32;    // floats of shared memory the transform CTAs need
  int sm_count = 0;
  int64_t code_bytes = 0, flops = 0;
  bool timing = false;
  std::vector<cudaEvent_t> ev;   // pairs (start, stop) around the decode kernels of each timed run
  size_t ev_used = 0;
};

namespace glqb {

// ------------------------------------------------------------------------------------------
// kernel variant tables
// ------------------------------------------------------------------------------------------
typedef void (*MvKernel)(const DevLinear*, int, long long, int, uint8_t*, int);

template <int K1, int K2>
static MvKernel trellis_kernel_nb(int nb) {
  switch (nb) {
    case 1: return trellis_mv_kernel<K1, K2, 1>;
    case 2: return trellis_mv_kernel<K1, K2, 2>;
    case 4: return trellis_mv_kernel<K1, K2, 4>;
    case 8: if constexpr (K2 == 0) return trellis_mv_kernel<K1, K2, 8>; else return nullptr;
  }
  return nullptr;
}

// table form of the single-stage batch-1 kernels (large launches only)
static MvKernel trellis_lut_kernel(int k1) {
  switch (k1) {
#ifndef GLQB_FAST_BUILD
    case 2: return trellis_mv_kernel<2, 0, 1, MV_LUT_STATES>;
    case 3: return trellis_mv_kernel<3, 0, 1, MV_LUT_STATES>;
#endif
    case 4: return trellis_mv_kernel<4, 0, 1, MV_LUT_STATES>;
  }
  return nullptr;
}
static long long trellis_lut_min_bytes() {
  // every CTA spends a microsecond or two filling its table, so small launches keep the arithmetic decode
  const char* e = getenv("GLQB_TRELLIS_LUT_MIN_BYTES");
  return e ? atoll(e) : (48ll << 20);
}

static MvKernel trellis_kernel(int k1, int k2, int nb) {
#define T_CASE(A, B) if (k1 == A && k2 == B) return trellis_kernel_nb<A, B>(nb);
#ifdef GLQB_FAST_BUILD   /* developer builds for kernel experiments: the 4-bit single-stage rate only */
  T_CASE(4, 0)
#else
  T_CASE(1, 0) T_CASE(2, 0) T_CASE(3, 0) T_CASE(4, 0)
  T_CASE(4, 1) T_CASE(4, 2) T_CASE(4, 3) T_CASE(4, 4)
#endif
#undef T_CASE
  return nullptr;
}

template <int NS>
static MvKernel e8_kernel_nb(int nb) {
  switch (nb) {
    case 1: return e8_mv_kernel<NS, 1>;
    case 2: return e8_mv_kernel<NS, 2>;
    case 4: return e8_mv_kernel<NS, 4>;
    case 8: if constexpr (NS <= 2) return e8_mv_kernel<NS, 8>; else return nullptr;
  }
  return nullptr;
}

static MvKernel e8_kernel(int ns, int nb) {
  switch (ns) {
    case 1: return e8_kernel_nb<1>(nb);
    case 2: return e8_kernel_nb<2>(nb);
    case 3: return e8_kernel_nb<3>(nb);
    case 4: return e8_kernel_nb<4>(nb);
  }
  return nullptr;
}

constexpr size_t FUSED_SMEM_LIMIT = 200 * 1024;
constexpr size_t FUSED_SMEM_MAX = 226 * 1024;       // one CTA per SM (the E8 form with a resident codebook); 1 KB left for static shared memory
static bool fused_enabled() {
  const char* e = getenv("GLQB_FUSED_DECODE");
  return !e || atoi(e) != 0;
}
// do two layers read the same transformed input?
static bool same_input(const GlqbLinearDesc& a, const GlqbLinearDesc& b) {
  return a.in_norm_weight == b.in_norm_weight && a.in_norm_dtype == b.in_norm_dtype && a.in_norm_eps == b.in_norm_eps &&
         a.in_gated_act == b.in_gated_act &&
         a.format == b.format && a.n_pad == b.n_pad && a.in_features == b.in_features && a.sv == b.sv &&
         a.batch == b.batch && a.x_offset == b.x_offset && a.x_stride == b.x_stride && a.x_dtype == b.x_dtype &&
         a.x_is_rotated == b.x_is_rotated && a.n_blocks_n == b.n_blocks_n &&
         memcmp(a.blocks_n, b.blocks_n, sizeof(int32_t) * a.n_blocks_n) == 0;
}

typedef void (*E8SmemKernel)(const DevLinear*, int, long long, int, uint8_t*, const uint32_t*, const uint32_t*, int, int);

template <int NS>
static E8SmemKernel e8_smem_kernel_nb(int nb) {
  switch (nb) {
    case 1: return e8_mv_smem_kernel<NS, 1>;
    case 2: return e8_mv_smem_kernel<NS, 2>;
    case 4: if constexpr (NS <= 2) return e8_mv_smem_kernel<NS, 4>; else return nullptr;
  }
  return nullptr;
}

static E8SmemKernel pick_e8_smem_kernel(const Segment& s) {
  switch (s.ns) {
    case 1: return e8_smem_kernel_nb<1>(s.nb);
    case 2: return e8_smem_kernel_nb<2>(s.nb);
    case 3: return e8_smem_kernel_nb<3>(s.nb);
    case 4: return e8_smem_kernel_nb<4>(s.nb);
  }
  return nullptr;
}

#ifndef GLQB_E8_SMEM_MAX_NB
#define GLQB_E8_SMEM_MAX_NB 2      // token-column blocks up to which the resident-table kernel is used
#endif
static long long e8_smem_min_bytes() {
  const char* e = getenv("GLQB_E8_SMEM_MIN_BYTES");
  // Filling the table costs every CTA about 224 KiB of L2 reads per launch (a few microseconds), so small launches
  // keep the global-memory gathers.  Measured, whole linears, gathers / resident: two stages of 4096 x 4096 (8 MiB, 16
  // tokens) 43 / 39 us, of 14336 x 4096 (28 MiB) one token 64 / 53, 16 tokens 79 / 63; 1024 x 4096 (2 MiB) 34 / 36.
  return e ? atoll(e) : (6ll << 20);
}
// the same for the tile decode of the prefill path (two stages of 14336 x 4096: 57 us either way; three stages of
// 5376 x 21504: 83 MiB of indices at 258 / 347 G indices per second)
static long long e8_tiles_smem_min_bytes() {
  const char* e = getenv("GLQB_E8_SMEM_MIN_BYTES");
  return e ? atoll(e) : (48ll << 20);
}

// Do all layers of the segment read one 65,536-entry table (and at most one small table)?  Also sums the
// index bytes of the segment.
static bool e8_uniform_tables(const std::vector<DevLinear>& dev, const Segment& s, const uint32_t** big_out,
                              const uint32_t** small_out, int* small_n_out, long long* bytes_out) {
  long long bytes = 0;
  const uint32_t* big = nullptr;
  const uint32_t* small = nullptr;
  int small_n = 0;
  for (int i = 0; i < s.count; ++i) {
    const DevLinear& L = dev[s.first + i];
    bytes += (long long)L.n_stages * L.m * (L.n / 8) * 2;
    for (int st = 0; st < L.n_stages; ++st) {
      if (L.table_entries[st] == 65536) {
        if (big && big != L.table[st]) return false;
        big = L.table[st];
      } else if (L.table_entries[st] <= 256) {
        if (small && (small != L.table[st] || small_n != L.table_entries[st])) return false;
        small = L.table[st];
        small_n = L.table_entries[st];
      } else {
        return false;
      }
    }
  }
  *big_out = big; *small_out = small; *small_n_out = small_n; *bytes_out = bytes;
  return big != nullptr;
}

static MvKernel pick_kernel(const Segment& s) {
  return s.format == GLQB_FMT_TRELLIS_3INST ? trellis_kernel(s.k1, s.k2, s.nb) : e8_kernel(s.ns, s.nb);
}

// token count from which E8 prefill decodes the weight tiles once instead of once per token tile
static int e8_two_phase_min_tokens() {
  const char* e = getenv("GLQB_E8_TWO_PHASE_MIN_TOKENS");
  return e ? atoi(e) : 129;     // measured on B200: above one 128-token tile the tile decode plus a copy-fed GEMM wins
}

// Trellis prefill decodes the weight tiles once, for the copy-fed GEMM, instead of once per 192-token tile into tensor
// memory (trellis_gemm_kernel), from this many flops per layer: the tile decode costs a launch and a write of the fp16
// weights (13 us at 11008 x 2048).  Measured, whole linears, tensor memory / tiles: 4096 x 4096, 1024 tokens (34 GFLOP)
// 65 / 65 us, 2048 tokens (69) 106 / 99; 11008 x 2048, 1024 tokens (46) 81 / 84, 2048 (92) 145 / 141; 2048 x 11008,
// 1024 tokens 94 / 103, 2048 tokens 186 / 149.
static double trellis_two_phase_min_flops() {
  const char* e = getenv("GLQB_TRELLIS_TWO_PHASE_MIN_FLOPS");
  return e ? atof(e) : 60e9;
}
// ... and while the tiles of a launch stay below 2 GiB of workspace (a sweep over a whole model keeps decoding into tensor memory)
constexpr size_t TRELLIS_TILES_MAX_BYTES = 2ull << 30;
static size_t tile_bytes(const GlqbLinearDesc& d) {
  return (size_t)((d.m_pad + GM_TILE_M - 1) / GM_TILE_M) * ((d.n_pad + GM_TILE_K - 1) / GM_TILE_K) * GM_A_BYTES;
}

// token tile of the tensor-core forms.  Pre-decoded tiles and E8: 128 or 256; trellis codes: at most 192, the tokens split
// evenly, in steps of 16.
static int tn_for_batch(int batch, bool codes) {
  if (batch <= DECODE_MAX_BATCH) return 0;
  return codes ? tile_tokens(batch) : batch <= 128 ? 128 : 256;
}

// Work of a segment's GEMM for at most `limit` tokens per layer: items (layer, 128-row tile, token tile, K range), and the
// K splits of every layer (`dev`: fixed_slots).  The SMs take the items in turn, so a split is chosen by the rounds it
// takes, in 64-column chunks (about 0.3 us each), plus the fp32 partial sums it writes and reads back at 5 TB/s.
// Splits for as many items as SMs, rounded up / by this rule, with the tokens rounded up to 512 / taken as they are: 333
// tokens of 2048 x 11008 80 / 43 us (192 items in two rounds of 148 / 128 in one).
//
// trellis_gemm_kernel may take two token tiles per item and decode their weights once; a chunk of such an item takes about 1.6
// times as long as one tile's (experts of two tiles of 128 tokens: 270 us a tile at a time, 215 us two), and there are half as
// many items: the same costs decide.
static void gemm_schedule(Segment& s, int limit, int sm_count, std::vector<DevLinear>& dev, std::vector<GemmItem>& items) {
  auto tokens_of = [&](const DevLinear& L) { return std::min(L.batch, limit); };
  auto tile_of = [&](const DevLinear& L) { return trellis_form(s) ? tile_tokens(tokens_of(L)) : s.tn; };
  auto splits = [](int kchunks, int ks, int& per) { per = (kchunks + ks - 1) / ks; return (kchunks + per - 1) / per; };
  const char* e = getenv("GLQB_GEMM_PAIRS");     // 0: single tiles, 1: pairs, whatever they cost
  const int forced = e ? atoi(e) : -1;
  int best = 1;
  bool pairs = false;                            // an item takes two token tiles
  double best_cost = 0;
  for (int ks = 1; ks <= 16; ++ks)
    for (int two = 0; two <= (trellis_form(s) ? 1 : 0); ++two) {
      if (forced >= 0 && trellis_form(s) && two != (forced != 0)) continue;
      long long n = 0;
      int longest = 0, per = 0;
      double sums = 0;
      bool ok = true, paired = false;
      for (int i = 0; i < s.count; ++i) {
        const DevLinear& L = dev[s.first + i];
        const int kchunks = (L.n + GM_TILE_K - 1) / GM_TILE_K, n_tiles = (tokens_of(L) + tile_of(L) - 1) / tile_of(L);
        ok = ok && ks <= std::max(1, kchunks / 8);
        const int k = splits(kchunks, ks, per);
        longest = std::max(longest, per);
        n += (long long)((L.m + GM_TILE_M - 1) / GM_TILE_M) * (two ? (n_tiles + 1) / 2 : n_tiles) * k;
        sums += (double)k * tokens_of(L) * L.m;
        paired = paired || (two && n_tiles > 1);
      }
      const double cost = (double)((n + sm_count - 1) / sm_count) * longest * (paired ? 1.6 : 1.0) + sums * 8 / 5e12 / 0.3e-6;
      if (best_cost == 0 || (ok && cost < best_cost)) { best = ks; pairs = two; best_cost = cost; }
    }
  s.item_first = (int)items.size();
  for (int i = 0; i < s.count; ++i) {
    DevLinear& L = dev[s.first + i];
    const int kchunks = (L.n + GM_TILE_K - 1) / GM_TILE_K, tn = tile_of(L), n_tiles = (tokens_of(L) + tn - 1) / tn;
    int per;
    L.fixed_slots = splits(kchunks, std::min(best, std::max(1, kchunks / 8)), per);
    for (int mt = 0; mt < (L.m + GM_TILE_M - 1) / GM_TILE_M; ++mt)
      for (int nt = 0; nt < n_tiles; nt += pairs ? 2 : 1)
        for (int k = 0; k < L.fixed_slots; ++k)
          items.push_back(GemmItem{s.first + i, mt, nt, k * per, std::min(kchunks, (k + 1) * per), k, 0, 0, 0, pairs && nt + 1 < n_tiles});
  }
  s.item_count = (int)items.size() - s.item_first;
  s.grid = std::min(s.item_count, sm_count);
}

// Two-stage trellis layers (whose weight decode costs twice as much) take 256-token tiles, decoded into shared memory by
// glq_gemm_kernel, where that saves a pass over the weights and there are 8 M of them.  Measured with 4 + 2 bits, whole
// plans, 192 / 256 tokens per tile: 256 tokens, 4096 x 4096 45 / 38 us, 11008 x 2048 57 / 42, 14336 x 4096 99 / 64,
// 2048 x 2048 21.4 / 22.1; 384 tokens (two passes either way) 48 / 49, 60 / 62, 104 / 107; 512 tokens 59 / 50, 63 / 65,
// 144 / 108; 1024 tokens of 2048 x 11008 143 / 127.
static bool trellis_two_stage_256(const GlqbLinearDesc& d) {
  const char* e = getenv("GLQB_TRELLIS_256_MIN_WEIGHTS");
  return d.n_stages > 1 && (d.batch + 255) / 256 < (d.batch + TG_TN - 1) / TG_TN &&
         (long long)d.m_pad * d.n_pad >= (e ? atoll(e) : (8ll << 20));
}

static int nb_for_batch(int batch) {
  if (batch <= 8) return 1;
  if (batch <= 16) return 2;
  if (batch <= 32) return 4;
  return 8;
}

static int validate(const GlqbLinearDesc& d, int idx) {
  if (d.format != GLQB_FMT_TRELLIS_3INST && d.format != GLQB_FMT_E8_SHELL)
    return fail(GLQB_E_INVALID, "layer %d: unknown format %d", idx, d.format);
  if (d.m_pad <= 0 || d.n_pad <= 0 || d.in_features <= 0 || d.out_features <= 0 ||
      d.in_features > d.n_pad || d.out_features > d.m_pad)
    return fail(GLQB_E_INVALID, "layer %d: bad dims m_pad=%d n_pad=%d in=%d out=%d", idx, d.m_pad, d.n_pad,
                d.in_features, d.out_features);
  if (d.batch < 1) return fail(GLQB_E_INVALID, "layer %d: batch %d", idx, d.batch);
  if (d.batch > 65535) return fail(GLQB_E_INVALID, "layer %d: batch %d exceeds 65535 tokens", idx, d.batch);
  if (!d.su || !d.sv || !d.codes[0]) return fail(GLQB_E_INVALID, "layer %d: null su/sv/codes", idx);
  // the kernels read the sign vectors and the trellis bit-streams with 16-byte accesses
  if ((reinterpret_cast<uintptr_t>(d.su) | reinterpret_cast<uintptr_t>(d.sv)) & 15)
    return fail(GLQB_E_INVALID, "layer %d: su / sv must be 16-byte aligned", idx);
  if (d.format == GLQB_FMT_TRELLIS_3INST) {
    if (d.m_pad % 32 || d.n_pad % 32)
      return fail(GLQB_E_INVALID, "layer %d: trellis needs m %% 32 == 0 and n %% 32 == 0 (got %d x %d)", idx,
                  d.m_pad, d.n_pad);
    if (d.n_stages < 1 || d.n_stages > 2) return fail(GLQB_E_INVALID, "layer %d: trellis stages %d", idx, d.n_stages);
    for (int s = 0; s < d.n_stages; ++s)
      if (d.bits[s] < 1 || d.bits[s] > 4 || !d.codes[s])
        return fail(GLQB_E_INVALID, "layer %d: trellis stage %d has K=%d (supported 1..4)", idx, s, d.bits[s]);
    for (int s = 0; s < d.n_stages; ++s)
      if (reinterpret_cast<uintptr_t>(d.codes[s]) & 15)
        return fail(GLQB_E_INVALID, "layer %d: trellis stage %d bit-stream must be 16-byte aligned", idx, s);
    if (!trellis_kernel(d.bits[0], d.n_stages > 1 ? d.bits[1] : 0, 1))
      return fail(GLQB_E_INVALID, "layer %d: no kernel for trellis rates K=%d+%d", idx, d.bits[0],
                  d.n_stages > 1 ? d.bits[1] : 0);
    if (d.in_features != d.n_pad) return fail(GLQB_E_INVALID, "layer %d: trellis layers are never padded", idx);
  } else {
    if (d.n_pad % 8) return fail(GLQB_E_INVALID, "layer %d: E8 needs n_pad %% 8 == 0", idx);
    if (d.n_stages < 1 || d.n_stages > 4) return fail(GLQB_E_INVALID, "layer %d: E8 stages %d", idx, d.n_stages);
    for (int s = 0; s < d.n_stages; ++s) {
      if (!d.codes[s] || !d.table[s]) return fail(GLQB_E_INVALID, "layer %d: E8 stage %d null codes/table", idx, s);
      if ((reinterpret_cast<uintptr_t>(d.codes[s]) & 1) || (reinterpret_cast<uintptr_t>(d.table[s]) & 15))
        return fail(GLQB_E_INVALID, "layer %d: E8 stage %d misaligned index matrix (2 bytes) or table (16 bytes)", idx, s);
      const int e = d.table_entries[s];
      if (e < 1 || e > 65536 || (e & (e - 1)))
        return fail(GLQB_E_INVALID, "layer %d: E8 table entries %d must be a power of two <= 65536", idx, e);
    }
  }
  int sn = 0, sm = 0;
  if (d.n_blocks_n < 1 || d.n_blocks_n > GLQB_MAX_BLOCKS || d.n_blocks_m < 1 || d.n_blocks_m > GLQB_MAX_BLOCKS)
    return fail(GLQB_E_INVALID, "layer %d: block counts %d/%d", idx, d.n_blocks_n, d.n_blocks_m);
  for (int i = 0; i < d.n_blocks_n; ++i) {
    const int b = d.blocks_n[i];
    if (b < 1 || (b & (b - 1)) || b > 32768) return fail(GLQB_E_INVALID, "layer %d: blocks_n[%d]=%d", idx, i, b);
    sn += b;
  }
  for (int i = 0; i < d.n_blocks_m; ++i) {
    const int b = d.blocks_m[i];
    if (b < 1 || (b & (b - 1)) || b > 32768) return fail(GLQB_E_INVALID, "layer %d: blocks_m[%d]=%d", idx, i, b);
    sm += b;
  }
  if (sn != d.n_pad || sm != d.m_pad)
    return fail(GLQB_E_INVALID, "layer %d: Hadamard blocks sum to %d/%d, expected n_pad=%d m_pad=%d", idx, sn, sm,
                d.n_pad, d.m_pad);
  if (d.x_dtype < 0 || d.x_dtype > 2 || d.y_dtype < 0 || d.y_dtype > 2)
    return fail(GLQB_E_INVALID, "layer %d: dtype", idx);
  if (d.stop_at_yrht && d.y_dtype != GLQB_DT_F32)
    return fail(GLQB_E_INVALID, "layer %d: rotated-domain output must be fp32", idx);
  if (d.in_gated_act < 0 || d.in_gated_act > 3 || (d.in_norm_weight && (d.in_norm_dtype < 0 || d.in_norm_dtype > 2)))
    return fail(GLQB_E_INVALID, "layer %d: input activation code %d / norm weight dtype %d", idx, d.in_gated_act, d.in_norm_dtype);
  if ((d.in_gated_act || d.in_norm_weight) && d.x_is_rotated)
    return fail(GLQB_E_INVALID, "layer %d: input fusions need an untransformed input", idx);
  if (d.y_accumulate && d.stop_at_yrht)
    return fail(GLQB_E_INVALID, "layer %d: the residual add applies to the final output only", idx);
  return GLQB_OK;
}

// packed bytes of a layer's codes (what a decode launch must read once)
static long long layer_code_bytes(const GlqbLinearDesc& d) {
  if (d.format == GLQB_FMT_TRELLIS_3INST) {
    long long b = 0;
    for (int s = 0; s < d.n_stages; ++s) b += (long long)d.m_pad * d.n_pad * d.bits[s] / 8;
    return b;
  }
  return (long long)d.n_stages * d.m_pad * (d.n_pad / 8) * 2;
}

// Does rht_out_plain_kernel serve every output item of the plan (rht_out_is_plain, host side)?  The static part is
// decided once; the alignment of this run's output is not known before.
static bool out_plain(const GlqbPlan* P, const uint8_t* y_base) {
  if (!P->out_plain_static) return false;
  for (const DevLinear& L : P->dev) {
    const int es = L.y_dtype == GLQB_DT_F32 ? 4 : 2;
    if (((L.y_off | L.y_stride) & 3) || (reinterpret_cast<uintptr_t>(y_base) & (4 * es - 1))) return false;
  }
  return true;
}

static int rht_smem(int max_elems) { return fht_words(max_elems) * 4 + 64; }

// Tokens per CTA of the transform kernels: a tile of 8192 values (fht_block), less when the launch, with `blocks` Hadamard
// blocks in all its layers, would leave SMs without work.
static int rht_tile_tokens(int block_size, int batch, long long blocks, int sm_count) {
  int t = std::min(std::max(1, std::min(64, 8192 / block_size)), batch);
  while (t > 1 && blocks * ((batch + t - 1) / t) < sm_count) t = (t + 1) / 2;
  return t;
}

// The blocks of one layer that a transform launch takes: those of at least 2^min_log values (the single-launch kernel
// transforms the shorter output blocks itself).
struct RhtLayer {
  int layer, nblocks;
  const int* logs;
  int batch, min_log;
};
// One item per (layer, block, tile of tokens); tracks the largest tile (floats) for the launch's smem.
// A block of more than 8192 values is shared by S = bs / 8192 CTAs per token, each producing one run of 8192 outputs
// (RhtItem::sub).
static void add_rht_items(std::vector<RhtItem>& items, const std::vector<RhtLayer>& layers, int sm_count, int& max_elems) {
  long long blocks = 0;
  for (const RhtLayer& r : layers)
    for (int b = 0; b < r.nblocks; ++b) blocks += r.logs[b] >= r.min_log;
  for (const RhtLayer& r : layers)
    for (int b = 0; b < r.nblocks; ++b) {
      if (r.logs[b] < r.min_log) continue;
      const int bs = 1 << r.logs[b];
      if (r.logs[b] > FHT_LOG) {
        for (int t = 0; t < r.batch; ++t)
          for (int k = 0; k < (bs >> FHT_LOG); ++k) items.push_back(RhtItem{r.layer, b, t, 1, k});
        max_elems = std::max(max_elems, 1 << FHT_LOG);
        continue;
      }
      const int tt = rht_tile_tokens(bs, r.batch, blocks, sm_count);
      for (int t0 = 0; t0 < r.batch; t0 += tt) {
        const int nt = std::min(tt, r.batch - t0);
        items.push_back(RhtItem{r.layer, b, t0, nt, -1});
        max_elems = std::max(max_elems, nt * bs);
      }
    }
}

constexpr int TICKET_SETS = 64;                  // sets allocated at a time
// Another TICKET_SETS sets.  `running`: for a run, which may be under capture (a stream of its own clears them; making one takes
// 0.2 ms, which a new plan does not pay).
static int add_ticket_sets(GlqbPlan* P, bool running) {
  const size_t n = P->n_tickets, bytes = n * TICKET_SETS * sizeof(int);
  int* p = nullptr;
  cudaStream_t st = nullptr;
  cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed;
  if (running) CUDA_TRY(cudaThreadExchangeStreamCaptureMode(&mode));
  cudaError_t e = cudaMalloc(&p, bytes);
  if (e == cudaSuccess) P->ticket_chunks.push_back(p);
  if (e == cudaSuccess && running) e = cudaStreamCreateWithFlags(&st, cudaStreamNonBlocking);
  if (e == cudaSuccess) e = running ? cudaMemsetAsync(p, 0, bytes, st) : cudaMemset(p, 0, bytes);
  if (e == cudaSuccess && running) e = cudaStreamSynchronize(st);
  if (st) cudaStreamDestroy(st);
  if (running) cudaThreadExchangeStreamCaptureMode(&mode);
  CUDA_TRY(e);
  for (int i = TICKET_SETS - 1; i >= 0; --i) P->free_tickets.push_back(p + i * n);
  return GLQB_OK;
}

// The tickets of a run in `workspace`.  A caller with ever new workspaces gets the sets of its earlier ones again, behind a
// device synchronisation; sets that a graph holds stay its own.
static int tickets_for(GlqbPlan* P, const void* workspace, cudaStream_t stream, int** out) {
  std::lock_guard<std::mutex> hold(P->ticket_mutex);
  cudaStreamCaptureStatus capture = cudaStreamCaptureStatusNone;
  CUDA_TRY(cudaStreamIsCapturing(stream, &capture));
  const bool captured = capture != cudaStreamCaptureStatusNone;
  for (GlqbPlan::TicketSet& t : P->ticket_sets)
    if (t.workspace == workspace) {
      t.captured = t.captured || captured;
      *out = t.tickets;
      return GLQB_OK;
    }
  if (P->free_tickets.empty() && !captured) {
    CUDA_TRY(cudaDeviceSynchronize());
    size_t kept = 0;
    for (const GlqbPlan::TicketSet& t : P->ticket_sets)
      if (t.captured) P->ticket_sets[kept++] = t;
      else P->free_tickets.push_back(t.tickets);
    P->ticket_sets.resize(kept);
  }
  if (P->free_tickets.empty()) {
    const int rc = add_ticket_sets(P, true);
    if (rc) return rc;
  }
  P->ticket_sets.push_back({workspace, P->free_tickets.back(), captured});
  P->free_tickets.pop_back();
  *out = P->ticket_sets.back().tickets;
  return GLQB_OK;
}

static int build_plan(GlqbPlan* P) {
  const int n = (int)P->descs.size();
  int dev_id = 0;
  CUDA_TRY(cudaGetDevice(&dev_id));
  CUDA_TRY(cudaDeviceGetAttribute(&P->sm_count, cudaDevAttrMultiProcessorCount, dev_id));

  // ---- segments: layers with the same kernel variant, in caller order inside a segment
  typedef std::tuple<int, int, int, int, int, int, int> Key;   // format, k1, k2, ns, nb, tn, two-phase
  const double tiles_min = trellis_two_phase_min_flops();
  auto by_flops = [&](const GlqbLinearDesc& d) { return 2.0 * d.batch * d.m_pad * d.n_pad >= tiles_min; };
  size_t trellis_tile_bytes = 0;
  for (const GlqbLinearDesc& d : P->descs)
    if (d.format == GLQB_FMT_TRELLIS_3INST && d.batch > DECODE_MAX_BATCH && by_flops(d)) trellis_tile_bytes += tile_bytes(d);
  auto trellis_tiles_once = [&](const GlqbLinearDesc& d) { return by_flops(d) && trellis_tile_bytes <= TRELLIS_TILES_MAX_BYTES; };
  std::map<Key, std::vector<int>> groups;
  std::vector<Key> key_order;
  for (int i = 0; i < n; ++i) {
    const GlqbLinearDesc& d = P->descs[i];
    Key k;
    const bool trellis = d.format == GLQB_FMT_TRELLIS_3INST;
    const bool tiles = d.batch > DECODE_MAX_BATCH && (trellis ? trellis_tiles_once(d) : d.batch >= e8_two_phase_min_tokens());
    const int tn = tn_for_batch(d.batch, trellis && !tiles && !trellis_two_stage_256(d));
    const int nb = tn ? 0 : nb_for_batch(d.batch);
    if (trellis)
      k = Key(d.format, d.bits[0], d.n_stages > 1 ? d.bits[1] : 0, d.n_stages, nb, tn, tiles ? 1 : 0);
    else
      k = Key(d.format, 0, 0, d.n_stages, nb, tn, tiles ? 1 : 0);
    if (!groups.count(k)) key_order.push_back(k);
    groups[k].push_back(i);
  }
  P->order.clear();
  P->segs.clear();
  for (const Key& k : key_order) {
    Segment s;
    s.format = std::get<0>(k); s.k1 = std::get<1>(k); s.k2 = std::get<2>(k);
    s.ns = std::get<3>(k); s.nb = std::get<4>(k); s.tn = std::get<5>(k); s.two_phase = std::get<6>(k);
    s.item_first = s.item_count = 0;
    s.first = (int)P->order.size();
    s.count = (int)groups[k].size();
    for (int i : groups[k]) P->order.push_back(i);
    if (s.tn ? !gemm_available(s) : !pick_kernel(s))
      return fail(GLQB_E_INVALID, "no kernel variant for format=%d K=%d+%d stages=%d token blocks=%d", s.format,
                  s.k1, s.k2, s.ns, s.nb);
    P->segs.push_back(s);
  }

  // ---- device table
  P->dev.assign(n, DevLinear());
  P->code_bytes = 0;
  P->flops = 0;
  P->max_batch = 1;
  for (int pos = 0; pos < n; ++pos) {
    const GlqbLinearDesc& d = P->descs[P->order[pos]];
    DevLinear& L = P->dev[pos];
    memset(&L, 0, sizeof L);
    for (int s = 0; s < GLQB_MAX_STAGES; ++s) {
      L.codes[s] = reinterpret_cast<const uint8_t*>(d.codes[s]);
      L.table[s] = d.table[s];
      L.table_entries[s] = d.table_entries[s];
      L.stage_scale[s] = d.stage_scale[s];
      L.bits[s] = d.bits[s];
    }
    L.su = reinterpret_cast<const __half*>(d.su);
    L.sv = reinterpret_cast<const __half*>(d.sv);
    L.row_scale = d.row_scale;
    L.wscale = d.wscale;
    L.format = d.format; L.m = d.m_pad; L.n = d.n_pad; L.in_f = d.in_features; L.out_f = d.out_features;
    L.n_stages = d.n_stages;
    L.batch = d.batch; L.x_dtype = d.x_dtype; L.y_dtype = d.y_dtype; L.stop_at_yrht = d.stop_at_yrht; L.x_is_rotated = d.x_is_rotated;
    L.x_stride = d.x_stride; L.y_stride = d.y_stride; L.x_off = d.x_offset; L.y_off = d.y_offset;
    L.in_norm_w = d.in_norm_weight; L.in_norm_dtype = d.in_norm_dtype; L.in_norm_eps = d.in_norm_eps;
    L.in_gated_act = d.in_gated_act; L.y_accumulate = d.y_accumulate;
    L.nbn = d.n_blocks_n; L.nbm = d.n_blocks_m;
    int off = 0;
    for (int i = 0; i < d.n_blocks_n; ++i) {
      L.bn_off[i] = off; L.bn_log[i] = ilog2(d.blocks_n[i]); off += d.blocks_n[i];
    }
    off = 0;
    for (int i = 0; i < d.n_blocks_m; ++i) {
      L.bm_off[i] = off; L.bm_log[i] = ilog2(d.blocks_m[i]); off += d.blocks_m[i];
    }
    if (d.format == GLQB_FMT_TRELLIS_3INST) {
      L.groups_per_strip = d.n_pad / 32;
      L.strips = d.m_pad / 32;
      for (int s = 0; s < d.n_stages; ++s) P->code_bytes += (int64_t)d.m_pad * d.n_pad * d.bits[s] / 8;
    } else {
      L.groups_per_strip = (d.n_pad + 255) / 256;
      L.strips = (d.m_pad + 15) / 16;
      P->code_bytes += (int64_t)d.n_stages * d.m_pad * (d.n_pad / 8) * 2;
    }
    P->flops += 2ll * d.batch * d.m_pad * d.n_pad;
    P->max_batch = std::max(P->max_batch, d.batch);
  }

  // ---- per segment: group prefix, range length per warp, grid
  P->gemm_items.clear();
  P->n_tickets = 0;
  for (Segment& s : P->segs) {
    if (!s.tn && s.nb == 1 && fused_enabled() && fused_available(s)) {
      // single-launch form: every layer of the segment reads the same input, at most 8 tokens, and the
      // activations plus the transform scratch fit in shared memory
      const GlqbLinearDesc& d0 = P->descs[P->order[s.first]];
      const bool e8 = s.format == GLQB_FMT_E8_SHELL;
      bool ok = !d0.x_is_rotated && d0.batch <= FUSED_MAX_TOKENS && s.count <= FUSED_MAX_LAYERS;
      {
        // The single-launch form is built for latency: strip-sized work units with a CTA-wide reduction each.  Large
        // launches are bound by streaming instead and keep the three-launch form (E8: with the resident table).
        static const long long max_bytes_trellis = [] { const char* e = getenv("GLQB_FUSED_MAX_BYTES"); return e ? atoll(e) : (1ll << 40); }();
        static const long long max_bytes_e8 = [] { const char* e = getenv("GLQB_FUSED_MAX_BYTES_E8"); return e ? atoll(e) : (16ll << 20); }();
        long long bytes = 0;
        for (int i = 0; i < s.count; ++i) bytes += layer_code_bytes(P->descs[P->order[s.first + i]]);
        ok = ok && bytes <= (e8 ? max_bytes_e8 : max_bytes_trellis);
      }
      for (int i = 1; i < s.count && ok; ++i) ok = same_input(d0, P->descs[P->order[s.first + i]]);
      if (!e8) ok = ok && d0.in_features == d0.n_pad;   // (trellis layers are never padded; the kernel's loads rely on it)
      // The transforms inside the kernel hold a warp's values at least (fht_fast: with fewer its shuffles would wait for lanes
      // that never come), and an output block holds whole strips: lists with blocks of less than 32 values take the other form.
      for (int i = 0; i < s.count && ok; ++i) {
        const GlqbLinearDesc& d = P->descs[P->order[s.first + i]];
        for (int b = 0; b < d.n_blocks_m; ++b) ok = ok && d.blocks_m[b] >= 32;
      }
      for (int b = 0; b < d0.n_blocks_n; ++b) ok = ok && d0.blocks_n[b] >= 32;
      // wide inputs are transformed once by rht_in_kernel (every CTA recomputing them would cost more than
      // the extra launch); so is a fused RMSNorm whose output block is too long for the in-kernel transform
      static const int in_max_n = [] { const char* e = getenv("GLQB_FUSED_IN_MAX_N"); return e ? atoi(e) : 4096; }();
      bool xr_global = d0.n_pad > in_max_n;
      for (int i = 0; i < d0.n_blocks_n; ++i) xr_global = xr_global || d0.blocks_n[i] > (1 << fused_in_max_log(e8));
      // Output blocks of at least 2^out_split_log rows are left to rht_out_kernel; shorter
      // ones are transformed inside the decode kernel by the CTA that completes them.  Measured on B200 (decoder
      // chain, SmolLM3-3B shapes): an extra launch costs more than the 8192-row transform it takes out of the
      // kernel's tail (101 vs 90 us per layer), so only blocks beyond 8192 rows are split off.
      static const int out_split_log = [] {
        const char* e = getenv("GLQB_FUSED_OUT_SPLIT_LOG");
        return std::max(12, std::min(e ? atoi(e) : FUSED_OUT_MAX_LOG + 1, FUSED_OUT_MAX_LOG + 1));
      }();
      static const int cta_factor = [] { const char* e = getenv("GLQB_FUSED_CTA_FACTOR"); return e ? std::max(1, atoi(e)) : 1; }();
      int scratch = 32;
      for (int i = 0; i < s.count && ok; ++i) {
        const GlqbLinearDesc& d = P->descs[P->order[s.first + i]];
        for (int b = 0; b < d.n_blocks_m; ++b)           // longer output blocks are left to rht_out_kernel
          if (d.blocks_m[b] < (1 << out_split_log)) scratch = std::max(scratch, d.blocks_m[b]);
      }
      if (!xr_global)
        for (int i = 0; i < d0.n_blocks_n; ++i) scratch = std::max(scratch, d0.blocks_n[i]);
      size_t smem = fused_smem_bytes(d0.n_pad, d0.batch, scratch, e8);
      size_t smem_limit = FUSED_SMEM_LIMIT;
      s.res_entries = 0;
      if (ok && e8 && smem <= FUSED_SMEM_LIMIT) {
        // E8 launches of a few MB and more keep as much of the codebook in shared memory as fits beside the
        // activations (one CTA per SM): otherwise every SM pulls most of the table through L2, one 32-byte sector
        // per gather
        const char* res_env = getenv("GLQB_E8_FUSED_RES_MIN_BYTES");          // (read per plan: the tests switch it)
        const long long res_min = res_env ? atoll(res_env) : (3ll << 20);
        long long bytes = 0;
        const uint32_t* big = nullptr;
        const uint32_t* small = nullptr;
        int small_n = 0;
        if (e8_uniform_tables(P->dev, s, &big, &small, &small_n, &bytes) && bytes >= res_min) {
          const size_t room = FUSED_SMEM_MAX > smem + 1024 ? FUSED_SMEM_MAX - smem - 1024 : 0;
          const int res = (int)std::min<size_t>(65536, room / 4 / 1024 * 1024);
          if (res >= 32768) {
            s.res_entries = res;
            s.big_table = big;
            s.small_table = small ? small : big;
            s.small_entries = small_n;
            smem += (size_t)res * 4 + 1024;
            smem_limit = FUSED_SMEM_MAX;
          }
        }
      }
      if (ok && smem <= smem_limit) {
        int resident = 0;
        CUDA_TRY(fused_prepare(s, smem_limit, smem, &resident));
        if (resident > 0) {
          // column groups per warp and unit: fewer for small layers, so that every SM gets work
          auto units_for = [&](int gpw) {
            long long u = 0;
            for (int i = 0; i < s.count; ++i) {
              const DevLinear& L = P->dev[s.first + i];
              u += (long long)L.strips * ((L.groups_per_strip + MV_WARPS * gpw - 1) / (MV_WARPS * gpw));
            }
            return u;
          };
          // (every CTA repeats the input transform, so more CTAs than SMs only pays when there is more
          // streaming work than one CTA per SM can take)
          // (an E8 group is 256 columns, a trellis group 32.)  No more groups per warp than keep all 8 warps of a
          // unit busy on the narrowest layer: a 4096-wide E8 layer has 16 groups per strip, two per warp.
          int gps_min = 1 << 30;
          for (int i = 0; i < s.count; ++i) gps_min = std::min(gps_min, P->dev[s.first + i].groups_per_strip);
          int gpw = std::min(e8 ? E8F_MAX_GPW : 8, std::max(1, (gps_min + MV_WARPS - 1) / MV_WARPS));
          while (gpw > (e8 ? 1 : 2) && units_for(gpw) < (long long)cta_factor * P->sm_count) gpw >>= 1;
          long long units = units_for(gpw);
          if (units < (1ll << 30)) {
            units = 0;
            for (int i = 0; i < s.count; ++i) {
              DevLinear& L = P->dev[s.first + i];
              const int kch = (L.groups_per_strip + MV_WARPS * gpw - 1) / (MV_WARPS * gpw);
              L.group_base = units;                       // first work unit of the layer
              L.fixed_slots = kch;
              L.slots = kch;
              L.per_warp = gpw;
              L.xr_global = xr_global ? 1 : 0;
              L.out_split_log = out_split_log;
              L.ticket_base = P->n_tickets;
              P->n_tickets += L.nbm;
              units += (long long)L.strips * kch;
            }
            s.fused = true;
            s.total_units = (int)units;
            s.scratch_elems = scratch;
            s.fused_smem = smem;
            s.grid = (int)std::min<long long>(units, (long long)P->sm_count * std::min(resident, 2));
            s.total_groups = 0;
            s.per_warp = 1;
            continue;
          }
        }
      }
    }
    if (s.tn) {
      for (int i = 0; i < s.count; ++i) {
        DevLinear& L = P->dev[s.first + i];
        L.gemm_tn = s.tn;
        L.gemm_even = trellis_form(s) ? 1 : 0;
        L.per_warp = 1;
        L.atile_off = s.two_phase ? -1 : 0;      // -1: allocate below
        P->max_batch_gemm = std::max(P->max_batch_gemm, L.batch);
      }
      gemm_schedule(s, P->max_batch, P->sm_count, P->dev, P->gemm_items);
      for (int i = 0; i < s.count; ++i) P->dev[s.first + i].slots = P->dev[s.first + i].fixed_slots;
      s.total_groups = 0;
      s.per_warp = 1;
      CUDA_TRY(gemm_prepare(s));
      if (s.two_phase && s.format == GLQB_FMT_E8_SHELL) {
        // tile decode with the codebook resident in shared memory
        long long bytes = 0;
        const uint32_t* big = nullptr;
        const uint32_t* small = nullptr;
        int small_n = 0;
        if (e8_uniform_tables(P->dev, s, &big, &small, &small_n, &bytes) && bytes >= e8_tiles_smem_min_bytes() &&
            tiles_smem_prepare(s.ns) == cudaSuccess) {
          s.smem_table = true;
          s.big_table = big;
          s.small_table = small ? small : big;
          s.small_entries = small_n;
        } else {
          cudaGetLastError();
        }
      }
      continue;
    }
    MvKernel kern = pick_kernel(s);
    int ctas_per_sm = 1;
    CUDA_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&ctas_per_sm, kern, MV_THREADS, 0));
    ctas_per_sm = std::max(1, std::min(ctas_per_sm, 4));
    long long warps_avail = (long long)P->sm_count * ctas_per_sm * MV_WARPS;
    int warps_per_cta = MV_WARPS;
    // E8: keep the codebook in shared memory when the launch is large enough to pay
    // for filling it and every stage reads either one shared 65,536-entry table or one small table
    if (s.format == GLQB_FMT_E8_SHELL && s.nb <= GLQB_E8_SMEM_MAX_NB && pick_e8_smem_kernel(s)) {
      long long bytes = 0;
      const uint32_t* big = nullptr;
      const uint32_t* small = nullptr;
      int small_n = 0;
      const bool ok = e8_uniform_tables(P->dev, s, &big, &small, &small_n, &bytes);
      if (ok && big && bytes >= e8_smem_min_bytes()) {
        E8SmemKernel ck = pick_e8_smem_kernel(s);
        CUDA_TRY(cudaFuncSetAttribute(ck, cudaFuncAttributeMaxDynamicSharedMemorySize, E8S_SMEM_BYTES));
        int resident = 0;
        if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&resident, ck, E8S_THREADS, E8S_SMEM_BYTES) == cudaSuccess &&
            resident > 0) {
          s.smem_table = true;
          s.big_table = big;
          s.small_table = small ? small : big;
          s.small_entries = small_n;
          warps_per_cta = E8S_THREADS / 32;
          warps_avail = (long long)P->sm_count * warps_per_cta;
        } else {
          cudaGetLastError();
        }
      }
    }
    if (s.format == GLQB_FMT_TRELLIS_3INST && s.nb == 1 && s.k2 == 0 && trellis_lut_kernel(s.k1)) {
      long long bytes = 0;
      for (int i = 0; i < s.count; ++i) bytes += (long long)P->dev[s.first + i].m * P->dev[s.first + i].n * s.k1 / 8;
      if (bytes >= trellis_lut_min_bytes() &&
          cudaFuncSetAttribute(trellis_lut_kernel(s.k1), cudaFuncAttributeMaxDynamicSharedMemorySize, MV_LUT_SMEM_BYTES) == cudaSuccess) {
        s.lut_table = true;
        warps_per_cta = MV_LUT_THREADS / 32;
        warps_avail = (long long)P->sm_count * warps_per_cta;
      } else {
        cudaGetLastError();
      }
    }
    long long total = 0;
    for (int i = 0; i < s.count; ++i) {
      DevLinear& L = P->dev[s.first + i];
      L.group_base = total;
      total += (long long)L.strips * L.groups_per_strip;
    }
    s.total_groups = total;
    const long long warps = warps_avail;
    long long per_warp = (total + warps - 1) / warps;
    if (per_warp < 1) per_warp = 1;
    s.per_warp = (int)per_warp;
    const long long used_warps = (total + per_warp - 1) / per_warp;
    s.grid = (int)((used_warps + warps_per_cta - 1) / warps_per_cta);
    for (int i = 0; i < s.count; ++i) {
      DevLinear& L = P->dev[s.first + i];
      L.per_warp = s.per_warp;
      L.slots = (L.groups_per_strip - 1) / s.per_warp + 2;
    }
  }

  // ---- the schedule of runs that need one token tile fewer (plans of one token count)
  std::vector<DevLinear> few;
  std::vector<GemmItem> few_items;
  P->few_tokens = 0;
  bool one_count = true, codes_in_gemm = false;
  for (const DevLinear& L : P->dev) { one_count = one_count && L.batch == P->max_batch; codes_in_gemm = codes_in_gemm || L.gemm_even; }
  const int tiles_most = (P->max_batch + TG_TN - 1) / TG_TN;
  if (one_count && codes_in_gemm && tiles_most > 1) {
    P->few_tokens = (tiles_most - 1) * TG_TN;
    P->few_segs = P->segs;
    few = P->dev;
    for (Segment& s : P->few_segs)
      if (s.tn) gemm_schedule(s, trellis_form(s) ? P->few_tokens : P->max_batch, P->sm_count, few, few_items);
    for (int pos = 0; pos < n; ++pos) P->dev[pos].slots = std::max(P->dev[pos].slots, few[pos].fixed_slots);
  }

  // ---- workspace: rotated activations (shared by layers with the same input) + partial sums
  size_t ws = 0;
  P->items_in.clear();
  P->items_in_gemm.clear();
  P->items_out.clear();
  std::vector<char> layer_fused(n, 0);
  for (const Segment& s : P->segs)
    if (s.fused)
      for (int i = 0; i < s.count; ++i) layer_fused[s.first + i] = 1;
  for (int pos = 0; pos < n; ++pos) {
    const GlqbLinearDesc& d = P->descs[P->order[pos]];
    // outside the single-launch form the input transform kernel applies the norm / activation (one token per
    // tile row, at most 8) and the output transform kernel the residual add: decode-sized layers only
    if (!layer_fused[pos] && (d.in_norm_weight || d.in_gated_act || d.y_accumulate) &&
        (d.batch > FUSED_MAX_TOKENS || P->dev[pos].gemm_tn))
      return fail(GLQB_E_INVALID,
                  "layer %d: the fused norm / activation / residual steps are served by the single-launch decode form only "
                  "(at most %d tokens, all layers of the call reading one input)", P->order[pos], FUSED_MAX_TOKENS);
  }
  std::vector<RhtLayer> rht_in, rht_in_gemm, rht_out;      // what the three transform launches of a run take
  for (int pos = 0; pos < n; ++pos) {
    DevLinear& L = P->dev[pos];
    const GlqbLinearDesc& d = P->descs[P->order[pos]];
    if (layer_fused[pos]) {                 // activations live in shared memory, transforms run inside the kernel
      ws = align_up(ws, 1024);
      L.xr_off = 0;
      if (L.xr_global) {                    // ... except wide inputs: transformed once into the workspace
        int first = pos;
        while (first > 0 && layer_fused[first - 1] && P->dev[first - 1].xr_global &&
               same_input(P->descs[P->order[first - 1]], d)) --first;
        if (first == pos) {
          L.xr_off = (long long)ws;
          ws = align_up(ws + (size_t)L.batch * L.n * sizeof(__half) * XR_TRELLIS_EXPAND, 1024);
          rht_in.push_back({pos, L.nbn, L.bn_log, L.batch, 0});
        } else {
          L.xr_off = P->dev[first].xr_off;
        }
      }
      L.part_off = (long long)ws;
      ws = align_up(ws + (size_t)L.slots * L.batch * L.m * sizeof(float), 256);
      L.rstd_off = (long long)ws;
      ws += 256;
      rht_out.push_back({pos, L.nbm, L.bm_log, L.batch, L.stop_at_yrht ? 64 : L.out_split_log});
      continue;
    }
    int same = -1;
    for (int q = 0; q < pos && same < 0; ++q) {
      if (layer_fused[q]) continue;
      const DevLinear& Q = P->dev[q];
      const GlqbLinearDesc& e = P->descs[P->order[q]];
      if (Q.format == L.format && Q.gemm_tn == L.gemm_tn && Q.gemm_even == L.gemm_even && Q.n == L.n && Q.in_f == L.in_f && Q.sv == L.sv &&
          Q.batch == L.batch &&
          Q.x_off == L.x_off && Q.x_stride == L.x_stride && Q.x_dtype == L.x_dtype && Q.nbn == L.nbn &&
          Q.x_is_rotated == L.x_is_rotated && Q.in_norm_w == L.in_norm_w && Q.in_norm_dtype == L.in_norm_dtype &&
          Q.in_norm_eps == L.in_norm_eps && Q.in_gated_act == L.in_gated_act &&
          memcmp(e.blocks_n, d.blocks_n, sizeof(int32_t) * d.n_blocks_n) == 0)
        same = q;
    }
    L.xr_global = 1;       // (three-launch form: a fused RMSNorm is complete in the transformed activations)
    if (same >= 0) {
      L.xr_off = P->dev[same].xr_off;
    } else {
      ws = align_up(ws, 1024);
      L.xr_off = (long long)ws;
      if (L.gemm_tn) {
        const size_t n_tiles = (L.batch + L.gemm_tn - 1) / L.gemm_tn, kchunks = (L.n + GM_TILE_K - 1) / GM_TILE_K;
        ws = align_up(ws + n_tiles * kchunks * L.gemm_tn * 128, 256);
        rht_in_gemm.push_back({pos, L.nbn, L.bn_log, L.batch, 0});
      } else {
        // E8 with several tokens interleaves groups of 8 tokens: round the token count up
        const size_t xr_tokens = (L.format == GLQB_FMT_E8_SHELL && L.batch > 1) ? (size_t)((L.batch + 7) / 8 * 8) : (size_t)L.batch;
        ws = align_up(ws + xr_tokens * L.n * sizeof(__half) *
                               (L.format == GLQB_FMT_TRELLIS_3INST ? XR_TRELLIS_EXPAND : 1), 256);
        rht_in.push_back({pos, L.nbn, L.bn_log, L.batch, 0});
      }
    }
    L.part_off = (long long)ws;
    ws = align_up(ws + (size_t)L.slots * L.batch * L.m * sizeof(float), 256);
    if (L.atile_off < 0) {
      ws = align_up(ws, 1024);
      L.atile_off = (long long)ws;
      ws += (size_t)((L.m + GM_TILE_M - 1) / GM_TILE_M) * ((L.n + GM_TILE_K - 1) / GM_TILE_K) * GM_A_BYTES;
    }
    rht_out.push_back({pos, L.nbm, L.bm_log, L.batch, 0});
  }
  add_rht_items(P->items_in, rht_in, P->sm_count, P->max_elems_in);
  add_rht_items(P->items_in_gemm, rht_in_gemm, P->sm_count, P->max_elems_in);
  add_rht_items(P->items_out, rht_out, P->sm_count, P->max_elems_out);
  // Launches of at most a tile per SM, without GEMM layers: the time of one tile counts, not the SMs' throughput.
  bool decode = true;
  for (const DevLinear& L : P->dev) decode = decode && L.gemm_tn == 0;
  // The GEMM works through the rows in rising order: the sums written last are still in L2 and are read first.  Rising / falling
  // order, whole calls: 2048 tokens of 11008 x 2048 149.1 / 146.0 us, of 14336 x 4096 (E8) 336.9 / 333.7; calls whose sums fit L2
  // anyway are the same (700 tokens of 5376 x 21504, three stages 299.9 / 299.6).
  if (!decode) std::reverse(P->items_out.begin(), P->items_out.end());
  // (inputs: only where norm or activation are computed on the way; plain loads of groups of four are the faster ones there)
  bool steps = false;
  for (const RhtItem& it : P->items_in) steps = steps || P->dev[it.layer].in_gated_act || P->dev[it.layer].in_norm_w;
  P->in_few = steps && P->items_in.size() <= (size_t)P->sm_count;
  P->out_few = decode && P->items_out.size() <= (size_t)P->sm_count;
  for (const RhtItem& it : P->items_out) P->out_few = P->out_few && !P->dev[it.layer].row_scale;
  P->ws_bytes = ws;
  P->out_wide = false;
  for (const DevLinear& L : P->dev) P->out_wide = P->out_wide || (long long)L.batch * L.m > 0xFFFFFFFFll;
  P->out_plain_static = true;
  for (const RhtItem& it : P->items_out) {
    const DevLinear& L = P->dev[it.layer];
    const int off = L.bm_off[it.block], bs = 1 << L.bm_log[it.block];
    P->out_plain_static = P->out_plain_static && !L.stop_at_yrht && ((L.m | off) & 3) == 0 && bs >= 4 && L.fixed_slots > 0 &&
                          it.sub < 0 && !L.row_scale && !L.y_accumulate && !(L.in_norm_w && !L.xr_global) && off + bs <= L.out_f;
  }

  // ---- upload
  if (P->few_tokens) {
    for (int pos = 0; pos < n; ++pos) {                    // the plan's buffers, the schedule's K splits
      const int slots = few[pos].fixed_slots;
      few[pos] = P->dev[pos];
      few[pos].fixed_slots = slots;
    }
    CUDA_TRY(cudaMalloc(&P->d_few_layers, sizeof(DevLinear) * n));
    CUDA_TRY(cudaMemcpy(P->d_few_layers, few.data(), sizeof(DevLinear) * n, cudaMemcpyHostToDevice));
    CUDA_TRY(cudaMalloc(&P->d_few_items, sizeof(GemmItem) * std::max<size_t>(1, few_items.size())));
    CUDA_TRY(cudaMemcpy(P->d_few_items, few_items.data(), sizeof(GemmItem) * few_items.size(), cudaMemcpyHostToDevice));
  }
  CUDA_TRY(cudaMalloc(&P->d_layers, sizeof(DevLinear) * n));
  CUDA_TRY(cudaMemcpy(P->d_layers, P->dev.data(), sizeof(DevLinear) * n, cudaMemcpyHostToDevice));
  CUDA_TRY(cudaMalloc(&P->d_items_in, sizeof(RhtItem) * std::max<size_t>(1, P->items_in.size())));
  CUDA_TRY(cudaMemcpy(P->d_items_in, P->items_in.data(), sizeof(RhtItem) * P->items_in.size(), cudaMemcpyHostToDevice));
  CUDA_TRY(cudaMalloc(&P->d_items_in_gemm, sizeof(RhtItem) * std::max<size_t>(1, P->items_in_gemm.size())));
  CUDA_TRY(cudaMemcpy(P->d_items_in_gemm, P->items_in_gemm.data(), sizeof(RhtItem) * P->items_in_gemm.size(),
                      cudaMemcpyHostToDevice));
  CUDA_TRY(cudaMalloc(&P->d_gemm_items, sizeof(GemmItem) * std::max<size_t>(1, P->gemm_items.size())));
  CUDA_TRY(cudaMemcpy(P->d_gemm_items, P->gemm_items.data(), sizeof(GemmItem) * P->gemm_items.size(),
                      cudaMemcpyHostToDevice));
  CUDA_TRY(cudaMalloc(&P->d_status, sizeof(int)));
  CUDA_TRY(cudaMemset(P->d_status, 0, sizeof(int)));
  if (P->n_tickets) {
    const int rc = add_ticket_sets(P, false);
    if (rc) return rc;
  }
  CUDA_TRY(cudaMalloc(&P->d_items_out, sizeof(RhtItem) * std::max<size_t>(1, P->items_out.size())));
  CUDA_TRY(cudaMemcpy(P->d_items_out, P->items_out.data(), sizeof(RhtItem) * P->items_out.size(), cudaMemcpyHostToDevice));
  return GLQB_OK;
}


}  // namespace glqb

// =============================================================================================
// exported C ABI
// =============================================================================================
extern "C" {

const char* glqb_last_error(void) { return g_err.c_str(); }
const char* glqb_version(void) { return "glq_b200 0.1 (sm_100a)"; }

int glqb_trellis_kernel_supported(int32_t m, int32_t n) { return (m > 0 && n > 0 && m % 32 == 0 && n % 32 == 0) ? 1 : 0; }

int glqb_plan_create(const GlqbLinearDesc* descs, int32_t count, GlqbPlan** out_plan) {
  if (!descs || count < 1 || !out_plan) return fail(GLQB_E_INVALID, "plan_create: bad arguments");
  for (int i = 0; i < count; ++i) {
    int rc = validate(descs[i], i);
    if (rc) return rc;
  }
  GlqbPlan* P = new GlqbPlan();
  P->descs.assign(descs, descs + count);
  // (a stream that is being captured must not keep another layout of the same call from getting its plan)
  cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed;
  cudaThreadExchangeStreamCaptureMode(&mode);
  int rc = build_plan(P);
  cudaThreadExchangeStreamCaptureMode(&mode);
  if (rc) {
    glqb_plan_destroy(P);
    return rc;
  }
  *out_plan = P;
  return GLQB_OK;
}

size_t glqb_plan_workspace_bytes(const GlqbPlan* plan) { return plan ? plan->ws_bytes : 0; }
int64_t glqb_plan_code_bytes(const GlqbPlan* plan) { return plan ? plan->code_bytes : 0; }
int64_t glqb_plan_flops(const GlqbPlan* plan) { return plan ? plan->flops : 0; }
int32_t glqb_plan_launches(const GlqbPlan* plan) {
  if (!plan) return 0;
  int n = (plan->items_in.empty() ? 0 : 1) + (plan->items_in_gemm.empty() ? 0 : 1) + (int)plan->segs.size() +
          (plan->items_out.empty() ? 0 : 1);
  for (const Segment& s : plan->segs) n += s.two_phase;
  return n;
}

int glqb_plan_set_timing(GlqbPlan* plan, int32_t enable) {
  if (!plan) return fail(GLQB_E_INVALID, "null plan");
  plan->timing = enable != 0;
  plan->ev_used = 0;
  return GLQB_OK;
}

int glqb_plan_kernel_ms(GlqbPlan* plan, double* total_ms_out, int32_t* runs_out) {
  if (!plan || !total_ms_out || !runs_out) return fail(GLQB_E_INVALID, "null argument");
  double total = 0.0;
  for (size_t i = 0; i + 1 < plan->ev_used; i += 2) {
    float ms = 0.f;
    CUDA_TRY(cudaEventSynchronize(plan->ev[i + 1]));
    CUDA_TRY(cudaEventElapsedTime(&ms, plan->ev[i], plan->ev[i + 1]));
    total += ms;
  }
  *total_ms_out = total;
  *runs_out = (int32_t)(plan->ev_used / 2);
  return GLQB_OK;
}

int glqb_plan_run(GlqbPlan* P, const void* x_base, void* y_base, void* workspace, size_t workspace_bytes,
                  void* stream) {
  return glqb_plan_run_tokens(P, x_base, y_base, INT32_MAX, workspace, workspace_bytes, stream);
}

int glqb_plan_run_tokens(GlqbPlan* P, const void* x_base, void* y_base, int32_t tokens, void* workspace,
                         size_t workspace_bytes, void* stream_) {
  if (!P || !x_base || !y_base) return fail(GLQB_E_INVALID, "plan_run: null argument");
  if (tokens < 1) return fail(GLQB_E_INVALID, "plan_run: %d tokens", tokens);
  for (const Segment& s : P->segs)
    if (s.fused && tokens < P->dev[s.first].batch)
      return fail(GLQB_E_INVALID, "plan_run: a plan of the single-launch form takes its %d tokens, not %d", P->dev[s.first].batch, tokens);
  const bool few = tokens <= P->few_tokens;
  const std::vector<Segment>& segs = few ? P->few_segs : P->segs;
  const DevLinear* d_layers = few ? P->d_few_layers : P->d_layers;
  const GemmItem* d_gemm_items = few ? P->d_few_items : P->d_gemm_items;
  if (P->ws_bytes && (!workspace || workspace_bytes < P->ws_bytes))
    return fail(GLQB_E_WORKSPACE, "workspace of %zu bytes needed, %zu given", P->ws_bytes, workspace_bytes);
  if (reinterpret_cast<uintptr_t>(workspace) & 255)
    return fail(GLQB_E_WORKSPACE, "workspace must be 256-byte aligned");
  cudaStream_t stream = reinterpret_cast<cudaStream_t>(stream_);
  uint8_t* ws = reinterpret_cast<uint8_t*>(workspace);
  int* tickets = nullptr;
  if (P->n_tickets) {
    const int rc = tickets_for(P, workspace, stream, &tickets);
    if (rc) return rc;
  }
  if (!P->items_in.empty()) {
    launch_chained(true, P->in_few ? rht_in_wide_kernel : rht_in_kernel<false>, (int)P->items_in.size(), P->in_few ? FHT_WIDE_THREADS : RHT_THREADS,
                   rht_smem(P->max_elems_in), stream, d_layers, P->d_items_in, reinterpret_cast<const uint8_t*>(x_base), ws, tokens);
  }
  if (!P->items_in_gemm.empty()) {
    launch_chained(true, rht_in_gemm_kernel, (int)P->items_in_gemm.size(), RHT_THREADS, rht_smem(P->max_elems_in), stream, d_layers,
                   P->d_items_in_gemm, reinterpret_cast<const uint8_t*>(x_base), ws, tokens);
  }
  if (P->timing) {
    while (P->ev.size() < P->ev_used + 2) {
      cudaEvent_t e;
      CUDA_TRY(cudaEventCreate(&e));
      P->ev.push_back(e);
    }
    CUDA_TRY(cudaEventRecord(P->ev[P->ev_used], stream));
  }
  for (const Segment& s : segs) {
    if (s.fused) {
      fused_launch(s, P->dev.data() + s.first, reinterpret_cast<const uint8_t*>(x_base), reinterpret_cast<uint8_t*>(y_base),
                   ws, tickets, P->comm ? comm_dev(P->comm) : nullptr, stream);
    } else if (s.tn) {
      gemm_launch(s, d_layers, d_gemm_items + s.item_first, ws, P->d_status, P->sm_count, tokens, stream);
    } else if (s.smem_table) {
      launch_chained(true, pick_e8_smem_kernel(s), s.grid, E8S_THREADS, E8S_SMEM_BYTES, stream, d_layers + s.first, s.count, s.total_groups,
                     s.per_warp, ws, s.big_table, s.small_table, s.small_entries, tokens);
    } else if (s.lut_table) {
      trellis_lut_kernel(s.k1)<<<s.grid, MV_LUT_THREADS, MV_LUT_SMEM_BYTES, stream>>>(d_layers + s.first, s.count, s.total_groups,
                                                                                     s.per_warp, ws, tokens);
    } else {
      pick_kernel(s)<<<s.grid, MV_THREADS, 0, stream>>>(d_layers + s.first, s.count, s.total_groups, s.per_warp, ws, tokens);
    }
  }
  if (P->timing) {
    CUDA_TRY(cudaEventRecord(P->ev[P->ev_used + 1], stream));
    P->ev_used += 2;
  }
  if (!P->items_out.empty()) {
    const int n_items = (int)P->items_out.size();
    uint8_t* yb = reinterpret_cast<uint8_t*>(y_base);
    if (P->out_few) {
      CUDA_TRY(launch_chained(true, rht_out_wide_kernel, n_items, FHT_WIDE_THREADS, rht_smem(P->max_elems_out), stream, d_layers,
                              P->d_items_out, ws, yb, tokens));
    } else if (out_plain(P, yb)) {
      CUDA_TRY(launch_chained(true, rht_out_plain_kernel, n_items, RHT_THREADS, rht_smem(P->max_elems_out), stream, d_layers, P->d_items_out, ws,
                              yb, tokens));
    } else {
      CUDA_TRY(launch_chained(true, P->out_wide ? rht_out_kernel<true> : rht_out_kernel<false>, n_items, RHT_THREADS,
                              rht_smem(P->max_elems_out), stream, d_layers, P->d_items_out, ws, yb, (const float*)nullptr, tokens));
    }
  }
  CUDA_TRY(cudaGetLastError());
  return GLQB_OK;
}

int glqb_plan_set_comm(GlqbPlan* P, GlqbComm* comm) {
  if (!P) return fail(GLQB_E_INVALID, "plan_set_comm: null plan");
  if (!comm) {
    for (DevLinear& L : P->dev) L.reduce = 0;
    P->comm = nullptr;
    return GLQB_OK;
  }
  const CommDev* C = comm_dev(comm);
  if (!C) return fail(GLQB_E_INVALID, "plan_set_comm: the communicator is not connected");
  // the sum runs where one CTA holds a whole output block: the single-launch form with every block inside the kernel
  if (!P->items_out.empty()) return fail(GLQB_E_INVALID, "plan_set_comm: the plan transforms outputs in a kernel of its own");
  long long floats = 0;
  int units = 0;
  for (const Segment& s : P->segs) {
    if (!s.fused)
      return fail(GLQB_E_INVALID, "plan_set_comm: only the single-launch decode form (trellis, at most %d tokens) sums over ranks",
                  FUSED_MAX_TOKENS);
    for (int i = s.first; i < s.first + s.count; ++i) {
      DevLinear& L = P->dev[i];
      if (L.stop_at_yrht) return fail(GLQB_E_INVALID, "plan_set_comm: layers that stop before the output transform have no sum");
      L.comm_off = (int)floats;
      L.comm_unit_base = units;
      floats += (long long)L.m * L.batch;
      units += L.nbm;
    }
    // every launch restarts at piece 0: launches of one stream follow one another, and areas alternate by epoch
    if (floats > C->max_floats || units > COMM_MAX_UNITS)
      return fail(GLQB_E_INVALID, "plan_set_comm: a launch exchanges %lld floats in %d pieces; the communicator holds %d and %d",
                  floats, units, C->max_floats, COMM_MAX_UNITS);
    floats = 0;
    units = 0;
  }
  for (DevLinear& L : P->dev) L.reduce = 1;
  P->comm = comm;
  return GLQB_OK;
}

int glqb_plan_status(GlqbPlan* plan, int32_t* status_out) {
  if (!plan || !status_out) return fail(GLQB_E_INVALID, "null argument");
  int v = 0;
  CUDA_TRY(cudaMemcpy(&v, plan->d_status, sizeof(int), cudaMemcpyDeviceToHost));
  *status_out = v;
  if (v) return fail(GLQB_E_DEVICE, "a kernel gave up waiting (status %d): results of that run are invalid", v);
  return GLQB_OK;
}

void glqb_plan_destroy(GlqbPlan* plan) {
  if (!plan) return;
  if (plan->d_layers) cudaFree(plan->d_layers);
  if (plan->d_few_layers) cudaFree(plan->d_few_layers);
  if (plan->d_few_items) cudaFree(plan->d_few_items);
  if (plan->d_items_in) cudaFree(plan->d_items_in);
  if (plan->d_items_out) cudaFree(plan->d_items_out);
  if (plan->d_items_in_gemm) cudaFree(plan->d_items_in_gemm);
  if (plan->d_gemm_items) cudaFree(plan->d_gemm_items);
  if (plan->d_status) cudaFree(plan->d_status);
  for (int* p : plan->ticket_chunks) cudaFree(p);
  for (cudaEvent_t e : plan->ev) cudaEventDestroy(e);
  delete plan;
}

int glqb_decompress_trellis_3inst(const void* packed, int32_t bits, const void* packed2, int32_t bits2,
                                  float inv_resid_scale2, int32_t m, int32_t n, void* out, int32_t out_dtype,
                                  void* stream_) {
  if (!packed || !out || m <= 0 || n <= 0 || m % 32 || n % 32)
    return fail(GLQB_E_INVALID, "decompress_trellis_3inst: needs m %% 32 == 0 and n %% 32 == 0 (got %d x %d)", m, n);
  if (bits < 1 || bits > 4) return fail(GLQB_E_INVALID, "decompress_trellis_3inst: K=%d unsupported (1..4)", bits);
  const int k2 = packed2 ? bits2 : 0;
  if (packed2 && (bits2 < 1 || bits2 > 4)) return fail(GLQB_E_INVALID, "decompress_trellis_3inst: K2=%d", bits2);
  if (out_dtype != GLQB_DT_F16 && out_dtype != GLQB_DT_F32) return fail(GLQB_E_INVALID, "out dtype");
  if (k2 && out_dtype != GLQB_DT_F32) return fail(GLQB_E_INVALID, "two-stage decode is written as fp32");
  cudaStream_t stream = reinterpret_cast<cudaStream_t>(stream_);
  const long long groups = (long long)(m / 32) * (n / 32);
  const int grid = (int)std::min<long long>((groups + MV_WARPS - 1) / MV_WARPS, 148 * 8);
  const uint8_t* p1 = reinterpret_cast<const uint8_t*>(packed);
  const uint8_t* p2 = reinterpret_cast<const uint8_t*>(packed2);
  const int f32 = out_dtype == GLQB_DT_F32;
#define D_CASE(A, B)                                                                                      \
  if (bits == A && k2 == B) {                                                                             \
    trellis_dump_kernel<A, B><<<grid, MV_THREADS, 0, stream>>>(p1, p2, inv_resid_scale2, m, n, out, f32); \
    CUDA_TRY(cudaGetLastError());                                                                         \
    return GLQB_OK;                                                                                       \
  }
#ifdef GLQB_FAST_BUILD   /* developer builds for kernel experiments: the 4-bit single-stage rate only */
  D_CASE(4, 0)
#else
  D_CASE(1, 0) D_CASE(2, 0) D_CASE(3, 0) D_CASE(4, 0)
  D_CASE(4, 1) D_CASE(4, 2) D_CASE(4, 3) D_CASE(4, 4)
#endif
#undef D_CASE
  return fail(GLQB_E_INVALID, "decompress_trellis_3inst: no kernel for K=%d+%d", bits, k2);
}

int glqb_dequant_e8(const void* const* qidxs, const uint32_t* const* tables, const int32_t* table_entries,
                    const float* stage_scale, int32_t n_stages, int32_t m, int32_t n, float* out, void* stream_) {
  if (!qidxs || !tables || !table_entries || !out || n_stages < 1 || n_stages > 4 || m <= 0 || n <= 0 || n % 8)
    return fail(GLQB_E_INVALID, "dequant_e8: bad arguments");
  E8DumpArgs A;
  memset(&A, 0, sizeof A);
  for (int s = 0; s < n_stages; ++s) {
    if (!qidxs[s] || !tables[s]) return fail(GLQB_E_INVALID, "dequant_e8: stage %d null", s);
    const int e = table_entries[s];
    if (e < 1 || e > 65536 || (e & (e - 1))) return fail(GLQB_E_INVALID, "dequant_e8: table entries %d", e);
    A.q[s] = reinterpret_cast<const uint16_t*>(qidxs[s]);
    A.table[s] = tables[s];
    A.entries[s] = e;
    A.scale[s] = (s && stage_scale) ? stage_scale[s] : 1.0f;
  }
  A.n_stages = n_stages; A.m = m; A.n = n;
  const long long total = (long long)m * (n / 8);
  const int grid = (int)std::min<long long>((total + 255) / 256, 148 * 16);
  e8_dump_kernel<<<grid, 256, 0, reinterpret_cast<cudaStream_t>(stream_)>>>(A, out);
  CUDA_TRY(cudaGetLastError());
  return GLQB_OK;
}

int glqb_e8_pack_table(const void* codebook_f16, int32_t entries, uint32_t* out_packed, void* stream_) {
  if (!codebook_f16 || !out_packed || entries < 1) return fail(GLQB_E_INVALID, "e8_pack_table: bad arguments");
  e8_pack_table_kernel<<<(entries + 255) / 256, 256, 0, reinterpret_cast<cudaStream_t>(stream_)>>>(
      reinterpret_cast<const __half*>(codebook_f16), entries, out_packed);
  CUDA_TRY(cudaGetLastError());
  return GLQB_OK;
}

// The unfused transform ops describe their one layer in kernel-parameter space (rht_in_single_kernel /
// rht_out_single_kernel): no device table, no allocation, no copy, nothing that would be illegal while the
// stream is being captured into a CUDA graph.  `offsets` (optional) gives the first column of every
// Hadamard block; without it the blocks are laid side by side.
static int run_rht_single(bool input, const void* src, int src_dtype, int64_t src_stride, const void* signs,
                          void* dst, int dst_dtype, int64_t dst_stride, int32_t feat, int32_t pad,
                          const int32_t* offsets, const int32_t* blocks, int32_t n_blocks, int32_t batch,
                          cudaStream_t stream) {
  if (!src || !signs || !dst || !blocks || n_blocks < 1 || n_blocks > GLQB_MAX_BLOCKS || batch < 1 || feat < 1 ||
      feat > pad)
    return fail(GLQB_E_INVALID, "rht: bad arguments (at most %d Hadamard blocks per call)", GLQB_MAX_BLOCKS);
  if (reinterpret_cast<uintptr_t>(signs) & 15) return fail(GLQB_E_INVALID, "rht: sign vector must be 16-byte aligned");
  DevLinear L;
  memset(&L, 0, sizeof L);
  RhtSingle S;
  memset(&S, 0, sizeof S);
  int off = 0, max_elems = 32, ctas = 0, dev_id = 0, sm_count = 0;
  CUDA_TRY(cudaGetDevice(&dev_id));
  CUDA_TRY(cudaDeviceGetAttribute(&sm_count, cudaDevAttrMultiProcessorCount, dev_id));
  for (int i = 0; i < n_blocks; ++i) {
    const int b = blocks[i];
    if (b < 1 || (b & (b - 1)) || b > 32768) return fail(GLQB_E_INVALID, "rht: block %d", b);
    const int o = offsets ? offsets[i] : off;
    if (o < 0 || o + b > pad) return fail(GLQB_E_INVALID, "rht: block %d at column %d exceeds %d columns", b, o, pad);
    if (input) { L.bn_off[i] = o; L.bn_log[i] = ilog2(b); } else { L.bm_off[i] = o; L.bm_log[i] = ilog2(b); }
    off += b;
    const int tt = rht_tile_tokens(b, batch, n_blocks, sm_count);
    S.first_cta[i] = ctas;
    S.tile_tokens[i] = tt;
    S.runs[i] = std::max(1, b >> FHT_LOG);
    ctas += (batch + tt - 1) / tt * S.runs[i];
    max_elems = std::max(max_elems, std::min(tt * b, 1 << FHT_LOG));
  }
  S.first_cta[n_blocks] = ctas;
  S.n_blocks = n_blocks;
  if (!offsets && off != pad) return fail(GLQB_E_INVALID, "rht: blocks sum to %d, expected %d", off, pad);
  L.format = GLQB_FMT_E8_SHELL;
  L.batch = batch;
  if (input) {
    L.n = pad; L.in_f = feat; L.sv = reinterpret_cast<const __half*>(signs);
    L.x_dtype = src_dtype; L.x_stride = src_stride; L.nbn = n_blocks; L.xr_off = 0;
  } else {
    L.m = pad; L.out_f = feat; L.su = reinterpret_cast<const __half*>(signs);
    L.y_dtype = dst_dtype; L.y_stride = dst_stride; L.nbm = n_blocks; L.wscale = 1.f;
  }
  const int smem = rht_smem(max_elems);
  if (input)
    rht_in_single_kernel<<<(unsigned)ctas, RHT_THREADS, smem, stream>>>(
        L, S, reinterpret_cast<const uint8_t*>(src), reinterpret_cast<uint8_t*>(dst));
  else
    rht_out_single_kernel<<<(unsigned)ctas, RHT_THREADS, smem, stream>>>(
        L, S, reinterpret_cast<uint8_t*>(dst), reinterpret_cast<const float*>(src));
  CUDA_TRY(cudaGetLastError());
  return GLQB_OK;
}

int glqb_input_rht(const void* x, int32_t x_dtype, int64_t x_stride, const void* sv, void* out_f32,
                   int32_t in_features, int32_t n_pad, const int32_t* blocks, int32_t n_blocks, int32_t batch,
                   void* stream) {
  return run_rht_single(true, x, x_dtype, x_stride, sv, out_f32, GLQB_DT_F32, n_pad, in_features, n_pad, nullptr,
                        blocks, n_blocks, batch, reinterpret_cast<cudaStream_t>(stream));
}

int glqb_output_rht(const float* y_rht, const void* su, void* out, int32_t out_dtype, int64_t out_stride,
                    int32_t out_features, int32_t m_pad, const int32_t* blocks, int32_t n_blocks, int32_t batch,
                    void* stream) {
  return run_rht_single(false, y_rht, GLQB_DT_F32, m_pad, su, out, out_dtype, out_stride, out_features, m_pad,
                        nullptr, blocks, n_blocks, batch, reinterpret_cast<cudaStream_t>(stream));
}

int glqb_output_rht_shards(const float* y_rht, const void* su, void* out, int32_t out_dtype, int64_t out_stride,
                           int32_t out_features, int32_t total_m, const int32_t* offsets, const int32_t* blocks,
                           int32_t n_blocks, int32_t batch, void* stream) {
  if (!offsets) return fail(GLQB_E_INVALID, "output_rht_shards: null offsets");
  return run_rht_single(false, y_rht, GLQB_DT_F32, total_m, su, out, out_dtype, out_stride, out_features, total_m,
                        offsets, blocks, n_blocks, batch, reinterpret_cast<cudaStream_t>(stream));
}

size_t glqb_linear_workspace_bytes(const GlqbLinearDesc* desc) {
  // Upper bound that does not depend on the device, with the roundings build_plan applies: activations
  // (E8 batches are padded to 8 tokens; the GEMM path stores whole token tiles of whole 64-column chunks),
  // the largest possible number of partial-sum slots (one per work group of a strip, plus one), and for
  // more than 128 tokens the decoded fp16 weight tiles.
  if (!desc) return 0;
  const size_t batch = (size_t)std::max(1, desc->batch);
  const int tn = tn_for_batch((int)batch, false);
  size_t ws = 1024;
  if (tn) {
    const size_t kchunks = ((size_t)desc->n_pad + GM_TILE_K - 1) / GM_TILE_K;
    const size_t tc = tn_for_batch((int)batch, true);       // either token tile may be the one: whole tiles of tn, or even ones
    const size_t rows = std::max((batch + tn - 1) / tn * tn, (batch + tc - 1) / tc * tc);
    ws += align_up(rows * kchunks * 128, 1024);
    ws += align_up(16 * batch * desc->m_pad * 4, 1024);                      // at most 16 K splits
    ws += align_up(tile_bytes(*desc), 1024) + 1024;                          // (the two-phase forms)
  } else {
    const size_t gps = desc->format == GLQB_FMT_TRELLIS_3INST ? desc->n_pad / 32 : (desc->n_pad + 255) / 256;
    ws += align_up(((batch + 7) / 8 * 8) * desc->n_pad * 2 * XR_TRELLIS_EXPAND, 1024);
    ws += align_up((gps + 1) * batch * desc->m_pad * 4, 1024);
  }
  return ws;
}

int glqb_fused_linear(const GlqbLinearDesc* desc, const void* x, void* y, void* workspace, size_t workspace_bytes,
                      void* stream) {
  // Stateless convenience form: builds a one-layer plan (which allocates its small device table), runs it,
  // waits for the stream and releases the plan.  It therefore synchronises and must not be called while the
  // stream is being captured; callers on a hot path keep a plan instead (glqb_plan_create once).
  GlqbPlan* P = nullptr;
  int rc = glqb_plan_create(desc, 1, &P);
  if (rc) return rc;
  rc = glqb_plan_run(P, x, y, workspace, workspace_bytes, stream);
  cudaError_t e = cudaStreamSynchronize(reinterpret_cast<cudaStream_t>(stream));
  glqb_plan_destroy(P);
  if (rc) return rc;
  if (e != cudaSuccess) return fail(GLQB_E_CUDA, "fused_linear: %s", cudaGetErrorString(e));
  return GLQB_OK;
}

}  // extern "C"
